"""Timed cases of the force, step-loop and ensemble entry points.

Every case is one call (or the few calls of one user step) through the
public Python entry points of nbody_gb300, on inputs made from a seed:

  force      nb.force(posMass, eps2): the stream-ordered force on a tensor
  row        nb.ComputeGravitation_GPU_GB300: the drop-in algorithm row
  newton3    nb.force_newton3
  slice      nb.force_rows: one rank's rows of a row-sharded evaluation
  loop       nb.force then nb.integrate_reference: a caller's own step loop
  reference  System with the reference integrator: state in, steps, state out
  kdk        System with the FP64 leapfrog: steps, then a snapshot (and the
             energies, when asked)
  ensemble   Ensemble: ticks of many systems, then every system's state

Sizes are the ones the benchmark, the studies, the serving stream and the
tests use, and ragged ones between them.
"""
import math
import random

import numpy as np
import torch

import nbody_gb300 as nb

# The reference driver's constants (softening 0.1, timestep 0.016, damping
# 0.95) for the reference integrator; the studies' for everything else.
REF_EPS2, REF_DT, REF_DAMPING = 0.01, 0.016, 0.95
EPS2 = 1e-4


def listed():
    return [
        # a small request's force on its own: launch and host latency
        {"name": "force_1000", "kind": "force", "bodies": "ball", "n": 1000},
        # the plain single system (uniform ball, masses 1/N)
        {"name": "force_16384", "kind": "force", "bodies": "equal_ball", "n": 16384},
        # a ragged mid-size evaluation
        {"name": "force_100003", "kind": "force", "bodies": "plummer", "n": 100003},
        # the plain large system, the headline workload
        {"name": "force_1048576", "kind": "force", "bodies": "plummer", "n": 1048576},
        # the drop-in row inside the reference driver (N a multiple of 1024,
        # its own bodies)
        {"name": "row_32768", "kind": "row", "bodies": "reference", "n": 32768},
        # the Newton's-third-law variant called by name
        {"name": "newton3_131072", "kind": "newton3", "bodies": "plummer", "n": 131072},
        # a caller's own loop at a small ragged size: force, then integrate
        {"name": "loop_10007", "kind": "loop", "bodies": "reference", "n": 10007},
        # the resident reference loop, one request: state in, 8 steps, out
        {"name": "reference_4096", "kind": "reference", "bodies": "reference", "n": 4096,
         "steps": 8},
        # the resident FP64 leapfrog at a serving size, 16 steps a snapshot
        {"name": "kdk_20000", "kind": "kdk", "bodies": "plummer", "n": 20000, "steps": 16,
         "dt": 0.005, "energies": False},
        # the precision study: leapfrog steps and an energy sample
        {"name": "kdk_262144_energies", "kind": "kdk", "bodies": "plummer", "n": 262144,
         "steps": 2, "dt": 0.002, "energies": True},
        # a batch of small systems of uneven size (the batched study's range)
        {"name": "ensemble_64_small", "kind": "ensemble", "bodies": "ball", "systems": 64,
         "n_lo": 64, "n_hi": 8192, "sizes": 4096, "steps": 20, "dt": 0.002, "newton3_min": 0},
        # the serving stream's main lane: few large systems, Newton-3 from 16,384
        {"name": "ensemble_8_large", "kind": "ensemble", "bodies": "plummer", "systems": 8,
         "n_lo": 8192, "n_hi": 65536, "sizes": 5, "steps": 4, "dt": 0.005,
         "newton3_min": 16384},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges (sizes log-uniform, mostly odd)."""
    kind = rng.choice(["force", "force", "row", "newton3", "slice", "loop", "reference", "kdk",
                       "ensemble"])
    if kind == "force":
        return {"kind": kind, "bodies": rng.choice(["ball", "equal_ball", "plummer"]),
                "n": _log_uniform(rng, 64, 600000)}
    if kind == "row":
        return {"kind": kind, "bodies": "reference", "n": 1024 * _log_uniform(rng, 1, 256)}
    if kind == "newton3":
        return {"kind": kind, "bodies": rng.choice(["ball", "plummer"]),
                "n": _log_uniform(rng, 1000, 400000)}
    if kind == "slice":
        n, world = _log_uniform(rng, 4096, 400000), rng.choice([2, 4, 8])
        rank, r = rng.randrange(world), -(-n // world)
        return {"kind": kind, "bodies": "plummer", "n": n, "begin": rank * r,
                "end": min(n, (rank + 1) * r)}
    if kind == "loop":
        return {"kind": kind, "bodies": "reference", "n": _log_uniform(rng, 256, 100000)}
    if kind == "reference":
        return {"kind": kind, "bodies": "reference", "n": _log_uniform(rng, 256, 65536),
                "steps": rng.randint(1, 5)}
    if kind == "kdk":
        n = _log_uniform(rng, 256, 200000)
        return {"kind": kind, "bodies": "plummer", "n": n,
                "steps": rng.randint(10, 24) if n < 40000 else rng.randint(1, 4), "dt": 0.002,
                "energies": rng.random() < 0.3}
    large = rng.random() < 0.4
    return {"kind": kind, "bodies": rng.choice(["ball", "plummer"]),
            "systems": rng.randint(3, 10) if large else rng.randint(16, 96),
            "n_lo": 4096 if large else 64, "n_hi": 65536 if large else 8192,
            "sizes": rng.randrange(1 << 20), "steps": rng.randint(3, 6) if large else
            rng.randint(8, 24), "dt": 0.005 if large else 0.002,
            "newton3_min": rng.choice([0, 16384]) if large else 0}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _directions(g, n):
    d = torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64)
    return d / d.norm(dim=1, keepdim=True)


def _bodies(what, n, seed):
    """(x, v, m): (n,3), (n,3), (n,) float64 CUDA tensors holding binary32
    values."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    u = torch.rand((n, 4), generator=g, device="cuda", dtype=torch.float64)
    if what == "plummer":  # scale radius 1, total mass 1, virial equilibrium
        r = (u[:, 0].clamp(1e-6, 0.999).pow(-2.0 / 3.0) - 1.0).rsqrt()
        x = _directions(g, n) * r[:, None]
        # speed / escape speed q has density q^2 (1 - q^2)^(7/2): q^2 is
        # Beta(3/2, 9/2), a ratio of sums of squared normals
        w = torch.randn((n, 12), generator=g, device="cuda", dtype=torch.float64).square()
        q = (w[:, :3].sum(1) / w.sum(1)).sqrt()
        v = _directions(g, n) * (q * math.sqrt(2.0) * (1.0 + r * r).pow(-0.25))[:, None]
        m = torch.full((n,), 1.0 / n, device="cuda", dtype=torch.float64)
    elif what == "reference":  # the reference driver's distribution
        scale = 0.9 * (n / 1024.0)
        x = _directions(g, n) * (scale * u[:, 0].pow(1.0 / 3.0))[:, None]
        v = _directions(g, n) * (0.9 * 8.0 * u[:, 1].pow(1.0 / 3.0))[:, None]
        m = 0.5 + 0.5 * u[:, 2]
    else:  # uniform ball of radius 1 at rest
        x = _directions(g, n) * u[:, 0].pow(1.0 / 3.0)[:, None]
        v = torch.zeros_like(x)
        m = torch.ones_like(u[:, 1]) if what == "equal_ball" else 0.5 + u[:, 1]
        m = m / n
    return tuple(t.float().double() for t in (x, v, m))


def _pm(x, m):
    return torch.cat([x, m[:, None]], 1).float().contiguous()


def _sizes(case):
    """The ensemble's system sizes: log-uniform, fixed by the case."""
    r = random.Random(case["sizes"])
    return [_log_uniform(r, case["n_lo"], case["n_hi"]) for _ in range(case["systems"])]


def _ensemble_bodies(case, seed):
    sizes = _sizes(case)
    if case["bodies"] == "plummer":
        return [_bodies("plummer", n, seed * 1009 + k) for k, n in enumerate(sizes)]
    x, v, m = _bodies("ball", sum(sizes), seed)
    at = np.cumsum([0] + sizes)
    # the ball's masses are 1/N of all bodies: each system's sum to about 1
    return [(x[a:b], v[a:b], (m[a:b] * (sum(sizes) / (b - a))).float().double())
            for a, b in zip(at[:-1], at[1:])]


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "ensemble":
        systems = [tuple(t.cpu().numpy() for t in b) for b in _ensemble_bodies(case, seed)]
        e = nb.Ensemble(sum(len(m) for _, _, m in systems), len(systems), EPS2)
        if case["newton3_min"]:
            e.set_newton3_min(case["newton3_min"])
        s["ens"] = e
        s["slots"] = [e.add(x, v, m.astype(np.float32), case["dt"], 1 << 40)
                      for x, v, m in systems]
        return s
    x, v, m = _bodies(case["bodies"], case["n"], seed)
    if kind in ("force", "row", "newton3", "slice"):
        s["pm"] = _pm(x, m)
        rows = case["end"] - case["begin"] if kind == "slice" else case["n"]
        s["out"] = torch.empty((rows, 4), device="cuda")
    elif kind == "loop":
        s["pm"], s["vel"] = _pm(x, m), _pm(v, 1.0 / m)
        s["out"] = torch.empty_like(s["pm"])
    elif kind == "reference":
        s["pm"], s["vel"] = _pm(x, m).cpu().numpy(), _pm(v, 1.0 / m).cpu().numpy()
        s["sys"] = nb.System(case["n"], nb.INTEGRATOR_REFERENCE, REF_EPS2, REF_DT, REF_DAMPING)
    elif kind == "kdk":
        s["sys"] = nb.System(case["n"], nb.INTEGRATOR_KDK64, EPS2, case["dt"], 1.0)
        s["sys"].set_state64(x.cpu().numpy(), v.cpu().numpy(), m.cpu().numpy())
    else:
        raise ValueError(kind)
    return s


def _eps2(case):
    return REF_EPS2 if case["bodies"] == "reference" else EPS2


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "force":
        return nb.force(s["pm"], _eps2(case), out=s["out"])
    if kind == "row":
        if not nb.ComputeGravitation_GPU_GB300(s["out"], s["pm"], _eps2(case), case["n"]) > 0.0:
            raise RuntimeError("the algorithm row failed")
        return s["out"]
    if kind == "newton3":
        return nb.force_newton3(s["pm"], _eps2(case), out=s["out"])
    if kind == "slice":
        return nb.force_rows(s["pm"], _eps2(case), case["begin"], case["end"], out=s["out"])
    if kind == "loop":
        nb.force(s["pm"], _eps2(case), out=s["out"])
        nb.integrate_reference(s["pm"], s["vel"], s["out"], REF_DT, REF_DAMPING)
        return {"force": s["out"], "pm": s["pm"], "vel": s["vel"]}
    if kind == "reference":
        s["sys"].set_state(s["pm"], s["vel"])
        s["sys"].step(case["steps"])
        pm, vel = s["sys"].get_state()
        return {"pm": pm, "vel": vel, "force": s["sys"].get_force()}
    if kind == "kdk":  # snapshots in the float4 arrays of the reference
        s["sys"].step(case["steps"])
        pm, vel = s["sys"].get_state()
        # velocities and inverse masses apart: 1/m = N would hide the former
        out = {"pm": pm, "v": vel[:, :3], "inv_mass": vel[:, 3]}
        if case["energies"]:
            d = s["sys"].diagnostics()
            out.update(kinetic=d["kinetic"], potential=d["potential"])
        return out
    s["ens"].tick(case["steps"])
    s["ens"].synchronize()
    got = [s["ens"].get_state(k) for k in s["slots"]]
    # snapshots in single precision, as the reference's float4 state
    return {"x": np.concatenate([p.astype(np.float32) for p, _, _ in got]),
            "v": np.concatenate([v.astype(np.float32) for _, v, _ in got]),
            "a": np.concatenate([a for _, _, a in got])}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """20 FLOP per interaction (N^2 a force pass, the reference's
    convention); inputs read once, outputs written once."""
    kind = case["kind"]
    if kind == "ensemble":
        sizes = _sizes(case)
        inter = float(sum(n * n for n in sizes)) * case["steps"]
        return {"bytes": sum(sizes) * (6 * 8 + 4 + 6 * 8 + 16.0), "flops": 20.0 * inter}
    n = float(case["n"])
    if kind in ("force", "row", "newton3"):
        return {"bytes": 32.0 * n, "flops": 20.0 * n * n}
    if kind == "slice":
        rows = case["end"] - case["begin"]
        return {"bytes": 16.0 * (n + rows), "flops": 20.0 * n * rows}
    if kind == "loop":
        return {"bytes": 80.0 * n, "flops": 20.0 * n * n}
    if kind == "reference":
        return {"bytes": 80.0 * n, "flops": 20.0 * n * n * case["steps"]}
    passes = case["steps"] + (1 if case["energies"] else 0)
    return {"bytes": (6 * 8 + 4 + 6 * 8 + 32.0) * n, "flops": 20.0 * n * n * passes}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _sum64(x, m, eps2, rows=None, potential=False):
    """sum_j m_j d_ij / (|d_ij|^2 + eps2)^(3/2) of the given rows (all), and
    -sum_{j != i} m_j / r_ij when asked."""
    eps2 = float(np.float32(eps2))
    n = x.shape[0]
    rows = slice(0, n) if rows is None else rows
    t = x[rows]
    xm = torch.cat([x, torch.ones_like(m[:, None])], 1) * m[:, None]
    force, phi = torch.empty_like(t), torch.empty_like(t[:, 0])
    step = max(1, min(t.shape[0], (1 << 23) // n))
    for a in range(0, t.shape[0], step):
        c = t[a:a + step]
        d2 = torch.full((c.shape[0], n), eps2, dtype=torch.float64, device=x.device)
        for k in range(3):
            d = c[:, k, None] - x[None, :, k]
            d2.addcmul_(d, d)
        inv = d2.rsqrt_()
        if potential:
            phi[a:a + step] = -(inv @ m)
        inv3 = (inv * inv).mul_(inv)
        s = inv3 @ xm
        force[a:a + step] = s[:, :3] - c * s[:, 3:]
    if potential:
        phi += m[rows] / math.sqrt(eps2)
    return force, phi


def _four(x, w):
    return torch.cat([x, w[:, None]], 1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        got = []
        for x, v, m in _ensemble_bodies(case, seed):
            f = _sum64(x, m, EPS2)[0]  # a system's first tick finds its accelerations
            for _ in range(case["steps"] - 1):
                v = v + f * (0.5 * case["dt"])
                x = x + v * case["dt"]
                f = _sum64(x, m, EPS2)[0]
                v = v + f * (0.5 * case["dt"])
            got.append((x, v, _four(f, torch.zeros_like(m))))
        return {k: torch.cat([g[i] for g in got]) for i, k in enumerate(("x", "v", "a"))}
    if case["n"] > 600000:
        return None
    x, v, m = _bodies(case["bodies"], case["n"], seed)
    eps2, zero = _eps2(case), torch.zeros_like(m)
    if kind in ("force", "row", "newton3"):
        return _four(_sum64(x, m, eps2)[0], zero)
    if kind == "slice":
        rows = slice(case["begin"], case["end"])
        return _four(_sum64(x, m, eps2, rows)[0], zero[rows])
    if kind in ("loop", "reference"):
        im = (1.0 / m).float().double()
        dt, damping = float(np.float32(REF_DT)), float(np.float32(REF_DAMPING))
        for _ in range(case.get("steps", 1)):
            f = _sum64(x, m, eps2)[0]
            v = (v + f * im[:, None] * dt) * damping
            x = x + v * dt
        return {"force": _four(f, zero), "pm": _four(x, m), "vel": _four(v, im)}
    dt = float(np.float32(case["dt"]))
    f = _sum64(x, m, eps2)[0]
    for k in range(case["steps"]):
        v = v + f * (0.5 * dt)
        x = x + v * dt
        f, phi = _sum64(x, m, eps2, potential=case["energies"] and k + 1 == case["steps"])
        v = v + f * (0.5 * dt)
    out = {"pm": _four(x, m), "v": v, "inv_mass": 1.0 / m}
    if case["energies"]:
        out.update(kinetic=float((0.5 * m * v.square().sum(1)).sum()),
                   potential=float((0.5 * m * phi).sum()))
    return out
