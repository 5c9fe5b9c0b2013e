"""Forces with each pair evaluated once (nbgb_force_newton3 at every N, the
default force at larger N) at the edges of its tiles, against FP64 and the
one-sided kernel: sets of 128 sources, rows of 512 targets (1,024
from N = 12,800 on), phases, and the forms for equal masses and
for positions far from the origin."""
import numpy as np
import pytest

from oracle import oracle as O

import nbody_gb300 as nb

pytestmark = pytest.mark.gpu

TOL_VS_FP64 = 5e-6   # the force gate of the other tests
ONE_SIDED = 25       # a one-sided configuration that takes masses of any sign


def _run(fn, pm, *args, **kw):
    import torch
    t = torch.from_numpy(np.ascontiguousarray(pm, np.float32)).cuda()
    out = fn(t, *args, **kw)
    torch.cuda.synchronize()
    return out.cpu().numpy()


def _err(out, pm, eps2, idx=None):
    f = O.ieee().forces_f64(pm, float(np.float32(eps2)), idx)
    o = out if idx is None else out[idx]
    assert np.all(o[:, 3] == 0)
    return (np.linalg.norm(o[:, :3] - f, axis=1) / np.linalg.norm(f, axis=1)).max()


@pytest.mark.parametrize("n", [2, 63, 64, 65, 127, 128, 129, 511, 512, 513, 641, 1025, 4097, 14335,
                               14336, 14463, 14465, 15489, 12799, 12800, 12801, 13311, 13313, 23935, 24577])
def test_edges_of_sets_and_rows(cuda, n):
    pm, _ = nb.ic_uniform_ball(n, 40 + n, 1.0, 0.5, 1.5)
    out = _run(nb.force_newton3, pm, 1e-4)
    assert nb.last_status() == 0
    assert _err(out, pm, 1e-4) <= TOL_VS_FP64
    assert np.array_equal(out, _run(nb.force_newton3, pm, 1e-4))  # deterministic
    if nb.force_kind(n)[0] == "pairs":
        assert np.array_equal(_run(nb.force, pm, 1e-4), out)


def test_kinds_and_launches(cuda):
    for n in (1, 1000, 4864):  # few bodies: one launch
        assert nb.force_kind(n) == ("onesided", 1)
    for n in (4865, 16384):
        assert nb.force_kind(n) == ("pairs", 2)
    kind, launches = nb.force_kind(400000)  # several phases
    assert kind == "pairs" and launches > 2 and launches % 2 == 0


def test_phases_against_the_one_sided_kernel(cuda):
    """N = 400,001: reaction pieces beyond one phase's workspace, carried
    sums, a ragged last row and set."""
    n = 400001
    _, _, pm, _ = nb.ic_plummer(n, 12)
    out = _run(nb.force, pm, 1e-4)
    assert nb.last_status() == 0
    idx = np.unique(np.concatenate([np.random.default_rng(2).choice(n, 200, replace=False),
                                    [0, 1023, 1024, 1407, 1408, n - 130, n - 1]]))
    assert _err(out, pm, 1e-4, idx) <= TOL_VS_FP64
    one = _run(nb.force, pm, 1e-4, config=ONE_SIDED)
    d = np.linalg.norm(out - one, axis=1) / np.linalg.norm(one, axis=1)
    assert d.max() <= TOL_VS_FP64


def _mass_case(case, n):
    pm, _ = nb.ic_uniform_ball(n, 5, 1.0, 0.5, 1.5)
    pm = pm.copy()
    if case == "equal":
        pm[:, 3] = np.float32(1.0 / n)
    elif case == "equal but one":  # one warp's targets and one set stay mixed
        pm[:, 3] = np.float32(1.0 / n)
        pm[2000, 3] *= 3
    elif case == "zeros":
        pm[::3, 3] = 0
    elif case == "equal in sets":  # each set of 128 equal, sets differ
        pm[:, 3] = (np.float32(1.0 / n) *
                    (1 + (np.arange(n) // 128) % 5)).astype(np.float32)
    elif case == "signed":
        pm[::7, 3] *= -1
    return pm


@pytest.mark.parametrize("case", ["equal", "equal but one", "zeros", "equal in sets", "signed"])
def test_mass_forms(cuda, case):
    n = 6500
    pm = _mass_case(case, n)
    out = _run(nb.force_newton3, pm, 1e-4)
    assert nb.last_status() == 0
    f = O.ieee().forces_f64(pm, float(np.float32(1e-4)))
    scale = np.linalg.norm(O.ieee().forces_f64(np.abs(pm), float(np.float32(1e-4))), axis=1)
    # signed masses cancel: errors relative to the unsigned system's forces
    ref = np.maximum(np.linalg.norm(f, axis=1), scale if case == "signed" else 0)
    assert (np.linalg.norm(out[:, :3] - f, axis=1) / ref).max() <= TOL_VS_FP64


@pytest.mark.parametrize("where", ["all", "some", "tiny"])
def test_far_positions_keep_the_one_sided_range(cuda, where):
    """Beyond 2^40 from the origin (or eps2 below 2^-80) (|d|^2+eps2)^-3/2
    alone leaves the binary32 range while m times it does not."""
    n = 6300
    pm, _ = nb.ic_uniform_ball(n, 6, 1.0, 0.5, 1.5)
    pm = pm.copy()
    k, eps2 = {"all": (43, 1e-4 * 2.0 ** 86), "some": (43, 1e-4), "tiny": (-45, 1e-4 * 2.0 ** -90)}[
        where]
    sel = slice(None) if where != "some" else slice(1000, 4000)
    pm[sel, :3] *= np.float32(2.0 ** k)
    pm[:, 3] *= np.float32(2.0 ** (60 if k > 0 else -60))
    out = _run(nb.force, pm, eps2)
    assert nb.force_kind(n)[0] == "pairs" and nb.last_status() == 0
    one = _run(nb.force, pm, eps2, config=ONE_SIDED)
    assert np.all(np.isfinite(out)) and np.any(one != 0)
    r = np.linalg.norm(one.astype(np.float64), axis=1)
    d = np.linalg.norm(out.astype(np.float64) - one, axis=1)
    assert np.all(d <= 2e-5 * r + 2e-5 * np.median(r) * (where == "some"))


@pytest.mark.parametrize("what,value", [("x", np.nan), ("x", np.inf), ("x", 1e20), ("m", np.inf)])
def test_special_values_as_the_one_sided_kernel(cuda, what, value):
    n = 6200
    pm, _ = nb.ic_uniform_ball(n, 7, 1.0, 0.5, 1.5)
    pm = pm.copy()
    pm[4321, 0 if what == "x" else 3] = value
    out = _run(nb.force, pm, 1e-4)
    one = _run(nb.force, pm, 1e-4, config=ONE_SIDED)
    nb.last_status()
    assert np.array_equal(np.isnan(out), np.isnan(one))
    assert np.array_equal(np.isinf(out), np.isinf(one))
    assert np.array_equal(np.sign(out[np.isinf(out)]), np.sign(one[np.isinf(one)]))


def test_negative_masses_stay_refused_by_the_stream_ordered_force(cuda):
    """As a log-domain plan: NaN forces and the status bit from nb.force; the
    drop-in evaluates again and takes any sign."""
    import torch
    n = 7000
    pm = _mass_case("signed", n)
    out = _run(nb.force, pm, 1e-4)
    assert nb.last_status() == 0x8 and np.all(np.isnan(out[:, :3]))
    t = torch.from_numpy(pm).cuda()
    f = torch.zeros_like(t)
    assert nb.ComputeGravitation_GPU_GB300(f, t, 1e-4, n) > 0.0
    assert nb.last_status() == 0
    assert np.array_equal(f.cpu().numpy(), _run(nb.force_newton3, pm, 1e-4))


@pytest.mark.parametrize("n", [6144, 9001])
def test_whole_row_slice_is_the_default_force(cuda, n):
    pm, _ = nb.ic_uniform_ball(n, 8, 1.0, 0.5, 1.5)
    assert np.array_equal(_run(nb.force_rows, pm, 1e-4, 0, n), _run(nb.force, pm, 1e-4))


def cancelling(n, row):
    """n bodies whose forces on the first `row` (massless, at the origin) are
    exact in every partial sum that keeps its remainder: sources at x = 2 and
    then at x = -2, eps2 lost in r^2 = 4, so every term is mass / 4, and masses
    of 16 bits that cancel but for one.  128 terms of a chain and the two
    halves of a fold fit 24 bits; a stretch's sum does not.  Returns posMass,
    eps2 and the exact force."""
    rng = np.random.default_rng(n)
    h = (n - row - 1) // 2
    k = rng.integers(1 << 15, 1 << 16, h)
    pm = np.zeros((n, 4), np.float32)
    pm[row:row + h, 0], pm[row:row + h, 3] = 2.0, k
    pm[row + h:row + 2 * h, 0], pm[row + h:row + 2 * h, 3] = -2.0, k[::-1]
    pm[row + 2 * h, 0], pm[row + 2 * h, 3] = 2.0, 12345.0
    pm[:, 3] *= 2.0 ** -16
    return pm, 1e-20, 12345.0 * 2.0 ** -18


@pytest.mark.parametrize("n", [8192, 12799, 16384, 40000, 300000])
def test_partial_sums_keep_their_remainders(cuda, n):
    pm, eps2, want = cancelling(n, 512 if n < 12800 else 1024)
    for fn in (nb.force, nb.force_newton3):
        out = _run(fn, pm, eps2)[:512]
        assert np.all(np.abs(out[:, 0] - want) <= 2.0 ** -23 * want), out[:, 0] - want
        assert np.all(out[:, 1:] == 0)


@pytest.mark.parametrize("n", [65537, 300001, 640003])
def test_phases_within_a_small_workspace(cuda, n):
    """The 32 MiB entry point: phases of at most 64 rows, down to one or two."""
    import torch
    _, _, pm, _ = nb.ic_plummer(n, 9)
    t = torch.from_numpy(pm).cuda()
    out = torch.full_like(t, float("nan"))
    assert nb.load().nbgb_force_static(out.data_ptr(), t.data_ptr(), 1e-4, n, 0) == 0
    torch.cuda.synchronize()
    assert nb.last_status() == 0 and bool(torch.isfinite(out).all())
    assert _err(out.cpu().numpy(), pm, 1e-4, np.arange(0, n, n // 300)) <= TOL_VS_FP64
