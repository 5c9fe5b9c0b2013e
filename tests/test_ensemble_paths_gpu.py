"""The ensemble's other paths beside its default plan: the one-sided queue under
explicit bucket plans (alone, mixed with pair systems, joining and leaving,
sub-cycled), and systems too large for the scratch arena (one-sided, and block
pairs with Newton-3)."""
import numpy as np
import pytest

from oracle import oracle as O

import nbody_gb300 as nb

pytestmark = pytest.mark.gpu

TOL_VS_FP64 = 5e-6  # the force gate of the other ensemble tests
EPS2 = 1e-4
# plans of the queue for some buckets; the rest keep the default (pairs, tasks)
PLANS = {
    "all one-sided": {b: (1, 256, 2) for b in range(6, 14)},
    "some one-sided": {8: (0, 128, 1), 12: (3, 512, 3), 13: (1, 256, 4)},
}


def _ball(n, seed):
    pm, _ = nb.ic_uniform_ball(n, seed, 1.0, 0.5, 1.5)
    p = pm[:, :3].astype(np.float64)
    return p, 0.1 * p[:, ::-1].copy(), pm[:, 3].copy(), pm


def _errors(a, pm, idx):
    f = O.ieee().forces_f64(pm, float(np.float32(EPS2)), idx)
    return (np.linalg.norm(a[idx, :3] - f, axis=1) / np.linalg.norm(f, axis=1)).max()


def _run(members, plans, steps, join_at=(), sub=()):
    """Final states of members (bodies: steps differ by none), joining at the
    tick join_at says and leaving when finished."""
    join_at, sub = dict(join_at), dict(sub)
    e = nb.Ensemble(60000, 8, EPS2, tuning=None)
    for b, plan in plans.items():
        e.set_bucket_plan(b, *plan)
    slots, out, t, pending = {}, {}, 0, sorted(members)
    while pending or slots:
        for n in list(pending):
            if join_at.get(n, 0) <= t:
                p, v, m, _ = _ball(n, n)
                slots[n] = e.add(p, v, m, 0.002, steps)
                if n in sub:
                    e.set_substeps(slots[n], sub[n])
                pending.remove(n)
                kind = "queue" if nb.bucket_of(n) in plans else "default"
                assert (e.slot_info(slots[n])["variant"] >= 0) == (kind == "queue"), n
        e.tick(1)
        t += 1
        assert t < 60
        for s in e.finished():
            n = next(k for k, v in slots.items() if v == s)
            out[n] = e.get_state(s)
            e.remove(s)
            del slots[n]
    assert nb.last_status() == 0
    e.close()
    return out


@pytest.mark.parametrize("which", list(PLANS))
def test_queue_and_pairs_in_one_ensemble(cuda, which):
    plans, sizes, steps = PLANS[which], [300, 700, 1500, 4100, 9000], 8
    alone = {n: _run([n], plans, steps)[n] for n in sizes}
    mixed = _run(sizes, plans, steps, {300: 0, 700: 1, 1500: 2, 4100: 3, 9000: 12})
    fewer = _run(sizes, plans, steps, {}, {300: 4, 1500: 8, 4100: 3})
    for n in sizes:
        for a, b, c in zip(alone[n], mixed[n], fewer[n]):
            assert np.array_equal(a, b) and np.array_equal(a, c), n
        # the last accelerations are the forces at the last positions
        p, _, acc = alone[n]
        now = np.concatenate([p, _ball(n, n)[2][:, None]], 1).astype(np.float32)
        assert _errors(acc, now, np.arange(n)) <= TOL_VS_FP64, n


@pytest.mark.parametrize("newton3,n,kind", [(0, 262143, "pairs"), (0, 283008, "pairs"),
                                            (0, 283009, "onesided"), (4096, 401152, "pairs"),
                                            (4096, 401153, "blockpairs")])
def test_largest_systems(cuda, newton3, n, kind):
    """Around the scratch arena's limits, beside smaller systems: first forces
    of sampled bodies against FP64, then two steps against the small systems
    alone and, sampled, against the accelerations."""
    assert nb.ensemble_kind(n, newton3 > 0)[0] == kind
    small = [700, 5000]
    e = nb.Ensemble(n + sum(small), 3, EPS2, tuning=None)
    e.set_newton3_min(newton3)
    p, v, m, pm = _ball(n, 5)
    big = e.add(p, v, m, 0.002, 2)
    slots = {}
    for k in small:
        q = _ball(k, k)
        slots[k] = e.add(*q[:3], 0.002, 2)
    assert big is not None
    e.tick(1)
    e.synchronize()
    idx = np.arange(3, n, n // 300)
    a0 = e.get_state(big)[2]
    assert np.all(np.isfinite(a0)) and _errors(a0, pm, idx) <= TOL_VS_FP64
    e.tick(2)
    e.synchronize()
    assert sorted(e.finished()) == sorted([big, *slots.values()]) and nb.last_status() == 0
    p2, v2, a2 = e.get_state(big)
    now = np.concatenate([p2, m[:, None]], 1).astype(np.float32)
    assert _errors(a2, now, idx) <= TOL_VS_FP64
    # two kick-drift-kick steps: x moves by 2 dt v + 2 dt^2 a to second order
    d = p2 - p - 0.004 * v - 2 * 0.002 ** 2 * a0[:, :3]
    assert np.abs(d).max() <= 0.1 * 2 * 0.002 ** 2 * np.abs(a0[:, :3]).max()
    # v moves by dt (a0 + 2 a1 + a2) / 2, a1 between the two
    dv = (v2 - v) - 0.002 * (a0[:, :3].astype(np.float64) + a2[:, :3])
    assert np.abs(dv).max() <= 0.1 * 0.004 * np.abs(a0[:, :3]).max()
    state = {k: e.get_state(s) for k, s in slots.items()}
    e.close()
    for k in small:
        f = nb.Ensemble(k, 1, EPS2, tuning=None)
        f.set_newton3_min(newton3)
        s = f.add(*_ball(k, k)[:3], 0.002, 2)
        f.tick(3)
        f.synchronize()
        for x, y in zip(state[k], f.get_state(s)):
            assert np.array_equal(x, y), k
        f.close()
