"""The ensemble's default plan (each pair once): edges of its sizes (warp tasks,
narrow and wide rows, sets of 128), against FP64, alone and mixed, with
sub-cycling, and systems whose scratch together exceeds the arena."""
import numpy as np
import pytest

from oracle import oracle as O

import nbody_gb300 as nb

pytestmark = pytest.mark.gpu

TOL_VS_FP64 = 5e-6  # the force gate of the other ensemble tests
EPS2 = 1e-4
SIZES = [1, 2, 127, 128, 129, 1023, 1024, 1025, 2047, 2048, 8191, 8192, 8193, 9857]


def _ball(n, seed):
    pm, _ = nb.ic_uniform_ball(n, seed, 1.0, 0.5, 1.5)
    p = pm[:, :3].astype(np.float64)
    return p, 0.1 * p[:, ::-1].copy(), pm[:, 3].copy(), pm


def _run(sizes, steps, sub=None):
    e = nb.Ensemble(sum(sizes), len(sizes), EPS2, tuning=None)
    slots = {}
    for n in sizes:
        p, v, m, _ = _ball(n, 900 + n)
        slots[n] = e.add(p, v, m, 0.002, steps)
        if sub:
            e.set_substeps(slots[n], sub[n % len(sub)])
    out, t = {}, 0
    while len(out) < len(sizes) and t < 4 + steps:
        e.tick(1)
        t += 1
        for s in e.finished():
            n = next(k for k, v in slots.items() if v == s)
            if n not in out:
                out[n] = e.get_state(s)
    assert nb.last_status() == 0
    e.close()
    return out


def test_first_forces_match_fp64_at_the_edges(cuda):
    e = nb.Ensemble(sum(SIZES), len(SIZES), EPS2, tuning=None)
    slots = {}
    for n in SIZES:
        p, v, m, _ = _ball(n, 900 + n)
        slots[n] = e.add(p, v, m, 0.01, 3)
    assert e.slot_info(slots[9857])["variant"] == -1
    e.tick(1)
    e.synchronize()
    for n in SIZES:
        p, v, _, pm = _ball(n, 900 + n)
        p1, v1, a = e.get_state(slots[n])
        assert np.array_equal(p1, p) and np.array_equal(v1, v)  # nothing moved yet
        f = O.ieee().forces_f64(pm, float(np.float32(EPS2)))
        if n == 1:
            assert np.all(a == 0)
            continue
        err = np.linalg.norm(a[:, :3] - f, axis=1) / np.linalg.norm(f, axis=1)
        assert err.max() <= TOL_VS_FP64, n
    e.close()


def test_alone_mixed_and_subcycled_are_bit_identical(cuda):
    sizes = [129, 700, 1024, 3000, 8193]
    mixed = _run(sizes, 6)
    sub = _run(sizes, 6, sub=[1, 4, 3])
    for n in sizes:
        alone = _run([n], 6)[n]
        for a, b, c in zip(alone, mixed[n], sub[n]):
            assert np.array_equal(a, b) and np.array_equal(a, c), n


def test_groups_beyond_the_scratch_arena(cuda):
    """Two systems of 200,000 bodies need more scratch than the arena has:
    evaluated one after the other, each as alone."""
    n = 200000
    e = nb.Ensemble(2 * n + 500, 3, EPS2, tuning=None)
    slots, pms = [], []
    for seed, k in ((1, n), (2, 500), (3, n)):
        p, v, m, pm = _ball(k, seed)
        slots.append(e.add(p, v, m, 0.01, 2))
        pms.append(pm)
    e.tick(1)
    e.synchronize()
    for s, pm in zip(slots, pms):
        _, _, a = e.get_state(s)
        idx = np.unique(np.random.default_rng(1).choice(len(pm), 200))
        f = O.ieee().forces_f64(pm, float(np.float32(EPS2)), idx)
        err = np.linalg.norm(a[idx, :3] - f, axis=1) / np.linalg.norm(f, axis=1)
        assert err.max() <= TOL_VS_FP64
    e.close()


@pytest.mark.parametrize("n", [1500, 20000, 70000])
def test_partial_sums_keep_their_remainders(cuda, n):
    from test_pair_gpu import cancelling
    pm, _, want = cancelling(n, 512 if n < 8192 else 1024)
    e = nb.Ensemble(n, 1, 1e-20, tuning=None)
    p = pm[:, :3].astype(np.float64)
    slot = e.add(p, np.zeros_like(p), pm[:, 3].copy(), 0.01, 3)
    e.tick(1)
    e.synchronize()
    a = e.get_state(slot)[2][:512]
    assert np.all(np.abs(a[:, 0] - want) <= 2.0 ** -23 * want), a[:, 0] - want
    assert np.all(a[:, 1:] == 0)
    e.close()


def test_warps_of_a_task_do_not_change_results(cuda):
    """One system's tiles are shared among four warps, those of hundreds taken
    by a warp or two each: the bits are the same (systems of 1 to 8 sets)."""
    sizes = [100, 200, 384, 500, 640, 768, 800, 1000]
    got = []
    for copies in (1, 200):
        e = nb.Ensemble(copies * sum(sizes), copies * len(sizes), EPS2, tuning=None)
        slots = {}
        for k in range(copies):
            for n in sizes:
                p, v, m, _ = _ball(n, 700 + n)
                slots[n, k] = e.add(p, v, m, 0.002, 6)
        e.tick(4)
        e.synchronize()
        got.append({n: e.get_state(slots[n, copies - 1]) for n in sizes})
        e.close()
    for n in sizes:
        for a, b in zip(got[0][n], got[1][n]):
            assert np.array_equal(a, b), n
