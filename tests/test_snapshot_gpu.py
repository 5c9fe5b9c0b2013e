"""State downloads: exact round trips on both sides of the line between pinned
and device buffers (512 KiB: 8,192 bodies of an ensemble's state, 10,922 of
FP64 state, 16,384 of float4 state), with one and with several chunks of 8 MiB
(174,762 bodies of FP64 state), odd remainders, and single outputs."""
import ctypes

import numpy as np
import pytest

import nbody_gb300 as nb

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 63, 8191, 8193, 10922, 10923, 16384, 16385, 174763, 349527]


def _state(n):
    rng = np.random.default_rng(n)
    return (rng.normal(size=(n, 3)), rng.normal(size=(n, 3)),
            rng.uniform(0.5, 1.0, n).astype(np.float32))


@pytest.mark.parametrize("n", SIZES)
def test_system_round_trip(cuda, n):
    x, v, m = _state(n)
    s = nb.System(n, nb.INTEGRATOR_KDK64, 1e-2, 0.01, 1.0)
    s.set_state64(x, v, m)
    p, q = s.get_state64()
    assert np.array_equal(p, x) and np.array_equal(q, v)
    pm, vm = s.get_state()
    assert np.array_equal(pm, np.c_[x.astype(np.float32), m])
    assert np.array_equal(vm, np.c_[v.astype(np.float32), np.float32(1) / m])
    only = np.full((n, 3), np.nan)
    assert s.lib.nbgb_system_get_state64(
        s.h, None, only.ctypes.data_as(ctypes.POINTER(ctypes.c_double))) == 0
    assert np.array_equal(only, v)
    s.close()
    s = nb.System(n, nb.INTEGRATOR_REFERENCE, 1e-2, 0.01, 1.0)
    vm[:, 3] = v[:, 0]
    s.set_state(pm, vm)
    a, b = s.get_state()
    assert np.array_equal(a, pm) and np.array_equal(b, vm)
    s.close()


@pytest.mark.parametrize("n", SIZES)
def test_ensemble_round_trip(cuda, n):
    e = nb.Ensemble(n + 7, 2)
    first = e.add(*_state(7), 0.01, 0)
    x, v, m = _state(n)
    k = e.add(x, v, m, 0.01, 0)
    p, q, _ = e.get_state(k)
    assert np.array_equal(p, x) and np.array_equal(q, v)
    assert np.array_equal(e.get_state(first)[0], _state(7)[0])
    e.close()
