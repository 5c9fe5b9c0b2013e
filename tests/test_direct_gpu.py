"""The single-launch force of a few thousand bodies: at the edges of its
targets per CTA (multiples of 4 x 152), of pairs and of shares of the sources,
against FP64 sums, and its special cases against the one-sided kernel's."""
import numpy as np
import pytest

from oracle import oracle as O

import nbody_gb300 as nb

pytestmark = pytest.mark.gpu

ONE_SIDED = 25  # a one-sided configuration that takes masses of any sign


def _run(pm, eps2, **kw):
    import torch
    out = nb.force(torch.from_numpy(pm).cuda(), eps2, **kw)
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("n", [1, 2, 3, 15, 16, 17, 255, 257, 607, 608, 609, 1216, 1217, 1824,
                               1825, 2432, 2433, 3040, 3041, 3648, 3649, 4256, 4257, 4864])
def test_edges(cuda, n):
    pm, _ = nb.ic_uniform_ball(n, 80 + n, 1.0, 0.5, 1.5)
    assert nb.force_kind(n) == ("onesided", 1)
    out = _run(pm, 1e-4)
    assert nb.last_status() == 0 and np.all(out[:, 3] == 0)
    f = O.ieee().forces_f64(pm, float(np.float32(1e-4)))
    # every term is good to some 3 ulp; FP32 sums of up to 38 of them, then
    # compensated: a few 1e-7 of the terms' magnitudes
    d = np.linalg.norm(out[:, :3] - f, axis=1)
    mag = np.zeros(n)
    for i in range(n):
        r = pm[:, :3].astype(np.float64) - pm[i, :3]
        s = (r * r).sum(1) + 1e-4
        mag[i] = (pm[:, 3] * np.sqrt((r * r).sum(1)) * s ** -1.5).sum()
    assert np.all(d <= 6e-7 * mag)
    assert np.array_equal(out, _run(pm, 1e-4))  # deterministic


@pytest.mark.parametrize("n", [33, 1001, 4864])
def test_steps_are_force_then_integrate(cuda, n):
    import torch
    pm, vm = nb.ic_reference(n, 5)
    s = nb.System(n, nb.INTEGRATOR_REFERENCE, 0.01, 0.016, 0.95)
    s.set_state(pm, vm)
    s.step(3)
    p, v = torch.from_numpy(pm).cuda(), torch.from_numpy(vm).cuda()
    for _ in range(3):
        f = nb.force(p, 0.01)
        nb.integrate_reference(p, v, f, 0.016, 0.95)
    torch.cuda.synchronize()
    a, b = s.get_state()
    assert np.array_equal(a, p.cpu().numpy()) and np.array_equal(b, v.cpu().numpy())
    assert np.array_equal(s.get_force(), f.cpu().numpy())
    s.close()


def test_refuses_negative_masses(cuda):
    n = 1500
    pm, _ = nb.ic_uniform_ball(n, 6, 1.0, 0.5, 1.5)
    pm = pm.copy()
    pm[1024, 3] = -1.0  # a pair that a log-domain source stream would refuse
    out = _run(pm, 1e-4)
    assert nb.last_status() != 0 and np.all(np.isnan(out[:, :3]))


@pytest.mark.parametrize("what,value", [("x", np.nan), ("x", np.inf), ("x", 1e20), ("m", np.inf),
                                        ("m", 0.0)])
def test_special_values(cuda, what, value):
    n = 1500
    pm, _ = nb.ic_uniform_ball(n, 7, 1.0, 0.5, 1.5)
    pm = pm.copy()
    pm[777, 0 if what == "x" else 3] = value
    out, one = _run(pm, 1e-4), _run(pm, 1e-4, config=ONE_SIDED)
    assert np.array_equal(np.isfinite(out), np.isfinite(one))
    ok = np.isfinite(one)
    assert np.allclose(out[ok], one[ok], rtol=2e-5, atol=2e-6 * np.abs(one[ok]).max())


@pytest.mark.parametrize("n", [2, 64, 1000, 2432, 4864, 4865, 20000, 270000])
def test_in_place(cuda, n):
    """Forces written over the bodies they are computed from, as the one-sided
    kernel takes them: every body is read before the first force is written
    (at 270,000 bodies a phase's bodies before its forces)."""
    import torch
    pm, _ = nb.ic_uniform_ball(n, 7 + n, 1.0, 0.5, 1.5)
    want = nb.force_newton3(torch.from_numpy(pm).cuda(), 1e-4)
    both = torch.from_numpy(pm).cuda()
    nb.force(both, 1e-4, out=both)
    assert torch.equal(both, want)
    row = torch.from_numpy(pm).cuda()
    assert nb.ComputeGravitation_GPU_GB300(row, row, 1e-4, n) > 0.0
    assert torch.equal(row, want)
