"""The diagnostics' potential, each pair evaluated once: at the edges of sets
(128) and rows (1,024), with several stretches per row and with late stretches
(34,011), against FP64 sums."""
import numpy as np
import pytest

from oracle import oracle as O

import nbody_gb300 as nb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 127, 129, 1023, 1024, 1025, 2049, 7000, 20011, 34011])
@pytest.mark.parametrize("equal", [True, False])
def test_potential_energy(cuda, n, equal):
    rng = np.random.default_rng(n)
    pm = rng.uniform(-1, 1, (n, 4)).astype(np.float32)
    pm[:, 3] = 1.0 / n if equal else rng.uniform(0, 2.0 / n, n)
    s = nb.System(n, nb.INTEGRATOR_REFERENCE, 1e-3, 0.01, 1.0)
    s.set_state(pm, np.zeros((n, 4), np.float32))
    d = s.diagnostics()
    phi = O.ieee().potential_f64(pm, float(np.float32(1e-3)))
    m = pm[:, 3].astype(np.float64)
    pe = 0.5 * (m * phi).sum()
    # Terms of one sign: rsqrt and the FP32 folds give at most some 2^-20 a
    # body; the self pair, subtracted, is m / eps of the sums.
    self_terms = 0.5 * (m * m).sum() / np.sqrt(1e-3)
    assert abs(d["potential"] - pe) <= 2e-6 * (abs(pe) + self_terms)
    assert s.diagnostics()["potential"] == d["potential"]
    s.close()
