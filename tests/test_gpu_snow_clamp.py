"""The snow return map on both sides of its 3D rule (G2P projects states with
|F^T F - I| < 0.4, k_project the others), against the f64 oracle."""
import numpy as np
import pytest

import oracle as O
from _gpu_util import gpu_sim, gpu_state, have_gpu, scale_rel

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA device")]

# one substep in f32 against f64, as in tests/test_gpu_parity.py
RTOL = 2e-5


@pytest.mark.parametrize("spread", [0.002, 0.02, 0.12, 0.2])
@pytest.mark.parametrize("dim", [2, 3])
def test_one_substep(dim, spread):
    n = 3000
    rng = np.random.default_rng(int(spread * 1e4))
    x = (0.3 + 0.4 * rng.random((n, dim))).astype(np.float32)
    v = rng.normal(0, 1, (n, dim)).astype(np.float32)
    F = np.eye(dim) + np.clip(rng.normal(0, spread, (n, dim, dim)), -0.3, 0.3)
    F = F[np.linalg.det(F) > 0.2]
    F = np.resize(F, (n, dim, dim)).astype(np.float32)
    C = rng.normal(0, 0.1, (n, dim, dim)).astype(np.float32)
    m = rng.uniform(0.5, 2.0, n).astype(np.float32)
    g = np.zeros(n, np.int32)
    kw = dict(plasticity="snow", theta_c=2.5e-2, theta_s=7.5e-3, hardening=10.0)
    sim = gpu_sim(dim, 1, 16, n, **kw)
    o = O.Oracle(dim, 1, 16, n, f64=True, plasticity=1, theta_c=2.5e-2, theta_s=7.5e-3, hardening=10.0)
    sim.set_particles(x=x, v=v, F=F, C=C, m=m, g=g)
    o.set_particles(x, v, F, C, m, g)
    sim.substep(1e-5)
    o.substep(1e-5)
    assert sim.errors() == 0
    p, q = gpu_state(sim), o.particles()
    for k in ("x", "v", "F", "C", "Jp"):
        assert scale_rel(p[k], q[k]) <= RTOL, (k, scale_rel(p[k], q[k]))
    assert np.abs(q["Jp"] - 1).max() > 1e-3 or spread < 0.01
    sim.close()
