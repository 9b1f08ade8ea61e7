"""Scenes from the sizes on at which the lattice and particle kernels launch two
and four times the resident CTAs (1M and 4M particles), one substep against the
f64 oracle."""
import numpy as np
import pytest

import oracle as O
from _gpu_util import gpu_sim, gpu_state, have_gpu, scale_rel

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA device")]

# one substep in f32 against f64, as in tests/test_gpu_parity.py
RTOL = 2e-5


@pytest.mark.parametrize("dim,n", [(2, 1_000_000), (2, 4_000_000), (3, 1_000_003)])
def test_large_scene(dim, n):
    rng = np.random.default_rng(n)
    coarsest = 1024 if dim == 2 else 64  # more blocks than one pass of the resident CTAs
    x = (0.05 + 0.9 * rng.random((n, dim))).astype(np.float32)
    v = rng.normal(0, 1, (n, dim)).astype(np.float32)
    F = np.tile(np.eye(dim, dtype=np.float32), (n, 1, 1))
    F += rng.normal(0, 0.02, F.shape).astype(np.float32)
    C = np.zeros((n, dim, dim), np.float32)
    m = np.ones(n, np.float32)
    g = np.where(x[:, 0] < 0.5, 1, 0).astype(np.int32)
    sim = gpu_sim(dim, 2, coarsest, n)
    o = O.Oracle(dim, 2, coarsest, n, f64=True)
    sim.set_particles(x=x, v=v, F=F, C=C, m=m, g=g)
    o.set_particles(x, v, F, C, m, g)
    sim.substep(1e-5)
    o.substep(1e-5)
    assert sim.errors() & ~2 == 0
    p, q = gpu_state(sim), o.particles()
    np.testing.assert_array_equal(p["fl"], q["fl"])
    for k in "xvFC":
        assert scale_rel(p[k], q[k]) <= RTOL, (k, scale_rel(p[k], q[k]))
    sim.close()
