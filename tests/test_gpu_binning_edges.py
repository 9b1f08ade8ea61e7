"""The lattice phases with few warps for much work: a scene that gets a handful
of CTAs in a batch beside a large one has more touched blocks than warps (the
dilation walks a block's levels in one warp instead of one warp a level) and
more bins than one pass of k_bins' warps, against the f64 oracle; its stepping
alone, with the whole chip, takes the other branch."""
import numpy as np
import pytest

import oracle as O
from _gpu_util import LO, gpu_grid, gpu_sim, gpu_state, have_gpu, scale_rel

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA device")]

# one substep in f32 against f64, as in tests/test_gpu_parity.py
RTOL = 2e-5


@pytest.mark.parametrize("dim,coarsest,level,n", [(2, 128, 2, 3000), (2, 128, 1, 1), (3, 16, 2, 2500), (3, 32, 1, 5000)])
def test_scattered_particles_in_a_small_share(dim, coarsest, level, n):
    from agimp.batch import SceneBatch
    rng = np.random.default_rng(n)
    x = rng.random((n, dim)).astype(np.float32) * 0.9 + 0.05
    v = rng.normal(0, 1, (n, dim)).astype(np.float32)
    m = rng.uniform(0.5, 2.0, n).astype(np.float32)
    # levels by a slab of the domain, the finest below 0.45
    g = np.where(x[:, 0] < 0.45, level - 1, 0).astype(np.int32)
    F = np.tile(np.eye(dim, dtype=np.float32), (n, 1, 1)) + rng.normal(0, 0.05, (n, dim, dim)).astype(np.float32)
    C = rng.normal(0, 0.1, (n, dim, dim)).astype(np.float32)
    big = 400000
    xb = (0.3 + 0.3 * rng.random((big, dim))).astype(np.float32)
    o = O.Oracle(dim, level, coarsest, n, f64=True)
    o.set_particles(x, v, F, C, m, g)
    o.substep(1e-5)
    q = o.particles()
    for alone in (True, False):
        sim = gpu_sim(dim, level, coarsest, n)
        sim.set_particles(x=x, v=v, F=F, C=C, m=m, g=g)
        if alone:
            sim.substep(1e-5)
        else:
            other = gpu_sim(dim, 1, 32, big)
            other.set_particles(x=xb, v=np.zeros_like(xb), F=np.tile(np.eye(dim, dtype=np.float32), (big, 1, 1)),
                                C=np.zeros((big, dim, dim), np.float32), m=np.ones(big, np.float32),
                                g=np.zeros(big, np.int32))
            batch = SceneBatch([other, sim])
            batch.substep(1e-5)
        assert sim.errors() & ~2 == 0
        p = gpu_state(sim)
        np.testing.assert_array_equal(p["fl"], q["fl"])
        for l in range(level):
            np.testing.assert_array_equal(gpu_grid(sim, l)[2], o.grid(l, LO, (coarsest << l) + 12)[2])
        for k in "xvFC":
            assert scale_rel(p[k], q[k]) <= RTOL, (alone, k, scale_rel(p[k], q[k]))
        if not alone:
            batch.close()
            other.close()
        sim.close()
