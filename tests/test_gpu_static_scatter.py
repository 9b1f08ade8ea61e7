"""Static scenes of scattered particles against the f64 oracle: the window of
cells looked up in the level map around every base cell (one word of recorded
base cells per block in 2D, five in 3D), with a warp per level and window (the
scene alone, more warps than touched blocks) and with all of them in one warp
(a small share of a batch)."""
import numpy as np
import pytest

import oracle as O
from _gpu_util import LO, gpu_grid, gpu_sim, gpu_state, have_gpu, scale_rel

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA device")]

# one substep in f32 against f64, as in tests/test_gpu_parity.py
RTOL = 2e-5


@pytest.mark.parametrize("dim,level,coarsest,n", [(3, 2, 16, 2500), (3, 3, 16, 4000), (3, 1, 16, 400), (2, 3, 64, 3000)])
def test_scattered_static_scene(dim, level, coarsest, n):
    from agimp import scenes
    from agimp.batch import SceneBatch
    from agimp.simulator import tabulate_level_map
    rng = np.random.default_rng(n + dim)
    # the whole domain to its edges, and one block full of particles
    x = 0.002 + 0.996 * rng.random((n, dim))
    x[: n // 8] = 0.5 + 4.0 / (coarsest << (level - 1)) * rng.random((n // 8, dim))
    x = x.astype(np.float32)
    v = rng.normal(0, 1, (n, dim)).astype(np.float32)
    m = rng.uniform(0.5, 2.0, n).astype(np.float32)
    F = np.tile(np.eye(dim, dtype=np.float32), (n, 1, 1)) + rng.normal(0, 0.05, (n, dim, dim)).astype(np.float32)
    C = rng.normal(0, 0.1, (n, dim, dim)).astype(np.float32)
    g = np.zeros(n, np.int32)
    box = (tuple([0.45] + [0.4] * (dim - 1)), tuple([0.6] * dim))
    table, H = tabulate_level_map(scenes.band_level_map([box], dim, level, coarsest), dim, level, coarsest)
    o = O.Oracle(dim, level, coarsest, n, f64=True)
    o.set_particles(x, v, F, C, m, g)
    o.set_level_map(table, H)
    o.substep(1e-5)
    q = o.particles()
    assert len(np.unique(q["fl"][q["fl"] >= 0])) == min(level, 3)
    big = 400000
    xb = (0.3 + 0.3 * rng.random((big, dim))).astype(np.float32)
    for alone in (True, False):
        sim = gpu_sim(dim, level, coarsest, n, table, H)
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
        assert sim.errors() == o.errors()
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
