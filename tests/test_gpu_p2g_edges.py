"""P2G's work items at their edges: cells holding one particle up to several
tasks' and items' worth, sparse and dense cells in one block, blocks at the
domain's edge, small and large scenes (their tasks differ in length), and a
radius below 1/2 (the general weights), against the f64 oracle."""
import numpy as np
import pytest

import oracle as O
from _gpu_util import gpu_grid, gpu_sim, gpu_state, have_gpu, scale_rel

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA device")]

# one substep in f32 against f64: sums of up to some hundred terms a node
# (tests/test_gpu_parity.py's one-substep bounds); 4e-4 of a node's sum of 1e5
# terms would be 1e5 eps / 2 if every rounding went the same way, and the
# observed order is its square root
RTOL = 2e-5


def _run(dim, x, coarsest, radius, level=1):
    n = len(x)
    rng = np.random.default_rng(n)
    v = rng.normal(0, 1, (n, dim)).astype(np.float32)
    F = (np.eye(dim) + rng.normal(0, 0.05, (n, dim, dim))).astype(np.float32)
    C = rng.normal(0, 0.1, (n, dim, dim)).astype(np.float32)
    m = rng.uniform(0.5, 2.0, n).astype(np.float32)
    g = np.full(n, level - 1, np.int32)
    sim = gpu_sim(dim, level, coarsest, n, radius=radius)
    o = O.Oracle(dim, level, coarsest, n, f64=True, radius=radius)
    sim.set_particles(x=x, v=v, F=F, C=C, m=m, g=g)
    o.set_particles(x, v, F, C, m, g)
    sim.substep(1e-5)
    o.substep(1e-5)
    assert sim.errors() == 0
    p, q = gpu_state(sim), o.particles()
    np.testing.assert_array_equal(p["fl"], q["fl"])
    mass = gpu_grid(sim, level - 1)[0]
    assert scale_rel(mass.sum(dtype=np.float64), m.sum(dtype=np.float64)) < 1e-5
    for k in "xvFC":
        assert scale_rel(p[k], q[k]) <= RTOL, (k, scale_rel(p[k], q[k]))
    sim.close()


@pytest.mark.parametrize("radius", [0.5, 0.3])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("counts", [(1,), (3, 4, 5), (8, 9, 7), (31, 32, 33), (39, 1, 40, 41), (79, 80, 81), (700,)])
def test_cells_of_given_counts(dim, counts, radius):
    """Cells at assorted places of a block (and of the next) with the given
    numbers of particles."""
    rng = np.random.default_rng(sum(counts))
    c = 16
    x = []
    for i, k in enumerate(counts):
        cell = np.array([4 + i % 3, 5 + 2 * i, 6 + (i * 3) % 5])[:dim]
        x.append((cell + 0.55 + 0.9 * rng.random((k, dim))) / c)
    _run(dim, np.concatenate(x).astype(np.float32), c, radius)


@pytest.mark.parametrize("dim", [2, 3])
def test_domain_edges(dim):
    rng = np.random.default_rng(5)
    x = rng.random((600, dim))
    x[:200, 0] *= 0.02
    x[200:400, -1] = 1 - 0.02 * x[200:400, -1]
    _run(dim, np.clip(x, 0, 1 - 1e-6).astype(np.float32), 16, 0.5)


@pytest.mark.parametrize("dim", [2, 3])
def test_large_scene(dim):
    """160,000 particles: a dense box (long tasks) and a sparse one."""
    rng = np.random.default_rng(9)
    a = 0.25 + 0.1 * rng.random((100000, dim))
    b = 0.45 + 0.4 * rng.random((60000, dim))
    _run(dim, np.concatenate([a, b]).astype(np.float32), 64 if dim == 2 else 32, 0.5)
