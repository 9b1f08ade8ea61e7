"""From ten million particles on the lattice and particle kernels launch eight
times the resident CTAs: eleven scenes of a million particles in one batch, each
against the same scene stepped alone (two times; checked against the oracle in
test_gpu_launch_waves.py)."""
import numpy as np
import pytest

from _gpu_util import gpu_sim, gpu_state, have_gpu, scale_rel

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA device")]

# one substep in f32: the two runs sum a node's particles in other orders; as in tests/test_gpu_parity.py
RTOL = 2e-5


@pytest.mark.parametrize("dim", [2, 3])
def test_batch_of_eleven_million(dim):
    from agimp.batch import SceneBatch
    n = 1_000_003
    rng = np.random.default_rng(dim)
    coarsest = 512 if dim == 2 else 64
    x = (0.05 + 0.9 * rng.random((n, dim))).astype(np.float32)
    F = np.tile(np.eye(dim, dtype=np.float32), (n, 1, 1)) + rng.normal(0, 0.02, (n, dim, dim)).astype(np.float32)
    s = dict(x=x, v=rng.normal(0, 1, (n, dim)).astype(np.float32), F=F, C=np.zeros((n, dim, dim), np.float32),
             m=np.ones(n, np.float32), g=np.where(x[:, 0] < 0.5, 1, 0).astype(np.int32))
    sims = [gpu_sim(dim, 2, coarsest, n) for _ in range(12)]
    for sim in sims:
        sim.set_particles(**s)
    alone, together = sims[0], sims[1:]
    batch = SceneBatch(together)
    batch.substep(1e-5)
    alone.substep(1e-5)
    q = gpu_state(alone)
    for sim in (together[0], together[5], together[10]):
        assert sim.errors() & ~2 == 0
        p = gpu_state(sim)
        np.testing.assert_array_equal(p["fl"], q["fl"])
        for k in "xvFC":
            assert scale_rel(p[k], q[k]) <= RTOL, (k, scale_rel(p[k], q[k]))
    batch.close()
    for sim in sims:
        sim.close()
