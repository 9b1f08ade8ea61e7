"""launches_per_substep against the kernels that a substep runs, traced on the
device: single scenes of every form that changes the number, batches, and the
surrogate's two kernels."""
import numpy as np
import pytest
import torch

from _gpu_util import gpu_sim, have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA device")]


def _scene(dim, level, plastic=False, static=False, n=3000):
    rng = np.random.default_rng(dim + level)
    x = (0.3 + 0.3 * rng.random((n, dim))).astype(np.float32)
    F = np.tile(np.eye(dim, dtype=np.float32), (n, 1, 1))
    sim = gpu_sim(dim, level, 16, n, plasticity="snow" if plastic else None)
    if static:
        sim.set_coarse_level_map(np.full((16,) * dim, level - 1, np.int8))
    sim.set_particles(x=x, v=np.zeros_like(x), F=F, C=np.zeros_like(F), m=np.ones(n, np.float32),
                      g=np.full(n, level - 1, np.int32))
    return sim


def _traced(step, n=3):
    step()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        for _ in range(n):
            step()
        torch.cuda.synchronize()
    names = [e.name for e in prof.events() if "agimp::" in e.name and "k_" in e.name]
    assert names and len(names) % n == 0, sorted(set(names))
    return len(names) // n


@pytest.mark.parametrize("dim,level,plastic,static", [(2, 1, False, False), (2, 3, True, False), (2, 3, False, True),
                                                      (3, 1, True, False), (3, 3, True, False), (3, 2, False, True)])
def test_single_scene(dim, level, plastic, static):
    sim = _scene(dim, level, plastic, static)
    assert sim.launches_per_substep() == _traced(lambda: sim.substep(1e-5))
    assert sim.launches_per_substep() == _traced(lambda: sim.profile_substep(1e-5))
    sim.close()


@pytest.mark.parametrize("surrogate", [False, True])
def test_batch_and_surrogate(surrogate):
    from agimp.batch import SceneBatch
    from agimp.surrogate import MLP
    sims = [_scene(2, 3, True), _scene(2, 2, False, True), _scene(2, 1)]
    mlp, one = MLP(), _scene(3, 2, True)
    batch = SceneBatch(sims)
    if surrogate:
        one.set_surrogate(mlp, [1.0] * 7)
        batch.set_surrogate(mlp, [1.0] * 7)
    assert batch.launches_per_substep() == _traced(lambda: batch.substep(1e-5))
    assert one.launches_per_substep() == _traced(lambda: one.substep(1e-5))
    batch.close()
    for s in sims + [one]:
        s.close()
