"""Launch tuning: a value that is not given stays as it is, and the autotuner
leaves alone the item size of 2D scenes, on which no 2D launch depends."""
import numpy as np
import pytest

from _gpu_util import gpu_sim, have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA device")]


def _scene(dim, n=4000):
    rng = np.random.default_rng(dim)
    x = (0.3 + 0.3 * rng.random((n, dim))).astype(np.float32)
    F = np.tile(np.eye(dim, dtype=np.float32), (n, 1, 1))
    sim = gpu_sim(dim, 2, 16, n)
    sim.set_particles(x=x, v=np.zeros_like(x), F=F, C=np.zeros_like(F), m=np.ones(n, np.float32),
                      g=np.ones(n, np.int32))
    return sim


@pytest.mark.parametrize("batched", [False, True])
def test_one_value_alone(batched):
    from agimp.batch import SceneBatch
    sims = [_scene(3), _scene(3)]
    t = SceneBatch(sims) if batched else sims[0]
    first = t.tuning
    t.set_tuning(ctas_per_sm=5)
    assert (t.tuning["chunk"], t.tuning["ctas_per_sm"]) == (first["chunk"], 5)
    t.set_tuning(chunk=64)
    assert (t.tuning["chunk"], t.tuning["ctas_per_sm"]) == (64, 5)
    t.set_tuning()
    assert (t.tuning["chunk"], t.tuning["ctas_per_sm"]) == (64, 5)
    if batched:
        t.close()
    for s in sims:
        s.close()


@pytest.mark.parametrize("chunk", [64, 128, 256, 512])
def test_autotune_2d_item_size(chunk):
    sim = _scene(2)
    sim.set_tuning(chunk, 3)
    best = sim.autotune(1e-5, trials=3)
    assert best["chunk"] == chunk and best["ctas_per_sm"] in (2, 3, 4, 8, 16)
    assert sim.tuning == best
    sim.close()
