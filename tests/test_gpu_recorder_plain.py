"""Arming the training-pair recorder leaves a run as it is: particles that share
no grid node (so that no order of additions comes in) get the same bits with
and without it, on both sides of the 3D rule for states near a rotation, and
the recorded pairs are the exact clamp of their trial states."""
import numpy as np
import pytest

from _gpu_util import gpu_sim, gpu_state, have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA device")]


def _isolated(dim, per_axis, dx, rng):
    i = np.stack(np.meshgrid(*[np.arange(per_axis)] * dim, indexing="ij"), -1).reshape(-1, dim)
    return ((4 * (i + 1) + 2 + rng.random(i.shape)) * dx).astype(np.float32)


@pytest.mark.parametrize("stride", [1, 3])
@pytest.mark.parametrize("dim,coarsest", [(3, 64), (2, 256)])
def test_same_bits_with_recorder(dim, coarsest, stride):
    import torch
    rng = np.random.default_rng(dim)
    x = _isolated(dim, coarsest // 4 - 2, 1.0 / coarsest, rng)
    n = len(x)
    spread = np.where(np.arange(n) % 4 == 0, 0.12, 0.02)[:, None, None]
    F = (np.eye(dim) + np.clip(rng.normal(0, 1, (n, dim, dim)), -2, 2) * spread).astype(np.float32)
    v = rng.normal(0, 1, (n, dim)).astype(np.float32)
    C = rng.normal(0, 0.1, (n, dim, dim)).astype(np.float32)
    m = rng.uniform(0.5, 2.0, n).astype(np.float32)
    jp = rng.uniform(0.8, 1.2, n).astype(np.float32)
    out = []
    for record in (False, True):
        sim = gpu_sim(dim, 1, coarsest, n, plasticity="snow", theta_c=2.5e-2, theta_s=7.5e-3, hardening=10.0)
        sim.set_particles(x=x, v=v, F=F, C=C, m=m, g=np.zeros(n, np.int32), Jp=jp)
        if record:
            X = torch.full((n, 7), float("nan"), device="cuda")
            T = torch.full((n, 4), float("nan"), device="cuda")
            sim.set_recorder(X, T, stride)
        sim.substep(1e-5)
        assert sim.errors() == 0
        out.append(gpu_state(sim))
        if record:
            k = sim.recorded()
            assert 0.5 * n < k * stride < 1.5 * n
            a, t = X[:k].cpu().numpy().astype(np.float64), T[:k].cpu().numpy().astype(np.float64)
            sig = 1 + 0.05 * a[:, :dim]
            c = np.clip(sig, 1 - 2.5e-2, 1 + 7.5e-3)
            np.testing.assert_allclose(t[:, :dim], (c - sig) / 0.02, atol=5e-5)
            np.testing.assert_allclose(t[:, 3], np.log(sig.prod(1) / c.prod(1)) / 0.02, atol=1e-4)
        sim.close()
    for k in ("x", "v", "F", "C", "Jp"):
        np.testing.assert_array_equal(out[0][k], out[1][k])
    assert (out[0]["Jp"] != jp).mean() > 0.5
