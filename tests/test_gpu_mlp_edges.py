"""The surrogate MLP's kernels at the edges of their branches: pre-activations
beyond the range of the shared reciprocal (|z| >= 40), infinite inputs, and
output buffers that are not 16-byte aligned."""
import ctypes

import numpy as np
import pytest

import mlp_ref as R
from _gpu_util import have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA device")]


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("gain", [1.0, 25.0, 100.0])
@pytest.mark.parametrize("n", [1, 129, 4099])
def test_forward_far_preactivations(n, gain):
    """Weights scaled so that pre-activations reach tens to hundreds: an
    activation may round to the neighbouring bf16 value (2^-8 of itself), which
    moves an output by at most that share of a term of its sum."""
    import torch

    from agimp.surrogate import MLP
    rng = np.random.default_rng(n)
    P = R.init_params(rng).astype(np.float32)
    P[: R.IN * R.H] *= gain
    X = rng.normal(0, 1, (n, R.IN)).astype(np.float32)
    m = MLP(params=P)
    Y = m.forward(torch.from_numpy(X).cuda()).cpu().numpy()
    assert m.errors() == 0
    ref, _ = R.forward(P, X)
    assert np.abs(Y - ref).max() <= 1e-2 * np.abs(ref).max() + 1e-3
    m.close()


def test_infinite_input_stays_in_its_row():
    """A row of infinities gives what the plain expression gives (no finite
    value), and the rows beside it are untouched."""
    import torch

    from agimp.surrogate import MLP
    rng = np.random.default_rng(3)
    P = R.init_params(rng).astype(np.float32)
    X = rng.normal(0, 1, (200, R.IN)).astype(np.float32)
    m = MLP(params=P)
    plain = m.forward(torch.from_numpy(X).cuda()).cpu().numpy()
    X[70] = np.inf
    Y = m.forward(torch.from_numpy(X).cuda()).cpu().numpy()
    assert not np.isfinite(Y[70]).any()
    keep = np.arange(200) != 70
    np.testing.assert_array_equal(Y[keep], plain[keep])
    m.close()


@pytest.mark.parametrize("n", [1, 128, 1000])
@pytest.mark.parametrize("shift", [1, 2, 3])
def test_unaligned_outputs(n, shift):
    import torch

    from agimp.surrogate import MLP
    rng = np.random.default_rng(n)
    m = MLP(params=R.init_params(rng).astype(np.float32))
    X = torch.from_numpy(rng.normal(0, 1, (n, R.IN)).astype(np.float32)).cuda()
    T = torch.from_numpy(rng.normal(0, 1, (n, R.OUT)).astype(np.float32)).cuda()
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    whole = m.forward(X)
    buf = torch.zeros(n * R.OUT + 8, device="cuda")
    assert m._L.agimp_mlp_forward(m._h, _ptr(X), _ptr(buf[shift:]), n, st) == 0
    assert torch.equal(buf[shift:shift + n * R.OUT].reshape(n, R.OUT), whole)
    assert not buf[:shift].any() and not buf[shift + n * R.OUT:].any()
    g = [torch.full((R.NPARAM + 8,), 7.0, device="cuda") for _ in range(2)]
    loss = torch.empty(2, device="cuda")
    for k, o in enumerate((0, shift)):
        assert m._L.agimp_mlp_grad(m._h, _ptr(X), _ptr(T), n, _ptr(g[k][o:]), _ptr(loss[k:]), st) == 0
    a, b = g[0][:R.NPARAM], g[1][shift:shift + R.NPARAM]
    # the same products; at most 8 CTAs add their sums in another order
    assert (a - b).norm() <= 1e-5 * a.norm()
    assert torch.allclose(loss[0], loss[1], rtol=1e-5)
    assert (g[1][:shift] == 7).all() and (g[1][shift + R.NPARAM:] == 7).all()
    m.close()
