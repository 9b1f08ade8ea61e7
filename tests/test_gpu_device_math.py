"""Device arithmetic that has a form of its own, run on the device: the
surrogate's activations (silu8: one reciprocal for two quotients) against the
rounded division they stand for, and the 3D snow return map near rotations
(hardware reciprocal root and quotient) against numpy's SVD in f64."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from _gpu_util import have_gpu
from conftest import REPO

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA device")]

LO, HI = np.float32(1 - 0.025), np.float32(1 + 0.0075)
EPS = 2.0 ** -23


def _harness(tmp_path_factory, name):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    out = str(tmp_path_factory.mktemp("harness") / ("lib%s.so" % name))
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "--expt-relaxed-constexpr",
                    "-Xcompiler", "-fPIC", "-shared", "-I", os.path.join(REPO, "include"),
                    os.path.join(REPO, "tests", "cuda_harness", name + ".cu"), "-o", out], check=True)
    return ctypes.CDLL(out)


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.fixture(scope="module")
def silu(tmp_path_factory):
    return _harness(tmp_path_factory, "silu_device")


def _activations(silu, z, deriv):
    import torch
    fast, plain = torch.empty_like(z), torch.empty_like(z)
    torch.cuda.synchronize()
    assert silu.h_silu(_ptr(z), _ptr(fast), _ptr(plain), ctypes.c_longlong(z.numel()), int(deriv)) == 0
    return fast, plain


def _arguments(kind):
    import torch
    n = 1 << 26
    g = torch.Generator(device="cuda").manual_seed(11)
    u = torch.rand(n, generator=g, device="cuda") * 2 - 1
    if kind == "uniform":
        return u * 39.99
    if kind == "normal":
        return torch.randn(n, generator=g, device="cuda").clamp(-39.9, 39.9)
    # magnitudes from 1e-30 to 39.9, unequal neighbours in a pair
    e = torch.rand(n, generator=g, device="cuda") * 31.6 - 30.0
    return torch.sign(u) * torch.pow(10.0, e).clamp(max=39.9)


@pytest.mark.parametrize("kind", ["uniform", "normal", "magnitudes"])
def test_silu_quotient(silu, kind):
    """The reciprocal has an error of a few units of its last place, one Newton
    step leaves about half of one, and the quotient is corrected by its exact
    remainder: before the last rounding it is within about 2^-45 of itself, so
    it rounds to another value only if it lies that near to the middle of two,
    once in 2^20 operands, and then to the neighbour."""
    import torch
    z = _arguments(kind)
    fast, plain = _activations(silu, z, False)
    ulps = (fast.view(torch.int32).long() - plain.view(torch.int32).long()).abs()
    ulps[(fast == 0) & (plain == 0)] = 0
    assert int(ulps.max()) <= 1
    assert int((ulps > 0).sum()) <= z.numel() >> 20


@pytest.mark.parametrize("kind", ["uniform", "normal", "magnitudes"])
def test_silu_derivative(silu, kind):
    """s (1 + z (1 - s)) moves by (1 + z (1 - 2 s)) ds when s moves by one unit,
    and its three roundings by at most as much again each."""
    import torch
    z = _arguments(kind)
    fast, plain = _activations(silu, z, True)
    s = torch.sigmoid(z.double())
    tol = 4 * EPS * s * (1 + z.double().abs())
    assert bool(((fast.double() - plain.double()).abs() <= tol).all())


def test_silu_beyond_the_shared_reciprocal(silu):
    """Groups of eight with any |z| >= 40, an infinity or NaN take the plain
    expressions."""
    import torch
    z = torch.linspace(-3, 3, 8 * 12, device="cuda").reshape(12, 8).clone()
    for i, v in enumerate((40.0, -40.0, 88.0, -88.0, 200.0, -200.0, 3e38, -3e38, float("inf"), float("-inf"),
                           float("nan"), 39.999)):
        z[i, i % 8] = v
    for deriv in (False, True):
        fast, plain = _activations(silu, z, deriv)
        torch.testing.assert_close(fast, plain, rtol=1e-6, atol=0, equal_nan=True)


@pytest.fixture(scope="module")
def snow(tmp_path_factory):
    return _harness(tmp_path_factory, "snow_device")


def _near(snow, F, jp0=1.25):
    import torch
    f = torch.from_numpy(np.ascontiguousarray(F, np.float32)).cuda()
    jp = torch.full((len(F),), jp0, device="cuda")
    ok = torch.zeros(len(F), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert snow.h_snow_near(_ptr(f), _ptr(jp), _ptr(ok), ctypes.c_float(LO), ctypes.c_float(HI), len(F)) == 0
    return f.cpu().numpy(), jp.cpu().numpy(), ok.cpu().numpy()


def _rotations(rng, n):
    q, r = np.linalg.qr(rng.normal(size=(n, 3, 3)))
    q = q * np.sign(np.einsum("nii->ni", r))[:, None, :]
    return q * np.linalg.det(q)[:, None, None]


def _check(snow, F):
    F = F.astype(np.float32)
    got, jp, ok = _near(snow, F)
    assert ok.all()
    u, s, vt = np.linalg.svd(F.astype(np.float64))
    c = np.clip(s, LO, HI)
    # the bounds of the host build's test
    assert np.abs(got - u @ (c[:, :, None] * vt)).max() < 1e-6
    assert np.abs(jp / (1.25 * (s / c).prod(1)) - 1).max() < 2e-6
    inside = ((s > LO + 1e-6) & (s < HI - 1e-6)).all(1)
    np.testing.assert_array_equal(got[inside], F[inside])
    assert (jp[inside] == 1.25).all()


@pytest.mark.parametrize("norm", [1e-6, 1e-3, 0.02, 0.1, 0.399])
def test_snow_against_svd(snow, norm):
    rng = np.random.default_rng(int(norm * 1e6))
    n = 20000
    e = rng.normal(size=(n, 3))
    e *= norm / np.linalg.norm(e, axis=1, keepdims=True)
    _check(snow, _rotations(rng, n) @ (np.sqrt(1 + e)[:, :, None] * _rotations(rng, n)))


def test_snow_repeated_and_axis_aligned(snow):
    rng = np.random.default_rng(4)
    I = np.eye(3)
    s = np.array([[1, 1, 1], [1.1, 1.1, 1.1], [0.9, 0.9, 1.1], [1.1, 0.9, 0.9], [0.9, 1.1, 0.9], [1, 1.05, 1],
                  [1.0 + 1e-7, 1, 1.1], [LO, HI, 1]])
    V = _rotations(rng, len(s))
    _check(snow, s[:, :, None] * I)
    _check(snow, s[:, :, None] * V)
    _check(snow, np.swapaxes(V, 1, 2) @ (s[:, :, None] * V))


def test_snow_refuses_far_and_inverted(snow):
    I = np.eye(3)
    far = np.stack([np.diag([1.2, 1, 1]), np.diag([0.7, 0.9, 1]), 0 * I, 1e20 * I, np.nan * I, np.diag([np.inf] * 3),
                    np.diag([-1.0, 1, 1]), -I])
    got, jp, ok = _near(snow, far)
    assert not ok.any()
    np.testing.assert_array_equal(got, far.astype(np.float32))
    assert (jp == 1.25).all()


@pytest.mark.parametrize("jp0", [float("inf"), float("-inf"), 0.0])
def test_snow_ratio_without_a_remainder(snow, jp0):
    F = np.tile(np.diag([1.1, 1.0, 1.0]), (3, 1, 1))
    got, jp, ok = _near(snow, F, jp0)
    assert ok.all()
    np.testing.assert_array_equal(jp, np.float32(jp0))
