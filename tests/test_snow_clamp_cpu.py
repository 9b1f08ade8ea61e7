"""The 3D snow return map near rotations (csrc/common.cuh: snow_clamp_near),
compiled as host code, against numpy's SVD in f64: norms up to its limit,
equal and axis-aligned singular values, and the states it must refuse."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import REPO

LO, HI = np.float32(1 - 0.025), np.float32(1 + 0.0075)


@pytest.fixture(scope="module")
def h(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    out = str(tmp_path_factory.mktemp("harness") / "libsnow_harness.so")
    subprocess.run([nvcc, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared",
                    "-I", os.path.join(REPO, "include"), os.path.join(REPO, "tests", "cuda_harness", "snow_harness.cu"),
                    "-o", out], check=True)
    return ctypes.CDLL(out)


def _near(h, F, lo=LO, hi=HI):
    F = np.ascontiguousarray(F, np.float32).copy()
    jp = np.full(len(F), 1.25, np.float32)
    ok = np.zeros(len(F), np.int32)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    h.h_snow_near(p(F), p(jp), p(ok), ctypes.c_float(lo), ctypes.c_float(hi), len(F))
    return F, jp, ok


def _rotations(rng, n):
    q, r = np.linalg.qr(rng.normal(size=(n, 3, 3)))
    q = q * np.sign(np.einsum("nii->ni", r))[:, None, :]
    return q * np.linalg.det(q)[:, None, None]


def _check(h, F):
    F = F.astype(np.float32)
    got, jp, ok = _near(h, F)
    assert ok.all()
    u, s, vt = np.linalg.svd(F.astype(np.float64))
    c = np.clip(s, LO, HI)
    # about ten roundings of numbers of order one in F' (eps = 6e-8); Jp: three
    # roots and six products, on sigmas with two roundings each
    assert np.abs(got - u @ (c[:, :, None] * vt)).max() < 1e-6
    assert np.abs(jp / (1.25 * (s / c).prod(1)) - 1).max() < 2e-6
    inside = ((s > LO + 1e-6) & (s < HI - 1e-6)).all(1)
    np.testing.assert_array_equal(got[inside], F[inside])
    assert (jp[inside] == 1.25).all()


@pytest.mark.parametrize("norm", [1e-6, 1e-3, 0.02, 0.1, 0.399])
def test_against_svd(h, norm):
    rng = np.random.default_rng(int(norm * 1e6))
    n = 3000
    e = rng.normal(size=(n, 3))
    e *= norm / np.linalg.norm(e, axis=1, keepdims=True)
    _check(h, _rotations(rng, n) @ (np.sqrt(1 + e)[:, :, None] * _rotations(rng, n)))


def test_repeated_and_axis_aligned(h):
    rng = np.random.default_rng(4)
    I = np.eye(3)
    s = np.array([[1, 1, 1], [1.1, 1.1, 1.1], [0.9, 0.9, 1.1], [1.1, 0.9, 0.9], [0.9, 1.1, 0.9], [1, 1.05, 1],
                  [1.0 + 1e-7, 1, 1.1], [LO, HI, 1]])
    V = _rotations(rng, len(s))
    _check(h, s[:, :, None] * I)
    _check(h, s[:, :, None] * V)
    _check(h, np.swapaxes(V, 1, 2) @ (s[:, :, None] * V))
    shear = I + 0.2 * np.array([[[0, 1, 0], [0, 0, 0], [0, 0, 0]], [[0, 0, 0], [0, 0, 0], [1, 0, 0]]])
    _check(h, shear)


def test_refuses_far_and_inverted(h):
    I = np.eye(3)
    far = np.stack([np.diag([1.2, 1, 1]), np.diag([0.7, 0.9, 1]), 0 * I, 1e20 * I, np.nan * I, np.diag([np.inf] * 3),
                    np.diag([-1.0, 1, 1]), -I])
    got, jp, ok = _near(h, far)
    assert not ok.any()
    np.testing.assert_array_equal(got, far.astype(np.float32))
    assert (jp == 1.25).all()
