"""The plastic volume ratio of the 3D snow return map near rotations at the ends
of its range (csrc/common.cuh: snow_clamp_near, compiled as host code): what
Jp det(F) / det(clamped F) gives, an infinite ratio (no hardening stress left)
included."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import REPO


def test_infinite_zero_and_tiny_ratio(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    out = str(tmp_path / "libsnow_harness.so")
    subprocess.run([nvcc, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared",
                    "-I", os.path.join(REPO, "include"), os.path.join(REPO, "tests", "cuda_harness", "snow_harness.cu"),
                    "-o", out], check=True)
    h = ctypes.CDLL(out)
    jp = np.array([np.inf, -np.inf, np.nan, 0.0, 3e38, 3.4e38, 1e-40, -1.25, 1.25], np.float32)
    F = np.tile(np.diag([1.1, 1.0, 1.0]).astype(np.float32), (len(jp), 1, 1))
    got, ok = jp.copy(), np.zeros(len(jp), np.int32)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    h.h_snow_near(p(F), p(got), p(ok), ctypes.c_float(0.975), ctypes.c_float(1.0075), len(jp))
    assert ok.all()
    # products that leave the range of 32 bits become infinite, as in
    # jp * Jo / Jn; the others to the bound of the return map's tests
    with np.errstate(over="ignore", invalid="ignore"):
        ref = (jp * np.float32(1.1)).astype(np.float64) / 1.0075
    fin = np.isfinite(ref)
    np.testing.assert_array_equal(got[~fin], ref[~fin].astype(np.float32))
    np.testing.assert_allclose(got[fin], ref[fin], rtol=2e-6, atol=3e-45)
