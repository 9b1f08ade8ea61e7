"""The 3D P2G stress around the norms where its form changes: |F F^T - I|_F =
0.1 (the series gets a Newton step) and 0.4 (polar iteration)."""
import ctypes

import numpy as np
import pytest
from test_device_math_cpu import f32p, h  # noqa: F401  (the compiled harness)


def _rotations(rng, n):
    q, r = np.linalg.qr(rng.normal(size=(n, 3, 3)))
    q = q * np.sign(np.einsum("nii->ni", r))[:, None, :]
    return q * np.linalg.det(q)[:, None, None]


@pytest.mark.parametrize("norm", [0.02, 0.0999, 0.1001, 0.25, 0.3999, 0.4001, 0.6])
def test_stress_at_norm(h, norm):  # noqa: F811
    """F = U sqrt(I + E) V with |E|_F = norm, against the polar rotation in
    f64.  The truncated series is off by less than 2.1e-8 below 0.1 and, after
    the Newton step, by half the square of 1.4e-4 below 0.4; the rest is the
    rounding of some ten operations on numbers of order one (eps = 6e-8)."""
    rng = np.random.default_rng(int(norm * 1e4))
    n = 2000
    e = rng.normal(size=(n, 3))
    e *= norm / np.linalg.norm(e, axis=1, keepdims=True)
    U, V = _rotations(rng, n), _rotations(rng, n)
    F = (U @ (np.sqrt(1 + e)[:, :, None] * V)).astype(np.float32)
    mu = 0.5
    tau = np.zeros_like(F)
    h.h_kirchhoff(3, f32p(F), ctypes.c_float(mu), ctypes.c_float(0.0), f32p(tau), n)
    Fd = F.astype(np.float64)
    u, s, vt = np.linalg.svd(Fd)
    ref = 2 * mu * (Fd - u @ vt) @ Fd.transpose(0, 2, 1)
    assert np.abs(tau - ref).max() < 1e-6
