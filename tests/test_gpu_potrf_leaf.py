"""The Cholesky leaf: factor and inverse of a 64 x 64 diagonal block from one elimination across four warps of 16 rows.

Sizes on both sides of the warps' rows and of the block; pivots that fail in every warp's rows; diagonal scalings far
from 1, which the pivots' reciprocal square root meets.  Tolerances: |U^T U - S| and |U X - I| are a small multiple of
n eps for these well-conditioned S (diagonal at least 2, off-diagonal row sums below 1): 1e-14 n.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spd(n, seed):
    rng = np.random.default_rng(seed)
    idx = np.arange(n)
    g = np.triu(rng.uniform(-1, 1, (n, n)), 1) * 0.3 * np.exp(-np.abs(idx[:, None] - idx[None, :]) / 1.5)
    return np.diag(rng.uniform(2, 3, n)) + g + g.T


def _factor(xe, s):
    import torch

    n = s.shape[0]
    b = torch.from_numpy(np.ascontiguousarray(s.T)).cuda()
    x = torch.full((n, n), 7.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    info = xe.dsygvd_factor_device(n, b.data_ptr(), n, x.data_ptr(), n)
    torch.cuda.synchronize()
    return info, np.triu(b.cpu().numpy().T), x.cpu().numpy().T


@pytest.mark.parametrize("n", [1, 2, 7, 15, 16, 17, 31, 33, 47, 49, 63, 64, 65, 80, 127, 129, 200])
def test_factor_and_inverse(xe, n):
    xe.set_device(0)
    s = _spd(n, 40 + n)
    info, u, x = _factor(xe, s)
    assert info == 0
    assert np.abs(u.T @ u - s).max() < 1e-14 * n + 1e-14
    assert np.abs(u @ x - np.eye(n)).max() < 1e-14 * n + 1e-14
    assert np.array_equal(np.tril(x, -1), np.zeros((n, n)))


@pytest.mark.parametrize("bad", [0, 1, 15, 16, 31, 32, 40, 63, 64, 100])
def test_pivot_that_fails(xe, bad):
    xe.set_device(0)
    s = _spd(130, 77)
    s[bad, bad] = -1.0
    info, _, _ = _factor(xe, s)
    assert info == 130 + bad + 1


def test_scaled_pivots(xe):
    """U = U0 D for S = D S0 D with powers of two on the diagonal (pivots from 2^-960 to 2^960)."""
    xe.set_device(0)
    n = 97
    s0 = _spd(n, 5)
    u0 = np.linalg.cholesky(s0).T
    e = np.linspace(-480, 480, n).round().astype(int)
    d = np.ldexp(1.0, e)
    info, u, _ = _factor(xe, d[:, None] * s0 * d[None, :])
    assert info == 0
    scaled = np.triu(u0) * d[None, :]
    np.testing.assert_allclose(np.diag(u), np.diag(scaled), rtol=1e-14 * n)
    # Entries relative to their column's scale (the largest row-wise product |U^T U| bounds the rounding).
    assert (np.abs(u - scaled) / d[None, :]).max() < 1e-14 * n
