"""The resident reduction with 1024 threads (n > 4096): rows in L2, four column pairs per thread up to n = 8192 and eight
above, where one code path serves five to eight active pairs.

The pairs past the active ones must not be touched: up to n = 14336 they lie in the next row.  Checked with eight random
vectors z of unit norm: |A Q z - Q T z| within n u |A| in the 2-norm (u the rounding unit; LAPACK's own bar is 30 times
that), |A| taken from the semicircle law, 2 sqrt(n / 3) for entries uniform on [-1, 1]; and Q^T Q = I on them within n u.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dtype", [(4099, np.float64), (9001, np.float64), (4101, np.float32), (10300, np.float32)])
def test_large_plans(xe, n, dtype):
    rng = np.random.default_rng(n)
    a = rng.random((n, n), dtype=dtype)
    a *= 2
    a -= 1
    i = np.arange(0, n, 512)
    for lo in i:  # symmetric: the upper triangle mirrored
        for up in i[i >= lo]:
            r, c = slice(lo, lo + 512), slice(up, up + 512)
            if lo == up:
                a[r, r] = np.triu(a[r, r]) + np.triu(a[r, r], 1).T
            else:
                a[c, r] = a[r, c].T
    ar = a.copy().T  # a symmetric matrix in Fortran order
    d, e, tau = np.zeros(n, dtype), np.zeros(n - 1, dtype), np.zeros(n - 1, dtype)
    sytrd, ormtr = (xe.xtb_dsytrd_upper, xe.xtb_dormtr_upper) if dtype == np.float64 else (xe.xtb_ssytrd_upper,
                                                                                          xe.xtb_sormtr_upper)
    sytrd(n, ar, n, d, e, tau)
    z = rng.standard_normal((n, 8))
    z /= np.linalg.norm(z, axis=0)
    tz = d[:, None] * z
    tz[:-1] += e[:, None].astype(float) * z[1:]
    tz[1:] += e[:, None].astype(float) * z[:-1]
    q = np.asfortranarray(np.hstack([z, tz]).astype(dtype))
    ormtr(n, 16, ar, n, tau, q, n)
    q = q.astype(float)
    res = a.astype(float, copy=False) @ q[:, :8]
    u = np.finfo(dtype).eps / 2
    norm = 2 * np.sqrt(n / 3)
    assert np.linalg.norm(res - q[:, 8:], axis=0).max() < n * u * norm
    assert np.abs(q[:, :8].T @ q[:, :8] - z.T @ z).max() < n * u
