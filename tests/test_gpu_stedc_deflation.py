"""GPU checks of the divide and conquer's deflation step over sizes on both sides of its shared-memory limit (merges of
6400), with spectra that deflate by small z, by close pairs and hardly at all.

Bars (backward error of a divide and conquer with 2^-53 rounding, LAPACK's own tests use 30 n u): residual
|T Z - Z diag(d)| <= 30 n u |T| and orthogonality |Z^T Z - I| <= 30 n u, in the largest entry.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def _tridiagonal(kind, n):
    rng = np.random.default_rng(n)
    if kind == "random":
        return rng.standard_normal(n), rng.standard_normal(n - 1)
    if kind == "wilkinson":  # glued copies of W21+: eigenvalues in close pairs
        d = np.resize(np.abs(np.arange(21) - 10.0), n)
        e = np.ones(n - 1)
        e[20::21] = 1e-8
        return d, e
    return np.full(n, 2.0), np.full(n - 1, -1.0)  # Toeplitz: small z at the ends, few deflations


@pytest.mark.parametrize("kind,n", [(k, n) for k in ("random", "wilkinson", "toeplitz") for n in (65, 129, 513, 1030, 2100)]
                         + [("wilkinson", 6500)])
def test_stedc_deflation(xe, kind, n):
    import torch

    d0, e0 = _tridiagonal(kind, n)
    d, z, info = xe.stedc(d0, e0)
    assert info == 0
    assert (np.diff(d) >= 0).all()
    zt, dt = torch.from_numpy(np.ascontiguousarray(z)).cuda(), torch.from_numpy(d).cuda()
    td, te = torch.from_numpy(d0).cuda(), torch.from_numpy(e0).cuda()
    tz = td[:, None] * zt
    tz[:-1] += te[:, None] * zt[1:]
    tz[1:] += te[:, None] * zt[:-1]
    norm = np.abs(d0).max() + 2 * np.abs(e0).max()
    assert float((tz - zt * dt[None, :]).abs().max()) <= 30 * n * U * norm
    assert float((zt.T @ zt - torch.eye(n, dtype=zt.dtype, device="cuda")).abs().max()) <= 30 * n * U
