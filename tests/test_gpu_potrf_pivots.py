"""The Cholesky pivots' roots, on diagonal S: U(k, k) = sqrt(S(k, k)) and X(k, k) = 1 / sqrt(S(k, k)).

Both end in one rounding (half an ulp) of a value whose own error, the cube of the hardware approximation's (at most about
2^-20), is a few hundredths of an ulp: 0.6 ulp against the roots in extended precision.  S spans the doubles, on both
sides of the bounds below which the argument is scaled.  For a dense S, U^T U against S in extended precision: the
elimination must not round an entry once for every product.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L = np.longdouble


def _factor(xe, s):
    import torch

    n = s.shape[0]
    b = torch.from_numpy(np.ascontiguousarray(s.T)).cuda()
    x = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    info = xe.dsygvd_factor_device(n, b.data_ptr(), n, x.data_ptr(), n)
    torch.cuda.synchronize()
    assert info == 0
    return np.triu(b.cpu().numpy().T), x.cpu().numpy().T


@pytest.mark.parametrize("lo,hi", [(1.0, 4.0), (1e-3, 1e3), (1e-251, 1e-249), (1e-281, 1e-279), (1e-300, 1e-290), (1e290, 1e300)])
def test_roots_of_the_pivots(xe, lo, hi):
    xe.set_device(0)
    n = 640
    d = np.exp(np.random.default_rng(17).uniform(np.log(lo), np.log(hi), n))
    u, x = _factor(xe, np.diag(d))
    root = np.sqrt(d.astype(L))
    rel = np.abs(np.diag(u).astype(L) - root) / np.spacing(root.astype(np.float64))
    # below 1e-280 d r is kept as it is: one rounding more
    assert rel.max() < (0.6 if lo > 1e-280 else 1.7)
    inv = 1 / root
    assert (np.abs(np.diag(x).astype(L) - inv) / np.spacing(inv.astype(np.float64))).max() < 0.6


@pytest.mark.parametrize("n", [37, 130, 300])
def test_factor_in_extended_precision(xe, n):
    """|U^T U - S| for S = 2 I + G with |G| row sums below 1: its rounding is that of a sum of about three numbers of size
    one per entry (bar: 4 u max S(k, k)), since the rows of U decay away from the diagonal."""
    xe.set_device(0)
    rng = np.random.default_rng(n)
    idx = np.arange(n)
    g = np.triu(rng.uniform(-1, 1, (n, n)), 1) * 0.3 * np.exp(-np.abs(idx[:, None] - idx[None, :]) / 1.5)
    s = np.diag(rng.uniform(2, 3, n)) + g + g.T
    u, x = _factor(xe, s)
    ul = u.astype(L)
    assert np.abs(ul.T @ ul - s).max() < 4 * 3 * 2.0**-53
    assert np.abs(ul @ x.astype(L) - np.eye(n)).max() < 4 * 2.0**-53
