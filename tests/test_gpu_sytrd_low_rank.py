"""The reduction of matrices whose trailing blocks vanish: rounding leaves about u |A|, u^2 |A|, ... of them step by step, down
to columns whose squares underflow.  The reflectors must stay orthogonal there.

Bars (LAPACK's own): |Q^T Q - I| <= 30 n u and |Q^T A Q - T| <= 30 n u |A| in the largest entry, u the rounding unit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(kind, n):
    if kind == "ones":
        return np.ones((n, n))
    if kind == "ramp":
        v = np.arange(1.0, n + 1)
        return np.outer(v, v) / n**2
    a = np.zeros((n, n))  # "corner": the reduction starts in an identity, the ones come later
    m = max(2, n // 2)
    a[:m, :m] = 1.0
    a[m:, m:] = np.eye(n - m)
    return a


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("kind", ["ones", "ramp", "corner"])
@pytest.mark.parametrize("scale", [1.0, 2.0**20])
def test_orthogonal_where_squares_underflow(xe, kind, dtype, scale):
    u = np.finfo(dtype).eps / 2
    for n in (3, 16, 33, 40, 64, 65, 66, 80, 97, 128, 129, 200, 260, 400, 700):
        a = (_matrix(kind, n) * scale).astype(dtype)
        f, d, e, tau = xe.sytrd_upper(a, dtype)
        q = xe.ormtr_upper(f, tau, np.eye(n, dtype=dtype, order="F"), dtype).astype(float)
        t = np.diag(d.astype(float)) + np.diag(e.astype(float), 1) + np.diag(e.astype(float), -1)
        assert np.abs(q.T @ q - np.eye(n)).max() <= 30 * n * u, n
        assert np.abs(q.T @ a.astype(float) @ q - t).max() <= 30 * n * u * np.linalg.norm(a.astype(float), 2), n
