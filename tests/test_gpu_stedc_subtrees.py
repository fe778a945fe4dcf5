"""The subtrees of at most 64 that one CTA solves: every size at which its leaves (at most 8) and levels change, alone and
below merge levels, on spectra with deflation of both kinds.

Bars as for the other tridiagonal tests: eigenvalues within 5e-14 n max(|d|, |e|) of LAPACK's dstedc, residual and
orthogonality within 1e-13 n, ascending order.
"""
import numpy as np
import pytest

from oracle import inputs, lapack, metrics

pytestmark = pytest.mark.gpu


def _check(xe, d, e):
    n = len(d)
    w_ref, _, info_ref = lapack.stedc(d, e)
    w, z, info = xe.stedc(d, e)
    assert info == 0 and info_ref == 0
    scale = max(np.abs(d).max(), np.abs(e).max() if n > 1 else 0.0, 1e-300) * n
    np.testing.assert_allclose(w, w_ref, rtol=0, atol=5e-14 * scale)
    assert np.all(np.diff(w) >= 0)
    t = np.diag(d) + np.diag(e, 1) + np.diag(e, -1)
    _, res, orth = metrics.eigen_accuracy(t, w_ref, w, z)
    assert res < 1e-13 * n and orth < 1e-13 * n


@pytest.mark.parametrize("n", [4, 7, 8, 9, 10, 15, 18, 24, 31, 33, 36, 40, 48, 56, 57, 61, 64, 66, 127, 128, 129, 250])
def test_sizes(xe, n):
    d, e = inputs.random_tridiagonal(n, 2100 + n)
    _check(xe, d, e)


@pytest.mark.parametrize("n", [12, 37, 64, 90])
@pytest.mark.parametrize("kind", ["zero_offdiag", "zeros", "ties", "split", "wilkinson", "toeplitz", "graded", "tiny", "huge"])
def test_hard(xe, n, kind):
    rng = np.random.default_rng(n)
    d, e = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n - 1)
    if kind == "zero_offdiag":
        e[:] = 0.0
    elif kind == "zeros":
        d[:] = 0.0
        e[:] = 0.0
    elif kind == "ties":
        d, e = np.resize(np.array([0.5, -0.25, 1.0]), n), 1e-9 * e
    elif kind == "split":
        e[::3] = 0.0
    elif kind == "wilkinson":
        d, e = np.abs(np.arange(n) - (n - 1) / 2), np.ones(n - 1)
    elif kind == "toeplitz":
        d, e = np.full(n, 2.0), np.full(n - 1, -1.0)
    elif kind == "graded":
        s = 10.0 ** np.linspace(0, -14, n)
        d, e = d * s, e * s[1:]
    elif kind == "tiny":
        d, e = d * 1e-150, e * 1e-150
    else:
        d, e = d * 1e150, e * 1e150
    _check(xe, d, e)


@pytest.mark.parametrize("n", [20, 64, 100])
def test_nan_input_ends(xe, n):
    """NaN in, an error or NaN out; the call returns and the next one is right."""
    d, e = inputs.random_tridiagonal(n, 3)
    bad = d.copy()
    bad[n // 2] = np.nan
    w, _, info = xe.stedc(bad, e)
    assert info != 0 or not np.all(np.isfinite(w))
    _check(xe, d, e)
