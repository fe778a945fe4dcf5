"""The resident reduction over its plans: thread and column counts change at n = 256, 512, 1024 and 2048, rows live in
registers, shared memory or L2 according to the rows per CTA.

Every plan is checked against LAPACK's spectrum (eigenvalues of the tridiagonal within 5e-14 n max|A|, the bar of the
other sytrd tests: LAPACK's and this reduction's backward errors are both a small multiple of n eps |A|) and against the
input (A Q = Q T through xtb_dormtr_upper, within 1e-13 n max|A| elementwise).  The sums of a column do not depend on how
its rows are dealt to CTAs, so a different grid gives the same bits.
"""
import numpy as np
import pytest

from oracle import inputs, lapack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [66, 129, 255, 256, 257, 511, 513, 593, 1023, 1025, 2047, 2049])
def test_plan_edges(xe, n):
    a = inputs.random_symmetric(n, seed=1300 + n)
    ar, d, e, tau = xe.sytrd_upper(a)
    scale = np.abs(a).max() * n
    w = lapack.stedc(d, e)[0]
    np.testing.assert_allclose(w, np.linalg.eigvalsh(a), rtol=0, atol=5e-14 * scale)
    q = xe.ormtr_upper(ar, tau, np.eye(n))
    t = np.diag(d) + np.diag(e, 1) + np.diag(e, -1)
    assert np.abs(a @ q - q @ t).max() < 1e-13 * scale
    assert np.abs(q.T @ q - np.eye(n)).max() < 1e-13 * n


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n,grids", [(130, (3, 20)), (300, (4, 17, 75)), (611, (16, 100)), (1100, (60, 148))])
def test_grid_does_not_change_the_bits(xe, n, grids, dtype):
    a = inputs.random_symmetric(n, seed=1400 + n).astype(dtype)
    old = xe.get_option("sytrd_grid")
    try:
        xe.set_option("sytrd_grid", 0)
        ref = xe.sytrd_upper(a, dtype)
        for g in grids:
            xe.set_option("sytrd_grid", g)
            for x, y in zip(ref, xe.sytrd_upper(a, dtype)):
                assert np.array_equal(x, y), g
    finally:
        xe.set_option("sytrd_grid", old)
