"""The accuracy of the Jacobi leaves (n <= 8: xtb_dstedc is one leaf), in extended precision.

About six sweeps of seven rounds, each of which rounds an entry of a, or of the vectors, a few times: the errors of 42
rounds add up like a random walk.  Residual: 3 u |T| a round, 2.2e-15 |T|, twice that at most over many inputs, and 1e-15
|T| for the off-diagonal part at which the sweeps stop: 5.5e-15 |T|.  Orthogonality: half a u a round from the update and
0.6 u from c^2 + s^2 = 1 give 5.1 u; the largest of 36 entries lies at about 2.2 times that: 1.25e-15 in the median.
"""
import numpy as np
import pytest

from oracle import inputs

pytestmark = pytest.mark.gpu

L = np.longdouble


@pytest.mark.parametrize("n", [2, 5, 7, 8])
def test_leaf_accuracy(xe, n):
    res, orth = [], []
    for seed in range(400):
        d, e = inputs.random_tridiagonal(n, 31000 + 1000 * n + seed)
        w, z, info = xe.stedc(d, e)
        assert info == 0
        t = (np.diag(d) + np.diag(e, 1) + np.diag(e, -1)).astype(L)
        zl = z.astype(L)
        res.append(np.abs(t @ zl - zl * w.astype(L)).max() / np.abs(w).max())
        orth.append(np.abs(zl.T @ zl - np.eye(n)).max())
    assert max(res) < 5.5e-15
    assert np.median(orth) < 1.25e-15
