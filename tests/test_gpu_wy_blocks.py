"""GPU checks of the compact-WY factors of ormtr (xtb_dormtr_upper, xtb_sormtr_upper) over block sizes that leave partial
tiles, partial pairs and a lone diagonal block when neighbours are joined.

Reference: the reflectors H(j) = I - tau v v^T applied one by one in FP64 on the host, from the same (rounded) v and tau,
tau = 2 / v^T v.  Each of the n - 1 applications perturbs a column by a few u of its norm in the blocked order as in the
plain one (the FP32 tau's own rounding changes a reflector by u), so a column may differ by 10 n u of its norm.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("nb,n", [(16, 41), (17, 41), (24, 25), (33, 130), (96, 300), (100, 300), (128, 300), (160, 333)])
def test_ormtr_block_sizes(xe, nb, n, dtype):
    rng = np.random.default_rng(nb + n)
    a = np.asfortranarray(rng.standard_normal((n, n)).astype(dtype))
    tau = np.zeros(n, dtype)
    ref = rng.standard_normal((n, 37)).astype(dtype).astype(np.float64)
    z = np.asfortranarray(ref.astype(dtype))
    norms = np.linalg.norm(ref, axis=0)
    for j in range(n - 1):
        v = np.zeros(n)
        v[:j] = a[:j, j + 1]
        v[j] = 1.0
        tau[j] = 2.0 / (v @ v)
        ref -= float(tau[j]) * np.outer(v, v @ ref)
    old = xe.get_option("ormtr_nb")
    xe.set_option("ormtr_nb", nb)
    try:
        out = xe.ormtr_upper(a, tau, z, dtype)
    finally:
        xe.set_option("ormtr_nb", old)
    u = np.finfo(dtype).eps / 2
    err = np.linalg.norm(out.astype(np.float64) - ref, axis=0)
    assert (err <= 10 * n * u * norms).all(), (err / norms).max()
