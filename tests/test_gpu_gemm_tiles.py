"""GPU checks of the grouped FP64 GEMM kernel (xtb_dgemm_device with the tensor-core split off) at the edges of its tiles.

A launch runs 32 x 32 or 64 x 64 output tiles by the number of tiles; K goes in steps of 16 through a four-deep pipeline,
and only a step at an edge of the matrix tests its elements.  Sizes: one element, tile edges of both kinds, K of a part
of a step, of one, four and five steps, and sizes on both sides of the choice of the tile (about 800), with all four
transpose combinations, odd leading dimensions and beta.  Reference: torch's FP64 product.  Both sum k products with
alpha and beta applied at the end, each with a rounding error of at most (k + 3) 2^-53 of the sum of absolute values, so
elementwise |difference| <= 2 (k + 3) 2^-53 (|alpha| |op(A)| |op(B)| + |beta C|).
"""
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (31, 33, 15), (32, 32, 16), (33, 65, 17), (64, 63, 64), (65, 64, 80), (130, 130, 130), (129, 7, 333),
         (776, 776, 50), (960, 961, 33), (1345, 1349, 20)]


@pytest.mark.parametrize("ta", [0, 1])
@pytest.mark.parametrize("tb", [0, 1])
@pytest.mark.parametrize("mnk", SIZES)
def test_dgemm_tile_edges(xe, ta, tb, mnk):
    import torch

    m, n, k = mnk
    dev = torch.device("cuda", 0)
    g = torch.Generator(device="cpu").manual_seed(m + 3 * n + 7 * k + ta + 2 * tb)
    ar, ac = (k, m) if ta else (m, k)
    br, bc = (n, k) if tb else (k, n)
    for pad, alpha, beta in ((0, 1.0, 0.0), (3, -0.5, 2.0)):
        lda, ldb, ldc = ar + pad, br + pad, m + pad
        A = torch.randn((ac, lda), generator=g, dtype=torch.float64).to(dev)
        B = torch.randn((bc, ldb), generator=g, dtype=torch.float64).to(dev)
        C = torch.randn((n, ldc), generator=g, dtype=torch.float64).to(dev)
        if beta == 0.0:
            C.fill_(float("nan"))  # C is not read
        a, b = A[:, :ar].T, B[:, :br].T
        opa, opb = (a.T if ta else a), (b.T if tb else b)
        ref, mag = alpha * (opa @ opb), abs(alpha) * (opa.abs() @ opb.abs())
        if beta != 0.0:
            ref, mag = ref + beta * C[:, :m].T, mag + abs(beta) * C[:, :m].T.abs()
        before = C.clone()
        torch.cuda.synchronize(dev)
        old = xe.get_option("dgemm_engine")
        xe.set_option("dgemm_engine", 0)
        try:
            rc = xe.dgemm_device(ta, tb, m, n, k, alpha, A.data_ptr(), lda, B.data_ptr(), ldb, beta, C.data_ptr(), ldc, 0)
        finally:
            xe.set_option("dgemm_engine", old)
        torch.cuda.synchronize(dev)
        assert rc == 0, xe.last_error()
        err = (C[:, :m].T - ref).abs()
        assert bool((err <= 2 * (k + 3) * 2.0 ** -53 * mag).all()), float((err / mag).max())
        if pad:
            assert torch.equal(C[:, m:], before[:, m:])
