"""16-bit products on pairs of SMs (more than 128 rows) at the edges of their tiles and splits, against float64 on the same operands.

Bar: what is left is fp32 accumulation, sixteen terms an addition: (K / 16 + 8) x 2^-24 of the sum of the terms' magnitudes bounds it, and
additions that truncate in a row of random terms stay a hundredth of that; 1e-5 of it, as for the other tensor-core products."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("M,N,K", [
    (129, 256, 8), (130, 264, 136), (256, 256, 64), (257, 300, 1000), (384, 1000, 72),      # rows of the second SM missing, ragged ends
    (512, 2560, 4096), (509, 2560, 9728), (512, 2592, 2560), (200, 512, 16384),               # split along k
    (512, 6176, 2560), (2048, 2576, 512), (2047, 5000, 264)])                                 # several tiles a pair
def test_pair_products(lib, pkg, dtype, M, N, K):
    g = torch.Generator().manual_seed(M + N)
    dt = getattr(torch, dtype)
    lda, ldb = K + 8, K + 16
    A, B = torch.randn(M, lda, generator=g).to(dt).cuda(), torch.randn(N, ldb, generator=g).to(dt).cuda()
    R = torch.randn(M, N, generator=g).cuda()
    A[:, K:] = float("nan")                                   # beyond K: never part of a sum
    B[:, K:] = float("nan")
    want = A[:, :K].double() @ B[:, :K].double().T
    size = A[:, :K].double().abs() @ B[:, :K].double().abs().T
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    fn = lib.b200_gemm_f16 if dtype == "float16" else lib.b200_gemm_bf16
    for resid in (False, True, True):
        c = torch.full((M + 1, N + 3), 7.0, device="cuda")
        a = pkg.GemmArgs()
        a.A, a.a_row, a.a_col, a.B, a.b_row, a.b_col = A.data_ptr(), lda, 1, B.data_ptr(), 1, ldb
        a.C, a.ldc, a.M, a.N, a.K, a.alpha, a.d_err = c.data_ptr(), N + 3, M, N, K, 0.5, err.data_ptr()
        if resid:
            a.R, a.ldr = R.data_ptr(), N
        assert fn(C.byref(a), None) == 0
        torch.cuda.synchronize()
        assert int(err) == 0 and (c[M] == 7.0).all() and (c[:, N:] == 7.0).all()
        w = want * 0.5 + (R.double() if resid else 0)
        assert ((c[:M, :N].double() - w).abs() <= 1e-5 * size + 1e-6).all()
    if dtype == "bfloat16" and N % 8 == 0:
        for relu2 in (0, 1):
            h = torch.zeros(M, N, dtype=dt, device="cuda")
            a = pkg.GemmArgs()
            a.A, a.a_row, a.a_col, a.B, a.b_row, a.b_col = A.data_ptr(), lda, 1, B.data_ptr(), 1, ldb
            a.Ch, a.ldch, a.M, a.N, a.K, a.alpha, a.d_err, a.relu2 = h.data_ptr(), N, M, N, K, 1.0, err.data_ptr(), relu2
            assert fn(C.byref(a), None) == 0
            w = want.clamp(min=0).square() if relu2 else want
            bar = 2 ** -8 * w.abs() + (2 * want.abs() if relu2 else 1) * 1e-5 * size + 1e-6      # one bfloat16 rounding
            assert ((h.double() - w).abs() <= bar).all() and int(err) == 0


# as pairs: one wave of tiles, split in three, less than a step; as tiles of one SM: a ragged end, several widths, many rows
@pytest.mark.parametrize("M,N,K", [(512, 19456, 2560), (300, 768, 3000), (130, 264, 136), (257, 300, 1000), (384, 3072, 512), (384, 4096, 512),
                                    (2048, 1024, 256)])
def test_products_on_either_side_of_the_cost_model(lib, pkg, M, N, K):
    """Two forms share these products by modelled time; both are held against float64 on shapes that the model gives them."""
    g = torch.Generator().manual_seed(M + N)
    A, B, R = torch.randn(M, K, generator=g).half().cuda(), torch.randn(N, K, generator=g).half().cuda(), torch.randn(M, N, generator=g).cuda()
    err, outs = torch.zeros(1, dtype=torch.int32, device="cuda"), []
    for _ in range(2):
        c = R.clone()
        a = pkg.GemmArgs()
        a.A, a.a_row, a.a_col, a.B, a.b_row, a.b_col = A.data_ptr(), K, 1, B.data_ptr(), 1, K
        a.C, a.ldc, a.R, a.ldr, a.M, a.N, a.K, a.alpha, a.d_err = c.data_ptr(), N, c.data_ptr(), N, M, N, K, 0.5, err.data_ptr()      # in place
        assert lib.b200_gemm_f16(C.byref(a), None) == 0
        torch.cuda.synchronize()
        outs.append(c)
    size = A.double().abs() @ B.double().abs().T
    assert int(err) == 0 and torch.equal(outs[0], outs[1])
    assert ((outs[0].double() - (0.5 * (A.double() @ B.double().T) + R.double())).abs() <= 1e-5 * size + 1e-6).all()
