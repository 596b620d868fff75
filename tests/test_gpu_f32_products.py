"""The CUDA-core fp32 product in every orientation at the edges of its tiles and splits, against float64 on the same operands.

Bar: K fp32 additions in a random walk, 2^-20 of the sum of the terms' magnitudes."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ak", [0, 1])
@pytest.mark.parametrize("bk", [0, 1])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (64, 64, 32), (65, 63, 33), (64, 1152, 6912), (64, 130, 1000), (7, 16, 2048), (1152, 300, 64)])
def test_f32_products(lib, pkg, ak, bk, M, N, K):
    g = torch.Generator().manual_seed(K + 3 * M)
    A, B, R = (torch.randn(*s, generator=g).cuda() for s in ((M, K), (K, N), (M, N)))
    a_mem, b_mem = (A.contiguous() if ak else A.T.contiguous()), (B.T.contiguous() if bk else B.contiguous())
    want, size = A.double() @ B.double(), A.double().abs() @ B.double().abs()
    outs = []
    for round_f16 in (0, 0, 1):
        c = R.clone()
        a = pkg.GemmArgs()
        a.A, a.a_row, a.a_col = a_mem.data_ptr(), K if ak else 1, 1 if ak else M
        a.B, a.b_row, a.b_col = b_mem.data_ptr(), 1 if bk else N, K if bk else 1
        a.C, a.ldc, a.R, a.ldr = c.data_ptr(), N, c.data_ptr(), N                   # in place
        a.M, a.N, a.K, a.alpha, a.round_f16 = M, N, K, -0.25, round_f16
        assert lib.b200_gemm_f32(C.byref(a), None) == 0
        torch.cuda.synchronize()
        outs.append(c)
    assert ((outs[0].double() - (R.double() - 0.25 * want)).abs() <= 2 ** -20 * (size + R.double().abs())).all()
    assert torch.equal(outs[0], outs[1])                      # the splits add in a fixed order
    assert torch.equal(outs[2], outs[0].half().float())


@pytest.mark.parametrize("ak", [0, 1])
@pytest.mark.parametrize("bk", [0, 1])
@pytest.mark.parametrize("M,N,K,pad", [(64, 1152, 769, 0), (33, 200, 257, 1), (64, 64, 1030, 3), (130, 70, 96, 1), (1, 700, 4100, 2)])
def test_f32_products_off_boundaries(lib, pkg, ak, bk, M, N, K, pad):
    """Operands, results and residuals that start `pad` floats behind a 16-byte boundary, in wider lines. Bar as above."""
    g = torch.Generator().manual_seed(K + M)

    def placed(t):
        rows, cols = t.shape
        whole = torch.full((rows * (cols + pad) + 4,), float("nan"), device="cuda")
        view = whole[pad:pad + rows * (cols + pad)].view(rows, cols + pad)[:, :cols]
        view.copy_(t)
        return whole, view

    A, B, R = (torch.randn(*s, generator=g).cuda() for s in ((M, K), (K, N), (M, N)))
    (_a, am), (_b, bm), (_r, rm), (_c, cm) = placed(A if ak else A.T), placed(B.T if bk else B), placed(R), placed(torch.zeros_like(R))
    a = pkg.GemmArgs()
    a.A, a.a_row, a.a_col = am.data_ptr(), am.stride(0) if ak else 1, 1 if ak else am.stride(0)
    a.B, a.b_row, a.b_col = bm.data_ptr(), 1 if bk else bm.stride(0), bm.stride(0) if bk else 1
    a.C, a.ldc, a.R, a.ldr = cm.data_ptr(), cm.stride(0), rm.data_ptr(), rm.stride(0)
    a.M, a.N, a.K, a.alpha = M, N, K, 1.0
    assert lib.b200_gemm_f32(C.byref(a), None) == 0
    torch.cuda.synchronize()
    want, size = A.double() @ B.double() + R.double(), A.double().abs() @ B.double().abs() + R.double().abs()
    assert ((cm.double() - want).abs() <= 2 ** -20 * size).all()
    assert torch.isnan(_c).sum() == _c.numel() - M * N        # nothing outside the result is written


@pytest.mark.parametrize("ak", [0, 1])
@pytest.mark.parametrize("bk", [0, 1])
@pytest.mark.parametrize("M,N,K", [(64, 2240, 700), (60, 1536, 700), (64, 1300, 800), (64, 960, 900), (130, 350, 1290), (64, 512, 4096),     # 3, 5, 6, 7, 6 and 8 blocks per tile
                                    (64, 512, 1536), (64, 3840, 1152), (64, 1152, 511), (300, 1152, 256),                                # splits of the turning form
                                    (700, 3700, 33), (2432, 1024, 64)])                                                                    # one, in several waves
def test_f32_products_in_every_number_of_blocks(lib, pkg, ak, bk, M, N, K):
    """Rows that do not share out evenly over the blocks of a tile, short and long k, few and many tiles. Bar as above."""
    g = torch.Generator().manual_seed(N + K)
    A, B, R = (torch.randn(*s, generator=g).cuda() for s in ((M, K), (K, N), (M, N)))
    a_mem, b_mem = (A.contiguous() if ak else A.T.contiguous()), (B.T.contiguous() if bk else B.contiguous())
    c = torch.full((M + 1, N), 7.0, device="cuda")
    a = pkg.GemmArgs()
    a.A, a.a_row, a.a_col = a_mem.data_ptr(), K if ak else 1, 1 if ak else M
    a.B, a.b_row, a.b_col = b_mem.data_ptr(), 1 if bk else N, K if bk else 1
    a.C, a.ldc, a.R, a.ldr = c.data_ptr(), N, R.data_ptr(), N
    a.M, a.N, a.K, a.alpha = M, N, K, 0.5
    assert lib.b200_gemm_f32(C.byref(a), None) == 0
    torch.cuda.synchronize()
    want, size = 0.5 * (A.double() @ B.double()) + R.double(), A.double().abs() @ B.double().abs() + R.double().abs()
    assert ((c[:M].double() - want).abs() <= 2 ** -20 * size).all() and (c[M] == 7.0).all()
