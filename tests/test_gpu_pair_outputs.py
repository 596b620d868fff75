"""What a pair product does with a sum on its way out, bit for bit: the sums themselves come from a launch with alpha 1 and nothing added, the rest is one
rounding for alpha, one for what is added, one for bfloat16. Widths and rows that end inside a block of 32 x 32 and inside a quad, rows that start
off a 16-byte boundary, tiles of every width that the model gives, one and several a pair, and splits."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SHAPES = [(129, 256, 64), (200, 257, 136), (259, 302, 264), (777, 2575, 256), (777, 6144, 256), (509, 2560, 4096), (192, 12296, 512), (1531, 2561, 1024), (513, 9736, 8)]


def product(lib, pkg, A, B, c, ldc, alpha, R=None, ldr=0, half=None, relu2=0):
    M, K = A.shape
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    a = pkg.GemmArgs()
    a.A, a.a_row, a.a_col, a.B, a.b_row, a.b_col = A.data_ptr(), K, 1, B.data_ptr(), 1, K
    a.M, a.N, a.K, a.alpha, a.d_err, a.relu2 = M, B.shape[0], K, alpha, err.data_ptr(), relu2
    if half is None:
        a.C, a.ldc = c, ldc
    else:
        a.Ch, a.ldch = half.data_ptr(), ldc
    if R is not None:
        a.R, a.ldr = R, ldr
    assert (lib.b200_gemm_bf16 if A.dtype == torch.bfloat16 else lib.b200_gemm_f16)(C.byref(a), None) == 0
    torch.cuda.synchronize()
    assert int(err) == 0


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_fp32_results(lib, pkg, M, N, K):
    g = torch.Generator().manual_seed(M + N)
    A, B = torch.randn(M, K, generator=g).half().cuda(), torch.randn(N, K, generator=g).half().cuda()
    alpha = torch.tensor(0.37, device="cuda")
    for off, pad in ((0, -N % 4), (1, 5)):                    # rows on 16-byte boundaries, and off them
        ld = N + pad
        buf = torch.full((3, M * ld + 8), 7.0, device="cuda")
        R = torch.randn(M * ld + 8, generator=g).cuda()
        rows = [b[off:off + M * ld].view(M, ld) for b in buf]
        where = R[off:off + M * ld].view(M, ld)
        at = [b.data_ptr() + 4 * off for b in buf]
        product(lib, pkg, A, B, at[0], ld, 1.0)
        product(lib, pkg, A, B, at[1], ld, 0.37)
        product(lib, pkg, A, B, at[2], ld, 0.37, R.data_ptr() + 4 * off, ld)
        sums = rows[0][:, :N]
        assert torch.equal(rows[1][:, :N], sums * alpha)
        assert torch.equal(rows[2][:, :N], sums * alpha + where[:, :N])
        for r, b in zip(rows, buf):
            assert (r[:, N:] == 7.0).all() and (b[:off] == 7.0).all() and (b[off + M * ld:] == 7.0).all()
        want = A.double() @ B.double().T
        assert ((sums.double() - want).abs() <= 1e-5 * (A.double().abs() @ B.double().abs().T) + 1e-6).all()


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("relu2", [0, 1])
def test_bfloat16_results(lib, pkg, M, N, K, relu2):
    g = torch.Generator().manual_seed(M + N)
    A, B = torch.randn(M, K, generator=g).bfloat16().cuda(), torch.randn(N, K, generator=g).bfloat16().cuda()
    ld = (N + 15) // 8 * 8
    half = torch.full((M + 1, ld), 7.0, dtype=torch.bfloat16, device="cuda")
    product(lib, pkg, A, B, None, ld, 1.0, half=half, relu2=relu2)
    want = A.double() @ B.double().T
    size = A.double().abs() @ B.double().abs().T
    w = want.clamp(min=0).square() if relu2 else want
    bar = 2 ** -8 * w.abs() + (2 * want.abs() if relu2 else 1) * 1e-5 * size + 1e-6 + (1e-5 * size) ** 2
    assert ((half[:M, :N].double() - w).abs() <= bar).all()
    assert (half[M] == 7.0).all() and (half[:M, N:] == 7.0).all()
