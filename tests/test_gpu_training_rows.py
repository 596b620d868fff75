"""Row steps of training at the edges of their fast forms (whole aligned quads, rows that a block holds in registers), against float64.

Bars: sums of up to 4097 fp32 squares in 17 levels and strides of 256, 2^-19 of the value; single values a few ulp of expf / tanhf, 2^-20."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [1024, 1025, 2560, 2561, 4096, 4097])
@pytest.mark.parametrize("rows", [1, 5])
def test_norms(lib, dim, rows):
    g = torch.Generator().manual_seed(dim)
    x, dy, old = (torch.randn(rows, dim + (3 if k == 1 else 0), generator=g).cuda() for k in range(3))
    gamma = (1 + 0.1 * torch.randn(dim, generator=g)).cuda()
    out, half = torch.empty(rows, dim, device="cuda"), torch.empty(rows, dim, dtype=torch.float16, device="cuda")
    assert lib.b200_rms_norm_rows_h(x.data_ptr(), gamma.data_ptr(), out.data_ptr(), half.data_ptr(), rows, dim, 1e-6, None) == 0
    xd = x.double().requires_grad_()
    want = xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-6) * gamma.double()
    assert ((out.double() - want).abs() <= 2 ** -19 * want.abs()).all() and torch.equal(half, out.half())
    want.backward(dy[:, :dim].double())
    for accumulate, clamp in ((0, 0.0), (1, 1.5)):
        dx, dh = old.clone(), torch.empty(rows, dim, dtype=torch.float16, device="cuda")
        assert lib.b200_rms_norm_bwd_rows_h(x.data_ptr(), dy.data_ptr(), dim + 3, gamma.data_ptr(), dx.data_ptr(), rows, dim, 1e-6, accumulate, clamp,
                                            dh.data_ptr(), 4.0, None) == 0
        torch.cuda.synchronize()
        full = xd.grad + (old.double() if accumulate else 0)
        w = full.clamp(-clamp, clamp) if clamp else full
        assert ((dx.double() - w).abs() <= 2 ** -19 * (full.abs() + x.double().abs() + dy[:, :dim].double().abs())).all()
        assert torch.equal(dh, (dx * 4).half())


@pytest.mark.parametrize("kind", ["silu", "gelu"])
@pytest.mark.parametrize("rows,inter", [(1, 4), (3, 6), (2, 1024), (5, 1028), (3, 1026), (2, 9728)])
def test_gated_activations(lib, kind, rows, inter):
    g = torch.Generator().manual_seed(inter)
    gu, dy = (2 * torch.randn(rows, 2 * inter, generator=g)).cuda(), torch.randn(rows, inter, generator=g).cuda()
    gd = gu.double().requires_grad_()
    a, u = gd[:, :inter], gd[:, inter:]
    act = a * torch.sigmoid(a) if kind == "silu" else 0.5 * a * (1 + torch.tanh(0.7978845608 * (a + 0.044715 * a ** 3)))
    (act * u).backward(dy.double())
    want = (act * u).detach()
    out, half = torch.empty(rows, inter, device="cuda"), torch.empty(rows, inter, dtype=torch.float16, device="cuda")
    d, dh = torch.empty(rows, 2 * inter, device="cuda"), torch.empty(rows, 2 * inter, dtype=torch.float16, device="cuda")
    if kind == "silu":
        assert lib.b200_silu_mul_rows_h(gu.data_ptr(), rows, inter, out.data_ptr(), half.data_ptr(), None) == 0
        assert lib.b200_silu_mul_bwd_rows_h(dy.data_ptr(), gu.data_ptr(), rows, inter, d.data_ptr(), dh.data_ptr(), 8.0, None) == 0
    else:
        assert lib.b200_gelu_mul_rows(gu.data_ptr(), rows, inter, out.data_ptr(), None) == 0
        assert lib.b200_gelu_mul_bwd_rows(dy.data_ptr(), gu.data_ptr(), rows, inter, d.data_ptr(), None) == 0
    torch.cuda.synchronize()
    size = (gu[:, :inter] * gu[:, inter:]).double().abs()                  # gelu: 1 + tanh cancels for negative arguments
    assert ((out.double() - want).abs() <= 2 ** -20 * (want.abs() + (size if kind == "gelu" else 0))).all()
    slope = torch.cat([dy.double() * gu[:, inter:].double(), dy.double() * gu[:, :inter].double()], 1).abs() * (1 + gu[:, :inter].double().abs().repeat(1, 2) ** 3)
    assert ((d.double() - gd.grad).abs() <= 2 ** -20 * (gd.grad.abs() + slope)).all()
    if kind == "silu":
        assert torch.equal(half, out.half()) and torch.equal(dh, (d * 8).half())


@pytest.mark.parametrize("rank,off", [(16, 0), (16, 1), (8, 0), (5, 0), (64, 0), (33, 0)])
@pytest.mark.parametrize("rows,cols", [(1, 1), (8, 256), (13, 300)])
def test_lora_add(lib, rank, off, rows, cols):
    g = torch.Generator().manual_seed(rank + cols)
    y, mid = torch.randn(rows, cols + 7, generator=g).cuda(), torch.randn(rows, rank + 2, generator=g).cuda()
    B = torch.zeros(cols * rank + 4, device="cuda")[off:off + cols * rank].view(cols, rank)
    B.copy_(torch.randn(cols, rank, generator=g))
    got = y.clone()
    assert lib.b200_lora_add(got.data_ptr(), cols + 7, 3, cols, mid.data_ptr(), rank + 2, B.data_ptr(), rank, 2.0, rows, None) == 0
    torch.cuda.synchronize()
    want = y.double().clone()
    want[:, 3:3 + cols] += 2 * mid[:, :rank].double() @ B.double().T
    size = y.double().abs()
    size[:, 3:3 + cols] += 2 * mid[:, :rank].double().abs() @ B.double().abs().T
    assert ((got.double() - want).abs() <= 2 ** -20 * size).all()
    assert torch.equal(got[:, :3], y[:, :3]) and torch.equal(got[:, 3 + cols:], y[:, 3 + cols:])


@pytest.mark.parametrize("rows", [1, 9])
@pytest.mark.parametrize("inter", [64, 252, 256, 260, 1024])
def test_gated_activations_in_both_forms(lib, rows, inter):
    """Either side of the width from which rows go in quads: operands on a 16-byte boundary and off it (always by elements) give the same bits."""
    g = torch.Generator().manual_seed(inter)
    gu, dy = 2 * torch.randn(rows * 2 * inter, generator=g), torch.randn(rows * inter, generator=g)
    got = []
    for off in (0, 2):                                       # pairs are read 8 bytes at a time in every form
        placed = [torch.zeros(t.numel() + 4).index_copy_(0, torch.arange(off, off + t.numel()), t).cuda() for t in (gu, dy)]
        at, back = (p.data_ptr() + 4 * off for p in placed)
        assert placed[0].data_ptr() % 16 == 0
        one, two = (torch.full((rows, n), float("nan"), device="cuda") for n in (inter, 2 * inter))
        half, pair = (t.half() for t in (one, two))
        gelu, slopes, rows_half = one.clone(), two.clone(), one.bfloat16()
        assert lib.b200_silu_mul_rows_h(at, rows, inter, one.data_ptr(), half.data_ptr(), None) == 0
        assert lib.b200_silu_mul_bwd_rows_h(back, at, rows, inter, two.data_ptr(), pair.data_ptr(), 8.0, None) == 0
        assert lib.b200_gelu_mul_rows(at, rows, inter, gelu.data_ptr(), None) == 0
        assert lib.b200_gelu_mul_bwd_rows(back, at, rows, inter, slopes.data_ptr(), None) == 0
        assert lib.b200_rows_gelu_mul(at, 2 * inter, rows, inter, 2, rows_half.data_ptr(), None) == 0
        torch.cuda.synchronize()
        got.append((one, two, half, pair, gelu, slopes, rows_half))
    for a, b in zip(*got):
        assert not torch.isnan(a).any() and torch.equal(a, b)
