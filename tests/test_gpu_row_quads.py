"""The row steps of a portion on rows of whole aligned quads, against float64: every number of quads a thread, parts of whole stretches, padding, earlier results.

Bars: a norm's square sum of up to 4096 fp32 terms added in 12 levels and stretches, 2^-20 of the value; bfloat16 results 2^-8; tanh and exp to a few ulp."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,ld,groups", [(4, 4, 1), (128, 128, 1), (132, 136, 1), (1024, 1024, 8), (1028, 1040, 1), (2048, 2048, 4), (2048, 2056, 16), (3072, 3072, 3), (4096, 4096, 1)])
@pytest.mark.parametrize("hist", [0, 1, 6])
def test_postnorm(lib, pkg, dim, ld, groups, hist):
    g, M = torch.Generator().manual_seed(dim + hist), 7

    def rows(n, pad=0):
        t = torch.full((M, n + pad), float("nan"))
        t[:, :dim] = torch.randn(M, dim, generator=g)
        return t.cuda()

    x, y, gate = rows(ld), rows(ld, 4), rows(ld, 8)
    bias, gamma = torch.randn(dim, generator=g).cuda(), torch.randn(dim, generator=g).cuda()
    hs, coef = torch.randn(max(hist, 1), M, ld, generator=g).cuda(), torch.randn(hist + 1, generator=g).cuda()
    post, out, half = (torch.full((M, ld), float("nan"), dtype=t, device="cuda") for t in (torch.float32, torch.float32, torch.bfloat16))
    a = pkg.RowsPostnormArgs()
    a.x, a.y, a.y_ld, a.gate, a.gate_ld, a.gate_bias, a.gamma = x.data_ptr(), y.data_ptr(), ld + 4, gate.data_ptr(), ld + 8, bias.data_ptr(), gamma.data_ptr()
    a.alpha, a.eps, a.rows, a.dim, a.ld, a.groups, a.norm_out = 1.5, 1e-4, M, dim, ld, groups, post.data_ptr()
    a.hist, a.hist_n, a.hist_stride, a.coef, a.out, a.out_h = hs.data_ptr(), hist, M * ld, coef.data_ptr(), out.data_ptr(), half.data_ptr()
    assert lib.b200_rows_postnorm(C.byref(a), None) == 0
    torch.cuda.synchronize()
    z = 1.5 * x[:, :dim].double() + torch.sigmoid(gate[:, :dim].double() + bias.double()) * y[:, :dim].double()
    parts = z.view(M, groups, -1)
    n = (parts * torch.rsqrt(parts.square().mean(-1, keepdim=True) + 1e-4)).view(M, dim) * gamma.double()
    want = n * coef[hist].double() + sum(coef[j].double() * hs[j, :, :dim].double() for j in range(hist)) if hist else n
    size = n.abs() + (want.abs() + sum(abs(float(coef[j])) * hs[j, :, :dim].double().abs() for j in range(hist)) if hist else 0)
    assert ((post[:, :dim].double() - n).abs() <= 2 ** -20 * (n.abs() + gamma.abs().double())).all()
    assert ((out[:, :dim].double() - want).abs() <= 2 ** -20 * (size + gamma.abs().double() * (1 + coef.abs().max().double()))).all()
    assert torch.equal(half[:, :dim], out[:, :dim].bfloat16())
    assert not post[:, dim:].any() and not out[:, dim:].any() and not half[:, dim:].any()


@pytest.mark.parametrize("dim,ld,groups", [(4, 4, 1), (132, 136, 1), (256, 256, 2), (1024, 1024, 8), (1028, 1040, 1), (1152, 1152, 3), (2048, 2048, 4), (2048, 2056, 16), (3072, 3072, 3),
                                           (4096, 4096, 1), (4096, 4096, 32)])
@pytest.mark.parametrize("hist", [0, 3])
def test_postnorm_adds_in_one_order(lib, pkg, dim, ld, groups, hist):
    """The same rows with one operand off the 16-byte boundary take the form of single elements: the same bits."""
    g, M = torch.Generator().manual_seed(dim + hist), 5
    x, gate = (torch.randn(M, ld, generator=g).cuda() for _ in range(2))
    y = torch.zeros(2, M * ld + 8, device="cuda")
    y[0, :M * ld] = torch.randn(M * ld, generator=g).cuda()
    y[1, 1:M * ld + 1] = y[0, :M * ld]
    bias, gamma = torch.randn(dim, generator=g).cuda(), torch.randn(dim, generator=g).cuda()
    hs, coef = torch.randn(max(hist, 1), M, ld, generator=g).cuda(), torch.randn(hist + 1, generator=g).cuda()
    post, out, half = (torch.full((2, M, ld), float("nan"), dtype=t, device="cuda") for t in (torch.float32, torch.float32, torch.bfloat16))
    for k in range(2):
        a = pkg.RowsPostnormArgs()
        a.x, a.y, a.y_ld, a.gate, a.gate_ld, a.gate_bias, a.gamma = x.data_ptr(), y[k].data_ptr() + 4 * k, ld, gate.data_ptr(), ld, bias.data_ptr(), gamma.data_ptr()
        a.alpha, a.eps, a.rows, a.dim, a.ld, a.groups, a.norm_out = 1.5, 1e-4, M, dim, ld, groups, post[k].data_ptr()
        a.hist, a.hist_n, a.hist_stride, a.coef, a.out, a.out_h = hs.data_ptr(), hist, M * ld, coef.data_ptr(), out[k].data_ptr(), half[k].data_ptr()
        assert y[k].data_ptr() % 16 == 0 and lib.b200_rows_postnorm(C.byref(a), None) == 0
    torch.cuda.synchronize()
    for t in (post, out, half):
        assert not torch.isnan(t).any() and torch.equal(t[0], t[1])


@pytest.mark.parametrize("wtype", [2, 3])
@pytest.mark.parametrize("rows,inter,pad", [(1, 4, 0), (3, 1020, 4), (5, 1024, 0), (2, 1028, 8), (33, 6144, 0), (3, 10, 2), (3, 12, 6)])
def test_gelu_mul(lib, wtype, rows, inter, pad):
    g = torch.Generator().manual_seed(inter)
    gu = (3 * torch.randn(rows, 2 * inter + pad, generator=g)).cuda()
    out = torch.full((rows + 1, inter), float("nan"), dtype=torch.bfloat16 if wtype == 2 else torch.float32, device="cuda")
    assert lib.b200_rows_gelu_mul(gu.data_ptr(), 2 * inter + pad, rows, inter, wtype, out.data_ptr(), None) == 0
    torch.cuda.synchronize()
    z, u = gu[:, 0:2 * inter:2].double(), gu[:, 1:2 * inter:2].double()
    want = 0.5 * z * (1 + torch.tanh(0.7978845608028654 * (z + 0.044715 * z ** 3))) * u
    bar = (2 ** -8 if wtype == 2 else 2 ** -20) * (want.abs() + (z * u).abs() * 2 ** -3)
    assert ((out[:rows].double() - want).abs() <= bar).all()
    assert torch.isnan(out[rows]).all()
