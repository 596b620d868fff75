"""The per-token products' input, assembled by all threads of a block, and their outputs in windows of rows, against float64.

Bars: a sum of fp32 products passes at most 64 additions of a thread, 5 of a warp's tree and 30 of warps, and the input's norms as many again: 2^-24 each, below
2^-16 of the terms' magnitude together."""
import ctypes as C

import numpy as np
import pytest

import test_gpu_hybrid_kernels as H
import test_gpu_latent_kernels as K

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
Q8, F16, BF16, F32 = 0, 1, 2, 3
BAR = 2.0 ** -16


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()


def packed(lib, w, wtype):
    """Rows as the kernel reads them and the values they hold."""
    rows, cols = w.shape
    stride = lib.b200_packed_row_stride(wtype, cols)
    d, src = torch.zeros(rows, stride, dtype=torch.uint8, device="cuda"), dev(w)
    call = lib.b200_q8_pack if wtype == Q8 else lib.b200_f16_pack
    assert call(src.data_ptr(), cols, rows, cols, d.data_ptr(), stride, 0, 1, None) == 0
    torch.cuda.synchronize()
    if wtype == F16:
        return d, stride, src.half().double()
    raw = d.cpu().numpy()
    quants = raw[:, :cols].view(np.int8).astype(np.float64)
    scales = np.ascontiguousarray(raw[:, cols:cols + cols // 16]).view(np.float16).astype(np.float64)
    return d, stride, torch.from_numpy(quants * np.repeat(scales, 32, axis=1)).cuda()


def resid_call(lib, pkg, d, stride, rows, cols, wtype, resid, slots, norm_at, final, grid=0, out_mode=None):
    a = pkg.MatvecArgs()
    a.d_w, a.row_stride, a.rows, a.cols, a.wtype, a.in_mode, a.out_mode, a.n_out, a.eps, a.grid = d.data_ptr(), stride, rows, cols, wtype, pkg.B200_IN_RESID, \
        pkg.B200_OUT_STORE if out_mode is None else out_mode, 1, 1e-5, grid
    out, kept = torch.full((rows,), float("nan"), device="cuda"), torch.full((cols,), float("nan"), device="cuda")
    a.d_out[0], a.d_resid_in, a.d_resid_out, a.n_slots, a.slot_stride = out.data_ptr(), resid.data_ptr(), kept.data_ptr(), len(slots), cols
    a.d_slots = slots.data_ptr() if len(slots) else None
    a.d_slot_norm_gamma = norm_at
    a.d_norm_gamma = final.data_ptr() if final is not None else None
    assert lib.b200_matvec(C.byref(a), None) == 0
    torch.cuda.synchronize()
    return out, kept


@pytest.mark.parametrize("wtype", [Q8, F16])
@pytest.mark.parametrize("cols", [32, 512, 2560, 4096, 5120, 9728])
@pytest.mark.parametrize("grid", [0, 3])
def test_slot_norm_weights_on_any_element(lib, pkg, wtype, cols, grid):
    """The weights of the slots' norm one to three elements behind a 16-byte boundary: the same bits."""
    g = torch.Generator().manual_seed(cols)
    w = torch.randn(37, cols, generator=g).numpy()
    d, stride, _ = packed(lib, w, wtype)
    resid, slots, gamma = torch.randn(cols, generator=g).cuda(), torch.randn(2, cols, generator=g).cuda(), torch.randn(cols, generator=g)
    got = []
    for off in range(4):
        room = torch.full((cols + 8,), float("nan"))
        room[off:off + cols] = gamma
        room = room.cuda()
        assert room.data_ptr() % 16 == 0
        got.append(resid_call(lib, pkg, d, stride, 37, cols, wtype, resid, slots, room.data_ptr() + 4 * off, None, grid))
    for out, kept in got:
        assert not torch.isnan(out).any() and torch.equal(out, got[0][0]) and torch.equal(kept, got[0][1])


def normed(v, weights):
    return weights * v * torch.rsqrt(v.square().mean() + 1e-5)


@pytest.mark.parametrize("wtype", [Q8, F16])
@pytest.mark.parametrize("cols", [32, 2560, 4096, 5120, 9728])
@pytest.mark.parametrize("n_slots,slot_norm,final", [(0, False, True), (1, False, False), (3, False, True), (2, True, False), (2, True, True)])
def test_residual_input(lib, pkg, wtype, cols, n_slots, slot_norm, final):
    """Vectors of up to five quads a thread: the residual kept and the product of what is assembled."""
    g = torch.Generator().manual_seed(cols + n_slots)
    d, stride, w = packed(lib, torch.randn(37, cols, generator=g).numpy(), wtype)
    resid, slots = 2 * torch.randn(cols, generator=g).cuda(), torch.randn(n_slots, cols, generator=g).cuda()
    sg, fg = (torch.randn(cols, generator=g).cuda() for _ in range(2))
    out, kept = resid_call(lib, pkg, d, stride, 37, cols, wtype, resid, slots, sg.data_ptr() if slot_norm else None, fg if final else None)
    add = slots.double().sum(0) if n_slots else torch.zeros_like(resid, dtype=torch.float64)
    add = normed(add, sg.double()) if slot_norm else add
    want = resid.double() + add
    assert ((kept.double() - want).abs() <= BAR * (resid.abs().double() + add.abs() + slots.abs().double().sum(0))).all()
    x = normed(want, fg.double()) if final else want
    assert ((out.double() - w @ x).abs() <= BAR * (w.abs() @ x.abs())).all()


@pytest.mark.parametrize("wtype", [BF16, F32])
@pytest.mark.parametrize("cols", [8, 64, 2560, 5120, 15360])
@pytest.mark.parametrize("n_slots,final", [(0, True), (3, False), (3, True)])
@pytest.mark.parametrize("grid", [0, 3])
def test_residual_input_of_other_types(lib, pkg, wtype, cols, n_slots, final, grid):
    """Stored sums and gated pairs; the norm over the whole vector, which has a kernel without parts."""
    g = torch.Generator().manual_seed(cols + n_slots)
    w = torch.randn(38, cols, generator=g).bfloat16().double()
    d, stride = K.pack(lib, w.numpy(), wtype, cols)
    w = w.cuda()
    resid, slots, fg = 2 * torch.randn(cols, generator=g).cuda(), torch.randn(n_slots, cols, generator=g).cuda(), torch.randn(cols, generator=g).cuda()
    want = resid.double() + (slots.double().sum(0) if n_slots else 0)
    x = normed(want, fg.double()) if final else want
    y, size = w @ x, w.abs() @ x.abs()
    out, kept = resid_call(lib, pkg, d, stride, 38, cols, wtype, resid, slots, None, fg if final else None, grid)
    assert ((kept.double() - want).abs() <= BAR * (resid.abs().double() + slots.abs().double().sum(0))).all()
    assert ((out.double() - y).abs() <= BAR * size).all()
    pairs, kept2 = resid_call(lib, pkg, d, stride, 38, cols, wtype, resid, slots, None, fg if final else None, grid, pkg.B200_OUT_GLU)
    act = y[0::2] * torch.sigmoid(y[0::2])
    assert ((pairs[:19].double() - act * y[1::2]).abs() <= BAR * (1.1 * size[0::2] * y[1::2].abs() + act.abs() * size[1::2] + (act * y[1::2]).abs())).all()
    assert torch.equal(kept, kept2) and torch.isnan(pairs[19:]).all()


@pytest.mark.parametrize("wtype", [Q8, F16])
@pytest.mark.parametrize("grid", [1, 2])
def test_pairs_in_several_windows(lib, pkg, wtype, grid):
    """One or two blocks for 3001 pairs: several windows of rows, several rows a thread."""
    g, rows, cols = torch.Generator().manual_seed(4), 6002, 64
    d, stride, w = packed(lib, 0.2 * torch.randn(rows, cols, generator=g).numpy(), wtype)
    x, out = torch.randn(cols, generator=g).cuda(), torch.full((rows // 2,), float("nan"), device="cuda")
    a = pkg.MatvecArgs()
    a.d_w, a.row_stride, a.rows, a.cols, a.wtype, a.in_mode, a.out_mode, a.n_out, a.grid = d.data_ptr(), stride, rows, cols, wtype, pkg.B200_IN_VEC, pkg.B200_OUT_GLU, 1, grid
    a.d_in_vec, a.d_out[0] = x.data_ptr(), out.data_ptr()
    assert lib.b200_matvec(C.byref(a), None) == 0
    torch.cuda.synchronize()
    y, size = w @ x.double(), w.abs() @ x.abs().double()
    gate, up = y[0::2], y[1::2]
    act = gate * torch.sigmoid(gate)                          # slope at most 1.1
    assert ((out.double() - act * up).abs() <= BAR * (1.1 * size[0::2] * up.abs() + act.abs() * size[1::2] + (act * up).abs())).all()


@pytest.mark.parametrize("wtype", [BF16, F32])
@pytest.mark.parametrize("grid", [1, 2])
def test_gates_and_streams_in_several_windows(lib, pkg, wtype, grid):
    """What a gated output adds, and the streams of a row, are fetched again for every window and for a thread's later rows."""
    g, rows, cols = np.random.default_rng(9), 5003, 40
    w, x, res, gate, bias = (g.standard_normal(s) for s in ((rows, cols), cols, rows, rows, rows))
    w, x = K.o.bf16(w), x.astype(np.float32).astype(np.float64)
    n = K.up8(rows)
    out = K.zeros(n)
    assert K.matvec(lib, pkg, w, wtype, cols, rows, d_in_vec=K.dev(x), out_mode=pkg.B200_OUT_GATED, d_out_resid=K.dev(res), d_out_gate=K.dev(gate),
                    d_out_gate_bias=K.dev(bias), resid_alpha=2.5, d_out=out, grid=grid) == 0
    size = np.abs(w) @ np.abs(x) + 2.5 * np.abs(res)
    assert (np.abs(K.host(out)[:rows] - (2.5 * res + K.o.logistic(gate + bias) * (w @ x))) <= BAR * size).all()
    assert not K.host(out)[rows:].any()
    for ns in (3, 8):
        c, old = H.connect(g, ns), g.standard_normal((ns, rows))
        new, u = H.zeros(ns, n), H.zeros(n)
        assert H.matvec(lib, pkg, w, wtype, d_in_vec=H.dev(x), out_mode=pkg.B200_OUT_STREAMS, d_out=u, d_streams_in=H.dev(H.padded(old, n)), streams_in_stride=n,
                        d_streams_out=new, streams_out_stride=n, d_connect=c[1], n_streams=ns, grid=grid) == 0
        want = H.o.connect(old[:, None], c[0], lambda u: u, lambda u: (w @ x)[None])[:, 0]
        terms = np.abs(c[0]["mix"]).T @ np.abs(old) + np.abs(c[0]["out"])[:, None] * (np.abs(w) @ np.abs(x))
        assert (np.abs(H.host(new)[:, :rows] - want) <= BAR * terms).all()
        assert (np.abs(H.host(u)[:rows] - c[0]["in"] @ want) <= BAR * (np.abs(c[0]["in"]) @ terms)).all()
        assert not H.host(new)[:, rows:].any() and not H.host(u)[rows:].any()
