"""Prompts in passes over the weights: the products, row kernels and attention of the Qwen3 / Gemma3 row path, each against the
same sums in float64, and whole prompts against the per-token path.

Bars. Two binary16 planes carry 22 bits of an element. Tensor cores truncate the accumulator at 2^-24 of its size with every
addition, at most 256 of them in a row: 256 x 2^-25 = 8e-6 of a result (measured up to 5e-6 on these inputs, whose terms differ by orders of
magnitude); bar 1e-5. One plane is the plain binary16 rounding of the activations: 2^-12 rms of each term, measured 2e-4, bar 6e-4."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_kernels import dev, pack, weights

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def planes_buffer(pkg, rows, cap, cols, planes, scaled=True):
    x = torch.full((planes * cap, cols), float("nan"), dtype=torch.float16, device="cuda")      # rows nobody wrote must not matter
    scale = torch.zeros(cap, dtype=torch.float32, device="cuda") if scaled else None
    return x, scale, pkg.RowPlanes(x.data_ptr(), cols, planes, cap, scale.data_ptr() if scaled else None)


def rel(a, b):
    a, b = a.double().cpu(), b.double().cpu()
    return float((a - b).norm() / b.norm())


def q8_values(lib, d_w, stride, rows, cols):
    raw = d_w.view(rows, stride)
    q = raw[:, :cols].contiguous().view(torch.int8).double().view(rows, cols // 32, 32)
    d = raw[:, cols:cols + cols // 16].contiguous().view(torch.float16).double()
    return (q * d[..., None]).view(rows, cols)


@pytest.mark.parametrize("wtype", ["q8", "f16"])
@pytest.mark.parametrize("planes", [2, 1])
@pytest.mark.parametrize("rows,cols,n", [
    (128, 64, 1), (136, 96, 16), (64, 32, 3),              # less than a tile, half a step of 64 columns
    (2560, 2560, 17), (512, 1536, 15), (6144, 2560, 33),   # few rows of x, tiles shared by clusters
    (1152, 6912, 130), (2560, 9728, 255), (2560, 4096, 257), (19456, 2560, 48), (1000, 2592, 512), (19456, 2560, 509), (384, 4096, 1531)])
def test_products(lib, pkg, synth, wtype, planes, rows, cols, n):
    wt = pkg.B200_WT_Q8 if wtype == "q8" else pkg.B200_WT_F16
    w = weights(synth, rows, cols, 3)
    w[:, : cols // 2] *= 10.0 ** (np.arange(rows) % 9 - 4)[:, None].astype(np.float32)      # rows and blocks of very different size
    d_w, stride = pack(lib, pkg, w, wt)
    exact_w = q8_values(lib, d_w, stride, rows, cols) if wtype == "q8" else d_w.view(torch.float16).view(rows, stride // 2)[:, :cols].double()
    g = torch.Generator().manual_seed(rows + n)
    x = torch.randn(n, cols, generator=g) * torch.exp(torch.randn(n, cols, generator=g))
    if planes == 2:
        x *= 10.0 ** (torch.arange(n) % 13 - 6)[:, None]   # one plane has no factor: binary16's own range
    x = x.cuda()
    cap = n + 5
    px, scale, args = planes_buffer(pkg, n, cap, cols, planes, planes == 2)
    assert lib.b200_rows_split_planes(x.data_ptr(), n, cols, C.byref(args), None) == 0
    ws = torch.zeros(rows, dtype=torch.float32, device="cuda")
    if wtype == "q8":
        assert lib.b200_q8_row_scale(d_w.data_ptr(), stride, rows, cols, ws.data_ptr(), None) == 0
    resid = torch.randn(n, rows, generator=g).cuda() * 1e-3
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    want = x.double() @ exact_w.T
    for use_resid in (False, True):
        out = torch.full((n + 1, rows), float("nan"), device="cuda")
        a = pkg.RowsMatmulArgs(wt, d_w.data_ptr(), stride, rows, cols, ws.data_ptr(), px.data_ptr(), cols, planes, cap,
                               scale.data_ptr() if scale is not None else None, n, out.data_ptr(), rows,
                               resid.data_ptr() if use_resid else None, rows, err.data_ptr(), 0)
        assert lib.b200_rows_matmul(C.byref(a), None) == 0
        torch.cuda.synchronize()
        assert int(err) == 0
        assert torch.isnan(out[n]).all()                   # nothing beyond the rows asked for
        bar = 1e-5 if planes == 2 else 6e-4
        full = want + resid.double() if use_resid else want
        # every row of x and of w on its own: neither may lean on a larger one
        by_x = (out[:n].double() - full).norm(dim=1) / full.norm(dim=1)
        size = x.double().norm(dim=1)[:, None] * exact_w.norm(dim=1)[None]
        by_w = (out[:n].double() - full).abs() / (size + full.abs())
        assert float(by_x.max()) <= bar and float(by_w.max()) <= (2e-6 if planes == 2 else 2 ** -11), (float(by_x.max()), float(by_w.max()))


def test_products_refuse_what_they_cannot_take(lib, pkg):
    a = pkg.RowsMatmulArgs()
    assert lib.b200_rows_matmul(C.byref(a), None) < 0
    x = torch.zeros(64, 64, dtype=torch.float16, device="cuda")
    out = torch.zeros(64, 64, device="cuda")
    good = dict(wtype=pkg.B200_WT_F16, d_w=x.data_ptr(), w_stride=128, rows=64, cols=64, d_x=x.data_ptr(), x_ld=64, planes=1, plane_rows=0, n=4,
                d_out=out.data_ptr(), out_ld=64)
    assert lib.b200_rows_matmul(C.byref(pkg.RowsMatmulArgs(**good)), None) == 0
    for change in (dict(cols=60), dict(x_ld=63), dict(x_ld=56), dict(planes=3), dict(planes=2), dict(w_stride=120), dict(wtype=pkg.B200_WT_F32),
                   dict(out_ld=63), dict(d_x=x.data_ptr() + 2), dict(n=0), dict(wtype=pkg.B200_WT_Q8)):
        assert lib.b200_rows_matmul(C.byref(pkg.RowsMatmulArgs(**{**good, **change})), None) < 0, change
    torch.cuda.synchronize()


@pytest.mark.parametrize("n_q,n_kv,hd", [(8, 2, 64), (8, 2, 128), (4, 1, 256), (3, 3, 128)])
@pytest.mark.parametrize("n_seq,seq_len,pos0", [(1, 1, 0), (1, 33, 0), (3, 64, 0), (1, 65, 31), (2, 17, 100), (1, 700, 0)])
def test_attention(lib, pkg, n_q, n_kv, hd, n_seq, seq_len, pos0):
    """Bar: a score is a sum of hd / 8 tensor-core additions, truncated at 2^-24 of scores up to about 50 here, and its error is the
    relative error of a weight: hd / 8 x 2^-25 x 50 = 5e-5 in the worst case, 6e-6 measured in 2-norm over a row; 2e-5."""
    max_seq, rows, heads = pos0 + seq_len + 3, n_seq * seq_len, n_q + 2 * n_kv
    g = torch.Generator().manual_seed(hd + seq_len)
    qkv = torch.randn(rows, heads, hd, generator=g).cuda()
    qg, kg = (1 + 0.3 * torch.randn(hd, generator=g)).cuda(), (1 + 0.3 * torch.randn(hd, generator=g)).cuda() * 3
    freq = torch.tensor([1.0 / 1e4 ** (2 * d / hd) for d in range(hd // 2)], dtype=torch.float32).cuda()
    kc = torch.full((n_seq, n_kv, max_seq, hd), float("nan"), dtype=torch.float16)
    vc = kc.clone()
    kc[:, :, :pos0] = torch.randn(n_seq, n_kv, pos0, hd, generator=g).half()
    vc[:, :, :pos0] = torch.randn(n_seq, n_kv, pos0, hd, generator=g).half()
    kc, vc = kc.cuda(), vc.cuda()
    q = torch.zeros(2 * rows * n_q * hd, dtype=torch.float16, device="cuda")
    qs = torch.zeros(rows * n_q, device="cuda")
    out = torch.full((rows, n_q, hd), float("nan"), device="cuda")
    a = pkg.RowsAttnArgs(n_q, n_kv, hd, max_seq, rows, seq_len, pos0, 1e-6, qkv.data_ptr(), qg.data_ptr(), kg.data_ptr(), freq.data_ptr(),
                         kc.data_ptr(), vc.data_ptr(), n_kv * max_seq * hd, q.data_ptr(), qs.data_ptr(), out.data_ptr())
    assert lib.b200_rows_attn(C.byref(a), None) == 0
    torch.cuda.synchronize()
    x = qkv.double().view(n_seq, seq_len, heads, hd)
    pos = torch.arange(pos0, pos0 + seq_len, device="cuda", dtype=torch.float32)
    ang = (pos[:, None] * freq).double()[None, :, None]

    def turn(t, gm):
        t = t * torch.rsqrt(t.square().mean(-1, keepdim=True) + 1e-6) * gm.double()
        u, v = t[..., : hd // 2], t[..., hd // 2:]
        return torch.cat([u * ang.cos() - v * ang.sin(), u * ang.sin() + v * ang.cos()], -1)
    qn, kn, vn = turn(x[:, :, :n_q], qg), turn(x[:, :, n_q:n_q + n_kv], kg), x[:, :, n_q + n_kv:]
    assert torch.equal(vc[:, :, pos0:pos0 + seq_len], vn.transpose(1, 2).half())
    # keys: one binary16 rounding of values that fp32 arithmetic gives to 2^-21 of a row's size
    assert float((kc[:, :, pos0:pos0 + seq_len].double() - kn.transpose(1, 2)).abs().max() / kn.abs().max()) < 2 ** -11
    assert torch.isnan(kc[:, :, pos0 + seq_len:]).all() and torch.isnan(vc[:, :, pos0 + seq_len:]).all()
    hide = torch.arange(pos0 + seq_len, device="cuda")[None, :] > torch.arange(pos0, pos0 + seq_len, device="cuda")[:, None]
    for h in range(n_q):
        k, v = kc[:, h // (n_q // n_kv), :pos0 + seq_len].double(), vc[:, h // (n_q // n_kv), :pos0 + seq_len].double()
        s = (qn[:, :, h] @ k.transpose(-1, -2) / hd ** 0.5).masked_fill(hide, -torch.inf)
        want = torch.softmax(s, -1) @ v
        got = out.view(n_seq, seq_len, n_q, hd)[:, :, h].double()
        assert float(((got - want).norm(dim=-1) / want.norm(dim=-1)).max()) < 2e-5


@pytest.mark.parametrize("planes", [2, 1])
@pytest.mark.parametrize("rows,dim", [(1, 64), (5, 2560), (3, 9728)])
def test_row_kernels(lib, pkg, planes, rows, dim):
    g = torch.Generator().manual_seed(dim)
    x, y = torch.randn(rows, dim, generator=g).cuda() * 1e5, torch.randn(rows, dim, generator=g).cuda() * 1e4
    gamma, post = torch.randn(dim, generator=g).cuda(), torch.randn(dim, generator=g).cuda()
    buf, scale, args = planes_buffer(pkg, rows, rows + 2, dim, planes)

    def value():
        b = buf.double().view(planes, rows + 2, dim)[:, :rows].sum(0)
        return b * scale[:rows, None].double()
    bar = 1e-6 if planes == 2 else 4e-4

    def norm(t, w):
        return t * torch.rsqrt(t.square().mean(-1, keepdim=True) + 1e-6) * w.double()
    for with_post in (False, True):
        xs = x.clone()
        assert lib.b200_rows_norm_planes(xs.data_ptr(), rows, dim, y.data_ptr(), post.data_ptr() if with_post else None, gamma.data_ptr(), None,
                                         1e-6, C.byref(args), None) == 0
        want = x.double() + (norm(y.double(), post) if with_post else y.double())
        assert rel(xs, want) < 1e-6 and rel(value(), norm(want, gamma)) < bar
    index = torch.tensor([rows - 1, 0][: rows], dtype=torch.int32, device="cuda")
    assert lib.b200_rows_norm_planes(xs.data_ptr(), len(index), dim, None, None, gamma.data_ptr(), index.data_ptr(), 1e-6, C.byref(args), None) == 0
    assert rel(value()[: len(index)], norm(xs.double()[index.long()], gamma)) < bar
    gu = torch.randn(rows, 2 * dim, generator=g).cuda() * 3
    for pairs in (0, 1):
        for gelu in (0, 1):
            gate, up = (gu[:, 0::2], gu[:, 1::2]) if pairs else (gu[:, :dim], gu[:, dim:])
            act = torch.nn.functional.gelu(gate.double(), approximate="tanh") if gelu else torch.nn.functional.silu(gate.double())
            assert lib.b200_rows_glu_planes(gu.data_ptr(), rows, dim, pairs, gelu, C.byref(args), None) == 0
            assert rel(value(), act * up.double()) < max(bar, 2e-6)
    # rows of zeros and rows with an infinity keep their values
    z = torch.zeros(rows, dim, device="cuda")
    z[0, 1] = torch.inf
    assert lib.b200_rows_split_planes(z.data_ptr(), rows, dim, C.byref(args), None) == 0
    torch.cuda.synchronize()
    assert torch.isinf(buf[0, 1]) and float(buf[1:rows].abs().sum()) == 0 and float(scale[0]) == 1.0


@pytest.mark.parametrize("family", ["tiny-qwen3", "tiny-gemma3"])
@pytest.mark.parametrize("fp16", [0, 1])
def test_prompt_equals_its_tokens(lib, pkg, synth, family, fp16):
    """Portions through the row path against the same tokens one by one: logits within 1e-3 of their spread (the caches are binary16 on
    both sides and agree to an ulp), any mix of portions, and the answer goes on from there."""
    sp = pkg.spec(family, gamma_jitter=0.1)
    gemma = "gemma" in family
    model = (synth.llmb200_synth_gemma3 if gemma else synth.llmb200_synth_qwen3)(C.byref(sp), 4)
    make = lib.inference_state_create_gemma3 if gemma else lib.inference_state_create
    s = make(model, 256, fp16)
    assert s
    V = sp.vocab_size
    toks = np.random.default_rng(5).integers(0, V, 150).astype(np.uint32)

    def feed(parts):
        lib.inference_state_reset(s)
        out, at = [], 0
        for n in parts:
            want = np.arange(n, dtype=np.int32)
            lg = np.zeros((n, V), np.float32)
            t = np.ascontiguousarray(toks[at:at + n])
            assert lib.inference_forward_tokens(s, t.ctypes.data_as(pkg.c_u32_p), n, want.ctypes.data_as(pkg.c_int_p), n,
                                                lg.ctypes.data_as(pkg.c_float_p)) == 0
            out.append(lg)
            at += n
        assert lib.llmb200_state_position(s) == len(toks) and lib.llmb200_state_error(s) == 0
        return np.concatenate(out)
    one = feed([1] * 150)
    spread = np.abs(one).max()
    for parts in ([150], [24, 5, 1, 64, 25, 31], [149, 1]):
        assert np.abs(feed(parts) - one).max() <= 1e-3 * spread, parts
    few = np.array([0, 77, 149], dtype=np.int32)                # the last layer is formed for these rows only; then the cache goes on
    lg = np.zeros((3, V), np.float32)
    lib.inference_state_reset(s)
    assert lib.inference_forward_tokens(s, toks.ctypes.data_as(pkg.c_u32_p), 150, few.ctypes.data_as(pkg.c_int_p), 3, lg.ctypes.data_as(pkg.c_float_p)) == 0
    assert np.abs(lg - one[few]).max() <= 1e-3 * spread
    lib.inference_state_reset(s)
    assert lib.inference_forward_tokens(s, toks.ctypes.data_as(pkg.c_u32_p), 149, None, 0, None) == 0
    after = np.ctypeslib.as_array(lib.inference_forward_token(s, int(toks[149])), (V,))
    assert np.abs(after - one[149]).max() <= 1e-3 * spread
    lib.inference_state_free(s)
    (synth.llmb200_synth_free_gemma3 if gemma else synth.llmb200_synth_free_qwen3)(model)


@pytest.mark.parametrize("cols", [32, 96, 2592])
@pytest.mark.parametrize("planes,n", [(1, 5), (2, 5), (2, 300)])
def test_an_odd_number_of_blocks_reads_no_padding(lib, pkg, synth, cols, planes, n):
    """The word that holds a row's last scale ends in padding that the packing kernels do not write: NaN there must not matter."""
    rows = 136
    stride = lib.b200_packed_row_stride(pkg.B200_WT_Q8, cols)
    d_w = torch.full((rows * stride,), 0xFF, dtype=torch.uint8, device="cuda")
    d_src = dev(weights(synth, rows, cols, 5))
    assert lib.b200_q8_pack(d_src.data_ptr(), cols, rows, cols, d_w.data_ptr(), stride, 0, 1, None) == 0
    exact_w = q8_values(lib, d_w, stride, rows, cols)
    x = torch.randn(n, cols, generator=torch.Generator().manual_seed(cols)).cuda()
    px, scale, args = planes_buffer(pkg, n, n, cols, planes, planes == 2)
    assert lib.b200_rows_split_planes(x.data_ptr(), n, cols, C.byref(args), None) == 0
    ws = torch.zeros(rows, dtype=torch.float32, device="cuda")
    assert lib.b200_q8_row_scale(d_w.data_ptr(), stride, rows, cols, ws.data_ptr(), None) == 0
    out = torch.zeros(n, rows, device="cuda")
    a = pkg.RowsMatmulArgs(pkg.B200_WT_Q8, d_w.data_ptr(), stride, rows, cols, ws.data_ptr(), px.data_ptr(), cols, planes, n,
                           scale.data_ptr() if scale is not None else None, n, out.data_ptr(), rows, None, rows, None, 0)
    assert lib.b200_rows_matmul(C.byref(a), None) == 0
    assert rel(out, x.double() @ exact_w.T) < (1e-5 if planes == 2 else 6e-4)


def test_q8_models_of_odd_block_counts(lib, pkg, synth):
    """Widths of 17 and 49 blocks; the memory that the state allocates holds what its last owner left there."""
    dirt = torch.full((1 << 28,), 0xFF, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    del dirt
    torch.cuda.empty_cache()
    sp = pkg.spec("tiny-qwen3", n_layers=2, d_model=544, intermediate_size=1568, gamma_jitter=0.1)
    model = synth.llmb200_synth_qwen3(C.byref(sp), 4)
    s = lib.inference_state_create(model, 64, 0)
    assert s
    toks = np.random.default_rng(5).integers(0, sp.vocab_size, 40).astype(np.uint32)
    one = np.stack([np.ctypeslib.as_array(lib.inference_forward_token(s, int(t)), (sp.vocab_size,)).copy() for t in toks])
    lib.inference_state_reset(s)
    lg = np.zeros_like(one)
    assert lib.inference_forward_tokens(s, toks.ctypes.data_as(pkg.c_u32_p), 40, np.arange(40, dtype=np.int32).ctypes.data_as(pkg.c_int_p), 40,
                                        lg.ctypes.data_as(pkg.c_float_p)) == 0
    assert np.abs(lg - one).max() <= 1e-3 * np.abs(one).max()
    lib.inference_state_free(s)
    synth.llmb200_synth_free_qwen3(model)


@pytest.mark.parametrize("hd,n_q,n_kv", [(64, 8, 2), (128, 4, 2), (256, 2, 1)])
@pytest.mark.parametrize("poison", [1e30, float("nan")])
def test_attention_leaves_later_values_out(lib, pkg, hd, n_q, n_kv, poison):
    """What one position's value or key holds reaches the rows that see it, as in the sums of the per-token path, and no other."""
    N, at, heads = 150, 75, n_q + 2 * n_kv
    g = torch.Generator().manual_seed(hd)
    qkv = torch.randn(N, heads, hd, generator=g).cuda()
    freq = torch.tensor([1.0 / 1e4 ** (2 * d / hd) for d in range(hd // 2)], dtype=torch.float32).cuda()

    def run(x, kc=None):
        kc = torch.zeros(n_kv, N, hd, dtype=torch.float16, device="cuda") if kc is None else kc
        vc = torch.zeros_like(kc)
        q = torch.zeros(2 * N * n_q * hd, dtype=torch.float16, device="cuda")
        qs, out = torch.zeros(N * n_q, device="cuda"), torch.zeros(N, n_q, hd, device="cuda")
        a = pkg.RowsAttnArgs(n_q, n_kv, hd, N, N, N, 0, 1e-6, x.data_ptr(), None, None, freq.data_ptr(), kc.data_ptr(), vc.data_ptr(), 0,
                             q.data_ptr(), qs.data_ptr(), out.data_ptr())
        assert lib.b200_rows_attn(C.byref(a), None) == 0
        torch.cuda.synchronize()
        return out
    plain = run(qkv)

    def same(out, rows):                                      # a tile with an infinity is summed in another order
        a, b = out[rows].double(), plain[rows].double()
        assert torch.isfinite(a).all() and float(((a - b).norm(dim=-1) / b.norm(dim=-1)).max()) < 2e-6
    bad = qkv.clone()
    bad[at, n_q + n_kv:, 3] = poison                          # one element of every value head
    out = run(bad)
    same(out, slice(0, at))
    assert rel(out[at:, :, 4:], plain[at:, :, 4:].double()) < 1e-6
    assert (torch.isnan(out[at:, :, 3]) if poison != poison else torch.isposinf(out[at:, :, 3])).all()
    bad = qkv.clone()
    bad[at, n_q:n_q + n_kv, :] = poison                       # a key: its scores are infinite or NaN
    same(run(bad), slice(0, at))
    bad = qkv.clone()
    bad[at, n_q:n_q + n_kv, 5] = poison                       # rows whose score with it is minus infinity give it no weight
    kc = torch.zeros(n_kv, N, hd, dtype=torch.float16, device="cuda")
    out = run(bad, kc)
    k = kc.double().repeat_interleave(n_q // n_kv, 0)
    x = bad[:, :n_q].double()
    ang = (torch.arange(N, device="cuda", dtype=torch.float32)[:, None] * freq).double()[:, None]
    x = torch.cat([x[..., : hd // 2] * ang.cos() - x[..., hd // 2:] * ang.sin(), x[..., : hd // 2] * ang.sin() + x[..., hd // 2:] * ang.cos()], -1)
    s = (x.transpose(0, 1)[:, :, None] * k[:, None]).sum(-1) / hd ** 0.5
    s = s.masked_fill(torch.ones(N, N, device="cuda").triu(1).bool(), -torch.inf)
    hit = torch.isfinite(torch.softmax(s, -1)).all(-1).transpose(0, 1)
    assert torch.equal(torch.isfinite(out).all(-1), hit) and (poison != poison or 0 < int(hit[at:].sum()) < hit[at:].numel())
    bad = qkv.clone()
    bad[at, :n_q, 5] = poison                                 # a query is its own row's only
    out = run(bad)
    assert torch.equal(out[:at], plain[:at]) and torch.equal(out[at + 1:], plain[at + 1:])


def test_planes_of_rows_with_infinities(lib, pkg):
    """An infinity is one plane's infinity and nothing in the other; it takes neither the range nor the bits of the row's other elements."""
    rows, dim = 3, 256
    x = torch.randn(rows, dim, generator=torch.Generator().manual_seed(1)) * 1e5
    x[0, 7], x[1, 9], x[2, 11] = torch.inf, -torch.inf, torch.nan
    finite = torch.isfinite(x)
    buf, scale, args = planes_buffer(pkg, rows, rows, dim, 2)
    d = x.cuda()
    assert lib.b200_rows_split_planes(d.data_ptr(), rows, dim, C.byref(args), None) == 0
    torch.cuda.synchronize()
    hi, lo = (p.double().cpu() for p in buf.view(2, rows, dim))
    value = (hi + lo) * scale.cpu()[:, None].double()
    assert ((value - x.double()).abs()[finite] <= 2 ** -22 * x.double().abs()[finite] + 2 ** -38 * 4e5).all()
    assert float(value[0, 7]) == float("inf") and float(value[1, 9]) == -float("inf") and torch.isnan(value[2, 11])
    assert float(lo[0, 7]) == 0 and float(lo[1, 9]) == 0


@pytest.mark.parametrize("planes", [1, 2])
@pytest.mark.parametrize("dim", [12288, 58016, 58112, 60000])
def test_rows_wider_than_shared_memory(lib, pkg, planes, dim):
    """Rows that just fill the 48 KB a kernel has without asking, and either side of the 58 048 values that it can be given beside its own."""
    g = torch.Generator().manual_seed(dim)
    gu, x, y = (torch.randn(2, n * dim, generator=g).cuda() for n in (2, 1, 1))
    gamma, post = torch.randn(dim, generator=g).cuda(), torch.randn(dim, generator=g).cuda()
    buf, scale, args = planes_buffer(pkg, 2, 2, dim, planes, planes == 2)

    def value():
        torch.cuda.synchronize()
        return buf.double().view(planes, 2, dim).sum(0) * (scale[:, None].double() if planes == 2 else 1.0)

    def norm(t, w):
        return t * torch.rsqrt(t.square().mean(-1, keepdim=True) + 1e-6) * w.double()
    bar = 2e-6 if planes == 2 else 4e-4
    for pairs in (0, 1):
        gate, up = (gu[:, 0::2], gu[:, 1::2]) if pairs else (gu[:, :dim], gu[:, dim:])
        assert lib.b200_rows_glu_planes(gu.data_ptr(), 2, dim, pairs, 0, C.byref(args), None) == 0
        assert rel(value(), torch.nn.functional.silu(gate.double()) * up.double()) < bar
    for with_post in (False, True):
        xs = x.clone()
        assert lib.b200_rows_norm_planes(xs.data_ptr(), 2, dim, y.data_ptr(), post.data_ptr() if with_post else None, gamma.data_ptr(), None, 1e-6,
                                         C.byref(args), None) == 0
        want = x.double() + (norm(y.double(), post) if with_post else y.double())
        assert rel(xs, want) < 1e-6 and rel(value(), norm(want, gamma)) < bar


def per_token(lib, pkg, d_w, stride, rows, cols, wt, x):
    out = torch.zeros(len(x), rows, device="cuda")
    for i in range(len(x)):
        a = pkg.MatvecArgs()
        a.d_w, a.row_stride, a.rows, a.cols, a.wtype = d_w.data_ptr(), stride, rows, cols, wt
        a.in_mode, a.d_in_vec = pkg.B200_IN_VEC, x[i].data_ptr()
        a.out_mode, a.n_out, a.eps = pkg.B200_OUT_STORE, 1, 1e-6
        a.d_out[0] = out[i].data_ptr()
        assert lib.b200_matvec(C.byref(a), None) == 0
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("wtype", ["q8", "f16"])
@pytest.mark.parametrize("rows,cols,n", [(512, 1536, 15), (2560, 2560, 4), (6144, 2560, 130), (2560, 9728, 48), (2560, 9728, 512), (2560, 4096, 1531)])
def test_products_stay_near_fp32_sums(lib, pkg, synth, wtype, rows, cols, n):
    """Against float64. Four truncated additions a step, half a unit each: up to 1.4e-7 of the result; the planes' last bits, 22 in either
    operand: 0.7e-7; up to 152 rounded additions in a random walk: 1.5e-7. Bar: their sum in squares and a third, 3e-7. The per-token kernel's fp32
    sums on the same operands are 1e-7 off and must not be more than three times as exact."""
    wt = pkg.B200_WT_Q8 if wtype == "q8" else pkg.B200_WT_F16
    d_w, stride = pack(lib, pkg, weights(synth, rows, cols, 3), wt)
    exact_w = q8_values(lib, d_w, stride, rows, cols) if wtype == "q8" else d_w.view(torch.float16).view(rows, stride // 2)[:, :cols].double()
    x = torch.randn(n, cols, generator=torch.Generator().manual_seed(n)).cuda()
    px, scale, args = planes_buffer(pkg, n, n, cols, 2)
    assert lib.b200_rows_split_planes(x.data_ptr(), n, cols, C.byref(args), None) == 0
    ws, err = torch.zeros(rows, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    if wtype == "q8":
        assert lib.b200_q8_row_scale(d_w.data_ptr(), stride, rows, cols, ws.data_ptr(), None) == 0
    out = torch.zeros(n, rows, device="cuda")
    a = pkg.RowsMatmulArgs(wt, d_w.data_ptr(), stride, rows, cols, ws.data_ptr(), px.data_ptr(), cols, 2, n, scale.data_ptr(), n, out.data_ptr(),
                           rows, None, rows, err.data_ptr(), 0)
    assert lib.b200_rows_matmul(C.byref(a), None) == 0
    torch.cuda.synchronize()
    want = x.double() @ exact_w.T
    few = min(n, 8)
    ours, theirs = rel(out, want), rel(per_token(lib, pkg, d_w, stride, rows, cols, wt, x[:few]), want[:few])
    assert int(err) == 0 and ours <= min(3e-7, 3 * theirs), (ours, theirs)


@pytest.mark.parametrize("n_q,n_kv,hd,N", [(8, 2, 64, 200), (8, 2, 128, 500), (4, 1, 256, 200)])
def test_attention_is_as_exact_as_the_per_token_kernel(lib, pkg, n_q, n_kv, hd, N):
    """Both against float64 over the keys and values that each left in its cache. Bar: the per-token kernel's error and a half of it again."""
    g, heads = torch.Generator().manual_seed(hd), n_q + 2 * n_kv
    qkv = torch.randn(N, heads, hd, generator=g).cuda()
    qg, kg = (1 + 0.3 * torch.randn(hd, generator=g)).cuda(), (1 + 0.3 * torch.randn(hd, generator=g)).cuda()
    freq = torch.tensor([1.0 / 1e4 ** (2 * d / hd) for d in range(hd // 2)], dtype=torch.float32).cuda()
    ang = (torch.arange(N, device="cuda", dtype=torch.float32)[:, None] * freq).double()[:, None]
    x = qkv[:, :n_q].double()
    x = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * qg.double()
    u, w = x[..., : hd // 2], x[..., hd // 2:]
    x = torch.cat([u * ang.cos() - w * ang.sin(), u * ang.sin() + w * ang.cos()], -1)
    errors = []
    for rows in (0, 1):
        kc, vc = (torch.zeros(n_kv, N, hd, dtype=torch.float16, device="cuda") for _ in range(2))
        out = torch.zeros(N, n_q, hd, device="cuda")
        if rows:
            q, qs = torch.zeros(2 * N * n_q * hd, dtype=torch.float16, device="cuda"), torch.zeros(N * n_q, device="cuda")
            a = pkg.RowsAttnArgs(n_q, n_kv, hd, N, N, N, 0, 1e-6, qkv.data_ptr(), qg.data_ptr(), kg.data_ptr(), freq.data_ptr(), kc.data_ptr(),
                                 vc.data_ptr(), 0, q.data_ptr(), qs.data_ptr(), out.data_ptr())
            assert lib.b200_rows_attn(C.byref(a), None) == 0
        else:
            scratch, tickets = torch.zeros(lib.b200_attn_scratch_floats(n_q, hd, 4), device="cuda"), torch.zeros(n_kv, dtype=torch.int32, device="cuda")
            pos = torch.arange(N, dtype=torch.int32, device="cuda")
            for i in range(N):
                a = pkg.AttnArgs(qkv[i].data_ptr(), qg.data_ptr(), kg.data_ptr(), freq.data_ptr(), kc.data_ptr(), vc.data_ptr(), out[i].data_ptr(),
                                 scratch.data_ptr(), tickets.data_ptr(), pos[i:].data_ptr(), n_q, n_kv, hd, N, 4, 1e-6, 0)
                assert lib.b200_attn_decode(C.byref(a), None) == 0
        torch.cuda.synchronize()
        k, v = (t.double().repeat_interleave(n_q // n_kv, 0) for t in (kc, vc))
        s = torch.einsum("ihd,hjd->hij", x, k) / hd ** 0.5
        s = s.masked_fill(torch.ones(N, N, device="cuda").triu(1).bool(), -torch.inf)
        errors.append(rel(out, torch.einsum("hij,hjd->ihd", torch.softmax(s, -1), v)))
    assert errors[1] <= 1.5 * errors[0], errors


@pytest.mark.parametrize("wtype", ["q8", "f16"])
def test_chained_products(lib, pkg, synth, wtype):
    """use_pdl: a product that starts while the kernel that makes its operand is still at it, over and over with other operands."""
    wt, rows, cols, n = pkg.B200_WT_Q8 if wtype == "q8" else pkg.B200_WT_F16, 1024, 2560, 40
    d_w, stride = pack(lib, pkg, weights(synth, rows, cols, 3), wt)
    ws = torch.zeros(rows, device="cuda")
    if wtype == "q8":
        assert lib.b200_q8_row_scale(d_w.data_ptr(), stride, rows, cols, ws.data_ptr(), None) == 0
    px, scale, args = planes_buffer(pkg, n, n, cols, 2)
    x = torch.randn(12, n, cols, generator=torch.Generator().manual_seed(1)).cuda()

    def run(pdl):
        out = torch.zeros(12, n, rows, device="cuda")
        torch.cuda.synchronize()
        for i in range(12):
            assert lib.b200_rows_split_planes(x[i].data_ptr(), n, cols, C.byref(args), None) == 0
            a = pkg.RowsMatmulArgs(wt, d_w.data_ptr(), stride, rows, cols, ws.data_ptr(), px.data_ptr(), cols, 2, n, scale.data_ptr(), n,
                                   out[i].data_ptr(), rows, None, rows, None, pdl)
            assert lib.b200_rows_matmul(C.byref(a), None) == 0
            if not pdl:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return out
    assert torch.equal(run(1), run(0))


def test_prompts_beyond_one_pass(lib, pkg, synth):
    """2500 tokens: a second pass over 452, wanted rows in both and at their edges, in a workspace that a short prompt made first."""
    sp = pkg.spec("tiny-qwen3", n_layers=2, gamma_jitter=0.1)
    model = synth.llmb200_synth_qwen3(C.byref(sp), 4)
    s = lib.inference_state_create(model, 4096, 1)
    assert s
    V = sp.vocab_size
    toks = np.random.default_rng(9).integers(0, V, 2500).astype(np.uint32)
    want = [0, 1000, 2047, 2048, 2300, 2499]
    one = []
    for i, t in enumerate(toks):
        lg = np.ctypeslib.as_array(lib.inference_forward_token(s, int(t)), (V,))
        if i in want:
            one.append(lg.copy())
    one = np.stack(one)

    def passes(n, want):
        lg = np.zeros((len(want), V), dtype=np.float32)
        lib.inference_state_reset(s)
        assert lib.inference_forward_tokens(s, toks.ctypes.data_as(pkg.c_u32_p), n, (C.c_int * len(want))(*want), len(want),
                                            lg.ctypes.data_as(pkg.c_float_p)) == 0
        return lg
    first = passes(40, [0])
    lg = passes(2500, want)
    assert np.abs(lg - one).max() <= 1e-3 * np.abs(one).max()
    assert np.abs(first[0] - one[0]).max() <= 1e-3 * np.abs(one).max()
    assert np.abs(passes(2500, [2499])[0] - one[-1]).max() <= 1e-3 * np.abs(one).max()
    many = passes(2500, list(range(1990, 2120)))               # more wanted rows than the head takes at once, in both passes
    assert np.abs(many[2047 - 1990] - one[2]).max() <= 1e-3 * np.abs(one).max() and np.abs(many[2048 - 1990] - one[3]).max() <= 1e-3 * np.abs(one).max()
    lib.inference_state_free(s)
    synth.llmb200_synth_free_qwen3(model)
