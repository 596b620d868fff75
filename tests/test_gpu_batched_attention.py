"""Attention of a step over many sequences: more (sequence, KV head) pairs than SMs, one block to each, which stores its results itself, or several that merge.

Off float64 over the cache rows that the kernel left: a score is a sum of hd fp32 products, 2^-17 of the terms' magnitude at the worst (64 .. 256 terms, magnitude
below 4 after the scale): 3e-5 of a weight, and so of the largest value."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("G", [1, 2, 4, 8])
@pytest.mark.parametrize("B,n_kv,pos", [(38, 4, 0), (19, 8, 7), (32, 8, 40), (150, 1, 131), (2, 3, 33)])
def test_many_sequences(lib, pkg, hd, G, B, n_kv, pos):
    max_seq, n_q = 160, G * n_kv
    g = torch.Generator().manual_seed(hd + G + pos)
    rows = n_q + 2 * n_kv
    qkv = torch.randn(B, rows, hd, generator=g).cuda()
    freq = (1e4 ** (-2.0 * torch.arange(hd // 2) / hd)).float().cuda()
    kc, vc = (torch.randn(B, n_kv, max_seq, hd, generator=g).half().cuda() for _ in range(2))
    kc[:, :, pos + 1:] = float("nan"); vc[:, :, pos + 1:] = float("nan")           # later rows: not read
    qg, kg = ((1 + 0.1 * torch.randn(hd, generator=g)).cuda() for _ in range(2))
    out = torch.full((B, n_q, hd), float("nan"), device="cuda")
    scratch = torch.full((B * lib.b200_attn_scratch_floats(n_q, hd, 1),), float("nan"), device="cuda")
    tickets = torch.zeros(B * n_kv, dtype=torch.int32, device="cuda")
    where = torch.tensor([pos], dtype=torch.int32, device="cuda")
    a = pkg.AttnArgs(qkv.data_ptr(), qg.data_ptr(), kg.data_ptr(), freq.data_ptr(), kc.data_ptr(), vc.data_ptr(), out.data_ptr(), scratch.data_ptr(),
                     tickets.data_ptr(), where.data_ptr(), n_q, n_kv, hd, max_seq, 1, 1e-6, 0, B, rows * hd, n_kv * max_seq * hd, n_q * hd)
    for _ in range(2):                                        # twice: nothing is left behind
        assert lib.b200_attn_decode(C.byref(a), None) == 0
    torch.cuda.synchronize()

    def rotated(x, gamma):
        x = x.double()
        x = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * gamma.double()
        ang = (pos * freq).double()
        lo, hi = x[..., :hd // 2], x[..., hd // 2:]
        return torch.cat([lo * ang.cos() - hi * ang.sin(), lo * ang.sin() + hi * ang.cos()], -1)

    q = rotated(qkv[:, :n_q], qg).view(B, n_kv, G, hd)
    k, v = kc[:, :, :pos + 1].double(), vc[:, :, :pos + 1].double()
    assert ((k[:, :, pos] - rotated(qkv[:, n_q:n_q + n_kv], kg)).abs() <= 2 ** -10 * k[:, :, pos].abs() + 1e-6).all()
    assert torch.equal(vc[:, :, pos], qkv[:, n_q + n_kv:].half())
    w = torch.softmax(q @ k.transpose(-1, -2) * hd ** -0.5, -1)
    want = (w @ v).view(B, n_q, hd)
    assert (out.double() - want).abs().max() <= 3e-5 * v.abs().max()
    assert (tickets == 0).all()


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("G", [1, 2, 4, 8])
@pytest.mark.parametrize("n_split", [1, 2])
@pytest.mark.parametrize("B,n_kv,pos", [(38, 4, 0), (19, 8, 7), (32, 8, 129), (150, 1, 131), (20, 8, 33)])
def test_a_sequence_is_the_same_in_any_company(lib, pkg, hd, G, n_split, B, n_kv, pos):
    """The step over all sequences and a step over each one alone: the same bits, whichever threads a block has, with one split and with several."""
    max_seq, n_q = 160, G * n_kv
    g = torch.Generator().manual_seed(hd + G + pos)
    rows = n_q + 2 * n_kv
    qkv = (2 * torch.randn(B, rows, hd, generator=g)).cuda()
    freq = (1e4 ** (-2.0 * torch.arange(hd // 2) / hd)).float().cuda()
    kc, vc = (torch.randn(B, n_kv, max_seq, hd, generator=g).half().cuda() for _ in range(2))
    out = torch.full((2, B, n_q, hd), float("nan"), device="cuda")
    scratch = torch.empty(B * lib.b200_attn_scratch_floats(n_q, hd, n_split), device="cuda")
    tickets = torch.zeros(B * n_kv, dtype=torch.int32, device="cuda")
    where = torch.tensor([pos], dtype=torch.int32, device="cuda")
    for first, n, to in [(0, B, 0)] + [(b, 1, 1) for b in range(B)]:
        a = pkg.AttnArgs(qkv[first].data_ptr(), 0, 0, freq.data_ptr(), kc[first].data_ptr(), vc[first].data_ptr(), out[to, first].data_ptr(), scratch.data_ptr(),
                         tickets.data_ptr(), where.data_ptr(), n_q, n_kv, hd, max_seq, n_split, 1e-6, 0, n, rows * hd, n_kv * max_seq * hd, n_q * hd)
        assert lib.b200_attn_decode(C.byref(a), None) == 0
    torch.cuda.synchronize()
    assert not torch.isnan(out).any()
    assert torch.equal(out[0], out[1])
