"""Training attention forward and backward over tile edges, against float64.

Bar: operands are split into TF32 pairs (22 bits) and sums of up to hd, 64 or N terms are fp32, truncated per eight terms: max(hd, 64) / 8 x 3 x 2^-24
of the terms bounds a tile's, fp32 adds join the tiles; 1e-6 measured in 2-norm over a tensor, 5e-6."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a.double() - b).norm() / b.norm())


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("S,N,Hq,Hkv,shift", [(1, 1, 2, 1, 0), (2, 63, 4, 2, 0), (3, 64, 2, 2, 0), (1, 65, 4, 1, 1), (2, 200, 4, 2, 0), (1, 509, 8, 2, 0)])
def test_forward_and_backward(lib, hd, S, N, Hq, Hkv, shift):
    g = torch.Generator().manual_seed(N + hd)
    M, G, scale, ld = S * N, Hq // Hkv, hd ** -0.5, (Hq + 2 * Hkv) * hd + 4
    qkv = torch.randn(M, ld, generator=g).cuda()

    def off(*shape):                                          # `shift` floats off a 16-byte boundary, where that was taken before
        t = torch.zeros(shape[0] * shape[1] + shift, device="cuda")[shift:].view(*shape)
        t.copy_(torch.randn(*shape, generator=g))
        return t
    q, k, d_out = off(M, Hq * hd), torch.randn(M, Hkv * hd, generator=g).cuda(), off(M, Hq * hd) * 1e-3
    if shift:
        d_out = off(M, Hq * hd)
        d_out *= 1e-3
    v = qkv[:, (Hq + Hkv) * hd:]
    probs, out = torch.full((S, Hq, N, N), 7.0, device="cuda"), torch.full((M, Hq * hd), 7.0, device="cuda")
    half = torch.zeros(M, Hq * hd, dtype=torch.float16, device="cuda")
    assert lib.b200_attn_train_fwd_h(q.data_ptr(), k.data_ptr(), v.data_ptr(), ld, S, N, Hq, Hkv, hd, scale, probs.data_ptr(), out.data_ptr(),
                                     half.data_ptr(), None) == 0
    dqkv = torch.full((M, ld), 7.0, device="cuda")
    d_score = torch.full((S * Hq * N * max(N, 2 * hd),), float("nan"), device="cuda")
    assert lib.b200_attn_train_bwd(d_out.data_ptr(), probs.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), ld, S, N, Hq, Hkv, hd, scale,
                                   d_score.data_ptr(), dqkv.data_ptr(), ld, None) == 0
    torch.cuda.synchronize()

    def heads(t, n):
        return t.double().reshape(S, N, n, hd).transpose(1, 2)
    Q, K, V = (t.detach().clone().requires_grad_() for t in (heads(q, Hq), heads(k, Hkv), heads(v[:, : Hkv * hd], Hkv)))
    s = Q @ K.repeat_interleave(G, 1).transpose(-1, -2) * scale
    p = torch.softmax(s.masked_fill(torch.ones(N, N, device="cuda").triu(1).bool(), -torch.inf), -1)
    o = p @ V.repeat_interleave(G, 1)
    o.backward(heads(d_out, Hq))

    def rows(t):
        return t.transpose(1, 2).reshape(M, -1)
    assert rel(probs, p.detach()) < 5e-6 and (probs.triu(1) == 0).all()
    assert rel(out, rows(o.detach())) < 5e-6 and torch.equal(half, out.half())
    got = [dqkv[:, :Hq * hd], dqkv[:, Hq * hd:(Hq + Hkv) * hd], dqkv[:, (Hq + Hkv) * hd:(Hq + 2 * Hkv) * hd]]
    for name, a, b in zip("qkv", got, (Q.grad, K.grad, V.grad)):
        size = 1e-3 * (hd * N) ** 0.5                          # one position: dQ and dK are zero up to rounding
        assert float((a.double() - rows(b)).norm()) <= 5e-6 * float(rows(b).norm()) + 1e-7 * size, name
    assert (dqkv[:, (Hq + 2 * Hkv) * hd:] == 7.0).all()


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("poison", [float("inf"), float("nan")])
@pytest.mark.parametrize("tc", [0, 1])
def test_other_rows_stay_out(lib, hd, poison, tc):
    """An infinity or NaN at one position reaches the sums that contain it and no other: later keys and values are left out, not weighted zero."""
    S, N, Hq, Hkv, at = 2, 200, 2, 1, 70
    g = torch.Generator().manual_seed(hd)
    M, ld = S * N, (Hq + 2 * Hkv) * hd
    qkv = torch.randn(M, ld, generator=g).cuda()
    tensors = dict(q=torch.randn(M, Hq * hd, generator=g).cuda(), k=torch.randn(M, Hkv * hd, generator=g).cuda(),
                   v=qkv, d=torch.randn(M, Hq * hd, generator=g).cuda())

    def run(t):
        v = t["v"][:, (Hq + Hkv) * hd:]
        probs, out = torch.zeros(S, Hq, N, N, device="cuda"), torch.zeros(M, Hq * hd, device="cuda")
        d_score, dqkv = torch.zeros(S * Hq * N * N, device="cuda"), torch.zeros(M, ld, device="cuda")
        fwd, bwd = (lib.b200_attn_train_fwd_tc, lib.b200_attn_train_bwd_tc) if tc else (lib.b200_attn_train_fwd_h, lib.b200_attn_train_bwd)
        assert fwd(t["q"].data_ptr(), t["k"].data_ptr(), v.data_ptr(), ld, S, N, Hq, Hkv, hd, hd ** -0.5, probs.data_ptr(), out.data_ptr(), None,
                   None) == 0
        assert bwd(t["d"].data_ptr(), probs.data_ptr(), t["q"].data_ptr(), t["k"].data_ptr(), v.data_ptr(), ld, S, N, Hq, Hkv, hd,
                   hd ** -0.5, d_score.data_ptr(), dqkv.data_ptr(), ld, None) == 0
        torch.cuda.synchronize()
        return out, dqkv[:, : Hq * hd], dqkv[:, Hq * hd:]
    plain = run(tensors)
    rows = torch.arange(M, device="cuda")
    others, before, after = rows != at, (rows < at) | (rows >= N), (rows > at)
    # which rows of (out, dQ, dK and dV) do not contain position `at` of the poisoned tensor
    free = dict(q=(others, others, after), k=(before, before, rows >= N), v=(before, before, rows >= N), d=(others, others, after))
    for name, keep in free.items():
        t = dict(tensors)
        t[name] = tensors[name].clone()
        t[name][at, -hd // 2:] = poison                       # of v's rows the last columns are the values
        for part, a, b, k in zip(("out", "dq", "dkv"), run(t), plain, keep):
            if tc:                                            # a fragment with an infinity is summed in fp32 instead
                assert torch.isfinite(a[k]).all() and rel(a[k], b[k].double()) < 2e-6, (name, part)
            else:
                assert torch.equal(a[k], b[k]), (name, part)


@pytest.mark.parametrize("tensor_cores", [False, True])
def test_the_engine_takes_the_form_it_was_asked_for(lib, pkg, tensor_cores):
    """With tensor cores off every product is fp32 on the CUDA cores, the attention's too: its probabilities are that form's to the bit."""
    import _sft_common as sc
    cfg, N, S = sc.SMALL, 40, 2
    Hq, Hkv, hd = cfg["n_q_heads"], cfg["n_kv_heads"], cfg["head_dim"]
    eng = sc.Engine(pkg, cfg, sc.make_weights(pkg, cfg), sc.make_lora(pkg, cfg, 4, b_std=0.02), N, S, 4, 8.0, tensor_cores=tensor_cores)
    ids = sc.tokens(pkg, N * S, 3, cfg["vocab_size"]).reshape(S, N)
    eng.forward_backward(ids, ids)
    q, k = (torch.from_numpy(eng.export(what, 1, N * S * h * hd)).cuda() for what, h in ((sc.Q_FINAL, Hq), (sc.K_FINAL, Hkv)))
    got = torch.from_numpy(eng.export(sc.PROBS, 1, S * Hq * N * N)).cuda()
    v, out, same = torch.zeros(N * S, Hkv * hd, device="cuda"), torch.zeros(N * S, Hq * hd, device="cuda"), []
    for fwd in (lib.b200_attn_train_fwd_h, lib.b200_attn_train_fwd_tc):
        probs = torch.zeros_like(got)
        assert fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), Hkv * hd, S, N, Hq, Hkv, hd, hd ** -0.5, probs.data_ptr(), out.data_ptr(), None, None) == 0
        torch.cuda.synchronize()
        same.append(torch.equal(probs, got))
    assert same == [not tensor_cores, tensor_cores]
    eng.close()


@pytest.mark.parametrize("S,N,Hq,Hkv,hd", [(2, 64, 8, 2, 128), (1, 509, 8, 2, 128), (1, 64, 4, 1, 256), (1, 200, 8, 2, 64)])
def test_tensor_cores_lose_nothing(lib, S, N, Hq, Hkv, hd):
    """Both forms against float64 on the same inputs. Bar of the fp32 form: some hundred fp32 roundings of 2^-25 in a random walk, 1e-6. Of the
    tensor-core form: the fp32 form's own error and a half of it again."""
    g = torch.Generator().manual_seed(N + hd)
    M, G, ld = S * N, Hq // Hkv, (Hq + 2 * Hkv) * hd
    qkv = torch.randn(M, ld, generator=g).cuda()
    q, k, d_out = (torch.randn(M, h * hd, generator=g).cuda() for h in (Hq, Hkv, Hq))
    v = qkv[:, (Hq + Hkv) * hd:]

    def heads(t, n):
        return t.double().reshape(S, N, n, hd).transpose(1, 2)
    Q, K, V = (t.detach().clone().requires_grad_() for t in (heads(q, Hq), heads(k, Hkv), heads(v[:, : Hkv * hd], Hkv)))
    s = Q @ K.repeat_interleave(G, 1).transpose(-1, -2) * hd ** -0.5
    p = torch.softmax(s.masked_fill(torch.ones(N, N, device="cuda").triu(1).bool(), -torch.inf), -1)
    o = p @ V.repeat_interleave(G, 1)
    o.backward(heads(d_out, Hq))
    rows = [t.transpose(1, 2).reshape(M, -1) for t in (o.detach(), Q.grad, K.grad, V.grad)]
    errors = []
    for fwd, bwd in ((lib.b200_attn_train_fwd_h, lib.b200_attn_train_bwd), (lib.b200_attn_train_fwd_tc, lib.b200_attn_train_bwd_tc)):
        probs, out = torch.zeros(S, Hq, N, N, device="cuda"), torch.zeros(M, Hq * hd, device="cuda")
        d_score, dqkv = torch.zeros(S * Hq * N * N, device="cuda"), torch.zeros(M, ld, device="cuda")
        assert fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), ld, S, N, Hq, Hkv, hd, hd ** -0.5, probs.data_ptr(), out.data_ptr(), None, None) == 0
        assert bwd(d_out.data_ptr(), probs.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), ld, S, N, Hq, Hkv, hd, hd ** -0.5,
                   d_score.data_ptr(), dqkv.data_ptr(), ld, None) == 0
        torch.cuda.synchronize()
        got = [out, dqkv[:, : Hq * hd], dqkv[:, Hq * hd:(Hq + Hkv) * hd], dqkv[:, (Hq + Hkv) * hd:]]
        errors.append([rel(probs, p.detach())] + [rel(a, b) for a, b in zip(got, rows)])
    assert max(errors[0]) < 1e-6, errors
    assert all(b <= 1.5 * a for a, b in zip(*errors)), errors
