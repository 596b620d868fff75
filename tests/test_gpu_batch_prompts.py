"""Prompts of the batched engine in passes: several passes with a shorter last one and products of more than 128 rows, memory that has no
room for a pass, wide activations, and device errors that the call must report. Reference: every sequence by itself on a single state with the
same binary16 weights (fp32 activations); logits within the 1e-2 that the engine's binary16 operands give."""
import ctypes as C

import numpy as np
import pytest

import _sft_common as sc

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def states(pkg, lib, cfg, B, G, max_seq, single=True):
    """A batch state and, over the same weights, a single one."""
    w = sc.make_weights(pkg, cfg)
    c = pkg.Config(pkg.MODEL_QWEN3, cfg["d_model"], cfg["n_q_heads"], cfg["n_kv_heads"], cfg["head_dim"], cfg["intermediate_size"],
                   cfg["vocab_size"], cfg["n_layers"], max_seq, 1)
    b = lib.llmb200_batch_begin(C.byref(c), B, G)
    s = lib.llmb200_state_begin(C.byref(c)) if single else None
    assert b and (s or not single)
    for i, l in enumerate(w["layers"]):
        r = pkg.LayerWeightRef()
        for name in ("q", "k", "v", "o", "gate", "up", "down"):
            setattr(r, name + "_proj", pkg.WeightRef(sc.fptr(l[name]), *l[name].shape))
        for name, field in (("input_norm", "input_norm_g"), ("post_attn_norm", "post_attn_norm_g"), ("q_norm", "q_norm_g"), ("k_norm", "k_norm_g")):
            setattr(r, field, sc.fptr(l[name]))
        r.d_model, r.head_dim = cfg["d_model"], cfg["head_dim"]
        assert lib.llmb200_batch_load_layer(b, i, C.byref(r), C.c_float(1e6)) == 0
        assert not single or lib.llmb200_state_load_layer(s, i, C.byref(r), C.c_float(1e6)) == 0
        lib.metal_flush()
    ends = [sc.fptr(w[k]) for k in ("lm_head", "final_norm", "emb")]
    assert lib.llmb200_batch_finish(b, *ends) == 0 and (not single or lib.llmb200_state_finish(s, *ends) == 0)
    lib.llmb200_batch_set_eos(b, None, 0)
    return b, s


def generate(pkg, lib, b, prompts, G):
    out = np.zeros((len(prompts), G), dtype=np.uint32)
    n = lib.llmb200_batch_generate(b, prompts.ctypes.data_as(pkg.c_u32_p), prompts.shape[1], out.ctypes.data_as(pkg.c_u32_p), G)
    return n, out


def logits_of(pkg, lib, b, B, V):
    got = np.zeros((B, V), dtype=np.float32)
    assert lib.llmb200_batch_logits(b, got.ctypes.data_as(pkg.c_float_p), got.size)
    return got


def check(pkg, lib, s, prompts, out, last, V):
    """`last`: the logits that the step over each sequence's last token but one left (position len(prompt) + len(out) - 2)."""
    for b in range(len(prompts)):
        seq = np.ascontiguousarray(np.concatenate([prompts[b], out[b][:-1]]).astype(np.uint32))
        lib.inference_state_reset(s)
        lg = np.zeros((1, V), dtype=np.float32)
        want = (C.c_int * 1)(len(seq) - 1)
        assert lib.inference_forward_tokens(s, seq.ctypes.data_as(pkg.c_u32_p), len(seq), want, 1, lg.ctypes.data_as(pkg.c_float_p)) == 0
        assert np.abs(lg[0] - last[b]).max() < 1e-2 * np.abs(lg).max(), b
        top = np.sort(lg[0])[-2:]
        assert int(np.argmax(lg[0])) == int(out[b][-1]) or top[1] - top[0] < 2e-2 * np.abs(lg).max(), b


# B, prompt: one pass of 32 x 64 rows, a second of 32 x 64, a last of 32 x 21; 3 x 682 and 3 x 17; a single row a pass boundary away; 2 x 130 rows
@pytest.mark.parametrize("B,P", [(32, 150), (3, 700), (32, 66), (2, 131)])
def test_several_passes(pkg, lib, B, P):
    cfg, G = dict(sc.SMALL, vocab_size=1024), 4
    b, s = states(pkg, lib, cfg, B, G, 1024)
    prompts = np.random.default_rng(P).integers(0, 1024, (B, P)).astype(np.uint32)
    short = np.ascontiguousarray(prompts[:, :9])
    assert generate(pkg, lib, b, short, G)[0] == G            # a small workspace first: the next call has to grow it
    n, out = generate(pkg, lib, b, prompts, G)
    assert n == G
    check(pkg, lib, s, prompts, out, logits_of(pkg, lib, b, B, 1024), 1024)
    again = generate(pkg, lib, b, prompts, G)[1]
    assert np.array_equal(out, again)
    lib.llmb200_batch_free(b)
    lib.inference_state_free(s)


def test_wide_feed_forward(pkg, lib):
    """Wider than a row in shared memory could be: the step needs none, and prompts go through as well. Reference: the restatement's forward."""
    cfg, B, G, P = dict(sc.SMALL, n_layers=1, d_model=64, intermediate_size=58624, vocab_size=256), 2, 3, 20
    b, _ = states(pkg, lib, cfg, B, G, 64, single=False)
    prompts = np.random.default_rng(P).integers(0, 256, (B, P)).astype(np.uint32)
    n, out = generate(pkg, lib, b, prompts, G)
    assert n == G
    last = logits_of(pkg, lib, b, B, 256)
    ow = sc.oracle_model(cfg, sc.make_weights(pkg, cfg))
    zero = sc.sft_oracle.LoRA(sc.make_lora(pkg, cfg, 4), 4, 8.0)
    for i in range(B):
        lg = sc.sft_oracle.forward(ow, zero, np.concatenate([prompts[i], out[i]])[:-1])[0][-1]
        assert np.abs(lg - last[i]).max() < 1e-2 * np.abs(lg).max()
    lib.llmb200_batch_free(b)


class Held:
    """Device memory taken until `room` bytes are left, by the runtime's own allocation call: no pool keeps or rounds it."""

    def __init__(self, room):
        self.rt, self.at = C.CDLL("libcudart.so.12"), []
        torch.cuda.empty_cache()
        for size in (8 << 30, 512 << 20, 32 << 20, 2 << 20):
            while torch.cuda.mem_get_info()[0] - size >= room:
                p = C.c_void_p()
                if self.rt.cudaMalloc(C.byref(p), C.c_size_t(size)) != 0:
                    self.rt.cudaGetLastError()
                    break
                self.at.append(p)

    def free(self):
        for p in self.at:
            self.rt.cudaFree(p)
        self.at = []


@pytest.mark.parametrize("room", [2 << 20, 64 << 20])
def test_prompts_without_memory_for_a_pass(pkg, lib, room):
    """A workspace that cannot be had: smaller passes, then the per-token path, and the same answer. Later calls get it back."""
    cfg, B, G, P = dict(sc.SMALL, intermediate_size=8192, vocab_size=1024), 32, 3, 300
    b, s = states(pkg, lib, cfg, B, G, 1024)
    rng = np.random.default_rng(4)
    prompts = rng.integers(0, 1024, (B, P)).astype(np.uint32)
    few = np.ascontiguousarray(prompts[:, :2])
    assert generate(pkg, lib, b, few, G)[0] == G              # graphs and kernels are loaded before memory runs short
    long = np.random.default_rng(5).integers(0, 1024, 900).astype(np.uint32)
    answer = np.zeros(4, dtype=np.uint32)
    lib.llmb200_state_set_eos(s, None, 0)

    def single():
        lg = np.zeros((2, 1024), dtype=np.float32)
        n = lib.inference_generate(s, long.ctypes.data_as(pkg.c_u32_p), 900, answer.ctypes.data_as(pkg.c_u32_p), 4)
        lib.inference_state_reset(s)
        rc = lib.inference_forward_tokens(s, long.ctypes.data_as(pkg.c_u32_p), 900, (C.c_int * 2)(450, 899), 2, lg.ctypes.data_as(pkg.c_float_p))
        return n, rc, lib.llmb200_state_position(s), lg
    assert lib.inference_generate(s, long.ctypes.data_as(pkg.c_u32_p), 3, answer.ctypes.data_as(pkg.c_u32_p), 4) == 4
    held = Held(room)
    try:
        n, rc, position, lg = single()
        tight, tight_out = generate(pkg, lib, b, prompts, G)
        tight_last = logits_of(pkg, lib, b, B, 1024)
    finally:
        held.free()
    assert n == 4 and rc == 0 and position == 900 and tight == G and lib.llmb200_state_error(s) == 0
    check(pkg, lib, s, prompts, tight_out, tight_last, 1024)
    n, rc, position, wide = single()
    assert n == 4 and rc == 0 and np.abs(wide - lg).max() <= 1e-3 * np.abs(wide).max()
    assert generate(pkg, lib, b, prompts, G)[0] == G
    lib.llmb200_batch_free(b)
    lib.inference_state_free(s)


def test_a_raised_error_word_fails_the_call(pkg, lib):
    """What a kernel whose wait ran out leaves behind: the answer of such a call is not an answer."""
    cfg, B, G, P = dict(sc.SMALL), 2, 3, 20
    b, _ = states(pkg, lib, cfg, B, G, 64, single=False)
    prompts = np.random.default_rng(P).integers(0, 512, (B, P)).astype(np.uint32)
    assert generate(pkg, lib, b, prompts, G)[0] == G and lib.llmb200_batch_error(b) == 0
    word, row = torch.full((4,), 0x7203, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert lib.b200_rows_gather(word.data_ptr(), 1, 4, row.data_ptr(), lib.llmb200_batch_error_word(b), None) == 0      # a copy of 16 bytes
    torch.cuda.synchronize()
    assert lib.llmb200_batch_error(b) == 0x7203 and generate(pkg, lib, b, prompts, G)[0] == 0
    assert generate(pkg, lib, b, np.ascontiguousarray(prompts[:, :2]), G)[0] == 0
    lib.llmb200_batch_free(b)
