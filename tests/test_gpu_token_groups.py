"""Several tokens in one launch of the whole-token kernel: the ids and the state they leave are those of single tokens, bit for bit, wherever a
group ends (end ids, the last position of the cache) and where the number of cache rows that a block stages at a time changes inside one."""
import ctypes as C

import numpy as np
import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def prompt_of(synth, n, vocab):
    p = np.zeros(n, dtype=np.uint32)
    synth.llmb200_synth_tokens(p.ctypes.data, n, 99, vocab)
    return p


def generate(lib, pkg, st, prompt, n):
    out = np.zeros(n, dtype=np.uint32)
    got = lib.inference_generate(st, prompt.ctypes.data_as(pkg.c_u32_p), len(prompt), out.ctypes.data_as(pkg.c_u32_p), n)
    assert lib.llmb200_state_error(st) == 0
    return out[:got]


def logits_after(lib, st, token, vocab):
    p = lib.inference_forward_token(st, int(token))
    assert p and lib.llmb200_state_error(st) == 0
    return np.ctypeslib.as_array(p, shape=(vocab,)).copy()


@pytest.mark.parametrize("fp16", [0, 1])
@pytest.mark.parametrize("name,max_seq,P,G", [("tiny-qwen3", 64, 16, 2), ("tiny-qwen3", 64, 3, 14), ("tiny-qwen3", 64, 59, 32), ("tiny-qwen3", 2048, 600, 23),
                                              ("tiny-gemma3", 64, 1, 9), ("tiny-gemma3", 4096, 420, 61)])
@pytest.mark.parametrize("narrow", ["0", "1"])
def test_groups_give_the_tokens_of_single_launches(lib, pkg, synth, monkeypatch, fp16, name, max_seq, P, G, narrow):
    monkeypatch.setenv("LLMB200_TK_NARROW", narrow)       # both widths of the kernel
    sp = pkg.spec(name, gamma_jitter=0.1)
    gemma = "gemma" in name
    model = (synth.llmb200_synth_gemma3 if gemma else synth.llmb200_synth_qwen3)(C.byref(sp), 8)
    st = (lib.inference_state_create_gemma3 if gemma else lib.inference_state_create)(model, max_seq, fp16)
    assert st
    try:
        V, prompt = sp.vocab_size, prompt_of(synth, P, sp.vocab_size)
        lib.llmb200_state_set_eos(st, None, 0)
        single, rows = list(generate(lib, pkg, st, prompt, 1)), []
        while len(single) < G and P + len(single) <= max_seq:
            rows.append(logits_after(lib, st, single[-1], V))
            single.append(int(rows[-1].argmax()))
        got = list(generate(lib, pkg, st, prompt, G))
        assert got == single[:len(got)] and len(got) == min(G, max_seq - P + 1)
        if len(got) > 2:                                  # stopped inside a group, then going on from there
            at = next((i for i in range(len(got) - 2, 0, -1) if got[i] not in got[:i]), None)
            if at is not None:
                eos = (C.c_int * 1)(int(got[at]))
                lib.llmb200_state_set_eos(st, eos, 1)
                assert list(generate(lib, pkg, st, prompt, G)) == got[:at + 1]
                assert lib.llmb200_state_position(st) == P + at
                assert np.array_equal(logits_after(lib, st, got[at], V), rows[at])
    finally:
        lib.inference_state_free(st)
        (synth.llmb200_synth_free_gemma3 if gemma else synth.llmb200_synth_free_qwen3)(model)


@pytest.mark.parametrize("fp16", [0, 1])
@pytest.mark.parametrize("name", ["tiny-qwen3", "tiny-gemma3"])
def test_widths_agree(lib, pkg, synth, monkeypatch, fp16, name):
    """640 and 320 consumer threads: the same sums in another order. A key or value that this moves across a border of the binary16 cache moves by
    2^-11 of itself, so that is what logits may move by."""
    sp = pkg.spec(name, gamma_jitter=0.1)
    gemma = "gemma" in name
    model = (synth.llmb200_synth_gemma3 if gemma else synth.llmb200_synth_qwen3)(C.byref(sp), 8)
    seen = []
    try:
        for narrow in "01":
            monkeypatch.setenv("LLMB200_TK_NARROW", narrow)
            st = (lib.inference_state_create_gemma3 if gemma else lib.inference_state_create)(model, 64, fp16)
            assert st
            seen.append([logits_after(lib, st, t, sp.vocab_size) for t in prompt_of(synth, 12, sp.vocab_size)])
            lib.inference_state_free(st)
    finally:
        (synth.llmb200_synth_free_gemma3 if gemma else synth.llmb200_synth_free_qwen3)(model)
    a, b = (np.array(x, dtype=np.float64) for x in seen)
    assert not np.array_equal(a, b) and np.abs(a - b).max() <= 2 ** -11 * np.abs(a).max()
