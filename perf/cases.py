"""The work by which the speed of this framework is judged: listed cases, a generator of more of the same ranges, and what each of
them has to give.

A case is one call, or the few calls that belong together, of a program that uses the library: answering a prompt, reading a long
document, decoding a batch, one training step. Every model is a cut of an architecture that the benchmarks run: full widths and heads,
fewer layers, and a vocabulary cut along with them, so that the LM head keeps about the share of a token that it has in the whole model.
Weights are random; the LM head is made so that the next token is clear-cut, as it mostly is for a trained model: greedy
continuations then do not hang on the last bit.
"""
import ctypes as C
import importlib.util
import json
import math
import os
import shutil
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG_NAME = "llmb200"


def package():
    if PKG_NAME not in sys.modules:
        where = os.path.join(ROOT, "llm.metal_b200")
        spec = importlib.util.spec_from_file_location(PKG_NAME, os.path.join(where, "__init__.py"), submodule_search_locations=[where])
        sys.modules[PKG_NAME] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[PKG_NAME])
    return sys.modules[PKG_NAME]


# ------------------------------------------------------------------ architectures (full widths; layers and vocabulary come with the case)

ARCHS = {
    "tiny-qwen3": dict(gemma=0, D=512, Hq=8, Hkv=2, hd=64, IS=1536, theta=1e6),
    "qwen3-4b": dict(gemma=0, D=2560, Hq=32, Hkv=8, hd=128, IS=9728, theta=1e6),
    "gemma3-1b": dict(gemma=1, D=1152, Hq=4, Hkv=1, hd=256, IS=6912, theta=1e6),
}
MORILORN = {256: dict(heads=4, dim=48, rot=16, vdim=64, rank=64, ff=512, window=64),
            2048: dict(heads=16, dim=128, rot=64, vdim=128, rank=512, ff=6144, window=1024)}
ZIDEPEL = {256: dict(heads=4, kv=1, dim=48, vdim=64, gla=24, rank=8, ff=512, streams=2),
           2048: dict(heads=16, kv=4, dim=128, vdim=128, gla=64, rank=16, ff=6144, streams=4)}
EPS = 1e-6
RANK_ALPHA = 2.0               # alpha / rank of the adapters (rank 16, alpha 32)
LR = 1e-4


def listed():
    four_b = dict(arch="qwen3-4b", layers=4, vocab=16384)
    return [
        # the smallest calls: a few tokens with a small model, launches and host work count
        dict(name="tiny-q8-chat", kind="generate", arch="tiny-qwen3", layers=4, vocab=4096, weights="q8", prompt=16, new=32),
        # an ordinary prompt read up to its first answer token, the default weight format
        dict(name="4b-q8-prompt", kind="prompt", weights="q8", prompt=512, **four_b),
        # a short question with a long answer: the per-token path
        dict(name="4b-q8-chat", kind="generate", weights="q8", prompt=48, new=256, **four_b),
        # a document of odd length, binary16 weights
        dict(name="4b-f16-document", kind="prompt", weights="f16", prompt=1531, **four_b),
        # Gemma3 blocks (four norms, GeGLU, heads of 256), binary16 weights, prompt and answer
        dict(name="gemma-f16-chat", kind="generate", arch="gemma3-1b", layers=6, vocab=32768, weights="f16", prompt=128, new=256),
        # many sequences at once
        dict(name="4b-batch32", kind="batch", batch=32, prompt=128, new=128, **four_b),
        # a training step of short sequences, and of one long ragged one
        dict(name="4b-lora-8x64", kind="lora", seqs=8, seq=64, rank=16, **four_b),
        dict(name="4b-lora-1x509", kind="lora", seqs=1, seq=509, rank=16, **four_b),
        # every weight trained, products in 32 bits
        dict(name="gemma-full-64", kind="full", arch="gemma3-1b", layers=2, vocab=8192, seq=64),
        # models from folders: a long prompt, a ragged one with an answer, and the 32-bit option
        dict(name="morilorn-prompt", kind="folder", model="morilorn", width=2048, layers=4, vocab=16384, dtype="bfloat16", prompt=2048, new=0),
        dict(name="zidepel-chat", kind="folder", model="zidepel", width=2048, layers=4, vocab=16384, dtype="bfloat16", prompt=777, new=64),
        dict(name="morilorn-f32-chat", kind="folder", model="morilorn", width=2048, layers=2, vocab=16384, dtype="float32", prompt=33, new=64),
    ]


def draw(rng):
    def log(lo, hi):
        return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))
    kind = rng.choice(["generate", "generate", "prompt", "prompt", "batch", "lora", "full", "folder", "folder", "folder"])
    if kind in ("generate", "prompt"):
        arch = rng.choice(["tiny-qwen3", "qwen3-4b", "gemma3-1b"])
        c = dict(kind=kind, arch=arch, layers=rng.randint(2, 6 if arch != "qwen3-4b" else 4), vocab=rng.choice([4096, 8192, 16384]),
                 weights=rng.choice(["q8", "f16"]), prompt=log(1 if kind == "generate" else 2, 256 if kind == "generate" else 1531))
        if kind == "generate":
            c["new"] = log(8, 192)
        return c
    if kind == "batch":
        return dict(kind="batch", arch=rng.choice(["tiny-qwen3", "qwen3-4b"]), layers=rng.randint(2, 4), vocab=rng.choice([4096, 8192, 16384]),
                    batch=rng.randint(1, 32), prompt=log(4, 128), new=log(4, 128))
    if kind == "lora":
        seq = log(16, 509)
        return dict(kind="lora", arch=rng.choice(["tiny-qwen3", "qwen3-4b"]), layers=rng.randint(2, 4), vocab=rng.choice([4096, 8192, 16384]),
                    seq=seq, seqs=rng.randint(1, max(1, 512 // seq)), rank=rng.choice([4, 8, 16]))
    if kind == "full":
        return dict(kind="full", arch=rng.choice(["tiny-qwen3", "gemma3-1b"]), layers=2, vocab=rng.choice([4096, 8192]), seq=log(8, 64))
    model, width = rng.choice(["morilorn", "zidepel"]), rng.choice([256, 2048])
    dtype = rng.choice(["bfloat16", "bfloat16", "float32"])
    new = rng.choice([0, log(4, 64)])
    return dict(kind="folder", model=model, width=width, layers=rng.randint(1, 2) * 2, vocab=rng.choice([4096, 8192, 16384]), dtype=dtype,
                prompt=log(8, (2048 if new == 0 else 800) if dtype == "bfloat16" else 64), new=new)


# ------------------------------------------------------------------ weights

POOL = 1 << 26
_kept = {}


def pool():
    """One block of normal values: every matrix is a stretch of it."""
    if "pool" not in _kept:
        g = torch.Generator().manual_seed(20)
        _kept["pool"] = torch.randn(POOL, generator=g)
    return _kept["pool"]


def stretch(shape, at, std):
    n = math.prod(shape)
    key = ("scaled", std)
    if key not in _kept:
        _kept[key] = pool() * std
    start = (at * 1048583 * 61) % (POOL - n)
    return _kept[key][start:start + n].view(shape)


def gamma(n, at):
    return (1.0 + 0.1 * stretch((n,), at, 1.0)).contiguous()


def successor(V):
    """The token that the model holds for the likeliest after each token: the LM head's row successor[t] leans on t's embedding."""
    return (torch.arange(V) * 5 + 1) % V


def embedding_and_head(V, D, emb_std, lean=0.02):
    emb = stretch((V, D), 900, emb_std)
    head = torch.empty(V, D)
    head[successor(V)] = emb * (lean / emb_std)
    return emb, head


def plain_model(case):
    """Weights of a Qwen3 or Gemma3 cut, 32-bit, on the host; kept for the process: a program loads its model once."""
    key = ("model", case["arch"], case["layers"], case["vocab"])
    if key in _kept:
        return _kept[key]
    for k in [k for k in _kept if k[0] == "model"]:
        del _kept[k]
    a, V = ARCHS[case["arch"]], case["vocab"]
    D, hd = a["D"], a["hd"]
    shapes = dict(q=(a["Hq"] * hd, D), k=(a["Hkv"] * hd, D), v=(a["Hkv"] * hd, D), o=(D, a["Hq"] * hd), gate=(a["IS"], D), up=(a["IS"], D),
                  down=(D, a["IS"]))
    layers = []
    for i in range(case["layers"]):
        w = {n: stretch(s, 1 + i * 16 + j, 0.02) for j, (n, s) in enumerate(shapes.items())}
        w.update({n: gamma(D, 500 + i * 16 + j) for j, n in enumerate(["input", "post_attn"] + (["pre_ff", "post_ff"] if a["gemma"] else []))})
        w.update(q_norm=gamma(hd, 700 + i), k_norm=gamma(hd, 750 + i))
        w["theta"] = 1e4 if a["gemma"] and i % 6 else a["theta"]
        layers.append(w)
    emb, head = embedding_and_head(V, D, 0.1 if a["gemma"] else 1.0)
    _kept[key] = dict(a=a, V=V, layers=layers, emb=emb, head=head, final=gamma(D, 800))
    return _kept[key]


def ptr(t):
    return C.cast(t.data_ptr(), package().c_float_p)


def layer_ref(m, w):
    pkg, a = package(), m["a"]
    r = pkg.LayerWeightRef()
    for name, k in (("q_proj", "q"), ("k_proj", "k"), ("v_proj", "v"), ("o_proj", "o"), ("gate_proj", "gate"), ("up_proj", "up"), ("down_proj", "down")):
        setattr(r, name, pkg.WeightRef(ptr(w[k]), *w[k].shape))
    r.input_norm_g, r.post_attn_norm_g, r.q_norm_g, r.k_norm_g = ptr(w["input"]), ptr(w["post_attn"]), ptr(w["q_norm"]), ptr(w["k_norm"])
    if a["gemma"]:
        r.pre_ff_norm_g, r.post_ff_norm_g = ptr(w["pre_ff"]), ptr(w["post_ff"])
    r.d_model, r.head_dim = a["D"], a["hd"]
    return r


def config(m, max_seq, use_fp16):
    a = m["a"]
    return package().Config(1 if a["gemma"] else 0, a["D"], a["Hq"], a["Hkv"], a["hd"], a["IS"], m["V"], len(m["layers"]), max_seq, use_fp16)


class Owned:
    """A handle of the library that is given back with the Python object."""

    def __init__(self, handle, free):
        if not handle:
            raise RuntimeError("the library refused to create the state")
        self.h, self._free = handle, free

    def __del__(self):
        if self.h:
            self._free(self.h)
            self.h = None


def ok(rc):
    if rc != 0:
        raise RuntimeError(f"a call failed with code {rc}")


def tokens(n, V, seed):
    return np.random.default_rng(seed).integers(0, V, n).astype(np.uint32)


def u32(a):
    return a.ctypes.data_as(package().c_u32_p)


# ------------------------------------------------------------------ decode states

def prepare_plain(case, seed):
    L, m = package().lib(), plain_model(case)
    cfg = config(m, 4096 if case["prompt"] > 512 else 1024, 1 if case["weights"] == "f16" else 0)
    s = Owned(L.llmb200_state_begin(C.byref(cfg)), L.inference_state_free)
    for i, w in enumerate(m["layers"]):
        ok(L.llmb200_state_load_layer(s.h, i, C.byref(layer_ref(m, w)), w["theta"]))
    ok(L.llmb200_state_finish(s.h, ptr(m["head"]), ptr(m["final"]), ptr(m["emb"])))
    L.llmb200_state_set_eos(s.h, None, 0)
    P = case["prompt"]
    return dict(case=case, L=L, s=s, tokens=tokens(P, m["V"], seed), out=np.zeros(case.get("new", 0), np.uint32),
                logits=np.zeros((2 if P > 2 else 1, m["V"]), np.float32))


def wanted(P):
    return [P // 2, P - 1] if P > 2 else [P - 1]


def run_plain(st):
    L, s, P = st["L"], st["s"].h, st["case"]["prompt"]
    if st["case"]["kind"] == "prompt":
        want = wanted(P)
        L.inference_state_reset(s)
        ok(L.inference_forward_tokens(s, u32(st["tokens"]), P, (C.c_int * len(want))(*want), len(want),
                                      st["logits"].ctypes.data_as(package().c_float_p)))
        return {"logits": st["logits"]}
    n = L.inference_generate(s, u32(st["tokens"]), P, u32(st["out"]), len(st["out"]))
    logits = L.inference_forward_token(s, int(st["out"][n - 1]))        # what comes after the answer
    return {"tokens": st["out"][:n], "logits": np.ctypeslib.as_array(logits, (st["logits"].shape[1],)).copy()}


# ------------------------------------------------------------------ batches

def prepare_batch(case, seed):
    L, m, B = package().lib(), plain_model(case), case["batch"]
    cfg = config(m, 512, 1)
    s = Owned(L.llmb200_batch_begin(C.byref(cfg), B, case["new"]), L.llmb200_batch_free)
    for i, w in enumerate(m["layers"]):
        ok(L.llmb200_batch_load_layer(s.h, i, C.byref(layer_ref(m, w)), w["theta"]))
    ok(L.llmb200_batch_finish(s.h, ptr(m["head"]), ptr(m["final"]), ptr(m["emb"])))
    L.llmb200_batch_set_eos(s.h, None, 0)
    return dict(case=case, L=L, s=s, tokens=tokens(B * case["prompt"], m["V"], seed), out=np.zeros((B, case["new"]), np.uint32),
                logits=np.zeros((B, m["V"]), np.float32))


def run_batch(st):
    c, L = st["case"], st["L"]
    if L.llmb200_batch_generate(st["s"].h, u32(st["tokens"]), c["prompt"], u32(st["out"]), c["new"]) != c["new"]:
        raise RuntimeError("batch generation failed")
    L.llmb200_batch_logits(st["s"].h, st["logits"].ctypes.data_as(package().c_float_p), st["logits"].size)
    return {"tokens": st["out"], "logits": st["logits"]}


# ------------------------------------------------------------------ training

class DeviceVector:
    """fp32 values that a state of the library owns, for torch.as_tensor, which keeps this object and with it the state."""

    def __init__(self, owner, address, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f4", "data": (address, False), "version": 2}


def adapters(m, rank):
    """A as after initialisation; B not zero: a step in the middle of training."""
    a = m["a"]
    return [(stretch((rank, a["D"]), 1000 + i * 4, 0.01), stretch((a["Hq"] * a["hd"], rank), 1001 + i * 4, 0.01),
             stretch((rank, a["D"]), 1002 + i * 4, 0.01), stretch((a["Hkv"] * a["hd"], rank), 1003 + i * 4, 0.01))
            for i in range(len(m["layers"]))]


def sequences(case, seed):
    n = case.get("seqs", 2)
    t = tokens(n * (case["seq"] + 1), case["vocab"], seed).reshape(n, case["seq"] + 1)
    return np.ascontiguousarray(t[:, :-1]), np.ascontiguousarray(t[:, 1:])


def prepare_lora(case, seed):
    pkg = package()
    L, m, R = pkg.lib(), plain_model(case), case["rank"]
    cfg = config(m, case["seq"], 1)
    s = Owned(L.llmb200_sft_begin(C.byref(cfg), case["seq"], case["seqs"], R, RANK_ALPHA * R), L.sft_state_free)
    for i, (w, ad) in enumerate(zip(m["layers"], adapters(m, R))):
        ok(L.llmb200_sft_load_layer(s.h, i, C.byref(layer_ref(m, w)), w["theta"], C.byref((pkg.c_float_p * 4)(*[ptr(x) for x in ad]))))
    ok(L.llmb200_sft_finish(s.h, ptr(m["head"]), ptr(m["final"]), ptr(m["emb"]), 0))
    views = []
    for call in (L.llmb200_sft_grad_vector, L.llmb200_sft_param_vector):
        p = C.c_void_p()
        n = call(s.h, C.byref(p))
        views.append(torch.as_tensor(DeviceVector(s, p.value, n), device="cuda"))
    return dict(case=case, L=L, s=s, io=sequences(case, seed), views=views)


def run_lora(st):
    loss = st["L"].llmb200_sft_train_batch(st["s"].h, u32(st["io"][0]), u32(st["io"][1]), LR)
    return {"loss": float(loss), "gradients": st["views"][0], "adapter": st["views"][1]}


def synthetic(case):
    """The library's own seeded model structure of a cut."""
    pkg = package()
    key = ("synth", case["arch"], case["layers"], case["vocab"])
    if key not in _kept:
        sp = pkg.spec(case["arch"], n_layers=case["layers"], vocab_size=case["vocab"], gamma_jitter=0.1)
        make = pkg.synth().llmb200_synth_gemma3 if ARCHS[case["arch"]]["gemma"] else pkg.synth().llmb200_synth_qwen3
        _kept[key] = (sp, make(C.byref(sp), min(16, os.cpu_count() or 1)))
    return _kept[key]


FULL_LR = 1e-2


def prepare_full(case, seed):
    L = package().lib()
    model = synthetic(case)[1]
    make = L.sft_state_create_gemma3_full if ARCHS[case["arch"]]["gemma"] else L.sft_state_create_full
    s = Owned(make(model, case["seq"]), L.sft_state_free)
    return dict(case=case, L=L, s=s, io=sequences(case, seed), logits=np.zeros((case["seq"], case["vocab"]), np.float32))


def run_full(st):
    """Two steps on two sequences: what the second one sees is the model that the first one stepped."""
    L, s, (x, y) = st["L"], st["s"].h, st["io"]
    losses = [float(L.sft_train_step(s, u32(x[i]), u32(y[i]), FULL_LR)) for i in range(2)]
    LOGITS = 100                                                        # LLMB200_SFT_LOGITS
    if L.llmb200_sft_export(s, LOGITS, 0, st["logits"].ctypes.data_as(package().c_float_p), st["logits"].size) == 0:
        raise RuntimeError("reading the logits failed")
    return {"losses": losses, "logits": st["logits"]}


# ------------------------------------------------------------------ models in folders

def folder_config(case):
    D, V = case["width"], case["vocab"]
    if case["model"] == "morilorn":
        z = MORILORN[D]
        layer = {"type": "latent_attention", "mlp": {"kind": "dense", "ff": z["ff"]},
                 "mixer": {"heads": z["heads"], "dim": z["dim"], "rot_dim": z["rot"], "vdim": z["vdim"], "kv_rank": z["rank"],
                           "mask": {"size": z["window"]}, "rot": {"base": 10000.0, "dims": z["rot"]}, "scale": (z["dim"] + z["rot"]) ** -0.5}}
        return {"architecture": "Morilorn", "vocab": V, "width": D, "embedding": {"scale": 8.0}, "norm": {"eps": EPS, "groups": 4},
                "postln_alpha": 2.0, "logit_softcap": 30.0, "layers": [layer] * case["layers"]}
    z = ZIDEPEL[D]
    attn = {"type": "attention", "mlp": {"kind": "dense", "ff": z["ff"]},
            "mixer": {"heads": z["heads"], "kv_heads": z["kv"], "dim": z["dim"], "vdim": z["vdim"], "scale": z["dim"] ** -0.5, "softcap": 40.0,
                      "q_temp": {"coef": 0.1, "every": 1000}}}
    rec = {"type": "gla", "mlp": {"kind": "dense", "ff": z["ff"]}, "mixer": {"heads": z["heads"], "dim": z["gla"], "vdim": z["vdim"], "tau": 16.0}}
    return {"architecture": "Zidepel", "vocab": V, "width": D, "streams": z["streams"], "max_positions": 4096, "norm": {"eps": EPS},
            "loop": {"start": 0, "stop": 2, "times": 2}, "layers": [rec if i % 4 == 0 else attn for i in range(case["layers"])]}


def folder_weights(case):
    """name -> bfloat16 values (as 32-bit), in the file's order."""
    key = ("model", case["model"], case["width"], case["layers"], case["vocab"])
    if key in _kept:
        return _kept[key]
    for k in [k for k in _kept if k[0] == "model"]:
        del _kept[k]
    D, V = case["width"], case["vocab"]
    w, at = {}, [0]

    def mat(name, *shape, std=0.02):
        at[0] += 1
        w[name] = stretch(shape, at[0], std)

    def vec(name, n, value, std):
        at[0] += 1
        w[name] = value + stretch((n,), at[0], 1.0) * std
    emb, head = embedding_and_head(V, D, 0.25 if case["model"] == "morilorn" else 1.0)
    w["embed"], w["head"] = emb, head
    vec("final.norm", D, 1.0, 0.1)
    if case["model"] == "morilorn":
        z = MORILORN[D]
        H, F = z["heads"], z["ff"]
        for i in range(case["layers"]):
            p = f"l{i}."
            for n in ("norm1", "norm2"):
                vec(p + n, D, 1.0, 0.1)
            for n in ("rg1", "rg2"):
                mat(p + n, D, D)
                vec(p + n + ".b", D, 0.0, 0.2)
            mat(p + "mix.q", H * (z["dim"] + z["rot"]), D, std=0.04)
            mat(p + "mix.dkv", z["rank"] + z["rot"], D, std=0.04)
            vec(p + "mix.dkv.norm", z["rank"], 1.0, 0.1)
            mat(p + "mix.uk", H * z["dim"], z["rank"], std=0.04)
            mat(p + "mix.uv", H * z["vdim"], z["rank"], std=0.04)
            mat(p + "mix.g", H * z["vdim"], D)
            mat(p + "mix.o", D, H * z["vdim"])
            mat(p + "mlp.gate", F, D)
            mat(p + "mlp.up", F, D)
            mat(p + "mlp.down", D, F)
            w[p + "dwa"] = torch.full((i + 2,), 0.125)
            w[p + "dwa"][-1] = 1.0
    else:
        z = ZIDEPEL[D]
        H, F, n = z["heads"], z["ff"], z["streams"]
        vec("embed.norm", D, 1.0, 0.1)
        mat("pos", 4096, D)
        for k in ("embed.norm.b", "final.norm.b"):
            vec(k, D, 0.0, 0.05)
        for i, layer in enumerate(folder_config(case)["layers"]):
            p = f"l{i}."
            for q in (1, 2):
                vec(f"{p}norm{q}", D, 1.0, 0.1)
                vec(f"{p}norm{q}.b", D, 0.0, 0.05)
                vec(f"{p}hc{q}.in", n, 1.0 / n, 0.05)
                vec(f"{p}hc{q}.out", n, 0.5, 0.1)
                at[0] += 1
                w[f"{p}hc{q}.mix"] = 0.9 * torch.eye(n) + 0.05 * stretch((n, n), at[0], 1.0)
            d = z["dim"] if layer["type"] == "attention" else z["gla"]
            mat(p + "mix.q", H * d, D)
            if layer["type"] == "attention":
                mat(p + "mix.k", z["kv"] * d, D)
                mat(p + "mix.v", z["kv"] * z["vdim"], D)
                vec(p + "mix.q.norm", d, 1.0, 0.1)
                vec(p + "mix.k.norm", d, 1.0, 0.1)
            else:
                w[p + "mix.k"] = 0.7 * w[p + "mix.q"] + 0.7 * stretch((H * d, D), at[0] + 300, 0.02)
                mat(p + "mix.v", H * z["vdim"], D)
                mat(p + "mix.g", H * z["vdim"], D)
                vec(p + "mix.norm", z["vdim"], 1.0, 0.1)
                mat(p + "mix.a1", z["rank"], D)
                mat(p + "mix.a2", H * d, z["rank"], std=0.25)
                vec(p + "mix.a2.b", H * d, 2.0, 1.0)
            mat(p + "mix.o", D, H * z["vdim"])
            mat(p + "mlp.up", F, D)
            mat(p + "mlp.down", D, F)
    _kept[key] = {k: v.to(torch.bfloat16) for k, v in w.items()}
    return _kept[key]


def prepare_folder(case, seed):
    pkg = package()
    w = folder_weights(case)
    folder = tempfile.mkdtemp(prefix="model-")
    try:
        with open(os.path.join(folder, "config.json"), "w") as f:
            json.dump(folder_config(case), f)
        header, at = {}, 0
        for k, v in w.items():
            header[k] = {"dtype": "BF16", "shape": list(v.shape), "data_offsets": [at, at + 2 * v.numel()]}
            at += 2 * v.numel()
        text = json.dumps(header).encode()
        with open(os.path.join(folder, "model.safetensors"), "wb") as f:
            f.write(len(text).to_bytes(8, "little") + text)
            for v in w.values():
                f.write(v.contiguous().view(torch.int16).numpy().data)
        model = pkg.DirModel(folder, 4096, case["dtype"])
    finally:
        shutil.rmtree(folder)
    s = Owned(model.state, pkg.lib().inference_state_free)
    return dict(case=case, s=s, model=model, tokens=tokens(case["prompt"], case["vocab"], seed).tolist())


def run_folder(st):
    c, m = st["case"], st["model"]
    if c["new"] == 0:
        m.reset()
        return {"logits": np.ctypeslib.as_array(m.feed(st["tokens"], wanted(c["prompt"])))}
    out = m.generate(st["tokens"], c["new"], eos=[])
    return {"tokens": np.array(out, dtype=np.int64), "logits": np.ctypeslib.as_array(m.feed([out[-1]], [0]))}


# ------------------------------------------------------------------ what the measurement calls

PREPARE = {"generate": prepare_plain, "prompt": prepare_plain, "batch": prepare_batch, "lora": prepare_lora, "full": prepare_full,
           "folder": prepare_folder}
RUN = {"generate": run_plain, "prompt": run_plain, "batch": run_batch, "lora": run_lora, "full": run_full, "folder": run_folder}


def prepare(case, seed):
    return PREPARE[case["kind"]](case, seed)


def run(state):
    return RUN[state["case"]["kind"]](state)


def parameters(case):
    """(weights of the layers as they run once for a token, weights of the LM head, width, cache values of a position)"""
    V = case["vocab"]
    if case["kind"] != "folder":
        a = ARCHS[case["arch"]]
        D, q, kv = a["D"], a["Hq"] * a["hd"], a["Hkv"] * a["hd"]
        return case["layers"] * ((q + 2 * kv) * D + q * D + 3 * a["IS"] * D), V * D, D, case["layers"] * 2 * kv
    D = case["width"]
    if case["model"] == "morilorn":
        z = MORILORN[D]
        H, r = z["heads"], z["rank"] + z["rot"]
        one = H * (z["dim"] + z["rot"]) * D + r * D + H * (z["dim"] + z["vdim"]) * z["rank"] + 2 * H * z["vdim"] * D + 3 * z["ff"] * D + 2 * D * D
        return case["layers"] * one, V * D, D, case["layers"] * r
    z, n, cache = ZIDEPEL[D], 0, 0
    kinds = [layer["type"] for layer in folder_config(case)["layers"]]
    for t in kinds[:2] * 2 + kinds[2:]:
        H = z["heads"]
        if t == "attention":
            n += H * z["dim"] * D + z["kv"] * (z["dim"] + z["vdim"]) * D + H * z["vdim"] * D + 2 * z["ff"] * D
            cache += z["kv"] * (z["dim"] + z["vdim"])
        else:
            n += 2 * H * z["gla"] * D + 3 * H * z["vdim"] * D + z["rank"] * (D + H * z["gla"]) + 2 * z["ff"] * D
    return n, V * D, D, cache


def work(case):
    body, head, D, cache = parameters(case)
    kind = case["kind"]
    if kind in ("lora", "full"):
        M = case["seq"] * case.get("seqs", 2)
        if kind == "lora":
            return {"bytes": 2.0 * (body + head) + 4.0 * M * D, "flops": 4.0 * M * (body + head)}
        return {"bytes": 2 * (2.0 + 2.0) * (body + head) + 4.0 * M * D + 2.0 * M * case["vocab"], "flops": 6.0 * M * (body + head)}
    size = {"q8": 34 / 32, "f16": 2.0, "bfloat16": 2.0, "float32": 4.0}[case.get("weights", case.get("dtype", "f16"))]
    store = {"float32": 4.0}.get(case.get("dtype"), 2.0)
    P, G, B = case["prompt"], case.get("new", 0), case.get("batch", 1)
    ends = len(wanted(P)) if G == 0 else 1
    steps = max(0, G - 1 + (kind != "batch" and G > 0))   # tokens after the prompt that go through the model one by one
    kv_read = sum(P + i for i in range(steps))
    return {"bytes": size * (body * (1 + steps) + head * (1 + steps)) + B * (4.0 * D * (P + steps) + store * cache * (P + steps + kv_read)),
            "flops": 2.0 * B * (body * (P + steps) + head * (ends + steps))}


def tolerance(case):
    """About four times the error measured against exact(): the binary16 cache of the single states (1e-4 to 2.2e-4), the binary16
    operands of batches (6e-4) and adapters (1e-3), the binary16 weights that a full step rounds to (3e-4), bfloat16 operands (1.8e-3), fp32."""
    if case["kind"] == "folder":
        rel = 1e-2 if case["dtype"] == "bfloat16" else 1e-5
    else:
        rel = {"generate": 1e-3, "prompt": 1e-3, "batch": 3e-3, "lora": 4e-3, "full": 1.5e-3}[case["kind"]]
    return {"rel": rel, "differ": 0.005}


# ------------------------------------------------------------------ the same in 64 bits

def q8(w):
    """Values of a matrix held as Q8_0: blocks of 32, a binary16 scale each."""
    b = w.float().view(w.shape[0], -1, 32)
    d = b.abs().amax(-1, keepdim=True) / 127.0
    q = torch.where(d > 0, b / torch.where(d > 0, d, torch.ones_like(d)), torch.zeros_like(b))
    q = torch.sign(q) * torch.floor(q.abs() + 0.5)
    return (q.clamp(-127, 127).double() * d.half().double()).view(w.shape)


def rms(x, g):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * g


def rotary(x, theta):
    """x [..., n, hd], halves."""
    n, hd = x.shape[-2:]
    d = torch.arange(hd // 2, device=x.device, dtype=torch.float32)
    f = (1.0 / torch.pow(torch.tensor(theta, device=x.device), 2 * d / hd)).float()
    ang = (torch.arange(n, device=x.device, dtype=torch.float32)[:, None] * f).double()
    c, s = ang.cos(), ang.sin()
    a, b = x[..., : hd // 2], x[..., hd // 2:]
    return torch.cat([a * c - b * s, a * s + b * c], -1)


def causal(q, k, v, scale, cap=None, window=None):
    """[..., H, n, d]; heads share keys in groups"""
    n = q.shape[-2]
    i = torch.arange(n, device=q.device)
    hide = (i[:, None] < i[None, :]) | ((i[:, None] - i[None, :] >= window) if window else False)
    out, g = [], q.shape[-3] // k.shape[-3]
    for h in range(q.shape[-3]):
        s = q[..., h, :, :] @ k[..., h // g, :, :].transpose(-1, -2) * scale
        s = cap * torch.tanh(s / cap) if cap else s
        out.append(torch.softmax(s.masked_fill(hide, -math.inf), -1) @ v[..., h // g, :, :])
    return torch.stack(out, -3)


def gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def plain_hidden(a, layers, emb, final, toks, lora=None):
    """Normed last hidden states [S, n, D] of tokens [S, n]."""
    x = emb[toks] * (float(np.sqrt(np.float32(a["D"]))) if a["gemma"] else 1.0)
    S, n, _ = x.shape

    def heads(t, h):
        return t.view(S, n, h, a["hd"]).transpose(1, 2)
    for i, w in enumerate(layers):
        h = rms(x, w["input"])
        q, k, v = h @ w["q"].T, h @ w["k"].T, h @ w["v"].T
        if lora is not None:
            aq, bq, av, bv = lora[i]
            q, v = q + RANK_ALPHA * (h @ aq.T @ bq.T), v + RANK_ALPHA * (h @ av.T @ bv.T)
        q, k = (rotary(rms(heads(t, c), g), w["theta"]) for t, c, g in ((q, a["Hq"], w["q_norm"]), (k, a["Hkv"], w["k_norm"])))
        o = causal(q, k, heads(v, a["Hkv"]), a["hd"] ** -0.5).transpose(1, 2).reshape(S, n, -1) @ w["o"].T
        x = x + (rms(o, w["post_attn"]) if a["gemma"] else o)
        h = rms(x, w["pre_ff"] if a["gemma"] else w["post_attn"])
        g, u = h @ w["gate"].T, h @ w["up"].T
        f = ((gelu(g) if a["gemma"] else g * torch.sigmoid(g)) * u) @ w["down"].T
        x = x + (rms(f, w["post_ff"]) if a["gemma"] else f)
    return rms(x, final)


MATS = ("q", "k", "v", "o", "gate", "up", "down")


def exact_weights(m, held):
    layers = [{k: (held(t.cuda()) if k in MATS else t if k == "theta" else t.cuda().double()) for k, t in w.items()} for w in m["layers"]]
    return layers, held(m["head"].cuda()), m["final"].cuda().double(), m["emb"].cuda().double()


def half_values(t):
    return t.half().double()


def chain(last, n, V):
    """n greedy tokens after `last`, as the LM head has them."""
    nxt, out = successor(V), []
    for _ in range(n):
        last = nxt[last]
        out.append(last)
    return torch.stack(out, -1)


def exact_plain(case, seed):
    m = plain_model(case)
    layers, head, final, emb = exact_weights(m, q8 if case.get("weights") == "q8" else half_values)
    B, P, G = case.get("batch", 1), case["prompt"], case.get("new", 0)
    t = torch.from_numpy(tokens(B * P, m["V"], seed).astype(np.int64)).view(B, P)
    if G:
        t = torch.cat([t, chain(t[:, -1], G, m["V"])], 1)
    if case["kind"] == "batch":
        hs = torch.cat([plain_hidden(m["a"], layers, emb, final, row[None, :-1].cuda())[:, -1] for row in t])
        return {"tokens": t[:, P:].numpy(), "logits": (hs @ head.T).cpu().numpy()}
    hs = plain_hidden(m["a"], layers, emb, final, t.cuda())[0]
    if case["kind"] == "prompt":
        return {"logits": (hs[wanted(P)] @ head.T).cpu().numpy()}
    return {"tokens": t[0, P:].numpy(), "logits": (hs[-1] @ head.T).cpu().numpy()}


def exact_lora(case, seed):
    m = plain_model(case)
    layers, head, final, emb = exact_weights(m, half_values)
    lora = [[x.cuda().double().requires_grad_() for x in ad] for ad in adapters(m, case["rank"])]
    flat = [x for ad in lora for x in ad]
    total, S = 0.0, case["seqs"]
    for x, y in zip(*sequences(case, seed)):
        x, y = (torch.from_numpy(v.astype(np.int64)).cuda() for v in (x, y))
        loss = torch.nn.functional.cross_entropy(plain_hidden(m["a"], layers, emb, final, x[None], lora)[0] @ head.T, y) / S
        loss.backward()
        total += float(loss)
    g = torch.cat([x.grad.reshape(-1) for x in flat])
    p = torch.cat([x.detach().reshape(-1) for x in flat])
    c = g / max(1.0, float(g.norm()))
    stepped = p - LR * (c / (c.abs() + 1e-8) + 0.01 * p)
    return {"loss": total, "gradients": g, "adapter": stepped}


def exact_full(case, seed):
    """The weights come from the same generator that fills the library's model structure."""
    pkg, (sp, _) = package(), synthetic(case)
    S, a, V = pkg.synth(), ARCHS[case["arch"]], case["vocab"]

    def mat(shape, at, mean=0.0, std=sp.weight_std):
        x = np.empty(math.prod(shape), np.float32)
        S.llmb200_synth_normal(x.ctypes.data, x.size, sp.seed, at, mean, std, min(16, os.cpu_count() or 1))
        return torch.from_numpy(x).view(shape).cuda()
    D, hd = a["D"], a["hd"]
    shapes = [(a["Hq"] * hd, D), (a["Hkv"] * hd, D), (a["Hkv"] * hd, D), (D, a["Hq"] * hd), (a["IS"], D), (a["IS"], D), (D, a["IS"])]
    layers = []
    norms = [("q_norm", hd, 7), ("k_norm", hd, 8), ("input", D, 9), ("post_attn", D, 10)] + ([("pre_ff", D, 11), ("post_ff", D, 12)] if a["gemma"] else [])
    for i in range(case["layers"]):
        w = {k: half_values(mat(s, S.llmb200_synth_tensor_id(i, j))) for j, (k, s) in enumerate(zip(MATS, shapes))}
        for k, n, at in norms:
            w[k] = mat((n,), S.llmb200_synth_tensor_id(i, at), 1.0, sp.gamma_jitter).double()
        w["theta"] = 1e4 if a["gemma"] and i % 6 else a["theta"]
        layers.append(w)
    emb = mat((V, D), S.llmb200_synth_tensor_id(0, 100))
    head = half_values(emb if a["gemma"] else mat((V, D), S.llmb200_synth_tensor_id(0, 101)))
    final = mat((D,), S.llmb200_synth_tensor_id(0, 102), 1.0, sp.gamma_jitter).double()
    xs, ys = (torch.from_numpy(v.astype(np.int64)).cuda() for v in sequences(case, seed))
    losses = []
    for x, y in zip(xs, ys):
        with torch.enable_grad():
            held = [w[k].requires_grad_() for w in layers for k in MATS] + [head.requires_grad_()]
            z = plain_hidden(a, layers, emb.double(), final, x[None])[0] @ head.T
            loss = torch.nn.functional.cross_entropy(z, y)
            grads = torch.autograd.grad(loss, held)
        losses.append(float(loss.detach()))
        stepped = [half_values((p - FULL_LR * g).detach()) for p, g in zip(held, grads)]
        head = stepped.pop()
        layers = [dict(w, **dict(zip(MATS, stepped[i * len(MATS):]))) for i, w in enumerate(layers)]
    return {"losses": losses, "logits": z.detach()}


def group_rms(x, g, groups):
    y = x.view(*x.shape[:-1], groups, -1)
    return (y * torch.rsqrt(y.square().mean(-1, keepdim=True) + EPS)).reshape(x.shape) * g


def pairs(x, base, dims):
    """[n, ..., d]: neighbouring pairs turned by their position's angle."""
    a = torch.arange(len(x), device=x.device).double()[:, None] * base ** (-torch.arange(0, dims, 2, device=x.device).double() / dims)
    c, s = (f.view(len(x), *[1] * (x.dim() - 2), -1) for f in (a.cos(), a.sin()))
    out = x.clone()
    e, o = x[..., 0:dims:2], x[..., 1:dims:2]
    out[..., 0:dims:2], out[..., 1:dims:2] = e * c - o * s, o * c + e * s
    return out


def morilorn_hidden(cfg, w, toks):
    x = w["embed"][toks] * cfg["embedding"]["scale"]
    n, groups, alpha, results = len(toks), cfg["norm"]["groups"], cfg["postln_alpha"], [x]
    for i, layer in enumerate(cfg["layers"]):
        m, p = layer["mixer"], f"l{i}."
        H, d, R, rot = m["heads"], m["dim"], m["kv_rank"], m["rot"]
        q = (x @ w[p + "mix.q"].T).view(n, H, -1)
        q = torch.cat([q[..., :d], pairs(q[..., d:], rot["base"], rot["dims"])], -1)
        kv = x @ w[p + "mix.dkv"].T
        c, kr = rms(kv[:, :R], w[p + "mix.dkv.norm"]), pairs(kv[:, R:], rot["base"], rot["dims"])
        k = torch.cat([(c @ w[p + "mix.uk"].T).view(n, H, d), kr[:, None].expand(n, H, -1)], -1)
        v = (c @ w[p + "mix.uv"].T).view(n, H, -1)
        o = causal(q.transpose(0, 1), k.transpose(0, 1), v.transpose(0, 1), m["scale"], window=m["mask"]["size"]).transpose(0, 1).reshape(n, -1)
        y = (o * torch.sigmoid(x @ w[p + "mix.g"].T)) @ w[p + "mix.o"].T
        u = group_rms(alpha * x + torch.sigmoid(x @ w[p + "rg1"].T + w[p + "rg1.b"]) * y, w[p + "norm1"], groups)
        y = (gelu(u @ w[p + "mlp.gate"].T) * (u @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T
        u = group_rms(alpha * u + torch.sigmoid(u @ w[p + "rg2"].T + w[p + "rg2.b"]) * y, w[p + "norm2"], groups)
        results.append(u)
        x = sum(float(a) * r for a, r in zip(w[p + "dwa"], results))
    return group_rms(x, w["final.norm"], groups)


def layer_norm(x, g, b):
    d = x - x.mean(-1, keepdim=True)
    return d * torch.rsqrt(d.square().mean(-1, keepdim=True) + EPS) * g + b


def zidepel_hidden(cfg, w, toks):
    n, loop = len(toks), cfg["loop"]
    x = layer_norm(w["embed"][toks] + w["pos"][:n], w["embed.norm"], w["embed.norm.b"])
    streams = torch.stack([x] * cfg["streams"])
    every = list(range(len(cfg["layers"])))
    for i in every[:loop["stop"]] + every[loop["start"]:loop["stop"]] * (loop["times"] - 1) + every[loop["stop"]:]:
        layer, p = cfg["layers"][i], f"l{i}."
        m = layer["mixer"]
        H, d, dv = m["heads"], m["dim"], m["vdim"]

        def attention(h):
            q = rms((h @ w[p + "mix.q"].T).view(n, H, d), w[p + "mix.q.norm"])
            at = torch.arange(n, device=h.device).double()
            q = q * (1.0 + m["q_temp"]["coef"] * torch.log(torch.floor((at + 1) / m["q_temp"]["every"]) + 1.0))[:, None, None]
            k = rms((h @ w[p + "mix.k"].T).view(n, m["kv_heads"], d), w[p + "mix.k.norm"])
            v = (h @ w[p + "mix.v"].T).view(n, m["kv_heads"], dv)
            o = causal(q.transpose(0, 1), k.transpose(0, 1), v.transpose(0, 1), m["scale"], cap=m["softcap"])
            return o.transpose(0, 1).reshape(n, -1) @ w[p + "mix.o"].T

        def linear(h):
            q, k = (h @ w[p + "mix.q"].T).view(n, H, d) * d ** -0.5, (h @ w[p + "mix.k"].T).view(n, H, d)
            v = (h @ w[p + "mix.v"].T).view(n, H, dv)
            a = torch.exp(torch.nn.functional.logsigmoid(h @ w[p + "mix.a1"].T @ w[p + "mix.a2"].T + w[p + "mix.a2.b"]) / m["tau"]).view(n, H, d)
            S, o = torch.zeros(H, d, dv, device=h.device, dtype=h.dtype), []
            for t in range(n):
                S = a[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
                o.append((q[t][:, None] @ S)[:, 0])
            g = h @ w[p + "mix.g"].T
            return (rms(torch.stack(o), w[p + "mix.norm"]).reshape(n, -1) * g * torch.sigmoid(g)) @ w[p + "mix.o"].T

        def feed_forward(h):
            return torch.relu(h @ w[p + "mlp.up"].T).square() @ w[p + "mlp.down"].T
        for q, sub in ((1, attention if layer["type"] == "attention" else linear), (2, feed_forward)):
            y = sub(layer_norm(torch.tensordot(w[f"{p}hc{q}.in"], streams, dims=1), w[f"{p}norm{q}"], w[f"{p}norm{q}.b"]))
            streams = torch.einsum("st,snd->tnd", w[f"{p}hc{q}.mix"], streams) + w[f"{p}hc{q}.out"][:, None, None] * y
    return layer_norm(streams.sum(0), w["final.norm"], w["final.norm.b"])


def exact_folder(case, seed):
    cfg, V, P, G = folder_config(case), case["vocab"], case["prompt"], case["new"]
    w = {k: v.cuda().double() for k, v in folder_weights(case).items()}
    t = torch.from_numpy(tokens(P, V, seed).astype(np.int64))
    if G:
        t = torch.cat([t, chain(t[-1], G, V)])
    hs = (morilorn_hidden if case["model"] == "morilorn" else zidepel_hidden)(cfg, w, t.cuda())
    z = hs[wanted(P) if G == 0 else [-1]] @ w["head"].T
    cap = cfg.get("logit_softcap")
    z = (cap * torch.tanh(z / cap) if cap else z).cpu().numpy().reshape(-1)
    return {"logits": z} if G == 0 else {"tokens": t[P:].numpy(), "logits": z}


def exact(case, seed):
    with torch.set_grad_enabled(case["kind"] == "lora"):
        make = {"lora": exact_lora, "full": exact_full, "folder": exact_folder}.get(case["kind"], exact_plain)
        return make(case, seed)
