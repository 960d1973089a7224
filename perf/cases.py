"""The framework's work as timed cases, through the calls a user makes: the op wrappers (`llama_cu_awq_b200.ops`), token-by-token
decoding (`Transformer.generate`, `Transformer.forward`), prompts in one pass (`Transformer.prefill`, `generate` with
`prompt_one_pass`), several sequences at once (`Batch`) and the sampled end of a token (classifier + `sample_topp`).

The models are slices of the configurations in `llama_cu_awq_b200.synth`: the full layer shapes, `layers` of their layers, and the
same share of their classifier (32 layers : 32000 words of the 7B model are 4 layers : 4000 words), so that every op keeps the
share of the time it has in the whole model. A slice and not the whole, because layers of random weights amplify the last bit of
a rounding: after 32 of them two correct implementations differ by 10 % in the logits, after 4 of them by 1 to 3 %.

Decoding is timed on given ids (the prompt is as long as the run): a generated id that two implementations round apart would
send them to different texts. The work of a position is the same either way.
"""
import random

import numpy as np
import torch

from llama_cu_awq_b200 import _lib, ops, synth
from llama_cu_awq_b200.model import Batch, Transformer


def listed():
    return [
        # one projection of a 7B layer for one token through the op wrapper: the smallest call there is
        {"name": "op_gemv_4096", "kind": "gemv", "K": 4096, "N": 4096},
        # a host program that kept its own token loop and calls the op wrappers one by one, in the middle of a conversation
        {"name": "op_layers_7b", "kind": "ops", "model": "llama2-7b", "layers": 2, "pos": 600},
        # the batched W4 product alone: gate|up of a 7B layer for 64 rows
        {"name": "op_gemm_m64", "kind": "gemm", "M": 64, "K": 4096, "N": 22016},
        # the end of a sampled token: classifier of the 7B model and the top-p sampler over 32000 words
        {"name": "op_sample_32000", "kind": "sample", "dim": 4096, "vocab": 32000, "temperature": 0.8, "topp": 0.9},
        # the headline use: the command line's token loop at batch 1 on the 7B shapes, short context
        {"name": "generate_7b", "kind": "generate", "model": "llama2-7b", "layers": 4, "tokens": 48, "one_pass": False},
        # batch-1 decode deep into the context window of the 7B model
        {"name": "decode_7b_long", "kind": "decode", "model": "llama2-7b", "layers": 2, "pos": 1800, "tokens": 16},
        # batch-1 decode of the largest model, 8 query heads per key/value head
        {"name": "decode_70b", "kind": "decode", "model": "llama2-70b", "layers": 2, "pos": 100, "tokens": 16},
        # time to the first token of a short, odd-sized prompt on the 13B shapes
        {"name": "first_token_13b", "kind": "generate", "model": "llama2-13b", "layers": 2, "tokens": 78, "one_pass": True},
        # a prompt of ordinary length in one pass
        {"name": "prefill_7b_512", "kind": "prefill", "model": "llama2-7b", "layers": 4, "start": 0, "tokens": 512},
        # the next message of a conversation: an odd number of tokens behind a history, 70B shapes
        {"name": "prefill_70b_next", "kind": "prefill", "model": "llama2-70b", "layers": 1, "start": 700, "tokens": 333},
        # a prompt that nearly fills the 7B model's context window
        {"name": "prefill_7b_2000", "kind": "prefill", "model": "llama2-7b", "layers": 2, "start": 0, "tokens": 2000},
        # eight sequences decoded together
        {"name": "batch8_7b", "kind": "batch", "model": "llama2-7b", "layers": 4, "seqs": 8, "tokens": 32},
    ]


def _log_between(rng, lo, hi, step=1):
    v = lo * (hi / lo) ** rng.random()
    return int(max(lo, min(hi, round(v / step) * step)))


def draw(rng: random.Random):
    kind = rng.choice(["gemv", "ops", "gemm", "sample", "generate", "decode", "decode", "first", "prefill", "prefill", "batch", "batch"])
    model = rng.choice(["llama2-7b", "llama2-7b", "llama2-13b", "llama2-70b"])
    layers = rng.randint(1, {"llama2-7b": 4, "llama2-13b": 3, "llama2-70b": 2}[model])
    if kind == "gemv":
        K = _log_between(rng, 512, 28672, 8)
        return {"kind": "gemv", "K": K, "N": _log_between(rng, 512, min(28672, 100_000_000 // K), 8)}
    if kind == "ops":
        return {"kind": "ops", "model": model, "layers": rng.randint(1, 2), "pos": _log_between(rng, 4, 1500)}
    if kind == "gemm":
        K = _log_between(rng, 1024, 14336, 128)
        return {"kind": "gemm", "M": _log_between(rng, 17, 1024), "K": K, "N": _log_between(rng, 1024, min(28672, 100_000_000 // K), 8)}
    if kind == "sample":
        return {"kind": "sample", "dim": rng.choice([2048, 4096, 5120]), "vocab": _log_between(rng, 2000, 50000, 8),
                "temperature": round(rng.uniform(0.5, 1.2), 2), "topp": round(rng.uniform(0.5, 0.95), 2)}
    if kind == "generate":
        return {"kind": "generate", "model": model, "layers": layers, "tokens": _log_between(rng, 6, 48), "one_pass": False}
    if kind == "decode":
        pos = _log_between(rng, 8, 1900)
        if pos > 300:   # (deep positions amplify roundings more: fewer layers)
            layers = min(layers, 1 if model == "llama2-70b" else 2)
        return {"kind": "decode", "model": model, "layers": layers, "pos": pos, "tokens": rng.randint(4, 16)}
    if kind == "first":
        return {"kind": "generate", "model": model, "layers": min(layers, 2), "tokens": _log_between(rng, 6, 400), "one_pass": True}
    if kind == "prefill":
        n = _log_between(rng, 20, 1400)
        if n > 300 or model == "llama2-70b":
            layers = min(layers, 1 if model == "llama2-70b" else 2)
        if model == "llama2-70b":
            n = min(n, 500)
        return {"kind": "prefill", "model": model, "layers": layers, "start": rng.choice([0, 0, rng.randint(1, 600)]), "tokens": n}
    return {"kind": "batch", "model": model, "layers": layers, "seqs": rng.randint(1, 16), "tokens": _log_between(rng, 6, 32)}


# ---------------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------------
def _config(case):
    """The slice: (dim, hidden, layers, heads, kv_heads, vocab, seq_len, theta)."""
    dim, hid, L, H, KV, V, S, theta = synth.CONFIGS[case["model"]]
    n = case["layers"]
    return dim, hid, n, H, KV, V * n // L // 32 * 32, S, theta      # (a vocabulary in whole 32s, as the full one is)


class _View:
    """A device buffer of the library as something torch can hold on to; `owner` keeps the buffer alive."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f2", "data": (int(ptr), False), "version": 2}


class _OpenBatch(Batch):
    """A Batch that gives its caches back when the program lets go of it."""

    def __del__(self):
        self.close()


def _model(case, seed):
    t = Transformer(None, synthetic=(_config(case), seed & 0x7FFFFFFF))
    logits = torch.as_tensor(_View(t.logits_device_ptr(), (t.config.vocab_size,), t), device="cuda")
    return t, logits


def _ids(case, seed, n):
    return np.random.default_rng(seed & 0x7FFFFFFF).integers(3, _config(case)[5], size=n, dtype=np.int32)


def _qweight(gen, K, N):
    """Packed weights as a checkpoint has them: nibbles and zero points uniform on 0..15, fp16 scales U[0.002, 0.02]."""
    pw, pz, g = synth.packed_dims(K)
    word = dict(dtype=torch.int32, device="cuda", generator=gen)
    scales = (torch.rand((N, g), device="cuda", generator=gen) * 0.018 + 0.002).half()
    return ops.QWeight(torch.randint(-(2**31), 2**31, (N, pw), **word), torch.randint(-(2**31), 2**31, (N, pz), **word), scales)


def _normal(gen, *shape, std=1.0):
    return (torch.randn(shape, device="cuda", generator=gen) * std).half()


def prepare(case, seed):
    kind = case["kind"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    s = {"kind": kind, "case": case}
    if kind == "gemv":
        s["w"] = _qweight(gen, case["K"], case["N"])
        s["x"] = _normal(gen, case["K"])
        s["y"] = torch.empty(case["N"], dtype=torch.float16, device="cuda")
    elif kind == "gemm":
        w = _qweight(gen, case["K"], case["N"])
        s["mm"] = ops.BatchedMatmul(w, case["K"], case["N"], case["M"])
        s["x"] = _normal(gen, case["M"], case["K"])
        s["y"] = torch.empty((case["M"], case["N"]), dtype=torch.float16, device="cuda")
    elif kind == "sample":
        # logits with a standard deviation of 6: a few dozen words hold nearly all of the probability, as in a language model
        s["w"] = _normal(gen, case["vocab"], case["dim"], std=0.02)
        s["x"] = _normal(gen, case["dim"], std=6.0 / (0.02 * case["dim"] ** 0.5))
        s["logits"] = torch.empty(case["vocab"], dtype=torch.float16, device="cuda")
        s["mail"] = torch.zeros(16, dtype=torch.int32).pin_memory()      # word 0: position, words 8..: token ids
        s["zero"], s["pos"] = (torch.zeros(1, dtype=torch.int32, device="cuda") for _ in range(2))
        s["coin"] = float(np.random.default_rng(seed).random())
        s["token"] = s["mail"][9:10]
    elif kind == "ops":
        dim, hid, L, H, KV, V, S, theta = _config(case)
        kvd = dim * KV // H
        s["cfg"] = (dim, hid, L, H, KV, kvd, S, theta)
        s["layers"] = [{n: _qweight(gen, k, m) for n, k, m in (("q", dim, dim), ("k", dim, kvd), ("v", dim, kvd), ("o", dim, dim),
                                                               ("gate", dim, hid), ("up", dim, hid), ("down", hid, dim))} for _ in range(L)]
        s["norm"] = torch.ones(dim, dtype=torch.float16, device="cuda")
        s["table"] = _normal(gen, V, dim, std=0.02)
        s["ids"] = torch.from_numpy(_ids(case, seed, S)).pin_memory()
        s["kc"], s["vc"] = _normal(gen, L, S, kvd), _normal(gen, L, S, kvd)
        s["x"], s["xb"], s["q"] = (torch.empty(dim, dtype=torch.float16, device="cuda") for _ in range(3))
        s["hb"] = torch.empty(hid, dtype=torch.float16, device="cuda")
        s["att"] = ops.attention_scratch(H, dim // H)
        s["pos"] = torch.tensor([case["pos"]], dtype=torch.int32, device="cuda")
    elif kind == "batch":
        t = Transformer(None, synthetic=(_config(case), seed & 0x7FFFFFFF))
        b = _OpenBatch(t, case["seqs"])
        s["b"], s["ids"] = b, _ids(case, seed, case["seqs"] * case["tokens"]).reshape(case["seqs"], case["tokens"])
        ptr = _lib.lib().q4_batch_logits(b.h)
        s["logits"] = torch.as_tensor(_View(ptr, (case["seqs"], t.config.vocab_size), b), device="cuda")
        b.reset(s["ids"])      # a server has taken a step before its first request
        b.forward()
    else:
        t, s["logits"] = _model(case, seed)
        s["t"] = t
        first = case.get("pos", case.get("start", 0))
        s["ids"] = _ids(case, seed, first + case["tokens"])
        if kind in ("generate", "decode"):
            s["path"] = t.best_path()
        if first:              # the conversation so far is in the cache
            t.reset(s["ids"], 0)
            t.prefill(first, gen_token=False)
        elif kind == "prefill" or case.get("one_pass"):   # a server has seen a prompt before this one
            t.reset(s["ids"], 0)
            t.prefill(case["tokens"], gen_token=False)
    return s


# ---------------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------------
def _run_layers(s):
    dim, hid, L, H, KV, kvd, S, theta = s["cfg"]
    hs, pos, x, xb = dim // H, s["pos"], s["x"], s["xb"]
    ops.copy_embedding(x, s["table"], dim, s["ids"].data_ptr(), pos)
    for l in range(L):
        w, loff = s["layers"][l], l * S * kvd
        ops.rmsnorm(xb, x, s["norm"], dim)
        ops.qkv_matvec(s["q"], s["kc"], s["vc"], xb, w["q"], w["k"], w["v"], dim, dim, loff, pos, kvSize=kvd)
        ops.RoPERotation(s["q"], s["kc"], H, KV, hs, pos, loff, theta)
        ops.MultiHeadAttention(xb, s["q"], s["kc"][l], s["vc"][l], s["att"], H, hs, H // KV, S, pos)
        ops.matmul(x, xb, w["o"], dim, dim, accum=True)
        ops.rmsnorm(xb, x, s["norm"], dim)
        ops.ffn_matvec_silu(s["hb"], xb, w["gate"], w["up"], dim, hid)
        ops.matmul(x, s["hb"], w["down"], hid, dim, accum=True)
    return {"x": x, "q": s["q"], "hb": s["hb"]}


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "gemv":
        ops.matmul(s["y"], s["x"], s["w"], case["K"], case["N"])
        return s["y"]
    if kind == "gemm":
        s["mm"](s["y"], s["x"], case["M"])
        return s["y"]
    if kind == "sample":
        mail = s["mail"].data_ptr()
        s["mail"][:1].copy_(s["zero"], non_blocking=True)     # a new sequence starts
        ops.matmul(s["logits"], s["x"], s["w"], case["dim"], case["vocab"])
        ops.sample_topp(s["logits"], case["vocab"], case["temperature"], case["topp"], s["coin"], mail + 32, mail, s["pos"])
        return {"probabilities": s["logits"], "token": s["token"]}
    if kind == "ops":
        return _run_layers(s)
    if kind == "batch":
        b = s["b"]
        b.reset(s["ids"])
        for _ in range(case["tokens"]):
            b.forward()
        return s["logits"]
    t = s["t"]
    if kind == "generate":
        t.generate(s["ids"], case["tokens"], path=s["path"], prompt_one_pass=case["one_pass"])
    elif kind == "decode":
        t.reset(s["ids"], case["pos"])
        for _ in range(case["tokens"]):
            t.forward(gen_token=False, path=s["path"])
    else:
        t.reset(s["ids"], case["start"])
        t.prefill(case["tokens"], gen_token=False)
    return s["logits"]


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------
def _layer(cfg):
    """(bytes of a layer's weights and norms, its weights)"""
    dim, hid, _, H, KV, _, _, _ = cfg
    kvd = dim * KV // H
    shapes = [(dim, dim), (dim, kvd), (dim, kvd), (dim, dim), (dim, hid), (dim, hid), (hid, dim)]
    return sum(synth.qweight_bytes(k, n) for k, n in shapes) + 4 * dim, sum(k * n for k, n in shapes)


def _rows_work(cfg, rows, history, logits):
    """`rows` consecutive positions behind `history` cached ones through the slice in one go, `logits` classifier rows."""
    dim, _, L, H, KV, V, _, _ = cfg
    kvd = dim * KV // H
    by, weights = _layer(cfg)
    keys = rows * history + rows * (rows + 1) // 2        # (query, key) pairs
    b = L * (by + 4 * kvd * (history + rows) + 4 * kvd * rows) + 2 * V * dim + 2 * dim + 2 * dim * rows + 2 * V * logits
    f = L * (2 * weights * rows + 4 * dim * keys) + 2 * V * dim * logits
    return b, f


def work(case):
    kind = case["kind"]
    if kind in ("gemv", "gemm"):
        M, K, N = case.get("M", 1), case["K"], case["N"]
        return {"bytes": synth.qweight_bytes(K, N) + 2 * M * (K + N), "flops": 2 * M * K * N}
    if kind == "sample":
        n, d = case["vocab"], case["dim"]
        return {"bytes": 2 * n * d + 2 * d + 2 * n, "flops": 2 * n * d}
    cfg = _config(case)
    if kind == "ops":
        b, f = _rows_work(cfg, 1, case["pos"], 0)
        return {"bytes": b - 2 * cfg[5] * cfg[0], "flops": f}
    if kind == "prefill" or case.get("one_pass"):
        b, f = _rows_work(cfg, case["tokens"], case.get("start", 0), 1)
        return {"bytes": b, "flops": f}
    # one position after the other: the weights once per position (and once for all sequences of a batch)
    dim, _, L, H, KV, V, _, _ = cfg
    n, first, seqs = case["tokens"], case.get("pos", 0), case.get("seqs", 1)
    b = f = 0
    for pos in range(first, first + n):
        one, ops_one = _rows_work(cfg, 1, pos, 1)
        own = L * 4 * (dim * KV // H) * (pos + 2) + 2 * dim * 2 + 2 * V      # what each sequence adds: cache, embedding, logits
        b += one + (seqs - 1) * own
        f += seqs * ops_one
    return {"bytes": b, "flops": f}


def tolerance(case):
    """fp16 weights, activations and results with 32-bit sums. One product: the roundings of its results and of the
    dequantised weights. Layers: each rounding is amplified by the random layers behind it (the per-op and the persistent
    decode path of one model, which both round where a single token's ops do, differ by 1 to 3 % at these depths).
    Sampling: the last place of an fp16 logit around 20 is 1/64, 2 % of that word's probability."""
    kind = case["kind"]
    if kind in ("gemv", "gemm"):
        return {"rel": 4e-3, "max": 3e-2}
    if kind == "ops":
        return {"rel": 1.5e-2, "max": 0.15}
    if kind == "sample":
        return {"rel": 2e-2, "max": 3e-2}
    return {"rel": 3e-2, "max": 0.3}
