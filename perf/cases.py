"""Performance cases: the work that programs built on this package have it do, through its public entry points.

A case is a dict of plain values.  Kinds:

  attn      one attention forward and backward over given q, k, v and dO (a training step of one layer)
  chain     the same with the RoPE + QK-Norm operator in front and its backward behind: projections in, gradients of
            the projections and of the norm's gains out
  ref       forward and backward through the reference-shaped entry points ([B x heads, T, D], no grouped heads)
  fwd       the forward alone (evaluation, scoring, activation recompute)
  qkprep    the RoPE + QK-Norm operator alone, forward and backward
  decode    one query token per sequence against a dense K/V cache
  generate  a sampler: prompt through every layer of a KVCache, then single tokens
  step      one layer's share of a sampling step over sequences of different lengths
  chunk     one layer's share of a chunked prefill: new tokens behind tokens already cached

Shapes come from the benchmark configurations (modern-llm-v1_b200/inputs.py), the tests and ranges around them.
"""
import math

import torch

import modern_llm_v1_b200 as m

BF16, F32 = torch.bfloat16, torch.float32
HEADS = ((6, 2), (16, 4), (8, 8), (12, 4), (8, 1), (4, 2))  # query heads, key/value heads
MAX_ATTN_FLOPS = 3.5 * 2.0 * 4 * 16 * 8192 * 8192 * 128  # the long-context training configuration
MAX_Q_ELEMS = 4 * 16 * 8192 * 128
MAX_CACHE_BYTES = 2 * 64 * 4 * 8192 * 64 * 2
EPS = 1e-5


def listed():
    return [
        # the plumbing configuration: a few hundred rows, where launches and host work are all there is
        {"name": "attn_small", "kind": "attn", "B": 2, "T": 128, "Hq": 6, "Hkv": 2, "D": 64, "layout": "BHTD"},
        # a layer of the 50M training configuration as the model runs it: projections in BF16, read where they lie
        {"name": "chain_50m", "kind": "chain", "B": 32, "T": 512, "Hq": 6, "Hkv": 2, "D": 64, "layout": "BTHD", "x": "bf16"},
        # the 300M-class training configuration, attention alone
        {"name": "attn_300m", "kind": "attn", "B": 16, "T": 1024, "Hq": 16, "Hkv": 4, "D": 64, "layout": "BHTD"},
        # the long-context training configuration: the largest amount of work in one call
        {"name": "attn_long", "kind": "attn", "B": 4, "T": 8192, "Hq": 16, "Hkv": 4, "D": 128, "layout": "BHTD"},
        # a caller of the reference's operators that has expanded its heads; a length that no tile divides
        {"name": "ref_ragged", "kind": "ref", "B": 32, "T": 1001, "D": 128},
        # scoring documents of one length: no gradients, heads where the projection left them
        {"name": "fwd_eval", "kind": "fwd", "B": 8, "T": 2000, "Hq": 16, "Hkv": 4, "D": 64, "layout": "BTHD"},
        # the operator in front of attention for a model whose projections are FP32
        {"name": "qkprep_f32", "kind": "qkprep", "B": 16, "T": 1024, "Hq": 16, "Hkv": 4, "D": 128, "layout": "BHTD", "x": "f32"},
        # the sampler's loop for one sequence on the 50M model's six layers
        {"name": "generate_one", "kind": "generate", "B": 1, "layers": 6, "T": 100, "tokens": 12, "Hq": 6, "Hkv": 2, "D": 64,
         "x": "f32"},
        # a single sequence with a medium cache: too few heads to fill the device without splitting the cache
        {"name": "decode_one", "kind": "decode", "B": 1, "L": 1500, "Hq": 16, "Hkv": 4, "D": 128},
        # the decode configuration: a batch of long caches, all HBM traffic
        {"name": "decode_batch", "kind": "decode", "B": 64, "L": 4096, "Hq": 16, "Hkv": 4, "D": 64},
        # a serving batch whose sequences have very different lengths
        {"name": "step_mixed", "kind": "step", "B": 48, "L": 6000, "Hq": 16, "Hkv": 4, "D": 64, "x": "bf16"},
        # a long prompt taken in chunks, one of the later ones
        {"name": "chunk_prefill", "kind": "chunk", "B": 2, "pos": 3000, "T": 500, "Hq": 16, "Hkv": 4, "D": 128, "x": "bf16"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("attn", "chain", "ref", "fwd", "qkprep", "decode", "generate", "step", "chunk"))
    Hq, Hkv = rng.choice(HEADS)
    D = rng.choice((64, 128))
    c = {"kind": kind, "B": _log_int(rng, 1, 64), "Hq": Hq, "Hkv": Hkv, "D": D}
    if kind in ("attn", "chain", "fwd", "qkprep"):
        c["T"] = _log_int(rng, 64, 8192)
        c["layout"] = rng.choice(("BHTD", "BTHD"))
    if kind == "ref":
        del c["Hq"], c["Hkv"]
        c["B"], c["T"] = _log_int(rng, 4, 256), _log_int(rng, 64, 4096)
    if kind in ("chain", "qkprep", "generate", "step", "chunk"):
        c["x"] = rng.choice(("bf16", "f32"))
    if kind in ("decode", "step"):
        c["L"] = _log_int(rng, 128, 8192)
    if kind == "generate":
        c["B"], c["layers"], c["T"], c["tokens"] = _log_int(rng, 1, 16), rng.randint(2, 8), _log_int(rng, 16, 1024), rng.randint(2, 16)
    if kind == "chunk":
        c["B"], c["T"], c["pos"] = _log_int(rng, 1, 8), _log_int(rng, 2, 1024), _log_int(rng, 64, 6000)
    while c["B"] > 1 and _too_large(c):
        c["B"] -= 1
    return c


def _too_large(c):
    w = work(c)
    rows = c.get("T", 1) + (c["tokens"] * c["layers"] if c["kind"] == "generate" else 0)
    if c["B"] * rows * c.get("Hq", 1) * c["D"] > MAX_Q_ELEMS:
        return True
    return w["flops"] > MAX_ATTN_FLOPS or (c["kind"] in ("decode", "step") and w["bytes"] > MAX_CACHE_BYTES)


# ---- what a pass cannot do without
def _pairs(T, pos=0):
    """(query, key) pairs of a causal block of T rows behind pos keys."""
    return T * pos + T * (T + 1) / 2


def _lengths(c):
    """The cache lengths of a mixed batch, the newest token included: spread evenly from an eighth of L up to L."""
    B, L = c["B"], c["L"]
    lo = max(1, L // 8)
    return [L if B == 1 else lo + (L - lo) * i // (B - 1) for i in range(B)]


def work(case):
    c = case
    k, B, D = c["kind"], c["B"], c["D"]
    Hq, Hkv = (1, 1) if k == "ref" else (c["Hq"], c["Hkv"])
    xb = {"f32": 4, "bf16": 2}[c.get("x", "bf16")]
    if k in ("attn", "ref", "chain", "fwd", "qkprep"):
        q, kv, rows = B * c["T"] * Hq * D, B * c["T"] * Hkv * D, B * c["T"]
        fwd_flops = 4.0 * B * Hq * _pairs(c["T"]) * D
        if k == "fwd":
            return {"bytes": 2 * (2 * q + 2 * kv) + 4 * rows * Hq, "flops": fwd_flops}
        if k == "qkprep":  # x in, y out; then dy and x in, dx out; rstd both ways; the tables once each way
            return {"bytes": (q + kv) * (3 * xb + 4) + 8 * rows * (Hq + Hkv) + 8 * c["T"] * D, "flops": 30.0 * (q + kv)}
        # q, k, v, dO in; O, logsumexp and the three gradients out
        attn_bytes = 2 * (4 * q + 4 * kv) + 4 * rows * Hq
        if k == "chain":  # q, k and their gradients are the projections'
            return {"bytes": 2 * (2 * q + 2 * kv) + 2 * xb * (q + kv) + 4 * rows * Hq + 4 * c["T"] * D, "flops": 3.5 * fwd_flops + 30.0 * (q + kv)}
        return {"bytes": attn_bytes, "flops": 3.5 * fwd_flops}
    if k == "decode":
        return {"bytes": 2 * (2 * B * Hkv * c["L"] * D + 2 * B * Hq * D) + 4 * B * Hq, "flops": 4.0 * B * Hq * c["L"] * D}
    new_q, new_kv = B * Hq * D, B * Hkv * D  # per new token: projections in; q, context and the cache rows out
    per_token = xb * (new_q + 2 * new_kv) + 2 * (2 * new_q + 2 * new_kv)
    if k == "step":
        keys = sum(_lengths(c))
        return {"bytes": per_token + 4 * keys * Hkv * D, "flops": 4.0 * keys * Hq * D}
    if k == "chunk":
        return {"bytes": c["T"] * (per_token + 4 * B * Hq) + 4 * B * c["pos"] * Hkv * D, "flops": 4.0 * B * Hq * _pairs(c["T"], c["pos"]) * D}
    if k == "generate":
        T, n = c["T"], c["tokens"]
        cached = sum(T + i for i in range(n))  # rows read back by the single tokens
        one = (T + n) * per_token + 4 * B * Hq * T + 4 * B * cached * Hkv * D
        return {"bytes": c["layers"] * one, "flops": c["layers"] * 4.0 * B * Hq * _pairs(T + n) * D}
    raise ValueError(k)


def tolerance(case):
    if case["kind"] == "qkprep":  # FP32 arithmetic; the BF16 outputs are rounded once
        return {"rel": 1e-3, "max": 1e-2}
    return {"rel": 1e-2}  # BF16 operands of every product, BF16 outputs


# ---- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(shape, g, dtype=F32, std=1.0):
    x = torch.randn(shape, generator=g, device="cuda", dtype=F32)
    if std != 1.0:
        x *= std
    return x.to(dtype)


def _normed(shape, g):
    """Query or key rows as QK-Norm leaves them (gain 1).  RoPE in front of the norm rotates independent normal pairs,
    which leaves their distribution as it is."""
    x = torch.randn(shape, generator=g, device="cuda", dtype=F32)
    return (x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS)).to(BF16)


def _gain(D, g):
    return 1.0 + 0.1 * torch.randn(D, generator=g, device="cuda", dtype=F32)


def _shape(c, H):
    return (c["B"], H, c["T"], c["D"]) if c["layout"] == "BHTD" else (c["B"], c["T"], H, c["D"])


def prepare(case, seed):
    return _PREPARE[case["kind"]](dict(case), _gen(seed))


def run(state):
    return _RUN[state["c"]["kind"]](state)


def _prepare_attn(c, g):
    sq, sk = _shape(c, c["Hq"]), _shape(c, c["Hkv"])
    s = {"c": c, "q": _normed(sq, g), "k": _normed(sk, g), "v": _randn(sk, g, BF16), "do": _randn(sq, g, BF16, 0.1)}
    s["o"], s["lse"] = torch.empty(sq, device="cuda", dtype=BF16), torch.empty((c["B"], c["Hq"], c["T"]), device="cuda")
    s["dq"], s["dk"], s["dv"] = torch.empty_like(s["q"]), torch.empty_like(s["k"]), torch.empty_like(s["v"])
    return s


def _run_attn(s):
    c = s["c"]
    dims = (c["B"], c["T"], c["Hq"], c["Hkv"], c["D"], c["layout"])
    m.flash_attn_forward_gqa(s["q"], s["k"], s["v"], s["o"], s["lse"], *dims)
    m.flash_attn_backward_gqa(s["q"], s["k"], s["v"], s["o"], s["lse"], s["do"], s["dq"], s["dk"], s["dv"], *dims)
    return s["o"], s["lse"], s["dq"], s["dk"], s["dv"]


def _prepare_fwd(c, g):
    sq, sk = _shape(c, c["Hq"]), _shape(c, c["Hkv"])
    s = {"c": c, "q": _normed(sq, g), "k": _normed(sk, g), "v": _randn(sk, g, BF16)}
    s["o"], s["lse"] = torch.empty(sq, device="cuda", dtype=BF16), torch.empty((c["B"], c["Hq"], c["T"]), device="cuda")
    return s


def _run_fwd(s):
    c = s["c"]
    m.flash_attn_forward_gqa(s["q"], s["k"], s["v"], s["o"], s["lse"], c["B"], c["T"], c["Hq"], c["Hkv"], c["D"], c["layout"])
    return s["o"], s["lse"]


def _prepare_ref(c, g):
    shape = (c["B"], c["T"], c["D"])
    s = {"c": c, "q": _normed(shape, g), "k": _normed(shape, g), "v": _randn(shape, g, BF16), "do": _randn(shape, g, BF16, 0.1)}
    s["o"], s["lse"] = torch.empty_like(s["q"]), torch.empty(shape[:2], device="cuda")
    s["dq"], s["dk"], s["dv"] = (torch.empty_like(s["q"]) for _ in range(3))
    return s


def _run_ref(s):
    c = s["c"]
    m.flash_attn_forward(s["q"], s["k"], s["v"], s["o"], s["lse"], c["B"], c["T"], c["D"])
    m.flash_attn_backward(s["q"], s["k"], s["v"], s["o"], s["lse"], s["do"], s["dq"], s["dk"], s["dv"], c["B"], c["T"], c["D"])
    return s["o"], s["lse"], s["dq"], s["dk"], s["dv"]


def _prepare_qkprep(c, g):
    """Projections [B, T, H, D] as a linear layer writes them; y and dy in the layout attention takes."""
    B, T, D = c["B"], c["T"], c["D"]
    xd = F32 if c["x"] == "f32" else BF16
    s = {"c": c, "gq": _gain(D, g), "gk": _gain(D, g)}
    s["cos"], s["sin"] = m.make_rope_cache(T, D)
    for n, H in (("q", c["Hq"]), ("k", c["Hkv"])):
        s["x" + n] = _randn((B, T, H, D), g, xd)
        s["dx" + n] = torch.empty_like(s["x" + n])
        s["y" + n] = torch.empty(_shape(c, H), device="cuda", dtype=BF16)
        s["dy" + n] = _randn(_shape(c, H), g, BF16, 0.1)
        s["rstd" + n] = torch.empty((B, H, T), device="cuda")
        s["dg" + n] = torch.zeros(D, device="cuda")
    return s


def _norm_forward(s):
    c = s["c"]
    m.rope_qknorm_forward_qk(s["xq"], s["xk"], s["cos"], s["sin"], s["gq"], s["gk"], EPS, s["yq"], s["yk"], s["rstdq"], s["rstdk"],
                             c["B"], c["T"], c["Hq"], c["Hkv"], c["D"], "BTHD", c["layout"])


def _norm_backward(s):
    """The gains' gradients are added to, as over the micro-batches of an optimizer step."""
    c = s["c"]
    m.rope_qknorm_backward_qk(s["dyq"], s["dyk"], s["xq"], s["xk"], s["cos"], s["sin"], s["gq"], s["gk"], s["rstdq"], s["rstdk"],
                              s["dxq"], s["dxk"], s["dgq"], s["dgk"], c["B"], c["T"], c["Hq"], c["Hkv"], c["D"], "BTHD", c["layout"])


def _run_qkprep(s):
    _norm_forward(s)
    _norm_backward(s)
    return s["yq"], s["yk"], s["rstdq"], s["rstdk"], s["dxq"], s["dxk"], s["dgq"], s["dgk"]


def _prepare_chain(c, g):
    s = _prepare_qkprep(c, g)
    sq, sk = _shape(c, c["Hq"]), _shape(c, c["Hkv"])
    s["v"], s["do"] = _randn(sk, g, BF16), _randn(sq, g, BF16, 0.1)
    s["o"], s["lse"], s["dv"] = torch.empty(sq, device="cuda", dtype=BF16), torch.empty((c["B"], c["Hq"], c["T"]), device="cuda"), torch.empty_like(s["v"])
    return s


def _run_chain(s):
    c = s["c"]
    dims = (c["B"], c["T"], c["Hq"], c["Hkv"], c["D"], c["layout"])
    _norm_forward(s)
    m.flash_attn_forward_gqa(s["yq"], s["yk"], s["v"], s["o"], s["lse"], *dims)
    m.flash_attn_backward_gqa(s["yq"], s["yk"], s["v"], s["o"], s["lse"], s["do"], s["dyq"], s["dyk"], s["dv"], *dims)
    _norm_backward(s)
    return s["o"], s["lse"], s["dxq"], s["dxk"], s["dv"], s["dgq"], s["dgk"]


def _prepare_decode(c, g):
    B, L, Hq, Hkv, D = c["B"], c["L"], c["Hq"], c["Hkv"], c["D"]
    s = {"c": c, "q": _normed((B, Hq, D), g), "k": _normed((B, Hkv, L, D), g), "v": _randn((B, Hkv, L, D), g, BF16)}
    s["o"], s["lse"] = torch.empty_like(s["q"]), torch.empty((B, Hq), device="cuda")
    return s


def _run_decode(s):
    c = s["c"]
    m.flash_attn_decode(s["q"], s["k"], s["v"], s["o"], s["lse"], c["B"], c["L"], c["Hq"], c["Hkv"], c["D"])
    return s["o"], s["lse"]


def _new_tokens(c, n, g):
    """The projections of n new tokens per sequence, and room for what attention makes of them."""
    B, Hq, Hkv, D = c["B"], c["Hq"], c["Hkv"], c["D"]
    xd = F32 if c["x"] == "f32" else BF16
    q = torch.empty((B, Hq, n, D), device="cuda", dtype=BF16)
    lse = torch.empty((B, Hq, n), device="cuda") if n > 1 else None
    return {"n": n, "x": tuple(_randn((B, n, H, D), g, xd) for H in (Hq, Hkv, Hkv)), "q": q, "ctx": torch.empty_like(q), "lse": lse}


def _cache(c, layers, L_cap, g):
    cache = m.KVCache(layers, c["B"], c["Hq"], c["Hkv"], c["D"], L_cap)
    return cache, _gain(c["D"], g), _gain(c["D"], g)


def _layer(s, layer, t):
    cache = s["cache"]
    cache.append(layer, *t["x"], s["gq"], s["gk"], t["q"])
    cache.attend(layer, t["q"], t["ctx"], t["lse"], n_new=t["n"])


def _prepare_step(c, g):
    L_cap = (c["L"] + 255) // 256 * 256
    cache, gq, gk = _cache(c, 1, L_cap, g)
    cache.k.copy_(_normed(cache.k.shape, g))
    cache.v.copy_(_randn(cache.v.shape, g, BF16))
    order = torch.randperm(c["B"], generator=g, device="cuda").tolist()
    lengths = _lengths(c)
    cache.set_lengths([lengths[i] - 1 for i in order])
    return {"c": c, "cache": cache, "gq": gq, "gk": gk, "t": _new_tokens(c, 1, g)}


def _run_step(s):
    _layer(s, 0, s["t"])
    return s["t"]["q"], s["t"]["ctx"], s["cache"].k, s["cache"].v


def _prepare_chunk(c, g):
    cache, gq, gk = _cache(c, 1, c["pos"] + c["T"], g)
    cache.k.copy_(_normed(cache.k.shape, g))
    cache.v.copy_(_randn(cache.v.shape, g, BF16))
    cache.advance(c["pos"])
    return {"c": c, "cache": cache, "gq": gq, "gk": gk, "t": _new_tokens(c, c["T"], g)}


def _run_chunk(s):
    _layer(s, 0, s["t"])
    return s["t"]["q"], s["t"]["ctx"], s["t"]["lse"], s["cache"].k, s["cache"].v


def _prepare_generate(c, g):
    cache, gq, gk = _cache(c, c["layers"], c["T"] + c["tokens"], g)
    prompt = [_new_tokens(c, c["T"], g) for _ in range(c["layers"])]
    tokens = [[_new_tokens(c, 1, g) for _ in range(c["layers"])] for _ in range(c["tokens"])]
    return {"c": c, "cache": cache, "gq": gq, "gk": gk, "prompt": prompt, "tokens": tokens}


def _run_generate(s):
    cache = s["cache"]
    cache.reset()
    for layer, t in enumerate(s["prompt"]):
        _layer(s, layer, t)
    cache.advance(s["c"]["T"])
    for token in s["tokens"]:
        for layer, t in enumerate(token):
            _layer(s, layer, t)
        cache.advance()
    # the contexts of the prompt and of the last token of every layer, and the caches that hold all the tokens
    last = s["tokens"][-1]
    return [t["ctx"] for t in s["prompt"]], [t["ctx"] for t in last], cache.k, cache.v


_PREPARE = {"attn": _prepare_attn, "chain": _prepare_chain, "ref": _prepare_ref, "fwd": _prepare_fwd, "qkprep": _prepare_qkprep,
            "decode": _prepare_decode, "generate": _prepare_generate, "step": _prepare_step, "chunk": _prepare_chunk}
_RUN = {"attn": _run_attn, "chain": _run_chain, "ref": _run_ref, "fwd": _run_fwd, "qkprep": _run_qkprep,
        "decode": _run_decode, "generate": _run_generate, "step": _run_step, "chunk": _run_chunk}
