"""The calls this package is used for, as cases that can be timed and compared.

Three ways in: the tensor-level ops (one fused op per call, driven by the caller's own layer code),
``DecodeEngine`` / ``EngineGroup`` steps (a caller that samples by itself feeds a token per sequence
and reads the logits), and ``prefill`` (a prompt into empty caches).  A model's depth only repeats its
layer, so the cases keep the width of a shape and a few of its layers: inputs are made quickly, and two
bf16 runs that add in another order stay close enough to be compared.

A case is a dict of sizes:
  kind     "mlp" | "attention" | "decode" | "prefill"
  dtype    "bf16" | "f32" | "int4" (int4-g128 factors, bf16 everything else)
  B        sequences (prefill: prompts, each of its own sequence)
  ctx      cached positions of the longest sequence (prefill: the prompt's length)
  step     sequence b holds ctx - b * step positions (0: all the same)
  d, H, Hk, Dh, I, Rqo, Rkv, Rmlp, vocab, layers   the model
  shared   layers 2i and 2i + 1 share their input-side factors
"""
import math

import torch

from flashsvd_b200 import ops, synthetic
from flashsvd_b200.engine import rope_tables
from flashsvd_b200.synthetic import ModelShape

STEPS = 4   # decode calls of one pass

# Llama-2-7B and Llama-2-70B shaped models with about 50 % / 40 % of the dense parameters
SHAPE_7B = dict(d=4096, H=32, Hk=32, Dh=128, I=11008, Rqo=1024, Rkv=1024, Rmlp=1488, vocab=32000, layers=4)
SHAPE_70B = dict(d=8192, H=64, Hk=8, Dh=128, I=28672, Rqo=1312, Rkv=224, Rmlp=2704, vocab=32000, layers=3)
SHAPE_SMALL = dict(d=1024, H=16, Hk=16, Dh=64, I=2816, Rqo=256, Rkv=256, Rmlp=376, vocab=32000, layers=4)


def _case(name, kind, shape, B, ctx, dtype="bf16", step=0, shared=False, **over):
    return dict(shape, name=name, kind=kind, dtype=dtype, B=B, ctx=ctx, step=step, shared=shared, **over)


def listed():
    return [
        # the smallest call: one fused low-rank SwiGLU MLP of a small model, a layer at a time
        _case("mlp_small_b1", "mlp", SHAPE_SMALL, 1, 0),
        # the attention half of a wide grouped-query layer at a long context, two ragged sequences
        _case("attention_gqa_b2", "attention", SHAPE_70B, 2, 4096, step=517),
        # fp32, the mode that reproduces greedy tokens exactly
        _case("decode_f32_b1", "decode", SHAPE_7B, 1, 256, dtype="f32"),
        # one user at a time: the plain interactive case
        _case("decode_b1", "decode", SHAPE_7B, 1, 512),
        # the same model with int4 factors, one user and a small server
        _case("decode_int4_b1", "decode", SHAPE_7B, 1, 512, dtype="int4"),
        _case("decode_int4_b16", "decode", SHAPE_7B, 16, 512, dtype="int4"),
        # a few and a few dozen sequences with shared bases at a long context
        _case("decode_b8_shared", "decode", SHAPE_7B, 8, 2048, shared=True),
        _case("decode_b32_shared", "decode", SHAPE_7B, 32, 2048, shared=True),
        # a full server: the widest batch, every sequence at a length of its own
        _case("decode_b128_ragged", "decode", SHAPE_7B, 128, 1023, step=6),
        # a large grouped-query model, long context
        _case("decode_70b_b8", "decode", SHAPE_70B, 8, 4096),
        # a long prompt of odd length, and several shorter prompts together
        _case("prefill_b1_long", "prefill", SHAPE_7B, 1, 2041),
        _case("prefill_b6", "prefill", SHAPE_7B, 6, 190),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _to8(x):
    return max(16, int(round(x / 8)) * 8)


def draw(rng):
    # widths from a 1024-wide to a 5120-wide model, MHA and grouped-query, odd tile remainders in the
    # intermediate size, the ranks and the vocabulary
    Dh = rng.choice([64, 128, 128])
    H = _log_int(rng, 1024, 5120) // Dh
    G = rng.choice([1, 1, 2, 4, 8])
    H = max(G, H // G * G)
    d = H * Dh
    I = _to8(d * rng.uniform(2.4, 3.6))
    ratio = rng.uniform(0.3, 0.65)
    Rqo = _to8(ratio * d / 2)
    Rkv = _to8(ratio * d * (H // G) * Dh / (d + (H // G) * Dh))
    Rmlp = _to8(ratio * d * I / (d + I))
    shape = dict(d=d, H=H, Hk=H // G, Dh=Dh, I=I, Rqo=Rqo, Rkv=Rkv, Rmlp=Rmlp, vocab=rng.randrange(4000, 40000),
                 layers=rng.randrange(2, 6))
    kind = rng.choice(["mlp", "attention", "decode", "decode", "decode", "decode", "decode", "prefill", "prefill"])
    dtype, shared, step = "bf16", False, 0
    if kind == "mlp":
        B, ctx = rng.randrange(1, 9), 0
    elif kind == "attention":
        B, ctx = rng.randrange(1, 9), _log_int(rng, 16, 6000)
    elif kind == "decode":
        dtype = rng.choice(["bf16", "bf16", "bf16", "bf16", "int4", "f32"])
        B = {"bf16": _log_int(rng, 1, 128), "int4": _log_int(rng, 1, 24), "f32": rng.randrange(1, 5)}[dtype]
        ctx = _log_int(rng, 32, min(4096, 200000 // B))
        shared = dtype == "bf16" and rng.random() < 0.3
    else:
        dtype = rng.choice(["bf16", "bf16", "bf16", "bf16", "int4"])
        B = 1 if rng.random() < 0.6 else rng.randrange(2, 9)
        ctx = _log_int(rng, 16, 2000 if B == 1 and dtype == "bf16" else 180)
    if kind in ("attention", "decode") and B > 1 and not (dtype == "int4" and B > 8) and rng.random() < 0.5:
        step = rng.randrange(1, max(2, (ctx - 8) // B + 1)) if ctx > 16 + B else 0
    return dict(shape, kind=kind, dtype=dtype, B=B, ctx=ctx, step=step, shared=shared)


def _shape(c):
    return ModelShape(d=c["d"], H=c["H"], Hk=c["Hk"], Dh=c["Dh"], I=c["I"], Rq=c["Rqo"], Rk=c["Rkv"], Rv=c["Rkv"],
                      Ro=c["Rqo"], Rg=c["Rmlp"], Ru=c["Rmlp"], Rd=c["Rmlp"], vocab=c["vocab"], n_layers=c["layers"])


def _lengths(c):
    return [c["ctx"] - b * c["step"] for b in range(c["B"])]


def _dims(c, S_max):
    return ops.make_dims(dtype=torch.bfloat16, B=c["B"], d=c["d"], H=c["H"], Hk=c["Hk"], Dh=c["Dh"], I=c["I"],
                         Rq=c["Rqo"], Rk=c["Rkv"], Rv=c["Rkv"], Ro=c["Rqo"], Rg=c["Rmlp"], Ru=c["Rmlp"], Rd=c["Rmlp"],
                         S_max=S_max)


def _new_rows(c, cache):
    """The rows of a cache that a pass of STEPS decode steps writes, [B, STEPS, Hk, Dh]."""
    B, S = cache.shape[:2]
    row = cache.stride(1)
    return cache.as_strided((B, STEPS, *cache.shape[2:]), (S * row - c["step"] * row, row, *cache.stride()[2:]),
                            cache.storage_offset() + c["ctx"] * row)


def prepare(case, seed):
    c, dev = case, torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(seed)

    def randn(*size, fan=1):
        return (torch.randn(*size, device=dev, generator=gen) / math.sqrt(fan)).to(torch.bfloat16)

    s = {"case": c}
    if c["kind"] == "mlp":
        R, I, d = c["Rmlp"], c["I"], c["d"]
        s.update(x=randn(c["B"], d), norm=torch.ones(d, device=dev, dtype=torch.bfloat16), upgate=randn(2 * R, d, fan=d),
                 gate=randn(I, R, fan=R), up=randn(I, R, fan=R), down_v=randn(R, I, fan=I), down_u=randn(d, R, fan=R),
                 ws=ops.make_workspace(_dims(c, 1), dev))
    elif c["kind"] == "attention":
        d, HD, KD, S = c["d"], c["H"] * c["Dh"], c["Hk"] * c["Dh"], c["ctx"] + 8
        cos, sin = rope_tables(S, c["Dh"], 10000.0, torch.bfloat16, dev)
        s.update(x=randn(c["B"], d), norm=torch.ones(d, device=dev, dtype=torch.bfloat16),
                 qkv_v=randn(c["Rqo"] + 2 * c["Rkv"], d, fan=d), q_u=randn(HD, c["Rqo"], fan=c["Rqo"]),
                 k_u=randn(KD, c["Rkv"], fan=c["Rkv"]), v_u=randn(KD, c["Rkv"], fan=c["Rkv"]),
                 o_v=randn(c["Rqo"], HD, fan=HD), o_u=randn(d, c["Rqo"], fan=c["Rqo"]),
                 k=randn(c["B"], S, c["Hk"], c["Dh"]), v=randn(c["B"], S, c["Hk"], c["Dh"]), cos=cos, sin=sin,
                 lens=torch.tensor(_lengths(c), dtype=torch.int32, device=dev), ws=ops.make_workspace(_dims(c, S), dev))
        s["out"] = [t.as_strided((c["B"], c["Hk"], c["Dh"]), ((S - c["step"]) * KD, c["Dh"], 1), c["ctx"] * KD)
                    for t in (s["k"], s["v"])]
    else:
        prompt = c["kind"] == "prefill"
        eng = synthetic.make_engine(_shape(c), device=dev, dtype=torch.float32 if c["dtype"] == "f32" else torch.bfloat16,
                                    batch=c["B"], ctx=0 if prompt else c["ctx"], max_new=c["ctx"] if prompt else STEPS,
                                    seed=seed, fill_cache=not prompt, share_pairs=c["shared"],
                                    factors="int4" if c["dtype"] == "int4" else "dense")
        s["eng"], s["group"] = eng, hasattr(eng, "engines")
        engines = eng.engines if s["group"] else [eng]
        n = c["ctx"] if prompt else STEPS
        s["ids"] = torch.randint(0, c["vocab"], (c["B"], n), device=dev, generator=gen, dtype=torch.int32)
        s["columns"] = [s["ids"][:, t].contiguous() for t in range(n)] if not prompt else None
        s["lens"] = torch.tensor(_lengths(c), dtype=torch.int32, device=dev)
        caches = [t for e in engines for pair in zip(e.key_cache, e.value_cache) for t in pair]
        s["logits"] = [e.logits for e in engines]
        s["out"] = [t[:, :n] for t in caches] if prompt else [_new_rows(c, t) for t in caches]
    return s


def run(s):
    c = s["case"]
    if c["kind"] == "mlp":
        return ops.mlp_swiglu_decode(s["x"], s["gate"], s["up"], s["down_v"], s["down_u"], s["ws"], upgate_v=s["upgate"],
                                     norm_w=s["norm"], residual=s["x"])
    if c["kind"] == "attention":
        q = ops.qkv_rope_append(s["x"], s["qkv_v"], s["q_u"], s["k_u"], s["v_u"], s["cos"], s["sin"], s["k"], s["v"],
                                s["lens"], s["ws"], num_heads=c["H"], num_kv_heads=c["Hk"], head_dim=c["Dh"],
                                ranks=(c["Rqo"], c["Rkv"], c["Rkv"]), norm_w=s["norm"])
        a = ops.flash_decode(q, s["k"], s["v"], s["lens"], s["ws"], seqlen_add=1)
        y = ops.lowrank_proj(a.view(c["B"], -1), s["o_v"], s["o_u"], s["ws"], residual=s["x"])
        return [y, q, *s["out"]]
    eng = s["eng"]
    if c["kind"] == "prefill":
        # new prompts take the places of finished ones
        if s["group"]:
            eng.fill_seqlens(0)
        else:
            eng.reset()
        eng.prefill(s["ids"])
        return [*(t.clone() for t in s["logits"]), *s["out"]]
    # sequences resume where they stood; the caller picks every next token by itself
    if s["group"]:
        eng.fill_seqlens(c["ctx"])
    else:
        eng.seqlens.copy_(s["lens"])
    for ids in s["columns"]:
        if s["group"]:
            eng.set_tokens(ids)
        else:
            eng.tokens.copy_(ids)
        eng.step(1)
    # (the logits are the engine's own memory: a caller that keeps them takes a copy)
    return [*(t.clone() for t in s["logits"]), *s["out"]]


def _factor_params(c):
    sh = _shape(c)
    HD, KD = sh.H * sh.Dh, sh.Hk * sh.Dh
    inner = sh.d * (sh.Rq + sh.Rk + sh.Rv + sh.Rg + sh.Ru) + HD * sh.Ro + sh.I * sh.Rd
    outer = HD * sh.Rq + KD * (sh.Rk + sh.Rv) + sh.d * sh.Ro + sh.I * (sh.Rg + sh.Ru) + sh.d * sh.Rd
    return inner, outer


def work(case):
    c = case
    inner, outer = _factor_params(c)
    es = 4 if c["dtype"] == "f32" else 2
    fb = 0.5 + 2 / 128 if c["dtype"] == "int4" else es    # bytes of one factor element
    row = c["Hk"] * c["Dh"] * es                           # one position of one cache
    if c["kind"] == "mlp":
        n = 3 * c["Rmlp"] * (c["d"] + c["I"])
        return {"bytes": 2 * n + 6 * c["B"] * c["d"], "flops": 2 * n * c["B"]}
    if c["kind"] == "attention":
        HD, KD = c["H"] * c["Dh"], c["Hk"] * c["Dh"]
        n = c["d"] * (c["Rqo"] + 2 * c["Rkv"]) + HD * c["Rqo"] + 2 * KD * c["Rkv"] + HD * c["Rqo"] + c["d"] * c["Rqo"]
        keys = sum(_lengths(c)) + c["B"]
        return {"bytes": 2 * n + 2 * keys * row + 6 * c["B"] * c["d"], "flops": 2 * n * c["B"] + 4 * keys * HD}
    L, head = c["layers"], c["vocab"] * c["d"]
    distinct = L * outer + (((L + 1) // 2) if c["shared"] else L) * inner
    if c["kind"] == "prefill":
        # every position through every layer, the head for the last one; the factors once, keys and
        # values written once and read once by the attention
        tokens, pairs = c["B"] * c["ctx"], c["B"] * c["ctx"] * (c["ctx"] + 1) // 2
        return {"bytes": distinct * fb + head * es + L * 4 * tokens * row,
                "flops": 2 * tokens * L * (inner + outer) + 2 * c["B"] * head + 4 * pairs * c["H"] * c["Dh"] * L}
    keys = sum(_lengths(c)) + c["B"]
    one = {"bytes": distinct * fb + head * es + L * 2 * keys * row + 4 * c["B"] * c["vocab"],
           "flops": 2 * c["B"] * (L * (inner + outer) + head) + 4 * keys * c["H"] * c["Dh"] * L}
    return {k: STEPS * v for k, v in one.items()}


def tolerance(case):
    if case["dtype"] == "f32":
        return {"rel": 2e-5}
    # one op: a few bf16 roundings; a model: about a dozen roundings a layer that add up like a random
    # walk over the layers (two orders of addition differ by 0.0075 sqrt(layers) in the logits)
    return {"rel": 1e-2} if case["kind"] in ("mlp", "attention") else {"rel": 0.012 * math.sqrt(case["layers"])}
