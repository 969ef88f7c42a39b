"""Timed cases: what a program built on this package has it do, from one operator to a whole prompt.

Kinds of case
  ops       one decoder layer driven operator by operator through ext.load() - what a program does that keeps its own
            step and swaps the operator module (embedding row, the six operators, nine launches and more)
  attention one paged decode-attention call for a batch of sequences of different lengths
  generate  Model.generate: a prompt, then greedy tokens, each read back as it is chosen
  decode    greedy steps that continue a sequence whose cache already holds `ctx` tokens
  prefill   Model.prefill: a prompt (or the next turn of a conversation) in one go; `score` asks for the logits of every
            position, as an evaluation of a text does
  quantize  QuantLinear: one fp16 matrix into the INT4 format (what loading a model does once per matrix)
  gptq      quantize_gptq: the same with a layer-input Hessian (what calibration does once per matrix)

Model shapes are the two of llm_decode_kernels_b200.shapes; the larger one runs with 8 of its layers, which keeps every
matrix at its size. Weights are N(0, 0.02). Embedding and LM head are made so that the logits have the clear maximum a
trained model's have: the head's row of token s(t) is the (scaled) embedding of t, for a random permutation s. Greedy
streams are then determined by the weights and not by the last bit of a logit. Caches that are filled beforehand hold
N(0, 1), as the context benchmarks of this repository do.
"""
import math
import random

import torch

from llm_decode_kernels_b200 import ext
from llm_decode_kernels_b200.model import DecodeConfig, Model, rope_tables
from llm_decode_kernels_b200.quant import QuantLinear, quantize_gptq
from llm_decode_kernels_b200.shapes import LLAMA3_70B, TINYLLAMA, config, random_llama_state

DEV = "cuda"
GROUP = 128
SHAPES = {"tinyllama": TINYLLAMA, "llama3_70b_8layers": dict(LLAMA3_70B, num_hidden_layers=8)}
EPS = 1e-5


def listed():
    return [
        # the smallest unit of work: one layer of the small model in mid-conversation, one call per operator
        {"name": "ops_layer_h2048_ctx512", "kind": "ops", "n_kv": 4, "inter": 5632, "ctx": 512},
        # a server's attention call: eight sequences of 128 .. 8192 tokens
        {"name": "attention_b8", "kind": "attention", "batch": 8, "n_q": 32, "n_kv": 4, "dim": 64, "lo": 128, "hi": 8192},
        # the headline workload: 128-token prompt, 256 greedy tokens
        {"name": "generate_128_256", "kind": "generate", "shape": "tinyllama", "prompt": 128, "new": 256,
         "prefill": False},
        # decoding behind an ordinary and behind a long context
        {"name": "decode_ctx2048", "kind": "decode", "shape": "tinyllama", "ctx": 2048, "new": 32},
        {"name": "decode_ctx8192", "kind": "decode", "shape": "tinyllama", "ctx": 8192, "new": 32},
        # decoding with the large model's matrices, which are bound by memory and not by latency
        {"name": "decode_70b_ctx4096", "kind": "decode", "shape": "llama3_70b_8layers", "ctx": 4096, "new": 16},
        # a short question, a page of text that is scored, a long document
        {"name": "prefill_77", "kind": "prefill", "shape": "tinyllama", "prompt": 77, "start": 0, "score": False},
        {"name": "prefill_512_score", "kind": "prefill", "shape": "tinyllama", "prompt": 512, "start": 0, "score": True},
        {"name": "prefill_4096", "kind": "prefill", "shape": "tinyllama", "prompt": 4096, "start": 0, "score": False},
        # a prompt for the large model, not a whole number of chunks
        {"name": "prefill_70b_1000", "kind": "prefill", "shape": "llama3_70b_8layers", "prompt": 1000, "start": 0,
         "score": False},
        # loading: the gate|up matrix with range clipping; calibrating: the down matrix
        {"name": "quantize_11264x2048_clip", "kind": "quantize", "rows": 11264, "cols": 2048, "group": 128, "clip": True},
        {"name": "gptq_2048x5632", "kind": "gptq", "rows": 2048, "cols": 5632, "clip": True},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    """A case of the same kinds: the kinds in the proportions of the list, sizes over their whole range."""
    kind = rng.choice(["ops", "attention", "generate", "decode", "decode", "decode", "prefill", "prefill", "prefill",
                       "prefill", "quantize", "gptq"])
    if kind == "ops":
        n_kv = rng.choice([1, 2, 4, 8])
        return {"kind": kind, "n_kv": n_kv, "inter": 128 * _log_int(rng, 8, 88), "ctx": _log_int(rng, 1, 8192)}
    if kind == "attention":
        n_q, n_kv, dim = rng.choice([(32, 4, 64), (64, 8, 128), (16, 8, 128), (8, 8, 64)])
        hi = _log_int(rng, 16, 8192)
        return {"kind": kind, "batch": rng.randint(1, 8), "n_q": n_q, "n_kv": n_kv, "dim": dim, "lo": max(1, hi // 64),
                "hi": hi}
    if kind == "generate":
        return {"kind": kind, "shape": "tinyllama", "prompt": _log_int(rng, 1, 128), "new": _log_int(rng, 8, 256),
                "prefill": rng.random() < 0.5}
    if kind == "decode":
        if rng.random() < 0.33:
            return {"kind": kind, "shape": "llama3_70b_8layers", "ctx": _log_int(rng, 16, 4096), "new": rng.randint(4, 16)}
        return {"kind": kind, "shape": "tinyllama", "ctx": _log_int(rng, 16, 16384), "new": rng.randint(8, 32)}
    if kind == "prefill":
        if rng.random() < 0.25:
            return {"kind": kind, "shape": "llama3_70b_8layers", "prompt": _log_int(rng, 8, 1000),
                    "start": rng.choice([0, 0, rng.randint(1, 1024)]), "score": False}
        prompt = _log_int(rng, 4, 4000)
        return {"kind": kind, "shape": "tinyllama", "prompt": prompt,
                "start": rng.choice([0, 0, rng.randint(1, max(1, 4096 - prompt))]),
                "score": prompt <= 1024 and rng.random() < 0.33}
    if kind == "quantize":
        return {"kind": kind, "rows": _log_int(rng, 256, 11264), "cols": 256 * rng.randint(2, 8),
                "group": rng.choice([64, 128, 128, 256]), "clip": rng.random() < 0.5}
    return {"kind": kind, "rows": _log_int(rng, 256, 2048), "cols": 128 * _log_int(rng, 4, 44),
            "clip": rng.random() < 0.5}


# ---------------------------------------------------------------------------------------------- preparation
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape, scale=1.0):
    return (torch.randn(*shape, generator=g, device=DEV) * scale).half()


def _model(shape, seed, ctx_cap, keep_packed):
    """A quantized model ready to decode up to ctx_cap, its step captured; and the generator the rest draws from."""
    c = config(SHAPES[shape])
    sd = random_llama_state(c, DEV, seed)
    g = _gen(seed + 1)
    succ = torch.randperm(c.vocab_size, generator=g, device=DEV)
    emb = sd["model.embed_tokens.weight"]
    sd["lm_head.weight"][succ] = emb          # logit of s(t) = <hidden, embedding of t>
    sd["model.embed_tokens.weight"] = emb * 200
    m = Model(sd, c, DecodeConfig(group=GROUP, max_ctx=ctx_cap, seed=seed, keep_packed=keep_packed))
    m.prepare(ctx_cap)
    return m, c, g


def _ids(c, n, seed):
    return torch.randint(0, c.vocab_size, (n,), generator=torch.Generator().manual_seed(seed))


def _prepare_ops(case, seed):
    g = _gen(seed)
    n_kv, inter, ctx, D, page = case["n_kv"], case["inter"], case["ctx"], 64, 16
    n_q = 8 * n_kv
    H, V = n_q * D, 32000
    s = {"K": ext.load(), "n_q": n_q, "n_kv": n_kv, "part_size": 256, "emb": _randn(g, V, H, scale=0.02)}
    for name, n, k in (("qkv", (n_q + 2 * n_kv) * D, H), ("o", H, H), ("gu", 2 * inter, H), ("down", H, inter)):
        s[name] = QuantLinear(_randn(g, n, k, scale=0.02), GROUP, keep_ref=False)
    pages = ctx // page + 1
    splits = -(-(ctx + 1) // s["part_size"])
    h16, f32 = dict(dtype=torch.half, device=DEV), dict(dtype=torch.float32, device=DEV)
    cos, sin = rope_tables(ctx + 2, D)
    s.update(kc=_randn(g, pages, n_kv, page, D), vc=_randn(g, pages, n_kv, page, D),
             bt=torch.randperm(pages, generator=g, device=DEV).int(), cos=cos.to(DEV), sin=sin.to(DEV),
             tok=torch.randint(0, V, (1,), generator=g, device=DEV), pos=torch.full((1,), ctx, dtype=torch.int32, device=DEV),
             ln1=_randn(g, H, scale=0.1) + 1, ln2=_randn(g, H, scale=0.1) + 1,
             x=torch.empty(H, **h16), normed=torch.empty(H, **h16), h_qkv=torch.empty((n_q + 2 * n_kv) * D, **h16),
             attn=torch.empty(n_q, D, **h16), h_o=torch.empty(H, **h16), h_gu=torch.empty(2 * inter, **h16),
             act=torch.empty(inter, **h16), h_down=torch.empty(H, **h16),
             o_part=torch.empty(n_q, splits, D, **f32), m_part=torch.empty(n_q, splits, **f32),
             l_part=torch.empty(n_q, splits, **f32))
    return s


def _prepare_attention(case, seed):
    g, rng = _gen(seed), random.Random(seed)
    B, n_q, n_kv, D, page = case["batch"], case["n_q"], case["n_kv"], case["dim"], 16
    ctxs = [rng.randint(case["lo"], case["hi"]) for _ in range(B)]
    pages = [-(-c // page) for c in ctxs]
    part = 256
    S = -(-max(ctxs) // part)
    pool = sum(pages)
    perm = torch.randperm(pool, generator=g, device=DEV).int().cpu()
    bt = torch.zeros(B, max(pages), dtype=torch.int32)
    at = 0
    for b, n in enumerate(pages):
        bt[b, :n] = perm[at:at + n]
        at += n
    f32 = dict(dtype=torch.float32, device=DEV)
    return {"K": ext.load(), "q": _randn(g, B, n_q, D), "kc": _randn(g, pool, n_kv, page, D),
            "vc": _randn(g, pool, n_kv, page, D), "bt": bt.to(DEV), "part_size": part,
            "pos": torch.tensor([c - 1 for c in ctxs], dtype=torch.int32, device=DEV),
            "o_part": torch.empty(B, n_q, S, D, **f32), "m_part": torch.empty(B, n_q, S, **f32),
            "l_part": torch.empty(B, n_q, S, **f32), "out": torch.empty(B, n_q, D, dtype=torch.half, device=DEV)}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ops":
        return dict(_prepare_ops(case, seed), kind=kind)
    if kind == "attention":
        return dict(_prepare_attention(case, seed), kind=kind)
    if kind == "generate":
        m, c, _ = _model(case["shape"], seed, case["prompt"] + case["new"] + 8, case["prefill"])
        return {"kind": kind, "m": m, "ids": _ids(c, case["prompt"], seed + 2), "new": case["new"],
                "prefill": case["prefill"]}
    if kind == "decode":
        m, c, g = _model(case["shape"], seed, case["ctx"] + case["new"] + 8, False)
        m.kv.normal_(generator=g)
        return {"kind": kind, "m": m, "ids": _ids(c, 1, seed + 2), "ctx": case["ctx"], "new": case["new"]}
    if kind == "prefill":
        m, c, g = _model(case["shape"], seed, case["start"] + case["prompt"] + 8, True)
        if case["start"]:
            m.kv.normal_(generator=g)
        return {"kind": kind, "m": m, "ids": _ids(c, case["prompt"], seed + 2), "start": case["start"],
                "score": case["score"]}
    g = _gen(seed)
    w = _randn(g, case["rows"], case["cols"], scale=0.02)
    if kind == "quantize":
        return {"kind": kind, "w": w, "group": case["group"], "clip": case["clip"]}
    # layer inputs as calibration sees them: correlated features of unequal size
    K = case["cols"]
    x = torch.randn(2048, K, generator=g, device=DEV)
    x = (x + 0.5 * x.roll(1, dims=1)) * torch.exp(0.5 * torch.randn(K, generator=g, device=DEV))
    return {"kind": kind, "w": w, "hess": 2 * (x.t() @ x) / x.shape[0], "clip": case["clip"]}


# ---------------------------------------------------------------------------------------------- one pass
def _run_ops(s):
    K, n_q, n_kv = s["K"], s["n_q"], s["n_kv"]

    def gemv(lin, x, y):
        K.gemv_w4a16(2, 0, 0, 0, lin.packed, lin.sz, x, y, GROUP)

    K.embed_row(s["emb"], s["tok"], s["x"])
    K.add_rmsnorm(s["x"], None, s["ln1"], s["normed"], EPS)
    gemv(s["qkv"], s["normed"], s["h_qkv"])
    K.rope_append(s["h_qkv"], s["cos"], s["sin"], s["pos"], s["bt"], s["kc"], s["vc"], n_q, n_kv)
    K.paged_attention(s["h_qkv"][: n_q * 64], s["kc"], s["vc"], s["bt"], s["pos"], s["part_size"], s["o_part"],
                      s["m_part"], s["l_part"], s["attn"], version=3)
    gemv(s["o"], s["attn"].view(-1), s["h_o"])
    K.add_rmsnorm(s["x"], s["h_o"], s["ln2"], s["normed"], EPS)
    gemv(s["gu"], s["normed"], s["h_gu"])
    K.swiglu(s["h_gu"], s["act"])
    gemv(s["down"], s["act"], s["h_down"])
    return {"x": s["x"], "down": s["h_down"], "kc": s["kc"], "vc": s["vc"]}


def run(state):
    s, kind = state, state["kind"]
    if kind == "ops":
        return _run_ops(s)
    if kind == "attention":
        s["K"].paged_attention_batched(s["q"], s["kc"], s["vc"], s["bt"], s["pos"], s["part_size"], s["o_part"],
                                       s["m_part"], s["l_part"], s["out"])
        return s["out"]
    if kind == "generate":
        m = s["m"]
        tokens = m.generate(s["ids"], s["new"], prefill=s["prefill"])
        return {"tokens": torch.tensor(tokens), "logits": m.logits, "kv": m.kv}
    if kind == "decode":
        m, ctx = s["m"], s["ctx"]
        m.reset(ctx)
        m.teacher_force(s["ids"])
        for _ in range(s["new"] - 1):
            m.run_step()
        return {"tokens": m.history[ctx:ctx + s["new"]], "logits": m.logits, "kv": m.kv}
    if kind == "prefill":
        m = s["m"]
        m.reset(s["start"])
        scores = m.prefill(s["ids"], collect_logits=s["score"])
        return {"next": m.tok, "logits": m.logits, "scores": scores, "kv": m.kv}
    if kind == "quantize":
        q = QuantLinear(s["w"], s["group"], keep_ref=False, clip=s["clip"])
        return {"packed": q.packed, "sz": q.sz}
    q, scale, zero = quantize_gptq(s["w"], s["hess"], GROUP, clip=s["clip"])
    return {"q": q, "scale": scale, "zero": zero}


# ---------------------------------------------------------------------------------------------- work and tolerance
def _int4_bytes(n, k, group=GROUP):
    return n * k // 2 + 4 * n * (k // group)


def _layer(c):
    """(bytes, flops per token) of one decoder layer's matrices."""
    H, I = c["hidden_size"], c["intermediate_size"]
    D = H // c["num_attention_heads"]
    n_att, n_qkv = c["num_attention_heads"] * D, (c["num_attention_heads"] + 2 * c["num_key_value_heads"]) * D
    mats = ((n_qkv, H), (H, n_att), (2 * I, H), (H, I))
    return sum(_int4_bytes(n, k) for n, k in mats) + 4 * H, 2 * sum(n * k for n, k in mats)


def _decode_work(c, first_ctx, tokens):
    """Steps at contexts first_ctx + 1 ... first_ctx + tokens (the step's own token included)."""
    H, V, L, n_q, n_kv = (c[k] for k in ("hidden_size", "vocab_size", "num_hidden_layers", "num_attention_heads",
                                         "num_key_value_heads"))
    D = H // n_q
    lb, lf = _layer(c)
    ctx_sum = tokens * first_ctx + tokens * (tokens + 1) // 2
    per_token = L * lb + _int4_bytes(V, H) + 4 * H + 2 * V
    return {"bytes": tokens * per_token + L * 4 * n_kv * D * ctx_sum,
            "flops": tokens * (L * lf + 2 * V * H) + L * 4 * n_q * D * ctx_sum}


def _prefill_work(c, start, T, score):
    H, V, L, n_q, n_kv = (c[k] for k in ("hidden_size", "vocab_size", "num_hidden_layers", "num_attention_heads",
                                         "num_key_value_heads"))
    D = H // n_q
    lb, lf = _layer(c)
    rows = T if score else 1
    ctx_sum = T * start + T * (T + 1) // 2
    return {"bytes": L * (lb + 4 * n_kv * D * (start + T)) + _int4_bytes(V, H) + 2 * H * T + 2 * V * rows,
            "flops": T * L * lf + rows * 2 * V * H + L * 4 * n_q * D * ctx_sum}


def work(case):
    kind = case["kind"]
    if kind == "ops":
        D, n_kv = 64, case["n_kv"]
        n_q = 8 * n_kv
        H, I = n_q * D, case["inter"]
        lb, lf = _layer(dict(hidden_size=H, intermediate_size=I, num_attention_heads=n_q, num_key_value_heads=n_kv))
        ctx = case["ctx"] + 1
        return {"bytes": lb + 4 * n_kv * D * ctx + 4 * H, "flops": lf + 4 * n_q * D * ctx}
    if kind == "attention":
        mean = (case["lo"] + case["hi"]) / 2
        B, n_q, n_kv, D = case["batch"], case["n_q"], case["n_kv"], case["dim"]
        return {"bytes": B * (4 * n_kv * D * mean + 4 * n_q * D), "flops": B * 4 * n_q * D * mean}
    if kind == "generate":
        c, steps = SHAPES[case["shape"]], case["new"] - 1
        a = (_prefill_work(c, 0, case["prompt"], False) if case["prefill"] else _decode_work(c, 0, case["prompt"]))
        b = _decode_work(c, case["prompt"], steps)
        return {k: a[k] + b[k] for k in a}
    if kind == "decode":
        return _decode_work(SHAPES[case["shape"]], case["ctx"], case["new"])
    if kind == "prefill":
        return _prefill_work(SHAPES[case["shape"]], case["start"], case["prompt"], case["score"])
    N, K = case["rows"], case["cols"]
    if kind == "quantize":
        return {"bytes": 2 * N * K + _int4_bytes(N, K, case["group"]), "flops": (7 if case["clip"] else 1) * 6 * N * K}
    # Cholesky of H, inverse, Cholesky of the inverse (K^3 / 3 multiply-adds each, and 2/3 for the inverse); the error of
    # every column goes onto all later ones
    return {"bytes": 2 * N * K + 4 * K * K + N * K + 4 * N * K // GROUP, "flops": 2 * K ** 3 * 4 / 3 + N * K * K}


def tolerance(case):
    kind = case["kind"]
    if kind == "ops":          # about ten fp16 roundings in a chain
        return {"rel": 4e-3}
    if kind == "attention":    # fp16 probabilities and output
        return {"rel": 2e-3}
    if kind == "quantize":
        # plain rounding is exact; with clipping two factors of nearly equal error may change places when the squares
        # are summed in another order, which changes a whole group
        return {"rel": 2e-3, "max": 0.6, "differ": 1e-3} if case["clip"] else "exact"
    if kind == "gptq":         # rounding decisions feed back: a level that flips moves the columns after it
        return {"rel": 1e-2, "max": 0.9, "differ": 1e-2}
    return {"rel": 1e-2}       # logits and cache rows behind a stack of fp16 layers; tokens are exact
