"""The work that users of this framework have it do, as cases that can be timed and checked.

Two levels are covered, because programs use both.  A host program that owns its projections calls the attention
operations over per-session paged caches: `decode_step` once per layer and token, `kv_append` + `attn_prefill` once per
layer and portion of a prompt.  A serving program gives token ids to a device model through `Engine.advance` and reads
logits: the dense F32 stack (Llama / Qwen3 class), and the mixed stack with Tumadra and Nurosun.

A case is a dict: "kind" says which of these, the rest are sizes.  `exact` restates every path in float64.
"""
import math
import random
import zlib

import numpy as np
import torch

import wayruntime_b200 as wr
from wayruntime_b200 import models
from wayruntime_b200.engine import Engine

HEAD_DIM = 128
THETA = {"decode": 5e5, "prefill": 5e5, "dense": 1e6}
EPS = 1e-6
MAX_ROWS = 2048                      # rows of a prompt that a model takes in one portion

#: width -> (feed-forward, query heads, kv heads, inner channels, dt rank): the sizes of the benchmark's models
SIZES = {1024: (3072, 8, 4, 2048, 64), 2048: (6144, 16, 4, 4096, 128), 4096: (12288, 32, 8, 8192, 256)}


def listed():
    qwen = {"kind": "dense", "width": 1024, "layers": 28, "heads": 16, "kv_heads": 8, "vocab": 151936}
    tumadra = {"kind": "tumadra", "width": 2048, "layers": 8, "vocab": 65536, "dtype": "bfloat16"}
    nurosun = {"kind": "nurosun", "width": 2048, "layers": 4, "vocab": 65536, "dtype": "bfloat16"}
    return [
        # one token of a chat with a small model whose projections stay on the host: rows cross from page-locked memory
        {"name": "decode_one_host", "kind": "decode", "sessions": 1, "heads": 16, "kv_heads": 8, "ctx_lo": 64, "ctx_hi": 192,
         "layers": 28, "host": True},
        # the batched decode step of an 8B-class model: 16 unequal sessions, four of its layers
        {"name": "decode_batch16", "kind": "decode", "sessions": 16, "heads": 32, "kv_heads": 8, "ctx_lo": 1024, "ctx_hi": 4096,
         "layers": 4, "host": False},
        # the same with long contexts: 2.1 GB of keys and values
        {"name": "decode_long16", "kind": "decode", "sessions": 16, "heads": 32, "kv_heads": 8, "ctx_lo": 32768, "ctx_hi": 32768,
         "layers": 1, "host": False},
        # a whole prompt, queries handed over in F16
        {"name": "prefill_2048", "kind": "prefill", "past": 0, "rows": 2048, "heads": 32, "kv_heads": 8, "layers": 4, "q": "float16"},
        # a portion in the middle of a long prompt, wide groups, sizes that align with nothing, F32 queries rotated in place
        {"name": "prefill_portion", "kind": "prefill", "past": 6001, "rows": 1999, "heads": 40, "kv_heads": 8, "layers": 2,
         "q": "float32"},
        # Qwen3-0.6B shape: a chat's next token, a full serving batch's next tokens, a prompt
        dict(qwen, name="dense_decode_1", phase="decode", sessions=1, ctx_lo=64, ctx_hi=192),
        dict(qwen, name="dense_decode_16", phase="decode", sessions=16, ctx_lo=200, ctx_hi=2000),
        dict(qwen, name="dense_prefill_1000", phase="prefill", sessions=1, ctx_lo=1000, ctx_hi=1000),
        # selective scans and differential attention in turn: a full portion of a prompt, a chat's next token
        dict(tumadra, name="tumadra_prefill_2048", phase="prefill", sessions=1, ctx_lo=2048, ctx_hi=2048),
        dict(tumadra, name="tumadra_decode_1", phase="decode", sessions=1, ctx_lo=256, ctx_hi=2000),
        # latent attention with experts: an odd prompt, a full serving batch's next tokens
        dict(nurosun, name="nurosun_prefill_1501", phase="prefill", sessions=1, ctx_lo=1501, ctx_hi=1501),
        dict(nurosun, name="nurosun_decode_16", phase="decode", sessions=16, ctx_lo=256, ctx_hi=2000),
    ]


def spread(rng, lo, hi):
    """A whole number in [lo, hi], even over its logarithm."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["decode"] * 3 + ["prefill"] * 2 + ["dense"] * 3 + ["tumadra"] * 2 + ["nurosun"] * 2)
    if kind == "decode":
        kv = rng.choice([1, 2, 4, 8, 8])
        heads = kv * rng.choice([1, 2, 4, 4, 5, 8])
        sessions, top = spread(rng, 1, 16), spread(rng, 64, 32768)
        most = max(1, int(2.1e9 / (512 * sessions * top * kv)))
        return {"kind": kind, "sessions": sessions, "heads": heads, "kv_heads": kv, "ctx_lo": max(1, top // rng.choice([1, 2, 4])),
                "ctx_hi": top, "layers": min(most, spread(rng, 1, 32)), "host": rng.random() < 0.25}
    if kind == "prefill":
        kv = rng.choice([1, 4, 8, 8])
        heads = kv * rng.choice([2, 4, 4, 5])
        rows = spread(rng, 17, 4096)
        past = 0 if rng.random() < 0.5 else spread(rng, 16, 8192)
        pairs = heads * rows * (past + rows / 2)
        return {"kind": kind, "past": past, "rows": rows, "heads": heads, "kv_heads": kv,
                "layers": max(1, min(rng.choice([1, 2, 4]), int(1.1e9 / pairs))), "q": rng.choice(["float16", "float32"])}
    phase = rng.choice(["decode", "prefill"])
    width = rng.choice([1024, 1024, 2048, 4096])
    dtype = "float32" if kind == "dense" or rng.random() < 0.15 else "bfloat16"
    layers = rng.choice([2, 4]) * (2 if width == 1024 else 1)
    if width == 4096:
        layers = 2
    if phase == "decode":
        sessions, top = spread(rng, 1, 16), spread(rng, 32, 2000)
        lo = max(2, top // rng.choice([1, 2, 8]))
    else:
        cost = 3 if width == 4096 else 1
        sessions, top = 1, spread(rng, 17, (768 if dtype == "float32" else 2048) // cost)
        lo = top
    case = {"kind": kind, "width": width, "layers": layers, "vocab": rng.choice([32003, 65536]), "phase": phase, "sessions": sessions,
            "ctx_lo": lo, "ctx_hi": top}
    if kind == "dense":
        kv = rng.choice([4, 8])
        return dict(case, heads=kv * rng.choice([1, 2, 4]), kv_heads=kv)
    return dict(case, dtype=dtype)


# ---- inputs

_CONTEXT = []


def context():
    """The process's one device context, as a program keeps it."""
    if not _CONTEXT:
        _CONTEXT.append(wr.Context(0, attn_max_seq=65536))
    return _CONTEXT[0]


def generator(*what):
    g = torch.Generator(device="cuda")
    g.manual_seed(zlib.crc32(repr(what).encode()))
    return g


def normal(shape, *what, dtype=torch.float32):
    return torch.randn(shape, generator=generator(*what), device="cuda", dtype=torch.float32).to(dtype)


def lengths(case, seed):
    """Keys that each session's new token attends, itself among them."""
    r = random.Random(seed)
    return [r.randint(case["ctx_lo"], case["ctx_hi"]) for _ in range(case["sessions"])]


def tokens(case, seed, n, *what):
    r = random.Random(zlib.crc32(repr((seed, n) + what).encode()))
    return [r.randrange(case["vocab"]) for _ in range(n)]


def cache_rows(case, seed, rows):
    """F16 keys (unit scale, as they are after the head norm) and values (as a projection of normed rows has them)
    of every layer: [layers][2][rows][kv heads][head dim]."""
    x = torch.empty((case["layers"], 2, rows, case["kv_heads"], HEAD_DIM), dtype=torch.float16, device="cuda")
    for i in range(case["layers"]):
        for which, scale in ((0, 1.0), (1, 0.64 if case["kind"] == "dense" else 1.0)):
            x[i, which] = normal(x.shape[2:], "cache", seed, i, which, dtype=torch.float16) * scale
    return x


def fill(case, seed, kvs, counts):
    rows = cache_rows(case, seed, sum(counts))
    torch.cuda.synchronize()
    for i in range(case["layers"]):
        lo = 0
        for kv, n in zip(kvs, counts):
            for which in (0, 1):
                if n:
                    kv.write_rows(i, which, 0, rows[i, which, lo:lo + n])
            lo += n
    context().sync()


def new_rows(case, seed, n):
    """F32 query, key and value rows of every layer as projections leave them."""
    shape = lambda h: (case["layers"], n, h, HEAD_DIM)  # noqa: E731
    return [normal(shape(h), name, seed) for name, h in (("q", case["heads"]), ("k", case["kv_heads"]), ("v", case["kv_heads"]))]


# ---- models: configurations, weights, and the last one that was built

def config(case):
    ff, heads, kv, inner, rank = SIZES[case["width"]]
    width, n, vocab = case["width"], case["layers"], case["vocab"]
    if case["kind"] == "dense":
        return {"architectures": ["Qwen3ForCausalLM"], "hidden_size": width, "intermediate_size": ff, "num_hidden_layers": n,
                "num_attention_heads": case["heads"], "num_key_value_heads": case["kv_heads"], "head_dim": HEAD_DIM,
                "vocab_size": vocab, "tie_word_embeddings": True, "rope_theta": THETA["dense"], "rms_norm_eps": EPS}
    if case["kind"] == "tumadra":
        mlp = {"kind": "dense", "ff": ff}
        attn = {"heads": heads, "kv_heads": kv, "dim": 64, "vdim": 128, "scale": 0.125, "diff": 0.5,
                "q_temp": {"coef": 0.1, "every": 1024}}
        scan = {"inner": inner, "state": 16, "dt_rank": rank, "conv": 4}
        return {"architecture": "Tumadra", "width": width, "vocab": vocab, "norm": {"groups": 4, "eps": 1e-5},
                "layers": [{"type": "attention", "mixer": attn, "mlp": mlp} if i % 2 else
                           {"type": "mamba1", "mixer": scan, "mlp": mlp} for i in range(n)]}
    mixer = {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": width // 2, "kv_rank": 512, "scale": 192 ** -0.5,
             "rot": {"base": 10000.0, "dims": 64}}
    moe = {"kind": "moe", "expert": {"ff": ff // 4, "limit": 7.0}, "router": {"experts": 32, "top": 4}}
    return {"architecture": "Nurosun", "width": width, "vocab": vocab, "norm": {"eps": 1e-5}, "embedding": {"scale": width ** 0.5},
            "residual_mult": 0.5,
            "layers": [{"type": "latent_attention", "mixer": dict(mixer, kv_from=i - 1), "mlp": moe} if i % 2 else
                       {"type": "latent_attention", "mixer": mixer, "mlp": {"kind": "dense", "ff": ff}} for i in range(n)]}


class Weights:
    """A checkpoint's answers, made from the tensor's name: matrices over the square root of their inputs, norms near
    one.  A Nurosun token carries its experts in the first columns of its embedding, which no layer writes and each
    layer's router reads in an order of its own: loads are even, and which expert a row takes hangs on no rounding."""

    def __init__(self, cfg, bf16):
        self.bf16 = bf16
        self.key = zlib.crc32(repr(cfg).encode())
        self.nurosun = cfg.get("architecture") == "Nurosun"
        self.experts = max([lay["mlp"]["router"]["experts"] for lay in cfg["layers"] if lay["mlp"]["kind"] == "moe"] + [0]) if self.nurosun else 0

    def __contains__(self, name):
        return True

    def make(self, name, shape):
        last = name.split(".")[-1]
        x = normal(shape, self.key, name)
        if "norm" in name:
            x = 1 + 0.1 * x
        elif last == "shift":
            x = torch.sigmoid(x)
        elif last == "A_log":
            x = x.clamp(-2, 2)
        elif last in ("lq1", "lk1", "lq2", "lk2"):
            x = 0.4 * x / math.sqrt(shape[0])
        elif name.endswith("dt.b"):
            x = x.clamp(-2, 2) - 2
        elif name == "embed" and self.nurosun:
            x /= math.sqrt(shape[1])
        elif len(shape) == 2 and "embed" not in name:
            x /= math.sqrt(shape[1])
        elif name != "embed" and "embed_tokens" not in name and last != "D":
            x *= 0.3
        if self.experts:
            e = self.experts
            if name == "embed":
                chosen = torch.rand((shape[0], e), generator=generator(self.key, "code"), device="cuda").argsort(1) < 4
                x[:, :e] = torch.where(chosen, 1.0, -0.125) * 2 / math.sqrt(shape[1])
            elif name.endswith("router"):
                x = torch.zeros(shape, device="cuda")
                at = torch.randperm(e, generator=generator(self.key, name), device="cuda")
                x[torch.arange(e, device="cuda"), at] = 1 + 0.1 * torch.rand(e, generator=generator(self.key, name, 1), device="cuda")
            elif name.endswith("router.b"):
                x = torch.zeros(shape, device="cuda")
            elif name.endswith(("mix.o", ".down")):
                x[:e] = 0
            elif name.endswith("norm1"):
                x[:e] = 1
        return x.to(torch.bfloat16) if self.bf16 else x

    def get(self, name, shape):
        x = self.make(name, shape)
        return x.view(torch.int16).cpu().numpy().view(np.uint16) if self.bf16 else x.cpu().numpy()

    f32 = get

    def f64(self, name, shape):
        return self.make(name, shape).double()


class Model:
    """A device model that is given back with its last user."""

    def __init__(self, case):
        cfg = config(case)
        self.key, self.dtype = repr(cfg) + self.format(case), self.format(case)
        self.model = models.build(context(), cfg, Weights(cfg, self.dtype == "bfloat16"), self.dtype, MAX_ROWS)

    @staticmethod
    def format(case):
        return case.get("dtype", "float32")

    def __del__(self):
        if getattr(self, "model", None):
            self.model.close()


_MODEL = []


def model_of(case):
    """The model of the case: weights are loaded once and serve all prompts, as in a program."""
    if not _MODEL or _MODEL[0].key != repr(config(case)) + Model.format(case):
        _MODEL.clear()
        _MODEL.append(Model(case))
    return _MODEL[0]


# ---- the cases themselves

def prepare(case, seed):
    if case["kind"] == "decode":
        n, lens = case["sessions"], lengths(case, seed)
        ctx = context()
        kvs = [ctx.kv_create(case["layers"], case["kv_heads"], HEAD_DIM, m) for m in lens]
        fill(case, seed, kvs, [m - 1 for m in lens])
        q, k, v = new_rows(case, seed, n)
        out = torch.zeros_like(q)
        if case["host"]:
            q, k, v, out = (x.cpu().pin_memory() for x in (q, k, v, out))
        torch.cuda.synchronize()
        positions = wr.Batch.u32([m - 1 for m in lens])
        return {"case": case, "kvs": wr.Batch(kvs), "positions": positions, "q": q, "k": k, "v": v, "out": out}
    if case["kind"] == "prefill":
        kv = context().kv_create(case["layers"], case["kv_heads"], HEAD_DIM, case["past"] + case["rows"])
        fill(case, seed, [kv], [case["past"]])
        q, k, v = new_rows(case, seed, case["rows"])
        if case["q"] == "float16":
            q = q.half()
        out = torch.zeros(q.shape, device="cuda")
        torch.cuda.synchronize()
        return {"case": case, "kv": kv, "q": q, "k": k, "v": v, "out": out}
    m = model_of(case)
    engine, lens = Engine(m.model), lengths(case, seed)
    if case["phase"] == "prefill":
        s = engine.session(lens[0])
        return {"case": case, "model": m, "engine": engine, "sessions": [s], "at": [0], "tokens": [tokens(case, seed, lens[0])]}
    sessions = [engine.session(n) for n in lens]
    if case["kind"] == "dense":
        fill(case, seed, [s.kv for s in sessions], [n - 1 for n in lens])
    else:
        for i, (s, n) in enumerate(zip(sessions, lens)):
            if n > 1:
                engine.advance([s], [tokens(case, seed, n, i)[:-1]], [[]])
    return {"case": case, "model": m, "engine": engine, "sessions": sessions, "at": [n - 1 for n in lens],
            "tokens": [tokens(case, seed, n, i)[-1:] for i, n in enumerate(lens)]}


def run(state):
    case = state["case"]
    if case["kind"] == "decode":
        ctx, q, k, v, out = context(), state["q"], state["k"], state["v"], state["out"]
        for i in range(case["layers"]):
            ctx.decode_step(state["kvs"], i, state["positions"], q[i], k[i], v[i], out[i], case["heads"], theta=THETA["decode"])
        return {"out": out, "q": q}                  # (device queries are rotated in place, on from where they stand)
    if case["kind"] == "prefill":
        ctx, kv, q, k, v, out = context(), state["kv"], state["q"], state["k"], state["v"], state["out"]
        rotate = case["q"] == "float32"
        for i in range(case["layers"]):
            ctx.kv_append([kv], i, [case["past"]], k[i], v[i], q[i] if rotate else None, case["heads"] if rotate else 0,
                          theta=THETA["prefill"], n_tokens=case["rows"])
            ctx.attn_prefill(kv, i, case["past"], case["rows"], q[i], out[i], case["heads"])
        return {"out": out, "q": q}
    for s, at in zip(state["sessions"], state["at"]):
        s.pos = at
    return state["engine"].advance(state["sessions"], state["tokens"])


def work(case):
    if case["kind"] == "decode":
        n, mean = case["sessions"], (case["ctx_lo"] + case["ctx_hi"]) / 2
        row, hq, kv = 4 * HEAD_DIM, case["heads"], case["kv_heads"]
        return {"bytes": case["layers"] * n * (mean * kv * row + (2 * hq + 2 * kv) * row),
                "flops": case["layers"] * n * mean * hq * 4 * HEAD_DIM}
    if case["kind"] == "prefill":
        p, n, hq, kv = case["past"], case["rows"], case["heads"], case["kv_heads"]
        q = 2 if case["q"] == "float16" else 4
        return {"bytes": case["layers"] * HEAD_DIM * ((p + n) * kv * 4 + n * kv * 8 + n * hq * (q + 4)),
                "flops": case["layers"] * 4 * HEAD_DIM * hq * (p * n + n * (n + 1) / 2)}
    ff, heads, kv, inner, rank = SIZES[case["width"]]
    d, size = case["width"], 4 if Model.format(case) == "float32" else 2
    mean = (case["ctx_lo"] + case["ctx_hi"]) / 2
    prompt = case["phase"] == "prefill"
    rows = mean if prompt else case["sessions"]
    pairs = mean * (mean + 1) / 2 if prompt else rows * mean             # (query, key) pairs per head
    held = 0 if prompt else rows * mean                                  # cache rows read
    used = touched = per_row = cache = 0
    for i in range(case["layers"]):
        if case["kind"] == "dense":
            hq, hk = case["heads"] * HEAD_DIM, case["kv_heads"] * HEAD_DIM
            w = d * (2 * hq + 2 * hk + 3 * ff)
            used, touched, per_row, cache = used + w, touched + w, per_row + 4 * hq * pairs / rows, cache + 4 * hk
        elif case["kind"] == "tumadra":
            w = 2 * d * ff
            if i % 2:
                w += d * (heads * 128 + kv * 128 + kv * 128 + heads * 128 + heads * 128)
                per_row += 2 * heads * (2 * 64 + 2 * 128) * pairs / rows
                cache += kv * 256 * (4 if size == 4 else 2)
            else:
                w += 3 * d * inner + inner * (2 * rank + 32)
                per_row += 8 * inner * 16
            used, touched = used + w, touched + w
        else:
            w = d * (d // 2) + (d // 2) * heads * 192 + 512 * heads * 256 + heads * 128 * d + (0 if i % 2 else d * 576)
            per_row += heads * 2 * (192 + 128) * pairs / rows
            cache += 576 * (4 if size == 4 else 2)
            if i % 2:
                expert = 3 * d * (ff // 4)
                used += w + 4 * expert
                touched += w + expert * 32 * (1 - (1 - 4 / 32) ** rows)
            else:
                used, touched = used + w + 3 * d * ff, touched + w + 3 * d * ff
    out_rows = 1 if prompt else rows
    head = d * case["vocab"]
    return {"bytes": size * (touched + head) + held * cache + out_rows * case["vocab"] * 4 + rows * d * size,
            "flops": rows * (2 * used + per_row) + 2 * head * out_rows}


def tolerance(case):
    """About four times the error seen against float64 (the larger of a kind's cases)."""
    if case["kind"] == "decode":
        return {"rel": 6e-6}                         # F32 sums over F16 keys and values: 1.5e-6 at 32768 keys
    if case["kind"] == "prefill":
        return {"rel": 1.2e-3}                       # F16 queries and weights: 3e-4
    if case["kind"] == "dense":                      # F32, prompts attend through the F16 kernel: 8e-7 and 2e-4
        return {"rel": 2e-5 if case["phase"] == "decode" else 8e-4}
    if case["dtype"] == "float32":
        return {"rel": 2e-5}
    if case["kind"] == "tumadra":                    # BF16: 5e-3
        return {"rel": 2e-2}
    return {"rel": 8e-3}                             # BF16: 1.6e-3, most of it from the prompt's portions


# ---- the same in float64

def truncated_half(x):
    """F16 of a float64 tensor, cut towards zero as the cache stores keys and values."""
    h = x.half()
    over = h.double().abs() > x.abs()
    return (h.view(torch.int16) - over.to(torch.int16)).view(torch.float16).double()


def rope_table(positions, dim, theta):
    """cos and sin that the dense path and the operations rotate with: their caches hold, bit for bit, what the reference's
    float32 series give (src/core/mathx.c:37-147), which near +-pi are far from the functions that they stand for."""
    f = np.float32
    ln2, pi, two_pi = f(0.6931471805599453), f(3.14159265358979), f(6.28318530717958)
    m, e = math.frexp(theta)
    m, e = f(2 * m), f(e - 1)
    t = (m - f(1)) / (m + f(1))
    t2 = t * t
    log = (f(2) * t) * (f(1) + t2 * (f(1) / f(3) + t2 * (f(1) / f(5) + t2 * (f(1) / f(7))))) + e * ln2
    x = np.arange(0, dim, 2).astype(f) / f(dim) * log
    k = (x / ln2 + f(0.5)).astype(np.int32)
    r = x - k.astype(f) * ln2
    r2 = r * r
    power = f(1) + r
    for term in (r2 * f(0.5), r2 * r * f(1 / 6), r2 * r2 * f(1 / 24), r2 * r2 * r * f(1 / 120)):
        power = power + term
    x = np.asarray(positions, f)[:, None] / (power * np.exp2(k).astype(f))
    while (far := x > pi).any():
        x[far] -= two_pi
    x2 = x * x
    x3, x4 = x2 * x, x2 * x2
    x5 = x3 * x2
    sin = x - x3 * f(1 / 6) + x5 * f(1 / 120) - x5 * x2 * f(1 / 5040)
    cos = f(1) - x2 * f(0.5) + x4 * f(1 / 24) - x4 * x2 * f(1 / 720)
    return [torch.from_numpy(v).double().cuda()[:, None, :] for v in (cos, sin)]


def turned_by(x, cos, sin):
    """x [rows, heads, dim]: components j and j + dim/2 turn by the row's j-th angle."""
    a, b = x.chunk(2, -1)
    return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)


def rotated(x, positions, theta):
    return turned_by(x, *rope_table(positions, x.shape[-1], theta))


def truly_rotated(x, positions, base):
    half = x.shape[-1] // 2
    turn = torch.as_tensor(positions, device="cuda", dtype=torch.float64)[:, None, None]
    turn = turn * base ** (-torch.arange(half, device="cuda", dtype=torch.float64) / half)
    return turned_by(x, turn.cos(), turn.sin())


def attend(q, k, v, scale, first):
    """q [n, heads, dim], k, v [keys, kv heads, dim]: row i sees keys up to first + i; one head after another."""
    group = q.shape[1] // k.shape[1]
    hidden = torch.arange(k.shape[0], device="cuda")[None, :] > first + torch.arange(q.shape[0], device="cuda")[:, None]
    out = [torch.softmax((q[:, h] @ k[:, h // group].T * scale).masked_fill_(hidden, -math.inf), -1) @ v[:, h // group]
           for h in range(q.shape[1])]
    return torch.stack(out, 1)


def exact(case, seed):
    if case["kind"] == "decode":
        return exact_decode(case, seed)
    if case["kind"] == "prefill":
        return exact_prefill(case, seed)
    lens = lengths(case, seed)
    cfg = config(case)
    w = Weights(cfg, Model.format(case) == "bfloat16")
    if case["kind"] == "dense":
        rows = exact_dense(case, seed, w, lens)
    else:
        prompt = case["phase"] == "prefill"
        ids = torch.zeros((len(lens), max(lens)), dtype=torch.long)
        for i, n in enumerate(lens):
            ids[i, :n] = torch.tensor(tokens(case, seed, n) if prompt else tokens(case, seed, n, i))
        rows = (exact_tumadra if case["kind"] == "tumadra" else exact_nurosun)(cfg, w, ids.cuda(), lens)
    return [row[None] for row in rows]


def exact_decode(case, seed):
    lens = lengths(case, seed)
    past = cache_rows(case, seed, sum(lens) - len(lens))
    q, k, v = (x.double() for x in new_rows(case, seed, case["sessions"]))
    at = [n - 1 for n in lens]
    out = torch.empty_like(q)
    turned = torch.empty_like(q)
    for i in range(case["layers"]):
        turned[i] = rotated(q[i], at, THETA["decode"])
        kr, vr, lo = truncated_half(rotated(k[i], at, THETA["decode"])), truncated_half(v[i]), 0
        for s, n in enumerate(at):
            kk = torch.cat([past[i, 0, lo:lo + n].double(), kr[s:s + 1]])
            vv = torch.cat([past[i, 1, lo:lo + n].double(), vr[s:s + 1]])
            out[i, s] = attend(turned[i, s:s + 1], kk, vv, HEAD_DIM ** -0.5, n)[0]
            lo += n
    return {"out": out, "q": q if case["host"] else turned}


def exact_prefill(case, seed):
    p, n = case["past"], case["rows"]
    past = cache_rows(case, seed, p)
    q, k, v = new_rows(case, seed, n)
    q = q.half().double() if case["q"] == "float16" else q.double()
    out, at = torch.empty_like(q), range(p, p + n)
    for i in range(case["layers"]):
        if case["q"] == "float32":
            q[i] = rotated(q[i], at, THETA["prefill"])
        kk = torch.cat([past[i, 0].double(), truncated_half(rotated(k[i].double(), at, THETA["prefill"]))])
        vv = torch.cat([past[i, 1].double(), truncated_half(v[i].double())])
        out[i] = attend(q[i], kk, vv, HEAD_DIM ** -0.5, p)
    return {"out": out, "q": q}


def rms(x, w, eps):
    return x / (x.square().mean(-1, keepdim=True) + eps).sqrt() * w


def silu(x):
    return x * torch.sigmoid(x)


def exact_dense(case, seed, w, lens):
    d, ff, hq, hk, vocab = case["width"], SIZES[case["width"]][0], case["heads"], case["kv_heads"], case["vocab"]
    prompt = case["phase"] == "prefill"
    ids = tokens(case, seed, lens[0]) if prompt else [tokens(case, seed, n, i)[-1] for i, n in enumerate(lens)]
    at = list(range(lens[0])) if prompt else [n - 1 for n in lens]
    embed = w.f64("model.embed_tokens.weight", (vocab, d))
    past = None if prompt else cache_rows(case, seed, sum(at))
    x = embed[torch.tensor(ids, device="cuda")]
    for i in range(case["layers"]):
        get = lambda name, *shape: w.f64(f"model.layers.{i}.{name}.weight", shape)  # noqa: B023, E731
        h = rms(x, get("input_layernorm", d), EPS)
        q, k, v = ((h @ get(f"self_attn.{n}_proj", m * HEAD_DIM, d).T).view(len(ids), m, HEAD_DIM) for n, m in (("q", hq), ("k", hk), ("v", hk)))
        q = rotated(rms(q, get("self_attn.q_norm", HEAD_DIM), EPS), at, THETA["dense"])
        k = truncated_half(rotated(rms(k, get("self_attn.k_norm", HEAD_DIM), EPS), at, THETA["dense"]))
        v = truncated_half(v)
        if prompt:
            a = attend(q, k, v, HEAD_DIM ** -0.5, 0)
        else:
            a, lo = torch.empty_like(q), 0
            for s, n in enumerate(at):
                kk, vv = (torch.cat([past[i, c, lo:lo + n].double(), new[s:s + 1]]) for c, new in ((0, k), (1, v)))
                a[s], lo = attend(q[s:s + 1], kk, vv, HEAD_DIM ** -0.5, n)[0], lo + n
        x = x + a.reshape(len(ids), -1) @ get("self_attn.o_proj", d, hq * HEAD_DIM).T
        h = rms(x, get("post_attention_layernorm", d), EPS)
        x = x + (silu(h @ get("mlp.gate_proj", ff, d).T) * (h @ get("mlp.up_proj", ff, d).T)) @ get("mlp.down_proj", d, ff).T
    x = x[-1:] if prompt else x
    return list(rms(x, w.f64("model.norm.weight", (d,)), EPS) @ embed.T)


def last_rows(x, lens):
    return x[torch.arange(len(lens), device="cuda"), torch.tensor(lens, device="cuda") - 1]


def causal_softmax(scores):
    hidden = torch.ones(scores.shape[-2:], device="cuda", dtype=torch.bool).triu(1)
    return torch.softmax(scores.masked_fill_(hidden, -math.inf), -1)


def exact_tumadra(cfg, w, ids, lens):
    """Whole sequences [sessions, tokens], shorter ones filled up behind; logits of each one's last token."""
    d, eps, groups = cfg["width"], cfg["norm"]["eps"], cfg["norm"]["groups"]
    n, t = ids.shape
    norm = lambda x, name: rms(x.unflatten(-1, (groups, -1)), 1.0, eps).flatten(-2) * w.f64(name, (d,))  # noqa: E731
    pos = torch.arange(t, device="cuda", dtype=torch.float64)
    col = torch.arange(d, device="cuda")
    angle = pos[:, None] * 10000.0 ** (-(2.0 * (col // 2)) / d)
    x = w.f64("embed", (cfg["vocab"], d))[ids] + torch.where(col % 2 == 0, angle.sin(), angle.cos())
    for i, lay in enumerate(cfg["layers"]):
        c, pre = lay["mixer"], f"l{i}."
        mix = lambda name, *shape: w.f64(f"{pre}mix.{name}", shape)  # noqa: B023, E731
        h = norm(x, pre + "norm1")
        before = torch.cat([torch.zeros_like(h[:, :1]), h[:, :-1]], 1)
        h = h + (before - h) * w.f64(pre + "shift", (d,))
        if lay["type"] == "attention":
            H, G, dim, vd = c["heads"], c["kv_heads"], c["dim"], c["vdim"]
            q = (h @ mix("q", H * 2 * dim, d).T + mix("q.b", H * 2 * dim)).view(n, t, H, 2, dim)
            k = (h @ mix("k", G * 2 * dim, d).T + mix("k.b", G * 2 * dim)).view(n, t, G, 2, dim)
            v = (h @ mix("v", G * vd, d).T + mix("v.b", G * vd)).view(n, t, G, vd)
            q = q * (1.0 + c["q_temp"]["coef"] * torch.log(torch.floor((pos + 1) / c["q_temp"]["every"]) + 1))[:, None, None, None]
            lam = torch.exp((mix("lq1", dim) * mix("lk1", dim)).sum()) - torch.exp((mix("lq2", dim) * mix("lk2", dim)).sum()) + c["diff"]
            heads = []
            for head in range(H):
                g = head // (H // G)
                a = [causal_softmax(q[:, :, head, m] @ k[:, :, g, m].mT * c["scale"]) @ v[:, :, g] for m in (0, 1)]
                heads.append(rms(a[0] - lam * a[1], 1.0, eps) * (1.0 - c["diff"]))
            y = torch.cat(heads, -1) * torch.sigmoid(h @ mix("g", H * vd, d).T)
            x = x + y @ mix("o", d, H * vd).T
        else:
            inner, state, rank, taps = c["inner"], c["state"], c["dt_rank"], c["conv"]
            u, z = (h @ mix("in", 2 * inner, d).T).split(inner, -1)
            taps_w, up = mix("conv", inner, taps), torch.nn.functional.pad(u, (0, 0, taps - 1, 0))
            u = silu(sum(up[:, j:j + t] * taps_w[:, j] for j in range(taps)) + mix("conv.b", inner))
            dt, B, C = (u @ mix("x", rank + 2 * state, inner).T).split([rank, state, state], -1)
            dt = torch.nn.functional.softplus(dt @ mix("dt", inner, rank).T + mix("dt.b", inner), threshold=1e9)
            A, s = -mix("A_log", inner, state).exp(), torch.zeros((n, inner, state), device="cuda", dtype=torch.float64)
            y, gain = torch.empty_like(u), dt * u
            for j in range(t):
                s = torch.exp(dt[:, j, :, None] * A).mul_(s).add_(gain[:, j, :, None] * B[:, j, None, :])
                y[:, j] = (s @ C[:, j, :, None])[..., 0]
            x = x + ((y + mix("D", inner) * u) * silu(z)) @ mix("o", d, inner).T
        h, ff = norm(x, pre + "norm2"), lay["mlp"]["ff"]
        u = h @ w.f64(pre + "mlp.up", (ff, d)).T
        a, b, c3, e = w.f64(pre + "mlp.act", (4,))
        u = a * rms(u, 1.0, eps) + b * rms(u ** 2, 1.0, eps) + c3 * rms(u ** 3, 1.0, eps) + e
        x = x + u @ w.f64(pre + "mlp.down", (d, ff)).T
    return list(norm(last_rows(x, lens), "final.norm") @ w.f64("head", (cfg["vocab"], d)).T)


def exact_nurosun(cfg, w, ids, lens):
    """As exact_tumadra."""
    d, eps = cfg["width"], cfg["norm"]["eps"]
    n, t = ids.shape
    def norm(x, name):
        x = x - x.mean(-1, keepdim=True)
        return rms(x, w.f64(name, (d,)), eps)
    turn = lambda v, base: truly_rotated(v.flatten(0, 1), list(range(t)) * n, base).unflatten(0, (n, t))  # noqa: E731
    x = w.f64("embed", (cfg["vocab"], d))[ids] * cfg["embedding"]["scale"]
    rows = None
    for i, lay in enumerate(cfg["layers"]):
        c, mlp, pre = lay["mixer"], lay["mlp"], f"l{i}."
        mix = lambda name, *shape: w.f64(f"{pre}mix.{name}", shape)  # noqa: B023, E731
        H, dim, rot, vd, rank, qr, base = c["heads"], c["dim"], c["rot_dim"], c["vdim"], c["kv_rank"], c["q_rank"], c["rot"]["base"]
        h = norm(x, pre + "norm1")
        if c.get("kv_from") is None:
            both = h @ mix("dkv", rank + rot, d).T
            rows = rms(both[..., :rank], mix("dkv.norm", rank), eps), turn(both[..., None, rank:], base)[:, :, 0]
        q = (rms(h @ mix("dq", qr, d).T, mix("dq.norm", qr), eps) @ mix("uq", H * (dim + rot), qr).T).view(n, t, H, dim + rot)
        turned = turn(q[..., dim:], base)
        uk, uv, heads = mix("uk", H * dim, rank), mix("uv", H * vd, rank), []
        for g in range(H):
            scores = q[:, :, g, :dim] @ (rows[0] @ uk[g * dim:(g + 1) * dim].T).mT + turned[:, :, g] @ rows[1].mT
            heads.append(causal_softmax(scores * c["scale"]) @ (rows[0] @ uv[g * vd:(g + 1) * vd].T))
        y = torch.cat(heads, -1) @ mix("o", d, H * vd).T
        if mlp["kind"] == "dense":
            g, u, down = (w.f64(f"{pre}mlp.{m}", s) for m, s in (("gate", (mlp["ff"], d)), ("up", (mlp["ff"], d)), ("down", (d, mlp["ff"]))))
            y = y + (silu(h @ g.T) * (h @ u.T)) @ down.T
        else:
            E, top, ff, limit = mlp["router"]["experts"], mlp["router"]["top"], mlp["expert"]["ff"], mlp["expert"]["limit"]
            flat = h.flatten(0, 1)
            value, chosen = (flat @ w.f64(pre + "mlp.router", (E, d)).T + w.f64(pre + "mlp.router.b", (E,))).topk(top, -1)
            weight, added = torch.softmax(value, -1), torch.zeros_like(flat)
            for e in range(E):
                at, slot = torch.nonzero(chosen == e, as_tuple=True)
                gate, up, down = (w.f64(f"{pre}mlp.e{e}.{m}", s) for m, s in (("gate", (ff, d)), ("up", (ff, d)), ("down", (d, ff))))
                g, u = (flat[at] @ gate.T).clamp(max=limit), (flat[at] @ up.T).clamp(-limit, limit)
                added[at] += weight[at, slot, None] * ((g * torch.sigmoid(1.702 * g) * (u + 1)) @ down.T)
            y = y + added.view(n, t, d)
        x = x + cfg["residual_mult"] * y
    return list(norm(last_rows(x, lens), "final.norm") @ w.f64("head", (cfg["vocab"], d)).T)
