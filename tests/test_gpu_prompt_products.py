"""GPU: the dense stack's products for more rows than a decode batch (gemm_f32.cu), against float64.

One layer; the attention rows that the call reports (attn_tap_out) are the fixed point in the middle:
    hidden_out = embed + attn @ wo^T + FFN(RMSNorm(.))
checks the split of plain and normed rows, the gate / up pairs and the sums in parts, and the V rows that reach the
cache check the three-segment product (to one F16 step: the cache truncates).

Tolerance (2-norm): a product rounds its result once, the sums in parts and the residual's additions up to four times more,
the norm's sum of squares, quotient and root at most eighteen times, SiLU and its product six: under 32 roundings of 2^-24
for what rows pass through.  The operands are within sqrt(k) 2^-31 of their rows' length and the digit products left out within 2^-28
of the largest ones (2^-31 in the mean square): below one rounding more for K up to 4096.
"""
import numpy as np
import pytest

import _gen
from test_gpu_model_glue import _after_attention, _model, _rms, _weights

pytestmark = pytest.mark.gpu
REL = 33 * 2.0 ** -24

SHAPES = [  # rows, hidden, q heads, kv heads, ffn
    (17, 132, 2, 1, 20),              # nothing aligns: one K block and a bit, eight-row groups half full
    (128, 256, 4, 2, 520), (129, 256, 4, 2, 524),
    (300, 1024, 8, 4, 1536),          # parts of K in both sums, several tiles
    (257, 2052, 16, 8, 4100),         # several tiles of 128 columns, K beyond a row's kept values
    (40, 512, 10, 2, 2052),           # short prompt, four parts
]


def _run(shape, rows, w, max_rows, tokens):
    import wayruntime_b200 as wr
    ctx = wr.Context(0)
    dm = _model(ctx, w, shape, max_rows=max_rows)
    kv = ctx.kv_create(shape["n_layers"], shape["n_kv_heads"], 128, rows)
    res = dm.forward(dm.FWD_PREFILL, [kv], [0], tokens, hidden=True, attn_tap=True)
    v = kv.read_rows(0, 1, 0, rows).reshape(rows, -1).view(np.float16).astype(np.float64)
    kv.close()
    dm.close()
    ctx.close()
    return res, v


def _check(res, v, w, tokens):
    emb = w["embed"][tokens]
    want = _after_attention(w, emb, res["attn"][0]) - emb
    got = res["hidden"].astype(np.float64) - emb
    assert np.linalg.norm(got - want) <= REL * (np.linalg.norm(want) + np.linalg.norm(emb))
    want = _rms(emb, w["l0.attn_norm"]) @ w["l0.wv"].astype(np.float64).T
    assert np.abs(v - want).max() <= 2.0 ** -10 * np.abs(want).max() * (1 + 1e-3)


@pytest.mark.parametrize("rows,hidden,n_q,n_kv,ffn", SHAPES)
def test_rows_match_float64(rows, hidden, n_q, n_kv, ffn):
    shape = dict(n_layers=1, hidden=hidden, n_q_heads=n_q, n_kv_heads=n_kv, head_dim=128, vocab=515, ffn=ffn)
    w = _weights(shape, 1200 + rows)
    tokens = [(29 * r + 3) % shape["vocab"] for r in range(rows)]
    res, v = _run(shape, rows, w, max(rows, 64), tokens)
    _check(res, v, w, tokens)


def test_rows_of_very_different_scale_keep_their_precision():
    """Weight rows from 1e-18 to 1e9, a row of zeros, large values beside small ones, a channel that the next weight undoes:
    every column of the result by its own norm."""
    shape = dict(n_layers=1, hidden=256, n_q_heads=4, n_kv_heads=2, head_dim=128, vocab=64, ffn=256)
    w = _weights(shape, 1300, tied=False)
    for name in ("l0.w_gate", "l0.w_up", "l0.wv"):
        w[name][3] *= 1e-18
        w[name][5] = 0.0
        w[name][7, 1] = 64.0
    w["l0.w_down"][9] *= 1e9
    w["l0.wo"][11] *= 1e-30
    w["l0.w_up"][13] *= 1024.0
    w["l0.w_down"][:, 13] /= 1024.0
    w["embed"][8] *= 1e-3
    tokens = [r % 64 for r in range(33)]
    res, v = _run(shape, 33, w, 64, tokens)
    emb = w["embed"][tokens]
    want = _after_attention(w, emb, res["attn"][0]) - emb
    err = np.linalg.norm(res["hidden"] - emb - want, axis=0)
    # (a column's sums are its terms' root sum of squares or less, the bound is by their size: a factor of 4)
    assert (err <= 4 * REL * (np.linalg.norm(want, axis=0) + np.linalg.norm(emb, axis=0))).all()


@pytest.mark.parametrize("rows,hidden,n_q,n_kv,ffn", [(200, 1024, 8, 4, 3072), (100, 2048, 16, 8, 4096), (33, 4096, 16, 8, 2048)])
def test_rows_are_no_further_from_float64_than_those_of_the_decode_kernels(rows, hidden, n_q, n_kv, ffn):
    import wayruntime_b200 as wr
    shape = dict(n_layers=1, hidden=hidden, n_q_heads=n_q, n_kv_heads=n_kv, head_dim=128, vocab=515, ffn=ffn)
    w = _weights(shape, 1400 + rows)
    tokens = [(29 * r + 3) % shape["vocab"] for r in range(rows)]
    emb = w["embed"][tokens]
    ctx = wr.Context(0)
    dm = _model(ctx, w, shape, max_rows=256)
    err = []
    for portion in (rows, 16):                       # (up to sixteen rows go through the F32 kernels)
        kv, got, attn = ctx.kv_create(1, n_kv, 128, rows), [], []
        for at in range(0, rows, portion):
            res = dm.forward(dm.FWD_PREFILL, [kv], [at], tokens[at:at + portion], hidden=True, attn_tap=True)
            got.append(res["hidden"])
            attn.append(res["attn"][0])
        want = _after_attention(w, emb, np.concatenate(attn))
        err.append(np.linalg.norm(np.concatenate(got) - want) / np.linalg.norm(want - emb))
        kv.close()
    dm.close()
    ctx.close()
    assert err[0] <= err[1], err


def test_weight_rows_of_one_entry_and_of_small_integers():
    """Products of one term and sums of whole multiples: nothing but the result's own rounding, and that of the activations
    to 2^-31 of their row's largest."""
    shape = dict(n_layers=1, hidden=256, n_q_heads=4, n_kv_heads=2, head_dim=128, vocab=64, ffn=256)
    w = _weights(shape, 1305, tied=False)
    w["embed"][:, :128] = 0.0                        # nothing to add the first channels to
    w["l0.w_down"][:128] = 0.0
    wo = w["l0.wo"]
    wo[:128] = 0.0
    for n in range(64):
        wo[n, 5 * n] = (3 + n) * 2.0 ** (n % 9 - 4)
    wo[64:128] = np.random.default_rng(1306).integers(-4, 5, (64, wo.shape[1]))
    tokens = [(5 * r + 1) % 64 for r in range(150)]
    res, _ = _run(shape, 150, w, 256, tokens)
    attn = res["attn"][0].astype(np.float64)
    want = attn @ wo[:128].astype(np.float64).T
    top = np.abs(attn).max(axis=1)[:, None] * np.abs(wo[:128].astype(np.float64)).sum(axis=1)
    assert (np.abs(res["hidden"][:, :128] - want) <= 2.0 ** -24 * np.abs(want) + 2.0 ** -31 * top).all()


def test_factors_far_from_one_do_not_overflow_on_the_way():
    """Feed-forward values near 2^-112 under weights near 2^110: the product is of ordinary size."""
    shape = dict(n_layers=1, hidden=256, n_q_heads=4, n_kv_heads=2, head_dim=128, vocab=64, ffn=512)
    w = _weights(shape, 1307, tied=False)
    w["l0.w_up"] *= np.float32(2.0 ** -112)
    w["l0.w_down"] *= np.float32(2.0 ** 112)
    tokens = [(5 * r + 1) % 64 for r in range(40)]
    res, v = _run(shape, 40, w, 64, tokens)
    _check(res, v, w, tokens)


def test_infinities_are_what_the_decode_kernels_make_of_them():
    """Infinite weights, and infinite feed-forward values: the same results are infinite, with the same sign, or not numbers."""
    import wayruntime_b200 as wr
    shape = dict(n_layers=1, hidden=1024, n_q_heads=16, n_kv_heads=2, head_dim=128, vocab=64, ffn=2052)
    w = _weights(shape, 1308, tied=False)
    down = w["l0.w_down"].copy()
    w["l0.w_down"][5, 2000] = -np.inf                # (sums of K's second part)
    w["l0.w_down"][6, 41] = np.nan
    w["l0.w_down"][700, 5], w["l0.w_down"][700, 1900] = np.inf, -np.inf
    tokens = [(5 * r + 1) % 64 for r in range(48)]
    ctx = wr.Context(0)

    def both():
        dm, out = _model(ctx, w, shape, max_rows=64), []
        for portion in (48, 16):
            kv = ctx.kv_create(1, 2, 128, 48)
            out.append(np.concatenate([dm.forward(dm.FWD_PREFILL, [kv], [at], tokens[at:at + portion], hidden=True)["hidden"]
                                       for at in range(0, 48, portion)]))
            kv.close()
        dm.close()
        kinds = [np.where(np.isnan(o), 2, np.where(np.isinf(o), np.sign(o), 0)) for o in out]
        assert np.array_equal(kinds[0], kinds[1])
        return kinds[0]

    kinds = both()
    assert all((kinds == i).any() for i in (-1, 0, 1, 2))
    w["l0.w_down"] = down
    w["l0.w_up"][43, 7] = np.inf
    kinds = both()
    assert all((kinds == i).any() for i in (-1, 1))
    ctx.close()


def test_a_row_with_an_infinity_ends_not_finite_and_leaves_the_rows_before_it():
    """(The attention kernel masks by a weight of zero, so rows of the same 128-row tile are not finite either.)"""
    shape = dict(n_layers=1, hidden=256, n_q_heads=4, n_kv_heads=2, head_dim=128, vocab=64, ffn=260)
    w = _weights(shape, 1301, tied=False)
    clean = [1 + r % 60 for r in range(150)]
    good, _ = _run(shape, 150, w, 256, clean)
    w["embed"][0, 5] = np.inf
    bad, _ = _run(shape, 150, w, 256, clean[:149] + [0])
    assert not np.isfinite(bad["hidden"][149]).any()
    assert np.array_equal(bad["hidden"][:128], good["hidden"][:128])


def test_a_rows_bits_do_not_depend_on_how_many_follow():
    shape = dict(n_layers=1, hidden=1024, n_q_heads=8, n_kv_heads=4, head_dim=128, vocab=300, ffn=1024)
    w = _weights(shape, 1302)
    tokens = [(7 * r + 1) % 300 for r in range(400)]
    many, _ = _run(shape, 400, w, 512, tokens)
    few, _ = _run(shape, 140, w, 512, tokens[:140])
    assert np.array_equal(many["attn"][0][:128], few["attn"][0][:128])
    assert np.array_equal(many["hidden"][:128], few["hidden"][:128])


def _like_normal(shape, seed, scale):
    """Large weights quickly: a period of normal values that no dimension here divides."""
    n = int(np.prod(shape))
    return np.resize(_gen.normal(seed, (1000003,), scale), n).reshape(shape)


def _run_in_portions(dm, kv, tokens, portion):
    res = [dm.forward(dm.FWD_PREFILL, [kv], [at], tokens[at:at + portion], hidden=True, attn_tap=True)
           for at in range(0, len(tokens), portion)]
    return np.concatenate([r["hidden"] for r in res]), np.concatenate([r["attn"] for r in res], axis=1)


def test_weights_are_split_for_each_call_in_models_too_large_to_keep_them():
    """Split weights are kept when they take a sixteenth of the device's memory or less; here they would take more, and the
    layers use one layer's memory in turn."""
    import torch
    import wayruntime_b200 as wr
    limit = torch.cuda.mem_get_info()[1] // 16
    one = dict(hidden=8192, n_q_heads=2, n_kv_heads=1, head_dim=128, vocab=64, ffn=24576)
    layer = 4 * 8192 * (6 * 128 + 3 * 24576)
    shape = dict(one, n_layers=limit // layer + 1)
    big = {n: _like_normal(s, 1320 + i, s[1] ** -0.5) for i, (n, s) in enumerate(
        dict(w_gate=(24576, 8192), w_up=(24576, 8192), w_down=(8192, 24576), wq=(256, 8192), wk=(128, 8192), wv=(128, 8192), wo=(8192, 256)).items())}
    w = {"embed": _gen.normal(1327, (64, 8192)), "final_norm": np.ones(8192, np.float32)}
    w["lm_head"] = w["embed"]
    for i in range(shape["n_layers"]):
        w.update({f"l{i}.{n}": a for n, a in big.items()})
        w[f"l{i}.wv"], w[f"l{i}.wo"] = big["wv"] * np.float32(2.0 ** (i % 3)), big["wo"] * np.float32(3.0 ** -(i % 3))
        if i % 2:
            w[f"l{i}.w_gate"], w[f"l{i}.w_up"] = big["w_up"], big["w_gate"]
        w.update({f"l{i}.{n}": np.ones(8192, np.float32) for n in ("attn_norm", "ffn_norm")})
    ctx = wr.Context(0)
    dm = _model(ctx, w, shape, max_rows=64)
    assert shape["n_layers"] * layer < dm.device_bytes < (shape["n_layers"] + 2) * layer
    tokens, got = [(7 * r + 1) % 64 for r in range(40)], []
    for portion in (40, 10):
        kv = ctx.kv_create(shape["n_layers"], 1, 128, 40)
        got.append(_run_in_portions(dm, kv, tokens, portion)[0])
        kv.close()
    assert np.abs(got[0] - got[1]).max() <= 2.0 ** -9 * np.abs(got[1]).max()        # (F16 keys and values)
    dm.close()
    ctx.close()


def test_products_that_split_their_weights_in_slices():
    """A feed-forward too wide for the digit sums (its down product takes the F32 kernels): no memory for prompts at all, and every other
    product splits its weights through a workspace that stays small.  q | k | v in two slices, gate and up in five."""
    import torch
    import wayruntime_b200 as wr
    hid, n_q, n_kv, ffn = 4096, 90, 30, 32772
    shape = dict(n_layers=1, hidden=hid, n_q_heads=n_q, n_kv_heads=n_kv, head_dim=128, vocab=64, ffn=ffn)
    w = {f"l0.{n}": _like_normal(s, 1330 + i, s[1] ** -0.5) for i, (n, s) in enumerate(
        dict(w_gate=(ffn, hid), w_up=(ffn, hid), w_down=(hid, ffn), wq=(n_q * 128, hid), wk=(n_kv * 128, hid), wv=(n_kv * 128, hid),
             wo=(hid, n_q * 128)).items())}
    w.update({"embed": _gen.normal(1338, (64, hid)), "final_norm": np.ones(hid, np.float32),
              "l0.attn_norm": 1 + _gen.normal(1339, (hid,), 0.1), "l0.ffn_norm": 1 + _gen.normal(1340, (hid,), 0.1)})
    w["lm_head"] = w["embed"]
    tokens = [(5 * r + 1) % 64 for r in range(24)]
    ctx = wr.Context(0)
    dm = _model(ctx, w, shape, max_rows=64)
    kv = ctx.kv_create(1, n_kv, 128, 24)
    free = torch.cuda.mem_get_info()[0]
    hidden, attn = _run_in_portions(dm, kv, tokens, 24)
    assert free - torch.cuda.mem_get_info()[0] <= 320 << 20
    v = kv.read_rows(0, 1, 0, 24).reshape(24, -1).view(np.float16).astype(np.float64)
    kv.close()
    dm.close()
    ctx.close()
    _check({"hidden": hidden, "attn": attn}, v, w, tokens)


def test_head_columns_in_slices_and_without_the_memory_for_them():
    """Mixed stack in F32, a head of 70003 columns for more rows than a decode batch: two slices through sums of their own.  A context
    without the memory takes the F32 kernels."""
    import torch
    import wayruntime_b200 as wr
    from _tumadra_models import attn, config, weights, with_mlp
    from test_gpu_tumadra import build
    cfg = config([with_mlp(attn(), 64)], width=1024, vocab=70003, groups=4)
    rng = np.random.default_rng(1350)
    w = weights(dict(cfg, vocab=8), 1351)
    w["embed"], w["head"] = _like_normal((70003, 1024), 1352, 1.0), _like_normal((70003, 1024), 1353, 1024 ** -0.5)
    tokens = [int(t) for t in rng.integers(0, 70003, 40)]

    def logits(ctx, m, places):
        kv = m.kv_create(64)
        out = m.forward(m.FWD_PREFILL, [kv], [0], tokens, logits=places)["logits"]
        kv.close()
        return out

    ctx = wr.Context(0)
    m = build(ctx, cfg, w, "float32", max_rows=64)
    few = np.concatenate([logits(ctx, m, list(range(lo, lo + 10))) for lo in range(0, 40, 10)])
    free = torch.cuda.mem_get_info()[0]
    many = logits(ctx, m, list(range(40)))
    assert free - torch.cuda.mem_get_info()[0] <= 320 << 20
    tol = 16 * 2.0 ** -24 * np.linalg.norm(few, axis=1, keepdims=True)
    assert (np.linalg.norm(many - few, axis=1, keepdims=True) <= tol).all()
    m.close()
    ctx.close()
    ctx = wr.Context(0)
    m = build(ctx, cfg, w, "float32", max_rows=64)
    logits(ctx, m, [0])
    torch.cuda.empty_cache()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (96 << 20), dtype=torch.uint8, device="cuda")
    for _ in range(2):
        short = logits(ctx, m, list(range(40)))
        assert (np.linalg.norm(short - few, axis=1, keepdims=True) <= tol).all()
    del hold
    torch.cuda.empty_cache()
    m.close()
    ctx.close()


@pytest.mark.parametrize("qk_norm", [True, False])
def test_prompt_rows_agree_with_those_of_small_portions(qk_norm):
    """The append of a prompt's rows (head norms or none, F16 queries) against the kernels for up to sixteen rows, two layers, a
    portion behind a past.  Keys and values are cut to F16 and queries rounded to it: an F16 step of the largest."""
    import wayruntime_b200 as wr
    ctx = wr.Context(0)
    shape = dict(n_layers=2, hidden=256, n_q_heads=6, n_kv_heads=2, head_dim=128, vocab=300, ffn=512)
    w = _weights(shape, 1310, qk_norm=qk_norm)
    dm = _model(ctx, w, shape, max_rows=256)
    tokens = [(7 * r + 1) % 300 for r in range(230)]
    got = []
    for portions in ([130, 100], [16] * 14 + [6]):
        kv, at, rows = ctx.kv_create(2, 2, 128, 230), 0, []
        for n in portions:
            rows.append(dm.forward(dm.FWD_PREFILL, [kv], [at], tokens[at:at + n], hidden=True)["hidden"])
            at += n
        got.append([np.concatenate(rows)] + [kv.read_rows(i, which, 0, 230).view(np.float16).astype(np.float64)
                                             for i in range(2) for which in range(2)])
        kv.close()
    for a, b in zip(*got):
        assert np.abs(a - b).max() <= 2.0 ** -9 * np.abs(b).max()
    dm.close()
    ctx.close()
