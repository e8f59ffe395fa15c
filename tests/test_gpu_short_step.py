"""GPU: the one-kernel attention step (attn_step_small.cu) around the session lengths at which its work is divided anew
(256 and 512 keys, 1024 is its last), for every number of q heads per kv head that it is built for.

A batch's rows carry the bits of each session alone, and agree with the norm / append / split-KV kernels, which
test_gpu_decode.py checks against the oracle: both sum at most 1025 products of weights and F16 values in F32
(2^-23 each, at random signs: 32 * 2^-23), and that path's weights are two F16 numbers (2^-22).
"""
import numpy as np
import pytest

from test_gpu_model_glue import _model, _prefill, _weights

pytestmark = pytest.mark.gpu
TOL = (32 * 2.0 ** -23 + 2.0 ** -22) * 4          # (values up to 4)


@pytest.mark.parametrize("n_q,n_kv", [(2, 2), (4, 2), (3, 1), (8, 2), (8, 1)])
def test_lengths_around_the_divisions(monkeypatch, n_q, n_kv):
    import wayruntime_b200 as wr
    ctx = wr.Context(0)
    shape = dict(n_layers=1, hidden=256, n_q_heads=n_q, n_kv_heads=n_kv, head_dim=128, vocab=515, ffn=128)
    w = _weights(shape, 1500 + n_q)
    dm = _model(ctx, w, shape, max_rows=256)
    lens = [0, 254, 255, 256, 300, 511, 512, 700, 1022, 1023, 1024]
    toks = [(31 * i + 7) % shape["vocab"] for i in range(len(lens))]

    def sessions():
        kvs = [ctx.kv_create(1, n_kv, 128, 1100) for _ in lens]
        for kv, n in zip(kvs, lens):
            if n:
                _prefill(dm, kv, [(11 * i + n) % shape["vocab"] for i in range(n)], chunk=256)
        return kvs

    a, b, c = sessions(), sessions(), sessions()
    alone = [dm.forward(dm.FWD_DECODE, [kv], [n], [t], logits=True, attn_tap=True) for kv, n, t in zip(a, lens, toks)]
    batch = dm.forward(dm.FWD_DECODE, b, lens, toks, logits=True, attn_tap=True)
    monkeypatch.setenv("WR_CUDA_STEP_SMALL_OFF", "1")
    other = dm.forward(dm.FWD_DECODE, c, lens, toks, attn_tap=True)
    for i, n in enumerate(lens):
        assert np.array_equal(batch["logits"][i].view(np.uint32), alone[i]["logits"][0].view(np.uint32)), n
        assert np.array_equal(batch["attn"][0][i].view(np.uint32), alone[i]["attn"][0][0].view(np.uint32)), n
        assert np.abs(batch["attn"][0][i] - other["attn"][0][i]).max() <= TOL, n
    for kv in a + b + c:
        kv.close()
    dm.close()
    ctx.close()


@pytest.mark.parametrize("qk_norm", [True, False])
def test_short_and_long_sessions_in_one_batch_over_three_layers(qk_norm):
    """Two streams per layer that meet before the next product: every step of every session has the bits it has alone."""
    import wayruntime_b200 as wr
    ctx = wr.Context(0)
    shape = dict(n_layers=3, hidden=256, n_q_heads=8, n_kv_heads=4, head_dim=128, vocab=515, ffn=128)
    w = _weights(shape, 1520, qk_norm=qk_norm)
    dm = _model(ctx, w, shape, max_rows=1024)
    lens = [60, 1500, 300, 2100, 1022, 1023, 1024, 5, 3000, 700]
    steps = 4                                        # (1022 and 1023 go from one kind to the other on the way)

    def sessions():
        kvs = [ctx.kv_create(3, 4, 128, n + steps) for n in lens]
        for kv, n in zip(kvs, lens):
            _prefill(dm, kv, [(11 * i + n) % shape["vocab"] for i in range(n)], chunk=1024)
        return kvs

    a, b = sessions(), sessions()
    for t in range(steps):
        pos, toks = [n + t for n in lens], [(31 * i + 7 * t) % shape["vocab"] for i in range(len(lens))]
        alone = [dm.forward(dm.FWD_DECODE, [kv], [p], [x], logits=True, attn_tap=True) for kv, p, x in zip(a, pos, toks)]
        batch = dm.forward(dm.FWD_DECODE, b, pos, toks, logits=True, attn_tap=True)
        for i, n in enumerate(lens):
            assert np.array_equal(batch["attn"][:, i].view(np.uint32), alone[i]["attn"][:, 0].view(np.uint32)), (t, n)
            assert np.array_equal(batch["logits"][i].view(np.uint32), alone[i]["logits"][0].view(np.uint32)), (t, n)
    for x, y in zip(a, b):
        n = lens[a.index(x)] + steps
        for layer in range(3):
            for which in (0, 1):
                assert np.array_equal(x.read_rows(layer, which, 0, n), y.read_rows(layer, which, 0, n))
    for kv in a + b:
        kv.close()
    dm.close()
    ctx.close()
