"""GPU: passes repeated by the thousand, none of which may take as long as a wait that ran out.

A lane that is left behind by its warp in a wait finds the phase after the next and sits the wait limit out; results are right and
no error is reported, so only the time shows it.  It took about one in 500 such prompts before waits of whole warps kept their lanes together."""
import time

import pytest

from _nurosun_models import Weights, config, dense, latent, tokens, weights
from _tumadra_models import attn, mamba, with_mlp
from _tumadra_models import config as tumadra_config
from _tumadra_models import weights as tumadra_weights

pytestmark = pytest.mark.gpu

LIMIT = 1_000_000_000        # cycles: half a second at the most a GPU clocks
HEADS = latent(heads=32, dim=128, rot=64, vdim=128, q_rank=64, kv_rank=64, scale=0.07, mlp=dense(64))


@pytest.mark.parametrize("cfg,make,rows,sessions,passes", [
    (config([HEADS], width=256), weights, 2048, 0, 2500),
    (tumadra_config([with_mlp(mamba(inner=256, state=16), 512), with_mlp(attn(heads=32, kv_heads=8, dim=64, vdim=128), 0)], width=256,
                    groups=4), tumadra_weights, 2048, 0, 2500),
    (config([HEADS], width=256), weights, 400, 16, 2500),
], ids=["latent prompt", "differential prompt", "latent steps"])
def test_no_pass_waits_for_a_limit(cfg, make, rows, sessions, passes):
    import wayruntime_b200 as wr
    from wayruntime_b200 import models
    ctx = wr.Context(0)
    ctx.set_wait_limit(LIMIT)
    m = models.build(ctx, cfg, Weights(make(cfg, 3)), "bfloat16", 2048)
    toks = tokens(cfg, rows, 4)
    kvs = [m.kv_create(rows + 1) for _ in range(sessions or 1)]
    for kv in kvs:
        m.forward(m.FWD_PREFILL, [kv], [0], toks, out_from=rows - 1, argmax=True)
    step = ((m.FWD_DECODE, kvs, [rows] * sessions, toks[:sessions], 0) if sessions else (m.FWD_PREFILL, kvs, [0], toks, rows - 1))
    slowest = 0.0
    for i in range(passes):
        begin = time.perf_counter()
        m.forward(*step[:4], out_from=step[4], argmax=True)
        if i:                                            # (the first one loads its kernels)
            slowest = max(slowest, time.perf_counter() - begin)
    for kv in kvs:
        kv.close()
    m.close()
    ctx.close()
    assert slowest < 0.4
