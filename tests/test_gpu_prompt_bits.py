"""GPU: the bits of prompts through PolyNorm.

The kernel that takes many rows spreads a row's sums over fewer threads than the one it stands for and adds them up in the
same order.  What it returns is pinned by digests of the residual rows, taken from the kernel with 512 threads per row of
commit 87bbae1.  How good the values are is tested elsewhere, against float64.
"""
import hashlib

import numpy as np
import pytest

from _tumadra_models import config, mamba, tokens, weights, with_mlp
from test_gpu_tumadra import build

pytestmark = pytest.mark.gpu

POLY = {
    333: "c0606011513c4a22",
    2048: "eadaadc1f087ad9f",
    2049: "1a442945a80d0eb5",
    4000: "ec7b0f84bbb8d8a2",
    4099: "ecd4ff6f1c229971",
    6144: "58d9b87e23e8712d",
    9000: "4ac19c2fc7c31215",
    12288: "46ed0570772d900a",
}


def digest_of(layer, groups, seed, dtype, cuts, zero=()):
    """Of all residual rows behind the one layer, the prompt in portions of `cuts` rows."""
    import wayruntime_b200 as wr
    ctx = wr.Context(0)
    cfg = config([layer], width=48, groups=groups)
    w = weights(cfg, seed)
    for name in zero:
        w[name][:] = 0
    toks = tokens(cfg, sum(cuts), seed + 1)
    m = build(ctx, cfg, w, dtype, max_rows=2048)
    kv, pos, h = m.kv_create(len(toks)), 0, hashlib.sha256()
    for n in cuts:
        tap = np.zeros((1, n, cfg["width"]), np.float32)
        m.set_hidden_tap(tap)
        m.forward(m.FWD_PREFILL, [kv], [pos], toks[pos:pos + n], out_from=n)
        h.update(tap.tobytes())
        pos += n
    m.set_hidden_tap(None)
    kv.close()
    m.close()
    ctx.close()
    return h.hexdigest()[:16]


def poly(ff):
    return digest_of(with_mlp(mamba(inner=8, state=2, dt_rank=1, conv=1), ff), 4, 3, "bfloat16", [500], ["l0.mix.o"])


@pytest.mark.parametrize("ff", POLY)
def test_polynorm_rows(ff):
    """One to six pieces of eight values per thread, the last of them short."""
    assert poly(ff) == POLY[ff]
