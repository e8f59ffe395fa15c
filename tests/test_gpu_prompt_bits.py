"""GPU: the bits of prompts through PolyNorm and through the scan's pieces.

The kernels that take many rows spread a row's sums over fewer threads than the ones they stand for and add them up in the
same order.  What they return is pinned by digests of the residual rows, taken from the kernels with 512 threads per row
(PolyNorm) and four states per thread (scan) of commit 87bbae1.  How good the values are is tested elsewhere, against float64.
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
SCAN = {
    (37, 5, (769,), "float32"): "2d72caa72068fbd2",
    (64, 8, (1024,), "float32"): "10fa9cbbacde648b",
    (130, 16, (1109,), "float32"): "076500faad7bb0b1",
    (130, 16, (20, 900), "float32"): "782dff9897688cea",
    (40, 17, (1025,), "float32"): "b70903b1d52bf054",
    (33, 32, (1300,), "float32"): "6f40708509d45e1f",
    (130, 16, (768,), "float32"): "d44f4aed0c0e7532",
    (130, 16, (700,), "float32"): "efa88c36983ac19b",
    (130, 16, (1109,), "bfloat16"): "150f5ac04db58962",
    (8200, 16, (900,), "float32"): "3784130df62c00a0",
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


def scan(inner, state, cuts, dtype):
    return digest_of(with_mlp(mamba(inner=inner, state=state, dt_rank=4, conv=3), 0), 3, 7, dtype, cuts)


@pytest.mark.parametrize("ff", POLY)
def test_polynorm_rows(ff):
    """One to six pieces of eight values per thread, the last of them short."""
    assert poly(ff) == POLY[ff]


@pytest.mark.parametrize("inner,state,cuts,dtype", SCAN)
def test_scan_pieces(inner, state, cuts, dtype):
    """One, two and four threads per channel with eight states each; whole pieces, pieces with a rest, one token in the last
    piece; portions that are not cut; a portion that goes on from a state; more states than a portion is cut for."""
    assert scan(inner, state, cuts, dtype) == SCAN[inner, state, cuts, dtype]
