"""GPU: selective scan of portions that are cut into pieces (more than 768 tokens here), against the float64 restatement:
state sizes around those that two, four and eight threads hold, pieces with remainders, a portion that goes on from a
state, and the decode step behind it.  Tolerances as for the mixer alone (test_gpu_tumadra.py)."""
import numpy as np
import pytest

import _plain_tumadra as plain
from _tumadra_models import config, mamba, tokens, weights, with_mlp
from test_gpu_tumadra import DTYPES, TOL, build, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("inner,state", [(37, 5), (64, 8), (130, 16), (40, 17), (33, 32)])
def test_portions_of_several_pieces(dtype, inner, state):
    import wayruntime_b200 as wr
    ctx = wr.Context(0)
    cfg = config([with_mlp(mamba(inner=inner, state=state, dt_rank=4, conv=3), 0)], width=48, groups=3)
    w = weights(cfg, 7)
    toks = tokens(cfg, 1110, 8)
    want = []
    plain.forward(cfg, w, toks, want)
    m = build(ctx, cfg, w, dtype, max_rows=2048)
    for cuts in ([1109, 1], [513, 596, 1], [300, 768, 41, 1], [300, 769, 40, 1], [20, 1089, 1]):
        kv, pos = m.kv_create(1200), 0
        for n in cuts:
            tap = np.zeros((1, n, 48), np.float32)
            m.set_hidden_tap(tap)
            m.forward(m.FWD_PREFILL if n > 1 else m.FWD_DECODE, [kv], [pos], toks[pos:pos + n], out_from=n)
            assert rel(tap[0], want[0][pos:pos + n]) <= TOL[dtype], (cuts, pos)
            pos += n
        m.set_hidden_tap(None)
        kv.close()
    m.close()
    ctx.close()
