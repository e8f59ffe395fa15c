"""GPU: selective scan of portions of some hundred tokens that are not cut into pieces: two states per thread, one state per thread,
and portions that go on from a state, against the float64 restatement.  Tolerances as for the mixer alone (test_gpu_tumadra.py)."""
import numpy as np
import pytest

import _plain_tumadra as plain
from _tumadra_models import config, mamba, tokens, weights, with_mlp
from test_gpu_tumadra import DTYPES, TOL, build, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("inner,state", [(8200, 16), (16392, 8), (300, 24)])
def test_portions_around_the_line(dtype, inner, state):
    import wayruntime_b200 as wr
    ctx = wr.Context(0)
    cfg = config([with_mlp(mamba(inner=inner, state=state, dt_rank=4, conv=3), 0)], width=48, groups=3)
    w = weights(cfg, 11)
    toks = tokens(cfg, 700, 12)
    want = []
    plain.forward(cfg, w, toks, want)
    m = build(ctx, cfg, w, dtype, max_rows=1024)
    for cuts in ([700], [640, 60], [58, 641, 1]):
        kv, pos = m.kv_create(800), 0
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
