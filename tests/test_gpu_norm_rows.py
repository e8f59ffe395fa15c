"""GPU: the norms of a prompt that take several rows per block, against the float64 restatements: both widths of a thread's share,
groups of one to several warps, blocks whose last rows are missing, the token shift across blocks and from a kept row; and rows
that are not numbers, which must leave the rows before them alone (those behind them see them through mixer and shift).

Tolerances as for one mixer (test_gpu_tumadra.py)."""
import numpy as np
import pytest

import _nurosun_models as nm
import _plain_tumadra as plain
import test_gpu_nurosun as tn
from _tumadra_models import config, mamba, tokens, weights, with_mlp
from test_gpu_tumadra import DTYPES, TOL, build, rel

pytestmark = pytest.mark.gpu

MIXER = mamba(inner=8, state=2, dt_rank=1, conv=1)


@pytest.fixture(scope="module")
def ctx():
    import wayruntime_b200 as wr
    c = wr.Context(0)
    yield c
    c.close()


def rows_of(m, cfg, toks, cuts):
    kv, pos, out = m.kv_create(len(toks)), 0, []
    for n in cuts:
        tap = np.zeros((1, n, cfg["width"]), np.float32)
        m.set_hidden_tap(tap)
        m.forward(m.FWD_PREFILL, [kv], [pos], toks[pos:pos + n], out_from=n)
        out.append(tap[0])
        pos += n
    m.set_hidden_tap(None)
    kv.close()
    return np.concatenate(out)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width,groups", [(64, 2), (1024, 4), (1024, 8), (2048, 1), (2080, 2), (4096, 8)])
def test_groups_and_token_shift(ctx, dtype, width, groups):
    cfg = config([with_mlp(MIXER, 24)], width=width, groups=groups)
    w = weights(cfg, 5)
    size = width // groups
    for g in range(groups):                              # groups of their own size: one that is taken for another shows
        w["embed"][:, g * size:(g + 1) * size] *= 2.0 ** (g % 4)
    toks = tokens(cfg, 77, 6)
    want = []
    plain.forward(cfg, w, toks, want)
    m = build(ctx, cfg, w, dtype)
    for cuts in ([17], [18], [19], [20], [77], [30, 19], [17, 17, 18]):
        n = sum(cuts)
        assert rel(rows_of(m, cfg, toks[:n], cuts), want[0][:n]) <= TOL[dtype], cuts
    m.close()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("width", [1024, 4096])
def test_rows_that_are_not_numbers(ctx, width, bad):
    """Group norm with token shift and PolyNorm (Tumadra), layer norm (Nurosun)."""
    tum = config([with_mlp(MIXER, 2100)], width=width, groups=4)
    nur = nm.config([nm.latent(mlp=nm.dense(40))], width=width)
    for cfg, make, builder in ((tum, weights, build), (nur, nm.weights, tn.build)):
        w = make(cfg, 5)
        w["embed"][7] = bad
        toks = [t if t != 7 else 8 for t in tokens(cfg, 40, 6)]
        m = builder(ctx, cfg, w, "bfloat16")
        clean = rows_of(m, cfg, toks, [40])
        assert np.isfinite(clean).all()
        for at in (1, 2, 3, 20, 39):
            got = rows_of(m, cfg, toks[:at] + [7] + toks[at + 1:], [40])
            assert np.array_equal(got[:at], clean[:at]) and not np.isfinite(got[at]).any(), at
        m.close()
