"""GPU: the products of a BF16 prompt (gemm_bf16.cu) where their tiles end: rows around one CTA's 128 and a pair's 256, output widths
below one tile, of several, and cut into wide and narrower ones, K-values that leave the last 64 half empty, a strip whose odd rank
has no rows.  One feed-forward (or gated pairs) against the float64 restatement.

Tolerance: what test_gpu_tumadra.py and test_gpu_nurosun.py allow a feed-forward of 16-bit products."""
import pytest

import _nurosun_models as nm
import _plain_nurosun
import _plain_tumadra
import test_gpu_nurosun as tn
import test_gpu_tumadra as tt
from _tumadra_models import config, mamba, tokens, weights, with_mlp

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import wayruntime_b200 as wr
    c = wr.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("width,ff,rows", [(52, 40, (128, 129)), (72, 264, (255, 256, 257)), (520, 1000, (130, 385)),
                                           (136, 8200, (200, 513)), (264, 2600, (2000, 2048))])
def test_feed_forward(ctx, width, ff, rows):
    cfg = config([with_mlp(mamba(inner=8, state=2, dt_rank=1, conv=1), ff)], width=width, groups=4)
    w = weights(cfg, 3)
    w["l0.mix.o"][:] = 0
    toks = tokens(cfg, max(rows), 4)
    want = []
    _plain_tumadra.forward(cfg, w, toks, want)
    m = tt.build(ctx, cfg, w, "bfloat16", max_rows=2048)
    for n in rows:
        kv = m.kv_create(2048)
        got = m.forward(m.FWD_PREFILL, [kv], [0], toks[:n], hidden=True)["hidden"]
        assert tt.rel(got, want[0][:n]) <= tt.TOL["bfloat16"] / 4, n
        kv.close()
    m.close()


@pytest.mark.parametrize("width,ff,rows", [(52, 333, (129, 257)), (200, 4104, (300, 769))])
def test_gated_pairs(ctx, width, ff, rows):
    cfg = nm.config([nm.latent(mlp=nm.dense(ff))], width=width)
    w = nm.weights(cfg, 3)
    tn.silence(w, 0, "mix.o")
    toks = nm.tokens(cfg, max(rows), 4)
    want = []
    _plain_nurosun.forward(cfg, w, toks, want)
    m = tn.build(ctx, cfg, w, "bfloat16", max_rows=1024)
    for n in rows:
        assert tn.rel(tn.residuals(m, cfg, toks[:n], [n], 1)[0], want[0][:n]) <= tn.TOL["bfloat16"] / 2, n
    m.close()
