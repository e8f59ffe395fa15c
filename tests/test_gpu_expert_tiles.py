"""GPU: experts' products of a BF16 prompt at sizes at which rings and accumulators are used again: K-blocks for several rounds of a
ring, more tiles than workers, experts with no row, one row, a tile and one row more, and prompts on both sides of the line
from which tiles have 256 rows (567 rows for 4 experts, one of which a row takes).  One layer against the float64 restatement.

Tolerance: what test_gpu_nurosun.py allows a feed-forward of 16-bit products."""
import numpy as np
import pytest

import _plain_nurosun
import test_gpu_nurosun as tn
from _nurosun_models import config, latent, moe, weights

pytestmark = pytest.mark.gpu

PATTERNS = np.array([[1, 1, 1], [1, -1, -1], [-1, 1, -1], [-1, -1, 1]], np.float32)


@pytest.mark.parametrize("width,ff", [(648, 2056), (2056, 520)])
def test_rows_of_experts(width, ff):
    import wayruntime_b200 as wr
    ctx = wr.Context(0)
    cfg = config([latent(mlp=moe(experts=4, top=1, ff=ff))], width=width, vocab=64)
    w = weights(cfg, 3)
    tn.silence(w, 0, "mix.o")
    rng = np.random.default_rng(4)
    w["embed"][:, :3] = PATTERNS[np.arange(64) % 4]      # token t goes to expert t % 4
    w["l0.mlp.router"][:] = 0
    w["l0.mlp.router"][:, :3] = 4 * PATTERNS
    w["l0.mlp.router.b"][:] = 0
    m = tn.build(ctx, cfg, w, "bfloat16", max_rows=1024)
    for counts in ((257, 1, 0, 308), (257, 1, 0, 309), (0, 256, 513, 130), (17, 0, 0, 1), (1000, 0, 0, 0)):
        toks = [int(4 * rng.integers(0, 16) + e) for e, n in enumerate(counts) for _ in range(n)]
        toks = [toks[i] for i in rng.permutation(len(toks))]
        want = []
        _plain_nurosun.forward(cfg, w, toks, want)
        got = tn.residuals(m, cfg, toks, [len(toks)], 1)[0]
        assert tn.rel(got, want[0]) <= tn.TOL["bfloat16"] / 2, counts
    m.close()
    ctx.close()
