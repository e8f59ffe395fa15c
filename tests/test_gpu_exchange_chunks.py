"""GPU: key shards of 129 to 256 keys go through merge warps, which receive the other ranks' rows and finish the output: a fused
step is one launch, and gives the bits of partial rows put together by a launch of their own."""
import numpy as np
import pytest

import _gen
from _cuda_util import make_cache, port

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [[129], [200, 256, 193], [256, 3000, 129, 192]])
@pytest.mark.parametrize("hq,hkv", [(8, 2), (8, 1), (16, 8)])
def test_short_shards_are_received_in_the_kernel(lens, hq, hkv):
    import torch
    import wayruntime_b200 as wr
    ctx, P, hd = wr.Context(0), port(), 128
    kvs = [make_cache(ctx, *(P.f32_to_f16(_gen.normal(700 + 10 * i + w, (n, hkv, hd))) for w in (0, 1))) for i, n in enumerate(lens)]
    rows = len(lens) * hq
    q = torch.from_numpy(_gen.normal(900, (len(lens), hq, hd))).cuda()
    triples = torch.empty((rows, wr.TRIPLE_PAD + hd), dtype=torch.float32, device="cuda")
    want = torch.empty((rows, hd), dtype=torch.float32, device="cuda")
    ctx.attn_decode_partial(kvs, 0, lens, q, triples, hq)
    ctx.attn_combine(1, rows, hd, triples, want)
    x = wr.Exchange(ctx, 1, 0, rows, hd)
    got = torch.full((len(lens), hq, hd), float("nan"), dtype=torch.float32, device="cuda")
    before = ctx.launch_count
    x.decode(kvs, 0, lens, q, got, hq)
    launched = ctx.launch_count - before
    ctx.sync()
    assert torch.equal(got.view(rows, hd), want)
    assert np.isfinite(want.cpu().numpy()).all()
    assert launched == 1
    x.close()
    for kv in kvs:
        kv.close()
    ctx.close()
