"""GPU: prompts whose work tiles hold one block of 128 rows (few rows or few heads) and prompts whose tiles hold two: a row's bits do
not depend on which.  The first rows of a long prompt against the same rows as a prompt of their own; odd and even groups, one and
many q heads per kv head, a last block of one row, behind a cache, with a window."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hq,hkv,past,window", [(32, 8, 0, 0), (40, 8, 0, 0), (40, 8, 130, 0), (16, 16, 64, 0), (28, 4, 0, 200), (64, 2, 700, 0)])
def test_rows_of_short_and_long_prompts_agree(hq, hkv, past, window):
    import wayruntime_b200 as wr
    ctx = wr.Context(0, attn_max_seq=8192)
    n = 1700
    g = torch.Generator(device="cuda").manual_seed(hq + past)
    kv = ctx.kv_create(1, hkv, 128, past + n)
    for which in (0, 1):
        kv.write_rows(0, which, 0, torch.randn((past + n, hkv, 128), generator=g, device="cuda").half())
    q = torch.randn((n, hq, 128), generator=g, device="cuda").half()

    def run(rows):
        out = torch.full((rows, hq, 128), float("nan"), device="cuda")
        torch.cuda.synchronize()
        ctx.attn_prefill(kv, 0, past, rows, q[:rows], out, hq, window=window)
        ctx.sync()
        return out.cpu().numpy().view(np.uint32)

    whole = run(n)
    for rows in (17, 128, 129, 300, 512, 513, 900):
        assert np.array_equal(run(rows), whole[:rows]), rows
    kv.close()
    ctx.close()
