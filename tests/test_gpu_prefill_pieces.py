"""GPU: prompt attention whose tiles are cut along the keys: a query row that is not a number is one result row that is not, and no
other row's bits move (the pieces of a tile are put together row by row)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("hq,hkv,past,n", [(40, 8, 6000, 17), (8, 1, 1000, 700), (40, 8, 6001, 1999)])
def test_a_bad_query_row_stays_alone(hq, hkv, past, n, bad):
    import wayruntime_b200 as wr
    ctx = wr.Context(0, attn_max_seq=8192)
    g = torch.Generator(device="cuda").manual_seed(hq + past)
    kv = ctx.kv_create(1, hkv, 128, past + n)
    for which in (0, 1):
        kv.write_rows(0, which, 0, torch.randn((past + n, hkv, 128), generator=g, device="cuda").half())
    q = torch.randn((n, hq, 128), generator=g, device="cuda").half()

    def run():
        out = torch.full((n, hq, 128), 7.0, device="cuda")
        torch.cuda.synchronize()
        ctx.attn_prefill(kv, 0, past, n, q, out, hq)
        ctx.sync()
        return out

    before = ctx.launch_count
    clean = run()
    assert ctx.launch_count - before == 2                # (attention, and the launch that puts pieces together)
    assert torch.isfinite(clean).all()
    for row, head in ((0, 0), (n // 2, hq // 2), (n - 1, hq - 1)):
        kept = q[row, head].clone()
        q[row, head] = bad
        got = run()
        q[row, head] = kept
        assert torch.isnan(got[row, head]).all()
        got[row, head] = clean[row, head]
        assert torch.equal(got.view(torch.int32), clean.view(torch.int32))
    kv.close()
    ctx.close()
