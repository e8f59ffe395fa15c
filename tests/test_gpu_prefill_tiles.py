"""GPU: prompts whose work tiles hold one block of 128 rows (few rows or few heads), two, or pieces of either along the keys.  The
first rows of a long prompt against the same rows as a prompt of their own; odd and even groups, one and many q heads per kv
head, a last block of one row, behind a cache, with a window.

Whole tiles of one and two blocks give a row the same bits (with a window, and behind few keys, none are cut).  Pieces have
reference maxima of their own: probabilities are F16 numbers below 2^8 times the largest, so each is off by at most 2^-11 of
itself either way, and a row of weights that add up to one moves by at most 2 * 2^-11 of the largest value; the sums' own
rounding (F32) is far below that."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hq,hkv,past,window,n,cuts", [
    (32, 8, 0, 0, 1700, (17, 128, 129, 300, 512)), (40, 8, 0, 0, 1700, (17, 300, 513)), (40, 8, 130, 0, 1700, (128, 257, 400)),
    (16, 16, 64, 0, 1700, (100, 385)), (28, 4, 3000, 200, 1700, (17, 513, 900)),
    (64, 2, 1500, 0, 1700, (17, 129, 300)), (16, 8, 6001, 0, 1999, (1, 100, 513, 1300)), (40, 8, 2000, 0, 1999, (128, 257, 700, 1111)),
    (5, 1, 4097, 0, 900, (1, 127, 255, 256, 640)), (8, 1, 777, 0, 2048, (30, 1100))])
def test_rows_of_short_and_long_prompts_agree(hq, hkv, past, window, n, cuts):
    import wayruntime_b200 as wr
    ctx = wr.Context(0, attn_max_seq=8192)
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
        return out

    # float64 over the same F16 rows, a kv head at a time
    k, v = (torch.from_numpy(kv.read_rows(0, which, 0, past + n).reshape(past + n, hkv, 128).view(np.float16)).cuda().double() for which in (0, 1))
    want = torch.empty((n, hq, 128), dtype=torch.float64, device="cuda")
    key, row = torch.arange(past + n, device="cuda")[None], past + torch.arange(n, device="cuda")[:, None]
    hidden = (key > row) | ((key + window <= row) if window else torch.zeros_like(key > row))
    for h in range(hq):
        s = (q[:, h].double() @ k[:, h * hkv // hq].T) / 128 ** 0.5
        want[:, h] = torch.softmax(s.masked_fill(hidden, float("-inf")), 1) @ v[:, h * hkv // hq]
    bound = 2 * 2.0 ** -11 * float(v.abs().max())
    whole = run(n)
    assert float((whole.double() - want).abs().max()) <= bound
    for rows in cuts:
        got = run(rows)
        assert float((got.double() - want[:rows]).abs().max()) <= bound, rows
        if window or past + rows <= 3 * 128:
            assert torch.equal(got.view(torch.int32), whole[:rows].view(torch.int32)), rows
    kv.close()
    ctx.close()
