"""GPU: the dense stack's products for a decode batch (gemv.cu): a row carries the bits that it has alone.

Rows around the row groups' sizes, widths around what stays in shared memory (eight rows up to 5184 values of K, four
up to 12416, staged in pieces beyond), K with quarters of unequal length, output widths that leave tiles half empty.
One row goes through gemv_splitk_kernel, whose results test_gpu_model_glue.py compares with float64.
"""
import numpy as np
import pytest

from test_gpu_model_glue import _model, _weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,hidden,ffn", [(5, 132, 20), (8, 256, 5184), (9, 260, 5188), (16, 1024, 1540), (13, 516, 12416),
                                             (16, 5188, 36), (11, 128, 12420), (6, 12420, 68)])
def test_batched_rows_carry_the_bits_of_a_row_alone(rows, hidden, ffn):
    import wayruntime_b200 as wr
    ctx = wr.Context(0)
    shape = dict(n_layers=1, hidden=hidden, n_q_heads=2, n_kv_heads=1, head_dim=128, vocab=515, ffn=ffn)
    w = _weights(shape, 1400 + rows)
    dm = _model(ctx, w, shape)
    tokens = [(61 * r + 7) % shape["vocab"] for r in range(rows)]
    kvs = [ctx.kv_create(1, 1, 128, 16) for _ in range(rows + 1)]
    want = [dm.forward(dm.FWD_DECODE, [kvs[rows]], [0], [t], hidden=True, logits=True) for t in tokens]
    got = dm.forward(dm.FWD_DECODE, kvs[:rows], [0] * rows, tokens, hidden=True, logits=True)
    for r in range(rows):
        assert np.array_equal(got["hidden"][r].view(np.uint32), want[r]["hidden"][0].view(np.uint32)), r
        assert np.array_equal(got["logits"][r].view(np.uint32), want[r]["logits"][0].view(np.uint32)), r
    for kv in kvs:
        kv.close()
    dm.close()
    ctx.close()
