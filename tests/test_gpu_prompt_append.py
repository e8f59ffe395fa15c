"""GPU: the append kernel of prompts (many tokens or heads, head_dim 128, 16-byte aligned rows) leaves the cache bytes and
rotated rows of the kernel that takes a token at a time, which test_gpu_kv_append.py checks against the oracle: blocks of one, two
and four tokens with remainders, several sessions in one call, heads that leave a thread's batch half full, partial and
no rotation, page borders, both sides of each line between the kernels; rows that are not aligned take the other kernel."""
import numpy as np
import pytest

import _gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_sess,n,hq,hkv,n_rot,rope,first", [
    (1, 64, 4, 4, 0, True, 0), (1, 63, 4, 4, 0, True, 2), (1, 130, 5, 1, 20, True, 61), (3, 200, 10, 2, 0, True, 30), (2, 600, 0, 3, 63, True, 5),
    (16, 5, 8, 8, 0, True, 127), (1, 1201, 16, 8, 1, True, 700), (1, 70, 4, 2, 0, False, 3),
    # 32 heads and more, from 64 tokens; fewer, from 8192 rows of heads or 1536 small CTAs
    (1, 64, 16, 8, 0, True, 0), (1, 63, 16, 8, 0, True, 2), (3, 50, 40, 1, 20, True, 61), (16, 5, 32, 8, 0, True, 127), (1, 130, 36, 2, 0, False, 3),
    (2, 683, 0, 3, 63, True, 5), (1, 1170, 5, 1, 7, True, 0), (1, 1535, 0, 1, 0, True, 3), (1, 1537, 0, 1, 0, True, 3), (1, 768, 2, 1, 64, True, 63)])
@pytest.mark.parametrize("aligned", [True, False])
def test_rows_and_bytes_of_the_token_kernel(n_sess, n, hq, hkv, n_rot, rope, first, aligned):
    import torch
    import wayruntime_b200 as wr
    ctx = wr.Context(0)
    pos = [first + 7 * s for s in range(n_sess)]

    def device(a):
        if aligned:
            return torch.from_numpy(a).cuda()
        t = torch.empty(a.size + 1, device="cuda")
        t[1:] = torch.from_numpy(a.ravel()).cuda()
        return t[1:].view(a.shape)

    k, v = (_gen.normal(1600 + i, (n_sess, n, hkv, 128)) for i in range(2))
    q = _gen.normal(1602, (n_sess, n, hq, 128)) if hq else None
    out = []
    for whole in (True, False):
        kvs = [ctx.kv_create(1, hkv, 128, p + n) for p in pos]
        kd, vd = device(k), device(v)
        qd = device(q) if hq else None
        torch.cuda.synchronize()
        if whole:
            ctx.kv_append(kvs, 0, pos, kd, vd, qd, hq, theta=1e6, n_rot_pairs=n_rot, rope=rope, n_tokens=n)
        else:
            for s in range(n_sess):
                for t in range(n):
                    ctx.kv_append([kvs[s]], 0, [pos[s] + t], kd[s, t], vd[s, t], qd[s, t] if hq else None, hq, theta=1e6,
                                  n_rot_pairs=n_rot, rope=rope)
        ctx.sync()
        out.append([kv.read_rows(0, w, 0, p + n) for kv, p in zip(kvs, pos) for w in (0, 1)] + ([qd.cpu().numpy()] if hq else []))
        for kv in kvs:
            kv.close()
    for a, b in zip(*out):
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
    ctx.close()
