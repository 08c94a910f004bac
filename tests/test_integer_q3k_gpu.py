"""The Q3_K kernel of few routed rows per expert at the edges of its passes (16 routed rows, eight to a group) and tiles (16 weight rows)."""
import numpy as np
import pytest
import torch

from edge0_b200.capi import TYPE_Q3_K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [256, 512, 768, 2048])
@pytest.mark.parametrize("N,counts,ne11", [(8, (17, 1, 0), 1), (40, (1, 7, 8, 9, 0, 2, 16, 17, 33, 3), 1), (264, (20, 3), 2), (1032, (2, 18), 1)])
def test_passes_and_tiles_keep_the_bits(K, N, counts, ne11, gpu_ctx, checker):
    """`counts` routed rows per expert, fewer than twelve on average, against the same rows one token at a time (the one-or-two-token
    kernel), and a sample of them against the reference's dot product.  Random bytes: scale * code meets both ends of its range."""
    rng = np.random.default_rng(K + N)
    E, n_ids = len(counts), ne11
    assert sum(counts) < 12 * E
    w = rng.integers(0, 256, (E, N, K // 256, 110), dtype=np.uint8)
    w[..., 108:110] = rng.normal(0, 1e-3, (E, N, K // 256, 1)).astype(np.float16).view(np.uint8)
    w[:, ::3, :, 96:108] = 0                                    # scales of -32 against codes of -4
    w[:, ::3, :, 0:32] = 0
    w = w.reshape(E, N, -1)
    rows = rng.permutation(np.repeat(np.arange(E), counts)).astype(np.int32)
    rows = rows[:len(rows) // n_ids * n_ids].reshape(-1, n_ids)
    b = rng.normal(0, 1, (len(rows), ne11, K)).astype(np.float32)
    b[0, 0, :256] = 0.0
    dw, db, ids = torch.from_numpy(w).cuda(), torch.from_numpy(b).cuda(), torch.from_numpy(rows).cuda()
    got = gpu_ctx.mul_mat_id(TYPE_Q3_K, dw, db, ids, K)
    one = torch.cat([gpu_ctx.mul_mat_id(TYPE_Q3_K, dw, db[t:t + 1], ids[t:t + 1], K) for t in range(len(rows))])
    gpu_ctx.synchronize()
    assert torch.equal(got, one)
    for t in rng.integers(0, len(rows), 6):
        aq = checker.quantize_activation(TYPE_Q3_K, b[t, 0])
        r = int(rng.integers(0, N))
        assert float(got[t, 0, r]) == checker.vec_dot(TYPE_Q3_K, K, w[rows[t, 0], r], aq)
