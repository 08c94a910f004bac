"""The NVFP4 integer kernel at the edges of its items: passes of one, two, three and four routed rows, ragged chunks of weight rows."""
import numpy as np
import pytest
import torch

from edge0_b200 import moe
from edge0_b200.capi import TYPE_NVFP4

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [256, 768, 2048, 4096])
@pytest.mark.parametrize("N,counts,ne11", [(8, (17, 0, 1), 1), (72, (1, 2, 3, 4, 5, 6, 7, 8, 9, 0, 33), 1), (264, (130, 3), 2), (1032, (2, 40), 1)])
def test_passes_and_chunks_keep_the_bits(K, N, counts, ne11, gpu_ctx, checker):
    """`counts` routed rows per expert against the same rows one token at a time (the one-or-two-token kernel), and a sample of them against
    the reference's dot product.  A block of zeros and a block scale of 0x7f (which decodes to zero) are among the operands."""
    rng = np.random.default_rng(K + N)
    E, n_ids = len(counts), ne11
    w = moe.quantize_nvfp4(rng.normal(0, 0.02, (E, N, K)).astype(np.float32))
    w[0, 0, 0] = 0x7f
    rows = rng.permutation(np.repeat(np.arange(E), counts)).astype(np.int32)
    rows = rows[:len(rows) // n_ids * n_ids].reshape(-1, n_ids)
    b = rng.normal(0, 1, (len(rows), ne11, K)).astype(np.float32)
    b[0, 0, :64] = 0.0
    dw, db, ids = torch.from_numpy(w).cuda(), torch.from_numpy(b).cuda(), torch.from_numpy(rows).cuda()
    got = gpu_ctx.mul_mat_id(TYPE_NVFP4, dw, db, ids, K)
    one = torch.cat([gpu_ctx.mul_mat_id(TYPE_NVFP4, dw, db[t:t + 1], ids[t:t + 1], K) for t in range(len(rows))])
    gpu_ctx.synchronize()
    assert torch.equal(got, one)
    for t in rng.integers(0, len(rows), 6):
        aq = checker.quantize_activation(TYPE_NVFP4, b[t, 0])
        r = int(rng.integers(0, N))
        assert float(got[t, 0, r]) == checker.vec_dot(TYPE_NVFP4, K, w[rows[t, 0], r], aq)
