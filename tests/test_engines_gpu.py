"""Kernels at the sizes where they can go wrong: edges of tiles, remainders, the ends of the range of a dispatch rule."""
import numpy as np
import pytest
import torch

from edge0_b200 import moe
from edge0_b200.capi import TYPE_NVFP4, TYPE_Q3_K

pytestmark = pytest.mark.gpu


def nvfp4_matrix(rng, *shape):
    return torch.from_numpy(moe.quantize_nvfp4(rng.normal(0, 0.02, shape).astype(np.float32))).cuda()


@pytest.mark.parametrize("K,N,T", [(4096, 1024, 256), (1024, 4096, 256), (2048, 2048, 100)])
def test_fp4_dense_product_is_repeatable(K, N, T, gpu_ctx):
    """Every token tile of a dense product reads the same matrix, which comes from L2: the tensor core, not memory, sets the pace, and
    a scale factor that is not in place when its instruction runs shows.  (Copies issued by a thread of their own lost up to one run
    in eight this way: a few features of one token tile off by half an RMS.)  The bar on the values is the FP4 engine's fp32
    accumulation error, 5e-5 of RMS, as for its other tests."""
    rng = np.random.default_rng(K + T)
    w, x = nvfp4_matrix(rng, N, K), torch.from_numpy(rng.normal(0, 1, (T, K)).astype(np.float32)).cuda()
    gpu_ctx.set_expert_path(1)
    try:
        exact = gpu_ctx.mul_mat(TYPE_NVFP4, w, x, K)
    finally:
        gpu_ctx.set_expert_path(0)
    first = gpu_ctx.mul_mat(TYPE_NVFP4, w, x, K)
    assert float((first - exact).abs().max() / exact.pow(2).mean().sqrt()) <= 5e-5
    differ = torch.zeros((), dtype=torch.int64, device="cuda")
    for _ in range(200):
        differ += (gpu_ctx.mul_mat(TYPE_NVFP4, w, x, K) != first).any()
    gpu_ctx.synchronize()
    assert int(differ) == 0


@pytest.mark.parametrize("K,N,counts,ne11", [
    (256, 8, (1, 7, 64, 65), 1), (512, 40, (8, 9, 63, 0), 2), (768, 72, (130, 0, 16, 33), 1), (2048, 64, (64, 129, 2, 31), 1), (2048, 768, (17,), 1)])
def test_q3k_matrix_instruction_keeps_the_bits(K, N, counts, ne11, gpu_ctx, checker):
    """mul_mat_id with `counts` routed rows per expert (edges of the 8-row and 64-row groups, ragged feature tiles, an idle expert):
    against the same rows one token at a time (the integer GEMV), and a sample of them against the reference's dot product.  Codes
    and scales are random bytes, so scale * code meets both ends of its range."""
    rng = np.random.default_rng(K + N)
    E, n_ids = len(counts), 2 if ne11 == 2 else 1
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
