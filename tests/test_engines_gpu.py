"""Kernels at the sizes where they can go wrong: edges of tiles, remainders, the ends of the range of a dispatch rule."""
import numpy as np
import pytest
import torch

from edge0_b200 import moe
from edge0_b200.capi import TYPE_NVFP4

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
