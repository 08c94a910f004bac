"""How the integer kernels cut their work over the CTAs, where its numbers leave 32 bits and where there are more experts than threads look."""
import numpy as np
import pytest
import torch

from edge0_b200 import moe
from edge0_b200.capi import TYPE_NVFP4, TYPE_Q3_K

pytestmark = pytest.mark.gpu


def matrix(rng, wtype, *shape):
    if wtype == TYPE_NVFP4:
        return moe.quantize_nvfp4(rng.normal(0, 0.02, shape).astype(np.float32))
    w = rng.integers(0, 256, shape[:-1] + (shape[-1] // 256, 110), dtype=np.uint8)
    w[..., 108:110] = rng.normal(0, 1e-3, shape[:-1] + (shape[-1] // 256, 1)).astype(np.float16).view(np.uint8)
    return w.reshape(shape[:-1] + (-1,))


def test_work_beyond_32_bits(gpu_ctx):
    """1300 tokens in 32 groups against 131072 weight rows: 2048 chunks of 5440 units each, times the CTAs.  Every token is one of 13, whose own
    products the kernel made of a hundredth of that work."""
    rng = np.random.default_rng(1)
    K, N = 256, 131072
    w = torch.from_numpy(matrix(rng, TYPE_NVFP4, 1, 1024, K)[0]).cuda().repeat(N // 1024, 1)
    w[:, 1] = torch.arange(N, device="cuda").remainder(97).to(torch.uint8)      # rows of their own: the second block scale
    x = torch.from_numpy(rng.normal(0, 1, (13, K)).astype(np.float32)).cuda()
    gpu_ctx.set_expert_path(1)
    try:
        want = gpu_ctx.mul_mat(TYPE_NVFP4, w, x, K)
        got = gpu_ctx.mul_mat(TYPE_NVFP4, w, x.repeat(100, 1), K)
        gpu_ctx.synchronize()
    finally:
        gpu_ctx.set_expert_path(0)
    assert all(torch.equal(got[13 * i:13 * i + 13], want) for i in range(100))


@pytest.mark.parametrize("wtype,K", [(TYPE_NVFP4, 256), (TYPE_Q3_K, 256), (TYPE_Q3_K, 512)])
@pytest.mark.parametrize("E,T,n_ids", [(1024, 700, 2), (1024, 12000, 2), (640, 5, 4)])
def test_more_experts_than_threads_look(wtype, K, E, T, n_ids, gpu_ctx):
    """Up to 1024 experts with rows, one row to an expert and more; against the kernel of few rows, sixteen at a time."""
    rng = np.random.default_rng(E + T + K)
    N = 24
    w = torch.from_numpy(matrix(rng, wtype, E, N, K)).cuda()
    b = torch.from_numpy(rng.normal(0, 1, (T, 1, K)).astype(np.float32)).cuda()
    ids = torch.from_numpy(np.argsort(rng.random((T, E)), axis=1)[:, :n_ids].astype(np.int32)).cuda()
    got = gpu_ctx.mul_mat_id(wtype, w, b, ids, K)
    at = range(0, T, 16 // n_ids) if T < 1000 else rng.integers(0, T - 16, 200)
    for t in at:
        t = int(t)
        few = gpu_ctx.mul_mat_id(wtype, w, b[t:t + 16 // n_ids].contiguous(), ids[t:t + 16 // n_ids].contiguous(), K)
        assert torch.equal(got[t:t + 16 // n_ids], few), t
    gpu_ctx.synchronize()
