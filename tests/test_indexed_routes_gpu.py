"""Indexed products of a few rows on either side of the line by what they read."""
import numpy as np
import pytest
import torch

from edge0_b200 import moe
from edge0_b200.capi import TYPE_NVFP4, TYPE_Q3_K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wtype,K,N,T", [(TYPE_NVFP4, 4096, 1896, 2), (TYPE_NVFP4, 256, 58264, 1), (TYPE_Q3_K, 768, 14304, 2), (TYPE_Q3_K, 2048, 10432, 2)])
def test_rows_that_read_much_are_grouped(wtype, K, N, T, gpu_ctx):
    """Eight rows to a token, most with an expert to themselves, against the first rows of the matrices, which the kernel of few rows takes."""
    rng = np.random.default_rng(K)
    E, few = 12, 1000
    gen = torch.Generator(device="cuda").manual_seed(K)
    if wtype == TYPE_NVFP4:
        w = torch.from_numpy(moe.quantize_nvfp4(rng.normal(0, 0.02, (1, 64, K)).astype(np.float32))).cuda().repeat(E, N // 64 + 1, 1)[:, :N].contiguous()
        w[..., 8:] = torch.randint(0, 256, w[..., 8:].shape, generator=gen, device="cuda", dtype=torch.uint8)
        w.view(E, N, -1, 36)[..., :4] &= 0x3f                   # block scales below 2
    else:
        w = torch.randint(0, 256, (E, N, K // 256, 110), generator=gen, device="cuda", dtype=torch.uint8)
        w[..., 108:110] = torch.full((1,), 1e-3, dtype=torch.float16, device="cuda").view(torch.uint8)
        w = w.reshape(E, N, -1)
    b = torch.from_numpy(rng.normal(0, 1, (T, 1, K)).astype(np.float32)).cuda()
    ids = torch.from_numpy(np.argsort(rng.random((T, E)), axis=1)[:, :8].astype(np.int32)).cuda()
    part = w[:, :few].contiguous()

    def kernels(experts):
        gpu_ctx.mul_mat_id(wtype, experts, b, ids, K)
        gpu_ctx.synchronize()
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            got = gpu_ctx.mul_mat_id(wtype, experts, b, ids, K)
            gpu_ctx.synchronize()
        return got, any("expert_few_rows" in e.key for e in prof.key_averages())

    whole, whole_few = kernels(w)
    first, first_few = kernels(part)
    assert first_few and not whole_few
    assert bool(torch.isfinite(whole).all()) and torch.equal(whole[..., :few], first)
