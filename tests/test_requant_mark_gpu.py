"""The marking of values whose rounding is in doubt, one and four rows to a warp: rows around the line and ragged last warps."""
import numpy as np
import pytest
import torch

from edge0_b200 import moe
from edge0_b200.capi import TYPE_NVFP4

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [2364, 2365, 2367, 2370, 4096])     # n_ff 1024: four rows to a warp from 2365 on
def test_marked_values_leave_the_integer_engines_output(T, gpu_ctx):
    """Path 7 (FP4 gate/up, fix-up, integer down) has the bits of path 1 only if every value in doubt was listed once, with its own row."""
    E, n_embd, n_ff = 16, 256, 1024
    rng = np.random.default_rng(T)
    mats = [torch.from_numpy(moe.quantize_nvfp4(rng.normal(0, 0.05, (E, r, c)).astype(np.float32))).cuda()
            for r, c in ((n_ff, n_embd), (n_ff, n_embd), (n_embd, n_ff))]
    layer = moe.MoeLayer(gpu_ctx, wtype=TYPE_NVFP4, top_k=1, router_w=rng.normal(0, 1, (E, n_embd)).astype(np.float32), gate=mats[0], up=mats[1], down=mats[2])
    x = rng.normal(0, 1, (T, n_embd)).astype(np.float32)
    x[T // 2] = 0.0
    xd = torch.from_numpy(x).cuda()
    outs = []
    for path in (1, 7):
        gpu_ctx.set_expert_path(path)
        try:
            outs.append(layer.forward(xd).clone())
            gpu_ctx.synchronize()
        finally:
            gpu_ctx.set_expert_path(0)
    assert torch.equal(outs[0], outs[1])
