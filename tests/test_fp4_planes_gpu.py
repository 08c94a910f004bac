"""Digit planes and their boxes on the FP4 engine: every number of routed rows a token tile and its four-row boxes can hold, the largest product
of code and significand, blocks far below their row's largest."""
import ctypes as C

import numpy as np
import pytest
import torch

from edge0_b200 import moe
from edge0_b200.capi import TYPE_NVFP4

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_embd,n_ff", [(256, 256), (768, 512), (1024, 768), (2048, 256)])
def test_tiles_boxes_and_largest_digits(n_embd, n_ff, gpu_ctx):
    """`hidden` and the output against the bit-identical engine, within the FP4 engine's fp32 accumulation error (5e-5 of RMS; the output, whose
    re-quantised input may differ in a few last bits of int8, 1e-2 of RMS)."""
    counts = [1, 2, 3, 4, 5, 7, 8, 9, 11, 12, 13, 14, 15, 16, 17, 0, 28, 29]
    rng = np.random.default_rng(n_embd + n_ff)
    E, T = len(counts), sum(counts)
    assert T < 14 * E
    mats = [torch.from_numpy(moe.quantize_nvfp4(rng.normal(0, 0.02, (E, r, c)).astype(np.float32))).cuda()
            for r, c in ((n_ff, n_embd), (n_ff, n_embd), (n_embd, n_ff))]
    layer = moe.MoeLayer(gpu_ctx, wtype=TYPE_NVFP4, top_k=1, router_w=np.zeros((E, n_embd), np.float32), gate=mats[0], up=mats[1], down=mats[2])
    x = rng.normal(0, 1, (T, n_embd)).astype(np.float32)
    x[0::4, :32] = 127 * 2047 * 2.0 ** -11 * rng.choice([-1, 1], 32)        # q = +-127 against a scale of significand 2047: 259969
    x[1::4, 32:64] *= 2.0 ** -16                                            # the smallest power of two a scale holds, and flushed blocks
    x[1::4, 64:96] *= 2.0 ** -30
    x[2::4, 96:128] = 0.0
    x[3] = 0.0
    xd = torch.from_numpy(x).cuda()
    ids = torch.from_numpy(rng.permutation(np.repeat(np.arange(E), counts)).astype(np.int32).reshape(T, 1)).cuda()
    w = torch.ones((T, 1), device="cuda")

    def run(path):
        s, ob = layer._observe(T, xd.device)
        out = torch.empty((T, n_embd), device="cuda")
        gpu_ctx.set_expert_path(path)
        try:
            gpu_ctx.check(gpu_ctx.lib.b200moe_ffn(gpu_ctx.handle, C.byref(layer.desc), xd.data_ptr(), 0, T, ids.data_ptr(), w.data_ptr(), out.data_ptr(),
                                                  C.byref(s), gpu_ctx._stream()))
            gpu_ctx.synchronize()
        finally:
            gpu_ctx.set_expert_path(0)
        return ob.hidden.squeeze(1).double(), out.double()

    (h, o), (h1, o1) = run(6), run(1)
    for got, want, bar in ((h, h1, 5e-5), (o, o1, 1e-2)):
        rms = want.pow(2).mean(dim=1, keepdim=True).sqrt().clamp(min=1e-30)  # of each row: some are large
        assert float(((got - want).abs() / rms)[want.abs().amax(dim=1) > 0].max()) <= bar
        assert bool((got[want.abs().amax(dim=1) == 0] == 0).all())
