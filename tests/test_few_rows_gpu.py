"""The kernel of one or two tokens: every weight row of ragged chunks against the reference's dot product, and layers whose launches overlap."""
import numpy as np
import pytest
import torch

from edge0_b200 import moe
from edge0_b200 import workloads as W
from edge0_b200.capi import TYPE_NVFP4, TYPE_Q3_K

pytestmark = pytest.mark.gpu


def matrix(rng, wtype, *shape):
    if wtype == TYPE_NVFP4:
        w = moe.quantize_nvfp4(rng.normal(0, 0.02, shape).astype(np.float32))
        w[0, 0, 0] = 0x7f                                       # decodes to zero
        return w
    w = rng.integers(0, 256, shape[:-1] + (shape[-1] // 256, 110), dtype=np.uint8)
    w[..., 108:110] = rng.normal(0, 1e-3, shape[:-1] + (shape[-1] // 256, 1)).astype(np.float16).view(np.uint8)
    return w.reshape(shape[:-1] + (-1,))


@pytest.mark.parametrize("wtype,K", [(TYPE_NVFP4, k) for k in (256, 512, 768, 1024, 2048, 4096)] + [(TYPE_Q3_K, k) for k in (256, 512, 768, 2048)])
@pytest.mark.parametrize("N,T,n_ids,ne11", [(8, 1, 1, 1), (40, 2, 3, 1), (264, 2, 2, 2)])
def test_rows_are_the_references(wtype, K, N, T, n_ids, ne11, gpu_ctx, checker):
    """mul_mat_id with ids that are a slice of a wider tensor, an expert that two tokens share and one that a token names twice."""
    rng = np.random.default_rng(K + N)
    E = 9
    w = matrix(rng, wtype, E, N, K)
    b = rng.normal(0, 1, (T, ne11, K)).astype(np.float32)
    b[0, 0, :32] = 0.0
    wide = rng.integers(0, E, (T, n_ids + 3)).astype(np.int32)
    wide[:, 0] = 5
    wide[-1, n_ids - 1] = 5
    got = gpu_ctx.mul_mat_id(wtype, torch.from_numpy(w).cuda(), torch.from_numpy(b).cuda(), torch.from_numpy(wide).cuda()[:, :n_ids], K)
    gpu_ctx.synchronize()
    for t in range(T):
        for s in range(n_ids):
            aq = checker.quantize_activation(wtype, b[t, s % ne11])
            want = [checker.vec_dot(wtype, K, w[wide[t, s], r], aq) for r in range(N)]
            assert np.array_equal(got[t, s].cpu().numpy(), np.array(want, np.float32)), (t, s)


@pytest.mark.parametrize("wtype", [TYPE_NVFP4, TYPE_Q3_K])
@pytest.mark.parametrize("K,N", [(256, 40), (768, 512), (2048, 1032)])
def test_dense_products_of_few_tokens(wtype, K, N, gpu_ctx, checker):
    """A token at a time up to the line, passes of the grouped kernel beyond it: the same bits."""
    rng = np.random.default_rng(K + N)
    w = matrix(rng, wtype, 1, N, K)[0]
    x = torch.from_numpy(rng.normal(0, 1, (6, K)).astype(np.float32)).cuda()
    dw = torch.from_numpy(w).cuda()
    gpu_ctx.set_expert_path(1)
    try:
        whole = gpu_ctx.mul_mat(wtype, dw, x, K)
        for n in (1, 2, 3, 4, 5):
            assert torch.equal(gpu_ctx.mul_mat(wtype, dw, x[:n].contiguous(), K), whole[:n]), n
    finally:
        gpu_ctx.set_expert_path(0)
    gpu_ctx.synchronize()
    aq = checker.quantize_activation(wtype, x[0].cpu().numpy())
    for r in (0, N - 1):
        assert float(whole[0, r]) == checker.vec_dot(wtype, K, w[r], aq)


@pytest.mark.parametrize("wtype", [TYPE_NVFP4, TYPE_Q3_K])
def test_tokens_share_a_large_matrix(wtype, gpu_ctx):
    """A dense product of a few tokens reads a matrix for each of them only while that is less than a pass of the grouped kernel (by the
    launches); the bits are the same on either side of the line."""
    K, row = 256, 144 if wtype == TYPE_NVFP4 else 110
    x = torch.randn((6, K), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    for T, line in ((1, 64 << 20), (3, 24 << 20)):
        N = line // (T * row) // 8 * 8
        w = torch.from_numpy(matrix(np.random.default_rng(T), wtype, 1, 512, K)[0]).cuda().repeat((N + 8 + 511) // 512, 1)
        gpu_ctx.set_expert_path(1)
        try:
            whole = gpu_ctx.mul_mat(wtype, w[:N + 8], x, K)
        finally:
            gpu_ctx.set_expert_path(0)
        for n, few in ((N, True), (N + 8, False)):
            before = gpu_ctx.launches()
            got = gpu_ctx.mul_mat(wtype, w[:n], x[:T].contiguous(), K)
            assert gpu_ctx.launches() - before == (1 if few else 3), (T, n)      # or: quantiser, groups, product
            assert torch.equal(got, whole[:T, :n]), (T, n)


@pytest.mark.parametrize("wtype", [TYPE_NVFP4, TYPE_Q3_K])
def test_rows_share_large_experts(wtype, gpu_ctx):
    """The same of indexed products of which each expert has several rows."""
    K, row, E = 256, 144 if wtype == TYPE_NVFP4 else 110, 4
    b = torch.randn((8, 1, K), generator=torch.Generator(device="cuda").manual_seed(2), device="cuda")
    N = (40 << 20) // (8 * row) // 8 * 8
    w = torch.from_numpy(matrix(np.random.default_rng(5), wtype, E, 512, K)).cuda().repeat(1, (N + 8 + 511) // 512, 1)
    for n, T, few in ((N, 8, True), (N + 8, 8, False), (N + 8, 7, True)):
        ids = (torch.arange(T, device="cuda") % E).reshape(T, 1).to(torch.int32)
        mats = w[:, :n].contiguous()
        before = gpu_ctx.launches()
        got = gpu_ctx.mul_mat_id(wtype, mats, b[:T].contiguous(), ids, K)
        assert gpu_ctx.launches() - before == (2 if few else 4), (n, T)       # quantiser, product, or counts and groups in between
        for t in range(T):
            assert torch.equal(got[t], gpu_ctx.mul_mat_id(wtype, mats, b[t:t + 1], ids[t:t + 1], K)[0]), (n, T, t)


def test_an_expert_that_does_not_exist_is_reported(gpu_ctx):
    rng = np.random.default_rng(1)
    w = torch.from_numpy(matrix(rng, TYPE_NVFP4, 9, 8, 256)).cuda()
    b = torch.zeros((1, 1, 256), device="cuda")
    gpu_ctx.mul_mat_id(TYPE_NVFP4, w, b, torch.tensor([[9, 0]], dtype=torch.int32, device="cuda"), 256)
    with pytest.raises(moe.B200MoeError):
        gpu_ctx.synchronize()
    gpu_ctx.mul_mat_id(TYPE_NVFP4, w, b, torch.tensor([[8, 0]], dtype=torch.int32, device="cuda"), 256)
    gpu_ctx.synchronize()


@pytest.mark.parametrize("wtype,T,shape", [(TYPE_NVFP4, 1, {}), (TYPE_Q3_K, 2, {}), (TYPE_NVFP4, 3, dict(n_latent=256)), (TYPE_NVFP4, 9, dict(n_ff_shexp=256)),
                                           (TYPE_Q3_K, 20, {}), (TYPE_NVFP4, 40, {})])
def test_overlapped_launches_keep_the_bits(wtype, T, shape, gpu_ctx):
    """Layers one behind the other, called one by one and replayed from a graph, against launches in series."""
    cfg = W.small_config(wtype, n_embd=512, n_expert=32, top_k=4, n_ff=256, seed=T, **shape)
    layers = [W.make_layer(cfg).to_device(gpu_ctx) for _ in range(2)]
    xs = [torch.from_numpy(W.make_tokens(cfg, T)).cuda() * (i + 1) for i in range(3)]
    outs = [torch.empty((T, 512), device="cuda") for _ in range(6)]

    def step():
        for i, o in enumerate(outs):
            layers[i % 2].forward(xs[i % 3], out=o)

    def bits():
        gpu_ctx.synchronize()
        return [o.clone() for o in outs]

    fresh = moe.Context(0)
    fresh.set_launch_overlap(False)
    serial = [W.make_layer(cfg).to_device(fresh).forward(x) for x in xs]
    fresh.synchronize()
    want = [serial[i % 3] for i in range(6)]
    for _ in range(30):
        step()
    got = bits()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    for o in outs:
        o.zero_()
    for _ in range(10):
        graph.replay()
    assert all(torch.equal(a, b) for a, b in zip(bits(), want))
