"""Kernels at the sizes where they can go wrong: edges of tiles, remainders, the ends of the range of a dispatch rule."""
import ctypes as C
import re

import numpy as np
import pytest
import torch

from edge0_b200 import moe
from edge0_b200 import workloads as W
from edge0_b200.capi import TYPE_NVFP4, TYPE_Q3_K
from edge0_b200.expert_parallel import SLOT_EXTRA_WORDS

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


@pytest.mark.parametrize("n_embd,n_ff", [(256, 256), (512, 768), (768, 512), (2048, 768)])
def test_q3k_matrix_instruction_gate_up(n_embd, n_ff, gpu_ctx):
    """The gate/up form in a layer with given routing: an expert of three 64-row tiles, ragged ones of 33, 9 and 1 rows and an idle one (one
    super-block to a row at 256 columns: the operand buffers change hands at every unit).  `hidden`, `down` and the output are those of a
    token at a time, on the integer GEMV."""
    counts = (130, 33, 0, 9, 1)
    rng = np.random.default_rng(n_embd + n_ff)
    E, T = len(counts), sum(counts)
    mats = []
    for r, c in ((n_ff, n_embd), (n_ff, n_embd), (n_embd, n_ff)):
        m = rng.integers(0, 256, (E, r, c // 256, 110), dtype=np.uint8)
        m[..., 108:110] = rng.normal(0, 3e-4, (E, r, c // 256, 1)).astype(np.float16).view(np.uint8)
        mats.append(m.reshape(E, r, -1))
    layer = moe.MoeLayer(gpu_ctx, wtype=TYPE_Q3_K, top_k=1, router_w=np.zeros((E, n_embd), np.float32), gate=mats[0], up=mats[1], down=mats[2])
    x = torch.from_numpy(rng.normal(0, 1, (T, n_embd)).astype(np.float32)).cuda()
    ids = torch.from_numpy(rng.permutation(np.repeat(np.arange(E), counts)).astype(np.int32).reshape(T, 1)).cuda()
    w = torch.from_numpy(rng.uniform(0.1, 1, (T, 1)).astype(np.float32)).cuda()

    def run(a, b):
        s, ob = layer._observe(b - a, x.device)
        out = torch.empty((b - a, n_embd), device="cuda")
        gpu_ctx.check(gpu_ctx.lib.b200moe_ffn(gpu_ctx.handle, C.byref(layer.desc), x[a:].data_ptr(), 0, b - a, ids[a:].data_ptr(), w[a:].data_ptr(),
                                              out.data_ptr(), C.byref(s), gpu_ctx._stream()))
        gpu_ctx.synchronize()
        return ob.hidden, ob.down, out

    whole = run(0, T)
    one = [torch.cat(t) for t in zip(*(run(t, t + 1) for t in range(T)))]
    assert bool(torch.isfinite(whole[2]).all()) and all(torch.equal(a, b) for a, b in zip(whole, one))


@pytest.mark.parametrize("T,n_ff,shape", [(96, 256, (512, 8, 2)), (108, 512, (256, 8, 2)), (109, 768, (768, 8, 2)), (433, 256, (512, 8, 2))])
def test_fp4_large_token_tile(T, n_ff, shape, gpu_ctx):
    """From 14 routed rows per expert on the FP4 kernels take tiles of 27 rows (N = 192, two blocks of plane scales): full, ragged and
    one-row tiles.  With the fix-up and the integer down kernel the layer keeps the integer engine's bits; without them `hidden` stays
    within the engine's fp32 accumulation error, 5e-5 of RMS."""
    n_embd, n_expert, top_k = shape
    cfg = W.small_config(TYPE_NVFP4, n_embd=n_embd, n_expert=n_expert, top_k=top_k, n_ff=n_ff, seed=T)
    layer = W.make_layer(cfg).to_device(gpu_ctx)
    x = torch.from_numpy(W.make_tokens(cfg, T)).cuda()
    got = {}
    try:
        for path in (1, 6, 7):
            gpu_ctx.set_expert_path(path)
            out, ob = layer.forward(x, observe=True)
            gpu_ctx.synchronize()
            got[path] = (out.clone(), ob.hidden.clone())
    finally:
        gpu_ctx.set_expert_path(0)
    assert torch.equal(got[7][0], got[1][0])
    want = got[1][1]
    assert float((got[6][1] - want).abs().max() / want.pow(2).mean().sqrt()) <= 5e-5


@pytest.mark.parametrize("T,top_k", [(1, 1), (1, 16), (2, 8), (16, 1), (5, 3)])
@pytest.mark.parametrize("wtype", [TYPE_NVFP4, TYPE_Q3_K])
def test_few_rows_summed_in_the_down_kernel(T, top_k, wtype, gpu_ctx, checker):
    """Up to 16 routed rows the CTA that finishes a token's last row sums them: the reference's bits, repeatedly."""
    cfg = W.small_config(wtype, n_embd=512, n_expert=16, top_k=top_k, n_ff=256, seed=T * 32 + top_k)
    layer = W.make_layer(cfg, quantize_q3k=(lambda w: checker.quantize(TYPE_Q3_K, w)) if wtype == TYPE_Q3_K else None)
    x = W.make_tokens(cfg, T)
    want = checker.moe_layer(x=x, **layer.checker_kwargs()).out
    dl = layer.to_device(gpu_ctx)
    for _ in range(3):
        out = dl.forward(torch.from_numpy(x).cuda())
        gpu_ctx.synchronize()
        assert np.array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("E,top_k", [(8, 2), (40, 4), (200, 8), (512, 10), (1000, 6)])
def test_routing_does_not_depend_on_the_batch(E, top_k, gpu_ctx):
    """Logits, probabilities, choice and weights of a token are the same bits whatever kernel and tile its batch takes (few-token chains,
    16 x 8 and 32 x 16 tiles, ragged edges, one block or several for the grouping), for fp32 and bf16 tokens."""
    rng = np.random.default_rng(E)
    none = np.zeros((E, 256, 144), np.uint8)
    layer = moe.MoeLayer(gpu_ctx, wtype=TYPE_NVFP4, top_k=top_k, router_w=rng.normal(0, 0.05, (E, 256)).astype(np.float32), gate=none, up=none, down=none)
    for dtype in (torch.float32, torch.bfloat16):
        x = torch.from_numpy(rng.normal(0, 1, (1201, 256)).astype(np.float32)).cuda().to(dtype)
        whole = None
        for n in (1201, 1, 2, 9, 17, 33, 130, 300):
            _, ob = layer.forward(x[:n].contiguous(), observe=True)
            gpu_ctx.synchronize()
            now = [ob.logits.clone(), ob.probs.clone(), ob.topk.clone(), ob.weights_norm.clone()]
            whole = whole or now
            assert all(torch.equal(a, b[:n]) for a, b in zip(now, whole)), n


@pytest.mark.parametrize("K", [256, 2048])
def test_block_of_nan_keeps_its_nan(K, gpu_ctx):
    """A block of 32 activations that are all NaN gets a NaN scale (a NaN among numbers is passed over), whether the quantiser takes one
    value or eight values per lane: 16-byte aligned rows against the same rows four bytes further on."""
    rng = np.random.default_rng(K)
    E, N, T = 4, 32, 24
    w = nvfp4_matrix(rng, E, N, K)
    ids = torch.from_numpy(rng.integers(0, E, (T, 1)).astype(np.int32)).cuda()
    flat = torch.from_numpy(rng.normal(0, 1, T * K + 4).astype(np.float32)).cuda()
    got = []
    for off in (0, 1):
        b = flat[off:off + T * K].view(T, 1, K)
        b.copy_(torch.from_numpy(np.random.default_rng(K + 1).normal(0, 1, (T, 1, K)).astype(np.float32)))
        b[3, 0, 32:64] = float("nan")
        b[5, 0, 7] = float("nan")
        got.append(gpu_ctx.mul_mat_id(TYPE_NVFP4, w, b, ids, K))
        gpu_ctx.synchronize()
    assert bool(torch.isnan(got[0][3]).all()) and int(torch.isnan(got[0]).sum()) == N
    assert torch.equal(torch.nan_to_num(got[0], nan=7.0), torch.nan_to_num(got[1], nan=7.0))


@pytest.mark.parametrize("T", [8, 120])     # token tiles of 14 and of 27 rows
@pytest.mark.parametrize("path", [0, 6, 7, 8])
def test_fp4_engine_keeps_what_is_not_finite(T, path, gpu_ctx):
    """An infinite activation, one whose block scale overflows fp16 (above 8.3e6) and a block of NaN have no digits in the planes: those
    tokens' outputs are not finite where the integer engine's are not, and the other tokens' outputs do not change."""
    cfg = W.small_config(TYPE_NVFP4, n_embd=512, n_expert=16, top_k=4, n_ff=256, seed=5)
    layer = W.make_layer(cfg).to_device(gpu_ctx)
    rng = np.random.default_rng(T)
    ids = torch.from_numpy(np.stack([rng.permutation(16)[:4] for _ in range(T)]).astype(np.int32)).cuda()
    w = torch.full((T, 4), 0.25, device="cuda")
    x = torch.from_numpy(W.make_tokens(cfg, T)).cuda()
    bad = x.clone()
    bad[1, 7], bad[3, 100], bad[5, 64:96] = float("inf"), 1e7, float("nan")
    got = {}
    try:
        for p, tokens in ((1, bad), (path, bad), (path, x)):
            gpu_ctx.set_expert_path(p)
            got[p, tokens is bad] = layer.ffn(tokens, ids, w)
            gpu_ctx.synchronize()
    finally:
        gpu_ctx.set_expert_path(0)
    assert not torch.isfinite(got[1, True][[1, 3, 5]]).any()
    assert torch.equal(torch.isfinite(got[path, True]), torch.isfinite(got[1, True]))
    good = [t for t in range(T) if t not in (1, 3, 5)]
    assert torch.equal(got[path, True][good], got[path, False][good])


@pytest.mark.parametrize("T,bar", [(512, 1e-2), (513, 2e-4)])
def test_width_4096_on_both_sides_of_the_fixup(T, bar, gpu_ctx, checker):
    """A plain layer of the widest rows at 4096 routed rows (the last size without the re-quantisation fix-up: the stated bar of the path)
    and beyond it (fix-up, then a tensor-core `down`: 2e-4 of RMS, the bar of its other tests).  Tokens are independent of each other, so
    the first and last few stand for all."""
    cfg = W.small_config(TYPE_NVFP4, n_embd=4096, n_expert=16, top_k=8, n_ff=256, seed=T)
    layer = W.make_layer(cfg)
    x = W.make_tokens(cfg, T)
    out, ob = layer.to_device(gpu_ctx).forward(torch.from_numpy(x).cuda(), observe=True)
    gpu_ctx.synchronize()
    some = [0, 1, 2, T - 3, T - 2, T - 1]
    want = checker.moe_layer(x=x[some], **layer.checker_kwargs())
    for got, ref, limit in ((ob.hidden, want.hidden, 5e-5), (out, want.out, bar)):
        got = got[some].cpu().numpy().astype(np.float64)
        assert np.abs(got - ref).max() / np.sqrt((ref.astype(np.float64) ** 2).mean()) <= limit


@pytest.mark.parametrize("wtype", [TYPE_NVFP4, TYPE_Q3_K])
def test_expert_parallel_kernels_follow_the_rows_that_exist(wtype, gpu_ctx):
    """The owner of 16 of 128 experts receives 8 x 80 slots of which 80 hold a row: five rows per expert, not forty.  The FP4 kernels take the
    tile of few rows and Q3_K the integer GEMV, as they do for 80 rows that come without empty slots; the results are the same bits
    whatever the expected number of rows."""
    cfg = W.small_config(wtype, n_embd=512, n_expert=16, top_k=1, n_ff=256, seed=8)
    rng = np.random.default_rng(8)
    none = np.zeros((16, 512), np.float32)
    if wtype == TYPE_NVFP4:
        mats = [nvfp4_matrix(rng, 16, r, c) for r, c in ((256, 512), (256, 512), (512, 256))]
    else:
        mats = []
        for r, c in ((256, 512), (256, 512), (512, 256)):
            m = rng.integers(0, 256, (16, r, c // 256, 110), dtype=np.uint8)
            m[..., 108:110] = rng.normal(0, 1e-4, (16, r, c // 256, 1)).astype(np.float16).view(np.uint8)
            mats.append(torch.from_numpy(m.reshape(16, r, -1)).cuda())
    layer = moe.MoeLayer(gpu_ctx, wtype=wtype, top_k=1, router_w=none, gate=mats[0], up=mats[1], down=mats[2])
    world, cap = 8, 80
    words = np.zeros((world, cap, cfg.n_embd + SLOT_EXTRA_WORDS), np.float32)
    words[..., :cfg.n_embd] = rng.normal(0, 1, (world, cap, cfg.n_embd))
    ids = np.full((world, cap), -1, np.int32)
    ids[:, :10] = rng.permutation(np.repeat(np.arange(16), 5)).reshape(world, 10)
    words.view(np.int32)[..., cfg.n_embd] = ids
    slots = torch.from_numpy(words.reshape(world * cap, -1).view(np.uint8)).cuda()
    taken = slots[torch.from_numpy(ids.reshape(-1) >= 0).cuda()].contiguous()
    few = "expert_gemm_fp4_kernel.*(14>|Li14E)" if wtype == TYPE_NVFP4 else "expert_gemv_kernel"
    many = "expert_gemm_fp4_kernel.*(27>|Li27E)" if wtype == TYPE_NVFP4 else "expert_mma_q3k_kernel"
    got = {}
    gpu_ctx.set_expert_path(8 if wtype == TYPE_NVFP4 else 0)
    try:
        for name, s, expected, want in (("all", slots, None, many), ("few", slots, cap, few), ("packed", taken, None, few)):
            layer.ep_expert_rows(s, expected_rows=expected)
            gpu_ctx.synchronize()
            with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
                got[name] = layer.ep_expert_rows(s, expected_rows=expected)
                gpu_ctx.synchronize()
            kernels = [e.key for e in prof.key_averages()]
            for pattern in (few, many):
                assert any(re.search(pattern, k) for k in kernels) == (pattern == want), (name, kernels)
    finally:
        gpu_ctx.set_expert_path(0)
    assert torch.equal(got["all"], got["few"])
    assert torch.equal(got["few"][torch.from_numpy(ids.reshape(-1) >= 0).cuda()], got["packed"])


@pytest.mark.parametrize("E,H", [(1200, 64), (4100, 96), (20000, 2112)])    # all warps resident; not; a matrix beyond the L2
def test_f32_product_of_few_tokens(E, H, gpu_ctx):
    """The F32 matmul gives a token the same bits in any batch, and a matrix that many warps share is read once for four tokens, not once
    for each (by the kernel that runs)."""
    gen = torch.Generator(device="cuda").manual_seed(E)
    w, x = torch.randn((E, H), generator=gen, device="cuda"), torch.randn((9, H), generator=gen, device="cuda")

    def product(n):
        d = torch.empty((n, E), device="cuda")
        gpu_ctx.check(gpu_ctx.lib.b200moe_op_mul_mat_f32(gpu_ctx.handle, w.data_ptr(), H, E, x.data_ptr(), n, d.data_ptr(), gpu_ctx._stream()))
        gpu_ctx.synchronize()
        return d

    whole = product(9)
    assert float((whole.double() - x.double() @ w.double().T).abs().max()) <= 1e-6 * H    # 32 chains of H / 32 fp32 steps of size ~1
    for n in (1, 2, 3, 4, 5, 8):
        assert torch.equal(product(n), whole[:n]), n
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        product(8)
    kernels = [e.key for e in prof.key_averages() if "router_logits" in e.key]
    assert kernels and all(bool(re.search("<4|ILi4E", k)) == (E > 1200) for k in kernels), kernels


@pytest.mark.parametrize("K", [256, 2048])      # four passes of 32 weight rows to a stage, and one
@pytest.mark.parametrize("E,N", [(1, 8), (1, 64), (8, 512), (13, 728), (16, 768)])
def test_integer_gemv_leaves_no_weight_row_out(K, E, N, gpu_ctx):
    """A warp that has no weight rows in a pass leaves it out.  From a row or two per CTA over half-filled passes to ragged chunks, the bits
    are those of a token at a time (the one-or-two-token kernel)."""
    T = 30
    rng = np.random.default_rng(E + N)
    w = nvfp4_matrix(rng, E, N, K)
    b = torch.from_numpy(rng.normal(0, 1, (T, 1, K)).astype(np.float32)).cuda()
    ids = torch.from_numpy(np.tile(np.arange(T)[:, None] % E, (1, 2)).astype(np.int32)).cuda()
    got = gpu_ctx.mul_mat_id(TYPE_NVFP4, w, b, ids, K)
    one = torch.cat([gpu_ctx.mul_mat_id(TYPE_NVFP4, w, b[t:t + 1], ids[t:t + 1], K) for t in range(T)])
    gpu_ctx.synchronize()
    assert torch.equal(got, one)
