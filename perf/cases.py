"""The calls whose speed matters to a user of this library, with inputs, required work and tolerances.

Every case goes through edge0_b200's public entry points: MoeLayer.forward / forward_host (router, experts, combine), the
expert-parallel step on one rank, and the indexed matmul Context.mul_mat_id.  `kind`:
  layer   plain MoE FFN layer on device tensors     host    the same through pinned host buffers, waiting for the result
  latent  layer with the shared latent projections  ep      the expert-parallel latent step, one rank
  mmid    one ggml_mul_mat_id with a gate-shaped expert tensor
`layers` layers with weights of their own run one after the other in a pass (a decode step walks a stack of layers, so that a
layer's weights are not in cache when it is reached); `graph` replays them from a CUDA graph captured in prepare().
"""
import math

import torch

from edge0_b200 import moe
from edge0_b200 import workloads as W
from edge0_b200.capi import TYPE_NVFP4, TYPE_Q3_K
from edge0_b200.expert_parallel import CudaBackend, ExpertParallelLayer

DEV = torch.device("cuda", 0)
WTYPE = {"nvfp4": TYPE_NVFP4, "q3_k": TYPE_Q3_K}

_PLAIN = dict(n_embd=2048, n_latent=0, n_expert=128, top_k=8, n_ff=768, n_ff_shexp=0, bias=False, layers=1, graph=False)
_LATENT = dict(n_embd=4096, n_latent=1024, n_expert=512, top_k=10, n_ff=1024, n_ff_shexp=0, bias=False, layers=1, graph=False)


def _case(base, kind, wtype, tokens, x, **more):
    return dict(base, kind=kind, wtype=wtype, tokens=tokens, x=x, **more)


def listed():
    return [
        # one sequence, one token: four layers of a decode step called one by one, as a graph executor does
        _case(_PLAIN, "layer", "q3_k", 1, "f32", layers=4, name="q3k_decode_1"),
        # the same from a captured CUDA graph, as a serving loop does
        _case(_PLAIN, "layer", "nvfp4", 1, "bf16", layers=4, graph=True, name="nvfp4_decode_1"),
        # a few sequences, tensors on the host
        _case(_PLAIN, "host", "nvfp4", 8, "bf16", name="nvfp4_host_8"),
        # batched decode
        _case(_PLAIN, "layer", "nvfp4", 64, "bf16", name="nvfp4_decode_64"),
        _case(_PLAIN, "layer", "q3_k", 32, "f32", name="q3k_decode_32"),
        # a layer with a shared expert and its sigmoid gate, an odd batch of fp32 activations
        _case(_PLAIN, "layer", "nvfp4", 17, "f32", n_ff_shexp=768, name="nvfp4_shexp_17"),
        # prompts: an ordinary ragged one for either weight type, and the longest, with a skewed router
        _case(_PLAIN, "layer", "nvfp4", 777, "bf16", name="nvfp4_prefill_777"),
        _case(_PLAIN, "layer", "q3_k", 1001, "f32", name="q3k_prefill_1001"),
        _case(_PLAIN, "layer", "nvfp4", 4096, "bf16", bias=True, name="nvfp4_prefill_4096"),
        # latent layer: a handful of sequences on the whole layer; through the expert-parallel step the 64 tokens that each of four
        # ranks has of a 256-token batch
        _case(_LATENT, "latent", "nvfp4", 3, "bf16", name="latent_decode_3"),
        _case(_LATENT, "ep", "nvfp4", 64, "bf16", name="latent_ep_64"),
        # the indexed matmul as an operator of its own
        _case(_PLAIN, "mmid", "nvfp4", 40, "f32", name="mul_mat_id_40"),
    ]


def _cost(c):
    w = work(c)
    return max(w["bytes"] / 6.5e12, w["flops"] / 1e14)


def draw(rng):
    most = max(_cost(c) for c in listed())
    q3_most = _cost(next(c for c in listed() if c["name"] == "q3k_prefill_1001"))
    while True:
        kind = rng.choice(("layer", "layer", "layer", "layer", "host", "latent", "ep", "mmid"))
        wtype = rng.choice(("nvfp4", "nvfp4", "q3_k")) if kind in ("layer", "host", "mmid") else "nvfp4"
        span = {"layer": 4096, "host": 512, "latent": 256, "ep": 256, "mmid": 512}[kind]
        tokens = int(round(math.exp(rng.uniform(0.0, math.log(span)))))
        if tokens > 4 and rng.random() < 0.6:
            tokens |= 1
        c = dict(kind=kind, wtype=wtype, tokens=tokens, x="f32" if kind == "mmid" else rng.choice(("bf16", "f32")), n_latent=0, n_ff_shexp=0,
                 bias=rng.random() < 0.3, layers=1, graph=False)
        if kind in ("latent", "ep"):
            c.update(n_embd=rng.choice((2048, 4096)), n_latent=rng.choice((512, 1024)), n_expert=rng.choice((64, 128, 256, 512)),
                     n_ff=rng.choice((512, 768, 1024)), top_k=rng.choice((4, 6, 8, 10)), bias=False)
        else:
            c.update(n_embd=rng.choice((512, 768, 2048) if wtype == "q3_k" else (512, 1024, 2048)), n_expert=rng.choice((16, 32, 64, 128, 256)),
                     n_ff=rng.choice((256, 512, 768)), top_k=rng.choice((2, 4, 6, 8, 10)))
            if kind == "layer" and rng.random() < 0.2:
                c["n_ff_shexp"] = rng.choice((512, 768))
            if kind == "layer" and tokens <= 2:
                c.update(layers=rng.randint(2, 4), graph=rng.random() < 0.5)
        if _cost(c) <= (q3_most if wtype == "q3_k" else most):
            return c


# ---- inputs ------------------------------------------------------------------------------------------------------------

def _nvfp4(gen, n, rows, cols, scaled):
    """uint8 [n][rows][cols / 64 * 36] quantised from N(0, 0.02) draws and the fp32 tensor scale of each matrix (None without)."""
    out = torch.empty((n, rows, cols // 64, 36), dtype=torch.uint8, device=DEV)
    scale = torch.empty(n, dtype=torch.float32, device=DEV)
    edges = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], device=DEV)
    step = max(1, (1 << 27) // (rows * cols))
    for a in range(0, n, step):
        b = min(n, a + step)
        w = torch.randn((b - a, rows, cols // 16, 16), generator=gen, device=DEV) * 0.02
        if scaled:
            s = w.abs().amax(dim=(1, 2, 3)) / (6 * 448)
            scale[a:b] = s
            w = w / s[:, None, None, None]
        d8 = (w.abs().amax(dim=-1) / 6).to(torch.float8_e4m3fn)
        d = d8.float().clamp(min=2.0 ** -9)[..., None]
        code = torch.bucketize((w / d).abs(), edges, out_int32=True).to(torch.uint8) | ((w < 0).to(torch.uint8) << 3)
        blk = out[a:b]
        blk[..., :4] = d8.view(torch.uint8).reshape(b - a, rows, cols // 64, 4)
        blk[..., 4:] = (code[..., :8] | (code[..., 8:] << 4)).reshape(b - a, rows, cols // 64, 32)
    return out.reshape(n, rows, -1), scale if scaled else None


def _q3_k(gen, n, rows, cols):
    """uint8 [n][rows][cols / 256 * 110] with the statistics of Q3_K blocks quantised from N(0, 0.02) draws."""
    out = torch.empty((n, rows, cols // 256, 110), dtype=torch.uint8, device=DEV)
    step = max(1, (1 << 26) // (rows * cols))
    for a in range(0, n, step):
        b = min(n, a + step)
        lead = (b - a, rows, cols // 256)
        code = (torch.randn(lead + (2, 4, 32), generator=gen, device=DEV) * 1.95 - 0.5).round().clamp(-4, 3).to(torch.int32) + 4
        sc = torch.randint(12, 32, lead + (16,), generator=gen, device=DEV, dtype=torch.int32)
        sc = sc * (torch.randint(0, 2, lead + (16,), generator=gen, device=DEV, dtype=torch.int32) * 2 - 1)
        at = torch.randint(0, 16, lead + (1,), generator=gen, device=DEV)
        sc = sc.scatter(-1, at, -32) + 32
        d = (torch.rand(lead, generator=gen, device=DEV) * 3e-4 + 3.5e-4) * (torch.randint(0, 2, lead, generator=gen, device=DEV) * 2 - 1)
        shift = torch.arange(4, device=DEV, dtype=torch.int32)
        bit = torch.arange(8, device=DEV, dtype=torch.int32).reshape(2, 4, 1)
        blk = out[a:b]
        blk[..., 0:32] = ((code >> 2) << bit).sum(dim=(-3, -2)).to(torch.uint8)
        blk[..., 32:96] = ((code & 3) << (2 * shift)[:, None]).sum(dim=-2).reshape(lead + (64,)).to(torch.uint8)
        blk[..., 96:104] = ((sc[..., :8] & 15) | ((sc[..., 8:] & 15) << 4)).to(torch.uint8)
        blk[..., 104:108] = ((sc >> 4).reshape(lead + (4, 4)) << (2 * shift)[:, None]).sum(dim=-2).to(torch.uint8)
        blk[..., 108:110] = d.half()[..., None].view(torch.uint8)
    return out.reshape(n, rows, -1)


def _matrices(gen, wtype, n, rows, cols, scaled=True):
    return _nvfp4(gen, n, rows, cols, scaled) if wtype == "nvfp4" else (_q3_k(gen, n, rows, cols), None)


def _weights(c, gen):
    E, H, I, n_in, wt = c["n_expert"], c["n_embd"], c["n_ff"], c["n_latent"] or c["n_embd"], c["wtype"]
    k = dict(router_w=torch.randn((E, H), generator=gen, device=DEV) * 0.02)
    if c["bias"]:
        k["router_bias"] = torch.randn(E, generator=gen, device=DEV)
    for name, rows, cols in (("gate", I, n_in), ("up", I, n_in), ("down", n_in, I)):
        k[name], k[name + "_scale"] = _matrices(gen, wt, E, rows, cols)
    if c["n_latent"]:
        for name, rows, cols in (("lat_down", n_in, H), ("lat_up", H, n_in)):
            q, k[name + "_scale"] = _matrices(gen, wt, 1, rows, cols)
            k[name] = q[0]
    if c["n_ff_shexp"]:
        S = c["n_ff_shexp"]
        for name, rows, cols in (("gate_shexp", S, H), ("up_shexp", S, H), ("down_shexp", H, S)):
            k[name] = _matrices(gen, wt, 1, rows, cols, scaled=False)[0][0]
        k["gate_inp_shexp"] = torch.randn(H, generator=gen, device=DEV) * 0.02
    return k


def prepare(case, seed):
    c = case
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    T, wt = c["tokens"], WTYPE[c["wtype"]]
    s = {"kind": c["kind"], "ctx": moe.Context(0), "graph": None}
    if c["kind"] == "mmid":
        s["w"] = _matrices(gen, c["wtype"], c["n_expert"], c["n_ff"], c["n_embd"], scaled=False)[0]
        s["b"] = torch.randn((T, 1, c["n_embd"]), generator=gen, device=DEV)
        s["ids"] = torch.rand((T, c["n_expert"]), generator=gen, device=DEV).topk(c["top_k"]).indices.to(torch.int32)
        s["wtype"], s["n_embd"] = wt, c["n_embd"]
        return s
    xs = [torch.randn((T, c["n_embd"]), generator=gen, device=DEV).to(torch.bfloat16 if c["x"] == "bf16" else torch.float32) for _ in range(c["layers"])]
    s["x"] = xs
    if c["kind"] == "ep":
        cfg = W.LayerConfig("ep", wt, n_embd=c["n_embd"], n_expert=c["n_expert"], top_k=c["top_k"], n_ff=c["n_ff"], n_latent=c["n_latent"])
        s["ep"] = ExpertParallelLayer(CudaBackend(s["ctx"], W.HostLayer(cfg, **_weights(c, gen))), cfg.n_expert, cfg.top_k)
        return s
    s["layers"] = [moe.MoeLayer(s["ctx"], wtype=wt, top_k=c["top_k"], **_weights(c, gen)) for _ in range(c["layers"])]
    if c["kind"] == "host":
        s["x"] = [x.cpu().pin_memory() for x in xs]
        s["out"] = torch.empty((T, c["n_embd"]), dtype=torch.float32).pin_memory()
    elif c["graph"]:
        s["out"] = [torch.empty((T, c["n_embd"]), dtype=torch.float32, device=DEV) for _ in xs]
        for l, x, o in zip(s["layers"], xs, s["out"]):
            l.forward(x, out=o)
        torch.cuda.synchronize()
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"]):
            for l, x, o in zip(s["layers"], xs, s["out"]):
                l.forward(x, out=o)
    return s


def run(state):
    s = state
    if s["kind"] == "mmid":
        return s["ctx"].mul_mat_id(s["wtype"], s["w"], s["b"], s["ids"], s["n_embd"])
    if s["kind"] == "ep":
        return s["ep"].forward(s["x"][0], return_routing=True)
    if s["kind"] == "host":
        return s["layers"][0].forward_host(s["x"][0], out=s["out"])
    if s["graph"] is not None:
        s["graph"].replay()
        return s["out"]
    return [l.forward(x) for l, x in zip(s["layers"], s["x"])]


def work(case):
    c = case
    T, k, E, H, I, n_in = c["tokens"], c["top_k"], c["n_expert"], c["n_embd"], c["n_ff"], c["n_latent"] or c["n_embd"]
    row = (lambda n: n // 64 * 36) if c["wtype"] == "nvfp4" else (lambda n: n // 256 * 110)
    touched = E * (1.0 - (1.0 - k / E) ** T)     # distinct experts of T tokens with k uniform choices each
    if c["kind"] == "mmid":
        return {"bytes": touched * I * row(H) + T * H * 4 + T * k * (I + 1) * 4, "flops": 2.0 * T * k * H * I}
    nbytes = touched * (2 * I * row(n_in) + n_in * row(I)) + E * H * 4 + T * H * ((2 if c["x"] == "bf16" else 4) + 4)
    flops = 2.0 * T * (k * 3 * n_in * I + E * H)
    if c["n_latent"]:
        nbytes += n_in * row(H) + H * row(n_in)
        flops += 4.0 * T * H * n_in
    if c["n_ff_shexp"]:
        S = c["n_ff_shexp"]
        nbytes += 2 * S * row(H) + H * row(S) + H * 4
        flops += 6.0 * T * S * H
    return {"bytes": nbytes * c["layers"], "flops": flops * c["layers"]}


def tolerance(case):
    c = case
    if c["kind"] == "mmid" or c["wtype"] == "q3_k" and not c["n_ff_shexp"] or c["tokens"] * c["top_k"] <= 16 and not c["n_latent"] and not c["n_ff_shexp"]:
        return "exact"      # integer dots summed in the reference's order: bit-identical by contract
    # Activations are re-quantised to int8 between the matmuls, so another order of the fp32 sums flips a few of those values.  The
    # default engines against the bit-identical one over 50 cases of these ranges: rel up to 3.3e-4, max up to 6.1e-3.
    return {"rel": 1e-3, "max": 2e-2}
