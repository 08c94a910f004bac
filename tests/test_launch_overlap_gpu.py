"""Which launches are programmatic dependents: never the one kernel of a call that stands alone, whatever ran on the context before."""
import ctypes as C

import pytest
import torch

from edge0_b200 import workloads as W
from edge0_b200.capi import TYPE_NVFP4

pytestmark = pytest.mark.gpu

CFG = W.small_config(TYPE_NVFP4, n_embd=512, n_expert=32, top_k=4, n_ff=256, seed=5)


def dependent_edges(graph):
    """programmatic dependencies among a captured graph's edges, and all its edges"""
    class EdgeData(C.Structure):            # cudaGraphEdgeData
        _fields_ = [("from_port", C.c_ubyte), ("to_port", C.c_ubyte), ("type", C.c_ubyte), ("reserved", C.c_ubyte * 5)]

    rt, raw, n = C.CDLL("libcudart.so.12"), C.c_void_p(graph.raw_cuda_graph()), C.c_size_t(0)
    assert rt.cudaGraphGetEdges_v2(raw, None, None, None, C.byref(n)) == 0
    ends, data = (C.c_void_p * (2 * n.value))(), (EdgeData * n.value)()
    assert rt.cudaGraphGetEdges_v2(raw, ends, C.byref(ends, n.value * C.sizeof(C.c_void_p)), data, C.byref(n)) == 0
    return sum(e.type == 1 for e in data), n.value          # 1: cudaGraphDependencyTypeProgrammatic


@pytest.mark.parametrize("behind", ["kernel", "copy", "join"])
def test_f32_product_is_an_ordinary_launch(behind, gpu_ctx):
    """One kernel, captured behind a kernel, a copy or a join with a second stream, after a layer call whose launches overlap."""
    layer = W.make_layer(CFG).to_device(gpu_ctx)
    gen = torch.Generator(device="cuda").manual_seed(3)
    w, y = torch.randn((64, 512), generator=gen, device="cuda"), torch.randn((3, 512), generator=gen, device="cuda")
    x, d = torch.zeros_like(y), torch.empty((3, 64), device="cuda")

    def product(src, dst):
        gpu_ctx.check(gpu_ctx.lib.b200moe_op_mul_mat_f32(gpu_ctx.handle, w.data_ptr(), 512, 64, src.data_ptr(), 3, dst.data_ptr(), gpu_ctx._stream()))

    want = torch.empty_like(d)
    product(2 * y if behind == "kernel" else y, want)
    layer.forward(torch.from_numpy(W.make_tokens(CFG, 1)).cuda())
    gpu_ctx.synchronize()
    side = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        if behind == "kernel":
            torch.mul(y, 2, out=x)
        elif behind == "copy":
            x.copy_(y)
        else:
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                torch.mul(y, 1, out=x)
            torch.cuda.current_stream().wait_stream(side)
        product(x, d)
    assert dependent_edges(graph) == (0, 1)
    graph.replay()
    gpu_ctx.synchronize()
    assert torch.equal(d, want)


def test_captured_layer_overlaps_inside_only(gpu_ctx):
    """The launches of a layer depend on one another programmatically; its first one depends on what is before it as any kernel does."""
    layer = W.make_layer(CFG).to_device(gpu_ctx)
    x, out = torch.from_numpy(W.make_tokens(CFG, 1)).cuda(), torch.empty((1, 512), device="cuda")
    layer.forward(x, out=out)
    gpu_ctx.synchronize()
    alone, behind = torch.cuda.CUDAGraph(keep_graph=True), torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(alone):
        layer.forward(x, out=out)
    with torch.cuda.graph(behind):
        x.mul_(1)
        layer.forward(x, out=out)
    inside, edges = dependent_edges(alone)
    assert inside == edges > 0
    assert dependent_edges(behind) == (inside, edges + 1)


@pytest.mark.parametrize("T", [1, 20])
def test_layer_waits_for_what_its_stream_waits_for(T, gpu_ctx):
    """x made on a second stream that the layer's stream has joined, right behind a copy, right behind a kernel, and on the host."""
    layer = W.make_layer(CFG).to_device(gpu_ctx)
    tokens = torch.from_numpy(W.make_tokens(CFG, T)).cuda()
    xs = [tokens * (i + 1) for i in range(4)]
    want = [layer.forward(x).clone() for x in xs]
    gpu_ctx.synchronize()
    x, out = torch.zeros_like(tokens), torch.empty((T, 512), device="cuda")
    host = [v.cpu().pin_memory() for v in xs]
    side, cur = torch.cuda.Stream(), torch.cuda.current_stream()
    busy = torch.randn((2048, 2048), device="cuda")
    for i in range(24):
        src, how = xs[i % 4], (i // 4) % 3
        if how == 0:
            side.wait_stream(cur)
            with torch.cuda.stream(side):
                busy @ busy                      # x arrives long after the host has launched the layer
                torch.mul(src, 1, out=x)
            cur.wait_stream(side)
        elif how == 1:
            busy @ busy
            x.copy_(host[i % 4], non_blocking=True)
        else:
            busy @ busy
            torch.mul(src, 1, out=x)
        layer.forward(x, out=out)
        assert torch.equal(out, want[i % 4]), i
        x.zero_()
    for i in range(8):
        assert torch.equal(layer.forward_host(host[i % 4]), want[i % 4].cpu()), i
