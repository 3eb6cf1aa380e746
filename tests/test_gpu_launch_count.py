"""``_lib.launch_count`` against the kernels that a captured layer call holds."""

import ctypes
import importlib

import pytest
import torch

import aiter_b200
from aiter_b200 import _lib

fm = importlib.import_module("aiter_b200.fused_moe")
pytestmark = pytest.mark.gpu
DEV = "cuda:0"
QT = aiter_b200.QuantType
FP8 = torch.float8_e4m3fn
SCALES = {QT.per_1x128: lambda E, N, K: (E, N // 128, K // 128), QT.per_Token: lambda E, N, K: (E, N, 1), QT.per_Tensor: lambda E, N, K: (E, 1)}


def _kernel_nodes(graph):
    """Number of kernel nodes of a captured graph (CU_GRAPH_NODE_TYPE_KERNEL is 0)."""
    cuda = ctypes.CDLL("libcuda.so.1")
    handle, n = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    assert cuda.cuGraphGetNodes(handle, None, ctypes.byref(n)) == 0
    nodes = (ctypes.c_void_p * n.value)()
    assert cuda.cuGraphGetNodes(handle, nodes, ctypes.byref(n)) == 0
    kinds = []
    for node in nodes:
        kind = ctypes.c_int(-1)
        assert cuda.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        kinds.append(kind.value)
    return kinds.count(0)


@pytest.mark.parametrize("qt", list(SCALES))
@pytest.mark.parametrize("x_dtype", [torch.bfloat16, FP8])
# up to 16384 routes, above; one block a CTA and pairs (b200_moe_debug_pairs)
@pytest.mark.parametrize("M,topk,E,I", [(40, 2, 8, 256), (8200, 2, 256, 256), (300, 2, 4, 1024), (8200, 2, 4, 1024)])
@pytest.mark.parametrize("pairs", [1, 2])
def test_count_is_what_a_graph_of_the_call_holds(qt, x_dtype, M, topk, E, I, pairs, monkeypatch):
    monkeypatch.setattr(fm, "_layer_sizes", fm._layer_sizes.__wrapped__)
    g = torch.Generator(device=DEV).manual_seed(1)
    H = 2048
    x, a1_scale = torch.randn((M, H), generator=g, device=DEV).to(torch.bfloat16), None
    if x_dtype == FP8:
        x, a1_scale = aiter_b200.get_hip_quant(qt)(x, quant_dtype=FP8)
    ids = torch.randint(0, E, (M, topk), generator=g, device=DEV, dtype=torch.int32)
    wts = torch.rand((M, topk), generator=g, device=DEV)
    w1, w2 = torch.zeros((E, 2 * I, H), device=DEV).to(FP8), torch.zeros((E, H, I), device=DEV).to(FP8)
    s1, s2 = torch.ones(SCALES[qt](E, 2 * I, H), device=DEV), torch.ones(SCALES[qt](E, H, I), device=DEV)

    def run():
        return aiter_b200.fused_moe(x, w1, w2, wts, ids, quant_type=qt, w1_scale=s1, w2_scale=s2, a1_scale=a1_scale)

    _lib.call_plain("b200_moe_debug_pairs", pairs)
    try:
        run()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        before = _lib.launch_count
        with torch.cuda.graph(graph):
            run()
    finally:
        _lib.call_plain("b200_moe_debug_pairs", 0)
    assert _lib.launch_count - before == _kernel_nodes(graph)
