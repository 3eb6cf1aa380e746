"""Layers whose row blocks are worked in pairs (moe_gemm_sorted.cu), against the same layer launched stage by stage, whose kernels
work one block a CTA. With one route a token no sum depends on the order of the reductions, so the two agree bit for bit."""

import importlib

import pytest
import torch

import aiter_b200
from aiter_b200 import _lib
from oracle import moe_oracle

fm = importlib.import_module("aiter_b200.fused_moe")
pytestmark = pytest.mark.gpu
DEV = "cuda:0"
QT = aiter_b200.QuantType
ACT = aiter_b200.ActivationType
FP8 = torch.float8_e4m3fn
SCALES = {QT.per_1x128: lambda E, N, K: (E, N // 128, K // 128), QT.per_Token: lambda E, N, K: (E, N, 1), QT.per_Tensor: lambda E, N, K: (E, 1)}


def _layer(counts, H, I, qt, act=ACT.Silu, x_dtype=torch.bfloat16, keep=None, live=None, topk=1):
    """Expert e has counts[e] routes, spread over the tokens at random."""
    g = torch.Generator(device=DEV).manual_seed(11)
    E, M = len(counts), sum(counts) // topk
    ids = torch.repeat_interleave(torch.arange(E, device=DEV), torch.tensor(counts, device=DEV))
    ids = ids[torch.randperm(ids.numel(), generator=g, device=DEV)].view(M, topk).int()
    wts = torch.rand((M, topk), generator=g, device=DEV) + 0.1
    x, a1_scale = torch.randn((M, H), generator=g, device=DEV).to(torch.bfloat16), None
    if x_dtype == FP8:
        x, a1_scale = aiter_b200.get_hip_quant(qt)(x, quant_dtype=FP8)
    else:
        x = x.to(x_dtype)
    sl = slice(*keep) if keep else slice(None)
    n = len(range(E)[sl])
    mask = None
    if keep:
        mask = torch.zeros(E, dtype=torch.int32, device=DEV)
        mask[sl] = 1
    w = {}
    for name, N, K in (("w1", 2 * I, H), ("w2", H, I)):
        w[name] = torch.randn((n, N, K), generator=g, device=DEV).mul_(60).to(FP8)
        w[name + "_scale"] = (torch.rand(SCALES[qt](n, N, K), generator=g, device=DEV) + 0.5) / (60 * K ** 0.5)
    nl = torch.tensor([live], dtype=torch.int32, device=DEV) if live is not None else None
    return lambda: aiter_b200.fused_moe(x, w["w1"], w["w2"], wts, ids, expert_mask=mask, activation=act, quant_type=qt, w1_scale=w["w1_scale"],
                                        w2_scale=w["w2_scale"], a1_scale=a1_scale, num_local_tokens=nl)


def _stages(run):
    fm.kernel_bench_events = []      # a list here selects the stage-by-stage launches
    try:
        return run()
    finally:
        fm.kernel_bench_events = None


EDGES = [129, 256, 1, 257, 0, 128, 384, 385]   # rows of an expert: around one, two and three blocks, none


@pytest.mark.parametrize("x_dtype", [torch.bfloat16, torch.float16, FP8])
@pytest.mark.parametrize("qt,H,I", [(QT.per_1x128, 384, 1024),     # half a tile of columns, K steps in fours
                                    (QT.per_1x128, 256, 1152),     # nine K steps
                                    (QT.per_Token, 2176, 4096), (QT.per_Tensor, 2048, 4224)])
def test_pairs_equal_single_blocks(qt, H, I, x_dtype):
    run = _layer(EDGES, H, I, qt, x_dtype=x_dtype, act=ACT.Gelu if x_dtype == torch.float16 else ACT.Silu)
    out, ref = run(), _stages(run)
    aiter_b200.check_device_status()
    assert float(ref.float().abs().max()) > 0
    if qt == QT.per_Tensor:
        # the stages repeat the one scale per row and per channel, so its two factors are multiplied in another order: 1e-7 of a
        # stage-1 value, which moves 3e-5 of them by a bf16 step, one in eight rows of 4224 by 6e-5 of its size, 2e-3 of the outputs
        s = moe_oracle.error_stats(out.float().to(torch.bfloat16), ref.float().to(torch.bfloat16).cpu())
        assert not s["has_nan"] and s["n_diff"] <= 1e-2 * s["numel"] and s["max_abs_over_rms"] <= 0.04, s
    else:
        assert torch.equal(out.view(torch.int16), ref.view(torch.int16))


@pytest.mark.parametrize("qt,H,I", [(QT.per_1x128, 256, 1024), (QT.per_Token, 2048, 4096)])
@pytest.mark.parametrize("counts,keep,live", [([700] * 4, (1, 3), None), ([300, 5, 900, 400], None, 1201), ([640] * 4, (0, 2), 0)])
def test_masked_and_padded_batches(qt, H, I, counts, keep, live):
    run = _layer(counts, H, I, qt, keep=keep, live=live)
    out, ref = run(), _stages(run)
    aiter_b200.check_device_status()
    assert torch.equal(out.view(torch.int16), ref.view(torch.int16))


@pytest.mark.parametrize("qt,H,I", [(QT.per_1x128, 4096, 1024), (QT.per_Token, 4096, 4096)])
def test_many_tiles_per_pair_of_ctas(qt, H, I):
    """More tiles than pairs of CTAs: every ring goes round and the staged rows are used again."""
    run = _layer([1500] * 8, H, I, qt)
    out, ref = run(), _stages(run)
    aiter_b200.check_device_status()
    assert torch.equal(out.view(torch.int16), ref.view(torch.int16))


@pytest.mark.parametrize("qt,H,I", [(QT.per_1x128, 256, 1024), (QT.per_Token, 2048, 4096)])
def test_waits_of_a_pair_run_out(qt, H, I):
    run = _layer([256, 300], H, I, qt)
    before = run()
    aiter_b200.check_device_status()
    try:
        _lib.call_plain("b200_moe_debug_config", 2_000_000, 1)    # ~1 ms at 1.9 GHz, producer stalled
        run()
        with pytest.raises(RuntimeError, match="gave up on a device-side wait"):
            aiter_b200.check_device_status()
    finally:
        _lib.call_plain("b200_moe_debug_config", 0, 0)
    after = run()
    aiter_b200.check_device_status()
    assert torch.equal(before.view(torch.int16), after.view(torch.int16))
