"""The one-call layer entry point (b200_fused_moe, what ``fused_moe`` uses) against the same layer launched stage by
stage: every quantisation type, input dtype and optional argument that changes the workspace map or a pointer."""

import importlib

import pytest
import torch

import aiter_b200
from oracle import inputs, moe_oracle

fm = importlib.import_module("aiter_b200.fused_moe")
pytestmark = pytest.mark.gpu
DEV = "cuda:0"
QT = aiter_b200.QuantType
FP8 = torch.float8_e4m3fn


@pytest.mark.parametrize("name,qt", [("cfg0", QT.per_1x128), ("cfg0_pt", QT.per_Token), ("cfg0_ptensor", QT.per_Tensor)])
@pytest.mark.parametrize("x_dtype", [torch.bfloat16, torch.float16, FP8])
@pytest.mark.parametrize("M,masked,live", [(1, False, None), (32, False, None), (9000, False, None), (32, True, 20)])
def test_one_call_equals_stages(name, qt, x_dtype, M, masked, live):
    c = inputs.make_config(name, seed=5, device=DEV, M=M)
    c = {k: (v.to(DEV) if isinstance(v, torch.Tensor) else v) for k, v in c.items()}
    E = c["cfg"]["E"]
    x, a1_scale = c["x"], None
    if x_dtype == FP8:
        x, a1_scale = aiter_b200.get_hip_quant(qt)(x, quant_dtype=FP8)
    else:
        x = x.to(x_dtype)
    sl = slice(0, E // 2) if masked else slice(None)
    mask = (torch.arange(E, device=DEV) < E // 2).to(torch.int32) if masked else None
    nl = torch.tensor([live], dtype=torch.int32, device=DEV) if live is not None else None

    def run():
        return aiter_b200.fused_moe(x, c["w1_q"][sl], c["w2_q"][sl], c["topk_weight"], c["topk_ids"], expert_mask=mask,
                                    quant_type=qt, w1_scale=c["w1_scale"][sl], w2_scale=c["w2_scale"][sl],
                                    a1_scale=a1_scale, num_local_tokens=nl)

    out = run()
    fm.kernel_bench_events = []      # a list here selects the stage-by-stage launches
    try:
        ref = run()
    finally:
        marks, fm.kernel_bench_events = fm.kernel_bench_events, None
    aiter_b200.check_device_status()
    assert len(marks) > 4 and out.dtype == ref.dtype == (torch.bfloat16 if x_dtype == FP8 else x_dtype)
    if live is not None:
        assert int((out[live:].view(torch.int16) != 0).sum()) == 0
    # the same kernels on the same inputs; only the order of stage 2's fp32 additions differs from run to run, which moves
    # isolated outputs by one step of the output type
    s = moe_oracle.error_stats(out.float().to(torch.bfloat16), ref.float().to(torch.bfloat16).cpu())
    assert not s["has_nan"] and s["n_diff"] <= 2e-3 * s["numel"] + 2 and s["max_abs_over_rms"] <= 0.04, s
