"""Sort and quantiser kernels at the edges of their work split: chunk and round boundaries of the sort, expert counts that
are odd, one or the maximum, masks and row limits; pieces per thread and cached row lengths of the quantisers. Bit-exact."""

import pytest
import torch

import aiter_b200
from oracle import moe_oracle
from test_gpu_sorting import DEV, check, run_sort

pytestmark = pytest.mark.gpu
FP8 = torch.float8_e4m3fn
QT = aiter_b200.QuantType


@pytest.mark.parametrize("M,topk,E,unit,masked,live", [
    (1, 1, 1, 1, False, None), (1023, 1, 7, 16, False, None), (1025, 1, 7, 128, True, None),   # one round | two
    (1024, 4, 33, 32, False, None), (4097, 1, 33, 32, True, 4096),                             # one chunk | two
    (2048, 8, 256, 128, False, 2047), (2049, 8, 256, 128, True, None),                         # one kernel | two
    (4100, 8, 1000, 64, True, 3), (6000, 6, 1024, 16, False, None), (20000, 2, 5, 128, False, 0),
])
def test_sort_edges(M, topk, E, unit, masked, live):
    g = torch.Generator().manual_seed(M + E)
    ids = torch.randint(0, E, (M, topk), generator=g, dtype=torch.int32)   # duplicates within a token are allowed
    ids[:: 3] = 0                                                          # a hot expert
    w = torch.rand((M, topk), generator=g)
    mask = (torch.arange(E) % 3 != 1).to(torch.int32) if masked else None
    nl = torch.tensor([live], dtype=torch.int32) if live is not None else None
    *out, local = run_sort(ids, w, E, unit, mask, nl, return_local_topk_ids=True)
    check(out, moe_oracle.moe_sorting_ref(ids, w, E, unit, mask, nl), f"{M}x{topk} E{E} unit {unit}")
    assert int(out[4].view(torch.int16).abs().max()) == 0 if out[4].numel() else True
    ref = moe_oracle.local_expert_ids(ids, mask if mask is not None else torch.ones(E, dtype=torch.int32)).to(torch.int32)
    if live is not None:
        ref[live:] = -1
    assert torch.equal(local.cpu(), ref)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,cols,limit", [(1, 128, None), (33, 384, 7), (2369, 4096, None), (2368, 4096, 2000)])
def test_group_quant_edges(dtype, rows, cols, limit):
    g = torch.Generator().manual_seed(rows)
    x = (torch.randn((rows, cols), generator=g) * 4).to(dtype)
    x[0, :8] = torch.tensor([0.0, -0.0, 1e-7, 448.0, -3.0, 0.5, 1e-30, 65504.0]).to(dtype)
    lim = torch.tensor([limit], dtype=torch.int32, device=DEV) if limit is not None else None
    n = rows if limit is None else limit
    q_ref, s_ref = moe_oracle.quant_1x128(x)
    for transpose in (False, True):
        q, s = aiter_b200.per_group_quant_hip(x.to(DEV), quant_dtype=FP8, num_rows=lim, transpose_scale=transpose)
        s = s.view(-1)[:n * (cols // 128)].view(cols // 128, n).t().contiguous() if transpose else s[:n]
        assert torch.equal(q[:n].cpu().view(torch.uint8), q_ref[:n].view(torch.uint8))
        assert torch.equal(s.cpu().view(torch.int32), s_ref[:n].view(torch.int32))


@pytest.mark.parametrize("rows,cols,limit", [(3, 8, None), (1, 4096, None), (5, 4104, None), (4, 16384, 3), (2, 16392, None),
                                             (3000, 256, 2999)])
def test_row_and_tensor_quant_edges(rows, cols, limit):
    g = torch.Generator().manual_seed(cols)
    x = (torch.randn((rows, cols), generator=g) * 4).to(torch.bfloat16)
    lim = torch.tensor([limit], dtype=torch.int32, device=DEV) if limit is not None else None
    n = rows if limit is None else limit
    q, s = aiter_b200.per_token_quant_hip(x.to(DEV), quant_dtype=FP8, num_rows=lim)
    q_ref, s_ref = moe_oracle.quant_per_token(x)
    assert torch.equal(q[:n].cpu().view(torch.uint8), q_ref[:n].view(torch.uint8))
    assert torch.equal(s[:n].cpu().view(torch.int32), s_ref[:n].view(torch.int32))
    q, s = aiter_b200.per_tensor_quant_hip(x.to(DEV), quant_dtype=FP8)
    q_ref, s_ref = moe_oracle.quant_per_tensor(x)
    assert torch.equal(q.cpu().view(torch.uint8), q_ref.view(torch.uint8)) and float(s) == float(s_ref)


@pytest.mark.parametrize("qt", [QT.per_1x128, QT.per_Token, QT.per_Tensor])
def test_quant_codes_at_extreme_scales(qt):
    """Codes are the correctly rounded quotients over the whole range of scales: around both limits between the two ways of
    dividing, where residuals are subnormal, and with quotients on and beside the middles between two codes."""
    g = torch.Generator().manual_seed(7)
    oracle = {QT.per_1x128: moe_oracle.quant_1x128, QT.per_Token: moe_oracle.quant_per_token,
              QT.per_Tensor: moe_oracle.quant_per_tensor}[qt]
    m = torch.randint(128, 256, (64, 128), generator=g).float() * 2.0 ** torch.randint(-18, 1, (64, 128), generator=g)
    x = m * torch.where(torch.rand((64, 128), generator=g) < 0.5, -1.0, 1.0)
    x[:, 0] = 448.0 * torch.randint(128, 256, (64,), generator=g) / 256     # scales of few bits: quotients hit the middles
    for top in (2.0 ** -120, 448e-30, 4.48e-27, 448e-24, 2.0 ** -70, 1.0, 2.0 ** 90, 448e30):
        t = (x.double() * (top / 448.0)).to(torch.bfloat16)
        q, s = aiter_b200.get_hip_quant(qt)(t.to(DEV), quant_dtype=FP8)
        q_ref, s_ref = oracle(t)
        assert torch.equal(s.cpu().view(-1).view(torch.int32), s_ref.reshape(-1).view(torch.int32)), top
        assert torch.equal(q.cpu().view(torch.uint8), q_ref.view(torch.uint8)), top
