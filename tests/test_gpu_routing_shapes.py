"""Group layouts of the grouped router that take its different branches: groups that are a power-of-two run of lanes, that
are not, that share a lane, expert counts that are no multiple of a vector load, and both types of bias."""

import pytest
import torch

import aiter_b200
from oracle import moe_oracle
from test_gpu_routing import DEV, compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,E,topk,groups,topk_group,bias_dtype", [
    (65, 256, 8, 32, 4, torch.float32),      # one group per lane
    (31, 256, 8, 1, 1, torch.bfloat16),      # one group over all lanes
    (40, 160, 6, 8, 3, torch.float32),       # 20 experts a group: a lane of 8 holds two groups' experts
    (17, 96, 4, 8, 2, torch.bfloat16),       # 12 a group over lanes of 4: three lanes a group
    (9, 30, 3, 3, 2, torch.float32),         # no vector loads, one expert a lane, 10 a group
    (5, 32, 4, 16, 8, torch.float32),        # groups of two experts on two lanes
    (3, 1024, 8, 16, 4, torch.float32),      # 32 experts a lane
])
def test_group_layouts(M, E, topk, groups, topk_group, bias_dtype):
    g = torch.Generator().manual_seed(E + groups)
    logits = torch.randn((M, E), generator=g)
    bias = (torch.randn((E,), generator=g) * 0.1).to(bias_dtype)
    w_ref, ids_ref = moe_oracle.biased_grouped_topk_ref(logits, bias.float(), topk, True, groups, topk_group, 2.5)
    w = torch.empty((M, topk), dtype=torch.float32, device=DEV)
    ids = torch.empty((M, topk), dtype=torch.int32, device=DEV)
    aiter_b200.biased_grouped_topk(logits.to(DEV), bias.to(DEV), w, ids, groups, topk_group, True, 2.5)
    compare(w, ids, w_ref, ids_ref, f"{M}x{E} in {groups} groups")
