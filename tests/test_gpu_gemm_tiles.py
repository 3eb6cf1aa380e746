"""The GEMM kernels at the edges of their tiles: output widths that leave half an output tile, blocks with
dead 32-row quarters, few tiles with long K, every scale type, against the oracle."""
import pytest
import torch

import aiter_b200 as ab
from oracle import moe_oracle

pytestmark = pytest.mark.gpu
QT = {"block": ab.QuantType.per_1x128, "token": ab.QuantType.per_Token, "tensor": ab.QuantType.per_Tensor}


def _weights(E, N, K, quant, g):
    w = torch.randn((E, N, K), generator=g) / K ** 0.5
    v = w.view(E, N // 128, 128, K // 128, 128)
    dims = {"block": (2, 4), "token": (3, 4), "tensor": (1, 2, 3, 4)}[quant]
    s = v.abs().amax(dim=dims, keepdim=True) / 448.0
    shape = {"block": (E, N // 128, K // 128), "token": (E, N, 1), "tensor": (E, 1)}[quant]
    return (v / s).to(torch.float8_e4m3fn).view(E, N, K), s.reshape(shape).contiguous()


def _deq(q, s, quant):
    E, N, K = q.shape
    q = q.double()
    if quant == "block":
        return (q.view(E, N // 128, 128, K // 128, 128) * s.double().view(E, N // 128, 1, K // 128, 1)).view(E, N, K)
    return q * s.double().view(E, -1, 1)


# H: half an output tile, one, odd counts of halves; rows per expert around the 32- and 128-row edges, and none
@pytest.mark.parametrize("quant", ["block", "token", "tensor"])
@pytest.mark.parametrize("H,I,E,rows", [(128, 128, 1, [3]), (256, 128, 3, [1, 31, 33]), (384, 256, 4, [97, 0, 128, 129]),
                                        (640, 384, 5, [64, 65, 0, 260, 1]), (1408, 128, 2, [32, 96]),
                                        # long K with fewer tiles than SMs; a second, partly filled round of tiles; few tiles in stage 2
                                        (7168, 384, 13, [1, 40, 130, 2, 3, 64, 7, 5, 1, 9, 33, 1, 2]),
                                        (2048, 1024, 20, [1 + 7 * i for i in range(20)]), (512, 2560, 6, [1, 128, 5, 70, 2, 33])])
def test_layer_at_tile_edges(quant, H, I, E, rows):
    g = torch.Generator().manual_seed(H + I)
    M = sum(rows)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(rows))[torch.randperm(M, generator=g)].to(torch.int32)[:, None]
    wts = torch.rand((M, 1), generator=g) + 0.5
    x = torch.randn((M, H), generator=g).to(torch.bfloat16)
    w1, s1 = _weights(E, 2 * I, H, quant, g)
    w2, s2 = _weights(E, H, I, quant, g)
    c = [t.cuda() for t in (x, w1, w2, wts, ids.contiguous(), s1, s2)]
    out = ab.fused_moe(c[0], c[1], c[2], c[3], c[4], quant_type=QT[quant], w1_scale=c[5], w2_scale=c[6])
    ab.check_device_status()

    def requant(t):   # the layer's activation quantisation, in fp32 as it is defined
        t = t.float()
        v = t.view(t.shape[0], -1, 128) if quant == "block" else t
        s = v.abs().amax(dim=None if quant == "tensor" else -1, keepdim=True) / 448.0
        s = torch.where(s == 0, torch.ones_like(s), s)
        return ((v / s).to(torch.float8_e4m3fn).double() * s.double()).view(t.shape)

    d1, d2, a1 = _deq(w1, s1, quant), _deq(w2, s2, quant), requant(x)
    h = torch.stack([d1[int(e)] @ a1[m] for m, e in enumerate(ids[:, 0])])
    a2 = requant((torch.nn.functional.silu(h[:, :I]) * h[:, I:]).to(torch.bfloat16))
    ref = torch.stack([d2[int(e)] @ a2[m] for m, e in enumerate(ids[:, 0])]) * wts.double()
    # bf16 result (2^-9 relative) plus single e4m3 codes of a2 that round the other way: the bars of the layer tests
    s = moe_oracle.error_stats(out, ref.to(torch.bfloat16))
    assert not s["has_nan"] and s["frac_within"] >= 0.995 and s["max_abs_over_rms"] <= 0.06, s


def test_padding_between_live_rows_of_one_cta():
    """Row scales: the requantiser's CTAs (8 an SM) stride over 7680 sorted rows of which they skip the padding, so a CTA meets
    live and padding rows in every order."""
    test_layer_at_tile_edges("token", 128, 640, 60, [(1, 40, 70, 128)[(i * i + i // 7) % 4] for i in range(60)])


def test_dead_quarters_between_live_ones_with_one_k_block():
    """Block scales, K = 128 in stage 1: a CTA has four tiles, in which a 32-row quarter is live and dead in every order."""
    test_layer_at_tile_edges("block", 128, 1280, 60, [(1, 40, 70, 128)[(i * i + i // 7) % 4] for i in range(60)])
