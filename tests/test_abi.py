"""The C-ABI library loads on a machine without a GPU and exports what include/*.h declares."""

import ctypes
import glob
import os
import re

import pytest
import torch

from conftest import ROOT

import aiter_b200
from aiter_b200 import _lib, build


@pytest.fixture(scope="module")
def lib():
    build.build()
    return _lib.lib()


def declared_functions():
    names = []
    for h in glob.glob(os.path.join(ROOT, "include", "*.h")):
        text = re.sub(r"/\*.*?\*/", "", open(h).read(), flags=re.S)
        names += re.findall(r"\b((?:aiter|b200)_[a-z0-9_]+)\s*\(", text)
    return sorted(set(names))


def test_header_and_library_agree(lib):
    decl = declared_functions()
    assert len(decl) >= 9
    for name in decl:
        assert hasattr(lib, name), f"{name} declared in include/ but not exported"
    assert set(_lib.exported_symbols()) == set(decl)


def test_ctypes_signatures_match_header(lib):
    """Every binding passes exactly as many arguments as the header declares."""
    text = ""
    for h in glob.glob(os.path.join(ROOT, "include", "*.h")):
        text += re.sub(r"/\*.*?\*/", "", open(h).read(), flags=re.S)
    for name, (_res, args) in _lib._SIGNATURES.items():
        m = re.search(r"\b" + name + r"\s*\(([^)]*)\)", text)
        assert m, name
        params = m.group(1).strip()
        n = 0 if params in ("", "void") else params.count(",") + 1
        assert n == len(args), f"{name}: header has {n} parameters, binding passes {len(args)}"


def test_abi_version_and_error_channel(lib):
    assert lib.aiter_ctypes_abi_version() == 4
    lib.aiter_clear_last_error()
    assert lib.aiter_get_last_error() is None
    # a call with a NULL tensor fails with status -1 and a message, without touching a GPU
    st = lib.b200_moe_quant_1x128(None, None, None, None, 1, 0, None)
    assert st == -1
    assert b"input must not be NULL" in lib.aiter_get_last_error()
    lib.aiter_clear_last_error()
    assert lib.aiter_get_last_error() is None


def test_tensor_struct_layout():
    # csrc/include/aiter_tensor.h:8-18 is a 160-byte POD
    assert ctypes.sizeof(_lib.aiter_tensor_t) == 160
    t = torch.zeros((3, 5), dtype=torch.int32)[:, ::2]
    s = _lib.to_aiter(t)
    assert (s.ndim, s.numel_, list(s.shape[:2]), list(s.strides[:2])) == (2, 9, [3, 3], [5, 2])
    assert s.dtype_ == 8 and s.device_id == -1
    assert _lib.to_aiter(None) is None


def test_workspace_size(lib):
    assert aiter_b200.moe_sorting_get_workspace_size(64, 256, 8) == 0
    ws = aiter_b200.moe_sorting_get_workspace_size(8192, 256, 8)
    assert ws == (16 * 256 + 256) * 4


# M, H, I, experts here, experts, topk, quant type, hidden dtype; kernels: sort (two above 16384 routes), quantiser (none for fp8, two for
# one scale per tensor), stage 1, requantisation of row scales, stage 2, final rounding; layers in pairs: two launches a stage, and with
# row scales the copy into sorted order
@pytest.mark.parametrize("sizes,kernels", [
    ((1, 4096, 1536, 128, 128, 8, 4, torch.bfloat16), 5), ((513, 1024, 512, 8, 8, 2, 1, torch.bfloat16), 7),
    ((32, 4096, 14336, 8, 8, 2, 2, torch.float16), 6), ((2048, 7168, 2048, 32, 256, 8, 4, torch.float8_e4m3fn), 4),
    ((3000, 7168, 512, 256, 256, 8, 4, torch.bfloat16), 6), ((4096, 4096, 14336, 8, 8, 2, 2, torch.bfloat16), 9),
    ((9000, 4096, 14336, 8, 8, 2, 1, torch.bfloat16), 11), ((16384, 4096, 1536, 128, 128, 8, 4, torch.bfloat16), 7)])
def test_kernels_of_a_layer_call(lib, sizes, kernels):
    assert lib.b200_fused_moe_launches(*sizes[:-1], _lib.AITER_DTYPE[sizes[-1]], 0) == kernels


# M, H, I, experts here, experts, topk, row scales, in pairs; both sides of every line of the rule
@pytest.mark.parametrize("M,H,I,local,E,topk,rows,pairs", [
    (4096, 4096, 1024, 32, 32, 8, False, True), (4096, 4096, 896, 32, 32, 8, False, False),          # inner dimension
    (2304, 7168, 2048, 128, 128, 8, False, True), (2303, 7168, 2048, 128, 128, 8, False, False),     # 144 rows an expert
    (527, 7168, 2048, 16, 16, 8, False, True), (528, 7168, 2048, 16, 16, 8, False, False),           # mostly three blocks from here
    (751, 7168, 2048, 16, 16, 8, False, False), (752, 7168, 2048, 16, 16, 8, False, True),           # ... to here
    (1056, 7168, 2048, 32, 32, 8, False, True), (1056, 6784, 2048, 32, 32, 8, False, False),         # ... which want twelve rounds
    (7104, 1024, 1024, 8, 8, 4, False, True), (7103, 1024, 1024, 8, 8, 4, False, False),             # six rounds of tiles
    (1000, 256, 1024, 4, 4, 1, False, False), (601, 4096, 4096, 4, 4, 1, False, False),              # small layers
    (8192, 7168, 2048, 32, 256, 8, False, True), (8192, 7168, 2048, 15, 256, 8, False, False),       # the share of this rank
    (592, 4096, 14336, 8, 8, 2, True, True), (578, 4096, 14336, 8, 8, 2, True, False),               # row scales
    (8192, 2048, 4096, 32, 32, 8, True, True), (8192, 1920, 4096, 32, 32, 8, True, False), (8192, 4096, 3968, 32, 32, 8, True, False),
    (2400, 4096, 4096, 32, 32, 8, True, False), (2400, 4096, 6144, 32, 32, 8, True, True),           # five blocks
    (1200, 4096, 10240, 8, 8, 2, True, True), (2400, 4096, 10112, 16, 16, 2, True, False),           # three blocks
    (1601, 4096, 4096, 8, 8, 2, True, False), (4096, 2048, 6144, 8, 8, 2, True, False), (4096, 4096, 8192, 8, 8, 2, True, True)])
def test_layers_in_pairs(lib, M, H, I, local, E, topk, rows, pairs):
    bf16 = _lib.AITER_DTYPE[torch.bfloat16]
    kernels = (9 if pairs else 6) if rows else (6 if pairs else 5)
    assert lib.b200_fused_moe_launches(M, H, I, local, E, topk, 2 if rows else 4, bf16, 0) == kernels + (M * topk > 16384)


def test_padded_batches_are_not_worked_in_pairs(lib):
    """The rows that pay for the pairs need not be there."""
    for quant, kernels in ((4, 6), (2, 7), (1, 8)):   # one kernel of them the count in front of the sort
        assert lib.b200_fused_moe_launches(9000, 4096, 14336, 8, 8, 2, quant, _lib.AITER_DTYPE[torch.bfloat16], 1) == kernels


def test_sizes_that_are_no_layer(lib):
    """The queries answer, whatever they are asked."""
    for sizes in ((0, 0, 0, 0, 0, 0), (-1, 4096, 4096, 8, 8, 2), (4096, 4096, 4096, 8, 0, 2)):
        assert lib.b200_fused_moe_launches(*sizes, 2, 0, 0) >= 4
        assert lib.b200_fused_moe_workspace_size(*sizes[:3], sizes[4], sizes[5], 2, 0) is not None


def test_workspace_of_a_layer(lib):
    """Bytes of a layer that is not worked in pairs: what its kernels use, buffer by buffer, and nothing for the pairs."""
    M, H, I, E, topk = 513, 1024, 640, 8, 2
    P = M * topk + E * 128 - topk
    def up(n):
        return -(-n // 256) * 256
    common = 2 * up(4 * P) + up(4 * (-(-P // 128))) + up(8) + 256 + up(4 * M * H) + up(M * H) + up(P * I)
    block = common + up(4 * M * H // 128) + up(4 * P * I // 128)
    rows = common + up(4 * M) + up(4 * P) + up(2 * P * I)
    bf16 = _lib.AITER_DTYPE[torch.bfloat16]
    assert lib.b200_fused_moe_workspace_size(M, H, I, E, topk, 4, bf16) == block
    assert lib.b200_fused_moe_workspace_size(M, H, I, E, topk, 2, bf16) == rows


def test_unsupported_options_are_named():
    x = torch.zeros((4, 256), dtype=torch.bfloat16)
    w1 = torch.zeros((2, 512, 256), dtype=torch.float8_e4m3fn)
    w2 = torch.zeros((2, 256, 256), dtype=torch.float8_e4m3fn)
    tw = torch.ones((4, 1))
    ti = torch.zeros((4, 1), dtype=torch.int32)
    QT, AT = aiter_b200.QuantType, aiter_b200.ActivationType
    with pytest.raises(NotImplementedError, match="quant_type"):
        aiter_b200.fused_moe(x, w1, w2, tw, ti, quant_type=QT.per_1x32)
    with pytest.raises(NotImplementedError, match="activation"):
        aiter_b200.fused_moe(x, w1, w2, tw, ti, quant_type=QT.per_1x128, activation=AT.Swiglu)
    with pytest.raises(NotImplementedError, match="bias1"):
        aiter_b200.fused_moe(x, w1, w2, tw, ti, quant_type=QT.per_1x128, bias1=torch.zeros(1))
    with pytest.raises(NotImplementedError, match="splitk"):
        aiter_b200.fused_moe(x, w1, w2, tw, ti, quant_type=QT.per_128x128, splitk=2)
    with pytest.raises(RuntimeError, match="CUDA"):
        aiter_b200.fused_moe(x, w1, w2, tw, ti, quant_type=QT.per_1x128,
                             w1_scale=torch.ones(1), w2_scale=torch.ones(1))
    with pytest.raises(NotImplementedError, match="flat"):
        aiter_b200.moe_sorting(ti, tw, 2, 256, torch.bfloat16, flat=True)
    with pytest.raises(RuntimeError, match="CUDA"):
        aiter_b200.moe_sorting(ti, tw, 2, 256, torch.bfloat16)


def test_enums_match_reference_values():
    QT, AT = aiter_b200.QuantType, aiter_b200.ActivationType
    assert (AT.No, AT.Silu, AT.Gelu, AT.Swiglu, AT.Situv2) == (-1, 0, 1, 2, 3)
    assert [q.value for q in QT] == list(range(8))
    assert QT.per_1x128 == 4 and QT.per_128x128 == 5


def test_registered_operator_fake_and_shuffle_hook():
    """The torch operator propagates shapes on meta tensors (aiter/fused_moe.py:579-619) and
    shuffle_weight keeps the is_shuffled protocol (aiter/ops/shuffle.py:148-209, aiter/fused_moe.py:747)."""
    x = torch.empty((4, 256), dtype=torch.bfloat16, device="meta")
    w1 = torch.empty((2, 512, 256), dtype=torch.float8_e4m3fn, device="meta")
    w2 = torch.empty((2, 256, 256), dtype=torch.float8_e4m3fn, device="meta")
    tw = torch.empty((4, 1), device="meta")
    ti = torch.empty((4, 1), dtype=torch.int32, device="meta")
    out = torch.ops.aiter_b200.fused_moe_(x, w1, w2, tw, ti, None, 0, 4, False, None, None, None, None, None)
    assert out.shape == (4, 256) and out.dtype == torch.bfloat16
    out = torch.ops.aiter_b200.fused_moe_(x.to(torch.float8_e4m3fn), w1, w2, tw, ti, None, 0, 4, False, None, None,
                                          None, None, torch.float16)
    assert out.dtype == torch.float16
    w = torch.zeros((2, 128, 128), dtype=torch.float8_e4m3fn)
    assert aiter_b200.shuffle_weight(w) is w and w.is_shuffled
    with pytest.raises(NotImplementedError):
        aiter_b200.shuffle_weight(w, use_int4=True)
