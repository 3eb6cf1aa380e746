"""The tests of test_gpu_pairs.py with the pairs asked for: its small layers, at the edges of blocks and tiles, are otherwise below the
size from which a layer is worked in pairs."""

import importlib

import pytest

from aiter_b200 import _lib
from test_gpu_pairs import (test_many_tiles_per_pair_of_ctas, test_masked_and_padded_batches, test_pairs_equal_single_blocks,  # noqa: F401
                            test_waits_of_a_pair_run_out)

fm = importlib.import_module("aiter_b200.fused_moe")
pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def pairs(monkeypatch):
    """Asks for pairs and sees that every layer call could have them."""
    asked, sizes_of = [], fm._layer_sizes.__wrapped__
    monkeypatch.setattr(fm, "_layer_sizes", lambda *sizes: asked.append(sizes) or sizes_of(*sizes))
    _lib.call_plain("b200_moe_debug_pairs", 1)
    yield
    counts = []
    for mode in (1, 2, 0):
        _lib.call_plain("b200_moe_debug_pairs", mode)
        counts.append([sizes_of(*sizes)[1] for sizes in asked])
    assert asked and all(a > b for a, b in zip(counts[0], counts[1]))
