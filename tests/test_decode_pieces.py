"""The decode attention of a layer-listed model with its keys in one, two, four and eight pieces."""
import pytest

import vunasun_models as vm
from test_vunasun_parity import DTYPES, built, check, exact, feed          # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("size, pieces", [(60, 1), (128, 2), (256, 4), (500, 8), (700, 8)])
def test_decode_attention_in_pieces(size, pieces, dtype):
    """Steps where all pieces but the first are empty, where the last key begins a piece, and across the edge of a chunk."""
    from megaqwen_b200.hybrid import HybridDecoder
    cfg = vm.config([(vm.attention(4, 2, 64, 32, size), None), (vm.attention(6, 1, 128, 64, size), 48)], width=64)
    w = vm.weights(cfg, 3)
    tiles = (min(size, 720) + 63) // 64
    assert pieces == (8 if tiles >= 8 else 4 if tiles >= 4 else 2 if tiles >= 2 else 1)
    dec = HybridDecoder(w, 720, 720, dtype=dtype)
    ids = vm.tokens(cfg, 715, 4)
    want = exact(cfg, w, ids)
    for start in sorted({0, 62, 127, size - 3, 2 * size - 2, 700}):
        if start + 6 > len(ids) or start < 0:
            continue
        got = feed(dec, ids[:start + 6], [start] if start else [])
        check(got[start:], want[start:start + 6], dtype, f"steps from {start}")
