"""Rules by which launches choose a kernel or a split, at the sizes that they were measured at (no GPU)."""
import pytest

from sglang_c_b200.csrc import ops


@pytest.mark.parametrize("keys,blocks,width,splits", [
    (64, 24, 128, 1), (128, 24, 128, 5), (256, 24, 128, 9), (512, 24, 128, 16), (1024, 24, 128, 16), (100, 96, 128, 4),
    (512, 48, 128, 8), (256, 64, 128, 4), (100, 128, 128, 2), (512, 32, 48, 8), (2000, 48, 128, 9), (128, 384, 128, 1),
    (100, 16, 256, 5), (512, 16, 256, 8), (256, 32, 256, 4), (100, 64, 256, 2)])
def test_a_tile_a_share_only_where_every_tile_has_one(keys, blocks, width, splits):
    assert ops.attention_ext_splits(keys, None, None, blocks, width) == splits
    assert ops.attention_ext_splits(4 * keys, keys, None, blocks, width) == splits          # (a window)
    assert ops.attention_ext_splits(4 * keys, None, keys, blocks, width) == splits          # (a chunk)
