"""The rule that picks the MXFP4 kernel of a call (mx_tile_tokens, prefill_mx8.cu): tiles of 32 tokens on fp8 pieces or of 128
on bf16 pieces, on the side that both were measured on. No device."""
import pytest

import pelica_b200 as pb

FP8, BF16 = 32, 128


@pytest.fixture(scope="module")
def tile():
    return pb.load_library().pm_debug_mx_tile_tokens


@pytest.mark.parametrize("groups,ff,pairs,want", [
    (32, 2880, 48, FP8), (32, 2880, 64, FP8), (32, 2880, 65, BF16), (32, 2880, 80, BF16), (32, 2880, 88, BF16),
    (24, 2880, 56, FP8), (24, 2880, 72, BF16), (64, 1024, 56, FP8), (64, 1024, 80, BF16), (128, 2880, 56, FP8),
    (128, 2880, 72, BF16), (16, 4096, 60, FP8), (16, 4096, 70, BF16), (32, 512, 72, BF16),
    # few tiles of 128 tokens: a third and more of the SMs would have no work
    (4, 2880, 88, FP8), (8, 2880, 88, FP8), (8, 1024, 88, FP8), (8, 2880, 89, BF16), (16, 2880, 80, FP8)])
def test_line(tile, groups, ff, pairs, want):
    assert tile(groups * pairs // 2, groups * pairs, groups, ff) == want


def test_short_calls_keep_every_bit(tile):
    assert all(tile(t, 4 * t, 1, 2880) == 16 for t in (1, 8, 31))
    assert tile(32, 128, 32, 2880) == FP8
    assert tile(40, 3, 8, 2880) == FP8  # fewer pairs than groups
    assert tile(0, 1, 1, 32) == tile(1, 0, 1, 32) == tile(1, 1, 0, 32) == tile(1, 1, 1, 0) == 0
