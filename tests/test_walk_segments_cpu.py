"""Rules of the chunk walks.  Segments: whole chunks, every token in one, none empty, one SM for each.  Batches left to one launch:
those of measured shapes on the right side of the line."""
import pytest

from b200attn import hybrid_ops


@pytest.mark.parametrize("chunk", [16, 32])
@pytest.mark.parametrize("groups", [1, 16, 64, 74, 148, 4096])
@pytest.mark.parametrize("length", [1, 33, 255, 256, 257, 1000, 4096, 32768])
def test_outer_walk_segments(length, groups, chunk):
    segment, count = hybrid_ops.outer_walk_segments(length, groups, 148, chunk)
    assert (count - 1) * segment < length <= count * segment
    if count > 1:
        assert segment % chunk == 0 and segment >= 128 and count * groups <= 148


@pytest.mark.parametrize("lengths,heads,outer,ssd", [
    ([33] + [16] * 31, 16, True, True), ([64] + [1] * 63, 16, True, True), ([48] + [8] * 127, 16, True, True),
    ([160] + [16] * 63, 16, False, True), ([33] + [32] * 31, 16, False, True),
    ([33] + [16] * 15, 16, False, False), ([33] * 32, 16, False, False), ([1024] + [16] * 31, 16, False, False),
    ([128] + [32] * 7, 16, False, False), ([256] + [1] * 63, 16, False, False), ([2048], 32, False, False)])
def test_batches_left_to_one_launch(lengths, heads, outer, ssd):
    args = sum(lengths), len(lengths), max(lengths), len(lengths) * heads, 148
    assert hybrid_ops.mostly_one_chunk(*args, 16, 16, 64) == outer
    assert hybrid_ops.mostly_one_chunk(*args, 32, 28, max(lengths)) == ssd
