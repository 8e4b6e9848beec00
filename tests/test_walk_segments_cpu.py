"""The rule that cuts sequences for the chunk walks: whole chunks, every token in a segment, no empty segment, one SM for each."""
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
