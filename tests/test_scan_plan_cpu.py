"""Head slices per CTA of the backward scan."""
import pytest

from state_space_models_neuron_b200.ops.cuda_ops import _PER_CHUNK, _pick_hpc, _segments, _walk_cost, _walk_states

GROUPS, CHUNKS = (1, 2, 3, 7, 8, 16, 24, 40, 48, 64, 80, 128), (1, 9, 16, 64, 128, 147, 148, 149, 256, 295, 296, 384, 512, 4096)


def test_divides_and_never_takes_more_waves_than_one_head_each():
    for group in GROUPS:
        for chunks in CHUNKS:
            hpc = _pick_hpc(group, chunks)
            assert 1 <= hpc <= group and group % hpc == 0
            assert -(-chunks * (group // hpc) // 148) <= -(-chunks * group // 148)
            assert hpc == 1 or chunks * group > 148              # heads are walked only when CTAs would queue
    assert _pick_hpc(80, 64) == 40 and _pick_hpc(16, 128) == 16 and _pick_hpc(16, 16) == 2


@pytest.mark.parametrize("group", GROUPS)
def test_sums_of_at_most_two_where_that_fills_the_chip(group):
    """More than two CTAs per group add to dB and dC in an order that changes from run to run."""
    for chunks in CHUNKS:
        if chunks >= 296 or (chunks >= 148 and group % 2 == 0):
            assert group // _pick_hpc(group, chunks) <= 2


def test_segments_are_never_empty_and_never_cost_more():
    for slices in (1, 8, 24, 32, 43, 44, 64, 96, 148, 149, 160, 320, 1280):
        for nc in (1, 2, 3, 4, 5, 8, 9, 16, 63, 64, 65, 256, 512):
            for per_chunk in _PER_CHUNK:
                count = _segments(slices, nc, per_chunk)
                assert 1 <= count <= min(32, nc) and (count - 1) * -(-nc // count) < nc
                assert _walk_cost(slices, nc, count, per_chunk) <= _walk_cost(slices, nc, 1, per_chunk)
            assert _walk_states(slices, nc) or (nc > 4 and slices * nc <= 512)       # a CTA per chunk for few chunks in all
