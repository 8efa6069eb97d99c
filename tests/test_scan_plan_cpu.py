"""Head slices per CTA of the backward scan."""
from state_space_models_neuron_b200.ops.cuda_ops import _pick_hpc


def test_divides_and_never_takes_more_waves_than_one_head_each():
    for group in (1, 2, 3, 7, 8, 16, 24, 80, 128):
        for chunks in (1, 9, 16, 64, 128, 147, 148, 149, 512, 4096):
            hpc = _pick_hpc(group, chunks)
            assert group % hpc == 0
            cost = lambda h: -(-chunks * (group // h) // 148) * (h + 1.5)
            assert all(cost(hpc) <= cost(h) for h in range(1, group + 1) if group % h == 0)
    assert _pick_hpc(80, 64) == 40 and _pick_hpc(16, 128) == 16 and _pick_hpc(16, 16) == 2
