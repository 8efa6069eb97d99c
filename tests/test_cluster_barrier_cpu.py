"""Cluster barriers are of the aligned form: all threads of a warp execute them together, also behind a branch for one thread."""
import os
import re

from state_space_models_neuron_b200.ops import native


def test_warps_converge_in_front_of_aligned_cluster_barriers():
    found = 0
    for name in sorted(os.listdir(native.CSRC)):
        if name.endswith((".cu", ".cuh", ".h")):
            with open(os.path.join(native.CSRC, name)) as f:
                source = re.sub(r"//.*", "", f.read())
            for m in re.finditer(r"barrier\.cluster\.arrive[\w.]*\.aligned", source):
                found += 1
                statements = [s.strip() for s in source[:m.start()].split(";")]
                assert statements[-2].endswith("__syncwarp()"), name
    assert found == 1              # the one helper that all kernels call
