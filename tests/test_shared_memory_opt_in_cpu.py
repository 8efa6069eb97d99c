"""Every device keeps a kernel's opt-in to large shared memory for itself: no flag of the process stands for all of them."""
import os
import re

from state_space_models_neuron_b200.ops import native


def test_opt_in_goes_by_device():
    calls = []
    for name in sorted(os.listdir(native.CSRC)):
        if name.endswith((".cu", ".cuh", ".h")):
            with open(os.path.join(native.CSRC, name)) as f:
                source = re.sub(r"//.*", "", f.read())
            calls += [name] * len(re.findall(r"cudaFuncSetAttribute\(", source))
            assert not re.findall(r"static bool \w+ = false", source), name
    assert calls == ["common.cuh"]             # SmemOptIn, which asks once per device
