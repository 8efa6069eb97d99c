"""Kernels that may start before their predecessors have finished read only with ordinary loads behind the wait."""
import os
import re

from state_space_models_neuron_b200.ops import native


def _kernels(source):
    """(name, parameters, body) of every __global__ function."""
    for m in re.finditer(r"__global__ void (?:__launch_bounds__\([^{;]*?\)\s+)?(\w+)\(([^{;]*?)\)\s*\{", source):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(source[i], 0)
            i += 1
        yield m.group(1), m.group(2), source[m.end():i]


def test_no_read_only_loads_in_dependent_kernels():
    seen = []
    for name in sorted(os.listdir(native.CSRC)):
        if not name.endswith(".cu"):
            continue
        with open(os.path.join(native.CSRC, name)) as f:
            source = re.sub(r"//.*", "", f.read())
        for kernel, parameters, body in _kernels(source):
            if "pdl_wait()" not in body:
                continue
            seen.append(kernel)
            for p in parameters.split(","):
                assert not ("const" in p and "__restrict__" in p), (kernel, p)
            assert "ld.global.nc" not in source and "__ldg" not in body, kernel
    assert {"gemm_rows_kernel", "gemm_cols_kernel", "decode_mixer_kernel", "decode_ssm_step_kernel", "decode_conv_step_kernel",
            "gated_rmsnorm_fwd_kernel", "add_rmsnorm_fwd_kernel", "norm_linear_kernel"} <= set(seen)
