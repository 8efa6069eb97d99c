"""Decode cache: per layer a rolling conv window and the SSM state.

Field names and shapes follow the `Mamba2Cache` of transformers 4.46 that the reference imports
(mamba2/mamba2_mixer.py:23) and the layouts its decode kernel uses
(mamba2/mamba2_kernel_inference.py:36-43): `conv_states[layer]` is `[B, conv_dim, K]` (oldest token
first), `ssm_states[layer]` is `[B, H, P, N]`; sizes are per tensor-parallel rank.
"""
from __future__ import annotations

import math
from typing import Optional

import torch

from ..parallel import state as ps


_PIECE = 64 << 20


def _zeros(count: int, shape, dtype, device):
    """`count` zero tensors of one shape.  Small ones whose sizes are whole 16-byte vectors share allocations and fills of at most
    64 MB (48 fills took 250 us of the host in front of a prompt through 24 layers); larger ones have one each, so that a cache needs
    no more memory in one piece than a layer's state, and a layer's state that is kept holds no more than that.  Each has a version
    counter of its own."""
    size = math.prod(shape) * dtype.itemsize
    each = _PIECE // size if size and size % 16 == 0 else 1
    if each < 2:
        return [torch.zeros(shape, device=device, dtype=dtype) for _ in range(count)]
    return [t.data for first in range(0, count, each)
            for t in torch.zeros((min(each, count - first), *shape), device=device, dtype=dtype).unbind(0)]


class Mamba2Cache:
    def __init__(self, config, batch_size: int, dtype: torch.dtype = torch.float16,
                 device: Optional[torch.device] = None, ssm_dtype: torch.dtype = torch.float32,
                 layer_indices=None):
        tp = ps.get_tensor_model_parallel_size()
        self.dtype = dtype
        self.seqlen_offset = 0
        self.conv_kernel_size = config.conv_kernel
        conv_dim = (config.intermediate_size + 2 * config.n_groups * config.state_size) // tp
        heads = config.num_heads // tp
        layers = range(config.num_hidden_layers) if layer_indices is None else layer_indices
        layers = list(layers)
        self.conv_states = dict(zip(layers, _zeros(len(layers), (batch_size, conv_dim, config.conv_kernel), dtype, device)))
        self.ssm_states = dict(zip(layers, _zeros(len(layers), (batch_size, heads, config.head_dim, config.state_size), ssm_dtype,
                                                  device)))

    def update_conv_state(self, layer_idx: int, new_conv_state: torch.Tensor) -> torch.Tensor:
        self.conv_states[layer_idx].copy_(new_conv_state.to(self.conv_states[layer_idx].dtype))
        return self.conv_states[layer_idx]

    def update_ssm_state(self, layer_idx: int, new_ssm_state: torch.Tensor) -> torch.Tensor:
        self.ssm_states[layer_idx].copy_(new_ssm_state.to(self.ssm_states[layer_idx].dtype))
        return self.ssm_states[layer_idx]

    def reset(self) -> None:
        self.seqlen_offset = 0
        for t in list(self.conv_states.values()) + list(self.ssm_states.values()):
            t.zero_()
