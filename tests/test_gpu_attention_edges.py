"""Attention at the edges of its tiling, forward and backward, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(q, k, v):
    ratio = q.shape[2] // k.shape[2]
    q, k, v = q.transpose(1, 2), k.transpose(1, 2).repeat_interleave(ratio, 1), v.transpose(1, 2).repeat_interleave(ratio, 1)
    s = q @ k.transpose(-1, -2) / q.shape[-1] ** 0.5
    s = s.masked_fill(torch.ones_like(s, dtype=torch.bool).triu(1), float("-inf"))
    return (torch.softmax(s, -1) @ v).transpose(1, 2)


@pytest.mark.parametrize("L", [128, 256, 384, 640])          # one tile, a pair, odd numbers of tiles
@pytest.mark.parametrize("Hq,Hkv", [(2, 2), (4, 1)])
@pytest.mark.parametrize("growing", [False, True])           # scores that grow along the keys: rows are rescaled often
def test_attention(L, Hq, Hkv, growing):
    from state_space_models_neuron_b200 import ops
    from state_space_models_neuron_b200.ops import cuda_ops
    gen = torch.Generator(device="cuda").manual_seed(L + Hq)
    make = lambda h: torch.randn(2, L, h, 128, device="cuda", generator=gen)
    q, k, v, do = make(Hq), make(Hkv), make(Hkv), make(Hq).bfloat16()
    if growing:
        q = q.abs() * 0.5
        k = k.abs() * torch.linspace(0.1, 6.0, L, device="cuda")[None, :, None, None]
    q, k, v = (t.bfloat16().requires_grad_() for t in (q, k, v))
    out = ops.attention(q, k, v)
    grads = torch.autograd.grad(out, (q, k, v), do)
    torch.cuda.synchronize()
    cuda_ops.check_status()
    Q, K, V = (t.detach().double().requires_grad_() for t in (q, k, v))
    ref = _reference(Q, K, V)
    want = torch.autograd.grad(ref, (Q, K, V), do.double())
    # P and dS are rounded to bf16 before their products (2^-9 relative each, independent over the sum), results once more
    for a, b in zip((out,) + grads, (ref,) + want):
        assert ((a.double() - b).norm() / b.norm()).item() < 2.0 ** -7
        assert (a.double() - b).abs().max().item() < 2.0 ** -4 * b.abs().max().item()
