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


def test_largest_probability_is_exact():
    """A row's largest probability is 1 before the division by the row sum, wherever the maximum stands: with it alone against
    a key whose value is zero, the result is rounded once."""
    from state_space_models_neuron_b200 import ops
    L, late = 384, 133
    gen = torch.Generator(device="cuda").manual_seed(5)
    q, k = torch.zeros(1, L, 1, 128, device="cuda"), torch.zeros(1, L, 1, 128, device="cuda")
    q[..., 0] = 8 + 8 * torch.rand(1, L, 1, device="cuda", generator=gen)
    k[..., 0] = -512.0                                        # scores below -350: nothing of these keys is left
    k[0, 0], k[0, late, 0, 0] = 0.0, 3.5                      # 0, and 2.5 to 5 from the second key tile on
    v = torch.randn(1, L, 1, 128, device="cuda", generator=gen).bfloat16()
    v[0, 0] = 0
    q, k = q.bfloat16(), k.bfloat16()
    out = ops.attention(q, k, v)[0, late:, 0].double()
    p = torch.sigmoid(q[0, late:, 0, :1].double() * 3.5 / 128 ** 0.5)
    want = p * v[0, late, 0].double()
    # half a bf16 step, and the fp32 exponential and division (2^-20 together)
    assert ((out - want).abs() <= (2.0 ** -9 + 2.0 ** -20) * 2.0 * want.abs()).all()
    # half a step is 2^-9 of the largest value with the same exponent, 2^-8 of the smallest: the mean tells the roundings apart
    assert ((out - want).norm() / want.norm()).item() < 1.1 * ((want.bfloat16().double() - want).norm() / want.norm()).item()


def test_nan_reaches_the_rows_that_see_it():
    from state_space_models_neuron_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(6)
    q, k, v = (torch.randn(1, 384, 2, 128, device="cuda", generator=gen).bfloat16() for _ in range(3))
    clean = ops.attention(q, k, v)
    k[0, 200, 1, 5] = float("nan")
    out = ops.attention(q, k, v)
    assert torch.equal(out[:, :, 0], clean[:, :, 0]) and torch.equal(out[:, :200], clean[:, :200])
    assert torch.isnan(out[:, 200:, 1]).all()
