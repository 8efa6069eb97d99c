"""`cuda_ops._apply`: the forward alone where autograd records nothing, the autograd Function everywhere else."""
import pytest
import torch

from state_space_models_neuron_b200.ops import cuda_ops


class _Double(torch.autograd.Function):
    contexts = []

    @staticmethod
    def forward(ctx, x):
        _Double.contexts.append(type(ctx).__name__)
        ctx.save_for_backward(x)
        ctx.factor = 2
        return x * ctx.factor

    @staticmethod
    def backward(ctx, g):
        return g * ctx.factor


def _ran_bare(fn):
    _Double.contexts.clear()
    out = fn()
    return _Double.contexts == ["_NoGrad"], out


def test_forward_alone_without_grad():
    x = torch.ones(3, requires_grad=True)
    for mode in (torch.no_grad(), torch.inference_mode()):
        with mode:
            bare, y = _ran_bare(lambda: cuda_ops._apply(_Double, x))
        assert bare and not y.requires_grad and torch.equal(y, torch.full((3,), 2.0))


def test_function_where_something_may_record():
    x = torch.ones(3, requires_grad=True)
    bare, y = _ran_bare(lambda: cuda_ops._apply(_Double, x))
    assert not bare
    y.sum().backward()
    assert torch.equal(x.grad, torch.full((3,), 2.0))
    with torch.no_grad():
        with torch.autograd.forward_ad.dual_level():
            dual = torch.autograd.forward_ad.make_dual(torch.ones(3), torch.ones(3))
            _Double.contexts.clear()
            try:
                cuda_ops._apply(_Double, dual)
            except (NotImplementedError, RuntimeError):      # the Function's own answer where it has no jvp
                pass
            assert "_NoGrad" not in _Double.contexts
        with pytest.raises(RuntimeError):                     # no vmap rule: refused, as before
            torch.vmap(lambda t: cuda_ops._apply(_Double, t))(torch.ones(2, 3))


class _Filled(torch.autograd.Function):
    """As the kernels: the output is made inside and filled through its address."""

    @staticmethod
    def forward(ctx, x):
        out = torch.empty_like(x)
        out.numpy()[:] = 2 * x.numpy()
        return out

    @staticmethod
    def backward(ctx, g):
        return 2 * g


def test_traced_without_grad():
    with torch.no_grad():
        traced = torch.jit.trace(lambda x: cuda_ops._apply(_Filled, x) + 1, torch.ones(4), check_trace=False)
        assert torch.equal(traced(torch.full((4,), 5.0)), torch.full((4,), 11.0))
        # the widening of logits takes the operation that a tracer can record
        traced = torch.jit.trace(lambda x: cuda_ops.widen(x) + 1, torch.ones(2, 8).bfloat16(), check_trace=False)
        assert torch.equal(traced(torch.full((2, 8), 5.0).bfloat16()), torch.full((2, 8), 6.0))
