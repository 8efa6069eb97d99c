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


def _block_parts(width=64, H=2, P=64, N=128):
    C, W = H * P + 2 * N, 2 * H * P + 2 * N + H
    make = lambda *s: torch.zeros(*s, dtype=torch.bfloat16)
    weights = dict(norm_w=make(width), in_w=make(W, width), in_b=make(W), conv_w=make(C, 1, 4), conv_b=make(C), dt_bias=make(H),
                   A_log=make(H), D=make(H), gate_w=make(H * P), out_w=make(width, H * P))
    return weights, make(1, C, 4), torch.zeros(1, H, P, N)


class _Elsewhere(torch.Tensor):
    """A tensor that answers as one of another device."""

    def get_device(self):
        return 1


def test_blocks_by_one_call_keep_to_one_device():
    """Addresses are passed on only where every tensor lies on the rows' device."""
    weights, window, state = _block_parts()
    here = window.get_device()
    given = lambda **kw: cuda_ops._block_weights(here, 64, 128, 1, 128, 64, 128, **{**weights, **kw})
    assert given() is not None and cuda_ops._block_states(here, 1, 384, 2, 64, 128, window, state) is not None
    for name, t in weights.items():
        assert given(**{name: t.as_subclass(_Elsewhere)}) is None, name
    assert cuda_ops._block_weights(0, 64, 128, 1, 128, 64, 128, **weights) is None
    assert cuda_ops._block_states(here, 1, 384, 2, 64, 128, window.as_subclass(_Elsewhere), state) is None
    assert cuda_ops._block_states(here, 1, 384, 2, 64, 128, window, state.as_subclass(_Elsewhere)) is None
    assert cuda_ops._block_states(0, 1, 384, 2, 64, 128, window, state) is None
    hidden = torch.zeros(1, 1, 64, dtype=torch.bfloat16)
    assert cuda_ops._block_rows(hidden, hidden.clone(), torch.bfloat16) is not None
    assert cuda_ops._block_rows(hidden, hidden.as_subclass(_Elsewhere), torch.bfloat16) is None


@pytest.mark.parametrize("module,name", [("norm", "weight"), ("mixer.conv1d", "weight"), ("mixer.conv1d", "bias"), ("mixer", "D"),
                                         ("mixer.norm", "weight"), ("mixer.in_proj", "weight"), ("mixer.out_proj", "weight"),
                                         ("mixer.out_proj", "bias")])
def test_blocks_by_one_call_want_plain_parameters(module, name):
    """A weight that is no parameter of its module (computed by a parametrisation or a pruning mask) keeps the calls one by one."""
    from state_space_models_neuron_b200.models import Mamba2Config
    from state_space_models_neuron_b200.models.modeling_mamba2 import Mamba2Block
    from state_space_models_neuron_b200.parallel import state as ps
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(1)
    cfg = Mamba2Config(num_heads=2, head_dim=64, vocab_size=64, hidden_size=64, state_size=128, num_hidden_layers=1, n_groups=1)
    block = Mamba2Block(cfg, 0)
    op = lambda *a: "one call"
    assert block._in_one_call(op, "step", None, None, None, None, None) == "one call"
    owner = block.get_submodule(module)
    value = getattr(owner, name)
    delattr(owner, name)
    setattr(owner, name, None if value is None else value.detach())
    assert block._in_one_call(op, "step", None, None, None, None, None) is None


@pytest.mark.parametrize("taps", [1, 2, 3, 5])
def test_other_numbers_of_taps_are_refused(taps):
    """The conv kernels read four taps per channel: any other weight is refused before a launch, in the mixer as in the conv itself."""
    H, P, N, L = 2, 64, 128, 128
    d, C = H * P, H * P + 2 * N
    make = lambda *s: torch.zeros(*s, dtype=torch.bfloat16)
    for cached in (False, True):
        with torch.no_grad(), pytest.raises(ValueError, match="taps"):
            cuda_ops.mamba2_mixer_core(make(1, L, d + C + H), make(C, 1, taps), make(C), make(H), make(H), make(H), make(d), d, 1, N, P,
                                       1e-5, None, 128, False, cached)
    with torch.no_grad(), pytest.raises(ValueError, match="taps"):
        cuda_ops.causal_conv1d_silu(make(1, L, C), make(C, 1, taps), make(C))
    with torch.no_grad(), pytest.raises(ValueError, match="taps"):         # four taps of fewer channels
        cuda_ops.causal_conv1d_silu(make(1, L, C), make(C // 2, 1, 4), make(C))


@pytest.mark.parametrize("where,name", [("Mamba2Mixer", "forward"), ("Mamba2Mixer", "step"), ("Mamba2Mixer", "_core_kwargs"),
                                        ("Mamba2Mixer", "__call__"), ("Mamba2RMSNorm", "forward_add"), ("ColumnParallelLinear", "forward"),
                                        ("RowParallelLinear", "forward"), ("RowParallelLinear", "__call__"), ("ops", "linear"),
                                        ("ops", "add_rmsnorm"), ("ops", "ssm_decode_step"), ("ops", "mamba2_mixer_core")])
def test_blocks_by_one_call_see_methods_replaced_on_classes(monkeypatch, where, name):
    """A method that a program or a test has set on a class, or an operation set in the package, is called as before."""
    from state_space_models_neuron_b200.models import Mamba2Config, modeling_mamba2
    from state_space_models_neuron_b200.parallel import state as ps
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(1)
    cfg = Mamba2Config(num_heads=2, head_dim=64, vocab_size=64, hidden_size=64, state_size=128, num_hidden_layers=1, n_groups=1)
    block = modeling_mamba2.Mamba2Block(cfg, 0)
    op = lambda *a: "one call"
    assert block._in_one_call(op, "step", None, None, None, None, None) == "one call"
    owner = getattr(modeling_mamba2, where)
    plain = getattr(owner, name)
    monkeypatch.setattr(owner, name, lambda *a, **kw: plain(*a, **kw))
    assert block._in_one_call(op, "step", None, None, None, None, None) is None
    monkeypatch.undo()
    assert block._in_one_call(op, "step", None, None, None, None, None) == "one call"


@pytest.mark.parametrize("batch", [0, 1, 7, 9, 130])
def test_cache_pieces(monkeypatch, batch):
    """Layers share memory in pieces of a limited size; a state above it has memory of its own."""
    from state_space_models_neuron_b200.models import Mamba2Cache, Mamba2Config, cache
    from state_space_models_neuron_b200.parallel import state as ps
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(1)
    monkeypatch.setattr(cache, "_PIECE", 1 << 20)
    cfg = Mamba2Config(num_heads=2, head_dim=64, vocab_size=64, hidden_size=64, state_size=128, num_hidden_layers=5, n_groups=1)
    c = Mamba2Cache(cfg, batch, dtype=torch.bfloat16)
    for states, shape in ((c.conv_states, (batch, 384, 4)), (c.ssm_states, (batch, 2, 64, 128))):
        assert list(states) == list(range(5))
        for i, t in states.items():
            assert tuple(t.shape) == shape and t.is_contiguous() and not t.any()
            assert t.untyped_storage().nbytes() <= max(1 << 20, t.numel() * t.element_size())
            version = states[(i + 1) % 5]._version
            t.fill_(i + 1)
            assert states[(i + 1) % 5]._version == version
        assert all(torch.equal(t, torch.full_like(t, i + 1)) for i, t in states.items())
