"""Prefill into caches whose tensors a program has made itself."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model_and_ids(B=2):
    from state_space_models_neuron_b200.models import Mamba2Config, Mamba2ForCausalLM
    from state_space_models_neuron_b200.parallel import state as ps
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(1)
    cfg = Mamba2Config(num_heads=8, head_dim=64, vocab_size=512, hidden_size=256, state_size=128, num_hidden_layers=2,
                       n_groups=1, initializer_range=0.02, dtype=torch.bfloat16)
    model = Mamba2ForCausalLM(cfg, device="cuda").to(torch.bfloat16).eval()
    return model, torch.randint(0, 512, (B, 256), device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))


@pytest.mark.parametrize("offset", [1, 2, 3, 4])               # elements of the windows behind a 16-byte boundary
@pytest.mark.parametrize("shift_state", [0, 1])
def test_cache_tensors_anywhere_in_memory(offset, shift_state):
    from state_space_models_neuron_b200.models import Mamba2Cache
    model, ids = _model_and_ids()
    want, plain = model.prefill(ids)
    cache = Mamba2Cache(model.config, 2, dtype=torch.bfloat16, device="cuda")
    for states, off in ((cache.conv_states, offset), (cache.ssm_states, shift_state)):
        for k, t in states.items():
            states[k] = torch.zeros(t.numel() + off, dtype=t.dtype, device="cuda")[off:].view(t.shape)
    logits, same = model.prefill(ids, cache)
    torch.cuda.synchronize()
    assert same is cache and torch.equal(logits, want)
    for k in plain.conv_states:
        assert torch.equal(cache.conv_states[k], plain.conv_states[k]) and torch.equal(cache.ssm_states[k], plain.ssm_states[k])


def test_gradient_through_an_overwritten_state_is_refused():
    model, ids = _model_and_ids()
    _, cache = model.prefill(ids)
    for states in (cache.conv_states, cache.ssm_states):
        scale = torch.ones((), device="cuda", requires_grad=True)
        y = (scale.to(states[1].dtype) * states[1]).sum()       # saves the state
        model.prefill(ids.flip(1), cache)
        with pytest.raises(RuntimeError, match="modified by an inplace operation"):
            y.backward()
