"""forward(labels=...) on the GPU: what hangs on the returned logits, and heads other than the plain one."""
import pytest
import torch

pytestmark = pytest.mark.gpu
V = 512


def _model(hybrid=False):
    from state_space_models_neuron_b200.models import Mamba2Config, Mamba2ForCausalLM, Mamba2HybridConfig, Mamba2HybridForCausalLM
    from state_space_models_neuron_b200.parallel import state as ps
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(1)
    kw = dict(num_heads=8, head_dim=64, vocab_size=V, hidden_size=256, state_size=128, n_groups=1, initializer_range=0.02,
              dtype=torch.bfloat16)
    if hybrid:
        cfg, build = Mamba2HybridConfig(num_hidden_layers=2, hybrid_override_pattern="M-", mlp_hidden_size=512, **kw), Mamba2HybridForCausalLM
    else:
        cfg, build = Mamba2Config(num_hidden_layers=1, **kw), Mamba2ForCausalLM
    return build(cfg, device="cuda").to(torch.bfloat16)


def _ids():
    ids = torch.randint(0, V, (2, 128), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    labels = ids.clone()
    labels[0, 5:9] = -100
    return ids, labels


def _loss_of(logits, labels):
    valid = labels[:, 1:].numel()
    return torch.nn.functional.cross_entropy(logits[:, :-1].reshape(-1, V), labels[:, 1:].reshape(-1), reduction="sum") / valid


@pytest.mark.parametrize("hybrid", [False, True])
def test_loss_hangs_on_the_logits(hybrid):
    model, (ids, labels) = _model(hybrid), _ids()
    out = model(input_ids=ids, labels=labels)
    seen = []
    out.logits.retain_grad()
    out.logits.register_hook(seen.append)
    out.loss.backward(retain_graph=True)
    leaf = out.logits.detach().double().requires_grad_()
    want, = torch.autograd.grad(_loss_of(leaf, labels), leaf)
    got = out.logits.grad
    # fp32 exponentials and one subtraction from a probability of at most 1
    assert got.dtype == torch.float32 and (got.double() - want).abs().max() <= 1e-5 * want.abs().max()
    assert len(seen) == 1 and torch.equal(seen[0], got)
    # a loss of the caller's own on the same logits: the two gradients meet in fp32, and are rounded to bf16 once
    w = model.lm_head.weight
    own = (out.logits * want.float().neg()).sum()
    both, = torch.autograd.grad(out.loss + own, w)
    alone, = torch.autograd.grad(_loss_of(model(input_ids=ids).logits, labels), w)
    assert both.float().norm() <= 1e-3 * alone.float().norm()


@pytest.mark.parametrize("head", ["linear", "bias", "gathered", "subclass", "hook", "forward"])
@pytest.mark.parametrize("grad", [True, False])
def test_other_heads(head, grad):
    from state_space_models_neuron_b200.parallel.layers import ColumnParallelLinear
    model, (ids, labels) = _model(), _ids()
    seen = []
    if head == "linear":
        model.set_output_embeddings(torch.nn.Linear(256, V, device="cuda", dtype=torch.bfloat16))
    elif head in ("bias", "gathered"):
        model.set_output_embeddings(ColumnParallelLinear(256, V, bias=head == "bias", gather_output=head == "gathered",
                                                         dtype=torch.bfloat16, device="cuda"))
    elif head == "subclass":
        class Scaled(ColumnParallelLinear):
            def forward(self, x):
                return 2 * super().forward(x)
        model.set_output_embeddings(Scaled(256, V, dtype=torch.bfloat16, device="cuda"))
    elif head == "hook":
        model.lm_head.register_forward_hook(lambda m, args, out: seen.append(out))
    else:
        plain = model.lm_head.forward
        model.lm_head.forward = lambda x: plain(x) + 1
    with torch.set_grad_enabled(grad):
        out = model(input_ids=ids, labels=labels)
    want = _loss_of(out.logits.detach().double(), labels)
    assert out.logits.shape == (2, 128, V) and out.logits.dtype == torch.float32
    assert abs(out.loss.item() - want.item()) <= 1e-5 * abs(want.item())
    assert out.loss.requires_grad == grad
    if head == "hook":
        assert len(seen) == 1 and torch.is_tensor(seen[0]) and torch.equal(seen[0].float(), out.logits)
