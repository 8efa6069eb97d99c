"""Gradient norm delivered by the kernels that write the gradients, the embedding's additions among them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tied", [True, False])
@pytest.mark.parametrize("ids_below", [512, 3, 1])           # spread, many equal ids, all equal
@pytest.mark.parametrize("passes", [1, 2])                   # stored, and accumulated over two backward passes
@pytest.mark.parametrize("vocab", [4096, 512])               # more and fewer than six rows per token
def test_norm_follows_the_embedding(tied, ids_below, passes, vocab):
    from state_space_models_neuron_b200 import parallel as nxd
    from state_space_models_neuron_b200.models import Mamba2Config, Mamba2ForCausalLM
    from state_space_models_neuron_b200.parallel import state as ps
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(1)
    cfg = nxd.parallel_config(1, {"zero_one_enabled": True}, init_seed=3)
    mc = Mamba2Config(num_heads=8, head_dim=64, vocab_size=vocab, hidden_size=256, state_size=128, num_hidden_layers=1, n_groups=1,
                      tie_word_embeddings=tied, initializer_range=0.02, dtype=torch.bfloat16)
    model = nxd.initialize_parallel_model(cfg, lambda: Mamba2ForCausalLM(mc, device="cuda").to(torch.bfloat16))
    opt = nxd.initialize_parallel_optimizer(cfg, nxd.AdamW_FP32OptimParams, [{"params": list(model.parameters())}], lr=1e-3)
    weight, follows = model.backbone.embeddings.weight, vocab >= 6 * 512
    for seed in range(2):
        opt.zero_grad()
        for k in range(passes):
            ids = torch.randint(0, ids_below, (2, 256), device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed + 7 * k))
            model(input_ids=ids, labels=ids, return_logits=False).loss.backward()
        # additions on top of stored gradients are followed; a product that accumulates is not, and the buffers are read instead
        assert weight.norm_tracked == (follows and (passes == 1 or not tied))
        total = opt._grad_norm_sq(opt.flat_grads).item()
        want = opt.flat_grads.double().square().sum().item()
        # fp32 sums of up to 2^18 squares in trees of threads, warps and blocks
        assert abs(total - want) <= 2e-5 * want
