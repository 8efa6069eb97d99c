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


# columns in one, four and more than four vectors per thread (256 threads of four values), more tokens than blocks, equal ids, ids of
# other ranks' rows
@pytest.mark.parametrize("D", [256, 1028, 4096, 5120, 8196])
@pytest.mark.parametrize("tokens", [1, 1300])
def test_additions_carry_the_norm_on(D, tokens):
    from state_space_models_neuron_b200.ops import cuda_ops as co
    gen = torch.Generator(device="cuda").manual_seed(D + tokens)
    rows = 96
    grad = torch.randn(rows, D, device="cuda", generator=gen)
    want = grad.double()
    norm = want.square().sum().float().reshape(1)
    moved = want.square().sum()                             # of all terms that enter the sum, without their signs
    for _ in range(2):
        ids = torch.randint(-3, rows + 3, (tokens,), device="cuda", generator=gen)
        g = torch.randn(tokens, D, device="cuda", generator=gen).bfloat16()
        co._run("ssm_embed_bwd", co._P(ids), co._P(g), co._ll(D), co._P(grad), co._ll(0), co._ll(rows), 1, tokens, tokens, D, 1, None, 0, 0,
                None, co._P(norm), co._P(co.status_tensor(grad.device)), co._st())
        mine = (ids >= 0) & (ids < rows)
        old, want = want, want.index_add(0, ids[mine], g[mine].double())
        moved = moved + (g[mine].double().abs() * (2 * torch.maximum(old.abs(), want.abs())[ids[mine]] + g[mine].double().abs())).sum()
    co.check_status()
    assert torch.allclose(grad.double(), want, rtol=0, atol=2.0 ** -24 * 64 * want.abs().max().item())     # up to 40 additions to a value
    # chains of about 100 additions per thread and of a few thousand to the accumulator, which round to either side
    assert abs(norm.item() - want.square().sum().item()) <= 2.0 ** -24 * 64 * moved.item()


@pytest.mark.parametrize("tied", [True, False])
@pytest.mark.parametrize("edit", ["none", "after", "between", "hook", "unused"])
def test_norm_of_edited_gradients(tied, edit):
    """What a program writes into the embedding's gradient between the backward pass and the step counts in the norm that clips."""
    from state_space_models_neuron_b200 import parallel as nxd
    from state_space_models_neuron_b200.models import Mamba2Config, Mamba2ForCausalLM
    from state_space_models_neuron_b200.parallel import state as ps
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(1)
    cfg = nxd.parallel_config(1, {"zero_one_enabled": True, "grad_clipping": True, "max_grad_norm": 1.0}, init_seed=3)
    mc = Mamba2Config(num_heads=8, head_dim=64, vocab_size=4096, hidden_size=256, state_size=128, num_hidden_layers=1, n_groups=1,
                      tie_word_embeddings=tied, initializer_range=0.02, dtype=torch.bfloat16)
    model = nxd.initialize_parallel_model(cfg, lambda: Mamba2ForCausalLM(mc, device="cuda").to(torch.bfloat16))
    more = [torch.nn.Parameter(torch.ones(64, 64, device="cuda", dtype=torch.bfloat16))] if edit == "unused" else []
    opt = nxd.initialize_parallel_optimizer(cfg, nxd.AdamW_FP32OptimParams, [{"params": [*model.parameters(), *more]}], lr=1e-3)
    weight = model.backbone.embeddings.weight
    ids = torch.randint(0, 4096, (2, 256), device="cuda", generator=torch.Generator(device="cuda").manual_seed(4))
    opt.zero_grad()
    for k in range(2 if edit == "between" else 1):
        model(input_ids=ids, labels=ids, return_logits=False).loss.backward()
        assert weight.norm_tracked == (k == 0)
        if edit in ("after", "between") and k == 0:
            with torch.no_grad():
                weight.main_grad[:2048] *= 8
    if edit == "hook":
        opt.post_reduce_hook = lambda o: weight.main_grad[:2048].mul_(8)
    opt.step()
    assert weight.norm_tracked == (edit in ("none", "unused"))
    want = opt.flat_grads.double().norm().item()
    assert abs(opt.last_grad_norm.item() - want) <= 1e-5 * want


@pytest.mark.parametrize("total", [0.0, 1e-20, 0.25, 1.0, 3.7e9, float("inf"), float("nan"), -1.0])
def test_clip_coefficient_equals_separate_operations(total):
    from state_space_models_neuron_b200.ops import cuda_ops
    sq = torch.tensor([total], device="cuda")
    step, skipped = torch.tensor([5], dtype=torch.int32, device="cuda"), torch.tensor([2], dtype=torch.int32, device="cuda")
    norm, clip = cuda_ops.clip_coefficient(sq, 0.7, step, skipped)
    want = torch.sqrt(sq.clamp(min=0))                   # below zero: sums that took each other back, but for rounding
    finite = torch.isfinite(want)
    assert torch.equal(norm.nan_to_num(9.0, 8.0), want.nan_to_num(9.0, 8.0))
    assert torch.equal(clip, torch.where(finite, torch.clamp(0.7 / (want + 1e-6), max=1.0), -torch.ones_like(want)))
    assert (step.item(), skipped.item()) == ((6, 2) if finite else (5, 3))


@pytest.mark.parametrize("rows", [1, 256, 257])
def test_row_loss_equals_separate_operations(rows):
    from state_space_models_neuron_b200.ops import cuda_ops
    gen = torch.Generator(device="cuda").manual_seed(rows)
    m, s, t = (torch.randn(rows, device="cuda", generator=gen) * 9 for _ in range(3))
    s = s.abs() + 1
    s[0], m[0] = (0.0, float("-inf")) if rows > 1 else (1.0, 0.0)
    labels = torch.randint(0, 3, (rows,), device="cuda", generator=gen)
    loss = cuda_ops.ce_row_loss(m, s, t, labels, 2)
    want = torch.where(labels != 2, torch.log(s) + m - t, torch.zeros_like(s))
    # the logarithm may be rounded to the other side: one step of it
    assert torch.allclose(loss, want, rtol=2.0 ** -23, atol=2.0 ** -23 * 6, equal_nan=True)
