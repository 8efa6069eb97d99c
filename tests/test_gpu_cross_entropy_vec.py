"""Cross-entropy kernels at the edges of their 16-byte path, and the loss taken in the LM head's GEMM."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [1, 7, 8, 9, 255, 2048, 2055, 50288])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("pad", [0, 8, 5])          # extra elements per row: aligned rows, and rows that are not
def test_partials_and_backward(V, dtype, pad):
    from state_space_models_neuron_b200.ops import cuda_ops
    rows, gen = 5, torch.Generator(device="cuda").manual_seed(V + pad)
    store = (torch.randn(rows, (V + 7) // 8 * 8 + pad, device="cuda", generator=gen) * 30).to(dtype)
    x = store[:, :V]
    x[1] = -200.0                                   # far from zero: the exponent is relative to the maximum
    x[2, : V // 2] = float("-inf")                  # masked entries
    labels = torch.randint(0, V, (rows,), device="cuda", generator=gen)
    labels[3], labels[4] = -100, V + 3              # ignored; another shard's id
    m, s, t = cuda_ops.ce_partials(x, labels, 0)
    ref = x.double()
    assert torch.equal(m.double(), ref.max(1).values)
    # fp32 exponentials (2 ulp) of arguments up to 2^8 (2^-24 relative each) and a sum of V terms
    assert torch.allclose(s.double(), (ref - ref.max(1, keepdim=True).values).exp().sum(1), rtol=1e-4)
    assert torch.equal(t[:3].double(), ref.gather(1, labels[:3, None])[:, 0]) and (t[3:] == 0).all()
    g = torch.rand(rows, device="cuda", generator=gen)
    grad = cuda_ops.ce_backward(x, labels, m, s, g, 0, -100)
    p = torch.softmax(ref, 1)
    p[torch.arange(3), labels[:3]] -= 1
    want = p * torch.where(labels == -100, 0.0, g.double())[:, None]
    assert torch.allclose(grad.double(), want, rtol=2 ** -8 if dtype == torch.bfloat16 else 2e-4, atol=2e-6)


@pytest.mark.parametrize("V", [512, 1000])
def test_loss_of_labelled_forward(V):
    """forward(labels=...) returns fp32 logits and the mean loss of the shifted labels, with the same gradients as the
    loss computed from those logits."""
    from state_space_models_neuron_b200.models import Mamba2Config, Mamba2ForCausalLM
    from state_space_models_neuron_b200.parallel import state as ps
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(1)
    cfg = Mamba2Config(num_heads=8, head_dim=64, vocab_size=V, hidden_size=256, state_size=128, num_hidden_layers=1,
                       n_groups=1, initializer_range=0.02, dtype=torch.bfloat16)
    model = Mamba2ForCausalLM(cfg, device="cuda").to(torch.bfloat16)
    ids = torch.randint(0, V, (2, 128), device="cuda")
    ids[0, 5:9] = -100
    inputs = ids.clamp(min=0)
    out = model(input_ids=inputs, labels=ids)
    valid = ids[:, 1:] != -100
    per_token = torch.nn.functional.cross_entropy(out.logits[:, :-1].reshape(-1, V), ids[:, 1:].reshape(-1), reduction="none",
                                                  ignore_index=-100)
    want = per_token.sum() / valid.numel()
    assert out.logits.dtype == torch.float32
    assert abs(out.loss.item() - want.item()) < 1e-5 * abs(want.item())
    w = model.lm_head.weight
    grad, = torch.autograd.grad(out.loss, w, retain_graph=True)
    ref, = torch.autograd.grad(want, w)
    # both round d(logits) to bf16 once and accumulate in fp32
    assert ((grad - ref).float().norm() / ref.float().norm()).item() < 2 ** -7
    with torch.no_grad():
        again = model(input_ids=inputs, labels=ids)
    assert torch.equal(again.logits, out.logits)


@pytest.mark.parametrize("M,V,K", [(5, 1000, 64), (300, 3004, 128)])
def test_statistics_of_rows_with_infinite_logits(M, V, K):
    """Row statistics out of the LM head's GEMM where the first logits of a row (a vector, a tile, all but one, all) are -inf."""
    from state_space_models_neuron_b200 import ops
    from state_space_models_neuron_b200.ops import cuda_ops
    from state_space_models_neuron_b200.parallel.cross_entropy import parallel_cross_entropy
    gen = torch.Generator(device="cuda").manual_seed(V)
    for first in (3, 8, 40, 520, V - 1, V):
        x, w = (torch.randn(*s, device="cuda", generator=gen).bfloat16() for s in ((M, K), (V, K)))
        x[:, 0] = 0
        x[1], x[1, 0], w[:, 0] = 0.5, 1e30, 0            # row 1 meets -1e60 in the first columns
        w[:first, 0] = -1e30
        labels = torch.randint(0, V, (M,), device="cuda", generator=gen)
        labels[1] = V - 1
        with torch.no_grad():
            y, (m, s, t) = ops.linear_ce(x, w, labels)
            loss = parallel_cross_entropy(y, labels, stats=(m, s, t))
        cuda_ops.check_status()
        ref = y.double()
        assert torch.equal(torch.isinf(ref).sum(1), torch.tensor([0, first] + [0] * (M - 2), device="cuda"))
        m2, s2, t2 = cuda_ops.ce_partials(y, labels, 0)          # the pass over the logits
        assert torch.equal(m, m2) and torch.equal(t, t2) and torch.allclose(s, s2, rtol=1e-5)
        want = torch.nn.functional.cross_entropy(ref, labels, reduction="none")
        assert torch.allclose(loss.double(), want, rtol=1e-5, atol=1e-5, equal_nan=True)
        assert torch.isfinite(loss[1]) == (first < V)


@pytest.mark.parametrize("N", [1, 2, 63, 64, 65, 191, 256, 257, 1001])
def test_statistics_at_the_edges_of_a_column_block(N):
    """Statistics out of the GEMM where N ends inside, at and just behind a 64-column block, with the labels of the rows at
    every column, and shards that begin at another id."""
    from state_space_models_neuron_b200.ops import cuda_ops
    gen = torch.Generator(device="cuda").manual_seed(N)
    M, K, start = 300, 64, 1000
    a, b = (torch.randn(*s, device="cuda", generator=gen).bfloat16() for s in ((M, K), (N, K)))
    labels = start - 1 + torch.arange(M, device="cuda") * (N + 1) // (M - 1)         # one before the shard .. one behind it
    y, (m, s, t) = cuda_ops.gemm_ce(a, b, labels, start)
    cuda_ops.check_status()
    ref, at = y.double(), labels - start
    inside = (at >= 0) & (at < N)
    assert torch.equal(m.double(), ref.max(1).values)
    assert torch.equal(t.double(), torch.where(inside, ref.gather(1, at.clamp(0, N - 1)[:, None])[:, 0], 0.0))
    # exponentials within 2 ulp and an argument below 2^7 rounded to 2^-24 of itself; sums of at most 1001 positive terms in
    # chains of at most 16 per block and 16 blocks
    assert torch.allclose(s.double(), (ref - ref.max(1, keepdim=True).values).exp().sum(1), rtol=2 ** -17 + 40 * 2 ** -24)


@pytest.mark.parametrize("V", [1, 3, 255, 2048, 8195, 50288])
@pytest.mark.parametrize("pad", [0, 4, 1])                   # rows on 16-byte boundaries, with a gap, and not on them
def test_row_maximum(V, pad):
    from state_space_models_neuron_b200.ops import cuda_ops
    gen = torch.Generator(device="cuda").manual_seed(V + pad)
    x = torch.randn(9, V + pad, device="cuda", generator=gen)[:, :V].clone(memory_format=torch.preserve_format) if pad == 0 else \
        torch.randn(9, V + pad, device="cuda", generator=gen)[:, :V]
    x[1] = float("-inf")
    x[2], x[2, V // 2:] = 1.0, 2.0                            # equal values: the first index
    x[3], x[3, V - 1] = -3.0, -2.0                            # all negative, the last one
    x[4], x[4, V // 3] = 0.0, -0.0                            # zeros of both signs are equal
    x[5, V // 4], x[5, V // 2] = float("nan"), float("nan")
    x[6, V - 1] = float("inf")
    val, idx = cuda_ops.row_max(x)
    want = x.cpu().max(dim=1)
    assert torch.equal(idx.cpu(), want.indices) and torch.equal(val.cpu().nan_to_num(7.0), want.values.nan_to_num(7.0))
    v3, i3 = cuda_ops.row_max(x.reshape(3, 3, V))
    assert torch.equal(i3.view(-1), idx) and v3.shape == (3, 3)
