"""A chain of kernels that start before their predecessors have finished, over the same buffers again and again."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 8, 16, 33, 128])           # every kernel of the few-row products
def test_chain_equals_one_by_one(M):
    from state_space_models_neuron_b200 import ops
    from state_space_models_neuron_b200.ops import cuda_ops
    D, inner, H, N = 768, 1536, 24, 128
    C = inner + 2 * N
    W = inner + C + H
    gen = torch.Generator(device="cuda").manual_seed(M)
    make = lambda *s, scale=1.0: (torch.randn(*s, device="cuda", generator=gen) * scale).bfloat16()
    w_in, w_out, norm, gate = make(W, D, scale=0.03), make(D, inner, scale=0.03), make(D), make(inner)
    conv_w, conv_b, head = make(C, 1, 4), make(C), [make(H), make(H).abs(), make(H)]
    x0, window0, state0 = make(M, D), make(M, C, 4), torch.randn(M, H, 64, N, device="cuda", generator=gen)
    zx, back = torch.empty(M, W, dtype=torch.bfloat16, device="cuda"), torch.empty(M, D, dtype=torch.bfloat16, device="cuda")
    out = []
    for wait in (lambda: None, torch.cuda.synchronize):
        x, window, state = x0.clone(), window0.clone(), state0.clone()
        for _ in range(40):
            h, x = ops.add_rmsnorm(x, back if _ else None, norm, 1e-5)
            wait()
            cuda_ops.gemm(h, w_in, out=zx)
            wait()
            y = ops.ssm_decode_step(zx, window, state, conv_w, conv_b, *head, gate, d_inner=inner, n_groups=1, d_state=N,
                                    head_dim=64, eps=1e-5, norm_group_size=None)
            wait()
            cuda_ops.gemm(y, w_out, out=back)
            wait()
        torch.cuda.synchronize()
        cuda_ops.check_status()
        out.append((x, window, state, back.clone()))
    for a, b in zip(*out):
        assert torch.equal(a, b)
    assert torch.isfinite(out[0][0].float()).all()
