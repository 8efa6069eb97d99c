"""GEMMs with few rows (csrc/gemm_skinny.cu) against a float64 product of the same bf16 operands."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 5, 8, 9, 16, 17, 32, 33, 64, 65, 128, 129])      # edges of the row classes; 129: the tiled kernel
@pytest.mark.parametrize("N,K", [(8, 8), (131, 72), (1000, 768), (3352, 776), (515, 5120), (57000, 128)])
def test_few_rows_match_float64(M, N, K):
    from state_space_models_neuron_b200.ops import cuda_ops
    gen = torch.Generator(device="cuda").manual_seed(M * 7919 + N + K)
    x = torch.randn(M, K + 8, device="cuda", generator=gen).bfloat16()[:, :K]          # row stride > K
    w = torch.randn(N, K, device="cuda", generator=gen).bfloat16()
    bias = torch.randn(N, device="cuda", generator=gen).bfloat16() if K == 768 else None
    ldo = (N + 7) // 8 * 8 + 8
    buf = torch.full((M, ldo), 7.0, dtype=torch.bfloat16, device="cuda")
    out = cuda_ops.gemm(x, w, out=buf[:, :N], bias=bias)
    again = cuda_ops.gemm(x, w, bias=bias)
    torch.cuda.synchronize()
    cuda_ops.check_status()
    ref = x.double() @ w.double().t() + (0 if bias is None else bias.double())
    # one bf16 rounding of the result (2^-8 relative covers its half unit) and fp32 accumulation of K products, whose
    # partial sums are at most the sum of magnitudes
    bound = 2.0 ** -8 * ref.abs() + 2.0 ** -21 * (x.double().abs() @ w.double().abs().t()) + 1e-6
    assert ((out.double() - ref).abs() <= bound).all()
    assert torch.equal(out, again)
    assert (buf[:, (N + 7) // 8 * 8:] == 7.0).all()          # nothing beyond the row's last 16 bytes
