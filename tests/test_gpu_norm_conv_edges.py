"""Norm and conv kernels at the edges of their thread and tile shapes, forward and backward, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _near(got, want, steps=3):
    # one bf16 rounding of the result; where a result is a difference, of its terms (the scale of the tensor)
    bound = steps * 2.0 ** -8 * (want.abs() + want.abs().mean())
    assert ((got.double() - want).abs() <= bound).all(), ((got.double() - want).abs() / bound).max().item()


@pytest.mark.parametrize("d,groups", [(8, 1), (264, 1), (2048, 1), (2056, 1), (5120, 1), (8192, 1), (4096, 8)])
@pytest.mark.parametrize("rows", [1, 297, 601])              # fewer rows than blocks, one more, an uneven share
@pytest.mark.parametrize("gate", [True, False])
def test_norms(d, groups, rows, gate):
    from state_space_models_neuron_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(d + rows)
    make = lambda *s: torch.randn(*s, device="cuda", generator=gen).bfloat16()
    y, z, w, dout = make(rows, d), make(rows, d), make(d), make(rows, d)
    for t in (y, z, w):
        t.requires_grad_()
    out = ops.gated_rmsnorm(y, z if gate else None, w, 1e-5, d // groups)
    Y, Z, W = (t.detach().double().requires_grad_() for t in (y, z, w))
    h = (Y * torch.nn.functional.silu(Z) if gate else Y).view(rows, groups, -1)
    ref = (h * torch.rsqrt(h.square().mean(-1, keepdim=True) + 1e-5)).view(rows, d) * W
    _near(out, ref)
    out.backward(dout)
    ref.backward(dout.double())
    _near(y.grad, Y.grad)
    _near(w.grad, W.grad)
    if gate:
        _near(z.grad, Z.grad)
    elif groups == 1:
        for rd in (torch.bfloat16, torch.float32):
            x, res, dres = make(rows, d).requires_grad_(), torch.randn(rows, d, device="cuda", generator=gen).to(rd), make(rows, d).to(rd)
            got, total = ops.add_rmsnorm(x, res, w, 1e-5, rd)
            s = (x.detach().double() + res.double()).to(rd).double().requires_grad_()
            want = s * torch.rsqrt(s.square().mean(-1, keepdim=True) + 1e-5) * W
            _near(got, want)
            gx, = torch.autograd.grad((got, total), x, (dout, dres))
            gs, = torch.autograd.grad(want, s, dout.double())
            _near(gx, gs + dres.double())


# blocks of the gated norm's backward kernel that walk more rows than their ring holds: stages are loaded again and their phase
# turns, by both thread counts (296, 592 and 148 blocks; rings of 3 or 4)
@pytest.mark.parametrize("rows,d,gs", [(296 * 8 + 1, 5120, 5120), (592 * 9 + 1, 264, 264), (592 * 5 + 7, 2048, 256), (148 * 9 + 1, 5128, 5128)])
@pytest.mark.parametrize("gate", [True, False])
def test_gated_norm_backward_of_many_rows(rows, d, gs, gate):
    from state_space_models_neuron_b200 import ops
    from state_space_models_neuron_b200.ops import cuda_ops
    gen = torch.Generator(device="cuda").manual_seed(rows)
    make = lambda *s: torch.randn(*s, device="cuda", generator=gen).bfloat16()
    y, z, w, dout = make(rows, d).requires_grad_(), make(rows, d).requires_grad_(), make(d).requires_grad_(), make(rows, d)
    ops.gated_rmsnorm(y, z if gate else None, w, 1e-5, gs).backward(dout)
    Y, Z, W = (t.detach().double().requires_grad_() for t in (y, z, w))
    h = (Y * torch.nn.functional.silu(Z) if gate else Y).view(rows, d // gs, gs)
    ((h * torch.rsqrt(h.square().mean(-1, keepdim=True) + 1e-5)).view(rows, d) * W).backward(dout.double())
    cuda_ops.check_status()
    _near(y.grad, Y.grad)
    _near(w.grad, W.grad)
    if gate:
        _near(z.grad, Z.grad)


@pytest.mark.parametrize("L", [1, 3, 8, 33, 35, 130])        # remainders of the token tiles and of the batches of four
@pytest.mark.parametrize("C", [8, 520, 10240])
@pytest.mark.parametrize("init", [True, False])
def test_conv(L, C, init):
    from state_space_models_neuron_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(L + C)
    make = lambda *s: torch.randn(*s, device="cuda", generator=gen).bfloat16()
    x, w, b, dy = make(2, L, C).requires_grad_(), make(C, 1, 4).requires_grad_(), make(C).requires_grad_(), make(2, L, C)
    before = make(2, 3, C) if init else None
    out = ops.causal_conv1d_silu(x, w, b, before)
    X, W, Bs = (t.detach().double().requires_grad_() for t in (x, w, b))
    pad = torch.cat([before.double() if init else X.new_zeros(2, 3, C), X], 1)
    ref = torch.nn.functional.silu(sum(pad[:, k:k + L] * W[:, 0, k] for k in range(4)) + Bs)
    _near(out, ref)
    if not init:                                               # the backward kernel takes the tokens before the first as zeros
        out.backward(dy)
        ref.backward(dy.double())
        for got, want in ((x, X), (w, W), (b, Bs)):
            _near(got.grad, want.grad)


@pytest.mark.parametrize("B,L,C,H", [(1, 128, 264, 3), (2, 256, 520, 8), (1, 1024, 5376, 13), (3, 2048, 2560, 80)])     # 8, 16 and 32 tokens a tile
@pytest.mark.parametrize("fp32", [False, True])
def test_conv_and_step_sizes_in_one_launch(B, L, C, H, fp32):
    """Conv, step sizes and conv window of ssm_conv_dt against one kernel each and against 64 bits."""
    from state_space_models_neuron_b200.ops import cuda_ops
    gen = torch.Generator(device="cuda").manual_seed(B + H)
    make = lambda *s: torch.randn(*s, device="cuda", generator=gen).bfloat16()
    ld = (C + H + 7) // 8 * 8
    rows = make(B, L, ld)
    xbc, raw = rows[..., :C], rows.view(B * L, ld)[:, C:C + H]
    w, bias = make(C, 4), make(C)
    A_log, D, dt_bias = (t.float() if fp32 else t for t in (make(H).abs(), make(H), make(H)))
    window = torch.empty(B, C, 4, dtype=torch.bfloat16, device="cuda")
    out, (dt, l, params) = cuda_ops._conv_dt(xbc, w, bias, raw, ld, A_log, D, dt_bias, window)
    assert torch.equal(out.view(B, L, C), cuda_ops._conv_fwd(xbc, w, bias, None))
    assert torch.equal(window, xbc[:, -4:].transpose(1, 2))
    dt2, l2, params2 = cuda_ops._dt_prep(raw, ld, A_log, D, dt_bias, B, L, H, True)
    assert torch.equal(dt, dt2) and torch.equal(l, l2) and all(torch.equal(a, b.float()) for a, b in zip(params, params2))
    A = -A_log.double().exp()
    want = torch.nn.functional.softplus(raw.double().view(B, L, H) + dt_bias.double()).permute(0, 2, 1)
    sums = (want * A[:, None]).view(B, H, L // 128, 128).cumsum(-1).view(B, H, L)
    # exponential and logarithm to a few ulp, sums of 128 in chains of 5 and 3
    assert torch.allclose(dt.double(), want, rtol=1e-5, atol=1e-6) and torch.allclose(l.double(), sums, rtol=2e-5, atol=1e-5)
    assert torch.allclose(params[0].double(), A, rtol=1e-6) and torch.equal(params[1], D.float()) and torch.equal(params[2], dt_bias.float())


@pytest.mark.parametrize("act", ["gelu", "silu"])
@pytest.mark.parametrize("rows,S", [(1, 8), (3, 2056), (2371, 16)])          # one vector, a second column block, more rows than blocks
def test_gated_linear_unit(rows, S, act):
    from state_space_models_neuron_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(rows + S)
    h = (torch.randn(rows, 2 * S, device="cuda", generator=gen) * 3).bfloat16().requires_grad_()
    dout = torch.randn(rows, S, device="cuda", generator=gen).bfloat16()
    H = h.detach().double().requires_grad_()
    f = torch.nn.functional.gelu if act == "gelu" else torch.nn.functional.silu
    out, ref = ops.glu(h, act), f(H[:, :S]) * H[:, S:]
    _near(out, ref)
    out.backward(dout)
    ref.backward(dout.double())
    _near(h.grad, H.grad)


def test_gelu_of_every_bf16_value():
    """All 65,536 values: below zero GELU is its Gaussian tail, where the result must not lose digits to 1 + erf."""
    from state_space_models_neuron_b200 import ops
    x = torch.arange(-32768, 32768, device="cuda", dtype=torch.int32).to(torch.int16).view(torch.bfloat16).requires_grad_()
    X = x.detach().double()
    y, cdf = ops.gelu(x), torch.special.erfc(-X / 2 ** 0.5) / 2
    Y = X * cdf
    d, = torch.autograd.grad(y, x, torch.ones_like(y))
    D = cdf + X * torch.exp(-X.square() / 2) * 0.3989422804014327
    ok = X.abs() < 12                                       # beyond: 0 or x, and a tail below what fp32 holds
    # half a step of 8 significant bits, and 2^-16 of the arithmetic (an argument of the exponential up to 104, rounded twice to
    # 2^-24 of itself)
    assert ((y.double() - Y).abs() <= (2.0 ** -8 + 2.0 ** -16) * Y.abs() + 1e-36)[ok].all()
    assert ((d.double() - D).abs() <= (2.0 ** -8 + 2.0 ** -16) * D.abs() + 2.0 ** -22)[ok].all()     # terms of the gradient cancel near -0.75
    big = (X.abs() >= 12) & X.isfinite()
    up, down = big & (X > 0), big & (X < 0)                 # x and 1; the rest of the tail, 12 phi(12) = 2^-102 at most
    assert torch.equal(y[up].double(), X[up]) and (d[up] == 1).all() and (y[down].abs() < 2.0 ** -101).all() and (d[down].abs() < 2.0 ** -97).all()
    assert y[X.isnan()].isnan().all() and y[X == float("inf")].item() == float("inf")
