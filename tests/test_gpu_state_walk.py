"""SSD kernels that walk the chunks, and fused decoding, against the kernels they stand for."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc", [1, 2, 3, 4, 7, 11])            # loads run three chunks ahead, two TMEM buffers
@pytest.mark.parametrize("H,P,G", [(4, 64, 1), (6, 128, 2)])   # a head of 128 channels is two slices
def test_walk_equals_separate_kernels(monkeypatch, nc, H, P, G):
    from state_space_models_neuron_b200.ops import cuda_ops
    B, L, d, Hv = 2, nc * 128, H * P, H * P // 64
    gen = torch.Generator(device="cuda").manual_seed(nc * 10 + H)
    C = d + 2 * G * 128
    xbc = torch.randn(B * L, C, device="cuda", generator=gen).bfloat16()
    dy = torch.randn(B * L, d, device="cuda", generator=gen).bfloat16()
    dt = torch.rand(B, H, L, device="cuda", generator=gen) * 0.1
    a = -torch.rand(H, device="cuda", generator=gen) * 8
    l = (dt * a[None, :, None]).view(B, H, nc, 128).cumsum(-1).reshape(B, H, L).contiguous()
    out = []
    for walk in (False, True):
        monkeypatch.setattr(cuda_ops, "_walk_states", lambda slices, n: walk)
        out.append(cuda_ops._chunk_states(xbc, C, d + G * 128, dy, d, dt, l, None, False, B, L, H, Hv, G, 1)[0])
    torch.cuda.synchronize()
    cuda_ops.check_status()
    # the same bf16 products and fp32 recurrence; only the contraction of a multiply and an add may differ: at most one
    # bf16 step of a state
    s0, s1 = out[0].float(), out[1].float()
    assert ((s0 - s1).abs() <= 2.0 ** -7 * s0.abs() + 1e-6).all()


@pytest.mark.parametrize("nc", [1, 2, 3, 4, 5, 9])             # two stages of loads, products of the next chunk ahead
@pytest.mark.parametrize("H,P,G", [(4, 64, 1), (6, 128, 2)])
def test_walk_scan_equals_separate_kernels(monkeypatch, nc, H, P, G):
    from state_space_models_neuron_b200.ops import cuda_ops
    B, L, d, Hv = 2, nc * 128, H * P, H * P // 64
    gen = torch.Generator(device="cuda").manual_seed(nc * 10 + H)
    xbc = torch.randn(B * L, d + 2 * G * 128, device="cuda", generator=gen).bfloat16()
    raw = torch.randn(B * L, 8, device="cuda", generator=gen).bfloat16()
    A, D, bias = -torch.rand(H, device="cuda", generator=gen) * 4, torch.rand(H, device="cuda"), torch.zeros(H, device="cuda")
    init = torch.randn(B, Hv, 128, 64, device="cuda", generator=gen)
    out = []
    for walk in (False, True):
        monkeypatch.setattr(cuda_ops, "_walk_states", lambda slices, n: walk)
        out.append(cuda_ops._ssd_forward(xbc, raw, 8, A, D, bias, B, L, d, G, H, Hv, init, True))
    bare = cuda_ops._ssd_forward(xbc, raw, 8, A, D, bias, B, L, d, G, H, Hv, init, True, want_states=False)
    torch.cuda.synchronize()
    cuda_ops.check_status()
    (y0, _, _, s0, f0, _), (y1, _, _, s1, f1, _) = out
    assert ((s0.float() - s1.float()).abs() <= 2.0 ** -7 * s0.float().abs() + 1e-6).all()
    assert torch.allclose(f0, f1, rtol=1e-5, atol=1e-5 * f0.abs().max().item())
    # y: one bf16 step of the result, and one of a state or a weight among the 128 terms of its sums
    assert ((y0.float() - y1.float()).abs() <= 2.0 ** -7 * (y0.float().abs() + y0.float().abs().mean())).all()
    assert bare[3] is None and torch.equal(bare[0], y1) and torch.equal(bare[4], f1)


@pytest.mark.parametrize("nc,count", [(2, 2), (5, 2), (7, 3), (7, 7), (11, 4)])       # equal segments, a short last one, one chunk each
@pytest.mark.parametrize("H,P,G", [(4, 64, 1), (6, 128, 2)])
def test_segments_equal_one_walk(monkeypatch, nc, count, H, P, G):
    from state_space_models_neuron_b200.ops import cuda_ops
    B, L, d, Hv = 2, nc * 128, H * P, H * P // 64
    gen = torch.Generator(device="cuda").manual_seed(nc * 10 + H)
    xbc = torch.randn(B * L, d + 2 * G * 128, device="cuda", generator=gen).bfloat16()
    dy = torch.randn(B * L, d, device="cuda", generator=gen).bfloat16()
    raw = torch.randn(B * L, 8, device="cuda", generator=gen).bfloat16() - 4           # decays that reach over several chunks
    A, D, bias = -torch.rand(H, device="cuda", generator=gen) * 0.5, torch.rand(H, device="cuda"), torch.zeros(H, device="cuda")
    init = torch.randn(B, Hv, 128, 64, device="cuda", generator=gen)
    monkeypatch.setattr(cuda_ops, "_walk_states", lambda slices, n: True)
    out = []
    for segments in (1, count):
        monkeypatch.setattr(cuda_ops, "_segments", lambda *a: segments)
        y, dt, l, s, f, _ = cuda_ops._ssd_forward(xbc, raw, 8, A, D, bias, B, L, d, G, H, Hv, init, True)
        back = cuda_ops._chunk_states(xbc, d + 2 * G * 128, d + G * 128, dy, d, dt, l, None, False, B, L, H, Hv, G, 1)[0]
        out.append((s, f, y, back))
    torch.cuda.synchronize()
    cuda_ops.check_status()
    (s0, f0, y0, b0), (s1, f1, y1, b1) = out
    # the recurrence in fp32, associated otherwise: at most one bf16 step of a state, of values that may have cancelled
    for a, b in ((s0, s1), (b0, b1)):
        assert ((a.float() - b.float()).abs() <= 2.0 ** -7 * a.float().abs() + 1e-5 * a.float().abs().max()).all()
    assert torch.allclose(f0, f1, rtol=1e-5, atol=1e-5 * f0.abs().max().item())
    assert ((y0.float() - y1.float()).abs() <= 2.0 ** -7 * (y0.float().abs() + y0.float().abs().mean())).all()


@pytest.mark.parametrize("B,H,P,G,fp32", [(1, 8, 64, 1, False), (3, 24, 64, 8, True), (5, 16, 128, 2, False)])
def test_decode_step_equals_separate_kernels(monkeypatch, B, H, P, G, fp32):
    """Conv, state update and window roll in the fused decoding kernels against one kernel each."""
    from state_space_models_neuron_b200 import ops
    from state_space_models_neuron_b200.ops import cuda_ops
    d, N = H * P, 128
    C = d + 2 * G * N
    gen = torch.Generator(device="cuda").manual_seed(B + H)
    make = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    kind = torch.float32 if fp32 else torch.bfloat16
    p = [make(C, 1, 4).bfloat16(), make(C).bfloat16(), make(H).to(kind), make(H).abs().to(kind), make(H).to(kind), make(d).bfloat16()]
    kw = dict(d_inner=d, n_groups=G, d_state=N, head_dim=P, eps=1e-5, norm_group_size=d // G)
    window, state = make(B, C, 4).bfloat16(), make(B, H, P, N)
    tokens = [torch.nn.functional.pad(make(B, d + C + H), (0, (-(d + C + H)) % 8)).bfloat16()[:, :d + C + H] for _ in range(3)]
    out = []
    mask = cuda_ops._head_param_mask
    for fused in (True, False):
        monkeypatch.setattr(cuda_ops, "_head_param_mask", mask if fused else (lambda *a: None))
        w, s = window.clone(), state.clone()
        ys = [ops.ssm_decode_step(t, w, s, *p, **kw) for t in tokens]
        out.append((ys, w, s))
    torch.cuda.synchronize()
    cuda_ops.check_status()
    assert torch.equal(out[0][1], out[1][1])                    # windows are moved, not computed: the last token, of four
    assert torch.equal(out[0][1], torch.stack([window[..., 3]] + [t[:, d:d + C] for t in tokens], -1))
    assert torch.allclose(out[0][2], out[1][2], rtol=1e-5, atol=1e-6)
    for a, b in zip(out[0][0], out[1][0]):
        assert ((a.float() - b.float()).abs() <= 2.0 ** -7 * (b.float().abs() + b.float().abs().mean())).all()


@pytest.mark.parametrize("nc", [1, 4, 5])                      # walked, walked, a CTA per chunk
@pytest.mark.parametrize("H,P,G", [(8, 64, 1), (8, 128, 2)])
def test_decoding_takes_the_final_state(nc, H, P, G):
    from state_space_models_neuron_b200 import ops
    B, L, N, d = 2, nc * 128, 128, H * P
    C = d + 2 * G * N
    gen = torch.Generator(device="cuda").manual_seed(nc + H)
    make = lambda *s: torch.randn(*s, device="cuda", generator=gen).bfloat16()
    head = [make(H), make(H).abs(), make(H)]                   # dt_bias, A_log, D
    y, state = ops.ssd_chunk_scan(make(B, L, H, P), make(B, L, H), -head[1].float().exp(), make(B, L, G, N), make(B, L, G, N),
                                  head[2], head[0], chunk_size=128, return_final_state=True)
    assert state.shape == (B, H, P, N) and state.is_contiguous()
    before = state.clone()
    ops.ssm_decode_step(make(B, d + C + H), make(B, C, 4), state, make(C, 1, 4), make(C), *head, make(d), d_inner=d, n_groups=G,
                        d_state=N, head_dim=P, eps=1e-5, norm_group_size=None)
    torch.cuda.synchronize()
    assert not torch.equal(state, before)


def _scan64(x, dt, A, Bm, Cm, D, bias):
    """The scan chunk by chunk in the precision of its inputs."""
    H, G = x.shape[2], Bm.shape[2]
    dt = torch.nn.functional.softplus(dt + bias)
    S, out = x.new_zeros(x.shape[0], H, 128, x.shape[3]), []
    Be, Ce = (t.repeat_interleave(H // G, 2) for t in (Bm, Cm))
    for t0 in range(0, x.shape[1], 128):
        at = slice(t0, t0 + 128)
        l, u = (A * dt)[:, at].cumsum(1).transpose(1, 2), (x[:, at] * dt[:, at, :, None]).transpose(1, 2)
        b, c = Be[:, at].transpose(1, 2), Ce[:, at].transpose(1, 2)
        decay = (l[..., :, None] - l[..., None, :]).tril().exp().tril()
        out.append(((c @ b.transpose(-1, -2) * decay) @ u + l.exp()[..., None] * (c @ S)).transpose(1, 2))
        S = l[..., -1:, None].exp() * S + b.transpose(-1, -2) @ (u * (l[..., -1:] - l).exp()[..., None])
    return torch.cat(out, 1) + D[:, None] * x


# a CTA of the backward scan walks one, some or all heads of a group; five and more chunks with few slices take the kernels
# of one CTA per chunk, the others walk
@pytest.mark.parametrize("B,L,H,P,G", [(1, 640, 6, 64, 1), (2, 256, 8, 64, 2), (1, 128, 4, 128, 1), (1, 768, 8, 128, 2)])
def test_scan_gradients_for_any_number_of_heads_per_cta(monkeypatch, B, L, H, P, G):
    from state_space_models_neuron_b200 import ops
    from state_space_models_neuron_b200.ops import cuda_ops
    gen = torch.Generator(device="cuda").manual_seed(L + H)
    make = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    ins = [make(B, L, H, P).bfloat16(), make(B, L, H).bfloat16(), -make(H).abs() * 4 - 1, make(B, L, G, 128).bfloat16(),
           make(B, L, G, 128).bfloat16(), make(H), make(H) - 3]
    dy = make(B, L, H, P).bfloat16()
    wide = [t.double().requires_grad_() for t in ins]
    want = _scan64(*wide)
    want = (want,) + torch.autograd.grad(want, wide, dy.double())
    group, first = H * P // 64 // G, None
    for hpc in [h for h in (1, 2, 3, group) if group % h == 0]:
        monkeypatch.setattr(cuda_ops, "_pick_hpc", lambda slices, chunks: hpc)
        leaf = [t.detach().clone().requires_grad_() for t in ins]
        y = ops.ssd_chunk_scan(*leaf, chunk_size=128)
        got = (y.detach(),) + torch.autograd.grad(y, leaf, dy)
        torch.cuda.synchronize()
        cuda_ops.check_status()
        # operands of the products and results are rounded to bf16 (2^-9 each at most, independent): three such roundings
        for a, b in zip(got, want):
            assert ((a.double() - b).norm() / b.norm()).item() < 3 * 2.0 ** -9
        first = first or got
        for i, (a, b) in enumerate(zip(got, first)):
            if i in (4, 5):                                    # dB and dC: another order of fp32 sums, rounded to bf16
                assert ((a - b).float().abs() <= 2.0 ** -7 * (b.float().abs() + 1e-3 * b.float().abs().mean())).all()
            else:                                              # a head's own
                assert torch.equal(a, b)
