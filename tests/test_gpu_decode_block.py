"""One token of a whole block by one native call, against the operations one by one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# rows of 64-column chunks and a remainder; both, one and no norm inside a product; parts of a head; groups of several warps
@pytest.mark.parametrize("B,width,H,P,G,gs,fp32", [(1, 256, 8, 64, 1, 512, False), (8, 768, 24, 64, 8, 192, True),
                                                   (5, 1000, 16, 128, 2, 1024, False), (2, 1032, 8, 64, 4, 128, True),
                                                   (3, 2560, 80, 64, 1, 5120, False), (9, 256, 8, 64, 1, 512, True),
                                                   (2, 256, 12, 64, 2, 96, False)])
def test_block_equals_separate_operations(B, width, H, P, G, gs, fp32):
    from state_space_models_neuron_b200 import ops
    from state_space_models_neuron_b200.ops import cuda_ops
    d, N = H * P, 128
    C = d + 2 * G * N
    gen = torch.Generator(device="cuda").manual_seed(B + width)
    make = lambda *s, scale=1.0: (torch.randn(*s, device="cuda", generator=gen) * scale).bfloat16()
    norm_w, gate_w = make(width), make(d)
    in_w, in_b, out_w = make(d + C + H, width, scale=width ** -0.5), make(d + C + H), make(width, d, scale=d ** -0.5)
    conv_w, conv_b, head = make(C, 1, 4), make(C), [make(H).float(), make(H).abs(), make(H)]
    window, state = make(B, C, 4), torch.randn(B, H, P, N, device="cuda", generator=gen)
    rd = torch.float32 if fp32 else None
    kw = dict(d_inner=d, n_groups=G, d_state=N, head_dim=P, eps=1e-5, norm_group_size=gs)
    w0, s0 = window.clone(), state.clone()
    hidden, residual = make(B, 1, width), None
    with torch.no_grad():
        for _ in range(3):
            window.copy_(w0), state.copy_(s0)                   # both sides from the same states
            out, res = ops.decode_block(hidden, residual, rd, window, state, norm_w, 1e-5, in_w, in_b, conv_w, conv_b, *head, gate_w,
                                        out_w, **kw)
            normed, want_res = ops.add_rmsnorm(hidden, residual, norm_w, 1e-5, rd)
            zx = ops.linear(normed, in_w, in_b)[:, 0]
            y = ops.ssm_decode_step(zx, w0, s0, conv_w, conv_b, *head, gate_w, **kw)
            want = ops.linear(y[:, None], out_w)
            torch.cuda.synchronize()
            cuda_ops.check_status()
            assert torch.equal(res, want_res) and out.shape == hidden.shape
            # in_proj's operands and results are rounded to bf16 once on both sides; that they are the same bits is tested below
            near = lambda a, b: ((a.double() - b.double()).norm() / b.double().norm()).item() < 2.0 ** -7
            assert near(window, w0) and torch.equal(window[..., :3], w0[..., :3]) and near(state, s0) and near(out, want)
            hidden, residual = want, want_res


# both norms inside the products: one and two vectors per thread of the norm kernel, whole and partial warps and chunks, groups of
# whole chunks, one to eight rows, several turns of the rows, no residual at first and then one of either type
@pytest.mark.parametrize("B,width,H,P,G,gs,fp32", [(1, 768, 24, 64, 1, 1536, True), (1, 1000, 8, 272, 1, 2176, False),
                                                   (8, 1024, 16, 64, 2, 1024, True), (5, 256, 32, 64, 1, 2048, False),
                                                   (1, 264, 16, 128, 1, 2048, True), (2, 64, 16, 64, 2, 512, False),
                                                   (1, 72, 8, 192, 4, 192, True), (4, 8, 8, 64, 1, 512, False),
                                                   (7, 104, 13, 64, 1, 832, True), (1, 1000, 8, 480, 1, 3840, False),
                                                   (8, 128, 64, 64, 1, 4096, False), (5, 128, 48, 64, 8, 384, True)])
def test_block_has_the_bits_of_separate_operations(B, width, H, P, G, gs, fp32):
    """Which norms run inside the products is a matter of time only: every sum and rounding is that of the separate kernels."""
    from state_space_models_neuron_b200 import ops
    from state_space_models_neuron_b200.ops import cuda_ops
    d, N = H * P, 128
    C = d + 2 * G * N
    assert all(cuda_ops._norms_in_products(B, width, d + C + H, d, gs, False))
    gen = torch.Generator(device="cuda").manual_seed(B + width)
    make = lambda *s, scale=1.0: (torch.randn(*s, device="cuda", generator=gen) * scale).bfloat16()
    norm_w, gate_w = make(width), make(d)
    in_w, in_b, out_w = make(d + C + H, width, scale=width ** -0.5), make(d + C + H), make(width, d, scale=d ** -0.5)
    conv_w, conv_b, head = make(C, 1, 4), make(C), [make(H).float(), make(H).abs(), make(H)]
    window, state = make(B, C, 4), torch.randn(B, H, P, N, device="cuda", generator=gen)
    rd = torch.float32 if fp32 else None
    kw = dict(d_inner=d, n_groups=G, d_state=N, head_dim=P, eps=1e-5, norm_group_size=gs)
    w0, s0 = window.clone(), state.clone()
    hidden, residual = make(B, 1, width), None
    with torch.no_grad():
        for _ in range(4):
            out, res = ops.decode_block(hidden, residual, rd, window, state, norm_w, 1e-5, in_w, in_b, conv_w, conv_b, *head, gate_w,
                                        out_w, **kw)
            normed, want_res = ops.add_rmsnorm(hidden, residual, norm_w, 1e-5, rd)
            y = ops.ssm_decode_step(ops.linear(normed, in_w, in_b)[:, 0], w0, s0, conv_w, conv_b, *head, gate_w, **kw)
            want = ops.linear(y[:, None], out_w)
            torch.cuda.synchronize()
            cuda_ops.check_status()
            for a, b in ((out, want), (res, want_res), (window, w0), (state, s0)):
                assert torch.equal(a, b)
            hidden, residual = out, res


def test_block_refuses_what_it_cannot_read():
    from state_space_models_neuron_b200 import ops
    B, width, H, P, N = 1, 256, 8, 64, 128
    d, C = H * P, H * P + 2 * N
    make = lambda *s: torch.randn(*s, device="cuda").bfloat16()
    good = dict(hidden=make(B, 1, width), residual=None, residual_dtype=None, conv_state=make(B, C, 4),
                ssm_state=torch.zeros(B, H, P, N, device="cuda"), norm_w=make(width), norm_eps=1e-5, in_w=make(d + C + H, width), in_b=None,
                conv_w=make(C, 1, 4), conv_b=None, dt_bias=make(H), A_log=make(H), D=make(H), gate_w=make(d), out_w=make(width, d))
    kw = dict(d_inner=d, n_groups=1, d_state=N, head_dim=P, eps=1e-5, norm_group_size=None)
    bad = dict(hidden=make(B, 1, width).float(), residual=make(B, 1, width).float(), conv_state=make(B, C, 8)[..., ::2],
               ssm_state=torch.zeros(B, H, N, P, device="cuda").transpose(2, 3), norm_w=make(width + 1)[1:], in_w=make(width, d + C + H).t(),
               in_b=make(3), out_w=make(width, d).float(), D=make(2 * H)[::2], gate_w=make(d + 8))
    with torch.no_grad():
        assert ops.decode_block(**good, **kw) is not None
        for name, value in bad.items():
            assert ops.decode_block(**{**good, name: value}, **kw) is None, name
    assert ops.decode_block(**good, **kw) is None               # recorded: autograd's operations stay


def test_hooks_and_replaced_modules_keep_their_calls():
    from state_space_models_neuron_b200.models import Mamba2Cache, Mamba2Config, Mamba2ForCausalLM
    from state_space_models_neuron_b200.parallel import state as ps
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(1)
    cfg = Mamba2Config(num_heads=8, head_dim=64, vocab_size=512, hidden_size=256, state_size=128, num_hidden_layers=2, n_groups=1,
                       initializer_range=0.02, dtype=torch.bfloat16)
    model = Mamba2ForCausalLM(cfg, device="cuda").to(torch.bfloat16).eval()
    token = torch.tensor([[3]], device="cuda")
    plain = model.step(token, Mamba2Cache(cfg, 1, dtype=torch.bfloat16, device="cuda"))
    seen = []
    block = model.backbone.layers[1]
    handle = block.mixer.out_proj.register_forward_hook(lambda *a: seen.append(a[2].shape))
    hooked = model.step(token, Mamba2Cache(cfg, 1, dtype=torch.bfloat16, device="cuda"))
    handle.remove()
    assert len(seen) == 1
    block.mixer.in_proj.forward = lambda x, f=block.mixer.in_proj.forward: seen.append(x.shape) or f(x)
    model.step(token, Mamba2Cache(cfg, 1, dtype=torch.bfloat16, device="cuda"))
    assert len(seen) == 2
    assert ((hooked - plain).norm() / plain.norm()).item() < 2.0 ** -6


# one chunk; heads of two slices and groups; several segments and few slices; a width that is no multiple of 64
@pytest.mark.parametrize("B,L,width,H,P,G,gs,fp32,cached", [(1, 128, 256, 8, 64, 1, 512, False, True), (2, 384, 512, 6, 128, 2, 384, True, True),
                                                            (1, 2176, 264, 4, 64, 1, 256, False, True), (3, 256, 256, 8, 64, 4, 512, True, False)])
def test_block_over_a_sequence_equals_separate_operations(B, L, width, H, P, G, gs, fp32, cached):
    from state_space_models_neuron_b200 import ops
    from state_space_models_neuron_b200.ops import cuda_ops
    d, N = H * P, 128
    C = d + 2 * G * N
    gen = torch.Generator(device="cuda").manual_seed(B + L)
    make = lambda *s, scale=1.0: (torch.randn(*s, device="cuda", generator=gen) * scale).bfloat16()
    norm_w, gate_w = make(width), make(d)
    in_w, in_b, out_w = make(d + C + H, width, scale=width ** -0.5), make(d + C + H), make(width, d, scale=d ** -0.5)
    conv_w, conv_b, head = make(C, 1, 4), make(C), [make(H).float(), make(H).abs(), make(H)]
    window, state = make(B, C, 4), torch.randn(B, H, P, N, device="cuda", generator=gen)
    rd = torch.float32 if fp32 else None
    kw = dict(d_inner=d, n_groups=G, d_state=N, head_dim=P, eps=1e-5, norm_group_size=gs)
    hidden, residual = make(B, L, width), None
    with torch.no_grad():
        for _ in range(2):
            versions = window._version, state._version
            out, res = ops.block_forward(hidden, residual, rd, window if cached else None, state if cached else None, norm_w, 1e-5, in_w, in_b,
                                         conv_w, conv_b, *head, gate_w, out_w, **kw)
            normed, want_res = ops.add_rmsnorm(hidden, residual, norm_w, 1e-5, rd)
            y, (w, s) = ops.mamba2_mixer_core(ops.linear(normed, in_w, in_b), conv_w, conv_b, *head, gate_w, return_final_states=True, **kw)
            want = ops.linear(y, out_w)
            torch.cuda.synchronize()
            cuda_ops.check_status()
            assert torch.equal(res, want_res) and out.shape == hidden.shape
            # the same kernels, but for the chunks' route: states in the order of another association, one bf16 step of a value
            near = lambda a, b: ((a.double() - b.double()).norm() / b.double().norm()).item() < 2.0 ** -8
            assert near(out, want)
            if cached:
                assert torch.equal(window, w) and near(state, s) and window._version > versions[0] and state._version > versions[1]
            hidden, residual = want, want_res
    assert ops.block_forward(hidden, residual, rd, None, None, norm_w, 1e-5, in_w, in_b, conv_w, conv_b, *head, gate_w, out_w, **kw) is None


def test_prompts_with_hooks_and_odd_caches_keep_their_calls():
    from state_space_models_neuron_b200.models import Mamba2Cache, Mamba2Config, Mamba2ForCausalLM
    from state_space_models_neuron_b200.parallel import state as ps
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(1)
    cfg = Mamba2Config(num_heads=8, head_dim=64, vocab_size=512, hidden_size=256, state_size=128, num_hidden_layers=2, n_groups=1,
                       initializer_range=0.02, dtype=torch.bfloat16)
    model = Mamba2ForCausalLM(cfg, device="cuda").to(torch.bfloat16).eval()
    ids = torch.randint(0, 512, (2, 128), device="cuda")
    plain, cache = model.prefill(ids)
    seen = []
    mixer = model.backbone.layers[1].mixer
    handles = [mixer.register_forward_hook(lambda *a: seen.append("mixer")), mixer.in_proj.register_forward_hook(lambda *a: seen.append("in"))]
    hooked, other = model.prefill(ids)
    [h.remove() for h in handles]
    assert seen == ["in", "mixer"] and torch.equal(hooked, plain)
    odd = Mamba2Cache(cfg, 2, dtype=torch.bfloat16, device="cuda", ssm_dtype=torch.bfloat16)
    again, _ = model.prefill(ids, odd)
    assert torch.equal(again, plain) and torch.equal(odd.ssm_states[1], cache.ssm_states[1].bfloat16())
    for i in range(2):
        assert torch.equal(cache.conv_states[i], other.conv_states[i]) and torch.equal(cache.ssm_states[i], other.ssm_states[i])
    host = Mamba2Cache(cfg, 2, dtype=torch.bfloat16, device="cpu")          # states of a prompt are copied into host memory
    again, _ = model.prefill(ids, host)
    assert torch.equal(again, plain) and all(torch.equal(host.ssm_states[i], cache.ssm_states[i].cpu()) for i in range(2))
