"""Performance cases: the work that users of the framework have it do, called the way their programs call it.

Sizes are those of the named configurations (`models/predefined_configs.py`), of `bench.py` and of
`mamba2_inference.py`; layer counts are cut so that a case holds a few GB, which leaves the work of a layer, of the
embedding, of the LM head and of the optimizer as it is.  Weights are random and token ids uniform, as in the benchmark.

Kinds of work
  train        one optimizer step replayed as a CUDA graph (`GraphedTrainStep`, what the launch scripts and the benchmark run)
  train_eager  the same step launched op by op (`train.py` without `--cuda_graph`)
  score        logits and loss of given texts without gradients (evaluation)
  prefill      a prompt through the chunked scan into a fresh cache (`Mamba2ForCausalLM.prefill`)
  decode       one greedy token for every sequence, replayed as a CUDA graph (`GraphedDecodeStep`)
  step         the same token launched op by op (`Mamba2ForCausalLM.step`, what `generate` calls)
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from state_space_models_neuron_b200 import parallel as nxd
from state_space_models_neuron_b200.models import Mamba2Cache, Mamba2ForCausalLM, Mamba2HybridForCausalLM, get_config
from state_space_models_neuron_b200.parallel import state as ps
from state_space_models_neuron_b200.parallel.graph import GraphedDecodeStep, GraphedTrainStep
from state_space_models_neuron_b200.utils.data import get_param_groups_by_weight_decay

STATE = 128          # d_state of every configuration
DEFAULTS = dict(head_dim=64, groups=1, vocab=50288, within=True, recompute=False, shard_of=1, pattern="", gated=False,
                rotary=False)


def _case(name, kind, model, layers, batch, seq, **options):
    return {"name": name, "kind": kind, "model": model, "layers": layers, "batch": batch, "seq": seq, **DEFAULTS, **options}


def listed():
    return [
        # one user typing at the smallest model: every layer is a chain of tiny kernels
        _case("decode_130m_b1", "decode", "Mamba130M", 24, 1, 128),
        # a serving batch of the benchmark's decode configuration: bound by the SSM states and the weights
        _case("decode_2.7b_b64", "decode", "Mamba3B", 12, 64, 128),
        # generate() without a captured graph, an odd number of sequences: host launches count
        _case("step_370m_b5", "step", "Mamba370M", 16, 5, 128),
        # a short chat prompt, one chunk
        _case("prefill_130m_1x128", "prefill", "Mamba130M", 24, 1, 128),
        # a batch of the benchmark's prompts
        _case("prefill_2.7b_16x2048", "prefill", "Mamba3B", 4, 16, 2048),
        # perplexity of texts of an odd number of chunks, fp32 logits, the preset's 128-channel heads
        _case("score_780m_3x896", "score", "Mamba780M", 4, 3, 896, head_dim=128, groups=8),
        # train.py with its defaults: smallest model, no graph
        _case("train_eager_130m_4x1152", "train_eager", "Mamba130M", 3, 4, 1152, vocab=50272),
        # data-parallel training of the 2.7B architecture, micro-batch 4
        _case("train_2.7b_4x2048", "train", "Mamba3B", 2, 4, 2048),
        # the headline benchmark: 7B, one 2048-token sequence
        _case("train_7b_1x2048", "train", "Mamba7B", 3, 1, 2048, groups=8, within=False),
        # one rank's share of the same model under TP=8
        _case("train_7b_share8_1x2048", "train", "Mamba7B", 4, 1, 2048, groups=8, within=False, shard_of=8),
        # hybrid 8B at its 4096-token length with rotary embedding and gated MLP
        _case("train_hybrid8b_1x4096", "train", "Mamba2Hybrid8B", 4, 1, 4096, groups=8, within=False, pattern="M-*-",
              gated=True, rotary=True),
        # hybrid 800M with the reference's plain MLP and no positions, longest supported context, mixer recomputed
        _case("train_hybrid800m_1x8192", "train", "Mamba2Hybrid800M", 4, 1, 8192, groups=8, recompute=True, pattern="M*-M"),
    ]


def draw(rng):
    """One more case of the ranges above: any kind, any configuration, batch and length spread over their logarithm."""
    most = [max(work(c)[k] for c in listed()) for k in ("bytes", "flops")]
    while True:
        kind = rng.choice(["decode", "step", "prefill", "score", "train_eager", "train", "train", "train"])
        hybrid = kind in ("train", "score") and rng.random() < 0.35
        model = rng.choice(["Mamba2Hybrid800M", "Mamba2Hybrid8B"] if hybrid else
                           ["Mamba130M", "Mamba370M", "Mamba780M", "Mamba1B", "Mamba3B", "Mamba7B"])
        pattern = rng.choice(["M*", "*-", "M-*", "M*-M", "M-*-"]) if hybrid else ""
        train = kind in ("train", "train_eager")
        layers = len(pattern) or (rng.randint(1, 3) if train else rng.randint(2, 12))
        width = get_config(model, 256).hidden_size
        head_dim = rng.choice([64, 64, 128])
        groups = rng.choice([g for g in (1, 2, 8) if (2 * width // head_dim) % g == 0])
        longest = 8192 if train or kind == "score" else 4096
        seq = 128 * max(1, round(2 ** rng.uniform(0, math.log2(longest // 128))))
        batch = max(1, round(2 ** rng.uniform(0, 6 if kind in ("decode", "step") else 3)))
        case = _case("", kind, model, layers, batch, 128 if kind in ("decode", "step") else seq, head_dim=head_dim,
                     groups=groups, vocab=rng.choice([50288, 50272, 32768, 16384]), within=rng.random() < 0.5,
                     recompute=train and rng.random() < 0.25, pattern=pattern,
                     shard_of=8 if groups == 8 and not hybrid and width >= 2048 and rng.random() < 0.25 else 1,
                     gated=hybrid and rng.random() < 0.5, rotary=hybrid and rng.random() < 0.5)
        del case["name"]
        w = work(case)
        if 2 * width // head_dim // case["shard_of"] % 8:       # single-token calls take multiples of eight heads
            continue
        if train and batch * seq < 512 or kind == "score" and batch * seq * case["vocab"] > 5e8:
            continue
        if w["bytes"] <= most[0] and w["flops"] <= most[1]:
            return case


def _config(case):
    more = {}
    if case["pattern"]:
        more = dict(hybrid_override_pattern=case["pattern"], gated_linear_unit=case["gated"],
                    mlp_hidden_act="silu" if case["gated"] else "gelu", rotary_emb_dim=128 if case["rotary"] else None)
    c = get_config(case["model"], case["vocab"], case["within"], case["groups"], dtype=torch.bfloat16,
                   head_dim=case["head_dim"], num_hidden_layers=case["layers"], initializer_range=0.02,
                   b200_recompute_mixer=case["recompute"], **more)
    k = case["shard_of"]
    if k > 1:      # as bench.py --shard_of
        c.num_heads, c.n_groups, c.vocab_size, c.expand = c.num_heads // k, max(1, c.n_groups // k), c.vocab_size // k, c.expand / k
    return c


_SERVED = []         # a small parameter of every layer of every model that has served a token


def prepare(case, seed):
    config = _config(case)
    parallel = nxd.parallel_config(1, {"zero_one_enabled": True, "grad_clipping": True, "max_grad_norm": 1.0}, init_seed=seed)
    if not ps.model_parallel_is_initialized():
        ps.initialize_model_parallel(1)
    build = Mamba2HybridForCausalLM if case["pattern"] else Mamba2ForCausalLM
    model = nxd.initialize_parallel_model(parallel, lambda: build(config, device="cuda").to(torch.bfloat16))
    gen = torch.Generator(device="cuda").manual_seed(seed)
    ids = torch.randint(0, config.vocab_size, (case["batch"], case["seq"]), device="cuda", generator=gen)
    state = {"kind": case["kind"], "model": model, "ids": ids}
    if case["kind"] in ("train", "train_eager"):
        model.train()
        opt = nxd.initialize_parallel_optimizer(parallel, nxd.AdamW_FP32OptimParams,
                                                get_param_groups_by_weight_decay(model, 0.1), lr=3e-5, betas=(0.9, 0.95))
        opt.zero_grad()
        state["opt"] = opt
        if case["kind"] == "train":
            state["step"] = GraphedTrainStep(model, opt, {"input_ids": ids, "labels": ids})
    else:
        model.eval()
        if case["kind"] in ("decode", "step"):
            # decoding keeps values made from the per-head parameters by address: a program that serves one model until
            # it ends never frees these, and the many models made here must not meet what was kept for another one
            _SERVED.extend(layer.mixer.dt_bias for layer in model.backbone.layers)
            _, cache = model.prefill(ids)
            state["cache"] = cache
            state["token"] = torch.randint(0, config.vocab_size, (case["batch"], 1), device="cuda", generator=gen)
            if case["kind"] == "decode":
                state["step"] = GraphedDecodeStep(model, cache, case["batch"])
    return state


def run(state):
    kind, model, ids = state["kind"], state["model"], state["ids"]
    if kind == "train":
        loss = state["step"]({"input_ids": ids, "labels": ids})
    elif kind == "train_eager":
        loss = model(input_ids=ids, labels=ids, return_logits=False).loss
        loss.backward()
        state["opt"].step()
        state["opt"].zero_grad()
    if "opt" in state:
        opt = state["opt"]
        return {"loss": loss.detach(), "gradients": opt.flat_grads, "weights": opt.master, "moments": [opt.exp_avg, opt.exp_avg_sq]}
    with torch.no_grad():
        if kind == "score":
            out = model(input_ids=ids, labels=ids)
            return {"loss": out.loss, "logits": out.logits}
        if kind == "prefill":
            logits, cache = model.prefill(ids)
        else:
            cache = state["cache"]
            if kind == "decode":
                state["step"](state["token"])
                logits = state["step"].logits
            else:
                logits = model.step(state["token"], cache)
    return {"logits": logits, "conv": list(cache.conv_states.values()), "ssm": list(cache.ssm_states.values())}


def _sizes(case):
    """(weights of all layers without embedding, their number that every token meets, recurrence operations of a token,
    attention operations of a token pair, values of the decode states of one sequence)."""
    c = _config(case)
    d, inner = c.hidden_size, c.intermediate_size
    weights = recurrence = attention = states = 0
    for kind in case["pattern"] or "M" * case["layers"]:
        if kind == "M":
            weights += d * c.in_proj_size + inner * d + c.conv_dim * 5 + inner
            recurrence += 4 * inner * STATE + 8 * c.conv_dim        # state update and read-out, conv
            states += inner * STATE * 4 + c.conv_dim * 4 * 2        # bytes: fp32 SSM state, bf16 conv window
        elif kind == "*":
            q, kv = c.attn_num_heads * c.attn_head_dim, c.attn_key_value_heads * c.attn_head_dim
            weights += d * (2 * q + 2 * kv)
            attention += 4 * q
        else:
            weights += d * c.mlp_hidden_size * (3 if case["gated"] else 2)
    return c, weights, recurrence, attention, states


def work(case):
    c, weights, recurrence, attention, states = _sizes(case)
    tokens, head = case["batch"] * case["seq"], c.vocab_size * c.hidden_size
    forward = tokens * (2 * weights + recurrence) + case["batch"] * case["seq"] ** 2 / 2 * attention
    if case["kind"] in ("train", "train_eager"):
        # bf16 weight in, fp32 gradient out, fp32 master weight and two moments in and out, ids
        return {"bytes": (weights + head) * (2 + 4 + 24) + 8 * tokens, "flops": 3 * (forward + 2 * tokens * head)}
    if case["kind"] == "score":
        return {"bytes": 2 * (weights + head) + 4 * tokens * c.vocab_size + 8 * tokens, "flops": forward + 2 * tokens * head}
    if case["kind"] == "prefill":
        return {"bytes": 2 * (weights + head) + case["batch"] * (states + 4 * c.vocab_size) + 8 * tokens,
                "flops": forward + 2 * case["batch"] * head}
    return {"bytes": 2 * (weights + head) + case["batch"] * (2 * states + 4 * c.vocab_size),
            "flops": case["batch"] * (2 * (weights + head) + recurrence)}


def tolerance(case):
    # Measured against the same model in PyTorch operations on the same card (bf16 tensors, cuBLAS, another order of every
    # sum): relative difference 0.008 to 0.014 of gradients and moments (2 to 4 layers), 0.009 to 0.011 of logits
    # (4 layers), 0.015 to 0.022 of logits and cached states (12 to 24 layers, where bf16 rounding of the residual stream
    # adds up); gradients of two runs of one implementation differ by 0.005 to 0.011 after three optimizer steps, because
    # AdamW's first steps move a weight by the sign of its gradient.  Largest single difference seen: 0.68.
    return {"rel": 0.03, "max": 0.9}


def _norm(x, weight, eps, group=None):
    grouped = x.unflatten(-1, (-1, group or x.shape[-1]))
    return (grouped * torch.rsqrt(grouped.square().mean(-1, keepdim=True) + eps)).flatten(-2) * weight


def _mixer(m, x, value, before):
    """Mamba-2 mixer over x [B, L, D] behind the state `before` = (conv window [B, 4, C], SSM state [B, H, P, N]) or None."""
    inner, bc, heads = m.intermediate_size_tp, m.n_groups_tp * STATE, m.num_heads_tp
    batch, length = x.shape[:2]
    z, xbc, dt = F.linear(x, value(m.in_proj.weight), value(m.in_proj.bias)).split([inner, inner + 2 * bc, heads], -1)
    window, S = before or (x.new_zeros(batch, 4, inner + 2 * bc), x.new_zeros(batch, heads, m.head_dim, STATE))
    window = torch.cat([window, xbc], 1)
    taps = value(m.conv1d.weight)[:, 0]
    pre = sum(window[:, k + 1:k + 1 + length] * taps[:, k] for k in range(4))
    act = F.silu(pre if m.conv1d.bias is None else pre + value(m.conv1d.bias))
    xs, Bm, Cm = (t.unflatten(-1, (n, -1)) for t, n in zip(act.split([inner, bc, bc], -1), (heads, m.n_groups_tp, m.n_groups_tp)))
    dt = F.softplus(dt + value(m.dt_bias))
    log_decay = -torch.exp(value(m.A_log)) * dt
    parts = []
    for t in range(0, length, 128):
        part = slice(t, t + 128)
        l = log_decay[:, part].cumsum(1).transpose(1, 2)                                       # [B, H, T]
        u = (xs[:, part] * dt[:, part, :, None]).transpose(1, 2)
        B, C = (v[:, part].transpose(1, 2).repeat_interleave(heads // m.n_groups_tp, 1) for v in (Bm, Cm))
        within = (l[..., :, None] - l[..., None, :]).tril().exp().tril()
        y = (C @ B.transpose(-1, -2) * within) @ u + l.exp()[..., None] * (C @ S.transpose(-1, -2))
        S = l[..., -1:, None].exp() * S + (u * (l[..., -1:] - l).exp()[..., None]).transpose(-1, -2) @ B
        parts.append(y.transpose(1, 2))
    y = (torch.cat(parts, 1) + value(m.D)[:, None] * xs).flatten(-2)
    y = _norm(y * F.silu(z), value(m.norm.weight), m.norm.eps, m.norm.group_size)
    return F.linear(y, value(m.out_proj.weight), value(m.out_proj.bias)), (window[:, -4:], S)


def _attention(a, x, value):
    q, k, v = (F.linear(x, value(p.weight)).unflatten(-1, (-1, a.head_dim)).transpose(1, 2) for p in (a.q_proj, a.k_proj, a.v_proj))
    if a.rotary_emb_dim:
        half = a.rotary_emb_dim // 2
        angle = torch.arange(x.shape[1], device=x.device, dtype=x.dtype)[:, None] * \
            a.rope_theta ** (-torch.arange(half, device=x.device, dtype=x.dtype) / half)
        cos, sin = angle.cos(), angle.sin()
        q, k = (torch.cat([t[..., :half] * cos - t[..., half:2 * half] * sin, t[..., half:2 * half] * cos + t[..., :half] * sin,
                           t[..., 2 * half:]], -1) for t in (q, k))
    ratio = a.num_heads // a.num_kv_heads
    out = [F.scaled_dot_product_attention(q[:, h], k[:, h // ratio], v[:, h // ratio], is_causal=True) for h in range(a.num_heads)]
    return F.linear(torch.cat(out, -1), value(a.o_proj.weight))


def _mlp(m, x, value):
    h = F.linear(x, value(m.gate_up_proj.weight))
    h = F.silu(h[..., :m.split_size]) * h[..., m.split_size:] if m.gated else F.gelu(h)
    return F.linear(h, value(m.down_proj.weight))


def _hidden(model, ids, value, before=None):
    """(last hidden states, states of the mixers) of tokens behind the mixers' states `before`."""
    x, states = F.embedding(ids, value(model.backbone.embeddings.weight)), []
    for block in model.backbone.layers:
        layer = block.mixer if hasattr(block, "mixer") else block.layer
        normed = _norm(x, value(block.norm.weight), model.config.layer_norm_epsilon)
        if hasattr(layer, "in_proj"):
            out, after = _mixer(layer, normed, value, before[len(states)] if before else None)
            states.append(after)
        else:
            out = (_attention if hasattr(layer, "q_proj") else _mlp)(layer, normed, value)
        x = x + out
    return _norm(x, value(model.backbone.norm_f.weight), model.config.layer_norm_epsilon), states


def exact(case, seed):
    """The first pass in 64 bits.  None for the captured training step, which stands behind two optimizer steps whose
    first moves of a weight follow the sign of its gradient, and for weights after such a move; the same gradients are
    those of the step launched op by op."""
    kind = case["kind"]
    if kind == "train" or case["batch"] * case["seq"] > 40000:
        return None
    state = prepare(case, seed)
    model, ids, wide = state["model"], state["ids"], {}

    def value(p):
        if p is not None and p not in wide:
            wide[p] = p.detach().double().requires_grad_(kind == "train_eager")
        return None if p is None else wide[p]

    def logits_of(hidden):
        return F.linear(hidden, value(model.lm_head.weight))

    def loss_of(logits):
        return F.cross_entropy(logits[:, :-1].flatten(0, 1), ids[:, 1:].flatten())

    if kind == "train_eager":
        loss = loss_of(logits_of(_hidden(model, ids, value)[0]))
        loss.backward()
        flat = torch.zeros(state["opt"].flat_grads.shape, dtype=torch.float64, device="cuda")
        for p, w in wide.items():
            flat[p.main_grad.storage_offset():][:p.numel()] = w.grad.flatten()
        clipped = flat * min(1.0, 1.0 / (float(flat.norm()) + 1e-6))
        return {"loss": loss.detach(), "gradients": flat, "weights": None, "moments": [0.1 * clipped, 0.05 * clipped.square()]}
    with torch.no_grad():
        hidden, states = _hidden(model, ids, value)
        if kind == "score":
            logits = logits_of(hidden)
            return {"loss": loss_of(logits), "logits": logits}
        if kind != "prefill":
            hidden, states = _hidden(model, state["token"], value, states)
        return {"logits": logits_of(hidden[:, -1:]), "conv": [w.transpose(1, 2) for w, _ in states], "ssm": [S for _, S in states]}
