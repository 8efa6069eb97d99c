"""Mamba-2 language model, HuggingFace `PreTrainedModel` compatible.

Module tree and state-dict keys match the reference (mamba2/modeling_mamba2.py:106-140,220-350,
359-531): `backbone.embeddings`, `backbone.layers.{i}.norm`, `backbone.layers.{i}.mixer.*`,
`backbone.norm_f`, `lm_head`.  Differences that matter to users: the full forward also serves
as decode prefill (fills a `Mamba2Cache`), `step()` works after it, and the pre-norm residual
add and RMSNorm of consecutive blocks run as one fused kernel on GPUs.
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import Optional, Tuple

import torch
import torch.nn as nn
from torch.nn.modules.module import _has_any_global_hook
from transformers import GenerationMixin, PreTrainedModel
from transformers.utils import ModelOutput

from .. import ops
from ..parallel import mappings as mp
from ..parallel import state as ps
from ..parallel.cross_entropy import parallel_argmax, parallel_cross_entropy
from ..parallel.layers import ColumnParallelLinear, ParallelEmbedding, RowParallelLinear, normal_init
from .cache import Mamba2Cache
from .configuration_mamba2 import Mamba2Config
from .mamba2_mixer import Mamba2Mixer, MambaRMSNormGated


class Mamba2RMSNorm(nn.Module):
    """fp32 RMSNorm.  Under sequence parallelism the weight only sees a slice of the sequence,
    so it is tagged and its gradient is summed over the TP group before the optimizer step
    (mamba2/modeling_mamba2.py:86-103)."""

    def __init__(self, hidden_size: int, eps: float = 1e-6, sequence_parallel_enabled: bool = False,
                 dtype=torch.float32, device=None):
        super().__init__()
        self.weight = nn.Parameter(torch.ones(hidden_size, dtype=dtype, device=device))
        self.variance_epsilon = eps
        if sequence_parallel_enabled:
            self.weight.sequence_parallel_enabled = True

    def forward(self, hidden_states):
        return ops.rmsnorm(hidden_states, self.weight, self.variance_epsilon)

    def forward_add(self, hidden_states, residual, residual_dtype=None):
        """(normed(residual + hidden_states), residual + hidden_states)"""
        return ops.add_rmsnorm(hidden_states, residual, self.weight, self.variance_epsilon, residual_dtype)


def _hooked(module) -> bool:
    return bool(module._forward_hooks or module._forward_pre_hooks or module._backward_hooks or module._backward_pre_hooks)


def _stood_for():
    """What a block's one native call stands for: methods of the classes and operations as they are now."""
    return (Mamba2Mixer.forward, Mamba2Mixer.step, Mamba2Mixer._core_kwargs, Mamba2Mixer.__call__, Mamba2RMSNorm.forward_add,
            ColumnParallelLinear.forward, ColumnParallelLinear.__call__, RowParallelLinear.forward, RowParallelLinear.__call__,
            ops.add_rmsnorm, ops.linear, ops.mamba2_mixer_core, ops.ssm_decode_step)


_STOOD_FOR = _stood_for()


class Mamba2Block(nn.Module):
    """Pre-norm residual block: h <- h + mixer(norm(h)).

    `forward(hidden, residual)` takes the previous block's branch output and the running
    residual stream and returns (this block's branch output, updated residual), so the add and
    the next norm fuse; the sum of the two is the block output of the reference
    (mamba2/modeling_mamba2.py:115-131)."""

    def __init__(self, config, layer_idx: int, device=None):
        super().__init__()
        self.config = config
        self.layer_idx = layer_idx
        self.residual_in_fp32 = config.residual_in_fp32
        self.norm = Mamba2RMSNorm(config.hidden_size, eps=config.layer_norm_epsilon,
                                  sequence_parallel_enabled=config.sequence_parallel_enabled,
                                  dtype=config.dtype or torch.float32, device=device)
        self.mixer = Mamba2Mixer(config, layer_idx=layer_idx, device=device)

    def _in_one_call(self, op, method: str, hidden_states, residual, residual_dtype, conv_state, ssm_state):
        """`op`, one native call that stands for `method` of the mixer and what surrounds it, where the block is made of the
        plain modules on one rank.  None where any is of another class, has a hook or a method set on it or on its class, holds a
        weight that is no parameter of its own (parametrised, pruned), or out_proj has a bias: these keep the calls one by one.  (The modules' own
        dictionaries: attribute lookups of a module cost the host more than the launches.)"""
        norm, m = self._modules["norm"], self._modules["mixer"]
        if type(m) is not Mamba2Mixer or type(norm) is not Mamba2RMSNorm:
            return None
        parts, own = m._modules, m._parameters
        gate, conv, first, last = parts["norm"], parts["conv1d"]._parameters, parts["in_proj"], parts["out_proj"]
        if (method in vars(m) or "_core_kwargs" in vars(m) or "forward_add" in vars(norm) or (method == "forward" and _hooked(m))
                or _has_any_global_hook() or _stood_for() != _STOOD_FOR
                or type(gate) is not MambaRMSNormGated or type(first) is not ColumnParallelLinear or type(last) is not RowParallelLinear
                or "forward" in vars(first) or "forward" in vars(last) or _hooked(first) or _hooked(last)
                or last._parameters.get("bias", last) is not None or ps.get_tensor_model_parallel_size() != 1):
            return None
        try:
            weights = (norm._parameters["weight"], norm.variance_epsilon, first._parameters["weight"], first._parameters["bias"],
                       conv["weight"], conv["bias"], own["dt_bias"], own["A_log"], own["D"], gate._parameters["weight"],
                       last._parameters["weight"])
        except KeyError:
            return None
        return op(hidden_states, residual, residual_dtype, conv_state, ssm_state, *weights, m.intermediate_size_tp, m.n_groups_tp,
                  m.ssm_state_size, m.head_dim, m.layer_norm_epsilon, gate.group_size)

    def forward(self, hidden_states, residual=None, cache_params=None):
        rd = torch.float32 if self.residual_in_fp32 else None
        if (not torch.is_grad_enabled() and hidden_states.dim() == 3 and (cache_params is None or type(cache_params) is Mamba2Cache)):
            states = (None, None) if cache_params is None else (cache_params.conv_states[self.layer_idx],
                                                                cache_params.ssm_states[self.layer_idx])
            done = self._in_one_call(ops.block_forward, "forward", hidden_states, residual, rd, *states)
            if done is not None:
                return done
        normed, residual = self.norm.forward_add(hidden_states, residual, rd)
        return self.mixer(normed, cache_params=cache_params), residual

    def step(self, hidden_states, residual, cache_params):
        rd = torch.float32 if self.residual_in_fp32 else None
        if hidden_states.dim() == 3 and hidden_states.shape[1] == 1:
            done = self._in_one_call(ops.decode_block, "step", hidden_states, residual, rd, cache_params.conv_states[self.layer_idx],
                                     cache_params.ssm_states[self.layer_idx])
            if done is not None:
                return done
        normed, residual = self.norm.forward_add(hidden_states, residual, rd)
        return self.mixer.step(normed, cache_params), residual


@dataclass
class Mamba2Output(ModelOutput):
    last_hidden_state: Optional[torch.FloatTensor] = None
    cache_params: Optional[Mamba2Cache] = None
    hidden_states: Optional[Tuple[torch.FloatTensor]] = None


@dataclass
class Mamba2CausalLMOutput(ModelOutput):
    loss: Optional[torch.FloatTensor] = None
    logits: Optional[torch.FloatTensor] = None
    cache_params: Optional[Mamba2Cache] = None
    hidden_states: Optional[Tuple[torch.FloatTensor]] = None


class Mamba2PreTrainedModel(PreTrainedModel):
    config_class = Mamba2Config
    base_model_prefix = "backbone"
    _no_split_modules = ["Mamba2Block"]
    # per-head SSM parameters are created in fp32 whatever the model dtype: loading must not round them
    _keep_in_fp32_modules_strict = ["dt_bias", "A_log", "D"]
    supports_gradient_checkpointing = False
    _is_stateful = True

    def _init_weights(self, module):
        # parameters are drawn in the layer constructors (TP-consistent global draw, then slice)
        return


def _rename_legacy_keys(state_dict, prefix, *args):
    """Accept `embedding.` for `embeddings.` (mamba2/modeling_mamba2.py:236-240)."""
    for k in list(state_dict.keys()):
        if "embedding." in k:
            state_dict[k.replace("embedding.", "embeddings.")] = state_dict.pop(k)


class Mamba2Model(Mamba2PreTrainedModel):
    def __init__(self, config, device=None):
        super().__init__(config)
        dtype = config.dtype or torch.float32
        self.embeddings = ParallelEmbedding(config.vocab_size, config.hidden_size,
                                            init_method=normal_init(config.initializer_range), dtype=dtype, device=device)
        self.layers = nn.ModuleList([Mamba2Block(config, layer_idx=i, device=device)
                                     for i in range(config.num_hidden_layers)])
        self.sequence_parallel_enabled = config.sequence_parallel_enabled and ps.get_tensor_model_parallel_size() > 1
        self.norm_f = Mamba2RMSNorm(config.hidden_size, eps=config.layer_norm_epsilon,
                                    sequence_parallel_enabled=config.sequence_parallel_enabled, dtype=dtype, device=device)
        self.gradient_checkpointing = False
        self._register_load_state_dict_pre_hook(_rename_legacy_keys)
        self.post_init()

    def get_input_embeddings(self):
        return self.embeddings

    def set_input_embeddings(self, new_embeddings):
        self.embeddings = new_embeddings

    def forward(self, input_ids=None, inputs_embeds=None, cache_params: Optional[Mamba2Cache] = None,
                use_cache: Optional[bool] = None, output_hidden_states: Optional[bool] = None,
                return_dict: Optional[bool] = None, **kwargs):
        if (input_ids is None) == (inputs_embeds is None):
            raise ValueError("pass exactly one of input_ids and inputs_embeds")
        sp = self.sequence_parallel_enabled
        if inputs_embeds is None:
            hidden = self.embeddings(input_ids, scatter_to_sequence_parallel=sp)
        else:
            hidden = mp.scatter_to_sequence_parallel_region(inputs_embeds) if sp else inputs_embeds
        if use_cache and cache_params is None:
            cache_params = Mamba2Cache(self.config, hidden.shape[0], dtype=hidden.dtype, device=hidden.device)
        if use_cache and cache_params.seqlen_offset > 0 and hidden.shape[1] == 1 and not self.training:
            # incremental decoding (what `generate()` does after the prompt): one token over the cached states
            residual = None
            for block in self.layers:
                hidden, residual = block.step(hidden, residual, cache_params)
            rd = torch.float32 if self.config.residual_in_fp32 else None
            hidden, _ = self.norm_f.forward_add(hidden, residual, rd)
            cache_params.seqlen_offset += 1
            return Mamba2Output(last_hidden_state=hidden, cache_params=cache_params)
        all_hidden = () if output_hidden_states else None
        residual = None
        for block in self.layers:
            hidden, residual = block(hidden, residual, cache_params=cache_params if use_cache else None)
            if output_hidden_states:
                all_hidden = all_hidden + ((hidden + residual).to(hidden.dtype),)
        rd = torch.float32 if self.config.residual_in_fp32 else None
        hidden, _ = self.norm_f.forward_add(hidden, residual, rd)
        if use_cache:
            cache_params.seqlen_offset += (input_ids if input_ids is not None else inputs_embeds).shape[1]
        if return_dict is False:
            return tuple(v for v in (hidden, cache_params, all_hidden) if v is not None)
        return Mamba2Output(last_hidden_state=hidden, cache_params=cache_params if use_cache else None,
                            hidden_states=all_hidden)

    @torch.no_grad()
    def step(self, input_ids, cache_params: Mamba2Cache):
        """One decode token through all blocks (mamba2/modeling_mamba2.py:337-350)."""
        if ps.get_tensor_model_parallel_size() > 1 and input_ids.is_cuda:
            from ..parallel import symm
            symm.advance_step(compact=True)      # fresh sequence numbers for this token's fused collectives
        hidden = self.embeddings(input_ids)
        residual = None
        for block in self.layers:
            hidden, residual = block.step(hidden, residual, cache_params)
        rd = torch.float32 if self.config.residual_in_fp32 else None
        hidden, _ = self.norm_f.forward_add(hidden, residual, rd)
        cache_params.seqlen_offset += 1
        return hidden


def _delivers_statistics(head) -> bool:
    """True for the plain head, whose GEMM can take the cross-entropy statistics along.  Any other module, a bias or a
    gathered output has no such form; a hook, or a forward set on the module, gets the tensor that the head returns."""
    return (type(head) is ColumnParallelLinear and head.bias is None and not head.gather_output and "forward" not in vars(head)
            and not (_hooked(head) or _has_any_global_hook()))


def _shift_labels(labels):
    shifted = torch.full_like(labels, -100)
    shifted[:, :-1] = labels[:, 1:]
    return shifted


def _mean_loss(logits, shifted, stats):
    return parallel_cross_entropy(logits, shifted, stats=stats).sum() / (shifted.shape[0] * (shifted.shape[1] - 1))


class Mamba2ForCausalLM(Mamba2PreTrainedModel, GenerationMixin):
    _tied_weights_keys = {"lm_head.weight": "backbone.embeddings.weight"}

    def __init__(self, config, device=None):
        super().__init__(config)
        dtype = config.dtype or torch.float32
        self.backbone = Mamba2Model(config, device=device)
        self.lm_head = ColumnParallelLinear(config.hidden_size, config.vocab_size, bias=False,
                                            init_method=normal_init(config.initializer_range), dtype=dtype,
                                            sequence_parallel_enabled=config.sequence_parallel_enabled, device=device)
        self.post_init()
        if config.tie_word_embeddings:
            self.lm_head.weight = self.backbone.embeddings.weight

    def get_output_embeddings(self):
        return self.lm_head

    def set_output_embeddings(self, new_embeddings):
        self.lm_head = new_embeddings

    def get_input_embeddings(self):
        return self.backbone.get_input_embeddings()

    def set_input_embeddings(self, new_embeddings):
        return self.backbone.set_input_embeddings(new_embeddings)

    def prepare_inputs_for_generation(self, input_ids, inputs_embeds=None, use_cache=None,
                                      cache_params: Optional[Mamba2Cache] = None, **kwargs):
        if cache_params is not None and cache_params.seqlen_offset > 0:
            input_ids = input_ids[:, -1:]
        model_inputs = {"input_ids": input_ids} if inputs_embeds is None or cache_params is not None \
            else {"inputs_embeds": inputs_embeds}
        model_inputs.update({"cache_params": cache_params, "use_cache": use_cache})
        return model_inputs

    def forward(self, input_ids=None, inputs_embeds=None, cache_params: Optional[Mamba2Cache] = None,
                labels=None, output_hidden_states=None, return_dict=None, use_cache=None, **kwargs):
        """Logits are `[B, L, V/TP]` fp32 (the local vocabulary shard under TP); the loss is the
        mean vocab-parallel cross entropy of logits[:, :-1] against labels[:, 1:]
        (mamba2/modeling_mamba2.py:498-510)."""
        out = self.backbone(input_ids=input_ids, inputs_embeds=inputs_embeds, cache_params=cache_params,
                            use_cache=use_cache, output_hidden_states=output_hidden_states, return_dict=True)
        hidden = out.last_hidden_state
        loss, logits = None, None
        if labels is not None and not kwargs.get("return_logits", True):
            loss = self.loss_from_hidden(hidden, labels)
        else:
            logits, loss = self.logits_and_loss(hidden, labels)
        if return_dict is False:
            return tuple(v for v in (loss, logits, out.cache_params, out.hidden_states) if v is not None)
        return Mamba2CausalLMOutput(loss=loss, logits=logits, cache_params=out.cache_params,
                                    hidden_states=out.hidden_states)

    def logits_and_loss(self, hidden, labels):
        """(fp32 logits, loss or None); the loss is a function of these logits in autograd.  Where the head's GEMM delivers
        the cross-entropy statistics of its rows the loss comes from them; a shifted copy of the fp32 logits and two passes
        over it took half of a scoring call."""
        tp = ps.get_tensor_model_parallel_size() if self.backbone.sequence_parallel_enabled else 1
        if (labels is not None and _delivers_statistics(self.lm_head) and hidden.is_cuda and hidden.dtype == torch.bfloat16
                and labels.device == hidden.device and labels.dtype == torch.int64
                and tuple(labels.shape) == (hidden.shape[0], hidden.shape[1] * tp)):
            shifted = _shift_labels(labels)
            logits, stats = self.lm_head(hidden, ce_labels=shifted)
            logits = ops.widen(logits)
            return logits, _mean_loss(logits, shifted, stats)
        logits = ops.widen(self.lm_head(hidden))
        if labels is None:
            return logits, None
        return logits, parallel_cross_entropy(logits[:, :-1, :], labels[:, 1:].to(logits.device)).mean()

    def loss_from_hidden(self, hidden, labels):
        """Loss without materialising fp32 logits for the caller: labels are shifted instead of
        the logits (position L-1 is ignored), the mean runs over the B*(L-1) real targets."""
        shifted = _shift_labels(labels).to(hidden.device)
        logits, stats = self.lm_head(hidden, ce_labels=shifted)
        return _mean_loss(logits, shifted, stats)

    @torch.no_grad()
    def prefill(self, input_ids, cache_params: Optional[Mamba2Cache] = None):
        """Run the chunked scan over a prompt, fill the cache, return last-token logits."""
        if cache_params is None:
            p = next(self.parameters())
            cache_params = Mamba2Cache(self.config, input_ids.shape[0], dtype=p.dtype, device=p.device)
        out = self.backbone(input_ids=input_ids, cache_params=cache_params, use_cache=True)
        return ops.widen(self.lm_head(out.last_hidden_state[:, -1:, :])), cache_params

    @torch.no_grad()
    def generate(self, inputs=None, max_new_tokens: Optional[int] = None, max_length: Optional[int] = None,
                 do_sample: bool = False, temperature: float = 1.0, top_k: Optional[int] = None,
                 eos_token_id: Optional[int] = None, input_ids=None, generator=None, **unused):
        """`GenerationMixin.generate`-style entry point on top of `generate_tokens` (the framework's own conv/SSM
        cache drives decoding; HuggingFace's generic loop would hand the model a KV cache object it cannot use).
        Supports greedy decoding and temperature / top-k sampling; other generation options are not implemented."""
        ids = inputs if inputs is not None else input_ids
        if ids is None:
            raise ValueError("generate() needs input ids")
        if unused:
            ignored = sorted(k for k in unused if unused[k] is not None)
            if ignored:
                import logging
                logging.getLogger(__name__).warning("generate(): ignoring unsupported options %s", ignored)
        if max_new_tokens is None:
            max_new_tokens = max(0, (max_length or ids.shape[1] + 20) - ids.shape[1])
        if eos_token_id is None:
            eos_token_id = getattr(self.generation_config, "eos_token_id", None) if hasattr(self, "generation_config") else None
            if isinstance(eos_token_id, (list, tuple)):
                eos_token_id = eos_token_id[0] if eos_token_id else None
        return self.generate_tokens(ids, max_new_tokens, temperature=temperature if do_sample else 0.0, top_k=top_k,
                                    eos_token_id=eos_token_id, generator=generator)

    @torch.no_grad()
    def generate_tokens(self, input_ids, max_new_tokens: int, temperature: float = 0.0, top_k: Optional[int] = None,
                        eos_token_id: Optional[int] = None, generator=None):
        """Prompt -> continuation with the cached decode path: the longest 128-multiple prefix of the prompt goes
        through the chunked scan (prefill), the rest of the prompt and every new token through `step`.
        temperature 0 = greedy.  Returns [B, L + new] token ids.  (HuggingFace's `generate()` plumbing is kept for
        API compatibility, but like in the reference it does not drive this cache.)"""
        B, L = input_ids.shape
        p = next(self.parameters())
        cache = Mamba2Cache(self.config, B, dtype=p.dtype, device=p.device)
        chunk = 128
        Lp = (L // chunk) * chunk
        logits = None
        if Lp:
            logits, cache = self.prefill(input_ids[:, :Lp], cache)
        for t in range(Lp, L):
            logits = self.step(input_ids[:, t:t + 1], cache)
        out = [input_ids]
        done = torch.zeros(B, dtype=torch.bool, device=input_ids.device)
        for _ in range(max_new_tokens):
            last = logits[:, -1].float()
            if temperature and temperature > 0:
                if ps.get_tensor_model_parallel_size() > 1:      # sampling needs the whole vocabulary
                    parts = [torch.empty_like(last) for _ in range(ps.get_tensor_model_parallel_size())]
                    torch.distributed.all_gather(parts, last.contiguous(), group=ps.get_tensor_model_parallel_group())
                    last = torch.cat(parts, dim=-1)
                last = last / temperature
                if top_k:
                    kth = torch.topk(last, top_k, dim=-1).values[:, -1:]
                    last = last.masked_fill(last < kth, float("-inf"))
                nxt = torch.multinomial(torch.softmax(last, -1), 1, generator=generator)
            else:
                nxt = parallel_argmax(last).unsqueeze(-1)
            out.append(nxt)
            if eos_token_id is not None:
                done |= nxt[:, 0] == eos_token_id
                if bool(done.all()):
                    break
            logits = self.step(nxt, cache)
        return torch.cat(out, dim=1)

    @torch.no_grad()
    def step(self, input_ids, cache_params: Mamba2Cache):
        """Single-token decode: logits for the next token (mamba2/modeling_mamba2.py:523-531)."""
        hidden = self.backbone.step(input_ids, cache_params)
        return ops.widen(self.lm_head(hidden))
