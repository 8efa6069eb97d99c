"""Autograd wrappers around the native sm_100a kernels (GPU path of `ops.functional`).

Tensors are passed to the C ABI as raw device pointers on the current CUDA stream.  The kernels
report asynchronous failures (a bounded wait that ran out) through a device status word; `check_status()`
reads it (this synchronises) and raises.
"""
from __future__ import annotations

import ctypes
import functools
import struct
from typing import Optional

import torch
from torch.autograd import forward_ad as _forward_ad

from . import native

_c = ctypes
_status = {}
_launches = [0]


def launch_count() -> int:
    """Number of native kernel launches issued by this process so far."""
    return _launches[0]


def _lib():
    return native.lib()


class _P:
    """Pointer argument that keeps its tensor alive until the launch call has returned: a temporary
    (`x.float()`, `.contiguous()`) must not be freed, and its block handed to the next temporary in the
    same argument list, before the kernel is enqueued."""
    __slots__ = ("t", "_as_parameter_")

    def __init__(self, t):
        self.t = t
        self._as_parameter_ = _c.c_void_p(0 if t is None else t.data_ptr())


def _p(t: Optional[torch.Tensor]):
    return _P(t)


def _st():
    return _c.c_void_p(torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice()))


def _ll(v):
    return _c.c_longlong(int(v))


def status_tensor(device=None) -> torch.Tensor:
    t = _status.get(device)                 # the device of a tensor carries its index: the key as it is stored
    if t is not None:
        return t
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    if device not in _status:
        _status[device] = torch.zeros(1, dtype=torch.int32, device=device)
    return _status[device]


def check_status() -> None:
    for dev, t in _status.items():
        code = int(t.item())
        if code != 0:
            t.zero_()
            raise RuntimeError(f"native kernel reported status {code} on {dev} "
                               "(1: mbarrier wait timed out, 2: flag wait timed out, 3: bad argument)")


_functions = {}


def _run(name: str, *args):
    fn = _functions.get(name)
    if fn is None:
        fn = getattr(_lib(), name)
        fn.restype = _c.c_int
        _functions[name] = fn
    code = fn(*args)
    _launches[0] += 1
    if code != 0:
        raise RuntimeError(f"{name} failed with code {code} (negative: argument check, positive: cudaError_t)")


class _NoGrad:
    """What a Function's forward gets in place of its context when nothing is recorded."""

    def save_for_backward(self, *tensors):
        pass

    def mark_non_differentiable(self, *tensors):
        pass


def _observed() -> bool:
    """True where forward-mode differentiation, a functorch transform or `torch.jit.trace` wants to see the call: a tracer
    that saw the tensors made inside would record them without the kernel that fills them through their addresses."""
    return (_forward_ad._current_level >= 0 or torch._C._are_functorch_transforms_active()
            or torch._C._get_tracing_state() is not None)


def _recording() -> bool:
    """True where autograd or one of the observers above may want to see the call."""
    return torch.is_grad_enabled() or _observed()


def _apply(function, *args):
    """`function.apply`, or its forward alone where autograd would record nothing: entering and leaving an autograd
    Function costs the host 5 to 10 us per call, half of a small kernel's launch.  Forward-mode differentiation, functorch
    transforms and tracing keep `apply`, which answers them."""
    if _recording():
        return function.apply(*args)
    return function.forward(_NoGrad(), *args)


def _require_bf16(*ts):
    for t in ts:
        if t is not None and t.dtype != torch.bfloat16:
            raise TypeError(f"GPU kernels take bfloat16 activations/weights, got {t.dtype}")


def _ceil8(n: int) -> int:
    return (n + 7) // 8 * 8


# ======================================================================================
# GEMM
# ======================================================================================
def _as_operand(t: torch.Tensor) -> torch.Tensor:
    """2D, unit inner stride, row stride % 8 == 0, 16-byte aligned base (TMA requirements)."""
    if t.dim() != 2:
        raise ValueError("GEMM operands are 2D")
    if t.stride(1) != 1 or t.stride(0) % 8 or t.data_ptr() % 16:
        cols = _ceil8(t.shape[1])
        buf = torch.zeros(t.shape[0], cols, dtype=t.dtype, device=t.device) if cols != t.shape[1] else \
            torch.empty(t.shape[0], cols, dtype=t.dtype, device=t.device)
        buf[:, :t.shape[1]].copy_(t)
        return buf[:, :t.shape[1]]
    return t


def gemm(a: torch.Tensor, b: torch.Tensor, a_mn: bool = False, b_mn: bool = False, out: Optional[torch.Tensor] = None,
         out_dtype=torch.bfloat16, accumulate: bool = False, bias: Optional[torch.Tensor] = None,
         gelu: bool = False, sumsq: Optional[torch.Tensor] = None) -> torch.Tensor:
    """C[M,N] = A B on tcgen05.  a is [M,K] (or [K,M] when a_mn), b is [N,K] (or [K,N] when b_mn).
    out: bf16 (fresh, row stride padded to 8) or fp32 (`accumulate` adds into `out`).
    sumsq (fp32 scalar tensor, fp32 store only): the kernel adds sum(C^2) to it."""
    _require_bf16(a, b, bias)
    a, b = _as_operand(a), _as_operand(b)
    M, K = (a.shape[1], a.shape[0]) if a_mn else (a.shape[0], a.shape[1])
    N, Kb = (b.shape[1], b.shape[0]) if b_mn else (b.shape[0], b.shape[1])
    if K != Kb:
        raise ValueError(f"GEMM inner dimensions differ: {K} vs {Kb}")
    if out is None:
        if out_dtype == torch.bfloat16:
            out = torch.empty(M, _ceil8(N), dtype=torch.bfloat16, device=a.device)[:, :N]
        else:
            out = torch.empty(M, (N + 3) // 4 * 4, dtype=torch.float32, device=a.device)[:, :N]
    if out.dtype == torch.float32 and (out.stride(0) % 4 or out.data_ptr() % 16) and out.stride(1) == 1:
        # TMA needs 16-byte aligned rows: go through a padded temporary
        tmp = gemm(a, b, a_mn=a_mn, b_mn=b_mn, out_dtype=torch.float32, sumsq=sumsq)
        if accumulate:
            out.add_(tmp)
        else:
            out.copy_(tmp)
        return out
    if out.dtype == torch.bfloat16:
        mode = 0
        if out.stride(1) != 1 or out.stride(0) % 8 or out.data_ptr() % 16:
            raise ValueError("bf16 GEMM output needs unit inner stride, row stride % 8 == 0, 16-byte base")
    else:
        mode = 2 if accumulate else 1
        if out.stride(1) != 1:
            raise ValueError("fp32 GEMM output needs unit inner stride")
    if sumsq is not None:
        if mode != 1 or sumsq.dtype != torch.float32:
            raise ValueError("sumsq needs an fp32 output that is stored, not accumulated")
        _run("ssm_gemm_bf16_ex", _p(a), _p(b), _p(out), M, N, K, _ll(a.stride(0)), _ll(b.stride(0)), _ll(out.stride(0)),
             int(a_mn), int(b_mn), mode, _p(bias), int(gelu), _p(status_tensor(a.device)), _st(), _p(sumsq))
        return out
    _run("ssm_gemm_bf16", _p(a), _p(b), _p(out), M, N, K, _ll(a.stride(0)), _ll(b.stride(0)), _ll(out.stride(0)),
         int(a_mn), int(b_mn), mode, _p(bias), int(gelu), _p(status_tensor(a.device)), _st())
    return out


def ce_epilogue_buffers(M: int, N: int, K: int, labels: torch.Tensor, vocab_start: int, rows_per_shard: int = 0):
    """Buffers for a GEMM whose epilogue emits cross-entropy statistics of its [M, N] output (the LM head):
    (arguments for the kernel, number of column tiles).  `labels` [M] int64 global ids, negative = ignored;
    `rows_per_shard`: shard rows when the GEMM is the all-gather variant (it decides the tile shape), else 0."""
    fn = _lib().ssm_gemm_ce_tiles
    fn.restype = _c.c_int
    tiles = int(fn(int(M), int(N), int(K), int(rows_per_shard)))
    dev = labels.device
    lab = labels.reshape(-1).contiguous()
    if lab.numel() != M or lab.dtype != torch.int64:
        raise ValueError("labels must be int64 with one entry per output row")
    return dict(labels=lab, vocab_start=int(vocab_start),
                tmax=torch.empty(tiles, M, dtype=torch.float32, device=dev),
                tsum=torch.empty(tiles, M, dtype=torch.float32, device=dev),
                tgt=torch.zeros(M, dtype=torch.float32, device=dev)), tiles


def ce_merge(ced, tiles: int):
    """Per-tile statistics -> (row max, row sum of exp(x - max), target logit or 0) for this vocabulary shard."""
    M = ced["tgt"].numel()
    m = torch.empty(M, dtype=torch.float32, device=ced["tgt"].device)
    s = torch.empty_like(m)
    _run("ssm_ce_merge_tiles", _p(ced["tmax"]), _p(ced["tsum"]), int(tiles), _ll(M), _p(m), _p(s), _st())
    return m, s, ced["tgt"]


def gemm_ce(a: torch.Tensor, b: torch.Tensor, labels: torch.Tensor, vocab_start: int):
    """y = a b^T (bf16, [M, N]) together with the cross-entropy statistics of its rows, produced by the GEMM
    epilogue (no second pass over the logits): returns (y, (max, sumexp, target))."""
    _require_bf16(a, b)
    a, b = _as_operand(a), _as_operand(b)
    M, K = a.shape
    N = b.shape[0]
    out = torch.empty(M, _ceil8(N), dtype=torch.bfloat16, device=a.device)[:, :N]
    ced, tiles = ce_epilogue_buffers(M, N, K, labels, vocab_start)
    _run("ssm_gemm_bf16_ce", _p(a), _p(b), _p(out), M, N, K, _ll(a.stride(0)), _ll(b.stride(0)), _ll(out.stride(0)),
         _p(status_tensor(a.device)), _st(), _p(ced["labels"]), _ll(ced["vocab_start"]), _p(ced["tmax"]),
         _p(ced["tsum"]), _p(ced["tgt"]))
    return out, ce_merge(ced, tiles)


def wgrad_to_main_grad(dy2: torch.Tensor, x2: torch.Tensor, w) -> bool:
    """dW = dY^T X written straight into the optimizer's fp32 `w.main_grad`: stored on the first contribution of a
    step (lazy zeroing), added afterwards.  When the optimizer has given the weight a norm accumulator (`w.norm_acc`)
    a stored gradient also adds its sum of squares to it (`w.norm_tracked` tells the optimizer that this weight's
    share of the gradient norm is already there).  False: no fp32 main_grad, the caller returns dW through autograd."""
    mg = getattr(w, "main_grad", None)
    if mg is None or mg.dtype != torch.float32:
        return False
    stale = getattr(w, "grad_stale", False)
    acc = getattr(w, "norm_acc", None) if stale else None
    if acc is not None and getattr(w, "scatter_added", False) and not _follow_norm(dy2.shape[0], w.shape[0]):
        acc = None
    if not stale:
        untrack_norm(w)
    gemm(dy2, x2, a_mn=True, b_mn=True, out=mg, accumulate=not stale, sumsq=acc)
    w.grad_stale = False
    if acc is not None:
        w.norm_tracked = True
        if getattr(w, "scatter_added", False):
            w.norm_version = mg._version
    return True


def _follow_norm(tokens: int, rows: int) -> bool:
    """Whether the additions of an embedding's gradient carry the gradient norm on (ssm_embed_bwd with an accumulator), or the norm
    of its rows is taken by a pass over all of them.  Additions that bring the old value back cost 25 to 40 us more, the pass reads 4
    bytes per value of the table (tokens x columns into rows: additions with and without, pass; us, cold): 2048 x 4096 into 50288
    49, 21, 144; 8192 x 4096 into 50288 96, 60, 143; 8192 x 2560 into 50288 84, 45, 100; 8192 x 1024 into 50288 53, 25, 45; 12288 x 2560
    into 50288 105, 63, 100; 4096 x 2560 into 16384 59, 27, 39; 4096 x 1024 into 16384 41, 16, 21; 2048 x 4096 into 6286 47, 21, 29.
    From six rows per token on following wins at every width; between three and six it wins or loses with the width and the table,
    and the pass, which takes no atomic additions with results, is kept there."""
    return tokens * 6 <= rows


def untrack_norm(w) -> None:
    """The gradient of `w` is about to change after a GEMM may already have added its sum of squares to the norm
    accumulator: mark the weight so that the optimizer recomputes the norm from the buffers this step."""
    if getattr(w, "norm_tracked", False):
        w.norm_tracked = False
        w.norm_dirty = True


def untrack_edited(w) -> None:
    """The same where operations of the program have written into the embedding's gradient since a kernel last added to the norm
    (rows of frozen tokens set to zero, say).  They are seen by the version counter, which the optimizer's flat buffer and all
    gradients in it share; writes through `.data` have a counter of their own and are not seen."""
    if getattr(w, "norm_tracked", False) and w.main_grad._version != w.norm_version:
        untrack_norm(w)


class _Linear(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, bias, ce_labels=None, ce_vocab_start=0):
        K = x.shape[-1]
        x2 = x.reshape(-1, K)
        ctx.save_for_backward(x2, w)
        ctx.has_bias = bias is not None
        ctx.xshape = x.shape
        if ce_labels is not None:
            y, stats = gemm_ce(x2, w, ce_labels, ce_vocab_start)
            ctx.mark_non_differentiable(*stats)
            return (y.reshape(*x.shape[:-1], w.shape[0]),) + tuple(stats)
        y = gemm(x2, w, bias=bias)
        return y.reshape(*x.shape[:-1], w.shape[0])

    @staticmethod
    def backward(ctx, dy, *unused):
        x2, w = ctx.saved_tensors
        N = w.shape[0]
        dy2 = dy.reshape(-1, N)
        dx = dw = db = None
        if ctx.needs_input_grad[0]:
            dx = gemm(dy2, w, b_mn=True).reshape(ctx.xshape)          # dX = dY W
        if ctx.needs_input_grad[1]:
            if not wgrad_to_main_grad(dy2, x2, w):                       # main_grad (+)= dY^T X
                dw = gemm(dy2, x2, a_mn=True, b_mn=True)
                if not dw.is_contiguous():
                    dw = dw.contiguous()
        if ctx.has_bias and ctx.needs_input_grad[2]:
            db = dy2.float().sum(0).to(dy.dtype)
        return dx, dw, db, None, None


def linear(x, w, bias=None):
    _require_bf16(x, w)
    return _apply(_Linear, x, w, bias)


def linear_ce(x, w, labels, vocab_start: int = 0):
    """(x w^T, (row max, row sum-exp, target logit)): the LM head with the cross-entropy statistics taken in the
    GEMM epilogue (mamba2/modeling_mamba2.py:498-510 computes them in separate passes over fp32 logits)."""
    _require_bf16(x, w)
    out = _apply(_Linear, x, w, None, labels, int(vocab_start))
    return out[0], tuple(out[1:])


# ======================================================================================
# conv
# ======================================================================================
def _conv_fwd(xBC, w2, bias, init, out=None):
    B, L, C = xBC.shape
    assert xBC.stride(2) == 1 and xBC.stride(0) == L * xBC.stride(1)
    if out is None:
        out = torch.empty(B, L, C, dtype=xBC.dtype, device=xBC.device)
    _run("ssm_conv1d_silu_fwd", _p(xBC), _ll(xBC.stride(1)), _p(w2), _p(bias), _p(init), _p(out), _ll(out.stride(1)),
         B, L, C, _st())
    return out


def _conv_bwd(xBC, w2, bias, dy16, dy32, c_split, dx_out, raw=False):
    """dx_out [B,L,C] view (row stride may exceed C); returns (dw [C,K], db [C]) fp32, or the per-tile partial
    buffer [tiles, C, 5] when `raw`."""
    B, L, C = xBC.shape
    tile = _lib().ssm_conv_bwd_tok_tile(B, L, C)
    ntile = (L + tile - 1) // tile
    part = torch.empty(B * ntile, C, 5, dtype=torch.float32, device=xBC.device)
    _run("ssm_conv1d_silu_bwd", _p(xBC), _ll(xBC.stride(1)), _p(w2), _p(bias), _p(dy16),
         _ll(dy16.stride(1) if dy16 is not None else 0), _p(dy32), _ll(dy32.stride(1) if dy32 is not None else 0),
         int(c_split), _p(dx_out), _ll(dx_out.stride(1)), _p(part), B, L, C, _st())
    if raw:
        return part
    s = part.sum(0)
    return s[:, :4], s[:, 4]


class _Conv(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, bias, init):
        C = x.shape[-1]
        w2 = w.reshape(C, -1).contiguous()
        if not (x.stride(2) == 1 and x.stride(0) == x.shape[1] * x.stride(1) and x.stride(1) % 8 == 0):
            x = x.contiguous()
        init3 = None if init is None else init[:, -3:, :].contiguous()
        out = _conv_fwd(x, w2, bias, init3)
        ctx.save_for_backward(x, w2, bias)
        ctx.wshape = w.shape
        return out

    @staticmethod
    def backward(ctx, dy):
        x, w2, bias = ctx.saved_tensors
        dy = dy.contiguous()
        dx = torch.empty(x.shape, dtype=x.dtype, device=x.device)
        dw, db = _conv_bwd(x, w2, bias, dy, None, x.shape[-1], dx)
        return dx, dw.to(w2.dtype).reshape(ctx.wshape), (None if bias is None else db.to(bias.dtype)), None


def _require_four_taps(weight, channels: int) -> None:
    if weight.numel() != 4 * channels:
        raise ValueError(f"the conv kernels are written for 4 taps of {channels} channels, got {tuple(weight.shape)}")


def causal_conv1d_silu(x, weight, bias, initial_state=None):
    _require_bf16(x, weight, bias)
    if weight.shape[-1] != 4:
        raise ValueError("the conv kernels are written for 4 taps")
    _require_four_taps(weight, x.shape[-1])
    return _apply(_Conv, x, weight, bias, initial_state)


# ======================================================================================
# norms
# ======================================================================================
_ROW_SLICES = 296


def _gated_fwd(y2, z2, w, eps, gs, out=None):
    rows, d = y2.shape
    if out is None:
        out = torch.empty(rows, d, dtype=y2.dtype, device=y2.device)
    _run("ssm_gated_rmsnorm_fwd", _p(y2), _ll(y2.stride(0)), _p(z2), _ll(z2.stride(0) if z2 is not None else 0), _p(w),
         _p(out), _ll(out.stride(0)), _ll(rows), d, gs, _c.c_float(eps), _st())
    return out


def _gated_bwd(y2, z2, w, dout2, eps, gs, dy_out, dz_out, raw=False):
    rows, d = y2.shape
    # one block per SM of the widest groups, two, or four of narrow rows (us with 148 / 296 / 592 slices, column sums included:
    # 2048 x 8192 43 / 52 / 61, 8192 x 5120 121 / 99 / 103, 2688 x 3072 35 / 28 / 32, 8192 x 2048 88 / 57 / 47, 4608 x 1536 42 / 31 / 25)
    slices = int(min(rows, _ROW_SLICES // 2 if gs > 5120 else _ROW_SLICES if d >= 2560 else _ROW_SLICES * 2))
    part = torch.empty(slices, d, dtype=torch.float32, device=y2.device)
    _run("ssm_gated_rmsnorm_bwd", _p(y2), _ll(y2.stride(0)), _p(z2), _ll(z2.stride(0) if z2 is not None else 0), _p(w),
         _p(dout2), _ll(dout2.stride(0)), _p(dy_out), _ll(dy_out.stride(0)), _p(dz_out),
         _ll(dz_out.stride(0) if dz_out is not None else 0), _p(part), slices, _ll(rows), d, gs, _c.c_float(eps),
         _p(status_tensor(y2.device)), _st())
    return part if raw else part.sum(0)


def _rows(t):
    """[..., d] -> 2D view with unit inner stride (copy only if needed)."""
    d = t.shape[-1]
    if t.dim() == 2 and t.stride(1) == 1:
        return t
    if t.stride(-1) == 1 and t.dim() == 3 and t.stride(0) == t.shape[1] * t.stride(1):
        return t.as_strided((t.shape[0] * t.shape[1], d), (t.stride(1), 1), t.storage_offset())
    return t.reshape(-1, d).contiguous()


class _GatedNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, y, z, w, eps, gs):
        y2, z2 = _rows(y), (None if z is None else _rows(z))
        out = _gated_fwd(y2, z2, w, eps, gs)
        ctx.save_for_backward(y2, z2, w)
        ctx.eps, ctx.gs, ctx.shape = eps, gs, y.shape
        return out.reshape(y.shape)

    @staticmethod
    def backward(ctx, dout):
        y2, z2, w = ctx.saved_tensors
        d2 = _rows(dout.contiguous())
        dy = torch.empty(y2.shape, dtype=y2.dtype, device=y2.device)
        dz = None if z2 is None else torch.empty(y2.shape, dtype=y2.dtype, device=y2.device)
        dw = _gated_bwd(y2, z2, w, d2, ctx.eps, ctx.gs, dy, dz)
        return dy.reshape(ctx.shape), (None if dz is None else dz.reshape(ctx.shape)), dw.to(w.dtype), None, None


def gated_rmsnorm(y, z, w, eps, group_size=None):
    _require_bf16(y, z, w)
    gs = y.shape[-1] if group_size is None else group_size
    return _apply(_GatedNorm, y, z, w, eps, gs)


class _AddRMSNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, residual, w, eps, res_dtype):
        D = x.shape[-1]
        x2 = x.reshape(-1, D).contiguous()
        rows = x2.shape[0]
        r2 = None if residual is None else residual.reshape(-1, D).contiguous()
        out = torch.empty_like(x2)
        res_out = torch.empty(rows, D, dtype=res_dtype, device=x.device)
        if r2 is not None and r2.dtype != res_dtype:
            r2 = r2.to(res_dtype)
        _run("ssm_add_rmsnorm_fwd", _p(x2), _p(r2), _p(w), _p(out), _p(res_out), _ll(rows), D, _c.c_float(eps),
             int(res_dtype == torch.float32), _st())
        ctx.save_for_backward(res_out, w)
        ctx.eps, ctx.shape, ctx.has_res = eps, x.shape, residual is not None
        ctx.x_dtype = x.dtype
        return out.reshape(x.shape), res_out.reshape(x.shape)

    @staticmethod
    def backward(ctx, dout, dres):
        res_out, w = ctx.saved_tensors
        rows, D = res_out.shape
        d2 = dout.reshape(rows, D).contiguous()
        dr2 = None if dres is None else dres.reshape(rows, D).contiguous()
        dsum = torch.empty_like(res_out)
        slices = int(min(rows, _ROW_SLICES))
        part = torch.empty(slices, D, dtype=torch.float32, device=res_out.device)
        _run("ssm_add_rmsnorm_bwd", _p(res_out), _p(w), _p(d2), _p(dr2), _p(dsum), _p(part), slices, _ll(rows), D,
             _c.c_float(ctx.eps), int(res_out.dtype == torch.float32), _st())
        dsum = dsum.reshape(ctx.shape)
        dx = dsum if dsum.dtype == ctx.x_dtype else dsum.to(ctx.x_dtype)
        mg = getattr(w, "main_grad", None)
        if mg is not None and mg.dtype == torch.float32 and w.is_leaf:
            _run("ssm_colsum", _p(part), slices, D, _p(mg), int(not getattr(w, "grad_stale", False)), _st())
            w.grad_stale = False
            return dx, (dsum if ctx.has_res else None), None, None, None
        return dx, (dsum if ctx.has_res else None), part.sum(0).to(w.dtype), None, None


def add_rmsnorm(x, residual, w, eps, residual_dtype=None):
    _require_bf16(x, w)
    rd = residual_dtype or x.dtype
    return _apply(_AddRMSNorm, x, residual, w, eps, rd)


def rmsnorm(x, w, eps):
    return add_rmsnorm(x, None, w, eps)[0]


# ======================================================================================
# GELU
# ======================================================================================
class _Gelu(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        xc = x.contiguous()
        y = torch.empty_like(xc)
        _run("ssm_gelu_fwd", _p(xc), _p(y), _ll(xc.numel()), _st())
        ctx.save_for_backward(xc)
        return y

    @staticmethod
    def backward(ctx, dy):
        (xc,) = ctx.saved_tensors
        dx = torch.empty_like(xc)
        _run("ssm_gelu_bwd", _p(xc), _p(dy.contiguous()), _p(dx), _ll(xc.numel()), _st())
        return dx


def gelu(x):
    _require_bf16(x)
    if x.numel() % 8:
        return torch.nn.functional.gelu(x)
    return _apply(_Gelu, x)


class _Glu(torch.autograd.Function):
    @staticmethod
    def forward(ctx, h, act):
        S = h.shape[-1] // 2
        h2 = h.reshape(-1, 2 * S)
        if h2.stride(1) != 1 or h2.stride(0) % 8 or h2.data_ptr() % 16:
            h2 = h2.contiguous()
        out = torch.empty(h2.shape[0], S, dtype=h.dtype, device=h.device)
        _run("ssm_glu_fwd", _p(h2), _ll(h2.stride(0)), _p(out), _ll(h2.shape[0]), S, act, _st())
        ctx.save_for_backward(h2)
        ctx.act, ctx.shape = act, h.shape
        return out.reshape(*h.shape[:-1], S)

    @staticmethod
    def backward(ctx, dout):
        (h2,) = ctx.saved_tensors
        S = h2.shape[1] // 2
        d2 = dout.reshape(-1, S).contiguous()
        dh = torch.empty(h2.shape[0], 2 * S, dtype=h2.dtype, device=h2.device)
        _run("ssm_glu_bwd", _p(h2), _ll(h2.stride(0)), _p(d2), _p(dh), _ll(h2.shape[0]), S, ctx.act, _st())
        return dh.reshape(ctx.shape), None


def glu(h, act: str = "silu"):
    """act(h[..., :S]) * h[..., S:] for h = [gate | up] in one kernel (forward and backward); act gelu or silu."""
    _require_bf16(h)
    if h.shape[-1] % 16 or act not in ("gelu", "silu", "swish"):
        raise ValueError("glu kernel needs an even split into multiples of 8 columns and act in {gelu, silu}")
    return _apply(_Glu, h, 0 if act == "gelu" else 1)


# ======================================================================================
# embedding
# ======================================================================================
def embed_grad_target(w, follow_norm: bool = False, tokens: int = 0):
    """(fp32 [V, D] buffer to accumulate into, direct, norm accumulator or None).  With an optimizer-owned `main_grad` the embedding
    backward adds into it in place (after the tied LM-head wgrad, which ran earlier in the backward pass).  follow_norm: the
    additions may go on with a gradient norm that the accumulator already holds (zeros, or what a GEMM stored and added);
    otherwise they make it stale."""
    mg = getattr(w, "main_grad", None)
    if mg is not None and mg.dtype == torch.float32 and mg.is_contiguous():
        untrack_edited(w)
        acc = getattr(w, "norm_acc", None) if follow_norm and not getattr(w, "norm_dirty", False) else None
        if getattr(w, "grad_stale", False):
            mg.zero_()
            w.grad_stale = False
            w.norm_tracked = acc is not None and _follow_norm(tokens, w.shape[0])
        if acc is None or not getattr(w, "norm_tracked", False):
            untrack_norm(w)             # scatter-added rows change the norm of a gradient a GEMM may have stored
            acc = None
        w.norm_version = mg._version
        return mg, True, acc
    return torch.zeros(w.shape, dtype=torch.float32, device=w.device), False, None


class _Embedding(torch.autograd.Function):
    @staticmethod
    def forward(ctx, ids, w, vocab_start):
        ids_c = ids.contiguous()
        out = torch.empty(*ids.shape, w.shape[1], dtype=w.dtype, device=w.device)
        _run("ssm_embed_lookup", _P(ids_c), _P(w), _ll(vocab_start), _ll(w.shape[0]), _P(out), _ll(ids_c.numel()),
             w.shape[1], _st())
        ctx.save_for_backward(ids_c)
        ctx.w, ctx.vocab_start = w, vocab_start
        return out

    @staticmethod
    def backward(ctx, g):
        (ids,), w = ctx.saved_tensors, ctx.w
        D = w.shape[1]
        g2 = g.reshape(-1, D)
        if g2.stride(1) != 1 or g2.stride(0) % 4:
            g2 = g2.contiguous()
        tgt, direct, acc = embed_grad_target(w, follow_norm=True, tokens=ids.numel())
        n = ids.numel()
        _run("ssm_embed_bwd", _P(ids), _P(g2), _ll(g2.stride(0)), _P(tgt), _ll(ctx.vocab_start), _ll(w.shape[0]), 1, n, n,
             D, 1, None, 0, 0, None, _P(acc), _P(status_tensor(w.device)), _st())
        return None, (None if direct else tgt.to(w.dtype)), None


def embedding(ids, w, vocab_start: int = 0):
    """Rows `w[ids - vocab_start]`, zeros for ids outside the local shard; the gradient is scatter-added in fp32."""
    if w.dtype != torch.bfloat16 or ids.dtype != torch.int64 or w.shape[1] % 8 or not w.is_contiguous():
        local = ids - vocab_start
        inside = (local >= 0) & (local < w.shape[0])
        return torch.nn.functional.embedding(torch.where(inside, local, torch.zeros_like(local)), w) \
            * inside[..., None].to(w.dtype)
    return _apply(_Embedding, ids, w, int(vocab_start))


# ======================================================================================
# cross entropy
# ======================================================================================
def ce_partials(logits, labels, vocab_start):
    rows, V = logits.shape
    assert logits.stride(1) == 1
    m = torch.empty(rows, dtype=torch.float32, device=logits.device)
    s, t = torch.empty_like(m), torch.empty_like(m)
    _run("ssm_ce_partials", _p(logits), _ll(logits.stride(0)), int(logits.dtype == torch.float32),
         _p(labels.contiguous()), _ll(rows), V, int(vocab_start), _p(m), _p(s), _p(t), _st())
    return m, s, t


def ce_backward(logits, labels, row_max, row_sum, grad_rows, vocab_start, ignore_index):
    rows, V = logits.shape
    ld = _ceil8(V)
    grad = torch.empty(rows, ld, dtype=logits.dtype, device=logits.device)[:, :V]
    if ld != V:
        grad.as_strided((rows, ld - V), (ld, 1), V).zero_()
    _run("ssm_ce_backward", _p(logits), _ll(logits.stride(0)), int(logits.dtype == torch.float32),
         _p(labels.contiguous()), _ll(rows), V, int(vocab_start), _ll(ignore_index), _p(row_max), _p(row_sum),
         _p(grad_rows.float().contiguous()), _p(grad), _ll(ld), _st())
    return grad


def ce_row_loss(m, s, tgt, labels, ignore_index):
    """log(s) + m - tgt per row, 0 where the label is ignored (fp32 statistics as ce_partials delivers them)."""
    rows = labels.numel()
    if (rows == 0 or labels.dtype != torch.int64 or labels.device != s.device or _observed()
            or not all(t.dtype == torch.float32 and t.is_contiguous() and t.numel() == rows for t in (m, s, tgt))):
        return torch.where(labels != ignore_index, torch.log(s) + m - tgt, torch.zeros_like(s))
    loss = torch.empty_like(s)
    _run("ssm_ce_row_loss", _p(m), _p(s), _p(tgt), _p(labels.contiguous()), _ll(ignore_index), _ll(rows), _p(loss), _st())
    return loss


def widen(x):
    """fp32 copy of bf16 `x` [..., n] (rows may be padded); inference only, the gradient path keeps `x.float()`."""
    if _observed():
        return x.float()
    n = x.shape[-1]
    x2 = x.reshape(-1, n) if x.dim() != 2 else x
    if (x.dtype != torch.bfloat16 or x2.shape[0] == 0 or x2.shape[0] > 65535 or n % 8 or n == 0 or x2.stride(1) != 1
            or x2.stride(0) % 8 or x2.data_ptr() % 16):
        return x.float()
    out = torch.empty(x.shape, dtype=torch.float32, device=x.device)
    _run("ssm_widen", _p(x2), _ll(x2.stride(0)), _p(out), _ll(x2.shape[0]), n, _st())
    return out


def row_max(x):
    """(largest value, its first index) of every row of fp32 x [..., V]; NaN counts as largest."""
    V = x.shape[-1]
    rows = x.numel() // V if V else 0
    x2 = x.reshape(-1, V) if x.dim() != 2 and rows else x
    if x.dtype != torch.float32 or rows == 0 or rows > 65535 or x2.stride(1) != 1 or V >= 2 ** 31 - 2 ** 16 or _observed():
        return x.float().max(dim=-1)
    val = torch.empty(x.shape[:-1], dtype=torch.float32, device=x.device)
    idx = torch.empty(x.shape[:-1], dtype=torch.int64, device=x.device)
    _run("ssm_row_max", _p(x2), _ll(x2.stride(0)), V, _ll(rows), _p(val), _p(idx), _st())
    return val, idx


# ======================================================================================
# optimizer
# ======================================================================================
def adamw_step(master, m, v, g, out, clip, lr, b1, b2, eps, wd, step, lr_dev=None, step_dev=None):
    """lr_dev (fp32 [1]) / step_dev (int32 [1]): device-resident values that override `lr` / `step`."""
    if master.dtype != torch.float32:
        raise TypeError("the fused AdamW keeps fp32 state")
    out16 = out if out.dtype == torch.bfloat16 else None
    out32 = out if out.dtype == torch.float32 else None
    _run("ssm_adamw", _p(master), _p(m), _p(v), _p(g), int(g.dtype == torch.float32), _p(out16), _p(out32),
         _ll(master.numel()), _p(clip), _c.c_float(lr), _c.c_float(b1), _c.c_float(b2), _c.c_float(eps),
         _c.c_float(wd), int(step), _p(lr_dev), _p(step_dev), _st())


def clip_coefficient(total, max_norm, step, skipped):
    """(gradient norm, clip coefficient or -1 where it is not finite) as fp32 [1] tensors from the norm's square; counts the step
    as applied (`step`) or skipped (int32 [1] tensors)."""
    norm, clip = torch.empty(1, dtype=torch.float32, device=total.device), torch.empty(1, dtype=torch.float32, device=total.device)
    _run("ssm_clip_coefficient", _p(total), _c.c_float(max_norm), _p(norm), _p(clip), _p(step), _p(skipped), _st())
    return norm, clip


def sumsq_accumulate(g, total):
    _run("ssm_sumsq", _p(g), int(g.dtype == torch.float32), _ll(g.numel()), _p(total), _st())


# ======================================================================================
# SSD scan and the fused mixer core
# ======================================================================================
_CT = 128


def _ssd_dims(d_inner, head_dim, n_groups, d_state):
    if d_state != 128:
        raise ValueError("the GPU SSD kernels are written for d_state = 128")
    if head_dim % 64:
        raise ValueError("the GPU SSD kernels need head_dim to be a multiple of 64")
    H = d_inner // head_dim
    psplit = head_dim // 64
    if H % n_groups:
        raise ValueError("heads must be divisible by groups")
    return H, psplit, H * psplit


def _chunk_states(conv_out, C, w_col0, v, v_stride, dt, l, init, want_final, B, L, H, Hv, G, mode):
    """(bf16 state [B, Hv, nc, 128, 64] on one side of every chunk, fp32 state [B, H, P, 128] behind the last one or None).  mode 0: states
    entering the chunks; mode 1: gradients of the states leaving them (the recurrence runs backwards)."""
    dev, nc, st = conv_out.device, L // _CT, status_tensor(conv_out.device)
    states = torch.empty(B, Hv, nc, 128, 64, dtype=torch.bfloat16, device=dev)
    if mode == 1 and _walk_states(B * Hv, nc):         # forwards, ssm_ssd_walk_scan walks and scans at once
        count = _segments(B * Hv, nc, _PER_CHUNK[1])
        ends = _segment_ends(conv_out, C, w_col0, v, v_stride, None, l, B, L, H, Hv, G, 0, count)
        _run("ssm_ssd_state_walk", _p(conv_out), _ll(C), C, w_col0, _p(v), _ll(v_stride), _p(None), _p(l), _p(states), B, L, H, Hv, G,
             0, count, _p(ends[0]), _p(ends[1]), _p(st), _st())
        return states, None
    final = torch.empty(B, Hv, 128, 64, dtype=torch.float32, device=dev) if want_final else None
    local = torch.empty(B, Hv, nc, 128, 64, dtype=torch.float32, device=dev)
    _run("ssm_ssd_chunk_state", _p(conv_out), _ll(C), C, w_col0, _p(v), _ll(v_stride), _p(dt), _p(l), _p(local),
         B, L, H, Hv, G, mode, _p(st), _st())
    _run("ssm_ssd_state_pass", _p(local), _p(l), _p(init), _p(states), _p(final), B, L, H, Hv, mode, _st())
    if want_final:
        final = final.transpose(2, 3).reshape(B, H, Hv // H * 64, 128)
    return states, final


def _walk_cost(slices: int, nc: int, count: int, per_chunk: float, sms: int = 148) -> float:
    """us of a walk of `count` segments: 5 us and the chunks of a segment for as many CTAs as there are SMs at once; with more
    than one segment also the launch that finds the states behind all but the last (1.35 us per chunk) and 0.7 us for each of
    these that a segment starts from."""
    length = -(-nc // count)
    cost = -(-slices * count // sms) * (5.0 + length * per_chunk)
    return cost if count == 1 else cost + -(-slices * (count - 1) // sms) * (5.0 + length * 1.35) + 0.7 * (count - 1)


_PER_CHUNK = (2.9, 1.35)               # us of a chunk of the forward walk, of the walk of the backward states


@functools.lru_cache(maxsize=4096)
def _segments(slices: int, nc: int, per_chunk: float) -> int:
    """Segments that the chunks of a walk are cut into (none of them empty).  Measured (us, with 4 us of other kernels forwards;
    slices x chunks: one / the count taken here): forward 16 x 64 165 / 51, 32 x 64 182 / 83, 64 x 16 47 / 44, 160 x 64 392 / 376,
    1 x 512 1189 / 101; backward states 16 x 64 90 / 36, 32 x 64 93 / 54."""
    return min((c for c in range(1, min(32, nc) + 1) if (c - 1) * -(-nc // c) < nc),
               key=lambda c: _walk_cost(slices, nc, c, per_chunk))


def _segment_ends(w, w_cols, w_col0, v, v_stride, dt, l, B, L, H, Hv, G, forward, count):
    """(states behind the segments from zero states, decays over them), or (None, None) for one segment."""
    if count == 1:
        return None, None
    fin = torch.empty(B, Hv, count, 128, 64, dtype=torch.float32, device=w.device)
    decay = torch.empty(B, Hv, count, dtype=torch.float32, device=w.device)
    _run("ssm_ssd_state_walk", _p(w), _ll(w_cols), w_cols, w_col0, _p(v), _ll(v_stride), _p(dt), _p(l), _p(None), B, L, H, Hv, G,
         forward, count, _p(fin), _p(decay), _p(status_tensor(w.device)), _st())
    return fin, decay


@functools.lru_cache(maxsize=4096)
def _walk_states(slices: int, nc: int) -> bool:
    """Kernels that walk the chunks of a head slice in segments, or one CTA per chunk and a recurrence kernel between, which take
    about 6 us, 55 ns per slice and chunk and 0.2 us per chunk forwards.  The separate kernels win for few chunks in all (us,
    separate / walk: 16 x 16 24 / 26, 2 x 64 30 / 42) and lose elsewhere (32 x 64 141 / 83, 48 x 64 198 / 106, 24 x 8 23 / 22, 1 x 512
    134 / 101).  The backward states follow the forward's line (16 x 16 14 / 20, 32 x 64 78 / 54).  Up to four chunks the launches
    saved decide."""
    return nc <= 4 or _walk_cost(slices, nc, _segments(slices, nc, _PER_CHUNK[0]), _PER_CHUNK[0]) < 6.0 + 0.055 * slices * nc + 0.2 * nc


def _dt_prep(dt_raw2, dt_raw_stride, A, D, dt_bias, B, L, H, log_a):
    """dt = softplus(dt_raw + dt_bias) and the running sums of A dt inside every chunk (fp32 [B, H, L]), and (A, D, dt_bias)
    in fp32.  log_a: A is A_log, of which the kernel takes -exp; the three may then be bf16 or fp32."""
    dev = dt_raw2.device
    if log_a:
        mask = _head_param_mask(A, D, dt_bias, H)
        if mask is None:
            return _dt_prep(dt_raw2, dt_raw_stride, -torch.exp(A.float()).contiguous(), D.float().contiguous(),
                            dt_bias.float().contiguous(), B, L, H, False)
        params = torch.empty(3, H, dtype=torch.float32, device=dev)
    else:
        mask, params = 0, None
    dt = torch.empty(B, H, L, dtype=torch.float32, device=dev)
    l = torch.empty_like(dt)
    _run("ssm_ssd_dt_prep", _p(dt_raw2), _ll(dt_raw_stride), _p(dt_bias), _p(A), _p(D), mask | (8 if log_a else 0), _p(params),
         _p(dt), _p(l), B, L, H, _st())
    return dt, l, (A, D, dt_bias) if params is None else params.unbind(0)


def _ssd_forward(conv_out, dt_raw2, dt_raw_stride, A, D, dt_bias, B, L, d_inner, G, H, Hv, init_state=None,
                 want_final=False, want_states=True, log_a=False, final_out=None, prepared=None):
    """conv_out [B*L, C] bf16 contiguous.  Returns y [B*L, d_inner], dt, l, S_in (None without want_states), final (or
    None), and (A, D, dt_bias) in fp32.  The backward pass wants S_in, the states entering the chunks.  final_out: contiguous
    fp32 [B, H, P, 128] that receives the final state.  prepared: what _dt_prep would return."""
    dev = conv_out.device
    C = conv_out.shape[1]
    nc = L // _CT
    st = status_tensor(dev)
    dt, l, params = prepared or _dt_prep(dt_raw2, dt_raw_stride, A, D, dt_bias, B, L, H, log_a)
    D = params[1]
    y = torch.empty(B * L, d_inner, dtype=torch.bfloat16, device=dev)
    if _walk_states(B * Hv, nc):
        s_in = torch.empty(B, Hv, nc, 128, 64, dtype=torch.bfloat16, device=dev) if want_states else None
        final = None
        if want_final:
            final = torch.empty(B, H, Hv // H * 64, 128, dtype=torch.float32, device=dev) if final_out is None else final_out
        count = _segments(B * Hv, nc, _PER_CHUNK[0])
        ends = _segment_ends(conv_out, C, d_inner, conv_out, C, dt, l, B, L, H, Hv, G, 1, count)
        _run("ssm_ssd_walk_scan", _p(conv_out), _ll(C), C, _p(s_in), _p(y), _ll(d_inner), _p(dt), _p(l), _p(D),
             _p(init_state), _p(final), B, L, H, Hv, G, d_inner, count, _p(ends[0]), _p(ends[1]), _p(st), _st())
        return y, dt, l, s_in, final, params
    s_in, final = _chunk_states(conv_out, C, d_inner, conv_out, C, dt, l, init_state, want_final, B, L, H, Hv, G, 0)
    if want_final:
        final = final.contiguous() if final_out is None else final_out.copy_(final)
    _run("ssm_ssd_chunk_scan_fwd", _p(conv_out), _ll(C), C, _p(s_in), _p(y), _ll(d_inner), _p(dt), _p(l), _p(D),
         B, L, H, Hv, G, d_inner, _p(st), _st())
    return y, dt, l, s_in, final, params


def _pick_hpc(hv_per_group, chunks, sms=148):
    """Head slices that one CTA of the backward scan walks (a divisor of the group's).  One CTA fits an SM and spends about
    one and a half heads on its set-up, B, C and the reduction of dB and dC, so the time is waves x (heads + 1.5): 64 chunks x
    80 slices take 350 us with 16 heads per CTA (three waves) and 313 us with 40 (one).
    The CTAs of a group add to the same dB and dC in the order in which they finish; with at most two of them the sums are
    the same in every run.  Where one or two per group fill the chip there are no more (by the count above five instead of
    two would save 9 % at 384 chunks x 80 slices)."""
    def cost(hpc):
        return -(-chunks * (hv_per_group // hpc) // sms) * (hpc + 1.5)
    most = 2 if chunks >= 2 * sms or (chunks >= sms and hv_per_group % 2 == 0) else hv_per_group
    return min((d for d in range(1, hv_per_group + 1) if hv_per_group % d == 0 and hv_per_group // d <= most), key=cost)


def _ssd_backward(conv_out, dy2, y2, dt, l, s_in, dt_raw2, dt_raw_stride, A, D, dt_bias, ddt_out, ddt_stride,
                  B, L, d_inner, G, H, Hv, raw=False):
    """Returns dx [B*L, d_inner] bf16, dBC fp32 [B*L, 2*G*128], dA, dD, d_dt_bias (fp32 [H]);
    d(dt_raw) goes to ddt_out (bf16, row stride ddt_stride, column h)."""
    dev = conv_out.device
    C = conv_out.shape[1]
    nc = L // _CT
    st = status_tensor(dev)
    psplit = Hv // H
    ds_out, _ = _chunk_states(conv_out, C, d_inner + G * 128, dy2, dy2.stride(0), dt, l, None, False, B, L, H, Hv, G, 1)
    dx = torch.empty(B * L, d_inner, dtype=torch.bfloat16, device=dev)
    dBC = torch.empty(B * L, 2 * G * 128, dtype=torch.float32, device=dev)
    hpart = torch.empty(B * nc, Hv, 3, dtype=torch.float32, device=dev)
    ddt32 = torch.empty(B, Hv, L, dtype=torch.float32, device=dev) if psplit > 1 else None
    hpc = _pick_hpc(Hv // G, nc * G * B)
    _run("ssm_ssd_chunk_scan_bwd", _p(conv_out), _ll(C), C, _p(dy2), _ll(dy2.stride(0)),
         _p(s_in), _p(ds_out), _p(dx), _ll(d_inner), _p(dBC), _p(hpart), _p(ddt_out), _ll(ddt_stride), _p(ddt32),
         _p(dt_raw2), _ll(dt_raw_stride), _p(dt_bias), _p(A), _p(dt), _p(l), _p(D), B, L, H, Hv, G, d_inner, hpc,
         _p(st), _st())
    if ddt32 is not None:
        summed = ddt32.reshape(B, H, psplit, L).sum(2).transpose(1, 2)           # [B, L, H]
        ddt_out.as_strided((B, L, H), (L * ddt_stride, ddt_stride, 1)).copy_(summed)
    if raw:
        return dx, dBC, hpart
    hp = hpart.sum(0).reshape(H, psplit, 3).sum(1)
    return dx, dBC, hp[:, 0], hp[:, 1], hp[:, 2]


def _conv_dt(xBC, w2, bias, dt_raw2, dt_raw_stride, A_log, D, dt_bias, window=None):
    """(conv output [B L, C], what _dt_prep returns for A_log) and, into `window` [B, C, 4], the last inputs of the conv."""
    B, L, C = xBC.shape
    H, dev = dt_raw2.shape[1], xBC.device
    mask = _head_param_mask(A_log, D, dt_bias, H)
    if mask is None:
        if window is not None:
            _run("ssm_conv_window", _p(xBC), _ll(xBC.stride(1)), _p(window), B, L, C, _st())
        return _conv_fwd(xBC, w2, bias, None).view(B * L, C), _dt_prep(dt_raw2, dt_raw_stride, A_log, D, dt_bias, B, L, H, True)
    out = torch.empty(B * L, C, dtype=xBC.dtype, device=dev)
    params = torch.empty(3, H, dtype=torch.float32, device=dev)
    dt = torch.empty(B, H, L, dtype=torch.float32, device=dev)
    l = torch.empty_like(dt)
    _run("ssm_conv_dt", _p(xBC), _ll(xBC.stride(1)), _p(w2), _p(bias), _p(out), _ll(C), _p(dt_raw2), _p(dt_bias), _p(A_log), _p(D),
         mask | 8, _p(params), _p(dt), _p(l), _p(window), B, L, C, H, _st())
    return out, (dt, l, params.unbind(0))


def _head_param_mask(A, D, dt_bias, H):
    """Bit i set: parameter i is bf16.  None where the kernels cannot read one of them as it is."""
    mask = 0
    for i, t in enumerate((A, D, dt_bias)):
        if t.dtype == torch.bfloat16:
            mask |= 1 << i
        elif t.dtype != torch.float32:
            return None
        if not t.is_contiguous() or t.numel() != H:
            return None
    return mask


class _MixerCore(torch.autograd.Function):
    @staticmethod
    def forward(ctx, zxBCdt, conv_w, conv_b, dt_bias, A_log, D, norm_w, d_inner, G, N, P, eps, gs, recompute,
                want_final, recorded, state_out):
        _require_bf16(zxBCdt, conv_w, conv_b, norm_w)
        H, psplit, Hv = _ssd_dims(d_inner, P, G, N)
        B, L, W = zxBCdt.shape
        C = d_inner + 2 * G * N
        if W != d_inner + C + H or L % _CT or d_inner % 8 or (G * N) % 8:
            raise ValueError("bad zxBCdt shape for the mixer core")
        _require_four_taps(conv_w, C)
        # rows may carry padding (row stride ld >= W, multiple of 8): that is how the GEMM epilogue writes them
        if (zxBCdt.stride(2) != 1 or zxBCdt.stride(1) % 8 or zxBCdt.stride(0) != L * zxBCdt.stride(1)
                or zxBCdt.data_ptr() % 16):
            buf = torch.empty(B * L, _ceil8(W), dtype=zxBCdt.dtype, device=zxBCdt.device)[:, :W]
            buf.copy_(zxBCdt.reshape(B * L, W))
            zxBCdt = buf.as_strided((B, L, W), (L * buf.stride(0), buf.stride(0), 1))
        ld = zxBCdt.stride(1)
        flat = zxBCdt.as_strided((B * L, W), (ld, 1))
        z2, xBC, dt_raw2 = flat[:, :d_inner], zxBCdt[..., d_inner:d_inner + C], flat[:, d_inner + C:]
        w2 = conv_w.reshape(C, -1).contiguous()
        window_out, final_out = state_out or (None, None)
        conv_state = None
        if want_final:
            conv_state = torch.empty(B, C, 4, dtype=zxBCdt.dtype, device=zxBCdt.device) if window_out is None else window_out
        conv_out, prepared = _conv_dt(xBC, w2, conv_b, dt_raw2, ld, A_log, D, dt_bias, conv_state)
        y, dt, l, s_in, final, (A, Df, bf) = _ssd_forward(
            conv_out, dt_raw2, ld, A_log, D, dt_bias, B, L, d_inner, G, H, Hv, want_final=want_final,
            want_states=recorded and not recompute, log_a=True, final_out=final_out, prepared=prepared)
        out = _gated_fwd(y, z2, norm_w, eps, gs)
        ctx.dims = (B, L, W, C, d_inner, G, N, P, H, Hv, eps, gs, recompute)
        if recompute:
            ctx.save_for_backward(zxBCdt, w2, conv_b, dt_bias, A_log, D, norm_w, A, Df, bf)
        else:
            ctx.save_for_backward(zxBCdt, w2, conv_b, dt_bias, A_log, D, norm_w, A, Df, bf, conv_out, y, dt, l, s_in)
        ctx.conv_w_shape = conv_w.shape
        ctx.conv_w_param = conv_w if conv_w.is_leaf else None
        out = out.view(B, L, d_inner)
        if want_final:
            ctx.mark_non_differentiable(conv_state, final)
            return out, conv_state, final
        return out

    @staticmethod
    def backward(ctx, dout, *unused):
        B, L, W, C, d_inner, G, N, P, H, Hv, eps, gs, recompute = ctx.dims
        saved = ctx.saved_tensors
        zxBCdt, w2, conv_b, dt_bias, A_log, D, norm_w, A, Df, bf = saved[:10]
        ld = zxBCdt.stride(1)
        flat = zxBCdt.as_strided((B * L, W), (ld, 1))
        z2, xBC, dt_raw2 = flat[:, :d_inner], zxBCdt[..., d_inner:d_inner + C], flat[:, d_inner + C:]
        if recompute:
            conv_out = _conv_fwd(xBC, w2, conv_b, None).view(B * L, C)
            y, dt, l, s_in, _, _ = _ssd_forward(conv_out, dt_raw2, ld, A, Df, bf, B, L, d_inner, G, H, Hv)
        else:
            conv_out, y, dt, l, s_in = saved[10:]
        dflat = torch.empty(B * L, ld, dtype=zxBCdt.dtype, device=zxBCdt.device)[:, :W]
        d_zx = dflat.as_strided((B, L, W), (L * ld, ld, 1))
        dout2 = dout.reshape(B * L, d_inner)
        if not dout2.is_contiguous():
            dout2 = dout2.contiguous()
        dy = torch.empty(B * L, d_inner, dtype=torch.bfloat16, device=dout.device)
        small = [ctx.conv_w_param, conv_b, norm_w, A_log, D, dt_bias]
        direct = all(p is None or (getattr(p, "main_grad", None) is not None and p.main_grad.dtype == torch.float32
                                   and p.main_grad.is_contiguous()) for p in small) and ctx.conv_w_param is not None
        if direct:
            # partial sums go straight into the fp32 main-gradient buffers with one finalisation kernel
            gpart = _gated_bwd(y, z2, norm_w, dout2, eps, gs, dy, dflat[:, :d_inner], raw=True)
            dx, dBC, hpart = _ssd_backward(conv_out, dy, y, dt, l, s_in, dt_raw2, ld, A, Df, bf,
                                           dflat[:, d_inner + C:], ld, B, L, d_inner, G, H, Hv, raw=True)
            cpart = _conv_bwd(xBC, w2, conv_b, dx.view(B, L, d_inner), dBC.view(B, L, 2 * G * N), d_inner,
                              d_zx[..., d_inner:d_inner + C], raw=True)
            mask = 0
            for bit, p in enumerate(small):
                if p is not None:
                    if not getattr(p, "grad_stale", False):
                        mask |= 1 << bit
                    p.grad_stale = False
            mg = [None if p is None else p.main_grad for p in small]
            _run("ssm_mixer_small_grads", _p(cpart), cpart.shape[0], C, _p(gpart), gpart.shape[0], d_inner, _p(hpart),
                 hpart.shape[0], Hv, H, _p(A), _p(mg[0]), _p(mg[1]), _p(mg[2]), _p(mg[3]), _p(mg[4]), _p(mg[5]),
                 mask, _st())
            return (d_zx,) + (None,) * 16
        dnorm_w = _gated_bwd(y, z2, norm_w, dout2, eps, gs, dy, dflat[:, :d_inner])
        dx, dBC, dA, dD, dbias = _ssd_backward(conv_out, dy, y, dt, l, s_in, dt_raw2, ld, A, Df, bf,
                                               dflat[:, d_inner + C:], ld, B, L, d_inner, G, H, Hv)
        dw, db = _conv_bwd(xBC, w2, conv_b, dx.view(B, L, d_inner), dBC.view(B, L, 2 * G * N), d_inner,
                           d_zx[..., d_inner:d_inner + C])
        dA_log = (dA * A).to(A_log.dtype)
        return (d_zx, dw.to(w2.dtype).reshape(ctx.conv_w_shape), None if conv_b is None else db.to(conv_b.dtype),
                dbias.to(dt_bias.dtype), dA_log, dD.to(D.dtype), dnorm_w.to(norm_w.dtype),
                None, None, None, None, None, None, None, None, None, None)


def mamba2_mixer_core(zxBCdt, conv_w, conv_b, dt_bias, A_log, D, norm_w, d_inner, n_groups, d_state, head_dim, eps,
                      norm_group_size, chunk_size, recompute, return_final_states, state_out=None):
    if chunk_size != _CT:
        raise ValueError("the GPU kernels use 128-token chunks")
    gs = d_inner if norm_group_size is None else norm_group_size
    if state_out is not None:
        B, H, C = zxBCdt.shape[0], d_inner // head_dim, d_inner + 2 * n_groups * d_state
        window, state = state_out
        if _recording() or not (window.dtype == zxBCdt.dtype and state.dtype == torch.float32 and window.is_contiguous()
                                and state.is_contiguous() and window.data_ptr() % 8 == 0     # the kernel stores whole windows
                                and window.device == state.device == zxBCdt.device
                                and tuple(window.shape) == (B, C, 4) and tuple(state.shape) == (B, H, head_dim, d_state)):
            state_out = None
    res = _apply(_MixerCore, zxBCdt, conv_w, conv_b, dt_bias, A_log, D, norm_w, d_inner, n_groups, d_state, head_dim,
                 eps, gs, recompute, return_final_states, torch.is_grad_enabled(), state_out)
    if return_final_states:
        if state_out is not None:          # written through their addresses: autograd learns of it here
            torch.autograd.graph.increment_version(state_out)
        return res[0], (res[1], res[2])
    return res


class _SSDScan(torch.autograd.Function):
    """Stand-alone scan op (tests, custom models): packs x|B|C into the layout the kernels read."""

    @staticmethod
    def forward(ctx, x, dt_raw, A, Bm, Cm, D, dt_bias, want_final, init_state):
        _require_bf16(x, Bm, Cm)
        Bsz, L, H, P = x.shape
        G, N = Bm.shape[2], Bm.shape[3]
        d_inner = H * P
        _, psplit, Hv = _ssd_dims(d_inner, P, G, N)
        conv_out = torch.cat([x.reshape(Bsz, L, d_inner), Bm.reshape(Bsz, L, G * N), Cm.reshape(Bsz, L, G * N)],
                             dim=-1).reshape(Bsz * L, -1).contiguous()
        Hp = _ceil8(H)
        dtr = torch.zeros(Bsz * L, Hp, dtype=torch.bfloat16, device=x.device)
        dtr[:, :H] = dt_raw.reshape(Bsz * L, H).to(torch.bfloat16)
        Af, Df, bf = A.float().contiguous(), D.float().contiguous(), dt_bias.float().contiguous()
        init = None
        if init_state is not None:   # [B,H,P,N] -> [B,Hv,128,64]
            init = init_state.float().reshape(Bsz, H, psplit, 64, N).permute(0, 1, 2, 4, 3).reshape(
                Bsz, Hv, N, 64).contiguous()
        y, dt, l, s_in, final, _ = _ssd_forward(conv_out, dtr, Hp, Af, Df, bf, Bsz, L, d_inner, G, H, Hv, init,
                                             want_final)
        ctx.save_for_backward(conv_out, y, dt, l, s_in, dtr, Af, Df, bf)
        ctx.dims = (Bsz, L, H, P, G, N, Hv, Hp)
        ctx.in_dtypes = (dt_raw.dtype, A.dtype, D.dtype, dt_bias.dtype)
        yv = y.view(Bsz, L, H, P)
        if want_final:
            ctx.mark_non_differentiable(final)
            return yv, final
        return yv

    @staticmethod
    def backward(ctx, dy, *unused):
        conv_out, y, dt, l, s_in, dtr, Af, Df, bf = ctx.saved_tensors
        Bsz, L, H, P, G, N, Hv, Hp = ctx.dims
        d_inner = H * P
        dy2 = dy.reshape(Bsz * L, d_inner).contiguous()
        ddt = torch.zeros(Bsz * L, Hp, dtype=torch.bfloat16, device=dy.device)
        dx, dBC, dA, dD, dbias = _ssd_backward(conv_out, dy2, y, dt, l, s_in, dtr, Hp, Af, Df, bf, ddt, Hp,
                                               Bsz, L, d_inner, G, H, Hv)
        t0, t1, t2, t3 = ctx.in_dtypes
        return (dx.view(Bsz, L, H, P), ddt[:, :H].reshape(Bsz, L, H).to(t0), dA.to(t1),
                dBC[:, :G * N].reshape(Bsz, L, G, N).to(dy.dtype), dBC[:, G * N:].reshape(Bsz, L, G, N).to(dy.dtype),
                dD.to(t2), dbias.to(t3), None, None)


def ssd_chunk_scan(x, dt_raw, A, Bm, Cm, D, dt_bias, chunk_size, initial_state, return_final_state):
    if chunk_size != _CT:
        raise ValueError("the GPU kernels use 128-token chunks")
    return _apply(_SSDScan, x, dt_raw, A, Bm, Cm, D, dt_bias, return_final_state, initial_state)


# ======================================================================================
# decode
# ======================================================================================
@torch.no_grad()
def ssm_decode_step(zxBCdt, conv_state, ssm_state, conv_w, conv_b, dt_bias, A_log, D, norm_w, d_inner, n_groups,
                    d_state, head_dim, eps, norm_group_size):
    _require_bf16(zxBCdt, conv_state, conv_w, norm_w)
    if ssm_state.dtype != torch.float32:
        raise TypeError("the decode kernel keeps the SSM state in fp32")
    B, W = zxBCdt.shape
    C = d_inner + 2 * n_groups * d_state
    H = d_inner // head_dim
    if conv_state.shape[-1] != 4 or not conv_state.is_contiguous() or not ssm_state.is_contiguous():
        raise ValueError("decode needs contiguous states and a 4-tap conv window")
    if zxBCdt.stride(1) != 1:
        zxBCdt = zxBCdt.contiguous()
    dev = zxBCdt.device
    y = torch.empty(B, d_inner, dtype=torch.bfloat16, device=dev)
    xBC, ld = zxBCdt[:, d_inner:], zxBCdt.stride(0)                     # x | B | C | dt
    w = conv_w.reshape(C, 4).contiguous()
    gs = d_inner if norm_group_size is None else norm_group_size
    mask = _head_param_mask(A_log, D, dt_bias, H)
    if mask is not None and W == d_inner + C + H and 2 * d_state + head_dim <= 12288:
        _run("ssm_decode_mixer_step", _p(xBC), _ll(ld), _p(conv_state), _p(w), _p(conv_b), _p(A_log), _p(D), _p(dt_bias), mask,
             _p(ssm_state), _p(y), B, C, H, head_dim, d_state, n_groups, d_inner, _st())
        out = torch.empty(B, d_inner, dtype=torch.bfloat16, device=dev)
        _run("ssm_gated_rmsnorm_roll", _p(y), _ll(d_inner), _p(zxBCdt), _ll(ld), _p(norm_w), _p(out), _ll(d_inner), _ll(B),
             d_inner, gs, _c.c_float(eps), _p(conv_state), _p(xBC), _ll(ld), d_inner, C, _st())
        return out
    act = torch.empty(B, C, dtype=torch.float32, device=dev)
    _run("ssm_decode_conv_step", _p(xBC), _ll(ld), _p(conv_state), _p(w), _p(conv_b), _p(act), B, C, _st())
    _run("ssm_decode_ssm_step", _p(act), _p(zxBCdt[:, d_inner + C:]), _ll(ld), _p(dt_bias.float().contiguous()),
         _p(-torch.exp(A_log.float()).contiguous()), _p(D.float().contiguous()), _p(ssm_state), _p(y), B, C, H, head_dim, d_state,
         n_groups, d_inner, _st())
    return _gated_fwd(y, zxBCdt[:, :d_inner], norm_w, eps, gs)


def _block_weights(dev, width, d_inner, n_groups, d_state, head_dim, gs, norm_w, in_w, in_b, conv_w, conv_b, dt_bias, A_log, D, gate_w,
                   out_w):
    """Addresses of a block's weights and the mask of its bf16 per-head parameters, or None where one of them is not as the
    kernels read it, or not on the GPU of this index."""
    C, H, bf16 = d_inner + 2 * n_groups * d_state, d_inner // head_dim, torch.bfloat16
    W = d_inner + C + H
    mask = _head_param_mask(A_log, D, dt_bias, H)
    for t in (norm_w, in_w, conv_w, gate_w, out_w, in_b, conv_b):        # (a generator costs the host more than the tests)
        if t is not None and (t.dtype is not bf16 or not t.is_contiguous() or t.get_device() != dev):
            return None
    if (mask is None or H % n_groups or width % 8 or d_inner % 8 or d_inner % gs or gs % 8 or max(width, gs) > 8192
            or A_log.get_device() != dev or D.get_device() != dev or dt_bias.get_device() != dev
            or in_w.shape != (W, width) or out_w.shape != (width, d_inner) or norm_w.numel() != width or gate_w.numel() != d_inner
            or conv_w.numel() != 4 * C or (in_b is not None and in_b.numel() != W) or (conv_b is not None and conv_b.numel() != C)):
        return None
    at = [norm_w.data_ptr(), in_w.data_ptr(), 0 if in_b is None else in_b.data_ptr(), conv_w.data_ptr(),
          0 if conv_b is None else conv_b.data_ptr(), A_log.data_ptr(), D.data_ptr(), dt_bias.data_ptr(), gate_w.data_ptr(),
          out_w.data_ptr()]
    if (at[0] | at[1] | at[8] | at[9]) & 15 or at[3] & 7:
        return None
    return at, mask


def _block_rows(hidden, residual, rd):
    """Addresses of a block's input rows, or None where they are not as the kernels read them."""
    if (hidden.dtype is not torch.bfloat16 or not hidden.is_contiguous() or not (rd is torch.bfloat16 or rd is torch.float32)
            or (residual is not None and (residual.dtype is not rd or not residual.is_contiguous() or residual.shape != hidden.shape
                                          or residual.get_device() != hidden.get_device()))):
        return None
    at = [hidden.data_ptr(), 0 if residual is None else residual.data_ptr()]
    return None if (at[0] | at[1]) & 15 else at


def _block_states(dev, B, C, H, P, N, conv_state, ssm_state):
    """Addresses of a layer's cached states, or None where the kernels cannot use them in place (a cache in host memory, which a
    prompt's states are copied into, is one such case)."""
    if (conv_state.dtype is not torch.bfloat16 or ssm_state.dtype is not torch.float32 or conv_state.shape != (B, C, 4)
            or ssm_state.shape != (B, H, P, N) or not conv_state.is_contiguous() or not ssm_state.is_contiguous()
            or conv_state.get_device() != dev or ssm_state.get_device() != dev):
        return None
    at = [conv_state.data_ptr(), ssm_state.data_ptr()]
    return None if at[0] & 7 or at[1] & 15 else at


@functools.lru_cache(maxsize=256)
def _scratch_offsets(*sizes):
    """Offsets of buffers of these sizes (bytes) in one allocation, on 256-byte boundaries, and its size."""
    at, end = [], 0
    for size in sizes:
        at.append(end)
        end += (size + 255) // 256 * 256
    return at, end


_BLOCK_FORWARD = struct.Struct("=26Qq11i2f")


def block_forward(hidden, residual, residual_dtype, conv_state, ssm_state, norm_w, norm_eps, in_w, in_b, conv_w, conv_b, dt_bias, A_log,
                  D, gate_w, out_w, d_inner, n_groups, d_state, head_dim, eps, norm_group_size):
    """A pre-norm block over whole sequences, `out_proj(mixer(norm(residual + hidden)))`, by one native call.  conv_state and
    ssm_state, which may be None, receive the states behind the last token.  Returns (branch output, new residual), or None
    where a tensor is not as the kernels read it; the caller then takes the separate operations."""
    B, L, width = hidden.shape
    C, H = d_inner + 2 * n_groups * d_state, d_inner // head_dim
    rd = residual_dtype or hidden.dtype
    gs = d_inner if norm_group_size is None else norm_group_size
    if L % _CT or L == 0 or B == 0 or B > 65535 or d_state != 128 or head_dim % 64 or hidden.numel() >= 2 ** 31:
        return None
    weights = _block_weights(hidden.get_device(), width, d_inner, n_groups, d_state, head_dim, gs, norm_w, in_w, in_b, conv_w, conv_b,
                             dt_bias, A_log, D, gate_w, out_w)
    rows = _block_rows(hidden, residual, rd)
    states = [0, 0] if conv_state is None else _block_states(hidden.get_device(), B, C, H, head_dim, d_state, conv_state, ssm_state)
    if weights is None or rows is None or states is None:
        return None
    dev, ld, T = hidden.device, _ceil8(d_inner + C + H), B * L
    count = _segments(T // L * d_inner // 64, L // _CT, _PER_CHUNK[0])
    segments = 0 if count == 1 else B * (d_inner // 64) * count
    at, end = _scratch_offsets(2 * T * max(width, d_inner), 2 * T * ld, 2 * T * C, 2 * T * d_inner, 12 * H, 4 * T * H, 4 * T * H,
                               segments * 4 * 128 * 64, segments * 4)
    scratch = torch.empty(end, dtype=torch.uint8, device=dev)
    base = scratch.data_ptr()
    out, res_out = torch.empty_like(hidden), torch.empty(hidden.shape, dtype=rd, device=dev)
    _run("ssm_block_forward", _BLOCK_FORWARD.pack(*rows, res_out.data_ptr(), *weights[0], *states, *[base + o for o in at], out.data_ptr(),
                                                  status_tensor(dev).data_ptr(), ld, B, L, width, d_inner, H, head_dim, n_groups, gs,
                                                  int(rd is torch.float32), weights[1], count, norm_eps, eps), _st())
    _launches[0] += 5 + (count > 1)
    if conv_state is not None:             # written through their addresses: autograd learns of it here
        torch.autograd.graph.increment_version((conv_state, ssm_state))
    return out, res_out


_BLOCK = struct.Struct("=20Qq11i2f")


@functools.lru_cache(maxsize=4096)
def _norms_in_products(B: int, width: int, in_cols: int, d_inner: int, gs: int, captured: bool):
    """Which norms of a decoding block are computed inside the product behind them (norm_linear_kernel, the same bits as two
    kernels): (first, gated).  Every block of it forms all rows, so few columns in all gain and many lose; two blocks of the first
    kind fit an SM, and a second wave of them costs what the launch saved (one kernel / two, us: in_proj 1 x 3352 x 768 3.0 / 3.8,
    1 x 4384 x 1024 3.5 / 4.5, 1 x 6176 x 1024 6.3 / 4.7, 2 x 4384 x 1024 3.7 / 4.5, 3 x 4384 x 1024 4.4 / 4.6, 5 x 4384 x 1024 5.4 / 4.7;
    out_proj from 1 x 1536 columns 3.5 / 4.6, 1 x 4096 7.5 / 8.4, 3 x 2048 5.5 / 5.7, 2 x 4096 8.9 / 8.7, 5 x 1536 5.7 / 5.6, 5 x 2048
    6.9 / 5.9; with eight groups 1 x 2048 5.0 / 5.2, 2 x 2048 5.4 / 5.3, 1 x 4096 8.5 / 8.2).  Where no graph is captured the host is
    the limit, which a launch less saves 3 us (370M, 5 sequences: 723 us a token with two kernels each, 642 with one)."""
    groups = d_inner // gs
    first, gated = (2048, 6144 if groups == 1 else 2048) if captured else (8192, 32768)
    return (B <= 8 and width <= 1024 and B * width <= first and (in_cols <= 16 * 2 * 148 or not captured),
            B <= 8 and d_inner <= 4096 and B * d_inner <= gated and (groups == 1 or (groups in (2, 4, 8) and gs % 64 == 0)))


def decode_block(hidden, residual, residual_dtype, conv_state, ssm_state, norm_w, norm_eps, in_w, in_b, conv_w, conv_b, dt_bias, A_log,
                 D, gate_w, out_w, d_inner, n_groups, d_state, head_dim, eps, norm_group_size):
    """One token of a pre-norm block, `out_proj(mixer(norm(residual + hidden)))`, by one native call of three to five kernels.
    Returns (branch output, new residual), or None where a tensor is not as the kernels read it; the
    caller then takes the separate operations, which convert or refuse it."""
    B, _, width = hidden.shape
    C, H = d_inner + 2 * n_groups * d_state, d_inner // head_dim
    rd = residual_dtype or hidden.dtype
    gs = d_inner if norm_group_size is None else norm_group_size
    if 2 * d_state + head_dim > 12288 or d_state % 4 or not 0 < B <= 65535:
        return None
    weights = _block_weights(hidden.get_device(), width, d_inner, n_groups, d_state, head_dim, gs, norm_w, in_w, in_b, conv_w, conv_b,
                             dt_bias, A_log, D, gate_w, out_w)
    rows = _block_rows(hidden, residual, rd)
    states = _block_states(hidden.get_device(), B, C, H, head_dim, d_state, conv_state, ssm_state)
    if weights is None or rows is None or states is None:
        return None
    dev, ld = hidden.device, _ceil8(d_inner + C + H)
    scratch = torch.empty(B * (ld + d_inner + max(width, d_inner)), dtype=torch.bfloat16, device=dev)
    out, res_out = torch.empty_like(hidden), torch.empty(hidden.shape, dtype=rd, device=dev)
    zx = scratch.data_ptr()
    first, gated = _norms_in_products(B, width, d_inner + C + H, d_inner, gs, True)
    if not (first and gated) and not torch.cuda.is_current_stream_capturing():
        first, gated = _norms_in_products(B, width, d_inner + C + H, d_inner, gs, False)
    _run("ssm_decode_block", _BLOCK.pack(*rows, res_out.data_ptr(), *weights[0], *states, zx, zx + 2 * B * ld, zx + 2 * B * (ld + d_inner),
                                         out.data_ptr(), status_tensor(dev).data_ptr(), ld, B, width, d_inner, H, head_dim, d_state,
                                         n_groups, gs, int(rd is torch.float32), weights[1], int(first) | 2 * int(gated), norm_eps, eps), _st())
    _launches[0] += 4 - first - gated
    return out, res_out


# ======================================================================================
# rotary position embedding
# ======================================================================================
_ROPE_TABLES = {}


def rotary_tables(seq_len: int, dim: int, theta: float, device, offset: int = 0):
    """fp32 cos / sin tables [seq_len, dim / 2], built once per (length, dim, theta, offset, device) and kept."""
    key = (int(seq_len), int(dim), float(theta), int(offset), str(device))
    if key not in _ROPE_TABLES:
        from . import oracle
        cos, sin = oracle.rotary_tables(seq_len, dim, theta, device=device, offset=offset)
        _ROPE_TABLES[key] = (cos.contiguous(), sin.contiguous())
    return _ROPE_TABLES[key]


def _rope_launch(x, cos, sin, inverse: bool):
    B, L, H, Dh = x.shape
    rd = cos.shape[-1] * 2
    x3 = x if (x.stride(3) == 1 and x.stride(2) == Dh and x.stride(0) == L * x.stride(1)) else x.contiguous()
    out = torch.empty(B, L, H, Dh, dtype=x.dtype, device=x.device)
    _run("ssm_rope", _p(x3), _ll(x3.stride(1)), _p(out), _ll(H * Dh), _p(cos), _p(sin), _ll(B * L), L, H, Dh, rd,
         int(inverse), _st())
    return out


class _Rope(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, cos, sin):
        ctx.save_for_backward(cos, sin)
        return _rope_launch(x, cos, sin, False)

    @staticmethod
    def backward(ctx, dy):
        cos, sin = ctx.saved_tensors
        return _rope_launch(dy, cos, sin, True), None, None


def apply_rotary(x, cos, sin):
    """Rotate-half rotary embedding on the first 2 * cos.shape[-1] channels of x [B, L, H, Dh] (bf16); cos / sin fp32
    [L, rd / 2].  The backward pass is the same kernel with the angle negated."""
    _require_bf16(x)
    rd = cos.shape[-1] * 2
    if x.shape[-1] % 8 or rd % 16 or cos.dtype != torch.float32 or cos.shape[0] != x.shape[1]:
        raise ValueError("rotary kernel needs head_dim % 8 == 0, rotary dim % 16 == 0 and fp32 tables of the sequence length")
    return _apply(_Rope, x, cos, sin)


# ======================================================================================
# attention
# ======================================================================================
class _Attention(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v):
        B, L, Hq, D = q.shape
        Hkv = k.shape[2]
        q2, k2, v2 = q.reshape(B * L, Hq * D), k.reshape(B * L, Hkv * D), v.reshape(B * L, Hkv * D)
        q2, k2, v2 = [t if t.is_contiguous() else t.contiguous() for t in (q2, k2, v2)]
        out = torch.empty_like(q2)
        lse = torch.empty(B, Hq, L, dtype=torch.float32, device=q.device)
        scale = 1.0 / (D ** 0.5)
        _run("ssm_attn_fwd", _p(q2), _p(k2), _p(v2), _p(out), _p(lse), B, L, Hq, Hkv, D, _c.c_float(scale),
             _p(status_tensor(q.device)), _st())
        ctx.save_for_backward(q2, k2, v2, out, lse)
        ctx.dims = (B, L, Hq, Hkv, D, scale)
        return out.view(B, L, Hq, D)

    @staticmethod
    def backward(ctx, dout):
        q2, k2, v2, out, lse = ctx.saved_tensors
        B, L, Hq, Hkv, D, scale = ctx.dims
        do2 = dout.reshape(B * L, Hq * D)
        if not do2.is_contiguous():
            do2 = do2.contiguous()
        delta = torch.empty(B, Hq, L, dtype=torch.float32, device=dout.device)
        _run("ssm_attn_delta", _p(do2), _p(out), _p(delta), B, L, Hq, D, _st())
        dq32 = torch.zeros(B * L, Hq * D, dtype=torch.float32, device=dout.device)
        dk, dv = torch.empty_like(k2), torch.empty_like(v2)
        _run("ssm_attn_bwd", _p(q2), _p(k2), _p(v2), _p(do2), _p(lse), _p(delta), _p(dq32), _p(dk), _p(dv), B, L, Hq, Hkv,
             D, _c.c_float(scale), _p(status_tensor(dout.device)), _st())
        return (dq32.to(torch.bfloat16).view(B, L, Hq, D), dk.view(B, L, Hkv, D), dv.view(B, L, Hkv, D))


def attention(q, k, v, causal=True):
    _require_bf16(q, k, v)
    if not causal:
        raise NotImplementedError("the GPU attention kernel is causal")
    if q.shape[-1] != 128 or q.shape[1] % 128 or q.shape[1] != k.shape[1]:
        raise ValueError("the GPU attention kernel needs head_dim 128 and equal q/k lengths that are multiples of 128")
    return _apply(_Attention, q, k, v)
