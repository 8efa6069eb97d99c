// Single-token decode over cached states for sm_100a (memory-bound: one pass over the SSM state).
//   mixer step: both of the following in one kernel per (head, batch), the form that decoding takes
//   conv step : roll the [C][4] window, depthwise conv + bias + SiLU for x, B and C alike
//   ssm step  : S <- S exp(A dt) + (dt x) (x) B ;  y = S C + D x ;  dt = softplus(dt_raw + bias) fused
// State layouts as in the cache: conv_state [B, C, 4] (oldest first), ssm_state [B, H, P, N] fp32, both
// updated in place.  The two separate steps serve heads that do not fit shared memory and parameters of other types.
// Reference: mamba2/mamba2_kernel_inference.py:13-23,26-104 (grid over batch only, softplus
// and gated norm outside); here the grid is (head, batch) and the state makes exactly one round trip.
#include "common.cuh"

namespace ssm {

__global__ void __launch_bounds__(256)
decode_conv_step_kernel(const __nv_bfloat16* xnew, long long xs, __nv_bfloat16* state, const __nv_bfloat16* w,
                        const __nv_bfloat16* bias, float* __restrict__ act, int C) {
  pdl_trigger();
  pdl_wait();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (c >= C) return;
  if (!SSM_INDEX_OK(c, xs)) return;               // the new token's row must hold all C channels
  uint2* sp = reinterpret_cast<uint2*>(state + ((long long)b * C + c) * 4);
  const uint2 s = *sp;
  const float x1 = bf16_hi(s.x), x2 = bf16_lo(s.y), x3 = bf16_hi(s.y);
  const __nv_bfloat16 xn = xnew[(long long)b * xs + c];
  const float x4 = __bfloat162float(xn);
  uint2 ns;
  ns.x = pack_bf16(x1, x2);
  ns.y = pack_bf16(x3, x4);
  *sp = ns;
  const uint2 wv = *reinterpret_cast<const uint2*>(w + (long long)c * 4);
  float pre = bias ? __bfloat162float(bias[c]) : 0.f;
  pre += bf16_lo(wv.x) * x1 + bf16_hi(wv.x) * x2 + bf16_lo(wv.y) * x3 + bf16_hi(wv.y) * x4;
  act[(long long)b * C + c] = silu_f(pre);
}

// State update and read-out of one head by 128 threads: warp w owns rows p = 4w .. 4w+3, 4w+16 .., ...; lanes own
// n = 4*lane + 128*r.  xh [P], Bv / Cv [N]: activations of the head (global or shared memory).
__device__ __forceinline__ void decode_ssm_head(const float* xh, const float* Bv, const float* Cv, float dt, float decay,
                                                float Dh, float* S, __nv_bfloat16* __restrict__ y, int P, int N) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // four rows per warp iteration: four independent 16-byte loads per lane are in flight before any arithmetic,
  // and the four row sums are reduced together (the state makes one round trip; this loop is latency-bound otherwise)
  for (int p0 = warp * 4; p0 < P; p0 += 16) {
    float4 s[4];
    float xs[4], acc[4];
    #pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int pp = p0 + r;
      xs[r] = pp < P ? xh[pp] : 0.f;
      acc[r] = 0.f;
    }
    for (int n = lane * 4; n < N; n += 128) {
      #pragma unroll
      for (int r = 0; r < 4; ++r)
        if (p0 + r < P) s[r] = *reinterpret_cast<const float4*>(S + (long long)(p0 + r) * N + n);
      const float4 bv = *reinterpret_cast<const float4*>(Bv + n);
      const float4 cv = *reinterpret_cast<const float4*>(Cv + n);
      #pragma unroll
      for (int r = 0; r < 4; ++r) {
        if (p0 + r < P) {
          const float dx = dt * xs[r];
          s[r].x = s[r].x * decay + dx * bv.x; s[r].y = s[r].y * decay + dx * bv.y;
          s[r].z = s[r].z * decay + dx * bv.z; s[r].w = s[r].w * decay + dx * bv.w;
          *reinterpret_cast<float4*>(S + (long long)(p0 + r) * N + n) = s[r];
          acc[r] += s[r].x * cv.x + s[r].y * cv.y + s[r].z * cv.z + s[r].w * cv.w;
        }
      }
    }
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      #pragma unroll
      for (int r = 0; r < 4; ++r) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], o);
    }
    if (lane < 4 && p0 + lane < P) {
      const float a = lane == 0 ? acc[0] : lane == 1 ? acc[1] : lane == 2 ? acc[2] : acc[3];
      const float x = lane == 0 ? xs[0] : lane == 1 ? xs[1] : lane == 2 ? xs[2] : xs[3];
      y[p0 + lane] = __float2bfloat16(a + Dh * x);
    }
  }
}

// grid (H, B), 128 threads, behind decode_conv_step_kernel
__global__ void __launch_bounds__(128)
decode_ssm_step_kernel(const float* act, const __nv_bfloat16* dt_raw, long long dts, const float* dt_bias, const float* A,
                       const float* D, float* state, __nv_bfloat16* __restrict__ y, int C, int H, int P, int N, int G, int d_in) {
  pdl_trigger();
  pdl_wait();
  const int h = blockIdx.x, b = blockIdx.y;
  const int g = h / (H / G);
  const float dt = softplus_f(__bfloat162float(dt_raw[(long long)b * dts + h]) + dt_bias[h]);
  const float* ab = act + (long long)b * C;
  // the activation row [x | B | C] must hold d_in + 2 G N values and the head's x slice must lie inside d_in
  if (!SSM_INDEX_OK(d_in + 2 * G * N - 1, C) || !SSM_INDEX_OK(h * P + P - 1, d_in)) return;
  decode_ssm_head(ab + h * P, ab + d_in + g * N, ab + d_in + G * N + g * N, dt, __expf(A[h] * dt), D[h],
                  state + (((long long)b * H + h) * P) * N, y + (long long)b * d_in + h * P, P, N);
}

// Conv and state update of one head in one kernel.  Every head computes the conv of its group's B and C channels for itself
// (2 N short dot products next to a 4 P N byte state) and rolls the windows of its own x channels; the B and C windows,
// which other heads still read, are rolled by the kernel behind this one (gated norm).  Bound by the state's round trip at
// large batches and by latency at small ones, where the conv kernel alone cost as much as this (130M, batch 1: 470 -> 450 us
// per token).  Few heads in all leave most SMs idle and every warp with P / 16 loads in series, so the P rows of a head are
// then dealt to up to four CTAs (decode_parts); rows are fetched a turn ahead, the first together with the inputs of the conv
// (130M, us per token: batch 1 303 -> 297, batch 8 419 -> 400).
struct DecodeParams { const void* A_log; const void* D; const void* dt_bias; int bf16_mask; };
__device__ __forceinline__ float decode_param(const void* p, int h, bool bf16) {
  return bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[h]) : reinterpret_cast<const float*>(p)[h];
}
__global__ void __launch_bounds__(128)
decode_mixer_kernel(const __nv_bfloat16* xnew, long long xs, __nv_bfloat16* window, const __nv_bfloat16* w,
                    const __nv_bfloat16* bias, const DecodeParams prm, float* state, __nv_bfloat16* __restrict__ y, int C, int H,
                    int rows, int parts, int N, int G, int d_in) {
  extern __shared__ __align__(16) float act[];         // B [N] | C [N] | x [P]
  pdl_trigger();
  const int h = blockIdx.x / parts, b = blockIdx.y, P = rows / parts;       // P: this CTA's rows of the head
  const int g = h / (H / G), x0 = blockIdx.x * P;                           // x0: its first x channel
  float* S = state + ((long long)b * H * rows + x0) * N;
  // the state on its way to L2 while the predecessor finishes and the conv is computed
  for (int i = threadIdx.x * 32; i < P * N; i += 128 * 32) prefetch_l2(S + i);
  pdl_wait();
  if (!SSM_INDEX_OK(d_in + 2 * G * N - 1, C) || !SSM_INDEX_OK(x0 + P - 1, d_in) || !SSM_INDEX_OK(C + h, xs)) return;
  const __nv_bfloat16* xr = xnew + (long long)b * xs;
  const float raw = __bfloat162float(xr[C + h]), bias_h = decode_param(prm.dt_bias, h, prm.bf16_mask & 4),
              log_a = decode_param(prm.A_log, h, prm.bf16_mask & 1), Dh = decode_param(prm.D, h, prm.bf16_mask & 2);
  // The usual state (128 values per row, rows in turns of 16): this warp's first rows are fetched together with the inputs of
  // the conv, and the next turn's before the present one is computed
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool whole = N == 128 && P % 16 == 0;
  float4 ahead[4];
  if (whole) {
    #pragma unroll
    for (int r = 0; r < 4; ++r) ahead[r] = *reinterpret_cast<const float4*>(S + (warp * 4 + r) * 128 + lane * 4);
  }
  // three channels per thread at a time (all of them at N = 128 and P <= 128): their loads go out together, in front of the
  // stores to the window, which they must not pass (2.7B, 64 sequences, us per token: 1218 one by one, 1184)
  for (int i0 = threadIdx.x; i0 < 2 * N + P; i0 += 3 * 128) {
    uint2 s[3], wv[3];
    float x4[3], pre[3];
    #pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int i = i0 + k * 128;
      if (i >= 2 * N + P) break;
      const int c = i >= 2 * N ? x0 + i - 2 * N : i < N ? d_in + g * N + i : d_in + G * N + g * N + i - N;
      s[k] = *reinterpret_cast<const uint2*>(window + ((long long)b * C + c) * 4);
      wv[k] = *reinterpret_cast<const uint2*>(w + (long long)c * 4);
      x4[k] = __bfloat162float(xr[c]);
      pre[k] = bias ? __bfloat162float(bias[c]) : 0.f;
    }
    #pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int i = i0 + k * 128;
      if (i >= 2 * N + P) break;
      const float x1 = bf16_hi(s[k].x), x2 = bf16_lo(s[k].y), x3 = bf16_hi(s[k].y);
      if (i >= 2 * N)                                    // this head's own x channels
        *reinterpret_cast<uint2*>(window + ((long long)b * C + x0 + i - 2 * N) * 4) = make_uint2(pack_bf16(x1, x2), pack_bf16(x3, x4[k]));
      pre[k] += bf16_lo(wv[k].x) * x1 + bf16_hi(wv[k].x) * x2 + bf16_lo(wv[k].y) * x3 + bf16_hi(wv[k].y) * x4[k];
      act[i] = silu_f(pre[k]);
    }
  }
  const float dt = softplus_f(raw + bias_h);
  const float A = -expf(log_a);
  __syncthreads();
  if (whole) {
    const float decay = __expf(A * dt);
    const float4 bv = *reinterpret_cast<const float4*>(act + lane * 4), cv = *reinterpret_cast<const float4*>(act + 128 + lane * 4);
    const float* xh = act + 256;
    __nv_bfloat16* yh = y + (long long)b * d_in + x0;
    for (int p0 = warp * 4; p0 < P; p0 += 16) {
      float4 s[4];
      float acc[4];
      #pragma unroll
      for (int r = 0; r < 4; ++r) s[r] = ahead[r];
      if (p0 + 16 < P) {
        #pragma unroll
        for (int r = 0; r < 4; ++r) ahead[r] = *reinterpret_cast<const float4*>(S + (p0 + 16 + r) * 128 + lane * 4);
      }
      #pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float dx = dt * xh[p0 + r];
        s[r].x = s[r].x * decay + dx * bv.x; s[r].y = s[r].y * decay + dx * bv.y;
        s[r].z = s[r].z * decay + dx * bv.z; s[r].w = s[r].w * decay + dx * bv.w;
        *reinterpret_cast<float4*>(S + (p0 + r) * 128 + lane * 4) = s[r];
        acc[r] = s[r].x * cv.x + s[r].y * cv.y + s[r].z * cv.z + s[r].w * cv.w;
      }
      #pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        #pragma unroll
        for (int r = 0; r < 4; ++r) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], o);
      }
      if (lane < 4) {
        const float a = lane == 0 ? acc[0] : lane == 1 ? acc[1] : lane == 2 ? acc[2] : acc[3];
        yh[p0 + lane] = __float2bfloat16(a + Dh * xh[p0 + lane]);
      }
    }
    return;
  }
  decode_ssm_head(act + 2 * N, act, act + N, dt, __expf(A * dt), Dh, S, y + (long long)b * d_in + x0, P, N);
}

}  // namespace ssm

using namespace ssm;
SSM_DEBUG_BOUNDS_GETTER(ssm_debug_bounds_decode)

extern "C" int ssm_decode_conv_step(const void* xnew, long long xs, void* state, const void* w, const void* bias,
                                    void* act, int B, int C, cudaStream_t st) {
  dim3 grid((C + 255) / 256, B);
  return launch_dependent(decode_conv_step_kernel, grid, dim3(256), 0, st, reinterpret_cast<const __nv_bfloat16*>(xnew), xs,
                          reinterpret_cast<__nv_bfloat16*>(state), reinterpret_cast<const __nv_bfloat16*>(w),
                          reinterpret_cast<const __nv_bfloat16*>(bias), reinterpret_cast<float*>(act), C);
}

extern "C" int ssm_decode_ssm_step(const void* act, const void* dt_raw, long long dts, const void* dt_bias,
                                   const void* A, const void* D, void* state, void* y, int B, int C, int H, int P,
                                   int N, int G, int d_in, cudaStream_t st) {
  if (N % 4 || H % G) return -SSM_ERR_BAD_ARG;
  dim3 grid(H, B);
  return launch_dependent(decode_ssm_step_kernel, grid, dim3(128), 0, st, reinterpret_cast<const float*>(act),
                          reinterpret_cast<const __nv_bfloat16*>(dt_raw), dts, reinterpret_cast<const float*>(dt_bias),
                          reinterpret_cast<const float*>(A), reinterpret_cast<const float*>(D),
                          reinterpret_cast<float*>(state), reinterpret_cast<__nv_bfloat16*>(y), C, H, P, N, G, d_in);
}

// CTAs per head: rows are dealt out while the grid does not fill the chip, in parts of at least 16 (one turn of the four warps)
static int decode_parts(int heads, int P) {
  int parts = 1;
  while (parts < 4 && heads * parts < 148 && P % (parts * 2) == 0 && P / (parts * 2) >= 16) parts *= 2;
  return parts;
}

// One token of a mixer up to the gated norm.  xnew: bf16 [B, C + H] (x | B | C | dt) with row stride xs; window bf16 [B,C,4]:
// the x channels are rolled, the rest is left for ssm_gated_rmsnorm_roll; A_log, D, dt_bias: bf16 where bit 0, 1, 2 of the
// mask is set, else fp32; state fp32 [B,H,P,N]; y bf16 [B, d_in].
extern "C" int ssm_decode_mixer_step(const void* xnew, long long xs, void* window, const void* w, const void* bias,
                                     const void* A_log, const void* D, const void* dt_bias, int bf16_mask, void* state, void* y,
                                     int B, int C, int H, int P, int N, int G, int d_in, cudaStream_t st) {
  const size_t smem = (size_t)(2 * N + P) * sizeof(float);
  if (N % 4 || H % G || smem > 48 * 1024 || B < 1 || B > 65535 || C != d_in + 2 * G * N) return -SSM_ERR_BAD_ARG;
  DecodeParams prm{A_log, D, dt_bias, bf16_mask};
  const int parts = decode_parts(H * B, P);
  return launch_dependent(decode_mixer_kernel, dim3(H * parts, B), dim3(128), smem, st, reinterpret_cast<const __nv_bfloat16*>(xnew), xs,
                          reinterpret_cast<__nv_bfloat16*>(window), reinterpret_cast<const __nv_bfloat16*>(w),
                          reinterpret_cast<const __nv_bfloat16*>(bias), prm, reinterpret_cast<float*>(state),
                          reinterpret_cast<__nv_bfloat16*>(y), C, H, P, parts, N, G, d_in);
}

// One token through a whole pre-norm block: residual add + norm, in_proj, conv and state update, gated norm, out_proj.
// Three to five kernels: the norms may be part of the products behind them.
extern "C" int ssm_add_rmsnorm_fwd(const void*, const void*, const void*, void*, void*, long long, int, float, int, cudaStream_t);
extern "C" int ssm_gemm_bf16(const void*, const void*, void*, int, int, int, long long, long long, long long, int, int, int,
                             const void*, int, int*, cudaStream_t);
extern "C" int ssm_gated_rmsnorm_roll(const void*, long long, const void*, long long, const void*, void*, long long, long long, int,
                                      int, float, void*, const void*, long long, int, int, cudaStream_t);
extern "C" int ssm_add_norm_linear(const void*, long long, const void*, void*, int, const void*, float, const void*, long long,
                                   const void*, void*, long long, int, int, int, cudaStream_t);
extern "C" int ssm_gated_norm_linear(const void*, long long, const void*, long long, const void*, int, float, const void*,
                                     long long, const void*, void*, long long, int, int, int, void*, const void*, long long, int,
                                     int, cudaStream_t);
struct DecodeBlock {                       // in the order in which cuda_ops.decode_block packs it
  const void *x, *res; void* res_out;      // bf16 [B, D], residual type [B, D] or null, residual type [B, D]
  const void *norm_w, *in_w, *in_b, *conv_w, *conv_b, *A_log, *Dp, *dt_bias, *gate_w, *out_w;
  void *window, *state;                    // bf16 [B, C, 4], fp32 [B, H, P, N]
  void *zx, *y, *normed, *out;             // scratch [B, zx_ld], [B, d_in], [B, max(D, d_in)]; result [B, D]
  int* status;
  long long zx_ld;
  int B, D, d_in, H, P, N, G, gs, res_fp32, bf16_mask, fused;       // bit 0, 1: first, gated norm inside the product behind it
  float eps_norm, eps_gate;
};
extern "C" int ssm_decode_block(const DecodeBlock* a, cudaStream_t st) {
  const int C = a->d_in + 2 * a->G * a->N, W = a->d_in + C + a->H;
  auto* zx = reinterpret_cast<__nv_bfloat16*>(a->zx);
  const void* xbc = zx + a->d_in;
  int r;
  if (a->fused & 1) {
    r = ssm_add_norm_linear(a->x, a->D, a->res, a->res_out, a->res_fp32, a->norm_w, a->eps_norm, a->in_w, a->D, a->in_b, a->zx,
                            a->zx_ld, a->B, W, a->D, st);
  } else {
    r = ssm_add_rmsnorm_fwd(a->x, a->res, a->norm_w, a->normed, a->res_out, a->B, a->D, a->eps_norm, a->res_fp32, st);
    if (r) return r;
    r = ssm_gemm_bf16(a->normed, a->in_w, a->zx, a->B, W, a->D, a->D, a->D, a->zx_ld, 0, 0, 0, a->in_b, 0, a->status, st);
  }
  if (r) return r;
  r = ssm_decode_mixer_step(xbc, a->zx_ld, a->window, a->conv_w, a->conv_b, a->A_log, a->Dp, a->dt_bias, a->bf16_mask, a->state,
                            a->y, a->B, C, a->H, a->P, a->N, a->G, a->d_in, st);
  if (r) return r;
  if (a->fused & 2)
    return ssm_gated_norm_linear(a->y, a->d_in, a->zx, a->zx_ld, a->gate_w, a->gs, a->eps_gate, a->out_w, a->d_in, nullptr, a->out,
                                 a->D, a->B, a->D, a->d_in, a->window, xbc, a->zx_ld, a->d_in, C, st);
  r = ssm_gated_rmsnorm_roll(a->y, a->d_in, a->zx, a->zx_ld, a->gate_w, a->normed, a->d_in, a->B, a->d_in, a->gs, a->eps_gate,
                             a->window, xbc, a->zx_ld, a->d_in, C, st);
  if (r) return r;
  return ssm_gemm_bf16(a->normed, a->out_w, a->out, a->B, a->D, a->d_in, a->d_in, a->d_in, a->D, 0, 0, 0, nullptr, 0, a->status, st);
}
