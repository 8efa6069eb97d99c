// Memory-bound kernels of the Mamba-2 block for sm_100a: causal depthwise conv1d + SiLU (fwd/bwd),
// gated group RMSNorm (fwd/bwd), residual-add + RMSNorm (fwd/bwd), GELU (fwd/bwd), vocab-shard cross
// entropy statistics and gradient, fused AdamW and sum of squares.  All io is 16-byte vectorised bf16,
// all arithmetic fp32.  Reference counterparts: mamba2/conv1d_grouped.py:65-194 (conv),
// mamba2/fused_kernel.py:76-175 (gated norm), mamba2/modeling_mamba2.py:94-103 (RMSNorm).
#include "common.cuh"
#include "dt_prep.cuh"
#include <type_traits>

namespace ssm {

__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&f)[8]) {
  unpack8(*reinterpret_cast<const uint4*>(p), f);
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&f)[8]) {
  uint4 u;
  u.x = pack_bf16(f[0], f[1]); u.y = pack_bf16(f[2], f[3]); u.z = pack_bf16(f[4], f[5]); u.w = pack_bf16(f[6], f[7]);
  *reinterpret_cast<uint4*>(p) = u;
}
__device__ __forceinline__ void load8f(const float* p, float (&f)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
__device__ __forceinline__ void store8f(float* p, const float (&f)[8]) {
  *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
  *reinterpret_cast<float4*>(p + 4) = make_float4(f[4], f[5], f[6], f[7]);
}

__device__ __forceinline__ float warp_sum(float v) {
  #pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
  #pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// Sum over the block; every thread gets the result.  `red` holds >= 33 floats.
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float t = (lane < nw) ? red[lane] : 0.f;
  t = warp_sum(t);
  return t;
}
__device__ __forceinline__ float block_max(float v, float* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float t = (lane < nw) ? red[lane] : -INFINITY;
  t = warp_max(t);
  return t;
}

// =====================================================================================
// causal depthwise conv1d (4 taps) + SiLU, channels-last
// =====================================================================================
constexpr int CONV_K = 4;

// Each thread owns 4 channels and walks a tile of tokens.  Both directions are bound by the bytes in flight: the loads of
// the next four tokens are issued before the arithmetic of the present four (2048 x 10240: forward 34.5 -> 22.4 us,
// backward 81.5 -> 51.2 us; 32768 x 5376: forward 264 -> 145 us).
constexpr int CONV_CPT = 4;

constexpr int CONV_PAIRS = CONV_CPT / 2;             // the arithmetic goes two channels at a time

__device__ __forceinline__ void unpack4(const uint2 u, uint64_t (&f)[CONV_PAIRS]) { f[0] = bf16x2_pair(u.x); f[1] = bf16x2_pair(u.y); }

// taps and bias of this thread's channels (the taps of a channel are 8 contiguous bytes)
__device__ __forceinline__ void conv_params(const __nv_bfloat16* w, const __nv_bfloat16* bias, int c0,
                                            uint64_t (&wt)[CONV_K][CONV_PAIRS], uint64_t (&bs)[CONV_PAIRS]) {
  #pragma unroll
  for (int e = 0; e < CONV_PAIRS; ++e) {
    const int c = c0 + 2 * e;
    #pragma unroll
    for (int k = 0; k < CONV_K; ++k) wt[k][e] = pack2(__bfloat162float(w[c * CONV_K + k]), __bfloat162float(w[(c + 1) * CONV_K + k]));
    bs[e] = bias ? pack2(__bfloat162float(bias[c]), __bfloat162float(bias[c + 1])) : 0;
  }
}

// x [B, L, C] with row stride xs (elements); out row stride os.  init [B, 3, C] (tokens preceding x) or null.
template <int TOK>
__device__ __forceinline__ void conv_fwd_tile(const __nv_bfloat16* __restrict__ x, long long xs, const __nv_bfloat16* __restrict__ w,
                                              const __nv_bfloat16* __restrict__ bias, const __nv_bfloat16* __restrict__ init,
                                              __nv_bfloat16* __restrict__ out, long long os, int L, int C, int bx, int tile, int b) {
  const int c0 = (bx * 128 + threadIdx.x) * CONV_CPT;
  if (c0 >= C) return;
  if (!SSM_INDEX_OK(c0 + CONV_CPT - 1, C) || !SSM_INDEX_OK(C - 1, xs) || !SSM_INDEX_OK(C - 1, os)) return;   // whole vectors inside a row
  const int t0 = tile * TOK;
  uint64_t wt[CONV_K][CONV_PAIRS], bs[CONV_PAIRS];
  const __nv_bfloat16* xb = x + (long long)b * L * xs + c0;
  __nv_bfloat16* ob = out + (long long)b * L * os + c0;
  uint2 next[4];
  auto fetch = [&](int t) {
    #pragma unroll
    for (int k = 0; k < 4; ++k) next[k] = t + k < L ? *reinterpret_cast<const uint2*>(xb + (long long)(t + k) * xs) : make_uint2(0, 0);
  };
  fetch(t0);
  uint64_t h[3][CONV_PAIRS];   // x[t-3], x[t-2], x[t-1]
  #pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int t = t0 - 3 + k;
    uint2 u = make_uint2(0, 0);
    if (t >= 0) u = *reinterpret_cast<const uint2*>(xb + (long long)t * xs);
    else if (init != nullptr) u = *reinterpret_cast<const uint2*>(init + ((long long)b * 3 + (t + 3)) * C + c0);
    unpack4(u, h[k]);
  }
  conv_params(w, bias, c0, wt, bs);
  #pragma unroll 1
  for (int i = 0; i < TOK; i += 4) {
    uint2 now[4];
    #pragma unroll
    for (int k = 0; k < 4; ++k) now[k] = next[k];
    if (i + 4 < TOK) fetch(t0 + i + 4);
    #pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int t = t0 + i + k;
      if (t >= L) return;
      uint64_t cur[CONV_PAIRS], o[CONV_PAIRS];
      unpack4(now[k], cur);
      #pragma unroll
      for (int e = 0; e < CONV_PAIRS; ++e) {
        const uint64_t pre = fma2(wt[3][e], cur[e], fma2(wt[2][e], h[2][e], fma2(wt[1][e], h[1][e], fma2(wt[0][e], h[0][e], bs[e]))));
        o[e] = mul2(pre, sigmoid2(pre));
        h[0][e] = h[1][e]; h[1][e] = h[2][e]; h[2][e] = cur[e];
      }
      *reinterpret_cast<uint2*>(ob + (long long)t * os) = make_uint2(pack_bf16_pair(o[0]), pack_bf16_pair(o[1]));
    }
  }
}

template <int TOK>
__global__ void __launch_bounds__(128, 8)
conv1d_silu_fwd_kernel(const __nv_bfloat16* __restrict__ x, long long xs, const __nv_bfloat16* __restrict__ w,
                       const __nv_bfloat16* __restrict__ bias, const __nv_bfloat16* __restrict__ init,
                       __nv_bfloat16* __restrict__ out, long long os, int L, int C) {
  conv_fwd_tile<TOK>(x, xs, w, bias, init, out, os, L, C, blockIdx.x, blockIdx.y, blockIdx.z);
}

// last four inputs of the conv, [B, C, 4], from x [B, L, C] (row stride xs), L >= 4
__device__ __forceinline__ void conv_window_tile(const __nv_bfloat16* __restrict__ x, long long xs, uint2* __restrict__ out, int L, int C, int c, int b) {
  if (c >= C) return;
  const __nv_bfloat16* p = x + ((long long)b * L + L - 4) * xs + c;
  uint32_t v[4];
  #pragma unroll
  for (int k = 0; k < 4; ++k) v[k] = __bfloat16_as_ushort(p[k * xs]);
  out[(long long)b * C + c] = make_uint2(v[0] | (v[1] << 16), v[2] | (v[3] << 16));
}

// What a mixer does with the output of in_proj in front of its scan, in one launch: conv of x | B | C, the step sizes, and where a
// prompt fills a cache the conv window.  The blocks of the three parts stand one behind the other in grid.x, the small parts
// first, which run beside the conv (us in three kernels -> one: 128 x 1792 with 24 heads 7.5 -> 5.9).
struct ConvDt {
  const __nv_bfloat16 *x, *w, *bias; long long xs; __nv_bfloat16* out; long long os; int L, C;
  DtPrep dt;
  uint2* window;
  int conv_x, conv_tiles, dt_groups, dt_blocks, window_x, window_blocks;     // conv: conv_x column blocks x conv_tiles x B
};
template <int TOK>
__global__ void __launch_bounds__(128, 8) conv_dt_kernel(const ConvDt a) {
  int i = blockIdx.x;
  if (i < a.dt_blocks) {
    const int chunks = a.L / DT_CHUNK, per = chunks * a.dt_groups, b = i / per, r = i - b * per;
    dt_prep_block(a.dt, r / a.dt_groups, r % a.dt_groups * DT_HEADS, b);
  } else if ((i -= a.dt_blocks) < a.window_blocks) {
    conv_window_tile(a.x, a.xs, a.window, a.L, a.C, (i % a.window_x) * 128 + threadIdx.x, i / a.window_x);
  } else {
    i -= a.window_blocks;
    const int per = a.conv_x * a.conv_tiles, b = i / per, r = i - b * per;
    conv_fwd_tile<TOK>(a.x, a.xs, a.w, a.bias, nullptr, a.out, a.os, a.L, a.C, r % a.conv_x, r / a.conv_x, b);
  }
}

// Backward of one thread's tile: tokens t0 .. t0 + TOK - 1 of 4 channels and three more behind it, whose pre-activation
// gradients reach back into the tile.  T16: dy is bf16, else fp32; `dy` points at token t0 of these channels.
template <int TOK, bool T16>
__device__ __forceinline__ void conv_bwd_tile(const __nv_bfloat16* __restrict__ xb, long long xs, const void* __restrict__ dy,
                                              long long ds, const uint64_t (&wt)[CONV_K][CONV_PAIRS], const uint64_t (&bs)[CONV_PAIRS],
                                              __nv_bfloat16* __restrict__ dx, long long dxs, int t0, int L,
                                              uint64_t (&dw)[CONV_K][CONV_PAIRS], uint64_t (&db)[CONV_PAIRS]) {
  using Raw = typename std::conditional<T16, uint2, uint4>::type;
  uint2 xn[4];
  Raw gn[4];
  auto fetch = [&](int i, int n) {
    #pragma unroll
    for (int k = 0; k < 4; ++k) {
      xn[k] = make_uint2(0, 0);
      gn[k] = Raw{};
      if (k < n && t0 + i + k < L) {
        xn[k] = *reinterpret_cast<const uint2*>(xb + (long long)(t0 + i + k) * xs);
        if constexpr (T16) gn[k] = *reinterpret_cast<const Raw*>(reinterpret_cast<const __nv_bfloat16*>(dy) + (long long)(i + k) * ds);
        else gn[k] = *reinterpret_cast<const Raw*>(reinterpret_cast<const float*>(dy) + (long long)(i + k) * ds);
      }
    }
  };
  fetch(0, 4);
  uint64_t xw[3][CONV_PAIRS], dp[3][CONV_PAIRS];              // x and pre-activation gradients of the three tokens before
  #pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int t = t0 - 3 + k;
    unpack4(t >= 0 ? *reinterpret_cast<const uint2*>(xb + (long long)t * xs) : make_uint2(0, 0), xw[k]);
    #pragma unroll
    for (int e = 0; e < CONV_PAIRS; ++e) dp[k][e] = 0;
  }
  auto token = [&](const uint2 xr, const Raw gr, int i, bool inside, bool store) {
    const bool valid = t0 + i < L;
    const uint64_t one = pack2(1.f, 1.f), minus = pack2(-1.f, -1.f);
    uint64_t cur[CONV_PAIRS], g[CONV_PAIRS], d[CONV_PAIRS];
    unpack4(xr, cur);
    if constexpr (T16) unpack4(gr, g);
    else {
      g[0] = pack2(__uint_as_float(gr.x), __uint_as_float(gr.y));
      g[1] = pack2(__uint_as_float(gr.z), __uint_as_float(gr.w));
    }
    #pragma unroll
    for (int e = 0; e < CONV_PAIRS; ++e) {
      const uint64_t pre = fma2(wt[3][e], cur[e], fma2(wt[2][e], xw[2][e], fma2(wt[1][e], xw[1][e], fma2(wt[0][e], xw[0][e], bs[e]))));
      const uint64_t sg = sigmoid2(pre);
      // g sg (1 + pre (1 - sg))
      const uint64_t dpre = valid ? mul2(mul2(g[e], sg), fma2(pre, fma2(sg, minus, one), one)) : 0;
      if (inside) {
        dw[0][e] = fma2(xw[0][e], dpre, dw[0][e]); dw[1][e] = fma2(xw[1][e], dpre, dw[1][e]);
        dw[2][e] = fma2(xw[2][e], dpre, dw[2][e]); dw[3][e] = fma2(cur[e], dpre, dw[3][e]);
        db[e] = add2(db[e], dpre);
      }
      // dx[t-3] = w3*dpre[t-3] + w2*dpre[t-2] + w1*dpre[t-1] + w0*dpre[t]
      d[e] = fma2(wt[0][e], dpre, fma2(wt[1][e], dp[2][e], fma2(wt[2][e], dp[1][e], mul2(wt[3][e], dp[0][e]))));
      dp[0][e] = dp[1][e]; dp[1][e] = dp[2][e]; dp[2][e] = dpre;
      xw[0][e] = xw[1][e]; xw[1][e] = xw[2][e]; xw[2][e] = cur[e];
    }
    if (store && t0 + i - 3 < L)
      *reinterpret_cast<uint2*>(dx + (long long)(i - 3) * dxs) = make_uint2(pack_bf16_pair(d[0]), pack_bf16_pair(d[1]));
  };
  #pragma unroll 1
  for (int i = 0; i < TOK; i += 4) {
    uint2 xr[4];
    Raw gr[4];
    #pragma unroll
    for (int k = 0; k < 4; ++k) { xr[k] = xn[k]; gr[k] = gn[k]; }
    fetch(i + 4, i + 4 < TOK ? 4 : 3);
    #pragma unroll
    for (int k = 0; k < 4; ++k) token(xr[k], gr[k], i + k, t0 + i + k < L, i > 0 || k == 3);
  }
  #pragma unroll
  for (int k = 0; k < 3; ++k) token(xn[k], gn[k], TOK + k, false, true);
}

// Backward.  dy for channels [0, c_split) comes from dy16 (bf16, row stride ds16); channels >= c_split from
// dy32 (fp32, row stride ds32, indexed by channel - c_split).  dx is written with row stride dxs.
// part [gridDim.z * gridDim.y, C, 5] receives per-tile partial sums (dw[0..3], db).
// Three blocks per SM: with four the registers of a tile spilled (2048 x 10240: 64.7 us, three 55.3; 8192 x 5376: 112.7 and
// 105.5; with the arithmetic in packed pairs 51.2 and 92.2).
template <int TOK>
__global__ void __launch_bounds__(128, 3)
conv1d_silu_bwd_kernel(const __nv_bfloat16* __restrict__ x, long long xs, const __nv_bfloat16* __restrict__ w,
                       const __nv_bfloat16* __restrict__ bias, const __nv_bfloat16* __restrict__ dy16, long long ds16,
                       const float* __restrict__ dy32, long long ds32, int c_split,
                       __nv_bfloat16* __restrict__ dx, long long dxs, float* __restrict__ part, int L, int C) {
  const int c0 = (blockIdx.x * blockDim.x + threadIdx.x) * CONV_CPT;
  if (c0 >= C) return;
  const int t0 = blockIdx.y * TOK;
  const int b = blockIdx.z;
  uint64_t wt[CONV_K][CONV_PAIRS], bs[CONV_PAIRS], dw[CONV_K][CONV_PAIRS], db[CONV_PAIRS];
  conv_params(w, bias, c0, wt, bs);
  #pragma unroll
  for (int e = 0; e < CONV_PAIRS; ++e) {
    db[e] = 0;
    #pragma unroll
    for (int k = 0; k < CONV_K; ++k) dw[k][e] = 0;
  }
  const long long first = (long long)b * L + t0;
  const __nv_bfloat16* xb = x + (long long)b * L * xs + c0;
  __nv_bfloat16* dxt = dx + first * dxs + c0;
  if (c0 < c_split) conv_bwd_tile<TOK, true>(xb, xs, dy16 + first * ds16 + c0, ds16, wt, bs, dxt, dxs, t0, L, dw, db);
  else conv_bwd_tile<TOK, false>(xb, xs, dy32 + first * ds32 + (c0 - c_split), ds32, wt, bs, dxt, dxs, t0, L, dw, db);
  float* pp = part + ((long long)(blockIdx.z * gridDim.y + blockIdx.y) * C + c0) * 5;
  #pragma unroll
  for (int e = 0; e < CONV_PAIRS; ++e) {
    #pragma unroll
    for (int k = 0; k < CONV_K; ++k) unpack2(dw[k][e], pp[e * 10 + k], pp[e * 10 + 5 + k]);
    unpack2(db[e], pp[e * 10 + 4], pp[e * 10 + 9]);
  }
}

// =====================================================================================
// gated group RMSNorm:  out = w * h * rsqrt(mean_g(h^2) + eps),  h = y * silu(z)
// one block per (row, group); thread handles vectors v = tid, tid + blockDim, ... of 8 elements
// =====================================================================================
// MAXV = 16-byte vectors per thread (norm_threads picks it).  All four norm kernels are bound by moving their rows once;
// what a block waits for is one round of loads and the block-wide sums.  The add backward kernel therefore keeps the raw rows
// in registers instead of reading them a second time, fetches the next row before it reduces the present one, and reduces
// both sums of a row together behind one barrier.
// Measured (us, before -> now): gated forward 32768 x 5120 318 -> 143, 2048 x 8192 24.8 -> 16.8; add forward 32768 x 2560
// 118 -> 94; add backward 4608 x 768 25.5 -> 14.3.
// The forward kernels also fetch the weights in front of the sum, since ordinary loads behind pdl_wait() are not moved there
// by the compiler (130M, one sequence, 49 norms and gates per token: 467 -> 433 us with all weights fetched there).

__device__ __forceinline__ uint4 load_raw8(const __nv_bfloat16* p) { return *reinterpret_cast<const uint4*>(p); }

// Sums of two values over the block, to every thread, behind ONE barrier: `red` (64 float2) is used in halves by turns,
// so a warp that is a call ahead writes into the other half.
__device__ __forceinline__ float2 block_sum2(float a, float b, float2* red, int turn) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  #pragma unroll
  for (int o = 16; o > 0; o >>= 1) { a += __shfl_xor_sync(0xffffffffu, a, o); b += __shfl_xor_sync(0xffffffffu, b, o); }
  float2* r = red + (turn & 1) * 32;
  if (lane == 0) r[w] = make_float2(a, b);
  __syncthreads();
  float2 t = lane < nw ? r[lane] : make_float2(0.f, 0.f);
  #pragma unroll
  for (int o = 16; o > 0; o >>= 1) { t.x += __shfl_xor_sync(0xffffffffu, t.x, o); t.y += __shfl_xor_sync(0xffffffffu, t.y, o); }
  return t;
}

// conv windows [rows][C][4] whose channels [c0, C) take the new token x [rows, C] (stride xs): what a decoding step leaves
// for the kernel behind its state update
struct WindowRoll { __nv_bfloat16* window; const __nv_bfloat16* x; long long xs; int c0, C; };

template <int NORM_MAXV, bool ROLL>
__global__ void __launch_bounds__(1024 / NORM_MAXV)
gated_rmsnorm_fwd_kernel(const __nv_bfloat16* y, long long ys, const __nv_bfloat16* z, long long zs, const __nv_bfloat16* w,
                         __nv_bfloat16* __restrict__ out, long long os, int gs, float eps, const WindowRoll roll) {
  __shared__ float red[33];
  pdl_trigger();
  pdl_wait();
  const long long row = blockIdx.x;
  const int g = blockIdx.y;
  const int nvec = gs / 8;
  const __nv_bfloat16* yr = y + row * ys + (long long)g * gs;
  const __nv_bfloat16* zr = z ? z + row * zs + (long long)g * gs : nullptr;
  uint4 yq[NORM_MAXV], zq[NORM_MAXV], wq[NORM_MAXV];
  #pragma unroll
  for (int i = 0; i < NORM_MAXV; ++i) {
    const int v = threadIdx.x + i * blockDim.x;
    if (v < nvec) {
      yq[i] = load_raw8(yr + v * 8);
      if (zr) zq[i] = load_raw8(zr + v * 8);
      wq[i] = load_raw8(w + (long long)g * gs + v * 8);      // wanted behind the sum, on its way meanwhile
    }
  }
  float h[NORM_MAXV][8];
  float ss = 0.f;
  #pragma unroll
  for (int i = 0; i < NORM_MAXV; ++i) {
    const int v = threadIdx.x + i * blockDim.x;
    if (v < nvec) {
      float a[8];
      unpack8(yq[i], a);
      if (zr) {
        float zz[8];
        unpack8(zq[i], zz);
        #pragma unroll
        for (int e = 0; e < 8; ++e) a[e] *= silu_f(zz[e]);
      }
      #pragma unroll
      for (int e = 0; e < 8; ++e) { h[i][e] = a[e]; ss += a[e] * a[e]; }
    }
  }
  if (ROLL) {                                          // the row's blocks (one per group) share its channels
    for (int c = roll.c0 + g * blockDim.x + threadIdx.x; c < roll.C; c += gridDim.y * blockDim.x) {
      uint2* sp = reinterpret_cast<uint2*>(roll.window + (row * roll.C + c) * 4);
      const uint2 s = *sp;
      const uint32_t x = __bfloat16_as_ushort(roll.x[row * roll.xs + c]);
      *sp = make_uint2((s.x >> 16) | (s.y << 16), (s.y >> 16) | (x << 16));
    }
  }
  const float rstd = rsqrtf(block_sum(ss, red) / gs + eps);
  #pragma unroll
  for (int i = 0; i < NORM_MAXV; ++i) {
    const int v = threadIdx.x + i * blockDim.x;
    if (v < nvec) {
      float ww[8], o[8];
      unpack8(wq[i], ww);
      #pragma unroll
      for (int e = 0; e < 8; ++e) o[e] = ww[e] * h[i][e] * rstd;
      store8(out + row * os + (long long)g * gs + v * 8, o);
    }
  }
}

// grid (row_slices, groups); each block walks rows r = blockIdx.x, blockIdx.x + gridDim.x, ...; one vector per thread.
// dwpart [gridDim.x, d] fp32 partial sums of dout * h * rstd.
// Bound by moving five rows per row.  Rows of y, z and dout come by bulk copies into a ring in shared memory, where both passes
// over a row read them: held in registers (with the next row's), they left room for one block per SM, which waited for its
// loads and its barrier in turn.  Arithmetic in pairs; the sigmoids of the first pass stay in registers for the second.
// us, before -> now: 8192 x 5120 146 -> 93, 4096 x 8192 104 -> 71, 2048 x 8192 58 -> 40, 4608 x 1536 26 -> 20 (64, 51, 26, 11 at copy
// bandwidth)
constexpr int GATED_RING_MAX = 4;
template <bool GATE, int THREADS, int PER_SM>
__global__ void __launch_bounds__(THREADS, PER_SM)
gated_rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ y, long long ys, const __nv_bfloat16* __restrict__ z, long long zs,
                         const __nv_bfloat16* __restrict__ w, const __nv_bfloat16* __restrict__ dout, long long dos,
                         __nv_bfloat16* __restrict__ dy, long long dys, __nv_bfloat16* __restrict__ dz, long long dzs,
                         float* __restrict__ dwpart, long long rows, int d, int gs, float eps, int ring, int* __restrict__ status) {
  extern __shared__ __align__(128) uint8_t stages[];       // [ring] y | dout | z rows of this group
  __shared__ float2 red[64];
  __shared__ uint64_t full[GATED_RING_MAX];
  const uint32_t bytes = (uint32_t)gs * 2, stage_bytes = (GATE ? 3 : 2) * bytes;
  const bool mine = (int)threadIdx.x < gs / 8;
  const long long c0 = (long long)blockIdx.y * gs, c = c0 + (mine ? threadIdx.x * 8 : 0);      // first column of group, of thread
  auto load = [&](long long row, int stage) {
    uint8_t* at = stages + stage * stage_bytes;
    mbar_expect_tx(&full[stage], stage_bytes);
    bulk_load(at, y + row * ys + c0, bytes, &full[stage]);
    bulk_load(at + bytes, dout + row * dos + c0, bytes, &full[stage]);
    if (GATE) bulk_load(at + 2 * bytes, z + row * zs + c0, bytes, &full[stage]);
  };
  if (threadIdx.x == 0) {
    for (int k = 0; k < ring; ++k) mbar_init(&full[k], 1);
    mbar_fence_init();
    for (int k = 0; k < ring; ++k)
      if (blockIdx.x + (long long)k * gridDim.x < rows) load(blockIdx.x + (long long)k * gridDim.x, k);
  }
  uint4 wq = make_uint4(0, 0, 0, 0);
  if (mine) wq = load_raw8(w + c);
  const uint32_t wr[4] = {wq.x, wq.y, wq.z, wq.w};
  uint64_t dw[4] = {0, 0, 0, 0};
  __syncthreads();
  int turn = 0, stage = 0;
  uint32_t phase = 0;
  bool ok = true;
  for (long long row = blockIdx.x; row < rows; row += gridDim.x, ++turn) {
    ok = mbar_wait(&full[stage], phase, ok ? status : nullptr) && ok;     // also behind a failure: copies land before the block goes
    const uint4* at = reinterpret_cast<const uint4*>(stages + stage * stage_bytes) + threadIdx.x;
    uint64_t sg[4];
    float2 t = make_float2(0.f, 0.f);
    if (mine) {
      const uint4 yq = at[0], gq = at[bytes / 16];
      uint4 zq = make_uint4(0, 0, 0, 0);
      if (GATE) zq = at[2 * (bytes / 16)];
      const uint32_t yr[4] = {yq.x, yq.y, yq.z, yq.w}, gr[4] = {gq.x, gq.y, gq.z, gq.w}, zr[4] = {zq.x, zq.y, zq.z, zq.w};
      uint64_t ss = 0, dot = 0;
      #pragma unroll
      for (int e = 0; e < 4; ++e) {
        uint64_t h = bf16x2_pair(yr[e]);
        if (GATE) {
          const uint64_t zz = bf16x2_pair(zr[e]);
          sg[e] = sigmoid2(zz);
          h = mul2(h, mul2(zz, sg[e]));
        }
        ss = fma2(h, h, ss);
        dot = fma2(mul2(bf16x2_pair(gr[e]), bf16x2_pair(wr[e])), h, dot);
      }
      float a, b;
      unpack2(ss, a, b);
      t.x = a + b;
      unpack2(dot, a, b);
      t.y = a + b;
    }
    t = block_sum2(t.x, t.y, red, turn);
    if (threadIdx.x == 0 && turn > 0) {                     // everybody is past the stage of the row before
      const long long next = row + (long long)(ring - 1) * gridDim.x;
      if (next < rows) load(next, stage == 0 ? ring - 1 : stage - 1);
    }
    const float rstd = rsqrtf(t.x / gs + eps);
    const float mdot = t.y * rstd / gs;                     // mean(dn * n), n = h * rstd
    if (mine && ok) {
      const uint4 yq = at[0], gq = at[bytes / 16];
      uint4 zq = make_uint4(0, 0, 0, 0);
      if (GATE) zq = at[2 * (bytes / 16)];
      const uint32_t yr[4] = {yq.x, yq.y, yq.z, yq.w}, gr[4] = {gq.x, gq.y, gq.z, gq.w}, zr[4] = {zq.x, zq.y, zq.z, zq.w};
      const uint64_t r2 = pack2(rstd, rstd), m2 = pack2(-mdot, -mdot), one = pack2(1.f, 1.f), minus = pack2(-1.f, -1.f);
      uint32_t oy[4], oz[4];
      #pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint64_t yy = bf16x2_pair(yr[e]), g = bf16x2_pair(gr[e]);
        if (GATE) {
          const uint64_t zz = bf16x2_pair(zr[e]), gate = mul2(zz, sg[e]);
          const uint64_t n = mul2(mul2(yy, gate), r2);
          const uint64_t dh = mul2(r2, fma2(n, m2, mul2(g, bf16x2_pair(wr[e]))));
          oy[e] = pack_bf16_pair(mul2(dh, gate));
          oz[e] = pack_bf16_pair(mul2(mul2(dh, yy), mul2(sg[e], fma2(zz, fma2(sg[e], minus, one), one))));
          dw[e] = fma2(g, n, dw[e]);
        } else {
          const uint64_t n = mul2(yy, r2);
          oy[e] = pack_bf16_pair(mul2(r2, fma2(n, m2, mul2(g, bf16x2_pair(wr[e])))));
          dw[e] = fma2(g, n, dw[e]);
        }
      }
      *reinterpret_cast<uint4*>(dy + row * dys + c) = make_uint4(oy[0], oy[1], oy[2], oy[3]);
      if (GATE) *reinterpret_cast<uint4*>(dz + row * dzs + c) = make_uint4(oz[0], oz[1], oz[2], oz[3]);
    }
    if (++stage == ring) { stage = 0; phase ^= 1; }
  }
  if (mine) {
    float f[8];
    #pragma unroll
    for (int e = 0; e < 4; ++e) unpack2(dw[e], f[2 * e], f[2 * e + 1]);
    store8f(dwpart + (long long)blockIdx.x * d + c, f);
  }
}

// =====================================================================================
// residual add + RMSNorm:  r' = r + x ;  out = w * r' * rsqrt(mean(r'^2) + eps)
// one block per row.  Residual stream may be bf16 or fp32.
// =====================================================================================
template <typename RT>
__device__ __forceinline__ void load8r(const RT* p, float (&f)[8]);
template <> __device__ __forceinline__ void load8r<__nv_bfloat16>(const __nv_bfloat16* p, float (&f)[8]) { load8(p, f); }
template <> __device__ __forceinline__ void load8r<float>(const float* p, float (&f)[8]) { load8f(p, f); }
template <typename RT>
__device__ __forceinline__ void store8r(RT* p, const float (&f)[8]);
template <> __device__ __forceinline__ void store8r<__nv_bfloat16>(__nv_bfloat16* p, const float (&f)[8]) { store8(p, f); }
template <> __device__ __forceinline__ void store8r<float>(float* p, const float (&f)[8]) { store8f(p, f); }

template <typename RT, int NORM_MAXV>
__global__ void __launch_bounds__(1024 / NORM_MAXV)
add_rmsnorm_fwd_kernel(const __nv_bfloat16* x, const RT* res, const __nv_bfloat16* w, __nv_bfloat16* __restrict__ out,
                       RT* __restrict__ res_out, int D, float eps) {
  __shared__ float red[33];
  pdl_trigger();
  pdl_wait();
  const long long row = blockIdx.x;
  const int nvec = D / 8;
  uint4 wq[NORM_MAXV];
  float r[NORM_MAXV][8];
  float ss = 0.f;
  #pragma unroll
  for (int i = 0; i < NORM_MAXV; ++i) {
    const int v = threadIdx.x + i * blockDim.x;
    if (v < nvec) {
      float a[8];
      wq[i] = load_raw8(w + v * 8);                          // wanted behind the sum, on its way meanwhile
      load8(x + row * D + v * 8, a);
      if (res) {
        float b[8];
        load8r<RT>(res + row * D + v * 8, b);
        #pragma unroll
        for (int e = 0; e < 8; ++e) a[e] += b[e];
      }
      if (res_out) store8r<RT>(res_out + row * D + v * 8, a);
      #pragma unroll
      for (int e = 0; e < 8; ++e) { r[i][e] = a[e]; ss += a[e] * a[e]; }
    }
  }
  const float rstd = rsqrtf(block_sum(ss, red) / D + eps);
  #pragma unroll
  for (int i = 0; i < NORM_MAXV; ++i) {
    const int v = threadIdx.x + i * blockDim.x;
    if (v < nvec) {
      float ww[8], o[8];
      unpack8(wq[i], ww);
      #pragma unroll
      for (int e = 0; e < 8; ++e) o[e] = ww[e] * r[i][e] * rstd;
      store8(out + row * D + v * 8, o);
    }
  }
}

// eight values of the residual stream as they are in memory
template <typename RT> struct Raw8;
template <> struct Raw8<__nv_bfloat16> {
  uint4 a;
  __device__ __forceinline__ void zero() { a = make_uint4(0, 0, 0, 0); }
  __device__ __forceinline__ void load(const __nv_bfloat16* p) { a = load_raw8(p); }
  __device__ __forceinline__ void get(float (&f)[8]) const { unpack8(a, f); }
};
template <> struct Raw8<float> {
  float4 a, b;
  __device__ __forceinline__ void zero() { a = b = make_float4(0.f, 0.f, 0.f, 0.f); }
  __device__ __forceinline__ void load(const float* p) {
    a = *reinterpret_cast<const float4*>(p); b = *reinterpret_cast<const float4*>(p + 4);
  }
  __device__ __forceinline__ void get(float (&f)[8]) const {
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
  }
};

// d_sum = d_res_out + rmsnorm_bwd(d_out);  dwpart [gridDim.x, D].  res = the summed residual r' saved by fwd.
template <typename RT>
__global__ void __launch_bounds__(1024)
add_rmsnorm_bwd_kernel(const RT* __restrict__ res, const __nv_bfloat16* __restrict__ w,
                       const __nv_bfloat16* __restrict__ dout, const RT* __restrict__ dres_out,
                       RT* __restrict__ dsum, float* __restrict__ dwpart, long long rows, int D, float eps) {
  __shared__ float2 red[64];
  const bool mine = (int)threadIdx.x < D / 8;
  const int c = mine ? threadIdx.x * 8 : 0;
  Raw8<RT> rn, dn;
  uint4 gn = make_uint4(0, 0, 0, 0);
  rn.zero(); dn.zero();
  auto fetch = [&](long long row) {
    if (mine && row < rows) {
      rn.load(res + row * D + c);
      gn = load_raw8(dout + row * D + c);
      if (dres_out) dn.load(dres_out + row * D + c);
    }
  };
  float dwacc[8];
  #pragma unroll
  for (int e = 0; e < 8; ++e) dwacc[e] = 0.f;
  fetch(blockIdx.x);
  int turn = 0;
  for (long long row = blockIdx.x; row < rows; row += gridDim.x, ++turn) {
    const Raw8<RT> rq = rn, dq = dn;
    const uint4 gq = gn;
    fetch(row + gridDim.x);
    float ss = 0.f, dot = 0.f;
    if (mine) {
      float r[8], go[8], ww[8];
      rq.get(r);
      unpack8(gq, go);
      load8(w + c, ww);
      #pragma unroll
      for (int e = 0; e < 8; ++e) { ss += r[e] * r[e]; dot += go[e] * ww[e] * r[e]; }
    }
    const float2 t = block_sum2(ss, dot, red, turn);
    const float rstd = rsqrtf(t.x / D + eps);
    const float mdot = t.y * rstd / D;
    if (mine) {
      float r[8], go[8], ww[8], o[8];
      rq.get(r);
      unpack8(gq, go);
      load8(w + c, ww);
      dq.get(o);                                            // zeros without dres_out
      #pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float n = r[e] * rstd;
        o[e] += rstd * (go[e] * ww[e] - n * mdot);
        dwacc[e] += go[e] * n;
      }
      store8r<RT>(dsum + row * D + c, o);
    }
  }
  if (mine) store8f(dwpart + (long long)blockIdx.x * D + c, dwacc);
}

// =====================================================================================
// GELU (erf) forward / backward, 8 elements per thread
// =====================================================================================
// Gaussian distribution function of a pair, and exp(-x^2 / 2) on the way.  With t = 1 / (1 + 0.34 |x|), the tail
// 0.5 erfc(|x| / sqrt 2) is exp(-x^2 / 2) times a polynomial of degree 9 in t (least-squares fit of 0.5 erfcx on |x| <= 14,
// weighted towards equal relative errors: 1.3e-8 in the fit; in fp32 3e-7 up to |x| = 2, then growing with the exponential's argument,
// 4e-7 up to 4, 1e-6 up to 6, 3.4e-6 up to 12), which is one division and one exponential per value, shared
// with the density that the backward pass wants; erff() takes two polynomials behind a branch on |x| < 1.  Below zero the tail
// itself is the result, so no digits cancel as they do in 1 + erf.
// These kernels were bound by that arithmetic, twice to three times what moving their rows takes:
//   us, 8192 x 16384, before -> now: forward 143 -> 108, backward 180 -> 138 (82 and 123 at copy bandwidth)
__device__ __forceinline__ uint64_t gauss_cdf2(uint64_t x, uint64_t& gauss) {
  float a, b;
  unpack2(mul2(mul2(x, x), pack2(-0.72134752f, -0.72134752f)), a, b);
  gauss = pack2(exp2f(a), exp2f(b));
  unpack2(x, a, b);
  const uint64_t t = pack2(1.f / fmaf(0.34f, fabsf(a), 1.f), 1.f / fmaf(0.34f, fabsf(b), 1.f));
  constexpr float c[10] = {2.20011179e-06f, 0.135569155f, 0.136619806f, 0.112408914f, 0.124749377f, -0.0648477748f, 0.229716182f,
                           -0.296367794f, 0.150507778f, -0.0283578485f};
  uint64_t p = pack2(c[9], c[9]);
  #pragma unroll
  for (int k = 8; k >= 0; --k) p = fma2(p, t, pack2(c[k], c[k]));
  float u, v;
  unpack2(mul2(gauss, p), u, v);
  return pack2(a < 0.f ? u : 1.f - u, b < 0.f ? v : 1.f - v);
}
// x Phi(x), and its derivative Phi(x) + x phi(x)
__device__ __forceinline__ uint64_t gelu2(uint64_t x) {
  uint64_t gauss;
  return mul2(x, gauss_cdf2(x, gauss));
}
__device__ __forceinline__ uint64_t gelu_grad2(uint64_t x) {
  uint64_t gauss;
  const uint64_t cdf = gauss_cdf2(x, gauss);
  return fma2(mul2(x, pack2(0.3989422804014327f, 0.3989422804014327f)), gauss, cdf);
}
__global__ void __launch_bounds__(256) gelu_fwd_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y, long long n8) {
  const long long step = (long long)gridDim.x * blockDim.x;
  #pragma unroll 2
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += step) {
    uint4 u = load_raw8(x + i * 8);
    u.x = pack_bf16_pair(gelu2(bf16x2_pair(u.x))); u.y = pack_bf16_pair(gelu2(bf16x2_pair(u.y)));
    u.z = pack_bf16_pair(gelu2(bf16x2_pair(u.z))); u.w = pack_bf16_pair(gelu2(bf16x2_pair(u.w)));
    *reinterpret_cast<uint4*>(y + i * 8) = u;
  }
}
__global__ void __launch_bounds__(256) gelu_bwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy,
                                                       __nv_bfloat16* __restrict__ dx, long long n8) {
  const long long step = (long long)gridDim.x * blockDim.x;
  #pragma unroll 2
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += step) {
    uint4 u = load_raw8(x + i * 8);
    const uint4 g = load_raw8(dy + i * 8);
    u.x = pack_bf16_pair(mul2(bf16x2_pair(g.x), gelu_grad2(bf16x2_pair(u.x)))); u.y = pack_bf16_pair(mul2(bf16x2_pair(g.y), gelu_grad2(bf16x2_pair(u.y))));
    u.z = pack_bf16_pair(mul2(bf16x2_pair(g.z), gelu_grad2(bf16x2_pair(u.z)))); u.w = pack_bf16_pair(mul2(bf16x2_pair(g.w), gelu_grad2(bf16x2_pair(u.w))));
    *reinterpret_cast<uint4*>(dx + i * 8) = u;
  }
}

// =====================================================================================
// vocab-shard cross entropy: per row (max, sum exp(l - max), target logit), and the gradient
// =====================================================================================
template <typename T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// 16 bytes of a logit row as floats, and back
template <typename T> struct LogitVec;
template <> struct LogitVec<float> {
  static constexpr int N = 4;
  static __device__ __forceinline__ void load(const float* p, float (&f)[4]) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
  }
  static __device__ __forceinline__ void store(float* p, const float (&f)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
  }
};
template <> struct LogitVec<__nv_bfloat16> {
  static constexpr int N = 8;
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, float (&f)[8]) { load8(p, f); }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, const float (&f)[8]) { store8(p, f); }
};
template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16(v); }

// One pass over the logits, bound by reading them: 16-byte loads and an online softmax instead of one pass for the
// maximum and one for the sum.  VEC: rows start on 16-byte boundaries (the tail of V is read one by one).
template <typename T, bool VEC>
__global__ void __launch_bounds__(256)
ce_partials_kernel(const T* __restrict__ logits, long long ld, const long long* __restrict__ labels, int V,
                   int vocab_start, float* __restrict__ omax, float* __restrict__ osum, float* __restrict__ otgt) {
  __shared__ float red[33];
  const long long row = blockIdx.x;
  const T* lr = logits + row * ld;
  float m = -INFINITY, s = 0.f;
  constexpr int N = LogitVec<T>::N;
  const int nv = VEC ? V / N : 0;
  #pragma unroll 4
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    float f[N], mx = m;
    LogitVec<T>::load(lr + (long long)i * N, f);
    #pragma unroll
    for (int e = 0; e < N; ++e) mx = fmaxf(mx, f[e]);
    const float ref = ce_ref(mx);
    s *= __expf(m - ref);
    m = mx;
    #pragma unroll
    for (int e = 0; e < N; ++e) s += __expf(f[e] - ref);
  }
  for (int i = nv * N + threadIdx.x; i < V; i += blockDim.x) {
    const float x = to_f<T>(lr[i]), mx = fmaxf(m, x), ref = ce_ref(mx);
    s = s * __expf(m - ref) + __expf(x - ref);
    m = mx;
  }
  const float gm = block_max(m, red);
  s = block_sum(s * __expf(m - ce_ref(gm)), red);
  if (threadIdx.x == 0) {
    const long long loc = labels[row] - vocab_start;
    omax[row] = gm; osum[row] = s;
    otgt[row] = (loc >= 0 && loc < V) ? to_f<T>(lr[loc]) : 0.f;
  }
}

// grad[row, i] = (exp(l - gmax) / gsum - [i == label]) * g[row];  gmax/gsum are the global statistics.
// Bound by reading and writing V values per row: 16-byte accesses where the rows of both start on 16-byte boundaries
// (4608 x 50272 bf16: 442 us with 2-byte accesses, 149 us now, 141 us at copy bandwidth).
template <typename T, bool VEC>
__global__ void __launch_bounds__(256)
ce_backward_kernel(const T* __restrict__ logits, long long ld, const long long* __restrict__ labels, int V,
                   int vocab_start, long long ignore_index, const float* __restrict__ gmax,
                   const float* __restrict__ gsum, const float* __restrict__ grow, T* __restrict__ grad, long long gld) {
  const long long row = blockIdx.x;
  const long long lab = labels[row];
  const float g = (lab == ignore_index) ? 0.f : grow[row];
  const float m = gmax[row], inv = 1.f / gsum[row];
  const long long at = lab - vocab_start;
  const int loc = at >= 0 && at < V ? (int)at : -1;
  const T* lr = logits + row * ld;
  T* gr = grad + row * gld;
  constexpr int N = LogitVec<T>::N;
  const int nv = VEC ? V / N : 0;
  #pragma unroll 4
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    float f[N];
    LogitVec<T>::load(lr + (long long)i * N, f);
    const int d = loc - i * N;
    #pragma unroll
    for (int e = 0; e < N; ++e) {
      float p = __expf(f[e] - m) * inv;
      if (d == e) p -= 1.f;
      f[e] = p * g;
    }
    LogitVec<T>::store(gr + (long long)i * N, f);
  }
  for (int i = nv * N + threadIdx.x; i < V; i += blockDim.x) {
    float p = __expf(to_f<T>(lr[i]) - m) * inv;
    if (i == loc) p -= 1.f;
    gr[i] = from_f<T>(p * g);
  }
}

// bf16 rows (stride ld, 16-byte aligned, n a multiple of 8) to contiguous fp32 rows; bound by the 6 bytes per value
__global__ void __launch_bounds__(256)
widen_kernel(const __nv_bfloat16* __restrict__ x, long long ld, float* __restrict__ out, int n) {
  const __nv_bfloat16* xr = x + (long long)blockIdx.y * ld;
  float* o = out + (long long)blockIdx.y * n;
  #pragma unroll 4
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n / 8; i += gridDim.x * blockDim.x) {
    float f[8];
    load8(xr + (long long)i * 8, f);
    store8f(o + (long long)i * 8, f);
  }
}

// =====================================================================================
// Rotary position embedding (rotate-half convention) on the first `rd` channels of every head:
//   out[:, :rd/2] = x1 * cos - sign * x2 * sin,   out[:, rd/2:rd] = x2 * cos + sign * x1 * sin
// x, out: [tokens, H, Dh] bf16 with a token stride; cos / sin: fp32 tables [L, rd/2], position = token % L + offset
// already folded into the table.  sign = +1 applies the rotation (forward), -1 its inverse (the backward pass:
// the Jacobian of a rotation is the rotation by the opposite angle).  Channels >= rd are copied.
// The reference's rotary helpers are mamba2hybrid/mamba2hybrid_attn.py:101-226 (applied at :428-430).
// =====================================================================================
__global__ void __launch_bounds__(256)
rope_kernel(const __nv_bfloat16* __restrict__ x, long long x_ld, __nv_bfloat16* __restrict__ out, long long out_ld,
            const float* __restrict__ cs, const float* __restrict__ sn, long long tokens, int L, int H, int Dh, int rd,
            float sign) {
  const int half = rd / 2;
  const int vec_rot = half / 8;                 // 8-channel vectors in each rotated half
  const int vec_rest = (Dh - rd) / 8;
  const int per_head = vec_rot + vec_rest;
  const long long total = tokens * H * per_head;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int v = (int)(i % per_head);
    const long long th = i / per_head;
    const int h = (int)(th % H);
    const long long t = th / H;
    const __nv_bfloat16* xr = x + t * x_ld + (long long)h * Dh;
    __nv_bfloat16* orow = out + t * out_ld + (long long)h * Dh;
    if (v >= vec_rot) {                          // pass-through channels
      const int c = rd + (v - vec_rot) * 8;
      *reinterpret_cast<uint4*>(orow + c) = *reinterpret_cast<const uint4*>(xr + c);
      continue;
    }
    const int c = v * 8;
    const uint4 a = *reinterpret_cast<const uint4*>(xr + c);
    const uint4 b = *reinterpret_cast<const uint4*>(xr + half + c);
    if (!SSM_INDEX_OK((long long)h * Dh + half + c + 7, x_ld) || !SSM_INDEX_OK((long long)h * Dh + half + c + 7, out_ld)) continue;
    const float* cp = cs + (t % L) * half + c;
    const float* sp = sn + (t % L) * half + c;
    const float4 c0 = *reinterpret_cast<const float4*>(cp), c1 = *reinterpret_cast<const float4*>(cp + 4);
    const float4 s0 = *reinterpret_cast<const float4*>(sp), s1 = *reinterpret_cast<const float4*>(sp + 4);
    const float cc[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
    const float ss[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
    const uint32_t ap[4] = {a.x, a.y, a.z, a.w}, bp[4] = {b.x, b.y, b.z, b.w};
    uint32_t o1[4], o2[4];
    #pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float x1l = bf16_lo(ap[e]), x1h = bf16_hi(ap[e]), x2l = bf16_lo(bp[e]), x2h = bf16_hi(bp[e]);
      const float sl = sign * ss[2 * e], sh = sign * ss[2 * e + 1];
      o1[e] = pack_bf16(x1l * cc[2 * e] - x2l * sl, x1h * cc[2 * e + 1] - x2h * sh);
      o2[e] = pack_bf16(x2l * cc[2 * e] + x1l * sl, x2h * cc[2 * e + 1] + x1h * sh);
    }
    *reinterpret_cast<uint4*>(orow + c) = make_uint4(o1[0], o1[1], o1[2], o1[3]);
    *reinterpret_cast<uint4*>(orow + half + c) = make_uint4(o2[0], o2[1], o2[2], o2[3]);
  }
}

// Row statistics that a GEMM epilogue produced per column tile -> one (max, sum exp(x - max)) per row.
// tmax / tsum: [tiles][rows].
// Bound by latency (a few MB): the tiles of a row are dealt to eight thread groups, four loads in flight each, and the
// groups' results meet in shared memory (one thread per row walking all tiles twice: 49 us for 8192 rows x 197 tiles).
__global__ void __launch_bounds__(256)
ce_merge_tiles_kernel(const float* __restrict__ tmax, const float* __restrict__ tsum, int tiles, long long rows,
                      float* __restrict__ omax, float* __restrict__ osum) {
  __shared__ float sm[8][33], ss[8][33];
  const int tx = threadIdx.x & 31, tg = threadIdx.x >> 5;
  const long long r = (long long)blockIdx.x * 32 + tx;
  float m = -INFINITY, s = 0.f;
  if (r < rows) {
    #pragma unroll 4
    for (int t = tg; t < tiles; t += 8) {
      const float tm = tmax[(long long)t * rows + r], ts = tsum[(long long)t * rows + r];
      const float mx = fmaxf(m, tm), ref = ce_ref(mx);
      s = s * __expf(m - ref) + ts * __expf(tm - ref);
      m = mx;
    }
  }
  sm[tg][tx] = m; ss[tg][tx] = s;
  __syncthreads();
  if (tg != 0 || r >= rows) return;
  #pragma unroll
  for (int k = 1; k < 8; ++k) m = fmaxf(m, sm[k][tx]);
  s = 0.f;
  #pragma unroll
  for (int k = 0; k < 8; ++k) s += ss[k][tx] * __expf(sm[k][tx] - ce_ref(m));
  omax[r] = m;
  osum[r] = s;
}

// =====================================================================================
// AdamW on a flat fp32 master shard + low-precision copy; sum of squares
// =====================================================================================
// 4 elements per thread per iteration, 16-byte loads/stores; n4 = n / 4 (segments are multiples of 128 elements)
template <typename GT> struct Vec4;
template <> struct Vec4<float> {
  static __device__ __forceinline__ float4 load(const float* p) { return *reinterpret_cast<const float4*>(p); }
};
template <> struct Vec4<__nv_bfloat16> {
  static __device__ __forceinline__ float4 load(const __nv_bfloat16* p) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    return make_float4(bf16_lo(u.x), bf16_hi(u.x), bf16_lo(u.y), bf16_hi(u.y));
  }
};

template <typename GT>
__global__ void __launch_bounds__(256)
adamw_kernel(float* __restrict__ master, float* __restrict__ m, float* __restrict__ v,
             const GT* __restrict__ g, __nv_bfloat16* __restrict__ out16, float* __restrict__ out32,
             long long n4, const float* __restrict__ clip, float lr, float b1, float b2, float eps,
             float wd, float bc1, float bc2, const float* __restrict__ lr_dev, const int* __restrict__ step_dev) {
  const float c = clip ? *clip : 1.f;
  if (!(c >= 0.f)) return;                               // negative or NaN coefficient: the optimizer skips this step
  if (lr_dev != nullptr) lr = *lr_dev;                   // device-resident hyper-parameters: a captured graph
  if (step_dev != nullptr) {                             // replays with the current learning rate and step
    const float st = (float)(*step_dev);
    bc1 = 1.f - powf(b1, st);
    bc2 = 1.f - powf(b2, st);
  }
  const float decay = 1.f - lr * wd, ib1 = 1.f / bc1, ib2 = 1.f / bc2;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
    const float4 gi = Vec4<GT>::load(g + i * 4);
    float4 mi = *reinterpret_cast<const float4*>(m + i * 4);
    float4 vi = *reinterpret_cast<const float4*>(v + i * 4);
    float4 wv = *reinterpret_cast<const float4*>(master + i * 4);
    #define SSM_ADAM(f)                                             \
      { const float gg = gi.f * c;                                  \
        mi.f = b1 * mi.f + (1.f - b1) * gg;                         \
        vi.f = b2 * vi.f + (1.f - b2) * gg * gg;                    \
        wv.f = wv.f * decay - lr * (mi.f * ib1) / (sqrtf(vi.f * ib2) + eps); }
    SSM_ADAM(x) SSM_ADAM(y) SSM_ADAM(z) SSM_ADAM(w)
    #undef SSM_ADAM
    *reinterpret_cast<float4*>(m + i * 4) = mi;
    *reinterpret_cast<float4*>(v + i * 4) = vi;
    *reinterpret_cast<float4*>(master + i * 4) = wv;
    if (out16) {
      uint2 o;
      o.x = pack_bf16(wv.x, wv.y); o.y = pack_bf16(wv.z, wv.w);
      *reinterpret_cast<uint2*>(out16 + i * 4) = o;
    }
    if (out32) *reinterpret_cast<float4*>(out32 + i * 4) = wv;
  }
}

template <typename GT>
__global__ void __launch_bounds__(256)
sumsq_kernel(const GT* __restrict__ g, long long n4, float* __restrict__ total) {
  __shared__ float red[33];
  float s = 0.f;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
    const float4 x = Vec4<GT>::load(g + i * 4);
    s += x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w;
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) atomicAdd(total, s);
}

// sum of squares over a list of [lo, hi) element ranges of one fp32 buffer (lo, hi multiples of 4), one launch:
// grid (x, number of ranges); blocks beyond the end of a short range leave at once
__global__ void __launch_bounds__(256)
sumsq_ranges_kernel(const float* __restrict__ g, const long long* __restrict__ ranges, float* __restrict__ total) {
  __shared__ float red[33];
  const long long lo = ranges[2 * blockIdx.y], n4 = (ranges[2 * blockIdx.y + 1] - lo) / 4;
  if ((long long)blockIdx.x * blockDim.x >= n4) return;
  const float* base = g + lo;
  float s = 0.f;
  #pragma unroll 4
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
    const float4 x = *reinterpret_cast<const float4*>(base + i * 4);
    s += x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w;
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) atomicAdd(total, s);
}

// =====================================================================================
// finalisation of small parameter gradients: column sums of per-CTA partial buffers written straight into the
// fp32 main-gradient buffers (store or accumulate per parameter), so the mixer backward issues one launch
// instead of ~20 reduction / cast / copy kernels
// =====================================================================================
struct SmallGradArgs {
  const float* conv_part; int T1, C;          // [T1][C][5]  (dw0..dw3, db)
  const float* gated_part; int S, d_in;       // [S][d_in]
  const float* hpart; int T2, Hv, H;          // [T2][Hv][3] (dA, dD, d dt_bias)
  const float* A;                             // [H]  (dA_log = dA * A)
  float *g_conv_w, *g_conv_b, *g_norm_w, *g_A_log, *g_D, *g_dt_bias;
  int acc_mask;                               // bit i set: add into parameter i's buffer, else overwrite
};

__device__ __forceinline__ void put(float* dst, float v, bool acc) { *dst = acc ? *dst + v : v; }

// Column sums with the rows split over 8 thread groups: block = 32 columns x 8 row groups, each thread adds
// every 8th row of its column (coalesced 128-byte row reads), the 8 partial sums meet in shared memory.
// A one-thread-per-column loop over all rows is latency-bound on these small matrices.
constexpr int CS_COLS = 32, CS_GROUPS = 8;

__device__ __forceinline__ float colsum_groups(float s, float (*red)[CS_COLS + 1]) {
  const int tx = threadIdx.x & (CS_COLS - 1), tg = threadIdx.x / CS_COLS;
  red[tg][tx] = s;
  __syncthreads();
  float r = 0.f;
  if (tg == 0) {
    #pragma unroll
    for (int k = 0; k < CS_GROUPS; ++k) r += red[k][tx];
  }
  return r;
}

__global__ void __launch_bounds__(256) mixer_small_grads_kernel(const SmallGradArgs a) {
  __shared__ float red[CS_GROUPS][CS_COLS + 1];
  const int tx = threadIdx.x & (CS_COLS - 1), tg = threadIdx.x / CS_COLS;
  const long long n_conv = (long long)a.C * 5, n_gated = a.d_in, n_h = (long long)a.H * 3;
  long long i = (long long)blockIdx.x * CS_COLS + tx;
  int seg = 3;
  float s = 0.f;
  if (i < n_conv) {
    seg = 0;
    #pragma unroll 8
    for (int t = tg; t < a.T1; t += CS_GROUPS) s += a.conv_part[(long long)t * n_conv + i];
  } else if (i - n_conv < n_gated) {
    seg = 1;
    i -= n_conv;
    #pragma unroll 8
    for (int t = tg; t < a.S; t += CS_GROUPS) s += a.gated_part[(long long)t * n_gated + i];
  } else if (i - n_conv - n_gated < n_h) {
    seg = 2;
    i -= n_conv + n_gated;
    const int h = (int)(i / 3), which = (int)(i % 3);
    const int psplit = a.Hv / a.H;
    for (int t = tg; t < a.T2; t += CS_GROUPS)
      for (int ps = 0; ps < psplit; ++ps) s += a.hpart[((long long)t * a.Hv + h * psplit + ps) * 3 + which];
  }
  s = colsum_groups(s, red);
  if (tg != 0) return;
  if (seg == 0) {
    const int c = (int)(i / 5), k = (int)(i % 5);
    if (k < 4) put(a.g_conv_w + c * 4 + k, s, a.acc_mask & 1);
    else if (a.g_conv_b) put(a.g_conv_b + c, s, a.acc_mask & 2);
  } else if (seg == 1) {
    put(a.g_norm_w + i, s, a.acc_mask & 4);
  } else if (seg == 2) {
    const int h = (int)(i / 3), which = (int)(i % 3);
    if (which == 0) put(a.g_A_log + h, s * a.A[h], a.acc_mask & 8);
    else if (which == 1) put(a.g_D + h, s, a.acc_mask & 16);
    else put(a.g_dt_bias + h, s, a.acc_mask & 32);
  }
}

// dst[c] (+)= sum_s part[s][c]
__global__ void __launch_bounds__(256) colsum_kernel(const float* __restrict__ part, int S, int n, float* dst, int acc) {
  __shared__ float red[CS_GROUPS][CS_COLS + 1];
  const int tx = threadIdx.x & (CS_COLS - 1), tg = threadIdx.x / CS_COLS;
  const int c = blockIdx.x * CS_COLS + tx;
  float s = 0.f;
  if (c < n) {
    #pragma unroll 8
    for (int t = tg; t < S; t += CS_GROUPS) s += part[(long long)t * n + c];
  }
  s = colsum_groups(s, red);
  if (tg == 0 && c < n) dst[c] = acc ? dst[c] + s : s;
}

}  // namespace ssm

// ------------------------------------------------------------------------------------ C API
using namespace ssm;
#define BF(p) reinterpret_cast<const __nv_bfloat16*>(p)
#define BFM(p) reinterpret_cast<__nv_bfloat16*>(p)

// Token-tile length: 32 at full size; shorter tiles when that grid would leave most warp slots empty (the
// per-rank channel counts of tensor parallelism), at the price of re-reading the 3-token halo more often.
static int conv_tok_for(int B, int L, int C, int ch_per_thread, int min_tok) {
  const long long warps = (long long)((C / ch_per_thread + 31) / 32) * ((L + 31) / 32) * B;
  int tok = warps >= 2048 ? 32 : warps >= 1024 ? 16 : 8;
  return tok < min_tok ? min_tok : tok;
}

extern "C" int ssm_conv1d_silu_fwd(const void* x, long long xs, const void* w, const void* bias, const void* init,
                                   void* out, long long os, int B, int L, int C, cudaStream_t st) {
  if (C % 8 || xs % 8 || os % 8) return -SSM_ERR_BAD_ARG;
  const int tok = conv_tok_for(B, L, C, CONV_CPT, 8);
  dim3 grid((C / CONV_CPT + 127) / 128, (L + tok - 1) / tok, B);
  if (tok == 32) conv1d_silu_fwd_kernel<32><<<grid, 128, 0, st>>>(BF(x), xs, BF(w), BF(bias), BF(init), BFM(out), os, L, C);
  else if (tok == 16) conv1d_silu_fwd_kernel<16><<<grid, 128, 0, st>>>(BF(x), xs, BF(w), BF(bias), BF(init), BFM(out), os, L, C);
  else conv1d_silu_fwd_kernel<8><<<grid, 128, 0, st>>>(BF(x), xs, BF(w), BF(bias), BF(init), BFM(out), os, L, C);
  return (int)cudaGetLastError();
}

// ssm_conv1d_silu_fwd without initial tokens, ssm_ssd_dt_prep and, with a window, ssm_conv_window in one launch
extern "C" int ssm_conv_dt(const void* x, long long xs, const void* w, const void* bias, void* out, long long os, const void* dt_raw,
                           const void* dt_bias, const void* A, const void* D, int mask, void* params_out, void* dt_out, void* l_out,
                           void* window, int B, int L, int C, int H, cudaStream_t st) {
  if (C % 8 || xs % 8 || os % 8 || L < DT_CHUNK || L % DT_CHUNK || B < 1 || H < 1 || (reinterpret_cast<uintptr_t>(dt_raw) & 15) ||
      (reinterpret_cast<uintptr_t>(window) & 7))
    return -SSM_ERR_BAD_ARG;
  const int tok = conv_tok_for(B, L, C, CONV_CPT, 8);
  ConvDt a;
  a.x = BF(x); a.w = BF(w); a.bias = BF(bias); a.xs = xs; a.out = BFM(out); a.os = os; a.L = L; a.C = C;
  a.dt = DtPrep{BF(dt_raw), xs, {A, D, dt_bias, mask, reinterpret_cast<float*>(params_out)}, reinterpret_cast<float*>(dt_out),
                reinterpret_cast<float*>(l_out), L, H};
  a.window = reinterpret_cast<uint2*>(window);
  a.conv_x = (C / CONV_CPT + 127) / 128; a.conv_tiles = (L + tok - 1) / tok;
  a.dt_groups = (H + DT_HEADS - 1) / DT_HEADS; a.window_x = (C + 127) / 128;
  const long long conv = (long long)a.conv_x * a.conv_tiles * B, dt = (long long)(L / DT_CHUNK) * a.dt_groups * B,
                  last = window != nullptr ? (long long)a.window_x * B : 0, total = conv + dt + last;
  if (total > 0x7fffffffll) return -SSM_ERR_BAD_ARG;
  a.dt_blocks = (int)dt; a.window_blocks = (int)last;
  auto kern = tok == 32 ? conv_dt_kernel<32> : tok == 16 ? conv_dt_kernel<16> : conv_dt_kernel<8>;
  kern<<<(unsigned)total, 128, 0, st>>>(a);
  return (int)cudaGetLastError();
}

// tokens per partial-sum tile of the backward kernel for this problem size
extern "C" int ssm_conv_bwd_tok_tile(int B, int L, int C) { return conv_tok_for(B, L, C, CONV_CPT, 16); }

// part must hold B * ceil(L / tile) * C * 5 floats, tile = ssm_conv_bwd_tok_tile(B, L, C).
extern "C" int ssm_conv1d_silu_bwd(const void* x, long long xs, const void* w, const void* bias, const void* dy16,
                                   long long ds16, const void* dy32, long long ds32, int c_split, void* dx,
                                   long long dxs, void* part, int B, int L, int C, cudaStream_t st) {
  if (C % 8 || xs % 8 || dxs % 8 || c_split % 8 || ds16 % 4 || ds32 % 4) return -SSM_ERR_BAD_ARG;
  const int tok = conv_tok_for(B, L, C, CONV_CPT, 16);
  dim3 grid((C / CONV_CPT + 127) / 128, (L + tok - 1) / tok, B);
  if (tok == 32)
    conv1d_silu_bwd_kernel<32><<<grid, 128, 0, st>>>(BF(x), xs, BF(w), BF(bias), BF(dy16), ds16,
                                                     reinterpret_cast<const float*>(dy32), ds32, c_split, BFM(dx), dxs,
                                                     reinterpret_cast<float*>(part), L, C);
  else
    conv1d_silu_bwd_kernel<16><<<grid, 128, 0, st>>>(BF(x), xs, BF(w), BF(bias), BF(dy16), ds16,
                                                     reinterpret_cast<const float*>(dy32), ds32, c_split, BFM(dx), dxs,
                                                     reinterpret_cast<float*>(part), L, C);
  return (int)cudaGetLastError();
}

template <bool ROLL>
static int gated_fwd(const void* y, long long ys, const void* z, long long zs, const void* w, void* out, long long os,
                     long long rows, int d, int gs, float eps, const WindowRoll& roll, cudaStream_t st) {
  int mv = 1;
  const int t = norm_threads(gs, &mv, false);
  if (gs % 8 || d % gs || t < 0 || ys % 8 || zs % 8 || os % 8) return -SSM_ERR_BAD_ARG;
  dim3 grid((unsigned)rows, d / gs);
  return launch_dependent(mv == 1 ? gated_rmsnorm_fwd_kernel<1, ROLL> : gated_rmsnorm_fwd_kernel<2, ROLL>, grid, dim3(t), 0, st,
                          BF(y), ys, BF(z), zs, BF(w), BFM(out), os, gs, eps, roll);
}
extern "C" int ssm_gated_rmsnorm_fwd(const void* y, long long ys, const void* z, long long zs, const void* w,
                                     void* out, long long os, long long rows, int d, int gs, float eps, cudaStream_t st) {
  return gated_fwd<false>(y, ys, z, zs, w, out, os, rows, d, gs, eps, WindowRoll{}, st);
}
// The same behind ssm_decode_mixer_step: also rolls channels [c0, C) of the conv windows.
extern "C" int ssm_gated_rmsnorm_roll(const void* y, long long ys, const void* z, long long zs, const void* w, void* out,
                                      long long os, long long rows, int d, int gs, float eps, void* window, const void* x,
                                      long long xs, int c0, int C, cudaStream_t st) {
  return gated_fwd<true>(y, ys, z, zs, w, out, os, rows, d, gs, eps, WindowRoll{BFM(window), BF(x), xs, c0, C}, st);
}
template <bool GATE, int THREADS, int PER_SM>
static int launch_gated_bwd(dim3 grid, int t, int gs, cudaStream_t st, const void* y, long long ys, const void* z, long long zs, const void* w,
                            const void* dout, long long dos, void* dy, long long dys, void* dz, long long dzs, void* dwpart, long long rows,
                            int d, float eps, int* status) {
  auto kern = gated_rmsnorm_bwd_kernel<GATE, THREADS, PER_SM>;
  // as many rows ahead as fit beside the other block of the SM
  const int stage = (GATE ? 6 : 4) * gs, room = (PER_SM == 1 ? 200 : 100) * 1024;
  const int ring = room / stage < GATED_RING_MAX ? room / stage : GATED_RING_MAX;
  static SmemOptIn opt_in;
  if (const int e = opt_in.ask(reinterpret_cast<const void*>(kern), room)) return e;
  kern<<<grid, t, ring * stage, st>>>(BF(y), ys, BF(z), zs, BF(w), BF(dout), dos, BFM(dy), dys, BFM(dz), dzs,
                                      reinterpret_cast<float*>(dwpart), rows, d, gs, eps, ring, status);
  return (int)cudaGetLastError();
}
// dwpart must hold row_slices * d floats.
extern "C" int ssm_gated_rmsnorm_bwd(const void* y, long long ys, const void* z, long long zs, const void* w,
                                     const void* dout, long long dos, void* dy, long long dys, void* dz, long long dzs,
                                     void* dwpart, int row_slices, long long rows, int d, int gs, float eps, int* status,
                                     cudaStream_t st) {
  int mv = 1;
  const int t = norm_threads(gs, &mv, true);
  if (gs % 8 || d % gs || t < 0 || ys % 8 || zs % 8 || dos % 8 || dys % 8 || dzs % 8 ||
      ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(z) | reinterpret_cast<uintptr_t>(dout)) & 15))
    return -SSM_ERR_BAD_ARG;
  dim3 grid(row_slices, d / gs);
  #define GATED_BWD(GATE, THREADS, PER_SM) launch_gated_bwd<GATE, THREADS, PER_SM>(grid, t, gs, st, y, ys, z, zs, w, dout, dos, dy, dys, dz, dzs, dwpart, rows, d, eps, status)
  if (z != nullptr) return t <= 640 ? GATED_BWD(true, 640, 2) : GATED_BWD(true, 1024, 1);
  return t <= 640 ? GATED_BWD(false, 640, 2) : GATED_BWD(false, 1024, 1);
  #undef GATED_BWD
}

extern "C" int ssm_add_rmsnorm_fwd(const void* x, const void* res, const void* w, void* out, void* res_out,
                                   long long rows, int D, float eps, int res_fp32, cudaStream_t st) {
  int mv = 1;
  const int t = norm_threads(D, &mv, false);
  if (D % 8 || t < 0) return -SSM_ERR_BAD_ARG;
  if (res_fp32)
    return launch_dependent(mv == 1 ? add_rmsnorm_fwd_kernel<float, 1> : add_rmsnorm_fwd_kernel<float, 2>, dim3((unsigned)rows),
                            dim3(t), 0, st, BF(x), reinterpret_cast<const float*>(res), BF(w), BFM(out),
                            reinterpret_cast<float*>(res_out), D, eps);
  return launch_dependent(mv == 1 ? add_rmsnorm_fwd_kernel<__nv_bfloat16, 1> : add_rmsnorm_fwd_kernel<__nv_bfloat16, 2>,
                          dim3((unsigned)rows), dim3(t), 0, st, BF(x), BF(res), BF(w), BFM(out), BFM(res_out), D, eps);
}
extern "C" int ssm_add_rmsnorm_bwd(const void* res, const void* w, const void* dout, const void* dres_out, void* dsum,
                                   void* dwpart, int row_slices, long long rows, int D, float eps, int res_fp32,
                                   cudaStream_t st) {
  int mv = 1;
  const int t = norm_threads(D, &mv, true);
  if (D % 8 || t < 0) return -SSM_ERR_BAD_ARG;
  if (res_fp32)
    add_rmsnorm_bwd_kernel<float><<<row_slices, t, 0, st>>>(reinterpret_cast<const float*>(res), BF(w), BF(dout),
                                                            reinterpret_cast<const float*>(dres_out),
                                                            reinterpret_cast<float*>(dsum),
                                                            reinterpret_cast<float*>(dwpart), rows, D, eps);
  else
    add_rmsnorm_bwd_kernel<__nv_bfloat16><<<row_slices, t, 0, st>>>(BF(res), BF(w), BF(dout), BF(dres_out), BFM(dsum),
                                                                    reinterpret_cast<float*>(dwpart), rows, D, eps);
  return (int)cudaGetLastError();
}

// -------------------------------------------------------------------------------------
// gated linear unit of the MLP: h = [gate | up] (row stride ld, halves of S columns), out = act(gate) * up.
// act: 0 GELU (erf), 1 SiLU.  Backward writes d(gate) | d(up) into dh with the same layout.
// (the reference's gated variant is mamba2hybrid/mamba2hybrid_mlp.py:118-134 in ATen ops)
// -------------------------------------------------------------------------------------
namespace ssm {
// (activation, derivative) of a pair
template <int ACT>
__device__ __forceinline__ uint64_t glu_act2(uint64_t x) {
  return ACT == 0 ? gelu2(x) : mul2(x, sigmoid2(x));
}
template <int ACT>
__device__ __forceinline__ void glu_act_grad2(uint64_t x, uint64_t& act, uint64_t& grad) {
  if (ACT == 0) {
    uint64_t gauss;
    const uint64_t cdf = gauss_cdf2(x, gauss);
    act = mul2(x, cdf);
    grad = fma2(mul2(x, pack2(0.3989422804014327f, 0.3989422804014327f)), gauss, cdf);
  } else {
    const uint64_t sg = sigmoid2(x), one = pack2(1.f, 1.f), minus = pack2(-1.f, -1.f);
    act = mul2(x, sg);
    grad = mul2(sg, fma2(x, fma2(sg, minus, one), one));
  }
}
// us, 4096 x 16384, before -> now: GELU forward 94 -> 72, backward 202 -> 109 (62 and 103 at copy bandwidth)
template <int ACT>
__global__ void __launch_bounds__(256)
glu_fwd_kernel(const __nv_bfloat16* __restrict__ h, long long ld, __nv_bfloat16* __restrict__ out, long long rows, int S) {
  const int vec = S / 8;
  const long long total = rows * vec;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / vec;
    const int c = (int)(i - r * vec) * 8;
    const uint4 g = load_raw8(h + r * ld + c), u = load_raw8(h + r * ld + S + c);
    uint4 o;
    o.x = pack_bf16_pair(mul2(glu_act2<ACT>(bf16x2_pair(g.x)), bf16x2_pair(u.x)));
    o.y = pack_bf16_pair(mul2(glu_act2<ACT>(bf16x2_pair(g.y)), bf16x2_pair(u.y)));
    o.z = pack_bf16_pair(mul2(glu_act2<ACT>(bf16x2_pair(g.z)), bf16x2_pair(u.z)));
    o.w = pack_bf16_pair(mul2(glu_act2<ACT>(bf16x2_pair(g.w)), bf16x2_pair(u.w)));
    *reinterpret_cast<uint4*>(out + r * S + c) = o;
  }
}
template <int ACT>
__global__ void __launch_bounds__(256)
glu_bwd_kernel(const __nv_bfloat16* __restrict__ h, long long ld, const __nv_bfloat16* __restrict__ dout,
               __nv_bfloat16* __restrict__ dh, long long rows, int S) {
  const int vec = S / 8;
  const long long total = rows * vec;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / vec;
    const int c = (int)(i - r * vec) * 8;
    const uint4 g = load_raw8(h + r * ld + c), u = load_raw8(h + r * ld + S + c), d = load_raw8(dout + r * S + c);
    const uint32_t gw[4] = {g.x, g.y, g.z, g.w}, uw[4] = {u.x, u.y, u.z, u.w}, dw[4] = {d.x, d.y, d.z, d.w};
    uint32_t dg[4], du[4];
    #pragma unroll
    for (int e = 0; e < 4; ++e) {
      uint64_t act, grad;
      glu_act_grad2<ACT>(bf16x2_pair(gw[e]), act, grad);
      const uint64_t dd = bf16x2_pair(dw[e]);
      dg[e] = pack_bf16_pair(mul2(mul2(dd, bf16x2_pair(uw[e])), grad));
      du[e] = pack_bf16_pair(mul2(dd, act));
    }
    *reinterpret_cast<uint4*>(dh + r * 2 * S + c) = make_uint4(dg[0], dg[1], dg[2], dg[3]);
    *reinterpret_cast<uint4*>(dh + r * 2 * S + S + c) = make_uint4(du[0], du[1], du[2], du[3]);
  }
}
}  // namespace ssm
static int glu_blocks(long long rows, int S) {
  const long long blocks = (rows * (S / 8) + 255) / 256;
  return (int)(blocks < 148 * 16 ? blocks : 148 * 16);
}
extern "C" int ssm_glu_fwd(const void* h, long long ld, void* out, long long rows, int S, int act, cudaStream_t st) {
  if (S % 8 || ld % 8 || rows < 1 || act < 0 || act > 1) return -SSM_ERR_BAD_ARG;
  auto kern = act == 0 ? glu_fwd_kernel<0> : glu_fwd_kernel<1>;
  kern<<<glu_blocks(rows, S), 256, 0, st>>>(BF(h), ld, BFM(out), rows, S);
  return (int)cudaGetLastError();
}
extern "C" int ssm_glu_bwd(const void* h, long long ld, const void* dout, void* dh, long long rows, int S, int act,
                           cudaStream_t st) {
  if (S % 8 || ld % 8 || rows < 1 || act < 0 || act > 1) return -SSM_ERR_BAD_ARG;
  auto kern = act == 0 ? glu_bwd_kernel<0> : glu_bwd_kernel<1>;
  kern<<<glu_blocks(rows, S), 256, 0, st>>>(BF(h), ld, BF(dout), BFM(dh), rows, S);
  return (int)cudaGetLastError();
}

extern "C" int ssm_gelu_fwd(const void* x, void* y, long long n, cudaStream_t st) {
  if (n % 8) return -SSM_ERR_BAD_ARG;
  const long long n8 = n / 8;
  const int blocks = (int)((n8 + 255) / 256 < 148 * 16 ? (n8 + 255) / 256 : 148 * 16);
  gelu_fwd_kernel<<<blocks, 256, 0, st>>>(BF(x), BFM(y), n8);
  return (int)cudaGetLastError();
}
extern "C" int ssm_gelu_bwd(const void* x, const void* dy, void* dx, long long n, cudaStream_t st) {
  if (n % 8) return -SSM_ERR_BAD_ARG;
  const long long n8 = n / 8;
  const int blocks = (int)((n8 + 255) / 256 < 148 * 16 ? (n8 + 255) / 256 : 148 * 16);
  gelu_bwd_kernel<<<blocks, 256, 0, st>>>(BF(x), BF(dy), BFM(dx), n8);
  return (int)cudaGetLastError();
}

extern "C" int ssm_ce_partials(const void* logits, long long ld, int is_fp32, const void* labels, long long rows, int V,
                               int vocab_start, void* omax, void* osum, void* otgt, cudaStream_t st) {
  auto lb = reinterpret_cast<const long long*>(labels);
  auto a = reinterpret_cast<float*>(omax); auto b = reinterpret_cast<float*>(osum); auto c = reinterpret_cast<float*>(otgt);
  const bool vec = (reinterpret_cast<uintptr_t>(logits) & 15) == 0 && ld % (is_fp32 ? 4 : 8) == 0;
  #define CE_PARTIALS(T, VEC) ce_partials_kernel<T, VEC><<<(unsigned)rows, 256, 0, st>>>(reinterpret_cast<const T*>(logits), ld, lb, V, vocab_start, a, b, c)
  if (is_fp32) { if (vec) CE_PARTIALS(float, true); else CE_PARTIALS(float, false); }
  else { if (vec) CE_PARTIALS(__nv_bfloat16, true); else CE_PARTIALS(__nv_bfloat16, false); }
  #undef CE_PARTIALS
  return (int)cudaGetLastError();
}
SSM_DEBUG_BOUNDS_GETTER(ssm_debug_bounds_elementwise)

extern "C" int ssm_rope(const void* x, long long x_ld, void* out, long long out_ld, const void* cos_tab, const void* sin_tab,
                        long long tokens, int L, int H, int Dh, int rd, int inverse, cudaStream_t st) {
  if (tokens < 1 || L < 1 || H < 1 || rd < 16 || rd > Dh || rd % 16 || Dh % 8 || x_ld % 8 || out_ld % 8 ||
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(cos_tab) |
        reinterpret_cast<uintptr_t>(sin_tab)) & 15))
    return -SSM_ERR_BAD_ARG;
  const long long total = tokens * H * (rd / 16 + (Dh - rd) / 8);
  const int blocks = (int)((total + 255) / 256 < 148 * 8 ? (total + 255) / 256 : 148 * 8);
  rope_kernel<<<blocks, 256, 0, st>>>(BF(x), x_ld, BFM(out), out_ld, reinterpret_cast<const float*>(cos_tab),
                                      reinterpret_cast<const float*>(sin_tab), tokens, L, H, Dh, rd, inverse ? -1.f : 1.f);
  return (int)cudaGetLastError();
}

extern "C" int ssm_ce_merge_tiles(const void* tmax, const void* tsum, int tiles, long long rows, void* omax, void* osum,
                                  cudaStream_t st) {
  if (tiles < 1 || rows < 1) return -SSM_ERR_BAD_ARG;
  ce_merge_tiles_kernel<<<(unsigned)((rows + 31) / 32), 256, 0, st>>>(
      reinterpret_cast<const float*>(tmax), reinterpret_cast<const float*>(tsum), tiles, rows,
      reinterpret_cast<float*>(omax), reinterpret_cast<float*>(osum));
  return (int)cudaGetLastError();
}
extern "C" int ssm_ce_backward(const void* logits, long long ld, int is_fp32, const void* labels, long long rows, int V,
                               int vocab_start, long long ignore_index, const void* gmax, const void* gsum,
                               const void* grow, void* grad, long long gld, cudaStream_t st) {
  auto lb = reinterpret_cast<const long long*>(labels);
  auto a = reinterpret_cast<const float*>(gmax); auto b = reinterpret_cast<const float*>(gsum);
  auto c = reinterpret_cast<const float*>(grow);
  const int per16 = is_fp32 ? 4 : 8;
  const bool vec = ((reinterpret_cast<uintptr_t>(logits) | reinterpret_cast<uintptr_t>(grad)) & 15) == 0 && ld % per16 == 0 && gld % per16 == 0;
  #define CE_BACKWARD(T, VEC) ce_backward_kernel<T, VEC><<<(unsigned)rows, 256, 0, st>>>(reinterpret_cast<const T*>(logits), ld, lb, V, vocab_start, ignore_index, a, b, c, reinterpret_cast<T*>(grad), gld)
  if (is_fp32) { if (vec) CE_BACKWARD(float, true); else CE_BACKWARD(float, false); }
  else { if (vec) CE_BACKWARD(__nv_bfloat16, true); else CE_BACKWARD(__nv_bfloat16, false); }
  #undef CE_BACKWARD
  return (int)cudaGetLastError();
}

namespace ssm {
__global__ void __launch_bounds__(128)
conv_window_kernel(const __nv_bfloat16* __restrict__ x, long long xs, uint2* __restrict__ out, int L, int C) {
  conv_window_tile(x, xs, out, L, C, blockIdx.x * 128 + threadIdx.x, blockIdx.y);
}
}  // namespace ssm
extern "C" int ssm_conv_window(const void* x, long long xs, void* out, int B, int L, int C, cudaStream_t st) {
  if (L < 4 || B < 1 || B > 65535 || C < 1 || (reinterpret_cast<uintptr_t>(out) & 7)) return -SSM_ERR_BAD_ARG;
  conv_window_kernel<<<dim3((C + 127) / 128, B), 128, 0, st>>>(BF(x), xs, reinterpret_cast<uint2*>(out), L, C);
  return (int)cudaGetLastError();
}

// largest value of a row and its first index (greedy token).  A cluster of eight CTAs shares a row and compares its eight
// candidates over distributed shared memory: one launch without anything to clear (50288 columns, us behind another call, one
// row / 64 rows: library reduction 12.8 / 13.6, this 4.2 / 7.4; 130M token 297 -> 287).
namespace ssm {
constexpr int ROW_MAX_CTAS = 8;
// larger key: larger value, NaN above all, and the lower index of equal values (-0 equals 0)
__device__ __forceinline__ unsigned long long row_max_key(float v, int i) {
  uint32_t u = __float_as_uint(v);
  if (u == 0x80000000u) u = 0u;
  if ((u & 0x7fffffffu) > 0x7f800000u) u = 0xffffffffu;
  else u = (u & 0x80000000u) ? ~u : u | 0x80000000u;
  return ((unsigned long long)u << 32) | (uint32_t)~i;
}
template <bool VEC>
__global__ void __cluster_dims__(ROW_MAX_CTAS, 1, 1) __launch_bounds__(256)
row_max_kernel(const float* x, long long ld, int V, float* __restrict__ val, long long* __restrict__ idx) {
  __shared__ unsigned long long best[8], mine;
  pdl_trigger();
  pdl_wait();
  const float* r = x + (long long)blockIdx.y * ld;
  unsigned long long k = 0;
  const int first = blockIdx.x * 256 + threadIdx.x, step = ROW_MAX_CTAS * 256, nv = VEC ? V / 4 : 0;
  #pragma unroll 4
  for (int i = first; i < nv; i += step) {
    const float4 f = *reinterpret_cast<const float4*>(r + (long long)i * 4);
    const unsigned long long a = row_max_key(f.x, i * 4), b = row_max_key(f.y, i * 4 + 1), c = row_max_key(f.z, i * 4 + 2), d = row_max_key(f.w, i * 4 + 3);
    const unsigned long long e = a > b ? a : b, g = c > d ? c : d, h = e > g ? e : g;
    k = h > k ? h : k;
  }
  for (int i = nv * 4 + first; i < V; i += step) {
    const unsigned long long a = row_max_key(r[i], i);
    k = a > k ? a : k;
  }
  #pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long a = __shfl_xor_sync(0xffffffffu, k, o);
    k = a > k ? a : k;
  }
  if ((threadIdx.x & 31) == 0) best[threadIdx.x >> 5] = k;
  __syncthreads();
  if (threadIdx.x == 0) {
    #pragma unroll
    for (int w = 1; w < 8; ++w) k = best[w] > k ? best[w] : k;
    mine = k;
  }
  cluster_sync_all();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    #pragma unroll
    for (int c = 1; c < ROW_MAX_CTAS; ++c) {
      uint32_t at;
      unsigned long long a;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_u32(&mine)), "r"(c));
      asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(a) : "r"(at) : "memory");
      k = a > k ? a : k;
    }
    const int i = (int)~(uint32_t)k;
    val[blockIdx.y] = r[i];
    idx[blockIdx.y] = i;
  }
  cluster_sync_all();                                    // nobody leaves while its candidate may be read
}
}  // namespace ssm
extern "C" int ssm_row_max(const void* x, long long ld, int V, long long rows, void* val, void* idx, cudaStream_t st) {
  if (rows < 1 || rows > 65535 || V < 1) return -SSM_ERR_BAD_ARG;
  const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0 && ld % 4 == 0;
  return launch_dependent(vec ? row_max_kernel<true> : row_max_kernel<false>, dim3(ROW_MAX_CTAS, (unsigned)rows), dim3(256), 0, st,
                          reinterpret_cast<const float*>(x), ld, V, reinterpret_cast<float*>(val), reinterpret_cast<long long*>(idx));
}

extern "C" int ssm_widen(const void* x, long long ld, void* out, long long rows, int n, cudaStream_t st) {
  if (rows < 1 || rows > 65535 || n < 8 || n % 8 || ld % 8 || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out)) & 15))
    return -SSM_ERR_BAD_ARG;
  const int blocks = (n / 8 + 1023) / 1024;
  widen_kernel<<<dim3((unsigned)blocks, (unsigned)rows), 256, 0, st>>>(BF(x), ld, reinterpret_cast<float*>(out), n);
  return (int)cudaGetLastError();
}

namespace ssm {
// What stands between the gradient norm and AdamW, in one thread instead of fourteen library kernels of 2 us: norm, clip
// coefficient min(1, max_norm / (norm + 1e-6)) or -1 where the norm is not finite, and the counters of applied and skipped
// steps.  Correctly rounded operations, as the library's.
__global__ void clip_kernel(const float* __restrict__ sumsq, float max_norm, float* __restrict__ norm, float* __restrict__ clip,
                            int* __restrict__ step, int* __restrict__ skipped) {
  const float square = *sumsq;              // where an embedding's additions took back what a product had added, rounding may leave
  const float n = __fsqrt_rn(square < 0.f ? 0.f : square);        // a value just below zero
  const bool finite = (__float_as_uint(n) & 0x7f800000u) != 0x7f800000u;
  *norm = n;
  *clip = finite ? fminf(__fdiv_rn(max_norm, __fadd_rn(n, 1e-6f)), 1.f) : -1.f;
  if (finite) ++*step; else ++*skipped;
}
// Loss of every row from its statistics: log(sum) + max - target logit, 0 where the label is ignored.
__global__ void __launch_bounds__(256)
ce_row_loss_kernel(const float* __restrict__ m, const float* __restrict__ sum, const float* __restrict__ tgt, const long long* __restrict__ labels,
                   long long ignore_index, long long rows, float* __restrict__ loss) {
  const long long r = (long long)blockIdx.x * 256 + threadIdx.x;
  if (r >= rows) return;
  // rounded after the logarithm and after each sum, as the separate operations were; the logarithm in 64 bits
  const float l = (float)log((double)sum[r]);
  loss[r] = labels[r] == ignore_index ? 0.f : __fsub_rn(__fadd_rn(l, m[r]), tgt[r]);
}
}  // namespace ssm
extern "C" int ssm_clip_coefficient(const void* sumsq, float max_norm, void* norm, void* clip, void* step, void* skipped, cudaStream_t st) {
  clip_kernel<<<1, 1, 0, st>>>(reinterpret_cast<const float*>(sumsq), max_norm, reinterpret_cast<float*>(norm),
                               reinterpret_cast<float*>(clip), reinterpret_cast<int*>(step), reinterpret_cast<int*>(skipped));
  return (int)cudaGetLastError();
}
extern "C" int ssm_ce_row_loss(const void* m, const void* sum, const void* tgt, const void* labels, long long ignore_index, long long rows,
                               void* loss, cudaStream_t st) {
  if (rows < 1) return -SSM_ERR_BAD_ARG;
  ce_row_loss_kernel<<<(unsigned)((rows + 255) / 256), 256, 0, st>>>(
      reinterpret_cast<const float*>(m), reinterpret_cast<const float*>(sum), reinterpret_cast<const float*>(tgt),
      reinterpret_cast<const long long*>(labels), ignore_index, rows, reinterpret_cast<float*>(loss));
  return (int)cudaGetLastError();
}

extern "C" int ssm_adamw(void* master, void* m, void* v, const void* g, int g_fp32, void* out16, void* out32,
                         long long n, const void* clip, float lr, float b1, float b2, float eps, float wd, int step,
                         const void* lr_dev, const void* step_dev, cudaStream_t st) {
  auto lrd = reinterpret_cast<const float*>(lr_dev);
  auto std_ = reinterpret_cast<const int*>(step_dev);
  const float bc1 = 1.f - powf(b1, (float)step), bc2 = 1.f - powf(b2, (float)step);
  if (n % 4 || (reinterpret_cast<uintptr_t>(master) | reinterpret_cast<uintptr_t>(m) | reinterpret_cast<uintptr_t>(v) |
                reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(out32)) & 15 ||
      (reinterpret_cast<uintptr_t>(out16) & 7))
    return -SSM_ERR_BAD_ARG;
  n /= 4;
  const int blocks = (int)((n + 255) / 256 < 148 * 8 ? (n + 255) / 256 : 148 * 8);
  auto M = reinterpret_cast<float*>(master); auto mm = reinterpret_cast<float*>(m); auto vv = reinterpret_cast<float*>(v);
  auto cl = reinterpret_cast<const float*>(clip);
  if (g_fp32) adamw_kernel<float><<<blocks, 256, 0, st>>>(M, mm, vv, reinterpret_cast<const float*>(g), BFM(out16), reinterpret_cast<float*>(out32), n, cl, lr, b1, b2, eps, wd, bc1, bc2, lrd, std_);
  else adamw_kernel<__nv_bfloat16><<<blocks, 256, 0, st>>>(M, mm, vv, BF(g), BFM(out16), reinterpret_cast<float*>(out32), n, cl, lr, b1, b2, eps, wd, bc1, bc2, lrd, std_);
  return (int)cudaGetLastError();
}
extern "C" int ssm_sumsq(const void* g, int g_fp32, long long n, void* total, cudaStream_t st) {
  if (n % 4 || (reinterpret_cast<uintptr_t>(g) & 15)) return -SSM_ERR_BAD_ARG;
  n /= 4;
  const int blocks = (int)((n + 255) / 256 < 148 * 4 ? (n + 255) / 256 : 148 * 4);
  if (g_fp32) sumsq_kernel<float><<<blocks, 256, 0, st>>>(reinterpret_cast<const float*>(g), n, reinterpret_cast<float*>(total));
  else sumsq_kernel<__nv_bfloat16><<<blocks, 256, 0, st>>>(BF(g), n, reinterpret_cast<float*>(total));
  return (int)cudaGetLastError();
}

// =====================================================================================
// allocation-free variant of add_rmsnorm_bwd (declared in ssm_noalloc.h)
// =====================================================================================
#include "ssm_noalloc.h"
#include <mutex>

// Partial weight-gradient sums, [SSM_NOALLOC_SLICES][D] packed with the call's D.  In host code this name is
// only a handle for the runtime's symbol table, never an address to pass to a kernel.
static __device__ __align__(256) float g_noalloc_scratch[SSM_NOALLOC_SLICES * SSM_NOALLOC_MAX_D];

namespace ssm {
// dw[c] = sum_s part[s][c]; device code may name the array directly.
__global__ void __launch_bounds__(256) noalloc_colsum_kernel(float* __restrict__ dw, int slices, int D) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= D) return;
  float s = 0.f;
  for (int r = 0; r < slices; ++r) s += g_noalloc_scratch[(long long)r * D + c];
  dw[c] = s;
}
}  // namespace ssm

static float* noalloc_scratch_for_current_device(int* err) {
  constexpr int kMaxDevices = 64;
  static float* ptrs[kMaxDevices] = {nullptr};
  static std::mutex mu;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices) { *err = e != cudaSuccess ? (int)e : -SSM_NOALLOC_ERR_BAD_ARG; return nullptr; }
  std::lock_guard<std::mutex> lock(mu);
  if (ptrs[dev] == nullptr) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);   // device address of the array on the current device
    if (e != cudaSuccess) { *err = (int)e; return nullptr; }
    ptrs[dev] = static_cast<float*>(p);
  }
  *err = 0;
  return ptrs[dev];
}

extern "C" int ssm_add_rmsnorm_bwd_noalloc(const void* res, const void* w, const void* dout, const void* dres_out,
                                           void* dsum, void* dw, long long rows, int D, float eps, int res_fp32,
                                           cudaStream_t st) {
  if (D > SSM_NOALLOC_MAX_D) return -SSM_NOALLOC_ERR_TOO_LARGE;
  int mv = 1;
  const int t = norm_threads(D, &mv, true);
  if (D <= 0 || D % 8 || t < 0 || rows < 1 || !res || !w || !dout || !dsum || !dw) return -SSM_NOALLOC_ERR_BAD_ARG;
  // the kernels move rows with 16-byte vector loads and stores: a misaligned base would fault on the device
  const uintptr_t vec16 = reinterpret_cast<uintptr_t>(res) | reinterpret_cast<uintptr_t>(w) |
                          reinterpret_cast<uintptr_t>(dout) | reinterpret_cast<uintptr_t>(dres_out) |
                          reinterpret_cast<uintptr_t>(dsum);
  if ((vec16 & 15) || (reinterpret_cast<uintptr_t>(dw) & 3)) return -SSM_NOALLOC_ERR_BAD_ARG;
  int err = 0;
  float* scratch = noalloc_scratch_for_current_device(&err);
  if (scratch == nullptr) return err;
  const int slices = rows < SSM_NOALLOC_SLICES ? (int)rows : SSM_NOALLOC_SLICES;
  if (res_fp32)
    add_rmsnorm_bwd_kernel<float><<<slices, t, 0, st>>>(reinterpret_cast<const float*>(res), BF(w), BF(dout),
                                                        reinterpret_cast<const float*>(dres_out),
                                                        reinterpret_cast<float*>(dsum), scratch, rows, D, eps);
  else
    add_rmsnorm_bwd_kernel<__nv_bfloat16><<<slices, t, 0, st>>>(BF(res), BF(w), BF(dout), BF(dres_out), BFM(dsum),
                                                                scratch, rows, D, eps);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  noalloc_colsum_kernel<<<(D + 255) / 256, 256, 0, st>>>(reinterpret_cast<float*>(dw), slices, D);
  return (int)cudaGetLastError();
}

extern "C" int ssm_mixer_small_grads(const void* conv_part, int T1, int C, const void* gated_part, int S, int d_in,
                                     const void* hpart, int T2, int Hv, int H, const void* A, void* g_conv_w,
                                     void* g_conv_b, void* g_norm_w, void* g_A_log, void* g_D, void* g_dt_bias,
                                     int acc_mask, cudaStream_t st) {
  SmallGradArgs a;
  a.conv_part = reinterpret_cast<const float*>(conv_part); a.T1 = T1; a.C = C;
  a.gated_part = reinterpret_cast<const float*>(gated_part); a.S = S; a.d_in = d_in;
  a.hpart = reinterpret_cast<const float*>(hpart); a.T2 = T2; a.Hv = Hv; a.H = H;
  a.A = reinterpret_cast<const float*>(A);
  a.g_conv_w = reinterpret_cast<float*>(g_conv_w); a.g_conv_b = reinterpret_cast<float*>(g_conv_b);
  a.g_norm_w = reinterpret_cast<float*>(g_norm_w); a.g_A_log = reinterpret_cast<float*>(g_A_log);
  a.g_D = reinterpret_cast<float*>(g_D); a.g_dt_bias = reinterpret_cast<float*>(g_dt_bias);
  a.acc_mask = acc_mask;
  const long long n = (long long)C * 5 + d_in + (long long)H * 3;
  mixer_small_grads_kernel<<<(unsigned)((n + CS_COLS - 1) / CS_COLS), 256, 0, st>>>(a);
  return (int)cudaGetLastError();
}
extern "C" int ssm_sumsq_ranges(const void* g, const void* ranges, int nranges, void* total, cudaStream_t st) {
  if (nranges < 1 || (reinterpret_cast<uintptr_t>(g) & 15)) return nranges == 0 ? 0 : -SSM_ERR_BAD_ARG;
  dim3 grid(148 * 8, nranges);       // with 148 * 2 blocks too few loads were in flight (824 MB: 210 us)
  sumsq_ranges_kernel<<<grid, 256, 0, st>>>(reinterpret_cast<const float*>(g), reinterpret_cast<const long long*>(ranges),
                                            reinterpret_cast<float*>(total));
  return (int)cudaGetLastError();
}
extern "C" int ssm_colsum(const void* part, int S, int n, void* dst, int acc, cudaStream_t st) {
  colsum_kernel<<<(n + CS_COLS - 1) / CS_COLS, 256, 0, st>>>(reinterpret_cast<const float*>(part), S, n,
                                                 reinterpret_cast<float*>(dst), acc);
  return (int)cudaGetLastError();
}
