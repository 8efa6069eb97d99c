// Step sizes of the SSD scan: dt = softplus(dt_raw + bias), l = inclusive running sum of A dt within each chunk of 128 tokens.
// A block of 128 threads serves one chunk of one sequence and up to eight heads, thread = token: the eight raw values of a token
// are one 16-byte load, where a block per head read a 32-byte sector of every row for one value.
#pragma once
#include "common.cuh"

namespace ssm {

constexpr int DT_CHUNK = 128, DT_HEADS = 8;

// Parameters as they are (bf16 where bit 0, 1, 2 of the mask is set for A, D, dt_bias; bit 3: A holds A_log); `out`
// (optional) receives (A, D, dt_bias) in fp32, [3][H], for the kernels behind this one.
struct HeadParams { const void* A; const void* D; const void* dt_bias; int mask; float* out; };
__device__ __forceinline__ float head_param(const void* p, int h, bool bf16) {
  return bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[h]) : reinterpret_cast<const float*>(p)[h];
}

struct DtPrep {
  const __nv_bfloat16* raw; long long row_stride;      // row (b L + t), column h; whole 16-byte vectors
  HeadParams prm;
  float *dt, *l;                                        // [B, H, L]
  int L, H;
};

// heads h0 .. h0 + 7 of chunk c of sequence b
__device__ __forceinline__ void dt_prep_block(const DtPrep& p, int c, int h0, int b) {
  __shared__ float ends[4][DT_HEADS];
  const int j = threadIdx.x, lane = j & 31, w = j >> 5;
  const long long t = (long long)c * DT_CHUNK + j;
  const int heads = p.H - h0 < DT_HEADS ? p.H - h0 : DT_HEADS;
  const __nv_bfloat16* at = p.raw + ((long long)b * p.L + t) * p.row_stride + h0;
  float v[DT_HEADS], a[DT_HEADS];
  if (heads == DT_HEADS) {
    unpack8(*reinterpret_cast<const uint4*>(at), v);
  } else {
    #pragma unroll
    for (int e = 0; e < DT_HEADS; ++e) v[e] = e < heads ? __bfloat162float(at[e]) : 0.f;
  }
  #pragma unroll
  for (int e = 0; e < DT_HEADS; ++e) {
    const int h = e < heads ? h0 + e : h0;
    float A = head_param(p.prm.A, h, p.prm.mask & 1);
    if (p.prm.mask & 8) A = -expf(A);
    const float bias = head_param(p.prm.dt_bias, h, p.prm.mask & 4);
    if (p.prm.out != nullptr && c == 0 && b == 0 && j == e && e < heads) {
      p.prm.out[h] = A;
      p.prm.out[p.H + h] = head_param(p.prm.D, h, p.prm.mask & 2);
      p.prm.out[2 * p.H + h] = bias;
    }
    v[e] = softplus_f(v[e] + bias);
    a[e] = A * v[e];
  }
  #pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    #pragma unroll
    for (int e = 0; e < DT_HEADS; ++e) {
      const float n = __shfl_up_sync(0xffffffffu, a[e], o);
      if (lane >= o) a[e] += n;
    }
  }
  if (lane == 31) {
    #pragma unroll
    for (int e = 0; e < DT_HEADS; ++e) ends[w][e] = a[e];
  }
  __syncthreads();
  #pragma unroll
  for (int e = 0; e < DT_HEADS; ++e) {
    if (e >= heads) break;
    float off = 0.f;
    for (int k = 0; k < w; ++k) off += ends[k][e];
    const long long o = ((long long)b * p.H + h0 + e) * p.L + t;
    p.dt[o] = v[e];
    p.l[o] = a[e] + off;
  }
}

}  // namespace ssm
