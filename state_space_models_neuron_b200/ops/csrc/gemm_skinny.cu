// bf16 GEMM with few rows (decoding, last-token logits): C[M,N] = X[M,K] W[N,K]^T, M <= 128, fp32 accumulation.
// Both kernels are bound by reading the weights once from HBM, so the work is cut for bytes in flight on every SM and
// not for tensor throughput: the 128-row tiles of gemm.cu leave most SMs idle here (N / 192 tiles) and pay a read-back
// of K slices through global memory.
//   M <= 8    (16 with few weights) gemm_rows_kernel: 16 weight rows per CTA, its eight warps share K and add up in shared
//             memory; operands go from global memory straight into mma.sync fragments (no descriptors, barriers or TMEM
//             to set up: at these sizes set-up latency is as long as the transfer).
//   M <= 128  gemm_cols_kernel: the weight rows are the 128-row side of a tcgen05 tile and X the 32-, 64- or 128-column
//             side; a cluster of up to eight CTAs shares K and adds the partial tiles over distributed shared memory.
// Sums run in a fixed order, so results are reproducible.
// Measured (weights from HBM, us; tiled kernel of gemm.cu -> these, single launches): 1 x 3352 x 768 11.5 -> 3.2, 1 x 50288 x 768
// 25.6 -> 17.2, 5 x 1024 x 2048 18.0 -> 5.9, 64 x 10576 x 2560 27.4 -> 16.1 (8.3 at copy bandwidth), 64 x 2560 x 5120
// 24.0 -> 12.1, 64 x 50288 x 2560 62.6 -> 48.2 (39.3), 128 x 768 x 1536 18.7 -> 8.0, 128 x 10576 x 2560 29.7 -> 19.8,
// 128 x 4096 x 8192 32.4 -> 21.6.
#include "common.cuh"

namespace ssm {

// ------------------------------------------------------------------------------------------------ M <= 8 (16)
constexpr int ROWS_WARPS = 8;
constexpr int ROWS_CHUNK = 64;       // K elements of one warp step: 128 bytes of every weight row

__device__ __forceinline__ void mma_16x8x16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                            uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
               "{%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// volatile: the loads of a step stay in front of its products (the compiler would otherwise sink each load to its use
// and leave two of them in flight).  The assembler does the same unless a __syncwarp() stands behind the loads: with it (us per
// call behind another call, one row) 768 x 1536 4.1 -> 2.7, 2560 x 5120 12.2 -> 7.2, 4096 x 8192 19.7 -> 12.3, 18560 x 4096
// 31.0 -> 24.8 (23.2 at copy bandwidth).  Ordinary loads, for X and the weights: see pdl_wait().
__device__ __forceinline__ uint4 ld8_if(bool in, const __nv_bfloat16* p) {
  uint4 u;
  asm volatile(
      "{\n\t"
      ".reg .pred q;\n\t"
      "setp.ne.s32 q, %5, 0;\n\t"
      "mov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
      "@q ld.global.v4.u32 {%0, %1, %2, %3}, [%4];\n\t"
      "}\n"
      : "=&r"(u.x), "=&r"(u.y), "=&r"(u.z), "=&r"(u.w) : "l"(p), "r"((int)in) : "memory");
  return u;
}

// Chunks that a warp fetches at once: its share of K in equal turns of at most four, so that no turn is nearly empty
static int rows_unroll(int per_warp) {
  const int turns = (per_warp + 3) / 4;
  return (per_warp + turns - 1) / turns;
}

// A lane holds 8 consecutive k of row lane / 4 (16 bytes); as the order of k inside a product does not matter, elements
// {0,1} and {2,3} of the eight are the two k pairs of one 16-wide step and {4..7} those of the next, for both operands.
template <int NT, int UNROLL>         // NT tiles of 8 rows of X, UNROLL chunks in flight
__global__ void __launch_bounds__(ROWS_WARPS * 32)
gemm_rows_kernel(const __nv_bfloat16* x, long long ldx, const __nv_bfloat16* w, long long ldw, const __nv_bfloat16* bias,
                 __nv_bfloat16* __restrict__ out, long long ldo, int M, int N, int K) {
  __shared__ float red[ROWS_WARPS][NT * 8][16 + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * 16;
  // rows beyond N or M read row 0; what they produce is not stored
  const __nv_bfloat16* wl = w + (long long)(n0 + g < N ? n0 + g : 0) * ldw + t * 8;
  const __nv_bfloat16* wh = w + (long long)(n0 + g + 8 < N ? n0 + g + 8 : 0) * ldw + t * 8;
  const __nv_bfloat16* xr[NT];
  #pragma unroll
  for (int i = 0; i < NT; ++i) xr[i] = x + (long long)(i * 8 + g < M ? i * 8 + g : 0) * ldx + t * 8;
  pdl_trigger();
  {
    // this warp's first weights on their way to L2 while the predecessor finishes: a 128-byte line per row and chunk
    const int k = (warp + (lane >> 4) * ROWS_WARPS) * ROWS_CHUNK, r = n0 + (lane & 15);
    if (k < K && r < N) prefetch_l2(w + (long long)r * ldw + k);
  }
  pdl_wait();
  float acc[NT][4];
  #pragma unroll
  for (int i = 0; i < NT; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
  const int chunks = (K + ROWS_CHUNK - 1) / ROWS_CHUNK;
  for (int c0 = warp; c0 < chunks; c0 += ROWS_WARPS * UNROLL) {
    uint4 a[UNROLL][2][2], b[UNROLL][2][NT];
    #pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const int k0 = (c0 + u * ROWS_WARPS) * ROWS_CHUNK;
      #pragma unroll
      for (int s = 0; s < 2; ++s) {
        const bool in = k0 + s * 32 + t * 8 < K;     // K is a multiple of 8
        const int k = k0 + s * 32;
        a[u][s][0] = ld8_if(in, wl + k);
        a[u][s][1] = ld8_if(in, wh + k);
        #pragma unroll
        for (int i = 0; i < NT; ++i) b[u][s][i] = ld8_if(in, xr[i] + k);
      }
    }
    __syncwarp();                             // all loads go out in front of it
    #pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      #pragma unroll
      for (int s = 0; s < 2; ++s) {
        const uint4 p = a[u][s][0], q = a[u][s][1];
        #pragma unroll
        for (int i = 0; i < NT; ++i) {
          mma_16x8x16(acc[i], p.x, q.x, p.y, q.y, b[u][s][i].x, b[u][s][i].y);
          mma_16x8x16(acc[i], p.z, q.z, p.w, q.w, b[u][s][i].z, b[u][s][i].w);
        }
      }
    }
  }
  #pragma unroll
  for (int i = 0; i < NT; ++i) {
    red[warp][i * 8 + 2 * t][g] = acc[i][0];
    red[warp][i * 8 + 2 * t + 1][g] = acc[i][1];
    red[warp][i * 8 + 2 * t][g + 8] = acc[i][2];
    red[warp][i * 8 + 2 * t + 1][g + 8] = acc[i][3];
  }
  __syncthreads();
  const int m = threadIdx.x >> 4, r = threadIdx.x & 15;
  if (m < M && m < NT * 8 && n0 + r < N) {
    float v = red[0][m][r];
    #pragma unroll
    for (int k = 1; k < ROWS_WARPS; ++k) v += red[k][m][r];
    if (bias != nullptr) v += __bfloat162float(bias[n0 + r]);
    out[(long long)m * ldo + n0 + r] = __float2bfloat16(v);
  }
}

// ------------------------------------------------------------------------------------------------ norm and product, M <= 8
// A norm in front of a product with at most eight rows, in one kernel with every rounding of the two that it stands for
// (the forward norms of elementwise.cu and gemm_rows_kernel): the sums of squares are taken in the order of a norm kernel's
// threads, an operand is bf16((wn h) rstd), and the products add up as in gemm_rows_kernel, so results are the same bits.
//   add    h = x + residual, the new residual is stored by the blocks in turn (64 columns c by block c mod gridDim.x)
//   gated  h = y silu(z); also rolls the conv windows of a decoding step (see WindowRoll in elementwise.cu)
// While a warp waits for its first weights it forms wn h of its share of the rows, in fp32 in shared memory, and its part of
// the sums; behind one barrier the operands are read from there.
// Every block reads the M rows for itself (from L2) next to 32 K bytes of weights, so this pays for narrow products, where a
// kernel's start and end cost more than its work, and not for wide ones; the caller has the rule and the times.
enum { NORM_ADD_BF16 = 0, NORM_ADD_FP32 = 1, NORM_GATED = 2 };

struct NormLinearParams {
  const __nv_bfloat16* a; long long lda;      // x, or y
  const void* b; long long ldb;               // residual (bf16 or fp32) or null, or z
  const __nv_bfloat16* wn;
  void* res_out;                              // add: [M, K] contiguous
  const __nv_bfloat16* w; long long ldw;
  const __nv_bfloat16* bias;
  __nv_bfloat16* out; long long ldo;
  int M, N, K, groups;                        // groups: equal parts of K, each a multiple of ROWS_CHUNK if more than one
  int threads;                                // a norm kernel's threads for one group
  float eps;
  __nv_bfloat16* window; const __nv_bfloat16* xnew; long long xs; int c0, C;      // gated: windows [M][C][4], channels [c0, C)
};
constexpr int NORM_PARTS = 8;                 // warps of a norm kernel's block at most 4096 columns
// floats of a row of wn h: four beyond the columns, so that two rows of a fragment meet no bank twice
__host__ __device__ constexpr int norm_row(int K) { return K + 4; }

__device__ __forceinline__ uint4 ld16_if(bool in, const void* p) { return ld8_if(in, reinterpret_cast<const __nv_bfloat16*>(p)); }

// VECS: 16-byte vectors of a row (or group) per thread of the norm kernel
template <int KIND, int UNROLL, int VECS>
__global__ void __launch_bounds__(ROWS_WARPS * 32, KIND == NORM_GATED ? 1 : 2)
norm_linear_kernel(const NormLinearParams p) {
  extern __shared__ __align__(16) float rows[];          // [M][norm_row(K)] wn h
  __shared__ float parts[8][8][NORM_PARTS];              // [row][group][warp of a norm kernel] sums of squares
  __shared__ float red[ROWS_WARPS][8][16 + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * 16, width = p.K / p.groups, chunks = (p.K + ROWS_CHUNK - 1) / ROWS_CHUNK;
  const __nv_bfloat16* wl = p.w + (long long)(n0 + g < p.N ? n0 + g : 0) * p.ldw + t * 8;
  const __nv_bfloat16* wh = p.w + (long long)(n0 + g + 8 < p.N ? n0 + g + 8 : 0) * p.ldw + t * 8;
  pdl_trigger();
  {
    // this warp's first weights on their way to L2 while the predecessor finishes: a 128-byte line per row and chunk
    const int r = n0 + (lane & 15);
    if (r < p.N) {
      #pragma unroll
      for (int u = 0; u < UNROLL; u += 2) {
        const int k = (warp + (u + (lane >> 4)) * ROWS_WARPS) * ROWS_CHUNK;
        if (k < p.K) prefetch_l2(p.w + (long long)r * p.ldw + k);
      }
    }
  }
  pdl_wait();
  uint4 wa[UNROLL][2], wb[UNROLL][2];
  auto fetch = [&](int c0) {
    #pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      #pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int k = (c0 + u * ROWS_WARPS) * ROWS_CHUNK + s * 32;
        const bool in = k + t * 8 < p.K;                 // K is a multiple of 8
        wa[u][s] = ld8_if(in, wl + k);
        wb[u][s] = ld8_if(in, wh + k);
      }
    }
    __syncwarp();                                        // all loads go out in front of it
  };
  fetch(warp);
  // ---- wn h and the sums of squares: an item stands for one warp of a norm kernel's block of one row and group; the vectors
  // of ITEMS of them are under way at once
  const int warps = p.threads >> 5, per_row = p.groups * warps, items = p.M * per_row;
  constexpr int ITEMS = KIND == NORM_GATED && VECS == 1 ? 3 : 1;
  for (int i0 = warp; i0 < items; i0 += ROWS_WARPS * ITEMS) {
    uint4 xa[ITEMS][VECS], xb[ITEMS][VECS], xc[ITEMS][VECS], nw[ITEMS][VECS];
    #pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const int i = i0 + j * ROWS_WARPS, m = i / per_row, rest = i - m * per_row, grp = rest / warps;
      #pragma unroll
      for (int q = 0; q < VECS; ++q) {
        const int v = (rest - grp * warps) * 32 + lane + q * p.threads, k = grp * width + v * 8;
        const bool in = i < items && v * 8 < width;
        xa[j][q] = ld16_if(in, p.a + m * p.lda + k);
        if (KIND == NORM_ADD_FP32) {
          const float* r = reinterpret_cast<const float*>(p.b) + m * p.ldb + k;
          xb[j][q] = ld16_if(in && p.b != nullptr, r);
          xc[j][q] = ld16_if(in && p.b != nullptr, r + 4);
        } else {
          xb[j][q] = ld16_if(in && p.b != nullptr, reinterpret_cast<const __nv_bfloat16*>(p.b) + m * p.ldb + k);
        }
        nw[j][q] = ld16_if(in, p.wn + k);
      }
    }
    __syncwarp();                                        // all loads go out in front of it
    #pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const int i = i0 + j * ROWS_WARPS, m = i / per_row, rest = i - m * per_row, grp = rest / warps, vw = rest - grp * warps;
      if (i >= items) break;
      float ss = 0.f;
      #pragma unroll
      for (int q = 0; q < VECS; ++q) {
        const int v = vw * 32 + lane + q * p.threads, k = grp * width + v * 8;
        float h[8], n[8], r[8];
        unpack8(xa[j][q], h);
        unpack8(nw[j][q], n);
        if (KIND == NORM_ADD_FP32) {
          const uint4 lo = xb[j][q], hi = xc[j][q];
          r[0] = __uint_as_float(lo.x); r[1] = __uint_as_float(lo.y); r[2] = __uint_as_float(lo.z); r[3] = __uint_as_float(lo.w);
          r[4] = __uint_as_float(hi.x); r[5] = __uint_as_float(hi.y); r[6] = __uint_as_float(hi.z); r[7] = __uint_as_float(hi.w);
        } else {
          unpack8(xb[j][q], r);
        }
        if (v * 8 < width) {
          if (KIND == NORM_GATED) {
            #pragma unroll
            for (int e = 0; e < 8; ++e) h[e] *= silu_f(r[e]);
          } else {
            if (p.b != nullptr) {
              #pragma unroll
              for (int e = 0; e < 8; ++e) h[e] += r[e];
            }
            if ((k / ROWS_CHUNK) % gridDim.x == blockIdx.x) {
              if (KIND == NORM_ADD_FP32) {
                float* o = reinterpret_cast<float*>(p.res_out) + (long long)m * p.K + k;
                *reinterpret_cast<float4*>(o) = make_float4(h[0], h[1], h[2], h[3]);
                *reinterpret_cast<float4*>(o + 4) = make_float4(h[4], h[5], h[6], h[7]);
              } else {
                *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.res_out) + (long long)m * p.K + k) =
                    make_uint4(pack_bf16(h[0], h[1]), pack_bf16(h[2], h[3]), pack_bf16(h[4], h[5]), pack_bf16(h[6], h[7]));
              }
            }
          }
          #pragma unroll
          for (int e = 0; e < 8; ++e) ss += h[e] * h[e];
          float4* o = reinterpret_cast<float4*>(rows + m * norm_row(p.K) + k);
          o[0] = make_float4(n[0] * h[0], n[1] * h[1], n[2] * h[2], n[3] * h[3]);
          o[1] = make_float4(n[4] * h[4], n[5] * h[5], n[6] * h[6], n[7] * h[7]);
        }
      }
      __syncwarp();
      #pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if (lane < NORM_PARTS && (lane == vw || lane >= warps)) parts[m][grp][lane] = lane == vw ? ss : 0.f;
    }
  }
  __syncthreads();
  // ---- the product
  const bool mine = g < p.M;                             // lanes of rows beyond M bring zeros
  const float* row = rows + (mine ? g : 0) * norm_row(p.K);
  float acc[4] = {0.f, 0.f, 0.f, 0.f}, rstd = 0.f;
  int have = -1;                                         // group of rstd
  for (int c0 = warp; c0 < chunks; c0 += ROWS_WARPS * UNROLL) {
    if (c0 != warp) fetch(c0);
    #pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const int k0 = (c0 + u * ROWS_WARPS) * ROWS_CHUNK, grp = p.groups == 1 ? 0 : k0 / width;
      if (k0 >= p.K) break;
      if (grp != have) {                                 // the sum over the warps as block_sum forms it
        const float* q = parts[mine ? g : 0][grp];
        rstd = rsqrtf((((q[0] + q[4]) + (q[2] + q[6])) + ((q[1] + q[5]) + (q[3] + q[7]))) / width + p.eps);
        have = grp;
      }
      #pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int k = k0 + s * 32 + t * 8;
        float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
        if (mine && k < p.K) { lo = *reinterpret_cast<const float4*>(row + k); hi = *reinterpret_cast<const float4*>(row + k + 4); }
        const uint4 q = wa[u][s], v = wb[u][s];
        mma_16x8x16(acc, q.x, v.x, q.y, v.y, pack_bf16(lo.x * rstd, lo.y * rstd), pack_bf16(lo.z * rstd, lo.w * rstd));
        mma_16x8x16(acc, q.z, v.z, q.w, v.w, pack_bf16(hi.x * rstd, hi.y * rstd), pack_bf16(hi.z * rstd, hi.w * rstd));
      }
    }
  }
  red[warp][2 * t][g] = acc[0];
  red[warp][2 * t + 1][g] = acc[1];
  red[warp][2 * t][g + 8] = acc[2];
  red[warp][2 * t + 1][g + 8] = acc[3];
  if (KIND == NORM_GATED) {
    const long long channels = p.C - p.c0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < p.M * channels; i += (long long)gridDim.x * blockDim.x) {
      const int r = (int)(i / channels), c = p.c0 + (int)(i % channels);
      uint2* sp = reinterpret_cast<uint2*>(p.window + ((long long)r * p.C + c) * 4);
      const uint2 s = *sp;
      const uint32_t x = __bfloat16_as_ushort(p.xnew[r * p.xs + c]);
      *sp = make_uint2((s.x >> 16) | (s.y << 16), (s.y >> 16) | (x << 16));
    }
  }
  __syncthreads();
  const int m = threadIdx.x >> 4, r = threadIdx.x & 15;
  if (m < p.M && n0 + r < p.N) {
    float v = red[0][m][r];
    #pragma unroll
    for (int k = 1; k < ROWS_WARPS; ++k) v += red[k][m][r];
    if (p.bias != nullptr) v += __bfloat162float(p.bias[n0 + r]);
    p.out[(long long)m * p.ldo + n0 + r] = __float2bfloat16(v);
  }
}

template <int KIND>
static int launch_norm_linear(NormLinearParams p, bool fp32, int sms, cudaStream_t stream) {
  // bases and strides of 16-byte vectors, groups of whole chunks
  const uintptr_t a = reinterpret_cast<uintptr_t>(p.a) | reinterpret_cast<uintptr_t>(p.b) | reinterpret_cast<uintptr_t>(p.wn) |
                      reinterpret_cast<uintptr_t>(p.w) | reinterpret_cast<uintptr_t>(p.res_out);
  const size_t smem = (size_t)p.M * norm_row(p.K) * sizeof(float);
  if (p.M < 1 || p.M > 8 || p.N < 1 || p.K < 8 || p.K > 4096 || p.K % 8 || (a & 15) || p.lda % 8 || p.ldw % 8 || p.ldb % (fp32 ? 4 : 8) ||
      !(p.groups == 1 || ((p.groups == 2 || p.groups == 4 || p.groups == 8) && p.K % (p.groups * ROWS_CHUNK) == 0)))
    return -SSM_ERR_BAD_ARG;
  int vecs = 1;
  p.threads = norm_threads(p.K / p.groups, &vecs, false);
  if (p.threads < 0 || p.threads > 32 * NORM_PARTS || (vecs == 2 && KIND != NORM_GATED)) return -SSM_ERR_BAD_ARG;
  const unsigned grid = (unsigned)((p.N + 15) / 16);
  const int unroll = rows_unroll(((p.K + ROWS_CHUNK - 1) / ROWS_CHUNK + ROWS_WARPS - 1) / ROWS_WARPS);
  const bool few = unroll <= 2 || grid > (unsigned)sms;
  auto kern = unroll == 1 && vecs == 1 ? norm_linear_kernel<KIND, 1, 1> : few ? norm_linear_kernel<KIND, 2, 1> : norm_linear_kernel<KIND, 3, 1>;
  int which = unroll == 1 && vecs == 1 ? 0 : few ? 1 : 2;
  if constexpr (KIND == NORM_GATED)
    if (vecs == 2) { kern = few ? norm_linear_kernel<KIND, 2, 2> : norm_linear_kernel<KIND, 3, 2>; which = few ? 3 : 4; }
  static SmemOptIn opt_in[5];
  if (smem > 40 * 1024)                                  // more than a kernel has without asking, beside its own tables
    if (const int e = opt_in[which].ask(reinterpret_cast<const void*>(kern), 8 * norm_row(4096) * (int)sizeof(float))) return e;
  return launch_dependent(kern, dim3(grid), dim3(ROWS_WARPS * 32), smem, stream, p);
}

// ------------------------------------------------------------------------------------------------ M <= 128
template <int NB, int STAGES>
struct ColsSmem {
  static constexpr int W_BYTES = 128 * 128;            // [128 weight rows][64 k]
  static constexpr int X_BYTES = NB * 128;             // [NB rows of X][64 k]
  static constexpr int STAGE_BYTES = W_BYTES + X_BYTES;
  static constexpr int BAR_OFF = STAGES * STAGE_BYTES;
  static constexpr int TOTAL = BAR_OFF + 128 + 1024;
  static_assert(NB * 128 * 4 <= BAR_OFF, "the partial tile reuses the ring");
};

constexpr int COLS_MAX_SPLIT = 8;    // CTAs of a cluster (portable size)

struct ColsParams {
  const __nv_bfloat16* bias;
  __nv_bfloat16* out;
  long long ldo;
  int M, N, kblocks, split;
  int* status;
};

__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t local_addr, uint32_t rank) {
  uint32_t a;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local_addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a)
               : "memory");
  return v;
}

// grid (split, tiles of 128 weight rows), clusters of `split` CTAs along K; 128 threads, PER_SM CTAs per SM.
template <int NB, int STAGES, int PER_SM>
__global__ void __launch_bounds__(128, PER_SM)
gemm_cols_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, const ColsParams p) {
  using S = ColsSmem<NB, STAGES>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + S::BAR_OFF);
  uint64_t* empty = full + STAGES;
  uint64_t* done = empty + STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int slice = blockIdx.x, n0 = blockIdx.y * 128;
  const int kb0 = (int)((long long)slice * p.kblocks / p.split), kb1 = (int)((long long)(slice + 1) * p.kblocks / p.split);
  constexpr int TMEM_COLS = NB < 32 ? 32 : NB;

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(done, 1);
    mbar_fence_init();
    tma_prefetch_desc(&tm_w); tma_prefetch_desc(&tm_x);
  }
  pdl_trigger();
  if (tid == 0)
    for (int kb = kb0; kb < kb1 && kb < kb0 + STAGES; ++kb) tma_prefetch_l2_2d(&tm_w, kb * 64, n0);
  if (warp == 1) { tmem_alloc(tmem_slot, TMEM_COLS); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  pdl_wait();

  if (warp == 0) {
    if (lane == 0) {
      int last[STAGES];
      #pragma unroll
      for (int s = 0; s < STAGES; ++s) last[s] = -1;
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&empty[stage], phase ^ 1, p.status)) { ok = false; break; }
        uint8_t* sw = smem + stage * S::STAGE_BYTES;
        mbar_expect_tx(&full[stage], S::STAGE_BYTES);
        tma_load_2d(sw, &tm_w, kb * 64, n0, &full[stage]);
        tma_load_2d(sw + S::W_BYTES, &tm_x, kb * 64, 0, &full[stage]);
        last[stage] = (int)phase;
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      if (!ok) {                       // let copies in flight land before the shared memory goes away
        #pragma unroll
        for (int s = 0; s < STAGES; ++s)
          if (last[s] >= 0) mbar_wait(&full[s], (uint32_t)last[s], nullptr);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = make_idesc_bf16(128, NB, 0, 0);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&full[stage], phase, p.status)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t sw = smem_u32(smem + stage * S::STAGE_BYTES);
        const uint64_t dw = make_smem_desc_sw128(sw, 16, 1024), dx = make_smem_desc_sw128(sw + S::W_BYTES, 16, 1024);
        #pragma unroll
        for (int kk = 0; kk < 4; ++kk) umma_bf16(tmem, dw + kk * 2, dx + kk * 2, idesc, (kb != kb0 || kk != 0) ? 1u : 0u);
        umma_commit(&empty[stage]);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      if (ok) umma_commit(done);
    }
    __syncwarp();
  }
  const bool ok = __syncthreads_and(mbar_wait(done, 0, p.status));
  tc_fence_after_sync();
  // thread = output column (weight row) n0 + tid, TMEM columns = rows of the output
  const int n = n0 + tid;
  float b = 0.f;
  if (p.bias != nullptr && n < p.N) b = __bfloat162float(p.bias[n]);
  float* part = reinterpret_cast<float*>(smem);        // [NB][128]; all loads have landed and all MMAs have read them
  if (ok) {
    #pragma unroll 1
    for (int h = 0; h < (NB + 31) / 32; ++h) {
      uint32_t v[32];
      tmem_ld32(tmem_addr(tmem, warp * 32, h * 32), v);
      tmem_ld_wait();
      if (p.split == 1) {
        #pragma unroll
        for (int e = 0; e < 32; ++e)
          if (h * 32 + e < p.M && n < p.N)
            p.out[(long long)(h * 32 + e) * p.ldo + n] = __float2bfloat16(__uint_as_float(v[e]) + b);
      } else {
        #pragma unroll
        for (int e = 0; e < 32; ++e) part[(h * 32 + e) * 128 + tid] = __uint_as_float(v[e]);
      }
    }
  }
  if (p.split > 1) {
    cluster_sync_all();
    // rows of the output are dealt to the CTAs of the cluster and their warps; a lane adds four columns, with the loads
    // from all slices in flight together
    const int c = n0 + lane * 4;
    if (ok && c < p.N) {
      float4 b4 = make_float4(0.f, 0.f, 0.f, 0.f);
      if (p.bias != nullptr) {
        b4.x = __bfloat162float(p.bias[c]);
        if (c + 1 < p.N) b4.y = __bfloat162float(p.bias[c + 1]);
        if (c + 2 < p.N) b4.z = __bfloat162float(p.bias[c + 2]);
        if (c + 3 < p.N) b4.w = __bfloat162float(p.bias[c + 3]);
      }
      const uint32_t base = smem_u32(part) + lane * 16;
      #pragma unroll 2
      for (int m = slice * 4 + warp; m < p.M; m += p.split * 4) {
        float4 v[COLS_MAX_SPLIT];
        #pragma unroll
        for (int s = 0; s < COLS_MAX_SPLIT; ++s)
          if (s < p.split) v[s] = ld_cluster_f32x4(base + m * 512, s);
        float4 t = b4;
        #pragma unroll
        for (int s = 0; s < COLS_MAX_SPLIT; ++s)
          if (s < p.split) { t.x += v[s].x; t.y += v[s].y; t.z += v[s].z; t.w += v[s].w; }
        __nv_bfloat16* o = p.out + (long long)m * p.ldo + c;
        if (c + 3 < p.N) {
          *reinterpret_cast<uint2*>(o) = make_uint2(pack_bf16(t.x, t.y), pack_bf16(t.z, t.w));
        } else {
          o[0] = __float2bfloat16(t.x);
          if (c + 1 < p.N) o[1] = __float2bfloat16(t.y);
          if (c + 2 < p.N) o[2] = __float2bfloat16(t.z);
        }
      }
    }
  }
  tc_fence_before_sync();
  if (p.split > 1) cluster_sync_all(); else __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, TMEM_COLS);
}

template <int NB, int STAGES, int PER_SM>
static int launch_cols(const void* X, long long ldx, const void* W, long long ldw, ColsParams p, int K, int sms,
                       cudaStream_t stream) {
  using S = ColsSmem<NB, STAGES>;
  auto kern = gemm_cols_kernel<NB, STAGES, PER_SM>;
  static SmemOptIn opt_in;
  if (const int e = opt_in.ask(reinterpret_cast<const void*>(kern), S::TOTAL)) return e;
  CUtensorMap tw, tx;
  int r = make_tmap_2d_bf16(&tw, W, (uint64_t)K, (uint64_t)p.N, (uint64_t)ldw * 2, 64, 128);
  if (r) return -200 - r;
  r = make_tmap_2d_bf16(&tx, X, (uint64_t)K, (uint64_t)p.M, (uint64_t)ldx * 2, 64, NB);
  if (r) return -100 - r;
  const int tiles = (p.N + 127) / 128;
  p.kblocks = (K + 63) / 64;
  // as many K slices as keep all CTAs resident at once with at least three k-blocks each
  p.split = COLS_MAX_SPLIT;
  while (p.split > 1 && ((long long)tiles * p.split > (long long)PER_SM * sms || p.kblocks / p.split < 3)) p.split /= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)p.split, (unsigned)tiles, 1);
  cfg.blockDim = dim3(128, 1, 1);
  cfg.dynamicSmemBytes = S::TOTAL;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)p.split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tw, tx, p);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

// Called by gemm.cu for plain bf16 products with K-major operands; bases 16-byte aligned, ldx and ldw multiples of 8.
// Returns false when the shape is not one of these kernels' (the caller then takes the tiled kernel).
bool gemm_skinny(const void* X, const void* W, void* C, int M, int N, int K, long long ldx, long long ldw, long long ldc,
                 const void* bias, int* status, int sms, cudaStream_t stream, int* code) {
  if (M > 128 || K % 8 || (N + 127) / 128 > 65535) return false;
  const auto* b = reinterpret_cast<const __nv_bfloat16*>(bias);
  auto* out = reinterpret_cast<__nv_bfloat16*>(C);
  // 9 to 16 rows: the direct kernel reads X once per 16 weight rows, which costs more than the set-up of the other one
  // once the weights are large (16 x 10576 x 2560: 16.4 us direct, 14.3 us tiled)
  if (M <= 8 || (M <= 16 && (long long)N * K <= (8 << 20))) {
    const auto* x = reinterpret_cast<const __nv_bfloat16*>(X);
    const auto* w = reinterpret_cast<const __nv_bfloat16*>(W);
    const unsigned grid = (unsigned)((N + 15) / 16);
    const int unroll = rows_unroll(((K + ROWS_CHUNK - 1) / ROWS_CHUNK + ROWS_WARPS - 1) / ROWS_WARPS);
    auto kern = M > 8 ? gemm_rows_kernel<2, 2> : unroll == 4 ? gemm_rows_kernel<1, 4> : unroll == 3 ? gemm_rows_kernel<1, 3>
              : gemm_rows_kernel<1, 2>;
    *code = launch_dependent(kern, dim3(grid), dim3(ROWS_WARPS * 32), 0, stream, x, ldx, w, ldw, b, out, ldc, M, N, K);
    return true;
  }
  ColsParams p;
  p.bias = b; p.out = out; p.ldo = ldc; p.M = M; p.N = N; p.kblocks = 0; p.split = 1; p.status = status;
  if (M <= 32)      *code = launch_cols<32, 3, 3>(X, ldx, W, ldw, p, K, sms, stream);
  else if (M <= 64) *code = launch_cols<64, 3, 3>(X, ldx, W, ldw, p, K, sms, stream);
  else              *code = launch_cols<128, 3, 2>(X, ldx, W, ldw, p, K, sms, stream);
  return true;
}

}  // namespace ssm

using namespace ssm;

static int device_sms() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 148;
  return sms;
}

// out[M, N] = rmsnorm(x + res) W^T (+ bias) and res_out = x + res, M <= 8.  x [M, K] bf16 (row stride ldx); res contiguous
// [M, K] of the residual type or null.  -SSM_ERR_BAD_ARG where the shape is not this kernel's.
extern "C" int ssm_add_norm_linear(const void* x, long long ldx, const void* res, void* res_out, int res_fp32, const void* wn,
                                   float eps, const void* w, long long ldw, const void* bias, void* out, long long ldo, int M,
                                   int N, int K, cudaStream_t st) {
  NormLinearParams p = {};
  p.a = reinterpret_cast<const __nv_bfloat16*>(x); p.lda = ldx; p.b = res; p.ldb = K;
  p.wn = reinterpret_cast<const __nv_bfloat16*>(wn); p.res_out = res_out; p.w = reinterpret_cast<const __nv_bfloat16*>(w);
  p.ldw = ldw; p.bias = reinterpret_cast<const __nv_bfloat16*>(bias); p.out = reinterpret_cast<__nv_bfloat16*>(out); p.ldo = ldo;
  p.M = M; p.N = N; p.K = K; p.groups = 1; p.eps = eps;
  return res_fp32 ? launch_norm_linear<NORM_ADD_FP32>(p, true, device_sms(), st) : launch_norm_linear<NORM_ADD_BF16>(p, false, device_sms(), st);
}

// out[M, N] = gated_rmsnorm(y, z) W^T (+ bias) behind ssm_decode_mixer_step, M <= 8; also rolls channels [c0, C) of the conv
// windows [M][C][4] with the new token xnew (row stride xs).
extern "C" int ssm_gated_norm_linear(const void* y, long long ldy, const void* z, long long ldz, const void* wn, int gs, float eps,
                                     const void* w, long long ldw, const void* bias, void* out, long long ldo, int M, int N, int K,
                                     void* window, const void* xnew, long long xs, int c0, int C, cudaStream_t st) {
  if (gs < 1 || K % gs) return -SSM_ERR_BAD_ARG;
  NormLinearParams p = {};
  p.a = reinterpret_cast<const __nv_bfloat16*>(y); p.lda = ldy; p.b = z; p.ldb = ldz;
  p.wn = reinterpret_cast<const __nv_bfloat16*>(wn); p.w = reinterpret_cast<const __nv_bfloat16*>(w);
  p.ldw = ldw; p.bias = reinterpret_cast<const __nv_bfloat16*>(bias); p.out = reinterpret_cast<__nv_bfloat16*>(out); p.ldo = ldo;
  p.M = M; p.N = N; p.K = K; p.groups = K / gs; p.eps = eps;
  p.window = reinterpret_cast<__nv_bfloat16*>(window); p.xnew = reinterpret_cast<const __nv_bfloat16*>(xnew); p.xs = xs;
  p.c0 = c0; p.C = C;
  if (z == nullptr) return -SSM_ERR_BAD_ARG;
  return launch_norm_linear<NORM_GATED>(p, false, device_sms(), st);
}
