// Causal grouped-query flash attention for sm_100a, head_dim 128, forward and backward, on tcgen05.
// Both directions are warp-specialised: loads, products and the softmax arithmetic of neighbouring tiles overlap.
// K/V heads are indexed (kv head = q head / ratio), never replicated in memory (the reference materialises
// repeat_kv before its NKI flash kernel: mamba2hybrid/mamba2hybrid_attn.py:440-447).
// q [B*L, Hq*128], k/v [B*L, Hkv*128], out [B*L, Hq*128], lse [B, Hq, L] (natural log, of scaled scores).
#include "common.cuh"

namespace ssm {

constexpr int AT = 128;                  // tile (queries / keys)
constexpr int AD = 128;                  // head dim
constexpr int ATILE = AT * AD * 2;       // bytes of one [128][128] bf16 tile (two 16 KiB swizzle blocks)
constexpr float LOG2E = 1.4426950408889634f;

__device__ __forceinline__ uint64_t adesc_k(uint32_t base, int kk) {     // K-major, two 64-wide atoms
  return make_smem_desc_sw128(base + (kk >> 2) * (ATILE / 2) + (kk & 3) * 32, 16, 1024);
}
__device__ __forceinline__ uint64_t adesc_mn(uint32_t base, int kk) {    // MN-major, two 64-wide blocks
  return make_smem_desc_sw128(base + kk * 2048, ATILE / 2, 1024);
}
__device__ __forceinline__ uint4 apack8(const float (&f)[8]) {
  uint4 u;
  u.x = pack_bf16(f[0], f[1]); u.y = pack_bf16(f[2], f[3]); u.z = pack_bf16(f[4], f[5]); u.w = pack_bf16(f[6], f[7]);
  return u;
}
// store 8 values of row `row`, columns [col, col+8) into a [128][128] swizzled tile
__device__ __forceinline__ void tile_store8(uint8_t* tile, int row, int col, const float (&f)[8]) {
  *reinterpret_cast<uint4*>(tile + (col >> 6) * (ATILE / 2) + sw128_offset(row, (col & 63) >> 3)) = apack8(f);
}

struct AttnFwdParams {
  float* lse;
  int L, Hq, Hkv;
  float scale;
  int* status;
};

// Forward: 320 threads for a pair of query tiles (256 queries) of one head.
//   warps 0-3, 4-7  softmax of the first / second query tile, thread = query row (the row's 128 scores in registers)
//   warp 8          issues all products;  warp 9  loads K and V tiles through a ring of three
// The two tiles take turns: while one group's exponentials keep the special-function units busy, the tensor cores work on
// the other's products.  S and O of both tiles fill the 512 TMEM columns.  The online softmax and the turns of two tiles are
// those of FlashAttention (Dao et al., 2022; Shah et al., 2024).  O is rescaled in TMEM for the warps in which a row's maximum
// has grown: the largest P of a row is then 1, which bf16 holds exactly.  Rescaling only past a growth of 2^8 took 652 us
// instead of 671 for 8192 queries of 32 heads, but put a rounding on that largest P: an error against 64 bits 1.5 % higher at
// 1024 queries.
// Bound by the exponentials (16 per clock and SM: as long as the products of a tile) and the softmax arithmetic around them.
// One 128-thread group doing everything in turn took 1537 us for 8192 queries of 32 heads, this 671 us (8192 x 16: 834 -> 386,
// 4096 x 32 with 8 key heads: 436 -> 213, 4 x 1024 x 16: 77.5 -> 47.2; one box, called back to back).
constexpr int ATTN_FWD_THREADS = 320;
constexpr int KV_RING = 3;
constexpr int ATTN_FWD_SMEM = (4 + KV_RING) * ATILE + 256 + 1024;

__global__ void __launch_bounds__(ATTN_FWD_THREADS, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o,
                const AttnFwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                                  // two query tiles
  uint8_t* sP = smem + 2 * ATILE;                      // two probability tiles, output staging at the end
  uint8_t* sKV = smem + 4 * ATILE;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (4 + KV_RING) * ATILE);
  uint64_t *q_full = bars, *full = bars + 1, *empty = full + KV_RING, *s_full = empty + KV_RING, *p_ready = s_full + 2,
           *o_done = p_ready + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_done + 2);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = blockIdx.y, b = blockIdx.z, hk = h / (p.Hq / p.Hkv);
  const int qtiles = p.L / AT;
  const int q0 = 2 * ((int)gridDim.x - 1 - (int)blockIdx.x);           // longest walks first
  const int n0 = q0 + 1, n1 = q0 + 1 < qtiles ? q0 + 2 : 0;            // key tiles of the two query tiles (n1 = 0: none)
  const int n = n1 > 0 ? n1 : n0;

  if (tid == 0) {
    mbar_init(q_full, 1);
    for (int k = 0; k < KV_RING; ++k) { mbar_init(&full[k], 1); mbar_init(&empty[k], 1); }
    for (int t = 0; t < 2; ++t) { mbar_init(&s_full[t], 1); mbar_init(&p_ready[t], 128); mbar_init(&o_done[t], 1); }
    mbar_fence_init();
    tma_prefetch_desc(&tm_q); tma_prefetch_desc(&tm_k); tma_prefetch_desc(&tm_v); tma_prefetch_desc(&tm_o);
  }
  if (warp == 8) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;                    // S of tile t at 128 t, O at 256 + 128 t

  // K and V tiles in the order in which they are used: K0, K1, V0, K2, V1, ..., V(n-1)
  if (warp == 9) {
    if (lane == 0) {
      const int qt_n = n1 > 0 ? 2 : 1;
      mbar_expect_tx(q_full, qt_n * ATILE);
      for (int t = 0; t < qt_n; ++t) {
        tma_load_2d(sQ + t * ATILE, &tm_q, h * AD, b * p.L + (q0 + t) * AT, q_full);
        tma_load_2d(sQ + t * ATILE + ATILE / 2, &tm_q, h * AD + 64, b * p.L + (q0 + t) * AT, q_full);
      }
      bool ok = true;
      int i = 0;
      for (; i < 2 * n && ok; ++i) {
        const int s = i % KV_RING;
        ok = mbar_wait(&empty[s], ((i / KV_RING) & 1) ^ 1, p.status);
        if (!ok) break;
        const bool is_v = i == 2 * n - 1 || (i > 0 && (i & 1) == 0);
        const int j = i == 2 * n - 1 ? n - 1 : is_v ? i / 2 - 1 : (i + 1) / 2;
        const CUtensorMap* tm = is_v ? &tm_v : &tm_k;
        uint8_t* dst = sKV + s * ATILE;
        mbar_expect_tx(&full[s], ATILE);
        tma_load_2d(dst, tm, hk * AD, b * p.L + j * AT, &full[s]);
        tma_load_2d(dst + ATILE / 2, tm, hk * AD + 64, b * p.L + j * AT, &full[s]);
      }
      if (!ok) {                                       // copies still in flight land before the CTA goes
        mbar_wait(q_full, 0, nullptr);
        for (int k = i > KV_RING ? i - KV_RING : 0; k < i; ++k) mbar_wait(&full[k % KV_RING], (k / KV_RING) & 1, nullptr);
      }
    }
    __syncwarp();
  } else if (warp == 8) {
    if (lane == 0) {
      const uint32_t id_s = make_idesc_bf16(128, 128, 0, 0), id_o = make_idesc_bf16(128, 128, 0, 1);
      auto scores = [&](int t, int slot) {             // S_t = Q_t K^T
        const uint32_t aq = smem_u32(sQ + t * ATILE), ak = smem_u32(sKV + slot * ATILE);
        #pragma unroll
        for (int kk = 0; kk < 8; ++kk) umma_bf16(tmem + t * 128, adesc_k(aq, kk), adesc_k(ak, kk), id_s, kk != 0);
        umma_commit(&s_full[t]);
      };
      bool ok = mbar_wait(q_full, 0, p.status) && mbar_wait(&full[0], 0, p.status);
      if (ok) {
        tc_fence_after_sync();
        scores(0, 0);
        if (n1 > 0) scores(1, 0);
        umma_commit(&empty[0]);
      }
      int used = 1;                                    // ring entries handed out so far
      for (int j = 0; j < n && ok; ++j) {
        const bool more = j + 1 < n;
        const int ik = used, iv = used + (more ? 1 : 0);
        used = iv + 1;
        const int sk = ik % KV_RING, sv = iv % KV_RING;
        bool k_here = false, v_here = false;
        #pragma unroll 1
        for (int t = 0; t < 2 && ok; ++t) {
          const int nt = t == 0 ? n0 : n1;
          if (j >= nt) continue;
          ok = mbar_wait(&p_ready[t], j & 1, p.status);
          if (ok && j + 1 < nt) {
            if (!k_here) { ok = mbar_wait(&full[sk], (ik / KV_RING) & 1, p.status); k_here = true; }
            tc_fence_after_sync();
            if (ok) scores(t, sk);
            if (ok && (t == 1 || n1 <= j + 1)) umma_commit(&empty[sk]);     // K(j+1) has no further reader
          }
          if (ok && !v_here) { ok = mbar_wait(&full[sv], (iv / KV_RING) & 1, p.status); v_here = true; }
          if (ok) {
            tc_fence_after_sync();
            const uint32_t ap = smem_u32(sP + t * ATILE), av = smem_u32(sKV + sv * ATILE);
            #pragma unroll
            for (int kk = 0; kk < 8; ++kk)
              umma_bf16(tmem + 256 + t * 128, adesc_k(ap, kk), adesc_mn(av, kk), id_o, (j | kk) != 0);
            umma_commit(&o_done[t]);
          }
        }
        if (ok) umma_commit(&empty[sv]);
      }
    }
    __syncwarp();
  } else {
    const int t = warp >> 2, row = tid & 127, nt = t == 0 ? n0 : n1;
    const uint32_t lanes = (uint32_t)(warp & 3) * 32;
    uint8_t* tile = sP + t * ATILE;
    const float c = p.scale * LOG2E;
    float m_run = 0.f, l_run = 0.f;
    bool ok = true;
    for (int j = 0; j < nt && ok; ++j) {
      ok = __all_sync(0xffffffffu, mbar_wait(&s_full[t], j & 1, p.status));
      if (!ok) break;
      tc_fence_after_sync();
      uint32_t v[4][32];
      #pragma unroll
      for (int i = 0; i < 4; ++i) tmem_ld32(tmem_addr(tmem, lanes, t * 128 + i * 32), v[i]);
      tmem_ld_wait();
      if (j == nt - 1) {                               // diagonal tile
        #pragma unroll
        for (int i = 0; i < 4; ++i)
          #pragma unroll
          for (int e = 0; e < 32; ++e)
            if (i * 32 + e > row) v[i][e] = 0xff800000u;          // -inf
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      #pragma unroll
      for (int e = 0; e < 32; ++e) {
        #pragma unroll
        for (int i = 0; i < 4; ++i) mx[i] = fmaxf(mx[i], __uint_as_float(v[i][e]));
      }
      const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      float alpha = 1.f;
      bool grow = false;
      if (j == 0) m_run = top;
      else if (top > m_run) {
        grow = true;
        alpha = exp2f((m_run - top) * c);
        m_run = top;
      }
      const float off = m_run * c;
      const uint64_t c2 = pack2(c, c), off2 = pack2(-off, -off);
      uint64_t sum2[4] = {0, 0, 0, 0};
      uint32_t pk[64];
      #pragma unroll
      for (int i = 0; i < 4; ++i) {
        #pragma unroll
        for (int e = 0; e < 32; e += 2) {
          float a0, a1;
          unpack2(fma2(pack2(__uint_as_float(v[i][e]), __uint_as_float(v[i][e + 1])), c2, off2), a0, a1);
          a0 = exp2f(a0); a1 = exp2f(a1);
          sum2[i] = add2(sum2[i], pack2(a0, a1));
          pk[i * 16 + e / 2] = pack_bf16(a0, a1);
        }
      }
      float sum[4];
      #pragma unroll
      for (int i = 0; i < 4; ++i) {
        float a0, a1;
        unpack2(sum2[i], a0, a1);
        sum[i] = a0 + a1;
      }
      l_run = l_run * alpha + ((sum[0] + sum[1]) + (sum[2] + sum[3]));
      if (j > 0) {                                     // P and O are in use until the previous product is complete
        ok = __all_sync(0xffffffffu, mbar_wait(&o_done[t], (j - 1) & 1, p.status));
        if (!ok) break;
        tc_fence_after_sync();
        if (__any_sync(0xffffffffu, grow)) {
          const uint64_t al2 = pack2(alpha, alpha);
          #pragma unroll 1
          for (int i = 0; i < 2; ++i) {
            uint32_t o[2][32];
            tmem_ld32(tmem_addr(tmem, lanes, 256 + t * 128 + i * 64), o[0]);
            tmem_ld32(tmem_addr(tmem, lanes, 256 + t * 128 + i * 64 + 32), o[1]);
            tmem_ld_wait();
            #pragma unroll
            for (int k = 0; k < 2; ++k)
              #pragma unroll
              for (int e = 0; e < 32; e += 2) {
                float a0, a1;
                unpack2(mul2(pack2(__uint_as_float(o[k][e]), __uint_as_float(o[k][e + 1])), al2), a0, a1);
                o[k][e] = __float_as_uint(a0); o[k][e + 1] = __float_as_uint(a1);
              }
            tmem_st32(tmem_addr(tmem, lanes, 256 + t * 128 + i * 64), o[0]);
            tmem_st32(tmem_addr(tmem, lanes, 256 + t * 128 + i * 64 + 32), o[1]);
          }
          tmem_st_wait();
        }
      }
      #pragma unroll
      for (int q = 0; q < 16; ++q)
        *reinterpret_cast<uint4*>(tile + (q >> 3) * (ATILE / 2) + sw128_offset(row, q & 7)) =
            make_uint4(pk[q * 4], pk[q * 4 + 1], pk[q * 4 + 2], pk[q * 4 + 3]);
      fence_proxy_async_smem();
      tc_fence_before_sync();
      mbar_arrive(&p_ready[t]);
    }
    if (nt > 0) {
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&o_done[t], (nt - 1) & 1, p.status));
      if (ok) {
        tc_fence_after_sync();
        const float inv = 1.f / l_run;
        #pragma unroll 1
        for (int i = 0; i < 4; ++i) {
          uint32_t o[32];
          tmem_ld32(tmem_addr(tmem, lanes, 256 + t * 128 + i * 32), o);
          tmem_ld_wait();
          #pragma unroll
          for (int q = 0; q < 4; ++q) {
            float f[8];
            #pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(o[q * 8 + e]) * inv;
            tile_store8(tile, row, i * 32 + q * 8, f);
          }
        }
        p.lse[((long long)b * p.Hq + h) * p.L + (q0 + t) * AT + row] = m_run * p.scale + logf(l_run);
        fence_proxy_async_smem();
      }
      asm volatile("bar.sync %0, 128;" ::"r"(1 + t) : "memory");
      if (row == 0 && ok) {
        tma_store_2d(&tm_o, tile, h * AD, b * p.L + (q0 + t) * AT);
        tma_store_2d(&tm_o, tile + ATILE / 2, h * AD + 64, b * p.L + (q0 + t) * AT);
        tma_store_commit();
        tma_store_wait_all();
      }
      tc_fence_before_sync();
    }
  }
  __syncthreads();
  if (warp == 8) tmem_dealloc(tmem, 512);
}

// ---------------------------------------------------------------------------------------------------
// Backward: one CTA per (128-key tile, kv head, batch) walks its group's query heads and their 64-query tiles at or below
// the diagonal.  Everything is transposed, TMEM lane = key (or channel for dQ): S^T = K Q^T and dP^T = V dO^T take 64
// columns each, twice, next to dV and dK (128 each): two tiles are under way, and the arithmetic of one runs under the
// products of the other.
//   warps 0-15   P and dS of a tile (row = key, 16 queries per warpgroup), back into the S^T columns they came from: P^T and
//                dS^T are the A operands of dV and dK there.  dS^T also goes to shared memory, as B operand of dQ^T
//   warps 16-19  read dQ^T back (it stands where dP^T was) and add it to fp32 dQ with one bulk reduction per tile
//   warp 20      issues all products, of whichever tile has its operands;  warp 21  loads, three tiles of Q and dO deep
// Bound by shared memory (288 KB per 64 x 128 tile, 2250 of about 2870 clocks: K and V as A operands 96, Q and dO as B 64, dS
// and dQ the rest).  us of the whole backward pass, 8192 queries of 32 heads / 4096 x 32: one 128-thread group doing everything
// in turn 3390 / 1046; these warps with one tile of scores 2362 / 651, two 1987 / 571, P and dS in TMEM 1913 / 563, and a third
// stage of Q and dO in the room they left 1701 / 561.  (dQ by a reduction per value instead of the staged bulk ones: +5 %.)
struct AttnBwdParams {
  const float* lse; const float* delta;     // [B, Hq, L]
  __nv_bfloat16* dk; __nv_bfloat16* dv;     // [B*L, Hkv*128]
  int L, Hq, Hkv;
  float scale;
  int* status;
};
constexpr int AQ = 64;                               // queries of a tile
constexpr int QTILE = AQ * AD * 2;                   // [64][128] bf16: two 8 KiB swizzle blocks
constexpr int PTILE = AT * AQ * 2;                   // [128 keys][64 queries] bf16
constexpr int BWD_STAGE = 2 * QTILE;                 // Q and dO
constexpr int BWD_RING = 3;
constexpr int ATTN_BWD_THREADS = 22 * 32;
constexpr int ATTN_BWD_SMEM = 2 * ATILE + BWD_RING * BWD_STAGE + 2 * PTILE + AQ * AD * 4 + BWD_RING * 2 * AQ * 4 + 256 + 1024;

__global__ void __launch_bounds__(ATTN_BWD_THREADS, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                const __grid_constant__ CUtensorMap tm_dq, const AttnBwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;
  uint8_t* sV = sK + ATILE;
  uint8_t* sStage = sV + ATILE;                        // [3] Q | dO
  uint8_t* sDS = sStage + BWD_RING * BWD_STAGE;        // [2] dS^T
  float* sdQ = reinterpret_cast<float*>(sDS + 2 * PTILE);              // [64 queries][128 channels]
  float* sStat = sdQ + AQ * AD;                        // [3] lse[64] | delta[64]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sStat + BWD_RING * 2 * AQ);
  uint64_t *kv_full = bars, *full = bars + 1, *empty = full + BWD_RING, *s_full = empty + BWD_RING, *ds_ready = s_full + 2,
           *dq_full = ds_ready + 2, *dq_free = dq_full + 2, *done = dq_free + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  const int hk = blockIdx.x % p.Hkv, b = blockIdx.x / p.Hkv, kt = blockIdx.y;      // longest walks first
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ratio = p.Hq / p.Hkv, per_head = p.L / AQ - 2 * kt, n = ratio * per_head;
  const int krow0 = b * p.L + kt * AT;

  if (tid == 0) {
    mbar_init(kv_full, 1);
    for (int k = 0; k < BWD_RING; ++k) { mbar_init(&full[k], 1); mbar_init(&empty[k], 1); }
    for (int k = 0; k < 2; ++k) {
      mbar_init(&s_full[k], 1); mbar_init(&ds_ready[k], 16);
      mbar_init(&dq_full[k], 1); mbar_init(&dq_free[k], 4);
    }
    mbar_init(done, 1);
    mbar_fence_init();
    tma_prefetch_desc(&tm_q); tma_prefetch_desc(&tm_k); tma_prefetch_desc(&tm_v); tma_prefetch_desc(&tm_do);
    tma_prefetch_desc(&tm_dq);
  }
  if (warp == 20) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;                    // stage s: S^T (then dQ^T) 128 s, dP^T 128 s + 64; dV 256, dK 384

  if (warp == 21) {
    if (lane == 0) {
      mbar_expect_tx(kv_full, 2 * ATILE);
      tma_load_2d(sK, &tm_k, hk * AD, krow0, kv_full);
      tma_load_2d(sK + ATILE / 2, &tm_k, hk * AD + 64, krow0, kv_full);
      tma_load_2d(sV, &tm_v, hk * AD, krow0, kv_full);
      tma_load_2d(sV + ATILE / 2, &tm_v, hk * AD + 64, krow0, kv_full);
      bool ok = true;
      int it = 0;
      for (; it < n; ++it) {
        const int st = it % BWD_RING, h = hk * ratio + it / per_head, q = (2 * kt + it % per_head) * AQ;
        ok = mbar_wait(&empty[st], ((it / BWD_RING) & 1) ^ 1, p.status);
        if (!ok) break;
        uint8_t* sq = sStage + st * BWD_STAGE;
        mbar_expect_tx(&full[st], BWD_STAGE + 2 * AQ * 4);
        tma_load_2d(sq, &tm_q, h * AD, b * p.L + q, &full[st]);
        tma_load_2d(sq + QTILE / 2, &tm_q, h * AD + 64, b * p.L + q, &full[st]);
        tma_load_2d(sq + QTILE, &tm_do, h * AD, b * p.L + q, &full[st]);
        tma_load_2d(sq + QTILE + QTILE / 2, &tm_do, h * AD + 64, b * p.L + q, &full[st]);
        const long long so = ((long long)b * p.Hq + h) * p.L + q;
        bulk_load(sStat + st * 2 * AQ, p.lse + so, AQ * 4, &full[st]);
        bulk_load(sStat + st * 2 * AQ + AQ, p.delta + so, AQ * 4, &full[st]);
      }
      if (!ok) {                                       // copies still in flight land before the CTA goes
        mbar_wait(kv_full, 0, nullptr);
        for (int k = it > BWD_RING ? it - BWD_RING : 0; k < it; ++k) mbar_wait(&full[k % BWD_RING], (k / BWD_RING) & 1, nullptr);
      }
    }
    __syncwarp();
  } else if (warp == 20) {
    if (lane == 0) {
      const uint32_t aK = smem_u32(sK), aV = smem_u32(sV);
      const uint32_t id_s = make_idesc_bf16(128, AQ, 0, 0), id_g = make_idesc_bf16(128, AD, 0, 1),
                     id_q = make_idesc_bf16(128, AQ, 1, 1);
      // descriptors of whole tiles; a k-step adds to the address field (16-byte units): 32 bytes inside an atom of 64 and
      // then the next atom (of 128 or of 64 rows), or 16 rows
      auto kstep = [](int kk) { return (uint64_t)((kk >> 2) * (ATILE / 2 / 16) + (kk & 3) * 2); };
      auto qstep = [](int kk) { return (uint64_t)((kk >> 2) * (QTILE / 2 / 16) + (kk & 3) * 2); };
      auto mstep = [](int kk) { return (uint64_t)(kk * 128); };
      const uint64_t dKk = adesc_k(aK, 0), dVk = adesc_k(aV, 0), dKm = adesc_mn(aK, 0);
      auto scores = [&](int it) {
        const uint32_t aQ = smem_u32(sStage + it % BWD_RING * BWD_STAGE), to = tmem + (it & 1) * 128;
        const uint64_t dQk = make_smem_desc_sw128(aQ, 16, 1024), dOk = make_smem_desc_sw128(aQ + QTILE, 16, 1024);
        #pragma unroll
        for (int kk = 0; kk < 8; ++kk) umma_bf16(to, dKk + kstep(kk), dQk + qstep(kk), id_s, kk != 0);
        #pragma unroll
        for (int kk = 0; kk < 8; ++kk) umma_bf16(to + 64, dVk + kstep(kk), dOk + qstep(kk), id_s, kk != 0);
        umma_commit(&s_full[it & 1]);
      };
      auto gradients = [&](int it) {
        const uint32_t aQ = smem_u32(sStage + it % BWD_RING * BWD_STAGE);
        const uint64_t dQm = make_smem_desc_sw128(aQ, QTILE / 2, 1024), dOm = make_smem_desc_sw128(aQ + QTILE, QTILE / 2, 1024);
        const uint64_t dDS = make_smem_desc_sw128(smem_u32(sDS + (it & 1) * PTILE), 16, 1024);
        const uint32_t ts = tmem + (it & 1) * 128;
        // k-step kk of P^T and dS^T is what warpgroup kk left in its own columns of S^T
        #pragma unroll
        for (int kk = 0; kk < 4; ++kk)      // dV[key][d] += sum_i P^T[key][i] dO[i][d]
          umma_bf16_ta(tmem + 256, ts + kk * 16, dOm + mstep(kk), id_g, (it | kk) != 0);
        #pragma unroll
        for (int kk = 0; kk < 4; ++kk)      // dK[key][d] += sum_i dS^T[key][i] Q[i][d]
          umma_bf16_ta(tmem + 384, ts + kk * 16 + 8, dQm + mstep(kk), id_g, (it | kk) != 0);
        #pragma unroll
        for (int kk = 0; kk < 8; ++kk)      // dQ^T[d][i] = sum_key K[key][d] dS^T[key][i], where dP^T of this tile was
          umma_bf16(ts + 64, dKm + mstep(kk), dDS + mstep(kk), id_q, kk != 0);
        umma_commit(&dq_full[it & 1]);      // also behind the readers of P^T and dS^T: their columns take the scores of it + 2
        umma_commit(&empty[it % BWD_RING]);
      };
      // Whatever is ready goes next: the scores of tile s (its operands have landed, its TMEM stage has been read for the last
      // time) or the gradients of tile g (P and dS are in shared memory).  The other of two stages stands for work meanwhile.
      bool ok = mbar_wait(kv_full, 0, p.status);
      uint64_t last = 0;
      int s = 0, g = 0;
      for (uint32_t idle = 1; g < n && ok; ++idle) {
        bool moved = false;
        if (s < n && s < g + 2 && mbar_test(&full[s % BWD_RING], (s / BWD_RING) & 1) && (s < 2 || mbar_test(&dq_free[s & 1], ((s >> 1) - 1) & 1))) {
          tc_fence_after_sync();
          scores(s++);
          moved = true;
        }
        if (g < s && mbar_test(&ds_ready[g & 1], (g >> 1) & 1)) {
          tc_fence_after_sync();
          gradients(g++);
          moved = true;
        }
        if (moved) {
          idle = 0;
        } else if ((idle & 1023u) == 0u) {             // bounded, as every wait here
          if (p.status != nullptr && *((volatile int*)p.status) != 0) ok = false;
          const uint64_t now = global_timer_ns();
          if (idle == 1024u) last = now;
          else if (now - last > SSM_WAIT_NS) { if (p.status != nullptr) atomicCAS(p.status, 0, SSM_ERR_TIMEOUT_MBAR); ok = false; }
        }
      }
      if (ok) umma_commit(done);
    }
    __syncwarp();
  } else if (warp >= 16) {
    // ---- dQ^T: thread = channel; [query][channel] rows in shared memory, one bulk reduction per tile
    const int d = tid - 512;
    bool ok = true;
    for (int it = 0; it < n && ok; ++it) {
      const int h = hk * ratio + it / per_head, q = (2 * kt + it % per_head) * AQ;
      ok = __all_sync(0xffffffffu, mbar_wait(&dq_full[it & 1], (it >> 1) & 1, p.status));
      tc_fence_after_sync();
      uint32_t v[2][32];
      if (ok) {
        tmem_ld32(tmem_addr(tmem, (warp & 3) * 32, (it & 1) * 128 + 64), v[0]);
        tmem_ld32(tmem_addr(tmem, (warp & 3) * 32, (it & 1) * 128 + 96), v[1]);
        tmem_ld_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&dq_free[it & 1]);  // the stage takes the scores of tile it + 2
      }
      if (d == 0) tma_store_wait_read();               // the previous tile has left the staging rows
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (ok) {
        #pragma unroll
        for (int i = 0; i < 2; ++i)
          #pragma unroll
          for (int e = 0; e < 32; ++e) sdQ[(i * 32 + e) * AD + d] = __uint_as_float(v[i][e]);
      }
      fence_proxy_async_smem();
      ok = barrier_and<1, 128>(ok);                    // the four warps meet at barriers: they leave together
      if (d == 0 && ok) {
        tma_add_2d(&tm_dq, sdQ, h * AD, b * p.L + q);
        tma_store_commit();
      }
    }
    if (d == 0) tma_store_wait_all();
  } else {
    // ---- P^T and dS^T: row = key
    const int row = tid & 127, wg = tid >> 7;
    const uint32_t lanes = (uint32_t)(warp & 3) * 32;
    const float c = p.scale * LOG2E;
    bool ok = true;
    for (int it = 0; it < n && ok; ++it) {
      const int st = it & 1, ring = it % BWD_RING, rel = (it % per_head) * AQ;      // first query relative to the key tile's first key
      // the loads of this stage (statistics included) complete on `full`, long before the scores; this thread observes the
      // phase before it reads what they wrote.  The scores are complete behind the gradients of tile it - 2, which were issued
      // in front of them: P, dS and the statistics of that tile have been read.
      ok = mbar_wait(&full[ring], (it / BWD_RING) & 1, p.status);
      ok = __all_sync(0xffffffffu, ok && mbar_wait(&s_full[st], (it >> 1) & 1, p.status));
      if (!ok) break;
      tc_fence_after_sync();
      uint32_t sv[16], dp[16];
      tmem_ld16(tmem_addr(tmem, lanes, st * 128 + wg * 16), sv);
      tmem_ld16(tmem_addr(tmem, lanes, st * 128 + 64 + wg * 16), dp);
      tmem_ld_wait();
      const float* lse = sStat + ring * 2 * AQ + wg * 16;
      const float* delta = lse + AQ;
      uint32_t pk[8], dk[8];
      #pragma unroll
      for (int e4 = 0; e4 < 4; ++e4) {
        const float4 ls = *reinterpret_cast<const float4*>(lse + e4 * 4), de = *reinterpret_cast<const float4*>(delta + e4 * 4);
        const uint64_t lv[2] = {pack2(ls.x, ls.y), pack2(ls.z, ls.w)}, dv[2] = {pack2(de.x, de.y), pack2(de.z, de.w)};
        float pv[4], ds[4];
        #pragma unroll
        for (int e = 0; e < 4; e += 2) {
          const int i = e4 * 4 + e;
          unpack2(fma2(pack2(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1])), pack2(c, c), mul2(lv[e / 2], pack2(-LOG2E, -LOG2E))),
                  pv[e], pv[e + 1]);
          pv[e] = exp2f(pv[e]); pv[e + 1] = exp2f(pv[e + 1]);
          if (rel < AT) {                                      // a tile on the diagonal: queries before the key
            pv[e] = rel + wg * 16 + i < row ? 0.f : pv[e];
            pv[e + 1] = rel + wg * 16 + i + 1 < row ? 0.f : pv[e + 1];
          }
          const uint64_t g = fma2(dv[e / 2], pack2(-1.f, -1.f), pack2(__uint_as_float(dp[i]), __uint_as_float(dp[i + 1])));
          unpack2(mul2(mul2(pack2(pv[e], pv[e + 1]), g), pack2(p.scale, p.scale)), ds[e], ds[e + 1]);
        }
        pk[e4 * 2] = pack_bf16(pv[0], pv[1]); pk[e4 * 2 + 1] = pack_bf16(pv[2], pv[3]);
        dk[e4 * 2] = pack_bf16(ds[0], ds[1]); dk[e4 * 2 + 1] = pack_bf16(ds[2], ds[3]);
      }
      tmem_st8(tmem_addr(tmem, lanes, st * 128 + wg * 16), pk);
      tmem_st8(tmem_addr(tmem, lanes, st * 128 + wg * 16 + 8), dk);
      uint8_t* sp = sDS + st * PTILE;
      #pragma unroll
      for (int q = 0; q < 2; ++q)
        *reinterpret_cast<uint4*>(sp + sw128_offset(row, wg * 2 + q)) = make_uint4(dk[q * 4], dk[q * 4 + 1], dk[q * 4 + 2], dk[q * 4 + 3]);
      tmem_st_wait();
      fence_proxy_async_smem();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ds_ready[st]);
    }
    if (ok) ok = __all_sync(0xffffffffu, mbar_wait(done, 0, p.status));
    if (ok) {
      tc_fence_after_sync();
      __nv_bfloat16* dst = (wg < 2 ? p.dv : p.dk) + (long long)(krow0 + row) * (p.Hkv * AD) + hk * AD + (wg & 1) * 64;
      #pragma unroll 1
      for (int db = 0; db < 2; ++db) {
        uint32_t v[32];
        tmem_ld32(tmem_addr(tmem, lanes, 256 + wg * 64 + db * 32), v);
        tmem_ld_wait();
        #pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
          float f[8];
          #pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(v[ch * 8 + e]);
          *reinterpret_cast<uint4*>(dst + db * 32 + ch * 8) = apack8(f);
        }
      }
    }
    tc_fence_before_sync();
  }
  __syncthreads();
  if (warp == 20) tmem_dealloc(tmem, 512);
}

// delta[b, h, t] = sum_d dout * out of a row; one warp per (row, head), bound by reading both once
__global__ void __launch_bounds__(256)
attn_delta_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ out, float* __restrict__ delta,
                  long long pairs, int L, int Hq) {
  const long long i = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);        // (row, head)
  if (i >= pairs) return;
  const int lane = threadIdx.x & 31;
  const uint2 a = *reinterpret_cast<const uint2*>(dout + i * AD + lane * 4), o = *reinterpret_cast<const uint2*>(out + i * AD + lane * 4);
  float s = bf16_lo(a.x) * bf16_lo(o.x) + bf16_hi(a.x) * bf16_hi(o.x) + bf16_lo(a.y) * bf16_lo(o.y) + bf16_hi(a.y) * bf16_hi(o.y);
  #pragma unroll
  for (int k = 16; k > 0; k >>= 1) s += __shfl_xor_sync(0xffffffffu, s, k);
  const long long row = i / Hq;
  const int h = (int)(i - row * Hq);
  const long long b = row / L;
  if (lane == 0) delta[(b * Hq + h) * L + (row - b * L)] = s;
}

}  // namespace ssm

using namespace ssm;

static int attn_maps(CUtensorMap* tq, CUtensorMap* tk, CUtensorMap* tv, CUtensorMap* tx, const void* q, const void* k,
                     const void* v, const void* x, int B, int L, int Hq, int Hkv, int q_rows) {
  int r = make_tmap_2d_bf16(tq, q, (uint64_t)Hq * AD, (uint64_t)B * L, (uint64_t)Hq * AD * 2, 64, q_rows);
  if (r) return -100 - r;
  r = make_tmap_2d_bf16(tk, k, (uint64_t)Hkv * AD, (uint64_t)B * L, (uint64_t)Hkv * AD * 2, 64, 128);
  if (r) return -200 - r;
  r = make_tmap_2d_bf16(tv, v, (uint64_t)Hkv * AD, (uint64_t)B * L, (uint64_t)Hkv * AD * 2, 64, 128);
  if (r) return -300 - r;
  r = make_tmap_2d_bf16(tx, x, (uint64_t)Hq * AD, (uint64_t)B * L, (uint64_t)Hq * AD * 2, 64, q_rows);
  if (r) return -400 - r;
  return 0;
}

extern "C" int ssm_attn_fwd(const void* q, const void* k, const void* v, void* out, void* lse, int B, int L, int Hq,
                            int Hkv, int D, float scale, int* status, cudaStream_t st) {
  if (D != AD || L % AT || Hq % Hkv) return -SSM_ERR_BAD_ARG;
  const int smem = ATTN_FWD_SMEM;
  static SmemOptIn opt_in;
  if (const int e = opt_in.ask(reinterpret_cast<const void*>(attn_fwd_kernel), smem)) return e;
  CUtensorMap tq, tk, tv, to;
  int r = attn_maps(&tq, &tk, &tv, &to, q, k, v, out, B, L, Hq, Hkv, AT);
  if (r) return r;
  AttnFwdParams p;
  p.lse = reinterpret_cast<float*>(lse); p.L = L; p.Hq = Hq; p.Hkv = Hkv; p.scale = scale; p.status = status;
  dim3 grid((L / AT + 1) / 2, Hq, B);
  attn_fwd_kernel<<<grid, ATTN_FWD_THREADS, smem, st>>>(tq, tk, tv, to, p);
  return (int)cudaGetLastError();
}

extern "C" int ssm_attn_delta(const void* dout, const void* out, void* delta, int B, int L, int Hq, int D, cudaStream_t st) {
  if (D != AD || B < 1 || L < 1 || Hq < 1 || ((reinterpret_cast<uintptr_t>(dout) | reinterpret_cast<uintptr_t>(out)) & 7)) return -SSM_ERR_BAD_ARG;
  const long long pairs = (long long)B * L * Hq;
  attn_delta_kernel<<<(unsigned)((pairs + 7) / 8), 256, 0, st>>>(reinterpret_cast<const __nv_bfloat16*>(dout),
                                                                reinterpret_cast<const __nv_bfloat16*>(out),
                                                                reinterpret_cast<float*>(delta), pairs, L, Hq);
  return (int)cudaGetLastError();
}

// dq32: fp32 [B*L, Hq*128], zero on entry; lse / delta: fp32 [B, Hq, L], 16-byte aligned
extern "C" int ssm_attn_bwd(const void* q, const void* k, const void* v, const void* dout, const void* lse,
                            const void* delta, void* dq32, void* dk, void* dv, int B, int L, int Hq, int Hkv, int D,
                            float scale, int* status, cudaStream_t st) {
  if (D != AD || L % AT || Hq % Hkv || L / AT > 65535 ||
      ((reinterpret_cast<uintptr_t>(lse) | reinterpret_cast<uintptr_t>(delta) | reinterpret_cast<uintptr_t>(dq32)) & 15))
    return -SSM_ERR_BAD_ARG;
  static SmemOptIn opt_in;
  if (const int e = opt_in.ask(reinterpret_cast<const void*>(attn_bwd_kernel), ATTN_BWD_SMEM)) return e;
  CUtensorMap tq, tk, tv, tdo, tdq;
  int r = attn_maps(&tq, &tk, &tv, &tdo, q, k, v, dout, B, L, Hq, Hkv, AQ);
  if (r) return r;
  r = make_tmap_2d(&tdq, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, dq32, (uint64_t)Hq * AD, (uint64_t)B * L, (uint64_t)Hq * AD * 4, AD,
                   AQ, CU_TENSOR_MAP_SWIZZLE_NONE);
  if (r) return -500 - r;
  AttnBwdParams p;
  p.lse = reinterpret_cast<const float*>(lse); p.delta = reinterpret_cast<const float*>(delta);
  p.dk = reinterpret_cast<__nv_bfloat16*>(dk); p.dv = reinterpret_cast<__nv_bfloat16*>(dv);
  p.L = L; p.Hq = Hq; p.Hkv = Hkv; p.scale = scale; p.status = status;
  attn_bwd_kernel<<<dim3(Hkv * B, L / AT), ATTN_BWD_THREADS, ATTN_BWD_SMEM, st>>>(tq, tk, tv, tdo, tdq, p);
  return (int)cudaGetLastError();
}
