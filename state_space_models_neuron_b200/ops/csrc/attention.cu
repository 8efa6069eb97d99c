// Causal grouped-query flash attention for sm_100a, head_dim 128, forward and backward, on tcgen05.
//   forward  : one CTA per (128-query tile, query head, batch); K/V tiles of 128 keys arrive by TMA (double
//              buffered); S = Q K^T and P V run on tcgen05 with TMEM accumulators; thread i owns query row i, so
//              the online softmax needs no cross-thread reductions; O stays in registers until the end.
//   backward : one CTA per (128-key tile, kv head, batch) walks the query heads of its group and the query tiles
//              at or below the diagonal; dK and dV accumulate in TMEM over the whole walk (deterministic), dQ is
//              added to an fp32 buffer with red.add.
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
// the other's products.  S and O of both tiles fill the 512 TMEM columns.  O is rescaled in TMEM only when a row's maximum
// has grown by more than 2^8 since its last rescaling (the sums use the same stale maximum, so the quotient is exact);
// P <= 2^8 keeps its relative precision in bf16.
// Bound by the exponentials (16 per clock and SM: as long as the products of a tile) and the softmax arithmetic around them.
// One 128-thread group doing everything in turn took 1541 us for 8192 queries of 32 heads, this 695 us (8192 x 16: 870 -> 424, 4096 x 32: 467 -> 248).
constexpr int ATTN_FWD_THREADS = 320;
constexpr int KV_RING = 3;
constexpr int ATTN_FWD_SMEM = (4 + KV_RING) * ATILE + 256 + 1024;
constexpr float RESCALE_LOG2 = 8.f;

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
      else if ((top - m_run) * c > RESCALE_LOG2) {
        grow = true;
        alpha = exp2f((m_run - top) * c);
        m_run = top;
      }
      const float off = m_run * c;
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t pk[64];
      #pragma unroll
      for (int i = 0; i < 4; ++i) {
        #pragma unroll
        for (int e = 0; e < 32; e += 2) {
          const float a0 = exp2f(fmaf(__uint_as_float(v[i][e]), c, -off));
          const float a1 = exp2f(fmaf(__uint_as_float(v[i][e + 1]), c, -off));
          sum[i] += a0 + a1;
          pk[i * 16 + e / 2] = pack_bf16(a0, a1);
        }
      }
      l_run = l_run * alpha + ((sum[0] + sum[1]) + (sum[2] + sum[3]));
      if (j > 0) {                                     // P and O are in use until the previous product is complete
        ok = __all_sync(0xffffffffu, mbar_wait(&o_done[t], (j - 1) & 1, p.status));
        if (!ok) break;
        tc_fence_after_sync();
        if (__any_sync(0xffffffffu, grow)) {
          #pragma unroll 1
          for (int i = 0; i < 4; ++i) {
            uint32_t o[32];
            tmem_ld32(tmem_addr(tmem, lanes, 256 + t * 128 + i * 32), o);
            tmem_ld_wait();
            #pragma unroll
            for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
            tmem_st32(tmem_addr(tmem, lanes, 256 + t * 128 + i * 32), o);
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
struct AttnBwdParams {
  const float* lse; const float* delta;     // [B, Hq, L]
  float* dq32;                              // [B*L, Hq*128] fp32, zero on entry
  __nv_bfloat16* dk; __nv_bfloat16* dv;     // [B*L, Hkv*128]
  int L, Hq, Hkv;
  float scale;
  int* status;
};

__global__ void __launch_bounds__(128, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                const AttnBwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;
  uint8_t* sV = smem + ATILE;
  uint8_t* sQ = smem + 2 * ATILE;
  uint8_t* sDO = smem + 3 * ATILE;
  uint8_t* sP = smem + 4 * ATILE;
  uint8_t* sDS = smem + 5 * ATILE;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 6 * ATILE);   // [0] kv, [1] q/do, [2] S,dP, [3] dV,dK,dQ
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 4);
  const int kt = blockIdx.x, hk = blockIdx.y, b = blockIdx.z, tid = threadIdx.x, warp = tid >> 5;
  const int ratio = p.Hq / p.Hkv;
  const int qtiles = p.L / AT;
  const int krow0 = b * p.L + kt * AT;

  if (tid == 0) {
    for (int k = 0; k < 4; ++k) mbar_init(&bars[k], 1);
    mbar_fence_init();
    tma_prefetch_desc(&tm_q); tma_prefetch_desc(&tm_k); tma_prefetch_desc(&tm_v); tma_prefetch_desc(&tm_do);
  }
  if (warp == 0) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  const uint32_t aK = smem_u32(sK), aV = smem_u32(sV), aQ = smem_u32(sQ), aDO = smem_u32(sDO), aP = smem_u32(sP),
                 aDS = smem_u32(sDS);
  if (tid == 0) {
    mbar_expect_tx(&bars[0], 2 * ATILE);
    tma_load_2d(sK, &tm_k, hk * AD, krow0, &bars[0]);
    tma_load_2d(sK + ATILE / 2, &tm_k, hk * AD + 64, krow0, &bars[0]);
    tma_load_2d(sV, &tm_v, hk * AD, krow0, &bars[0]);
    tma_load_2d(sV + ATILE / 2, &tm_v, hk * AD + 64, krow0, &bars[0]);
  }
  const float c = p.scale * LOG2E;
  bool ok = true;
  int it = 0;
  for (int hr = 0; hr < ratio && ok; ++hr) {
    const int h = hk * ratio + hr;
    for (int qt = kt; qt < qtiles && ok; ++qt, ++it) {
      const uint32_t par = it & 1;
      const int qrow0 = b * p.L + qt * AT;
      if (tid == 0) {
        mbar_expect_tx(&bars[1], 2 * ATILE);
        tma_load_2d(sQ, &tm_q, h * AD, qrow0, &bars[1]);
        tma_load_2d(sQ + ATILE / 2, &tm_q, h * AD + 64, qrow0, &bars[1]);
        tma_load_2d(sDO, &tm_do, h * AD, qrow0, &bars[1]);
        tma_load_2d(sDO + ATILE / 2, &tm_do, h * AD + 64, qrow0, &bars[1]);
        bool good = (it > 0) || mbar_wait(&bars[0], 0, p.status);
        good = good && mbar_wait(&bars[1], par, p.status);
        if (good) {
          tc_fence_after_sync();
          const uint32_t id = make_idesc_bf16(128, 128, 0, 0);
          #pragma unroll
          for (int kk = 0; kk < 8; ++kk) umma_bf16(tmem, adesc_k(aQ, kk), adesc_k(aK, kk), id, kk != 0);           // S
          #pragma unroll
          for (int kk = 0; kk < 8; ++kk) umma_bf16(tmem + 128, adesc_k(aDO, kk), adesc_k(aV, kk), id, kk != 0);   // dP
          umma_commit(&bars[2]);
        }
      }
      __syncwarp();
      ok = __syncthreads_and(mbar_wait(&bars[2], par, p.status));
      tc_fence_after_sync();
      if (!ok) break;
      const long long so = ((long long)b * p.Hq + h) * p.L + qt * AT + tid;
      const float lse2 = p.lse[so] * LOG2E, dlt = p.delta[so];
      const bool diag = (qt == kt);
      #pragma unroll 1
      for (int jb = 0; jb < 4; ++jb) {
        uint32_t sv[32], dp[32];
        tmem_ld32(tmem_addr(tmem, warp * 32, jb * 32), sv);
        tmem_ld32(tmem_addr(tmem, warp * 32, 128 + jb * 32), dp);
        tmem_ld_wait();
        #pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
          float pf[8], df[8];
          #pragma unroll
          for (int e = 0; e < 8; ++e) {
            const int col = jb * 32 + ch * 8 + e;
            const float pv = (!diag || col <= tid) ? exp2f(__uint_as_float(sv[ch * 8 + e]) * c - lse2) : 0.f;
            pf[e] = pv;
            df[e] = pv * (__uint_as_float(dp[ch * 8 + e]) - dlt) * p.scale;
          }
          tile_store8(sP, tid, jb * 32 + ch * 8, pf);
          tile_store8(sDS, tid, jb * 32 + ch * 8, df);
        }
      }
      fence_proxy_async_smem();
      tc_fence_before_sync();
      __syncthreads();
      if (tid == 0) {
        tc_fence_after_sync();
        const uint32_t id_t = make_idesc_bf16(128, 128, 1, 1);
        #pragma unroll
        for (int kk = 0; kk < 8; ++kk)      // dV[key][d] += sum_i P[i][key] dO[i][d]
          umma_bf16(tmem + 256, adesc_mn(aP, kk), adesc_mn(aDO, kk), id_t, (it | kk) != 0);
        #pragma unroll
        for (int kk = 0; kk < 8; ++kk)      // dK[key][d] += sum_i dS[i][key] Q[i][d]
          umma_bf16(tmem + 384, adesc_mn(aDS, kk), adesc_mn(aQ, kk), id_t, (it | kk) != 0);
        const uint32_t id_q = make_idesc_bf16(128, 128, 0, 1);
        #pragma unroll
        for (int kk = 0; kk < 8; ++kk)      // dQ[i][d] = sum_key dS[i][key] K[key][d]
          umma_bf16(tmem, adesc_k(aDS, kk), adesc_mn(aK, kk), id_q, kk != 0);
        umma_commit(&bars[3]);
      }
      __syncwarp();
      ok = __syncthreads_and(mbar_wait(&bars[3], par, p.status));
      tc_fence_after_sync();
      if (!ok) break;
      float* dq = p.dq32 + (long long)(qrow0 + tid) * (p.Hq * AD) + h * AD;
      #pragma unroll 1
      for (int db = 0; db < 4; ++db) {
        uint32_t v[32];
        tmem_ld32(tmem_addr(tmem, warp * 32, db * 32), v);
        tmem_ld_wait();
        #pragma unroll
        for (int k4 = 0; k4 < 8; ++k4)
          asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dq + db * 32 + k4 * 4),
                       "f"(__uint_as_float(v[k4 * 4])), "f"(__uint_as_float(v[k4 * 4 + 1])),
                       "f"(__uint_as_float(v[k4 * 4 + 2])), "f"(__uint_as_float(v[k4 * 4 + 3])) : "memory");
      }
      tc_fence_before_sync();
      __syncthreads();       // Q, dO, P, dS tiles and TMEM[0,256) are free for the next iteration
    }
  }
  if (ok) {
    tc_fence_after_sync();
    #pragma unroll 1
    for (int which = 0; which < 2; ++which) {
      __nv_bfloat16* dst = (which == 0 ? p.dv : p.dk) + (long long)(krow0 + tid) * (p.Hkv * AD) + hk * AD;
      #pragma unroll 1
      for (int db = 0; db < 4; ++db) {
        uint32_t v[32];
        tmem_ld32(tmem_addr(tmem, warp * 32, 256 + which * 128 + db * 32), v);
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
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

}  // namespace ssm

using namespace ssm;

static int attn_maps(CUtensorMap* tq, CUtensorMap* tk, CUtensorMap* tv, CUtensorMap* tx, const void* q, const void* k,
                     const void* v, const void* x, int B, int L, int Hq, int Hkv) {
  int r = make_tmap_2d_bf16(tq, q, (uint64_t)Hq * AD, (uint64_t)B * L, (uint64_t)Hq * AD * 2, 64, 128);
  if (r) return -100 - r;
  r = make_tmap_2d_bf16(tk, k, (uint64_t)Hkv * AD, (uint64_t)B * L, (uint64_t)Hkv * AD * 2, 64, 128);
  if (r) return -200 - r;
  r = make_tmap_2d_bf16(tv, v, (uint64_t)Hkv * AD, (uint64_t)B * L, (uint64_t)Hkv * AD * 2, 64, 128);
  if (r) return -300 - r;
  r = make_tmap_2d_bf16(tx, x, (uint64_t)Hq * AD, (uint64_t)B * L, (uint64_t)Hq * AD * 2, 64, 128);
  if (r) return -400 - r;
  return 0;
}

extern "C" int ssm_attn_fwd(const void* q, const void* k, const void* v, void* out, void* lse, int B, int L, int Hq,
                            int Hkv, int D, float scale, int* status, cudaStream_t st) {
  if (D != AD || L % AT || Hq % Hkv) return -SSM_ERR_BAD_ARG;
  static bool cfg = false;
  const int smem = ATTN_FWD_SMEM;
  if (!cfg) {
    cudaError_t e = cudaFuncSetAttribute(attn_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    cfg = true;
  }
  CUtensorMap tq, tk, tv, to;
  int r = attn_maps(&tq, &tk, &tv, &to, q, k, v, out, B, L, Hq, Hkv);
  if (r) return r;
  AttnFwdParams p;
  p.lse = reinterpret_cast<float*>(lse); p.L = L; p.Hq = Hq; p.Hkv = Hkv; p.scale = scale; p.status = status;
  dim3 grid((L / AT + 1) / 2, Hq, B);
  attn_fwd_kernel<<<grid, ATTN_FWD_THREADS, smem, st>>>(tq, tk, tv, to, p);
  return (int)cudaGetLastError();
}

extern "C" int ssm_attn_bwd(const void* q, const void* k, const void* v, const void* dout, const void* lse,
                            const void* delta, void* dq32, void* dk, void* dv, int B, int L, int Hq, int Hkv, int D,
                            float scale, int* status, cudaStream_t st) {
  if (D != AD || L % AT || Hq % Hkv) return -SSM_ERR_BAD_ARG;
  static bool cfg = false;
  const int smem = 6 * ATILE + 128 + 1024;
  if (!cfg) {
    cudaError_t e = cudaFuncSetAttribute(attn_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    cfg = true;
  }
  CUtensorMap tq, tk, tv, tdo;
  int r = attn_maps(&tq, &tk, &tv, &tdo, q, k, v, dout, B, L, Hq, Hkv);
  if (r) return r;
  AttnBwdParams p;
  p.lse = reinterpret_cast<const float*>(lse); p.delta = reinterpret_cast<const float*>(delta);
  p.dq32 = reinterpret_cast<float*>(dq32);
  p.dk = reinterpret_cast<__nv_bfloat16*>(dk); p.dv = reinterpret_cast<__nv_bfloat16*>(dv);
  p.L = L; p.Hq = Hq; p.Hkv = Hkv; p.scale = scale; p.status = status;
  dim3 grid(L / AT, Hkv, B);
  attn_bwd_kernel<<<grid, 128, smem, st>>>(tq, tk, tv, tdo, p);
  return (int)cudaGetLastError();
}
