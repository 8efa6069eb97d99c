// SSD (state-space duality) chunked scan for sm_100a, forward and backward, chunk = 128 tokens,
// d_state N = 128, head slices of P = 64 channels (a head of 128 channels is two slices sharing dt/A/D).
//
// Per (batch b, head slice h, chunk c), with l_i = cumsum(A dt) inside the chunk:
//   forward   Y = (CB^T o Lambda o dt_j) X + exp(l_i) C S_in + D x           (Lambda_ij = exp(l_i - l_j), j <= i)
//             S_local = sum_j exp(l_T - l_j) dt_j B_j (x) x_j ;  S_in[c+1] = exp(l_T) S_in[c] + S_local[c]
//   backward  see ssd_chunk_scan_bwd_kernel.
// All 128x128x{64,128} products run on tcgen05 with fp32 accumulators in TMEM; operands come straight from
// TMA (B, C, x, dY, states) or are built by the arithmetic warps in the 128-byte-swizzled layout
// (decay-weighted CB^T, scaled x / dY).  The decay factors are always formed as exp of a difference of
// cumulative sums, never as a ratio of exponentials.
// Reference math: mamba2/mamba2_kernel.py:15-62,138-169 (forward), :358-480 (backward).
#include "common.cuh"
#include "dt_prep.cuh"

namespace ssm {

constexpr int CT = 128;      // chunk length
constexpr int NS = 128;      // d_state
constexpr int PS = 64;       // channels per head slice
constexpr int TILE128 = 128 * 128 * 2;   // bytes of a [128][128] bf16 tile (two 16 KiB swizzle blocks)
constexpr int TILE64 = 128 * 64 * 2;     // bytes of a [128][64] bf16 tile

// descriptor helpers ------------------------------------------------------------------------------
// K-major operand tile [rows][K] made of 64-wide K atoms of [rows][128 B]; k-step kk covers K = 16*kk..
__device__ __forceinline__ uint64_t desc_kmajor(uint32_t base, int kk, uint32_t atom_bytes) {
  return make_smem_desc_sw128(base + (kk >> 2) * atom_bytes + (kk & 3) * 32, 16, 1024);
}
// MN-major operand tile [K rows][MN] made of 64-wide MN blocks of [K rows][128 B] `block_bytes` apart.
__device__ __forceinline__ uint64_t desc_mnmajor(uint32_t base, int kk, uint32_t block_bytes) {
  return make_smem_desc_sw128(base + kk * 2048, block_bytes, 1024);
}

__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 u;
  u.x = pack_bf16(f[0], f[1]); u.y = pack_bf16(f[2], f[3]); u.z = pack_bf16(f[4], f[5]); u.w = pack_bf16(f[6], f[7]);
  return u;
}

__device__ __forceinline__ void load8f_smem(const float* p, float (&f)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}

// block-wide helpers for 128 threads -----------------------------------------------------------------
__device__ __forceinline__ float warp_sum128(float v) {
  #pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// sum over the 128 threads, result to all; red has >= 4 floats; contains two __syncthreads
__device__ __forceinline__ float block_sum128(float v, float* red) {
  v = warp_sum128(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  return red[0] + red[1] + red[2] + red[3];
}

// =====================================================================================
// dt and its running sums (dt_prep.cuh).   grid (nc, heads / 8, B), 128 threads
// =====================================================================================
__global__ void __launch_bounds__(DT_CHUNK) ssd_dt_prep_kernel(const DtPrep p) { dt_prep_block(p, blockIdx.x, blockIdx.y * DT_HEADS, blockIdx.z); }

// =====================================================================================
// chunk states:  S[n][p] = sum_j W[j][n] * s_j * V[j][p]
//   mode 0 (forward):   W = B, V = x,  s_j = exp(l_T - l_j) * dt_j
//   mode 1 (backward):  W = C, V = dY, s_j = exp(l_j)
// grid (nc, Hv, B), 128 threads.  out fp32 [B, Hv, nc, 128, 64].
// =====================================================================================
struct ChunkStateParams {
  const __nv_bfloat16* v; long long v_row_stride;  // V rows: (b*L + t) * v_row_stride + hv*64
  const float* dt; const float* l;                 // [B, H, L]
  float* out;
  int L, H, Hv, G, nc, w_col0, mode;
  int* status;
};

__global__ void __launch_bounds__(128)
ssd_chunk_state_kernel(const __grid_constant__ CUtensorMap tm_w, const ChunkStateParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sW = smem;                      // [128 j][128 n]  (two blocks)
  uint8_t* sV = smem + TILE128;            // [128 j][64 p]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + TILE128 + TILE64);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2);
  const int c = blockIdx.x, hv = blockIdx.y, b = blockIdx.z, tid = threadIdx.x, warp = tid >> 5;
  const int psplit = p.Hv / p.H, h = hv / psplit, g = h / (p.H / p.G);
  const long long row0 = (long long)b * p.L + (long long)c * CT;

  if (tid == 0) { mbar_init(&bars[0], 1); mbar_init(&bars[1], 1); mbar_fence_init(); }
  if (warp == 0) { tmem_alloc(tmem_slot, 64); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;

  if (tid == 0) {
    mbar_expect_tx(&bars[0], TILE128);
    tma_load_2d(sW, &tm_w, p.w_col0 + g * NS, (int)row0, &bars[0]);
    tma_load_2d(sW + TILE128 / 2, &tm_w, p.w_col0 + g * NS + 64, (int)row0, &bars[0]);
  }
  // scaled V row j -> smem (MN-major B operand: rows = j (K), 64 contiguous p)
  {
    const long long lo = ((long long)b * p.H + h) * p.L + (long long)c * CT;
    const float lj = p.l[lo + tid];
    float s;
    if (p.mode == 0) s = __expf(p.l[lo + CT - 1] - lj) * p.dt[lo + tid];
    else s = __expf(lj);
    const __nv_bfloat16* vr = p.v + (row0 + tid) * p.v_row_stride + (long long)hv * PS;
    #pragma unroll
    for (int ch = 0; ch < 8; ++ch) {
      float f[8];
      unpack8(*reinterpret_cast<const uint4*>(vr + ch * 8), f);
      #pragma unroll
      for (int e = 0; e < 8; ++e) f[e] *= s;
      *reinterpret_cast<uint4*>(sV + sw128_offset(tid, ch)) = pack8(f);
    }
  }
  fence_proxy_async_smem();
  __syncthreads();
  bool ok = true;
  if (tid == 0) {
    ok = mbar_wait(&bars[0], 0, p.status);
    if (ok) {
      tc_fence_after_sync();
      const uint32_t idesc = make_idesc_bf16(128, PS, 1, 1);
      const uint32_t a = smem_u32(sW), bb = smem_u32(sV);
      #pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        umma_bf16(tmem, desc_mnmajor(a, kk, TILE128 / 2), desc_mnmajor(bb, kk, 0), idesc, kk != 0);
      umma_commit(&bars[1]);
    }
  }
  __syncwarp();
  ok = __syncthreads_and(mbar_wait(&bars[1], 0, p.status));
  tc_fence_after_sync();
  if (ok) {
    float* o = p.out + ((((long long)b * p.Hv + hv) * p.nc + c) * NS + tid) * PS;
    #pragma unroll
    for (int half = 0; half < 2; ++half) {
      uint32_t v[32];
      tmem_ld32(tmem_addr(tmem, warp * 32, half * 32), v);
      tmem_ld_wait();
      #pragma unroll
      for (int q = 0; q < 8; ++q)
        *reinterpret_cast<float4*>(o + half * 32 + q * 4) =
            make_float4(__uint_as_float(v[q * 4]), __uint_as_float(v[q * 4 + 1]), __uint_as_float(v[q * 4 + 2]),
                        __uint_as_float(v[q * 4 + 3]));
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 64);
}

// =====================================================================================
// inter-chunk recurrence (elementwise over the N*P state entries):
//   forward:  in[c] = run ; run = exp(l_T[c]) * run + local[c]       c = 0 .. nc-1
//   reverse:  in[c] = run ; run = exp(l_T[c]) * run + local[c]       c = nc-1 .. 0
// in: bf16 [B,Hv,nc,N*P] (MMA operand), final: fp32 [B,Hv,N*P] (optional), init fp32 [B,Hv,N*P] (optional).
// grid (N*P/4/256, Hv, B), 256 threads.
// =====================================================================================
__global__ void __launch_bounds__(256)
ssd_state_pass_kernel(const float* __restrict__ local, const float* __restrict__ l, const float* __restrict__ init,
                      __nv_bfloat16* __restrict__ in16, float* __restrict__ fin, int L, int H, int Hv, int nc,
                      int reverse) {
  const int hv = blockIdx.y, b = blockIdx.z;
  const int h = hv / (Hv / H);
  const int e = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
  const long long base = ((long long)b * Hv + hv) * nc;
  const float* lrow = l + ((long long)b * H + h) * L;
  float4 run = make_float4(0.f, 0.f, 0.f, 0.f);
  if (init) run = *reinterpret_cast<const float4*>(init + ((long long)b * Hv + hv) * (NS * PS) + e);
  for (int k = 0; k < nc; ++k) {
    const int c = reverse ? nc - 1 - k : k;
    const long long o = (base + c) * (NS * PS) + e;
    uint2 pk;
    pk.x = pack_bf16(run.x, run.y); pk.y = pack_bf16(run.z, run.w);
    *reinterpret_cast<uint2*>(in16 + o) = pk;
    const float dec = __expf(lrow[(long long)c * CT + CT - 1]);
    const float4 s = *reinterpret_cast<const float4*>(local + o);
    run.x = dec * run.x + s.x; run.y = dec * run.y + s.y; run.z = dec * run.z + s.z; run.w = dec * run.w + s.w;
  }
  if (fin) *reinterpret_cast<float4*>(fin + ((long long)b * Hv + hv) * (NS * PS) + e) = run;
}

// =====================================================================================
// the backward pass's states in one kernel (mode 1 of the two kernels above without the fp32 states in between):
//   in[c] = run ; run = exp(l_T[c]) * run + sum_j exp(l_j) C[j][n] dY[j][p]       c descending
// One CTA per (head slice, batch) walks the chunks; the running state stays in registers (256 threads: row n = tid & 127,
// 32 of the 64 channels each).  Loads run three chunks ahead; the products of the next chunk run on tcgen05 (two TMEM
// buffers) while this one's state is stored and updated.
// Bound by latency per chunk (wait, scale V, products, update) at few heads, by HBM at many (V in, bf16 states out): the
// fp32 states, written and read back, were two thirds of the bytes.
// Few head slices leave most SMs idle while each walks all its chunks, so the chunks are cut into segments: a first launch
// finds the state behind every segment but the last from a zero state (`finals`), and the launch that wants the states
// (this kernel backwards, ssd_walk_scan_kernel forwards) starts a segment from those behind the earlier ones.
// 32 slices x 64 chunks (us): forward 178 in one walk, 137 with a CTA per chunk, 79 in four segments; backward states 93, 78, 54.
// =====================================================================================
struct Segments {
  int count, len;                        // of consecutive steps, `len` chunks each (the last one may be shorter)
  float* fin;                            // [B, Hv, count][128 n][64 p] state behind a segment that began with zeros
  float* decay;                          // [B, Hv, count] decay over a segment
};
// the state that enters segment `seg`: V consecutive channels of row `row` from `at` on, entered with `run`
template <int V>
__device__ __forceinline__ void segment_entry(const Segments& sg, long long slice, int seg, int row, int at, float (&run)[V]) {
  for (int r = 0; r < seg; ++r) {
    const float d = sg.decay[slice * sg.count + r];
    const float4* f = reinterpret_cast<const float4*>(sg.fin + ((slice * sg.count + r) * NS + row) * PS + at);
    #pragma unroll
    for (int e = 0; e < V; e += 4) {
      const float4 v = f[e / 4];
      run[e] = d * run[e] + v.x; run[e + 1] = d * run[e + 1] + v.y; run[e + 2] = d * run[e + 2] + v.z; run[e + 3] = d * run[e + 3] + v.w;
    }
  }
}
struct StateWalkParams {
  const float* dt; const float* l;       // [B, H, L]; dt forwards only
  int L, H, Hv, G, nc, w_col0;
  int forward, finals;                   // forward: W = B, V = x, ascending; finals: no states, only what Segments wants
  Segments seg;
  int* status;
};
constexpr int WALK_STAGES = 3;
constexpr int WALK_STAGE_BYTES = TILE128 + TILE64;
constexpr int WALK_SMEM = WALK_STAGES * WALK_STAGE_BYTES + 2 * TILE64 + 128 + 1024;

__global__ void __launch_bounds__(256, 1)
ssd_state_walk_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_v,
                      const __grid_constant__ CUtensorMap tm_in, const StateWalkParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sOut = smem + WALK_STAGES * WALK_STAGE_BYTES;                 // two staging tiles for the bf16 states
  uint64_t* full = reinterpret_cast<uint64_t*>(sOut + 2 * TILE64);       // [stage] loads landed
  uint64_t* done = full + WALK_STAGES;                                   // [2] products of a TMEM buffer complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 2);
  const int hv = blockIdx.x, b = blockIdx.y, seg = blockIdx.z, tid = threadIdx.x, warp = tid >> 5;
  const int first = seg * p.seg.len, n = p.nc - first < p.seg.len ? p.nc - first : p.seg.len;      // steps of this segment
  const int row = tid & 127, half = tid >> 7;
  const int h = hv / (p.Hv / p.H), g = h / (p.H / p.G);
  const float* lh = p.l + ((long long)b * p.H + h) * p.L;
  const float* dth = p.dt + ((long long)b * p.H + h) * p.L;
  auto chunk = [&](int k) { return p.forward ? first + k : p.nc - 1 - first - k; };      // chunk of step k

  if (tid == 0) {
    for (int s = 0; s < WALK_STAGES; ++s) mbar_init(&full[s], 1);
    mbar_init(&done[0], 1); mbar_init(&done[1], 1);
    mbar_fence_init();
    tma_prefetch_desc(&tm_w); tma_prefetch_desc(&tm_v); tma_prefetch_desc(&tm_in);
  }
  if (warp == 0) { tmem_alloc(tmem_slot, 128); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;

  auto load = [&](int k) {                                               // thread 0
    const int st = k % WALK_STAGES, r = b * p.L + chunk(k) * CT;
    uint8_t* sw = smem + st * WALK_STAGE_BYTES;
    mbar_expect_tx(&full[st], WALK_STAGE_BYTES);
    tma_load_2d(sw, &tm_w, p.w_col0 + g * NS, r, &full[st]);
    tma_load_2d(sw + TILE128 / 2, &tm_w, p.w_col0 + g * NS + 64, r, &full[st]);
    tma_load_2d(sw + TILE128, &tm_v, hv * PS, r, &full[st]);
  };
  int loaded = 0;                                                        // steps whose loads have been issued (thread 0)
  if (tid == 0)
    for (; loaded < WALK_STAGES && loaded < n; ++loaded) load(loaded);
  // scaling of a step: l_j and dt_j of this thread's row and l_T, fetched a step ahead
  float lj = 0.f, lT = 0.f, dj = 1.f, lsum = 0.f;
  auto fetch = [&](int k) {
    if (k >= n) return;
    const long long o = (long long)chunk(k) * CT;
    lj = lh[o + row]; lT = lh[o + CT - 1];
    if (p.forward) dj = dth[o + row];
    lsum += lT;
  };
  // V rows of step k scaled in place, then its products issued into TMEM buffer k & 1
  bool ok = true;
  auto scale_and_issue = [&](int k) {
    const int st = k % WALK_STAGES;
    uint8_t* sw = smem + st * WALK_STAGE_BYTES;
    uint8_t* sv = sw + TILE128;
    const float s = p.forward ? __expf(lT - lj) * dj : __expf(lj);
    ok = mbar_wait(&full[st], (k / WALK_STAGES) & 1, p.status);
    if (ok) {
      #pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint4* at = reinterpret_cast<uint4*>(sv + sw128_offset(row, half * 4 + q));
        float f[8];
        unpack8(*at, f);
        #pragma unroll
        for (int e = 0; e < 8; ++e) f[e] *= s;
        *at = pack8(f);
      }
    }
    fence_proxy_async_smem();
    ok = __syncthreads_and(ok);
    if (tid == 0 && ok) {
      tc_fence_after_sync();
      const uint32_t idesc = make_idesc_bf16(128, PS, 1, 1);
      const uint32_t aw = smem_u32(sw), av = smem_u32(sv);
      #pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        umma_bf16(tmem + (k & 1) * 64, desc_mnmajor(aw, kk, TILE128 / 2), desc_mnmajor(av, kk, 0), idesc, kk != 0);
      umma_commit(&done[k & 1]);
    }
    __syncwarp();
  };

  float run[32];
  #pragma unroll
  for (int e = 0; e < 32; ++e) run[e] = 0.f;
  const long long slice = (long long)b * p.Hv + hv;
  if (!p.finals) segment_entry<32>(p.seg, slice, seg, row, half * 32, run);
  fetch(0);
  float dec = __expf(lT);                                                // of the step whose products are in flight
  scale_and_issue(0);
  fetch(1);
  for (int k = 0; k < n && ok; ++k) {
    const float dec_k = dec;
    // the state that enters step k's chunk
    uint8_t* so = sOut + (k & 1) * TILE64;
    if (!p.finals) {
      #pragma unroll
      for (int q = 0; q < 4; ++q) {
        float f[8];
        #pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = run[q * 8 + e];
        *reinterpret_cast<uint4*>(so + sw128_offset(row, half * 4 + q)) = pack8(f);
      }
    }
    if (k + 1 < n) {
      dec = __expf(lT);
      scale_and_issue(k + 1);                                            // its barrier also covers the staging tile
      if (!ok) break;
      fetch(k + 2);
    } else {
      fence_proxy_async_smem();
      __syncthreads();
    }
    if (tid == 0 && !p.finals) {
      tma_store_2d(&tm_in, so, 0, ((b * p.Hv + hv) * p.nc + chunk(k)) * NS);
      tma_store_commit();
    }
    ok = mbar_wait(&done[k & 1], (k >> 1) & 1, p.status);
    ok = __all_sync(0xffffffffu, ok);
    tc_fence_after_sync();
    if (tid == 0 && ok && loaded < n) { load(loaded); ++loaded; }        // step k's stage is free again
    if (ok) {
      uint32_t v[32];
      tmem_ld32(tmem_addr(tmem, (warp & 3) * 32, (k & 1) * 64 + half * 32), v);
      tmem_ld_wait();
      #pragma unroll
      for (int e = 0; e < 32; ++e) run[e] = dec_k * run[e] + __uint_as_float(v[e]);
    }
    tc_fence_before_sync();
    if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");   // step k - 1's tile has been read
    ok = __syncthreads_and(ok);                                          // TMEM buffer and staging tile are free again
  }
  if (p.finals && ok) {
    float4* f = reinterpret_cast<float4*>(p.seg.fin + ((slice * p.seg.count + seg) * NS + row) * PS + half * 32);
    #pragma unroll
    for (int e = 0; e < 32; e += 4) f[e / 4] = make_float4(run[e], run[e + 1], run[e + 2], run[e + 3]);
    if (tid == 0) p.seg.decay[slice * p.seg.count + seg] = __expf(lsum);
  }
  if (tid == 0) {
    tma_store_wait_all();
    if (!ok)                                                             // copies still in flight land before the CTA goes
      for (int k = loaded > WALK_STAGES ? loaded - WALK_STAGES : 0; k < loaded; ++k)
        mbar_wait(&full[k % WALK_STAGES], (k / WALK_STAGES) & 1, nullptr);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 128);
}

// =====================================================================================
// forward chunk scan.  grid (nc, Hv, B), 128 threads, 2 CTAs / SM.
// TMEM: [0,128) CB^T product, [128,192) Y_diag, [192,256) Y_off.
// smem: C tile | B tile | x tile | S_in tile ; the decay-weighted matrix reuses the C tile, the output
// staging reuses the B tile.
// =====================================================================================
struct ScanFwdParams {
  const float* dt; const float* l; const float* D;   // dt,l [B,H,L]; D [H]
  int L, H, Hv, G, nc, d_in;
  int* status;
};

__global__ void __launch_bounds__(128)
ssd_chunk_scan_fwd_kernel(const __grid_constant__ CUtensorMap tm_xbc, const __grid_constant__ CUtensorMap tm_sin,
                          const __grid_constant__ CUtensorMap tm_y, const ScanFwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sC = smem;                          // [128 i][128 n]; later M [128 i][128 j]
  uint8_t* sB = smem + TILE128;                // [128 j][128 n]; later y staging [128 i][64 p]
  uint8_t* sX = smem + 2 * TILE128;            // [128 j][64 p]
  uint8_t* sS = smem + 2 * TILE128 + TILE64;   // [128 n][64 p]
  float* s_l = reinterpret_cast<float*>(smem + 2 * TILE128 + 2 * TILE64);
  float* s_dt = s_l + CT;
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_dt + CT);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 3);
  const int c = blockIdx.x, hv = blockIdx.y, b = blockIdx.z, tid = threadIdx.x, warp = tid >> 5;
  const int psplit = p.Hv / p.H, h = hv / psplit, g = h / (p.H / p.G);
  const int row0 = b * p.L + c * CT;

  if (tid == 0) {
    mbar_init(&bars[0], 1); mbar_init(&bars[1], 1); mbar_init(&bars[2], 1);
    mbar_fence_init();
    tma_prefetch_desc(&tm_xbc); tma_prefetch_desc(&tm_sin); tma_prefetch_desc(&tm_y);
  }
  if (warp == 0) { tmem_alloc(tmem_slot, 256); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;

  if (tid == 0) {
    mbar_expect_tx(&bars[0], 2 * TILE128 + 2 * TILE64);
    const int cB = p.d_in + g * NS, cC = p.d_in + p.G * NS + g * NS;
    tma_load_2d(sC, &tm_xbc, cC, row0, &bars[0]);
    tma_load_2d(sC + TILE128 / 2, &tm_xbc, cC + 64, row0, &bars[0]);
    tma_load_2d(sB, &tm_xbc, cB, row0, &bars[0]);
    tma_load_2d(sB + TILE128 / 2, &tm_xbc, cB + 64, row0, &bars[0]);
    tma_load_2d(sX, &tm_xbc, hv * PS, row0, &bars[0]);
    tma_load_2d(sS, &tm_sin, 0, ((b * p.Hv + hv) * p.nc + c) * NS, &bars[0]);
  }
  {
    const long long lo = ((long long)b * p.H + h) * p.L + (long long)c * CT;
    s_l[tid] = p.l[lo + tid];
    s_dt[tid] = p.dt[lo + tid];
  }
  __syncthreads();
  bool ok = true;
  if (tid == 0) {
    ok = mbar_wait(&bars[0], 0, p.status);
    if (ok) {
      tc_fence_after_sync();
      const uint32_t aC = smem_u32(sC), aB = smem_u32(sB), aS = smem_u32(sS);
      const uint32_t id_cb = make_idesc_bf16(128, 128, 0, 0);
      #pragma unroll
      for (int kk = 0; kk < 8; ++kk)      // CB^T[i][j] = sum_n C[i][n] B[j][n]
        umma_bf16(tmem, desc_kmajor(aC, kk, TILE128 / 2), desc_kmajor(aB, kk, TILE128 / 2), id_cb, kk != 0);
      const uint32_t id_off = make_idesc_bf16(128, PS, 0, 1);
      #pragma unroll
      for (int kk = 0; kk < 8; ++kk)      // Y_off[i][p] = sum_n C[i][n] S_in[n][p]
        umma_bf16(tmem + 192, desc_kmajor(aC, kk, TILE128 / 2), desc_mnmajor(aS, kk, 0), id_off, kk != 0);
      umma_commit(&bars[1]);
    }
  }
  __syncwarp();
  ok = __syncthreads_and(mbar_wait(&bars[1], 0, p.status));
  tc_fence_after_sync();
  const int i = tid;
  if (ok) {
    // decay-weighted lower-triangular matrix, row i, written over the C tile (K-major A operand, K = j)
    const float li = s_l[i];
    #pragma unroll 1
    for (int jb = 0; jb < 4; ++jb) {
      if (jb > warp) {      // columns j > i for every row of this warp: the causal mask zeroes the whole block
        #pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
          const int jc = jb * 32 + ch * 8;
          *reinterpret_cast<uint4*>(sC + (jc >> 6) * (TILE128 / 2) + sw128_offset(i, (jc & 63) >> 3)) = make_uint4(0, 0, 0, 0);
        }
        continue;
      }
      uint32_t v[32];
      tmem_ld32(tmem_addr(tmem, warp * 32, jb * 32), v);
      tmem_ld_wait();
      #pragma unroll
      for (int ch = 0; ch < 4; ++ch) {
        float f[8];
        #pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int j = jb * 32 + ch * 8 + e;
          f[e] = (j <= i) ? __uint_as_float(v[ch * 8 + e]) * __expf(li - s_l[j]) * s_dt[j] : 0.f;
        }
        const int jc = jb * 32 + ch * 8;
        *reinterpret_cast<uint4*>(sC + (jc >> 6) * (TILE128 / 2) + sw128_offset(i, (jc & 63) >> 3)) = pack8(f);
      }
    }
  }
  fence_proxy_async_smem();
  tc_fence_before_sync();
  __syncthreads();
  if (tid == 0 && ok) {
    tc_fence_after_sync();
    const uint32_t aM = smem_u32(sC), aX = smem_u32(sX);
    const uint32_t id = make_idesc_bf16(128, PS, 0, 1);
    #pragma unroll
    for (int kk = 0; kk < 8; ++kk)        // Y_diag[i][p] = sum_j M[i][j] x[j][p]
      umma_bf16(tmem + 128, desc_kmajor(aM, kk, TILE128 / 2), desc_mnmajor(aX, kk, 0), id, kk != 0);
    umma_commit(&bars[2]);
  }
  __syncwarp();
  ok = __syncthreads_and(ok && mbar_wait(&bars[2], 0, p.status));
  tc_fence_after_sync();
  if (ok) {
    const float al = __expf(s_l[i]);
    const float Dh = p.D[h];
    #pragma unroll
    for (int half = 0; half < 2; ++half) {
      uint32_t yd[32], yo[32];
      tmem_ld32(tmem_addr(tmem, warp * 32, 128 + half * 32), yd);
      tmem_ld32(tmem_addr(tmem, warp * 32, 192 + half * 32), yo);
      tmem_ld_wait();
      #pragma unroll
      for (int ch = 0; ch < 4; ++ch) {
        float xv[8], f[8];
        unpack8(*reinterpret_cast<const uint4*>(sX + sw128_offset(i, half * 4 + ch)), xv);
        #pragma unroll
        for (int e = 0; e < 8; ++e)
          f[e] = __uint_as_float(yd[ch * 8 + e]) + al * __uint_as_float(yo[ch * 8 + e]) + Dh * xv[e];
        *reinterpret_cast<uint4*>(sB + sw128_offset(i, half * 4 + ch)) = pack8(f);
      }
    }
  }
  fence_proxy_async_smem();
  tc_fence_before_sync();
  __syncthreads();
  if (tid == 0 && ok) {
    tma_store_2d(&tm_y, sB, hv * PS, row0);
    tma_store_commit();
    tma_store_wait_all();
  }
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 256);
}

// =====================================================================================
// forward scan in one kernel: the state walk (ascending) and the chunk scan of the same chunk.  One CTA per (head slice,
// batch); x, B and C of a chunk are read once, the state that enters it goes from registers through shared memory into the
// product with C, and to HBM only where a backward pass will want it.
//   warps 0-15  row = token / state row, a quarter of the columns each.  Chunk k:
//                 c  decay-weighted C B^T                     -> M
//                 e  state update, C S_in read back
//                 a  of chunk k + 1: x scaled for the state, entering state to shared memory
//                 f  y = M x + exp(l_i) C S_in + D x, in place of x
//   warp 16     issues the products: state and C S_in of k + 1 behind a, M x of k and C B^T of k + 1 behind c
//   warp 17     loads (two stages) and stores
// so that every product runs under the arithmetic of another step.  Bound by that arithmetic (one exponential per pair of
// tokens), the products' reads of shared memory and the hand-overs.  States and scan in kernels of their own wrote and read
// the states and read x and B twice: 128 slices x 16 chunks 86 -> 51 us, 320 x 16 232 -> 158, 1280 x 16 808 -> 472.
// TMEM: [0,128) and [128,256) C B^T by turns, [256,320) state, [320,384) C S_in, [384,448) M x.
// =====================================================================================
struct WalkScanParams {
  const float* dt; const float* l; const float* D;    // [B, H, L]; D [H]
  const float* init; float* fin;         // fp32 [B, Hv, 128 n, 64 p] in, [B, Hv, 64 p, 128 n] out, or null
  int store_states;                      // write the bf16 state entering every chunk
  int L, H, Hv, G, nc, d_in;
  Segments seg;                          // one CTA per (head slice, batch, segment)
  int* status;
};
constexpr int WS_THREADS = 18 * 32;
constexpr int WS_STAGE = 2 * TILE128 + TILE64;                           // B | C | x
constexpr int WS_USED = 2 * WS_STAGE + 2 * TILE64 + TILE128 + 2 * 2 * CT * 4 + 128;
constexpr int WS_SMEM = 227 * 1024;                                      // all of it: what is left aligns the tiles

__global__ void __launch_bounds__(WS_THREADS, 1)
ssd_walk_scan_kernel(const __grid_constant__ CUtensorMap tm_xbc, const __grid_constant__ CUtensorMap tm_in,
                     const __grid_constant__ CUtensorMap tm_y, const WalkScanParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sXs = smem + 2 * WS_STAGE;                  // scaled x [128 j][64 p]
  uint8_t* sS = sXs + TILE64;                          // entering state [128 n][64 p]
  uint8_t* sM = sS + TILE64;                           // M [128 i][128 j]
  float* sLD = reinterpret_cast<float*>(sM + TILE128); // [2] l[128] | dt[128] of a stage's chunk
  uint64_t* bars = reinterpret_cast<uint64_t*>(sLD + 2 * 2 * CT);
  uint64_t *full = bars, *cb_done = bars + 2, *st_done = bars + 4, *y_done = bars + 5, *xs_ready = bars + 6,
           *m_ready = bars + 7, *y_ready = bars + 8, *s_free = bars + 10;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 11);
  if (smem - smem_raw > WS_SMEM - WS_USED) {           // uniform; cannot happen while dynamic shared memory starts on 1 KiB
    if (threadIdx.x == 0) atomicCAS(p.status, 0, SSM_ERR_BAD_ARG);
    return;
  }
  const int hv = blockIdx.x, b = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int c0 = blockIdx.z * p.seg.len, n = p.nc - c0 < p.seg.len ? p.nc - c0 : p.seg.len;        // this segment's chunks
  const int h = hv / (p.Hv / p.H), g = h / (p.H / p.G);

  if (tid == 0) {
    for (int k = 0; k < 6; ++k) mbar_init(&bars[k], 1);
    for (int k = 6; k < 10; ++k) mbar_init(&bars[k], 16);
    mbar_init(s_free, 1);
    mbar_fence_init();
    tma_prefetch_desc(&tm_xbc); tma_prefetch_desc(&tm_in); tma_prefetch_desc(&tm_y);
  }
  if (warp == 16) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;

  if (warp == 17) {
    if (lane == 0) {
      const long long lo = ((long long)b * p.H + h) * p.L + (long long)c0 * CT;
      auto load = [&](int k) {
        uint8_t* sb = smem + (k & 1) * WS_STAGE;
        uint64_t* bar = &full[k & 1];
        const int r = b * p.L + (c0 + k) * CT, cB = p.d_in + g * NS, cC = p.d_in + p.G * NS + g * NS;
        mbar_expect_tx(bar, WS_STAGE + 2 * CT * 4);
        tma_load_2d(sb, &tm_xbc, cB, r, bar);
        tma_load_2d(sb + TILE128 / 2, &tm_xbc, cB + 64, r, bar);
        tma_load_2d(sb + TILE128, &tm_xbc, cC, r, bar);
        tma_load_2d(sb + TILE128 + TILE128 / 2, &tm_xbc, cC + 64, r, bar);
        tma_load_2d(sb + 2 * TILE128, &tm_xbc, hv * PS, r, bar);
        bulk_load(sLD + (k & 1) * 2 * CT, p.l + lo + (long long)k * CT, CT * 4, bar);
        bulk_load(sLD + (k & 1) * 2 * CT + CT, p.dt + lo + (long long)k * CT, CT * 4, bar);
      };
      int loaded = 0;
      for (; loaded < 2 && loaded < n; ++loaded) load(loaded);
      bool ok = true;
      for (int k = -1; k < n && ok; ++k) {
        if (p.store_states && k + 1 < n) {          // the state entering chunk k + 1 is in shared memory
          ok = mbar_wait(xs_ready, (k + 1) & 1, p.status);
          if (!ok) break;
          tma_store_2d(&tm_in, sS, 0, ((b * p.Hv + hv) * p.nc + c0 + k + 1) * NS);
          tma_store_commit();
          tma_store_wait_read();
          mbar_arrive(s_free);
        }
        if (k >= 0) {                                  // y of chunk k stands in its x tile
          ok = mbar_wait(&y_ready[k & 1], (k >> 1) & 1, p.status);
          if (!ok) break;
          tma_store_2d(&tm_y, smem + (k & 1) * WS_STAGE + 2 * TILE128, hv * PS, b * p.L + (c0 + k) * CT);
          tma_store_commit();
          if (loaded < n) { tma_store_wait_read(); load(loaded); ++loaded; }
        }
      }
      tma_store_wait_all();
      if (!ok)                                         // copies still in flight land before the CTA goes
        for (int k = loaded > 2 ? loaded - 2 : 0; k < loaded; ++k) mbar_wait(&full[k & 1], (k >> 1) & 1, nullptr);
    }
    __syncwarp();
  } else if (warp == 16) {
    if (lane == 0) {
      const uint32_t id_cb = make_idesc_bf16(128, 128, 0, 0), id_st = make_idesc_bf16(128, PS, 1, 1),
                     id_off = make_idesc_bf16(128, PS, 0, 1);
      const uint64_t dXs = desc_mnmajor(smem_u32(sXs), 0, 0), dS = desc_mnmajor(smem_u32(sS), 0, 0);
      // descriptor steps (16-byte units) of a k-step: 32 bytes inside an atom of 64, then the next atom; 16 rows
      auto kstep = [](int kk) { return (uint64_t)((kk >> 2) * (TILE128 / 2 / 16) + (kk & 3) * 2); };
      auto issue_cb = [&](int k) {
        const uint32_t aB = smem_u32(smem + (k & 1) * WS_STAGE);
        const uint64_t dC = desc_kmajor(aB + TILE128, 0, TILE128 / 2), dB = desc_kmajor(aB, 0, TILE128 / 2);
        #pragma unroll
        for (int kk = 0; kk < 8; ++kk) umma_bf16(tmem + (k & 1) * 128, dC + kstep(kk), dB + kstep(kk), id_cb, kk != 0);
        umma_commit(&cb_done[k & 1]);
      };
      bool ok = mbar_wait(&full[0], 0, p.status);
      if (ok) { tc_fence_after_sync(); issue_cb(0); }
      auto issue_state = [&](int k) {
        ok = mbar_wait(xs_ready, k & 1, p.status);
        if (!ok) return;
        tc_fence_after_sync();
        const uint32_t aB = smem_u32(smem + (k & 1) * WS_STAGE);
        const uint64_t dBm = desc_mnmajor(aB, 0, TILE128 / 2), dC = desc_kmajor(aB + TILE128, 0, TILE128 / 2);
        #pragma unroll
        for (int kk = 0; kk < 8; ++kk)                 // S_local[n][p] = sum_j B[j][n] xs[j][p]
          umma_bf16(tmem + 256, dBm + (uint64_t)(kk * 128), dXs + (uint64_t)(kk * 128), id_st, kk != 0);
        #pragma unroll
        for (int kk = 0; kk < 8; ++kk)                 // Y_off[i][p] = sum_n C[i][n] S_in[n][p]
          umma_bf16(tmem + 320, dC + kstep(kk), dS + (uint64_t)(kk * 128), id_off, kk != 0);
        umma_commit(st_done);
      };
      if (ok) issue_state(0);
      for (int k = 0; k < n && ok; ++k) {
        ok = mbar_wait(m_ready, k & 1, p.status);
        if (!ok) break;
        tc_fence_after_sync();
        const uint64_t dM = desc_kmajor(smem_u32(sM), 0, TILE128 / 2),
                       dX = desc_mnmajor(smem_u32(smem + (k & 1) * WS_STAGE + 2 * TILE128), 0, 0);
        #pragma unroll
        for (int kk = 0; kk < 8; ++kk)                 // Y_diag[i][p] = sum_j M[i][j] x[j][p]
          umma_bf16(tmem + 384, dM + kstep(kk), dX + (uint64_t)(kk * 128), id_off, kk != 0);
        umma_commit(y_done);
        if (k + 1 < n) {
          ok = mbar_wait(&full[(k + 1) & 1], ((k + 1) >> 1) & 1, p.status);
          if (!ok) break;
          tc_fence_after_sync();
          issue_cb(k + 1);
          issue_state(k + 1);
        }
      }
    }
    __syncwarp();
  } else {
    const int rw = warp & 3, wq = warp >> 2, row = rw * 32 + lane;      // quarter wq: 16 channels, 32 tokens
    const uint32_t lanes = (uint32_t)rw * 32;
    const float Dh = p.D[h];
    float run[16];
    #pragma unroll
    for (int e = 0; e < 16; e += 4) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (p.init != nullptr)
        v = *reinterpret_cast<const float4*>(p.init + ((long long)b * p.Hv + hv) * (NS * PS) + row * PS + wq * 16 + e);
      run[e] = v.x; run[e + 1] = v.y; run[e + 2] = v.z; run[e + 3] = v.w;
    }
    segment_entry<16>(p.seg, (long long)b * p.Hv + hv, blockIdx.z, row, wq * 16, run);
    bool ok = true;
    // what the other warps do with these writes starts when all sixteen warps have arrived
    auto arrive = [&](uint64_t* bar) {
      fence_proxy_async_smem();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    auto wait = [&](uint64_t* bar, int phase) {
      ok = __all_sync(0xffffffffu, mbar_wait(bar, phase & 1, p.status));
      tc_fence_after_sync();
    };
    float li = 0.f, lT = 0.f;                          // of the chunk whose x has been scaled last
    auto prepare = [&](int k) {                        // a
      wait(&full[k & 1], k >> 1);
      if (ok && p.store_states && k > 0) wait(s_free, k - 1);
      if (!ok) return;
      const float* sl = sLD + (k & 1) * 2 * CT;
      li = sl[row]; lT = sl[CT - 1];
      const float sx = __expf(lT - li) * sl[CT + row];
      const uint8_t* sX = smem + (k & 1) * WS_STAGE + 2 * TILE128;
      #pragma unroll
      for (int q = 0; q < 2; ++q) {
        const uint32_t off = sw128_offset(row, wq * 2 + q);
        float f[8];
        unpack8(*reinterpret_cast<const uint4*>(sX + off), f);
        #pragma unroll
        for (int e = 0; e < 8; ++e) f[e] *= sx;
        *reinterpret_cast<uint4*>(sXs + off) = pack8(f);
        #pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = run[q * 8 + e];
        *reinterpret_cast<uint4*>(sS + off) = pack8(f);
      }
      arrive(xs_ready);
    };
    prepare(0);
    for (int k = 0; k < n && ok; ++k) {
      const float lik = li, dec = __expf(lT);
      const float* sl = sLD + (k & 1) * 2 * CT + wq * 32;
      // ---- c
      wait(&cb_done[k & 1], k >> 1);
      if (!ok) break;
      uint8_t* m_at = sM + (wq >> 1) * (TILE128 / 2);
      if (wq > rw) {                                   // tokens j > i for every row of this warp
        #pragma unroll
        for (int ch = 0; ch < 4; ++ch)
          *reinterpret_cast<uint4*>(m_at + sw128_offset(row, (wq & 1) * 4 + ch)) = make_uint4(0, 0, 0, 0);
      } else {
        uint32_t v[32];
        tmem_ld32(tmem_addr(tmem, lanes, (k & 1) * 128 + wq * 32), v);
        tmem_ld_wait();
        #pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
          float lv[8], dv[8], f[8];
          load8f_smem(sl + ch * 8, lv);
          load8f_smem(sl + CT + ch * 8, dv);
          #pragma unroll
          for (int e = 0; e < 8; ++e)
            f[e] = (wq * 32 + ch * 8 + e <= row) ? __uint_as_float(v[ch * 8 + e]) * __expf(lik - lv[e]) * dv[e] : 0.f;
          *reinterpret_cast<uint4*>(m_at + sw128_offset(row, (wq & 1) * 4 + ch)) = pack8(f);
        }
      }
      arrive(m_ready);
      // ---- e
      wait(st_done, k);
      if (!ok) break;
      uint32_t v[16], yo[16];
      tmem_ld16(tmem_addr(tmem, lanes, 256 + wq * 16), v);
      tmem_ld16(tmem_addr(tmem, lanes, 320 + wq * 16), yo);
      tmem_ld_wait();
      #pragma unroll
      for (int e = 0; e < 16; ++e) run[e] = dec * run[e] + __uint_as_float(v[e]);
      // ---- a of the next chunk
      if (k + 1 < n) { prepare(k + 1); if (!ok) break; }
      // ---- f
      wait(y_done, k);
      if (!ok) break;
      tmem_ld16(tmem_addr(tmem, lanes, 384 + wq * 16), v);
      tmem_ld_wait();
      const float al = __expf(lik);
      uint8_t* sX = smem + (k & 1) * WS_STAGE + 2 * TILE128;
      #pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint4* at = reinterpret_cast<uint4*>(sX + sw128_offset(row, wq * 2 + q));
        float xv[8], f[8];
        unpack8(*at, xv);
        #pragma unroll
        for (int e = 0; e < 8; ++e)
          f[e] = __uint_as_float(v[q * 8 + e]) + al * __uint_as_float(yo[q * 8 + e]) + Dh * xv[e];
        *at = pack8(f);
      }
      arrive(&y_ready[k & 1]);                         // two barriers: the store of a chunk may lag one chunk behind
    }
    if (ok && p.fin != nullptr && c0 + n == p.nc) {                      // channel rows, as a decoding cache holds them
      float* fin = p.fin + ((long long)b * p.Hv + hv) * (NS * PS) + (wq * 16) * NS + row;
      #pragma unroll
      for (int e = 0; e < 16; ++e) fin[e * NS] = run[e];
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 16) tmem_dealloc(tmem, 512);
}

// =====================================================================================
// backward chunk scan.  grid (nc, G * splits, B), 1 CTA / SM; the CTA walks `hpc` head slices
// of one group.  Given dY and, per chunk, S_in (state entering the chunk) and dS_out (gradient of the state
// leaving the chunk):
//   CB = C B^T ; dM = dY X^T ; M0 = CB o Lambda ; dCB = dM o Lambda o dt_j
//   dU   = M0^T dY + exp(l_T - l_j) (B dS_out)                      dx = dt_j dU + D dY
//   dB  += dCB^T C + (exp(l_T - l_j) dt_j X) dS_out^T               dC += dCB B + (exp(l_i) dY) S_in^T
//   ddt_j = sum_p x dU + A da_j ;  da_j = sum_{k >= j} dl_k + E
//   dl_k = sum_{j<k} W[k][j] - sum_{i>k} W[i][k] + exp(l_k) sum_p dY (C S_in) - exp(l_T - l_k) dt_k sum_p x (B dS_out),
//          W = dM o M0 o dt_j   (row sums in-thread, column sums by a warp butterfly; no cancellation of large terms)
//   E = exp(l_T) <dS_out, S_in> + sum_j exp(l_T - l_j) dt_j sum_p x (B dS_out)
//   dA += sum_j dt_j da_j ; dD += sum dY x ; d(dt_raw) = ddt sigmoid(dt_raw + bias)
//   warps 0-15  row = token, a quarter of the columns each (16 channels, 32 tokens):
//                 1  exp(l_T - l_j) dt_j x and exp(l_i) dY       2  M0, dCB and the row / column sums of W
//                 3  dx and the per-token sums                   4  (warps 0-3, a thread per row) ddt, dA, dD, d dt_bias
//   warp 16     issues the products: CB, dM behind the loads; dU, C S_in and then dB, dC behind 2
//   warp 17     loads and the store of dx
// The arithmetic of 2 goes two values at a time (fma.rn.f32x2 and the like): 124 -> 116 us at 128 slices x 16 chunks.
// The loads of the next head start as soon as the last product that reads a tile is complete, 3 runs under the products of
// dB and dC, 4 under the next head's 1.  Bound by the per-pair arithmetic of 2 and the hand-overs between the steps: with
// 128-token tiles and four operands per head in shared memory there is room for one head only.
// TMEM: [0,128) CB then dU_diag | dU_state, [128,256) dM then C S_in, [256,384) dB, [384,512) dC
// (dB, dC accumulate over the CTA's heads and go to the fp32 output by bulk stores, or reductions where CTAs share a group).
// =====================================================================================
struct ScanBwdParams {
  const float* dt; const float* l; const float* D; const float* A; const float* dt_bias;
  const __nv_bfloat16* dt_raw; long long dt_raw_stride;     // [B*L rows], column h
  __nv_bfloat16* ddt_raw; long long ddt_stride;             // d(dt_raw): row (b*L+t)*stride + h  (bf16, atomic-free when psplit == 1)
  float* ddt32;                                             // [B, Hv, L] fp32 per head slice (summed on the host when psplit > 1)
  float* hpart;                                             // fp32 [B*nc, Hv, 3]  (dA, dD, d dt_bias partials)
  int L, H, Hv, G, nc, d_in, hpc;
  int* status;
};

constexpr int BWD_THREADS = 18 * 32;
// C, B | x, dY, S_in, dS_out | M0, dCB | scaled x, scaled dY | l, dt | sums
constexpr int BWD_USED = 2 * TILE128 + 4 * TILE64 + 2 * TILE128 + 2 * TILE64 + 2 * CT * 4 + 48 * 4 + 128;
constexpr int BWD_SMEM = 227 * 1024;                 // all of it: what is left aligns the tiles

__global__ void __launch_bounds__(BWD_THREADS, 1)
ssd_chunk_scan_bwd_kernel(const __grid_constant__ CUtensorMap tm_xbc, const __grid_constant__ CUtensorMap tm_dy,
                          const __grid_constant__ CUtensorMap tm_sin, const __grid_constant__ CUtensorMap tm_dsout,
                          const __grid_constant__ CUtensorMap tm_dx, const __grid_constant__ CUtensorMap tm_dbc,
                          const ScanBwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sC = smem;
  uint8_t* sB = sC + TILE128;
  uint8_t* sX = sB + TILE128;
  uint8_t* sDY = sX + TILE64;
  uint8_t* sSin = sDY + TILE64;
  uint8_t* sDS = sSin + TILE64;
  uint8_t* sM0 = sDS + TILE64;         // M0; once dU is complete: dx staging | sums
  uint8_t* sDCB = sM0 + TILE128;
  uint8_t* sXs = sDCB + TILE128;       // exp(l_T - l_j) dt_j x
  uint8_t* sDYs = sXs + TILE64;        // exp(l_i) dY
  float* s_l = reinterpret_cast<float*>(sDYs + TILE64);
  float* s_dt = s_l + CT;
  float* s_red = s_dt + CT;            // [16] share of E per warp, [16] dD per warp, [4] suffix totals, [4] dA, [4] d dt_bias
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_red + 48);
  uint64_t *cb_full = bars, *a_full = bars + 1, *b_full = bars + 2, *s_done = bars + 3, *u_done = bars + 4, *g_done = bars + 5,
           *m0_free = bars + 6, *ops_ready = bars + 7, *e_done = bars + 8;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 9);
  float* s_col = reinterpret_cast<float*>(sM0 + TILE64);               // [4 row-warps][128] column sums of W
  float* s_part = s_col + 4 * CT;                                      // [4 sums][4 quarters][128 rows]
  if (smem - smem_raw > BWD_SMEM - BWD_USED) {         // uniform; cannot happen while dynamic shared memory starts on 1 KiB
    if (threadIdx.x == 0) atomicCAS(p.status, 0, SSM_ERR_BAD_ARG);
    return;
  }
  const int c = blockIdx.x, b = blockIdx.z, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int psplit = p.Hv / p.H;
  const int hv_per_group = (p.H / p.G) * psplit;
  const int splits = hv_per_group / p.hpc;
  const int g = blockIdx.y / splits;
  const int hv0 = g * hv_per_group + (blockIdx.y % splits) * p.hpc;
  const int row0 = b * p.L + c * CT;
  const int GN = p.G * NS;

  if (tid == 0) {
    for (int k = 0; k < 7; ++k) mbar_init(&bars[k], 1);
    mbar_init(ops_ready, 16); mbar_init(e_done, 16);
    mbar_fence_init();
    tma_prefetch_desc(&tm_xbc); tma_prefetch_desc(&tm_dy); tma_prefetch_desc(&tm_sin);
    tma_prefetch_desc(&tm_dsout); tma_prefetch_desc(&tm_dx); tma_prefetch_desc(&tm_dbc);
  }
  if (warp == 16) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;

  if (warp == 17) {
    if (lane == 0) {
      auto load_a = [&](int it) {                      // x, dY, l, dt
        const int hv = hv0 + it, h = hv / psplit;
        const long long lo = ((long long)b * p.H + h) * p.L + (long long)c * CT;
        mbar_expect_tx(a_full, 2 * TILE64 + 2 * CT * 4);
        tma_load_2d(sX, &tm_xbc, hv * PS, row0, a_full);
        tma_load_2d(sDY, &tm_dy, hv * PS, row0, a_full);
        bulk_load(s_l, p.l + lo, CT * 4, a_full);
        bulk_load(s_dt, p.dt + lo, CT * 4, a_full);
      };
      auto load_b = [&](int it) {                      // S_in, dS_out
        const int srow = ((b * p.Hv + hv0 + it) * p.nc + c) * NS;
        mbar_expect_tx(b_full, 2 * TILE64);
        tma_load_2d(sSin, &tm_sin, 0, srow, b_full);
        tma_load_2d(sDS, &tm_dsout, 0, srow, b_full);
      };
      const int cB = p.d_in + g * NS, cC = p.d_in + GN + g * NS;
      mbar_expect_tx(cb_full, 2 * TILE128);
      tma_load_2d(sC, &tm_xbc, cC, row0, cb_full);
      tma_load_2d(sC + TILE128 / 2, &tm_xbc, cC + 64, row0, cb_full);
      tma_load_2d(sB, &tm_xbc, cB, row0, cb_full);
      tma_load_2d(sB + TILE128 / 2, &tm_xbc, cB + 64, row0, cb_full);
      load_a(0);
      load_b(0);
      bool ok = true;
      int na = 1, nb = 1;
      for (int it = 0; it < p.hpc; ++it) {
        const bool more = it + 1 < p.hpc;
        ok = mbar_wait(u_done, it & 1, p.status);
        if (!ok) break;
        if (more) { load_a(it + 1); ++na; }
        ok = mbar_wait(g_done, it & 1, p.status);
        if (!ok) break;
        if (more) { load_b(it + 1); ++nb; }
        ok = mbar_wait(e_done, it & 1, p.status);
        if (!ok) break;
        tma_store_2d(&tm_dx, sM0, (hv0 + it) * PS, row0);
        tma_store_commit();
        tma_store_wait_read();
        mbar_arrive(m0_free);
      }
      tma_store_wait_all();
      if (!ok) {                                       // copies still in flight land before the CTA goes
        mbar_wait(cb_full, 0, nullptr);
        mbar_wait(a_full, (na - 1) & 1, nullptr);
        mbar_wait(b_full, (nb - 1) & 1, nullptr);
      }
    }
    __syncwarp();
  } else if (warp == 16) {
    if (lane == 0) {
      // descriptors of the tiles in the roles they have; a k-step adds to the address field: 32 bytes inside an atom of 64,
      // then the next atom (kstep), or 16 rows (mstep)
      const uint64_t dCk = desc_kmajor(smem_u32(sC), 0, TILE128 / 2), dBk = desc_kmajor(smem_u32(sB), 0, TILE128 / 2),
                     dCm = desc_mnmajor(smem_u32(sC), 0, TILE128 / 2), dBm = desc_mnmajor(smem_u32(sB), 0, TILE128 / 2),
                     dXk = desc_kmajor(smem_u32(sX), 0, 0), dYk = desc_kmajor(smem_u32(sDY), 0, 0),
                     dYm = desc_mnmajor(smem_u32(sDY), 0, 0), dSink = desc_kmajor(smem_u32(sSin), 0, 0),
                     dSinm = desc_mnmajor(smem_u32(sSin), 0, 0), dDSk = desc_kmajor(smem_u32(sDS), 0, 0),
                     dDSm = desc_mnmajor(smem_u32(sDS), 0, 0), dM0m = desc_mnmajor(smem_u32(sM0), 0, TILE128 / 2),
                     dCBm = desc_mnmajor(smem_u32(sDCB), 0, TILE128 / 2), dCBk = desc_kmajor(smem_u32(sDCB), 0, TILE128 / 2),
                     dXsk = desc_kmajor(smem_u32(sXs), 0, 0), dYsk = desc_kmajor(smem_u32(sDYs), 0, 0);
      auto kstep = [](int kk) { return (uint64_t)((kk >> 2) * (TILE128 / 2 / 16) + (kk & 3) * 2); };
      auto mstep = [](int kk) { return (uint64_t)(kk * 128); };
      const uint32_t id_cb = make_idesc_bf16(128, 128, 0, 0), id_u1 = make_idesc_bf16(128, PS, 1, 1),
                     id_u2 = make_idesc_bf16(128, PS, 0, 1), id_b1 = make_idesc_bf16(128, 128, 1, 1),
                     id_c1 = make_idesc_bf16(128, 128, 0, 1);
      bool ok = mbar_wait(cb_full, 0, p.status);
      for (int it = 0; it < p.hpc && ok; ++it) {
        ok = mbar_wait(a_full, it & 1, p.status) && (it == 0 || mbar_wait(e_done, (it - 1) & 1, p.status));
        if (!ok) break;
        tc_fence_after_sync();
        #pragma unroll
        for (int kk = 0; kk < 8; ++kk)                            // CB[i][j] = sum_n C[i][n] B[j][n]
          umma_bf16(tmem, dCk + kstep(kk), dBk + kstep(kk), id_cb, kk != 0);
        #pragma unroll
        for (int kk = 0; kk < 4; ++kk)                            // dM[i][j] = sum_p dY[i][p] x[j][p]
          umma_bf16(tmem + 128, dYk + kstep(kk), dXk + kstep(kk), id_cb, kk != 0);
        umma_commit(s_done);
        ok = mbar_wait(ops_ready, it & 1, p.status) && mbar_wait(b_full, it & 1, p.status);
        if (!ok) break;
        tc_fence_after_sync();
        #pragma unroll
        for (int kk = 0; kk < 8; ++kk)                            // dU_diag[j][p] = sum_i M0[i][j] dY[i][p]
          umma_bf16(tmem, dM0m + mstep(kk), dYm + mstep(kk), id_u1, kk != 0);
        #pragma unroll
        for (int kk = 0; kk < 8; ++kk)                            // dU_state[j][p] = sum_n B[j][n] dS_out[n][p]
          umma_bf16(tmem + 64, dBk + kstep(kk), dDSm + mstep(kk), id_u2, kk != 0);
        #pragma unroll
        for (int kk = 0; kk < 8; ++kk)                            // Yoff[i][p] = sum_n C[i][n] S_in[n][p]
          umma_bf16(tmem + 128, dCk + kstep(kk), dSinm + mstep(kk), id_u2, kk != 0);
        umma_commit(u_done);
        #pragma unroll
        for (int kk = 0; kk < 8; ++kk)                            // dB[j][n] += sum_i dCB[i][j] C[i][n]
          umma_bf16(tmem + 256, dCBm + mstep(kk), dCm + mstep(kk), id_b1, (it | kk) != 0);
        #pragma unroll
        for (int kk = 0; kk < 4; ++kk)                            // dB[j][n] += sum_p xs[j][p] dS_out[n][p]
          umma_bf16(tmem + 256, dXsk + kstep(kk), dDSk + kstep(kk), id_cb, 1);
        #pragma unroll
        for (int kk = 0; kk < 8; ++kk)                            // dC[i][n] += sum_j dCB[i][j] B[j][n]
          umma_bf16(tmem + 384, dCBk + kstep(kk), dBm + mstep(kk), id_c1, (it | kk) != 0);
        #pragma unroll
        for (int kk = 0; kk < 4; ++kk)                            // dC[i][n] += sum_p dYs[i][p] S_in[n][p]
          umma_bf16(tmem + 384, dYsk + kstep(kk), dSink + kstep(kk), id_cb, 1);
        umma_commit(g_done);
      }
    }
    __syncwarp();
  } else {
    const int rw = warp & 3, wq = warp >> 2, row = rw * 32 + lane;
    const uint32_t lanes = (uint32_t)rw * 32;
    bool ok = true;
    auto arrive = [&](uint64_t* bar) {
      fence_proxy_async_smem();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    auto wait = [&](uint64_t* bar, int phase) {
      ok = __all_sync(0xffffffffu, mbar_wait(bar, phase & 1, p.status));
      tc_fence_after_sync();
    };
    auto all_ok = [](bool mine) { return barrier_and<1, 512>(mine); };
    for (int it = 0; it < p.hpc; ++it) {
      const int hv = hv0 + it, h = hv / psplit;
      // dt_raw of this row: wanted in 4, on its way meanwhile
      const float raw = wq == 0 ? __bfloat162float(p.dt_raw[(long long)(row0 + row) * p.dt_raw_stride + h]) : 0.f;
      const float Dh = p.D[h];
      float dti = 0.f, a_left = 0.f, a_right = 0.f;
      do {                                             // a wait that ran out leaves here: all warps meet at the barrier
        // ---- 1
        wait(a_full, it);
        if (!ok) break;
        const float li = s_l[row], lT = s_l[CT - 1];
        dti = s_dt[row]; a_left = __expf(li); a_right = __expf(lT - li);
        uint4 xrow[2], grow[2];
        #pragma unroll
        for (int q = 0; q < 2; ++q) {
          const uint32_t off = sw128_offset(row, wq * 2 + q);
          xrow[q] = *reinterpret_cast<const uint4*>(sX + off);
          grow[q] = *reinterpret_cast<const uint4*>(sDY + off);
        }
        if (it > 0) { wait(g_done, it - 1); if (!ok) break; }      // the products of the head before have read what follows
        #pragma unroll
        for (int q = 0; q < 2; ++q) {
          const uint32_t off = sw128_offset(row, wq * 2 + q);
          float f[8];
          unpack8(xrow[q], f);
          #pragma unroll
          for (int e = 0; e < 8; ++e) f[e] *= a_right * dti;
          *reinterpret_cast<uint4*>(sXs + off) = pack8(f);
          unpack8(grow[q], f);
          #pragma unroll
          for (int e = 0; e < 8; ++e) f[e] *= a_left;
          *reinterpret_cast<uint4*>(sDYs + off) = pack8(f);
        }
        wait(b_full, it);
        if (!ok) break;
        float dot_ss = 0.f;                  // share of <dS_out, S_in> (row n = `row`, 16 channels)
        #pragma unroll
        for (int q = 0; q < 2; ++q) {
          const uint32_t off = sw128_offset(row, wq * 2 + q);
          float f[8], f2[8];
          unpack8(*reinterpret_cast<const uint4*>(sSin + off), f);
          unpack8(*reinterpret_cast<const uint4*>(sDS + off), f2);
          #pragma unroll
          for (int e = 0; e < 8; ++e) dot_ss += f[e] * f2[e];
        }
        // ---- 2: row i of M0 and dCB, columns 32 wq .. + 31
        wait(s_done, it);
        if (!ok) break;
        if (it > 0) { wait(m0_free, it - 1); if (!ok) break; }
        float r1 = 0.f, col[2] = {0.f, 0.f};             // this thread's share of sum_{j<i} W[i][j]; column sums over the warp
        uint8_t* m_at = sM0 + (wq >> 1) * (TILE128 / 2);
        uint8_t* d_at = sDCB + (wq >> 1) * (TILE128 / 2);
        if (wq > rw) {                                   // tokens j > i for every row of this warp
          #pragma unroll
          for (int ch = 0; ch < 4; ++ch) {
            const uint32_t off = sw128_offset(row, (wq & 1) * 4 + ch);
            *reinterpret_cast<uint4*>(m_at + off) = make_uint4(0, 0, 0, 0);
            *reinterpret_cast<uint4*>(d_at + off) = make_uint4(0, 0, 0, 0);
          }
        } else {
          #pragma unroll
          for (int half = 0; half < 2; ++half) {
            uint32_t cb[16], dm[16];
            float wv[16];
            tmem_ld16(tmem_addr(tmem, lanes, wq * 32 + half * 16), cb);
            tmem_ld16(tmem_addr(tmem, lanes, 128 + wq * 32 + half * 16), dm);
            tmem_ld_wait();
            #pragma unroll
            for (int ch = 0; ch < 2; ++ch) {
              const int j0 = wq * 32 + half * 16 + ch * 8;
              float lv[8], dv[8], m0[8], dc[8];
              load8f_smem(s_l + j0, lv);
              load8f_smem(s_dt + j0, dv);
              #pragma unroll
              for (int e = 0; e < 8; e += 2) {
                const int i = ch * 8 + e;
                float lam0, lam1;
                unpack2(exp_diff2(pack2(li, li), pack2(lv[e], lv[e + 1])), lam0, lam1);
                if (wq == rw) {                        // the diagonal block
                  lam0 = half * 16 + i <= lane ? lam0 : 0.f;
                  lam1 = half * 16 + i + 1 <= lane ? lam1 : 0.f;
                }
                const uint64_t lam = pack2(lam0, lam1);
                const uint64_t mm = mul2(pack2(__uint_as_float(cb[i]), __uint_as_float(cb[i + 1])), lam);
                const uint64_t dd = mul2(pack2(__uint_as_float(dm[i]), __uint_as_float(dm[i + 1])), pack2(dv[e], dv[e + 1]));
                unpack2(mm, m0[e], m0[e + 1]);
                unpack2(mul2(dd, lam), dc[e], dc[e + 1]);
                // W[i][j] = dM[i][j] * (CB Lambda dt_j)[i][j], strictly below the diagonal
                unpack2(mul2(dd, mm), wv[i], wv[i + 1]);
                if (wq == rw) {
                  wv[i] = half * 16 + i < lane ? wv[i] : 0.f;
                  wv[i + 1] = half * 16 + i + 1 < lane ? wv[i + 1] : 0.f;
                }
              }
              const uint32_t off = sw128_offset(row, (wq & 1) * 4 + half * 2 + ch);
              *reinterpret_cast<uint4*>(m_at + off) = pack8(m0);
              *reinterpret_cast<uint4*>(d_at + off) = pack8(dc);
            }
            #pragma unroll
            for (int e = 0; e < 16; ++e) r1 += wv[e];
            // column sums over the warp's rows: recursive halving, lanes l and l + 16 end with column l
            #pragma unroll
            for (int sft = 8; sft >= 1; sft >>= 1) {
              const bool up = (lane & sft) != 0;
              #pragma unroll
              for (int k = 0; k < sft; ++k) {
                const float keep = up ? wv[k + sft] : wv[k];
                const float send = up ? wv[k] : wv[k + sft];
                wv[k] = keep + __shfl_xor_sync(0xffffffffu, send, sft);
              }
            }
            col[half] = wv[0] + __shfl_xor_sync(0xffffffffu, wv[0], 16);
          }
        }
        arrive(ops_ready);
        // ---- 3: row j, 16 channels
        wait(u_done, it);
        if (!ok) break;
        float ddt_direct = 0.f, r2 = 0.f, q = 0.f, dD = 0.f;
        {
          uint32_t ud[16], us[16], yo[16];
          tmem_ld16(tmem_addr(tmem, lanes, wq * 16), ud);
          tmem_ld16(tmem_addr(tmem, lanes, 64 + wq * 16), us);
          tmem_ld16(tmem_addr(tmem, lanes, 128 + wq * 16), yo);
          tmem_ld_wait();
          #pragma unroll
          for (int ch = 0; ch < 2; ++ch) {
            float xv[8], gy[8], o[8];
            unpack8(xrow[ch], xv);
            unpack8(grow[ch], gy);
            #pragma unroll
            for (int e = 0; e < 8; ++e) {
              const float usr = __uint_as_float(us[ch * 8 + e]);
              const float dU = __uint_as_float(ud[ch * 8 + e]) + a_right * usr;
              ddt_direct += xv[e] * dU;
              q += xv[e] * usr;
              r2 += gy[e] * __uint_as_float(yo[ch * 8 + e]);
              dD += gy[e] * xv[e];
              o[e] = dti * dU + Dh * gy[e];
            }
            *reinterpret_cast<uint4*>(sM0 + sw128_offset(row, wq * 2 + ch)) = pack8(o);      // M0 is dead
          }
        }
        if (lane < 16) {
          s_col[rw * CT + wq * 32 + lane] = col[0];
          s_col[rw * CT + wq * 32 + 16 + lane] = col[1];
        }
        s_part[wq * CT + row] = r1;
        s_part[(4 + wq) * CT + row] = ddt_direct;
        s_part[(8 + wq) * CT + row] = r2;
        s_part[(12 + wq) * CT + row] = q;
        // E = exp(l_T) <dS_out, S_in> + sum_j a_right dt_j q_j
        const float e_share = warp_sum128(__expf(lT) * dot_ss + a_right * dti * q), d_share = warp_sum128(dD);
        if (lane == 0) { s_red[warp] = e_share; s_red[16 + warp] = d_share; }
      } while (false);
      ok = all_ok(ok);
      if (!ok) break;
      if (wq != 0) { arrive(e_done); continue; }
      // ---- 4
      float E = 0.f;
      #pragma unroll
      for (int k = 0; k < 16; ++k) E += s_red[k];
      float sum[4], c1 = 0.f;
      #pragma unroll
      for (int i = 0; i < 4; ++i) {
        sum[i] = (s_part[i * 4 * CT + row] + s_part[(i * 4 + 1) * CT + row]) + (s_part[(i * 4 + 2) * CT + row] + s_part[(i * 4 + 3) * CT + row]);
        c1 += s_col[i * CT + row];
      }
      arrive(e_done);                                  // nothing of M0 is read after this
      // suffix sum of dl over the 128 rows
      float suf = sum[0] + a_left * sum[2] - c1 - a_right * dti * sum[3];
      #pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float n = __shfl_down_sync(0xffffffffu, suf, o);
        if (lane + o < 32) suf += n;
      }
      if (lane == 0) s_red[32 + rw] = suf;
      asm volatile("bar.sync 2, 128;" ::: "memory");
      float tail = 0.f;
      for (int w = rw + 1; w < 4; ++w) tail += s_red[32 + w];
      const float da = suf + tail + E;
      const float ddt = sum[1] + p.A[h] * da;
      const float ddr = ddt * sigmoid_f(raw + p.dt_bias[h]);
      if (p.ddt32 != nullptr) p.ddt32[((long long)b * p.Hv + hv) * p.L + (long long)c * CT + row] = ddr;
      else p.ddt_raw[(long long)(row0 + row) * p.ddt_stride + h] = __float2bfloat16(ddr);
      const float a_share = warp_sum128(dti * da), b_share = warp_sum128(ddr);
      if (lane == 0) { s_red[36 + rw] = a_share; s_red[40 + rw] = b_share; }
      asm volatile("bar.sync 2, 128;" ::: "memory");
      if (tid == 0) {
        float sD = 0.f;
        #pragma unroll
        for (int k = 0; k < 16; ++k) sD += s_red[16 + k];
        float* hp = p.hpart + (((long long)b * p.nc + c) * p.Hv + hv) * 3;
        hp[0] = s_red[36] + s_red[37] + s_red[38] + s_red[39];
        hp[1] = sD;
        hp[2] = s_red[40] + s_red[41] + s_red[42] + s_red[43];
      }
    }
    // ---- dB (quarters 0, 1) and dC (2, 3): 64 columns each, staged where C .. dS_out were
    if (ok) wait(g_done, p.hpc - 1);
    if (ok) {
      #pragma unroll 1
      for (int i = 0; i < 2; ++i) {
        uint32_t v[32];
        tmem_ld32(tmem_addr(tmem, lanes, 256 + wq * 64 + i * 32), v);
        tmem_ld_wait();
        uint8_t* blk = smem + (wq * 2 + i) * TILE64;   // [128 rows][32 fp32]
        #pragma unroll
        for (int k4 = 0; k4 < 8; ++k4)
          *reinterpret_cast<uint4*>(blk + sw128_offset(row, k4)) = make_uint4(v[k4 * 4], v[k4 * 4 + 1], v[k4 * 4 + 2], v[k4 * 4 + 3]);
      }
    }
    fence_proxy_async_smem();
    ok = all_ok(ok);
    if (tid == 0 && ok) {
      for (int k = 0; k < 8; ++k)
        if (splits > 1) tma_add_2d(&tm_dbc, smem + k * TILE64, (k >> 2) * GN + g * NS + (k & 3) * 32, row0);
        else tma_store_2d(&tm_dbc, smem + k * TILE64, (k >> 2) * GN + g * NS + (k & 3) * 32, row0);
      tma_store_commit();
      tma_store_wait_all();
    }
    tc_fence_before_sync();
  }
  __syncthreads();
  if (warp == 16) tmem_dealloc(tmem, 512);
}

}  // namespace ssm

// ------------------------------------------------------------------------------------ C API
using namespace ssm;

// A, D, dt_bias, mask, params_out: see HeadParams
extern "C" int ssm_ssd_dt_prep(const void* dt_raw, long long row_stride, const void* dt_bias, const void* A, const void* D,
                               int mask, void* params_out, void* dt_out, void* l_out, int B, int L, int H, cudaStream_t st) {
  if (L % CT || row_stride % 8 || (reinterpret_cast<uintptr_t>(dt_raw) & 15)) return -SSM_ERR_BAD_ARG;
  const DtPrep p{reinterpret_cast<const __nv_bfloat16*>(dt_raw), row_stride, {A, D, dt_bias, mask, reinterpret_cast<float*>(params_out)},
                 reinterpret_cast<float*>(dt_out), reinterpret_cast<float*>(l_out), L, H};
  ssd_dt_prep_kernel<<<dim3(L / CT, (H + DT_HEADS - 1) / DT_HEADS, B), DT_CHUNK, 0, st>>>(p);
  return (int)cudaGetLastError();
}

// w_src: bf16 [B*L, w_cols] (row stride w_stride) holding W (B or C of every group) starting at column w_col0.
// v: bf16 rows (b*L+t)*v_stride + hv*64.   out fp32 [B,Hv,nc,128,64].
extern "C" int ssm_ssd_chunk_state(const void* w_src, long long w_stride, int w_cols, int w_col0, const void* v,
                                   long long v_stride, const void* dt, const void* l, void* out, int B, int L, int H,
                                   int Hv, int G, int mode, int* status, cudaStream_t st) {
  if (L % CT || Hv % H || H % G || w_stride % 8 || v_stride % 8) return -SSM_ERR_BAD_ARG;
  const int smem = TILE128 + TILE64 + 64 + 1024;
  static SmemOptIn opt_in;
  if (const int e = opt_in.ask(reinterpret_cast<const void*>(ssd_chunk_state_kernel), smem)) return e;
  CUtensorMap tm;
  int r = make_tmap_2d_bf16(&tm, w_src, (uint64_t)w_cols, (uint64_t)B * L, (uint64_t)w_stride * 2, 64, 128);
  if (r) return -100 - r;
  ChunkStateParams p;
  p.v = reinterpret_cast<const __nv_bfloat16*>(v); p.v_row_stride = v_stride;
  p.dt = reinterpret_cast<const float*>(dt); p.l = reinterpret_cast<const float*>(l);
  p.out = reinterpret_cast<float*>(out);
  p.L = L; p.H = H; p.Hv = Hv; p.G = G; p.nc = L / CT; p.w_col0 = w_col0; p.mode = mode; p.status = status;
  dim3 grid(L / CT, Hv, B);
  ssd_chunk_state_kernel<<<grid, 128, smem, st>>>(tm, p);
  return (int)cudaGetLastError();
}

extern "C" int ssm_ssd_state_pass(const void* local, const void* l, const void* init, void* in16, void* fin, int B,
                                  int L, int H, int Hv, int reverse, cudaStream_t st) {
  dim3 grid(NS * PS / 4 / 256, Hv, B);
  ssd_state_pass_kernel<<<grid, 256, 0, st>>>(reinterpret_cast<const float*>(local), reinterpret_cast<const float*>(l),
                                              reinterpret_cast<const float*>(init),
                                              reinterpret_cast<__nv_bfloat16*>(in16), reinterpret_cast<float*>(fin), L,
                                              H, Hv, L / CT, reverse);
  return (int)cudaGetLastError();
}

// `count` segments cover the nc chunks; the buffers are wanted for more than one
static bool segments_ok(int nc, int count, const void* fin, const void* decay, Segments* sg) {
  if (count < 1 || count > nc || count > 64 || (count > 1 && (fin == nullptr || decay == nullptr || (reinterpret_cast<uintptr_t>(fin) & 15))))
    return false;
  sg->count = count; sg->len = (nc + count - 1) / count;
  sg->fin = reinterpret_cast<float*>(const_cast<void*>(fin)); sg->decay = reinterpret_cast<float*>(const_cast<void*>(decay));
  return (count - 1) * sg->len < nc;               // none is empty
}

// Backwards (forward = 0): mode 1 of ssm_ssd_chunk_state (w_src: C) and ssm_ssd_state_pass in one; v: bf16 [B*L, Hv*64] (row
// stride v_stride); in16 bf16 [B,Hv,nc,128,64] is written.  Without in16: the states behind the first `count` - 1 segments
// from zero states, seg_fin fp32 [B,Hv,count,128,64] and seg_decay fp32 [B,Hv,count], either way (forward: w_src B, v x).
extern "C" int ssm_ssd_state_walk(const void* w_src, long long w_stride, int w_cols, int w_col0, const void* v, long long v_stride,
                                  const void* dt, const void* l, void* in16, int B, int L, int H, int Hv, int G, int forward,
                                  int count, void* seg_fin, void* seg_decay, int* status, cudaStream_t st) {
  Segments sg;
  if (L % CT || Hv % H || H % G || w_stride % 8 || v_stride % 8 || B < 1 || B > 65535 || (forward && (in16 != nullptr || dt == nullptr)) ||
      !segments_ok(L / CT, count, seg_fin, seg_decay, &sg) || (in16 == nullptr && count < 2))
    return -SSM_ERR_BAD_ARG;
  static SmemOptIn opt_in;
  if (const int e = opt_in.ask(reinterpret_cast<const void*>(ssd_state_walk_kernel), WALK_SMEM)) return e;
  const int nc = L / CT;
  CUtensorMap tw, tv, ti;
  int r = make_tmap_2d_bf16(&tw, w_src, (uint64_t)w_cols, (uint64_t)B * L, (uint64_t)w_stride * 2, 64, 128);
  if (r) return -100 - r;
  r = make_tmap_2d_bf16(&tv, v, (uint64_t)Hv * PS, (uint64_t)B * L, (uint64_t)v_stride * 2, 64, 128);
  if (r) return -200 - r;
  ti = tv;
  if (in16 != nullptr) r = make_tmap_2d_bf16(&ti, in16, 64, (uint64_t)B * Hv * nc * NS, 128, 64, 128);
  if (r) return -300 - r;
  StateWalkParams p;
  p.dt = reinterpret_cast<const float*>(dt); p.l = reinterpret_cast<const float*>(l);
  p.L = L; p.H = H; p.Hv = Hv; p.G = G; p.nc = nc; p.w_col0 = w_col0; p.status = status;
  p.forward = forward; p.finals = in16 == nullptr; p.seg = sg;
  ssd_state_walk_kernel<<<dim3(Hv, B, p.finals ? count - 1 : count), 256, WALK_SMEM, st>>>(tw, tv, ti, p);
  return (int)cudaGetLastError();
}

// The whole forward scan.  xbc as in ssm_ssd_chunk_scan_fwd; s_in (bf16 [B,Hv,nc,128,64], written) or null; init fp32
// [B,Hv,128 n,64 p] and fin fp32 [B,Hv,64 p,128 n] are optional; y as in ssm_ssd_chunk_scan_fwd; more than one segment wants
// what ssm_ssd_state_walk left in seg_fin and seg_decay.
extern "C" int ssm_ssd_walk_scan(const void* xbc, long long xbc_stride, int xbc_cols, void* s_in, void* y, long long y_stride,
                                 const void* dt, const void* l, const void* D, const void* init, void* fin, int B, int L,
                                 int H, int Hv, int G, int d_in, int count, const void* seg_fin, const void* seg_decay, int* status,
                                 cudaStream_t st) {
  Segments sg;
  if (L % CT || Hv % H || H % G || xbc_stride % 8 || y_stride % 8 || B < 1 || B > 65535 ||
      !segments_ok(L / CT, count, seg_fin, seg_decay, &sg) ||
      ((reinterpret_cast<uintptr_t>(dt) | reinterpret_cast<uintptr_t>(l)) & 15))
    return -SSM_ERR_BAD_ARG;
  static SmemOptIn opt_in;
  if (const int e = opt_in.ask(reinterpret_cast<const void*>(ssd_walk_scan_kernel), WS_SMEM)) return e;
  const int nc = L / CT;
  CUtensorMap tx, ts, ty;
  int r = make_tmap_2d_bf16(&tx, xbc, (uint64_t)xbc_cols, (uint64_t)B * L, (uint64_t)xbc_stride * 2, 64, 128);
  if (r) return -100 - r;
  ts = tx;
  if (s_in != nullptr) r = make_tmap_2d_bf16(&ts, s_in, 64, (uint64_t)B * Hv * nc * NS, 128, 64, 128);
  if (r) return -200 - r;
  r = make_tmap_2d_bf16(&ty, y, (uint64_t)Hv * PS, (uint64_t)B * L, (uint64_t)y_stride * 2, 64, 128);
  if (r) return -300 - r;
  WalkScanParams p;
  p.dt = reinterpret_cast<const float*>(dt); p.l = reinterpret_cast<const float*>(l);
  p.D = reinterpret_cast<const float*>(D);
  p.init = reinterpret_cast<const float*>(init); p.fin = reinterpret_cast<float*>(fin);
  p.store_states = s_in != nullptr;
  p.L = L; p.H = H; p.Hv = Hv; p.G = G; p.nc = nc; p.d_in = d_in; p.status = status; p.seg = sg;
  ssd_walk_scan_kernel<<<dim3(Hv, B, count), WS_THREADS, WS_SMEM, st>>>(tx, ts, ty, p);
  return (int)cudaGetLastError();
}

// xbc: conv output bf16 [B*L, xbc_cols] (x | B | C), row stride xbc_stride.  s_in bf16 [B*Hv*nc*128, 64].
// y: bf16 [B*L, Hv*64] row stride y_stride (written).
extern "C" int ssm_ssd_chunk_scan_fwd(const void* xbc, long long xbc_stride, int xbc_cols, const void* s_in, void* y,
                                      long long y_stride, const void* dt, const void* l, const void* D, int B, int L,
                                      int H, int Hv, int G, int d_in, int* status, cudaStream_t st) {
  if (L % CT || Hv % H || H % G || xbc_stride % 8 || y_stride % 8) return -SSM_ERR_BAD_ARG;
  const int smem = 2 * TILE128 + 2 * TILE64 + 2 * CT * 4 + 64 + 1024;
  static SmemOptIn opt_in;
  if (const int e = opt_in.ask(reinterpret_cast<const void*>(ssd_chunk_scan_fwd_kernel), smem)) return e;
  const int nc = L / CT;
  CUtensorMap tx, ts, ty;
  int r = make_tmap_2d_bf16(&tx, xbc, (uint64_t)xbc_cols, (uint64_t)B * L, (uint64_t)xbc_stride * 2, 64, 128);
  if (r) return -100 - r;
  r = make_tmap_2d_bf16(&ts, s_in, 64, (uint64_t)B * Hv * nc * NS, 128, 64, 128);
  if (r) return -200 - r;
  r = make_tmap_2d_bf16(&ty, y, (uint64_t)Hv * PS, (uint64_t)B * L, (uint64_t)y_stride * 2, 64, 128);
  if (r) return -300 - r;
  ScanFwdParams p;
  p.dt = reinterpret_cast<const float*>(dt); p.l = reinterpret_cast<const float*>(l);
  p.D = reinterpret_cast<const float*>(D);
  p.L = L; p.H = H; p.Hv = Hv; p.G = G; p.nc = nc; p.d_in = d_in; p.status = status;
  dim3 grid(nc, Hv, B);
  ssd_chunk_scan_fwd_kernel<<<grid, 128, smem, st>>>(tx, ts, ty, p);
  return (int)cudaGetLastError();
}

// dy: bf16 [B*L, Hv*64] (row stride dy_stride).  dx: bf16 [B*L, Hv*64] written (row stride dx_stride).
// dBC: fp32 [B*L, 2*G*128], written whole.  hpart: fp32 [B*nc, Hv, 3].
// ddt: if ddt32 != null it receives fp32 [B,Hv,L]; else bf16 values are written to ddt_raw rows.
extern "C" int ssm_ssd_chunk_scan_bwd(const void* xbc, long long xbc_stride, int xbc_cols, const void* dy,
                                      long long dy_stride, const void* s_in,
                                      const void* ds_out, void* dx, long long dx_stride, void* dBC, void* hpart,
                                      void* ddt_raw, long long ddt_stride, void* ddt32, const void* dt_raw,
                                      long long dt_raw_stride, const void* dt_bias, const void* A, const void* dt,
                                      const void* l, const void* D, int B, int L, int H, int Hv, int G, int d_in,
                                      int hpc, int* status, cudaStream_t st) {
  if (L % CT || Hv % H || H % G || xbc_stride % 8 || dy_stride % 8 || dx_stride % 8 ||
      ((reinterpret_cast<uintptr_t>(dt) | reinterpret_cast<uintptr_t>(l) | reinterpret_cast<uintptr_t>(dBC)) & 15))
    return -SSM_ERR_BAD_ARG;
  const int hv_per_group = Hv / G;
  if (hpc <= 0 || hv_per_group % hpc) return -SSM_ERR_BAD_ARG;
  static SmemOptIn opt_in;
  if (const int e = opt_in.ask(reinterpret_cast<const void*>(ssd_chunk_scan_bwd_kernel), BWD_SMEM)) return e;
  const int nc = L / CT;
  CUtensorMap tx, tdy, ts, tds, tdx;
  int r = make_tmap_2d_bf16(&tx, xbc, (uint64_t)xbc_cols, (uint64_t)B * L, (uint64_t)xbc_stride * 2, 64, 128);
  if (r) return -100 - r;
  r = make_tmap_2d_bf16(&tdy, dy, (uint64_t)Hv * PS, (uint64_t)B * L, (uint64_t)dy_stride * 2, 64, 128);
  if (r) return -200 - r;
  r = make_tmap_2d_bf16(&ts, s_in, 64, (uint64_t)B * Hv * nc * NS, 128, 64, 128);
  if (r) return -300 - r;
  r = make_tmap_2d_bf16(&tds, ds_out, 64, (uint64_t)B * Hv * nc * NS, 128, 64, 128);
  if (r) return -400 - r;
  r = make_tmap_2d_bf16(&tdx, dx, (uint64_t)Hv * PS, (uint64_t)B * L, (uint64_t)dx_stride * 2, 64, 128);
  if (r) return -500 - r;
  CUtensorMap tdbc;
  r = make_tmap_2d(&tdbc, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, dBC, (uint64_t)2 * G * NS, (uint64_t)B * L, (uint64_t)2 * G * NS * 4, 32, 128);
  if (r) return -600 - r;
  ScanBwdParams p;
  p.dt = reinterpret_cast<const float*>(dt); p.l = reinterpret_cast<const float*>(l);
  p.D = reinterpret_cast<const float*>(D); p.A = reinterpret_cast<const float*>(A);
  p.dt_bias = reinterpret_cast<const float*>(dt_bias);
  p.dt_raw = reinterpret_cast<const __nv_bfloat16*>(dt_raw); p.dt_raw_stride = dt_raw_stride;
  p.ddt_raw = reinterpret_cast<__nv_bfloat16*>(ddt_raw); p.ddt_stride = ddt_stride;
  p.ddt32 = reinterpret_cast<float*>(ddt32);
  p.hpart = reinterpret_cast<float*>(hpart);
  p.L = L; p.H = H; p.Hv = Hv; p.G = G; p.nc = nc; p.d_in = d_in; p.hpc = hpc; p.status = status;
  if (hpc < hv_per_group) {                            // CTAs of a group add to it
    const cudaError_t e = cudaMemsetAsync(dBC, 0, (size_t)B * L * 2 * G * NS * sizeof(float), st);
    if (e != cudaSuccess) return (int)e;
  }
  dim3 grid(nc, G * (hv_per_group / hpc), B);
  ssd_chunk_scan_bwd_kernel<<<grid, BWD_THREADS, BWD_SMEM, st>>>(tx, tdy, ts, tds, tdx, tdbc, p);
  return (int)cudaGetLastError();
}
