// Whole pre-norm blocks over a full sequence, launched by one call.  No kernels of its own: at a few hundred tokens the kernels
// of a block take 3 to 8 us each and a launch from Python about 20, so the chain is put together here.
// 130M, one prompt of 128 tokens, 24 layers: 4717 us with ten launches per block from Python, 1380 to 1430 (830 of them kernels) so.
#include "common.cuh"

extern "C" {
int ssm_add_rmsnorm_fwd(const void*, const void*, const void*, void*, void*, long long, int, float, int, cudaStream_t);
int ssm_gemm_bf16(const void*, const void*, void*, int, int, int, long long, long long, long long, int, int, int, const void*, int,
                  int*, cudaStream_t);
int ssm_conv_dt(const void*, long long, const void*, const void*, void*, long long, const void*, const void*, const void*, const void*,
                int, void*, void*, void*, void*, int, int, int, int, cudaStream_t);
int ssm_ssd_state_walk(const void*, long long, int, int, const void*, long long, const void*, const void*, void*, int, int, int, int,
                       int, int, int, void*, void*, int*, cudaStream_t);
int ssm_ssd_walk_scan(const void*, long long, int, void*, void*, long long, const void*, const void*, const void*, const void*, void*,
                      int, int, int, int, int, int, int, const void*, const void*, int*, cudaStream_t);
int ssm_gated_rmsnorm_fwd(const void*, long long, const void*, long long, const void*, void*, long long, long long, int, int, float,
                          cudaStream_t);

struct BlockForward {                      // in the order in which cuda_ops.block_forward packs it
  const void *x, *res; void* res_out;      // bf16 [B L, D], residual type [B L, D] or null, residual type [B L, D]
  const void *norm_w, *in_w, *in_b, *conv_w, *conv_b, *A_log, *Dp, *dt_bias, *gate_w, *out_w;
  void *window, *final_state;              // bf16 [B, C, 4] and fp32 [B, H, P, 128], or null
  void *normed, *zx, *conv, *y;            // bf16 scratch [B L, max(D, d_in)], [B L, zx_ld], [B L, C], [B L, d_in]
  void *params, *dt, *l;                   // fp32 scratch [3, H], [B, H, L], [B, H, L]
  void *seg_fin, *seg_decay;               // fp32 scratch of more than one segment
  void* out;                               // bf16 [B L, D]
  int* status;
  long long zx_ld;
  int B, L, D, d_in, H, P, G, gs, res_fp32, bf16_mask, count;
  float eps_norm, eps_gate;
};

int ssm_block_forward(const BlockForward* a, cudaStream_t st) {
  const int N = 128, C = a->d_in + 2 * a->G * N, W = a->d_in + C + a->H, Hv = a->d_in / 64, rows = a->B * a->L;
  auto* zx = reinterpret_cast<__nv_bfloat16*>(a->zx);
  auto* params = reinterpret_cast<float*>(a->params);
  int r = ssm_add_rmsnorm_fwd(a->x, a->res, a->norm_w, a->normed, a->res_out, rows, a->D, a->eps_norm, a->res_fp32, st);
  if (!r) r = ssm_gemm_bf16(a->normed, a->in_w, zx, rows, W, a->D, a->D, a->D, a->zx_ld, 0, 0, 0, a->in_b, 0, a->status, st);
  if (!r) r = ssm_conv_dt(zx + a->d_in, a->zx_ld, a->conv_w, a->conv_b, a->conv, C, zx + a->d_in + C, a->dt_bias, a->A_log, a->Dp,
                          a->bf16_mask | 8, params, a->dt, a->l, a->window, a->B, a->L, C, a->H, st);
  if (!r && a->count > 1)
    r = ssm_ssd_state_walk(a->conv, C, C, a->d_in, a->conv, C, a->dt, a->l, nullptr, a->B, a->L, a->H, Hv, a->G, 1, a->count, a->seg_fin,
                           a->seg_decay, a->status, st);
  if (!r) r = ssm_ssd_walk_scan(a->conv, C, C, nullptr, a->y, a->d_in, a->dt, a->l, params + a->H, nullptr, a->final_state, a->B, a->L,
                                a->H, Hv, a->G, a->d_in, a->count, a->seg_fin, a->seg_decay, a->status, st);
  if (!r) r = ssm_gated_rmsnorm_fwd(a->y, a->d_in, zx, a->zx_ld, a->gate_w, a->normed, a->d_in, rows, a->d_in, a->gs, a->eps_gate, st);
  if (!r) r = ssm_gemm_bf16(a->normed, a->out_w, a->out, rows, a->D, a->d_in, a->d_in, a->d_in, a->D, 0, 0, 0, nullptr, 0, a->status, st);
  return r;
}
}
