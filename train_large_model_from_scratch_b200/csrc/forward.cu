// Forward pass of a run of dense transformer blocks without gradients, issued by one call.
//
// The kernels are the ones the per-op path launches; what goes away is the host work between them (an autograd node, a
// handful of allocations and a foreign-function call each: about 30 us per kernel, where a 333-token prompt keeps the GPU
// busy for 9 us per kernel) and, with no backward to come, the store of gate | up.
#include "common.cuh"

using namespace tlm;

TLM_API int tlm_add_rmsnorm_fwd(const float* x, const void* delta, const void* w, float* x_new, void* h, float* rstd, int rows,
                                int D, float eps, cudaStream_t st);
TLM_API int tlm_gemm_heads(const void* A, const void* B, int M, int N, int K, long long lda, long long ldb, int b_mn,
                           void* const* dst_ptrs, int n_dst, int batch, int rows_per_batch, int dst_rows, int dst_heads,
                           int row_off, int Hq, int Hkv, int q_l, int kv_l, int hd, int n_rot, const void* cs, int kv_rep,
                           const float* cosT, const float* sinT, cudaStream_t stream);
TLM_API int tlm_attn_fwd(const void* qkv, void* o, float* lse, int B, int T, int Hq, int Hkv, int hd, float scale, cudaStream_t st);
TLM_API int tlm_gemm(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb, long long ldc,
                     int a_mn, int b_mn, int epi, cudaStream_t stream);
TLM_API int tlm_gemm_swiglu(const void* x, const void* w_gu, void* gate_up, void* act, int M, int I, int K, long long lda,
                            long long ldb, cudaStream_t stream);

// `layers`: six weights per block (first norm, q|k|v projection, output projection, second norm, gate|up, down), bf16,
// contiguous. x: residual stream [B T, D] fp32, not written. xa / xb: two more of its size; on return the residual stream
// is in xa and `delta` [B T, D] bf16 holds the last branch output, not added yet. h [B T, D], qkv [B T, (Hq + 2 Hkv) hd],
// o [B T, D], act [B T, I] bf16 and lse [B Hq T], rstd [B T] fp32 are scratch. cs / cosT / sinT: see tlm_gemm_heads.
// Returns the first error code; what was launched before it stays launched.
TLM_API int tlm_blocks_forward(const void* const* layers, int n_layers, const float* x, float* xa, float* xb, void* delta, void* h,
                               void* qkv, void* o, void* act, float* lse, float* rstd, int B, int T, int D, int Hq, int Hkv,
                               int hd, int I, float eps, float scale, const void* cs, const float* cosT, const float* sinT,
                               cudaStream_t st) {
  const int M = B * T, Ht = Hq + 2 * Hkv;
  if (n_layers <= 0 || layers == nullptr || D != Hq * hd) return -6;
  const float* cur = x;
  void* dst[1] = {qkv};
  int e = 0;
  for (int l = 0; l < n_layers; ++l) {
    const void* const* w = layers + 6 * l;
    // the residual stream alternates: xa after a block's second norm, xb after the next block's first
    if (l == 0) e = tlm_add_rmsnorm_fwd(cur, nullptr, w[0], const_cast<float*>(cur), h, rstd, M, D, eps, st);   // nothing to add: x is not stored
    else { e = tlm_add_rmsnorm_fwd(cur, delta, w[0], xb, h, rstd, M, D, eps, st); cur = xb; }
    if (e) return e;
    if ((e = tlm_gemm_heads(h, w[1], M, Ht * hd, D, D, D, 0, dst, 1, B, T, T, Ht, 0, Hq, Hkv, Hq, Hkv, hd, Hq + Hkv, cs, 1, cosT, sinT, st))) return e;
    if ((e = tlm_attn_fwd(qkv, o, lse, B, T, Hq, Hkv, hd, scale, st))) return e;
    if ((e = tlm_gemm(o, w[2], delta, M, D, D, D, D, D, 0, 0, 0, st))) return e;
    if ((e = tlm_add_rmsnorm_fwd(cur, delta, w[3], xa, h, rstd, M, D, eps, st))) return e;
    cur = xa;
    if ((e = tlm_gemm_swiglu(h, w[4], nullptr, act, M, I, D, D, D, st))) return e;
    if ((e = tlm_gemm(act, w[5], delta, M, D, I, I, I, D, 0, 0, 0, st))) return e;
  }
  return 0;
}
