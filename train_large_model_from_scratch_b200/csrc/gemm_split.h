// GEMMs whose 256-wide tiles cannot fill the chip: small tiles, the reduction split over a cluster (gemm_split.cu).
#pragma once

#include <cuda_runtime.h>

namespace tlm {

enum SplitEpilogue { SPLIT_BF16 = 0, SPLIT_F32_ACC = 1, SPLIT_HEADS = 3, SPLIT_SWIGLU = 4, SPLIT_SWIGLU_BWD = 5 };

struct SplitGemm {
  const void* A;                 // [M, K] (pitch lda), or [K, M] when a_mn
  const void* B;                 // [N, K] (pitch ldb), or [K, N] when b_mn; SPLIT_SWIGLU: [2 N, K], gate rows then up rows
  int M, N, K;                   // SPLIT_SWIGLU: N = columns of act
  long long lda, ldb;
  bool a_mn, b_mn;
  int epi;
  void* C;                       // bf16 or fp32 result (pitch ldc); SwiGLU: gate|up (or null) / d(gate)|d(up), pitch ldc = 2 N
  long long ldc;
  void* act;                     // SPLIT_SWIGLU: silu(gate) * up, [M, N]
  const void* aux;               // SPLIT_SWIGLU_BWD: gate|up, [M, 2 N]
  // SPLIT_HEADS: columns are heads of hd columns, rows are [batch][rows_per_batch]; C is [batch, dst_rows, dst_heads, hd],
  // head h of row (b, t) goes to C[b, row_off + t, h, :]; heads below n_rot are rotated with the fp32 tables [rows_per_batch, hd]
  int hd, rows_per_batch, dst_rows, dst_heads, row_off, n_rot;
  const float* cosT;
  const float* sinT;
};

struct SplitPlan { int bn, split; };          // tile width (64 / 128), CTAs that share one tile's reduction; bn == 0: not this path

// The plan for a product of that size, or bn == 0 where the 256-wide tiles of gemm.cu are faster: they would take `wide_us`.
SplitPlan split_plan(const SplitGemm& g, double wide_us);
int split_run(const SplitGemm& g, const SplitPlan& plan, cudaStream_t st);

}  // namespace tlm
