// Which products run on the small tiles of gemm_split.cu and on which plan (estimated times), and how far a GEMM reads ahead:
// without device code, so that a host test can walk over sizes (tests/test_gemm_cost_cpu.py).
#pragma once

#ifdef __CUDACC__
#define TLM_COST_HD __host__ __device__ __forceinline__
#else
#define TLM_COST_HD inline
#endif

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

// End of the part of a block's reduction [lo, hi) whose weights are asked for while the kernel in front still runs (few rows: the
// weights are the larger operand and come out of memory). What the ring takes first, six k-blocks of 64; over the whole chip that
// is 28 MB, which L2 keeps until it is read. The whole reduction instead (786 k-blocks of an LM head's data gradient, up to 309 MB)
// put the first loads behind thousands of requests and read lines twice: 1024 x 1024, K 50304 291 us, 235 this way and without;
// 333 x 1024 82, 64 and 64; 333 x 3072 300, 234 and 234. Logits of prompts whose weights do not stay in L2, without -> six
// k-blocks (twelve gave the same): 10 layers of 2048, 32 rows 716 -> 696 us; 16 of 768, 329 rows 790 -> 780; 8 of 2048, 200 rows
// 656 -> 644; 12 of 1024, 333 rows 672 -> 669.
constexpr int WEIGHTS_AHEAD = 6 * 64;
TLM_COST_HD constexpr int weights_ahead_end(int lo, int hi) { return hi - lo > WEIGHTS_AHEAD ? lo + WEIGHTS_AHEAD : hi; }

// Estimated time (us) of a product on the wide tiles of gemm.cu, `tile_m` x `tile_n` outputs each, taken by `walkers`:
// 5.4 us around the main loops (fp32 accumulation 7.2), 0.28 us per k-block of a tile, one wave of tiles after another.
inline double wide_rule(int M, int N, int tile_m, int tile_n, int K, int walkers, int splits) {
  const long long items = (long long)((M + tile_m - 1) / tile_m) * ((N + tile_n - 1) / tile_n) * (splits > 0 ? splits : 1);
  return (splits > 0 ? 7.2 : 5.4) + (double)((items + walkers - 1) / walkers) * ((K + 63) / 64) * 0.28;
}

// Estimated time in us, fitted to 380 products (M 1 - 8192, N 256 - 50304, K 8 - 8000; every plan and the wide tiles timed with
// operands in L2 and with weights and gradients out of memory). A k-block takes 0.24 us (64 columns, four stages) or 0.33 us
// (128 columns: 0.27 out of L2, 0.36 where three stages are not enough for the latency of memory: 966 x 1536, K 6784 took 41.5 us
// on 128 columns, 33.7 on 64, 35.9 on wide tiles) of a CTA, and no less than all CTAs' blocks take at 17.6 TB/s out of the whole
// L2 (7.5 TB/s when the operands do not stay in it: 2560 x 512, K 50304 on 80 CTAs took 273 us against 224 us on wide tiles),
// 1.3 times as long when the rows of a K-major operand do not start on 128-byte lines (2436 x 512, K 1384: 16.4 us, wide tiles
// 14.5); plus what surrounds the main loop and the exchange of the partial tiles. Few rows: when all of A is less than 128 KB, its
// lines come from too few places in L2, and the CTAs wait for each other there, 3.5 ns each per k-block (6000 gate | up columns,
// K 2048, on 188 CTAs: 28 us at 24 rows, 12.3 us at 32; wide tiles 14.8). A weight gradient's C is read and written by the
// reductions, 4 bytes at 6.5 TB/s (1024 x 3872, K 80: 9.1 us, wide tiles 7.7), and has to win clearly: the wide tiles add
// whole TMA boxes.
// The figures are those of rings of three and four stages and of MMAs issued by one lane. With deep rings (launch_split) a plan that
// has its SMs to itself takes up to a quarter less than estimated, so some products stay on wide tiles that a plan would now beat
// (1024 x 1024, K 50304: 225 us, 163 on two CTAs per 128-wide tile). 520 random products take 0.910 of the time that they took then.
// A plan also fixes the order in which a result's fp32 sums are added: other figures here give other last bits.
inline SplitPlan split_rule(const SplitGemm& g, double wide_us, int sms) {
  SplitPlan best{0, 0};
  const long long kblocks = (g.K + 63) / 64, slots = 2LL * sms;
  const double operand_bytes = 2.0 * g.K * ((double)g.M + (g.epi == SPLIT_SWIGLU ? 2.0 : 1.0) * g.N);
  const double lines = (!g.a_mn && g.lda % 64 != 0) || (!g.b_mn && g.ldb % 64 != 0) ? 1.3 : 1.0;
  const double l2_rate = operand_bytes > 64e6 ? 7.5e6 : 17.6e6;        // bytes per us
  const double per_cta = !g.a_mn && 2.0 * g.M * g.K < 131072.0 ? 0.0035 : 0.0;
  const double c_us = g.epi == SPLIT_F32_ACC ? 4.0 * g.M * g.N / 6.5e6 : 0.0;
  static const double exchange[2][4] = {{0.0, 1.5, 1.3, 2.8}, {0.0, 2.2, 2.0, 2.3}};       // S = 1, 2, 4, 8
  double best_us = (g.epi == SPLIT_F32_ACC ? 0.85 : 0.95) * wide_us;
  for (int bn = 64; bn <= 128; bn *= 2) {
    if (g.epi == SPLIT_HEADS && (g.hd > bn || bn % g.hd != 0)) continue;
    const int tile_n = g.epi == SPLIT_SWIGLU ? bn / 2 : bn;
    const long long tiles = (long long)((g.M + 127) / 128) * ((g.N + tile_n - 1) / tile_n);
    for (int i = 0, s = 1; s <= 8 && s <= kblocks; ++i, s *= 2) {
      const long long ctas = tiles * s, resident = ctas < slots ? ctas : slots;
      if (ctas > (s > 1 ? sms : slots)) continue;          // a second wave of clusters costs more than it saves
      double block = bn == 64 ? 0.24 : 0.33;
      const double shared = (double)resident * (bn == 64 ? 24576.0 : 32768.0) / l2_rate, queue = (double)resident * per_cta;
      if (shared > block) block = shared;
      if (queue > block) block = queue;
      const double us = (bn == 64 ? 3.4 : 3.8) + (g.a_mn ? 1.0 : 0.0) + exchange[bn / 128][i] + c_us +
                        (double)((kblocks + s - 1) / s) * lines * block;
      if (us < best_us) { best_us = us; best = {bn, s}; }
    }
  }
  return best;
}

}  // namespace tlm
