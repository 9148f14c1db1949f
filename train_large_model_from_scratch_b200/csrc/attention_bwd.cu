// Causal GQA flash attention, backward, on tcgen05 / TMEM.
//
// Inputs: packed qkv[B,T,Hq+2Hkv,hd], o[B,T,Hq,hd], do[B,T,Hq,hd] (bf16),
// lse[B,Hq,T] (fp32). Output: dqkv[B,T,Hq+2Hkv,hd] (bf16) in the packed layout,
// so the QKV projection's dgrad/wgrad GEMMs consume one tensor.
//
// Three launches:
//   1. delta[b,h,t] = sum_d do*o; the dQ accumulator is zeroed on the way (few rows: by a memset)
//   2. main kernel: one CTA per (128-row KV tile, batch, KV head). The CTA walks over every query head of the group and
//      every query tile at or below the diagonal. Per step five products run on the tensor cores, scores transposed:
//                      S^T = K Q^T,  dP^T = V dO^T       (TMEM, fp32; rows = keys, columns = queries)
//                      dV += P^T dO,  dK += dS^T Q       (TMEM accumulators; P^T / dS^T are TMEM operands)
//                      dQ  = dS K                        (TMEM, flushed per step)
//      so P never leaves tensor memory and only dS goes through shared memory, as the [kv][q] bf16 tile that dQ reads
//      MN-major. Q / dO / K / V tiles are used as loaded.
//      Warps: 0 loads (Q, dO by TMA; -lse log2 e and -delta of the step's rows by the warp), 1 issues the products,
//      2 - 17 softmax (32 keys x 32 queries each: P, dS), 18 - 21 take dQ out: tiles are added to an fp32 buffer with TMA
//      reduce-add tile stores because several KV tiles contribute to one query row.
//      With few KV tiles a cluster of CTAs shares a tile's steps (SPLIT, see split_for).
//   3. dq (fp32, [B,Hq,T,hd]) -> bf16 into dqkv; with RoPE tables this pass also applies the transposed rotation to
//      dQ (from the fp32 accumulator) and to the dK slots the main kernel wrote, so the packed gradient that leaves
//      is the gradient of the UN-rotated q and k and no separate RoPE pass runs.
// A second instantiation of the main kernel (SCATTER) serves Ulysses sequence parallelism: its dK / dV epilogue
// rotates dK itself and stores the rows straight into the sequence owners' packed gradient buffers, and the
// conversion pass does the same for dQ.
// Every wait is bounded; on a timeout the CTA records a status code, leaves its
// loops and still releases its tensor memory.
#include "common.cuh"
#include <cstdlib>

namespace tlm {

constexpr int AB_TILE = 128, AB_THREADS = 704, AB_MAX_DST = 8;

struct AttnBwdDst {
  __nv_bfloat16* p[AB_MAX_DST];
  int n, rows, heads;
};

struct AttnBwdParams {
  __nv_bfloat16* dqkv;
  float* dq_acc;            // [B,Hq,T,hd] fp32, zeroed before the main kernel
  const __nv_bfloat16* qkv;
  const float* lse;
  const float* delta;
  int B, T, Hq, Hkv;
  float scale, scale_log2;
  unsigned int* status;
  int hd;                   // head dim in memory; the SCATTER form runs 32 on its HD = 64 kernel with zero-filled upper columns
  // Transposed RoPE on the way out (tables cos / sin [T, hd], fp32, row = position; nullptr: off):
  //   dx[j] = dy[j] c[j] + dy[j+h] s[j+h],  dx[j+h] = dy[j+h] c[j+h] - dy[j] s[j]   (h = hd / 2).
  const float* cosT;
  const float* sinT;
  // SCATTER instantiation only: head -> sequence return of the packed gradient (Ulysses backward). Row t of local
  // head slot s is stored into
  //   dst[t / dst_rows][b, t % dst_rows, head(s), :]     (bf16 [B, dst_rows, dst_heads, hd] per rank)
  // with head(s) = dst_q0 + s for q slots, dst_k0 + s for k, dst_v0 + s for v (peer-mapped addresses, plain
  // 16-byte stores).
  __nv_bfloat16* dst[AB_MAX_DST];
  int n_dst, dst_rows, dst_heads, dst_q0, dst_k0, dst_v0;
  int split;               // SPLIT instantiation: CTAs of the cluster that share one KV tile's steps
  int head_group;          // (batch, KV head) pairs per group of the heavy-first block order (see heavy_first_decode)
};

// delta[b, h, t] = sum_c o[b, t, h, c] * dout[b, t, h, c]. One block per (b, 32 consecutive t): that slab of o
// and dout is contiguous, hd / 8 lanes share a row with 16-byte loads (four rows in flight per lane), the row sums
// are staged in shared memory so that the [B, Hq, T] output is written as whole 128-byte lines.
constexpr int DELTA_T = 32, DELTA_THREADS = 256;

__global__ void __launch_bounds__(DELTA_THREADS)
attn_delta_kernel(const __nv_bfloat16* o, const __nv_bfloat16* dout,
                  float* __restrict__ delta, float* __restrict__ dq_acc, int B, int T, int Hq, int hd) {
  griddep_wait();
  griddep_launch();
  extern __shared__ float delta_s[];                       // [Hq][DELTA_T + 1]
  const int tiles_t = (T + DELTA_T - 1) / DELTA_T;
  const int b = blockIdx.x / tiles_t, t0 = (blockIdx.x % tiles_t) * DELTA_T;
  const int nt = min(DELTA_T, T - t0);
  const int lpr = hd >> 3;                                 // lanes per row: 4, 8 or 16
  const int sub = threadIdx.x % lpr, slot = threadIdx.x / lpr, slots = DELTA_THREADS / lpr;
  const int rows = nt * Hq;                                // row rr = tl * Hq + h
  const long long base = ((long long)b * T + t0) * Hq * hd;
  // this slab of the dQ accumulator starts at zero: stores that nothing waits for, beside the loads of the row sums
  const int vec_h = nt * hd / 4;                           // float4 of one head: its nt rows are contiguous
  for (int h = 0; dq_acc != nullptr && h < Hq; ++h) {
    float4* z = reinterpret_cast<float4*>(dq_acc + (((long long)b * Hq + h) * T + t0) * hd);
    for (int i = threadIdx.x; i < vec_h; i += DELTA_THREADS) z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  const uint4* op = reinterpret_cast<const uint4*>(o + base) + sub;
  const uint4* dp = reinterpret_cast<const uint4*>(dout + base) + sub;
  for (int rb = 0; rb < rows; rb += 4 * slots) {          // trip count is uniform: the shuffles below need whole warps
    const int r0 = rb + slot;
    uint4 a[4], d[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int rr = r0 + u * slots;
      if (rr < rows) { a[u] = op[(long long)rr * lpr]; d[u] = dp[(long long)rr * lpr]; }
      else { a[u] = make_uint4(0, 0, 0, 0); d[u] = a[u]; }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t aw[4] = {a[u].x, a[u].y, a[u].z, a[u].w}, dw[4] = {d[u].x, d[u].y, d[u].z, d[u].w};
      float acc = 0.f;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 x = unpack_bf16(aw[k]), y = unpack_bf16(dw[k]);
        acc = fmaf(x.x, y.x, fmaf(x.y, y.y, acc));
      }
      for (int off = lpr >> 1; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
      const int rr = r0 + u * slots;
      if (sub == 0 && rr < rows) delta_s[(rr % Hq) * (DELTA_T + 1) + rr / Hq] = acc;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < Hq * DELTA_T; i += DELTA_THREADS) {
    const int h = i / DELTA_T, tl = i % DELTA_T;
    if (tl < nt) delta[((long long)b * Hq + h) * T + t0 + tl] = delta_s[h * (DELTA_T + 1) + tl];
  }
}

// dq_acc (fp32 [B, Hq, T, hd]) * scale -> bf16 q-head slots of dqkv, 8 low columns and their 8 partner columns
// (j + hd / 2) per thread so that the transposed rotation (see AttnBwdParams) can be applied on the way.
// `rot_k` (only without a head -> sequence return): the Hkv k-head slots of dqkv, written as bf16 by the main kernel, are
// rotated in place by further work items (heads Hq .. Hq + Hkv - 1).
// Index: 32 bits while the items fit (three 64-bit divisions per item took longer than the item's 64 bytes).
template <typename Index>
__global__ void attn_dq_convert_kernel(const float* dq_acc, __nv_bfloat16* __restrict__ dqkv, int B, int T,
                                       int Hq, int heads_total, int hd, float scale, const float* cosT,
                                       const float* sinT, const AttnBwdDst d, int dst_q0, int rot_k) {
  griddep_wait();
  griddep_launch();
  const int half = hd / 2, vec_log = hd == 32 ? 1 : hd == 64 ? 2 : 3;          // hd / 16 items per row
  const int heads = Hq + rot_k;
  const Index total = ((Index)B * heads * T) << vec_log, step = (Index)gridDim.x * blockDim.x;
  for (Index i = blockIdx.x * (Index)blockDim.x + threadIdx.x; i < total; i += step) {
    const int j = (int)(i & ((1 << vec_log) - 1)) * 8;
    Index r = i >> vec_log;
    const Index bh = r / (Index)T;
    const int t = (int)(r - bh * (Index)T);
    const long long b = (long long)(bh / (Index)heads);
    const int h = (int)(bh - (Index)b * heads);
    float lo[8], hi[8];
    if (h < Hq) {
      const float* src = dq_acc + (((long long)b * Hq + h) * T + t) * hd + j;
      *reinterpret_cast<float4*>(lo) = *reinterpret_cast<const float4*>(src);
      *reinterpret_cast<float4*>(lo + 4) = *reinterpret_cast<const float4*>(src + 4);
      *reinterpret_cast<float4*>(hi) = *reinterpret_cast<const float4*>(src + half);
      *reinterpret_cast<float4*>(hi + 4) = *reinterpret_cast<const float4*>(src + half + 4);
#pragma unroll
      for (int k = 0; k < 8; ++k) { lo[k] *= scale; hi[k] *= scale; }
    } else {                                             // a k head: bf16 in, rotated bf16 out, same place
      const __nv_bfloat16* src = dqkv + ((b * T + t) * heads_total + h) * (long long)hd + j;
      const uint4 a = *reinterpret_cast<const uint4*>(src), c = *reinterpret_cast<const uint4*>(src + half);
      const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, cw[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 x = unpack_bf16(aw[k]), y = unpack_bf16(cw[k]);
        lo[2 * k] = x.x; lo[2 * k + 1] = x.y; hi[2 * k] = y.x; hi[2 * k + 1] = y.y;
      }
    }
    if (cosT != nullptr) {
      const float* c = cosT + (long long)t * hd + j;
      const float* sn = sinT + (long long)t * hd + j;
      float cl[8], ch[8], sl[8], sh[8];
      *reinterpret_cast<float4*>(cl) = *reinterpret_cast<const float4*>(c);
      *reinterpret_cast<float4*>(cl + 4) = *reinterpret_cast<const float4*>(c + 4);
      *reinterpret_cast<float4*>(ch) = *reinterpret_cast<const float4*>(c + half);
      *reinterpret_cast<float4*>(ch + 4) = *reinterpret_cast<const float4*>(c + half + 4);
      *reinterpret_cast<float4*>(sl) = *reinterpret_cast<const float4*>(sn);
      *reinterpret_cast<float4*>(sl + 4) = *reinterpret_cast<const float4*>(sn + 4);
      *reinterpret_cast<float4*>(sh) = *reinterpret_cast<const float4*>(sn + half);
      *reinterpret_cast<float4*>(sh + 4) = *reinterpret_cast<const float4*>(sn + half + 4);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float a = lo[k], bb = hi[k];
        lo[k] = a * cl[k] + bb * sh[k];
        hi[k] = bb * ch[k] - a * sl[k];
      }
    }
    __nv_bfloat16* dst;
    if (d.n > 0) {
      const int owner = t / d.rows, tl = t - owner * d.rows;
      if (owner >= d.n) continue;
      dst = d.p[owner] + ((b * d.rows + tl) * d.heads + dst_q0 + h) * (long long)hd + j;
    } else {
      dst = dqkv + ((b * T + t) * heads_total + h) * (long long)hd + j;
    }
    *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16(lo[0], lo[1]), pack_bf16(lo[2], lo[3]), pack_bf16(lo[4], lo[5]), pack_bf16(lo[6], lo[7]));
    *reinterpret_cast<uint4*>(dst + half) = make_uint4(pack_bf16(hi[0], hi[1]), pack_bf16(hi[2], hi[3]), pack_bf16(hi[4], hi[5]), pack_bf16(hi[6], hi[7]));
  }
}

// What a step consists of, and what bounds it. Every step is taken in two halves of 64 query columns, each with its own eight
// softmax warps and barriers: while one half's exponentials run, the other half's products do. For head dims 32 and 64 there
// are three score tiles for the two halves, so a half's scores of its next step are there before its warps ask for them
// (two tiles: 1048 us against 974 at the first shape below); dP^T of the next step is issued as soon as a half has published
// P^T and dS^T, and its warps come to it only after their exponentials. Head dim 128 (WIDE) has 256 tensor-memory columns
// beside dV and dK: scores of both halves, and dP^T in turns with dQ; a step's chain is dQ -> its way out, beside dV, dK and
// the next scores -> dP^T -> dS, and the exponentials of the next step run beside the last link.
// Cycles per 128 x 128 step, head dim 64 / 32 / 128: products 1664 / 832 / 2560, exponentials 1024 (16 a cycle); shared memory
// moves 300 / 184 KB at head dim 64 / 32, 128 B a cycle. By ncu (B 8, T 4096, 16 / 8 heads: 457 steps and 14 blocks an SM) 2750 / 2630 / 5190, what
// surrounds a block's steps included, about five steps each; tensor pipe 48 / 25 / 51 %, exponential unit 45 / 46 / 23 %, shared
// memory 47 / 26 / 39 % of its cycles. Long runs are under the power cap at 1.5 - 1.7 GHz, so what counts is energy: without the dQ
// reductions to L2 head dim 64 would take 8 % less, without any other part 2 - 4 %.
// In us with the delta and conversion passes, in sequence, against the form before (scores [q][kv], P and dS through shared
// memory, eight softmax warps that also flushed dQ, products issued by one lane's own code, a smaller last group of heads):
//   B 8, T 4096, 16 / 8 heads of 64: 1098 -> 930     B 1, T 32768, the same: 7400 -> 6040
//   B 8, T 4096, 32 / 4 heads of 32: 2055 -> 1350    B 2, T 4096, 24 / 8 heads of 128: 929 -> 667
// The parts were not timed one by one. What was measured is that a step's products, issued by one lane's own code, took 76 cycles
// each whatever their size (see umma_bf16_w), more than those of 64 columns run.
template <int HD>
struct AttnBwdCfg {
  static constexpr bool WIDE = HD == 128;
  static constexpr int KB = WIDE ? 2 : 1;                     // 64-wide blocks of a tile (HD 32: one of 32)
  static constexpr int STAGES = WIDE ? 2 : 3;                 // Q / lse / delta ring
  static constexpr int DO_STAGES = WIDE ? 1 : 3;
  static constexpr int DS_BUFS = WIDE ? 1 : 2;
  static constexpr int NS = WIDE ? 2 : 3;                     // score tiles (half steps)
  static constexpr bool KV_TMEM = HD == 32;                   // K and V as operands in tensor memory
  static constexpr int TILE_BYTES = AB_TILE * HD * 2;
  static constexpr int OFF_K = 0;
  static constexpr int OFF_V = OFF_K + TILE_BYTES;
  static constexpr int OFF_Q = OFF_V + (KV_TMEM ? 0 : TILE_BYTES);
  static constexpr int OFF_DO = OFF_Q + STAGES * TILE_BYTES;
  static constexpr int OFF_DS = OFF_DO + DO_STAGES * TILE_BYTES;   // buffers of [2 query halves][128 kv][64 q] bf16
  static constexpr int DS_BYTES = AB_TILE * AB_TILE * 2;
  static constexpr int OFF_DQS = OFF_DS + DS_BUFS * DS_BYTES;  // dQ staging: [32 rows][32 fp32] boxes of the four flush warps
  static constexpr int BOXES = WIDE ? 2 : 1;
  static constexpr int OFF_ROW = OFF_DQS + 4 * BOXES * 4096;
  static constexpr int OFF_BAR = OFF_ROW + STAGES * 2 * AB_TILE * 4;
  static constexpr int TOTAL = OFF_BAR + 256;
  static_assert(TOTAL <= 232448, "shared memory of one block");
  static constexpr int PART_PITCH = 2 * HD + 4;                // SPLIT: floats per row of this CTA's dV | dK, from OFF_Q on
  static_assert(AB_TILE * PART_PITCH * 4 <= (WIDE ? OFF_ROW : OFF_DS) - OFF_Q, "the partial dV | dK fits behind K and V");
  // tensor memory: NS tiles of S^T (a half step's P^T and dS^T replace them as bf16), two of dP^T, dV, dK, dQ, K and V.
  // WIDE: dQ takes turns with dP^T.
  static constexpr uint32_t S_COL = 0, DP_COL = NS * 64, DV_COL = DP_COL + 128, DK_COL = DV_COL + HD, DQ_COL = WIDE ? DP_COL : DK_COL + HD;
  static constexpr uint32_t K_COL = DQ_COL + HD, V_COL = K_COL + HD / 2;
  static_assert((WIDE ? DK_COL + HD : KV_TMEM ? V_COL + HD / 2 : DQ_COL + HD) <= 512, "tensor memory");
  static constexpr int OUT_COLS = HD / 4;                      // columns of dV and of dK one softmax warp carries out
};

// P of 32 query columns of one KV row: scores from tensor memory, -lse of the columns from shared memory; columns below
// `masked` come before the row (DIAG).
template <bool DIAG>
__device__ __forceinline__ void attn_bwd_p(uint32_t t_s, const float* nlse, float2 sc2, int masked, float2* pr) {
#pragma unroll
  for (int c = 0; c < 32; c += 16) {
    uint32_t sv[16];
    tmem_ld16(t_s + c, sv);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 16; i += 4) {
      const float4 nl = *reinterpret_cast<const float4*>(nlse + c + i);
      const float2 x = ffma2(make_float2(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1])), sc2, make_float2(nl.x, nl.y));
      const float2 y = ffma2(make_float2(__uint_as_float(sv[i + 2]), __uint_as_float(sv[i + 3])), sc2, make_float2(nl.z, nl.w));
      float2* o = pr + ((c + i) >> 1);
      o[0] = make_float2(ex2_approx(x.x), ex2_approx(x.y));
      o[1] = make_float2(ex2_approx(y.x), ex2_approx(y.y));
      if (DIAG) {
        if (c + i < masked) o[0].x = 0.f;
        if (c + i + 1 < masked) o[0].y = 0.f;
        if (c + i + 2 < masked) o[1].x = 0.f;
        if (c + i + 3 < masked) o[1].y = 0.f;
      }
    }
  }
}

// SPLIT: a cluster of p.split CTAs works on one KV tile, each on its share of the (query head, query tile) steps; every CTA
// leaves its fp32 dV | dK in its own shared memory and the cluster adds them up, in fixed order. See split_for.
template <int HD, bool SCATTER, bool SPLIT>
__global__ void __launch_bounds__(AB_THREADS, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tm_qkv, const __grid_constant__ CUtensorMap tm_do,
                const __grid_constant__ CUtensorMap tm_dq, const AttnBwdParams p) {
  using C = AttnBwdCfg<HD>;
  constexpr uint32_t TMEM_COLS = 512;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t sbase = smem_u32(smem_raw);
  uint8_t* sal = smem_raw;
  if (sbase & 1023u) {                                // swizzled tiles need a 1024-byte aligned base
    griddep_wait();
    if (threadIdx.x == 0) report_status(p.status, (20u << 8) | 2u);
    return;
  }
  const uint32_t bar0 = sbase + C::OFF_BAR;
  // barriers; [n] of a half, buffer, stage or score tile
  enum { KV_FULL = 0, KV_TMEM = 1, DP_FULL = 2 /* [2] */, PDS = 4 /* [2]: P^T, dS^T published */, DQ_FULL = 6 /* [2] */, DQ_FREE = 8,
         RING_FULL = 9 /* [3] */, RING_EMPTY = 12 /* [3] */, S_FULL = 15 /* [3] */, DO_FULL = 18, DO_EMPTY = 19, ALL_DONE = 20, N_BARS = 21 };
  auto bar = [&](int i) { return bar0 + 8u * i; };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sal + C::OFF_BAR + 192);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int n_tiles = (p.T + AB_TILE - 1) / AB_TILE;
  int j, bh;                                                  // KV tile (tile 0 has the most query tiles), (batch, KV head)
  const int split = SPLIT ? p.split : 1, rank = SPLIT ? (int)cluster_ctarank() : 0;
  heavy_first_decode((int)blockIdx.x / split, n_tiles, p.B * p.Hkv, p.head_group, j, bh);
  const int b = bh / p.Hkv, kvh = bh % p.Hkv;
  const int rep = p.Hq / p.Hkv;
  const int per_head = n_tiles - j;                           // query tiles j..n_tiles-1
  const int it0 = SPLIT ? rep * per_head * rank / split : 0;                                       // this CTA's steps
  const int n_it = SPLIT ? rep * per_head * (rank + 1) / split - it0 : rep * per_head;             // (SPLIT: may be none)
  const int heads_total = p.Hq + 2 * p.Hkv;

  if (threadIdx.x == 0) {
    for (int i = 0; i < N_BARS; ++i)
      mbar_init(bar(i), i == KV_TMEM ? 16 : (i == PDS || i == PDS + 1) ? 8 : i == DQ_FREE ? 4 : (i >= RING_FULL && i < RING_EMPTY) ? 2 : 1);
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tm_qkv);
    tma_prefetch_desc(&tm_do);
    tma_prefetch_desc(&tm_dq);
  }
  if (warp == 1) { tmem_alloc(smem_u32(tmem_slot), TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  griddep_wait();

  if (warp == 0) {
    // ---------------------------------------------------------------- producer: Q, dO by TMA; -lse, -delta by the warp
    if (lane == 0) {
      mbar_expect_tx(bar(KV_FULL), (C::KV_TMEM ? 1 : 2) * C::TILE_BYTES);
#pragma unroll
      for (int kb = 0; kb < C::KB; ++kb) {
        tma_load_4d(sbase + C::OFF_K + kb * 16384, &tm_qkv, bar(KV_FULL), kb * 64, p.Hq + kvh, j * AB_TILE, b);
        if (!C::KV_TMEM) tma_load_4d(sbase + C::OFF_V + kb * 16384, &tm_qkv, bar(KV_FULL), kb * 64, p.Hq + p.Hkv + kvh, j * AB_TILE, b);
      }
    }
    for (int it = 0; it < n_it; ++it) {
      const int st = it % C::STAGES;
      const int hq = kvh * rep + (it0 + it) / per_head, qi = j + (it0 + it) % per_head;
      if (!mbar_wait_warp(bar(RING_EMPTY + st), ((uint32_t)(it / C::STAGES) & 1u) ^ 1u, 21, abort_flag, p.status)) break;
      if (lane == 0) {
        mbar_expect_tx(bar(RING_FULL + st), (C::WIDE ? 1 : 2) * C::TILE_BYTES);
#pragma unroll
        for (int kb = 0; kb < C::KB; ++kb)
          tma_load_4d(sbase + C::OFF_Q + st * C::TILE_BYTES + kb * 16384, &tm_qkv, bar(RING_FULL + st), kb * 64, hq, qi * AB_TILE, b);
        if (!C::WIDE) tma_load_4d(sbase + C::OFF_DO + st * C::TILE_BYTES, &tm_do, bar(RING_FULL + st), 0, hq, qi * AB_TILE, b);
      }
      constexpr float LOG2E = 1.4426950408889634f;
      const long long r0 = ((long long)b * p.Hq + hq) * p.T;
      float* rows = reinterpret_cast<float*>(sal + C::OFF_ROW) + st * 2 * AB_TILE;
      float l[4], d[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int t = qi * AB_TILE + 32 * k + lane;
        l[k] = t < p.T ? p.lse[r0 + t] * -LOG2E : -INFINITY;               // rows past the end: P = 0
        d[k] = t < p.T ? -p.delta[r0 + t] : 0.f;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) { rows[32 * k + lane] = l[k]; rows[AB_TILE + 32 * k + lane] = d[k]; }
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(RING_FULL + st));
      if constexpr (C::WIDE) {
        if (!mbar_wait_warp(bar(DO_EMPTY), ((uint32_t)it & 1u) ^ 1u, 35, abort_flag, p.status)) break;
        if (lane == 0) {
          mbar_expect_tx(bar(DO_FULL), C::TILE_BYTES);
#pragma unroll
          for (int kb = 0; kb < C::KB; ++kb)
            tma_load_4d(sbase + C::OFF_DO + kb * 16384, &tm_do, bar(DO_FULL), kb * 64, hq, qi * AB_TILE, b);
        }
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer
    const uint32_t el = elect_one();
    constexpr uint32_t idesc_s = umma_idesc_bf16(AB_TILE, 64, 0, 0);          // S^T, dP^T of one half: B K-major
    constexpr uint32_t idesc_t = umma_idesc_bf16(AB_TILE, HD, 0, 1);          // dV, dK: A from tensor memory, B MN-major
    constexpr uint32_t idesc_q = umma_idesc_bf16(AB_TILE, HD, 1, 1);          // dQ    : A, B MN-major
    const uint64_t dk_mn = attn_desc_mn<HD>(sbase + C::OFF_K);
    // Half step h = 2 it + s: query columns 64 s .. 64 s + 63 of step it, scores in tile h % NS. Which tile and which ring stage
    // is carried along instead of computed from h, and s is a constant of the unrolled body: both keep the operands uniform.
    const uint64_t dk_k = attn_desc_k<HD>(sbase + C::OFF_K), dv_k = attn_desc_k<HD>(sbase + C::OFF_V);
    const uint64_t q_k = attn_desc_k<HD>(sbase + C::OFF_Q), do_k = attn_desc_k<HD>(sbase + C::OFF_DO);
    const uint64_t q_mn = attn_desc_mn<HD>(sbase + C::OFF_Q), do_mn = attn_desc_mn<HD>(sbase + C::OFF_DO);
    auto issue_sp = [&](uint32_t d, uint32_t a_tmem, uint64_t a_smem, uint64_t db) {
#pragma unroll
      for (int t = 0; t < HD / 16; ++t) {
        if constexpr (C::KV_TMEM) umma_bf16_ts_w(el, d, a_tmem + t * 8, umma_desc_advance(db, t * 32), idesc_s, t > 0);
        else umma_bf16_w(el, d, umma_desc_advance(a_smem, t * 32), umma_desc_advance(db, t * 32), idesc_s, t > 0);
      }
    };
    auto ring = [&](int it, int st) -> bool {
      const bool r = mbar_wait_warp(bar(RING_FULL + st), (uint32_t)(it / C::STAGES) & 1u, 22, abort_flag, p.status);
      tc_fence_after();
      return r;
    };
    auto issue_s = [&](int sb, int st, int s) {
      issue_sp(tmem + C::S_COL + sb * 64, tmem + C::K_COL, dk_k, umma_desc_advance(q_k, st * C::TILE_BYTES + s * (C::TILE_BYTES / 2)));
      umma_commit_w(el, bar(S_FULL + sb));
    };
    auto issue_dp = [&](int st, int s) {
      issue_sp(tmem + C::DP_COL + s * 64, tmem + C::V_COL, dv_k, umma_desc_advance(do_k, st * C::TILE_BYTES + s * (C::TILE_BYTES / 2)));
      umma_commit_w(el, bar(DP_FULL + s));
    };
    bool ok = mbar_wait_warp(bar(KV_FULL), 0, 23, abort_flag, p.status);
    if (ok && C::KV_TMEM) ok = mbar_wait_warp(bar(KV_TMEM), 0, 34, abort_flag, p.status);
    tc_fence_after();
    if constexpr (C::WIDE) {
      // One order of five products a step; S^T and dP^T of both halves in one piece (half the reads of K and V).
      constexpr uint32_t idesc_w = umma_idesc_bf16(AB_TILE, AB_TILE, 0, 0);
      auto issue_kk = [&](uint32_t d, uint64_t a, uint64_t bm) {
#pragma unroll
        for (int t = 0; t < HD / 16; ++t) {
          const uint32_t off = (t >> 2) * 16384 + (t & 3) * 32;
          umma_bf16_w(el, d, umma_desc_advance(a, off), umma_desc_advance(bm, off), idesc_w, t > 0);
        }
      };
      auto issue_dp_w = [&](int it) -> bool {
        if (!mbar_wait_warp(bar(DO_FULL), (uint32_t)it & 1u, 36, abort_flag, p.status)) return false;
        tc_fence_after();
        issue_kk(tmem + C::DP_COL, dv_k, do_k);
        umma_commit_w(el, bar(DP_FULL));
        return true;
      };
      const uint64_t dds_mn = umma_smem_desc(sbase + C::OFF_DS, 16384, 1024);
      if (ok && n_it > 0 && (ok = ring(0, 0))) {
        issue_kk(tmem + C::S_COL, dk_k, q_k);
        umma_commit_w(el, bar(S_FULL));
        ok = issue_dp_w(0);
      }
      for (int it = 0; it < n_it && ok; ++it) {
        const int st = it & 1;
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          if (!(ok = mbar_wait_warp(bar(PDS + s), (uint32_t)it & 1u, 26, abort_flag, p.status))) break;
          tc_fence_after();
          if (s == 1) {                                 // first, so that its way out runs beside the products after it
#pragma unroll
            for (int t = 0; t < AB_TILE / 16; ++t)
              umma_bf16_w(el, tmem + C::DQ_COL, umma_desc_advance(dds_mn, t * 2048), umma_desc_advance(dk_mn, t * 2048), idesc_q, t > 0);
            umma_commit_w(el, bar(DQ_FULL));
          }
          const uint64_t dq = umma_desc_advance(q_mn, st * C::TILE_BYTES + s * 8192), ddo = umma_desc_advance(do_mn, s * 8192);
          const uint32_t t_s = tmem + C::S_COL + s * 64;
#pragma unroll
          for (int t = 0; t < 4; ++t)
            umma_bf16_ts_w(el, tmem + C::DV_COL, t_s + (t >> 1) * 32 + (t & 1) * 8, umma_desc_advance(ddo, t * 2048), idesc_t, (it > 0) | (s > 0) | (t > 0));
          if (s == 1) umma_commit_w(el, bar(DO_EMPTY));
#pragma unroll
          for (int t = 0; t < 4; ++t)
            umma_bf16_ts_w(el, tmem + C::DK_COL, t_s + 16 + (t >> 1) * 32 + (t & 1) * 8, umma_desc_advance(dq, t * 2048), idesc_t, (it > 0) | (s > 0) | (t > 0));
        }
        if (!ok) break;
        umma_commit_w(el, bar(RING_EMPTY + st));
        if (it + 1 < n_it) {
          if (!(ok = ring(it + 1, st ^ 1))) break;
          issue_kk(tmem + C::S_COL, dk_k, umma_desc_advance(q_k, (st ^ 1) * C::TILE_BYTES));
          umma_commit_w(el, bar(S_FULL));
          if (!(ok = mbar_wait_warp(bar(DQ_FREE), (uint32_t)it & 1u, 27, abort_flag, p.status))) break;     // dQ(it) is out of the dP columns
          if (!(ok = issue_dp_w(it + 1))) break;
        }
      }
    } else {
      if (ok && n_it > 0 && (ok = ring(0, 0))) {
        issue_s(0, 0, 0);
        issue_dp(0, 0);
        issue_s(1, 0, 1);
        issue_dp(0, 1);
        if (n_it > 1 && (ok = ring(1, 1))) issue_s(2, 1, 0);
      }
      int st = 0, sb = 0;
      for (int it = 0; it < n_it && ok; ++it) {
        const int st1 = st == C::STAGES - 1 ? 0 : st + 1, st2 = st1 == C::STAGES - 1 ? 0 : st1 + 1;
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          if (!(ok = mbar_wait_warp(bar(PDS + s), (uint32_t)it & 1u, 26, abort_flag, p.status))) break;
          tc_fence_after();
          if (it + 1 < n_it) issue_dp(st1, s);           // needed first; its columns were read before P^T and dS^T were published
          const uint64_t dq = umma_desc_advance(q_mn, st * C::TILE_BYTES + s * (C::TILE_BYTES / 2));
          const uint64_t ddo = umma_desc_advance(do_mn, st * C::TILE_BYTES + s * (C::TILE_BYTES / 2));
          const uint32_t t_s = tmem + C::S_COL + sb * 64;
#pragma unroll
          for (int t = 0; t < 4; ++t)
            umma_bf16_ts_w(el, tmem + C::DV_COL, t_s + (t >> 1) * 32 + (t & 1) * 8, umma_desc_advance(ddo, t * attn_mn_step<HD>()), idesc_t, (it > 0) | (s > 0) | (t > 0));
#pragma unroll
          for (int t = 0; t < 4; ++t)
            umma_bf16_ts_w(el, tmem + C::DK_COL, t_s + 16 + (t >> 1) * 32 + (t & 1) * 8, umma_desc_advance(dq, t * attn_mn_step<HD>()), idesc_t, (it > 0) | (s > 0) | (t > 0));
          // the tensor pipe works in order: these scores replace the P^T / dS^T that were just read
          if (s == 0) {
            if (it + 1 < n_it) issue_s(sb, st1, 1);
          } else if (it + 2 < n_it) {
            if (!(ok = ring(it + 2, st2))) break;
            issue_s(sb, st2, 0);
          }
          sb = sb == C::NS - 1 ? 0 : sb + 1;
        }
        if (!ok) break;
        if (it > 0 && !(ok = mbar_wait_warp(bar(DQ_FREE), ((uint32_t)it & 1u) ^ 1u, 27, abort_flag, p.status))) break;     // dQ(it-1) is in registers
        tc_fence_after();
        const uint64_t dds_mn = umma_smem_desc(sbase + C::OFF_DS + (it & 1) * C::DS_BYTES, 16384, 1024);
#pragma unroll
        for (int t = 0; t < AB_TILE / 16; ++t)
          umma_bf16_w(el, tmem + C::DQ_COL, umma_desc_advance(dds_mn, t * 2048), umma_desc_advance(dk_mn, t * attn_mn_step<HD>()), idesc_q, t > 0);
        umma_commit_w(el, bar(DQ_FULL + (it & 1)));       // dQ ready, this dS buffer free
        umma_commit_w(el, bar(RING_EMPTY + st));
        st = st1;
      }
    }
    if (ok && n_it > 0) umma_commit_w(el, bar(ALL_DONE));
    griddep_launch();
  } else if (warp < 18) {
    // ---------------------------------------------------------------- softmax warps: 32 query columns of 32 KV rows each
    const int q4 = warp & 3, g = (warp - 2) >> 2, s = g >> 1;
    const int row = q4 * 32 + lane;                           // row of the KV tile
    const int t_row = j * AB_TILE + row;
    const uint32_t t_lane = tmem + ((uint32_t)(q4 * 32) << 16);
    bool ok = true;
    if constexpr (C::KV_TMEM) {   // K (warps of half 0) and V (half 1) rows become tensor-memory operands, half a row per warp
      static_assert(HD == 32, "half a row is 16 columns, 8 words; p.hd is HD (the scatter form has wider tiles)");
      const int c0 = (g & 1) * 16;
      const __nv_bfloat16* src = p.qkv + (((long long)b * p.T + t_row) * heads_total + p.Hq + s * p.Hkv + kvh) * HD + c0;
      uint32_t w[8];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const uint4 v = t_row < p.T ? reinterpret_cast<const uint4*>(src)[c] : make_uint4(0, 0, 0, 0);
        w[4 * c] = v.x; w[4 * c + 1] = v.y; w[4 * c + 2] = v.z; w[4 * c + 3] = v.w;
      }
      tmem_st8(t_lane + (s == 0 ? C::K_COL : C::V_COL) + c0 / 2, w);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(KV_TMEM));
    }
    const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
    const int col0 = (g & 1) * 32;                             // of the half's 64 query columns
    for (int it = 0; it < n_it; ++it) {
      const int st = it % C::STAGES, qi = j + (it0 + it) % per_head;
      const float* rows = reinterpret_cast<const float*>(sal + C::OFF_ROW) + st * 2 * AB_TILE + s * 64 + col0;
      uint8_t* drow = sal + C::OFF_DS + (C::WIDE ? 0 : it & 1) * C::DS_BYTES + s * 16384 + row * 128;
      if (!mbar_wait_warp(bar(RING_FULL + st), (uint32_t)(it / C::STAGES) & 1u, 28, abort_flag, p.status)) { ok = false; break; }
      const int h = 2 * it + s, sb = C::WIDE ? 0 : h % C::NS;
      const uint32_t t_s = t_lane + C::S_COL + (C::WIDE ? s : sb) * 64 + col0, t_dp = t_lane + C::DP_COL + s * 64 + col0;
      if (!mbar_wait_warp(bar(S_FULL + sb), (uint32_t)(C::WIDE ? it : h / C::NS) & 1u, 29, abort_flag, p.status)) { ok = false; break; }
      tc_fence_after();
      float2 pr[16];
      // two copies: the compare and select of the diagonal tiles doubled the instructions of a pair in all the others
      if (qi == j) attn_bwd_p<true>(t_s, rows, sc2, row - s * 64 - col0, pr);
      else attn_bwd_p<false>(t_s, rows, sc2, 0, pr);
      {
        uint32_t pp[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) pp[i] = pack_bf16(pr[i].x, pr[i].y);
        tmem_st16(t_s, pp);
      }
      if (!mbar_wait_warp(bar(DP_FULL + (C::WIDE ? 0 : s)), (uint32_t)it & 1u, 33, abort_flag, p.status)) { ok = false; break; }
      tc_fence_after();
      uint32_t dd[16];
#pragma unroll
      for (int c = 0; c < 32; c += 16) {
        uint32_t dp[16];
        tmem_ld16(t_dp + c, dp);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
          const float4 nd = *reinterpret_cast<const float4*>(rows + AB_TILE + c + i);
          // dS = P (dP - delta); the softmax scale is applied once, when dQ and dK leave their accumulators
          const float2 d0 = fmul2(pr[(c + i) >> 1], fadd2(make_float2(__uint_as_float(dp[i]), __uint_as_float(dp[i + 1])), make_float2(nd.x, nd.y)));
          const float2 d1 = fmul2(pr[((c + i) >> 1) + 1], fadd2(make_float2(__uint_as_float(dp[i + 2]), __uint_as_float(dp[i + 3])), make_float2(nd.z, nd.w)));
          dd[(c + i) >> 1] = pack_bf16(d0.x, d0.y);
          dd[((c + i) >> 1) + 1] = pack_bf16(d1.x, d1.y);
        }
      }
      tmem_st16(t_s + 16, dd);
      if (!C::WIDE && it > 1 && !mbar_wait_warp(bar(DQ_FULL + (it & 1)), ((uint32_t)(it >> 1) & 1u) ^ 1u, 30, abort_flag, p.status)) { ok = false; break; }
#pragma unroll
      for (int ch = 0; ch < 4; ++ch)
        *reinterpret_cast<uint4*>(drow + ((((col0 >> 3) + ch) ^ (row & 7)) << 4)) = make_uint4(dd[4 * ch], dd[4 * ch + 1], dd[4 * ch + 2], dd[4 * ch + 3]);
      fence_proxy_async_smem();
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(PDS + s));
    }
    if (ok && n_it > 0) ok = mbar_wait_warp(bar(ALL_DONE), 0, 31, abort_flag, p.status);
    tc_fence_after();
    constexpr int W = C::OUT_COLS;
    const int out0 = g * W;                                    // first of this warp's columns of dV and dK
    auto load_out = [&](uint32_t col, uint32_t* r) {
      if constexpr (W == 8) tmem_ld8(t_lane + col, r);
      else if constexpr (W == 16) tmem_ld16(t_lane + col, r);
      else tmem_ld32(t_lane + col, r);
      tmem_ld_wait();
    };
    if (ok && !SPLIT) {
      // dV, dK accumulators -> bf16 rows of the packed gradient tensor
#pragma unroll
      for (int which = 0; which < 2; ++which) {
        const float osc = which == 0 ? 1.f : p.scale;
        __nv_bfloat16* dst = p.dqkv + (((long long)b * p.T + t_row) * heads_total + (which == 0 ? p.Hq + p.Hkv : p.Hq) + kvh) * p.hd + out0;
        bool dst_ok = t_row < p.T && out0 < p.hd;
        if (SCATTER && p.n_dst > 0) {
          const int owner = t_row / p.dst_rows, tl = t_row - owner * p.dst_rows;
          dst_ok = dst_ok && owner < p.n_dst;
          if (dst_ok)
            dst = p.dst[owner] + (((long long)b * p.dst_rows + tl) * p.dst_heads + (which == 0 ? p.dst_v0 : p.dst_k0) + kvh) * p.hd + out0;
        }
        uint32_t r[W];
        load_out((which == 0 ? C::DV_COL : C::DK_COL) + out0, r);
        if (SCATTER && which == 1 && p.cosT != nullptr && out0 < p.hd) {
          // transposed RoPE on dK (fp32): column j pairs with j +- hd / 2 (the condition is the warp's, as the load needs)
          const bool low = out0 < p.hd / 2;
          const int pc = low ? out0 + p.hd / 2 : out0 - p.hd / 2;      // partner's first column
          uint32_t q2[W];
          load_out(C::DK_COL + pc, q2);
          if (t_row < p.T) {
            const float* cr = p.cosT + (long long)t_row * p.hd;
            const float* sr = p.sinT + (long long)t_row * p.hd;
#pragma unroll
            for (int i = 0; i < W; ++i) {
              const float a = __uint_as_float(r[i]), bb = __uint_as_float(q2[i]);
              r[i] = __float_as_uint(low ? a * cr[out0 + i] + bb * sr[pc + i] : a * cr[out0 + i] - bb * sr[pc + i]);
            }
          }
        }
        if (dst_ok) {
#pragma unroll
          for (int i = 0; i < W; i += 8) {
            uint4 v;
            v.x = pack_bf16(__uint_as_float(r[i]) * osc, __uint_as_float(r[i + 1]) * osc);
            v.y = pack_bf16(__uint_as_float(r[i + 2]) * osc, __uint_as_float(r[i + 3]) * osc);
            v.z = pack_bf16(__uint_as_float(r[i + 4]) * osc, __uint_as_float(r[i + 5]) * osc);
            v.w = pack_bf16(__uint_as_float(r[i + 6]) * osc, __uint_as_float(r[i + 7]) * osc);
            *reinterpret_cast<uint4*>(dst + i) = v;
          }
        }
      }
    }
    if constexpr (SPLIT) {
      // this CTA's dV | dK, over the Q / dO ring: every MMA and every row of the ring has been read (WIDE: over the dQ boxes too)
      if (C::WIDE) {
        __syncwarp();
        asm volatile("bar.sync 1, 640;" ::: "memory");
      }
      float* part = reinterpret_cast<float*>(sal + C::OFF_Q) + row * C::PART_PITCH + out0;
#pragma unroll
      for (int which = 0; which < 2; ++which) {
        uint32_t r[W];
        load_out((which == 0 ? C::DV_COL : C::DK_COL) + out0, r);
#pragma unroll
        for (int i = 0; i < W; i += 4)
          *reinterpret_cast<uint4*>(part + which * HD + i) =
              n_it > 0 ? make_uint4(r[i], r[i + 1], r[i + 2], r[i + 3]) : make_uint4(0, 0, 0, 0);      // no step: nothing was accumulated
      }
    }
  } else {
    // ---------------------------------------------------------------- dQ of every step -> fp32 accumulator in global memory
    const int q4 = warp & 3;
    const uint32_t t_lane = tmem + ((uint32_t)(q4 * 32) << 16);
    const int box0 = C::OFF_DQS + q4 * C::BOXES * 4096;
    for (int it = 0; it < n_it; ++it) {
      const int hq = kvh * rep + (it0 + it) / per_head, qi = j + (it0 + it) % per_head;
      const int y0 = qi * AB_TILE + q4 * 32;                  // first of this warp's 32 query rows
      if (!mbar_wait_warp(bar(DQ_FULL + (C::WIDE ? 0 : it & 1)), (uint32_t)(C::WIDE ? it : it >> 1) & 1u, 32, abort_flag, p.status)) break;
      tc_fence_after();
      constexpr int COLS = HD < 64 ? HD : 64;                 // in registers at a time
#pragma unroll
      for (int c0 = 0; c0 < HD; c0 += COLS) {
        uint32_t r[COLS];
#pragma unroll
        for (int c = 0; c < COLS; c += 32) tmem_ld32(t_lane + C::DQ_COL + c0 + c, r + c);
        tmem_ld_wait();
        if (c0 + COLS == HD) {                                // all of it has been read: the columns are free
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(DQ_FREE));
        }
#pragma unroll
        for (int c = 0; c < COLS; c += 32 * C::BOXES) {
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");      // staging boxes free again
          __syncwarp();
#pragma unroll
          for (int x = 0; x < C::BOXES; ++x) {
            uint8_t* rowp = sal + box0 + x * 4096 + lane * 128;
            const uint32_t* v = r + c + 32 * x;
#pragma unroll
            for (int ch = 0; ch < 8; ++ch)
              *reinterpret_cast<uint4*>(rowp + ((ch ^ (lane & 7)) << 4)) = make_uint4(v[4 * ch], v[4 * ch + 1], v[4 * ch + 2], v[4 * ch + 3]);
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
#pragma unroll
            for (int x = 0; x < C::BOXES; ++x)
              if (y0 < p.T && c0 + c + 32 * x < p.hd)
                asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4}], [%1];"
                             ::"l"((uint64_t)&tm_dq), "r"(sbase + box0 + x * 4096), "r"(c0 + c + 32 * x), "r"(y0), "r"(b * p.Hq + hq) : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        }
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");      // dQ reductions have left shared memory and landed
    if (SPLIT && C::WIDE) {
      __syncwarp();
      asm volatile("bar.sync 1, 640;" ::: "memory");
    }
  }
  if constexpr (SPLIT) {
    __syncwarp();
    tc_fence_before();
    cluster_sync_all();
    // rows [128 rank / split, 128 (rank + 1) / split) of the sum, in place (nobody else reads these rows of this CTA's part)
    float* base = reinterpret_cast<float*>(sal + C::OFF_Q);
    const int rows = AB_TILE / split, r0 = rank * rows;
    for (int i = threadIdx.x; i < rows * (HD / 2); i += AB_THREADS) {
      const int r = r0 + i / (HD / 2), c = (i % (HD / 2)) * 4;
      const uint32_t off = sbase + C::OFF_Q + (uint32_t)(r * C::PART_PITCH + c) * 4u;
      float4 a[8];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (q < split) a[q] = ld_cluster_f4(mapa_shared(off, (uint32_t)q));
#pragma unroll
      for (int q = 1; q < 8; ++q)
        if (q < split) { a[0].x += a[q].x; a[0].y += a[q].y; a[0].z += a[q].z; a[0].w += a[q].w; }
      *reinterpret_cast<float4*>(base + r * C::PART_PITCH + c) = a[0];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < rows * (HD / 4); i += AB_THREADS) {
      const int r = r0 + i / (HD / 4), c = (i % (HD / 4)) * 8, t_row = j * AB_TILE + r;
      if (t_row >= p.T) continue;
      const bool is_k = c >= HD;
      const float osc = is_k ? p.scale : 1.f;
      const float* v = base + r * C::PART_PITCH + c;
      uint4 o;
      o.x = pack_bf16(v[0] * osc, v[1] * osc); o.y = pack_bf16(v[2] * osc, v[3] * osc);
      o.z = pack_bf16(v[4] * osc, v[5] * osc); o.w = pack_bf16(v[6] * osc, v[7] * osc);
      *reinterpret_cast<uint4*>(p.dqkv + (((long long)b * p.T + t_row) * heads_total + (is_k ? p.Hq : p.Hq + p.Hkv) + kvh) * p.hd + (c - (is_k ? HD : 0))) = o;
    }
    cluster_sync_all();                // no CTA leaves while another may still read its part
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, TMEM_COLS); }
}

// CTAs per KV tile. One CTA per KV tile walks over all its query heads and tiles, so the tile with the most steps bounds the
// launch from below however idle the chip is. A cluster divides that, but every CTA of a cluster costs about 5.4 steps
// (start-up and the exchange of dV and dK while its SM has no other CTA). The estimate is the longer of a CTA's own time and the
// work per SM; its pick was within 1 % of the fastest of 1, 2, 4, 8 on seventeen measured shapes of all head dims. With delta and
// conversion passes, in us, unsplit -> picked: 1 x 8192, 8 / 1 heads of 64 680 -> 194; 4 x 777, 16 / 2 94 -> 51; 3 x 1001, 12 / 4
// 50 -> 40; 1 x 1074, 8 / 2 of 128 108 -> 41; 2 x 256, 8 / 2 of 32 20 -> 14.
static int split_for(int n_tiles, int heads_kv, int rep) {
  const char* v = getenv("TLM_ATTN_BWD_SPLIT");          // 1, 2, 4 or 8: for tests and measurements
  const int forced = v != nullptr ? atoi(v) : 0;
  if (forced == 1 || forced == 2 || forced == 4 || forced == 8) return forced;
  const double heaviest = (double)rep * n_tiles, tiles = (double)n_tiles * heads_kv, total = heaviest * (n_tiles + 1) / 2 * heads_kv;
  const double sms = num_sms();
  int best = 1;
  double best_cost = heaviest > total / sms ? heaviest : total / sms;
  for (int s = 2; s <= 8; s *= 2) {
    const double own = heaviest / s + 3.0, shared = (total + 5.4 * tiles * s) / sms, cost = own > shared ? own : shared;
    if (cost < best_cost) { best_cost = cost; best = s; }
  }
  return best;
}

template <int HD, bool SCATTER, bool SPLIT = false>
static int launch_bwd(const CUtensorMap& mq, const CUtensorMap& mdo, const CUtensorMap& mdq, const AttnBwdParams& p,
                      cudaStream_t st) {
  constexpr int smem = AttnBwdCfg<HD>::TOTAL;
  auto kern = attn_bwd_kernel<HD, SCATTER, SPLIT>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  const int grid = ((p.T + AB_TILE - 1) / AB_TILE) * p.B * p.Hkv;
  return launch_overlapped(kern, dim3((unsigned)(grid * (SPLIT ? p.split : 1))), dim3(AB_THREADS), smem, st, SPLIT ? p.split : 1, mq, mdo, mdq, p);
}

}  // namespace tlm

using namespace tlm;

// dq_acc: fp32 scratch [B,Hq,T,hd]; delta: fp32 scratch [B,Hq,T]. Both are owned by the caller.
// cosT / sinT (optional, fp32 [T, hd]): the transposed RoPE is applied to dQ and dK on the way out.
// dst_ptrs (optional, n_dst > 0): head -> sequence return, see AttnBwdParams; dqkv may then be null.
static int attn_bwd_impl(const void* qkv, const void* o, const void* dout, const float* lse, void* dqkv,
                         float* dq_acc, float* delta, int B, int T, int Hq, int Hkv, int hd, float scale,
                         const float* cosT, const float* sinT, void* const* dst_ptrs, int n_dst, int dst_rows,
                         int dst_heads, int dst_q0, int dst_k0, int dst_v0, cudaStream_t st) {
  if (hd != 32 && hd != 64 && hd != 128) return -4;
  if (Hq % Hkv != 0) return -5;
  if ((size_t)Hq * (DELTA_T + 1) * 4 > 48 * 1024) return -6;
  // Few blocks would take longer over the zeroes than a memset (48 heads of 64, 16 rows: one block, 3 us more)
  const int delta_blocks = B * ((T + DELTA_T - 1) / DELTA_T);
  const bool fused_zero = delta_blocks >= num_sms();
  if (!fused_zero) {
    const cudaError_t ce = cudaMemsetAsync(dq_acc, 0, (size_t)B * T * Hq * hd * 4, st);
    if (ce != cudaSuccess) return (int)ce;
  }
  int le = launch_overlapped(attn_delta_kernel, dim3(delta_blocks), dim3(DELTA_THREADS), (size_t)Hq * (DELTA_T + 1) * 4, st, 1,
      (const __nv_bfloat16*)o, (const __nv_bfloat16*)dout, delta, fused_zero ? dq_acc : nullptr, B, T, Hq, hd);
  if (le) return le;
  CUtensorMap mq, mdo;
  const int box_cols = hd == 32 && n_dst == 0 ? 32 : 64;
  int e = make_qkv_map(&mq, qkv, B, T, Hq + 2 * Hkv, hd, AB_TILE, box_cols);
  if (e) return e;
  e = make_qkv_map(&mdo, dout, B, T, Hq, hd, AB_TILE, box_cols);
  if (e) return e;
  if ((cosT == nullptr) != (sinT == nullptr)) return -6;
  if (n_dst < 0 || n_dst > AB_MAX_DST || (n_dst > 0 && (dst_ptrs == nullptr || dst_rows <= 0 || (long long)dst_rows * n_dst < T)))
    return -6;
  if (n_dst == 0 && dqkv == nullptr) return -6;
  AttnBwdParams p{};
  p.qkv = (const __nv_bfloat16*)qkv; p.dqkv = (__nv_bfloat16*)dqkv; p.dq_acc = dq_acc; p.lse = lse; p.delta = delta; p.B = B; p.T = T; p.Hq = Hq; p.Hkv = Hkv;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f; p.status = status_word(); p.hd = hd; p.cosT = cosT; p.sinT = sinT;
  p.n_dst = n_dst; p.dst_rows = dst_rows; p.dst_heads = dst_heads; p.dst_q0 = dst_q0; p.dst_k0 = dst_k0; p.dst_v0 = dst_v0;
  // per (batch, KV head): Q, dO, dQ (fp32 accumulator + bf16 result) of its query heads, K, V, dK, dV. In us with the delta and
  // conversion passes: B 8, T 4096, 16 / 8 heads of 64: 910 - 925 with groups of 4 - 16, 957 with 32, 1055 with all 64.
  // What is left for the last group counts (even_group): 24 / 8 heads of 128, B 2, T 4096, 4 x 4 650, 5 + 5 + 5 + 1 730, 6 + 6 + 4 720,
  // 2 x 8 650; 32 / 4 heads of 32, B 8, 4 x 8 1345, 10 + 10 + 10 + 2 1515, 5 x 6 + 2 1478, 2 x 16 1367
  p.head_group = attn_head_group("TLM_ATTN_BWD_GROUP", (long long)T * hd * (10LL * (Hq / Hkv) + 8), 112LL << 20, B * Hkv);
  AttnBwdDst dd{};
  dd.n = n_dst; dd.rows = dst_rows; dd.heads = dst_heads;
  for (int i = 0; i < n_dst; ++i) { p.dst[i] = (__nv_bfloat16*)dst_ptrs[i]; dd.p[i] = p.dst[i]; }
  CUtensorMap mdq;                                     // fp32 [B*Hq, T, hd] accumulator, box 32 x 32 x 1
  {
    uint64_t dims[3] = {(uint64_t)hd, (uint64_t)T, (uint64_t)B * Hq};
    uint64_t strides[2] = {(uint64_t)hd * 4, (uint64_t)T * hd * 4};
    uint32_t box[3] = {32, 32, 1};
    e = make_tmap_f32(&mdq, dq_acc, 3, dims, strides, box);
    if (e) return e;
  }
  if (n_dst > 0) e = hd == 128 ? launch_bwd<128, true>(mq, mdo, mdq, p, st) : launch_bwd<64, true>(mq, mdo, mdq, p, st);
  else {
    p.split = split_for((T + AB_TILE - 1) / AB_TILE, B * Hkv, Hq / Hkv);
    if (p.split > 1) e = hd == 128 ? launch_bwd<128, false, true>(mq, mdo, mdq, p, st) : hd == 64 ? launch_bwd<64, false, true>(mq, mdo, mdq, p, st)
                                                                                                   : launch_bwd<32, false, true>(mq, mdo, mdq, p, st);
    else e = hd == 128 ? launch_bwd<128, false>(mq, mdo, mdq, p, st) : hd == 64 ? launch_bwd<64, false>(mq, mdo, mdq, p, st)
                                                                                : launch_bwd<32, false>(mq, mdo, mdq, p, st);
  }
  if (e) return e;
  // without a return scatter the main kernel has written un-rotated dK into dqkv: this pass rotates it in place
  const int rot_k = (n_dst == 0 && cosT != nullptr) ? Hkv : 0;
  const long long items = (long long)B * T * (Hq + rot_k) * (hd / 16);
  int cb = (int)((items + 255) / 256 < num_sms() * 16 ? (items + 255) / 256 : num_sms() * 16);
  auto conv = items + 256LL * cb < (1LL << 32) ? attn_dq_convert_kernel<unsigned> : attn_dq_convert_kernel<long long>;
  return launch_overlapped(conv, dim3(cb), dim3(256), 0, st, 1, (const float*)dq_acc, (__nv_bfloat16*)dqkv, B, T, Hq, Hq + 2 * Hkv, hd, scale, cosT, sinT,
                           dd, dst_q0, rot_k);
}

TLM_API int tlm_attn_bwd(const void* qkv, const void* o, const void* dout, const float* lse, void* dqkv,
                         float* dq_acc, float* delta, int B, int T, int Hq, int Hkv, int hd, float scale,
                         const float* cosT, const float* sinT, cudaStream_t st) {
  return attn_bwd_impl(qkv, o, dout, lse, dqkv, dq_acc, delta, B, T, Hq, Hkv, hd, scale, cosT, sinT, nullptr, 0, 0, 0, 0, 0, 0, st);
}

// Attention backward whose gradient rows leave for the sequence owners' packed buffers (see AttnBwdParams):
// dst_ptrs[r]: bf16 [B, dst_rows, dst_heads, hd] on rank r; q slot s -> head dst_q0 + s, k -> dst_k0 + s, v -> dst_v0 + s.
TLM_API int tlm_attn_bwd_scatter(const void* qkv, const void* o, const void* dout, const float* lse, float* dq_acc,
                                 float* delta, int B, int T, int Hq, int Hkv, int hd, float scale, const float* cosT,
                                 const float* sinT, void* const* dst_ptrs, int n_dst, int dst_rows, int dst_heads,
                                 int dst_q0, int dst_k0, int dst_v0, cudaStream_t st) {
  if (n_dst < 1) return -6;
  return attn_bwd_impl(qkv, o, dout, lse, nullptr, dq_acc, delta, B, T, Hq, Hkv, hd, scale, cosT, sinT, dst_ptrs, n_dst,
                       dst_rows, dst_heads, dst_q0, dst_k0, dst_v0, st);
}
