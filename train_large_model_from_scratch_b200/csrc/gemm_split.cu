// Small bf16 GEMMs: C[M,N] (=|+=) A[M,K] * B[N,K]^T with few output tiles.
//
// gemm.cu's 128 x 256 (pairs: 256 x 256) tiles leave most SMs without work when M and N are small, and whoever has a
// tile walks the whole reduction alone: the data gradient of a 50304-wide LM head over 512 tokens of width 256 was two
// tiles of 786 k-blocks. Here a tile is 128 x 64 or 128 x 128 and a cluster of S = 1, 2, 4 or 8 CTAs shares its
// reduction, each CTA an equal share of the k-blocks. Every CTA leaves its fp32 partial tile in its own shared memory,
// and after a cluster barrier CTA r adds up rows [128 r / S, 128 (r + 1) / S) of all S partials (distributed shared
// memory, fixed order, so the result does not depend on timing) and applies the epilogue. No workspace, no second
// launch, no atomics between the parts.
//
// Roles as in gemm.cu: warp 0 TMA producer, warp 1 MMA issuer and tensor-memory owner, warps 2-5 move the accumulator
// to shared memory; then all six warps reduce and store. Two CTAs fit an SM, so one's prologue and epilogue run beside
// the other's main loop. Waits are bounded.
#include "common.cuh"
#include "gemm_split.h"

namespace tlm {

constexpr int SP_BM = 128, SP_BK = 64, SP_THREADS = 192;
constexpr int SP_A_BYTES = SP_BM * SP_BK * 2;
constexpr int SP_BOX_MN = 64 * SP_BK * 2;                 // one 64(mn) x 64(k) MN-major box
constexpr int SP_ALONE = 117 * 1024;                      // shared memory of which an SM has room for one

template <int BN>
struct SplitCfg {
  // 96 KB ring: two CTAs per SM. A CTA that has an SM to itself takes as deep a one as it has k-blocks for (see launch_split).
  static constexpr int STAGES = BN == 64 ? 4 : 3, MAX_STAGES = BN == 64 ? 9 : 6;
  static constexpr int STAGE_BYTES = SP_A_BYTES + BN * SP_BK * 2;
  static constexpr int PITCH = BN + 4;                    // floats per row of the partial tile (reuses the ring)
  static constexpr int REST = 1024 /*align slack*/ + 256 /*barriers*/;
  static_assert(SP_BM * PITCH * 4 <= STAGES * STAGE_BYTES, "the partial tile reuses the operand ring");
  static_assert(MAX_STAGES * STAGE_BYTES + REST <= 227 * 1024, "shared memory of one block");
};

struct SplitParams {
  SplitGemm g;
  int tiles_m, tiles_n, stages;
  unsigned int* status;
};

template <bool A_MN, bool B_MN, int EPI, int BN, int S>
__global__ void __launch_bounds__(SP_THREADS, 2)
gemm_split_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const SplitParams p) {
  using C = SplitCfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sal = smem_raw + (sbase - smem_u32(smem_raw));
  // barriers: full[MAX_STAGES], empty[MAX_STAGES], accumulator full
  const int ring = p.stages * C::STAGE_BYTES;
  const uint32_t bar0 = sbase + ring;
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (C::MAX_STAGES + s); };
  const uint32_t acc_bar = bar0 + 8u * (2 * C::MAX_STAGES);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sal + ring + 8 * (2 * C::MAX_STAGES + 1));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const SplitGemm& g = p.g;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int rank = S > 1 ? (int)cluster_ctarank() : 0;
  const int tile = (int)blockIdx.x / S;
  const int tm = tile % p.tiles_m, tn = tile / p.tiles_m;
  constexpr int TILE_N = EPI == SPLIT_SWIGLU ? BN / 2 : BN;       // output columns (SwiGLU: as many of gate and of up)
  const int m0 = tm * SP_BM, n0 = tn * TILE_N;
  const int kblocks = (g.K + SP_BK - 1) / SP_BK;
  const int kb_lo = (int)((long long)kblocks * rank / S), kb_hi = (int)((long long)kblocks * (rank + 1) / S);

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2 * C::MAX_STAGES + 1; ++i) mbar_init(bar0 + 8u * i, 1);
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) { tmem_alloc(smem_u32(tmem_slot), BN); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  // Few rows: the first of this block's weights into L2 while the kernel in front still runs (see weights_ahead_end), asked for by
  // a warp that is idle until the accumulator is there. Into L2 only, so it does not matter whether that kernel writes them.
  // 3003 rows of 768 (weights in L2 anyway) lost 1 % and stay without.
  if (!A_MN && threadIdx.x == 64 && tm == 0 && g.M <= g.N) {
    const int end = weights_ahead_end(kb_lo * SP_BK, kb_hi * SP_BK);
    for (int k0 = kb_lo * SP_BK; k0 < end; k0 += SP_BK) {
      if (B_MN) {
#pragma unroll
        for (int j = 0; j < BN / 64; ++j) tma_prefetch_2d(&tmB, n0 + 64 * j, k0);
      } else {
        tma_prefetch_2d(&tmB, k0, n0);
        if (EPI == SPLIT_SWIGLU) tma_prefetch_2d(&tmB, k0, g.N + n0);
      }
    }
  }
  griddep_wait();

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0; uint32_t phase = 0;
      for (int kb = kb_lo; kb < kb_hi; ++kb) {
        if (!mbar_wait(empty_bar(stage), phase ^ 1u, 81, abort_flag, p.status)) break;
        const int k0 = kb * SP_BK;
        const uint32_t sa = sbase + stage * C::STAGE_BYTES, sb = sa + SP_A_BYTES, fb = full_bar(stage);
        mbar_expect_tx(fb, C::STAGE_BYTES);
        if (A_MN) {
#pragma unroll
          for (int j = 0; j < SP_BM / 64; ++j) tma_load_2d(sa + j * SP_BOX_MN, &tmA, fb, m0 + 64 * j, k0);
        } else {
          tma_load_2d(sa, &tmA, fb, k0, m0);
        }
        if (B_MN) {
#pragma unroll
          for (int j = 0; j < BN / 64; ++j) tma_load_2d(sb + j * SP_BOX_MN, &tmB, fb, n0 + 64 * j, k0);
        } else if (EPI == SPLIT_SWIGLU) {         // gate rows, then the matching up rows
          tma_load_2d(sb, &tmB, fb, k0, n0);
          tma_load_2d(sb + BN * SP_BK, &tmB, fb, k0, g.N + n0);
        } else {
          tma_load_2d(sb, &tmB, fb, k0, n0);
        }
        if (++stage == p.stages) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1) {
    // by the whole warp (see umma_bf16_w): four MMAs of 48 (BN 64) or 64 cycles took 76 each to issue from one lane's own code.
    // In us, weights out of memory: 333 x 1024 x 4096 11.6 -> 11.1, 333 x 1024 x 1024 7.2 -> 6.7, 512 x 256 x 256 3.7 -> 3.4
    const uint32_t el = elect_one();
    constexpr uint32_t idesc = umma_idesc_bf16(SP_BM, BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
    int stage = 0; uint32_t phase = 0;
    bool ok = true;
    for (int kb = kb_lo; kb < kb_hi; ++kb) {
      if (!mbar_wait_warp(full_bar(stage), phase, 82, abort_flag, p.status)) { ok = false; break; }
      tc_fence_after();
      const uint32_t sa = sbase + stage * C::STAGE_BYTES, sb = sa + SP_A_BYTES;
      const uint64_t ad = A_MN ? umma_smem_desc(sa, SP_BOX_MN, 1024) : umma_smem_desc(sa, 16, 1024);
      const uint64_t bd = B_MN ? umma_smem_desc(sb, SP_BOX_MN, 1024) : umma_smem_desc(sb, 16, 1024);
#pragma unroll
      for (int kk = 0; kk < SP_BK / 16; ++kk)
        umma_bf16_w(el, tmem, umma_desc_advance(ad, kk * (A_MN ? 2048 : 32)), umma_desc_advance(bd, kk * (B_MN ? 2048 : 32)), idesc, (kb > kb_lo) | (kk > 0));
      umma_commit_w(el, empty_bar(stage));
      if (++stage == p.stages) { stage = 0; phase ^= 1u; }
    }
    if (ok) umma_commit_w(el, acc_bar);
    griddep_launch();
  } else {
    // accumulator -> this CTA's partial tile in shared memory (every operand read of the ring has retired by then)
    const int row = (warp & 3) * 32 + lane;
    if (mbar_wait_warp(acc_bar, 0, 83, abort_flag, p.status)) {
      tc_fence_after();
      const uint32_t taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
      float* dst = reinterpret_cast<float*>(sal) + row * C::PITCH;
#pragma unroll
      for (int c = 0; c < BN; c += 32) {
        uint32_t r[32];
        tmem_ld32(taddr + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; j += 4) *reinterpret_cast<uint4*>(dst + c + j) = make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
      }
    }
    tc_fence_before();
  }
  __syncwarp();
  if (S > 1) cluster_sync_all(); else __syncthreads();

  // ---- sum of the S partial tiles, in place: this CTA's rows of its own partial are read by nobody else. Neighbouring lanes
  // read neighbouring 16-byte pieces, which is what the shared-memory network between SMs wants (S = 8, 32-byte pieces read
  // by the epilogue itself: 3 us more).
  constexpr int ROWS = SP_BM / S;
  if constexpr (S > 1) {
    constexpr int P4 = BN / 4;
    for (int i = threadIdx.x; i < ROWS * P4; i += SP_THREADS) {
      const int r = rank * ROWS + i / P4, c = (i % P4) * 4;
      if (m0 + r >= g.M) break;                              // rows ascend with i
      const uint32_t off = sbase + (uint32_t)(r * C::PITCH + c) * 4u;
      float4 a[S];
#pragma unroll
      for (int s = 0; s < S; ++s) a[s] = ld_cluster_f4(mapa_shared(off, (uint32_t)s));
#pragma unroll
      for (int s = 1; s < S; ++s) { a[0].x += a[s].x; a[0].y += a[s].y; a[0].z += a[s].z; a[0].w += a[s].w; }
      *reinterpret_cast<float4*>(reinterpret_cast<float*>(sal) + r * C::PITCH + c) = a[0];
    }
    __syncthreads();
  }

  // ---- epilogue, 8 columns per item
  constexpr bool PAIRED = EPI == SPLIT_HEADS || EPI == SPLIT_SWIGLU;      // items own 8 columns and their 8 partner columns
  constexpr int PER_ROW = PAIRED ? BN / 16 : BN / 8;
  auto load8 = [&](int r, int c, float* v) {
    const float* src = reinterpret_cast<const float*>(sal) + r * C::PITCH + c;
    *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(src);
    *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(src + 4);
  };
  auto pack8 = [](const float* v) {
    return make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
  };
  const int half = EPI == SPLIT_HEADS ? g.hd >> 1 : 0;
  // What other kernels wrote (rotation tables, gate / up) comes through plain loads: the read-only path may only be used for
  // memory that nothing writes while this kernel lives, and it lives from before griddep_wait. A plain load does not pass a
  // store, so the loads of BATCH items are issued before the first of their stores; one after the other, their latency was
  // most of the epilogue.
  constexpr int BATCH = EPI == SPLIT_HEADS ? 2 : EPI == SPLIT_SWIGLU_BWD ? 4 : 1;
  constexpr int ITEMS = ROWS * PER_ROW;
  float4 pre[EPI == SPLIT_HEADS ? BATCH * 8 : 1];            // per item: cos, sin of the lower, cos, sin of the upper columns
  uint4 pre_gu[EPI == SPLIT_SWIGLU_BWD ? BATCH * 2 : 1];     // per item: gate, up
  for (int i0 = threadIdx.x; i0 < ITEMS; i0 += BATCH * SP_THREADS) {
    if constexpr (BATCH > 1) {
#pragma unroll
      for (int u = 0; u < BATCH; ++u) {
        const int i = i0 + u * SP_THREADS, r = rank * ROWS + i / PER_ROW, ch = i % PER_ROW;
        const long long row = m0 + r;
        if (i >= ITEMS || row >= g.M) continue;
        if constexpr (EPI == SPLIT_HEADS) {
          const int per_half = half >> 3, hh = ch / per_half, j = (ch - hh * per_half) * 8;
          if (n0 + hh * g.hd >= g.N || n0 / g.hd + hh >= g.n_rot) continue;
          const long long at = (long long)(row % g.rows_per_batch) * g.hd + j;
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            pre[u * 8 + k] = *reinterpret_cast<const float4*>(g.cosT + at + 4 * k);
            pre[u * 8 + 2 + k] = *reinterpret_cast<const float4*>(g.sinT + at + 4 * k);
            pre[u * 8 + 4 + k] = *reinterpret_cast<const float4*>(g.cosT + at + half + 4 * k);
            pre[u * 8 + 6 + k] = *reinterpret_cast<const float4*>(g.sinT + at + half + 4 * k);
          }
        } else {
          if (n0 + ch * 8 >= g.N) continue;
          const __nv_bfloat16* gp = reinterpret_cast<const __nv_bfloat16*>(g.aux) + row * 2 * g.N + n0 + ch * 8;
          pre_gu[u * 2] = *reinterpret_cast<const uint4*>(gp);
          pre_gu[u * 2 + 1] = *reinterpret_cast<const uint4*>(gp + g.N);
        }
      }
    }
#pragma unroll
    for (int ub = 0; ub < BATCH; ++ub) {
      const int i = i0 + ub * SP_THREADS, r = rank * ROWS + i / PER_ROW, ch = i % PER_ROW;
      const long long row = m0 + r;
      if (i >= ITEMS || row >= g.M) continue;
      float v[8];
      if constexpr (EPI == SPLIT_BF16 || EPI == SPLIT_F32_ACC) {
        const int col = n0 + ch * 8;
        if (col >= g.N) continue;
        if constexpr (EPI == SPLIT_BF16) {
          load8(r, ch * 8, v);
          *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(g.C) + row * g.ldc + col) = pack8(v);
        } else {
          // one reduction per element: nothing waits for C, and the result does not depend on timing
          float* out = reinterpret_cast<float*>(g.C) + row * g.ldc + col;
          load8(r, ch * 8, v);
          asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(out), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]) : "memory");
          asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(out + 4), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
        }
      } else if constexpr (EPI == SPLIT_HEADS) {
        const int per_half = half >> 3;                        // 8-column pieces of half a head
        const int hh = ch / per_half, j = (ch - hh * per_half) * 8, c = hh * g.hd + j;
        if (n0 + c >= g.N) continue;                           // N is a multiple of hd
        const int head = n0 / g.hd + hh;
        const int bi = (int)(row / g.rows_per_batch), t = (int)(row - (long long)bi * g.rows_per_batch);
        const bool rot = head < g.n_rot;
        float u[8];
        load8(r, c, v);
        load8(r, c + half, u);
        if (rot) {
          const float *cl = reinterpret_cast<const float*>(pre + ub * 8), *sl = cl + 8, *chh = cl + 16, *sh = cl + 24;
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const float a = v[k], b = u[k];
            v[k] = a * cl[k] - b * sl[k];
            u[k] = b * chh[k] + a * sh[k];
          }
        }
        __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(g.C) + (((long long)bi * g.dst_rows + g.row_off + t) * g.dst_heads + head) * g.hd + j;
        *reinterpret_cast<uint4*>(out) = pack8(v);
        *reinterpret_cast<uint4*>(out + half) = pack8(u);
      } else if constexpr (EPI == SPLIT_SWIGLU) {
        const int col = n0 + ch * 8;
        if (col >= g.N) continue;
        float u[8];
        load8(r, ch * 8, v);
        load8(r, BN / 2 + ch * 8, u);
        // as in gemm.cu: the products are rounded to bf16 first, so the numbers equal those of separate kernels
        const uint4 gp = pack8(v), up = pack8(u);
        const uint32_t gw[4] = {gp.x, gp.y, gp.z, gp.w}, uw[4] = {up.x, up.y, up.z, up.w};
        uint32_t o[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) o[k] = swiglu2(gw[k], uw[k]);
        if (g.C != nullptr) {
          __nv_bfloat16* gu = reinterpret_cast<__nv_bfloat16*>(g.C) + row * g.ldc + col;
          *reinterpret_cast<uint4*>(gu) = gp;
          *reinterpret_cast<uint4*>(gu + g.N) = up;
        }
        *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(g.act) + row * g.N + col) = make_uint4(o[0], o[1], o[2], o[3]);
      } else {
        const int col = n0 + ch * 8;
        if (col >= g.N) continue;
        const uint4 gv = pre_gu[ub * 2], uv = pre_gu[ub * 2 + 1];
        load8(r, ch * 8, v);
        const uint4 dv = pack8(v);
        const uint32_t dw[4] = {dv.x, dv.y, dv.z, dv.w}, gw[4] = {gv.x, gv.y, gv.z, gv.w}, uw[4] = {uv.x, uv.y, uv.z, uv.w};
        uint32_t og[4], ou[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) swiglu_bwd2(dw[k], gw[k], uw[k], og[k], ou[k]);
        __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(g.C) + row * g.ldc + col;
        *reinterpret_cast<uint4*>(out) = make_uint4(og[0], og[1], og[2], og[3]);
        *reinterpret_cast<uint4*>(out + g.N) = make_uint4(ou[0], ou[1], ou[2], ou[3]);
      }
    }
  }

  // no CTA leaves while another may still read its partial tile
  __syncwarp();
  if (S > 1) cluster_sync_all(); else __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, BN); }
}

// ---- host side ----------------------------------------------------------------------------------
// Has every CTA of a plan an SM to itself? Always up to one CTA per SM without a cluster; with one only where whole clusters of
// them surely fit (144 CTAs in clusters of four took a second wave).
static bool one_per_sm(long long ctas, int split) { return split == 1 ? ctas <= num_sms() : ctas * 4 <= num_sms() * 3; }

template <bool A_MN, bool B_MN, int EPI, int BN, int S>
static int launch_split(const CUtensorMap& ma, const CUtensorMap& mb, SplitParams p, cudaStream_t st) {
  auto kern = gemm_split_kernel<A_MN, B_MN, EPI, BN, S>;
  using C = SplitCfg<BN>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::MAX_STAGES * C::STAGE_BYTES + C::REST);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  const int ctas = p.tiles_m * p.tiles_n * S, per_cta = ((p.g.K + SP_BK - 1) / SP_BK + S - 1) / S;
  // A grid that starts beside the last blocks of the kernel in front would pair up on the free SMs; with more than half of an
  // SM's shared memory each block gets its own (333 x 1024 x 4096: 13.8 -> 11 us). And a ring as deep as there are k-blocks or
  // room for: 96 KB in flight do not cover the latency of memory. Same product 10.1 -> 9.0 us, 512 x 256 x 50304 40.1 -> 31.0,
  // 1000 x 768 x 50304 141 -> 112.
  const bool alone = one_per_sm(ctas, S);
  p.stages = !alone || per_cta <= C::STAGES ? C::STAGES : per_cta < C::MAX_STAGES ? per_cta : C::MAX_STAGES;
  int smem = p.stages * C::STAGE_BYTES + C::REST;
  if (alone && smem < SP_ALONE) smem = SP_ALONE;
  return launch_overlapped<2>(kern, dim3((unsigned)ctas), dim3(SP_THREADS), smem, st, S, ma, mb, p);
}

static int split_map(CUtensorMap* m, const void* ptr, long long rows, long long k, long long ld, bool mn, int box_rows) {
  uint64_t dims[2] = {(uint64_t)(mn ? rows : k), (uint64_t)(mn ? k : rows)}, strides[1] = {(uint64_t)ld * 2};
  uint32_t box[2] = {64, (uint32_t)(mn ? SP_BK : box_rows)};
  return make_tmap_bf16(m, ptr, 2, dims, strides, box);
}

// everything the epilogues load and store in 16-byte pieces (absent tensors are null)
static bool aligned_ok(const SplitGemm& g) {
  return g.N % 8 == 0 && g.ldc % 8 == 0 && aligned16(g.C) && aligned16(g.act) && aligned16(g.aux) && aligned16(g.cosT) && aligned16(g.sinT);
}

int split_run(const SplitGemm& g, const SplitPlan& plan, cudaStream_t st) {
  const int bn = plan.bn, tile_n = g.epi == SPLIT_SWIGLU ? bn / 2 : bn;
  const int kblocks = (g.K + SP_BK - 1) / SP_BK;
  if ((bn != 64 && bn != 128) || plan.split < 1 || plan.split > kblocks) return -4;
  if (!aligned_ok(g)) return -4;
  if (g.epi == SPLIT_HEADS && (g.hd > bn || bn % g.hd != 0 || g.hd % 16 != 0)) return -4;
  CUtensorMap ma, mb;
  int e = split_map(&ma, g.A, g.M, g.K, g.lda, g.a_mn, SP_BM);
  if (e) return e;
  e = split_map(&mb, g.B, g.epi == SPLIT_SWIGLU ? 2LL * g.N : g.N, g.K, g.ldb, g.b_mn, tile_n);
  if (e) return e;
  SplitParams p{g, (g.M + SP_BM - 1) / SP_BM, (g.N + tile_n - 1) / tile_n, 0, status_word()};
#define TLM_SPLIT_S(A, B, E, BN)                                   \
  switch (plan.split) {                                            \
    case 1: return launch_split<A, B, E, BN, 1>(ma, mb, p, st);    \
    case 2: return launch_split<A, B, E, BN, 2>(ma, mb, p, st);    \
    case 4: return launch_split<A, B, E, BN, 4>(ma, mb, p, st);    \
    case 8: return launch_split<A, B, E, BN, 8>(ma, mb, p, st);    \
    default: return -4;                                            \
  }
#define TLM_SPLIT(A, B, E)                                                                             \
  if (g.a_mn == A && g.b_mn == B && g.epi == E) {                                                      \
    if (bn == 64) TLM_SPLIT_S(A, B, E, 64) else TLM_SPLIT_S(A, B, E, 128)                              \
  }
  TLM_SPLIT(false, false, SPLIT_BF16) TLM_SPLIT(false, true, SPLIT_BF16) TLM_SPLIT(true, true, SPLIT_F32_ACC)
  TLM_SPLIT(false, false, SPLIT_HEADS) TLM_SPLIT(false, false, SPLIT_SWIGLU) TLM_SPLIT(false, true, SPLIT_SWIGLU_BWD)
#undef TLM_SPLIT
#undef TLM_SPLIT_S
  return -2;
}

SplitPlan split_plan(const SplitGemm& g, double wide_us) {
  if (!aligned_ok(g)) return SplitPlan{0, 0};
  return split_rule(g, wide_us, num_sms());
}

}  // namespace tlm

using namespace tlm;

// tlm_gemm (same arguments) with the tile width and the split given: for tests and measurements.
TLM_API int tlm_gemm_split(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                           long long ldc, int a_mn, int b_mn, int epi, int bn, int split, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (epi != SPLIT_BF16 && epi != SPLIT_F32_ACC) return -2;
  SplitGemm g{};
  g.A = A; g.B = B; g.M = M; g.N = N; g.K = K; g.lda = lda; g.ldb = ldb; g.a_mn = a_mn != 0; g.b_mn = b_mn != 0;
  g.epi = epi; g.C = C; g.ldc = ldc;
  return split_run(g, SplitPlan{bn, split}, stream);
}
// The fused epilogues with the plan given, for the same purpose. heads: C = [M / rows, rows, N / hd, hd], the first n_rot heads
// rotated; forward SwiGLU: C = gate|up [M, 2 N] (or null), act [M, N]; backward: A = dy, B = w_down [K, N], aux = gate|up,
// C = d(gate)|d(up).
TLM_API int tlm_gemm_split_heads(const void* A, const void* B, void* C, int M, int N, int K, int hd, int rows, int n_rot,
                                 const float* cosT, const float* sinT, int bn, int split, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (hd <= 0 || N % hd != 0 || rows <= 0 || M % rows != 0 || (n_rot > 0 && (cosT == nullptr || sinT == nullptr))) return -5;
  SplitGemm g{};
  g.A = A; g.B = B; g.M = M; g.N = N; g.K = K; g.lda = K; g.ldb = K; g.epi = SPLIT_HEADS; g.C = C; g.ldc = hd;
  g.hd = hd; g.rows_per_batch = rows; g.dst_rows = rows; g.dst_heads = N / hd; g.n_rot = n_rot; g.cosT = cosT; g.sinT = sinT;
  return split_run(g, SplitPlan{bn, split}, stream);
}
TLM_API int tlm_gemm_split_swiglu(const void* A, const void* B, void* C, void* act, const void* aux, int M, int N, int K,
                                  int backward, int bn, int split, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (backward ? (C == nullptr || aux == nullptr) : act == nullptr) return -5;
  SplitGemm g{};
  g.A = A; g.B = B; g.M = M; g.N = N; g.K = K; g.lda = K; g.ldb = backward ? N : K; g.b_mn = backward != 0;
  g.epi = backward ? SPLIT_SWIGLU_BWD : SPLIT_SWIGLU; g.C = C; g.ldc = 2LL * N; g.act = act; g.aux = aux;
  return split_run(g, SplitPlan{bn, split}, stream);
}
