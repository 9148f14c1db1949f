// Shared helpers for the sm_100a kernel library: launch bookkeeping, bounded
// waits, and thin inline-PTX wrappers for mbarrier, TMA (non-multicast forms
// only) and tcgen05 (alloc / mma / commit / ld / fences).
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "flag_protocol.h"
#include "tile_order.h"

#define TLM_API extern "C" __attribute__((visibility("default")))

namespace tlm {

// ---- launch bookkeeping ------------------------------------------------------
// Every launcher bumps this counter once per kernel launch; Python reads it to
// report how many kernels of this library ran inside a timed region.
extern unsigned long long g_launches;
extern int g_deterministic;        // nonzero: no order-dependent floating-point atomics (see tlm_set_deterministic)
inline void count_launch(int n = 1) { g_launches += (unsigned long long)n; }

// Status word in mapped pinned host memory. Kernels that give up on a wait
// write a nonzero code there (first writer wins) and return, so the context
// stays usable and the host can read the word at any time.
// code = (site << 8) | detail. `status_word()` returns the device-visible pointer.
unsigned int* status_word();

// Kernels launched through launch_overlapped may start before the kernel in front of them in the stream is done, and call
// griddep_wait() before they touch memory that another kernel reads or writes: it returns when that kernel has ended and its
// writes can be seen (and, as that kernel waited in the same way, those before it). griddep_launch() lets the next kernel
// start; it takes effect when every block of the grid has called it or ended, so no block of a grid is ever kept out by its
// successor. A kernel that uses tensor memory calls it after its own allocation, in the warp that allocates: a block of the
// next kernel that takes the rest of an SM's columns, or waits for them, then holds up nobody it waits for itself. The GEMM
// and attention kernels call it when their last MMA has been issued, so that launch, barriers, tensor memory and descriptor
// fetch of the next kernel run beside the epilogue; norms at their start. Called at the start by all of them (the next kernel's
// blocks then sit on the few SMs that are free, two on one SM) a 333-token prompt took 703 us, not called 686, so 668.
// Early blocks pile up on the SMs that happen to be free, so a grid of more blocks than starts_early allows is launched as an
// ordinary kernel, which also gives up the launch hidden behind the end of the kernel in front. Both sides, us: norms of 3003 rows
// 5.7 (6.2 early), norm and GEMM of 32768 x 1024 107.6 (119.9), of 8192 x 1024 32.9 (35.5); norms of 1500 rows alone 5.4 (5.1), but
// with the GEMM behind them 12.3 (13.1). Small-tile GEMMs run two blocks per SM by design and pile up no further: 1000 x 2048,
// K 256 5.8 ordinary, 4.9 early; eleven such products 0.92 of the time, a step of 13 layers of 512 2529 -> 2478. Clusters start
// early whatever their grid: split attention backward 51.3 (ordinary 52.7) for 4 x 777, 16 / 2 heads of 64, 65.0 (66.3) for
// 2 x 1699, 8 / 4 of 128, 193 (194) for 1 x 8192, 8 / 1 of 64. Attention forward of 149 - 296 blocks is ordinary: in a row with itself
// it loses 1 us (3 x 1001, 12 heads of 64 16.4, early 15.2), between its GEMMs and a norm it does not (36.3, early 37.3; 1 x 3000
// 55.6, early 61.2). So are the delta and conversion passes of its backward: 1 us in a row, 172.8 (early 188.7) for 4 x 2048 behind
// a GEMM.
// Steps of 512 tokens (tiny model) 1163 -> 1064 us, of 6006 tokens (8 layers of 768) 6930 -> 6580 us.
// The kernel lives from before that wait, so what other kernels write is not read-only for its whole life: such kernels take
// their inputs as plain pointers (no const __restrict__, from which the compiler may make read-only loads that need not stay
// behind the wait; no __ldg).
int num_sms();
#ifdef __CUDACC__
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// PER_SM: see starts_early
template <int PER_SM = 1, typename... P, typename... A>
inline int launch_overlapped(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, int cluster, A&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = !starts_early(grid.x, cluster, PER_SM, num_sms()) ? 0 : cluster > 1 ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, P(args)...);
  count_launch();
  return (int)(e != cudaSuccess ? e : cudaPeekAtLastError());
}
#endif

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

inline int launch_status() {
  cudaError_t e = cudaPeekAtLastError();
  return (int)e;
}

// ---- small device utilities --------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void report_status(unsigned int* status, unsigned int code) {
  if (status != nullptr) atomicCAS_system(status, 0u, code);
}

// ---- flags in peer-visible memory ----------------------------------------------------
__device__ __forceinline__ void st_release_sys(int* addr, int v) {
  asm volatile("st.release.sys.global.s32 [%0], %1;" ::"l"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_acquire_sys(const int* addr) {
  int v;
  asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(addr) : "memory");
  return v;
}

// "Parameters ready" flags of the sharded optimizer step (one symmetric int32 array of READY_INTS words per flat
// buffer). Word [bucket * READY_STRIDE + r] of a rank's array is written by rank r, into every rank's copy, once
// all of r's parameter stores of that bucket's update have been issued and fenced; it holds the number of updates
// done so far. Words READY_EPOCH0 + bucket (how many updates this rank itself has done: the value consumers wait
// for) and READY_CNT0 + bucket (blocks-finished counter of the update kernel) are only used locally.
// Memory policy of the flag protocols (flag_protocol.h) on the device: system-scope acquire loads / release stores.
struct DeviceMem {
  static __device__ __forceinline__ int load_acquire(const int* p) { return ld_acquire_sys(p); }
  static __device__ __forceinline__ void store_release(int* p, int v) { st_release_sys(p, v); }
};

constexpr int READY_STRIDE = 16, READY_MAX_BUCKETS = 16;
constexpr int READY_EPOCH0 = READY_STRIDE * READY_MAX_BUCKETS, READY_CNT0 = READY_EPOCH0 + READY_MAX_BUCKETS;
constexpr int READY_INTS = 512;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack_bf16(uint32_t u) {
  __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162*>(&u);
  return __bfloat1622float2(v);
}

// ---- mbarrier -------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// CLUSTER: also acquires what the other CTA of the cluster published with its (cluster-scope) arrival
template <bool CLUSTER = false>
__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  if (CLUSTER)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
  return ok;
}

// Wait with a time limit. Returns false (after recording `site`) when the
// phase did not complete within the limit; callers then leave their loops,
// skip further waits and fall through to the common teardown.
// The limit is counted in SM cycles (`clock64`, a cheap register read) and only
// looked at every 1024 failed polls: reading %globaltimer costs on the order of a
// microsecond, which on a wait that sits on a pipeline's critical path (and
// almost every wait fails its first poll) is more than the work between waits.
constexpr uint64_t kWaitLimitNs = 2000000000ull;            // 2 s (flag waits on peers, timed with %globaltimer)

// Lanes 0..n-1 of the calling warp wait (bounded) until every rank's "parameters ready" word of `bucket` has
// reached this rank's own update count. Returns false on the lanes that gave up (status `site << 8 | rank`).
__device__ __forceinline__ bool wait_params_ready(const int* ready_local, int bucket, int n, int lane,
                                                  unsigned int* status, unsigned int site) {
  bool ok = true;
  if (lane < n) {
    const int expect = reinterpret_cast<const volatile int*>(ready_local)[READY_EPOCH0 + bucket];
    const proto::ReadyLayout layout{READY_STRIDE, READY_EPOCH0, READY_CNT0};
    const uint64_t t0 = globaltimer_ns();
    uint32_t spins = 0;
    while (!proto::ready_from<DeviceMem>(ready_local, bucket, layout, lane, expect)) {
      if ((++spins & 0x3f) == 0 && globaltimer_ns() - t0 > kWaitLimitNs) {
        report_status(status, (site << 8) | (unsigned int)lane);
        ok = false;
        break;
      }
    }
  }
  return ok;
}
constexpr long long kWaitLimitCycles = 4000000000ll;        // ~2-3 s of SM cycles
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, unsigned int site,
                                          volatile int* abort_flag, unsigned int* status) {
  if (mbar_try_wait<CLUSTER>(bar, parity)) return true;
  long long t0 = 0;
  uint32_t spins = 0;
  while (!mbar_try_wait<CLUSTER>(bar, parity)) {
    if ((++spins & 0x3ff) == 0) {
      if (*abort_flag) return false;
      const long long now = clock64();
      if (t0 == 0) {
        t0 = now;
      } else if (now - t0 > kWaitLimitCycles) {
        *abort_flag = 1;
        report_status(status, (site << 8) | 1u);
        return false;
      }
    }
  }
  return true;
}

// The same by a whole warp that stays together: all lanes get the same answer. In front of warp-wide instructions (tcgen05.ld / st,
// MMAs by an elected lane, __syncwarp, named barriers) it has to be this one: while an abort is under way one lane may see the
// phase complete and another the flag, and a warp that splits there never meets again. The vote costs the attention kernels'
// softmax warps -1 to +1 %; voting on the first poll already changes nothing beyond the noise.
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, unsigned int site, volatile int* abort_flag,
                                               unsigned int* status) {
  return __all_sync(0xffffffffu, mbar_wait<CLUSTER>(bar, parity, site, abort_flag, status));
}

// ---- TMA (tiled, no multicast) ------------------------------------------------------
__device__ __forceinline__ void tma_load_2d(uint32_t smem_dst, const CUtensorMap* map, uint32_t bar,
                                            int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_dst), "l"((uint64_t)map), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t smem_dst, const CUtensorMap* map, uint32_t bar,
                                            int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_dst), "l"((uint64_t)map), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t smem_dst, const CUtensorMap* map, uint32_t bar,
                                            int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_dst), "l"((uint64_t)map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
// The box of tma_load_2d into L2 only
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap* map, int c0, int c1) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"((uint64_t)map), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void tma_prefetch_3d(const CUtensorMap* map, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"((uint64_t)map), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)map) : "memory");
}

// ---- tcgen05 ----------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_result), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// One lane of a converged warp, the same one every time (nonzero on that lane).
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
  return r;
}
// MMA and commit of a whole converged warp, issued by the lane whose `elected` is nonzero. Issued by one lane's own code, MMAs of any
// size took 76 cycles each (clock reads around a step's issue); issued like this they take what they run. The likely reason:
// an MMA's operands live in uniform registers, and are computed there only where the code around it is the warp's.
// D[tmem] (+)= A[smem] * B[smem], bf16 inputs, fp32 accumulate.
__device__ __forceinline__ void umma_bf16_w(uint32_t elected, uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(elected)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void umma_bf16_ts_w(uint32_t elected, uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                               uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(elected)
      : "memory");
}
// Arrive on an mbarrier once all previously issued MMAs of the elected lane retire.
__device__ __forceinline__ void umma_commit_w(uint32_t elected, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
      ::"r"(bar), "r"(elected) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// 32 lanes x 32 consecutive fp32 columns: thread t of the warp gets lane (base_lane + t).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}

// ---- UMMA descriptors --------------------------------------------------------------------------
// Shared-memory matrix descriptor, 128-byte swizzle, sm_100 version field = 1.
//   K-major  : rows of 64 bf16 (128 B); 8-row groups 1024 B apart  -> SBO = 1024, LBO unused (1)
//   MN-major : [k][64 mn] rows of 128 B; 8-k groups 1024 B apart (SBO); next 64 mn `lbo_bytes` apart
__device__ __forceinline__ uint64_t umma_smem_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;        // descriptor version (Blackwell)
  d |= (uint64_t)2 << 61;        // SWIZZLE_128B
  return d;
}
// Tiles of 32 bf16 columns, 64-byte swizzle: rows of 64 B, 8-row (K-major) or 8-k (MN-major) groups 512 B apart. One tile
// is 32 wide in its contiguous direction, so there is no second stride.
__device__ __forceinline__ uint64_t umma_smem_desc_sw64(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(512 >> 4) << 32;
  d |= (uint64_t)1 << 46;        // descriptor version (Blackwell)
  d |= (uint64_t)4 << 61;        // SWIZZLE_64B
  return d;
}
// Operand tiles of the attention kernels: [128 rows][HD columns], HD 32 in one 64-byte-swizzled block, HD 64 / 128 in 64-wide
// 128-byte-swizzled blocks 16 KB apart. K-major view (reduction over the columns) and MN-major view (reduction over the rows).
template <int HD>
__device__ __forceinline__ uint64_t attn_desc_k(uint32_t addr) {
  return HD == 32 ? umma_smem_desc_sw64(addr) : umma_smem_desc(addr, 16, 1024);
}
template <int HD>
__device__ __forceinline__ uint64_t attn_desc_mn(uint32_t addr) {
  return HD == 32 ? umma_smem_desc_sw64(addr) : umma_smem_desc(addr, 16384, 1024);
}
template <int HD>
constexpr uint32_t attn_mn_step() { return HD == 32 ? 1024 : 2048; }      // bytes of 16 rows of such a block
// Descriptor of the same tile `byte_off` bytes further on. The start-address field holds (addr >> 4) in its
// low 14 bits and shared-memory addresses stay below 2^18, so the field cannot carry into its neighbours and
// the whole update is one add. The thread that issues the MMAs is a serial bottleneck (one instruction
// stream feeds the tensor pipe), so descriptors are built once per tile and advanced this way.
__device__ __forceinline__ uint64_t umma_desc_advance(uint64_t desc, uint32_t byte_off) {
  return desc + (uint64_t)(byte_off >> 4);
}
// ---- CTA pairs (cta_group::2) --------------------------------------------------------------------
// Two CTAs of one cluster (ranks 0 and 1, neighbouring SMs) run one M = 256 MMA: each CTA stages its own 128 rows of A
// and its own half of B's N rows in its own shared memory at the same offsets, the MMA is issued by one thread of
// rank 0 (the leader) and fills 128 accumulator lanes in each CTA's tensor memory. Loads are plain tiled TMA loads
// (no multicast) that may complete on the leader's mbarrier.
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// Every thread of the cluster. The `.aligned` form needs a whole warp at the instruction together, and callers come out of
// loops whose lanes leave at different turns, so the warp is joined here.
__device__ __forceinline__ void cluster_sync_all() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of the same shared-memory offset in CTA `rank` of this cluster
__device__ __forceinline__ uint32_t mapa_shared(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// 16 bytes of another CTA's shared memory (address from mapa_shared)
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
// `bar` is a shared::cluster address (the leader's barrier, see mapa_shared); `smem_dst` is this CTA's own memory
__device__ __forceinline__ void tma_load_2d_pair(uint32_t smem_dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_dst), "l"((uint64_t)map), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(uint32_t smem_dst, const CUtensorMap* map, uint32_t bar, int c0, int c1,
                                                 int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_dst), "l"((uint64_t)map), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
// tensor-memory management of a pair: the same warp of BOTH CTAs issues each of these
__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_result), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// by a converged warp, as umma_bf16_w
__device__ __forceinline__ void umma_bf16_pair_w(uint32_t elected, uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                                 uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(elected)
      : "memory");
}
// Arrive on the mbarrier at offset `bar` in BOTH CTAs of the pair once all MMAs issued so far by the elected lane retire.
__device__ __forceinline__ void umma_commit_pair_w(uint32_t elected, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}"
      ::"r"(bar), "h"((uint16_t)3), "r"(elected)
      : "memory");
}

// Instruction descriptor for kind::f16 with bf16 A/B and fp32 D.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int M, int N, int a_mn_major, int b_mn_major) {
  return (1u << 4)                       // D format: f32
         | (1u << 7)                     // A format: bf16
         | (1u << 10)                    // B format: bf16
         | ((uint32_t)a_mn_major << 15)  // A major: 0 = K, 1 = MN
         | ((uint32_t)b_mn_major << 16)  // B major
         | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// ---- host: tensor-map encoding through the driver entry point -----------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn get_encode_tiled();

// rank-N bf16 tensor map with 128B swizzle. dims/strides innermost first;
// strides[i] is the byte stride of dimension i+1.
int make_tmap_bf16(CUtensorMap* map, const void* base, int rank, const uint64_t* dims, const uint64_t* strides_bytes,
                   const uint32_t* box);

// same for fp32 elements (inner box extent <= 32 elements with the 128-byte swizzle)
int make_tmap_f32(CUtensorMap* map, const void* base, int rank, const uint64_t* dims, const uint64_t* strides_bytes,
                  const uint32_t* box);

// Heads per group of the attention kernels' heavy-first block order (heavy_first_decode): as many heads as keep the
// group's tensors (`bytes_per_head` each) within `budget_bytes` of L2, or the value of the environment variable `env`
// (read on every call: a handful of launches per step); clamped to [1, n_heads].
int attn_head_group(const char* env, long long bytes_per_head, long long budget_bytes, int n_heads);

// 4-D bf16 map over a packed [B, T, heads, hd] tensor: dims (hd, heads, T, B), box (box_cols, 1, box_rows, 1).
int make_qkv_map(CUtensorMap* map, const void* base, int B, int T, int heads, int hd, int box_rows, int box_cols = 64);

// Packed fp32 pairs (sm_100: one issue slot for two lanes of fma / add / mul). The softmax warps of the attention
// kernels are bound by instruction issue, so their scale-and-shift, row-sum and dS arithmetic runs on pairs.
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(*reinterpret_cast<unsigned long long*>(&d))
      : "l"(*reinterpret_cast<const unsigned long long*>(&a)), "l"(*reinterpret_cast<const unsigned long long*>(&b)),
        "l"(*reinterpret_cast<const unsigned long long*>(&c)));
  return d;
}
__device__ __forceinline__ float2 fadd2(float2 a, float2 b) {
  float2 d;
  asm("add.rn.f32x2 %0, %1, %2;"
      : "=l"(*reinterpret_cast<unsigned long long*>(&d))
      : "l"(*reinterpret_cast<const unsigned long long*>(&a)), "l"(*reinterpret_cast<const unsigned long long*>(&b)));
  return d;
}
__device__ __forceinline__ float2 fmul2(float2 a, float2 b) {
  float2 d;
  asm("mul.rn.f32x2 %0, %1, %2;"
      : "=l"(*reinterpret_cast<unsigned long long*>(&d))
      : "l"(*reinterpret_cast<const unsigned long long*>(&a)), "l"(*reinterpret_cast<const unsigned long long*>(&b)));
  return d;
}

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// 1 / x with the hardware's approximation (about 1 ulp; 0 for infinities and where the result would be denormal)
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// SwiGLU on pairs of columns. The GEMM epilogues that apply it are bound by instruction issue (30 instructions per element
// with scalar arithmetic and __fdividef, 10 - 12 here), not by the exponentials. 32768 x 4096 columns, K 1024, in a training
// step: forward 451 -> 415 us, backward 357 -> 322 us.
__device__ __forceinline__ float2 sigmoid2(float2 a) {
  const float2 x = fmul2(a, make_float2(-1.4426950408889634f, -1.4426950408889634f));
  const float2 den = fadd2(make_float2(ex2_approx(x.x), ex2_approx(x.y)), make_float2(1.f, 1.f));
  return make_float2(rcp_approx(den.x), rcp_approx(den.y));
}
// packed bf16 pairs in and out: silu(gate) * up
__device__ __forceinline__ uint32_t swiglu2(uint32_t gate, uint32_t up) {
  const float2 a = unpack_bf16(gate);
  const float2 o = fmul2(fmul2(a, sigmoid2(a)), unpack_bf16(up));
  return pack_bf16(o.x, o.y);
}
// d(gate), d(up) from d(act), gate, up
__device__ __forceinline__ void swiglu_bwd2(uint32_t dact, uint32_t gate, uint32_t up, uint32_t& dgate, uint32_t& dup) {
  const float2 a = unpack_bf16(gate), s = sigmoid2(a), one = make_float2(1.f, 1.f);
  const float2 ps = fmul2(unpack_bf16(dact), s);                                         // d(act) * sigmoid
  const float2 u = ffma2(a, ffma2(s, make_float2(-1.f, -1.f), one), one);                // 1 + gate (1 - sigmoid)
  const float2 og = fmul2(fmul2(ps, unpack_bf16(up)), u), ou = fmul2(ps, a);
  dgate = pack_bf16(og.x, og.y);
  dup = pack_bf16(ou.x, ou.y);
}

}  // namespace tlm
