// Block order of the causal attention grids and the choice of grids that start early, written once for the device and for
// host tests (tests/tile_order_host_test.cpp, tests/test_tile_order_cpu.py).
#pragma once

#ifdef __CUDACC__
#define TLM_TILE_HD __host__ __device__ __forceinline__
#else
#define TLM_TILE_HD inline
#endif

namespace tlm {

// Heavy-first order for causal attention grids. Tiles of one (batch, head) differ in work by the causal mask (rank 0
// heaviest); blocks start in linear order, so the order decides the tail: with all tiles of one head adjacent, the last
// head's heaviest tiles start when the grid is almost drained and run alone. Here the heads are taken in groups of
// `group` (few enough that the group's tensors stay in L2), and inside a group all heads' rank-0 tiles come first, then
// all rank-1 tiles, ...: every group, the last one included, ends on its lightest tiles.
//   linear block id in [0, n_tiles * n_heads) -> (rank of the tile within its head, head); a bijection.
TLM_TILE_HD void heavy_first_decode(int linear, int n_tiles, int n_heads, int group, int& tile_rank, int& head) {
  const int per_group = n_tiles * group;
  const int g = linear / per_group, r = linear - g * per_group;
  const int left = n_heads - g * group;
  const int g_heads = group < left ? group : left;            // the last group may be smaller
  tile_rank = r / g_heads;
  head = g * group + (r - tile_rank * g_heads);
}

// Group size for at most `most` heads a group: the smallest that needs no more groups, so that the last group, which takes what is
// left, is as large as that allows. The chip runs dry at the end of the last group, from the heaviest of its tiles on, and a
// small rest of heads has too few tiles to fill it beside those: 32 heads of 8 x 32 steps in groups of 10 + 10 + 10 + 2 took 1104
// steps' time on 148 SMs, in four of 8 949 (total / 148 is 913). A small rest can remain: 16 heads of at most 3 are 5 x 3 + 1.
TLM_TILE_HD int even_group(int n_heads, int most) {
  const int groups = (n_heads + most - 1) / most;
  return (n_heads + groups - 1) / groups;
}

// May a grid start beside the last blocks of the kernel in front (see launch_overlapped)? `per_sm`: blocks of it that share an SM
// without loss.
TLM_TILE_HD constexpr bool starts_early(long long blocks, int cluster, int per_sm, int sms) { return cluster > 1 || blocks <= (long long)per_sm * sms; }

}  // namespace tlm
