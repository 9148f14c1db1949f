// GEMMs whose 256-wide tiles cannot fill the chip: small tiles, the reduction split over a cluster (gemm_split.cu).
#pragma once

#include <cuda_runtime.h>

#include "gemm_cost.h"

namespace tlm {

// The plan for a product of that size, or bn == 0 where the 256-wide tiles of gemm.cu are faster: they would take `wide_us`.
SplitPlan split_plan(const SplitGemm& g, double wide_us);
int split_run(const SplitGemm& g, const SplitPlan& plan, cudaStream_t st);

}  // namespace tlm
