// The packed marching-cubes case table in global memory (one copy per
// translation unit that includes this header): every reader indexes it by
// lane, which constant memory would serve one address at a time.
#pragma once
#include <cstdint>
#include "mc_tables.h"

namespace daxgb {
static __device__ const uint64_t kMcCase[256] = DAX_GB300_MC_CASE_WORDS;

__device__ __forceinline__ int mc_num_tris(int cs) { return (int)(__ldg(kMcCase + cs) >> 60); }
__device__ __forceinline__ int mc_edge(uint64_t word, int n) { return (int)((word >> (4 * n)) & 0xF); }
}  // namespace daxgb
