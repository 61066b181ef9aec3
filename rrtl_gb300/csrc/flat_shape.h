// Shape of the flat gate kernel (gate_flat.h), shared by the kernel, the
// program builder (flatprog.cpp) and the host runtime.
#pragma once

#include <stdint.h>

namespace rrtl {

constexpr uint32_t kFlatComputeThreads = 512;  // 16 compute warps (flatprog.h kFlatWarps)
constexpr uint32_t kFlatServiceThreads = 128;
constexpr uint32_t kFlatThreads = kFlatComputeThreads + kFlatServiceThreads;
#ifndef RRTL_FLAT_PREFETCH
#define RRTL_FLAT_PREFETCH 4
#endif
constexpr uint32_t kFlatPrefetch = RRTL_FLAT_PREFETCH;  // entries a warp loads ahead
constexpr uint32_t kFlatMaxVectors = 4;  // vectors per tile of 4-word rows (one for narrower rows)
constexpr uint64_t kFlatMinCycles = 4;   // shorter runs stay on one launch of the fused kernel
// Entry flags (bits of word y): a level barrier before it, three-input cells.
constexpr uint32_t kFlatDevSync = 1u << 16, kFlatDevThree = 1u << 24;
constexpr uint32_t kFlatConst0 = 0xFFFFFFFEu, kFlatConst1 = 0xFFFFFFFFu;  // constant rows of the commit list

// Shared memory of the CTA: all of an SM's, so that the distance of the
// tile's N planes is a compile-time constant.
constexpr uint32_t kFlatSmem = 227 * 1024;
constexpr uint32_t kFlatHeader = 512;  // detection state, the queue's item and job
#if defined(__CUDACC__)
__host__ __device__
#endif
constexpr uint32_t flat_plane_bytes(uint32_t N) {
  return (kFlatSmem - kFlatHeader) / N & ~127u;
}

}  // namespace rrtl
