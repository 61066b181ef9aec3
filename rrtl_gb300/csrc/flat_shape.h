// Shape of the flat gate kernel (gate_flat.h), shared by the kernel, the
// program builder (flatprog.cpp) and the host runtime.
#pragma once

#include <stdint.h>

namespace rrtl {

constexpr uint32_t kFlatComputeThreads = 512;  // 16 compute warps
constexpr uint32_t kFlatServiceThreads = 128;
constexpr uint32_t kFlatThreads = kFlatComputeThreads + kFlatServiceThreads;
// Tiles of one or two words (without forces) need so few registers that a run
// of its own takes 24 compute warps: 50,000 gates 24.6k -> 23.7k (one word)
// and 28.7k -> 28.0k clocks a tile-cycle, 200,000 gates 66.9k -> 59.1k and
// 80.9k -> 74.3k; 28 warps are slower again (65.8k and 74.8k before the byte
// offsets, against 63.2k and 74.4k). Programs of few entries a level use the
// warps they have entries for.
constexpr uint32_t kFlatNarrowThreads = 768;
#ifndef RRTL_FLAT_PREFETCH
#define RRTL_FLAT_PREFETCH 4
#endif
constexpr uint32_t kFlatPrefetch = RRTL_FLAT_PREFETCH;  // entries a warp loads ahead
constexpr uint32_t kFlatMaxVectors = 4;  // vectors per tile of 4-word rows (one for narrower rows)
constexpr uint64_t kFlatMinCycles = 4;   // shorter runs stay on one launch of the fused kernel
// One-word rows whose byte offset fits 16 bits are named by it in the entries:
// a tile-cycle of narrow rows is bound by ALU instructions (two scheduler
// slots each), of which the address of a row is one less. With the entry
// batches no longer copied (flat_tile), a tile-cycle of one word takes 25.9k
// -> 24.6k clocks at 50,000 gates, 70.5k -> 66.9k at 200,000.
constexpr uint32_t kFlatByteRows = 1u << 14;
// Entry flags (bits of word y): a level barrier before it, three-input cells.
constexpr uint32_t kFlatDevSync = 1u << 16, kFlatDevThree = 1u << 24;
constexpr uint32_t kFlatConst0 = 0xFFFFFFFEu, kFlatConst1 = 0xFFFFFFFFu;  // constant rows of the commit list

// Shared memory of the CTA: all of an SM's, so that the distance of the
// tile's N planes is a compile-time constant.
constexpr uint32_t kFlatSmem = 227 * 1024;
constexpr uint32_t kFlatHeader = 512;  // detection state, the queue's item and job
#if defined(__CUDACC__)
#define RRTL_FLAT_HD __host__ __device__
#else
#define RRTL_FLAT_HD
#endif
RRTL_FLAT_HD constexpr uint32_t flat_plane_bytes(uint32_t N) {
  return (kFlatSmem - kFlatHeader) / N & ~127u;
}

// The part of a run that is block `block`'s k-th (n = 0: it has no more): n
// cycles from c0 of one tile. Tiles laid end to end, each as long as the run's
// cycles, are cut into equal shares, one a block, so a tile is split between
// two blocks at most: the later block takes its first cycles before anything
// else, the earlier one its last cycles after everything else, when those are
// done (a share is no shorter than a tile).
struct FlatPart {
  uint32_t tile;
  bool first, last;  // the first or last cycles of a split tile
  uint64_t c0, n;
};
RRTL_FLAT_HD inline FlatPart flat_part(uint32_t n_tiles, uint64_t cycles, uint32_t block, uint32_t blocks, uint32_t k) {
  const uint64_t total = n_tiles * cycles, share = (total + blocks - 1) / blocks;
  const uint64_t lo = block * share, end = lo + share < total ? lo + share : total;
  FlatPart p{};
  if (lo >= total) return p;
  const uint64_t tile = lo / cycles + k, at = tile * cycles;
  if (at >= end) return p;
  p.tile = (uint32_t)tile;
  p.first = lo > at;
  p.last = end < at + cycles;
  p.n = (p.last ? end : at + cycles) - (p.first ? lo : at);
  p.c0 = p.last ? cycles - p.n : 0;
  return p;
}

}  // namespace rrtl
