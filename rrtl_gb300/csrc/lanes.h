// Lanes of a batch's 32-lane words, shared by the gate kernels, the compiled
// gate kernels (this header is handed to NVRTC) and their CPU tests.
#pragma once

#include <stdint.h>

#include "stim.h"

namespace rrtl {

// Lanes of 32-lane word gw that exist in a batch of `lanes` lanes.
RRTL_HD uint32_t valid_mask(uint32_t gw, uint32_t lanes) {
  uint32_t base = gw * 32u;
  if (base >= lanes) return 0u;
  uint32_t n = lanes - base;
  return n >= 32u ? 0xFFFFFFFFu : ((1u << n) - 1u);
}

// Lanes of word gw with a first-detection cycle in `detect`, which has one
// entry a lane and no more (a caller's buffer, in runs on device pointers).
RRTL_HD uint32_t detected_lanes(const uint32_t* detect, uint32_t gw, uint32_t lanes) {
  const uint32_t have = valid_mask(gw, lanes);
  uint32_t det = 0u;
  for (uint32_t b = 0; b < 32u; ++b)
    if ((have >> b & 1u) && detect[gw * 32u + b] != 0xFFFFFFFFu) det |= 1u << b;
  return det;
}

}  // namespace rrtl
