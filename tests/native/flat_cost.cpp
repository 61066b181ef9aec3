// Modelled clocks of a tile-cycle of each flat shape (test infrastructure).
#include <cstdint>
#include <cstdio>

#include "../../rrtl_gb300/csrc/design.h"
#include "../../rrtl_gb300/csrc/flatprog.h"

using namespace rrtl;

// shapes: V, N, Q, narrow; the statistics are those of the 4-word program, as for any design that fits one.
extern "C" int flat_costs(const char* json, size_t len, const char* top, uint32_t n, const uint32_t* shapes, double* clocks) {
  try {
    Design d = design_from_json(json, len);
    GateProgram gp = build_gate_program(lower_to_machine_program(lower_to_packed_program(d, top)), 8);
    FlatProgram fp = build_flat_program(gp, 4);
    for (uint32_t i = 0; i < n; ++i) {
      FlatShape x;
      x.V = shapes[4 * i];
      x.N = shapes[4 * i + 1];
      x.Q = shapes[4 * i + 2];
      x.narrow = shapes[4 * i + 3] != 0;
      clocks[i] = flat_tile_cost(fp, 4, x);
    }
    return 0;
  } catch (const std::exception&) {
    return 1;
  }
}
