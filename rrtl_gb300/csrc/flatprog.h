// Flat gate program: the per-cycle form of a GateProgram for the flat fused
// kernel (gate_flat.h).
//
// The fused kernel of gate_fused.h evaluates runs of cells that share one
// truth table, so its groups are drawn from small buckets and every run pays
// a dispatch. Here a cell carries its own function as coefficient bits, so
// any cells of a level may share a warp step:
//
//  1. Packing: within a cycle only the recorded and committed nets can be
//     observed, so inverters and buffers are folded into their readers and a
//     net with a single reader is folded into that reader where the result
//     still has at most three inputs. (FlatOptions::settle: the closing
//     settle's program, which computes every signal and writes it back;
//     FlatOptions::observe: a row for every signal, for stuck-at forces.)
//  2. Register folding: a cell that computes a register's next value writes
//     the register's own row, with the synchronous reset in its function, at
//     a level after every other read of the register. Registers for which
//     no such level exists stay on a commit list.
//  3. Rows ("slots") of V words by liveness; cells grouped by G = 32/V so
//     that the rows read at one operand position, and the rows written, fall
//     on distinct bank residues (slot mod G).
//     The 50,000-gate netlist: 51,300 cells unpacked, 36,900 packed; 16,500
//     wavefronts per 4-word vector and cycle, 4% above one per group and row
//     position (the fused program's 8-word groups take 47,100 per two vectors).
//  4. A schedule: per warp a stream of 16-byte-per-lane entries in level
//     order, each with the number of level barriers to pass before it.
#pragma once

#include <cstdint>
#include <vector>

#include "flat_shape.h"
#include "gateprog.h"

namespace rrtl {

// One lane of a stream entry.
//  two cells of two inputs: x = a | b << 16, y = out | meta; z, w the second
//  one cell of three inputs (kFlatDevThree): x = a | b << 16, y = out | meta,
//    z = c, w = coefficients
// meta (y bits 16-31): kFlatDevSync, kFlatDevThree, and the coefficients of a
// two-input function f = k0 ^ a k1 ^ b k2 ^ ab k3 in bits 23 (k0), 31 (k1),
// 22 (k2), 30 (k3): byte sign bits, which one byte permute turns into a mask.
// Three inputs: f = g0 ^ c g1, coefficient j of g0 in bit 8j + 7 of w, of g1
// in bit 8j + 6. An entry without cells writes scratch rows.
struct FlatLane {
  uint32_t x = 0, y = 0, z = 0, w = 0;
};

struct FlatCell {
  uint32_t in[3] = {0, 0, 0};  // nets
  uint32_t out = 0;            // net (a folded register's Q net)
  uint8_t lut = 0;             // over a <-> 0xF0, b <-> 0xCC, c <-> 0xAA
  uint8_t n = 0;               // inputs
  int32_t level = 0;
  int32_t reg = -1;            // register written in place, -1: none
};

struct FlatProgram {
  uint32_t V = 4, G = 8;
  uint32_t warps = 16;                    // streams: warps of the set that walks the program
  uint32_t n_levels = 0;
  std::vector<int32_t> net_slot;          // -1: not resident
  std::vector<uint8_t> recordable;        // net holds its value in its slot when the cycle's settle ends
  uint32_t n_slots = 0;                   // the first G are scratch rows of idle lanes
  std::vector<int32_t> net_level;         // level a cell writes the net's row at, -1: none does
  std::vector<uint8_t> net_warp;          // warp that does
  std::vector<uint32_t> source_nets;      // loaded at the start of a run, written back at its end
  std::vector<uint32_t> commit;           // GateProgram::regs indices not folded
  std::vector<FlatLane> stream;           // [entry][32 lanes]
  std::vector<uint32_t> stream_net;       // settle: [entry][32][2] signal net each cell writes back, ~0: none
  std::vector<uint32_t> warp_begin;       // per warp: first entry (a multiple of kFlatPrefetch); size warps + 1
  std::vector<uint32_t> warp_tail;        // level barriers after a warp's last entry
  // shared-memory wavefronts of one row vector's cell accesses, and their floor
  uint64_t wavefronts = 0, floor_wavefronts = 0;
  uint32_t n_two = 0, n_three = 0, n_entries = 0;
};

struct FlatOptions {
  bool pack = true;       // (false: only for the CPU tests of the other parts, as below)
  bool fold_regs = true;
  bool settle = false;   // a closing settle: every signal computed and written back, no registers committed
  bool observe = false;  // every signal keeps a row of its own (stuck-at forces act on any of them)
  uint32_t max_warps = kFlatComputeThreads / 32;  // of the set; a program of few entries a level uses fewer
  uint32_t max_slots = 0;  // above this, a row is placed at any residue before the slot array grows (0: no limit)
};

FlatProgram build_flat_program(const GateProgram& gp, uint32_t V, const FlatOptions& opt = {});

// A shape of the flat kernel: row width V (0: none), vectors per warp set N,
// warp sets Q.
struct FlatShape {
  uint32_t V = 0, N = 1, Q = 1;
  bool narrow = false;  // on the kFlatNarrow program
  uint32_t words() const { return V * N * Q; }
};

// Clocks of one tile-cycle, from the statistics of the program built for row
// width `base`.
double flat_tile_cost(const FlatProgram& fp, uint32_t base, const FlatShape& x);

}  // namespace rrtl
