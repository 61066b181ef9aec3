// Per-design compiled gate kernels: emitter (see gate_jit.h).
//
// The emitted kernel follows the gate engine's cycle exactly as the fused and
// plain kernels do (gate_kernels.cu): stimulus into the source nets, every
// cell in level order, record (trace word, hash term, detection against lane
// 0 of the word, trace checks), then the register commit with synchronous
// reset select; the closing settle re-evaluates the cells and the launch
// writes back the sources and every signal net.
#include "gate_jit.h"

#include <algorithm>
#include <cstdio>

#include "../../include/rrtl_cuda.h"

namespace rrtl {

namespace {

std::string u(uint64_t v) { return std::to_string(v) + "u"; }
std::string n(uint32_t net) {
  if (net == kNetConst0) return "0u";
  if (net == kNetConst1) return "0xFFFFFFFFu";
  return "n" + std::to_string(net);
}

// The cells in level order, each net a constant of the enclosing block; with
// `store`, every signal net is written back as it is computed, so that the
// closing settle keeps no more nets live than a cycle does.
void cells(std::string& o, const GateProgram& gp, bool store) {
  for (const GateCell& c : gp.cells) {
    if (c.pad) continue;
    char lut[8];
    snprintf(lut, sizeof lut, "0x%02x", c.lut);
    o += "    const uint32_t " + n(c.out) + " = lop3<" + lut + ">(" + n(c.in[0]) + ", " + n(c.in[1]) + ", " + n(c.in[2]) +
         ");\n";
    if (store && gp.net_signal[c.out] >= 0) o += "    G[(size_t)" + u(c.out) + " * wp] = " + n(c.out) + ";\n";
  }
}

}  // namespace

// The tables' values as bytes: looked up on every run, before its first copy
// (as text, a run of 40 entries on 64 lanes took 50.0 instead of 48.2 us).
std::string GateRunTables::key() const {
  std::string k;
  auto put = [&](const auto& v) { k.append(reinterpret_cast<const char*>(&v), sizeof v); };
  k.reserve(16 + stim.size() * 16 + rec.size() * 4);
  put(mode);
  put((uint32_t)stim.size());
  for (const GateStimDev& t : stim) {
    put(t.net);
    put(t.kind);
    put(t.param);
  }
  for (const GateRecDev& t : rec) put(t.net);
  return k;
}

namespace {

// Work of a block's service warps: stimulus entries by kind (drawn, uniform,
// traced) in buffer order, and whether the run records anything.
struct Service {
  uint32_t warps = 0;
  std::vector<size_t> stim;  // run.stim entries, random first, then uniform, then traced
  size_t n_random = 0, n_uniform = 0;
};

bool run_records(const GateRunTables& run) {
  return !run.rec.empty() && (run.mode & (RRTL_REC_HASH | RRTL_REC_TRACE | RRTL_REC_DETECT | RRTL_REC_CHECK));
}

Service plan_service(const GateRunTables& run, uint32_t service) {
  Service S;
  if (!service) return S;
  for (uint32_t kind : {RRTL_STIM_RANDOM, RRTL_STIM_RANDOM_UNIFORM, RRTL_STIM_TRACE}) {
    for (size_t i = 0; i < run.stim.size(); ++i)
      if (run.stim[i].kind == kind) S.stim.push_back(i);
    if (kind == RRTL_STIM_RANDOM) S.n_random = S.stim.size();
    if (kind == RRTL_STIM_RANDOM_UNIFORM) S.n_uniform = S.stim.size() - S.n_random;
  }
  // about two entries a warp and cycle
  const size_t items = S.stim.size() + (run_records(run) ? run.rec.size() : 0);
  S.warps = (uint32_t)std::min<size_t>(service, (items + 1) / 2);
  return S;
}

}  // namespace

// A block is 32 words: warp 0 keeps every net of its words in registers and
// evaluates the cells; the other warps draw the next cycle's stimulus and
// finish the last cycle's record, each for the same 32 words, through shared
// memory rows written one cycle and read the next (one barrier a cycle).
//
// Bound: latency. A batch is few warps (262,144 lanes are 256 blocks), so one
// warp's chain of instructions per cycle decides, and with stimulus and hash
// in that chain it was mostly those; and the instruction cache: the code of a
// cycle has to fit it, or every SM streams it from L2 (service loops unrolled
// per entry: 16-bit ALU planes, 17 hashed outputs, 1.0 us a cycle on one SM,
// 2.1 on 152; rolled 0.76 on either). Nets are constants of the cycle's block
// and the closing settle stores each as it is computed: kept live across the
// loop they spilled (12 KB of stack; the ALU planes 5.1 us a cycle without
// records, 0.87 now on one warp, 0.68 with service warps). us per cycle,
// before and now: crc32 (195 cells, 8 random inputs, 32 hashed outputs) at
// 65,536 lanes 2.51 and 0.65, at 262,144 2.50 and 1.06, at 1,048,576 3.11 and
// 2.28; ALU planes (646 cells, hashed) at 65,536 lanes 6.7 and 0.75, at
// 1,048,576 19.6 and 2.9.
// A cycle's hash sums are kept in shared memory and added to the run's hashes
// by one burst of atomics a block every 32 cycles (each block's on a cycle of
// its own), not by an atomic per cycle and warp: all blocks add to the same
// addresses, and a burst per service warp cost crc32 at 155,648
// lanes 0.2 us a cycle.
std::string gate_jit_source(const GateProgram& gp, const GateRunTables& run, uint32_t service) {
  const uint32_t mode = run.mode;
  const bool trace = mode & RRTL_REC_TRACE, hash = mode & RRTL_REC_HASH, detect = mode & RRTL_REC_DETECT,
             check = mode & RRTL_REC_CHECK;
  const Service S = plan_service(run, service);
  const uint32_t H = S.warps;
  const size_t ns = S.stim.size(), nr = run_records(run) ? run.rec.size() : 0;
  std::vector<int> buffer_of(run.stim.size(), -1);
  for (size_t i = 0; i < ns; ++i) buffer_of[S.stim[i]] = (int)i;
  std::string o;
  o += "// Compiled gate kernel (generated from the design's gate program and one run's tables).\n";
  o += "#include \"gate_common.h\"\n";
  o += "extern \"C\" __global__ void __launch_bounds__(" + std::to_string(gate_jit_threads(run, service)) +
       ", 1) rrtl_gate_jit(const rrtl::GateRunDev R) {\n";
  o += "  using namespace rrtl;\n";
  if (ns) {
    o += "  __shared__ uint32_t stim_rows[2][" + u(ns) + "][32];  // drawn for the next cycle\n";
    o += "  __shared__ unsigned long long stim_key[" + u(ns) + "];  // stream keys, or the column of a traced input\n";
  }
  if (nr && H) o += "  __shared__ uint32_t rec_rows[2][" + u(nr) + "][32];  // recorded in the last cycle\n";
  if (nr && hash) o += "  __shared__ unsigned long long hash_rows[" + u(std::max(1u, H)) + "][64][4];  // of the last 64 cycles\n";
  o += "  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;\n";
  o += "  const uint32_t w = blockIdx.x * 32u + lane;  // 32-lane word\n";
  o += "  const bool own = w < R.words_pad;\n";
  o += "  const uint32_t cycles = (uint32_t)R.cycles;\n";
  const std::string hash_end =
      "        if (w >= R.words) h = 0ull;  // (once, so that the terms' chains interleave)\n"
      "        h += __shfl_xor_sync(0xFFFFFFFFu, h, 16);\n        h += __shfl_xor_sync(0xFFFFFFFFu, h, 8);\n"
      "        h += __shfl_xor_sync(0xFFFFFFFFu, h, 4);\n";
  if (nr && hash) {
    // The sums of the cycles since the last burst that end with cycle e, added to the run's hashes: lane l takes e - l.
    o += "  auto burst = [&](uint32_t e) {\n";
    o += "    if (lane <= ((e + blockIdx.x) & 31u) && lane <= e) {\n";
    o += "      unsigned long long t = 0ull;\n";
    o += "      for (uint32_t k = 0; k < " + u(std::max(1u, H)) + "; ++k)\n";
    o += "        for (uint32_t j = 0; j < 4u; ++j) t += hash_rows[k][(e - lane) & 63u][(lane + j) & 3u];\n";
    o += "      if (t) atomicAdd(R.out_hash + (R.cycle_base + e - lane), t);\n    }\n  };\n";
  }
  auto detect_state = [&](const char* cond) {
    // lanes detected by an earlier launch of the run stay detected
    o += std::string("    uint32_t det = ") + cond + "detected_lanes(R.detect, w, R.lanes)" + (*cond ? " : 0u" : "") + ";\n";
  };
  const std::string detect_end =
      "        uint32_t nb = w < R.words ? diff & ~det & vm : 0u;\n        det |= nb;\n"
      "        while (nb) { const uint32_t b = __ffs(nb) - 1u; R.detect[w * 32u + b] = (uint32_t)c; nb &= nb - 1u; }\n";
  const std::string columns = u(run.rec.size());
  const bool inline_record = nr && !H;
  // ---- service warps: rolled loops over the entries (unrolled, an entry of each
  // kind for every warp, the code no longer fits the instruction cache)
  if (H) {
    o += "  if (warp != 0u) {\n";
    o += "    const uint32_t me = warp - 1u;\n";
    if (nr) o += "    const uint32_t vm = valid_mask(w, R.lanes);\n";
    if (nr && detect) detect_state("me == 0u ? ");
    if (ns) {
      o += "    if (me == 0u && lane == 0u) {\n";
      for (size_t i = 0; i < ns; ++i) {
        const GateStimDev& t = run.stim[S.stim[i]];
        char buf[64];
        snprintf(buf, sizeof buf, "0x%llxull", (unsigned long long)t.param);
        o += "      stim_key[" + std::to_string(i) + "] = " +
             (t.kind == RRTL_STIM_TRACE ? std::string(buf) : "stim_stream_key(R.seed, " + std::string(buf) + ")") + ";\n";
      }
      o += "    }\n";
      o += "    __syncwarp();\n    asm volatile(\"bar.sync 1, " + std::to_string(32 * H) + ";\" ::: \"memory\");\n";
      o += "    auto draw = [&](unsigned long long c, uint32_t (*rows)[32]) {\n";
      const size_t e0 = S.n_random, e1 = e0 + S.n_uniform;
      if (e0)
        o += "#pragma unroll 2\n      for (uint32_t s = me; s < " + u(e0) + "; s += " + u(H) +
             ") rows[s][lane] = stim_key_word(stim_key[s], c, R.word_base + w);\n";
      if (e1 > e0)
        o += "      for (uint32_t s = " + u(e0) + " + me; s < " + u(e1) + "; s += " + u(H) +
             ") rows[s][lane] = 0u - (stim_key_word(stim_key[s], c, 0ull) & 1u);\n";
      if (ns > e1)
        o += "      for (uint32_t s = " + u(e1) + " + me; s < " + u(ns) + "; s += " + u(H) +
             ") rows[s][lane] = w < R.words ? R.in_trace[((size_t)c * R.n_trace_cols + stim_key[s]) * R.words + w] : 0u;\n";
      o += "    };\n";
    }
    if (nr) {
      o += "    auto record = [&](uint32_t i, uint32_t (*rows)[32]) {\n";
      o += "      const unsigned long long c = R.cycle_base + i;\n";
      if (hash || trace || check) {
        if (hash) o += "      unsigned long long h = 0ull, salts = 0ull;  // salts: one per lane, shared by shuffles\n";
        o += "#pragma unroll 4\n";
        o += "      for (uint32_t k = me, t = 0; k < " + u(nr) + "; k += " + u(H) + ", ++t) {\n";
        if (hash) o += "        if ((t & 31u) == 0u) salts = hash_salt(c, k + lane * " + u(H) + ");\n";
        o += "        const uint32_t v = rows[k][lane] & vm;\n";
        if (trace) o += "        if (w < R.words) R.out_trace[((size_t)c * " + columns + " + k) * R.words + w] = v;\n";
        if (hash) o += "        h += hash_term_salted(__shfl_sync(0xFFFFFFFFu, salts, t & 31u), R.word_base + w, v);\n";
        if (check) o += "        if (w < R.words) check_word(R, c, k, w, v);\n";
        o += "      }\n";
        if (hash) o += hash_end + "        if (lane < 4u) hash_rows[me][i & 63u][lane] = h;\n";
      }
      if (detect) {
        o += "      if (me == 0u) {\n        uint32_t diff = 0u;\n#pragma unroll 4\n";
        o += "        for (uint32_t k = 0; k < " + u(nr) + "; ++k) { const uint32_t v = rows[k][lane] & vm; diff |= v ^ (0u - (v & 1u)); }\n";
        o += detect_end + "      }\n";
      }
      o += "    };\n";
    }
    if (ns) o += "    if (cycles) draw(R.cycle_base, stim_rows[0]);\n";
    o += "    __syncthreads();\n";
    o += "    for (uint32_t i = 0; i < cycles; ++i) {\n";
    if (ns) o += "      if (i + 1u < cycles) draw(R.cycle_base + i + 1u, stim_rows[(i + 1u) & 1u]);\n";
    if (nr && hash) o += "      if (me == 0u && i > 1u && ((i - 2u + blockIdx.x) & 31u) == 31u) burst(i - 2u);\n";
    if (nr) o += "      if (i) record(i - 1u, rec_rows[(i - 1u) & 1u]);\n";
    o += "      __syncthreads();\n    }\n";
    if (nr) o += "    if (cycles) record(cycles - 1u, rec_rows[(cycles - 1u) & 1u]);\n";
    if (nr && hash) {
      o += "    __syncwarp();\n    asm volatile(\"bar.sync 1, " + std::to_string(32 * H) + ";\" ::: \"memory\");\n";
      o += "    if (me == 0u && cycles) {\n";
      o += "      if (cycles > 1u && ((cycles - 2u + blockIdx.x) & 31u) == 31u) burst(cycles - 2u);\n";
      o += "      burst(cycles - 1u);\n    }\n";
    }
    o += "    return;\n  }\n";
  }
  // ---- the compute warp: every net a register; sources loaded, cell outputs declared
  o += "  uint32_t* G = R.nets + w;\n";
  o += "  const size_t wp = R.words_pad;\n";
  std::vector<uint8_t> produced(gp.n_nets, 0);
  for (const GateCell& c : gp.cells)
    if (!c.pad) produced[c.out] = 1;
  std::vector<uint32_t> sources;
  for (uint32_t k = 2; k < gp.n_nets; ++k)
    if (gp.net_is_source[k] && !produced[k]) sources.push_back(k);
  for (uint32_t k : sources) o += "  uint32_t " + n(k) + " = own ? G[(size_t)" + u(k) + " * wp] : 0u;\n";
  if (inline_record) {
    o += "    const uint32_t vm = valid_mask(w, R.lanes);\n";
    if (detect) detect_state("");
  }
  if (H) o += "  __syncthreads();\n";
  o += "  unsigned long long c = R.cycle_base;\n";
  o += "  for (uint32_t i = 0; i < cycles; ++i, ++c) {\n";
  for (size_t k = 0; k < run.stim.size(); ++k) {
    const GateStimDev& s = run.stim[k];
    if (s.kind == RRTL_STIM_HOLD) continue;
    if (buffer_of[k] >= 0) {
      o += "    " + n(s.net) + " = stim_rows[i & 1u][" + std::to_string(buffer_of[k]) + "][lane];\n";
      continue;
    }
    char buf[160];
    snprintf(buf, sizeof buf, "GateStimDev{0u, %uu, %uu, 0u, 0x%llxull}", s.net, s.kind, (unsigned long long)s.param);
    o += "    " + n(s.net) + " = stim_value(" + buf + ", R, c, w, " + n(s.net) + ");\n";
  }
  cells(o, gp, false);
  if (inline_record) {
    o += "    {\n";
    if (hash) o += "        unsigned long long h = 0ull;\n";
    if (detect) o += "        uint32_t diff = 0u;\n";
    for (size_t q = 0; q < nr; ++q) {
      const std::string salt = "salt" + std::to_string(q / 32);
      if (hash && q % 32 == 0)  // the cycle's hash salts, one per lane of the warp, shared by shuffles
        o += "        const unsigned long long " + salt + " = hash_salt(c, " + u(q) + " + lane);\n";
      o += "        { const uint32_t v = " + n(run.rec[q].net) + " & vm;";
      if (trace) o += " if (w < R.words) R.out_trace[((size_t)c * " + columns + " + " + u(q) + ") * R.words + w] = v;";
      if (hash) o += " h += hash_term_salted(__shfl_sync(0xFFFFFFFFu, " + salt + ", " + u(q % 32) + "), R.word_base + w, v);";
      if (detect) o += " diff |= v ^ (0u - (v & 1u));";
      if (check) o += " if (w < R.words) check_word(R, c, " + u(q) + ", w, v);";
      o += " }\n";
    }
    if (hash) {
      o += hash_end + "        if (lane < 4u) hash_rows[0][i & 63u][lane] = h;\n";
      o += "        if (((i + blockIdx.x) & 31u) == 31u || i + 1u == cycles) {\n";
      o += "          __syncwarp();\n          burst(i);\n          __syncwarp();\n        }\n";
    }
    if (detect) o += detect_end;
    o += "    }\n";
  }
  for (size_t k = 0; k < nr && !inline_record; ++k)
    o += "    rec_rows[i & 1u][" + std::to_string(k) + "][lane] = " + n(run.rec[k].net) + ";\n";
  // commit: every register's next value from the pre-commit nets, then all at once
  if (!gp.regs.empty()) {
    o += "    {\n";
    for (size_t k = 0; k < gp.regs.size(); ++k) {
      const GateReg& r = gp.regs[k];
      std::string e = n(r.d_net);
      if (r.has_reset) {
        // m = reset asserted per lane; next = (m & reset value) | (~m & d)
        const std::string m = r.active_low ? "(~" + n(r.rst_net) + ")" : n(r.rst_net);
        const std::string rv = r.reset_value ? "0xFFFFFFFFu" : "0u";
        e = "((" + m + " & " + rv + ") | (~" + m + " & " + n(r.d_net) + "))";
      }
      o += "      const uint32_t q" + std::to_string(k) + " = " + e + ";\n";
    }
    for (size_t k = 0; k < gp.regs.size(); ++k) o += "      " + n(gp.regs[k].q_net) + " = q" + std::to_string(k) + ";\n";
    o += "    }\n";
  }
  if (H) o += "    __syncthreads();\n";
  o += "  }\n";
  o += "  if (!own) return;\n";
  for (uint32_t k : sources) o += "  G[(size_t)" + u(k) + " * wp] = " + n(k) + ";\n";
  o += "  if (R.final_settle) {\n";
  cells(o, gp, true);
  o += "  }\n";
  o += "}\n";
  return o;
}

uint32_t gate_jit_threads(const GateRunTables& run, uint32_t service) { return 32u * (1u + plan_service(run, service).warps); }

void gate_jit_build(const GateProgram& gp, const GateRunTables& run, uint32_t service, int device, JitKernel* J) {
  if (gp.n_real_cells > kGateJitMaxCells) {
    J->error = "gate program of " + std::to_string(gp.n_real_cells) + " cells runs on the fused kernel";
    return;
  }
  J->threads = gate_jit_threads(run, service);
  jit_build_kernel(gate_jit_source(gp, run, service), device, "rrtl_gate_jit", J);
}

cudaError_t launch_gate_jit(const JitKernel& J, const GateRunDev& R, cudaStream_t st) {
  GateRunDev r = R;
  void* args[] = {&r};
  return cudaLaunchKernel(reinterpret_cast<const void*>(J.fn), dim3((R.words_pad + 31u) / 32u), dim3(J.threads), args, 0, st);
}

std::string gate_fused_jit_source(const GateProgram& gp) {
  std::vector<uint8_t> used(256, 0);
  used[0] = 1;  // an empty run (header word 0) dispatches to class 0
  for (const GateCell& c : gp.cells) used[c.lut] = 1;
  // the kernel's shape as the host library was built with it (launch size, shares)
  std::string o = "// rrtl_gate_fused_jit: gate_fused_kernel<" + std::to_string(gp.tile_words) +
                  "> for one design's truth-table classes\n#define RRTL_FUSED_WARPS " +
                  std::to_string(kGateFusedWarps) + "\n#define RRTL_FUSED_CTAS_PER_SM " +
                  std::to_string(kGateFusedCtasPerSm) + "\n#define RRTL_FUSED_V " + std::to_string(RRTL_FUSED_V) +
                  "\n#define RRTL_LUT_CLASSES(X)";
  for (int l = 0; l < 256; ++l)
    if (used[l]) o += " X(" + std::to_string(l) + ")";
  o += "\n#include \"gate_fused.h\"\n";
  o += "extern \"C\" __global__ void __launch_bounds__(rrtl::kFusedThreads, rrtl::kGateFusedCtasPerSm)\n";
  o += "rrtl_gate_fused_jit(rrtl::GateProgDev P, rrtl::GateRunDev R) {\n";
  o += "  rrtl::fused_kernel_body<" + std::to_string(gp.tile_words) + ", true>(P, R);\n}\n";
  return o;
}

void gate_fused_jit_build(const GateProgram& gp, int device, JitKernel* J) {
  for (const GateCell& c : gp.cells)
    if (!lut_is_canonical(c.lut)) {
      J->error = "a cell's truth table is not a class representative";
      return;
    }
  jit_build_kernel(gate_fused_jit_source(gp), device, "rrtl_gate_fused_jit", J);
}

cudaError_t launch_gate_fused_jit(const JitKernel& J, const GateProgDev& P, const GateRunDev& R, uint32_t grid,
                                  size_t smem, cudaStream_t st) {
  GateProgDev p = P;
  GateRunDev r = R;
  void* args[] = {&p, &r};
  return cudaLaunchKernel(reinterpret_cast<const void*>(J.fn), dim3(grid), dim3(kGateFusedWarps * 32u), args, smem, st);
}

}  // namespace rrtl
