// CPU emulation of the flat gate kernel's program (test infrastructure).
//
// Runs the per-warp entry streams of a FlatProgram as the kernel decodes
// them, level by level, over `lanes` lanes, with the register commit list,
// and checks what the kernel relies on without checking it: every warp passes
// the same level barriers, no lane reads or writes a row that another lane
// writes in the same level, rows stay inside the slot array. Stimulus and
// the per-cycle output hash follow stim.h.
#include <cstdint>
#include <cstdio>
#include <map>
#include <string>
#include <vector>

#include "../../include/rrtl_cuda.h"
#include "../../rrtl_gb300/csrc/design.h"
#include "../../rrtl_gb300/csrc/flatprog.h"
#include "../../rrtl_gb300/csrc/stim.h"

using namespace rrtl;

namespace {

struct Fail {
  std::string msg;
};

uint32_t mask_of(uint32_t w, int bit) { return (w >> bit) & 1u ? 0xFFFFFFFFu : 0u; }

uint32_t two(uint32_t meta, uint32_t a, uint32_t b) {
  const uint32_t k0 = mask_of(meta, 23), k1 = mask_of(meta, 31), k2 = mask_of(meta, 22), k3 = mask_of(meta, 30);
  return k0 ^ (a & k1) ^ (b & k2) ^ (a & b & k3);
}

}  // namespace

// Parts of a run over `blocks` blocks: every tile's cycles once and in order, a
// split tile's first part its block's first, its last part waiting for it and
// never before the time it is done at equal speed. 0: as stated.
extern "C" int emu_flat_parts(uint32_t n_tiles, uint64_t cycles, uint32_t blocks) {
  std::vector<uint64_t> first(n_tiles, 0), last(n_tiles, 0), done(n_tiles, 0);
  const uint64_t share = (n_tiles * cycles + blocks - 1) / blocks;
  for (int pass = 0; pass < 2; ++pass)
    for (uint32_t b = 0; b < blocks; ++b) {
      uint64_t t = 0;
      for (uint32_t k = 0;; ++k) {
        const FlatPart p = flat_part(n_tiles, cycles, b, blocks, k);
        if (!p.n) break;
        if (p.tile >= n_tiles || p.c0 + p.n > cycles || (p.first && p.last)) return 1;
        if (p.first != (p.c0 == 0 && p.n < cycles) || p.last != (p.c0 > 0)) return 2;
        if (p.first && k) return 3;
        if (pass == 0) (p.last ? last : first)[p.tile] += p.n;
        if (p.first) done[p.tile] = p.n;
        if (pass && p.last && (p.c0 != first[p.tile] || done[p.tile] > t)) return 4;
        t += p.n;
      }
      if (t > share) return 5;
    }
  for (uint32_t i = 0; i < n_tiles; ++i)
    if (first[i] + last[i] != cycles) return 6;
  return 0;
}

extern "C" int emu_flat_run(const char* json, size_t len, const char* top, uint32_t V, uint32_t pack, uint32_t fold,
                            uint32_t max_warps, uint32_t max_slots, uint32_t lanes, uint64_t cycles, uint64_t seed,
                            uint64_t lane_base, uint32_t n_stim, const uint32_t* stim_sig, const uint32_t* stim_kind,
                            const uint64_t* stim_param, uint32_t n_rec, const uint32_t* rec_sig, uint64_t* out_hash,
                            uint32_t* stats, char* err, size_t errcap) {
  try {
    Design d = design_from_json(json, len);
    MachineProgram mp = lower_to_machine_program(lower_to_packed_program(d, top));
    GateProgram gp = build_gate_program(mp, 8);
    FlatOptions opt;
    opt.pack = pack != 0;
    opt.observe = pack == 2;  // 2: every signal keeps a row
    opt.settle = pack == 3;   // 3: the closing settle's program, its signal nets taken from its write-back
    opt.fold_regs = fold != 0;
    opt.max_warps = max_warps;
    opt.max_slots = max_slots;
    FlatProgram fp = build_flat_program(gp, V, opt);
    for (uint32_t s = 0; opt.observe && s < gp.n_signals; ++s) {
      const uint32_t net = gp.signal_net[s];
      if (!gp.net_is_source[net] && fp.net_slot[net] >= 0 && fp.net_level[net] < 0) throw Fail{"a row no cell writes"};
    }
    const uint32_t warps = fp.warps;
    if (warps < 1 || warps > max_warps) throw Fail{"streams"};
    if (stats) {
      const uint32_t s[] = {fp.n_two,   fp.n_three, fp.n_levels, fp.n_slots, fp.n_entries, (uint32_t)fp.wavefronts,
                            (uint32_t)fp.floor_wavefronts, (uint32_t)fp.commit.size()};
      for (size_t i = 0; i < sizeof s / 4; ++i) stats[i] = s[i];
    }
    auto fail = [](const std::string& m) { throw Fail{m}; };
    const uint32_t words = (lanes + 31) / 32;
    const uint64_t word_base = lane_base / 32;
    std::vector<uint32_t> S((size_t)fp.n_slots * words, 0u);
    auto row = [&](uint32_t s) {
      if (s >= fp.n_slots) throw Fail{"a row outside the slot array"};
      return &S[(size_t)s * words];
    };
    std::vector<uint32_t> rec_net(n_rec), stim_net(n_stim);
    for (uint32_t i = 0; i < n_rec; ++i) {
      rec_net[i] = gp.signal_net.at(rec_sig[i]);
      if (!opt.settle && !fp.recordable[rec_net[i]]) fail("a recorded net is not recordable");
    }
    for (uint32_t i = 0; i < n_stim; ++i) stim_net[i] = gp.signal_net.at(stim_sig[i]);
    if (fp.warp_begin.size() != warps + 1) fail("warp table size");
    for (uint32_t w = 0; w < warps; ++w)
      if ((fp.warp_begin[w + 1] - fp.warp_begin[w]) % kFlatPrefetch) fail("a stream is not a multiple of the prefetch");
    if (fp.stream_net.size() != (opt.settle ? fp.stream.size() * 2 : 0)) fail("write-back table size");
    if (opt.settle && !fp.commit.empty()) fail("a settle commits registers");
    std::vector<std::vector<uint32_t>> back(opt.settle ? gp.n_nets : 0);
    std::map<std::pair<uint32_t, uint32_t>, uint32_t> row_net;  // level and row written -> net
    for (uint32_t n = 0; opt.settle && n < gp.n_nets; ++n)
      if (!gp.net_is_source[n] && fp.net_level[n] >= 0) row_net[{(uint32_t)fp.net_level[n], (uint32_t)fp.net_slot[n]}] = n;
    auto value = [&](uint32_t net) -> const uint32_t* {  // a net's words at the end of the cycle
      if (!opt.settle || gp.net_is_source[net]) return row((uint32_t)fp.net_slot[net]);
      if (back[net].empty()) throw Fail{"a net that is not written back"};
      return back[net].data();
    };
    std::vector<uint32_t> commit = fp.commit;
    for (uint32_t k = 0; opt.settle && k < gp.regs.size(); ++k) commit.push_back(k);
    std::vector<uint64_t> wrote(fp.n_slots, ~0ull), read(fp.n_slots, ~0ull);  // lane that touched the row in this level
    for (uint64_t c = 0; c < cycles; ++c) {
      for (auto& v : back) v.clear();
      for (uint32_t i = 0; i < n_stim; ++i)
        for (uint32_t w = 0; w < words; ++w) {
          uint32_t& v = row((uint32_t)fp.net_slot[stim_net[i]])[w];
          switch (stim_kind[i]) {
            case RRTL_STIM_RANDOM: v = stim_word(seed, stim_param[i], c, word_base + w); break;
            case RRTL_STIM_RANDOM_UNIFORM: v = stim_uniform_word(seed, stim_param[i], c); break;
            case RRTL_STIM_PULSE: v = c < stim_param[i] ? 0xFFFFFFFFu : 0u; break;
            case RRTL_STIM_CONST: v = (stim_param[i] & 1u) ? 0xFFFFFFFFu : 0u; break;
            case RRTL_STIM_HOLD: break;
            default: fail("stimulus kind outside the emulator");
          }
        }
      std::vector<uint32_t> at(warps), level(warps, 0);
      for (uint32_t w = 0; w < warps; ++w) at[w] = fp.warp_begin[w];
      for (uint32_t L = 0; L < fp.n_levels; ++L) {
        std::fill(wrote.begin(), wrote.end(), ~0ull);
        std::fill(read.begin(), read.end(), ~0ull);
        for (uint32_t w = 0; w < warps; ++w)
          for (; at[w] < fp.warp_begin[w + 1]; ++at[w]) {
            const FlatLane* e = &fp.stream[(size_t)at[w] * 32];
            const uint32_t sync = e[0].y & kFlatDevSync ? 1u : 0u, three = e[0].y & kFlatDevThree;
            if (level[w] + sync > L) break;
            level[w] += sync;
            for (uint32_t l = 0; l < 32; ++l) {
              if (((e[l].y & kFlatDevSync) != 0) != (sync != 0) || (e[l].y & kFlatDevThree) != three)
                fail("an entry's lanes disagree");
              const int parts = three ? 1 : 2;
              for (int h = 0; h < parts; ++h) {
                const uint32_t x = h ? e[l].z : e[l].x, y = h ? e[l].w : e[l].y;
                const uint32_t sl[3] = {x & 0xFFFFu, x >> 16, e[l].z};
                const uint64_t id = ((uint64_t)at[w] * 2 + (uint64_t)h) * 32 + l;
                const uint32_t so = y & 0xFFFFu;
                for (int k = 0; k < (three ? 3 : 2); ++k) {
                  row(sl[k]);
                  if (sl[k] < fp.G || so < fp.G) continue;  // scratch rows; an idle lane's result is never read
                  if (wrote[sl[k]] != ~0ull && wrote[sl[k]] != id) fail("a lane reads a row written in its own level");
                  read[sl[k]] = read[sl[k]] == ~0ull || read[sl[k]] == id ? id : ~0ull - 1;
                }
                if (so >= fp.G) {
                  if (wrote[so] != ~0ull) fail("a row is written twice in a level");
                  if (read[so] != ~0ull && read[so] != id) fail("a lane writes a row read in its own level");
                  wrote[so] = id;
                }
                std::vector<uint32_t> out(words);
                for (uint32_t q = 0; q < words; ++q) {
                  const uint32_t a = row(sl[0])[q], b = row(sl[1])[q];
                  if (!three) {
                    out[q] = two(y, a, b);
                  } else {
                    const uint32_t cc = row(sl[2])[q], W = e[l].w;
                    const uint32_t g0 = mask_of(W, 7) ^ (a & mask_of(W, 15)) ^ (b & mask_of(W, 23)) ^ (a & b & mask_of(W, 31));
                    const uint32_t g1 = mask_of(W, 6) ^ (a & mask_of(W, 14)) ^ (b & mask_of(W, 22)) ^ (a & b & mask_of(W, 30));
                    out[q] = g0 ^ (cc & g1);
                  }
                }
                for (uint32_t q = 0; q < words; ++q) row(so)[q] = out[q];
                const uint32_t net = opt.settle ? fp.stream_net[((size_t)at[w] * 32 + l) * 2 + (uint32_t)h] : ~0u;
                if (opt.settle && so >= fp.G) {
                  const uint32_t made = row_net.at({L, so});
                  if (net != (gp.net_signal[made] >= 0 ? made : ~0u)) fail("a write-back of another net");
                  back[made] = out;
                } else if (net != ~0u) {
                  fail("an idle lane writes back");
                }
              }
            }
          }
      }
      for (uint32_t w = 0; w < warps; ++w) {
        if (at[w] != fp.warp_begin[w + 1]) fail("a stream was not finished");
        if (fp.n_levels && level[w] + fp.warp_tail[w] != fp.n_levels - 1) fail("warps pass different barriers");
      }
      unsigned long long hs = 0ull;
      for (uint32_t k = 0; k < n_rec; ++k)
        for (uint32_t w = 0; w < words; ++w) {
          const uint32_t left = lanes - w * 32, vm = left >= 32 ? 0xFFFFFFFFu : (1u << left) - 1u;
          hs += hash_term(c, k, word_base + w, value(rec_net[k])[w] & vm);
        }
      out_hash[c] = hs;
      for (uint32_t s = 0; opt.settle && s < gp.n_signals; ++s)
        if (gp.signal_net[s] > kNetConst1) value(gp.signal_net[s]);
      for (uint32_t k : commit) {
        const GateReg& r = gp.regs[k];
        for (uint32_t w = 0; w < words; ++w) {
          uint32_t v = r.d_net == kNetConst0 ? 0u : r.d_net == kNetConst1 ? 0xFFFFFFFFu : value(r.d_net)[w];
          if (r.has_reset) {
            uint32_t m = r.rst_net == kNetConst0 ? 0u : r.rst_net == kNetConst1 ? 0xFFFFFFFFu
                                                                               : value(r.rst_net)[w];
            if (r.active_low) m = ~m;
            v = r.reset_value ? v | m : v & ~m;
          }
          row((uint32_t)fp.net_slot[r.q_net])[w] = v;
        }
      }
    }
    return 0;
  } catch (const Fail& f) {
    if (err && errcap) snprintf(err, errcap, "%s", f.msg.c_str());
    return 1;
  } catch (const std::exception& e) {
    if (err && errcap) snprintf(err, errcap, "error: %s", e.what());
    return 2;
  }
}
