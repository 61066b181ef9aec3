// Flat gate program lowering (see flatprog.h).
#include "flatprog.h"

#include <algorithm>
#include <array>

namespace rrtl {

namespace {

const uint8_t kVar[3] = {0xF0, 0xCC, 0xAA};

// Table `tt` evaluated on three 8-bit variable masks.
uint8_t apply3(uint8_t tt, uint8_t x, uint8_t y, uint8_t z) {
  uint8_t r = 0;
  for (int p = 0; p < 8; ++p) {
    const int idx = (((x >> p) & 1) << 2) | (((y >> p) & 1) << 1) | ((z >> p) & 1);
    if ((tt >> idx) & 1) r |= (uint8_t)(1u << p);
  }
  return r;
}

bool depends(uint8_t tt, int i) {
  const uint8_t v = kVar[i];
  const int sh = i == 0 ? 4 : i == 1 ? 2 : 1;
  return (uint8_t)((tt & v) >> sh) != (uint8_t)(tt & (uint8_t)~v);
}

// Drop inputs the table does not depend on (and repeated ones) and renumber.
void simplify(FlatCell& c) {
  for (int i = 0; i < c.n; ++i)
    for (int j = i + 1; j < c.n; ++j)
      if (c.in[i] == c.in[j]) {  // merge j into i
        uint8_t m[3] = {kVar[0], kVar[1], kVar[2]};
        m[j] = kVar[i];
        c.lut = apply3(c.lut, m[0], m[1], m[2]);
      }
  uint32_t in[3];
  uint8_t m[3] = {0, 0, 0};
  int k = 0;
  for (int i = 0; i < c.n; ++i)
    if (depends(c.lut, i)) {
      m[i] = kVar[k];
      in[k++] = c.in[i];
    }
  c.lut = apply3(c.lut, m[0], m[1], m[2]);
  for (int i = 0; i < k; ++i) c.in[i] = in[i];
  c.n = (uint8_t)k;
  if (k == 0) c.lut = (c.lut & 1) ? 0xFF : 0x00;
}

// Input `pos` of y replaced by the function of cell x; false when the result
// would read more than three nets.
bool compose(const FlatCell& y, int pos, const FlatCell& x, FlatCell* out) {
  uint32_t u[6];
  int n = 0;
  for (int i = 0; i < y.n; ++i)
    if (i != pos) u[n++] = y.in[i];
  for (int i = 0; i < x.n; ++i) {
    bool seen = false;
    for (int j = 0; j < n; ++j) seen |= u[j] == x.in[i];
    if (!seen) u[n++] = x.in[i];
  }
  if (n > 3) return false;
  auto mask = [&](uint32_t net) -> uint8_t {
    for (int j = 0; j < n; ++j)
      if (u[j] == net) return kVar[j];
    return 0;
  };
  uint8_t mx[3] = {0, 0, 0}, my[3] = {0, 0, 0};
  for (int i = 0; i < x.n; ++i) mx[i] = mask(x.in[i]);
  const uint8_t tx = apply3(x.lut, mx[0], mx[1], mx[2]);
  for (int i = 0; i < y.n; ++i) my[i] = i == pos ? tx : mask(y.in[i]);
  *out = y;
  out->lut = apply3(y.lut, my[0], my[1], my[2]);
  out->n = (uint8_t)n;
  for (int i = 0; i < n; ++i) out->in[i] = u[i];
  simplify(*out);
  return true;
}

// Algebraic normal form of a table over (a, b) at fixed c: bits k0, ka, kb, kab.
std::array<uint32_t, 4> anf2(uint8_t lut, int c) {
  auto f = [&](int a, int b) { return (uint32_t)((lut >> ((a << 2) | (b << 1) | c)) & 1); };
  const uint32_t k0 = f(0, 0), ka = f(1, 0) ^ k0, kb = f(0, 1) ^ k0;
  return {k0, ka, kb, f(1, 1) ^ ka ^ kb ^ k0};
}

uint32_t two_meta(uint8_t lut) {
  const auto k = anf2(lut, 0);
  return (k[0] << 23) | (k[1] << 31) | (k[2] << 22) | (k[3] << 30);
}

uint32_t three_coef(uint8_t lut) {
  const auto g0 = anf2(lut, 0), h = anf2(lut, 1);
  uint32_t w = 0;
  for (int j = 0; j < 4; ++j) w |= (g0[j] << (8 * j + 7)) | ((g0[j] ^ h[j]) << (8 * j + 6));
  return w;
}

// The packed, register-folded, levelized cells of a gate program.
struct Logic {
  const GateProgram& gp;
  std::vector<FlatCell> cells;
  std::vector<uint8_t> alive;
  std::vector<int32_t> cell_of;  // net -> cell, -1
  std::vector<uint8_t> root;     // net must be in its own row at the end of a cycle
  std::vector<uint32_t> commit;  // registers left on the commit list
  uint32_t n_levels = 0;
  bool observe = false, settle = false;

  explicit Logic(const GateProgram& g) : gp(g) {}

  // A net whose row nothing but its readers sees.
  bool hidden(uint32_t net) const { return !(observe && gp.net_signal[net] >= 0); }

  void collect() {
    for (const GateCell& c : gp.cells) {
      if (c.pad) continue;
      FlatCell f;
      f.lut = c.lut;
      f.n = 3;
      f.out = c.out;
      uint8_t m[3];
      for (int i = 0; i < 3; ++i) {
        f.in[i] = c.in[i];
        m[i] = c.in[i] == kNetConst0 ? 0x00 : c.in[i] == kNetConst1 ? 0xFF : kVar[i];
      }
      f.lut = apply3(f.lut, m[0], m[1], m[2]);
      simplify(f);
      cells.push_back(f);  // gp.cells are in level order: producers come first
    }
    alive.assign(cells.size(), 1);
    cell_of.assign(gp.n_nets, -1);
    for (size_t i = 0; i < cells.size(); ++i) cell_of[cells[i].out] = (int32_t)i;
    root.assign(gp.n_nets, 0);
    for (uint32_t n = 0; n < gp.n_nets; ++n)
      if (cell_of[n] >= 0 && gp.net_end_live[n]) root[n] = 1;
  }

  std::vector<uint32_t> fanout() const {
    std::vector<uint32_t> f(gp.n_nets, 0);
    for (size_t i = 0; i < cells.size(); ++i)
      if (alive[i])
        for (int k = 0; k < cells[i].n; ++k) ++f[cells[i].in[k]];
    return f;
  }

  void drop_dead() {
    std::vector<uint32_t> f = fanout();
    for (size_t i = cells.size(); i-- > 0;) {
      if (!alive[i] || root[cells[i].out] || f[cells[i].out] || (settle && gp.net_signal[cells[i].out] >= 0)) continue;
      alive[i] = 0;
      for (int k = 0; k < cells[i].n; ++k) --f[cells[i].in[k]];
    }
  }

  void pack() {
    // inverters, buffers and constants into their readers
    for (size_t i = 0; i < cells.size(); ++i) {
      FlatCell& y = cells[i];
      for (int k = 0; k < y.n;) {
        const int32_t x = cell_of[y.in[k]];
        FlatCell z;
        if (x >= 0 && cells[x].n <= 1 && hidden(cells[x].out) && compose(y, k, cells[x], &z)) {
          y = z;
          k = 0;
        } else {
          ++k;
        }
      }
    }
    drop_dead();
    // single-reader nets into their reader, the smallest support first
    std::vector<uint32_t> f = fanout();
    for (size_t i = 0; i < cells.size(); ++i) {
      if (!alive[i]) continue;
      FlatCell& y = cells[i];
      for (;;) {
        int best = -1;
        FlatCell bz;
        for (int k = 0; k < y.n; ++k) {
          const int32_t x = cell_of[y.in[k]];
          if (x < 0 || root[cells[x].out] || f[cells[x].out] != 1 || !hidden(cells[x].out)) continue;
          FlatCell z;
          if (compose(y, k, cells[x], &z) && (best < 0 || z.n < bz.n)) {
            best = k;
            bz = z;
          }
        }
        if (best < 0) break;
        const int32_t x = cell_of[y.in[best]];
        // readers of y's inputs and of x's inputs become readers through y alone
        for (int k = 0; k < y.n; ++k) --f[y.in[k]];
        for (int k = 0; k < cells[x].n; ++k) --f[cells[x].in[k]];
        alive[x] = 0;
        y = bz;
        for (int k = 0; k < y.n; ++k) ++f[y.in[k]];
      }
    }
    drop_dead();
  }

  int32_t asap(const FlatCell& c) const {
    int32_t lv = 0;
    for (int k = 0; k < c.n; ++k) {
      const int32_t p = cell_of[c.in[k]];
      if (p >= 0) lv = std::max(lv, cells[p].level + 1);
    }
    return lv;
  }

  void levelize() {
    int32_t top = -1;
    for (size_t i = 0; i < cells.size(); ++i)
      if (alive[i]) {
        cells[i].level = asap(cells[i]);
        top = std::max(top, cells[i].level);
      }
    n_levels = (uint32_t)(top + 1);
  }

  // Registers written in place. A register's next-value cell may write the
  // register's row at a level after every other cell that reads it; the row
  // is then not a record of the D net any more, so a D net that something
  // else observes (an output, another register, another cell) gets a cell of
  // its own for the register. Levels are relaxed to a fixpoint; a register
  // that would need a level past the last one is left on the commit list.
  void fold_registers(bool enable) {
    const size_t nr = gp.regs.size();
    std::vector<uint32_t> f = fanout();
    std::vector<uint32_t> d_uses(gp.n_nets, 0);
    std::vector<uint8_t> is_rst(gp.n_nets, 0);
    for (const GateReg& r : gp.regs) {
      ++d_uses[r.d_net];
      if (r.has_reset) is_rst[r.rst_net] = 1;
    }
    struct Fold {
      uint32_t reg;
      int32_t cell;       // the D cell, rewritten in place, or -1: a new cell
      FlatCell next;      // the register's next value
    };
    std::vector<Fold> folds;
    for (uint32_t r = 0; r < nr; ++r) {
      const GateReg& g = gp.regs[r];
      const int32_t dc = cell_of[g.d_net];
      const bool is_out = gp.net_is_output[g.d_net];
      FlatCell next;
      bool own = false;
      if (dc >= 0 && alive[dc] && d_uses[g.d_net] == 1 && f[g.d_net] == 0 && !is_rst[g.d_net] && !is_out &&
          hidden(g.d_net)) {
        next = cells[dc];
        own = add_reset(g, &next);
      }
      if (!own) {
        next = FlatCell{};
        next.n = 1;
        next.in[0] = g.d_net;
        next.lut = kVar[0];
        if (g.d_net == kNetConst0 || g.d_net == kNetConst1) {
          next.n = 0;
          next.lut = g.d_net == kNetConst1 ? 0xFF : 0x00;
        }
        add_reset(g, &next);
      }
      next.out = g.q_net;
      next.reg = (int32_t)r;
      folds.push_back(Fold{r, own ? dc : -1, next});
    }
    if (!enable || n_levels == 0) {
      for (uint32_t r = 0; r < nr; ++r) commit.push_back(r);
      return;
    }
    // last level at which a cell other than the register's own reads each net
    std::vector<uint8_t> out_of(folds.size(), 0);  // unfolded
    std::vector<int32_t> lev(folds.size(), 0);
    std::vector<uint8_t> owned(cells.size(), 0);
    for (const Fold& x : folds)
      if (x.cell >= 0) owned[x.cell] = 1;
    std::vector<int32_t> fixed_last(gp.n_nets, -1);
    for (size_t i = 0; i < cells.size(); ++i)
      if (alive[i] && !owned[i])
        for (int k = 0; k < cells[i].n; ++k)
          fixed_last[cells[i].in[k]] = std::max(fixed_last[cells[i].in[k]], cells[i].level);
    std::vector<std::vector<uint32_t>> readers(gp.n_nets);  // folds that read a net
    for (uint32_t i = 0; i < folds.size(); ++i) {
      lev[i] = asap(folds[i].next);
      for (int k = 0; k < folds[i].next.n; ++k) readers[folds[i].next.in[k]].push_back(i);
    }
    for (bool changed = true; changed;) {
      changed = false;
      for (uint32_t i = 0; i < folds.size(); ++i) {
        if (out_of[i]) continue;
        const uint32_t q = folds[i].next.out;
        int32_t need = std::max(lev[i], fixed_last[q] + 1);
        for (uint32_t j : readers[q]) {
          if (j == i) continue;  // its own old value is read in the same step
          need = std::max(need, (out_of[j] ? unfolded_level(folds[j].cell) : lev[j]) + 1);
        }
        if (need >= (int32_t)n_levels) {
          out_of[i] = 1;
          changed = true;
        } else if (need != lev[i]) {
          lev[i] = need;
          changed = true;
        }
      }
    }
    for (uint32_t i = 0; i < folds.size(); ++i) {
      if (out_of[i]) {
        commit.push_back(folds[i].reg);
        continue;
      }
      FlatCell c = folds[i].next;
      c.level = lev[i];
      if (folds[i].cell >= 0) {
        cell_of[cells[folds[i].cell].out] = -1;
        root[cells[folds[i].cell].out] = 0;
        cells[folds[i].cell] = c;
      } else {
        cells.push_back(c);
        alive.push_back(1);
      }
    }
  }
  // Level at which a register on the commit list reads its D cell's inputs
  // (without a cell of its own it reads its D net after the last level).
  int32_t unfolded_level(int32_t cell) const { return cell >= 0 ? cells[cell].level : (int32_t)n_levels; }

  // The register's next value with its synchronous reset; false (cell
  // unchanged) when that reads more than three nets.
  static bool add_reset(const GateReg& g, FlatCell* c) {
    if (!g.has_reset) return true;
    if (g.rst_net == kNetConst0 || g.rst_net == kNetConst1) {
      const bool active = (g.rst_net == kNetConst1) != g.active_low;
      if (active) {
        c->n = 0;
        c->lut = g.reset_value ? 0xFF : 0x00;
      }
      return true;
    }
    int pos = -1;
    for (int k = 0; k < c->n; ++k)
      if (c->in[k] == g.rst_net) pos = k;
    if (pos < 0) {
      if (c->n == 3) return false;
      pos = c->n;
      c->in[c->n++] = g.rst_net;
    }
    const uint8_t act = g.active_low ? (uint8_t)~kVar[pos] : kVar[pos];
    c->lut = (uint8_t)(g.reset_value ? (c->lut | act) : (c->lut & ~act));
    simplify(*c);
    return true;
  }
};

struct Group {
  std::vector<uint32_t> cells;
};

// Cells of one level and kind into groups of G whose operand rows (and rows
// written at a fixed residue) fall on distinct residues where possible. A
// group is a matching of the bipartite multigraph with a node per residue on
// either side and a cell per edge (operand a's residue, operand b's): edges
// are oriented to even out the node degrees (a cell may read its inputs in
// any order), then matchings are peeled off, the busiest residues first, as
// an edge colouring with as few colours as the largest degree needs.
struct Grouper {
  uint32_t G;
  std::vector<FlatCell>& cells;
  const std::vector<int32_t>& slot;

  uint32_t res(const FlatCell& c, int k) const { return (uint32_t)slot[c.in[k]] % G; }
  int fixed_out(const FlatCell& c) const { return c.reg >= 0 ? (int)((uint32_t)slot[c.out] % G) : -1; }

  static void swap_inputs(FlatCell& c, int i, int j) {
    uint8_t m[3] = {kVar[0], kVar[1], kVar[2]};
    std::swap(m[i], m[j]);
    c.lut = apply3(c.lut, m[0], m[1], m[2]);
    std::swap(c.in[i], c.in[j]);
  }

  // Distinct rows per residue at each position: the wavefronts of the group.
  uint32_t cost(const Group& g, int n) const {
    uint32_t total = 0;
    uint32_t rows[32];
    for (int p = 0; p < n; ++p) {
      uint8_t per[32] = {0};
      uint32_t mx = 0, nr = 0;
      for (uint32_t ci : g.cells) {
        const FlatCell& c = cells[ci];
        if (p >= c.n) continue;
        const uint32_t s = (uint32_t)slot[c.in[p]];
        bool seen = false;
        for (uint32_t q = 0; q < nr && !seen; ++q) seen = rows[q] == s;
        if (seen) continue;
        rows[nr++] = s;
        mx = std::max<uint32_t>(mx, ++per[s % G]);
      }
      total += std::max(mx, 1u);
    }
    uint8_t per[32] = {0};
    uint32_t mx = 1;
    for (uint32_t ci : g.cells) {
      const int o = fixed_out(cells[ci]);
      if (o >= 0) mx = std::max<uint32_t>(mx, ++per[o]);
    }
    return total + mx;
  }

  void orient(const std::vector<uint32_t>& list, int n) {
    std::vector<std::vector<int32_t>> deg(n, std::vector<int32_t>(G, 0));
    for (uint32_t ci : list)
      for (int p = 0; p < cells[ci].n; ++p) ++deg[p][res(cells[ci], p)];
    for (int pass = 0; pass < 4; ++pass) {
      bool any = false;
      for (uint32_t ci : list) {
        FlatCell& c = cells[ci];
        for (int i = 0; i < c.n; ++i)
          for (int j = i + 1; j < c.n; ++j) {
            const uint32_t ri = res(c, i), rj = res(c, j);
            if (ri == rj) continue;
            // moving ri from position i to j and rj from j to i
            const int32_t d = (deg[i][rj] - deg[i][ri]) + (deg[j][ri] - deg[j][rj]) + 2;
            if (d < 0) {
              --deg[i][ri];
              --deg[j][rj];
              ++deg[i][rj];
              ++deg[j][ri];
              swap_inputs(c, i, j);
              any = true;
            }
          }
      }
      if (!any) break;
    }
  }

  std::vector<Group> build(std::vector<uint32_t> list, int n) {
    std::vector<Group> out;
    if (list.empty()) return out;
    orient(list, n);
    // bucket[ra * G + rb]; a cell of fewer than two inputs reads its one row at both positions
    std::vector<std::vector<uint32_t>> bucket((size_t)G * G);
    std::vector<uint32_t> dl(G, 0), dr(G, 0);
    size_t left = list.size();
    std::vector<uint32_t> none;  // constants: no operand
    for (uint32_t ci : list) {
      const FlatCell& c = cells[ci];
      if (c.n == 0) {
        none.push_back(ci);
        continue;
      }
      const uint32_t a = res(c, 0), b = res(c, c.n >= 2 ? 1 : 0);
      bucket[(size_t)a * G + b].push_back(ci);
      ++dl[a];
      ++dr[b];
    }
    left -= none.size();
    std::vector<int32_t> ml(G), mr(G);
    std::vector<uint8_t> seen(G);
    std::vector<uint32_t> lo(G), ro(G);
    while (left) {
      for (uint32_t r = 0; r < G; ++r) lo[r] = ro[r] = r;
      std::stable_sort(lo.begin(), lo.end(), [&](uint32_t x, uint32_t y) { return dl[x] > dl[y]; });
      std::stable_sort(ro.begin(), ro.end(), [&](uint32_t x, uint32_t y) { return dr[x] > dr[y]; });
      std::fill(ml.begin(), ml.end(), -1);
      std::fill(mr.begin(), mr.end(), -1);
      auto augment = [&](auto&& self, uint32_t a) -> bool {
        for (uint32_t b : ro) {
          if (seen[b] || bucket[(size_t)a * G + b].empty()) continue;
          seen[b] = 1;
          if (mr[b] < 0 || self(self, (uint32_t)mr[b])) {
            mr[b] = (int32_t)a;
            ml[a] = (int32_t)b;
            return true;
          }
        }
        return false;
      };
      for (uint32_t a : lo) {
        if (!dl[a]) break;
        std::fill(seen.begin(), seen.end(), 0);
        augment(augment, a);
      }
      Group g;
      std::vector<uint8_t> used_c(G, 0), used_o(G, 0);
      for (uint32_t a = 0; a < G; ++a) {
        if (ml[a] < 0) continue;
        std::vector<uint32_t>& bk = bucket[(size_t)a * G + (uint32_t)ml[a]];
        // of the bucket's cells, one whose third operand and fixed row are free in the group
        size_t pick = bk.size() - 1;
        uint32_t pc = ~0u;
        for (size_t k = bk.size(); k-- > 0 && bk.size() - k <= 48;) {
          const FlatCell& c = cells[bk[k]];
          const int o = fixed_out(c);
          const uint32_t x = (c.n == 3 && used_c[res(c, 2)] ? 2u : 0u) + (o >= 0 && used_o[o] ? 1u : 0u);
          if (x < pc) {
            pc = x;
            pick = k;
            if (!x) break;
          }
        }
        const uint32_t ci = bk[pick];
        bk.erase(bk.begin() + (long)pick);
        if (cells[ci].n == 3) used_c[res(cells[ci], 2)] = 1;
        const int o = fixed_out(cells[ci]);
        if (o >= 0) used_o[o] = 1;
        --dl[a];
        --dr[(uint32_t)ml[a]];
        --left;
        g.cells.push_back(ci);
      }
      out.push_back(std::move(g));
    }
    // constants wherever a lane is idle
    for (size_t k = 0, gi = 0; k < none.size(); ++k) {
      while (gi < out.size() && out[gi].cells.size() >= G) ++gi;
      if (gi == out.size()) out.push_back(Group{});
      out[gi].cells.push_back(none[k]);
    }
    merge_small(out, n);
    return out;
  }

  // Three-input cells: a group takes cells one at a time, each in an input
  // order whose three residues (and fixed row) are still free in the group,
  // the cells with the busiest residues first. Candidates are the first
  // kLook cells left; a group that finds none stays short.
  std::vector<Group> build_three(const std::vector<uint32_t>& list) {
    static const int orders[6][3] = {{0, 1, 2}, {0, 2, 1}, {1, 0, 2}, {1, 2, 0}, {2, 0, 1}, {2, 1, 0}};
    const size_t kLook = 256;
    std::vector<Group> out;
    std::vector<uint32_t> pool(list);
    std::vector<uint32_t> deg(G, 0);  // operand rows left per residue
    for (uint32_t ci : pool)
      for (int p = 0; p < 3; ++p) ++deg[res(cells[ci], p)];
    while (!pool.empty()) {
      Group g;
      uint32_t used[4] = {0, 0, 0, 0};  // residues taken at each position, rows written
      while (g.cells.size() < G) {
        size_t best = pool.size();
        int best_order = 0;
        uint32_t best_score = 0;
        for (size_t k = 0; k < pool.size() && k < kLook; ++k) {
          const FlatCell& c = cells[pool[k]];
          const int o = fixed_out(c);
          if (o >= 0 && (used[3] >> o & 1u)) continue;
          const uint32_t r[3] = {res(c, 0), res(c, 1), res(c, 2)};
          const uint32_t score = 1 + deg[r[0]] + deg[r[1]] + deg[r[2]];
          if (score <= best_score) continue;
          for (int q = 0; q < 6; ++q)
            if (!((used[0] >> r[orders[q][0]] | used[1] >> r[orders[q][1]] | used[2] >> r[orders[q][2]]) & 1u)) {
              best = k;
              best_order = q;
              best_score = score;
              break;
            }
        }
        if (best == pool.size()) break;
        FlatCell& c = cells[pool[best]];
        const FlatCell old = c;
        uint8_t m[3] = {0, 0, 0};
        for (int p = 0; p < 3; ++p) {
          c.in[p] = old.in[orders[best_order][p]];
          m[orders[best_order][p]] = kVar[p];
          const uint32_t r = res(c, p);
          used[p] |= 1u << r;
          --deg[r];
        }
        c.lut = apply3(old.lut, m[0], m[1], m[2]);
        const int o = fixed_out(c);
        if (o >= 0) used[3] |= 1u << o;
        g.cells.push_back(pool[best]);
        pool.erase(pool.begin() + (long)best);
      }
      out.push_back(std::move(g));
    }
    merge_small(out, 3);
    return out;
  }

  // The last matchings are small: two groups become one where that costs
  // fewer wavefronts than the two apart.
  void merge_small(std::vector<Group>& gs, int n) const {
    std::stable_sort(gs.begin(), gs.end(), [](const Group& a, const Group& b) { return a.cells.size() > b.cells.size(); });
    for (size_t i = gs.size(); i-- > 1;) {
      const uint32_t ci = cost(gs[i], n);
      size_t best = gs.size();
      int32_t gain = 0;
      for (size_t j = 0; j < i; ++j) {
        if (gs[j].cells.size() + gs[i].cells.size() > G) continue;
        Group m = gs[j];
        m.cells.insert(m.cells.end(), gs[i].cells.begin(), gs[i].cells.end());
        const int32_t d = (int32_t)(cost(gs[j], n) + ci) - (int32_t)cost(m, n);
        if (d > gain) {
          gain = d;
          best = j;
        }
      }
      if (best < gs.size()) {
        gs[best].cells.insert(gs[best].cells.end(), gs[i].cells.begin(), gs[i].cells.end());
        gs.erase(gs.begin() + (long)i);
      }
    }
  }
};

}  // namespace

FlatProgram build_flat_program(const GateProgram& gp, uint32_t V, const FlatOptions& opt) {
  if (V != 4 && V != 2 && V != 1) throw RrtlError("E_GATE_SCOPE", "row vectors are 4, 2 or 1 words");
  FlatProgram fp;
  fp.V = V;
  const uint32_t G = fp.G = 32 / V;
  Logic lg(gp);
  lg.observe = opt.observe || opt.settle;
  lg.settle = opt.settle;
  lg.collect();
  if (opt.pack) lg.pack();
  else lg.drop_dead();
  lg.levelize();
  lg.fold_registers(opt.fold_regs && !opt.settle);
  std::vector<FlatCell>& cells = lg.cells;
  const uint32_t NL = fp.n_levels = lg.n_levels;
  fp.commit = lg.commit;

  // ---- liveness in levels: a net is read at levels up to last[n]; NL = the end of the cycle
  const int32_t kEnd = (int32_t)NL;
  std::vector<int32_t> last(gp.n_nets, -1), made(gp.n_nets, -1), q_write(gp.n_nets, -1);
  std::vector<std::vector<uint32_t>> at(NL);
  for (uint32_t i = 0; i < cells.size(); ++i) {
    if (!lg.alive[i]) continue;
    const FlatCell& c = cells[i];
    at[c.level].push_back(i);
    for (int k = 0; k < c.n; ++k) last[c.in[k]] = std::max(last[c.in[k]], c.level);
    if (c.reg >= 0) q_write[c.out] = c.level;
    else made[c.out] = c.level;
  }
  for (uint32_t r : lg.commit) {
    q_write[gp.regs[r].q_net] = kEnd;
    if (opt.settle) continue;  // no row is read after the levels
    last[gp.regs[r].d_net] = kEnd;
    if (gp.regs[r].has_reset) last[gp.regs[r].rst_net] = kEnd;
  }
  if (opt.settle) fp.commit.clear();
  for (uint32_t n = 0; n < gp.n_nets && !opt.settle; ++n)
    if (made[n] >= 0 && lg.root[n] && (gp.net_is_output[n] || last[n] >= kEnd)) last[n] = kEnd;

  // ---- residue balance: rows read per (level, residue)
  std::vector<uint32_t> reads((size_t)NL * G, 0);
  std::vector<uint32_t> use_off(gp.n_nets + 1, 0), use_level;
  for (uint32_t L = 0; L < NL; ++L)
    for (uint32_t i : at[L])
      for (int k = 0; k < cells[i].n; ++k) ++use_off[cells[i].in[k] + 1];
  for (uint32_t n = 0; n < gp.n_nets; ++n) use_off[n + 1] += use_off[n];
  use_level.resize(use_off[gp.n_nets]);
  {
    std::vector<uint32_t> fill(use_off.begin(), use_off.end() - 1);
    for (uint32_t L = 0; L < NL; ++L)
      for (uint32_t i : at[L])
        for (int k = 0; k < cells[i].n; ++k) use_level[fill[cells[i].in[k]]++] = L * 2 + (cells[i].n == 3);
  }
  reads.assign((size_t)NL * 2 * G, 0);
  auto read_cost = [&](uint32_t n, uint32_t r) {
    uint64_t c = 0;
    for (uint32_t i = use_off[n]; i < use_off[n + 1]; ++i) c += reads[(size_t)use_level[i] * G + r];
    return c;
  };
  auto placed = [&](uint32_t n, uint32_t r) {
    for (uint32_t i = use_off[n]; i < use_off[n + 1]; ++i) ++reads[(size_t)use_level[i] * G + r];
  };

  // ---- slots
  std::vector<int32_t>& slot = fp.net_slot;
  slot.assign(gp.n_nets, -1);
  uint32_t next_slot = G;  // slots 0..G-1: scratch rows
  std::vector<uint32_t> src_next(G), src_count(G, 0);
  for (uint32_t r = 0; r < G; ++r) src_next[r] = G + r;
  std::vector<uint8_t> is_q(gp.n_nets, 0);
  for (const GateReg& r : gp.regs) is_q[r.q_net] = 1;
  struct Free {
    uint32_t slot;
    int32_t until;  // a net may use the slot when it is last read below this level
  };
  std::vector<std::vector<Free>> free_q(G);
  std::vector<std::vector<uint32_t>> free_all(G);
  std::vector<std::vector<uint32_t>> q_free_at(NL + 1);  // register nets whose row is free from this level on
  uint32_t n_src = 0;
  for (uint32_t n = 2; n < gp.n_nets; ++n) {
    if (!gp.net_is_source[n]) continue;
    uint32_t best = 0;
    uint64_t bc = ~0ull;
    for (uint32_t r = 0; r < G; ++r) {
      const uint64_t c = read_cost(n, r) * 1000000u + src_count[r];
      if (c < bc && src_count[r] <= n_src / G + 8) {
        bc = c;
        best = r;
      }
    }
    placed(n, best);
    ++src_count[best];
    ++n_src;
    slot[n] = (int32_t)src_next[best];
    src_next[best] += G;
    next_slot = std::max(next_slot, (uint32_t)slot[n] + 1);
    fp.source_nets.push_back(n);
  }
  for (uint32_t r = 0; r < G; ++r)
    for (uint32_t s = src_next[r]; s < next_slot; s += G) free_all[r].push_back(s);
  for (uint32_t n = 2; n < gp.n_nets; ++n)
    if (is_q[n] && q_write[n] > 0 && last[n] + 1 < q_write[n]) q_free_at[last[n] + 1].push_back(n);
  std::vector<std::vector<uint32_t>> dying(NL + 1);
  for (uint32_t n = 0; n < gp.n_nets; ++n)
    if (made[n] >= 0) {
      last[n] = std::max(last[n], made[n]);
      if (last[n] < kEnd) dying[last[n]].push_back(n);
    }
  std::vector<int32_t> slot_until;  // per slot: kEnd + 1, or the level its register is written at
  auto until_of = [&](uint32_t s) { return s < slot_until.size() && slot_until[s] ? slot_until[s] : kEnd + 1; };
  slot_until.assign(next_slot, 0);
  for (uint32_t n = 2; n < gp.n_nets; ++n)
    if (is_q[n]) slot_until[slot[n]] = std::max(q_write[n], 0) ? q_write[n] : 0;
  auto fits_q = [&](uint32_t r, int32_t lu) -> int {
    const std::vector<Free>& v = free_q[r];
    int best = -1;  // the slot whose register is written soonest after the net's last read
    for (size_t k = 0; k < v.size(); ++k)
      if (v[k].until > lu && (best < 0 || v[k].until < v[(size_t)best].until)) best = (int)k;
    return best;
  };
  auto take = [&](uint32_t n, uint32_t r) -> uint32_t {
    const int k = fits_q(r, last[n]);
    if (k >= 0) {
      const uint32_t s = free_q[r][k].slot;
      free_q[r].erase(free_q[r].begin() + k);
      return s;
    }
    if (!free_all[r].empty()) {
      const uint32_t s = free_all[r].back();
      free_all[r].pop_back();
      return s;
    }
    while (next_slot % G != r) {
      free_all[next_slot % G].push_back(next_slot);
      ++next_slot;
    }
    return next_slot++;
  };
  auto release = [&](uint32_t s) {
    const int32_t u = until_of(s);
    if (u <= kEnd) free_q[s % G].push_back(Free{s, u});
    else free_all[s % G].push_back(s);
  };

  // An entry without cells: every lane reads a scratch row and writes one of its own residue.
  auto push_idle = [&](std::vector<FlatLane>& st, uint32_t meta) {
    for (uint32_t l = 0; l < 32; ++l) st.push_back(FlatLane{0u, (l % G) | meta, 0u, l % G});
  };

  const bool tight = opt.max_slots != 0;

  // ---- levels: group and place
  fp.net_level.assign(gp.n_nets, -1);
  fp.net_warp.assign(gp.n_nets, 0);
  Grouper grouper{G, cells, slot};
  std::vector<uint8_t> used_res(G);
  struct Entry {
    std::vector<FlatLane> lanes;
    std::vector<uint32_t> outs;  // nets written
    std::vector<uint32_t> nets;  // settle: signal net per lane and cell
    double cost = 0;
  };
  std::vector<std::vector<Entry>> entries(NL);
  for (uint32_t L = 0; L < NL; ++L) {
    for (uint32_t n : q_free_at[L]) release((uint32_t)slot[n]);
    if (L > 0)
      for (uint32_t n : dying[L - 1]) release((uint32_t)slot[n]);
    std::vector<uint32_t> two, three;
    for (uint32_t i : at[L]) (cells[i].n == 3 ? three : two).push_back(i);
    std::vector<Group> g2 = grouper.build(two, 2), g3 = grouper.build_three(three);
    fp.n_two += (uint32_t)two.size();
    fp.n_three += (uint32_t)three.size();
    // rows written: distinct residues within a group, cheapest for the readers
    for (auto* gs : {&g2, &g3})
      for (Group& g : *gs) {
        std::fill(used_res.begin(), used_res.end(), 0);
        std::vector<uint32_t> open;
        for (uint32_t ci : g.cells) {
          if (cells[ci].reg >= 0) used_res[(uint32_t)slot[cells[ci].out] % G] = 1;
          else open.push_back(ci);
        }
        // nets with the most readers choose first
        std::stable_sort(open.begin(), open.end(), [&](uint32_t x, uint32_t y) {
          const uint32_t a = cells[x].out, b = cells[y].out;
          return use_off[a + 1] - use_off[a] > use_off[b + 1] - use_off[b];
        });
        for (uint32_t ci : open) {
          const uint32_t n = cells[ci].out;
          uint32_t best = G;
          uint64_t bc = ~0ull;
          for (uint32_t r = 0; r < G; ++r) {
            if (used_res[r]) continue;
            // a row a register leaves free is taken before one any net could use
            const bool q = fits_q(r, last[n]) >= 0, has = q || !free_all[r].empty();
            const uint64_t c = read_cost(n, r) * 2u + (has ? 0u : 1u) + (tight && !q ? 1u << 16 : 0u);
            if (c < bc) {
              bc = c;
              best = r;
            }
          }
          if (best == G) best = (uint32_t)(next_slot % G);  // fixed rows filled the residues: a conflict
          if (opt.max_slots && next_slot + G > opt.max_slots && free_all[best].empty() && fits_q(best, last[n]) < 0)
            for (uint32_t r = 0; r < G; ++r)  // a write conflict rather than a longer slot array
              if (!free_all[r].empty() || fits_q(r, last[n]) >= 0) {
                best = r;
                break;
              }
          used_res[best] = 1;
          placed(n, best);
          slot[n] = (int32_t)take(n, best);
        }
        fp.wavefronts += grouper.cost(g, gs == &g2 ? 2 : 3);
        fp.floor_wavefronts += gs == &g2 ? 3 : 4;
      }
    // entries of this level: V groups fill a warp's lanes
    std::vector<Entry>& es = entries[L];
    auto lane_fill = [&](const std::vector<Group>& gs, size_t g0, auto&& put) {
      for (uint32_t h = 0; h < V; ++h) {
        const size_t gi = g0 + h;
        uint8_t used[32] = {0};
        uint32_t pad_a = 0, pad_b = 0, pad_c = 0;
        size_t k = 0;
        if (gi < gs.size()) {
          const Group& g = gs[gi];
          for (; k < g.cells.size(); ++k) {
            const FlatCell& c = cells[g.cells[k]];
            const uint32_t a = c.n > 0 ? (uint32_t)slot[c.in[0]] : 0, b = c.n > 1 ? (uint32_t)slot[c.in[1]] : a;
            const uint32_t cc = c.n > 2 ? (uint32_t)slot[c.in[2]] : a, o = (uint32_t)slot[c.out];
            used[o % G] = 1;
            if (c.n > 0 || k == 0) pad_a = a, pad_b = b, pad_c = cc;
            put(h * G + (uint32_t)k, a, b, cc, o, c.lut);
          }
        }
        // idle lanes read a row the group reads anyway and write a scratch row of a free residue
        for (uint32_t r = 0; k < G; ++k) {
          while (r < G && used[r]) ++r;
          const uint32_t o = r < G ? r : 0;
          if (r < G) used[r] = 1;
          put(h * G + (uint32_t)k, pad_a, pad_b, pad_c, o, 0);
        }
      }
    };
    auto outs_of = [&](Entry& e, const std::vector<Group>& gs, size_t g0, size_t n) {
      if (opt.settle) e.nets.assign(64, 0xFFFFFFFFu);
      for (size_t g = g0; g < std::min(gs.size(), g0 + n); ++g)
        for (size_t k = 0; k < gs[g].cells.size(); ++k) {
          const uint32_t net = cells[gs[g].cells[k]].out;
          e.outs.push_back(net);
          const size_t at_lane = g - g0;  // groups fill the lanes of the first cell, then those of the second
          if (opt.settle && gp.net_signal[net] >= 0) e.nets[2 * (at_lane % V * G + k) + at_lane / V] = net;
        }
    };
    for (size_t g = 0; g < g2.size(); g += 2 * V) {
      Entry e;
      e.lanes.resize(32);
      outs_of(e, g2, g, 2 * V);
      lane_fill(g2, g, [&](uint32_t l, uint32_t a, uint32_t b, uint32_t, uint32_t o, uint8_t lut) {
        e.lanes[l].x = a | (b << 16);
        e.lanes[l].y = o | two_meta(lut);
      });
      lane_fill(g2, g + V, [&](uint32_t l, uint32_t a, uint32_t b, uint32_t, uint32_t o, uint8_t lut) {
        e.lanes[l].z = a | (b << 16);
        e.lanes[l].w = o | two_meta(lut);
      });
      e.cost = g + V < g2.size() ? 7.0 : 4.0;  // row accesses and the entry itself
      es.push_back(std::move(e));
    }
    for (size_t g = 0; g < g3.size(); g += V) {
      Entry e;
      e.lanes.resize(32);
      outs_of(e, g3, g, V);
      lane_fill(g3, g, [&](uint32_t l, uint32_t a, uint32_t b, uint32_t c, uint32_t o, uint8_t lut) {
        e.lanes[l].x = a | (b << 16);
        e.lanes[l].y = o | kFlatDevThree;
        e.lanes[l].z = c;
        e.lanes[l].w = three_coef(lut);
      });
      e.cost = 5.0;
      es.push_back(std::move(e));
    }
    fp.n_entries += (uint32_t)es.size();
  }
  // ---- schedule: as many warps as a level has entries on average. A warp
  // without an entry in a level still spends an idle one on its barrier: 10,000
  // gates (4.7 entries a level), clocks per tile-cycle of one-word and of
  // 4-word tiles: 16 warps 17.7k and 27.0k, 8 14.5k and 20.9k, 6 12.5k and
  // 17.2k, 5 12.4k and 17.4k.
  const uint32_t warps = fp.warps = std::max(1u, std::min(opt.max_warps, NL ? (fp.n_entries + NL - 1) / NL : 1u));
  std::vector<std::vector<FlatLane>> streams(warps);
  std::vector<std::vector<uint32_t>> stream_nets(warps);
  std::vector<uint32_t> last_level(warps, 0);
  for (uint32_t L = 0; L < NL; ++L) {
    std::vector<Entry>& es = entries[L];
    // longest first onto the least loaded warp; warps rotate so that no warp is always the longest
    std::stable_sort(es.begin(), es.end(), [](const Entry& a, const Entry& b) { return a.cost > b.cost; });
    std::vector<double> load(warps, 0.0);
    double sched[4] = {0, 0, 0, 0};  // per warp scheduler (warp mod 4)
    for (Entry& e : es) {
      uint32_t w = 0;
      for (uint32_t k = 0; k < warps; ++k) {
        const uint32_t c = (k + L) % warps;
        if (k == 0 || load[c] < load[w] || (load[c] == load[w] && sched[c % 4] < sched[w % 4])) w = c;
      }
      load[w] += e.cost;
      sched[w % 4] += e.cost;
      for (uint32_t n : e.outs) {
        fp.net_warp[n] = (uint8_t)w;
        fp.net_level[n] = (int32_t)L;
      }
      uint32_t syncs = L - last_level[w];
      last_level[w] = L;
      for (; syncs > 1; --syncs) push_idle(streams[w], kFlatDevSync);  // levels in which the warp has no entry
      for (FlatLane& l : e.lanes) {
        if (syncs) l.y |= kFlatDevSync;
        streams[w].push_back(l);
      }
      if (opt.settle) {
        stream_nets[w].resize((streams[w].size() - 32) * 2, 0xFFFFFFFFu);
        stream_nets[w].insert(stream_nets[w].end(), e.nets.begin(), e.nets.end());
      }
    }
  }
  if (next_slot > kMaxSlots) next_slot = kMaxSlots + 1;
  fp.n_slots = next_slot;
  fp.warp_begin.assign(warps + 1, 0);
  fp.warp_tail.assign(warps, 0);
  for (uint32_t w = 0; w < warps; ++w) {
    while (streams[w].size() % (32 * kFlatPrefetch)) push_idle(streams[w], 0u);
    fp.warp_tail[w] = NL ? NL - 1 - last_level[w] : 0;
    fp.warp_begin[w + 1] = fp.warp_begin[w] + (uint32_t)(streams[w].size() / 32);
    fp.stream.insert(fp.stream.end(), streams[w].begin(), streams[w].end());
    if (opt.settle) {
      stream_nets[w].resize(streams[w].size() * 2, 0xFFFFFFFFu);
      fp.stream_net.insert(fp.stream_net.end(), stream_nets[w].begin(), stream_nets[w].end());
    }
  }
  fp.recordable.assign(gp.n_nets, 0);
  for (uint32_t n = 2; n < gp.n_nets; ++n) {
    if (made[n] >= 0 && last[n] >= kEnd) fp.recordable[n] = 1;
    if (gp.net_is_source[n] && !is_q[n]) fp.recordable[n] = 1;
  }
  return fp;
}

// A tile-cycle costs a boundary (stimulus, record, two barriers), a part per
// level, one per entry and, in wide tiles, one per vector and its wavefronts.
// Clocks, fitted to one wave of tiles on ten netlists of 3,000 to 200,000 gates
// and 11 to 158 levels; the fit is within 8% of every one- and two-word tile
// and 11% of every wider one (without the boundary: 41%, too low at 11 levels).
// Measured, clocks a tile-cycle at 10,000 gates and 11 / 41 / 155 levels and at
// 50,000 and 200,000 gates and 41 levels: one word 7.4k / 12.1k / 34.8k / 23.4k /
// 58.9k (in the queue, 16 warps: 7.4k / 11.8k / 34.1k / 24.9k / 66.9k), two
// 9.1k / 13.7k / 36.9k / 27.9k / 74.3k (8.9k / 13.7k / 36.7k / 29.3k / 80.9k),
// one 4-word vector 10.9k / 17.5k / 44.5k / 36.6k / 105k, two 16.1k / 25.2k /
// 56.8k / 56.2k, three 21.2k / 32.5k / 77.1k / 76.5k, four as two warp sets of
// two 22.0k / 36.9k / 77.9k / 95.8k.
double flat_tile_cost(const FlatProgram& fp, uint32_t base, const FlatShape& x) {
  const double L = fp.n_levels, E = fp.n_entries;
  if (x.V == 1) return x.narrow ? 3060.0 + 162.0 * L + 15.1 * E : 2880.0 + 147.0 * L + 17.4 * E;
  if (x.V == 2) return x.narrow ? 3800.0 + 157.0 * L + 19.7 * E : 3550.0 + 159.0 * L + 21.2 * E;
  const double vec4 = (double)fp.wavefronts * (base == 4 ? 1.0 : base == 2 ? 1.9 : 3.6);  // wavefronts of 4-word rows
  return 3280.0 + 158.0 * L + 8.3 * E + x.N * x.Q * (935.0 + 49.0 * L + 1.06 * vec4);
}

}  // namespace rrtl
