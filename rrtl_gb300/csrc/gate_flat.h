// Device code of the flat gate kernel: cycles of a flat gate program
// (flatprog.h) over tiles of N vectors of V words.
//
// One CTA per SM: 16 compute warps (24 for tiles of one or two words) walk the
// levels, four service warps prepare
// the next cycle's stimulus and finish the last cycle's record (hash, trace,
// detection) while the levels run, so a cycle boundary is two barriers and
// the row copies. Rows ("slots") are V words; the vectors of a tile lie in
// planes a fixed distance apart, so a cell's row address is computed once,
// the planes are immediate offsets, and a decoded entry serves N row
// operations. With Q = 2 two sets of eight warps walk the program
// independently over N planes each, so one set's barriers and decoding
// overlap the other's row accesses. A compute warp's entries come straight
// from L2 into registers, kFlatPrefetch entries ahead: each is read by one
// lane once per cycle, so staging them in shared memory would only add
// wavefronts to the pipe that bounds the kernel.
//
// Bound: the shared-memory pipe (one 128-byte wavefront a clock) and, close
// behind, the integer pipe (3 LOP3 a two-input cell word, 7 a three-input
// one). 50,000 gates, one tile per SM, clocks per 32-lane word and cycle: 6.0k
// at 16 words (4.1k of them wavefronts), 6.4k at 12, 6.9k at 8, 9.2k at 4,
// 14.0k at 2, 23.7k at 1; the fused kernel compiled for the design took 10.1k at 8.
// 65,536 lanes x 1,000 cycles: 79.6 -> 42.5 ms with the closing settle and
// the flip-flop read-back (47.9 before tiles were split between blocks); 200
// lanes x 100 cycles 2.97 -> 1.29 ms; 200,000 gates, 10,007 lanes x 100 cycles
// 20.4 -> 5.0 ms.
//
// What decided the form, 50,000 gates at 8 words, clocks per tile-cycle: entry
// loads issued one by one into a rotating queue 85.6k (each waits behind the
// others' scoreboard), in a batch per four entries 69.3k; type dispatch and a
// barrier count per entry 70.6k, one flag bit each and a uniform vote 62.8k;
// the function as C expressions 62.8k, as explicit LOP3s 56.4k; skipping the
// accesses of lane groups without a cell 68.6k (the branches cost more than
// the wavefronts); one loop body instead of four unrolled entries 58.5k;
// eight entries ahead instead of four 115k (the code leaves the instruction cache).
#pragma once

#include <stdint.h>

#include "../../include/rrtl_cuda.h"
#include "flat_shape.h"
#include "gate_common.h"
#include "gate_dev.h"

namespace rrtl {

template <int V>
struct FlatVec;
template <>
struct FlatVec<1> {
  using T = uint32_t;
};
template <>
struct FlatVec<2> {
  using T = uint2;
};
template <>
struct FlatVec<4> {
  using T = uint4;
};

__device__ __forceinline__ uint32_t flat_sign_mask3(uint32_t x) {  // bit 31 of x over the word
  uint32_t d;
  asm("prmt.b32 %0, %1, 0, 0xBBBB;" : "=r"(d) : "r"(x));
  return d;
}
__device__ __forceinline__ uint32_t flat_sign_mask2(uint32_t x) {  // bit 23
  uint32_t d;
  asm("prmt.b32 %0, %1, 0, 0xAAAA;" : "=r"(d) : "r"(x));
  return d;
}
__device__ __forceinline__ uint32_t flat_sign_mask1(uint32_t x) {  // bit 15
  uint32_t d;
  asm("prmt.b32 %0, %1, 0, 0x9999;" : "=r"(d) : "r"(x));
  return d;
}
__device__ __forceinline__ uint32_t flat_sign_mask0(uint32_t x) {  // bit 7
  uint32_t d;
  asm("prmt.b32 %0, %1, 0, 0x8888;" : "=r"(d) : "r"(x));
  return d;
}

// A two-input function by its algebraic normal form: 3 LOP3 for any table.
struct FlatTwo {
  uint32_t k0, k1, k2, k3;
  __device__ __forceinline__ explicit FlatTwo(uint32_t y) {
    const uint32_t z = y << 1;
    k0 = flat_sign_mask2(y);
    k1 = flat_sign_mask3(y);
    k2 = flat_sign_mask2(z);
    k3 = flat_sign_mask3(z);
  }
  __device__ __forceinline__ uint32_t operator()(uint32_t a, uint32_t b) const {
    return lop3<0x6A>(b, lop3<0x6A>(a, k3, k2), lop3<0x6A>(a, k1, k0));  // 0x6A: (x & y) ^ z
  }
  __device__ __forceinline__ uint2 operator()(uint2 a, uint2 b) const {
    return make_uint2((*this)(a.x, b.x), (*this)(a.y, b.y));
  }
  __device__ __forceinline__ uint4 operator()(uint4 a, uint4 b) const {
    return make_uint4((*this)(a.x, b.x), (*this)(a.y, b.y), (*this)(a.z, b.z), (*this)(a.w, b.w));
  }
};

// A three-input function f = g0 ^ c g1: 7 LOP3.
struct FlatThree {
  uint32_t p0, p1, p2, p3, q0, q1, q2, q3;
  __device__ __forceinline__ explicit FlatThree(uint32_t w) {
    const uint32_t z = w << 1;
    p0 = flat_sign_mask0(w);
    p1 = flat_sign_mask1(w);
    p2 = flat_sign_mask2(w);
    p3 = flat_sign_mask3(w);
    q0 = flat_sign_mask0(z);
    q1 = flat_sign_mask1(z);
    q2 = flat_sign_mask2(z);
    q3 = flat_sign_mask3(z);
  }
  __device__ __forceinline__ uint32_t operator()(uint32_t a, uint32_t b, uint32_t c) const {
    const uint32_t g0 = lop3<0x6A>(b, lop3<0x6A>(a, p3, p2), lop3<0x6A>(a, p1, p0));
    const uint32_t g1 = lop3<0x6A>(b, lop3<0x6A>(a, q3, q2), lop3<0x6A>(a, q1, q0));
    return lop3<0x6A>(c, g1, g0);
  }
  __device__ __forceinline__ uint2 operator()(uint2 a, uint2 b, uint2 c) const {
    return make_uint2((*this)(a.x, b.x, c.x), (*this)(a.y, b.y, c.y));
  }
  __device__ __forceinline__ uint4 operator()(uint4 a, uint4 b, uint4 c) const {
    return make_uint4((*this)(a.x, b.x, c.x), (*this)(a.y, b.y, c.y), (*this)(a.z, b.z, c.z), (*this)(a.w, b.w, c.w));
  }
};

__device__ __forceinline__ uint4 flat_load_entry(const uint4* p) {
  uint4 r;
  asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
  return r;
}

// The barrier between levels of one warp set (ids from 2), for as many
// threads as the program has streams; kFull is that count where it is every
// warp of the set (as an immediate the barrier is cheaper: 2% of a
// tile-cycle of 16 words), 0 where it is known at run time only.
template <int kFull>
struct FlatBar {
  uint32_t id, threads;
  // Passed when `go` is not zero (the same on every lane of the warp).
  __device__ __forceinline__ void pass(uint32_t go) const {
    if constexpr (kFull > 0)
      asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %0, 0;\n @p bar.sync %1, %2;\n}\n" ::"r"(go), "r"(id), "n"(kFull)
                   : "memory");
    else
      asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %0, 0;\n @p bar.sync %1, %2;\n}\n" ::"r"(go), "r"(id), "r"(threads)
                   : "memory");
  }
};

__device__ __forceinline__ void flat_bar_service() {
  __syncwarp();
  asm volatile("bar.sync 1, %0;" ::"n"(kFlatServiceThreads) : "memory");
}

// Row `slot` of the slot array (kBytes: its byte offset).
template <int V, bool kBytes>
__device__ __forceinline__ const typename FlatVec<V>::T* flat_row(const uint8_t* S, uint32_t slot) {
  return reinterpret_cast<const typename FlatVec<V>::T*>(S + (kBytes ? slot : slot * (V * 4u)));
}

// Entries of two cells per lane (two inputs) and one cell per lane (three
// inputs), each over the set's N vectors. Cells of a level never read each
// other's rows, so every load of an entry may precede its stores (which the
// compiler cannot know). Functions and row addresses are decoded before the
// level barrier the entry may wait for.
// `out` sees every row vector written: out(which cell, plane, value).
template <int V, int N, int Q, bool kBytes, class Bar, class Out>
__device__ __forceinline__ void flat_pair2(uint8_t* S, const uint4& r, uint32_t go, const Bar& bar, const Out& out) {
  using T = typename FlatVec<V>::T;
  constexpr uint32_t kStep = flat_plane_bytes(N * Q) / sizeof(T);
  constexpr int H = N > 2 ? 2 : N;  // planes whose operands are in registers at once
  const FlatTwo f(r.y), g(r.w);
  const T* const pa = flat_row<V, kBytes>(S, r.x & 0xFFFFu);
  const T* const pb = flat_row<V, kBytes>(S, r.x >> 16);
  const T* const pc = flat_row<V, kBytes>(S, r.z & 0xFFFFu);
  const T* const pd = flat_row<V, kBytes>(S, r.z >> 16);
  T* const po = const_cast<T*>(flat_row<V, kBytes>(S, r.y & 0xFFFFu));
  T* const pq = const_cast<T*>(flat_row<V, kBytes>(S, r.w & 0xFFFFu));
  bar.pass(go);
#pragma unroll
  for (int p0 = 0; p0 < N; p0 += H) {
    T a[H], b[H], c[H], d[H];
#pragma unroll
    for (int p = 0; p < H; ++p) {
      if (p0 + p >= N) break;
      a[p] = pa[(p0 + p) * kStep];
      b[p] = pb[(p0 + p) * kStep];
      c[p] = pc[(p0 + p) * kStep];
      d[p] = pd[(p0 + p) * kStep];
    }
#pragma unroll
    for (int p = 0; p < H; ++p) {
      if (p0 + p >= N) break;
      const T v = f(a[p], b[p]), w = g(c[p], d[p]);
      po[(p0 + p) * kStep] = v;
      pq[(p0 + p) * kStep] = w;
      out(0, p0 + p, v);
      out(1, p0 + p, w);
    }
  }
}

template <int V, int N, int Q, bool kBytes, class Bar, class Out>
__device__ __forceinline__ void flat_one3(uint8_t* S, const uint4& r, uint32_t go, const Bar& bar, const Out& out) {
  using T = typename FlatVec<V>::T;
  constexpr uint32_t kStep = flat_plane_bytes(N * Q) / sizeof(T);
  constexpr int H = N > 2 ? 2 : N;
  const FlatThree f(r.w);
  const T* const pa = flat_row<V, kBytes>(S, r.x & 0xFFFFu);
  const T* const pb = flat_row<V, kBytes>(S, r.x >> 16);
  const T* const pc = flat_row<V, kBytes>(S, r.z);
  T* const po = const_cast<T*>(flat_row<V, kBytes>(S, r.y & 0xFFFFu));
  bar.pass(go);
#pragma unroll
  for (int p0 = 0; p0 < N; p0 += H) {
    T a[H], b[H], c[H];
#pragma unroll
    for (int p = 0; p < H; ++p) {
      if (p0 + p >= N) break;
      a[p] = pa[(p0 + p) * kStep];
      b[p] = pb[(p0 + p) * kStep];
      c[p] = pc[(p0 + p) * kStep];
    }
#pragma unroll
    for (int p = 0; p < H; ++p) {
      if (p0 + p >= N) break;
      const T v = f(a[p], b[p], c[p]);
      po[(p0 + p) * kStep] = v;
      out(0, p0 + p, v);
    }
  }
}

struct FlatNoOut {
  template <class T>
  __device__ __forceinline__ void operator()(int, int, const T&) const {}
};

// Stuck-at forces of the comb nets one warp writes, applied by that warp when
// it finished a level, before the level's barrier: no barrier of their own.
// The list is sorted by level; each lane holds one force of a 32-force
// window, which moves on once its last force's level is done.
struct FlatForces {
  const uint4* base;
  uint32_t n, at, due;  // due: next level with a force
  uint4 f;
  __device__ __forceinline__ void load(uint32_t lane) {
    f = at + lane < n ? __ldg(base + at + lane) : make_uint4(0u, 0u, 0u, 0xFFFFFFFFu);
  }
  __device__ __forceinline__ void begin(uint32_t lane, bool first) {
    if (first || at) {
      at = 0u;
      load(lane);
    }
    due = __reduce_min_sync(0xFFFFFFFFu, f.w);
  }
  __device__ __forceinline__ void set(uint8_t* S, uint32_t level) const {
    if (f.w == level) {
      uint32_t& v = *reinterpret_cast<uint32_t*>(S + f.x);
      v = (v & ~f.y) | (f.z & f.y);
    }
  }
  // Before the level's barrier: the forces of `level`.
  __device__ __forceinline__ void apply(uint8_t* S, uint32_t level, uint32_t lane) {
    if (level != due) return;
    __syncwarp();  // the warp's rows of this level are written
    set(S, level);
    while (at + 32u < n && last() <= level) {
      at += 32u;
      load(lane);
      set(S, level);
    }
  }
  // After it, where the other warps' row accesses cover the latency: the next level due.
  __device__ __forceinline__ void advance(uint32_t level) {
    if (level == due) due = __reduce_min_sync(0xFFFFFFFFu, f.w > level ? f.w : 0xFFFFFFFFu);
  }
  __device__ __forceinline__ uint32_t last() const { return __shfl_sync(0xFFFFFFFFu, f.w, 31); }
};

template <int kCompute>
__device__ __forceinline__ void flat_bar_compute() {
  __syncwarp();
  asm volatile("bar.sync 6, %0;" ::"n"(kCompute) : "memory");
}

// Source rows of a tile of W words in (words past the padded batch read as zero).
template <int V, uint32_t W, uint32_t kPlane>
__device__ __forceinline__ void flat_load_sources(const FlatProgDev& P, const GateRunDev& R, uint32_t col0, uint8_t* S) {
  for (uint32_t i = threadIdx.x; i < P.n_src * W; i += blockDim.x) {
    const uint32_t k = i / W, ww = i % W;
    *reinterpret_cast<uint32_t*>(S + (ww / V) * kPlane + __ldg(P.src_slot + k) * (V * 4u) + (ww % V) * 4u) =
        col0 + ww < R.words_pad ? R.nets[(size_t)__ldg(P.src_net + k) * R.words_pad + col0 + ww] : 0u;
  }
}

// Closing settle of one tile (V * N words): the levels once, every signal net
// written back to the run's global rows as it is computed. Bound: the
// write-back (4 bytes a signal and word) and, in small batches, the level
// chain. As a separate fused-kernel launch at its widest tile the settle left
// most SMs idle in small batches and stored word by word: whole runs that end
// with this one instead went from 1.51 to 1.41 ms (50,000 gates, 200 lanes,
// 100 cycles), 3.26 to 3.11 (5,003 lanes, 200 cycles), 7.04 to 6.35 (200,000
// gates, 10,007 lanes, 100 cycles) and 47.5 to 47.2 (65,536 lanes, 1,000).
template <int V, int N>
__device__ __forceinline__ void flat_settle_tile(const FlatProgDev& P, const GateRunDev& R, uint32_t tile, uint8_t* smem) {
  using T = typename FlatVec<V>::T;
  constexpr uint32_t W = V * N;
  constexpr int D = (int)kFlatPrefetch;
  uint8_t* const S = smem + kFlatHeader;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, col0 = tile * W;
  flat_load_sources<V, W, flat_plane_bytes(N)>(P, R, col0, S);
  __syncthreads();
  if (warp < P.warps) {
    const FlatBar<0> bar{2u, P.warps * 32u};
    const uint32_t begin = __ldg(P.warp_begin + warp), n = __ldg(P.warp_begin + warp + 1) - begin;
    const uint4* const base = P.stream + (size_t)begin * 32u + lane;
    const uint2* const nets = P.stream_net + (size_t)begin * 32u + lane;
    uint4 q[D];
    uint2 w[D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      q[d] = n ? flat_load_entry(base + d * 32) : make_uint4(0u, 0u, 0u, 0u);
      w[d] = n ? __ldg(nets + d * 32) : make_uint2(0u, 0u);
    }
    for (uint32_t e = 0; e < n; e += D) {
      const uint32_t ahead = e + D < n ? e + D : 0u;
      uint4 nx[D];
      uint2 wx[D];
#pragma unroll
      for (int d = 0; d < D; ++d) {
        nx[d] = flat_load_entry(base + (size_t)(ahead + d) * 32u);
        wx[d] = __ldg(nets + (size_t)(ahead + d) * 32u);
      }
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const uint4 r = q[d];
        const uint2 id = w[d];
        auto out = [&](int h, int plane, const T& v) {
          const uint32_t net = h ? id.y : id.x, col = col0 + (uint32_t)plane * V;
          if (net != 0xFFFFFFFFu && col < R.words_pad) *reinterpret_cast<T*>(R.nets + (size_t)net * R.words_pad + col) = v;
        };
        const uint32_t go = r.y & kFlatDevSync;
        if (__any_sync(0xFFFFFFFFu, r.y & kFlatDevThree)) flat_one3<V, N, 1, false>(S, r, go, bar, out);
        else flat_pair2<V, N, 1, false>(S, r, go, bar, out);
      }
#pragma unroll
      for (int d = 0; d < D; ++d) {
        q[d] = nx[d];
        w[d] = wx[d];
      }
    }
    for (uint32_t k = __ldg(P.warp_tail + warp); k; --k) bar.pass(1u);
  }
  __syncthreads();
}

// Cycles [c0, c0 + ncyc) of one tile (V * N * Q words) of a run; F: with
// stuck-at forces; kFull: the program has a stream for every warp of a set;
// kBytes: its entries hold byte offsets; kCompute: compute threads.
// Source nets are read from and written back to the run's global rows; the
// caller settles the other nets (the closing settle) afterwards.
template <int V, int N, int Q, bool F, bool kFull, bool kBytes, int kCompute>
__device__ __forceinline__ void flat_tile(const FlatProgDev& P, const GateRunDev& R, uint32_t tile, uint64_t c0,
                                          uint64_t ncyc, uint8_t* smem) {
  constexpr uint32_t W = V * N * Q;
  constexpr uint32_t kPlane = flat_plane_bytes(N * Q);
  constexpr int D = (int)kFlatPrefetch;
  uint32_t* dstate = reinterpret_cast<uint32_t*>(smem);  // diff[16], detected[16]
  uint8_t* const S = smem + kFlatHeader;
  const uint32_t tid = threadIdx.x, lane = tid & 31u;
  const uint32_t col0 = tile * W;
  auto word_at = [&](uint32_t slot, uint32_t ww) -> uint32_t& {  // word ww of the tile
    return *reinterpret_cast<uint32_t*>(S + (ww / V) * kPlane + slot * (V * 4u) + (ww % V) * 4u);
  };
  flat_load_sources<V, W, kPlane>(P, R, col0, S);
  if (tid < 16u) {
    // lanes already detected by an earlier part of this run stay detected
    dstate[tid] = 0u;
    dstate[16 + tid] = (R.mode & RRTL_REC_DETECT) && tid < W ? detected_lanes(R.detect, col0 + tid, R.lanes) : 0u;
  }
  __syncthreads();
  const bool serial = F || P.n_commit != 0 || R.flat_serial;
  if (tid < kCompute) {
    constexpr uint32_t kSetWarps = kCompute / 32 / Q;
    const uint32_t set = Q == 1 ? 0u : tid / (kCompute / Q), warp = (tid >> 5) % kSetWarps;
    uint8_t* const Sq = S + set * (N * kPlane);  // the set's planes
    const FlatBar<kFull ? kCompute / Q : 0> bar{2u + set, P.warps * 32u};
    const bool active = warp < P.warps;  // a program of few cells a level has fewer streams than the set has warps
    const uint32_t begin = active ? __ldg(P.warp_begin + warp) : 0u, n = active ? __ldg(P.warp_begin + warp + 1) - begin : 0u;
    const uint32_t tail = active ? __ldg(P.warp_tail + warp) : 0u;
    const uint4* const base = P.stream + (size_t)begin * 32u + lane;
    FlatForces forces{};
    uint32_t begin0 = 0, end0 = 0;  // forces of registers; the thread's first stays in registers
    uint4 first0{};
    if constexpr (F) {
      const uint32_t k = (tile * Q + set) * P.warps + warp;
      forces.base = R.flat_forces + (active ? __ldg(R.flat_off + k) : 0u);
      forces.n = active ? __ldg(R.flat_off + k + 1) - __ldg(R.flat_off + k) : 0u;
      forces.begin(lane, true);
      begin0 = __ldg(R.flat_off0 + tile);
      end0 = __ldg(R.flat_off0 + tile + 1);
      if (begin0 + tid < end0) first0 = __ldg(R.flat_forces0 + begin0 + tid);
    }
    uint4 q[D];
#pragma unroll
    for (int d = 0; d < D; ++d) q[d] = n ? flat_load_entry(base + d * 32) : make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();  // first cycle's stimulus in place
    for (uint64_t c = 0; c < ncyc; ++c) {
      uint32_t level = 0;
      if constexpr (F) forces.begin(lane, false);
      // entries [e, e + D) from `cur`, the D after them (the next cycle's first behind the last) into `nx`
      auto batch = [&](const uint4 (&cur)[D], uint4 (&nx)[D], uint32_t e) {
        const uint4* const ahead = base + (size_t)(e + D < n ? e + D : 0u) * 32u;
#pragma unroll
        for (int d = 0; d < D; ++d) nx[d] = flat_load_entry(ahead + d * 32);
#pragma unroll
        for (int d = 0; d < D; ++d) {
          const uint4 r = cur[d];
          const uint32_t go = r.y & kFlatDevSync;
          if constexpr (F) {
            if (go) forces.apply(S, level, lane);  // the same on every lane
          }
          // (the vote makes the branch a warp-uniform one)
          if (__any_sync(0xFFFFFFFFu, r.y & kFlatDevThree)) flat_one3<V, N, Q, kBytes>(Sq, r, go, bar, FlatNoOut{});
          else flat_pair2<V, N, Q, kBytes>(Sq, r, go, bar, FlatNoOut{});
          if constexpr (F) {
            if (go) forces.advance(level++);
          }
        }
      };
      uint4 nx[D];
      if constexpr (V < 4 && !F) {
        // narrow rows are bound by the instructions of an entry: two batches a turn, in place of the copies
        for (uint32_t e = 0; e < n; e += 2 * D) {
          batch(q, nx, e);
          if (e + D < n) {
            batch(nx, q, e + D);
          } else {
#pragma unroll
            for (int d = 0; d < D; ++d) q[d] = nx[d];
          }
        }
      } else {
        for (uint32_t e = 0; e < n; e += D) {
          batch(q, nx, e);
#pragma unroll
          for (int d = 0; d < D; ++d) q[d] = nx[d];
        }
      }
      for (uint32_t k = tail; k; --k) {
        if constexpr (F) forces.apply(S, level, lane);
        bar.pass(1u);
        if constexpr (F) forces.advance(level++);
      }
      if constexpr (F) forces.apply(S, level, lane);
      __syncthreads();  // every level done
      if (serial) {
        // registers left on the commit list
        for (uint32_t i = tid; i < P.n_commit * W; i += kCompute) {
          const uint4 rr = __ldg(reinterpret_cast<const uint4*>(P.commit) + i / W);
          const uint32_t ww = i % W;
          uint32_t d = rr.y == kFlatConst0 ? 0u : rr.y == kFlatConst1 ? 0xFFFFFFFFu : word_at(rr.y, ww);
          if (rr.w & 1u) {
            uint32_t m = rr.z == kFlatConst0 ? 0u : rr.z == kFlatConst1 ? 0xFFFFFFFFu : word_at(rr.z, ww);
            if (rr.w & 2u) m = ~m;
            d = (rr.w & 4u) ? d | m : d & ~m;
          }
          word_at(rr.x, ww) = d;
        }
        if constexpr (F) {
          if (P.n_commit) flat_bar_compute<kCompute>();
          for (uint32_t i = begin0 + tid; i < end0; i += kCompute) {
            const uint4 f = i == begin0 + tid ? first0 : __ldg(R.flat_forces0 + i);
            uint32_t& v = *reinterpret_cast<uint32_t*>(S + f.x);
            v = (v & ~f.y) | (f.z & f.y);
          }
        }
        __syncthreads();
      }
      __syncthreads();  // next cycle's stimulus in place
    }
  } else {
    const uint32_t st = tid - kCompute;
    constexpr int KS = 10, KR = 8;  // stimulus and record words a thread holds in registers
    const uint32_t n_stim = R.n_stim * W, n_rec = R.n_rec * W;
    uint32_t sv[KS], rv[KR];
    auto stim_of = [&](uint32_t i, uint64_t c) -> uint32_t {  // never HOLD
      const GateStimDev& s = R.stim[i / W];
      return s.kind == RRTL_STIM_HOLD ? 0u : stim_value(s, R, c, col0 + i % W, 0u);
    };
    auto stim_prepare = [&](uint64_t c) {
#pragma unroll
      for (int j = 0; j < KS; ++j) {
        const uint32_t i = st + j * kFlatServiceThreads;
        sv[j] = i < n_stim ? stim_of(i, c) : 0u;
      }
    };
    auto stim_store = [&](uint64_t c) {
#pragma unroll
      for (int j = 0; j < KS; ++j) {
        const uint32_t i = st + j * kFlatServiceThreads;
        if (i < n_stim && R.stim[i / W].kind != RRTL_STIM_HOLD) word_at(R.stim[i / W].slot, i % W) = sv[j];
      }
      for (uint32_t i = st + KS * kFlatServiceThreads; i < n_stim; i += kFlatServiceThreads)
        if (R.stim[i / W].kind != RRTL_STIM_HOLD) word_at(R.stim[i / W].slot, i % W) = stim_of(i, c);
    };
    unsigned long long hs = 0ull;
    auto record_word = [&](uint64_t c, uint32_t i, uint32_t v) {
      const uint32_t k = i / W, ww = i % W, gw = col0 + ww;
      v &= valid_mask(gw, R.lanes);
      if (gw >= R.words) return;
      if (R.mode & RRTL_REC_TRACE) R.out_trace[((size_t)c * R.n_rec + k) * R.words + gw] = v;
      if (R.mode & RRTL_REC_HASH) hs += hash_term(c, k, R.word_base + gw, v);
      if (R.mode & RRTL_REC_DETECT) atomicOr(&dstate[ww], v ^ (0u - (v & 1u)));
      if (R.mode & RRTL_REC_CHECK) check_word(R, c, k, gw, v);
    };
    stim_prepare(c0);
    stim_store(c0);
    __syncthreads();
    for (uint64_t c = 0; c < ncyc; ++c) {
      const bool more = c + 1 < ncyc;
      if (more) stim_prepare(c0 + c + 1);
      __syncthreads();  // every level done
      hs = 0ull;
#pragma unroll
      for (int j = 0; j < KR; ++j) {
        const uint32_t i = st + j * kFlatServiceThreads;
        rv[j] = i < n_rec ? word_at(R.rec[i / W].slot, i % W) : 0u;
      }
      for (uint32_t i = st + KR * kFlatServiceThreads; i < n_rec; i += kFlatServiceThreads)
        record_word(c0 + c, i, word_at(R.rec[i / W].slot, i % W));
      if (serial) __syncthreads();
      if (more) stim_store(c0 + c + 1);
      __syncthreads();
      if (R.n_rec) {
#pragma unroll
        for (int j = 0; j < KR; ++j) {
          const uint32_t i = st + j * kFlatServiceThreads;
          if (i < n_rec) record_word(c0 + c, i, rv[j]);
        }
        if (R.mode & RRTL_REC_HASH) {
          for (int o = 16; o > 0; o >>= 1) hs += __shfl_xor_sync(0xFFFFFFFFu, hs, o);
          if (lane == 0 && hs) atomicAdd(R.out_hash + c0 + c, hs);
        }
        if (R.mode & RRTL_REC_DETECT) {
          flat_bar_service();
          if (st < W) {
            const uint32_t gw = col0 + st;
            uint32_t nb = dstate[st] & ~dstate[16 + st] & valid_mask(gw, R.lanes);
            dstate[16 + st] |= nb;
            dstate[st] = 0u;
            while (nb) {
              const uint32_t b = __ffs(nb) - 1u;
              R.detect[gw * 32u + b] = (uint32_t)(c0 + c);
              nb &= nb - 1u;
            }
          }
        }
      }
    }
  }
  __syncthreads();
  for (uint32_t i = tid; i < P.n_src * W; i += blockDim.x) {
    const uint32_t k = i / W, ww = i % W;
    if (col0 + ww < R.words_pad) R.nets[(size_t)__ldg(P.src_net + k) * R.words_pad + col0 + ww] = word_at(__ldg(P.src_slot + k), ww);
  }
  __syncthreads();
}

}  // namespace rrtl
