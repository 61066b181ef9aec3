// Flat gate kernel (gate_flat.h): launchers per row width V and vectors per
// tile N.
#include <cuda_runtime.h>

#include "gate_flat.h"

namespace rrtl {

// Waits until another block has run the first cycles of a tile split with it
// (flat_part). That block began them before anything else, so they are
// normally done. Bounded by far more than the run can take (a tile-cycle is
// under 0.2 ms); false when the bound ran out.
__device__ __forceinline__ bool flat_wait_part(const uint32_t* done, uint64_t cycles) {
  bool ok = true;
  if (threadIdx.x == 0) {
    uint32_t v = 0;
    for (uint64_t left = (1ull << 22) + cycles * 1024ull; left; --left) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(done) : "memory");
      if (v) break;
      __nanosleep(500);
    }
    ok = v != 0;
  }
  return __syncthreads_and(ok);
}

template <int V, bool F>
constexpr uint32_t flat_compute_threads() { return V < 4 && !F ? kFlatNarrowThreads : kFlatComputeThreads; }

// Blocks take equal shares of the run (flat_part) where its tiles do not fill
// the last round. A split tile costs one more load and store of its sources
// (one to two cycles), a last round up to all of the run: 200,000 gates, 10,007
// lanes x 100 cycles (157 tiles of 2 words on 152 SMs) 6.35 -> 5.36 ms; 50,000
// gates, 5,003 x 200 (157 of 1) 3.11 -> 2.91. At 65,536 lanes x 1,000 it makes
// 171 tiles of 12 words (42.5 ms) better than 128 of 16 (47.0), which leave 24
// SMs without a tile.
template <int V, int N, int Q, bool F, bool kFull, bool kBytes>
__global__ void __launch_bounds__(flat_compute_threads<V, F>() + kFlatServiceThreads, 1) gate_flat_kernel(FlatProgDev P, GateRunDev R) {
  extern __shared__ __align__(128) uint8_t smem[];
  for (uint32_t k = 0;; ++k) {
    FlatPart p{};
    if (R.flat_done) {
      p = flat_part(R.n_tiles, R.cycles, blockIdx.x, gridDim.x, k);
    } else {
      p.tile = blockIdx.x + k * gridDim.x;
      p.n = p.tile < R.n_tiles ? R.cycles : 0ull;
    }
    if (!p.n) break;
    if (p.last && !flat_wait_part(R.flat_done + p.tile, R.cycles)) {
      if (threadIdx.x == 0) atomicExch(R.err, (uint32_t)RRTL_E_TIMEOUT);
      break;
    }
    flat_tile<V, N, Q, F, kFull, kBytes, flat_compute_threads<V, F>()>(P, R, p.tile, R.cycle_base + p.c0, p.n, smem);
    if (p.first && threadIdx.x == 0) {
      __threadfence();  // the tile's state, written before flat_tile's last barrier
      asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(R.flat_done + p.tile), "r"(1u) : "memory");
    }
  }
}

template <int V, int N, int Q, bool F, bool kFull, bool kBytes>
static cudaError_t launch_f(const FlatProgDev& P, const GateRunDev& R, uint32_t grid, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(gate_flat_kernel<V, N, Q, F, kFull, kBytes>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFlatSmem);
  if (e != cudaSuccess) return e;
  constexpr uint32_t threads = flat_compute_threads<V, F>() + kFlatServiceThreads;
  if (R.flat_done) {
    // blocks wait for one another: all of them resident, or whole tiles
    void* args[] = {const_cast<FlatProgDev*>(&P), const_cast<GateRunDev*>(&R)};
    e = cudaLaunchCooperativeKernel(gate_flat_kernel<V, N, Q, F, kFull, kBytes>, dim3(grid), dim3(threads), args, kFlatSmem, st);
    if (e != cudaErrorCooperativeLaunchTooLarge && e != cudaErrorNotSupported) return e;
    cudaGetLastError();
    GateRunDev whole = R;
    whole.flat_done = nullptr;
    gate_flat_kernel<V, N, Q, F, kFull, kBytes><<<grid, threads, kFlatSmem, st>>>(P, whole);
    return cudaGetLastError();
  }
  gate_flat_kernel<V, N, Q, F, kFull, kBytes><<<grid, threads, kFlatSmem, st>>>(P, R);
  return cudaGetLastError();
}

template <int V, int N, int Q>
static cudaError_t launch(const FlatProgDev& P, const GateRunDev& R, uint32_t grid, cudaStream_t st) {
  const bool full = P.warps == flat_compute_threads<V, false>() / 32 / Q;
  if constexpr (V == 1) {
    if (P.row_bytes) {
      if (R.has_forces) return launch_f<V, N, Q, true, false, true>(P, R, grid, st);
      return full ? launch_f<V, N, Q, false, true, true>(P, R, grid, st) : launch_f<V, N, Q, false, false, true>(P, R, grid, st);
    }
  }
  if (R.has_forces) return launch_f<V, N, Q, true, false, false>(P, R, grid, st);
  return full ? launch_f<V, N, Q, false, true, false>(P, R, grid, st) : launch_f<V, N, Q, false, false, false>(P, R, grid, st);
}

cudaError_t launch_gate_flat(uint32_t V, uint32_t N, uint32_t Q, const FlatProgDev& P, const GateRunDev& R, uint32_t grid,
                             cudaStream_t st) {
  switch (V * 100 + N * 10 + Q) {
    case 411: return launch<4, 1, 1>(P, R, grid, st);
    case 421: return launch<4, 2, 1>(P, R, grid, st);
    case 431: return launch<4, 3, 1>(P, R, grid, st);
    case 422: return launch<4, 2, 2>(P, R, grid, st);
    case 211: return launch<2, 1, 1>(P, R, grid, st);
    case 111: return launch<1, 1, 1>(P, R, grid, st);
    default: return cudaErrorInvalidValue;
  }
}

template <int V, int N>
__global__ void __launch_bounds__(kFlatThreads, 1) gate_flat_settle_kernel(FlatProgDev P, GateRunDev R) {
  extern __shared__ __align__(128) uint8_t smem[];
  for (uint32_t tile = blockIdx.x; tile < R.n_tiles; tile += gridDim.x) flat_settle_tile<V, N>(P, R, tile, smem);
}

template <int V, int N>
static cudaError_t launch_settle(const FlatProgDev& P, const GateRunDev& R, uint32_t grid, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(gate_flat_settle_kernel<V, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFlatSmem);
  if (e != cudaSuccess) return e;
  gate_flat_settle_kernel<V, N><<<grid, kFlatThreads, kFlatSmem, st>>>(P, R);
  return cudaGetLastError();
}

cudaError_t launch_gate_flat_settle(uint32_t V, uint32_t N, const FlatProgDev& P, const GateRunDev& R, uint32_t grid,
                                    cudaStream_t st) {
  switch (V * 10 + N) {
    case 42: return launch_settle<4, 2>(P, R, grid, st);
    case 41: return launch_settle<4, 1>(P, R, grid, st);
    case 21: return launch_settle<2, 1>(P, R, grid, st);
    case 11: return launch_settle<1, 1>(P, R, grid, st);
    default: return cudaErrorInvalidValue;
  }
}

// Persistent queue kernel: CTAs take (job, tile) items, all cycles of the
// job, from a device list (longest first) until it is empty. The job's
// descriptor lies in the header of shared memory, behind the detection state.
template <int V, int N, int Q>
__device__ __forceinline__ void queue_tile(const FlatJobDev& J, const GateItemDev& item, uint8_t* smem) {
  if (J.settle) {
    if constexpr (Q == 1) flat_settle_tile<V, N>(J.P, J.R, item.tile, smem);
    return;
  }
  if constexpr (V == 1) {
    if (J.P.row_bytes) {
      if (J.R.has_forces) flat_tile<V, N, Q, true, false, true, kFlatComputeThreads>(J.P, J.R, item.tile, item.c0, item.ncyc, smem);
      else flat_tile<V, N, Q, false, false, true, kFlatComputeThreads>(J.P, J.R, item.tile, item.c0, item.ncyc, smem);
      return;
    }
  }
  if (J.R.has_forces) flat_tile<V, N, Q, true, false, false, kFlatComputeThreads>(J.P, J.R, item.tile, item.c0, item.ncyc, smem);
  else flat_tile<V, N, Q, false, false, false, kFlatComputeThreads>(J.P, J.R, item.tile, item.c0, item.ncyc, smem);
}

__global__ void __launch_bounds__(kFlatThreads, 1) gate_flat_queue_kernel(FlatQueueDev L) {
  extern __shared__ __align__(128) uint8_t smem[];
  uint32_t& s_item = *reinterpret_cast<uint32_t*>(smem + 128);
  FlatJobDev& J = *reinterpret_cast<FlatJobDev*>(smem + 136);
  static_assert(136 + sizeof(FlatJobDev) <= kFlatHeader, "the job descriptor overflows the header");
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(L.next, 1u);
    __syncthreads();
    const uint32_t it = s_item;
    if (it >= L.n_items) break;
    const GateItemDev item = L.items[it];
    for (uint32_t i = threadIdx.x; i < sizeof(FlatJobDev) / 4; i += blockDim.x)
      reinterpret_cast<uint32_t*>(&J)[i] = reinterpret_cast<const uint32_t*>(L.jobs + item.job)[i];
    __syncthreads();  // also orders the s_item read before its next write
    switch (J.shape) {
      case 422: queue_tile<4, 2, 2>(J, item, smem); break;
      case 421: queue_tile<4, 2, 1>(J, item, smem); break;
      case 411: queue_tile<4, 1, 1>(J, item, smem); break;
      case 211: queue_tile<2, 1, 1>(J, item, smem); break;
      case 111: queue_tile<1, 1, 1>(J, item, smem); break;
      default: break;
    }
  }
}

cudaError_t launch_gate_flat_queue(const FlatQueueDev& L, uint32_t grid, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(gate_flat_queue_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFlatSmem);
  if (e != cudaSuccess) return e;
  gate_flat_queue_kernel<<<grid, kFlatThreads, kFlatSmem, st>>>(L);
  return cudaGetLastError();
}

}  // namespace rrtl
