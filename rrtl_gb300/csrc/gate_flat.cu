// Flat gate kernel (gate_flat.h): launchers per row width V and vectors per
// tile N.
#include <cuda_runtime.h>

#include "gate_flat.h"

namespace rrtl {

template <int V, int N, int Q, bool F, bool kFull>
__global__ void __launch_bounds__(kFlatThreads, 1) gate_flat_kernel(FlatProgDev P, GateRunDev R) {
  extern __shared__ __align__(128) uint8_t smem[];
  for (uint32_t tile = blockIdx.x; tile < R.n_tiles; tile += gridDim.x)
    flat_tile<V, N, Q, F, kFull>(P, R, tile, R.cycle_base, R.cycles, smem);
}

template <int V, int N, int Q, bool F, bool kFull>
static cudaError_t launch_f(const FlatProgDev& P, const GateRunDev& R, uint32_t grid, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(gate_flat_kernel<V, N, Q, F, kFull>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFlatSmem);
  if (e != cudaSuccess) return e;
  gate_flat_kernel<V, N, Q, F, kFull><<<grid, kFlatThreads, kFlatSmem, st>>>(P, R);
  return cudaGetLastError();
}

template <int V, int N, int Q>
static cudaError_t launch(const FlatProgDev& P, const GateRunDev& R, uint32_t grid, cudaStream_t st) {
  if (R.has_forces) return launch_f<V, N, Q, true, false>(P, R, grid, st);
  return P.warps == kFlatComputeThreads / 32 / Q ? launch_f<V, N, Q, false, true>(P, R, grid, st)
                                                 : launch_f<V, N, Q, false, false>(P, R, grid, st);
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
  if (J.R.has_forces) flat_tile<V, N, Q, true, false>(J.P, J.R, item.tile, item.c0, item.ncyc, smem);
  else flat_tile<V, N, Q, false, false>(J.P, J.R, item.tile, item.c0, item.ncyc, smem);
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
