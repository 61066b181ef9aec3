// Flat gate kernel (gate_flat.h): launchers per row width V and vectors per
// tile N.
#include <cuda_runtime.h>

#include "gate_flat.h"

namespace rrtl {

template <int V, int N, int Q, bool F>
__global__ void __launch_bounds__(kFlatThreads, 1) gate_flat_kernel(FlatProgDev P, GateRunDev R) {
  extern __shared__ __align__(128) uint8_t smem[];
  for (uint32_t tile = blockIdx.x; tile < R.n_tiles; tile += gridDim.x)
    flat_tile<V, N, Q, F>(P, R, tile, R.cycle_base, R.cycles, smem);
}

template <int V, int N, int Q, bool F>
static cudaError_t launch_f(const FlatProgDev& P, const GateRunDev& R, uint32_t grid, cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(gate_flat_kernel<V, N, Q, F>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFlatSmem);
  if (e != cudaSuccess) return e;
  gate_flat_kernel<V, N, Q, F><<<grid, kFlatThreads, kFlatSmem, st>>>(P, R);
  return cudaGetLastError();
}

template <int V, int N, int Q>
static cudaError_t launch(const FlatProgDev& P, const GateRunDev& R, uint32_t grid, cudaStream_t st) {
  return R.has_forces ? launch_f<V, N, Q, true>(P, R, grid, st) : launch_f<V, N, Q, false>(P, R, grid, st);
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

}  // namespace rrtl
