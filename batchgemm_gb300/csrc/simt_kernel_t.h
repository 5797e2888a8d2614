// simt_kernel_t.h -- the persistent FP32 SIMT kernel for plans with transposed operands (A stored
// K x M, B stored N x K): one instantiation and one translation unit per
// combination, so that the tile code carries no per-operand branches and the
// three compile side by side.
#include "simt_tile.h"

namespace bgemm {
namespace {

__global__ void __launch_bounds__(simt::kThreads, 2)
    simt_persistent_kernel_t(const __grid_constant__ SimtParams p) {
  simt::persistent_body<BGEMM_SIMT_TA, BGEMM_SIMT_TB>(p);
}

}  // namespace

cudaError_t BGEMM_SIMT_LAUNCH(const SimtParams& p, int grid, cudaStream_t stream) {
  static bool attr_done = false;
  if (!attr_done) {
    const cudaError_t e =
        cudaFuncSetAttribute(simt_persistent_kernel_t, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             simt::kSmemBytes);
    if (e != cudaSuccess) return e;
    attr_done = true;
  }
  simt_persistent_kernel_t<<<grid, simt::kThreads, simt::kSmemBytes, stream>>>(p);
  return cudaGetLastError();
}

}  // namespace bgemm
