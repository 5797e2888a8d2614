// simt_kernel.cu -- persistent FP32 SIMT kernel for column-major vbatched SGEMM.
//
// Replaces the reference's dense-grid dispatcher (CUDA/framework/kernel.h:11-43,
// launched over (max tiles M, max tiles N, batch) at CUDA/framework/gemm.cu:181-200)
// and its tile bodies (CUDA/framework/kernel_128_new.h, kernel_256_new.h,
// CUDA/batching/kernel_256.h): one wave of persistent CTAs pulls work items
// from a largest-first tile queue with an atomic counter, so no CTA is
// launched for a tile outside its matrix.  The tiles themselves and the way a
// CTA's warps share the queue are in simt_tile.h; this file instantiates the
// reference's layout (both operands untransposed), simt_kernel_tn.cu, _nt.cu
// and _tt.cu the transposed ones.
#include "simt_tile.h"

namespace bgemm {
namespace {

__global__ void __launch_bounds__(simt::kThreads, 2)
    simt_persistent_kernel(const __grid_constant__ SimtParams p) {
  simt::persistent_body<false, false>(p);
}

}  // namespace

cudaError_t simt_launch_tn(const SimtParams& p, int grid, cudaStream_t stream);
cudaError_t simt_launch_nt(const SimtParams& p, int grid, cudaStream_t stream);
cudaError_t simt_launch_tt(const SimtParams& p, int grid, cudaStream_t stream);

static cudaError_t simt_attributes() {
  static bool done = false;
  if (done) return cudaSuccess;
  const cudaError_t e =
      cudaFuncSetAttribute(simt_persistent_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           simt::kSmemBytes);
  done = e == cudaSuccess;
  return e;
}

cudaError_t simt_launch(const SimtParams& p, int grid, cudaStream_t stream, bool ta, bool tb) {
  if (ta && tb) return simt_launch_tt(p, grid, stream);
  if (ta) return simt_launch_tn(p, grid, stream);
  if (tb) return simt_launch_nt(p, grid, stream);
  const cudaError_t e = simt_attributes();
  if (e != cudaSuccess) return e;
  simt_persistent_kernel<<<grid, simt::kThreads, simt::kSmemBytes, stream>>>(p);
  return cudaGetLastError();
}

cudaError_t simt_launch_behind(const SimtParams& p, int grid, cudaStream_t stream) {
  const cudaError_t e = simt_attributes();
  if (e != cudaSuccess) return e;
  return pdl_launch(simt_persistent_kernel, grid, simt::kThreads, simt::kSmemBytes, stream, p);
}

int simt_ctas_per_sm() {
  int n = 0;
  cudaFuncSetAttribute(simt_persistent_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       simt::kSmemBytes);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, simt_persistent_kernel, simt::kThreads,
                                                    simt::kSmemBytes) != cudaSuccess)
    return 1;
  // the transposed kernels have the same launch bounds and shared memory
  return n > 0 ? n : 1;
}

}  // namespace bgemm
