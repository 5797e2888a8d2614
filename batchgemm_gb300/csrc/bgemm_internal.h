// bgemm_internal.h -- structures shared by the host planner and the kernels.
#pragma once
#include <stdint.h>

#include <cuda_runtime.h>

namespace bgemm {

// Per-matrix descriptor, uploaded once per plan (32 bytes).
struct MatDesc {
  int M, N, K;
  int lda, ldb, ldc;
  int cfg;    // tile configuration id of the plan's mode
  int aux;    // flag bits below (plan paths); size bin (device-built framework path)
};
// MatDesc::aux flags: op(A) = A^T (A stored K x M), op(B) = B^T (B stored
// N x K); bit 30 is the tensor-core modes' operand swap.
constexpr int kTransAFlag = 1 << 28;
constexpr int kTransBFlag = 1 << 29;

// floor(4 * log2(x)) for x >= 1 (0 for smaller x), from the float's exponent
// and mantissa bits with fixed quarter-octave edges, so that the host
// replays of the device planners bin exactly as the device does (log2f of
// the host C library and of CUDA may differ in the last bit).
__host__ __device__ inline int quarter_octave(float x) {
  if (!(x >= 1.0f)) return 0;
  union {
    float f;
    uint32_t u;
  } v;
  v.f = x;
  const int e = (int)((v.u >> 23) & 0xffu) - 127;
  v.u = (v.u & 0x007fffffu) | 0x3f800000u;  // mantissa in [1, 2)
  const int q = (v.f >= 1.18920712f) + (v.f >= 1.41421356f) + (v.f >= 1.68179283f);
  return 4 * e + q;
}

// One work item of the largest-first tile queue (8 bytes).
struct TileItem {
  int mat;
  uint16_t tm, tn;  // tile coordinates along M and N (tensor-core swapped
                    // orientation: along the MMA's M and N)
};

// ------------------------------------------- programmatic dependent launch --
// The kernels of one call follow one another in a stream.  A kernel launched
// with pdl_launch may be set up once every CTA of the kernel before it has
// passed pdl_trigger() (or ended); all it does with memory stands behind its
// pdl_wait(), which waits for the end of that kernel.  So only the launch and
// the set-up overlap: two hand-overs of the device-size call (planner,
// expansion, SIMT kernel) took 2.5 us off its 47.5.
#ifdef __CUDACC__
__device__ __forceinline__ void pdl_trigger() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... Params, typename... Args>
cudaError_t pdl_launch(void (*kernel)(Params...), int grid, int threads, size_t smem,
                       cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid, 1, 1);
  cfg.blockDim = dim3((unsigned)threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}
#endif

// ---------------------------------------------------------------- SIMT ----
// Tile configurations of the FP32 SIMT kernel.  Ids 0 and 1 are computed by one
// warp (eight run side by side in a CTA), the others by a CTA of 256 threads.
struct SimtCfg {
  int bm, bn;  // tile
  int lm, ln;  // log2 of these
  int gm, gn;  // steps in which a ragged edge's outputs are skipped
};
constexpr int kSimtNumCfgs = 10;
constexpr SimtCfg kSimtCfgs[kSimtNumCfgs] = {
    {16, 16, 4, 4, 16, 16},  {32, 32, 5, 5, 16, 16},  {64, 32, 6, 5, 16, 16},
    {32, 64, 5, 6, 16, 16},  {64, 64, 6, 6, 16, 16},  {128, 64, 7, 6, 16, 16},
    {64, 128, 6, 7, 16, 16}, {128, 128, 7, 7, 32, 16}, {8, 128, 3, 7, 8, 16},
    {128, 8, 7, 3, 16, 8},
};
__host__ __device__ constexpr bool simt_warp_cfg(int cfg) { return cfg < 2; }
// What the planners choose from: ids 2 to 6 run only when forced (64 x 64 as a
// choice of its own gained a third on one batch in 90, a large matrix of odd
// leading dimensions among 49 small ones, and lost on as many as it won of the
// others); a thin matrix takes a thin tile or, where even that is mostly padding, 16 x 16 ones (K = 4096 and M or
// N <= 8, two batches of about 100 each: 568 and 474 us in thin tiles, 664 and
// 610 in 16 x 16, 857 and 875 in 32 x 32).
__host__ __device__ constexpr bool simt_auto_cfg(int cfg, int M, int N) {
  return cfg == 0 || (cfg == 8 ? M <= 8 : cfg == 9 ? N <= 8
                                                   : (cfg == 1 || cfg == 7) && M > 8 && N > 8);
}

struct SimtParams {
  const MatDesc* descs;
  const TileItem* items;
  int n_items;
  const int* n_items_dev;  // if set, the item count is read from the device
  int* counters;  // [0]: next work item, [1]: CTAs finished (self-reset)
  float alpha, beta;
  const float* const* A;
  const float* const* B;
  float* const* C;
};

// ta / tb: the plan's matrices carry kTransAFlag / kTransBFlag
cudaError_t simt_launch(const SimtParams& p, int grid, cudaStream_t stream, bool ta = false,
                        bool tb = false);
// behind a kernel that triggers (the device planner's)
cudaError_t simt_launch_behind(const SimtParams& p, int grid, cudaStream_t stream);
int simt_ctas_per_sm();

}  // namespace bgemm
