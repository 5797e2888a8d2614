// framework.cu -- drop-in for the reference framework's kernel entry
//   gemm<<<grid, 256, 16 KB>>>(M, N, K, A, B, C, T_strategy)
// (CUDA/framework/kernel.h:11, launched at CUDA/framework/gemm.cu:200): the
// sizes are device arrays, C_i += A_i * B_i column-major with lda = M_i,
// ldb = K_i, ldc = M_i.
//
// Because the sizes live on the device, the tile queue is built there too:
//   1. fw_plan_kernel (one CTA) picks each matrix's SIMT tile configuration
//      with the host planner's model and rule (tile_table.h), buckets matrices
//      by modelled tile time (quarter-octave bins) and reserves each matrix a
//      contiguous range of the queue, longest tiles first;
//   2. fw_expand_kernel writes the work items (one warp per matrix);
//   3. the persistent SIMT kernel reads the item count from the device.
// The three launches allocate nothing and can be captured in a CUDA graph;
// the queue scratch is owned by the library (one buffer per device, grown
// when a call needs more).
#include <algorithm>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "bgemm.h"
#include "bgemm_internal.h"
#include "plan_internal.h"
#include "tile_table.h"

namespace bgemm {
namespace {

constexpr int kBins = 64;
constexpr int kPlanThreads = 1024;

__constant__ SimtCfg c_cfgs[kSimtNumCfgs];
__constant__ TileCost c_cost[kSimtNumCfgs];

struct FwScratch {
  int* err;         // bit 0: a size was negative or above max_dim
  int* n_items;
  int* counters;    // 2 ints: queue head, CTAs finished
  MatDesc* descs;   // [cap_batch]
  int* mat_start;   // [cap_batch] first queue slot of each matrix (-1: none)
  TileItem* items;  // [cap_items]
};

// A size that is negative or above max_dim: the matrix is skipped.
__host__ __device__ inline bool fw_bad(int M, int N, int K, int max_dim) {
  return M < 0 || N < 0 || K < 0 || M > max_dim || N > max_dim;
}
__host__ __device__ inline int fw_bin(int K, TileCost t) {
  const int q = quarter_octave(simt_tile_ns(K, t)) - 24;
  return q < 0 ? 0 : q > kBins - 1 ? kBins - 1 : q;
}

// Sum of a 64-bit value over the warp, in pieces that 32 lanes cannot overflow.
__device__ __forceinline__ long long warp_sum(long long v) {
  const unsigned long long u = (unsigned long long)v;
  const unsigned m = (1u << 27) - 1;
  const unsigned long long a = __reduce_add_sync(0xffffffffu, (unsigned)u & m);
  const unsigned long long b = __reduce_add_sync(0xffffffffu, (unsigned)(u >> 27) & m);
  const unsigned long long c = __reduce_add_sync(0xffffffffu, (unsigned)(u >> 54));
  return (long long)(a + (b << 27) + (c << 54));
}

// One thread per matrix.  One CTA, so its latency counts, not its throughput:
// a matrix's candidates are modelled once and stay in registers (in batches of
// more than kPlanThreads, where a thread takes several in turn, once a pass);
// the sums of every limit step are formed in one pass, per warp without
// atomics; warps that a small batch leaves idle share the steps; the bins'
// prefix sums run in parallel.  256 matrices: 16.5 us with 64-bit shared
// atomics and one thread's loop over the bins, 12.6 with all steps in the
// eight warps that had matrices and the candidates modelled three times,
// 9.1 as it is.
__global__ void __launch_bounds__(kPlanThreads)
    fw_plan_kernel(const int* __restrict__ dM, const int* __restrict__ dN,
                   const int* __restrict__ dK, int batch, int max_dim, int slots, FwScratch s) {
  constexpr int kPlanWarps = kPlanThreads / 32;
  static_assert(kPlanWarps == 32 && kSimtSteps < 32, "a warp per step, a lane per warp");
  __shared__ int bin_tiles[kBins];
  __shared__ int bin_start[kBins];
  __shared__ long long work_w[kPlanWarps][kSimtSteps + 1];
  __shared__ float longest_w[kPlanWarps][kSimtSteps + 1];
  __shared__ float makespan[kSimtSteps + 1];
  __shared__ float longest;
  __shared__ float limit;
  pdl_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the warps stand side by side over the matrices, as often as they go (each
  // such group takes every groups-th step)
  const int span = min((batch + 31) / 32, kPlanWarps);
  const int group = warp / span, groups = kPlanWarps / span;
  const int first = (warp - group * span) * 32 + lane;
  const bool once = batch <= kPlanThreads;
  int M = 0, N = 0, K = 0;  // the thread's matrix
  bool any = false;
  SimtCands e;
  auto fetch = [&](int i) {
    M = i < batch ? dM[i] : 0;
    N = i < batch ? dN[i] : 0;
    K = i < batch ? dK[i] : 0;
    any = !fw_bad(M, N, K, max_dim) && M > 0 && N > 0;
    if (any) simt_cands(M, N, K, -1, &e);
  };
  if (once && group < groups) fetch(first);
  if (threadIdx.x < kBins) bin_tiles[threadIdx.x] = 0;
  if (lane <= kSimtSteps) {
    work_w[warp][lane] = 0;
    longest_w[warp][lane] = 0.0f;
  }
  __syncwarp();
  auto sums = [&](int from, int to) {
    if (group < groups) {
      for (int i0 = first; i0 - lane < batch; i0 += span * 32) {
        if (!once) fetch(i0);
        float T = from == 0 ? 3e38f : simt_limit(longest, from + group);
        for (int j = from + group; j <= to; j += groups) {
          float w = 0.0f, l = 0.0f;
          if (any && simt_pick(e, T, &w, &l) < 0) w = l = 0.0f;
          const long long v = warp_sum((long long)w);
          // (no time is negative: ordered as their bits are)
          l = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(l)));
          if (lane == 0) {
            work_w[warp][j] += v;
            longest_w[warp][j] = fmaxf(longest_w[warp][j], l);
          }
          T = simt_limit(T, groups);
        }
      }
    }
    __syncthreads();
    if (warp >= from && warp <= to) {  // step `warp`, every warp's part
      const long long v = warp_sum(work_w[lane][warp]);
      const float l = __uint_as_float(
          __reduce_max_sync(0xffffffffu, __float_as_uint(longest_w[lane][warp])));
      if (lane == 0) {
        if (warp == 0) longest = l;
        makespan[warp] = simt_makespan(v, l, slots);
      }
    }
    __syncthreads();
  };
  sums(0, 0);
  sums(1, kSimtSteps);
  if (threadIdx.x == 0) limit = simt_choose_limit(makespan, longest);
  __syncthreads();
  // each matrix reserves its tiles in the bin of its tile time
  int start = -1, bin = 0;
  auto reserve = [&](int i) {
    MatDesc d{M, N, K, max(M, 1), max(K, 1), max(M, 1), 0, 0};
    start = -1;
    if (fw_bad(M, N, K, max_dim)) {
      atomicOr(s.err, 1);
    } else if (any) {
      float w, l;
      const int c = simt_pick(e, limit, &w, &l);
      if (c >= 0) {
        d.cfg = c;
        d.aux = bin = fw_bin(K, c_cost[c]);
        start = atomicAdd(&bin_tiles[bin], (int)simt_tiles(M, N, c_cfgs[c]));
      }
    }
    s.descs[i] = d;
  };
  if (once) {
    if (group == 0 && first < batch) reserve(first);
  } else {
    for (int i = threadIdx.x; i < batch; i += kPlanThreads) {
      fetch(i);
      reserve(i);
      s.mat_start[i] = start;
    }
  }
  __syncthreads();
  if (threadIdx.x < kBins) {  // longest tiles first
    int run = 0;
#pragma unroll 16
    for (int b = 0; b < kBins; ++b) run += b > (int)threadIdx.x ? bin_tiles[b] : 0;
    bin_start[threadIdx.x] = run;
    if (threadIdx.x == 0) *s.n_items = run + bin_tiles[0];
  }
  __syncthreads();
  if (once) {
    if (group == 0 && first < batch) s.mat_start[first] = start < 0 ? -1 : bin_start[bin] + start;
  } else {
    for (int i = threadIdx.x; i < batch; i += kPlanThreads) {
      const int off = s.mat_start[i];
      if (off >= 0) s.mat_start[i] = bin_start[s.descs[i].aux] + off;
    }
  }
}

__global__ void fw_expand_kernel(int batch, FwScratch s) {
  pdl_trigger();
  pdl_wait();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= batch) return;
  const int start = s.mat_start[warp];
  if (start < 0) return;
  const MatDesc d = s.descs[warp];
  const int tmx = simt_tiles_m(d.M, c_cfgs[d.cfg]), tnx = simt_tiles_n(d.N, c_cfgs[d.cfg]);
  const int tiles = tmx * tnx;
  for (int t = lane; t < tiles; t += 32)
    s.items[start + t] = TileItem{warp, (uint16_t)(t % tmx), (uint16_t)(t / tmx)};
}

struct FwContext {
  void* mem = nullptr;
  size_t cap_batch = 0;
  size_t cap_items = 0;
  FwScratch s{};
  bool consts = false;
};

std::mutex g_fw_mu;
std::unordered_map<int, FwContext> g_fw;

}  // namespace
}  // namespace bgemm

using namespace bgemm;

extern "C" bgemm_status_t bgemm_framework_gemm(const int* dM, const int* dN, const int* dK,
                                               float* const* dA, float* const* dB,
                                               float* const* dC, const int* dT, int batch,
                                               int max_dim, bgemm_stream_t stream) {
  (void)dT;  // tile choice is this library's own
  if (batch < 0) return set_error(BGEMM_ERROR_INVALID_VALUE, 8, -1, "batch < 0");
  if (batch == 0) return BGEMM_SUCCESS;
  if (!dM) return set_error(BGEMM_ERROR_INVALID_VALUE, 1, -1, "M is NULL");
  if (!dN) return set_error(BGEMM_ERROR_INVALID_VALUE, 2, -1, "N is NULL");
  if (!dK) return set_error(BGEMM_ERROR_INVALID_VALUE, 3, -1, "K is NULL");
  if (!dA) return set_error(BGEMM_ERROR_INVALID_VALUE, 4, -1, "A is NULL");
  if (!dB) return set_error(BGEMM_ERROR_INVALID_VALUE, 5, -1, "B is NULL");
  if (!dC) return set_error(BGEMM_ERROR_INVALID_VALUE, 6, -1, "C is NULL");
  if (max_dim < 1 || max_dim > (1 << 20))
    return set_error(BGEMM_ERROR_INVALID_VALUE, 9, -1, "max_dim = %d not in [1, 2^20]",
                     max_dim);
  DeviceFacts df;
  bgemm_status_t st = device_facts(&df);
  if (st != BGEMM_SUCCESS) return st;

  // worst-case queue: every matrix max_dim x max_dim in 16 x 16 tiles, 8
  // bytes per item (batch = 1024, max_dim = 65536 would be 128 GB)
  const size_t per = (size_t)((max_dim + 15) / 16);
  const size_t need_items = (size_t)batch * per * per;
  if (need_items > (size_t)INT32_MAX)
    return set_error(BGEMM_ERROR_NOT_SUPPORTED, 9, -1,
                     "batch * ceil(max_dim/16)^2 = %zu queue items exceeds 2^31 - 1; pass a "
                     "tighter max_dim",
                     need_items);
  std::lock_guard<std::mutex> lk(g_fw_mu);
  FwContext& ctx = g_fw[df.device];
  if (!ctx.consts) {
    cudaError_t e = cudaMemcpyToSymbol(c_cfgs, kSimtCfgs, sizeof(kSimtCfgs));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_cost, kSimtCost, sizeof(kSimtCost));
    if (e != cudaSuccess) return cuda_error(e, "framework constants");
    ctx.consts = true;
  }
  if ((size_t)batch > ctx.cap_batch || need_items > ctx.cap_items) {
    const size_t cb = std::max((size_t)batch, ctx.cap_batch);
    const size_t ci = std::max(need_items, ctx.cap_items);
    const size_t off_descs = 256;
    const size_t off_start = off_descs + ((sizeof(MatDesc) * cb + 255) & ~size_t(255));
    const size_t off_items = off_start + ((sizeof(int) * cb + 255) & ~size_t(255));
    const size_t total = off_items + sizeof(TileItem) * ci;
    if (ctx.mem) cudaFree(ctx.mem);  // waits for kernels still using it
    ctx.mem = nullptr;
    ctx.cap_batch = ctx.cap_items = 0;
    cudaError_t e = cudaMalloc(&ctx.mem, total);
    if (e != cudaSuccess)
      return set_error(BGEMM_ERROR_ALLOC, 0, -1, "framework queue of %zu bytes: %s", total,
                       cudaGetErrorString(e));
    e = cudaMemset(ctx.mem, 0, 256);
    if (e != cudaSuccess) return cuda_error(e, "framework queue init");
    char* b = static_cast<char*>(ctx.mem);
    ctx.s.err = reinterpret_cast<int*>(b);
    ctx.s.n_items = reinterpret_cast<int*>(b + 4);
    ctx.s.counters = reinterpret_cast<int*>(b + 128);
    ctx.s.descs = reinterpret_cast<MatDesc*>(b + off_descs);
    ctx.s.mat_start = reinterpret_cast<int*>(b + off_start);
    ctx.s.items = reinterpret_cast<TileItem*>(b + off_items);
    ctx.cap_batch = cb;
    ctx.cap_items = ci;
  }
  const int grid = df.num_sms * df.simt_ctas_per_sm;
  fw_plan_kernel<<<1, kPlanThreads, 0, stream>>>(dM, dN, dK, batch, max_dim, grid, ctx.s);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_error(e, "framework plan kernel");
  e = pdl_launch(fw_expand_kernel, (batch + 7) / 8, 256, 0, stream, batch, ctx.s);
  if (e != cudaSuccess) return cuda_error(e, "framework expand kernel");
  SimtParams sp{ctx.s.descs, ctx.s.items, 0, ctx.s.n_items, ctx.s.counters, 1.0f, 1.0f,
                const_cast<const float* const*>(dA), const_cast<const float* const*>(dB), dC};
  e = simt_launch_behind(sp, grid, stream);
  if (e != cudaSuccess) return cuda_error(e, "framework SIMT launch");
  return BGEMM_SUCCESS;
}

namespace bgemm {

// Runs the three launches of the device-queue path on scratch the caller
// provides: `base` holds counters, descriptors, per-matrix queue offsets and
// up to `cap_items` work items for up to `cap_batch` matrices (layout below,
// fw_scratch_bytes gives its size); `err` receives bit 0 for a size that is
// negative or above max_dim.  Allocates nothing.
size_t fw_scratch_bytes(size_t cap_batch, size_t cap_items) {
  const size_t off_descs = 256;
  const size_t off_start = off_descs + ((sizeof(MatDesc) * cap_batch + 255) & ~size_t(255));
  const size_t off_items = off_start + ((sizeof(int) * cap_batch + 255) & ~size_t(255));
  return off_items + sizeof(TileItem) * cap_items;
}

cudaError_t fw_launch_on_scratch(const int* dM, const int* dN, const int* dK, float* const* dA,
                                 float* const* dB, float* const* dC, int batch, int max_dim,
                                 void* base, size_t cap_batch, int* err, int grid,
                                 cudaStream_t stream) {
  const size_t off_descs = 256;
  const size_t off_start = off_descs + ((sizeof(MatDesc) * cap_batch + 255) & ~size_t(255));
  const size_t off_items = off_start + ((sizeof(int) * cap_batch + 255) & ~size_t(255));
  char* b = static_cast<char*>(base);
  FwScratch s;
  s.err = err;
  s.n_items = reinterpret_cast<int*>(b + 4);
  s.counters = reinterpret_cast<int*>(b + 128);
  s.descs = reinterpret_cast<MatDesc*>(b + off_descs);
  s.mat_start = reinterpret_cast<int*>(b + off_start);
  s.items = reinterpret_cast<TileItem*>(b + off_items);
  {
    std::lock_guard<std::mutex> lk(g_fw_mu);
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    FwContext& ctx = g_fw[dev];
    if (!ctx.consts) {
      e = cudaMemcpyToSymbol(c_cfgs, kSimtCfgs, sizeof(kSimtCfgs));
      if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_cost, kSimtCost, sizeof(kSimtCost));
      if (e != cudaSuccess) return e;
      ctx.consts = true;
    }
  }
  fw_plan_kernel<<<1, kPlanThreads, 0, stream>>>(dM, dN, dK, batch, max_dim, grid, s);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  e = pdl_launch(fw_expand_kernel, (batch + 7) / 8, 256, 0, stream, batch, s);
  if (e != cudaSuccess) return e;
  SimtParams sp{s.descs, s.items, 0, s.n_items, s.counters, 1.0f, 1.0f,
                const_cast<const float* const*>(dA), const_cast<const float* const*>(dB), dC};
  return simt_launch_behind(sp, grid, stream);
}

}  // namespace bgemm

extern "C" bgemm_status_t bgemm_framework_release(void) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_error(e, "cudaGetDevice");
  {
    std::lock_guard<std::mutex> lk(g_fw_mu);
    auto it = g_fw.find(dev);
    if (it != g_fw.end() && it->second.mem) {
      e = cudaFree(it->second.mem);  // waits for kernels still using it
      it->second.mem = nullptr;
      it->second.cap_batch = it->second.cap_items = 0;
      if (e != cudaSuccess) return cuda_error(e, "framework scratch release");
    }
  }
  return fwtc_release(dev);
}

extern "C" bgemm_status_t bgemm_framework_check_device(bgemm_stream_t stream) {
  int dev = 0;
  cudaGetDevice(&dev);
  cudaError_t e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return cuda_error(e, "cudaStreamSynchronize");
  bgemm_status_t st = fwtc_check_device(dev);
  if (st != BGEMM_SUCCESS) return st;
  std::lock_guard<std::mutex> lk(g_fw_mu);
  auto it = g_fw.find(dev);
  if (it == g_fw.end() || !it->second.mem) return BGEMM_SUCCESS;
  int err = 0;
  e = cudaMemcpy(&err, it->second.s.err, sizeof(int), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return cuda_error(e, "framework error word");
  if (err) {
    cudaMemset(it->second.s.err, 0, sizeof(int));
    return set_error(BGEMM_ERROR_INVALID_VALUE, 1, -1,
                     "a matrix size was negative or above max_dim; such matrices were skipped");
  }
  return BGEMM_SUCCESS;
}

// Host replay of fw_plan_kernel + fw_expand_kernel (tests without a GPU): the
// same per-matrix choices and rebalance rounds, reserved in matrix order
// instead of by atomics; `slots` is the persistent SIMT grid the entry uses.
extern "C" int bgemm_debug_framework_plan(const int* M, const int* N, const int* K, int batch,
                                          int max_dim, int slots, int* cfg_out, int* items_out,
                                          int max_items, int* err) {
  if (batch < 0 || !err || slots < 1 || (batch > 0 && (!M || !N || !K))) return -1;
  std::vector<int> cfg(batch, -1);
  std::vector<int> start(batch, -1);
  std::vector<int> bin(batch, 0);
  std::vector<SimtCands> cand(batch);
  int bin_tiles[kBins] = {};
  long long work[kSimtSteps + 1] = {};
  float longest[kSimtSteps + 1] = {};
  *err = 0;
  auto any = [&](int i) { return !fw_bad(M[i], N[i], K[i], max_dim) && M[i] > 0 && N[i] > 0; };
  for (int i = 0; i < batch; ++i) {
    if (fw_bad(M[i], N[i], K[i], max_dim)) *err |= 1;
    if (any(i)) simt_cands(M[i], N[i], K[i], -1, &cand[i]);
  }
  for (int j = 0; j <= kSimtSteps; ++j)
    for (int i = 0; i < batch; ++i) {
      float w, l;
      if (!any(i) ||
          simt_pick(cand[i], j == 0 ? 3e38f : simt_limit(longest[0], j), &w, &l) < 0)
        continue;
      work[j] += (long long)w;
      longest[j] = std::max(longest[j], l);
    }
  const float limit = simt_choose_limit(work, longest, slots);
  for (int i = 0; i < batch; ++i) {
    float w, l;
    if (any(i)) cfg[i] = simt_pick(cand[i], limit, &w, &l);
    if (cfg_out) cfg_out[i] = cfg[i];
    if (cfg[i] < 0) continue;
    bin[i] = fw_bin(K[i], kSimtCost[cfg[i]]);
    start[i] = bin_tiles[bin[i]];
    bin_tiles[bin[i]] += (int)simt_tiles(M[i], N[i], kSimtCfgs[cfg[i]]);
  }
  int bin_start[kBins], n = 0;
  for (int b = kBins - 1; b >= 0; --b) {
    bin_start[b] = n;
    n += bin_tiles[b];
  }
  if (items_out && n > max_items) return -1;
  for (int i = 0; items_out && i < batch; ++i) {
    if (start[i] < 0) continue;
    const int tmx = (M[i] + kSimtCfgs[cfg[i]].bm - 1) / kSimtCfgs[cfg[i]].bm;
    const int tnx = (N[i] + kSimtCfgs[cfg[i]].bn - 1) / kSimtCfgs[cfg[i]].bn;
    const int s0 = bin_start[bin[i]] + start[i];
    for (int t = 0; t < tmx * tnx; ++t) {
      items_out[3 * (s0 + t)] = i;
      items_out[3 * (s0 + t) + 1] = t % tmx;
      items_out[3 * (s0 + t) + 2] = t / tmx;
    }
  }
  return n;
}
