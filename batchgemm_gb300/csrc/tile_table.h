// tile_table.h -- per-tile cost model consumed by the planners.
//
// Time of one work item of configuration c on a matrix with inner dimension
// K is modelled as  t = a_c + b_c * K  (nanoseconds for the CTA -- or CTA
// pair -- that runs it, with every other persistent CTA busy too).  The
// planner picks, per matrix, the configuration with the least total time and
// then splits the largest tiles until no single tile is longer than the
// average load of one persistent CTA (the parallelism rebalance).
//
// tile_table_tuned.inc, written by batchgemm_gb300/autotune.py from
// measurements on the GPU, replaces the defaults below when present.
#pragma once
#include <math.h>

#include <utility>

#include "bgemm_internal.h"

namespace bgemm {

struct TileCost {
  float a_ns;  // fixed cost per tile (prologue, epilogue, latency)
  float b_ns;  // cost per unit of K
};

// Tensor-core cost tables are indexed [mode - 1][cfg]: TF32, TF32X3, BF16X3;
// cfg 0..7 one-SM tiles, 8..15 CTA-pair tiles.  b = 0 marks a configuration
// the mode does not run.
#if defined(BGEMM_HAVE_TUNED_TABLE)
#include "tile_table_tuned.inc"
#else
// Defaults from a first-principles model.  SIMT: 2 CTAs per SM share 128
// FP32 lanes at ~1.9 GHz, b = BM*BN / (64 lanes * 1.9 GHz) / efficiency.
constexpr TileCost kSimtCost[10] = {
    {1500.f, 16 * 16 / 64 / 1.9f / 0.20f},    {1600.f, 32 * 32 / 64 / 1.9f / 0.45f},
    {1700.f, 64 * 32 / 64 / 1.9f / 0.60f},    {1700.f, 32 * 64 / 64 / 1.9f / 0.60f},
    {1800.f, 64 * 64 / 64 / 1.9f / 0.70f},    {2000.f, 128 * 64 / 64 / 1.9f / 0.80f},
    {2000.f, 64 * 128 / 64 / 1.9f / 0.80f},   {2200.f, 128 * 128 / 64 / 1.9f / 0.85f},
    {1600.f, 8 * 128 / 64 / 1.9f / 0.45f},    {1600.f, 128 * 8 / 64 / 1.9f / 0.45f},
};
// Tensor cores: per 128-byte K slice a tile streams its operands from L2,
// which bounds the narrow tiles, so a tile costs at least what a 128-wide
// (one SM) or 256-wide (pair) tile costs for the same K.  TF32 runs 4096
// flops/clk/SM (BF16 8192) at ~1.9 GHz.
#define BGEMM_TC1(bn, prod, rate) {1500.f, 2.f * 128 * ((bn) > 128 ? (bn) : 128) * (prod) / (rate)}
#define BGEMM_TC2(bn, prod, rate) {2500.f, 2.f * 256 * (0.6f * 256 + 0.4f * (bn)) * (prod) / (2 * (rate))}
#define BGEMM_TC_ROW(prod, rate, pairs)                                                          \
  {BGEMM_TC1(16, prod, rate), BGEMM_TC1(32, prod, rate), BGEMM_TC1(64, prod, rate),             \
   BGEMM_TC1(128, prod, rate), BGEMM_TC1(16, prod, rate), BGEMM_TC1(32, prod, rate),            \
   BGEMM_TC1(64, prod, rate), BGEMM_TC1(128, prod, rate),                                        \
   pairs ? TileCost BGEMM_TC2(64, prod, rate) : TileCost{0.f, 0.f},                              \
   pairs ? TileCost BGEMM_TC2(128, prod, rate) : TileCost{0.f, 0.f},                             \
   pairs ? TileCost BGEMM_TC2(256, prod, rate) : TileCost{0.f, 0.f}, TileCost{0.f, 0.f},         \
   pairs ? TileCost BGEMM_TC2(64, prod, rate) : TileCost{0.f, 0.f},                              \
   pairs ? TileCost BGEMM_TC2(128, prod, rate) : TileCost{0.f, 0.f},                             \
   pairs ? TileCost BGEMM_TC2(256, prod, rate) : TileCost{0.f, 0.f}, TileCost{0.f, 0.f}}
constexpr TileCost kTcCost[3][16] = {
    BGEMM_TC_ROW(1, 7782.f, false),
    BGEMM_TC_ROW(3, 7782.f, true),
    BGEMM_TC_ROW(3, 15564.f, true),
};
#undef BGEMM_TC_ROW
#undef BGEMM_TC2
#undef BGEMM_TC1
#endif

// Promotion schedule of the split tensor-core modes on CTA pairs, indexed
// [mode - 1][bucket of K] (see TcSchedule in tc_common.h): 128-byte K slices
// per promotion group, 0 = promote every MMA of K and keep lo*lo.  The
// single-product TF32 row is unused.  Defaults: the small-K path up to
// K = 64, groups of two slices above; the autotuner replaces them with the
// fastest groups whose error against FP64 stays within the FP32 SIMT path's.
#if !defined(BGEMM_TUNED_HAS_SCHEDULE)
constexpr unsigned char kTcGroupTable[3][8] = {
    {0, 2, 2, 2, 2, 2, 2, 2}, {0, 2, 2, 2, 2, 2, 2, 2}, {0, 2, 2, 2, 2, 2, 2, 2}};
#endif

// Compile-time schedule parameters, swept by the autotuner with a rebuild per
// candidate:
//   kSimtRingCap      cp.async ring stages of a SIMT tile: a tile takes as
//                     many 16-k stages as the CTA's shared memory holds, up
//                     to this cap (the 128 x 128 tile always has 4);
//   kTcCPrefetchLead  beta != 0: promotion groups before the end of a pair
//                     tile at which its C lines are prefetched into L2 (0:
//                     none; the epilogue's pipelined reads then go to HBM).
#if !defined(BGEMM_TUNED_HAS_BUILD_PARAMS)
constexpr int kSimtRingCap = 4;
constexpr int kTcCPrefetchLead = 0;
#endif

// ------------------------------------------------- SIMT planning model --
// Shared by the host planner, the device planner and its host replay, which
// decide alike: single precision with explicit fmaf, work summed as whole
// nanoseconds.
//
// For each matrix the configuration with the least work (modelled time on the
// CTAs) among those whose single tile takes no longer than a limit T, with T
// chosen for the batch: the makespan is modelled as the average load of a
// persistent CTA plus the longest tile (kSimtTail of it), and T runs down from
// the longest tile of the unlimited choice in steps of sqrt(2).
constexpr float kSimtTail = 1.0f;     // share of kSimtTailNs that counts
// time per k that a skipped edge saves (125 batches: with 0 1.005 times as long
// as with 0.35 in the geometric mean, one 1.10; 0.2 1.001; 0.6 1.003, one 1.47)
constexpr float kSimtFma = 0.35f;
constexpr int kSimtSteps = 12;

// (bm, bn, gm and gn are powers of two; unsigned, since sizes go up to the
// largest int and simt_fits has to refuse those)
__host__ __device__ inline int simt_tiles_m(int M, SimtCfg g) {
  return (int)(((unsigned)M + (unsigned)(g.bm - 1)) >> g.lm);
}
__host__ __device__ inline int simt_tiles_n(int N, SimtCfg g) {
  return (int)(((unsigned)N + (unsigned)(g.bn - 1)) >> g.ln);
}
__host__ __device__ inline bool simt_fits(int M, int N, SimtCfg g) {
  // TileItem holds 16-bit tile coordinates
  return simt_tiles_m(M, g) <= 65535 && simt_tiles_n(N, g) <= 65535;
}
__host__ __device__ inline long long simt_tiles(int M, int N, SimtCfg g) {
  return (long long)simt_tiles_m(M, g) * simt_tiles_n(N, g);
}
// One full tile's share of a CTA's time.
__host__ __device__ inline float simt_tile_ns(int K, TileCost t) {
  return fmaf(t.b_ns, (float)K, t.a_ns);
}
// What the longest tile adds to the makespan: about the time that it takes
// beside few others, as those of a short queue and the last ones of a long one
// do.  (With an SM to itself, K of 64 to 4096, the mean over aligned and odd
// leading dimensions and every storage: 16.0, 35.3, 97, 22.5 and 20.5 ns per k
// for ids 0, 1, 7, 8, 9.  125 batches of 1 to 2000 matrices of sizes up to
// 2000, against one build's times, with 25, 45 and 120 for the first three
// 0.922 in the geometric mean, with 36, 51 and 126 0.927.  Id 0 has its own 16
// since it takes slices of 32 k at any K: 149 batches of up to 4 GFLOP 0.975
// against 25; a first part of 1500 ns instead 0.970, but 1.24 and 1.11 on two
// of the uniform ones, of 2200 0.995.  Ids 2 to 6, which are only forced, have
// theirs alone.)
constexpr TileCost kSimtTailNs[kSimtNumCfgs] = {
    {1900.0f, 16.0f}, {2400.0f, 45.0f}, {2100.0f, 30.0f}, {2100.0f, 30.0f}, {2700.0f, 45.0f},
    {3400.0f, 70.0f}, {3400.0f, 70.0f}, {3664.0f, 120.0f}, {2400.0f, 22.5f}, {2100.0f, 20.5f}};
// All tiles of a matrix.  A ragged edge's FMAs are skipped in steps of gm x gn
// outputs, its copies are not.
__host__ __device__ inline float simt_work_ns(int M, int N, int K, SimtCfg g, TileCost t) {
  const float tiles = (float)simt_tiles(M, N, g);
  const float done = (float)((M + g.gm - 1) & -g.gm) * (float)((N + g.gn - 1) & -g.gn);
  const float part = done / (tiles * (float)(g.bm * g.bn));
  return fmaf(t.b_ns * tiles * fmaf(kSimtFma, part, 1.0f - kSimtFma), (float)K, t.a_ns * tiles);
}
// The candidates of one matrix (M, N > 0); lat < 0: not one.
struct SimtCands {
  float work[kSimtNumCfgs], lat[kSimtNumCfgs];
};
template <int C>
__host__ __device__ inline void simt_cand(int M, int N, int K, int force, SimtCands* e) {
  constexpr SimtCfg g = kSimtCfgs[C];
  constexpr TileCost t = kSimtCost[C];
  e->work[C] = 0.0f;
  e->lat[C] = -1.0f;
  if ((force >= 0 ? C != force : !simt_auto_cfg(C, M, N)) || !simt_fits(M, N, g)) return;
  e->work[C] = simt_work_ns(M, N, K, g, t);
  e->lat[C] = simt_tile_ns(K, kSimtTailNs[C]);
}
template <int... C>
__host__ __device__ inline void simt_cands_of(std::integer_sequence<int, C...>, int M, int N,
                                              int K, int force, SimtCands* e) {
  (simt_cand<C>(M, N, K, force, e), ...);
}
__host__ __device__ inline void simt_cands(int M, int N, int K, int force, SimtCands* e) {
  simt_cands_of(std::make_integer_sequence<int, kSimtNumCfgs>{}, M, N, K, force, e);
}
// Least work with a tile of at most T, or else the shortest tile (-1: none).
__host__ __device__ inline int simt_pick(const SimtCands& e, float T, float* work, float* lat) {
  int best = -1, any = -1;
  float bw = 0.0f, bl = 0.0f, sl = 0.0f, sw = 0.0f;
#pragma unroll
  for (int c = kSimtNumCfgs - 1; c >= 0; --c) {
    if (e.lat[c] < 0.0f) continue;
    if (any < 0 || e.lat[c] < sl) {
      any = c;
      sl = e.lat[c];
      sw = e.work[c];
    }
    if (e.lat[c] <= T && (best < 0 || e.work[c] < bw)) {
      best = c;
      bw = e.work[c];
      bl = e.lat[c];
    }
  }
  *work = best >= 0 ? bw : sw;
  *lat = best >= 0 ? bl : sl;
  return best >= 0 ? best : any;
}
// The limit of step j > 0, from the longest tile of step 0 (which has none).
__host__ __device__ inline float simt_limit(float longest, int step) {
  float t = longest;
  for (int j = 0; j < step; ++j) t *= 0.70710678f;
  return t;
}
// The modelled makespan of a step on `slots` CTAs from its sums, and T from
// every step's.
__host__ __device__ inline float simt_makespan(long long work, float longest, int slots) {
  return fmaf(kSimtTail, longest, (float)work / (float)slots);
}
__host__ __device__ inline float simt_choose_limit(const float* makespan, float longest) {
  float best = 0.0f, limit = longest, T = 3e38f;  // limit: step j - 1's
  for (int j = 0; j <= kSimtSteps; ++j) {
    if (j > 0 && kSimtTail * limit <= 0.02f * best) break;
    if (j > 0) limit *= 0.70710678f;
    if (j == 0 || makespan[j] < best) {
      best = makespan[j];
      T = j == 0 ? 3e38f : limit;
    }
  }
  return T;
}

inline float simt_choose_limit(const long long* work, const float* longest, int slots) {
  float makespan[kSimtSteps + 1];
  for (int j = 0; j <= kSimtSteps; ++j) makespan[j] = simt_makespan(work[j], longest[j], slots);
  return simt_choose_limit(makespan, longest[0]);
}

}  // namespace bgemm
