// simt_tile.h -- the persistent FP32 SIMT kernel (simt_kernel.cu): operand
// staging, the FMA loop, the C read and write, and how a CTA's warps share
// the tile queue.
//
// A tile is computed by a team: one warp for the 16 x 16 and 32 x 32 tiles, so
// that a small tile still gives every thread 8 to 32 outputs and eight tiles
// run side by side in a CTA, the whole CTA (256 threads) for all others.  A
// warp's lanes form an LX x LY grid and each thread owns TM x TN outputs.  The
// thin tiles (8 x 128, 128 x 8) are bound by the bytes they read for a few
// FMAs each: all eight warps share one tile's long operand, in slices of 32 k,
// so that a CTA keeps 55 KB on the way and a long K ends soon (run_thin).
// Operands stream through a cp.async ring of BK k-slices:
//   A slice: [k][BM]      rows contiguous, 16-byte cp.async when lda % 4 == 0
//                         and A is 16-byte aligned, 4-byte otherwise
//   B slice: [n][BK + 4]  k contiguous, as B is stored: 16-byte cp.async on
//                         the same condition; rows of BK + 4 floats (20 or 36)
//                         put the float4 reads of eight lanes on distinct banks
//                         (the 128 x 128 tile: [k][BN + 4])
// An operand stored the other way round from its slice (A as K x M) is
// transposed by 4-byte copies; B as N x K is staged as [k][BN + 4].  Edges are
// zero-filled by the cp.async source size, so any M, N, K >= 0 and any leading
// dimension work.
//
// Every output element is a single fma chain over k in order (bit-exact with
// the reference's tile bodies, CUDA/framework/kernel_128_new.h,
// kernel_256_new.h, CUDA/batching/kernel_256.h, and with the oracle).  Two
// rows' chains run in one packed fma.rn.f32x2: the FP32 pipe does the same 128
// FMAs per SM and clock, but half the issue slots stay free for the fragment
// loads and copies.
//
// The code is kept short on purpose: loops over copies, k and C are rolled.
// A batch of small tiles runs each shape's code only a few times in a row,
// and with every loop unrolled (ten shapes, each about 25 KB) the warps waited
// for instructions more than for anything else: config "256 matrices of 16 to
// 256" took 138 us unrolled.
#pragma once
#include <stdint.h>

#include "bgemm_internal.h"
#include "tile_table.h"

namespace bgemm {
namespace simt {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
// Shared memory of a CTA: 14 KB per warp, so that two CTAs share an SM's
// 227 KB; a warp's tile uses its own 14 KB, a CTA tile all of it.
constexpr int kWarpFloats = 3584;
// Behind it the CTA's control words: the item of the next round, the number of
// CTA tiles that warps left, those tiles, and which warp pulls first.
constexpr int kCtlItem = 0, kCtlPosts = 1, kCtlPost = 2, kCtlTurn = 10, kCtlInts = 16;
static_assert(kCtlPost + kWarps <= kCtlTurn, "control words");
constexpr int kSmemBytes = kWarps * kWarpFloats * 4 + kCtlInts * 4;
static_assert(kSimtRingCap >= 2 && kSimtRingCap <= 32, "SIMT ring cap out of range");

// A pair of FP32 values in one 64-bit register pair (low half first).
using f32x2 = unsigned long long;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// src_bytes of 0 reads nothing from src and writes zeros.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src),
               "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, int src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src),
               "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ void fma2(f32x2& d, f32x2 a, f32x2 b) {
  asm volatile("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ bool vec16(const float* X, int ldx) {
  return ((reinterpret_cast<uintptr_t>(X) & 15u) == 0) && ((ldx & 3) == 0);
}

// The thread index, read anew: the compiler would otherwise compute every
// shape's thread coordinates and shared-memory addresses once, ahead of the
// persistent loop, and spill them there.
__device__ __forceinline__ int thread_index() {
  int t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}

// Tile shape, ring geometry and index maps of a team of WM x WN warps, each of
// LX x (32 / LX) lanes.  TA / TB: A stored K x M, B stored N x K.  CT: the tile
// is computed as C^T = B^T A^T, that is, all of the below is said of B^T, A^T
// and C^T.  SHIFT: B's slice holds each row from the 16-byte boundary before it.
template <int WM_, int WN_, int LX_, int TM_, int TN_, bool TA_, bool TB_, int BK_ = 0,
          bool CT_ = false, bool SHIFT_ = false>
struct Shape {
  static constexpr int WM = WM_, WN = WN_, LX = LX_, TM = TM_, TN = TN_;
  static constexpr bool TA = TA_, TB = TB_, CT = CT_, SHIFT = SHIFT_;
  static constexpr int NT = 32 * WM * WN, LY = 32 / LX;
  static constexpr int WBM = LX * TM, WBN = LY * TN;  // a warp's part of the tile
  static constexpr int BM = WM * WBM, BN = WN * WBN;
  static_assert(NT == 32 || NT == kThreads, "a team is a warp or the CTA");
  static_assert(TM % 4 == 0 && (TN % 4 == 0 || TN <= 2), "register tile");
  static_assert(!SHIFT || (TN == 1 && !TB), "one offset per thread");
  static constexpr int kBudget = NT == 32 ? kWarpFloats : kWarps * kWarpFloats;
  // B's slice by rows of n (else of k): as an N x K operand is stored, and
  // wherever 64 accumulators leave no registers for fragments of several k
  static constexpr bool BROWS = TB || TM * TN >= 64;
  static constexpr int LDA = TA ? BM + 4 : BM;
  static constexpr int stage(int bk) {
    return bk * LDA + (BROWS ? bk * (BN + 4) : BN * (bk + 4));
  }
  static constexpr int BK = BK_ ? BK_ : 16;
  static constexpr int LDB = BROWS ? BN + 4 : BK + 4;
  static constexpr int A_STAGE = BK * LDA;
  static constexpr int STAGE = stage(BK);
  // A warp's part of C is staged as WBN columns of LDC floats behind the ring
  // stages that the prologue fills.
  static constexpr int LDC = WBM + 4;
  static constexpr int C_ALL = WBN * LDC * (NT / 32);
  static constexpr int fit(int ns) {
    return (ns - 1) * STAGE + (C_ALL > STAGE ? C_ALL : STAGE) <= kBudget ? ns : fit(ns - 1);
  }
  static constexpr int NS = fit(kSimtRingCap);
  static_assert(NS >= 2 && STAGE % 4 == 0 && A_STAGE % 4 == 0, "ring geometry");
  // (fragments are read up to one k behind a slice)
  static_assert((NS - 1) * STAGE + A_STAGE + LDA <= kBudget && NS * STAGE + LDB <= kBudget,
                "reads ahead");

  // A lane's place in the grid: eight consecutive lanes take 4 x 2 places, so
  // that a 16-byte fragment read moves 64 and 32 distinct bytes per quarter
  // warp and two quarters share a shared-memory wavefront (lane % LX gives 128
  // bytes of A per quarter and four wavefronts a read).
  static __device__ __forceinline__ int lane_x(int lane) {
    if constexpr (LX == 8) return (lane & 1) | ((lane >> 1) & 6);
    if constexpr (LX == 4) return (lane & 1) | ((lane >> 1) & 2);
    return lane % LX;
  }
  static __device__ __forceinline__ int lane_y(int lane) {
    if constexpr (LX == 8) return ((lane >> 1) & 1) | ((lane >> 3) & 2);
    if constexpr (LX == 4) return ((lane >> 1) & 1) | ((lane >> 2) & 6);
    return lane / LX;
  }
  // column of the warp's part that lane row ly holds as its j-th
  static __device__ __forceinline__ int n_of(int ly, int j) {
    if constexpr (!BROWS) return j * LY + ly;
    if constexpr (TN <= 2) return ly * TN + j;
    return (j / 4) * (LY * 4) + ly * 4 + j % 4;
  }
  static __device__ __forceinline__ void sync() {
    if constexpr (NT == 32)
      __syncwarp();
    else
      __syncthreads();
  }
};

// N copies of BYTES (16 or 4) per thread, copy i from src + i * step * ld to
// dst + i * DSTEP bytes.  `bytes` of each are read (the rest zero-filled), of
// the copies from `left` on (counted in units of `unit` per copy) none; FULL:
// there are no such copies.  Blocks of 16 (the whole, or half of the thin tiles' long
// slices) took the 2048-matrix batch from 2.78 ms, in blocks of four, to 2.59.
template <int BYTES, int N, int STEP, int DSTEP, int UNIT, bool FULL>
__device__ __forceinline__ void copy_run(uint32_t dst, const float* src, int ld, int bytes,
                                         int left) {
  constexpr int U = N < 16 ? N : 16;
  static_assert(N % U == 0, "copies in blocks");
#pragma unroll 1
  for (int i0 = 0; i0 < N; i0 += U) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const float* q = src + (long long)ld * (u * STEP);
      const int b = FULL || u * UNIT < left ? bytes : 0;
      if constexpr (BYTES == 16)
        cp_async16(dst + u * DSTEP, q, b);
      else
        cp_async4(dst + u * DSTEP, q, b);
    }
    src += (long long)ld * (U * STEP);
    dst += U * DSTEP;
    left -= U * UNIT;
  }
}
template <int BYTES, int N, int STEP, int DSTEP, int UNIT>
__device__ __forceinline__ void copies(uint32_t dst, const float* src, int ld, int bytes, int left,
                                       bool full) {
  if (full)
    copy_run<BYTES, N, STEP, DSTEP, UNIT, true>(dst, src, ld, bytes, left);
  else
    copy_run<BYTES, N, STEP, DSTEP, UNIT, false>(dst, src, ld, bytes, left);
}

// BK k-slices of R operand rows into s[k][LDS] when element (r, k) sits at
// X[r + k*ldx] (rows contiguous), X being the tile's first row at the slices'
// first k.  Elements beyond `rows` and `ks` are zero-filled.  Each thread
// keeps one row position (or one per NT rows) and walks k.
template <int NT, int R, int LDS, int BK>
__device__ __forceinline__ void load_rows_contig(const float* X, int ldx, int rows, int ks,
                                                 float* s, bool vec, int tid) {
  const bool full = ks >= BK;
  if (vec) {
    constexpr int RC = R / 4;  // 16-byte chunks per k
    static_assert(NT % RC == 0, "one row position per thread");
    constexpr int KS = NT / RC;
    const int rr = (tid % RC) * 4, kk0 = tid / RC;
    const int valid = min(max(rows - rr, 0), 4) * 4;
    const float* src = X + (long long)kk0 * ldx + rr;
    const uint32_t dst = smem_u32(s + kk0 * LDS + rr);
    if (BK % KS == 0 || kk0 < BK)
      copies<16, (BK + KS - 1) / KS, KS, KS * LDS * 4, KS>(dst, src, ldx, valid, ks - kk0, full);
  } else {
    static_assert(NT >= R, "one row position per thread");
    constexpr int KS = NT / R;
    const int rr = tid % R, kk0 = tid / R;
    const float* src = X + (long long)kk0 * ldx + rr;
    const uint32_t dst = smem_u32(s + kk0 * LDS + rr);
    if (BK % KS == 0 || kk0 < BK)
      copies<4, (BK + KS - 1) / KS, KS, KS * LDS * 4, KS>(dst, src, ldx, rr < rows ? 4 : 0,
                                                          ks - kk0, full);
  }
}

// The same slices when element (r, k) sits at X[k + r*ldx] (k contiguous),
// into s[r][LDS], or transposed into s[k][LDS] (SCATTER: 4-byte copies only).
// Each thread keeps one k position and walks the rows.
template <int NT, int R, int LDS, int BK, bool SCATTER>
__device__ __forceinline__ void load_k_contig(const float* X, int ldx, int rows, int ks, float* s,
                                              bool vec, int tid) {
  const bool full = rows >= R;
  if (vec && !SCATTER) {
    constexpr int KC = BK / 4, RS = NT / KC;
    const int kq = (tid % KC) * 4, rr0 = tid / KC;
    const int valid = min(max(ks - kq, 0), 4) * 4;
    const float* src = X + (long long)rr0 * ldx + kq;
    const uint32_t dst = smem_u32(s + rr0 * LDS + kq);
    if (R % RS == 0 || rr0 < R)
      copies<16, (R + RS - 1) / RS, RS, RS * LDS * 4, RS>(dst, src, ldx, valid, rows - rr0, full);
  } else {
    constexpr int RS = NT / BK;
    const int kk = tid % BK, rr0 = tid / BK;
    const float* src = X + (long long)rr0 * ldx + kk;
    const uint32_t dst = smem_u32(SCATTER ? s + kk * LDS + rr0 : s + rr0 * LDS + kk);
    constexpr int DR = (SCATTER ? 1 : LDS) * 4;  // bytes from row to row
    if (R % RS == 0 || rr0 < R)
      copies<4, (R + RS - 1) / RS, RS, RS * DR, RS>(dst, src, ldx, kk < ks ? 4 : 0, rows - rr0,
                                                    full);
  }
}

// Floats from the 16-byte boundary at or before X to X.
__device__ __forceinline__ int floats_off(const float* X) {
  return (int)(reinterpret_cast<uintptr_t>(X) >> 2) & 3;
}
// The same slices, k contiguous, rows that start anywhere: 16-byte copies from
// the boundary at or before each row's k on, so that s[r][LDS] holds the slice
// from float floats_off(row) on.  What lies before the row's first element
// (`first`: the slices start there) and behind its last is not read.
template <int NT, int R, int LDS, int BK>
__device__ __forceinline__ void load_k_shifted(const float* X, int ldx, int rows, int ks, float* s,
                                               bool first, int tid) {
  constexpr int KC = BK / 4, RS = NT / KC;  // chunks of a row, the last one apart
  static_assert(LDS >= BK + 4 && R % RS == 0 && RS % 4 == 0 && R <= NT, "chunks");
  const int c = tid % KC, rr0 = tid / KC;
  const float* row = X + (long long)rr0 * ldx;
  const int off = floats_off(row);  // that of every RS-th row
  const uint32_t dst = smem_u32(s + rr0 * LDS + c * 4);
  if (first && c == 0 && off > 0) {
#pragma unroll 1
    for (int r = 0; r < R; r += RS)
      for (int q = off; q < 4; ++q)
        cp_async4(dst + (r * LDS + q) * 4, row + (long long)r * ldx + (q - off),
                  rr0 + r < rows && q - off < ks ? 4 : 0);
  } else {
    copies<16, R / RS, RS, RS * LDS * 4, RS>(dst, row - off + c * 4, ldx,
                                             min(max(ks + off - c * 4, 0), 4) * 4, rows - rr0,
                                             rows >= R);
  }
  if (tid < R) {
    const float* last = X + (long long)tid * ldx;
    const int o = floats_off(last);
    if (o > 0)
      cp_async16(smem_u32(s + tid * LDS + BK), last - o + BK,
                 tid < rows ? min(max(ks + o - BK, 0), 4) * 4 : 0);
  }
}

// One k of the register tile's first HM * 4 rows and NJ columns: the row pair
// stays the operand of NJ FMAs in a row and the columns run back and forth, so
// that consecutive FMAs share register operands (measured on FFMA2 alone,
// 8 x 8: 123 of 128 FMAs per SM and clock in this order, 109 column by column).
template <int HM, int NJ, int TM, int TN>
__device__ __forceinline__ void fma_tile(const f32x2 (&a)[TM / 2], const float (&b)[TN],
                                         f32x2 (&acc)[TM / 2][TN]) {
  f32x2 bb[NJ];
#pragma unroll
  for (int j = 0; j < NJ; ++j) bb[j] = pack2(b[j], b[j]);
#pragma unroll
  for (int i = 0; i < 2 * HM; ++i)
#pragma unroll
    for (int q = 0; q < NJ; ++q) {
      const int j = (i & 1) ? NJ - 1 - q : q;
      fma2(acc[i][j], a[i], bb[j]);
    }
}

// acc += A slice * B slice, k in order, for the first HM of the TM / 4 row
// groups and NJ of the TN columns a thread owns; sA and sB are at the thread's
// first row and column (SHIFT: sB at the boundary `off` floats before it).
template <class S, int HM, int NJ>
__device__ __forceinline__ void compute_part(const float* sA, const float* sB, int off, int ks,
                                             f32x2 (&acc)[S::TM / 2][S::TN]) {
  constexpr int TM = S::TM, TN = S::TN;
  // long slices end with the matrix's K, rounded up to 4
  constexpr bool kLong = S::BK > 16;
  const int k_end = kLong ? min(S::BK, (ks + 3) & ~3) : S::BK;
  auto load_a = [&](int k, f32x2(&a)[TM / 2]) {
#pragma unroll
    for (int h = 0; h < HM; ++h) {
      const ulonglong2 v =
          *reinterpret_cast<const ulonglong2*>(sA + k * S::LDA + h * (S::LX * 4));
      a[2 * h] = v.x;
      a[2 * h + 1] = v.y;
    }
  };
  constexpr int UN = kLong ? 2 : S::BK / 4;
  if constexpr (!S::BROWS) {
    float4 ahead;
    if constexpr (S::SHIFT) ahead = *reinterpret_cast<const float4*>(sB);
#pragma unroll UN
    for (int kq = 0; kq < k_end; kq += 4) {
      float b[4][TN];
      if constexpr (S::SHIFT) {
        // eight floats in two aligned reads, the row's four by selects (four
        // 4-byte reads of 16 lanes' rows would take eight wavefronts, not two)
        const float4 u = ahead;
        ahead = *reinterpret_cast<const float4*>(sB + kq + 4);
        const bool two = (off & 2) != 0, one = (off & 1) != 0;
        const float t0 = two ? u.z : u.x, t1 = two ? u.w : u.y, t2 = two ? ahead.x : u.z;
        const float t3 = two ? ahead.y : u.w, t4 = two ? ahead.z : ahead.x;
        b[0][0] = one ? t1 : t0; b[1][0] = one ? t2 : t1;
        b[2][0] = one ? t3 : t2; b[3][0] = one ? t4 : t3;
      } else {
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          const float4 v = *reinterpret_cast<const float4*>(sB + j * S::LY * S::LDB + kq);
          b[0][j] = v.x; b[1][j] = v.y; b[2][j] = v.z; b[3][j] = v.w;
        }
      }
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        f32x2 a[TM / 2];
        load_a(kq + kk, a);
        fma_tile<HM, NJ, TM, TN>(a, b[kk], acc);
      }
    }
  } else {
    auto load_b = [&](int k, float(&b)[TN]) {
      if constexpr (TN == 1) {
        b[0] = sB[k * S::LDB];
      } else if constexpr (TN == 2) {
        const float2 v = *reinterpret_cast<const float2*>(sB + k * S::LDB);
        b[0] = v.x; b[1] = v.y;
      } else {
#pragma unroll
        for (int h = 0; h < NJ / 4; ++h) {
          const float4 v = *reinterpret_cast<const float4*>(sB + k * S::LDB + h * (S::LY * 4));
          b[4 * h] = v.x; b[4 * h + 1] = v.y; b[4 * h + 2] = v.z; b[4 * h + 3] = v.w;
        }
      }
    };
    // the fragments of the next k are read while this one's FMAs run (those of
    // the row behind the last are never used)
    f32x2 a[2][TM / 2];
    float b[2][TN];
    load_a(0, a[0]);
    load_b(0, b[0]);
#pragma unroll UN
    for (int kq = 0; kq < k_end; kq += 4) {
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        load_a(kq + kk + 1, a[(kk + 1) & 1]);
        load_b(kq + kk + 1, b[(kk + 1) & 1]);
        fma_tile<HM, NJ, TM, TN>(a[kk & 1], b[kk & 1], acc);
      }
    }
  }
}

// The part of the register tile that a ragged edge leaves: half the rows and
// half the columns are skipped where they are all outside the matrix, and the
// whole where nothing is inside (mrem and nrem: rows and columns left from the
// warp's first on; ks: k left).  A skipped FMA's issue slots go to the SM's
// other warps.
template <class S>
__device__ __forceinline__ void compute_stage(const float* sA, const float* sB, int off, int mrem,
                                              int nrem, int ks,
                                              f32x2 (&acc)[S::TM / 2][S::TN]) {
  constexpr int HM = S::TM / 4, TN = S::TN;
  if (mrem <= 0 || nrem <= 0) return;
  const bool half_m = HM == 2 && mrem <= S::LX * 4;
  constexpr bool kHalfN = S::BROWS ? TN == 8 : TN >= 2;
  const bool half_n = kHalfN && nrem <= S::WBN / 2;
  if (!half_m && !half_n)
    compute_part<S, HM, TN>(sA, sB, off, ks, acc);
  else if (!half_m)
    compute_part<S, HM, kHalfN ? TN / 2 : TN>(sA, sB, off, ks, acc);
  else if (!half_n)
    compute_part<S, 1, TN>(sA, sB, off, ks, acc);
  else
    compute_part<S, 1, kHalfN ? TN / 2 : TN>(sA, sB, off, ks, acc);
}

// How a warp walks its part of C, lanes along consecutive rows: access e of E
// covers CPI columns (parts of fewer than 32 rows) or a 32-row piece of one.
// CT: lanes along consecutive columns of C^T, which are C's rows.
template <class S>
struct CWalk {
  static constexpr int CPI = S::WBM < 32 ? 32 / S::WBM : 1;
  static constexpr int RPC = S::WBM < 32 ? 1 : S::WBM / 32;
  static constexpr int E = S::WBN / CPI * RPC;
  static_assert(S::WBN % CPI == 0 && E % 4 == 0 && (!S::CT || S::WBN < 32), "C walk");
  // aligned C: four rows per lane, CPI4 columns per access
  static constexpr int CPI4 = 128 / S::WBM, E4 = S::WBN / CPI4;
  static_assert(S::CT || S::WBN % CPI4 == 0, "C walk");
  int lm, lc;
  __device__ __forceinline__ explicit CWalk(int lane)
      : lm(S::CT ? lane / S::WBN : S::WBM < 32 ? lane % S::WBM : lane),
        lc(S::CT ? lane % S::WBN : S::WBM < 32 ? lane / S::WBM : 0) {}
  __device__ __forceinline__ int m(int e) const {
    return lm + (S::CT ? e * (32 / S::WBN) : e % RPC * 32);
  }
  __device__ __forceinline__ int n(int e) const { return S::CT ? lc : e / RPC * CPI + lc; }
};
template <class S>
__device__ __forceinline__ long long c_at(const MatDesc& d, int m, int n) {
  return S::CT ? (long long)m * d.ldc + n : (long long)n * d.ldc + m;
}

// The warp's part of C (first row and column m0, n0) into sC, zero outside the
// matrix: asynchronous copies, all in flight together.
template <class S>
__device__ __forceinline__ void fetch_c(const float* C, const MatDesc& d, int m0, int n0,
                                        float* sC, int lane) {
  using W = CWalk<S>;
  if (!S::CT && vec16(C, d.ldc)) {
    const int lm = lane % (32 / W::CPI4) * 4, lc = lane / (32 / W::CPI4);
    const int valid = min(max(d.M - m0 - lm, 0), 4) * 4;
#pragma unroll 4
    for (int e = 0; e < W::E4; ++e) {
      const int nl = e * W::CPI4 + lc, n = n0 + nl;
      cp_async16(smem_u32(sC + nl * S::LDC + lm), C + (long long)n * d.ldc + (m0 + lm),
                 n < d.N ? valid : 0);
    }
    return;
  }
  const W w(lane);
#pragma unroll 4
  for (int e = 0; e < W::E; ++e) {
    const int m = m0 + w.m(e), n = n0 + w.n(e);
    cp_async4(smem_u32(sC + w.n(e) * S::LDC + w.m(e)), C + c_at<S>(d, m, n),
              m < d.M && n < d.N ? 4 : 0);
  }
}

// Matrix `mat` of the queue (CT: of the transposed product).
template <class S>
__device__ __forceinline__ MatDesc desc_of(const SimtParams& p, int mat) {
  const MatDesc d = p.descs[mat];
  if constexpr (S::CT) return MatDesc{d.N, d.M, d.K, d.ldb, d.lda, d.ldc, d.cfg, d.aux};
  return d;
}

__device__ __forceinline__ volatile int* control() {
  extern __shared__ __align__(16) float smem_all[];
  return reinterpret_cast<volatile int*>(smem_all + kWarps * kWarpFloats);
}
// The next item of the queue (the CTAs' first items are their block indexes).
__device__ __forceinline__ int pull_item(const SimtParams& p) {
  return atomicAdd(p.counters, 1) + (int)gridDim.x;
}
constexpr int kNoItem = 0x7fffffff;

// One tile of matrix `mat` whose first row and column are m0 and n0, by the
// calling team.  With `pull` the team's first thread takes its next item while
// C is written (the atomic's round trip is then hidden) and gets it back; a
// warp takes none when another warp of the CTA waits with a CTA tile.  A real
// call: inlined beside one another the shapes spilled in their k loops, by
// another amount after every edit (the 2048-matrix beta = 0.5 batch took 2.77
// ms with calls, 2.87 to 3.75 ms inlined).
template <class S>
__device__ __noinline__ int run_tile(const SimtParams& p, int mat, int m0, int n0, bool pull) {
  constexpr int TM = S::TM, TN = S::TN, NS = S::NS, BK = S::BK;
  extern __shared__ __align__(16) float smem_all[];
  const int thread = thread_index(), lane = thread & 31;
  const int tid = S::NT == 32 ? lane : thread;
  const int lx = S::lane_x(lane), ly = S::lane_y(lane);
  const int warp = thread >> 5;
  const int wm = S::NT == 32 ? 0 : warp % S::WM * S::WBM;  // the warp's part
  const int wn = S::NT == 32 ? 0 : warp / S::WM * S::WBN;
  float* ring = S::NT == 32 ? smem_all + warp * kWarpFloats : smem_all;
  float* sC = ring + (NS - 1) * S::STAGE + (S::NT == 32 ? 0 : warp * (S::WBN * S::LDC));

  f32x2 acc[TM / 2][TN];
  {
    const MatDesc d = desc_of<S>(p, mat);
    const float* A = S::CT ? p.B[mat] : p.A[mat];
    const float* B = S::CT ? p.A[mat] : p.B[mat];
    const bool a_vec = vec16(A, d.lda), b_vec = vec16(B, d.ldb);
    // the tile's first row and column at the k of the next stage to load
    A += S::TA ? (long long)m0 * d.lda : (long long)m0;
    B += S::TB ? (long long)n0 : (long long)n0 * d.ldb;
    const int mrem = d.M - m0, nrem = d.N - n0;
    const int b_off = S::SHIFT ? floats_off(B + (long long)(wn + ly) * d.ldb) : 0;

    // alpha = beta = 1: the chains start from C, as the reference's do; its
    // old values come in behind the prologue's stages
    const bool inplace = p.alpha == 1.0f && p.beta == 1.0f;
    if (inplace) {
      fetch_c<S>(p.C[mat], d, m0 + wm, n0 + wn, sC, lane);
    } else if (!S::CT && p.beta != 0.0f) {
      const float* C = p.C[mat];
      for (int c = lane; c < S::WBN; c += 32) {
        const int n = n0 + wn + c, m = m0 + wm;
        if (n < d.N && m < d.M) {
          const float* q = C + (long long)n * d.ldc + m;
          const int last = min(S::WBM, d.M - m) - 1;
#pragma unroll 1
          for (int r = 0; r < last; r += 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(q + r));
          asm volatile("prefetch.global.L2 [%0];" ::"l"(q + last));
        }
      }
    }
    cp_async_commit();

    int lda = d.lda, ldb = d.ldb;
    int to_load = d.K;  // k that no stage holds yet
    auto load_stage = [&](int slot) {
      float* sA = ring + slot * S::STAGE;
      float* sB = sA + S::A_STAGE;
      // opaque in each stage: the compiler would otherwise keep one address
      // per copy in registers across the k loop
      asm volatile("" : "+r"(lda), "+r"(ldb));
      if constexpr (S::TA)
        load_k_contig<S::NT, S::BM, S::LDA, BK, true>(A, lda, mrem, to_load, sA, false, tid);
      else
        load_rows_contig<S::NT, S::BM, S::LDA, BK>(A, lda, mrem, to_load, sA, a_vec, tid);
      if constexpr (S::TB)
        load_rows_contig<S::NT, S::BN, S::LDB, BK>(B, ldb, nrem, to_load, sB, b_vec, tid);
      else if constexpr (S::SHIFT)
        load_k_shifted<S::NT, S::BN, S::LDB, BK>(B, ldb, nrem, to_load, sB, to_load == d.K, tid);
      else
        load_k_contig<S::NT, S::BN, S::LDB, BK, S::BROWS>(B, ldb, nrem, to_load, sB, b_vec, tid);
      A += S::TA ? (long long)BK : (long long)BK * lda;
      B += S::TB ? (long long)BK * ldb : (long long)BK;
      to_load -= BK;
    };
#pragma unroll 1
    for (int s = 0; s < NS - 1; ++s) {
      if (to_load > 0) load_stage(s);
      cp_async_commit();
    }
    // C and the first stage are in; the last slot, where C is, is overwritten
    // only after the next sync
    cp_async_wait<NS - 2>();
    S::sync();
#pragma unroll
    for (int j = 0; j < TN; ++j)
#pragma unroll
      for (int h = 0; h < TM / 4; ++h) {
        ulonglong2 v = make_ulonglong2(0, 0);
        if (inplace)
          v = *reinterpret_cast<const ulonglong2*>(sC + S::n_of(ly, j) * S::LDC +
                                                   h * (S::LX * 4) + lx * 4);
        acc[2 * h][j] = v.x;
        acc[2 * h + 1][j] = v.y;
      }

    int rd_slot = 0, wr_slot = NS - 1;
#pragma unroll 1
    for (int k_left = d.K; k_left > 0; k_left -= BK) {
      cp_async_wait<NS - 2>();
      S::sync();
      if (to_load > 0) load_stage(wr_slot);
      cp_async_commit();
      const float* sA = ring + rd_slot * S::STAGE;
      compute_stage<S>(sA + wm + lx * 4,
                       sA + S::A_STAGE + (S::BROWS ? wn + S::n_of(ly, 0) : (wn + ly) * S::LDB),
                       b_off, mrem - wm, nrem - wn, k_left, acc);
      rd_slot = rd_slot + 1 == NS ? 0 : rd_slot + 1;
      wr_slot = wr_slot + 1 == NS ? 0 : wr_slot + 1;
    }
    cp_async_wait<0>();
    S::sync();
  }

  // C <- alpha * acc + beta * C (acc itself when its chains started from C).
  // The outputs pass through shared memory, so that lanes walk consecutive
  // rows; old values of C come in there first.  The matrix is read again
  // instead of being held through the k loop.
  const MatDesc d = desc_of<S>(p, mat);
  float* C = p.C[mat];
  int next = kNoItem;
  if (pull && tid == 0 && (S::NT != 32 || control()[kCtlPosts] == 0)) next = pull_item(p);
  {
    const float alpha = p.alpha, beta = p.beta;
    const bool inplace = alpha == 1.0f && beta == 1.0f, rd = !inplace && beta != 0.0f;
    if (rd) {
      fetch_c<S>(C, d, m0 + wm, n0 + wn, sC, lane);
      cp_async_commit();
      cp_async_wait<0>();
      __syncwarp();
    }
#pragma unroll
    for (int j = 0; j < TN; ++j)
#pragma unroll
      for (int h = 0; h < TM / 4; ++h) {
        float4* q =
            reinterpret_cast<float4*>(sC + S::n_of(ly, j) * S::LDC + h * (S::LX * 4) + lx * 4);
        const float2 lo = unpack2(acc[2 * h][j]), hi = unpack2(acc[2 * h + 1][j]);
        float4 v = make_float4(lo.x, lo.y, hi.x, hi.y);
        if (rd) {
          const float4 c = *q;
          v = make_float4(fmaf(alpha, v.x, beta * c.x), fmaf(alpha, v.y, beta * c.y),
                          fmaf(alpha, v.z, beta * c.z), fmaf(alpha, v.w, beta * c.w));
        } else if (!inplace) {
          v = make_float4(alpha * v.x, alpha * v.y, alpha * v.z, alpha * v.w);
        }
        *q = v;
      }
    __syncwarp();
  }
  using W = CWalk<S>;
  if (!S::CT && vec16(C, d.ldc)) {
    const int lm = lane % (32 / W::CPI4) * 4, lc = lane / (32 / W::CPI4);
    const int m = m0 + wm + lm;
#pragma unroll 4
    for (int e = 0; e < W::E4; ++e) {
      const int nl = e * W::CPI4 + lc, n = n0 + wn + nl;
      const float4 v = *reinterpret_cast<const float4*>(sC + nl * S::LDC + lm);
      float* q = C + (long long)n * d.ldc + m;
      if (n < d.N) {
        if (m + 4 <= d.M) {
          *reinterpret_cast<float4*>(q) = v;
        } else {
          if (m < d.M) q[0] = v.x;
          if (m + 1 < d.M) q[1] = v.y;
          if (m + 2 < d.M) q[2] = v.z;
        }
      }
    }
    return next;
  }
  const W w(lane);
#pragma unroll 4
  for (int e = 0; e < W::E; ++e) {
    const int m = m0 + wm + w.m(e), n = n0 + wn + w.n(e);
    if (m < d.M && n < d.N) C[c_at<S>(d, m, n)] = sC[w.n(e) * S::LDC + w.m(e)];
  }
  return next;
}

// An 8 x 128 tile of A B (CT: of B^T A^T, a 128 x 8 tile of C).  The long
// operand decides the form: where its k is contiguous it is staged as it lies,
// each lane with a row of it; else as slices of k, each lane with four rows,
// which is the 128 x 8 form of the transposed product.  Copies of 4 bytes pass
// through the L1, of which two CTAs' shared memory leaves 26 KB: rows that
// start anywhere take 16-byte copies from the boundary before them and selects
// (600 matrices of 8 x 1024 x 512 at odd leading dimensions: 524 us with 4-byte
// copies, 377 so; their transposes 600 and 376, on 16 bytes 467 and 297).
template <bool TA, bool TB, bool CT>
__device__ __forceinline__ int run_thin(const SimtParams& p, int mat, int m0, int n0, bool pull) {
  if constexpr (TB) {
    return run_tile<Shape<8, 1, 4, 4, 1, false, !TA, 32, !CT>>(p, mat, n0, m0, pull);
  } else {
    const bool vec = CT ? vec16(p.A[mat], p.descs[mat].lda) : vec16(p.B[mat], p.descs[mat].ldb);
    return vec ? run_tile<Shape<1, 8, 2, 4, 1, TA, false, 32, CT>>(p, mat, m0, n0, pull)
               : run_tile<Shape<1, 8, 2, 4, 1, TA, false, 32, CT, true>>(p, mat, m0, n0, pull);
  }
}

// Tiles that run only when a plan asks for them, by the CTA as well.
template <bool TA, bool TB>
__device__ __noinline__ int run_forced(const SimtParams& p, TileItem ti, int cfg, bool pull) {
  switch (cfg) {
    case 2:
      return run_tile<Shape<2, 4, 8, 4, 2, TA, TB>>(p, ti.mat, ti.tm * 64, ti.tn * 32, pull);
    case 3:
      return run_tile<Shape<2, 4, 4, 4, 2, TA, TB>>(p, ti.mat, ti.tm * 32, ti.tn * 64, pull);
    case 4:
      return run_tile<Shape<2, 4, 8, 4, 4, TA, TB>>(p, ti.mat, ti.tm * 64, ti.tn * 64, pull);
    case 5:
      return run_tile<Shape<4, 2, 4, 8, 4, TA, TB>>(p, ti.mat, ti.tm * 128, ti.tn * 64, pull);
    default:
      return run_tile<Shape<2, 4, 4, 8, 4, TA, TB>>(p, ti.mat, ti.tm * 64, ti.tn * 128, pull);
  }
}

// The persistent kernel's body.  CTAs pull items of the largest-first queue
// with an atomic counter.  A CTA tile occupies all eight warps.  When the
// pulled item is a warp tile, the warps go on by themselves, each pulling and
// computing tiles of its own, until one of them pulls a CTA tile or the queue
// is empty: that warp leaves the tile among the control words, the others stop
// after the tile they are at, and the CTA computes what was left together.
template <bool TA, bool TB>
__device__ __forceinline__ void persistent_body(const SimtParams& p) {
  pdl_wait();
  volatile int* ctl = control();
  const int lane = threadIdx.x & 31;
  const int n_items = p.n_items_dev ? *p.n_items_dev : p.n_items;
  // With no more items than CTAs each CTA has its own: nobody pulls (a count of
  // CTA tiles that is not zero keeps the warps from it) and the queue's
  // counters are not touched.  16 matrices of at most 32: 4.7 us a launch with
  // every warp's pull and the count of the CTAs that finished, 3.5 without.
  // Else no more warps of a CTA pull at its start than items fall to it, all
  // eight of the first CTAs would pull a short queue empty; and they take turns
  // from the quarter of the SM on whose scheduler the SM's other CTA does not
  // start, since two warps of 32 x 32 tiles on one take twice as long.  (512
  // tiles of 8 matrices of 256 x 256 x 1024 on 304 CTAs: 112 us with eight
  // pullers, 66 with two, 45 with their turns; only speed hangs on the slots.)
  if (threadIdx.x == 0) {
    ctl[kCtlPosts] = n_items > (int)gridDim.x ? 0 : -1;
    int slot;  // of the SM's warps; warp w of a CTA has quarter (slot + w) % 4
    asm volatile("mov.u32 %0, %%warpid;" : "=r"(slot));
    ctl[kCtlTurn] = slot + (slot & 8) / 4;
  }
  __syncthreads();
  int it = (int)blockIdx.x;
#pragma unroll 1
  while (it < n_items) {
    int posts = 1;  // CTA tiles to compute: `it`, or those that warps left
    const bool left = simt_warp_cfg(p.descs[p.items[it].mat].cfg);
    if (left) {
      const int warp = threadIdx.x >> 5;
      const int turn = ((warp + ctl[kCtlTurn]) & 3) | (warp & 4);
      if (turn != 0)
        it = n_items > turn * (int)gridDim.x || (it != (int)blockIdx.x && n_items > (int)gridDim.x)
                 ? __shfl_sync(0xffffffffu, lane == 0 ? pull_item(p) : 0, 0)
                 : kNoItem;
#pragma unroll 1
      while (it < n_items) {
        const TileItem ti = p.items[it];
        const int cfg = p.descs[ti.mat].cfg;
        int next;
        if (!simt_warp_cfg(cfg)) {
          if (lane == 0)
            ctl[kCtlPost + atomicAdd(const_cast<int*>(ctl) + kCtlPosts, 1)] = it;
          break;
        }
        // (16 x 16: slices of 32 k, fewer waits and address sums per k.  One tile
        // of K = 4096 66 us, in slices of 16 78.  Both forms, by a line at K =
        // 256, cost batches that run only one of them up to a tenth: 546 matrices
        // of up to 109 11.3 us, 9.9 and 10.7 with either alone.)
        if (cfg == 0)
          next = run_tile<Shape<1, 1, 4, 4, 2, TA, TB, 32>>(p, ti.mat, ti.tm * 16, ti.tn * 16, true);
        else
          next = run_tile<Shape<1, 1, 4, 8, 4, TA, TB>>(p, ti.mat, ti.tm * 32, ti.tn * 32, true);
        __syncwarp();  // the staged C has been read: the next tile's copies may land there
        it = __shfl_sync(0xffffffffu, next, 0);
      }
      __syncthreads();
      posts = ctl[kCtlPosts];
      if (posts <= 0) break;  // every warp found the queue empty
    }
    int next = kNoItem;
#pragma unroll 1
    for (int q = 0; q < posts; ++q) {
      if (q > 0) __syncthreads();  // the ring is free again
      const TileItem ti = p.items[left ? ctl[kCtlPost + q] : it];
      const int cfg = p.descs[ti.mat].cfg;
      const bool pull = q == posts - 1 && n_items > (int)gridDim.x;
      if (cfg == 8)
        next = run_thin<TA, TB, false>(p, ti.mat, ti.tm * 8, ti.tn * 128, pull);
      else if (cfg == 9)
        next = run_thin<!TB, !TA, true>(p, ti.mat, ti.tn * 8, ti.tm * 128, pull);
      else if (cfg == 7)
        next = run_tile<Shape<2, 4, 8, 8, 8, TA, TB>>(p, ti.mat, ti.tm * 128, ti.tn * 128, pull);
      else
        next = run_forced<TA, TB>(p, ti, cfg, pull);
    }
    if (threadIdx.x == 0) {
      ctl[kCtlItem] = next;
      ctl[kCtlPosts] = 0;
    }
    __syncthreads();
    it = ctl[kCtlItem];
    // (the next round writes the control words only behind another barrier or,
    // a warp's post, after every thread has passed this one)
  }
  // The last CTA to leave resets the queue, so the next launch (or graph
  // replay) starts from item 0 without a memset.  Every pull of a CTA has
  // returned before its thread 0 gets here: each warp that leaves the loop
  // alone does so through the barrier above.
  if (n_items > (int)gridDim.x && threadIdx.x == 0) {
    const unsigned prev = atomicAdd(reinterpret_cast<unsigned*>(p.counters) + 1, 1u);
    if (prev == gridDim.x - 1) {
      atomicExch(p.counters, 0);
      atomicExch(p.counters + 1, 0);
    }
  }
}

}  // namespace simt
}  // namespace bgemm
