// tc2_kernel.cu -- the split-precision tensor-core GEMM on CTA pairs
// (tcgen05 cta_group::2, two SMs per output tile).
//
// Each cluster of two CTAs owns a 256 x BN output tile (BN = 64, 128 or 256)
// of one matrix: CTA r loads rows [128r, 128r + 128) of the A side and rows
// [r*BN/2, (r+1)*BN/2) of the B side (hi and lo halves) with TMA into its own
// shared memory, the leader CTA issues every cta_group::2 MMA, and each CTA
// receives its 128 x BN slice of the accumulator in its own TMEM.  Per
// 128-byte K slice a CTA loads at most 64 KB for 128 x 256 outputs -- half
// the L2 traffic per flop of the one-SM kernel (tc_kernel.cu), which is what
// bounds that kernel.
//
// Accumulation is group-promoted as in tc_kernel.cu: each group accumulates
// into a fresh 256-column TMEM buffer (2-deep ring) with the small products
// first, and the epilogue warps of both CTAs add it into FP32 registers with
// round-to-nearest.  The group length per bucket of K comes from the launch's
// autotuned TcSchedule (a number of 128-byte K slices, or one MMA with lo*lo
// kept on the small-K path).
//
// Scheduling is dynamic: the leader CTA's producer pulls the next item of
// the largest-first queue with one atomic (fetched a tile ahead, so its
// latency hides behind the current tile's loads) and publishes it in a
// 4-slot ring in the shared memory of both CTAs (a remote store plus a
// release.cluster arrive on the peer's barrier).  The leader's MMA lane, the
// 16 epilogue warps of both CTAs and the peer's producer read each slot and
// acknowledge it on the leader's sempty barrier; -1 ends the walk.  The last
// cluster to finish resets the queue head, so graph replays need no memset.
//
// Synchronisation across the pair:
//   full[s]   leader only: its producer expects the bytes of both CTAs; the
//             peer's TMA completes on the leader's barrier (cta_group::2 TMA);
//   empty[s]  both CTAs: the leader's commit is multicast to the pair;
//   tfull[b]  both CTAs: multicast commit when a group's MMAs finish;
//   tempty[b] leader only: 16 arrivals (8 epilogue warps x 2 CTAs), relaxed:
//             each warp's TMEM loads have completed before it arrives;
//   sfull[j]  both CTAs: the leader's producer published schedule slot j;
//   sempty[j] leader only: 18 arrivals (leader MMA lane, peer producer,
//             8 epilogue warps x 2 CTAs) once slot j has been read.
// All waits are bounded as in tc_kernel.cu.
#include <stdint.h>

#include "tc_epilogue.h"
#include "tc_ptx.h"
#include "tc_split.h"
#include "tile_table.h"

namespace bgemm {
namespace {

constexpr int kRows = 128;                 // A-side rows per CTA
constexpr int kA = kRows * 128;            // 16 KB per part
constexpr int kB = 128 * 128;              // B-side half: up to 128 rows
constexpr int kNAcc = 2;                   // 256-column accumulator buffers
constexpr int kSched = 4;                  // schedule slots (items published ahead)
// Packing warps (warps 2 and 3, otherwise idle): each loads a strip of 32 packed rows in chunks
// of 32 k through a ring of four buffers, [k][33] floats where rows are
// contiguous in memory and [row][32] where k is.
constexpr int kPackWarps = 2, kPackBufs = 4, kPackK2 = 32;
constexpr int kPackFloats = kPackK2 * 33;
// K from which a strip with contiguous k is walked in chunks of 8 rows x 128 k
// instead of 32 x 32.
constexpr int kPackWideK = 256;
constexpr int kPackBytes = kPackFloats * 4;
// Stage ring of 3 stages of 64 KB, two parts per side: the split modes' hi and
// lo halves of one 128-byte K slice, or two consecutive K slices of the
// single-product TF32 mode (four TMA boxes per stage either way: one thread
// keeps ~150 GB/s per SM in flight with four boxes per stage, ~100 with two).
template <int SPLIT>
struct Geo2 {
  static constexpr int NP = 2;
  static constexpr int STAGE = NP * (kA + kB);
  static constexpr int S = 3;
  static constexpr int NBAR = 2 * S + 2 * kNAcc + 1 + 2 * kSched;
  // barriers | TMEM address, abort flag (16 B) | schedule slots | packing
  // warps' buffers (16-byte aligned) | alignment of the whole
  static constexpr int PACK = (S * STAGE + NBAR * 8 + 16 + 4 * kSched + 15) / 16 * 16;
  static constexpr int SMEM = PACK + kPackWarps * kPackBufs * kPackBytes + 1024;
};
constexpr int kSmemMax = Geo2<1>::SMEM > Geo2<0>::SMEM ? Geo2<1>::SMEM : Geo2<0>::SMEM;
constexpr int kEpiWarps2 = 8;              // 2 per TMEM lane quadrant
constexpr int kCols = 128;                 // accumulator columns per epilogue warp
// Three warpgroups: warpgroup 0 = producer (warp 0), MMA issuer (warp 1) and
// two packing warps; warpgroups 1 and 2 = the 8 epilogue warps.  At launch every
// thread gets 168 registers (3 warps per SM sub-partition); warpgroup 0 gives
// most of its share to the epilogue warps, whose 128 accumulator columns per
// lane would otherwise spill: 128 x 72 + 256 x 216 = 384 x 168.  (At 56 and
// 224 the packing warps spilled: batch stream 6846 us, 6812 this way.)
constexpr int kThreads2 = 384;
constexpr int kEpiWarp0 = 4;               // first epilogue warp
constexpr uint32_t kRegsCtl = 72, kRegsEpi = 216, kRegsLaunch = 168;
static_assert(128 * kRegsCtl + 256 * kRegsEpi <= kThreads2 * kRegsLaunch, "register split");
// Promotion groups of the split modes come per bucket of K from the launch's
// TcSchedule (autotuned table): group g > 0 = g 128-byte K slices per TMEM
// buffer, g = 0 = the small-K path (promote every MMA, keep lo*lo).
__device__ __forceinline__ int group_slices(const TcGemmParams& p, int K) {
  return p.sched.group(tc_sched_bucket(K));
}
// beta != 0: promotion groups before the tile's end at which C is prefetched
// into L2 (autotuned, tile_table.h; 0 = no prefetch)
constexpr int kCPrefetchLead = kTcCPrefetchLead;
static_assert(kCPrefetchLead >= 0 && kCPrefetchLead <= 16, "C prefetch lead out of range");

// MMA width of a tile along the B side: bn, or for the matrix's last tile
// column its remaining width rounded up to 16 (the pair MMA's N step), so
// that the padding of a ragged edge is not multiplied.  CTA r then loads
// B-side rows [tn*bn + r*n/2, +n/2), the columns stay contiguous.
__device__ __forceinline__ int tile_n(const MatDesc& d, int tn, int bn) {
  const int rem = (tc_cfg_swap(d.cfg) ? d.M : d.N) - tn * bn;
  return min(bn, (rem + 15) & ~15);
}

template <int KIND>
__device__ __forceinline__ uint32_t make_idesc_pair(int n) {
  constexpr uint32_t fmt = (KIND == kKindTF32) ? 2u : 1u;
  return (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(256 >> 4) << 24);
}

__device__ __forceinline__ void cp4(uint32_t dst, const float* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void cp16(uint32_t dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes)
               : "memory");
}

// A packing warp: pulls strips behind the pre-pass kernel's and splits them as
// tc_pack_kernel does, three chunks on their way while one is written.  A
// finished strip is published by a release on its matrix's count, behind a
// proxy fence: the readers are TMA loads.
// Bound by the issue of one warp: alone on the chip the 304 of them split the
// skewed batch's 5.5 GB of operands in 3.5 ms (4.2 ms before inner chunks lost
// their bounds), beside the GEMM in 5.7.  What it costs the GEMM is the packed
// stores: half of it their way into L2, half their way on to HBM, from where
// the GEMM reads them back (the operands in use at a time are larger than L2);
// the copies into shared memory cost little.  Skewed batch, pre-pass then GEMM
// 9.45 ms, this way 8.6 to 8.9; a limit on how far packing runs ahead of the
// tiles (one to eight waves), stores that bypass a cache and L2 prefetch by the
// producers changed nothing or made it slower.
template <int KIND, int SPLIT>
__device__ __forceinline__ void pack_strips(const TcGemmParams& p, float* buf, int lane,
                                            volatile int* abort) {
  const int n_jobs = *p.n_jobs, n_head = *p.n_head;
  if (n_head >= n_jobs) return;
#pragma unroll 1
  for (;;) {
    int j = 0;
    if (lane == 0) j = *abort ? n_jobs : n_head + atomicAdd(p.counters + 2, 1);
    j = __shfl_sync(0xffffffffu, j, 0);
    if (j >= n_jobs) return;
    const PackJob job = p.jobs[j];
    const bool is_a = job.op == 0;
    int K, rows, ld;
    bool rows_contig;
    {
      const MatDesc d = p.descs[job.mat];
      K = d.K;
      rows = (is_a ? d.M : d.N) - job.r0;
      ld = is_a ? d.lda : d.ldb;
      rows_contig = is_a ? !(d.aux & kTransAFlag) : (d.aux & kTransBFlag) != 0;
    }
    const float* X = is_a ? p.A[job.mat] : p.B[job.mat];
    X += rows_contig ? (long long)job.r0 : (long long)job.r0 * ld;
    const bool vec = ((reinterpret_cast<uintptr_t>(X) & 15u) == 0) && (ld & 3) == 0;
    // A chunk: 32 rows of 32 k or, where k is contiguous and long, 8 rows of
    // 128 k.  The packed stores are what packing costs the GEMM (skewed batch
    // 8.6 ms, 6.8 without them, 6.5 without packing at all), and rows of 256 or
    // 512 bytes cost less than pieces of 64 or 128: row-major NT of 96 matrices
    // of 97 to 1501 in BF16 521 -> 507 us, the skewed batch 9.00 -> 8.92 ms.
    // Lines at K = 128 or 512: row 504 and 508 us, the skewed batch 0.3 and 0.8
    // % slower than at 256.  The single product keeps the 32 x 32 chunks: no
    // faster with the others (1227 and 1224 us, 128 matrices of N = K = 1024).
    const bool wide = SPLIT && !rows_contig && K >= kPackWideK;
    const int kc = wide ? 128 : kPackK2, rc = wide ? 8 : 32;
    const int rows_end = K > 0 ? min(rows, 32) : 0;
    // one chunk's copies; inner ones carry no bounds
    auto load = [&](int k0, int r, float* s) {
      const uint32_t dst = smem_u32(s) + lane * 4;
      const int ks = K - k0;
      if (wide) {
        const float* src = X + (long long)r * ld + k0;
        if (vec) {
          const int bytes = min(max(ks - 4 * lane, 0), 4) * 4;
#pragma unroll
          for (int i = 0; i < 8; ++i)
            cp16(dst + (i * 128 + 3 * lane) * 4, src + (long long)ld * i + 4 * lane,
                 r + i < rows ? bytes : 0);
        } else if (ks >= 128 && r + 8 <= rows) {
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int q = 0; q < 4; ++q)
              cp4(dst + (i * 128 + q * 32) * 4, src + (long long)ld * i + q * 32 + lane, 4);
        } else {
#pragma unroll 1
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int q = 0; q < 4; ++q)
              cp4(dst + (i * 128 + q * 32) * 4, src + (long long)ld * i + q * 32 + lane,
                  r + i < rows && q * 32 + lane < ks ? 4 : 0);
        }
      } else if (rows_contig) {
        const float* src = X + (long long)k0 * ld + lane;
        const int bytes = lane < rows ? 4 : 0;
        if (ks >= kPackK2) {
#pragma unroll
          for (int k = 0; k < kPackK2; ++k) cp4(dst + k * 132, src + (long long)ld * k, bytes);
        } else {
#pragma unroll 4
          for (int k = 0; k < kPackK2; ++k)
            cp4(dst + k * 132, src + (long long)ld * k, k < ks ? bytes : 0);
        }
      } else if (vec) {
        const int kq = (lane & 7) * 4, r0 = lane >> 3;
        const int bytes = min(max(ks - kq, 0), 4) * 4;
        const float* src = X + (long long)r0 * ld + k0 + kq;
#pragma unroll
        for (int r = 0; r < 32; r += 4)
          cp16(smem_u32(s) + ((r0 + r) * kPackK2 + kq) * 4, src + (long long)ld * r,
               r0 + r < rows ? bytes : 0);
      } else {
        const float* src = X + k0 + lane;
        const int bytes = lane < ks ? 4 : 0;
        if (rows >= 32) {
#pragma unroll
          for (int r = 0; r < 32; ++r) cp4(dst + r * 128, src + (long long)ld * r, bytes);
        } else {
#pragma unroll 4
          for (int r = 0; r < 32; ++r)
            cp4(dst + r * 128, src + (long long)ld * r, r < rows ? bytes : 0);
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const PackDesc* pd = p.pdescs + job.mat;
    const int kpad = pd->kpad;
    constexpr int E = KIND == kKindTF32 ? 4 : 2;  // bytes of a packed element
    // four k a lane: eight lanes to a packed row and four rows at a time, or
    // the warp to a row
    const int r4 = wide ? 0 : lane >> 3, kq = (wide ? lane : lane & 7) * 4;
    const int rstep = wide ? 1 : 4;
    const long long step = (long long)rstep * kpad;  // elements
    char* const hi0 = p.ws + (is_a ? pd->a_hi : pd->b_hi);
    char* const lo0 = p.ws + (is_a ? pd->a_lo : pd->b_lo);
    int lk = 0, lr = 0;  // the next chunk to load
    auto load_next = [&](int b) {
      if (lr < rows_end) {
        load(lk, lr, buf + b * kPackFloats);
        lk += kc;
        if (lk >= K) {
          lk = 0;
          lr += rc;
        }
      } else {
        asm volatile("cp.async.commit_group;" ::: "memory");
      }
    };
#pragma unroll 1
    for (int c = 0; c < kPackBufs - 1; ++c) load_next(c);
    int rd = 0, wr = kPackBufs - 1, k0 = 0, r0 = 0;
#pragma unroll 1
    while (r0 < rows_end) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kPackBufs - 2) : "memory");
      __syncwarp();  // (and every lane is done with the buffer that is filled next)
      load_next(wr);
      const long long at = (long long)(job.r0 + r0 + r4) * kpad + k0 + kq;
      char* hi = hi0 + at * E;
      char* lo = lo0 + at * E;
      // (k contiguous: r4 * 32 + kq, or kq, are 4 * lane in either form)
      const float* s = buf + rd * kPackFloats + (rows_contig ? kq * 33 + r4 : 4 * lane);
      auto fetch = [&](int it, float(&x)[4]) {
        if (rows_contig) {
#pragma unroll
          for (int i = 0; i < 4; ++i) x[i] = s[i * 33 + it * 4];
        } else {
          const float4 v = *reinterpret_cast<const float4*>(s + it * 4 * kPackK2);
          x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
        }
      };
      if (rows - r0 >= rc && k0 + kc <= K) {
        // (four rows of fragments at a time, for their latencies to overlap)
#pragma unroll
        for (int i0 = 0; i0 < 8; i0 += 4) {
          float x[4][4];
#pragma unroll
          for (int i = 0; i < 4; ++i) fetch(i0 + i, x[i]);
#pragma unroll
          for (int i = 0; i < 4; ++i) put4<KIND, SPLIT>(hi, lo, (i0 + i) * step, x[i]);
        }
      } else {
#pragma unroll 1
        for (int it = 0; it < 8; ++it) {
          const int left = K - k0 - kq;
          if (r0 + it * rstep + r4 < rows && left > 0) {
            float x[4];
            fetch(it, x);
            if (left >= 4) {
              put4<KIND, SPLIT>(hi, lo, it * step, x);
            } else {
#pragma unroll
              for (int i = 0; i < 3; ++i)
                if (i < left) put<KIND, SPLIT>(hi, lo, it * step + i, x[i]);
            }
          }
        }
      }
      k0 += kc;
      if (k0 >= K) {
        k0 = 0;
        r0 += rc;
      }
      rd = rd + 1 == kPackBufs ? 0 : rd + 1;
      wr = wr + 1 == kPackBufs ? 0 : wr + 1;
    }
    __syncwarp();
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __threadfence();
    asm volatile("fence.proxy.async.global;" ::: "memory");
    __syncwarp();
    if (lane == 0)
      asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(p.ready + job.mat) : "memory");
  }
}

// Waits (bounded) until `need` strips of a matrix are packed.
__device__ __forceinline__ bool wait_packed(const int* ready, int need, int* err,
                                            volatile int* abort, unsigned long long limit_ns) {
  auto done = [&]() {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(ready) : "memory");
    return v >= need;
  };
  if (!done()) {
    const uint64_t t0 = gtimer();
    while (!done()) {
      __nanosleep(100);
      if (*abort) return false;
      if (gtimer() - t0 > limit_ns) {
        atomicOr(err, 1);
        *abort = 1;
        return false;
      }
    }
  }
  asm volatile("fence.proxy.async.global;" ::: "memory");
  return true;
}

// BETA: the launch's beta is nonzero (C is read, eight reads ahead of the
// stores; the L2 prefetch of kCPrefetchLead is off in the tuned table).  The
// beta = 0 form is a separate instantiation that keeps the
// plain epilogue's code (the read path's registers slowed it by ~4 %).
template <int KIND, int SPLIT, bool BETA>
__global__ void __launch_bounds__(kThreads2, 1) tc2_gemm_kernel(const TcGemmParams p) {
  using G = Geo2<SPLIT>;
  constexpr int kS = G::S;
  constexpr int kStage = G::STAGE;
  constexpr int kNBar = G::NBAR;
  constexpr int KE = (KIND == kKindTF32) ? 32 : 64;  // elements per 128-byte slice
  constexpr int NSUB = 4;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t pad = (1024u - (raw & 1023u)) & 1023u;
  uint8_t* smem = smem_raw + pad;
  const uint32_t sbase = raw + pad;
  const uint32_t bar0 = sbase + kS * kStage;
  auto full = [&](int s) { return bar0 + 8u * s; };
  auto empty = [&](int s) { return bar0 + 8u * (kS + s); };
  auto tfull = [&](int s) { return bar0 + 8u * (2 * kS + s); };
  auto tempty = [&](int s) { return bar0 + 8u * (2 * kS + kNAcc + s); };
  const uint32_t drain = bar0 + 8u * (2 * kS + 2 * kNAcc);
  auto sfull = [&](int j) { return bar0 + 8u * (2 * kS + 2 * kNAcc + 1 + j); };
  auto sempty = [&](int j) { return bar0 + 8u * (2 * kS + 2 * kNAcc + 1 + kSched + j); };
  volatile uint32_t* tmem_slot =
      reinterpret_cast<volatile uint32_t*>(smem + kS * kStage + kNBar * 8);
  volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* slots = reinterpret_cast<volatile int*>(tmem_slot + 4);
  const uint32_t slots_addr = smem_u32(const_cast<int*>(slots));

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int ncl = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kS; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), 1);
    }
    for (int s = 0; s < kNAcc; ++s) {
      mbar_init(tfull(s), 1);
      mbar_init(tempty(s), 2 * kEpiWarps2);
    }
    for (int j = 0; j < kSched; ++j) {
      mbar_init(sfull(j), 1);
      mbar_init(sempty(j), 2 + 2 * kEpiWarps2);
    }
    mbar_init(drain, 1);
    *abort = 0;
    fence_mbar_init();
  }
  cluster_sync();
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_wait();  // (all of the above runs beside the pre-pass's last CTAs)
  const int n_items = p.n_items_dev ? *p.n_items_dev : p.n_items;
  if (p.cta_times && threadIdx.x == 0) p.cta_times[2 * blockIdx.x] = gtimer();

  // Each warpgroup sets its register budget at one point that all four of
  // its warps execute (setmaxnreg is warpgroup-aligned), ahead of the roles'
  // code, so that the compiler allocates every role for its budget.
  if (warp < kEpiWarp0) {
    regs_shrink<kRegsCtl>();
    if (warp == 0) {
      // ------------------------------------------------------------ producer
      if (lane == 0) {
        Ring st, sc;
        // stages with a load in flight, and the phase each was loaded in (bit s)
        uint32_t inflight = 0, inflight_phase = 0;
        bool ok = true;
        int last_mat = -1;
        // The leader publishes each item one tile ahead of its own loads, so
        // the peer's producer and the consumers find the next item ready.
        auto pull = [&]() {
          const int v = atomicAdd(p.counters, 1);
          return v < n_items ? v : -1;
        };
        auto publish = [&](int v) {
          if (!wait_bounded_cluster(sempty(sc.idx), sc.phase ^ 1u, p.error, abort, p.timeout_ns))
            return false;
          slots[sc.idx] = v;
          st_cluster_u32(mapa_shared(slots_addr + 4u * sc.idx, 1), (uint32_t)v);
          mbar_arrive(sfull(sc.idx));
          mbar_arrive_cluster(mapa_shared(sfull(sc.idx), 1));
          sc.next(kSched);
          return true;
        };
        int cur = -1, nxt = -1;
        if (leader) {
          cur = pull();
          ok = publish(cur);
          if (ok && cur >= 0) nxt = pull();
        }
        while (ok) {
          int it;
          if (leader) {
            it = cur;
            if (it < 0) break;
            if (!publish(nxt)) {
              ok = false;
              break;
            }
            const int after = nxt >= 0 ? pull() : -1;
            cur = nxt;
            nxt = after;
          } else {
            if (!wait_bounded_cluster(sfull(sc.idx), sc.phase, p.error, abort, p.timeout_ns)) {
              ok = false;
              break;
            }
            it = slots[sc.idx];
            mbar_arrive_cluster(mapa_shared(sempty(sc.idx), 0));
            sc.next(kSched);
            if (it < 0) break;
          }
          const TileItem ti = p.items[it];
          const MatDesc d = p.descs[ti.mat];
          const int bn = tc2_cfg_bn(d.cfg);
          const int hb = bn >> 1;
          const CUtensorMap* tm = p.tmaps + 4 * ti.mat;
          if (ti.mat != last_mat && d.K > 0) {
            const int await = p.jobs ? p.pdescs[ti.mat].await : 0;
            for (int q = 0; q < 4; ++q) tmap_acquire(tm + q);
            if (await > 0 &&
                !wait_packed(p.ready + ti.mat, await, p.error, abort, p.timeout_ns)) {
              ok = false;
              break;
            }
            last_mat = ti.mat;
          }
          const int nk = (d.K + KE - 1) / KE;           // 128-byte K slices
          const int nst = SPLIT ? nk : (nk + 1) / 2;     // stages
          const int row_a = ti.tm * 256 + (int)rank * kRows;
          const int row_b = ti.tn * bn + (int)rank * (tile_n(d, ti.tn, bn) >> 1);
          for (int kb = 0; kb < nst; ++kb) {
            // single product: slices 2kb and (if it exists) 2kb + 1
            const int parts = SPLIT ? 2 : (2 * kb + 1 < nk ? 2 : 1);
            const uint32_t tx = 2u * parts * (uint32_t)(kA + hb * 128);  // both CTAs
            if (!wait_bounded(empty(st.idx), st.phase ^ 1u, p.error, abort, p.timeout_ns)) {
              ok = false;
              break;
            }
            const uint32_t sa = sbase + st.idx * kStage;
            const uint32_t sb = sa + G::NP * kA;
            const uint32_t fb = mapa_shared(full(st.idx), 0);
            if (leader) {
              mbar_arrive_expect_tx(full(st.idx), tx);
              inflight |= 1u << st.idx;
              inflight_phase = (inflight_phase & ~(1u << st.idx)) | (st.phase << st.idx);
            }
            if (SPLIT) {
              tma_load_2d_pair(sa, tm + 0, kb * KE, row_a, fb);
              tma_load_2d_pair(sb, tm + 2, kb * KE, row_b, fb);
              tma_load_2d_pair(sa + kA, tm + 1, kb * KE, row_a, fb);
              tma_load_2d_pair(sb + kB, tm + 3, kb * KE, row_b, fb);
            } else {
              for (int j = 0; j < parts; ++j) {
                tma_load_2d_pair(sa + j * kA, tm + 0, (2 * kb + j) * KE, row_a, fb);
                tma_load_2d_pair(sb + j * kB, tm + 2, (2 * kb + j) * KE, row_b, fb);
              }
            }
            st.next(kS);
          }
          if (!ok) break;
        }
        // The leader's full barriers count the bytes of both CTAs: once every
        // phase it expected has completed, no copy of either CTA is in flight.
        if (leader) {
          for (int s = 0; s < kS; ++s)
            if ((inflight >> s) & 1u)
              wait_bounded(full(s), (inflight_phase >> s) & 1u, p.error, nullptr, p.timeout_ns);
        }
        if (!ok) {
          const uint64_t t0 = gtimer();  // aborted: give stray copies time to land
          while (gtimer() - t0 < 200000ull) {
          }
        }
      }
      __syncwarp();
    } else if (warp == 1) {
      // -------------------------------------------------- MMA issue (leader)
      if (lane == 0 && leader) {
        Ring st, acc, sc;
        bool ok = true;
        while (ok) {
          if (!wait_bounded(sfull(sc.idx), sc.phase, p.error, abort, p.timeout_ns)) break;
          const int it = slots[sc.idx];
          mbar_arrive(sempty(sc.idx));
          sc.next(kSched);
          if (it < 0) break;
          const TileItem ti = p.items[it];
          const MatDesc d = p.descs[ti.mat];
          const int bn = tc2_cfg_bn(d.cfg);
          const uint32_t idesc = make_idesc_pair<KIND>(tile_n(d, ti.tn, bn));
          const int nk = (d.K + KE - 1) / KE;
          const int nsub = (d.K + KE / NSUB - 1) / (KE / NSUB);
          const int gs = SPLIT ? group_slices(p, d.K) : 1;
          const bool fine = SPLIT && gs == 0;
          int kg = 0;  // slice within the current promotion group
          // A 256-column buffer holds P = 256 / bn promotion groups side by
          // side (sub-accumulators at column stride bn), so narrow tiles run P
          // groups ahead before waiting on the epilogue's drain.
          const int P = 256 / bn;
          int sub = 0;        // promotion group within the current buffer
          uint32_t gbuf = 0;  // TMEM address of the current group
          auto begin_group = [&]() {
            if (sub == 0) {
              if (!wait_bounded(tempty(acc.idx), acc.phase ^ 1u, p.error, abort, p.timeout_ns))
                return false;
              tc_fence_after();
            }
            gbuf = tmem + acc.idx * 256u + (uint32_t)(sub * bn);
            return true;
          };
          auto end_group = [&](bool last) {
            if (++sub == P || last) {
              mma_commit_pair(tfull(acc.idx));
              acc.next(kNAcc);
              sub = 0;
            }
          };
          const int nst = SPLIT ? nk : (nk + 1) / 2;  // stages (the producer's count)
          for (int kb = 0; kb < nst; ++kb) {
            if (!wait_bounded(full(st.idx), st.phase, p.error, abort, p.timeout_ns)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t sa = sbase + st.idx * kStage;
            const uint32_t sb = sa + G::NP * kA;
            const int s_end = min(NSUB, nsub - kb * NSUB);
            if (!SPLIT) {
              // one product: a single accumulator per tile, the 2-deep ring
              // alternating between tiles; the stage holds K slices 2kb, 2kb+1
              if (kb == 0) {
                if (!wait_bounded(tempty(acc.idx), acc.phase ^ 1u, p.error, abort, p.timeout_ns)) {
                  ok = false;
                  break;
                }
                tc_fence_after();
              }
              const uint32_t buf = tmem + acc.idx * 256u;
              for (int j = 0; j < 2 && 2 * kb + j < nk; ++j) {
                const int slice = 2 * kb + j;
                const int se = min(NSUB, nsub - slice * NSUB);
                for (int s = 0; s < se; ++s)
                  mma_pair<KIND>(buf, sw128_desc(sa + j * kA + 32u * s),
                                 sw128_desc(sb + j * kB + 32u * s), idesc,
                                 (slice > 0 || s > 0) ? 1u : 0u);
              }
              if (kb == nst - 1) {
                mma_commit_pair(tfull(acc.idx));
                acc.next(kNAcc);
              }
            } else if (fine) {
              for (int s = 0; s < s_end && ok; ++s) {
                if (!begin_group()) {
                  ok = false;
                  break;
                }
                const uint32_t buf = gbuf;
                // small K: the split error dominates, so lo*lo is kept too
                mma_pair<KIND>(buf, sw128_desc(sa + kA + 32u * s), sw128_desc(sb + kB + 32u * s),
                               idesc, 0u);
                mma_pair<KIND>(buf, sw128_desc(sa + kA + 32u * s), sw128_desc(sb + 32u * s), idesc,
                               1u);
                mma_pair<KIND>(buf, sw128_desc(sa + 32u * s), sw128_desc(sb + kB + 32u * s), idesc,
                               1u);
                mma_pair<KIND>(buf, sw128_desc(sa + 32u * s), sw128_desc(sb + 32u * s), idesc, 1u);
                end_group(kb == nk - 1 && s == s_end - 1);
              }
              if (!ok) break;
            } else {
              // a group spans gs slices; small products of each slice first
              const bool first = kg == 0;
              if (first && !begin_group()) {
                ok = false;
                break;
              }
              const uint32_t buf = gbuf;
              for (int s = 0; s < s_end; ++s) {
                mma_pair<KIND>(buf, sw128_desc(sa + kA + 32u * s), sw128_desc(sb + 32u * s), idesc,
                               (first && s == 0) ? 0u : 1u);
                mma_pair<KIND>(buf, sw128_desc(sa + 32u * s), sw128_desc(sb + kB + 32u * s), idesc,
                               1u);
              }
              for (int s = 0; s < s_end; ++s)
                mma_pair<KIND>(buf, sw128_desc(sa + 32u * s), sw128_desc(sb + 32u * s), idesc, 1u);
              if (++kg == gs || kb == nk - 1) {
                end_group(kb == nk - 1);
                kg = 0;
              }
            }
            mma_commit_pair(empty(st.idx));
            st.next(kS);
          }
        }
        mma_commit_pair(drain);
        wait_bounded(drain, 0, p.error, nullptr, p.timeout_ns);
      }
      __syncwarp();
    } else if (p.jobs) {
      // ------------------------------------------- packing (both CTAs)
      pack_strips<KIND, SPLIT>(
          p, reinterpret_cast<float*>(smem + G::PACK + (warp - 2) * kPackBufs * kPackBytes), lane,
          abort);
    }
  } else {
    // -------------------------------------------- epilogue (both CTAs)
    regs_grow<kRegsEpi>();
    const int q = warp & 3;  // TMEM lanes 32q .. 32q + 31
    const int half = (warp - kEpiWarp0) >> 2;
    Ring acc, sc;
    const float alpha = p.alpha, beta = p.beta;
    // Reads the next schedule slot (lane 0) and acknowledges it to the
    // leader.  The acknowledgment is a cluster-scope release, which waits for
    // this lane's earlier global stores; so the next item is fetched before a
    // tile's C stores, never right after them.
    auto fetch = [&]() {
      int v = -1;
      if (lane == 0) {
        // the peer's slots are written by the leader's producer (release.cluster)
        const bool got = leader ? wait_bounded(sfull(sc.idx), sc.phase, p.error, abort,
                                               p.timeout_ns)
                                : wait_bounded_cluster(sfull(sc.idx), sc.phase, p.error, abort,
                                                       p.timeout_ns);
        if (got) {
          v = slots[sc.idx];
          mbar_arrive_cluster(mapa_shared(sempty(sc.idx), 0));
        }
      }
      sc.next(kSched);
      return __shfl_sync(0xffffffffu, v, 0);
    };
    int it = fetch();
    while (it >= 0) {
      const TileItem ti = p.items[it];
      const MatDesc d = p.descs[ti.mat];
      float* C = p.C[ti.mat];
      const int bn = tc2_cfg_bn(d.cfg);
      const bool swap = tc_cfg_swap(d.cfg);
      const int row0 = ti.tm * 256 + (int)rank * kRows + q * 32;  // A-side row of lane 0
      const long long ldc = d.ldc;
      const int c_lo = half * kCols;
      const int ncols = max(0, min(kCols, tile_n(d, ti.tn, bn) - c_lo));
      const int col_base = ti.tn * bn + c_lo;
      if constexpr (!BETA) {
        // (never taken: this form is launched with beta = 0; the guarded
        // tile-start prefetch keeps its code as measured fastest)
        if (beta != 0.0f) c_prefetch<kCols>(C, ldc, d.M, d.N, swap, row0, col_base, ncols, lane);
      }
      const int nk = (d.K + KE - 1) / KE;
      const int nsub = (d.K + KE / NSUB - 1) / (KE / NSUB);
      const int gs = SPLIT ? group_slices(p, d.K) : 1;
      const int ngroups = !SPLIT ? (nk > 0 ? 1 : 0) : gs == 0 ? nsub : (nk + gs - 1) / gs;
      float r[kCols];
#pragma unroll
      for (int j = 0; j < kCols; ++j) r[j] = 0.0f;
      int ok = 1;
      // beta != 0: C is pulled into L2 kCPrefetchLead groups before the tile
      // ends (earlier, the operand stream evicts it again before c_store)
      const int g_pf = (BETA && kCPrefetchLead > 0) ? max(0, ngroups - kCPrefetchLead) : -1;
      if (BETA && kCPrefetchLead > 0 && ngroups == 0)
        c_prefetch<kCols>(C, ldc, d.M, d.N, swap, row0, col_base, ncols, lane);
      // buffers of up to P = 256 / bn promotion groups each (see the MMA lane);
      // the groups are added in K order, as if each had a buffer of its own
      const int P = SPLIT ? 256 / bn : 1;
      for (int g0 = 0; g0 < ngroups; g0 += P) {
        if (lane == 0) ok = wait_bounded(tfull(acc.idx), acc.phase, p.error, abort, p.timeout_ns);
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (!ok) break;
        tc_fence_after();
        const int nsubs = min(P, ngroups - g0);
        for (int sg = 0; sg < nsubs; ++sg) {
          if (BETA && g0 + sg == g_pf)
            c_prefetch<kCols>(C, ldc, d.M, d.N, swap, row0, col_base, ncols, lane);
          const uint32_t tb =
              tmem + ((uint32_t)(q * 32) << 16) + acc.idx * 256u + (uint32_t)(sg * bn) + c_lo;
#pragma unroll
          for (int c = 0; c < kCols / 16; c += 2) {
            if (c * 16 < ncols) {
              float v0[16], v1[16];
              tmem_ld16(tb + c * 16, v0);
              tmem_ld16(tb + (c + 1) * 16, v1);
              tmem_wait_ld();
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                r[c * 16 + j] += v0[j];
                r[(c + 1) * 16 + j] += v1[j];
              }
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster_relaxed(mapa_shared(tempty(acc.idx), 0));
        acc.next(kNAcc);
      }
      if (!ok) break;
      it = fetch();
      if constexpr (BETA)
        c_store_pipe<kCols, 8>(r, C, ldc, d.M, d.N, swap, row0, col_base, ncols, alpha, beta, lane);
      else
        c_store<kCols>(r, C, ldc, d.M, d.N, swap, row0, col_base, ncols, alpha, beta, lane);
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync();
  tc_fence_after();
  if (warp == 1) tmem_dealloc_pair(tmem, 512);
  if (leader) {
    // the last cluster to finish resets the queues for the next launch (every
    // leader has pulled its final item, and every packing warp published its
    // last strip, before it gets here)
    if (threadIdx.x == 0) {
      __threadfence();
      const unsigned prev = atomicAdd(reinterpret_cast<unsigned*>(p.counters) + 1, 1u);
      const bool last = prev == (unsigned)ncl - 1;
      if (last) {
        atomicExch(p.counters, 0);
        atomicExch(p.counters + 1, 0);
        atomicExch(p.counters + 2, 0);
        __threadfence();
      }
      slots[0] = last ? 1 : 0;
    }
    if (p.jobs && *p.n_head < *p.n_jobs) {
      __syncthreads();
      if (slots[0])
        for (int i = threadIdx.x; i < p.n_ready; i += kThreads2) p.ready[i] = 0;
    }
  }
  if (p.cta_times && threadIdx.x == 0) p.cta_times[2 * blockIdx.x + 1] = gtimer();
}

// As bounded_wait_selftest_kernel (tc_kernel.cu), of wait_packed.
__global__ void packed_wait_selftest_kernel(int* err, int* out, unsigned long long limit_ns) {
  __shared__ int abort_flag;
  if (threadIdx.x == 0) {
    abort_flag = 0;
    out[1] = wait_packed(out + 2, 1, err, &abort_flag, limit_ns) ? 1 : 0;
    out[0] = 1;
  }
}

template <int KIND, int SPLIT, bool BETA>
cudaError_t launch2(const TcGemmParams& p, int grid, cudaStream_t s) {
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(tc2_gemm_kernel<KIND, SPLIT, BETA>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         Geo2<SPLIT>::SMEM);
    if (e != cudaSuccess) return e;
    attr = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid, 1, 1);
  cfg.blockDim = dim3(kThreads2, 1, 1);
  cfg.dynamicSmemBytes = Geo2<SPLIT>::SMEM;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, tc2_gemm_kernel<KIND, SPLIT, BETA>, p);
}

template <int KIND, int SPLIT>
cudaError_t launch2b(const TcGemmParams& p, int grid, cudaStream_t s) {
  return p.beta != 0.0f ? launch2<KIND, SPLIT, true>(p, grid, s)
                        : launch2<KIND, SPLIT, false>(p, grid, s);
}

}  // namespace

cudaError_t tc2_gemm_launch(int kind, int split, const TcGemmParams& p, int grid,
                            cudaStream_t s) {
  if (grid < 2 || (grid & 1)) return cudaErrorInvalidValue;
  if (kind == kKindTF32 && !split) return launch2b<kKindTF32, 0>(p, grid, s);
  if (kind == kKindTF32) return launch2b<kKindTF32, 1>(p, grid, s);
  if (kind == kKindBF16 && split) return launch2b<kKindBF16, 1>(p, grid, s);
  return cudaErrorInvalidValue;
}

cudaError_t tc2_wait_selftest_launch(int* err, int* out, unsigned long long limit_ns,
                                     cudaStream_t s) {
  packed_wait_selftest_kernel<<<1, 32, 0, s>>>(err, out, limit_ns);
  return cudaGetLastError();
}

int tc2_max_clusters() {
  int n = 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2, 1, 1);
  cfg.blockDim = dim3(kThreads2, 1, 1);
  cfg.dynamicSmemBytes = kSmemMax;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaFuncSetAttribute(tc2_gemm_kernel<kKindTF32, 1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       kSmemMax);
  if (cudaOccupancyMaxActiveClusters(&n, tc2_gemm_kernel<kKindTF32, 1, true>, &cfg) != cudaSuccess)
    return 0;
  return n;
}

}  // namespace bgemm
