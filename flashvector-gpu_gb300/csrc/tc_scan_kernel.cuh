// tc_scan_kernel.cuh -- the tcgen05 scan kernel template shared by the fp16
// and fp8 translation units (tc_scan_fp16.cu, tc_scan_fp8.cu), which each
// instantiate one precision so the two compile in parallel.
//
// Warp roles (64 + 128 G threads, one CTA per SM; G = 1, 2 or 4 epilogue
// groups, see below):
//   warp 0    TMA producer: per K block, a 128-query tile (A) and a 256-row
//             base tile (B), 128-byte-swizzled, into a STAGES-deep ring;
//   warp 1    TMEM owner + single-thread tcgen05.mma issuer (M=128, N=256,
//             fp32 accumulators, two 256-column buffers so the epilogue of
//             tile i overlaps the MMAs of tile i+1);
//   warps 2.. epilogue, 4 warps per group: thread r of a group owns query r
//             of the block (TMEM lane r),
//             turns dot products into distances, applies the slot mask and
//             keeps that query's best kl (distance, slot) keys: appended to a
//             list where an admission bound is known, else in a shared-memory
//             max-heap. No distance matrix ever reaches HBM.
//
// Shared bound (scans without an admission bound). Every query owns kl global "slots"; a CTA that keeps a key
// also lowers slot hash(row) of its query to the key's distance (red.min).
// Each slot then holds a distance of a distinct real row, so the maximum
// over the kl slots is >= the query's global kl-th best distance: a row
// farther than it cannot be in the shortlist, and every CTA scanning the
// query drops it. The maximum sits near rank kl * H(kl) of all rows scanned
// so far, so after the first tiles almost no row reaches the heap.
#pragma once

#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include <type_traits>

#include "common.cuh"
#include "kernels.h"
#include "tc_ptx.cuh"
#include "topk.cuh"

namespace fv {

constexpr int TC_M = 128;                  // queries per CTA (TMEM lanes)
constexpr int TC_N = 256;                  // base rows per tile (MMA N)
constexpr int RUN = 8;                     // consecutive rows of a minima-pass tile
constexpr int RUNS = TC_N / RUN;           // runs of a minima-pass tile
constexpr int KB_BYTES = 128;              // K bytes per stage row (one 128B swizzle atom)
constexpr int A_STAGE = TC_M * KB_BYTES;   // 16 KB
constexpr int B_STAGE = TC_N * KB_BYTES;   // 32 KB

// threads of a scan CTA with G epilogue groups: warp 0 TMA, warp 1 MMA,
// 4 epilogue warps per group
__host__ __device__ constexpr int scan_threads(int G) { return 64 + 128 * G; }

struct TcScanArgs {
  uint32_t n, nq, kblocks, nqb, splits;
  const float* xnorm;    // [n] ||x||^2 of the fp32 rows (L2, cosine)
  const float* xscale;   // [n] per-row fp8 scale (FP8 only)
  const float* qnorm;    // [nq] ||q||^2
  const float* qscale;   // [nq] per-query fp8 scale (FP8 only)
  const uint32_t* mask;
  uint64_t* partial;     // [nq][splits][kl]
  uint32_t* tslot;       // [nq][tslot_stride] shared-bound slots (float_order distances)
  uint32_t tslot_stride; // kl rounded up to a multiple of 4 (padding slots hold 0)
  uint32_t kl;           // heap entries used (<= KL); == shortlist when the bound is shared
  uint32_t share;        // 1: the CTAs of a query share the slot bound (kl == shortlist)
  uint32_t* status;
  const QueryFilter* filters;  // per-query filters over slots (== logical ids), or null
  const float* qbound;         // per-query admission bound (distance), or null
  const uint32_t* active;      // per-query flags: only flagged queries are scanned (null: all)
  float floor;                 // L2: lower limit of a distance (0, or -inf for a ranking value that may be negative)
  uint64_t wait_ns;            // limit of the pipeline's waits (the drains keep their own)
  // minima pass only (PASS_MIN): scans every run_stride-th run of RUN rows (a
  // sample when > 1), 256 / RUN runs to a tile; the smallest distance of `gran`
  // columns (8, 16, 32, 64 or 128), [nq][pm_stride], in tile order
  uint32_t run_stride;
  float* pmin;
  uint32_t pm_stride, gran;
};

enum { PASS_HEAP = 0, PASS_MIN = 1, PASS_LIST = 2 };
// heap capacities that select the passes without shared-memory heaps
constexpr int kMinima = 0, kLists = -1;

// PAIR: a CTA of a cta_group::2 pair holds half of each 256-row base tile.
// NCOL: per-column arrays that the epilogue stages (norms, scales, cosine's
// factors; none in the fused fp8 forms, whose accumulator is the ranking
// value). A_STAGES: query-tile buffers (1 where the query tile is always
// resident).
template <int KL, int STAGES, int G, bool PAIR = false, int NCOL = 2, int A_STAGES = STAGES>
struct ScanSmem {
  static constexpr size_t b_stage = PAIR ? B_STAGE / 2 : B_STAGE;
  static constexpr size_t a_off = 0;
  static constexpr size_t b_off = a_off + (size_t)A_STAGES * A_STAGE;
  static constexpr size_t heap_off = b_off + (size_t)STAGES * b_stage;
  static constexpr size_t col_off = heap_off + (size_t)G * KL * TC_M * 8;  // [4G warps][NCOL][TC_N] floats
  static constexpr size_t cmask_off = col_off + (size_t)4 * G * NCOL * TC_N * 4;  // [4G warps][8] words
  static constexpr size_t bar_off = cmask_off + 4 * G * 8 * 4;          // barriers
  static constexpr size_t nbars = 2 * STAGES + 5;
  static constexpr size_t misc_off = bar_off + nbars * 8;
  static constexpr size_t bytes = misc_off + 16 + 1024;                 // + alignment slack
};

// The fused fp8 forms (table scale, L2 / inner product): the accumulator is
// the ranking value, so no column data is staged.
template <bool FP8, int METRIC, bool TS>
constexpr bool kFusedScan = FP8 && TS && METRIC != METRIC_COSINE;

// G = 4 runs only the fused fp8 forms with one K block per tile, whose query
// tile is resident: one query-tile buffer.
template <bool FP8, int KL, int STAGES, int METRIC, int G, bool PAIR, bool TS>
using ScanLayout = ScanSmem<KL, STAGES, G, PAIR, kFusedScan<FP8, METRIC, TS> ? 0 : FP8 && METRIC == METRIC_COSINE ? 3 : 2,
                            G == 4 ? 1 : STAGES>;

// Sift `key` down from position i of a max-heap of kl keys stored with stride
// HS (TC_M in shared memory, one heap per query row of the block; 1 in global
// memory).
template <int HS>
static __device__ __forceinline__ void heap_down(uint64_t* h, int kl, int i, uint64_t key) {
  while (true) {
    int l = 2 * i + 1;
    if (l >= kl) break;
    uint64_t cv = h[l * HS];
    int c = l;
    if (l + 1 < kl) {
      uint64_t rv = h[(l + 1) * HS];
      if (rv > cv) { cv = rv; c = l + 1; }
    }
    if (cv <= key) break;
    h[i * HS] = cv;
    i = c;
  }
  h[i * HS] = key;
}

// Turns kl unordered keys into a max-heap (bottom-up).
template <int HS>
static __device__ __forceinline__ void heap_build(uint64_t* h, int kl) {
  for (int i = kl / 2 - 1; i >= 0; --i) heap_down<HS>(h, kl, i, h[i * HS]);
}

// A range's list that has just filled (or is full): its heap, the rare part
// of a bounded scan, out of the way of the common one. Returns the distance of
// the worst key kept.
static __device__ __noinline__ float list_full(uint64_t* list, int kl, uint64_t key, bool build) {
  if (build)
    heap_build<1>(list, kl);
  else
    heap_down<1>(list, kl, 0, key);  // replaces the root
  return key_dist(list[0]);
}

// v[j] for a lane-varying j without local memory: a 5-level select tree.
static __device__ __forceinline__ float select32(const float* v, int j) {
  float t[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) t[i] = (j & 1) ? v[2 * i + 1] : v[2 * i];
#pragma unroll
  for (int i = 0; i < 8; ++i) t[i] = (j & 2) ? t[2 * i + 1] : t[2 * i];
#pragma unroll
  for (int i = 0; i < 4; ++i) t[i] = (j & 4) ? t[2 * i + 1] : t[2 * i];
#pragma unroll
  for (int i = 0; i < 2; ++i) t[i] = (j & 8) ? t[2 * i + 1] : t[2 * i];
  return (j & 16) ? t[1] : t[0];
}

// G epilogue groups, each with its own heaps, dumped as separate lists
// (partial row split * G + g). With G = 2 both groups drain every tile, group
// g the columns [128 g, 128 g + 128) of it, so the MMA of tile i + 1 (the
// other accumulator buffer) runs while tile i is drained.
//
// G = 4 (fused fp8 with one K block per tile, shortlists above 48 keys; that
// call's minima pass runs G = 2): 16 epilogue warps, group g draining the
// 32-column chunks g and g + 4 of every tile. Heaps of at most 32 keys fit
// four groups' heaps in shared memory; interleaved chunks spread runs of
// consecutive slots over the groups.
//
// PAIR: the CTA is one of a cluster of two (a cta_group::2 pair) sharing the
// same base range: CTA r holds query block 2p + r and rows [128 r, 128 r +
// 128) of every 256-row tile; the even CTA issues M=256 MMAs whose 128
// accumulator lanes land in each CTA's TMEM, so each SM streams 16 KB of
// base per K block instead of 32 KB and the ring gets deeper. Both CTAs'
// TMA loads count on the even CTA's full barriers; the even CTA's commits
// are multicast to both CTAs' barriers; the odd CTA's epilogue arrives on
// the even CTA's accumulator barriers.
//
// PASS_HEAP: the heaps live in shared memory (a scan without a bound, where
// every range keeps replacing its worst key).
// PASS_LIST: a bounded scan, whose ranges hold a few keys and seldom fill: a
// range's keys are appended to its list in the output itself, which becomes a
// heap only when it fills. The 64 to 128 KB of shared memory that four groups'
// heaps took hold base tiles instead: with two stages the ring could not
// cover the latency of a tile.
// PASS_MIN: the pass that finds every query's admission bound. No heaps: the
// epilogue reduces each tile's accumulators to the smallest distance of every
// `gran` columns and stores those, so its cost per tile is the minimum tree
// alone and the freed shared memory holds a deeper ring. The r-th smallest
// of a query's minima is >= the r-th smallest distance scanned (minima of
// disjoint columns are distances of distinct rows), so it bounds from above. It
// is a tight bound while the r best rows lie in nearly as many minima, and bases
// are often stored in an order that keeps a query's best rows together. So a
// tile is 32 runs of 8 rows, spread evenly over the base (whole sectors of norms
// and bytes of masks still), and a minimum of 8 or 16 columns takes one row of
// each run. (Tiles of 256 consecutive rows and minima of consecutive columns:
// 1,000,000 x 96 fp16 stored by cluster, 500 queries, L2, k 10: 1,235 us a call,
// 523 with the runs.)
// Keeping the sample's best r keys in heaps instead spent the pass filling
// them: 123 us for 1/32 of a 1M x 768 scan of 1,024 queries.
template <bool FP8, int KL, int STAGES, int METRIC, int G, bool PAIR, bool TS, int PASS>
__global__ void __launch_bounds__(scan_threads(G), 1)
    tc_scan_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, TcScanArgs a) {
  constexpr bool MINP = PASS == PASS_MIN;
  constexpr int HS = PASS == PASS_LIST ? 1 : TC_M;  // stride of a range's keys
  using L = ScanLayout<FP8, KL, STAGES, METRIC, G, PAIR, TS>;
  constexpr uint32_t b_stage = (uint32_t)L::b_stage;
  constexpr int SCAN_THREADS = scan_threads(G);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sA = sm + L::a_off;
  uint8_t* sB = sm + L::b_off;
  uint64_t* heap = reinterpret_cast<uint64_t*>(sm + L::heap_off);
  float* colbuf = reinterpret_cast<float*>(sm + L::col_off);
  uint32_t* colmask = reinterpret_cast<uint32_t*>(sm + L::cmask_off);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + L::bar_off);
  uint64_t* full = bars;
  uint64_t* empty = bars + STAGES;
  uint64_t* acc_full = bars + 2 * STAGES;
  uint64_t* acc_empty = acc_full + 2;
  uint64_t* mma_done = acc_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + L::misc_off);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t qb, split, rank = 0;
  if constexpr (PAIR) {
    rank = tc::cluster_ctarank();
    const uint32_t c = blockIdx.x >> 1, npairs = (a.nqb + 1) / 2;
    qb = 2 * (c % npairs) + rank;
    split = c / npairs;
  } else {
    qb = blockIdx.x % a.nqb;
    split = blockIdx.x / a.nqb;
  }
  if (!PAIR && a.active) {
    // a re-scan of flagged queries: a block holding none of them leaves at once
    int any = 0;
    for (int r = threadIdx.x; r < TC_M; r += SCAN_THREADS) {
      const uint32_t q = qb * TC_M + r;
      any |= (q < a.nq && a.active[q]) ? 1 : 0;
    }
    if (!__syncthreads_or(any)) return;
  }
  constexpr bool col_split = G >= 2;
  const uint32_t ntiles = MINP ? a.n / (TC_N * a.run_stride) : (a.n + TC_N - 1) / TC_N;
  // A range is every splits-th tile, so that rows which a base's order keeps
  // together are shared out over the ranges, their lists and their threads. (1M x
  // 96 as above: 523 us a call with ranges of consecutive tiles, 274 like this;
  // 200,000 x 768 by cluster, 512 queries, k 100: 2,204, and three quarters of
  // the best 100 found, to 802 and all of them.)
  const uint32_t my_tiles = split < ntiles ? (ntiles - split - 1) / a.splits + 1 : 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(&acc_full[b], 1);
      // the epilogue warps (of both CTAs) that drain buffer b
      tc::mbar_init(&acc_empty[b], PAIR ? 8 : (col_split ? 4 * G : 4));
    }
    tc::mbar_init(mma_done, 1);
    *abort_flag = 0;
    tc::fence_mbar_init();
  }
  if (warp == 1) {
    if constexpr (PAIR)
      tc::tmem_alloc_pair(tmem_slot, 512);
    else
      tc::tmem_alloc(tmem_slot, 512);
    tc::tc_fence_before();
  }
  __syncthreads();
  if constexpr (PAIR) tc::cluster_sync();  // both CTAs' barriers exist before either signals the other's
  tc::tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  // K blocks that fit the query-tile buffers: the query tile is loaded once
  // (block kb with the first base tile's, into buffer kb) and stays resident;
  // only base tiles stream after it (with two K blocks and the query tile
  // reloaded, a third of the L2 traffic was query tiles)
  constexpr uint32_t A_BUFS = G == 4 ? 1 : STAGES;
  const bool a_resident = !PAIR && a.kblocks <= A_BUFS;

  if (warp == 0) {
    // ------------------------------------------------------ TMA producer
    if (lane == 0) {
      tc::prefetch_tmap(&tmA);
      tc::prefetch_tmap(&tmB);
      const uint64_t pol_a = tc::policy_evict_last();
      const uint64_t pol_b = tc::policy_evict_first();
      const int kb_elems = FP8 ? 128 : 64;
      uint32_t stage = 0, phase = 0;
      int32_t issued_parity[STAGES];
#pragma unroll
      for (int s = 0; s < STAGES; ++s) issued_parity[s] = -1;
      bool ok = true;
      for (uint32_t i = 0; ok && i < my_tiles; ++i) {
        const int32_t tile_b = (int32_t)(split + i * a.splits), row_b = tile_b * TC_N;
        for (uint32_t kb = 0; kb < a.kblocks; ++kb) {
          if (!tc::mbar_wait(&empty[stage], phase ^ 1, abort_flag, a.status, a.wait_ns)) {
            ok = false;
            break;
          }
          if constexpr (PAIR) {
            const uint32_t fb = tc::mapa(tc::smem_addr(&full[stage]), 0);  // the even CTA's full barrier
            if (rank == 0) tc::mbar_arrive_expect_tx(&full[stage], 2 * (A_STAGE + b_stage));
            tc::tma_load_2d_pair(sA + stage * A_STAGE, &tmA, fb, (int32_t)(kb * kb_elems), (int32_t)(qb * TC_M),
                                 pol_a);
            if constexpr (MINP)
              tc::tma_load_4d_pair(sB + stage * b_stage, &tmB, fb, (int32_t)(kb * kb_elems), 0, tile_b,
                                   (int32_t)(rank * (RUNS / 2)), pol_b);
            else
              tc::tma_load_2d_pair(sB + stage * b_stage, &tmB, fb, (int32_t)(kb * kb_elems),
                                   row_b + (int32_t)(rank * (TC_N / 2)), pol_b);
          } else {
            const bool load_a = !a_resident || i == 0;
            tc::mbar_arrive_expect_tx(&full[stage], (load_a ? A_STAGE : 0) + B_STAGE);
            if (load_a)
              tc::tma_load_2d(sA + (a_resident ? kb : stage) * A_STAGE, &tmA, &full[stage], (int32_t)(kb * kb_elems),
                              (int32_t)(qb * TC_M), pol_a);
            if constexpr (MINP)
              tc::tma_load_4d(sB + stage * B_STAGE, &tmB, &full[stage], (int32_t)(kb * kb_elems), 0, tile_b, 0, pol_b);
            else
              tc::tma_load_2d(sB + stage * B_STAGE, &tmB, &full[stage], (int32_t)(kb * kb_elems), row_b, pol_b);
          }
          issued_parity[stage] = (int32_t)phase;
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      // drain: every copy issued must have landed before the CTA may exit
      // (normally they all have; after an abort this waits a bounded time).
      // A pair's copies all count on the even CTA's barriers, which it drains.
      uint32_t no_abort = 0;
      if (!PAIR || rank == 0) {
#pragma unroll
        for (int s = 0; s < STAGES; ++s)
          if (issued_parity[s] >= 0)
            tc::mbar_wait(&full[s], (uint32_t)issued_parity[s], &no_abort, a.status, 100000000ull);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------- MMA issuer
    if (lane == 0 && (!PAIR || rank == 0)) {
      constexpr uint32_t idesc = tc::idesc_f32acc(0, 0, PAIR ? 2 * TC_M : TC_M, TC_N);
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      for (uint32_t i = 0; ok && i < my_tiles; ++i) {
        const uint32_t buf = i & 1, use = i >> 1;
        if (!tc::mbar_wait(&acc_empty[buf], (use & 1) ^ 1, abort_flag, a.status, a.wait_ns)) break;
        tc::tc_fence_after();
        const uint32_t d_tmem = tmem + buf * TC_N;
        for (uint32_t kb = 0; kb < a.kblocks; ++kb) {
          if (!tc::mbar_wait(&full[stage], phase, abort_flag, a.status, a.wait_ns)) {
            ok = false;
            break;
          }
          tc::tc_fence_after();
          const uint32_t a_base = tc::smem_addr(sA + (a_resident ? kb : stage) * A_STAGE);
          const uint32_t b_base = tc::smem_addr(sB + stage * b_stage);
#pragma unroll
          for (uint32_t kk = 0; kk < 4; ++kk) {
            if constexpr (PAIR)
              tc::mma_pair<FP8>(d_tmem, tc::sdesc_k_sw128(a_base + kk * 32), tc::sdesc_k_sw128(b_base + kk * 32),
                                idesc, (kb | kk) != 0);
            else
              tc::mma<FP8>(d_tmem, tc::sdesc_k_sw128(a_base + kk * 32), tc::sdesc_k_sw128(b_base + kk * 32), idesc,
                           (kb | kk) != 0);
          }
          if constexpr (PAIR)
            tc::mma_commit_pair(&empty[stage], 3);
          else
            tc::mma_commit(&empty[stage]);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (ok) {
          if constexpr (PAIR)
            tc::mma_commit_pair(&acc_full[buf], 3);
          else
            tc::mma_commit(&acc_full[buf]);
        }
      }
      if constexpr (PAIR)
        tc::mma_commit_pair(mma_done, 3);
      else
        tc::mma_commit(mma_done);
    }
  } else {
    // --------------------------------------------------------- epilogue
    const int quad = warp & 3;                    // TMEM lane quadrant of this warp
    const int grp = (warp - 2) >> 2;              // epilogue group
    const int row = quad * 32 + lane;             // query row in the block
    const uint32_t q = qb * TC_M + row;
    const bool qvalid = q < a.nq && (a.active == nullptr || a.active[q] != 0u);
    const int kl = MINP ? 0 : (int)a.kl;
    uint64_t* const list = a.partial + (((size_t)q * a.splits + split) * G + grp) * kl;  // this range's output
    uint64_t* h = PASS == PASS_LIST ? list : heap + (size_t)grp * KL * TC_M + row;
    if (PASS == PASS_HEAP)
      for (int i = 0; i < kl; ++i) h[i * HS] = kSentinelKey;
    const float qn = qvalid ? __ldg(a.qnorm + q) : 0.f;
    const QueryFilter qf = (a.filters && qvalid) ? load_filter(a.filters, q) : QueryFilter{nullptr, 0u, 0u};
    const float qs = (FP8 && qvalid) ? __ldg(a.qscale + q) : 1.f;
    // fp8 L2 and inner product over a table-scale table: the accumulator is
    // the ranking value in the table's units (L2: the norm digits fold
    // -||x||^2 / (2 s s_q) into the dot product), v = sc * acc with
    // sc = -2 s s_q (L2) or -s s_q (IP), a power of two, so the scaling is
    // exact and no per-row data is read. A per-row-scale table reads each
    // row's scale (and norm) per value instead.
    constexpr bool fused = FP8 && METRIC != METRIC_COSINE && TS;
    const float sc = fused ? (METRIC == METRIC_L2 ? -2.0f : -1.0f) * qs * __ldg(a.xscale) : 1.f;
    const float inv_sc = fused ? __fdiv_rn(1.0f, sc) : 1.f;
    float worst = kSentinelDist;  // this CTA's kl-th best distance (1e30 until the heap is full)
    // admission bound: the query's pre-pass bound, lowered by the shared slots
    float bound = (a.qbound && qvalid) ? __ldg(a.qbound + q) : kSentinelDist;
    uint32_t* slots = (!MINP && a.share && qvalid) ? a.tslot + (size_t)q * a.tslot_stride : nullptr;

    // Until kl keys are held the heap is an unordered list (appends cost
    // one store); on the kl-th key it is heapified once and from then on a
    // key replaces the root. The kept set is the same either way.
    int fill = 0;
    auto keep = [&](float dist, uint32_t slot) {
      const uint64_t key = make_key(dist, slot);
      if constexpr (PASS == PASS_LIST) {
        // (worst stays at 1e30, and the threshold where it is, until it fills)
        if (fill < kl) {
          h[fill] = key;
          if (++fill < kl) return;
          worst = list_full(h, kl, key, true);
        } else {
          worst = list_full(h, kl, key, false);
        }
        return;
      }
      if (fill < kl) {
        h[fill * HS] = key;
        if (++fill == kl) {
          heap_build<HS>(h, kl);
          worst = key_dist(h[0]);
        }
      } else {
        heap_down<HS>(h, kl, 0, key);  // replaces the root
        worst = key_dist(h[0]);
      }
      if (slots) atomicMin(slots + __umulhi(slot * 2654435761u, (uint32_t)kl), float_order(dist));
    };
    // admission threshold in the v domain, refreshed when worst or bound
    // moves: every v whose distance could enter (D(v) < worst and D(v) <=
    // bound) has v <= thr (for L2 the subtraction of the query norm is padded
    // by a relative slack, so thr errs on the admitting side; exact tests
    // follow). Fused fp8 tests the accumulator instead: v <= thr <=> acc >=
    // thr / sc (sc < 0, a power of two), padded the same way against underflow.
    //
    // Cosine: a division and a square root per value bounded the pass (64,931
    // x 859, 16 queries: 159 us a call, now 76). Where sqrt(|q|^2 |x|^2) >= 0.01 for a tile's
    // columns, v = -dot / |x| from a factor staged per column ranks within
    // kCosPad of the distance 1 + v / |q| (the factors' few ulps, and 1e-8
    // against 0.01), so v <= cthr, raised by it, admits every candidate and
    // the exact distance is evaluated for those alone. Nor does |q|^2 |x|^2
    // overflow for any of them: the distance would then be 1 at every angle. Rows
    // of zeros, whose distance is 1 too, have the factor 0 (|x|^2 underflows below
    // |x| = 1e-22: with |q| < 1e8 the dot is then nothing against the 1e-8). (600,000
    // x 64 with a row of zeros in most tiles, 200 queries: 626 us without that,
    // 225 with it.)
    constexpr float kCosPad = 4e-6f;
    const float q_over = METRIC == METRIC_COSINE ? sqrtf(qn) / (FP8 ? qs : 1.f) : 1.f;
    const float q_inv = METRIC == METRIC_COSINE ? __fdiv_rn(1.f, q_over) : 1.f;
    // the range of the warp's squared query norms
    [[maybe_unused]] float q_least = qvalid ? qn : INFINITY, q_most = qvalid ? qn : 0.f;
    if (METRIC == METRIC_COSINE) {
#pragma unroll
      for (int o = 16; o; o >>= 1) {
        q_least = fminf(q_least, __shfl_xor_sync(0xffffffffu, q_least, o));
        q_most = fmaxf(q_most, __shfl_xor_sync(0xffffffffu, q_most, o));
      }
    }
    // (A bound of -inf, where products overflowed, admits the rows at -inf: the
    // thresholds stay finite, or their slack would make them NaN.)
    constexpr float kLowest = -3.402823466e38f;
    float thr = 0.f, cthr = 0.f;
    auto refresh = [&]() {
      const float w = fmaxf(fminf(worst, bound), kLowest);
      thr = METRIC == METRIC_L2 ? (w - qn) + 1e-6f * (fabsf(w) + fabsf(qn)) + 1e-30f : w;
      if (METRIC == METRIC_COSINE) {
        cthr = fmaxf((w - 1.0f + kCosPad) * q_over, kLowest);
        cthr += 1e-6f * fabsf(cthr);
      }
      if (fused) {
        thr *= inv_sc;
        thr -= 1e-6f * fabsf(thr) + 1e-37f;
      }
    };

    // per-warp copy of the current tile's column data (norms, fp8 factors,
    // mask words): staged by the warp itself, so the epilogue warps never
    // wait on one another. The global loads for tile i + 1 are issued into
    // registers while tile i is processed (lane l holds columns l + 32 r).
    constexpr int kCols = kFusedScan<FP8, METRIC, TS> ? 0 : FP8 && METRIC == METRIC_COSINE ? 3 : 2;
    float* cb = colbuf + (warp - 2) * kCols * TC_N;
    float* cf = cb + (kCols - 1) * TC_N;  // cosine: -1 / |x| (times the row's scale)
    uint32_t* cm = colmask + (warp - 2) * 8;
    // this group's columns [c_lo, c_hi) of each tile; only its own columns'
    // data is staged
    const int c_lo = col_split ? grp * (TC_N / G) : 0;
    const int c_hi = col_split ? c_lo + TC_N / G : TC_N;
    float pre_n[TC_N / 32], pre_s[TC_N / 32];
    uint32_t pre_m = 0;
    // minima pass: the first row of run r of a tile
    auto run_row = [&](uint32_t tile, uint32_t r) { return RUN * a.run_stride * (tile + r * ntiles); };
    auto prefetch = [&](uint32_t tile) {
      const uint32_t v0n = tile * TC_N;
#pragma unroll
      for (int r = 0; r < TC_N / 32; ++r) {
        const uint32_t slot = MINP ? run_row(tile, (lane + 32 * r) / RUN) + lane % RUN : v0n + lane + 32 * r;
        const bool in = slot < a.n && 32 * r >= c_lo && 32 * r < c_hi;
        pre_n[r] = (METRIC != METRIC_INNER_PRODUCT && !fused && in) ? __ldg(a.xnorm + slot) : 0.f;
        // per-column factor of the scaled dot: -2 xs (L2), -xs (IP), xs
        // (cosine) for per-row scales; a table-scale table needs none
        const float xs = (FP8 && !fused && in) ? __ldg(a.xscale + slot) : 0.f;
        pre_s[r] = METRIC == METRIC_L2 ? -2.0f * xs : (METRIC == METRIC_INNER_PRODUCT ? -xs : xs);
      }
      pre_m = 0;
      if (MINP && lane < 8) {
        pre_m = 0xFFFFFFFFu;
        if (a.mask) {
          pre_m = 0;
#pragma unroll
          for (int b = 0; b < 32 / RUN; ++b) {
            const uint32_t row = run_row(tile, 32 / RUN * lane + b);
            pre_m |= ((__ldg(a.mask + (row >> 5)) >> (row & 31u)) & 0xFFu) << (RUN * b);
          }
        }
      } else if (lane < 8) {
        const uint32_t c0 = v0n + lane * 32;
        if (c0 < a.n) {
          const uint32_t cnt = min(32u, a.n - c0);
          pre_m = cnt == 32 ? 0xFFFFFFFFu : ((1u << cnt) - 1u);
          if (a.mask) pre_m &= __ldg(a.mask + (c0 >> 5));
        }
      }
    };
    if (my_tiles) prefetch(split);
    uint32_t tile = split;
    for (uint32_t i = 0; i < my_tiles; ++i, tile += a.splits) {
      const uint32_t buf = i & 1, use = i >> 1;
      const uint32_t v0 = tile * TC_N;
      __syncwarp();
      [[maybe_unused]] bool by_factor = true;  // cosine: all norms of the tile allow it
#pragma unroll
      for (int r = 0; r < TC_N / 32; ++r) {
        if (32 * r < c_lo || 32 * r >= c_hi) continue;
        if (METRIC != METRIC_INNER_PRODUCT && !fused) cb[lane + 32 * r] = pre_n[r];
        if (FP8 && !fused) cb[TC_N + lane + 32 * r] = pre_s[r];
        if (METRIC == METRIC_COSINE) {
          // (a row of zeros has the distance 1, the factor 0; a NaN passes, as it has
          // no distance either way)
          const bool zero = pre_n[r] == 0.f;
          cf[lane + 32 * r] = zero ? 0.f : -rsqrtf(pre_n[r]) * (FP8 ? pre_s[r] : 1.f);
          if (MINP || v0 + lane + 32 * r < a.n)
            by_factor = by_factor && (zero ? q_most < 1e16f : !(pre_n[r] * q_least < 1e-4f) && !(pre_n[r] * q_most >= 1e38f));
        }
      }
      if (METRIC == METRIC_COSINE) by_factor = __all_sync(0xffffffffu, by_factor);
      if (lane < 8) cm[lane] = pre_m;
      __syncwarp();
      if (i + 1 < my_tiles) prefetch(tile + a.splits);
      // the shared bound, loaded before the accumulator wait hides its latency
      uint32_t smax = 0;
      if (slots)
        for (uint32_t s4 = 0; s4 < a.tslot_stride; s4 += 4) {
          const uint4 w = __ldcg(reinterpret_cast<const uint4*>(slots + s4));
          smax = max(smax, max(max(w.x, w.y), max(w.z, w.w)));
        }
      if (!tc::mbar_wait(&acc_full[buf], use & 1, abort_flag, a.status, a.wait_ns)) break;
      tc::tc_fence_after();
      if (slots && smax != 0xFFFFFFFFu) bound = fminf(bound, order_float(smax));
      refresh();

      const uint32_t t_row = tmem + ((uint32_t)(quad * 32) << 16) + buf * TC_N;
      // hands the accumulator buffer back as soon as this warp's last values
      // are in registers, before they are looked at: a tile whose slowest warp
      // held candidates otherwise kept the next MMA waiting (10M x 96 fp8,
      // 10,000 queries: 16.9 ms, of which 6.3 were such waits)
      auto hand_back = [&]() {
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          // relaxed: the buffer's TMEM values are in registers (wait::ld); the
          // arrival must not wait for this lane's shared-bound red.min updates
          if (PAIR && rank != 0)
            tc::mbar_arrive_cluster_relaxed(tc::mapa(tc::smem_addr(&acc_empty[buf]), 0));
          else
            tc::mbar_arrive_relaxed(&acc_empty[buf]);
        }
      };
      if constexpr (G == 4) {
        // fused fp8, the group's 32-column chunks at 32 g and 128 + 32 g: the
        // accumulator is the ranking value (v = sc * acc, sc < 0), so a
        // larger accumulator is better; a chunk whose largest value cannot
        // enter is skipped whole
        auto chunk32 = [&](const uint32_t (&rr)[32], uint32_t col, uint32_t m32) {
          if (m32 == 0u) return;
          auto max3 = [](float x, float y, float z) {
            float d;
            asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(x), "f"(y), "f"(z));
            return d;
          };
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(rr[j]);
          float t1[11];
#pragma unroll
          for (int j = 0; j < 10; ++j) t1[j] = max3(v[3 * j], v[3 * j + 1], v[3 * j + 2]);
          t1[10] = fmaxf(v[30], v[31]);
          const float top = fmaxf(max3(max3(t1[0], t1[1], t1[2]), max3(t1[3], t1[4], t1[5]), max3(t1[6], t1[7], t1[8])),
                                  fmaxf(t1[9], t1[10]));
          if (!(top >= thr)) return;
          // (four chains of eight: one chain of 32 was most of the mask's latency)
          uint32_t p4[4] = {0u, 0u, 0u, 0u};
#pragma unroll
          for (int j = 0; j < 32; ++j) p4[j >> 3] |= (uint32_t)(v[j] >= thr) << j;
          uint32_t pass = ((p4[0] | p4[1]) | (p4[2] | p4[3])) & m32;
          while (pass) {
            const int j = __ffs(pass) - 1;
            pass &= pass - 1;
            const float x = select32(v, j) * sc;
            const float d = METRIC == METRIC_L2 ? fmaxf(0.f, qn + x) : x;
            if (d < worst && d <= bound) {
              keep(d, v0 + col + (uint32_t)j);
              if (PASS != PASS_LIST) refresh();
            }
          }
        };
        uint32_t ra[32], rb[32];
        const uint32_t col = 32u * (uint32_t)grp;
        __syncwarp();  // tcgen05.ld is warp-collective: reconverge after the divergent insertions
        tc::tmem_ld32_async(t_row + col, ra);
        tc::tmem_ld32_async(t_row + 128u + col, rb);
        uint32_t ma = qvalid ? cm[col >> 5] : 0u, mb = qvalid ? cm[(128u + col) >> 5] : 0u;
        if (qf.words) {
          ma &= filter_word(qf, (v0 + col) >> 5);
          mb &= filter_word(qf, (v0 + 128u + col) >> 5);
        }
        tc::tmem_wait_ld(ra);
        tc::reg_fence(rb);
        hand_back();
        chunk32(ra, col, ma);
        chunk32(rb, 128u + col, mb);
      } else {
        [[maybe_unused]] float m[8];  // minima pass: of 128 columns (64 where gran is 8)
#pragma unroll 1
        for (int c0 = c_lo; c0 < c_hi; c0 += 64) {
          uint32_t ra[32], rb[32];
          __syncwarp();  // tcgen05.ld is warp-collective: reconverge after the divergent insertions
          tc::tmem_ld32_async(t_row + c0, ra);
          tc::tmem_ld32_async(t_row + c0 + 32, rb);
          uint64_t mw = qvalid ? ((uint64_t)cm[(c0 >> 5) + 1] << 32 | cm[c0 >> 5]) : 0ull;
          if (qf.words) {
            uint64_t fw = 0;
            if constexpr (MINP) {
#pragma unroll
              for (int b = 0; b < 64 / RUN; ++b) {
                const uint32_t row = run_row(tile, c0 / RUN + b);
                fw |= (uint64_t)((filter_word(qf, row >> 5) >> (row & 31u)) & 0xFFu) << (RUN * b);
              }
            } else {
              const uint32_t w0 = (v0 + (uint32_t)c0) >> 5;
              fw = ((uint64_t)filter_word(qf, w0 + 1) << 32) | filter_word(qf, w0);
            }
            mw &= fw;
          }
          tc::tmem_wait_ld(ra);
          tc::reg_fence(rb);
          if (c0 + 64 >= c_hi) hand_back();
          if (!MINP && mw == 0ull) continue;
          // the chunk's admission test and insertions; FU: the accumulator is
          // the ranking value (fp8 table-scale tables)
          // AP: cosine by the staged factors
          auto chunk = [&](auto fu_tag, auto ap_tag) {
            constexpr bool FU = decltype(fu_tag)::value, AP = decltype(ap_tag)::value;
            // per-column values v, v[0..32) columns c0.., v[32..64) columns
            // c0+32..; the distance is D(v): L2  D(v) = max(floor, ||q||^2 + v) with
            // v = ||x||^2 - 2 <q, x> (the query's norm is added after the
            // minimum, D being monotone), IP  D(v) = v = -<q, x>, cosine the
            // full expression. FP8 cosine dots carry the query and table scales.
            float v[64];
            if constexpr (FU) {
#pragma unroll
              for (int j = 0; j < 64; ++j) v[j] = __uint_as_float(j < 32 ? ra[j] : rb[j - 32]);
            } else if constexpr (AP) {
              const float4* fb = reinterpret_cast<const float4*>(cf + c0);
#pragma unroll
              for (int j4 = 0; j4 < 16; ++j4) {
                const float4 f4 = fb[j4];
                const float fv[4] = {f4.x, f4.y, f4.z, f4.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const int j = 4 * j4 + e;
                  v[j] = __uint_as_float(j < 32 ? ra[j] : rb[j - 32]) * fv[e];
                }
              }
            } else if (METRIC == METRIC_COSINE) {
#pragma unroll
              for (int j = 0; j < 64; ++j) {
                float dot = __uint_as_float(j < 32 ? ra[j] : rb[j - 32]);
                if (FP8) dot = dot * (qs * cb[TC_N + c0 + j]);
                v[j] = 1.0f - dot / (sqrtf(qn * cb[c0 + j]) + 1e-8f);
              }
            } else {
              const float4* nb = reinterpret_cast<const float4*>(cb + c0);
              const float4* sb = reinterpret_cast<const float4*>(cb + TC_N + c0);
#pragma unroll
              for (int j4 = 0; j4 < 16; ++j4) {
                const float4 n4 = METRIC == METRIC_L2 ? nb[j4] : make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 s4 = FP8 ? sb[j4] : make_float4(0.f, 0.f, 0.f, 0.f);
                const float nv[4] = {n4.x, n4.y, n4.z, n4.w};
                const float sv[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const int j = 4 * j4 + e;
                  const float dot = __uint_as_float(j < 32 ? ra[j] : rb[j - 32]);
                  if constexpr (FP8) {
                    // per-row scales: -2 xs (L2) or -xs (IP) in sv; two columns an
                    // instruction, each rounded as alone (10M x 96, 10,000 queries,
                    // L2: 36.3 ms a call one by one, 35.9 in pairs; IP 29.7 and 28.3)
                    if (e & 1) continue;
                    const float dot1 = __uint_as_float(j < 32 ? ra[(j + 1) & 31] : rb[(j + 1) & 31]);
                    const uint64_t d2 = tc::mul2(tc::pack2(dot, dot1), tc::pack2(qs, qs));
                    const uint64_t s2 = tc::pack2(sv[e], sv[e + 1]);
                    tc::unpack2(METRIC == METRIC_L2 ? tc::fma2(d2, s2, tc::pack2(nv[e], nv[e + 1])) : tc::mul2(d2, s2),
                                v[j], v[j + 1]);
                  } else {
                    v[j] = METRIC == METRIC_L2 ? fmaf(-2.0f, dot, nv[e]) : -dot;
                  }
                }
              }
            }
            // D: distance from v (fused fp8: from the accumulator, v = sc * acc;
            // cosine by factors: an upper bound)
            auto D = [&](float x) {
              if (AP) return fmaf(x, q_inv, 1.0f + kCosPad);
              if (FU) x *= sc;
              return METRIC == METRIC_L2 ? fmaxf(a.floor, qn + x) : x;
            };
            // better(x, y): the smaller v, i.e. the larger accumulator when fused
            auto better = [](float x, float y) { return FU ? fmaxf(x, y) : fminf(x, y); };
            auto may = [&](float x) { return FU ? x >= thr : x <= (AP ? cthr : thr); };
            // a tree of three-input bests: a 64-column batch whose best cannot
            // enter is skipped whole (the common case once warm); the pairwise
            // bests (j, j + 32) are formed only for a batch that passes
            // best of three in one instruction (three-input min / max)
            auto best3 = [](float x, float y, float z) {
              float d;
              if (FU)
                asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(x), "f"(y), "f"(z));
              else
                asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(x), "f"(y), "f"(z));
              return d;
            };
            if constexpr (MINP) {
              // the smallest distance of 8 columns, one of each run (none where the
              // mask admits none), then of `gran`: with the other 64 columns' runs
              // first, then of neighbours in a run. Columns whose product is NaN (an
              // fp16 row that overflowed times a zero, a NaN row) drop out of a
              // minimum: what starts it is no distance, not L2's floor.
              const float none = FU ? -INFINITY : INFINITY;
              if (mw != ~0ull) {
#pragma unroll
                for (int j = 0; j < 64; ++j) v[j] = ((mw >> j) & 1ull) ? v[j] : none;
              }
              if (a.gran == 8 || (c0 & 64) == 0) {
#pragma unroll
                for (int j = 0; j < 8; ++j) m[j] = none;
              }
#pragma unroll
              for (int j = 0; j < 8; ++j)
                m[j] = best3(best3(v[j], v[j + 8], v[j + 16]), best3(v[j + 24], v[j + 32], v[j + 40]),
                             best3(v[j + 48], v[j + 56], m[j]));
              if (!qvalid || (a.gran != 8 && (c0 & 64) == 0)) return;
              const uint32_t at = tile * TC_N + (uint32_t)c0;  // scanned column
              float* o = a.pmin + (size_t)q * a.pm_stride + (a.gran == 8 ? at : at & ~127u) / a.gran;
              if (a.gran <= 16) {
                reinterpret_cast<float4*>(o)[0] = make_float4(D(m[0]), D(m[1]), D(m[2]), D(m[3]));
                reinterpret_cast<float4*>(o)[1] = make_float4(D(m[4]), D(m[5]), D(m[6]), D(m[7]));
                return;
              }
              const float p0 = better(m[0], m[4]), p1 = better(m[1], m[5]), p2 = better(m[2], m[6]),
                          p3 = better(m[3], m[7]);
              if (a.gran == 32)
                *reinterpret_cast<float4*>(o) = make_float4(D(p0), D(p1), D(p2), D(p3));
              else if (a.gran == 64)
                *reinterpret_cast<float2*>(o) = make_float2(D(better(p0, p2)), D(better(p1, p3)));
              else
                *o = D(better(better(p0, p2), better(p1, p3)));
              return;
            } else {
            float r[22], s8[8];
#pragma unroll
            for (int i = 0; i < 21; ++i) r[i] = best3(v[3 * i], v[3 * i + 1], v[3 * i + 2]);
            r[21] = v[63];
#pragma unroll
            for (int i = 0; i < 7; ++i) s8[i] = best3(r[3 * i], r[3 * i + 1], r[3 * i + 2]);
            s8[7] = r[21];
            const float top = best3(best3(s8[0], s8[1], s8[2]), best3(s8[3], s8[4], s8[5]), better(s8[6], s8[7]));
            if (!(mw != 0ull && may(top))) return;
            float m1[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) m1[j] = better(v[j], v[j + 32]);
            // pairs (j, j+32) that may hold a candidate, walked lane-parallel
            uint32_t pass = 0;
#pragma unroll
            for (int j = 0; j < 32; ++j) pass |= (uint32_t)may(m1[j]) << j;
            pass &= (uint32_t)mw | (uint32_t)(mw >> 32);
            while (pass) {
              const int j = __ffs(pass) - 1;
              pass &= pass - 1;
              float dlo, dhi;
              if constexpr (AP) {
                auto exact = [&](const uint32_t (&rr)[32], int c) {
                  float f[32];
#pragma unroll
                  for (int t = 0; t < 32; ++t) f[t] = __uint_as_float(rr[t]);
                  float dot = select32(f, j);
                  if (FP8) dot = dot * (qs * cb[TC_N + c]);
                  return 1.0f - dot / (sqrtf(qn * cb[c]) + 1e-8f);
                };
                dlo = exact(ra, c0 + j);
                dhi = exact(rb, c0 + j + 32);
              } else {
                dlo = D(select32(v, j));
                dhi = D(select32(v + 32, j));
              }
              if (((mw >> j) & 1ull) && dlo < worst && dlo <= bound) {
                keep(dlo, v0 + c0 + j);
                refresh();
              }
              if (((mw >> (j + 32)) & 1ull) && dhi < worst && dhi <= bound) {
                keep(dhi, v0 + c0 + j + 32);
                refresh();
              }
            }
            }
          };
          if constexpr (METRIC == METRIC_COSINE) {
            if (by_factor)
              chunk(std::false_type{}, std::true_type{});
            else
              chunk(std::false_type{}, std::false_type{});
          } else {
            chunk(std::integral_constant<bool, fused>{}, std::false_type{});
          }
        }
      }
    }
    if (!MINP && qvalid) {
      // entry 0 of a dumped list is its largest key (the select kernel tests
      // it for overflow): a full heap has it there already; a list that never
      // filled gets one of its sentinels moved there
      if (fill > 0 && fill < kl) {
        h[fill * HS] = h[0];
        h[0] = kSentinelKey;
        ++fill;
      }
      if (PASS == PASS_LIST) {
        for (int i = fill; i < kl; ++i) h[i] = kSentinelKey;
      } else {
        for (int i = 0; i < kl; ++i) list[i] = h[i * HS];
      }
    }
  }

  __syncthreads();
  if (warp == 1) {
    // all MMAs must have retired before the accumulators are released; this
    // wait ignores the abort flag (bounded by time only)
    uint32_t no_abort = 0;
    tc::mbar_wait(mma_done, 0, &no_abort, a.status, 100000000ull);
    __syncwarp();
    tc::tc_fence_after();
    if constexpr (PAIR)
      tc::tmem_dealloc_pair(tmem, 512);
    else
      tc::tmem_dealloc(tmem, 512);
  }
  // a pair's CTAs read each other's shared memory (MMA operands, barriers):
  // neither leaves before the other is done
  if constexpr (PAIR) tc::cluster_sync();
}


template <bool FP8, int KL, int STAGES, int METRIC, int G, bool PAIR = false, bool TS = true, int PASS = PASS_HEAP>
cudaError_t launch_scan_kernel(const CUtensorMap& ta, const CUtensorMap& tb, const TcScanArgs& a, uint32_t grid,
                               cudaStream_t stream) {
  using L = ScanLayout<FP8, KL, STAGES, METRIC, G, PAIR, TS>;
  static_assert(L::bytes <= 227 * 1024, "scan shared memory above the 227 KB per-CTA limit");
  auto kern = tc_scan_kernel<FP8, KL, STAGES, METRIC, G, PAIR, TS, PASS>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::bytes);
  if (e != cudaSuccess) return e;
  if constexpr (PAIR) {
    // grid = 2 CTAs per (query-block pair, split), clusters of two
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(scan_threads(G), 1, 1);
    cfg.dynamicSmemBytes = L::bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, kern, ta, tb, a);
    note_launch();
    return e;
  }
  kern<<<grid, scan_threads(G), L::bytes, stream>>>(ta, tb, a);
  note_launch();
  return cudaGetLastError();
}

// groups == 2 (short K: one or two K blocks per tile, where the epilogue
// rather than the MMA bounds a tile) halves the stage ring and caps the heap
// at 48 entries so that two groups' heaps fit next to it; groups == 4 (fused
// fp8, one K block) caps it at 32. groups == -1 selects the CTA-pair
// variant (grid = 2 CTAs per cluster).
template <bool FP8, int METRIC, bool TS>
cudaError_t dispatch_scan_kl(int kl, int groups, const CUtensorMap& ta, const CUtensorMap& tb, const TcScanArgs& a,
                             uint32_t grid, cudaStream_t stream) {
  if (kl == kMinima) {
    if (groups == -1) return launch_scan_kernel<FP8, 0, 6, METRIC, 1, true, TS, PASS_MIN>(ta, tb, a, grid, stream);
    if (groups == 1) return launch_scan_kernel<FP8, 0, 4, METRIC, 1, false, TS, PASS_MIN>(ta, tb, a, grid, stream);
    return launch_scan_kernel<FP8, 0, 4, METRIC, 2, false, TS, PASS_MIN>(ta, tb, a, grid, stream);
  }
  if (kl == kLists) {
    if (groups == -1) return launch_scan_kernel<FP8, 0, 6, METRIC, 1, true, TS, PASS_LIST>(ta, tb, a, grid, stream);
    if (groups == 1) return launch_scan_kernel<FP8, 0, 4, METRIC, 1, false, TS, PASS_LIST>(ta, tb, a, grid, stream);
    if (groups == 2) return launch_scan_kernel<FP8, 0, 4, METRIC, 2, false, TS, PASS_LIST>(ta, tb, a, grid, stream);
    if constexpr (kFusedScan<FP8, METRIC, TS>)
      return launch_scan_kernel<FP8, 0, 6, METRIC, 4, false, TS, PASS_LIST>(ta, tb, a, grid, stream);
    return cudaErrorInvalidValue;
  }
  if (groups == -1) {
    // cta_group::2 pairs (one epilogue group): 16 KB of base per stage frees
    // room for 4-6 stages
    switch (kl) {
      case 16: return launch_scan_kernel<FP8, 16, 6, METRIC, 1, true, TS>(ta, tb, a, grid, stream);
      case 32: return launch_scan_kernel<FP8, 32, 5, METRIC, 1, true, TS>(ta, tb, a, grid, stream);
      case 48: return launch_scan_kernel<FP8, 48, 5, METRIC, 1, true, TS>(ta, tb, a, grid, stream);
      default: return launch_scan_kernel<FP8, 64, 4, METRIC, 1, true, TS>(ta, tb, a, grid, stream);
    }
  }
  if (groups == 4) {
    // fused fp8 with one K block per tile only (the layout keeps one
    // query-tile buffer); heaps of 16 or 32 keys
    if constexpr (kFusedScan<FP8, METRIC, TS>) {
      if (a.kblocks != 1) return cudaErrorInvalidValue;
      if (kl <= 16) return launch_scan_kernel<FP8, 16, 4, METRIC, 4, false, TS>(ta, tb, a, grid, stream);
      return launch_scan_kernel<FP8, 32, 2, METRIC, 4, false, TS>(ta, tb, a, grid, stream);
    }
    return cudaErrorInvalidValue;
  }
  if (groups == 2) {
    switch (kl) {
      case 16: return launch_scan_kernel<FP8, 16, 3, METRIC, 2, false, TS>(ta, tb, a, grid, stream);
      case 32: return launch_scan_kernel<FP8, 32, 2, METRIC, 2, false, TS>(ta, tb, a, grid, stream);
      default: return launch_scan_kernel<FP8, 48, 2, METRIC, 2, false, TS>(ta, tb, a, grid, stream);
    }
  }
  switch (kl) {
    case 16: return launch_scan_kernel<FP8, 16, 4, METRIC, 1, false, TS>(ta, tb, a, grid, stream);
    case 32: return launch_scan_kernel<FP8, 32, 3, METRIC, 1, false, TS>(ta, tb, a, grid, stream);
    case 48: return launch_scan_kernel<FP8, 48, 3, METRIC, 1, false, TS>(ta, tb, a, grid, stream);
    default: return launch_scan_kernel<FP8, 64, 3, METRIC, 1, false, TS>(ta, tb, a, grid, stream);
  }
}

template <bool FP8>
cudaError_t dispatch_scan(int kl, int groups, int metric, bool table_scale, const CUtensorMap& ta,
                          const CUtensorMap& tb, const TcScanArgs& a, uint32_t grid, cudaStream_t stream) {
  // TS (fp8 only): false for a per-row-scale table, whose L2 / IP epilogue
  // reads each row's scale and norm; cosine reads them either way
  if constexpr (FP8) {
    if (!table_scale && metric == METRIC_INNER_PRODUCT)
      return dispatch_scan_kl<FP8, METRIC_INNER_PRODUCT, false>(kl, groups, ta, tb, a, grid, stream);
    if (!table_scale && metric == METRIC_L2)
      return dispatch_scan_kl<FP8, METRIC_L2, false>(kl, groups, ta, tb, a, grid, stream);
  }
  switch (metric) {
    case METRIC_INNER_PRODUCT:
      return dispatch_scan_kl<FP8, METRIC_INNER_PRODUCT, true>(kl, groups, ta, tb, a, grid, stream);
    case METRIC_COSINE: return dispatch_scan_kl<FP8, METRIC_COSINE, true>(kl, groups, ta, tb, a, grid, stream);
    default: return dispatch_scan_kl<FP8, METRIC_L2, true>(kl, groups, ta, tb, a, grid, stream);
  }
}

}  // namespace fv
