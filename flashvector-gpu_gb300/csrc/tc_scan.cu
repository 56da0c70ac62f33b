// tc_scan.cu -- tensor-core flat scan (FP16 and FP8-E4M3) fused with top-k,
// followed by an exact fp32 rescore of an over-fetched shortlist and an
// fp64 re-rank of the candidates that straddle the k-th distance.
//
// Replaces the reference's fp16_tc_wmma_search_kernel / launch_fp16_tc_search
// (ivf_quant_lookup.cu:894-1058): same inputs (Fp16GpuTables) and result
// layout; the reference scores 16 queries x 64 rows per step with wmma and
// re-streams the whole fp16 base set once per 16 queries.
//
// The scan kernel itself (tc_scan_kernel.cuh) is instantiated per precision
// in tc_scan_fp16.cu / tc_scan_fp8.cu. Machine mapping (one CTA per SM,
// 64 + 128 G threads for G epilogue groups):
//   warp 0    TMA producer: per K block, a 128-query tile (A) and a 256-row
//             base tile (B), 128-byte-swizzled, into a STAGES-deep ring;
//   warp 1    TMEM owner + single-thread tcgen05.mma issuer (M=128, N=256,
//             fp32 accumulators, two 256-column buffers so the epilogue of
//             tile i overlaps the MMAs of tile i+1);
//   warps 2.. epilogue, 4 warps per group: thread r of a group owns query r
//             of the block (TMEM lane r),
//             turns dot products into distances, applies the slot mask and
//             keeps that query's best (distance, slot) keys. No distance
//             matrix ever reaches HBM.
// A call first finds a bound per query from column minima (of a sample of the
// base, or of all of it) and then scans with it: a range's few keys under the
// bound are appended to its list. A CTA scans a range of base tiles, every so many;
// the lists are merged by tc_select_kernel, which also rescores them in fp32.
#include <cmath>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cudaTypedefs.h>

#include "../../include/fv_bridge.h"
#include "tc_scan_kernel.cuh"

namespace fv {

namespace {

// ---------------------------------------------------------------------------
// Query preparation: fp32 -> fp16 (round to nearest even, as the reference
// converts queries: ivf_quant_lookup.cu:953) or fp32 -> e4m3 with a per-query
// power-of-two scale s_q = 2^a: the smallest with max|q| <= 448 s_q, raised
// where needed to 2^(b - 8) (s = 2^b the table's scale) so that the L2
// norm-digit factor -s / s_q = -2^(b - a) is an e4m3 value; it goes into
// columns dim..dim+2 against the table's norm digits (0 there for inner
// product and cosine, and for L2 where b - a < -9: a query so much larger
// than every row that the rows' norms no longer order the candidates);
// ||q||^2 of the fp32 query (the reference's :922-928, here summed across
// the warp: it only enters the scan's approximate distance). One warp per
// query.
// ---------------------------------------------------------------------------
template <bool FP8>
__global__ void __launch_bounds__(256) tc_prep_queries_kernel(const float* __restrict__ q, uint32_t nq, uint32_t dim,
                                                              uint32_t pd, void* __restrict__ out,
                                                              float* __restrict__ qnorm, float* __restrict__ qscale,
                                                              uint32_t* __restrict__ tslot, uint32_t kl,
                                                              uint32_t stride, const float* __restrict__ xscale,
                                                              int metric, uint32_t nq_rows, bool table_scale) {
  const uint32_t qi = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (qi >= nq_rows) return;
  if (qi >= nq) {
    // padding rows up to a whole query block: zero codes, so that every TMA
    // load of a query tile is in bounds (an out-of-bounds fill of most of a
    // 128-row tile, reloaded per K block, slowed a one-query scan by 40%)
    const size_t row_bytes = (size_t)pd * (FP8 ? 1 : 2);
    uint8_t* o = static_cast<uint8_t*>(out) + (size_t)qi * row_bytes;
    for (size_t b = (size_t)lane * 16; b < row_bytes; b += 32 * 16) *reinterpret_cast<uint4*>(o + b) = make_uint4(0, 0, 0, 0);
    return;
  }
  const float* src = q + (size_t)qi * dim;
  // shared-bound slots: empty (all ones) for the kl used, 0 for the padding
  for (uint32_t s = lane; s < stride; s += 32) tslot[(size_t)qi * stride + s] = s < kl ? 0xFFFFFFFFu : 0u;
  {
    // ||q||^2 of the scan's approximate distance (L2 and cosine); the exact
    // fp32 rescore recomputes distances in the reference's order
    float s = 0.f;
    for (uint32_t d = lane; d < dim; d += 32) s = fmaf(src[d], src[d], s);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) qnorm[qi] = s;
  }
  if (FP8) {
    float amax = 0.f;
    for (uint32_t d = lane; d < dim; d += 32) amax = fmaxf(amax, fabsf(src[d]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (!table_scale) {
      // per-row-scale table: the query's scale amax / 448, no norm digits
      const float scale = amax > 0.f ? amax / 448.0f : 1.0f;
      if (lane == 0) qscale[qi] = scale;
      uint8_t* o8 = static_cast<uint8_t*>(out) + (size_t)qi * pd;
      for (uint32_t d = lane; d < pd; d += 32)
        o8[d] = d < dim ? (uint8_t)__nv_cvt_float_to_fp8(src[d] / scale, __NV_SATFINITE, __NV_E4M3) : (uint8_t)0;
      return;
    }
    const int b = ilogbf(__ldg(xscale));
    int a = b - 8;
    if (amax > 0.f) {
      int ap = ilogbf(amax) - 8;
      for (int it = 0; it < 4 && ldexpf(448.0f, ap) < amax; ++it) ++ap;
      for (int it = 0; it < 4 && ldexpf(448.0f, ap - 1) >= amax; ++it) --ap;
      a = max(a, ap);
    }
    if (lane == 0) qscale[qi] = ldexpf(1.0f, a);
    const float digit = (metric == METRIC_L2 && b - a >= -9) ? -ldexpf(1.0f, b - a) : 0.f;
    uint8_t* o8 = static_cast<uint8_t*>(out) + (size_t)qi * pd;
    for (uint32_t d = lane; d < pd; d += 32) {
      const float v = d < dim ? ldexpf(src[d], -a) : (d < dim + 3 ? digit : 0.f);
      o8[d] = (uint8_t)__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3);
    }
  } else {
    __half* o16 = static_cast<__half*>(out) + (size_t)qi * pd;
    for (uint32_t d = lane; d < pd; d += 32) o16[d] = d < dim ? __float2half_rn(src[d]) : __float2half_rn(0.f);
  }
}

// fp64 distance in the warp's lane-strided order (only the candidates at the
// k-th boundary go through here).
__device__ double warp_distance_f64(const float* __restrict__ q, const float* __restrict__ x, uint32_t dim, int lane,
                                    int metric) {
  double a = 0.0, b = 0.0, c = 0.0;
  constexpr int B = 8;  // loads in flight ahead of the (ordered) accumulation
  for (uint32_t d0 = lane; d0 < dim; d0 += 32 * B) {
    float qa[B], xa[B];
#pragma unroll
    for (int i = 0; i < B; ++i) {
      const uint32_t d = d0 + 32 * i;
      qa[i] = d < dim ? q[d] : 0.f;
      xa[i] = d < dim ? __ldg(x + d) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < B; ++i) {
      if (d0 + 32 * i >= dim) break;
      const double u = qa[i], w = xa[i];
      if (metric == METRIC_L2) {
        const double t = u - w;
        a += t * t;
      } else {
        a += u * w;
        b += u * u;
        c += w * w;
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
    c += __shfl_xor_sync(0xffffffffu, c, o);
  }
  if (metric == METRIC_L2) return a;
  if (metric == METRIC_INNER_PRODUCT) return -a;
  return 1.0 - a / (sqrt(b) * sqrt(c) + 1e-300);
}

struct SelectArgs {
  const uint64_t* partial;   // [nq][lists][KL]
  uint32_t lists, kl, cap, shortlist, k;  // cap: keys that fit the block's shared memory (power of two)
  const float* queries;      // fp32 queries (rescore)
  const float* vectors;      // fp32 rows (null: no rescore)
  uint32_t dim;
  int metric;
  uint32_t boundary;
  float eps;
  GpuSearchResult* out;
  uint32_t* status;
  const float* tau;          // per-query admission bound of the scan (null: none)
  uint32_t* redo;            // set for a bounded query that kept too few keys
  const uint32_t* only;      // process only the flagged queries (null: all)
  uint32_t* incomplete_q;    // per-query flag set when a range heap may have dropped keys (or null)
};

constexpr int BAND_MAX = 64;

// One CTA per query: merge the per-range heaps, keep the best `shortlist`
// keys, rescore them in fp32 (the reference's warp-order distance), sort,
// re-rank the band |d - d_k| <= eps * scale in fp64, write the top k.
// NT: 256 threads, or 1,024 where the queries leave SMs idle (1 query of 1M x
// 768: 22 us with 256, most of it the rows' latency).
template <int NT>
__global__ void __launch_bounds__(NT) tc_select_kernel(SelectArgs s) {
  extern __shared__ __align__(16) uint64_t keys[];
  __shared__ double band_d[BAND_MAX];
  __shared__ int band_lo, band_hi;
  __shared__ int incomplete;
  const uint32_t q = blockIdx.x;
  if (s.only && s.only[q] == 0u) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t total = s.lists * s.kl;
  const uint64_t* src = s.partial + (size_t)q * total;
  __shared__ uint32_t n_live;
  if (threadIdx.x == 0) incomplete = 0;
  // only the kept keys are sorted (lists that stayed partly empty hold
  // sentinels); sorted they are the same sequence as the whole table sorted
  const uint32_t kp = min(s.shortlist, total);
  uint32_t live = block_compact_keys(src, total, keys, &n_live, s.cap);
  if (live > s.cap) {
    // more keys than the launch foresaw (an unlucky sample, rows in an order
    // that fills one range): keep the best kp by their kp-th key
    const uint64_t limit = block_kth_key(src, total, kp);
    live = block_compact_keys(src, total, keys, &n_live, s.cap, limit);
  }
  const uint32_t sp2 = next_pow2_dev(max(max(live, kp), 2u));
  for (uint32_t i = live + threadIdx.x; i < sp2; i += NT) keys[i] = kSentinelKey;
  __syncthreads();
  block_bitonic_sort(keys, sp2);
  if (s.kl < kp) {
    // a range whose heap stayed full and whose worst kept key still beats the
    // kp-th merged key may have dropped keys that belong in the shortlist
    const uint64_t cut = keys[kp - 1];
    for (uint32_t l = threadIdx.x; l < s.lists; l += NT) {
      const uint64_t root = src[(size_t)l * s.kl];
      if (root != kSentinelKey && root < cut) incomplete = 1;
    }
  }
  __syncthreads();
  if (incomplete && threadIdx.x == 0) {
    set_status(s.status, kStatusOverflow);
    if (s.incomplete_q) s.incomplete_q[q] = 1u;
  }
  // a bounded scan kept too few rows (see plan_tc_scan): the query is scanned
  // again unbounded
  if (s.redo && threadIdx.x == 0 && keys[kp - 1] == kSentinelKey && s.tau[q] < kSentinelDist &&
      (!incomplete || keys[min(s.k, kp) - 1] == kSentinelKey))
    s.redo[q] = 1u;

  const float* qv = s.queries + (size_t)q * s.dim;
  if (s.vectors) {
    // four candidates per warp pass (two of 32 warps), so that as many rows'
    // gathers are in flight
    constexpr uint32_t NW = NT / 32, R = NT == 256 ? 4 : 2;
    for (uint32_t c0 = warp; c0 < kp; c0 += R * NW) {
      if (keys[c0] == kSentinelKey) break;  // sorted: the rest are sentinels too
      const float* rows[R];
      uint32_t slot[R];
#pragma unroll
      for (uint32_t r = 0; r < R; ++r) {
        // a missing candidate re-reads the first one and is not stored
        const uint32_t c = c0 + r * NW;
        const uint64_t key = c < kp ? keys[c] : kSentinelKey;
        slot[r] = key_slot(key != kSentinelKey ? key : keys[c0]);
        rows[r] = s.vectors + (size_t)slot[r] * s.dim;
      }
      float d[R];
      warp_metric_distances<R, NT == 256 ? 4 : 8>(qv, rows, s.dim, lane, (MetricType)s.metric, d);
      __syncwarp();
      if (lane == 0) {
#pragma unroll
        for (uint32_t r = 0; r < R; ++r) {
          const uint32_t c = c0 + r * NW;
          if (c < kp && keys[c] != kSentinelKey) keys[c] = d[r] < kSentinelDist ? make_key(d[r], slot[r]) : kSentinelKey;
        }
      }
    }
    const uint32_t p2 = next_pow2_dev(kp);
    for (uint32_t i = kp + threadIdx.x; i < p2; i += NT) keys[i] = kSentinelKey;
    __syncthreads();
    block_bitonic_sort(keys, p2);

    if (s.boundary && s.k <= kp && keys[s.k - 1] != kSentinelKey) {
      // ||q||^2 for the band's width, summed by warp 0 (lane-strided, tree)
      float qn = 0.f;
      if (warp == 0) {
        for (uint32_t d = lane; d < s.dim; d += 32) qn = fmaf(qv[d], qv[d], qn);
        qn = warp_tree_sum(qn);
      }
      if (threadIdx.x == 0) {
        const float dk = key_dist(keys[s.k - 1]);
        // scale of the accumulated terms: |d_k| for L2; |q||x| bounds |dot|
        float scale = fabsf(dk) + (s.metric == METRIC_L2 ? 0.f : sqrtf(qn) * 2.0f);
        const float band = s.eps * scale;
        int lo = (int)s.k - 1, hi = (int)s.k;
        while (lo > 0 && key_dist(keys[lo - 1]) >= dk - band) --lo;
        while (hi < (int)kp && keys[hi] != kSentinelKey && key_dist(keys[hi]) <= dk + band) ++hi;
        if (hi - lo > BAND_MAX || hi - lo < 2) lo = hi = 0;
        band_lo = lo;
        band_hi = hi;
      }
      __syncthreads();
      const int lo = band_lo, hi = band_hi;
      for (int c = lo + warp; c < hi; c += NT / 32) {
        const double d = warp_distance_f64(qv, s.vectors + (size_t)key_slot(keys[c]) * s.dim, s.dim, lane, s.metric);
        if (lane == 0) band_d[c - lo] = d;
      }
      __syncthreads();
      if (threadIdx.x == 0 && hi > lo) {
        // insertion sort of the band by (fp64 distance, slot); distances
        // reported for the band are the fp64 values rounded to fp32
        for (int i = lo + 1; i < hi; ++i) {
          const double di = band_d[i - lo];
          const uint64_t ki = keys[i];
          int j = i - 1;
          while (j >= lo && (band_d[j - lo] > di || (band_d[j - lo] == di && key_slot(keys[j]) > key_slot(ki)))) {
            band_d[j + 1 - lo] = band_d[j - lo];
            keys[j + 1] = keys[j];
            --j;
          }
          band_d[j + 1 - lo] = di;
          keys[j + 1] = ki;
        }
        for (int i = lo; i < hi; ++i) keys[i] = make_key((float)band_d[i - lo], key_slot(keys[i]));
      }
      __syncthreads();
    }
  }
  for (uint32_t r = threadIdx.x; r < s.k; r += NT)
    s.out[(size_t)q * s.k + r] = key_to_result(r < kp ? keys[r] : kSentinelKey, nullptr);
}

// The admission bound of each query: the r-th smallest of its `cnt` minima
// (no bound, 1e30, when fewer than r of them are distances), raised by a few
// ulps so that the scan admits every row behind it. NV values per thread in
// registers (the rest re-read from L2), the answer built bit by bit from the
// top of the ordered representation by counting values. Also clears the
// query's re-scan flag. A scan whose distances carry an error raises the bound
// b to b + m.rel |b| + m.per_norm qnorm[q] + m.abs.
struct TauMargin {
  float rel = 1e-6f, per_norm = 0.f, abs = 0.f;
  const float* qnorm = nullptr;
};
//
// Up to 2,048 minima a query is one warp's, without barriers (2,000 queries of
// 512: 12 us with a block each); more take a block of 128 threads.
constexpr int TAU_THREADS = 128;
template <int NV, bool WARP>
__global__ void __launch_bounds__(TAU_THREADS) tc_tau_kernel(const float* __restrict__ pmin, uint32_t nq, uint32_t cnt,
                                                             uint32_t stride, uint32_t r, TauMargin m,
                                                             float* __restrict__ tau, uint32_t* __restrict__ redo) {
  constexpr int LANES = WARP ? 32 : TAU_THREADS;  // threads of a query
  __shared__ uint32_t part[2][TAU_THREADS / 32];
  const uint32_t q = WARP ? blockIdx.x * (TAU_THREADS / 32) + (threadIdx.x >> 5) : blockIdx.x;
  const uint32_t tid = WARP ? threadIdx.x & 31u : threadIdx.x;
  if (q >= nq) return;  // (whole warps)
  const float* src = pmin + (size_t)q * stride;
  uint32_t u[NV], lo = 0xFFFFFFFFu, hi = 0;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const uint32_t at = (uint32_t)i * LANES + tid;
    u[i] = at < cnt ? float_order(__ldcg(src + at)) : 0xFFFFFFFFu;
    lo = min(lo, u[i]);
    if (at < cnt) hi = max(hi, u[i]);
  }
  // bits above the highest in which two values differ are common to all
  int top = 31;
  uint32_t ans = 0;
  if (WARP) {
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    top = 31 - __clz(lo ^ hi);
    ans = top < 0 ? lo : lo & ~((2u << top) - 1u);
  }
#pragma unroll 1
  for (int bit = top; bit >= 0; --bit) {
    const uint32_t test = ans | ((1u << bit) - 1u);
    uint32_t c = 0;
#pragma unroll
    for (int i = 0; i < NV; ++i) c += u[i] <= test;
    if (!WARP)
      for (uint32_t at = NV * LANES + tid; at < cnt; at += LANES) c += float_order(__ldcg(src + at)) <= test;
    c = __reduce_add_sync(0xffffffffu, c);
    if (!WARP) {
      if ((tid & 31) == 0) part[bit & 1][tid >> 5] = c;
      __syncthreads();
      c = 0;
#pragma unroll
      for (int w = 0; w < TAU_THREADS / 32; ++w) c += part[bit & 1][w];
    }
    if (c < r) ans |= 1u << bit;
  }
  if (tid == 0) {
    const float t = order_float(ans);
    const float up = m.rel * fabsf(t) + m.abs + (m.qnorm ? m.per_norm * fabsf(m.qnorm[q]) : 0.f);
    tau[q] = t < kSentinelDist ? (t > -INFINITY ? t + up : t) : kSentinelDist;  // (-inf + inf is NaN)
    redo[q] = 0u;
  }
}

void launch_tau(const float* pmin, uint32_t nq, uint32_t cnt, uint32_t stride, uint32_t r, const TauMargin& m,
                float* tau, uint32_t* redo, cudaStream_t stream) {
  auto go = [&](auto kern, uint32_t per_block) {
    kern<<<(nq + per_block - 1) / per_block, TAU_THREADS, 0, stream>>>(pmin, nq, cnt, stride, r, m, tau, redo);
  };
  constexpr uint32_t W = TAU_THREADS / 32;
  if (cnt <= 256)
    go(tc_tau_kernel<8, true>, W);
  else if (cnt <= 512)
    go(tc_tau_kernel<16, true>, W);
  else if (cnt <= 1024)
    go(tc_tau_kernel<32, true>, W);
  else if (cnt <= 2048)
    go(tc_tau_kernel<64, true>, W);
  else
    go(tc_tau_kernel<32, false>, 1);
}

// cuTensorMapEncodeTiled resolved through the runtime, so the library does
// not link libcuda (it must load on hosts without a driver).
PFN_cuTensorMapEncodeTiled_v12000 tmap_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

bool encode_tmap(CUtensorMap* m, const void* ptr, bool fp8, uint64_t inner_elems, uint64_t rows, uint64_t row_bytes,
                 uint32_t box_rows) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = tmap_encoder();
  if (!enc) return false;
  cuuint64_t dims[2] = {inner_elems, rows};
  cuuint64_t strides[1] = {row_bytes};
  cuuint32_t box[2] = {(cuuint32_t)(fp8 ? 128 : 64), box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(m, fp8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
                                      const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                      CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// The base as the minima pass reads it: tile t of `tiles` holds the runs of RUN
// rows t, t + tiles, t + 2 tiles, .. of every stride-th one (box_runs of the RUNS
// a box); every coordinate inside the table, as RUNS RUN stride tiles <= n.
bool encode_runs(CUtensorMap* m, const void* ptr, bool fp8, uint64_t inner_elems, uint64_t row_bytes, uint32_t stride,
                 uint32_t tiles, uint32_t box_runs) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = tmap_encoder();
  if (!enc) return false;
  const cuuint64_t run_bytes = (cuuint64_t)RUN * stride * row_bytes;
  cuuint64_t dims[4] = {inner_elems, RUN, tiles, RUNS};
  cuuint64_t strides[3] = {row_bytes, run_bytes, run_bytes * tiles};
  cuuint32_t box[4] = {(cuuint32_t)(fp8 ? 128 : 64), RUN, 1, box_runs};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  return enc(m, fp8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void*>(ptr), dims,
             strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// ---------------------------------------------------------------------------
// Committed autotuner results (flashvector-gpu_gb300/tuning/gb300.json,
// compiled in by build.py as tuning_table.inc): per shape range, the CTA-pair
// choice, the pre-pass choice and stride, and the over-fetch that reached
// recall@10 >= 0.99 fastest on this GPU. Explicit knobs (fv_tune_set) and
// explicit scan options take precedence; "tc.table" = 0 ignores the table.
// ---------------------------------------------------------------------------
struct TuneEntry {
  int fp8, metric;
  uint32_t dim_lo, dim_hi;
  uint64_t n_lo, n_hi;
  uint32_t nq_lo, nq_hi, k_lo, k_hi;
  int pair, prepass, stride, overfetch;
};
const TuneEntry kTuneTable[] = {
#include "tuning_table.inc"
    {-1, -1, 0, 0, 0, 0, 0, 0, 0, 0, -1, -1, 0, 0}};

const TuneEntry* tune_lookup(bool fp8, int metric, uint32_t dim, uint64_t n, uint32_t nq, uint32_t k) {
  if (tune_value("tc.table", 1) == 0) return nullptr;
  for (const TuneEntry& e : kTuneTable) {
    if (e.fp8 < 0) break;
    if (e.fp8 == (fp8 ? 1 : 0) && e.metric == metric && dim >= e.dim_lo && dim <= e.dim_hi && n >= e.n_lo &&
        n <= e.n_hi && nq >= e.nq_lo && nq <= e.nq_hi && k >= e.k_lo && k <= e.k_hi)
      return &e;
  }
  return nullptr;
}

// Sampled rank for the pre-pass bound. A sample of every stride-th run of rows
// holds each of a query's top (shortlist - 1) rows with probability
// 1 / stride, so the number of them in the sample is about Poisson(lambda =
// shortlist / stride); the sample's r-th best distance is below the query's
// shortlist-th distance (and the query needs the re-scan) only when that
// count reaches r. Returns the smallest r whose Poisson tail P(X >= r) is
// below `tail`.
uint32_t poisson_rank(double lambda, double tail) {
  double term = std::exp(-lambda), cdf = 0.0;
  uint32_t r = 0;
  while (1.0 - cdf >= tail && r < 4096) {
    cdf += term;
    ++r;
    term *= lambda / r;
  }
  return r;
}

// One CTA per SM at a time: a grid of nqb * splits CTAs runs in
// ceil(nqb * splits / sms) waves, the last one possibly part-empty. Among
// split counts in [s_min, max(2 s_min, 32)] (within the tile count and the
// select kernel's 16,384-key sort), take the smallest whose waves are at
// least 1% fuller than those of every smaller candidate (a grid of 79 query
// blocks x 1 split fills 53% of 148 SMs; x 13 splits, 99%).
uint32_t fill_waves(uint32_t s_min, uint32_t nqb, uint32_t ntiles, uint32_t sms, uint32_t keys_per_split) {
  auto fullness = [&](uint32_t s) {
    const uint64_t ctas = (uint64_t)nqb * s, waves = (ctas + sms - 1) / sms;
    return (double)ctas / (double)(waves * sms);
  };
  uint32_t best = s_min;
  double best_f = fullness(s_min);
  for (uint32_t s = s_min + 1; s <= std::max(2 * s_min, 32u) && s <= ntiles; ++s) {
    if ((uint64_t)s * keys_per_split > 16384u) break;
    const double f = fullness(s);
    if (f > best_f + 0.01) {
      best = s;
      best_f = f;
    }
  }
  return best;
}

}  // namespace

// rank > 0: a collecting pass (launch_tc_collect): the bound is for the rank
// best rows, and the heaps have room for k.
TcPlan plan_tc_scan(const TcTables& t, uint32_t nq, uint32_t k, MetricType metric, const FvScanOptions& opt,
                    uint32_t rank) {
  TcPlan P{};
  const bool fp8 = t.fp8;
  const uint32_t elem = fp8 ? 1 : 2;
  const uint32_t kb_elems = fp8 ? 128 : 64;
  const uint32_t kblocks = (t.padded_dim + kb_elems - 1) / kb_elems;
  const TuneEntry* te = rank ? nullptr : tune_lookup(fp8, (int)metric, t.dim, t.n, nq, k);
  const uint32_t overfetch = opt.overfetch ? opt.overfetch : (te && te->overfetch > 0 ? (uint32_t)te->overfetch : 4u);
  const uint32_t shortlist = t.vectors ? std::min<uint32_t>(std::max(k, overfetch * k), 4096u) : k;
  // short K (at most two 64-element fp16 / 128-element fp8 blocks per tile):
  // a tile costs the MMA little and the epilogue much, so two epilogue
  // groups drain the two accumulator buffers in parallel. Fused fp8 with one
  // K block and a shortlist above 48 keys (where two groups' heaps hold less
  // than the shortlist too) runs four ("tc.groups": -1 auto, 2 or 4).
  const bool fused_fp8 = fp8 && t.fp8_table_scale && metric != METRIC_COSINE && kblocks == 1;
  const int64_t groups_knob = tune_value("tc.groups", -1);
  const bool four = fused_fp8 && (groups_knob == 4 || (groups_knob < 0 && shortlist > 48u));
  const int groups = kblocks > 2 ? 1 : (four ? 4 : 2);
  const uint32_t kl_cap = groups == 4 ? 32u : (groups == 2 ? 48u : 64u);
  const uint32_t kl = std::min<uint32_t>(kl_cap, shortlist);         // heap entries per (query, range, group)
  const uint32_t kl_tmpl = std::min<uint32_t>(kl_cap, (kl + 15) / 16 * 16);  // heap capacity (template)
  const uint32_t nqb = (nq + TC_M - 1) / TC_M;
  const uint32_t ntiles = (t.n + TC_N - 1) / TC_N;
  const int sms = device_sm_count();
  // CTA pairs (cta_group::2) for long rows: two query blocks share each
  // base tile, each SM streaming half of it
  int64_t pair_knob = tune_value("tc.pair", -1);
  if (pair_knob < 0 && te && te->pair >= 0) pair_knob = te->pair;
  const bool pair = groups == 1 && pair_knob != 0;
  const uint32_t nqb_grid = pair ? 2 * ((nqb + 1) / 2) : nqb;  // CTAs per split
  uint32_t splits = opt.splits ? opt.splits : std::max<uint32_t>(1u, (uint32_t)sms / nqb_grid);
  if (!opt.splits && shortlist > kl) {
    // a (query, range, group) heap keeps kl keys: split the base so that each
    // heap holds, in expectation, a third of its share of the shortlist (a
    // heap that still overflows is reported through the status word)
    splits = std::max<uint32_t>(splits, (3 * shortlist + kl * groups - 1) / (kl * groups));
  }
  splits = std::max(1u, std::min(splits, ntiles));
  if (!opt.splits) splits = fill_waves(splits, nqb_grid, ntiles, (uint32_t)sms, groups * kl);
  // the select kernel sorts lists*kl keys in shared memory: <= 16384
  while (splits > 1 && next_pow2(splits * groups * kl) > 16384u) --splits;
  const uint32_t tps = (ntiles + splits - 1) / splits;
  splits = (ntiles + tps - 1) / tps;

  // Pre-pass: each query's admission bound for the scan, from the minima pass
  // over every pstride-th run of 8 rows. A sample of stride s holds each of the
  // query's top (shortlist - 1) rows with probability 1 / s; the bound is the
  // r-th smallest minimum, r from the Poisson tail below (or ceil(margin *
  // shortlist / stride) when the margin knob is set), and the sampled r-th
  // distance is an upper bound on the shortlist-th distance unless the sample
  // is unlucky (probability < 1e-7 per query); with s = 1 it always is, at
  // r = shortlist (the same accumulators, hence the same distances, are
  // behind the bound and the scan). The scan then admits only rows within it.
  // Queries whose bounded scan comes up short are scanned again without the
  // bound (device-side, no host round trip): the bound was too tight (s > 1), or a
  // range's list, which holds less than the shortlist where that is above 48 or
  // 64, filled up (rows that the base's order puts into one tile). The scan without
  // a bound loses the same rows to a full list, so that one is no reason while
  // there are k keys.
  //
  // Automatic stride. Long rows are bound by the MMA, whose pass costs 1 / s
  // of the scan again: 64 sampled tiles. Short rows (at most two K blocks)
  // are bound by the candidate path, which a tighter bound shortens: 256
  // tiles. At most 32 either way (the share of the scan is then 3% and the
  // bound admits rows of rank ~8 shortlists), more only to keep a query's
  // minima within 4,096.
  int64_t pp_knob = tune_value("tc.prepass", -1);
  if (pp_knob < 0 && te && te->prepass >= 0) pp_knob = te->prepass;
  int64_t stride_knob = tune_value("tc.prepass_stride", 0);
  if (stride_knob <= 0 && te && te->stride > 0) stride_knob = te->stride;
  const uint32_t auto_stride = std::max(std::min(32u, std::max(1u, ntiles / (kblocks > 2 ? 64u : 256u))),
                                        (ntiles + 2047u) / 2048u);
  uint32_t pstride =
      stride_knob > 0 ? (uint32_t)std::min<int64_t>(std::max<int64_t>(2, stride_knob), 1 << 20) : auto_stride;
  const int64_t pmargin = rank ? 0 : tune_value("tc.prepass_margin", 0);
  const uint32_t ranked = rank ? rank : shortlist;  // rows that the bound is for
  const size_t part_bytes = align_up((size_t)nq * splits * groups * kl * 8, 256);
  // The coarsest minima (fewest to store and to select from) that still number
  // 8 r, so that two of a query's r best rows seldom share one: with c minima the
  // bound admits about -c ln(1 - r / c) rows, 1.07 r for 8 r and 1.4 r for 2 r. Up
  // to 512, which cost nothing to select from, 32 r: a minimum of 128 columns
  // holds eight neighbours of a run, which a base in order of distance all has
  // among the best (60,000 x 128 in order of norm, 200 queries, L2, k 10: 290 us a
  // call with 8 r, 208 so).
  // They live in the space of the range heaps, which are written after the bound
  // is known: a call takes no more scratch than its unbounded scan. Where 8 r do
  // not fit there, the most that fit down to 2 r; where those do not either, the
  // sample is thinned until they do (4M x 96 fp8 rows, 4,000 queries, a stride of
  // 8 asked for: 14.2 ms without a bound, 7.4 with one).
  uint32_t pgran = 0, pcount = 0, psampled = 0, pr = 0;
  while (true) {
    psampled = t.n / (TC_N * pstride);
    pr = std::max<uint32_t>(1u, pmargin > 0 ? (uint32_t)((pmargin * ranked + pstride - 1) / pstride)
                                            : (pstride == 1 ? ranked : poisson_rank((double)ranked / pstride, 1e-7)));
    for (uint32_t g = 128; g >= 8 && !pgran; g >>= 1) {
      const uint32_t c = psampled * (TC_N / g);
      if ((c >= std::max(8 * pr, std::min(32 * pr, 512u)) || g == 8) && (size_t)nq * c * 4 <= part_bytes) {
        pgran = g;
        pcount = c;
      }
    }
    for (uint32_t g = 16; g <= 128 && !pgran; g <<= 1) {
      const uint32_t c = psampled * (TC_N / g);
      if (c >= 2 * pr && (size_t)nq * c * 4 <= part_bytes) {
        pgran = g;
        pcount = c;
      }
    }
    if (pgran || psampled < 64) break;
    pstride *= 2;
  }
  // Off where the base is so small that the minima cannot bound (the heaps then
  // hold about every row anyway), and where the heaps of a few keys, with the bound
  // that ranges share, cost less than the pass (us a call with and without it):
  // shortlists of 4 for one or two queries, which fill one lane (100,000 x 768: 78
  // and 61; 300,000 x 64: 56 and 50), of 8 there over long rows of larger bases (78
  // and 68), and of 4 for many queries over larger bases (866 of 300,000 x 156, half
  // masked: 225 and 189; 1M x 64: 299 and 274; for 128 queries it is 61 and 111).
  // The knob turns it off, or on, anywhere.
  const bool long_rows = kblocks > 2, one_lane = nq <= 2, many = nqb >= 4;
  const bool quick = !rank && ((shortlist <= 4 && ((one_lane && (long_rows || ntiles >= 1024)) ||
                                                   (many && ntiles >= (long_rows ? 256u : 2048u)))) ||
                               (shortlist <= 8 && one_lane && long_rows && ntiles >= 256));
  const bool prepass = pp_knob != 0 && (pp_knob > 0 || !quick) && pgran && pcount >= 2 * pr;
  psampled = std::max(1u, psampled);
  uint32_t psplits = std::max<uint32_t>(1u, std::min<uint32_t>((uint32_t)sms / nqb_grid, psampled));
  psplits = fill_waves(psplits, nqb_grid, psampled, (uint32_t)sms, 0);
  const uint32_t ptps = (psampled + psplits - 1) / psplits;
  psplits = (psampled + ptps - 1) / ptps;

  // scratch: prepared queries | ||q||^2 | q scales | minima, then range heaps |
  //          bounds and re-scan flags (pre-pass), or shared-bound slots
  // prepared queries padded with zero rows to whole query blocks (of the
  // CTA pairs' grid when pairs run)
  const uint32_t nq_rows = nqb_grid * TC_M;
  const size_t q_bytes = align_up((size_t)nq_rows * t.padded_dim * elem, 1024);
  const size_t qn_bytes = align_up((size_t)nq * 4, 256);
  const uint32_t slot_stride = prepass ? 0u : (kl + 3) / 4 * 4;
  const size_t slot_bytes = align_up((size_t)nq * slot_stride * 4, 256);
  const size_t tau_bytes = prepass ? align_up((size_t)nq * 8, 256) : 0;
  P.fp8 = fp8;
  P.elem = elem;
  P.kblocks = kblocks;
  P.shortlist = shortlist;
  P.groups = groups;
  P.kl = kl;
  P.kl_tmpl = kl_tmpl;
  P.nqb = nqb;
  P.pair = pair;
  P.nqb_grid = nqb_grid;
  P.splits = splits;
  P.prepass = prepass;
  P.pstride = pstride;
  P.pr = pr;
  P.ptiles = psampled;
  P.pgran = pgran;
  P.pcount = pcount;
  P.psplits = psplits;
  P.nq_rows = nq_rows;
  P.q_bytes = q_bytes;
  P.qn_bytes = qn_bytes;
  P.part_bytes = part_bytes;
  P.slot_stride = slot_stride;
  P.slot_bytes = slot_bytes;
  P.tau_bytes = tau_bytes;
  P.scratch_bytes = q_bytes + 2 * qn_bytes + part_bytes + slot_bytes + tau_bytes;
  return P;
}

size_t tc_scan_scratch_bytes(const TcTables& t, uint32_t nq, uint32_t k, MetricType metric,
                             const FvScanOptions& opt) {
  return plan_tc_scan(t, nq, k, metric, opt).scratch_bytes;
}

int launch_tc_scan(const TcTables& t, const float* queries, uint32_t nq, uint32_t k, MetricType metric,
                   const uint32_t* mask, GpuSearchResult* out, const FvScanOptions& opt, cudaStream_t stream,
                   const QueryFilter* filters) {
  const TcPlan P = plan_tc_scan(t, nq, k, metric, opt);
  void* scratch = scratch_get(stream, P.scratch_bytes);
  if (!scratch) return (int)cudaErrorMemoryAllocation;
  return launch_tc_scan_planned(P, t, queries, nq, k, metric, mask, out, opt, stream, filters, scratch, nullptr);
}

int launch_tc_scan_planned(const TcPlan& P, const TcTables& t, const float* queries, uint32_t nq, uint32_t k,
                           MetricType metric, const uint32_t* mask, GpuSearchResult* out, const FvScanOptions& opt,
                           cudaStream_t stream, const QueryFilter* filters, void* scratch_at,
                           uint32_t* incomplete_q) {
  const bool fp8 = P.fp8;
  const uint32_t elem = P.elem, kblocks = P.kblocks, shortlist = P.shortlist, kl = P.kl, kl_tmpl = P.kl_tmpl;
  const int groups = P.groups;
  const uint32_t nqb = P.nqb, nqb_grid = P.nqb_grid, splits = P.splits;
  const bool pair = P.pair, prepass = P.prepass;
  const uint32_t nq_rows = P.nq_rows, slot_stride = P.slot_stride;
  const size_t q_bytes = P.q_bytes, qn_bytes = P.qn_bytes, part_bytes = P.part_bytes;
  uint8_t* scratch = static_cast<uint8_t*>(scratch_at);
  void* qprep = scratch;
  float* qnorm = reinterpret_cast<float*>(scratch + q_bytes);
  float* qscale = reinterpret_cast<float*>(scratch + q_bytes + qn_bytes);
  uint64_t* partial = reinterpret_cast<uint64_t*>(scratch + q_bytes + 2 * qn_bytes);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(scratch + q_bytes + 2 * qn_bytes + part_bytes);
  float* tau = prepass ? reinterpret_cast<float*>(tslot) : nullptr;
  uint32_t* redo = prepass ? tslot + nq : nullptr;

  {
    ProfScope ps(fp8 ? "tc_prep_queries_fp8" : "tc_prep_queries_fp16", stream);
    const uint32_t blocks = (nq_rows * 32 + 255) / 256;
    // the shared-bound slots serve a scan without the pre-pass (none with it:
    // slot_stride is 0)
    const uint32_t slot_kl = kl;
    if (fp8)
      tc_prep_queries_kernel<true><<<blocks, 256, 0, stream>>>(queries, nq, t.dim, t.padded_dim, qprep, qnorm, qscale,
                                                               tslot, slot_kl, slot_stride, t.scales, (int)metric,
                                                               nq_rows, t.fp8_table_scale);
    else
      tc_prep_queries_kernel<false><<<blocks, 256, 0, stream>>>(queries, nq, t.dim, t.padded_dim, qprep, qnorm,
                                                                qscale, tslot, slot_kl, slot_stride, nullptr,
                                                                (int)metric, nq_rows, false);
    note_launch();
  }

  const uint64_t row_bytes = (uint64_t)t.padded_dim * elem;
  CUtensorMap ta, tb, tb_half, tb_runs;
  if (!encode_tmap(&ta, qprep, fp8, t.padded_dim, nq_rows, row_bytes, TC_M) ||
      !encode_tmap(&tb, t.base, fp8, t.padded_dim, t.n, row_bytes, TC_N) ||
      (pair && !encode_tmap(&tb_half, t.base, fp8, t.padded_dim, t.n, row_bytes, TC_N / 2)) ||
      (prepass && !encode_runs(&tb_runs, t.base, fp8, t.padded_dim, row_bytes, P.pstride, P.ptiles,
                               pair ? RUNS / 2 : RUNS)))
    return FV_ERR_ARG;

  TcScanArgs a{};
  a.n = t.n;
  a.nq = nq;
  a.kblocks = kblocks;
  a.nqb = nqb;
  a.xnorm = t.norms;
  a.xscale = t.scales;
  a.qnorm = qnorm;
  a.qscale = qscale;
  a.mask = mask;
  a.tslot = tslot;
  a.tslot_stride = slot_stride;
  a.status = status_word();
  a.filters = filters;
  // "tc.wait_limit_ns" (0: 2 s) bounds the pipeline's waits; a wait that runs
  // out ends the scan early and is reported through the status word
  const int64_t wl = tune_value("tc.wait_limit_ns", 0);
  a.wait_ns = wl > 0 ? (uint64_t)wl : 2000000000ull;
  // use_pair: the CTA-pair variant (not for the re-scan of flagged queries,
  // whose blocks leave independently)
  auto scan = [&](const TcScanArgs& args, int kl_t, uint32_t splits_n, const char* name, bool use_pair,
                  int groups_n) -> cudaError_t {
    ProfScope ps(name, stream);
    const int g = use_pair ? -1 : groups_n;
    const uint32_t grid = (use_pair ? nqb_grid : nqb) * splits_n;
    const CUtensorMap& b = kl_t == kMinima ? tb_runs : use_pair ? tb_half : tb;
    return fp8 ? dispatch_tc_scan_fp8(kl_t, g, (int)metric, t.fp8_table_scale, ta, b, args, grid, stream)
               : dispatch_tc_scan_fp16(kl_t, g, (int)metric, true, ta, b, args, grid, stream);
  };
  cudaError_t e;
  if (prepass) {
    TcScanArgs p = a;
    p.splits = P.psplits;
    p.run_stride = P.pstride;
    p.pmin = reinterpret_cast<float*>(partial);
    p.pm_stride = P.pcount;
    p.gran = P.pgran;
    e = scan(p, kMinima, P.psplits, fp8 ? "tc_prepass_fp8" : "tc_prepass_fp16", pair, groups > 2 ? 2 : groups);
    if (e != cudaSuccess) return (int)e;
    {
      ProfScope ps("tc_tau", stream);
      launch_tau(p.pmin, nq, P.pcount, P.pcount, P.pr, TauMargin{}, tau, redo, stream);
      note_launch();
    }
  }
  a.splits = splits;
  a.partial = partial;
  a.kl = kl;
  a.share = (kl == shortlist && !prepass) ? 1u : 0u;
  a.qbound = tau;
  e = scan(a, prepass ? kLists : (int)kl_tmpl, splits, fp8 ? "tc_scan_fp8" : "tc_scan_fp16", pair, groups);
  if (e != cudaSuccess) return (int)e;

  // The keys that a block sorts: all of them without a bound; with one, about
  // r s rows pass it, within 5 standard deviations of the sampled rank (a
  // query beyond that selects by its kp-th key). Room for every list instead
  // (up to 128 KB) left one block per SM.
  const uint32_t all_keys = next_pow2(splits * groups * kl);
  const double foreseen = (double)P.pstride * (P.pr + (P.pstride > 1 ? 5.0 * std::sqrt((double)P.pr) : 0.125 * P.pr));
  const uint32_t foreseen_keys = next_pow2((uint32_t)std::min(foreseen, 16384.0) + 64u);
  const uint32_t sel_keys = std::max(std::max(2u, next_pow2(shortlist)), prepass ? std::min(all_keys, foreseen_keys) : all_keys);
  SelectArgs s{partial, splits * groups, kl, sel_keys, shortlist, k, queries, t.vectors, t.dim,
               (int)metric,
               opt.boundary_fp64 ? 1u : 0u, 0.f, out, status_word(), tau, redo, nullptr, incomplete_q};
  s.eps = opt.boundary_eps > 0.f ? opt.boundary_eps : (float)((t.dim + 31) / 32 + 5) * 2.0f * 5.960464477539063e-08f;
  size_t sel_smem = (size_t)sel_keys * 8;
  const int sel_threads = nq <= 2u * (uint32_t)device_sm_count() ? 1024 : 256;
  auto select = sel_threads == 1024 ? tc_select_kernel<1024> : tc_select_kernel<256>;
  e = cudaFuncSetAttribute(select, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sel_smem);
  if (e != cudaSuccess) return (int)e;
  {
    ProfScope ps("tc_select_rescore", stream);
    select<<<nq, sel_threads, sel_smem, stream>>>(s);
    note_launch();
  }
  if (prepass && (P.pstride > 1 || kl < shortlist)) {
    // queries whose bound was too tight, or whose range it admits overflowed:
    // scanned again without it (blocks holding none of them exit at once), then
    // selected again
    TcScanArgs f = a;
    f.qbound = nullptr;
    f.active = redo;
    f.share = 0;
    e = scan(f, (int)kl_tmpl, splits, fp8 ? "tc_rescan_fp8" : "tc_rescan_fp16", false, groups);
    if (e != cudaSuccess) return (int)e;
    SelectArgs r = s;
    r.cap = std::max(sel_keys, all_keys);
    sel_smem = (size_t)r.cap * 8;
    e = cudaFuncSetAttribute(select, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sel_smem);
    if (e != cudaSuccess) return (int)e;
    r.tau = nullptr;
    r.redo = nullptr;
    r.only = redo;
    ProfScope ps("tc_select_rescore", stream);
    select<<<nq, sel_threads, sel_smem, stream>>>(r);
    note_launch();
  }
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Collecting pass (flat_tc.cu): the minima pass and the bounded scan over
// prepared fp16 rows and queries, ranking by max(floor, qnorm + norm -
// 2 dot). Leaves the range lists and the bounds for the caller to finish.
// ---------------------------------------------------------------------------
bool plan_tc_collect(TcCollect& c) {
  const TcTables t{false, c.rows16, c.row_norms, nullptr, nullptr, c.n, c.dim, c.padded_dim};
  c.plan = plan_tc_scan(t, c.nq, c.room, METRIC_L2, FvScanOptions{0, 0, 0.f, 0}, c.rank);
  c.query_rows = c.plan.nq_rows;
  c.bytes = c.plan.part_bytes + c.plan.tau_bytes;
  return c.plan.prepass;
}

int launch_tc_collect(TcCollect& c, void* scratch, cudaStream_t stream) {
  const TcPlan& P = c.plan;
  c.partial = static_cast<uint64_t*>(scratch);
  c.bound = reinterpret_cast<float*>(static_cast<uint8_t*>(scratch) + P.part_bytes);
  c.flags = reinterpret_cast<uint32_t*>(c.bound + c.nq);
  c.lists = P.splits * P.groups;
  c.kl = P.kl;
  const uint64_t row_bytes = (uint64_t)c.padded_dim * 2;
  CUtensorMap ta, tb, tb_half, tb_runs;
  if (!encode_tmap(&ta, c.q16, false, c.padded_dim, P.nq_rows, row_bytes, TC_M) ||
      !encode_tmap(&tb, c.rows16, false, c.padded_dim, c.n, row_bytes, TC_N) ||
      (P.pair && !encode_tmap(&tb_half, c.rows16, false, c.padded_dim, c.n, row_bytes, TC_N / 2)) ||
      !encode_runs(&tb_runs, c.rows16, false, c.padded_dim, row_bytes, P.pstride, P.ptiles, P.pair ? RUNS / 2 : RUNS))
    return FV_ERR_ARG;
  TcScanArgs a{};
  a.n = c.n;
  a.nq = c.nq;
  a.kblocks = P.kblocks;
  a.nqb = P.nqb;
  a.xnorm = c.row_norms;
  a.qnorm = c.qnorm;
  a.mask = c.mask;
  a.floor = c.floor;
  a.status = c.status;
  const int64_t wl = tune_value("tc.wait_limit_ns", 0);
  a.wait_ns = wl > 0 ? (uint64_t)wl : 2000000000ull;
  auto scan = [&](const TcScanArgs& args, int kl_t, uint32_t splits_n, const char* name) -> cudaError_t {
    ProfScope ps(name, stream);
    return dispatch_tc_scan_fp16(kl_t, P.pair ? -1 : P.groups, METRIC_L2, true, ta,
                                 kl_t == kMinima ? tb_runs : P.pair ? tb_half : tb, args,
                                 (P.pair ? P.nqb_grid : P.nqb) * splits_n, stream);
  };
  TcScanArgs p = a;
  p.splits = P.psplits;
  p.xnorm = c.row_norms_min;
  p.run_stride = P.pstride;
  p.pmin = reinterpret_cast<float*>(c.partial);
  p.pm_stride = P.pcount;
  p.gran = P.pgran;
  cudaError_t e = scan(p, kMinima, P.psplits, "tc_prepass_fp16");
  if (e != cudaSuccess) return (int)e;
  {
    ProfScope ps("tc_tau", stream);
    const TauMargin m{c.margin_rel, c.margin_norm, c.margin_abs, c.qnorm};
    launch_tau(p.pmin, c.nq, P.pcount, P.pcount, P.pr, m, c.bound, c.flags, stream);
    note_launch();
  }
  a.splits = P.splits;
  a.partial = c.partial;
  a.kl = P.kl;
  a.qbound = c.bound;
  return (int)scan(a, kLists, P.splits, "tc_scan_fp16");
}

}  // namespace fv

extern "C" int fv_tune_lookup(int fp8, MetricType metric, uint32_t dim, uint64_t num_vectors, uint32_t num_queries,
                              uint32_t top_k, int32_t* out_knobs) {
  if (!out_knobs) return FV_ERR_NULL;
  const fv::TuneEntry* e = fv::tune_lookup(fp8 != 0, (int)metric, dim, num_vectors, num_queries, top_k);
  if (!e) return FV_ERR_ARG;
  out_knobs[0] = e->pair;
  out_knobs[1] = e->prepass;
  out_knobs[2] = e->stride;
  out_knobs[3] = e->overfetch;
  return 0;
}

