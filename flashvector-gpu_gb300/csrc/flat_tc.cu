// flat_tc.cu -- exact fp32 flat scan of a batch behind a tensor-core filter.
//
// The plain exact scan (flat_fp32.cu) evaluates every (query, row) pair on the
// CUDA cores, three separately rounded operations per dimension: 100,000 x
// 128 x 1,000 takes 1.5 ms of which 1.0 ms is that arithmetic. Here the
// tensor cores evaluate a LOWER BOUND of every pair's distance from fp16
// copies of the rows, made per call, and only the rows whose lower bound does
// not exceed a bound on the query's k-th distance are evaluated exactly, with
// the plain scan's operations in the plain scan's order. The answer is the
// plain scan's bit for bit:
//
//   * rows and queries are scaled by powers of two (L2 also centred on the
//     mean of a sample, cosine normalised), X and Q; A is the distance in
//     that scale: ||Q - X||^2 (L2), -2 <Q, X> (inner product, cosine);
//   * the pass ranks by a = (norm terms) - 2 <fp16(Q), fp16(X)> - e H, with
//     H = |Q|^2 + |X|^2, which is at most A as the plain scan would round it:
//     with |Q||X| <= H / 2, the fp16 rounding of both sides (2^-11 each)
//     moves -2 <Q, X> by at most (2^-10 + 2^-22) H, values below fp16's
//     normal range by 2^-24 sqrt(dim) (1 + H), the fp32 accumulation by
//     dim 2^-23 H, the norms by dim 2^-24 H, the additions and the centring
//     by 2^-21 H, the plain scan's own rounding by dim 2^-24 H (inner
//     product; for L2 it is relative and tested below; cosine adds its
//     normalisation and its 1e-8). e sums these with slack (error_bound);
//   * a row that was not collected has a >= B, the query's bound (lowered to
//     the largest key of any list that filled up), hence A >= B: when the
//     k-th exact distance among the collected rows is below B the collected
//     rows hold the answer. A query that fails this test, or whose values
//     leave fp16's range, is flagged, and the plain scan answers it; so are
//     all of a call one of whose passes gave up a wait;
//   * a row that leaves fp16's range, or is not finite, has no such bound: it
//     gets zero codes, no part in the minima and a = -inf in the scan, so that
//     every query collects it. (One such row in 100,000 x 128 x 1,000 used to
//     flag every query: 1,698 us, plain scan 1,612; now 173.)
//
// Measured: 100,000 x 128 x 1,000, k 10: 1,592 -> 160 us (encoding 37, minima
// pass 37, scan 50, finish 15); 200,000 x 512 x 100: 1,131 -> 263 us. Bounded
// by the epilogues of the two tensor-core passes and, for few queries, by the
// encoding (6 bytes a value).
#include <cuda_fp16.h>

#include <cmath>

#include "../../include/fv_bridge.h"
#include "common.cuh"
#include "kernels.h"
#include "topk.cuh"

namespace fv {

namespace {

constexpr uint32_t SAMPLE = 256;     // rows behind the centre and the scale
constexpr int CEN_GROUPS = 32;       // row groups of a centring block
constexpr int PREP_WARPS = 8;
constexpr uint32_t PREP_ROWS = 4;    // rows in flight per lane group
constexpr int FIN_THREADS = 128;
constexpr uint32_t FIN_KEYS = 1024;  // collected rows of a query that are evaluated
constexpr float kMaxNorm = 3.0e4f;   // of a scaled row or query: no fp16 value overflows
constexpr float kUnit = 256.f;       // norm of a scaled unit vector (cosine)

// words of the call's shared state
enum { W_MIN_NORM = 0, W_STATUS = 1, W_COUNT = 2 };  // smallest row norm (cosine), status bits of the scans

struct QueryInfo {
  float to_a;    // A = to_a * distance (cosine: to_a * (distance - 1))
  float norm;    // |q| unscaled (cosine)
  float scaled;  // |Q|
  float pad;
};

// mu[d] and the variance about it (inner product, cosine: 0 and the mean
// square), over up to 256 evenly spaced rows (values that are not finite left
// out: any centre and scale will do). A block owns 32 dimensions.
__global__ void __launch_bounds__(32 * CEN_GROUPS) flat_tc_center_kernel(const float* __restrict__ x, uint32_t n,
                                                                         uint32_t dim, int metric,
                                                                         float* __restrict__ mu,
                                                                         float* __restrict__ var,
                                                                         uint32_t* __restrict__ words) {
  __shared__ float part[CEN_GROUPS][33];
  const uint32_t lane = threadIdx.x & 31, g = threadIdx.x >> 5;
  const uint32_t d = blockIdx.x * 32 + lane;
  const uint32_t s = min(n, SAMPLE);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    words[W_MIN_NORM] = 0x7f800000u;  // +inf
    words[W_STATUS] = 0u;
  }
  auto total = [&](float v) {  // over the row groups, to every thread of the dimension
    part[g][lane] = v;
    __syncthreads();
    float sum = 0.f;
#pragma unroll
    for (int r = 0; r < CEN_GROUPS; ++r) sum += part[r][lane];
    __syncthreads();
    return sum;
  };
  float m = 0.f, acc = 0.f;
  if (metric == METRIC_L2) {
    if (d < dim) {
#pragma unroll 8
      for (uint32_t i = g; i < s; i += CEN_GROUPS) {
        const float v = __ldg(x + (size_t)((uint64_t)i * n / s) * dim + d);
        acc += fabsf(v) < INFINITY ? v : 0.f;
      }
    }
    m = total(acc) / (float)s;
  }
  acc = 0.f;
  if (d < dim) {
#pragma unroll 8
    for (uint32_t i = g; i < s; i += CEN_GROUPS) {
      const float v = __ldg(x + (size_t)((uint64_t)i * n / s) * dim + d) - m;
      acc = fabsf(v) < INFINITY ? fmaf(v, v, acc) : acc;
    }
  }
  acc = total(acc) / (float)s;
  if (g == 0 && d < dim) {
    mu[d] = m;
    var[d] = acc;
  }
}

// power of two that takes a norm to [256, 512) (1 for zero and non-finite)
__device__ __forceinline__ float scale_for(float norm) {
  if (!(norm > 0.f) || !(norm < 3.0e38f)) return 1.f;
  return ldexpf(1.f, max(-60, min(60, 8 - ilogbf(norm))));
}

struct PrepArgs {
  const float* x;
  const float* q;
  uint32_t n, nq, nq_rows, dim, pd;
  int metric;
  float e, e_abs;
  const float* mu;
  const float* var;
  __half* x16;
  __half* q16;
  float* xnorm;       // of the scan: -inf for a row out of range
  float* xnorm_min;   // of the minima pass: inf there
  float* qnorm;
  QueryInfo* info;
  const uint32_t* mask;
  uint32_t* words;
};

// Rows [0, n) are base rows, then nq_rows queries (those past nq zero). LPR
// lanes take a row, E = 4 (VEC) or 1 consecutive dimensions each, so short
// rows share a warp; PREP_ROWS rows of a lane group are in flight together
// (one row at a time, a warp per row, moved 3 TB/s).
template <bool VEC, int LPR>
__global__ void __launch_bounds__(32 * PREP_WARPS) flat_tc_prep_kernel(PrepArgs a) {
  constexpr int E = VEC ? 4 : 1;
  constexpr uint32_t R = PREP_ROWS;
  const uint32_t lane = threadIdx.x & 31, sub = lane % LPR;
  const uint64_t rows = (uint64_t)a.n + a.nq_rows;
  auto group_sum = [](float v) {
#pragma unroll
    for (int o = LPR / 2; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  };
  float s = 1.f;
  if (a.metric != METRIC_COSINE) {
    float v = 0.f;
    for (uint32_t d = lane; d < a.dim; d += 32) v += __ldg(a.var + d);
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    s = scale_for(sqrtf(v));
  }
  // smallest row norm (cosine) of the warp's rows: one atomic a warp, and only
  // where it moves the word (an atomic per row took 40 us for 100,000 rows)
  uint32_t w_min = 0x7f800000u;
  constexpr uint64_t WARP_ROWS = (uint64_t)R * (32 / LPR);
  for (uint64_t wb = ((uint64_t)blockIdx.x * PREP_WARPS + (threadIdx.x >> 5)) * WARP_ROWS; wb < rows;
       wb += (uint64_t)gridDim.x * PREP_WARPS * WARP_ROWS) {
    const uint64_t w0 = wb + lane / LPR * R;
    // row i of this lane group: its source (null: a padding query, or no row) and multiplier
    const float* src[R];
    float mult[R], norm[R];
    bool odd[R];
    bool own = false;  // some row's scale comes from its own norm
#pragma unroll
    for (uint32_t i = 0; i < R; ++i) {
      const uint64_t w = w0 + i;
      const bool is_q = w >= a.n;
      const uint64_t r = is_q ? w - a.n : w;
      src[i] = w >= rows || (is_q && r >= a.nq) ? nullptr : (is_q ? a.q : a.x) + r * a.dim;
      mult[i] = s;
      norm[i] = 0.f;
      odd[i] = false;
      own = own || (a.metric == METRIC_INNER_PRODUCT && is_q);
    }
    if (__any_sync(0xffffffffu, own || a.metric == METRIC_COSINE)) {
      float v[R], amax[R];
#pragma unroll
      for (uint32_t i = 0; i < R; ++i) v[i] = amax[i] = 0.f;
      for (uint32_t d = sub; d < a.dim; d += LPR) {
#pragma unroll
        for (uint32_t i = 0; i < R; ++i) {
          const float f = src[i] ? __ldg(src[i] + d) : 0.f;
          v[i] = fmaf(f, f, v[i]);
          amax[i] = fmaxf(amax[i], fabsf(f));
        }
      }
#pragma unroll
      for (uint32_t i = 0; i < R; ++i) {
#pragma unroll
        for (int o = LPR / 2; o; o >>= 1) amax[i] = fmaxf(amax[i], __shfl_xor_sync(0xffffffffu, amax[i], o));
        const float nr = sqrtf(group_sum(v[i]));
        if (a.metric == METRIC_COSINE) {
          norm[i] = nr;
          mult[i] = nr > 0.f ? __fdiv_rn(kUnit, nr) : 0.f;
          // a norm outside [1e-18, 1e18] (zero apart) has lost digits
          odd[i] = amax[i] > 0.f && !(nr > 1e-18f && nr < 1e18f);
        } else if (w0 + i >= a.n) {
          mult[i] = scale_for(nr);  // an inner-product query has a scale of its own
        }
      }
    }
    float n2[R];
#pragma unroll
    for (uint32_t i = 0; i < R; ++i) n2[i] = 0.f;
    for (uint32_t d = E * sub; d < a.pd; d += E * LPR) {
      float m[E], v[R][E];
#pragma unroll
      for (int e = 0; e < E; ++e) m[e] = 0.f;
      if (d < a.dim) {  // (VEC: dim is a multiple of 4)
        if constexpr (VEC) {
          const float4 t = __ldg(reinterpret_cast<const float4*>(a.mu + d));
          m[0] = t.x;
          m[1] = t.y;
          m[2] = t.z;
          m[3] = t.w;
        } else {
          m[0] = __ldg(a.mu + d);
        }
      }
#pragma unroll
      for (uint32_t i = 0; i < R; ++i) {
        if constexpr (VEC) {
          float4 t = make_float4(m[0], m[1], m[2], m[3]);
          if (src[i] && d < a.dim) t = __ldg(reinterpret_cast<const float4*>(src[i] + d));
          v[i][0] = t.x;
          v[i][1] = t.y;
          v[i][2] = t.z;
          v[i][3] = t.w;
        } else {
          v[i][0] = src[i] && d < a.dim ? __ldg(src[i] + d) : m[0];
        }
      }
#pragma unroll
      for (uint32_t i = 0; i < R; ++i) {
#pragma unroll
        for (int e = 0; e < E; ++e) {
          v[i][e] = __fmul_rn(__fsub_rn(v[i][e], m[e]), mult[i]);
          n2[i] = fmaf(v[i][e], v[i][e], n2[i]);
        }
        const uint64_t w = w0 + i;
        if (w >= rows) continue;
        __half* dst = (w >= a.n ? a.q16 + (w - a.n) * a.pd : a.x16 + w * a.pd) + d;
        if constexpr (VEC) {
          const __half2 h0 = __floats2half2_rn(v[i][0], v[i][1]), h1 = __floats2half2_rn(v[i][2], v[i][3]);
          uint2 o;
          o.x = *reinterpret_cast<const uint32_t*>(&h0);
          o.y = *reinterpret_cast<const uint32_t*>(&h1);
          *reinterpret_cast<uint2*>(dst) = o;
        } else {
          *dst = __float2half_rn(v[i][0]);
        }
      }
    }
#pragma unroll
    for (uint32_t i = 0; i < R; ++i) {
      const float nn = group_sum(n2[i]);
      if (!src[i]) continue;
      const uint64_t w = w0 + i;
      const float low = a.metric == METRIC_L2 ? nn - a.e * nn : -a.e * nn;
      if (w >= a.n) {
        if (sub) continue;
        const uint64_t r = w - a.n;
        a.qnorm[r] = low;
        QueryInfo inf;
        inf.to_a = a.metric == METRIC_L2 ? s * s
                                         : a.metric == METRIC_INNER_PRODUCT ? 2.f * s * mult[i] : 2.f * kUnit * kUnit;
        inf.norm = norm[i];
        inf.scaled = odd[i] ? INFINITY : sqrtf(nn);
        inf.pad = 0.f;
        a.info[r] = inf;
        continue;
      }
      const bool out = odd[i] || !(sqrtf(nn) < kMaxNorm);
      if (out) {
        // (each lane over what it wrote)
        for (uint32_t d = E * sub; d < a.pd; d += E * LPR) {
#pragma unroll
          for (int e = 0; e < E; ++e) a.x16[w * a.pd + d + e] = __float2half_rn(0.f);
        }
      }
      if (sub) continue;
      a.xnorm[w] = out ? -INFINITY : low - a.e_abs;
      a.xnorm_min[w] = out ? INFINITY : low - a.e_abs;
      if (a.metric == METRIC_COSINE && !out && norm[i] > 0.f && mask_allows(a.mask, (uint32_t)w))
        w_min = min(w_min, __float_as_uint(norm[i]));
    }
  }
  w_min = __reduce_min_sync(0xffffffffu, w_min);
  if (lane == 0 && w_min < __ldcg(a.words + W_MIN_NORM)) atomicMin(a.words + W_MIN_NORM, w_min);
}

// The plain scan's distance of one row (flat_f32_scan_kernel): separately
// rounded operations in dimension order. qv in shared memory.
template <int METRIC, bool VEC>
__device__ __forceinline__ float exact_distance(const float* qv, const float* __restrict__ x, uint32_t dim,
                                                float qnorm) {
  float acc = 0.f, xn = 0.f;
  auto term = [&](float q, float v) {
    if (METRIC == METRIC_L2) {
      const float diff = __fsub_rn(q, v);
      acc = __fadd_rn(acc, __fmul_rn(diff, diff));
    } else {
      acc = __fadd_rn(acc, __fmul_rn(q, v));
      if (METRIC == METRIC_COSINE) xn = __fadd_rn(xn, __fmul_rn(v, v));
    }
  };
  uint32_t d = 0;
  if constexpr (VEC) {
    for (; d + 32 <= dim; d += 32) {
      float4 v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = __ldg(reinterpret_cast<const float4*>(x + d) + i);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 q = *reinterpret_cast<const float4*>(qv + d + 4 * i);
        term(q.x, v[i].x);
        term(q.y, v[i].y);
        term(q.z, v[i].z);
        term(q.w, v[i].w);
      }
    }
  } else {
    for (; d + 16 <= dim; d += 16) {
      float v[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = __ldg(x + d + i);
#pragma unroll
      for (int i = 0; i < 16; ++i) term(qv[d + i], v[i]);
    }
  }
  for (; d < dim; ++d) term(qv[d], __ldg(x + d));
  if (METRIC == METRIC_L2) return acc;
  if (METRIC == METRIC_INNER_PRODUCT) return -acc;
  const float denom = __fadd_rn(__fmul_rn(sqrtf(qnorm), sqrtf(xn)), 1e-8f);
  return __fsub_rn(1.0f, __fdiv_rn(acc, denom));
}

struct FinishArgs {
  const float* x;
  const float* q;
  const uint32_t* vec_ids;
  uint32_t n, dim, k;
  const uint64_t* partial;
  uint32_t lists, kl;
  const float* bound;
  const QueryInfo* info;
  const uint32_t* words;
  float slack;  // relative (L2) or absolute margin of the final test
  uint32_t* flags;
  GpuSearchResult* out;
};

// One block per query: the collected rows' exact distances, the first k by
// (distance, slot), and the test that no other row can be among them.
template <int METRIC, bool VEC>
__global__ void __launch_bounds__(FIN_THREADS) flat_tc_finish_kernel(FinishArgs a) {
  extern __shared__ __align__(16) float qv[];  // [dim]
  __shared__ __align__(16) uint64_t keys[FIN_KEYS];
  __shared__ uint32_t n_live, s_low;
  __shared__ float s_qnorm;
  const uint32_t q = blockIdx.x, tid = threadIdx.x;
  for (uint32_t d = tid; d < a.dim; d += FIN_THREADS) qv[d] = __ldg(a.q + (size_t)q * a.dim + d);
  if (tid == 0) s_low = float_order(a.bound[q]);
  __syncthreads();
  if (METRIC == METRIC_COSINE && tid == 32) {
    float s = 0.f;
    for (uint32_t d = 0; d < a.dim; ++d) s = __fadd_rn(s, __fmul_rn(qv[d], qv[d]));
    s_qnorm = s;
  }
  const uint32_t total = a.lists * a.kl;
  const uint64_t* src = a.partial + (size_t)q * total;
  for (uint32_t l = tid; l < a.lists; l += FIN_THREADS) {
    const uint64_t root = src[(size_t)l * a.kl];
    if (root != kSentinelKey) atomicMin(&s_low, (uint32_t)(root >> 32));
  }
  uint32_t live = block_compact_keys(src, total, keys, &n_live, FIN_KEYS);
  if (live > FIN_KEYS) {
    const uint64_t limit = block_kth_key(src, total, FIN_KEYS);
    live = block_compact_keys(src, total, keys, &n_live, FIN_KEYS, limit);
    if (tid == 0) atomicMin(&s_low, (uint32_t)(limit >> 32));
  }
  __syncthreads();
  const float qnorm = METRIC == METRIC_COSINE ? s_qnorm : 0.f;
  for (uint32_t c = tid; c < live; c += FIN_THREADS) {
    const uint32_t slot = key_slot(keys[c]);
    const float d = exact_distance<METRIC, VEC>(qv, a.x + (size_t)slot * a.dim, a.dim, qnorm);
    keys[c] = d < kSentinelDist ? make_key(d, slot) : kSentinelKey;
  }
  const uint32_t sp2 = next_pow2_dev(max(max(live, a.k), 2u));
  for (uint32_t i = live + tid; i < sp2; i += FIN_THREADS) keys[i] = kSentinelKey;
  __syncthreads();
  block_bitonic_sort(keys, sp2);
  for (uint32_t r = tid; r < a.k; r += FIN_THREADS) a.out[(size_t)q * a.k + r] = key_to_result(keys[r], a.vec_ids);
  if (tid == 0) {
    const QueryInfo inf = a.info[q];
    const float low = order_float(s_low);
    // (a pass that gave up a wait has not seen every row)
    bool ok = a.words[W_STATUS] == 0u && inf.scaled < kMaxNorm;
    if (METRIC == METRIC_COSINE) ok = ok && inf.norm * __uint_as_float(a.words[W_MIN_NORM]) > 8.2e-5f;
    if (ok && low < kSentinelDist) {  // else every admissible row was collected
      const uint64_t kth = keys[a.k - 1];
      const float t = key_dist(kth);
      ok = kth != kSentinelKey &&
           (METRIC == METRIC_L2 ? t * inf.to_a < low * (1.f - a.slack)
                                : inf.to_a * (METRIC == METRIC_COSINE ? t - 1.f : t) < low - a.slack * fabsf(low));
    }
    if (!ok) a.flags[q] = 1u;
  }
}

// e of the file comment.
float error_bound(uint32_t dim, MetricType metric) {
  const double d = dim, sub = std::ldexp(std::sqrt(d), -24);
  if (metric == METRIC_COSINE) return (float)(std::ldexp(1.0, -10) + 1.5 * std::ldexp(d, -22) + std::ldexp(1.0, -12) + sub);
  return (float)(std::ldexp(1.0, -10) + 1.25 * std::ldexp(d, -22) + std::ldexp(1.0, -20) + sub);
}

// Pairs x dimensions from which the filter is the faster way: below, its eight
// launches and the encoding outweigh the arithmetic that it saves (50,000 x 64
// x 32: 70 against 54 us; 20,000 x 64 x 100, 1.3e8: 68 against 88).
constexpr uint64_t kFlatTcWork = 120000000ull;
// The copies and lists live in the stream's scratch (scratch_try), which keeps
// up to a quarter more until it is released.
constexpr size_t kMaxScratch = (size_t)1 << 30;

}  // namespace

FlatTcPlan plan_flat_tc(uint32_t n, uint32_t dim, uint32_t nq, uint32_t k, MetricType metric) {
  FlatTcPlan P;
  const int64_t knob = tune_value("flat.tc", -1);
  const bool forced = knob == 1;
  if (knob == 0 || nq < 32 || n < 2048 || dim < 8 || dim > 4096) return P;
  if (!forced && (uint64_t)nq * n * dim < kFlatTcWork) return P;
  P.pd = (dim + 15) / 16 * 16;
  const size_t table = (size_t)n * P.pd * 2;
  if (table > kMaxScratch) return P;
  P.f = plan_flat_f32(n, nq, k, 0);
  TcCollect& c = P.c;
  c.n = n;
  c.dim = dim;
  c.padded_dim = P.pd;
  c.nq = nq;
  c.rank = k;
  c.room = 2 * k + 64;
  const float e = error_bound(dim, metric);
  // how far a bound on the lower bounds is raised so that it is, as a rule,
  // also a bound on the distances themselves: the k best rows have A <= a +
  // 2 e H with H about 3 |Q|^2 + 2 A (L2; they are near the query) or the
  // norms' sum
  if (metric == METRIC_L2) {
    c.floor = 0.f;
    c.margin_rel = 8.f * e;
    c.margin_norm = 8.f * e;
    c.margin_abs = 1.f;
  } else {
    c.floor = -INFINITY;
    c.margin_rel = 0.f;
    c.margin_norm = metric == METRIC_COSINE ? 0.f : 3.f;  // qnorm holds -e |Q|^2
    c.margin_abs = metric == METRIC_COSINE ? 5.f * e * kUnit * kUnit : 2.f * e * 524288.f;
  }
  if (!plan_tc_collect(c)) return P;
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t o = at;
    at = (at + bytes + 1023) / 1024 * 1024;
    return o;
  };
  P.x16 = take(table);
  P.xnorm = take((size_t)n * 4);
  P.xnorm_min = take((size_t)n * 4);
  P.q16 = take((size_t)c.query_rows * P.pd * 2);
  P.qnorm = take((size_t)nq * 4);
  P.info = take((size_t)nq * sizeof(QueryInfo));
  P.mu = take((size_t)dim * 4);
  P.var = take((size_t)dim * 4);
  P.words = take(W_COUNT * 4);
  P.collect = take(c.bytes);
  P.plain = take(P.f.scratch_bytes);
  if (at <= kMaxScratch) P.bytes = at;
  return P;
}

int launch_flat_tc(const FlatTcPlan& P, const float* vectors, const uint32_t* vec_ids, uint32_t n, uint32_t dim,
                   const float* queries, uint32_t nq, uint32_t k, MetricType metric, const uint32_t* mask,
                   GpuSearchResult* out, void* scratch, cudaStream_t stream) {
  uint8_t* base = static_cast<uint8_t*>(scratch);
  const bool vec = dim % 4 == 0 && (uintptr_t)vectors % 16 == 0 && (uintptr_t)queries % 16 == 0;
  float* mu = reinterpret_cast<float*>(base + P.mu);
  float* var = reinterpret_cast<float*>(base + P.var);
  uint32_t* words = reinterpret_cast<uint32_t*>(base + P.words);
  PrepArgs p{};
  p.x = vectors;
  p.q = queries;
  p.n = n;
  p.nq = nq;
  p.nq_rows = P.c.query_rows;
  p.dim = dim;
  p.pd = P.pd;
  p.metric = (int)metric;
  p.e = error_bound(dim, metric);
  p.e_abs = (float)std::ldexp(std::sqrt((double)dim), -23);
  p.mu = mu;
  p.var = var;
  p.x16 = reinterpret_cast<__half*>(base + P.x16);
  p.q16 = reinterpret_cast<__half*>(base + P.q16);
  p.xnorm = reinterpret_cast<float*>(base + P.xnorm);
  p.xnorm_min = reinterpret_cast<float*>(base + P.xnorm_min);
  p.mask = mask;
  p.qnorm = reinterpret_cast<float*>(base + P.qnorm);
  p.info = reinterpret_cast<QueryInfo*>(base + P.info);
  p.words = words;
  {
    ProfScope ps("flat_tc_prep", stream);
    flat_tc_center_kernel<<<(dim + 31) / 32, 32 * CEN_GROUPS, 0, stream>>>(vectors, n, dim, (int)metric, mu, var,
                                                                           words);
    const uint64_t rows = (uint64_t)n + P.c.query_rows;
    auto prep = [&](auto kern, uint32_t lanes) {
      const uint64_t per_block = (uint64_t)PREP_WARPS * PREP_ROWS * (32 / lanes);
      const uint32_t blocks = (uint32_t)std::min<uint64_t>((rows + per_block - 1) / per_block, 8ull * device_sm_count());
      kern<<<blocks, 32 * PREP_WARPS, 0, stream>>>(p);
    };
    if (vec) {
      if (P.pd <= 16)
        prep(flat_tc_prep_kernel<true, 4>, 4);
      else if (P.pd <= 32)
        prep(flat_tc_prep_kernel<true, 8>, 8);
      else if (P.pd <= 64)
        prep(flat_tc_prep_kernel<true, 16>, 16);
      else
        prep(flat_tc_prep_kernel<true, 32>, 32);
    } else if (P.pd <= 16) {
      prep(flat_tc_prep_kernel<false, 16>, 16);
    } else {
      prep(flat_tc_prep_kernel<false, 32>, 32);
    }
    note_launch(2);
  }
  TcCollect c = P.c;
  c.rows16 = p.x16;
  c.row_norms = p.xnorm;
  c.row_norms_min = p.xnorm_min;
  c.q16 = p.q16;
  c.qnorm = p.qnorm;
  c.mask = mask;
  c.status = words + W_STATUS;
  int rc = launch_tc_collect(c, base + P.collect, stream);
  if (rc) return rc;
  const float slack = metric == METRIC_L2 ? (float)std::ldexp((double)dim + 2, -23) : 1e-6f;
  FinishArgs f{vectors, queries, vec_ids, n, dim, k, c.partial, c.lists, c.kl, c.bound, p.info, words, slack,
               c.flags, out};
  {
    ProfScope ps("flat_tc_finish", stream);
    const size_t smem = (size_t)dim * 4;
    auto go = [&](auto kern) { kern<<<nq, FIN_THREADS, smem, stream>>>(f); };
    switch (metric) {
      case METRIC_INNER_PRODUCT:
        vec ? go(flat_tc_finish_kernel<METRIC_INNER_PRODUCT, true>)
            : go(flat_tc_finish_kernel<METRIC_INNER_PRODUCT, false>);
        break;
      case METRIC_COSINE:
        vec ? go(flat_tc_finish_kernel<METRIC_COSINE, true>) : go(flat_tc_finish_kernel<METRIC_COSINE, false>);
        break;
      default: vec ? go(flat_tc_finish_kernel<METRIC_L2, true>) : go(flat_tc_finish_kernel<METRIC_L2, false>); break;
    }
    note_launch();
  }
  return launch_flat_f32_planned(P.f, vectors, vec_ids, n, dim, queries, nq, k, metric, mask, out, false,
                                 P.f.scratch_bytes ? base + P.plain : nullptr, stream, nullptr, c.flags);
}

}  // namespace fv
