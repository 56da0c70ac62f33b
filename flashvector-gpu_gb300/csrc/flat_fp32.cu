// flat_fp32.cu -- exact fp32 flat scan fused with top-k.
//
// Replaces the reference's flat_scan_kernel / launch_flat_scan
// (sparse_hybrid.cu:13-107). Same contract, different machine mapping:
//
//  * a CTA owns QT queries (8, 16, 32 or 64) and a contiguous range of base
//    tiles (128 rows); every base tile is staged once in shared memory and
//    scored against all its queries (the reference re-streams the whole base
//    set per query);
//  * each thread accumulates up to a 4 x 8 block of (query, row) distances,
//    walking the dimensions in ascending order with separately rounded
//    subtract / multiply / add -- the order of the reference's own exact
//    search RecallEvaluator::exact_knn (metrics.rs:103-135), so distances
//    are bit-identical to it;
//  * per query the running top-k is a sorted list of (distance, slot) keys in
//    shared memory (ties -> lower slot, as the reference's strict `<`
//    insertion in slot order); after each tile every thread tests its own
//    block against the queries' current k-th keys and appends only the keys
//    that can enter to a per-query candidate list, which a warp sorts in
//    registers and merges into the query's list;
//  * when the base range is split over several CTAs the per-split lists go
//    to scratch and a second kernel merges them.
#include <mutex>
#include <type_traits>

#include "../../include/fv_bridge.h"
#include "common.cuh"
#include "kernels.h"
#include "topk.cuh"

namespace fv {

namespace {

constexpr int QT_MAX = 64;  // queries per CTA: 8, 16, 32 or 64
constexpr int VT = 128;     // base rows per tile
constexpr int DK = 32;      // dimensions per staged chunk
constexpr int NT = 256;     // threads per CTA
constexpr int NW = NT / 32;

struct FlatArgs {
  const float* vectors;
  const uint32_t* vec_ids;
  uint32_t n, dim;
  const float* queries;
  uint32_t nq, k;
  const uint32_t* mask;
  GpuSearchResult* out;   // written directly when splits == 1
  uint64_t* partial;      // [nq][splits][k] sorted lists when splits > 1
  uint32_t splits, tiles_per_split;
  const QueryFilter* filters;  // per-query filters over logical ids (vec_ids[slot], or slot), or null
  const uint32_t* active;      // only the flagged queries (blocks without one leave at once), or null
};

// Merges the m (<= 128) candidates of one query's tile into its sorted list
// list[0, k); returns the new k-th key. Warp-collective. Short lists (k <= 32)
// take the candidates 32 at a time, one key a lane; longer ones all at once,
// four keys a lane. In each step min(list[i], candidates[last - i]) keeps the
// smallest keys of both as one bitonic sequence, which a merge then sorts. A
// handful of candidates (the usual tile once the list is warm) are inserted
// one by one instead: a ballot finds the place, a shuffle moves the tail.
constexpr uint32_t INSERT_MAX = 6;  // a merge of 32 candidates costs about as much as 12 insertions
template <int NR>
__device__ __forceinline__ uint64_t list_insert(uint64_t* list, uint32_t k, const float* cd, const uint8_t* cr,
                                                uint32_t m, uint32_t v0) {
  const uint32_t lane = threadIdx.x & 31u;
  uint64_t l[NR];  // key 32 j + lane
#pragma unroll
  for (int j = 0; j < NR; ++j) l[j] = 32 * j + lane < k ? list[32 * j + lane] : kSentinelKey;
  for (uint32_t i = 0; i < m; ++i) {
    const uint64_t c = make_key(cd[i], v0 + cr[i]);
    uint32_t at = 0;  // keys before c
#pragma unroll
    for (int j = 0; j < NR; ++j) at += __popc(__ballot_sync(0xffffffffu, l[j] < c));
#pragma unroll
    for (int j = NR - 1; j >= 0; --j) {
      uint64_t prev = __shfl_up_sync(0xffffffffu, l[j], 1);
      if (j > 0) {
        const uint64_t edge = __shfl_sync(0xffffffffu, l[j > 0 ? j - 1 : 0], 31);
        if (lane == 0) prev = edge;
      }
      const uint32_t i0 = 32 * j + lane;
      if (i0 == at) l[j] = c;
      if (i0 > at) l[j] = prev;
    }
  }
#pragma unroll
  for (int j = 0; j < NR; ++j)
    if (32 * j + lane < k) list[32 * j + lane] = l[j];
  __syncwarp();
  return list[k - 1];
}
__device__ __forceinline__ uint64_t list_merge(uint64_t* list, uint32_t k, const float* cd, const uint8_t* cr,
                                               uint32_t m, uint32_t v0) {
  const uint32_t lane = threadIdx.x & 31u;
  if (m <= INSERT_MAX) {
    if (k <= 32) return list_insert<1>(list, k, cd, cr, m, v0);
    if (k <= 128) return list_insert<4>(list, k, cd, cr, m, v0);
    return list_insert<8>(list, k, cd, cr, m, v0);
  }
  if (k <= 32) {
    uint64_t l = lane < k ? list[lane] : kSentinelKey;
    for (uint32_t b = 0; b < m; b += 32) {
      const uint32_t i = b + lane;
      uint64_t c = i < m ? make_key(cd[i], v0 + cr[i]) : kSentinelKey;
      c = warp_bitonic_sort32(c);
      c = __shfl_sync(0xffffffffu, c, 31 - lane);
      l = l < c ? l : c;
#pragma unroll
      for (int stride = 16; stride > 0; stride >>= 1) {
        const uint64_t o = __shfl_xor_sync(0xffffffffu, l, stride);
        if ((o < l) == ((lane & stride) == 0)) l = o;
      }
    }
    if (lane < k) list[lane] = l;
    return __shfl_sync(0xffffffffu, l, k - 1);
  }
  auto idx = [&](int e) { return 64u * (e >> 1) + 2 * lane + (e & 1); };
  uint64_t c[4], a[4], b[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const uint32_t i = idx(e);
    c[e] = i < m ? make_key(cd[i], v0 + cr[i]) : kSentinelKey;
    a[e] = i < k ? list[i] : kSentinelKey;
    b[e] = 128 + i < k ? list[128 + i] : kSentinelKey;
  }
  // descending order of c is c reversed: element e of lane l <-> element 3 - e of lane 31 - l
  warp128_sort(c, true);
  auto low = [&](uint64_t (&x)[4], uint64_t (&y)[4]) {  // x: the 128 smallest of both; y: the 128 largest (bitonic)
    uint64_t r[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) r[e] = __shfl_sync(0xffffffffu, y[3 - e], 31 - lane);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const uint64_t lo = x[e] < r[e] ? x[e] : r[e];
      y[e] = x[e] < r[e] ? r[e] : x[e];
      x[e] = lo;
    }
    warp128_merge<64>(x, true, true);
  };
  if (k > 128) {
    low(b, c);  // the best of the list's upper half and the candidates
    low(a, b);  // a: the 128 smallest of all, b: the rest
    warp128_merge<64>(b, true, true);
  } else {
    low(a, c);
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const uint32_t i = idx(e);
    if (i < k) list[i] = a[e];
    if (128 + i < k) list[128 + i] = b[e];
  }
  __syncwarp();
  return list[k - 1];
}

// Shared memory of a CTA: the staged chunk (rows [DK][VT], queries [DK][QT]),
// whose space holds the tile's candidate distances [QT][VT] after it is
// scored; then the lists.
template <int QT>
struct FlatSmem {
  static constexpr int XS = VT + (QT == QT_MAX ? 4 : 0), QS = QT + (QT == QT_MAX ? 4 : 0);  // row strides
  static constexpr size_t stage_floats = (size_t)DK * XS + (size_t)DK * QS;
  static constexpr size_t cand_floats = (size_t)QT * VT;
  static constexpr size_t floats = (stage_floats > cand_floats ? stage_floats : cand_floats) + QT + VT;
  static size_t bytes(uint32_t k) {
    return floats * 4 + (size_t)k * QT * 8 + QT * 8 + QT * 4 + (size_t)QT * VT;
  }
};

// FUSED = false: separately rounded sub/mul/add in dimension order (the
// reference's exact search). FUSED = true: fmaf(diff, diff, acc) in
// dimension order (the reference's coarse quantizer, ivf_rerank.cuh:80-84).
//
// The rows of a chunk are stored dimension-major. Below 64 queries the groups
// of four rows are permuted by the dimension group, which spreads the
// transposing stores over the banks; with 64 the arithmetic hides them and a
// padded stride saves the address arithmetic. Below 64 queries the next chunk's global loads are in
// flight while one is scored (64 have no registers left for it and are bound
// by the arithmetic: 100,000 x 128 x 1,000 took 1,725 us with, 1,592 without).
template <int QT, int METRIC, bool VEC4, bool FUSED = false>
__global__ void __launch_bounds__(NT, QT >= 32 ? 2 : 3) flat_f32_scan_kernel(FlatArgs a) {
  constexpr int QPT = QT >= 16 ? QT / 16 : 1;  // queries per thread
  constexpr int RPT = QT >= 16 ? 8 : 4;        // rows per thread (QT = 8: half the tile)
  constexpr bool SWZ = QT < QT_MAX;
  constexpr int XS = FlatSmem<QT>::XS, QS = FlatSmem<QT>::QS;
  auto x_at = [](int group, int dd) { return dd * XS + 4 * (SWZ ? group ^ (dd >> 2) : group); };
  auto q_at = [](int qi, int dd) {
    return dd * QS + 4 * (SWZ ? (qi >> 2) ^ ((dd >> 2) & (QT / 4 - 1)) : qi >> 2) + (qi & 3);
  };
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* xs = reinterpret_cast<float*>(smem_raw);  // [DK][VT]
  float* qs = xs + DK * XS;                        // [DK][QT]
  float* cd = xs;                                  // [QT][VT] candidate distances of a tile
  float* qn = xs + (FlatSmem<QT>::floats - QT - VT);      // [QT]
  float* xn = qn + QT;                                    // [VT]
  uint64_t* list = reinterpret_cast<uint64_t*>(xn + VT);  // [QT][k] sorted keys
  uint64_t* wq = list + (size_t)a.k * QT;                 // [QT] current k-th key per query
  uint32_t* cnt = reinterpret_cast<uint32_t*>(wq + QT);   // [QT] candidates of the tile per query
  uint8_t* cr = reinterpret_cast<uint8_t*>(cnt + QT);     // [QT][VT] their rows within the tile

  const int tid = threadIdx.x, warp = tid >> 5;
  const int ty = tid >> 4, tx = tid & 15;
  const int tq = QT >= 16 ? ty * QPT : (ty & 7);     // first query of this thread
  const int xh = QT >= 16 ? 0 : (ty >> 3) * 16;      // QT = 8: row group offset of this thread's half
  const uint32_t q0 = blockIdx.x * QT;
  if (a.active && !__syncthreads_or(tid < QT && q0 + tid < a.nq && a.active[q0 + tid] != 0u)) return;
  const uint32_t k = a.k;
  const uint32_t ntiles = (a.n + VT - 1) / VT;
  const uint32_t t_begin = blockIdx.y * a.tiles_per_split;
  const uint32_t t_end = min(t_begin + a.tiles_per_split, ntiles);

  for (uint32_t i = tid; i < k * QT; i += NT) list[i] = kSentinelKey;
  if (tid < QT) {
    wq[tid] = kSentinelKey;
    cnt[tid] = 0;
  }
  QueryFilter qf[QPT];  // filters of this thread's queries
#pragma unroll
  for (int i = 0; i < QPT; ++i) {
    const uint32_t q = q0 + tq + i;
    qf[i] = (a.filters && q < a.nq) ? load_filter(a.filters, q) : QueryFilter{nullptr, 0u, 0u};
  }
  float qnorm = 0.f;  // cosine: ||q||^2 of query tid - VT, summed over the first tile's chunks

  // staged elements of this thread: VEC4 four rows' worth of float4 (row e >> 3,
  // dimensions 4 (e & 7)..), else single floats (row e / DK, dimension e % DK)
  constexpr int XR = VT * DK / NT, QR = QT * DK / NT;  // floats per thread
  constexpr bool QV = QR >= 4;                         // QT >= 32: whole float4s of queries per thread
  constexpr int XL = VEC4 ? XR / 4 : XR;
  constexpr int QL = VEC4 ? (QV ? QR / 4 : 1) : QR;
  float4 xv4[VEC4 ? XL : 1], qv4[VEC4 ? QL : 1];
  float xv1[VEC4 ? 1 : XL], qv1[VEC4 ? 1 : QL];
  auto load = [&](uint32_t v0, uint32_t d0) {
    if constexpr (VEC4) {
#pragma unroll
      for (int r = 0; r < XL; ++r) {
        const int e = tid + NT * r, vi = e >> 3, dd = (e & 7) * 4;
        xv4[r] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (v0 + vi < a.n && d0 + dd < a.dim)
          xv4[r] = __ldg(reinterpret_cast<const float4*>(a.vectors + (size_t)(v0 + vi) * a.dim + d0 + dd));
      }
#pragma unroll
      for (int r = 0; r < QL; ++r) {
        const int e = tid + NT * r, qi = e >> 3, dd = (e & 7) * 4;
        qv4[r] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (qi < QT && q0 + qi < a.nq && d0 + dd < a.dim)
          qv4[r] = __ldg(reinterpret_cast<const float4*>(a.queries + (size_t)(q0 + qi) * a.dim + d0 + dd));
      }
    } else {
#pragma unroll
      for (int r = 0; r < XL; ++r) {
        const int e = tid + NT * r, vi = e / DK, dd = e % DK;
        xv1[r] = (v0 + vi < a.n && d0 + dd < a.dim) ? __ldg(a.vectors + (size_t)(v0 + vi) * a.dim + d0 + dd) : 0.f;
      }
#pragma unroll
      for (int r = 0; r < QL; ++r) {
        const int e = tid + NT * r, qi = e / DK, dd = e % DK;
        qv1[r] = (q0 + qi < a.nq && d0 + dd < a.dim) ? __ldg(a.queries + (size_t)(q0 + qi) * a.dim + d0 + dd) : 0.f;
      }
    }
  };
  auto put_x = [&](int vi, int dd, float v) { xs[x_at(vi >> 2, dd) + (vi & 3)] = v; };
  auto put_q = [&](int qi, int dd, float v) { qs[q_at(qi, dd)] = v; };
  auto store = [&]() {
    if constexpr (VEC4) {
#pragma unroll
      for (int r = 0; r < XL; ++r) {
        const int e = tid + NT * r, vi = e >> 3, dd = (e & 7) * 4;
        put_x(vi, dd, xv4[r].x);
        put_x(vi, dd + 1, xv4[r].y);
        put_x(vi, dd + 2, xv4[r].z);
        put_x(vi, dd + 3, xv4[r].w);
      }
#pragma unroll
      for (int r = 0; r < QL; ++r) {
        const int e = tid + NT * r, qi = e >> 3, dd = (e & 7) * 4;
        if (qi < QT) {
          put_q(qi, dd, qv4[r].x);
          put_q(qi, dd + 1, qv4[r].y);
          put_q(qi, dd + 2, qv4[r].z);
          put_q(qi, dd + 3, qv4[r].w);
        }
      }
    } else {
#pragma unroll
      for (int r = 0; r < XL; ++r) put_x((tid + NT * r) / DK, (tid + NT * r) % DK, xv1[r]);
#pragma unroll
      for (int r = 0; r < QL; ++r) put_q((tid + NT * r) / DK, (tid + NT * r) % DK, qv1[r]);
    }
  };

  constexpr bool PREFETCH = QT < QT_MAX;
  if (PREFETCH && t_begin < t_end) load(t_begin * VT, 0);
  for (uint32_t t = t_begin; t < t_end; ++t) {
    const uint32_t v0 = t * VT;
    float acc[QPT][RPT];
#pragma unroll
    for (int i = 0; i < QPT; ++i)
#pragma unroll
      for (int j = 0; j < RPT; ++j) acc[i][j] = 0.f;
    float xnorm = 0.f;

    for (uint32_t d0 = 0; d0 < a.dim; d0 += DK) {
      const uint32_t dk = min((uint32_t)DK, a.dim - d0);
      __syncthreads();  // previous chunk fully consumed (or the previous tile's candidates)
      if constexpr (!PREFETCH) load(v0, d0);
      store();
      if constexpr (PREFETCH) {
        if (d0 + DK < a.dim)
          load(v0, d0 + DK);
        else if (t + 1 < t_end)
          load(v0 + VT, 0);
      }
      __syncthreads();

      if (METRIC == METRIC_COSINE) {
        if (tid < VT) {
          for (uint32_t dd = 0; dd < dk; ++dd) {
            const float x = xs[x_at(tid >> 2, dd) + (tid & 3)];
            xnorm = __fadd_rn(xnorm, __fmul_rn(x, x));
          }
        } else if (t == t_begin && tid < VT + QT) {
          const int qi = tid - VT;
          for (uint32_t dd = 0; dd < dk; ++dd) {
            const float q = qs[q_at(qi, dd)];
            qnorm = __fadd_rn(qnorm, __fmul_rn(q, q));
          }
        }
      }

      auto step = [&](int dd) {
        // this thread's queries and its rows (columns 4 tx.. and, for QT >= 16,
        // 64 + 4 tx..) of dimension dd
        const float* qp = qs + q_at(tq, dd);
        float qv[QPT], xv[RPT];
        if constexpr (QPT == 4) {
          const float4 v = *reinterpret_cast<const float4*>(qp);
          qv[0] = v.x;
          qv[1] = v.y;
          qv[2] = v.z;
          qv[3] = v.w;
        } else if constexpr (QPT == 2) {
          const float2 v = *reinterpret_cast<const float2*>(qp);
          qv[0] = v.x;
          qv[1] = v.y;
        } else {
          qv[0] = *qp;
        }
#pragma unroll
        for (int j = 0; j < RPT; j += 4) {
          const float4 v = *reinterpret_cast<const float4*>(xs + x_at(tx + xh + 4 * j, dd));
          xv[j] = v.x;
          xv[j + 1] = v.y;
          xv[j + 2] = v.z;
          xv[j + 3] = v.w;
        }
#pragma unroll
        for (int i = 0; i < QPT; ++i)
#pragma unroll
          for (int j = 0; j < RPT; ++j) {
            if (METRIC == METRIC_L2) {
              const float diff = __fsub_rn(qv[i], xv[j]);
              acc[i][j] = FUSED ? fmaf(diff, diff, acc[i][j]) : __fadd_rn(acc[i][j], __fmul_rn(diff, diff));
            } else {
              acc[i][j] = __fadd_rn(acc[i][j], __fmul_rn(qv[i], xv[j]));
            }
          }
      };
      if (dk == DK) {
#pragma unroll 8
        for (int dd = 0; dd < DK; ++dd) step(dd);
      } else {
        for (uint32_t dd = 0; dd < dk; ++dd) step((int)dd);
      }
    }

    if (METRIC == METRIC_COSINE) {
      if (tid < VT)
        xn[tid] = xnorm;
      else if (t == t_begin && tid < VT + QT)
        qn[tid - VT] = qnorm;
    }
    __syncthreads();  // the chunk is consumed (cd takes its place), xn and qn are visible

#pragma unroll
    for (int i = 0; i < QPT; ++i) {
      const int qi = tq + i;
      const uint64_t wk = wq[qi];
#pragma unroll
      for (int j = 0; j < RPT; ++j) {
        const int vi = 4 * (tx + xh) + (j < 4 ? 0 : 64) + (j & 3);  // the row of acc[.][j] (see step)
        float dist;
        if (METRIC == METRIC_L2) {
          dist = acc[i][j];
        } else if (METRIC == METRIC_INNER_PRODUCT) {
          dist = -acc[i][j];
        } else {
          float denom = __fadd_rn(__fmul_rn(sqrtf(qn[qi]), sqrtf(xn[vi])), 1e-8f);
          dist = __fsub_rn(1.0f, __fdiv_rn(acc[i][j], denom));
        }
        const uint32_t slot = v0 + vi;
        // a key that cannot beat the query's current k-th key never enters
        // (the k-th key only decreases, so testing against an older one
        // admits a superset); NaN fails `<`
        if (dist < kSentinelDist && make_key(dist, slot) < wk && slot < a.n && mask_allows(a.mask, slot) &&
            (!a.filters || filter_allows(qf[i], a.vec_ids ? __ldg(a.vec_ids + slot) : slot))) {
          const uint32_t pos = atomicAdd(cnt + qi, 1u);
          cd[qi * VT + pos] = dist;
          cr[qi * VT + pos] = (uint8_t)vi;
        }
      }
    }
    __syncthreads();

    // the tile's candidates into the lists, one query per warp at a time
    for (int qi = warp; qi < QT; qi += NW) {
      const uint32_t m = cnt[qi];  // uniform over the warp
      if (m == 0) continue;
      const uint64_t w = list_merge(list + (size_t)qi * k, k, cd + qi * VT, cr + qi * VT, m, v0);
      __syncwarp();
      if ((tid & 31) == 0) {
        wq[qi] = w;
        cnt[qi] = 0;
      }
    }
  }
  __syncthreads();

  for (uint32_t i = tid; i < QT * k; i += NT) {
    const uint32_t q = q0 + i / k, r = i % k;
    if (q >= a.nq) break;
    if (a.active && a.active[q] == 0u) continue;
    if (a.splits == 1)
      a.out[(size_t)q * k + r] = key_to_result(list[i], a.vec_ids);
    else
      a.partial[((size_t)q * a.splits + blockIdx.y) * k + r] = list[i];
  }
}

}  // namespace

// Merges `lists` lists of `k` keys per query into the
// ascending top-k; one CTA per query, bitonic sort in shared memory.
__global__ void __launch_bounds__(256) merge_partial_topk_kernel(const uint64_t* __restrict__ partial, uint32_t lists,
                                                                 uint32_t k, uint32_t pow2, const uint32_t* vec_ids,
                                                                 GpuSearchResult* __restrict__ out, uint32_t out_k,
                                                                 const uint32_t* __restrict__ active) {
  extern __shared__ __align__(16) uint64_t keys[];
  const uint32_t q = blockIdx.x;
  if (active && active[q] == 0u) return;
  const uint32_t total = lists * k;
  const uint64_t* src = partial + (size_t)q * total;
  for (uint32_t i = threadIdx.x; i < pow2; i += blockDim.x) keys[i] = i < total ? src[i] : kSentinelKey;
  __syncthreads();
  block_bitonic_sort(keys, pow2);
  for (uint32_t r = threadIdx.x; r < out_k; r += blockDim.x) out[(size_t)q * out_k + r] = key_to_result(keys[r], vec_ids);
}

// Queries per CTA. Whole blocks of 64 use the cores best (four queries a
// thread share each row operand); a smaller block wins where rounding the
// batch up to 64 would add more than a sixth of work, and for a handful of
// queries, which the staging of the rows bounds whatever the block.
static uint32_t flat_query_tile(uint32_t nq) {
  if (nq <= 8) return 8;
  if (nq <= 16) return 16;
  if (nq <= 32) return 32;
  const uint32_t p32 = (nq + 31) / 32 * 32, p64 = (nq + 63) / 64 * 64;
  return 6 * p64 > 7 * p32 ? 32 : 64;
}

FlatPlan plan_flat_f32(uint32_t n, uint32_t nq, uint32_t k, uint32_t forced_splits) {
  const uint32_t nqb64 = (nq + QT_MAX - 1) / QT_MAX;
  const uint32_t ntiles = (n + VT - 1) / VT;
  int sms = device_sm_count();
  const uint32_t pow2k = next_pow2(k);
  const uint32_t smax = std::max(1u, std::min(ntiles, 8192u / pow2k));  // merge sorts splits * k keys
  // CTA slots of a wave (two 64-query blocks per SM by registers, three or
  // more of the smaller ones), and the fewest splits that give every slot a
  // CTA, or a few more when that fills the last wave better (a query block
  // count just above the slot count otherwise leaves a nearly empty wave)
  auto choose = [&](uint32_t nqb, uint32_t per_sm, uint32_t cap) {
    const uint64_t slots = (uint64_t)per_sm * (uint64_t)sms;
    const uint32_t s0 = (uint32_t)std::max<uint64_t>(1, (slots + nqb - 1) / nqb);
    auto fullness = [&](uint32_t sp) {
      const uint64_t ctas = (uint64_t)nqb * sp, waves = (ctas + slots - 1) / slots;
      return (double)ctas / (double)(waves * slots);
    };
    uint32_t splits = std::min(s0, cap);
    double best = fullness(splits);
    for (uint32_t sp = splits + 1; sp <= std::min(std::max(2 * s0, 8u), cap); ++sp) {
      const double f = fullness(sp);
      if (f > best + 0.01) {
        best = f;
        splits = sp;
      }
    }
    return splits;
  };
  auto clamp = [&](uint32_t splits) {
    splits = std::max(1u, std::min(splits, smax));
    const uint32_t tps = (ntiles + splits - 1) / splits;
    return (ntiles + tps - 1) / tps;
  };
  // the scratch is that of 64-query blocks, whose split count bounds the others'
  const uint32_t splits64 = clamp(forced_splits ? forced_splits : choose(nqb64, 2, smax));
  FlatPlan p;
  p.query_tile = flat_query_tile(nq);
  p.splits = splits64;
  if (!forced_splits && p.query_tile != QT_MAX)
    p.splits = clamp(choose((nq + p.query_tile - 1) / p.query_tile, 3, splits64));
  p.tiles_per_split = (ntiles + p.splits - 1) / p.splits;
  p.scratch_bytes = splits64 > 1 ? (size_t)nq * splits64 * k * 8 : 0;
  return p;
}

int launch_flat_f32(const float* vectors, const uint32_t* vec_ids, uint32_t n, uint32_t dim, const float* queries,
                    uint32_t nq, uint32_t k, MetricType metric, const uint32_t* mask, GpuSearchResult* out,
                    uint32_t forced_splits, cudaStream_t stream, const QueryFilter* filters) {
  void* scratch = nullptr;
  if (!filters && !forced_splits) {
    const FlatTcPlan t = plan_flat_tc(n, dim, nq, k, metric);
    // (a caller's arena that only fits the plain scan keeps it, as does one that
    // is not 16-byte aligned, which the filter's TMA and vector accesses need, and
    // a capture or a full device, where the arena cannot grow for the filter)
    if (t.bytes && (scratch = scratch_try(stream, t.bytes)) != nullptr && (uintptr_t)scratch % 16 == 0)
      return launch_flat_tc(t, vectors, vec_ids, n, dim, queries, nq, k, metric, mask, out, scratch, stream);
  }
  const FlatPlan p = plan_flat_f32(n, nq, k, forced_splits);
  if (p.scratch_bytes) {
    scratch = scratch_get(stream, p.scratch_bytes);
    if (!scratch) return (int)cudaErrorMemoryAllocation;
  }
  return launch_flat_f32_planned(p, vectors, vec_ids, n, dim, queries, nq, k, metric, mask, out, false, scratch,
                                 stream, filters);
}

int launch_flat_f32_planned(const FlatPlan& p, const float* vectors, const uint32_t* vec_ids, uint32_t n,
                            uint32_t dim, const float* queries, uint32_t nq, uint32_t k, MetricType metric,
                            const uint32_t* mask, GpuSearchResult* out, bool fused, void* scratch,
                            cudaStream_t stream, const QueryFilter* filters, const uint32_t* active) {
  const uint32_t qt = p.query_tile, nqb = (nq + qt - 1) / qt;
  const uint32_t splits = p.splits, tps = p.tiles_per_split;
  FlatArgs a{vectors, vec_ids, n, dim, queries, nq, k, mask, out, static_cast<uint64_t*>(scratch), splits, tps,
             filters, active};
  if (splits > 1 && !a.partial) return (int)cudaErrorMemoryAllocation;

  const bool vec4 = (dim % 4 == 0) && ((uintptr_t)vectors % 16 == 0) && ((uintptr_t)queries % 16 == 0);
  dim3 grid(nqb, splits);
  auto go = [&](auto kern, size_t smem) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    kern<<<grid, NT, smem, stream>>>(a);
  };
  auto by_metric = [&](auto qt_tag, auto vec_tag) {
    constexpr int Q = decltype(qt_tag)::value;
    constexpr bool V = decltype(vec_tag)::value;
    const size_t smem = FlatSmem<Q>::bytes(k);
    if (fused) return go(flat_f32_scan_kernel<Q, METRIC_L2, V, true>, smem);
    switch (metric) {
      case METRIC_INNER_PRODUCT: return go(flat_f32_scan_kernel<Q, METRIC_INNER_PRODUCT, V>, smem);
      case METRIC_COSINE: return go(flat_f32_scan_kernel<Q, METRIC_COSINE, V>, smem);
      default: return go(flat_f32_scan_kernel<Q, METRIC_L2, V>, smem);
    }
  };
  auto by_tile = [&](auto vec_tag) {
    switch (qt) {
      case 8: return by_metric(std::integral_constant<int, 8>{}, vec_tag);
      case 16: return by_metric(std::integral_constant<int, 16>{}, vec_tag);
      case 32: return by_metric(std::integral_constant<int, 32>{}, vec_tag);
      default: return by_metric(std::integral_constant<int, 64>{}, vec_tag);
    }
  };
  ProfScope ps(fused ? "coarse_f32_scan" : "flat_f32_scan", stream);
  if (vec4)
    by_tile(std::true_type{});
  else
    by_tile(std::false_type{});
  note_launch();
  if (splits > 1) {
    const uint32_t pow2 = next_pow2(splits * k);
    const size_t msmem = (size_t)pow2 * 8;
    cudaFuncSetAttribute(merge_partial_topk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)msmem);
    merge_partial_topk_kernel<<<nq, 256, msmem, stream>>>(a.partial, splits, k, pow2, vec_ids, out, k, active);
    note_launch();
  }
  return (int)cudaGetLastError();
}


// ===========================================================================
// Allocation-free variant of the exact flat scan.
//
// Some callers of this library cannot call cudaMalloc: code that runs while
// another thread is capturing a CUDA graph in global capture mode (where an
// allocation is an illegal call), latency-critical serving threads that
// must not take the allocator's locks or risk its implicit device
// synchronisation, and hosts that hand all device memory to one pool of
// their own. For them fv_flat_scan_batch_noalloc keeps the per-split heaps
// of the scan in the fixed array below instead of the per-stream arena.
//
// The array is a file-scope device variable: every GPU that loads this
// library holds its kNoAllocScratchBytes until the process exits. In host
// code its name is only a host-side stand-in, not a device address, so the
// address handed to the kernels is looked up once per device with
// cudaGetSymbolAddress (with that device current) on the first call made
// on the device; make that first call before any stream capture begins.
// The looked-up address is kept for the life of the process: after a
// cudaDeviceReset the array may sit elsewhere in the new context, so a
// process that resets a device must not call this entry point on it again.
// All calls share the one array and it keeps whatever the last call wrote;
// the scan writes every slot it later reads, so nothing needs clearing, but
// calls whose work overlaps on the GPU (different streams, or host threads
// racing on one device) overwrite each other's heaps -- serialise them.
// ===========================================================================
namespace {
constexpr size_t kNoAllocScratchBytes = 8u << 20;  // 8 MiB per device
static __device__ __align__(256) uint64_t g_flat_noalloc_scratch[kNoAllocScratchBytes / 8];

constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mu;
uint64_t* g_noalloc_addr[kMaxDevices] = {};

cudaError_t noalloc_scratch_address(uint64_t** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_addr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_flat_noalloc_scratch);
    if (e != cudaSuccess) return e;
    g_noalloc_addr[dev] = static_cast<uint64_t*>(p);
  }
  *out = g_noalloc_addr[dev];
  return cudaSuccess;
}
}  // namespace

// Same work split and kernels as launch_flat_f32's plain scan (never the
// tensor-core filter), with the per-split lists in the fixed array; refuses
// (FV_ERR_SCRATCH_LIMIT) a call whose lists would not fit instead of allocating.
int launch_flat_f32_noalloc(const float* vectors, const uint32_t* vec_ids, uint32_t n, uint32_t dim,
                            const float* queries, uint32_t nq, uint32_t k, MetricType metric, const uint32_t* mask,
                            GpuSearchResult* out, cudaStream_t stream) {
  const FlatPlan p = plan_flat_f32(n, nq, k, 0);
  if (p.scratch_bytes > kNoAllocScratchBytes) return FV_ERR_SCRATCH_LIMIT;
  uint64_t* heaps = nullptr;
  if (p.scratch_bytes) {
    cudaError_t e = noalloc_scratch_address(&heaps);
    if (e != cudaSuccess) return (int)e;
  }
  return launch_flat_f32_planned(p, vectors, vec_ids, n, dim, queries, nq, k, metric, mask, out, false, heaps,
                                 stream);
}

}  // namespace fv

extern "C" int fv_flat_scan_batch_noalloc(const float* d_vectors, const uint32_t* d_vec_ids, uint32_t num_vectors,
                                          uint32_t dim, const float* d_queries, uint32_t num_queries, uint32_t top_k,
                                          MetricType metric, const uint32_t* d_valid_mask,
                                          GpuSearchResult* d_out_results, void* stream) {
  if (!d_queries || !d_out_results) return -1;
  if (num_vectors > 0 && !d_vectors) return -1;
  if (num_queries == 0 || top_k == 0) return 0;
  if (top_k > (uint32_t)fv::kMaxTopK) top_k = fv::kMaxTopK;
  cudaStream_t s = (cudaStream_t)stream;
  if (num_vectors == 0)
    return (int)cudaMemsetAsync(d_out_results, 0xFF, (size_t)num_queries * top_k * sizeof(GpuSearchResult), s);
  if (dim == 0) return -2;
  return fv::launch_flat_f32_noalloc(d_vectors, d_vec_ids, num_vectors, dim, d_queries, num_queries, top_k, metric,
                                     d_valid_mask, d_out_results, s);
}

