// ivf.cu -- IVF-PQ, IVF-SQ8 and IVF-RaBitQ inverted-list scans.
//
// Replaces launch_ivf_pq_search / launch_ivf_sq_search /
// launch_ivf_rabitq_search and their kernels (ivf_pq_lookup.cu:14-444,
// ivf_quant_lookup.cu:18-870, ivf_rerank.cuh:49-160) with the same inputs,
// clamps and result semantics:
//   * top_k <= 256; nprobe clamped to [1, nlist];
//     shortlist = rerank_k ? rerank_k : top_k, >= top_k, <= 10240;
//     exact rerank when rerank_k != 1 and fp32 rows are present;
//   * coarse probe: the nprobe nearest centroids by squared L2 accumulated
//     with fmaf in dimension order (ivf_rerank.cuh:78-84) -- exact here, by
//     (distance, list id);
//   * PQ: residual LUT[m][c] = sum_sd fmaf(((q - centroid) - codeword)^2)
//     per (query, list) in shared memory (ivf_pq_lookup.cu:150-162), ADC =
//     the LUT entries of a row's codes added in sub-space order (:176-178);
//     SQ8: sum_d fmaf over (q - centroid) - fmaf(code, scale, min)
//     (ivf_quant_lookup.cu:83-87), L2 whatever the metric;
//     RaBitQ: the query rotated once per query (three rounds of sign flip,
//     Walsh-Hadamard butterflies, 1/sqrt(P) scale: ivf_quant_lookup.cu:
//     337-376), per (query, list) its rotated residual quantised to 4 bits
//     over [min, max] as four bit-planes (:381-460), per posting the
//     popcount estimate (:462-489) with its roundings fixed
//     (rabitq_estimate below);
//   * shortlist = the best `shortlist` (approx distance, id) keys; rerank
//     with the reference's warp-order fp32 distance; the first top_k by
//     (distance, id) are returned.
// Because every distance is evaluated in the reference's operation order,
// the results are bit-identical to the oracle's restatement.
//
// Machine mapping. The coarse probe is the exact flat scan kernel in its
// fused-FMA mode (a Q x nlist tiled scan with a fused top-nprobe), or the
// tensor-core candidates below. The list scan is one persistent launch: CTAs
// pull queries from a device work counter. The query's probed lists are taken
// up to 32 at a time; their postings form one sequence that the CTA's threads
// walk together, so a list costs no barriers of its own and short lists share
// a round (most lists of a Zipf base hold a fraction of one). What a list
// needs first is made for all of them at once: RaBitQ query codes one warp per
// list; SQ8 subtracts the centroid on the fly. PQ builds the 256-entry tables
// only for lists with enough postings to use them (they read the whole
// codebook, 128 KB at m = 32) and evaluates the few table entries that a short
// list needs in place, in the same operations. A running shortlist is kept in
// shared memory: rows whose key cannot beat its worst key are dropped, the
// rest are appended to a buffer; when it fills, the best of both are kept.
#include <type_traits>

#include <cuda_fp16.h>

#include "../../include/fv_bridge.h"
#include "common.cuh"
#include "kernels.h"
#include "topk.cuh"

namespace fv {

namespace {

constexpr int IVF_THREADS = 256;
constexpr uint32_t IVF_BUF = 1536;         // candidate buffer entries (>= 1.5 rounds of 1,024 postings)
constexpr uint32_t MAX_SHORTLIST = 10240;  // reference clamp (ivf_rerank.cuh:12)
// Keys of which a flush selects the shortlist from registers. Up to 512 a sort
// is the quicker (5 queries, 20,000 x 128: 57 us sorting, 67 selecting), from
// 1,024 the selection (2,000 RaBitQ queries over 1M rows: list scan 788 us
// sorting, 646 selecting); past 2,048 the registers do not hold them.
constexpr uint32_t KEEP_MIN = 512, KEEP_MAX = 2048;

enum IvfMode { IVF_PQ = IVF_MODE_PQ, IVF_SQ8 = IVF_MODE_SQ8, IVF_RABITQ = IVF_MODE_RABITQ };

struct IvfArgs {
  const float* centroids;   // [nlist][dim]
  const float* codebooks;   // PQ: [m][256][sub]
  const float* sq_mins;     // SQ8: [dim]
  const float* sq_scales;   // SQ8: [dim]
  const uint8_t* codes;     // [N][code_bytes] by id, or by list position when list_major
                            // (RaBitQ: the sign bits, code_bytes = 4 W)
  const uint32_t* offsets;  // [nlist + 1]
  const uint32_t* vec_ids;  // [N] ids in list order
  const float* vectors;     // fp32 rows (rerank) or null
  uint32_t num_vectors, dim, nlist, m_pq, sub_dim, code_bytes;
  const float* queries;
  uint32_t nq, top_k, nprobe, rerank_k, list_major;
  int metric;
  const uint32_t* mask;
  // the mask in list order: bit i of this array = mask bit of vec_ids[i], for
  // list positions i < list_n (null when there is no mask; positions past the
  // lists hold 0); one shared word per 32 postings replaces a dependent id +
  // mask-word load per posting
  const uint32_t* list_allow;
  uint32_t list_n;
  // the admitted list positions in list order (compacted from list_allow),
  // and per bit word the count of admitted positions before it: a list
  // whose mask admits under half of its postings is scanned over these
  // positions only (null when there is no mask)
  const uint32_t* adm_pos;
  const uint32_t* adm_prefix;  // [ceil(list_n / 32) + 1]
  const uint32_t* q_topk;         // per-query top_k / nprobe / rerank_k, or null (uniform)
  const uint32_t* q_nprobe;
  const uint32_t* q_rerank;
  const QueryFilter* filters;     // per-query filters over ids, or null
  const GpuSearchResult* probes;  // [nq][nprobe] coarse result (id = list)
  uint32_t* work;                 // work counter (zeroed before the launch)
  const uint32_t* order;          // queries in the order they are pulled, or null (as given)
  GpuSearchResult* out;
  uint32_t* status;
  uint32_t keys_pow2;             // pow2(largest shortlist + IVF_BUF)
  uint32_t list_chunk;            // probed lists walked as one sequence (<= 32)
  uint32_t keep_at;               // byte offset of the flush's selection scratch (0: flushes sort)
  uint32_t items_per_q;           // G: a query's probed postings are cut into G ranges
  uint64_t* partial;              // G > 1: [nq * G][part_stride] shortlists of the ranges
  uint32_t part_stride;           // >= every query's shortlist
  // RaBitQ
  const float* rot_centroids;     // [nlist][P]
  const float* rq_meta;           // [N][4] by id, or by list position when list_major
  const float* rot_signs;         // [3][P]
  uint32_t P, W;                  // rotated dimension (power of two), words of bits per row
  float inv_sqrt_p;               // 1.0f / sqrtf(P), correctly rounded
};

// Index of list position p in the compacted admitted positions (the count of
// admitted positions before p). p <= list_n.
__device__ __forceinline__ uint32_t adm_index(const IvfArgs& a, uint32_t p) {
  const uint32_t w = p >> 5, b = p & 31u;
  return __ldg(a.adm_prefix + w) + (b ? __popc(__ldg(a.list_allow + w) & ((1u << b) - 1u)) : 0u);
}

// The postings of list l as the scan walks them: [beg, end) list positions
// (compact = false), or [beg, end) indices into adm_pos (compact = true)
// when the list-order mask admits under half of the list.
struct ListSpan {
  uint32_t beg, end;
  bool compact;
};
__device__ __forceinline__ ListSpan list_span(const IvfArgs& a, uint32_t l) {
  const uint32_t lbeg = __ldg(a.offsets + l), lend = __ldg(a.offsets + l + 1);
  if (a.adm_pos != nullptr && lend > lbeg) {
    const uint32_t a0 = adm_index(a, lbeg), a1 = adm_index(a, lend);
    if (2 * (a1 - a0) < lend - lbeg) return ListSpan{a0, a1, true};
  }
  return ListSpan{lbeg, lend, false};
}

// Rerank of a query's shortlist keys[0, S) (in any order, sentinels last) with
// the reference's warp-order fp32 distance, sort, and the query's top k into
// out[q][0, top_k) (sentinels past k). Block-collective.
template <int NT, uint32_t R, int B>
__device__ void ivf_finish_query(const IvfArgs& a, uint64_t* keys, uint32_t q, uint32_t S, uint32_t kq,
                                 bool do_rerank, const float* qv, KeepScratch* keep) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (do_rerank) {
    // R candidates per warp pass (c, c + NW, .., all owned by warp c % NW as
    // with one at a time), so R rows' gathers, B loads ahead each, are in
    // flight per warp.
    constexpr uint32_t NW = NT / 32;
    for (uint32_t c0 = warp; c0 < S; c0 += R * NW) {
      if (keys[c0] == kSentinelKey) break;  // the rest are sentinels too
      const float* rows[R];
      uint32_t slot[R];
      bool any = false;
#pragma unroll
      for (uint32_t r = 0; r < R; ++r) {
        const uint32_t c = c0 + r * NW;
        const uint64_t key = c < S ? keys[c] : kSentinelKey;
        const bool ok = key != kSentinelKey && key_slot(key) < a.num_vectors;
        // an unused slot reads row 0 and its result is dropped
        slot[r] = ok ? key_slot(key) : kInvalidId;
        rows[r] = a.vectors + (size_t)(ok ? slot[r] : 0u) * a.dim;
        any = any || ok;
      }
      if (!any) continue;
      float d[R];
      warp_metric_distances<R, B>(qv, rows, a.dim, lane, (MetricType)a.metric, d);
      __syncwarp();
      if (lane == 0) {
#pragma unroll
        for (uint32_t r = 0; r < R; ++r)
          if (slot[r] != kInvalidId) keys[c0 + r * NW] = make_key(d[r], slot[r]);
      }
    }
    __syncthreads();
  }
  uint32_t sorted = S;
  if (keep && S > 2 * kq && S > KEEP_MIN && S <= KEEP_MAX) {
    block_keep_smallest<NT, KEEP_MAX / NT>(keys, S, kq, *keep);
    sorted = kq;
  }
  const uint32_t p2 = next_pow2_dev(sorted);
  for (uint32_t i = sorted + tid; i < p2; i += NT) keys[i] = kSentinelKey;
  __syncthreads();
  block_bitonic_sort(keys, p2);
  for (uint32_t r = tid; r < a.top_k; r += NT)
    a.out[(size_t)q * a.top_k + r] = key_to_result(r < S && r < kq ? keys[r] : kSentinelKey, nullptr);
}

// The reference's clamps (ivf_pq_lookup.cu:351-362) for one query: returns
// the shortlist length; top_k and nprobe are clamped in place.
__host__ __device__ __forceinline__ uint32_t ivf_clamps(uint32_t& top_k, uint32_t& nprobe, uint32_t rerank_k,
                                                        uint32_t nlist) {
  top_k = top_k < (uint32_t)kMaxTopK ? top_k : (uint32_t)kMaxTopK;
  nprobe = nprobe == 0 ? 1u : nprobe;
  nprobe = nprobe < nlist ? nprobe : nlist;
  uint32_t s = rerank_k == 0 ? top_k : rerank_k;
  s = s > top_k ? s : top_k;
  return s < MAX_SHORTLIST ? s : MAX_SHORTLIST;
}

constexpr uint32_t LIST_CHUNK = 32;

// staging of SQ8 rows, see sq8_rows
constexpr uint32_t SQ_STRIDE = 80;                  // bytes per row of a 64-dimension chunk: 16-byte steps off the same bank
constexpr uint32_t SQ_WORDS = 32 / 4 + 1;           // words per row of a 32-dimension chunk that starts at any byte
constexpr uint32_t SQ_BUF_BYTES = 64 * SQ_WORDS * 4;  // of two chunks of 32 dimensions each
constexpr uint32_t SQ_WARP_BYTES = 64 * SQ_STRIDE;
static_assert(2 * SQ_BUF_BYTES <= SQ_WARP_BYTES, "both forms in one area");

struct IvfSmem {
  // [keys_pow2] u64 keys | table | query (dim f32) | PQ: query residual to the
  // probed centroid (dim f32) | the lists of a chunk: first posting, list,
  // postings before it (3 LC + 1 u32)
  // table: PQ LUT (m*256 f32); SQ8 mins+scales+residual (3*dim f32); RaBitQ rotated
  //        query (P f32) + per list of a chunk its query code (4*W u32
  //        bit-planes, min, delta, sum u, centroid distance)
  __host__ __device__ static size_t table_floats(int mode, uint32_t dim, uint32_t m_pq, uint32_t P, uint32_t lc) {
    return mode == IVF_PQ ? (size_t)m_pq * 256
                          : mode == IVF_SQ8 ? (size_t)3 * dim : (size_t)P + (size_t)lc * (P / 8 + 4);
  }
  static size_t bytes(int mode, uint32_t keys_pow2, uint32_t dim, uint32_t m_pq, uint32_t P, uint32_t lc) {
    size_t b = (size_t)keys_pow2 * 8;
    b += table_floats(mode, dim, m_pq, P, lc) * 4;
    b += ((size_t)dim + 3) / 4 * 16;
    if (mode == IVF_PQ) b += (size_t)dim * 4;
    return b + (3 * lc + 1) * 4;
  }
  // SQ8 with staged rows: the warps' staging areas follow, 16-byte aligned
  static size_t staged_bytes(uint32_t keys_pow2, uint32_t dim, uint32_t lc) {
    return (bytes(IVF_SQ8, keys_pow2, dim, 0, 0, lc) + 15) / 16 * 16 + (size_t)(IVF_THREADS / 32) * SQ_WARP_BYTES;
  }
};

// RaBitQ: the query rotated into rq[0, P) (block-collective). The rounds of
// the reference's rotation (sign flip; butterflies x + y, x - y at half
// length 1, 2, ..., P/2; scale by 1/sqrt(P)) with each round's scale and
// the next round's sign flip applied in one pass -- the same two roundings.
__device__ void rabitq_rotate_query(float* rq, const float* qs, const IvfArgs& a) {
  const int tid = threadIdx.x;
  const uint32_t P = a.P;
  for (uint32_t d = tid; d < P; d += IVF_THREADS) rq[d] = __fmul_rn(d < a.dim ? qs[d] : 0.f, __ldg(a.rot_signs + d));
  __syncthreads();
  for (int st = 0; st < 3; ++st) {
    for (uint32_t h = 1; h < P; h <<= 1) {
      for (uint32_t i = tid; i < P / 2; i += IVF_THREADS) {
        const uint32_t x0 = ((i & ~(h - 1)) << 1) | (i & (h - 1));  // (i / h) * 2h + i % h
        const float x = rq[x0], y = rq[x0 + h];
        rq[x0] = __fadd_rn(x, y);
        rq[x0 + h] = __fsub_rn(x, y);
      }
      __syncthreads();
    }
    const float* next = st < 2 ? a.rot_signs + (size_t)(st + 1) * P : nullptr;
    for (uint32_t d = tid; d < P; d += IVF_THREADS) {
      const float v = __fmul_rn(rq[d], a.inv_sqrt_p);
      rq[d] = next ? __fmul_rn(v, __ldg(next + d)) : v;
    }
    __syncthreads();
  }
}

// RaBitQ: the 4-bit code of the rotated query residual to list l
// (ivf_quant_lookup.cu:381-460): diff = rq - rot_centroid over all P
// coordinates, u = clamp(rint((diff - min) * (15 / range)), 0, 15) (all 0
// when range <= 1e-12), bit-plane j word w bit l = bit j of u[32 w + l].
// Writes planes[4][W], then min, delta = range / 15, sum u (exact: at most
// 15 * 4096) and the query's distance to the centroid. Warp-collective.
__device__ void rabitq_query_code(const float* rq, uint32_t* code, const IvfArgs& a, uint32_t l, float qc) {
  const int lane = threadIdx.x & 31;
  const float* rc = a.rot_centroids + (size_t)l * a.P;
  float lo = 1e30f, hi = -1e30f;
  for (uint32_t d = lane; d < a.P; d += 32) {
    const float v = __fsub_rn(rq[d], __ldg(rc + d));
    lo = fminf(lo, v);
    hi = fmaxf(hi, v);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  const float range = __fsub_rn(hi, lo);
  const bool live = range > 1e-12f;
  const float delta = live ? __fdiv_rn(range, 15.0f) : 0.f;
  const float inv = live ? __fdiv_rn(15.0f, range) : 0.f;
  uint32_t su = 0;
  for (uint32_t w = 0; w < a.W; ++w) {
    uint32_t u = 0;
    if (delta > 0.f) {
      const float v = __fsub_rn(rq[w * 32 + lane], __ldg(rc + w * 32 + lane));
      const int qi = __float2int_rn(__fmul_rn(__fsub_rn(v, lo), inv));
      u = (uint32_t)min(max(qi, 0), 15);
    }
    su += u;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t pj = __ballot_sync(0xffffffffu, (u >> j) & 1u);
      if (lane == 0) code[j * a.W + w] = pj;
    }
  }
  su = __reduce_add_sync(0xffffffffu, su);
  if (lane == 0) {
    float* par = reinterpret_cast<float*>(code + 4 * a.W);
    par[0] = lo;
    par[1] = delta;
    par[2] = (float)su;
    par[3] = qc;
  }
}

// RaBitQ estimate of one posting from s_bu = sum_j 2^j popc(bits & plane_j)
// and its meta m = {|r|^2, rescale, popcount, |x|^2}
// (ivf_quant_lookup.cu:462-489). The reference leaves the roundings to the
// compiler; here they are fixed:
//   t = fmaf(delta, 2 s_bu - sum_u, q_min * (2 popcount - P))
//   est_l2 = (q_c + |r|^2) - 2 (rescale * t)
//   IP: -0.5 ((|q|^2 + |x|^2) - est_l2); cosine: 0.5 est_l2.
__device__ __forceinline__ float rabitq_estimate(uint32_t s_bu, float4 m, float P, float qmin, float delta,
                                                 float sum_u, float qc, float qn, int metric) {
  const float A = __fsub_rn(__fmul_rn(2.f, m.z), P);
  const float B = __fsub_rn(__fmul_rn(2.f, (float)s_bu), sum_u);
  const float t = __fmaf_rn(delta, B, __fmul_rn(qmin, A));
  const float est = __fsub_rn(__fadd_rn(qc, m.x), __fmul_rn(2.f, __fmul_rn(m.y, t)));
  if (metric == METRIC_INNER_PRODUCT) return __fmul_rn(-0.5f, __fsub_rn(__fadd_rn(qn, m.w), est));
  if (metric == METRIC_COSINE) return __fmul_rn(0.5f, est);
  return est;
}

// s_bu of a row of MW 16-byte words of bits held in registers. The masked
// words of the four planes are added bitwise before they are counted: a full
// adder turns three words of one weight into a sum and a carry of twice the
// weight (two logic instructions), so nine population counts (a quarter-rate
// unit) replace sixteen per 128 bits.
__device__ __forceinline__ void full_add(uint32_t a, uint32_t b, uint32_t c, uint32_t& sum, uint32_t& carry) {
  sum = a ^ b ^ c;
  carry = (a & b) | (c & (a | b));
}
template <int MW>
__device__ __forceinline__ uint32_t rabitq_sbu(const uint32_t* planes, const uint4 (&b)[MW]) {
  uint32_t acc = 0;
#pragma unroll
  for (int w = 0; w < MW; ++w) {
    uint32_t x[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint4 p = *reinterpret_cast<const uint4*>(planes + j * 4 * MW + 4 * w);
      x[j][0] = b[w].x & p.x;
      x[j][1] = b[w].y & p.y;
      x[j][2] = b[w].z & p.z;
      x[j][3] = b[w].w & p.w;
    }
    uint32_t s1, c2, s2, t2, c4a, c4b, s4, t4, c8a, c8b, s8, t8, c16a, c16b;
    full_add(x[0][0], x[0][1], x[0][2], s1, c2);      // weight 1: s1, x[0][3]
    full_add(x[1][0], x[1][1], x[1][2], t2, c4a);
    full_add(t2, x[1][3], c2, s2, c4b);               // weight 2: s2
    full_add(x[2][0], x[2][1], x[2][2], s4, c8a);
    full_add(x[2][3], c4a, c4b, t4, c8b);             // weight 4: s4, t4
    full_add(x[3][0], x[3][1], x[3][2], s8, c16a);
    full_add(x[3][3], c8a, c8b, t8, c16b);            // weight 8: s8, t8
    acc += (__popc(s1) + __popc(x[0][3])) + (__popc(s2) << 1) + ((__popc(s4) + __popc(t4)) << 2) +
           ((__popc(s8) + __popc(t8)) << 3) + ((__popc(c16a) + __popc(c16b)) << 4);
  }
  return acc;
}

// s_bu of a row read word by word (any W, any alignment)
__device__ __forceinline__ uint32_t rabitq_sbu_any(const uint32_t* planes, const uint32_t* __restrict__ row,
                                                   uint32_t W) {
  uint32_t c[4] = {0, 0, 0, 0};
  for (uint32_t w = 0; w < W; ++w) {
    const uint32_t b = __ldg(row + w);
#pragma unroll
    for (int j = 0; j < 4; ++j) c[j] += __popc(b & planes[j * W + w]);
  }
  return c[0] + (c[1] << 1) + (c[2] << 2) + (c[3] << 3);
}

// PQ: ADC of one row from its code bytes; LUT rows of 256 floats.
__device__ __forceinline__ float adc_row(const float* __restrict__ lut, const uint8_t* __restrict__ row, uint32_t m_pq,
                                         bool vec16) {
  float s = 0.f;
  if (vec16) {
    for (uint32_t m0 = 0; m0 < m_pq; m0 += 16) {
      const uint4 w = __ldg(reinterpret_cast<const uint4*>(row + m0));
      const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int b = 0; b < 16; ++b) {
        const uint32_t c = (ws[b >> 2] >> ((b & 3) * 8)) & 0xFFu;
        s = __fadd_rn(s, lut[(m0 + b) * 256 + c]);
      }
    }
  } else {
    for (uint32_t m = 0; m < m_pq; ++m) s = __fadd_rn(s, lut[m * 256 + __ldg(row + m)]);
  }
  return s;
}

// PQ: ADC of a code row already in registers (MW 16-byte words, m_pq = 16 MW),
// sub-spaces added in order as adc_row does.
template <int MW>
__device__ __forceinline__ float adc_words(const float* __restrict__ lut, const uint4 (&w)[MW]) {
  float s = 0.f;
#pragma unroll
  for (int j = 0; j < MW; ++j) {
    const uint32_t ws[4] = {w[j].x, w[j].y, w[j].z, w[j].w};
#pragma unroll
    for (int b = 0; b < 16; ++b) {
      const uint32_t c = (ws[b >> 2] >> ((b & 3) * 8)) & 0xFFu;
      s = __fadd_rn(s, lut[(j * 16 + b) * 256 + c]);
    }
  }
  return s;
}

// PQ: ADC of one row without tables: the entry of each sub-space evaluated in
// place with the table's operations (the residual to the list's centroid
// rounded once per dimension, fmaf in sub-dimension order), added in sub-space
// order. Four sub-spaces' codewords are in flight at a time where rows of
// four dimensions load as float4 (v4).
template <typename CodeAt>
__device__ __forceinline__ float adc_direct(const IvfArgs& a, const float* qs, const float* __restrict__ cent,
                                            CodeAt code, bool v4) {
  float s = 0.f;
  if (v4) {
    const float4* cb = reinterpret_cast<const float4*>(a.codebooks);
    const float4* cc = reinterpret_cast<const float4*>(cent);
    constexpr uint32_t B = 4;
    for (uint32_t m0 = 0; m0 < a.m_pq; m0 += B) {
      float4 w[B], c[B];
#pragma unroll
      for (uint32_t b = 0; b < B; ++b) {
        const uint32_t m = min(m0 + b, a.m_pq - 1);
        w[b] = __ldg(cb + (size_t)m * 256 + code(m));
        c[b] = __ldg(cc + m);
      }
#pragma unroll
      for (uint32_t b = 0; b < B; ++b) {
        if (m0 + b >= a.m_pq) break;
        const float4 q = *reinterpret_cast<const float4*>(qs + (m0 + b) * 4);
        const float t0 = __fsub_rn(__fsub_rn(q.x, c[b].x), w[b].x), t1 = __fsub_rn(__fsub_rn(q.y, c[b].y), w[b].y);
        const float t2 = __fsub_rn(__fsub_rn(q.z, c[b].z), w[b].z), t3 = __fsub_rn(__fsub_rn(q.w, c[b].w), w[b].w);
        s = __fadd_rn(s, fmaf(t3, t3, fmaf(t2, t2, fmaf(t1, t1, fmaf(t0, t0, 0.f)))));
      }
    }
    return s;
  }
  for (uint32_t m = 0; m < a.m_pq; ++m) {
    const float* cb = a.codebooks + ((size_t)m * 256 + code(m)) * a.sub_dim;
    float e = 0.f;
    for (uint32_t sd = 0; sd < a.sub_dim; ++sd) {
      const uint32_t d = m * a.sub_dim + sd;
      const float t = __fsub_rn(__fsub_rn(qs[d], __ldg(cent + d)), __ldg(cb + sd));
      e = fmaf(t, t, e);
    }
    s = __fadd_rn(s, e);
  }
  return s;
}

// SQ8: squared L2 between the query's residual to the list's centroid and the
// decoded row, in dimension order; one row per thread (where the staging below
// does not fit).
__device__ __forceinline__ float sq8_row(const float* qs, const float* __restrict__ cent, const float* mins,
                                         const float* scales, const uint8_t* __restrict__ row, uint32_t dim) {
  float s = 0.f;
  for (uint32_t d = 0; d < dim; ++d) {
    const float rec = fmaf((float)__ldg(row + d), scales[d], mins[d]);
    const float t = __fsub_rn(__fsub_rn(qs[d], __ldg(cent + d)), rec);
    s = fmaf(t, t, s);
  }
  return s;
}

// SQ8, staged: a warp scores 2 x 32 rows, each lane two of them (one where no
// lane has a second). The rows' codes come in through shared memory by whole
// segments (a lane reading its own row touches one line per 16 bytes: 32 L1
// wavefronts where the segment takes 8), and one read of the query, centroid
// and decoding parameters serves both rows. RES: qs already holds the residual
// to the centroid that all rows share. A byte becomes a float by taking the
// mantissa's place in 2^23. row[i]: the lane's rows (null: none).
// Warp-collective.
//   PIPE: 32 dimensions at a time, the next ones copied while these are scored,
// which is what a call of few warps waits for (8 queries x 64 lists of 768
// dimensions 268 -> 232 us). Rows may start at any byte: words are copied
// aligned and shifted into place (397 dimensions, 300 queries: 2,588 -> 2,239). A
// word that holds a row's first or last byte is copied whole, so that up to 3
// bytes before and behind the table are read with it, and dropped; a word never
// crosses into another page or allocation. (Copying only a row's bytes of each word, by
// cp.async's source size, costs up to 15%: 100 dimensions, 3,000 queries: 2,167 us a
// call, 2,544.)
//   Otherwise 16-byte-aligned rows, 64 dimensions at a time: fewer steps, for
// calls whose warps cover each other's loads (2,000 queries, 128 dimensions:
// 2,721 us, and 3,081 with PIPE).
__device__ __forceinline__ void cp_async16(void* dst, uint64_t src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, uint64_t src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
template <bool RES, bool PIPE>
__device__ __forceinline__ void sq8_rows(const float* qs, const float* const (&cent)[2], const float* mins,
                                         const float* scales, const uint8_t* const (&row)[2], uint32_t dim,
                                         bool aligned, bool cent16, uint8_t* stage, float (&out)[2]) {
  const uint32_t lane = threadIdx.x & 31u;
  const int rows = __any_sync(0xffffffffu, row[1] != nullptr) ? 2 : 1;
  constexpr uint32_t CHUNK = PIPE ? 32 : 64;
  out[0] = out[1] = 0.f;
  // dimensions [d0, d0 + CHUNK) of the rows into buffer buf
  auto copy = [&](uint32_t d0, uint8_t* buf) {
    const uint32_t nd = min(CHUNK, dim - d0);
    for (int i = 0; i < rows; ++i) {
      const uint64_t mine = (uint64_t)(uintptr_t)(i ? row[1] : row[0]);
      if (aligned) {
        // two lanes a row, 16 bytes each; a row's halves change places every
        // four rows, which puts eight lanes' halves on different banks
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const uint32_t r = 16 * j + (lane >> 1), c = (lane & 1u) * 16;
          const uint64_t p = __shfl_sync(0xffffffffu, mine, r);
          if (p && c < nd) cp_async16(buf + (i * 32 + r) * 32 + (c ^ ((r & 4u) * 4)), p + d0 + c);
        }
      } else {
        // eight lanes a row, one aligned word each, and a ninth word where the
        // row's chunk reaches into it
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint32_t r = 4 * j + (lane >> 3), w = lane & 7u;
          const uint64_t p = __shfl_sync(0xffffffffu, mine, r);
          const uint64_t at = ((p + d0) & ~(uint64_t)3) + 4 * w;
          if (p && at < p + d0 + nd) cp_async4(buf + ((i * 32 + r) * SQ_WORDS + w) * 4, at);
        }
        const uint64_t at = ((mine + d0) & ~(uint64_t)3) + CHUNK;
        if (mine && at < mine + d0 + nd) cp_async4(buf + ((i * 32 + lane) * SQ_WORDS + SQ_WORDS - 1) * 4, at);
      }
    }
  };
  auto copy64 = [&](uint32_t d0) {
    const uint32_t nd = min(CHUNK, dim - d0);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if (i == rows) break;
      // four lanes a row, 16 bytes each
      uint4 w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t r = 8 * j + (lane >> 2), c = (lane & 3u) * 16;
        const uint64_t p = __shfl_sync(0xffffffffu, (uint64_t)(uintptr_t)row[i], r);
        w[j] = p && c < nd ? __ldg(reinterpret_cast<const uint4*>(p + d0 + c)) : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t r = 8 * j + (lane >> 2), c = (lane & 3u) * 16;
        *reinterpret_cast<uint4*>(stage + (i * 32 + r) * SQ_STRIDE + c) = w[j];
      }
    }
  };
  __syncwarp();  // the buffers are free
  if constexpr (PIPE) {
    copy(0, stage);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  uint32_t which = 0;
  for (uint32_t d0 = 0; d0 < dim; d0 += CHUNK, which ^= 1u) {
    const uint32_t nd = min(CHUNK, dim - d0);
    if constexpr (PIPE) {
      if (d0 + CHUNK < dim) copy(d0 + CHUNK, stage + (which ^ 1u) * SQ_BUF_BYTES);
      asm volatile("cp.async.commit_group;" ::: "memory");
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      copy64(d0);
    }
    __syncwarp();
    const uint8_t* buf = PIPE ? stage + which * SQ_BUF_BYTES : stage;
    const uint32_t stride = !PIPE ? SQ_STRIDE : aligned ? 32u : SQ_WORDS * 4;
    const uint32_t sh0 = 8 * ((uint32_t)((uintptr_t)row[0] + d0) & 3u), sh1 = 8 * ((uint32_t)((uintptr_t)row[1] + d0) & 3u);
    const uint8_t* st0 = buf + lane * stride;
    const uint8_t* st1 = st0 + 32 * stride;
    const uint32_t swap = PIPE ? (lane & 4u) * 4 : 0u;
    auto term = [&](float& s, uint32_t w, int b, float qd, float cd, float m, float k) {
      const float code = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u + b)) - 8388608.0f;  // exact
      const float t = __fsub_rn(RES ? qd : __fsub_rn(qd, cd), fmaf(code, k, m));
      s = fmaf(t, t, s);
    };
    auto score = [&](auto two) {
      constexpr bool TWO = decltype(two)::value;
      if ((!PIPE || aligned) && cent16) {
        for (uint32_t d = 0; d < nd; d += 16) {
          const uint4 wa = *reinterpret_cast<const uint4*>(st0 + (d ^ swap));
          const uint4 wb = TWO ? *reinterpret_cast<const uint4*>(st1 + (d ^ swap)) : wa;
          const uint32_t a4[4] = {wa.x, wa.y, wa.z, wa.w}, b4[4] = {wb.x, wb.y, wb.z, wb.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint32_t at = d0 + d + 4 * j;
            const float4 q = *reinterpret_cast<const float4*>(qs + at);
            const float4 mn = *reinterpret_cast<const float4*>(mins + at);
            const float4 sc = *reinterpret_cast<const float4*>(scales + at);
            float4 ca = q, cb = q;
            if (!RES) {
              ca = __ldg(reinterpret_cast<const float4*>(cent[0] + at));
              if (TWO) cb = cent[1] == cent[0] ? ca : __ldg(reinterpret_cast<const float4*>(cent[1] + at));
            }
            term(out[0], a4[j], 0, q.x, ca.x, mn.x, sc.x);
            if (TWO) term(out[1], b4[j], 0, q.x, cb.x, mn.x, sc.x);
            term(out[0], a4[j], 1, q.y, ca.y, mn.y, sc.y);
            if (TWO) term(out[1], b4[j], 1, q.y, cb.y, mn.y, sc.y);
            term(out[0], a4[j], 2, q.z, ca.z, mn.z, sc.z);
            if (TWO) term(out[1], b4[j], 2, q.z, cb.z, mn.z, sc.z);
            term(out[0], a4[j], 3, q.w, ca.w, mn.w, sc.w);
            if (TWO) term(out[1], b4[j], 3, q.w, cb.w, mn.w, sc.w);
          }
        }
      } else {
        for (uint32_t d = 0; d < nd; d += 4) {
          // (aligned rows, whose halves may have changed places: shifted by 0)
          const uint32_t at4 = !PIPE || aligned ? d ^ swap : d;
          const uint32_t* pa = reinterpret_cast<const uint32_t*>(st0 + at4);
          const uint32_t* pb = reinterpret_cast<const uint32_t*>(st1 + at4);
          const uint32_t wa = __funnelshift_r(pa[0], pa[1], sh0);
          const uint32_t wb = TWO ? __funnelshift_r(pb[0], pb[1], sh1) : 0u;
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            const uint32_t at = d0 + d + b;
            if (at >= dim) break;
            const float q = qs[at], mn = mins[at], sc = scales[at];
            float ca = q, cb = q;
            if (!RES) {
              ca = __ldg(cent[0] + at);
              if (TWO) cb = cent[1] == cent[0] ? ca : __ldg(cent[1] + at);
            }
            term(out[0], wa, b, q, ca, mn, sc);
            if (TWO) term(out[1], wb, b, q, cb, mn, sc);
          }
        }
      }
    };
    if (rows == 2)
      score(std::true_type{});
    else
      score(std::false_type{});
    __syncwarp();  // this buffer is consumed
  }
}

// A PQ list of at least this many postings gets its tables: building them
// reads the whole codebook and costs about as much as evaluating 128 rows in
// place (32 of the 8,192 entries each).
constexpr uint32_t PQ_TABLE_MIN = 128;
// A longer list of the other modes is walked by itself too: one list's query
// code (RaBitQ) or residual (SQ8) serves every posting without a search for
// its list. Below, a round of the CTA would be part empty.
constexpr uint32_t LIST_ALONE_MIN = 1024;

// Resident CTAs per SM each variant is compiled for (its register budget:
// 4 -> 64, 3 -> 85, 2 -> 128 registers per thread): the list scans are
// load-latency bound, so occupancy is worth more than registers.
template <int MODE, int MW>
constexpr int ivf_min_blocks() {
  return MODE == IVF_PQ ? (MW == 4 ? 2 : 3) : MODE == IVF_SQ8 || (MODE == IVF_RABITQ && MW >= 4) ? 3 : 4;
}

// MODE: PQ, SQ8 or RaBitQ. MW > 0: code rows of 16 * MW bytes at 16-byte-
// aligned rows (PQ m_pq = 16, 32, 64; RaBitQ P = 128 MW with 16-byte-aligned
// meta rows; SQ8 with staged rows, R = 2: MW = 1 the rows in turn, MW = 2 the next
// ones copied meanwhile), R postings per thread per
// round, all their loads before any is scored.
template <int MODE, int MW, int R>
__global__ void __launch_bounds__(IVF_THREADS, ivf_min_blocks<MODE, MW>()) ivf_scan_kernel(IvfArgs a) {
  // a round offers at most IVF_THREADS * R candidates, appended after the
  // shortlist; the buffer is flushed between rounds, so one round must fit
  static_assert((uint32_t)IVF_THREADS * R <= IVF_BUF, "a round of postings must fit the candidate buffer");
  constexpr uint32_t step = IVF_THREADS * R;
  constexpr int MWW = MW > 0 && MODE != IVF_SQ8 ? MW : 1;
  extern __shared__ __align__(16) uint8_t smem[];
  uint64_t* keys = reinterpret_cast<uint64_t*>(smem);
  float* tab = reinterpret_cast<float*>(smem + (size_t)a.keys_pow2 * 8);
  float* qs = tab + IvfSmem::table_floats(MODE, a.dim, a.m_pq, a.P, a.list_chunk);
  float* qres = qs + (a.dim + 3) / 4 * 4;  // PQ only: q - centroid of the probed list
  uint32_t* s_beg = reinterpret_cast<uint32_t*>(qres + (MODE == IVF_PQ ? a.dim : 0));
  uint32_t* s_list = s_beg + a.list_chunk;     // top bit: s_beg indexes the admitted positions
  uint32_t* s_cum = s_list + a.list_chunk;     // [chunk + 1] postings of the sequence before each list
  __shared__ uint32_t s_q, s_cnt, s_long, s_used;
  __shared__ uint64_t s_tau;
  __shared__ unsigned long long s_total;
  __shared__ float s_red[MODE == IVF_RABITQ ? IVF_THREADS : 1];

  KeepScratch* keep = a.keep_at ? reinterpret_cast<KeepScratch*>(smem + a.keep_at) : nullptr;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  float* mins = tab;                     // SQ8 only
  float* scales = tab + a.dim;
  float* rq = tab;                       // RaBitQ only: rotated query, list codes
  uint32_t* codes = reinterpret_cast<uint32_t*>(tab + a.P);
  const uint32_t code_words = 4 * a.W + 4;
  const bool cb4 = MODE == IVF_PQ && a.sub_dim == 4 && ((uintptr_t)a.codebooks % 16u) == 0;
  const bool vec16 = (a.code_bytes % 16u) == 0 && ((uintptr_t)a.codes % 16u) == 0;
  const bool cent16 = a.dim % 4 == 0 && ((uintptr_t)a.centroids % 16u) == 0;
  uint8_t* stage = smem + ((reinterpret_cast<uint8_t*>(s_cum + a.list_chunk + 1) - smem) + 15) / 16 * 16 +
                   warp * SQ_WARP_BYTES;  // SQ8, MW > 0

  if (MODE == IVF_SQ8) {
    for (uint32_t d = tid; d < a.dim; d += IVF_THREADS) {
      mins[d] = __ldg(a.sq_mins + d);
      scales[d] = __ldg(a.sq_scales + d);
    }
  }

  const uint32_t G = a.items_per_q;
  while (true) {
    __syncthreads();
    if (tid == 0) s_q = atomicAdd(a.work, 1u);
    __syncthreads();
    const uint32_t item = s_q;
    if (item >= a.nq * G) break;
    const uint32_t q = a.order ? __ldg(a.order + item / G) : item / G, g = item % G;
    uint32_t kq = a.q_topk ? __ldg(a.q_topk + q) : a.top_k;
    uint32_t npq = a.q_nprobe ? __ldg(a.q_nprobe + q) : a.nprobe;
    const uint32_t rrq = a.q_rerank ? __ldg(a.q_rerank + q) : a.rerank_k;
    const uint32_t S = ivf_clamps(kq, npq, rrq, a.nlist);
    npq = min(npq, a.nprobe);
    kq = min(kq, a.top_k);
    const bool do_rerank = rrq != 1u && a.vectors != nullptr;
    const QueryFilter qf = load_filter(a.filters, q);
    const GpuSearchResult* probes = a.probes + (size_t)q * a.nprobe;

    const float* qv = a.queries + (size_t)q * a.dim;
    for (uint32_t d = tid; d < a.dim; d += IVF_THREADS) qs[d] = __ldg(qv + d);
    for (uint32_t i = tid; i < S; i += IVF_THREADS) keys[i] = kSentinelKey;
    if (tid == 0) {
      s_cnt = 0;
      s_tau = kSentinelKey;
    }
    if (G > 1 && warp == 0) {
      // the query's probed postings, to cut this item's range out of
      unsigned long long total = 0;
      for (uint32_t p = lane; p < npq; p += 32) {
        const uint32_t l = probes[p].id;
        if (l < a.nlist) {
          const ListSpan sp = list_span(a, l);
          total += sp.end - sp.beg;
        }
      }
#pragma unroll
      for (int o = 16; o; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
      if (lane == 0) s_total = total;
    }
    __syncthreads();
    float qn = 0.f;  // RaBitQ, inner product: ||q||^2
    if constexpr (MODE == IVF_RABITQ) {
      if (a.metric == METRIC_INNER_PRODUCT) {
        // in the order of the reference's 256-thread block
        // (ivf_quant_lookup.cu:686-697): strided fmaf partials, pairwise fold
        float part = 0.f;
        for (uint32_t d = tid; d < a.dim; d += IVF_THREADS) part = __fmaf_rn(qs[d], qs[d], part);
        s_red[tid] = part;
        __syncthreads();
        for (int st = IVF_THREADS / 2; st > 0; st >>= 1) {
          if (tid < st) s_red[tid] = __fadd_rn(s_red[tid], s_red[tid + st]);
          __syncthreads();
        }
        qn = s_red[0];
      }
      rabitq_rotate_query(rq, qs, a);
    }
    // this item's range of the query's probed postings (lists in probe order)
    const uint64_t lo = G > 1 ? s_total * g / G : 0ull;
    const uint64_t hi = G > 1 ? s_total * (g + 1) / G : ~0ull;
    uint64_t cum = 0;  // postings of the lists before this chunk (warp 0)

    auto flush = [&]() {
      // keys[0, S) the shortlist, keys[S, S + cnt) new candidates
      const uint32_t cnt = s_cnt;  // block-uniform (read after a barrier)
      if (cnt == 0) return;
      uint64_t tau;
      if (keep && S + cnt > KEEP_MIN && S + cnt <= KEEP_MAX) {
        tau = block_keep_smallest<IVF_THREADS, KEEP_MAX / IVF_THREADS>(keys, S + cnt, S, *keep);
      } else {
        const uint32_t p2 = next_pow2_dev(S + cnt);  // sort only the occupied prefix
        for (uint32_t i = S + cnt + tid; i < p2; i += IVF_THREADS) keys[i] = kSentinelKey;
        __syncthreads();
        block_bitonic_sort(keys, p2);
        tau = keys[S - 1];
      }
      if (tid == 0) {
        s_cnt = 0;
        s_tau = tau;
      }
      __syncthreads();
    };
    // Barrier at a round's end; whether another round might not fit the buffer.
    // The thread that appended last sees the full count, and the decision is
    // the barrier's: read after it, the count could already hold candidates of
    // a faster warp's next round.
    auto round_full = [&]() { return __syncthreads_or(s_cnt > IVF_BUF - step) != 0; };
    // one posting per lane into the buffer (warp-collective): `at` is its id,
    // or its list position when the id has not been needed so far
    auto offer = [&](bool pass, float d, uint32_t at, bool is_pos, uint64_t tau) {
      pass = pass && d < kSentinelDist && float_order(d) <= (uint32_t)(tau >> 32);
      uint64_t key = 0;
      if (pass) {
        key = make_key(d, is_pos ? __ldg(a.vec_ids + at) : at);
        pass = key <= tau;
      }
      const uint32_t m = __ballot_sync(0xffffffffu, pass);
      if (m == 0u) return;
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(&s_cnt, (uint32_t)__popc(m));
      base = __shfl_sync(0xffffffffu, base, 0);
      if (pass) keys[S + base + __popc(m & ((1u << lane) - 1u))] = key;
    };
    // Posting i of a span: whether it exists and, where the mask's list-order
    // bits cover it, is admitted (its code row is loaded then), whether it is
    // to be scored (also the id-based mask and the query's filter), its list
    // position, and its id where that was needed.
    struct Post {
      uint32_t pos, id;
      bool in, ok, has_id;
    };
    auto fetch = [&](uint32_t i, bool in, bool compact) {
      Post p;
      bool bits = true;
      p.pos = i;
      if (compact) {  // i indexes the admitted positions: all pass the mask
        p.pos = in ? __ldg(a.adm_pos + i) : 0u;
      } else if (a.mask != nullptr) {
        bits = a.list_allow != nullptr && i < a.list_n;
        if (in && bits) in = (__ldg(a.list_allow + (i >> 5)) >> (i & 31u)) & 1u;
      }
      p.has_id = !a.list_major || qf.words != nullptr || !bits;
      p.id = in && p.has_id ? __ldg(a.vec_ids + p.pos) : 0u;
      p.in = p.ok = in;
      if (p.has_id && in) p.ok = (bits || mask_allows(a.mask, p.id)) && filter_allows(qf, p.id);
      return p;
    };

    for (uint32_t c0 = 0; c0 < npq; c0 += a.list_chunk) {
      const uint32_t nl = min(a.list_chunk, npq - c0);
      if (warp == 0) {
        // this item's part of each list, one list per lane
        uint32_t l = 0xFFFFFFFFu, beg = 0, len = 0;
        bool compact = false;
        if (lane < (int)nl) {
          l = probes[c0 + lane].id;
          if (l < a.nlist) {
            const ListSpan sp = list_span(a, l);
            beg = sp.beg;
            len = sp.end - sp.beg;
            compact = sp.compact;
          }
        }
        unsigned long long before = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const unsigned long long y = __shfl_up_sync(0xffffffffu, before, o);
          if (lane >= o) before += y;
        }
        const unsigned long long all = __shfl_sync(0xffffffffu, before, 31);
        before = cum + before - len;
        const uint64_t s0 = max((uint64_t)before, lo), s1 = min((uint64_t)before + len, hi);
        cum += all;
        if (s0 < s1) {
          beg += (uint32_t)(s0 - before);
          len = (uint32_t)(s1 - s0);
        } else {
          len = 0;
        }
        const uint32_t used = __ballot_sync(0xffffffffu, len > 0);
        // a list that is worth a walk of its own leaves the common sequence
        const bool tables = MODE == IVF_PQ ? len >= PQ_TABLE_MIN : MW > 0 && len >= LIST_ALONE_MIN;
        const uint32_t longs = __ballot_sync(0xffffffffu, tables);
        uint32_t x = tables ? 0u : len;
        const uint32_t own = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
          if (lane >= o) x += y;
        }
        if (lane < (int)nl) {
          s_beg[lane] = beg;
          s_list[lane] = (l & 0x7FFFFFFFu) | (compact ? 0x80000000u : 0u);
          s_cum[lane] = tables ? len : x - own;  // (such a list's entry: its length, see below)
        }
        if (lane == 0) {
          s_long = longs;
          s_used = used;
        }
        if (lane == (int)nl - 1) s_cum[nl] = x;
      }
      if constexpr (MODE == IVF_RABITQ) {
        // (of 64 ranges each has postings of a few lists: 40,000 x 3,000, 8 queries
        // of 64 lists: 794 us with all lists' codes in every range, 367 without)
        uint32_t used = ~0u;
        if (G > 1) {
          __syncthreads();
          used = s_used;
        }
        for (uint32_t p = warp; p < nl; p += IVF_THREADS / 32) {
          if (!((used >> p) & 1u)) continue;
          const GpuSearchResult pr = probes[c0 + p];
          if (pr.id < a.nlist) rabitq_query_code(rq, codes + p * code_words, a, pr.id, pr.distance);
        }
      }
      __syncthreads();

      if constexpr (MODE == IVF_PQ || MW > 0) {
        uint32_t longs = s_long;  // uniform over the block
        while (longs) {
          const uint32_t p = __ffs(longs) - 1;
          longs &= longs - 1;
          const uint32_t l = s_list[p] & 0x7FFFFFFFu, beg = s_beg[p], end = beg + s_cum[p];
          const bool compact = s_list[p] >> 31;
          const float* cent = a.centroids + (size_t)l * a.dim;
          if constexpr (MODE == IVF_PQ) {
            // LUT[m][c] = sum_sd ((q - centroid) - codeword)^2 with fmaf in
            // sub-dimension order; q - centroid is rounded once per dimension, as
            // the reference's expression rounds it (ivf_pq_lookup.cu:150-162)
            for (uint32_t d = tid; d < a.dim; d += IVF_THREADS) qres[d] = qs[d] - __ldg(cent + d);
            __syncthreads();
            const uint32_t entries = a.m_pq * 256;
            if (cb4) {
              const float4* cbv = reinterpret_cast<const float4*>(a.codebooks);
              auto entry = [&](uint32_t e, float4 w) {  // codeword (m, c) = row e of 4 floats
                const float* r = qres + (e >> 8) * 4;
                const float t0 = r[0] - w.x, t1 = r[1] - w.y, t2 = r[2] - w.z, t3 = r[3] - w.w;
                tab[e] = fmaf(t3, t3, fmaf(t2, t2, fmaf(t1, t1, fmaf(t0, t0, 0.f))));
              };
              // B codeword loads in flight per thread before any is used (the
              // codebooks, 16 KB per sub-space, stream from L2 for every list)
              constexpr uint32_t B = 8;
              uint32_t e0 = tid;
              for (; e0 + (B - 1) * IVF_THREADS < entries; e0 += B * IVF_THREADS) {
                float4 w[B];
#pragma unroll
                for (uint32_t b = 0; b < B; ++b) w[b] = __ldg(cbv + e0 + b * IVF_THREADS);
#pragma unroll
                for (uint32_t b = 0; b < B; ++b) entry(e0 + b * IVF_THREADS, w[b]);
              }
              for (uint32_t e = e0; e < entries; e += IVF_THREADS) entry(e, __ldg(cbv + e));
            } else {
              for (uint32_t e = tid; e < entries; e += IVF_THREADS) {
                const uint32_t m = e >> 8, c = e & 255u;
                const float* cb = a.codebooks + ((size_t)m * 256 + c) * a.sub_dim;
                float s = 0.f;
                for (uint32_t sd = 0; sd < a.sub_dim; ++sd) {
                  const float t = qres[m * a.sub_dim + sd] - __ldg(cb + sd);
                  s = fmaf(t, t, s);
                }
                tab[e] = s;
              }
            }
          } else if constexpr (MODE == IVF_SQ8) {
            float* res = tab + 2 * a.dim;
            for (uint32_t d = tid; d < a.dim; d += IVF_THREADS) res[d] = __fsub_rn(qs[d], __ldg(cent + d));
          }
          [[maybe_unused]] const uint32_t* code = codes + p * code_words;
          [[maybe_unused]] float4 par = make_float4(0.f, 0.f, 0.f, 0.f);
          if constexpr (MODE == IVF_RABITQ) par = *reinterpret_cast<const float4*>(code + 4 * a.W);
          __syncthreads();
          for (uint32_t base = beg; base < end; base += step) {
            Post post[R];
            uint4 w[R][MWW];
            float4 mt[MODE == IVF_RABITQ ? R : 1];
#pragma unroll
            for (int r = 0; r < R; ++r) {
              const uint32_t i = base + r * IVF_THREADS + tid;
              post[r] = fetch(i, i < end, compact);
              if constexpr (MODE == IVF_RABITQ)
                mt[r] = post[r].in ? __ldg(reinterpret_cast<const float4*>(a.rq_meta) +
                                           (a.list_major ? post[r].pos : post[r].id))
                                   : make_float4(0.f, 0.f, 0.f, 0.f);
              if constexpr (MW > 0 && MODE != IVF_SQ8) {
                const uint4* row = reinterpret_cast<const uint4*>(
                    a.codes + (size_t)(a.list_major ? post[r].pos : post[r].id) * (16u * MW));
#pragma unroll
                for (int j = 0; j < MWW; ++j) w[r][j] = post[r].in ? __ldg(row + j) : make_uint4(0u, 0u, 0u, 0u);
              }
            }
            const uint64_t tau = s_tau;
            [[maybe_unused]] float sq[2] = {0.f, 0.f};
            if constexpr (MODE == IVF_SQ8) {
              const uint8_t* rows[2];
#pragma unroll
              for (int r = 0; r < 2; ++r)
                rows[r] = post[r].ok ? a.codes + (size_t)(a.list_major ? post[r].pos : post[r].id) * a.code_bytes : nullptr;
              const float* const none[2] = {nullptr, nullptr};
              if (__any_sync(0xffffffffu, post[0].ok || post[1].ok))
                sq8_rows<true, MW == 2>(tab + 2 * a.dim, none, mins, scales, rows, a.dim, vec16, a.dim % 4 == 0, stage, sq);
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
              float d = 0.f;
              if constexpr (MODE == IVF_SQ8) {
                d = sq[r & 1];
              } else if (post[r].ok) {
                if constexpr (MODE == IVF_RABITQ)
                  d = rabitq_estimate(rabitq_sbu<MWW>(code, w[r]), mt[r], (float)a.P, par.x, par.y, par.z, par.w, qn,
                                      a.metric);
                else if constexpr (MW > 0)
                  d = adc_words<MWW>(tab, w[r]);
                else
                  d = adc_row(tab, a.codes + (size_t)(a.list_major ? post[r].pos : post[r].id) * a.code_bytes, a.m_pq,
                              vec16);
              }
              offer(post[r].ok, d, post[r].has_id ? post[r].id : post[r].pos, !post[r].has_id, tau);
            }
            if (round_full()) flush();
          }
        }
        if (s_long) {
          // the lists walked alone drop out of the sequence: their prefix entry
          // is the next list's
          __syncthreads();
          if (tid == 0)
            for (int p = (int)nl - 1; p >= 0; --p)
              if ((s_long >> p) & 1u) s_cum[p] = s_cum[p + 1];
          __syncthreads();
        }
      }

      // the sequence of the chunk's (other) postings
      const uint32_t total = s_cum[nl];
      uint32_t at_list = 0;  // the list of this thread's last posting (they only move on)
      for (uint32_t base = 0; base < total; base += step) {
        uint32_t lp[R];
        Post post[R];
        uint4 w[R][MWW];
        float4 mt[MODE == IVF_RABITQ ? R : 1];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const uint32_t t = base + r * IVF_THREADS + tid;
          // the last list whose prefix is <= t (empty lists repeat a prefix)
          uint32_t p = at_list;
          if (p + 1 < nl && s_cum[p + 1] <= t) {
            p = 0;
#pragma unroll
            for (uint32_t h = LIST_CHUNK / 2; h; h >>= 1)
              if (p + h < nl && s_cum[p + h] <= t) p += h;
          }
          lp[r] = at_list = p;
          post[r] = fetch(s_beg[p] + (t - s_cum[p]), t < total, s_list[p] >> 31);
          const size_t row = a.list_major ? post[r].pos : post[r].id;
          if constexpr (MODE != IVF_SQ8 && MW > 0) {
            const uint4* rw = reinterpret_cast<const uint4*>(a.codes + row * (16u * MW));
#pragma unroll
            for (int j = 0; j < MWW; ++j) w[r][j] = post[r].in ? __ldg(rw + j) : make_uint4(0u, 0u, 0u, 0u);
            if constexpr (MODE == IVF_RABITQ)
              mt[r] = post[r].in ? __ldg(reinterpret_cast<const float4*>(a.rq_meta) + row)
                                 : make_float4(0.f, 0.f, 0.f, 0.f);
          }
        }
        const uint64_t tau = s_tau;
        [[maybe_unused]] float sq[2] = {0.f, 0.f};
        if constexpr (MODE == IVF_SQ8 && MW > 0) {
          static_assert(R == 2, "two rows a lane");
          const uint8_t* rows[2];
          const float* cents[2];
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            rows[r] = post[r].ok ? a.codes + (size_t)(a.list_major ? post[r].pos : post[r].id) * a.code_bytes : nullptr;
            // (an unused row is scored against list 0's centroid and dropped)
            cents[r] = a.centroids + (post[r].ok ? (size_t)(s_list[lp[r]] & 0x7FFFFFFFu) * a.dim : 0);
          }
          if (__any_sync(0xffffffffu, post[0].ok || post[1].ok))
            sq8_rows<false, MW == 2>(qs, cents, mins, scales, rows, a.dim, vec16, cent16, stage, sq);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float d = 0.f;
          if (MODE == IVF_SQ8 && MW > 0) {
            d = sq[r & 1];
          } else if (post[r].ok) {
            const size_t row = a.list_major ? post[r].pos : post[r].id;
            const uint32_t l = s_list[lp[r]] & 0x7FFFFFFFu;
            if constexpr (MODE == IVF_RABITQ) {
              const uint32_t* code = codes + lp[r] * code_words;
              const float4 par = *reinterpret_cast<const float4*>(code + 4 * a.W);  // min, delta, sum u, distance
              if constexpr (MW > 0) {
                d = rabitq_estimate(rabitq_sbu<MWW>(code, w[r]), mt[r], (float)a.P, par.x, par.y, par.z, par.w, qn,
                                    a.metric);
              } else {
                const float* mp = a.rq_meta + row * 4;
                const float4 meta = make_float4(__ldg(mp), __ldg(mp + 1), __ldg(mp + 2), __ldg(mp + 3));
                const uint32_t sbu =
                    rabitq_sbu_any(code, reinterpret_cast<const uint32_t*>(a.codes + row * a.code_bytes), a.W);
                d = rabitq_estimate(sbu, meta, (float)a.P, par.x, par.y, par.z, par.w, qn, a.metric);
              }
            } else if constexpr (MODE == IVF_PQ) {
              const float* cent = a.centroids + (size_t)l * a.dim;
              if constexpr (MW > 0) {
                // (the code bytes again, from the cache: indexing the registers
                // by sub-space would spill them)
                const uint32_t* cw = reinterpret_cast<const uint32_t*>(a.codes + row * (16u * MW));
                d = adc_direct(a, qs, cent, [&](uint32_t m) { return (__ldg(cw + (m >> 2)) >> (8 * (m & 3))) & 255u; },
                               cb4 && cent16);
              } else {
                const uint8_t* cw = a.codes + row * a.code_bytes;
                d = adc_direct(a, qs, cent, [&](uint32_t m) { return (uint32_t)__ldg(cw + m); }, cb4 && cent16);
              }
            } else {
              d = sq8_row(qs, a.centroids + (size_t)l * a.dim, mins, scales, a.codes + row * a.code_bytes, a.dim);
            }
          }
          offer(post[r].ok, d, post[r].has_id ? post[r].id : post[r].pos, !post[r].has_id, tau);
        }
        if (round_full()) flush();
      }
      __syncthreads();  // the chunk's lists and codes are replaced
    }
    flush();
    if (G > 1) {
      // a range's shortlist goes to the merge kernel
      uint64_t* dst = a.partial + ((size_t)q * G + g) * a.part_stride;
      for (uint32_t i = tid; i < S; i += IVF_THREADS) dst[i] = keys[i];
      continue;
    }
    // (PQ has the registers for four rows in flight per warp: 2,000 queries with
    // 400 candidates 539 -> 506 us; two in the others' 64)
    ivf_finish_query<IVF_THREADS, MODE == IVF_PQ ? 4 : 2, 4>(a, keys, q, S, kq, do_rerank, qv, keep);
  }
}

// The order in which CTAs pull queries when there are more than run at once:
// most probed postings first, by half octaves (a counting sort: one warp per
// query counts and takes a place in its bucket, a second launch turns places
// into positions). A query over a Zipf base's head list takes several times
// the mean, and one pulled last had the GPU to itself: 2,000 RaBitQ queries
// over 1M rows, list scan 1,004 us in the given order.
constexpr uint32_t ORDER_BUCKETS = 62;  // next to the work counter in its 64 words

__device__ __forceinline__ uint32_t order_bucket(unsigned long long postings) {
  const uint32_t v = (uint32_t)min(postings, 0x7FFFFFFFull) | 1u;
  const uint32_t top = 31u - __clz(v);
  return min(2 * top + (top ? (v >> (top - 1)) & 1u : 0u), ORDER_BUCKETS - 1);
}

__global__ void __launch_bounds__(256) ivf_order_count_kernel(IvfArgs a, uint32_t* __restrict__ hist,
                                                              uint32_t* __restrict__ place) {
  const uint32_t q = (blockIdx.x * 256 + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (q >= a.nq) return;
  uint32_t kq = a.top_k, npq = a.q_nprobe ? __ldg(a.q_nprobe + q) : a.nprobe;
  ivf_clamps(kq, npq, 1u, a.nlist);
  npq = min(npq, a.nprobe);
  unsigned long long total = 0;
  for (uint32_t p = lane; p < npq; p += 32) {
    const uint32_t l = a.probes[(size_t)q * a.nprobe + p].id;
    if (l < a.nlist) {
      const ListSpan sp = list_span(a, l);
      total += sp.end - sp.beg;
    }
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
  if (lane == 0) {
    const uint32_t b = order_bucket(total);
    place[q] = atomicAdd(hist + b, 1u) << 6 | b;
  }
}

__global__ void __launch_bounds__(256) ivf_order_kernel(uint32_t nq, const uint32_t* __restrict__ hist,
                                                        const uint32_t* __restrict__ place,
                                                        uint32_t* __restrict__ order) {
  __shared__ uint32_t first[ORDER_BUCKETS];
  if (threadIdx.x < ORDER_BUCKETS) {
    uint32_t n = 0;  // queries in larger buckets
    for (uint32_t b = threadIdx.x + 1; b < ORDER_BUCKETS; ++b) n += __ldg(hist + b);
    first[threadIdx.x] = n;
  }
  __syncthreads();
  const uint32_t q = blockIdx.x * 256 + threadIdx.x;
  if (q < nq) {
    const uint32_t p = place[q];
    order[first[p & 63u] + (p >> 6)] = q;
  }
}

// G > 1: one CTA per query merges the G range shortlists (top S of their
// union, by key), reranks and writes the top k -- the same answer as one
// range holding every posting.
// NT: 256, or 1,024 where the queries leave SMs idle (more rows of the rerank
// are then in flight: 8 queries, 100 rows of 768: 57 us with 256).
template <int NT>
__global__ void __launch_bounds__(NT) ivf_merge_kernel(IvfArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  uint64_t* keys = reinterpret_cast<uint64_t*>(smem);
  const uint32_t q = blockIdx.x, G = a.items_per_q;
  uint32_t kq = a.q_topk ? __ldg(a.q_topk + q) : a.top_k;
  uint32_t npq = a.q_nprobe ? __ldg(a.q_nprobe + q) : a.nprobe;
  const uint32_t rrq = a.q_rerank ? __ldg(a.q_rerank + q) : a.rerank_k;
  const uint32_t S = ivf_clamps(kq, npq, rrq, a.nlist);
  kq = min(kq, a.top_k);
  const bool do_rerank = rrq != 1u && a.vectors != nullptr;
  __shared__ KeepScratch keep;
  const uint32_t total = G * S;
  const uint64_t* src = a.partial + (size_t)q * G * a.part_stride;
  for (uint32_t i = threadIdx.x; i < total; i += NT) keys[i] = __ldcg(src + (size_t)(i / S) * a.part_stride + i % S);
  // The S smallest of the ranges' shortlists: selected from registers (64
  // ranges of 100 took 127 us as one sort of 8,192 keys), or sorted where
  // that is the quicker, or the registers do not hold them.
  __syncthreads();
  if (total > KEEP_MIN && total <= 2048) {
    block_keep_smallest<NT, 2048 / NT>(keys, total, S, keep);
  } else if (total > KEEP_MIN && total <= 8192) {
    block_keep_smallest<NT, 8192 / NT>(keys, total, S, keep);
  } else {
    const uint32_t p2 = next_pow2_dev(total);
    for (uint32_t i = total + threadIdx.x; i < p2; i += NT) keys[i] = kSentinelKey;
    __syncthreads();
    block_bitonic_sort(keys, p2);
  }
  ivf_finish_query<NT, NT == 256 ? 4 : 2, 8>(a, keys, q, S, kq, do_rerank, a.queries + (size_t)q * a.dim, &keep);
}

// The mask in list order (one word per 32 list positions), for one call.
// Only positions inside the lists (< offsets[nlist]) read an id: vec_ids may
// be shorter than the id space n (an engine whose slots carry remapped ids).
__global__ void __launch_bounds__(256) ivf_list_mask_kernel(const uint32_t* __restrict__ vec_ids,
                                                            const uint32_t* __restrict__ offsets, uint32_t nlist,
                                                            uint32_t n, const uint32_t* __restrict__ mask,
                                                            uint32_t* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t postings = min(n, __ldg(offsets + nlist));
  const bool b = i < postings && mask_allows(mask, __ldg(vec_ids + i));
  const uint32_t w = __ballot_sync(0xffffffffu, b);
  if ((threadIdx.x & 31u) == 0 && i < n) out[i >> 5] = w;
}

// Compaction of the list-order mask (three launches): per 1,024-word block
// the count of admitted positions; an exclusive scan of those counts; per
// word the exclusive prefix count and the admitted positions themselves,
// in list order.
constexpr uint32_t ADM_BLOCK = 1024;

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t x, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  return x;
}

// exclusive prefix of v over the block (ADM_BLOCK threads), plus the block total
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* total) {
  __shared__ uint32_t s_warp[ADM_BLOCK / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t x = warp_incl_scan(v, lane);
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  if (warp == 0) s_warp[lane] = warp_incl_scan(s_warp[lane], lane);
  __syncthreads();
  const uint32_t excl = (warp ? s_warp[warp - 1] : 0u) + x - v;
  *total = s_warp[ADM_BLOCK / 32 - 1];
  __syncthreads();
  return excl;
}

__global__ void __launch_bounds__(ADM_BLOCK) adm_count_kernel(const uint32_t* __restrict__ words, uint32_t nwords,
                                                              uint32_t* __restrict__ block_sums) {
  const uint32_t w = blockIdx.x * ADM_BLOCK + threadIdx.x;
  uint32_t total;
  block_excl_scan(w < nwords ? __popc(__ldg(words + w)) : 0u, &total);
  if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

// in place, one block, ADM_BLOCK entries at a time with a running carry
__global__ void __launch_bounds__(ADM_BLOCK) adm_scan_kernel(uint32_t* __restrict__ sums, uint32_t n) {
  uint32_t carry = 0;
  for (uint32_t base = 0; base < n; base += ADM_BLOCK) {
    const uint32_t i = base + threadIdx.x;
    uint32_t total;
    const uint32_t excl = block_excl_scan(i < n ? sums[i] : 0u, &total);
    if (i < n) sums[i] = carry + excl;
    carry += total;
  }
}

__global__ void __launch_bounds__(ADM_BLOCK) adm_compact_kernel(const uint32_t* __restrict__ words, uint32_t nwords,
                                                                const uint32_t* __restrict__ block_off,
                                                                uint32_t* __restrict__ prefix,
                                                                uint32_t* __restrict__ pos) {
  const uint32_t w = blockIdx.x * ADM_BLOCK + threadIdx.x;
  uint32_t bits = w < nwords ? __ldg(words + w) : 0u, total;
  const uint32_t o = __ldg(block_off + blockIdx.x) + block_excl_scan(__popc(bits), &total);
  if (w < nwords) {
    prefix[w] = o;
    if (w == nwords - 1) prefix[nwords] = o + __popc(bits);
    for (uint32_t k = o; bits; ++k) {
      const uint32_t b = __ffs(bits) - 1;
      bits &= bits - 1;
      pos[k] = w * 32 + b;
    }
  }
}

// ---------------------------------------------------------------------------
// Tensor-core coarse probe (large nlist). The exact coarse probe is a Q x
// nlist fp32 scan; here an fp16 tensor-core scan of the centred queries
// (q - mu) against the centred centroids (c - mu; L2 distances do not move
// under the shift, the fp16 rounding error shrinks with the magnitudes)
// returns each query's K best lists by that approximate distance, their
// exact distances are recomputed with the exact probe's arithmetic (fmaf of
// q - c in dimension order), and the first nprobe by (distance, list) are
// kept. That is the exact probe list whenever no list outside the K can
// reach the nprobe-th place: every list outside has approximate distance
// >= t16 (the K-th approximate distance), an approximate distance is within
// `err` of the exact one (a bound from the fp16 unit roundoff, the fp32
// accumulation and the norms), so d_nprobe < (t16 - err) (1 - dim 2^-22)
// proves it. A query that fails the test, or whose candidate heaps may have
// dropped a key, is recomputed by the exact scan (coarse_exact_kernel).
constexpr int CO_THREADS = 256;
constexpr uint32_t CO_CHUNK = 2048;  // centroids per step of the exact fallback

// mu: the mean of up to 1,024 evenly spaced centroids (any shift is exact
// for L2; the mean keeps the fp16 values small). A block owns 32 dimensions
// and 32 strided row groups, so a thread's chain is 32 additions with
// independent loads: one thread per dimension over all 1,024 rows was a
// single block bound by that serial chain (4,096 x 128: 525 us of a 2,085 us
// search of 2,000 queries, now 1,584 us).
constexpr int MU_ROWS = 32;
__global__ void __launch_bounds__(32 * MU_ROWS) coarse_mu_kernel(const float* __restrict__ cent, uint32_t nlist,
                                                                 uint32_t dim, float* __restrict__ mu) {
  __shared__ float part[MU_ROWS][33];
  const uint32_t lane = threadIdx.x & 31, g = threadIdx.x >> 5;
  const uint32_t d = blockIdx.x * 32 + lane;
  const uint32_t s = min(nlist, 1024u);
  float acc = 0.f;
  if (d < dim) {
#pragma unroll 8
    for (uint32_t i = g; i < s; i += MU_ROWS) acc += __ldg(cent + (size_t)((uint64_t)i * nlist / s) * dim + d);
  }
  part[g][lane] = acc;
  __syncthreads();
  if (g == 0 && d < dim) {
    float sum = 0.f;
    for (int r = 0; r < MU_ROWS; ++r) sum += part[r][lane];
    mu[d] = sum / (float)s;
  }
}

// One block per row: rows [0, nlist) are centroids -> fp16 (c - mu) padded to
// pd, ||c - mu||^2, and the largest ||c - mu|| (float bits, atomicMax);
// rows [nlist, nlist + nq) are queries -> q - mu in fp32.
__global__ void __launch_bounds__(128) coarse_prep_kernel(const float* __restrict__ cent, uint32_t nlist,
                                                          const float* __restrict__ queries, uint32_t nq,
                                                          uint32_t dim, uint32_t pd, const float* __restrict__ mu,
                                                          __half* __restrict__ c16, float* __restrict__ cnorm,
                                                          uint32_t* __restrict__ cmax, float* __restrict__ qc) {
  const uint32_t r = blockIdx.x;
  if (r >= nlist) {
    const uint32_t q = r - nlist;
    for (uint32_t d = threadIdx.x; d < dim; d += 128)
      qc[(size_t)q * dim + d] = __fsub_rn(__ldg(queries + (size_t)q * dim + d), mu[d]);
    return;
  }
  __shared__ float s_red[4];
  float part = 0.f;
  for (uint32_t d = threadIdx.x; d < pd; d += 128) {
    const float v = d < dim ? __fsub_rn(__ldg(cent + (size_t)r * dim + d), mu[d]) : 0.f;
    c16[(size_t)r * pd + d] = __float2half_rn(v);
    part = fmaf(v, v, part);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = part;
  __syncthreads();
  if (threadIdx.x == 0) {
    const float n2 = (s_red[0] + s_red[1]) + (s_red[2] + s_red[3]);
    cnorm[r] = n2;
    atomicMax(cmax, __float_as_uint(sqrtf(n2)));
  }
}

// exact coarse distance of query row qv (shared) to centroid c: the exact
// probe's arithmetic (flat_f32_scan_kernel, FUSED)
__device__ __forceinline__ float coarse_exact(const float* qv, const float* __restrict__ c, uint32_t dim) {
  float acc = 0.f;
  uint32_t d = 0;
  if (dim % 4 == 0 && (uintptr_t)c % 16 == 0) {
    for (; d + 32 <= dim; d += 32) {  // eight 16-byte loads in flight
      float4 v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = __ldg(reinterpret_cast<const float4*>(c + d) + i);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 q = *reinterpret_cast<const float4*>(qv + d + 4 * i);
        const float d0 = __fsub_rn(q.x, v[i].x), d1 = __fsub_rn(q.y, v[i].y);
        const float d2 = __fsub_rn(q.z, v[i].z), d3 = __fsub_rn(q.w, v[i].w);
        acc = fmaf(d0, d0, acc);
        acc = fmaf(d1, d1, acc);
        acc = fmaf(d2, d2, acc);
        acc = fmaf(d3, d3, acc);
      }
    }
  }
  for (; d < dim; ++d) {
    const float diff = __fsub_rn(qv[d], __ldg(c + d));
    acc = fmaf(diff, diff, acc);
  }
  return acc;
}

// Per query: exact distances of the K candidates, the first nprobe, and the
// exactness test. flags[q] = 1 sends the query to the exact fallback. NT
// threads (>= K, and at least 64): one candidate each; blocks of 256 for 48
// candidates left most threads idle and two thirds of the queries waiting
// (2,000 queries: 61 us).
template <int NT>
__global__ void __launch_bounds__(NT) coarse_finish_kernel(const float* __restrict__ queries,
                                                                   const float* __restrict__ cent, uint32_t nlist,
                                                                   uint32_t dim, const GpuSearchResult* __restrict__ cand,
                                                                   uint32_t K, uint32_t nprobe,
                                                                   const float* __restrict__ qc,
                                                                   const uint32_t* __restrict__ cmax,
                                                                   uint32_t force_exact, uint32_t* __restrict__ flags,
                                                                   GpuSearchResult* __restrict__ probes) {
  extern __shared__ __align__(16) uint8_t co_smem[];
  uint64_t* keys = reinterpret_cast<uint64_t*>(co_smem);          // [NT]
  float* qv = reinterpret_cast<float*>(co_smem + NT * 8);         // [dim]
  __shared__ float s_red[NT / 32];
  const uint32_t q = blockIdx.x;
  const int tid = threadIdx.x;
  float part = 0.f;
  for (uint32_t d = tid; d < dim; d += NT) {
    qv[d] = __ldg(queries + (size_t)q * dim + d);
    const float c = __ldg(qc + (size_t)q * dim + d);
    part = fmaf(c, c, part);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  if ((tid & 31) == 0) s_red[tid >> 5] = part;
  __syncthreads();
  const GpuSearchResult* cq = cand + (size_t)q * K;
  if (tid < (int)K) {
    const uint32_t id = cq[tid].id;
    keys[tid] = id < nlist ? make_key(coarse_exact(qv, cent + (size_t)id * dim, dim), id) : kSentinelKey;
  } else {
    keys[tid] = kSentinelKey;
  }
  __syncthreads();
  block_bitonic_sort(keys, NT);
  for (uint32_t j = tid; j < nprobe; j += NT) probes[(size_t)q * nprobe + j] = key_to_result(keys[j], nullptr);
  if (tid == 0 && K < nlist) {
    float qn2 = 0.f;
    for (int w = 0; w < NT / 32; ++w) qn2 += s_red[w];
    const float qn = sqrtf(qn2), cm = __uint_as_float(*cmax);
    const GpuSearchResult last = cq[K - 1];
    const float dnp = key_dist(keys[nprobe - 1]);
    bool ok = last.id < nlist && keys[nprobe - 1] != kSentinelKey && qn < 3.0e4f && cm < 3.0e4f;
    if (ok) {
      const float t16 = last.distance;
      const float fd = (float)dim;
      // |q.c - fp16(q).fp16(c)| <= (2.01 u16 + dim 2^-23) |q| |c| + dim 2^-25 (|q| + |c|)
      const float e_dot = (2.01f * 4.8828125e-4f + fd * 1.1920929e-7f) * qn * cm + fd * 2.9802322e-8f * (qn + cm);
      const float e_norm = fd * 1.1920929e-7f * (qn2 + cm * cm);
      const float e_add = 4.7683716e-7f * (qn2 + cm * cm + 2.f * qn * cm);
      const float err = 2.f * e_dot + e_norm + e_add;
      ok = dnp < (t16 - err) * (1.f - fd * 2.3841858e-7f);
    }
    if (!ok || force_exact) flags[q] = 1u;
  }
}

// The exact probe of a flagged query (the others return at once): every
// centroid's exact distance, the running best nprobe kept by sorting it
// with each chunk of CO_CHUNK new keys.
__global__ void __launch_bounds__(CO_THREADS) coarse_exact_kernel(const float* __restrict__ queries,
                                                                  const float* __restrict__ cent, uint32_t nlist,
                                                                  uint32_t dim, uint32_t nprobe,
                                                                  const uint32_t* __restrict__ flags,
                                                                  GpuSearchResult* __restrict__ probes) {
  const uint32_t q = blockIdx.x;
  if (flags[q] == 0u) return;
  extern __shared__ __align__(16) uint8_t co_smem[];
  constexpr uint32_t NK = 4096;                                    // pow2 >= 256 + CO_CHUNK
  uint64_t* keys = reinterpret_cast<uint64_t*>(co_smem);          // [NK]
  float* qv = reinterpret_cast<float*>(co_smem + NK * 8);         // [dim]
  const int tid = threadIdx.x;
  for (uint32_t d = tid; d < dim; d += CO_THREADS) qv[d] = __ldg(queries + (size_t)q * dim + d);
  for (uint32_t i = tid; i < 256; i += CO_THREADS) keys[i] = kSentinelKey;
  __syncthreads();
  for (uint32_t c0 = 0; c0 < nlist; c0 += CO_CHUNK) {
    for (uint32_t i = tid; i < NK - 256; i += CO_THREADS) {
      const uint32_t c = c0 + i;
      keys[256 + i] = (i < CO_CHUNK && c < nlist) ? make_key(coarse_exact(qv, cent + (size_t)c * dim, dim), c)
                                                  : kSentinelKey;
    }
    __syncthreads();
    block_bitonic_sort(keys, NK);
  }
  for (uint32_t j = tid; j < nprobe; j += CO_THREADS) probes[(size_t)q * nprobe + j] = key_to_result(keys[j], nullptr);
}

__global__ void relayout_codes_kernel(const uint8_t* __restrict__ by_id, const uint32_t* __restrict__ vec_ids,
                                      uint32_t n, uint32_t row_bytes, uint8_t* __restrict__ by_list) {
  const uint64_t total = (uint64_t)n * row_bytes;
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t pos = e / row_bytes, b = e % row_bytes;
    by_list[e] = by_id[(uint64_t)__ldg(vec_ids + pos) * row_bytes + b];
  }
}

size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

// Committed autotuner results for the IVF scans (tuning/gb300.json
// "ivf_entries", compiled in by build.py as tuning_ivf.inc): per shape range
// the posting-range split and the coarse probe that searched fastest (every
// choice gives the same answer; the pipelining they also record belonged to
// an earlier list scan). Knobs set with fv_tune_set take precedence;
// "tc.table" = 0 ignores the table.
struct IvfTuneEntry {
  int mode;
  uint32_t dim_lo, dim_hi;
  uint64_t n_lo, n_hi;
  uint32_t nlist_lo, nlist_hi, nq_lo, nq_hi, np_lo, np_hi;
  int pipeline, split, tc_coarse;
};
const IvfTuneEntry kIvfTuneTable[] = {
#include "tuning_ivf.inc"
    {-1, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, -1, -1, -1}};

const IvfTuneEntry* ivf_tune_lookup(int mode, uint32_t dim, uint64_t n, uint32_t nlist, uint32_t nq,
                                    uint32_t nprobe) {
  if (tune_value("tc.table", 1) == 0) return nullptr;
  for (const IvfTuneEntry& e : kIvfTuneTable) {
    if (e.mode < 0) break;
    if (e.mode == mode && dim >= e.dim_lo && dim <= e.dim_hi && n >= e.n_lo && n <= e.n_hi && nlist >= e.nlist_lo &&
        nlist <= e.nlist_hi && nq >= e.nq_lo && nq <= e.nq_hi && nprobe >= e.np_lo && nprobe <= e.np_hi)
      return &e;
  }
  return nullptr;
}

// A knob's value: the explicit setting, else the table entry's, else `dflt`
// (-1 in both means automatic).
int64_t ivf_knob(const char* key, int table_value, int64_t dflt) {
  const int64_t v = tune_value(key, -1);
  if (v >= 0) return v;
  if (table_value >= 0) return table_value;
  return dflt;
}

// Every size of one IVF search call, computed once: launch_ivf_search
// launches from it and the serving loop admits a batch by scratch_bytes.
// rc: 0 to launch, 1 when the call has nothing to do, else an error code.
struct IvfPlan {
  int rc = 0;
  uint32_t P = 0, top_k = 0, nprobe = 0, shortlist = 0, G = 1, sms = 0, list_n = 0, nwords = 0, adm_blocks = 0;
  // tensor-core coarse probe: candidates per query and the byte offsets of
  // its buffers in the coarse part of the scratch
  bool tcc = false, force_exact = false;
  uint32_t K = 0;
  size_t co_mu = 0, co_c16 = 0, co_cnorm = 0, co_qc = 0, co_cand = 0, co_flags = 0, co_cmax = 0, co_tc = 0;
  TcPlan tc;
  FlatPlan cp;
  size_t coarse_bytes = 0, probe_bytes = 0, part_bytes = 0, allow_bytes = 0, scratch_bytes = 0;
};

IvfPlan plan_ivf_search(int mode, const IvfLaunch& L) {
  IvfPlan Q{};
  auto refuse = [&](int rc) {
    Q.rc = rc;
    return Q;
  };
  if (L.nq == 0 || L.top_k == 0 || L.nlist == 0 || L.dim == 0 || (mode == IVF_PQ && L.m_pq == 0)) return refuse(1);
  const uint32_t P = mode == IVF_RABITQ ? L.padded_dim : 0;
  if (mode == IVF_RABITQ && (P < 32 || P > 4096 || (P & (P - 1)) || P < L.dim)) return refuse(FV_ERR_ARG);
  // uniform batch: the clamps of the call; heterogeneous batch: top_k,
  // nprobe and rerank_k are the batch maxima and bound every query's values
  uint32_t top_k = L.top_k, nprobe = L.nprobe;
  uint32_t shortlist = ivf_clamps(top_k, nprobe, L.rerank_k, L.nlist);
  if (L.q_rerank) shortlist = std::min(std::max(std::max(L.rerank_k, top_k), shortlist), MAX_SHORTLIST);
  if (nprobe > (uint32_t)kMaxTopK) return refuse(FV_ERR_ARG);  // coarse selection keeps <= 256 lists
  if (mode == IVF_PQ && (L.sub_dim == 0 || L.m_pq * L.sub_dim > L.dim)) return refuse(FV_ERR_ARG);

  // Work items: with fewer queries than ~4 CTAs per SM, each query's probed
  // postings are cut into G equal ranges (a Zipf-giant list spreads over G
  // CTAs); each range keeps its own shortlist and ivf_merge_kernel joins
  // them. "ivf.split": -1 automatic, 0 / 1 never, G > 1 force G.
  const uint32_t sms = (uint32_t)device_sm_count();
  const IvfTuneEntry* te = ivf_tune_lookup(mode, L.dim, L.num_vectors, L.nlist, L.nq, nprobe);
  const int64_t split_knob = ivf_knob("ivf.split", te ? te->split : -1, -1);
  uint32_t G = 1;
  if (split_knob > 1)
    G = (uint32_t)split_knob;
  else if (split_knob < 0 && L.nq < 4 * sms) {
    // A few queries are cut into as many ranges as run at once (equal ones: a
    // range too many is a second wave); more queries into somewhat more, whose
    // unequal lists the CTAs even out by pulling.
    const uint32_t slots = (mode == IVF_RABITQ ? 4u : 3u) * sms;
    G = 8 * L.nq <= slots ? slots / L.nq : (4 * sms + L.nq - 1) / L.nq;
  }
  G = std::max(1u, std::min<uint32_t>(std::min(G, 64u), 16384u / next_pow2(shortlist)));

  // coarse probe: exact fp32 scan, or the tensor-core candidates + exact
  // rescore ("ivf.tc_coarse": -1 automatic, 0 off, 1 on, 2 on with every
  // query sent to the exact fallback -- a check of the fallback)
  const int64_t tcc_knob = ivf_knob("ivf.tc_coarse", te ? te->tc_coarse : -1, -1);
  const uint32_t K = std::min<uint32_t>(std::min(256u, nprobe + 16), L.nlist);
  // (tables of at least one 256-row tile and one 64-element K block, so no
  // TMA box is larger than the tensor it reads)
  const bool tcc_fits = L.nlist >= 256 && L.dim >= 64;
  const bool tcc = tcc_fits && (tcc_knob > 0 || (tcc_knob < 0 && L.nlist >= 2048 && L.nq >= 256 &&
                                                  K == nprobe + 16 && K < L.nlist));
  const uint32_t pd16 = (L.dim + 15) / 16 * 16;
  TcTables ct{false, nullptr, nullptr, nullptr, nullptr, L.nlist, L.dim, pd16};
  const FvScanOptions copt{0, 0, 0.f, 0};
  size_t tc_bytes = 0;
  if (tcc) {
    Q.co_mu = 0;
    Q.co_c16 = align256(Q.co_mu + (size_t)L.dim * 4);
    Q.co_cnorm = (Q.co_c16 + (size_t)L.nlist * pd16 * 2 + 1023) / 1024 * 1024;
    Q.co_qc = align256(Q.co_cnorm + (size_t)L.nlist * 4);
    Q.co_cand = align256(Q.co_qc + (size_t)L.nq * L.dim * 4);
    Q.co_flags = align256(Q.co_cand + (size_t)L.nq * K * 8);
    Q.co_cmax = align256(Q.co_flags + (size_t)L.nq * 4);
    Q.co_tc = (Q.co_cmax + 256 + 1023) / 1024 * 1024;
    Q.tc = plan_tc_scan(ct, L.nq, K, METRIC_L2, copt);
    tc_bytes = Q.co_tc + Q.tc.scratch_bytes;
  }
  Q.tcc = tcc;
  Q.K = K;
  Q.force_exact = tcc_knob == 2;

  // scratch: coarse heaps | probes | range shortlists | work counter
  const FlatPlan cp = plan_flat_f32(L.nlist, L.nq, nprobe, 0);
  const size_t coarse_bytes = tcc ? (tc_bytes + 1023) / 1024 * 1024 : align256(cp.scratch_bytes);
  const size_t probe_bytes = align256((size_t)L.nq * nprobe * sizeof(GpuSearchResult));
  const size_t part_bytes = G > 1 ? align256((size_t)L.nq * G * shortlist * 8) : 0;
  const uint32_t list_n = L.mask ? L.num_vectors : 0u;
  const size_t nwords = ((size_t)list_n + 31) / 32;
  const size_t allow_bytes = align256(nwords * 4);
  // compaction of the admitted positions ("ivf.compact" 0 turns it off)
  const bool compact = list_n > 0 && tune_value("ivf.compact", 1) != 0;
  const uint32_t adm_blocks = compact ? (uint32_t)((nwords + ADM_BLOCK - 1) / ADM_BLOCK) : 0u;
  const size_t adm_bytes = compact ? align256((size_t)adm_blocks * 4) + align256((nwords + 1) * 4) +
                                         align256((size_t)list_n * 4)
                                   : 0;
  Q.P = P;
  Q.top_k = top_k;
  Q.nprobe = nprobe;
  Q.shortlist = shortlist;
  Q.G = G;
  Q.sms = sms;
  Q.list_n = list_n;
  Q.cp = cp;
  Q.coarse_bytes = coarse_bytes;
  Q.probe_bytes = probe_bytes;
  Q.part_bytes = part_bytes;
  Q.allow_bytes = allow_bytes;
  Q.adm_blocks = adm_blocks;
  Q.nwords = (uint32_t)nwords;
  Q.scratch_bytes = coarse_bytes + probe_bytes + part_bytes + 256 + allow_bytes + adm_bytes;
  return Q;
}

}  // namespace

// The tensor-core coarse probe of one call into probes[nq][nprobe] (exact:
// see coarse_finish_kernel); its buffers are the coarse part of `scratch`.
static int launch_coarse_tc(const IvfPlan& Q, const IvfLaunch& L, uint8_t* scratch, GpuSearchResult* probes,
                     cudaStream_t stream) {
  ProfScope ps("coarse_tc", stream);
  float* mu = reinterpret_cast<float*>(scratch + Q.co_mu);
  __half* c16 = reinterpret_cast<__half*>(scratch + Q.co_c16);
  float* cnorm = reinterpret_cast<float*>(scratch + Q.co_cnorm);
  float* qc = reinterpret_cast<float*>(scratch + Q.co_qc);
  GpuSearchResult* cand = reinterpret_cast<GpuSearchResult*>(scratch + Q.co_cand);
  uint32_t* flags = reinterpret_cast<uint32_t*>(scratch + Q.co_flags);
  uint32_t* cmax = reinterpret_cast<uint32_t*>(scratch + Q.co_cmax);
  const uint32_t pd16 = (L.dim + 15) / 16 * 16;
  cudaError_t e = cudaMemsetAsync(flags, 0, (size_t)L.nq * 4, stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(cmax, 0, 4, stream);
  if (e != cudaSuccess) return (int)e;
  coarse_mu_kernel<<<(L.dim + 31) / 32, 32 * MU_ROWS, 0, stream>>>(L.centroids, L.nlist, L.dim, mu);
  coarse_prep_kernel<<<L.nlist + L.nq, 128, 0, stream>>>(L.centroids, L.nlist, L.queries, L.nq, L.dim, pd16, mu, c16,
                                                         cnorm, cmax, qc);
  note_launch(2);
  const TcTables ct{false, c16, cnorm, nullptr, nullptr, L.nlist, L.dim, pd16};
  const FvScanOptions copt{0, 0, 0.f, 0};
  int rc = launch_tc_scan_planned(Q.tc, ct, qc, L.nq, Q.K, METRIC_L2, nullptr, cand, copt, stream, nullptr,
                                  scratch + Q.co_tc, flags);
  if (rc != 0) return rc;
  const uint32_t fthreads = Q.K <= 64 ? 64u : 256u;
  const size_t fsmem = fthreads * 8 + (size_t)L.dim * 4;
  auto finish = fthreads == 64 ? coarse_finish_kernel<64> : coarse_finish_kernel<256>;
  const size_t xsmem = 4096 * 8 + (size_t)L.dim * 4;
  e = cudaFuncSetAttribute(finish, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fsmem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(coarse_exact_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)xsmem);
  if (e != cudaSuccess) return (int)e;
  finish<<<L.nq, fthreads, fsmem, stream>>>(L.queries, L.centroids, L.nlist, L.dim, cand, Q.K, Q.nprobe, qc, cmax,
                                            Q.force_exact ? 1u : 0u, flags, probes);
  coarse_exact_kernel<<<L.nq, CO_THREADS, xsmem, stream>>>(L.queries, L.centroids, L.nlist, L.dim, Q.nprobe, flags,
                                                          probes);
  note_launch(2);
  return (int)cudaGetLastError();
}

int ivf_tune_query(int mode, uint32_t dim, uint64_t n, uint32_t nlist, uint32_t nq, uint32_t nprobe,
                   int32_t* out3) {
  const IvfTuneEntry* e = ivf_tune_lookup(mode, dim, n, nlist, nq, nprobe);
  if (!e) return FV_ERR_ARG;
  out3[0] = e->pipeline;
  out3[1] = e->split;
  out3[2] = e->tc_coarse;
  return 0;
}

size_t ivf_search_scratch_bytes(int mode, const IvfLaunch& L) {
  const IvfPlan Q = plan_ivf_search(mode, L);
  return Q.rc == 0 ? Q.scratch_bytes : 0;
}

int launch_ivf_search(int mode, const IvfLaunch& L, cudaStream_t stream) {
  const IvfPlan Q = plan_ivf_search(mode, L);
  if (Q.rc) return Q.rc == 1 ? 0 : Q.rc;
  const uint32_t P = Q.P, top_k = Q.top_k, nprobe = Q.nprobe, shortlist = Q.shortlist, G = Q.G, sms = Q.sms;
  const uint32_t list_n = Q.list_n;
  const FlatPlan& cp = Q.cp;
  const size_t coarse_bytes = Q.coarse_bytes, probe_bytes = Q.probe_bytes, part_bytes = Q.part_bytes;
  uint8_t* scratch = static_cast<uint8_t*>(scratch_get(stream, Q.scratch_bytes));
  if (!scratch) return (int)cudaErrorMemoryAllocation;
  uint32_t* list_allow =
      list_n ? reinterpret_cast<uint32_t*>(scratch + coarse_bytes + probe_bytes + part_bytes + 256) : nullptr;
  GpuSearchResult* probes = reinterpret_cast<GpuSearchResult*>(scratch + coarse_bytes);
  uint64_t* partial = G > 1 ? reinterpret_cast<uint64_t*>(scratch + coarse_bytes + probe_bytes) : nullptr;
  uint32_t* work = reinterpret_cast<uint32_t*>(scratch + coarse_bytes + probe_bytes + part_bytes);

  int rc = 0;
  if (Q.tcc) {
    rc = launch_coarse_tc(Q, L, scratch, probes, stream);
  } else {
    rc = launch_flat_f32_planned(cp, L.centroids, nullptr, L.nlist, L.dim, L.queries, L.nq, nprobe, METRIC_L2,
                                 nullptr, probes, true, cp.scratch_bytes ? scratch : nullptr, stream);
  }
  if (rc != 0) return rc;
  cudaError_t e = cudaMemsetAsync(work, 0, 256, stream);  // the counter and the order's buckets
  if (e != cudaSuccess) return (int)e;
  if (list_n) {
    ProfScope ps("ivf_list_mask", stream);
    ivf_list_mask_kernel<<<(list_n + 255) / 256, 256, 0, stream>>>(L.vec_ids, L.offsets, L.nlist, list_n, L.mask,
                                                                     list_allow);
    note_launch();
  }
  uint32_t *adm_prefix = nullptr, *adm_pos = nullptr;
  if (Q.adm_blocks) {
    uint32_t* adm_sums = list_allow + Q.allow_bytes / 4;
    adm_prefix = adm_sums + align256((size_t)Q.adm_blocks * 4) / 4;
    adm_pos = adm_prefix + align256(((size_t)Q.nwords + 1) * 4) / 4;
    ProfScope ps("ivf_mask_compact", stream);
    adm_count_kernel<<<Q.adm_blocks, ADM_BLOCK, 0, stream>>>(list_allow, Q.nwords, adm_sums);
    adm_scan_kernel<<<1, ADM_BLOCK, 0, stream>>>(adm_sums, Q.adm_blocks);
    adm_compact_kernel<<<Q.adm_blocks, ADM_BLOCK, 0, stream>>>(list_allow, Q.nwords, adm_sums, adm_prefix, adm_pos);
    note_launch(3);
  }

  IvfArgs a{};
  a.centroids = L.centroids;
  a.codebooks = L.codebooks;
  a.sq_mins = L.sq_mins;
  a.sq_scales = L.sq_scales;
  a.codes = L.codes;
  a.offsets = L.offsets;
  a.vec_ids = L.vec_ids;
  a.vectors = L.vectors;
  a.num_vectors = L.num_vectors;
  a.dim = L.dim;
  a.nlist = L.nlist;
  a.m_pq = L.m_pq;
  a.sub_dim = L.sub_dim;
  a.code_bytes = mode == IVF_PQ ? L.m_pq : mode == IVF_SQ8 ? L.dim : P / 8;
  if (mode == IVF_RABITQ) {
    a.codes = reinterpret_cast<const uint8_t*>(L.rq_bits);
    a.rot_centroids = L.rot_centroids;
    a.rq_meta = L.rq_meta;
    a.rot_signs = L.rot_signs;
    a.P = P;
    a.W = P / 32;
    a.inv_sqrt_p = rabitq_inv_sqrt(P);
  }
  a.queries = L.queries;
  a.nq = L.nq;
  a.top_k = top_k;
  a.nprobe = nprobe;
  a.rerank_k = L.rerank_k;
  a.list_major = L.list_major ? 1u : 0u;
  a.metric = (int)L.metric;
  a.mask = L.mask;
  a.list_allow = list_allow;
  a.list_n = list_n;
  a.adm_pos = adm_pos;
  a.adm_prefix = adm_prefix;
  a.q_topk = L.q_topk;
  a.q_nprobe = L.q_nprobe;
  a.q_rerank = L.q_rerank;
  a.filters = L.filters;
  a.probes = probes;
  a.work = work;
  a.out = L.out;
  a.status = status_word();
  a.keys_pow2 = next_pow2(shortlist + IVF_BUF);
  a.items_per_q = G;
  a.partial = partial;
  a.part_stride = shortlist;

  // (calls near the limit walk four lists at a time, in the shared memory that
  // one list's tables take)
  a.list_chunk = LIST_CHUNK;
  size_t smem = IvfSmem::bytes(mode, a.keys_pow2, L.dim, L.m_pq, P, a.list_chunk);
  if (smem > 224 * 1024) {
    a.list_chunk = 4;
    smem = IvfSmem::bytes(mode, a.keys_pow2, L.dim, L.m_pq, P, a.list_chunk);
  }
  if (smem > 227 * 1024) return FV_ERR_ARG;
  const size_t staged = mode == IVF_SQ8 ? IvfSmem::staged_bytes(a.keys_pow2, L.dim, a.list_chunk) : 0;
  // (1 KB short of the limit, which the kernel's static shared memory counts against)
  const bool stage_rows = staged > 0 && staged <= 226 * 1024;
  if (stage_rows) smem = staged;
  // scratch of the flushes' selection, where shortlist and buffer fit its
  // registers (and the block has room: else they sort)
  const size_t keep_at = (smem + 15) / 16 * 16;
  if (shortlist + IVF_BUF <= KEEP_MAX && keep_at + sizeof(KeepScratch) <= 224 * 1024) {
    a.keep_at = (uint32_t)keep_at;
    smem = keep_at + sizeof(KeepScratch);
  }
  const bool rows16 = mode == IVF_PQ && ((uintptr_t)L.codes % 16u) == 0;
  // SQ8: rows copied ahead where they may start at any byte, or where all
  // ranges run at once and their warps are too few to cover the loads
  const bool sq_rows16 = a.code_bytes % 16 == 0 && (uintptr_t)L.codes % 16 == 0;
  auto kern = !stage_rows                                          ? ivf_scan_kernel<IVF_SQ8, 0, 1>
              : sq_rows16 && (uint64_t)L.nq * G > 3ull * sms ? ivf_scan_kernel<IVF_SQ8, 1, 2>
                                                             : ivf_scan_kernel<IVF_SQ8, 2, 2>;
  if (mode == IVF_RABITQ) {
    // bits rows of P/8 bytes as 16-byte words when they and the meta rows
    // are 16-byte aligned; R postings per thread per round as registers allow
    const bool al = ((uintptr_t)L.rq_bits % 16u) == 0 && ((uintptr_t)L.rq_meta % 16u) == 0;
    kern = ivf_scan_kernel<IVF_RABITQ, 0, 1>;
    if (al && P == 128) kern = ivf_scan_kernel<IVF_RABITQ, 1, 4>;
    if (al && P == 256) kern = ivf_scan_kernel<IVF_RABITQ, 2, 2>;
    if (al && P == 512) kern = ivf_scan_kernel<IVF_RABITQ, 4, 2>;
    if (al && P == 1024) kern = ivf_scan_kernel<IVF_RABITQ, 8, 1>;
  }
  if (mode == IVF_PQ) {
    kern = ivf_scan_kernel<IVF_PQ, 0, 1>;
    if (rows16 && L.m_pq == 16) kern = ivf_scan_kernel<IVF_PQ, 1, 4>;
    if (rows16 && L.m_pq == 32) kern = ivf_scan_kernel<IVF_PQ, 2, 4>;
    if (rows16 && L.m_pq == 64) kern = ivf_scan_kernel<IVF_PQ, 4, 2>;
  }
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, IVF_THREADS, smem);
  const uint32_t slots = (uint32_t)(std::max(1, per_sm) * sms);
  const uint32_t grid = std::max(1u, (uint32_t)std::min<uint64_t>((uint64_t)L.nq * G, slots));
  if ((uint64_t)L.nq * G > slots && coarse_bytes >= (size_t)L.nq * 8 && L.nq < (1u << 26)) {
    // (the coarse probe's part of the scratch is free by now)
    uint32_t* place = reinterpret_cast<uint32_t*>(scratch);
    uint32_t* order = place + L.nq;
    ivf_order_count_kernel<<<(L.nq + 7) / 8, 256, 0, stream>>>(a, work + 1, place);
    ivf_order_kernel<<<(L.nq + 255) / 256, 256, 0, stream>>>(L.nq, work + 1, place, order);
    note_launch(2);
    a.order = order;
  }
  {
    ProfScope ps(mode == IVF_PQ ? "ivf_pq_scan" : mode == IVF_SQ8 ? "ivf_sq8_scan" : "ivf_rabitq_scan", stream);
    kern<<<grid, IVF_THREADS, smem, stream>>>(a);
    note_launch();
  }
  if (G > 1) {
    const size_t msmem = (size_t)next_pow2(G * shortlist) * 8;
    auto merge = L.nq <= 2 * sms ? ivf_merge_kernel<1024> : ivf_merge_kernel<256>;
    e = cudaFuncSetAttribute(merge, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)msmem);
    if (e != cudaSuccess) return (int)e;
    ProfScope ps("ivf_merge", stream);
    merge<<<L.nq, L.nq <= 2 * sms ? 1024 : 256, msmem, stream>>>(a);
    note_launch();
  }
  return (int)cudaGetLastError();
}

int launch_relayout_codes(const uint8_t* by_id, const uint32_t* vec_ids, uint32_t n, uint32_t row_bytes,
                          uint8_t* by_list, cudaStream_t stream) {
  if (n == 0 || row_bytes == 0) return 0;
  const uint64_t total = (uint64_t)n * row_bytes;
  const uint32_t blocks = (uint32_t)std::min<uint64_t>((total + 255) / 256, 65535ull * 16);
  relayout_codes_kernel<<<blocks, 256, 0, stream>>>(by_id, vec_ids, n, row_bytes, by_list);
  note_launch();
  return (int)cudaGetLastError();
}

}  // namespace fv

extern "C" int fv_tune_lookup_ivf(int mode, uint32_t dim, uint64_t num_vectors, uint32_t nlist, uint32_t num_queries,
                                  uint32_t nprobe, int32_t* out_knobs) {
  if (!out_knobs) return FV_ERR_NULL;
  return fv::ivf_tune_query(mode, dim, num_vectors, nlist, num_queries, nprobe, out_knobs);
}
