// encode.cu -- device-side encoders of the reduced-precision flat tables.
//
//  * fp16: the reference's host encoder encode_fp16_padded / f32_to_f16_bits
//    (crates/engine/src/quant.rs:239-274, 306-327) restated for the GPU:
//    mantissa rounded half-up (not round-to-even), subnormals truncated,
//    rows zero-padded to padded_dim, ||x||^2 as the sequential fp32 sum of
//    the squares (separately rounded multiply and add, as Rust evaluates).
//  * fp8 (no reference counterpart): one power-of-two scale s = 2^b for the
//    whole table, the smallest with max_v ||x_v||^2 <= 896 s^2 (so every
//    code is below 30 in magnitude, far inside e4m3's range: the relative
//    precision of a normal e4m3 code does not depend on the scale, so this
//    equals per-row power-of-two scaling for every code that stays normal);
//    codes = e4m3(x / s) round-to-nearest-even; columns dim, dim + 1,
//    dim + 2 hold three e4m3 "norm digits" n1 + n2 + n3 ~ ||x||^2 / (2 s^2)
//    (each the round-to-nearest-even e4m3 value of what the previous ones
//    left, residual <= 2^-12 relative), so that a query row carrying
//    -s / s_q in those columns makes the tensor-core dot product equal
//    <q, x> / (s s_q) - ||x||^2 / (2 s s_q) -- the L2 ranking value up to
//    the per-query factor -2 s s_q and the query's norm; remaining columns
//    zero; ||x||^2 by compensated (Neumaier) fp32 summation; every entry of
//    the scale array holds s.
//  * fp8, per-row scales (the other layout, selected by the table's
//    scale_mode): s_v = max|x_v| / 448, codes e4m3(x / s_v), no digits.
#include <cuda_fp8.h>

#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace fv {

namespace {

__device__ __forceinline__ uint16_t f32_to_f16_halfup(float x) {
  const uint32_t bits = __float_as_uint(x);
  const uint16_t sign = (uint16_t)((bits >> 16) & 0x8000u);
  const int32_t exp = (int32_t)((bits >> 23) & 0xffu);
  const uint32_t mant = bits & 0x007fffffu;
  if (exp == 255) return (uint16_t)(sign | (mant == 0 ? 0x7c00u : 0x7e00u));
  const int32_t e = exp - 127 + 15;
  if (e >= 31) return (uint16_t)(sign | 0x7c00u);
  if (e <= 0) {
    if (e < -10) return sign;
    return (uint16_t)(sign | (uint16_t)((mant | 0x00800000u) >> (14 - e)));
  }
  const uint32_t r = mant + 0x1000u;
  if (r & 0x00800000u) return (uint16_t)(e + 1 >= 31 ? (sign | 0x7c00u) : (sign | (uint16_t)((e + 1) << 10)));
  return (uint16_t)(sign | (uint16_t)(e << 10) | (uint16_t)(r >> 13));
}

// Four values at once: magnitudes in [2^-14, 65504 + rounding) share one
// exponent shift, and a mantissa that rounds over carries into the exponent
// (up to infinity) by itself; anything else takes the general conversion.
__device__ __forceinline__ uint32_t f32_to_f16_normal(uint32_t b, bool& normal) {
  const uint32_t a = (b & 0x7fffffffu) - 0x38800000u;  // 113 << 23: the exponent of 2^-14
  normal = normal && a < 0x0f000000u;                  // below 143 << 23: the exponent of 2^16
  return ((a + 0x00801000u) >> 13) | ((b >> 16) & 0x8000u);
}
__device__ __forceinline__ uint2 f32_to_f16_halfup4(float4 v) {
  bool normal = true;
  uint32_t h[4] = {f32_to_f16_normal(__float_as_uint(v.x), normal), f32_to_f16_normal(__float_as_uint(v.y), normal),
                   f32_to_f16_normal(__float_as_uint(v.z), normal), f32_to_f16_normal(__float_as_uint(v.w), normal)};
  if (!normal) {
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
      const float f = i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w;
      const uint32_t c = f32_to_f16_halfup(f);
      h[0] = i == 0 ? c : h[0];
      h[1] = i == 1 ? c : h[1];
      h[2] = i == 2 ? c : h[2];
      h[3] = i == 3 ? c : h[3];
    }
  }
  return make_uint2(h[0] | (h[1] << 16), h[2] | (h[3] << 16));
}
__device__ __forceinline__ uint16_t f32_to_f16_halfup_fast(float v) {
  bool normal = true;
  const uint32_t h = f32_to_f16_normal(__float_as_uint(v), normal);
  return normal ? (uint16_t)h : f32_to_f16_halfup(v);
}

// A warp encodes 8 rows, 128 dimensions at a time: the chunk is read with
// whole-row segments (16-byte loads where VEC), converted and stored, and its
// squares are transposed through shared memory so that lane r adds row r's
// squares in dimension order. The next chunk's loads are in flight meanwhile.
// ||x||^2 is a sequential fp32 sum, so the transposition is what lets rows
// advance together: with one lane per row reading its row alone, 500,000 x 768
// took 2,221 us. Eight rows a warp rather than 32 keep small tables in enough
// warps (10,357 x 633: 37 us at the start, 172 us with 32 rows a warp).
constexpr int E16_WARPS = 8, E16_DIMS = 128;
template <bool VEC, int E16_ROWS>
__global__ void __launch_bounds__(32 * E16_WARPS, 3) encode_fp16_kernel(const float* __restrict__ x, uint32_t n,
                                                                        uint32_t dim, uint32_t pd,
                                                                        uint16_t* __restrict__ out,
                                                                        float* __restrict__ norms) {
  // (a stride of 132 floats: 16-byte stores, and the eight summing lanes on
  // different banks)
  __shared__ __align__(16) float sq[E16_WARPS][E16_ROWS][E16_DIMS + 4];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint64_t row0 = ((uint64_t)blockIdx.x * E16_WARPS + warp) * E16_ROWS;
  if (row0 >= n) return;
  const int rows = (int)min((uint64_t)E16_ROWS, n - row0);
  float(*t)[E16_DIMS + 4] = sq[warp];
  const float* src = x + row0 * dim;
  uint16_t* dst = out + row0 * pd;
  float sum = 0.f;
  constexpr int NV = VEC ? 1 : 4;  // loads per row of a chunk: a float4, or four floats 32 apart
  using V = typename std::conditional<VEC, float4, float>::type;
  V cur[E16_ROWS][NV];
  auto load = [&](uint32_t d0) {
#pragma unroll
    for (int r = 0; r < E16_ROWS; ++r) {
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const uint32_t d = d0 + (VEC ? 4 * lane : lane + 32 * i);
        if constexpr (VEC)
          cur[r][i] = r < rows && d < dim ? __ldg(reinterpret_cast<const float4*>(src + (size_t)r * dim + d))
                                          : make_float4(0.f, 0.f, 0.f, 0.f);
        else
          cur[r][i] = r < rows && d < dim ? __ldg(src + (size_t)r * dim + d) : 0.f;
      }
    }
  };
  load(0);
  for (uint32_t d0 = 0; d0 < pd; d0 += E16_DIMS) {
    __syncwarp();  // the previous chunk is summed
#pragma unroll
    for (int r = 0; r < E16_ROWS; ++r) {
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const uint32_t c = VEC ? 4 * lane : lane + 32 * i;
        const V v = cur[r][i];
        if constexpr (VEC) {
          *reinterpret_cast<float4*>(&t[r][c]) =
              make_float4(__fmul_rn(v.x, v.x), __fmul_rn(v.y, v.y), __fmul_rn(v.z, v.z), __fmul_rn(v.w, v.w));
          // dim is a multiple of 4: four columns in or out together
          if (r < rows && d0 + c < pd)
            *reinterpret_cast<uint2*>(dst + (size_t)r * pd + d0 + c) =
                d0 + c < dim ? f32_to_f16_halfup4(v) : make_uint2(0u, 0u);
        } else {
          t[r][c] = __fmul_rn(v, v);
          if (r < rows && d0 + c < pd)
            dst[(size_t)r * pd + d0 + c] = d0 + c < dim ? f32_to_f16_halfup_fast(v) : (uint16_t)0;
        }
      }
    }
    if (d0 + E16_DIMS < dim) load(d0 + E16_DIMS);
    __syncwarp();
    if (lane < E16_ROWS) {
      const int m = d0 < dim ? (int)min((uint32_t)E16_DIMS, dim - d0) : 0;
      int j = 0;
      for (; j + 16 <= m; j += 16) {
        float4 w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = *reinterpret_cast<const float4*>(&t[lane][j + 4 * i]);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, w[i].x), w[i].y), w[i].z), w[i].w);
      }
      for (; j < m; ++j) sum = __fadd_rn(sum, t[lane][j]);
    }
  }
  if (norms && lane < rows) norms[row0 + lane] = sum;
}

// Neumaier accumulation of one term.
__device__ __forceinline__ void neumaier_add(float& sum, float& comp, float v) {
  const float t = sum + v;
  if (fabsf(sum) >= fabsf(v))
    comp += (sum - t) + v;
  else
    comp += (v - t) + sum;
  sum = t;
}

// smallest b in [-62, 62] with mx <= 896 * 4^b (0 for an all-zero table)
__device__ __forceinline__ int fp8_table_exponent(float mx) {
  if (!(mx > 0.f)) return 0;
  int b = max(-62, min(62, (ilogbf(mx) - 9) / 2));
  while (b < 62 && ldexpf(896.0f, 2 * b) < mx) ++b;
  while (b > -62 && ldexpf(896.0f, 2 * (b - 1)) >= mx) --b;
  return b;
}

// One step of the butterfly over the lanes' compensated sums, for rows r and
// r + H at once: the lower half of each 2o lanes goes on with row r, the upper
// half with row r + H. A row's left operand is the lower lane's, as in a
// butterfly of one row read at lane 0.
template <int H>
__device__ __forceinline__ void neumaier_halve(float* sum, float* comp, int o, int lane) {
  const bool up = (lane & o) != 0;
#pragma unroll
  for (int r = 0; r < H; ++r) {
    const float os = __shfl_xor_sync(0xffffffffu, up ? sum[r] : sum[r + H], o);
    const float oc = __shfl_xor_sync(0xffffffffu, up ? comp[r] : comp[r + H], o);
    float a = up ? os : sum[r], c = up ? oc : comp[r];
    neumaier_add(a, c, up ? sum[r + H] : os);
    c += up ? comp[r + H] : oc;
    sum[r] = a;
    comp[r] = c;
  }
}

// ||x||^2 of each row (compensated), and the largest of them as ordered
// bits in *max_bits (norms are >= 0, so the bit patterns order like the values).
// Bound by the read of the table: a warp takes R = 8 rows at a time (eight
// loads in flight, and three of the five steps across the lanes shared by all
// eight) and raises the maximum once for all its rows: 47 us for 328,756 x 157.
// With a row and an atomic on one word per warp the whole encoder took 307 us
// there and takes 120 (500,000 x 768: 972 and 612 us; two reads and the write
// at the measured copy rate: 510). Tables of fewer and longer rows, whose warps
// of eight rows would not fill the GPU, take two rows or one a warp and as many
// loads in flight.
template <int R>
__global__ void __launch_bounds__(256) fp8_norms_kernel(const float* __restrict__ x, uint32_t n, uint32_t dim,
                                                        float* __restrict__ norms, uint32_t* __restrict__ max_bits) {
  constexpr int B = 8 / R, LPR = 32 / R;  // loads of a row in flight; lanes that end with a row
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  const int lane = threadIdx.x & 31;
  uint32_t top = 0;
  for (uint64_t row0 = (uint64_t)(((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * R; row0 < n;
       row0 += (uint64_t)warps * R) {
    float sum[R], comp[R];
    const float* src[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      sum[r] = comp[r] = 0.f;
      src[r] = x + min(row0 + r, (uint64_t)n - 1) * dim;
    }
    // (the next 32 B dimensions of every row are in flight while these are added)
    auto load = [&](float (&v)[R][B], uint32_t d) {
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int b = 0; b < B; ++b) v[r][b] = d + 32 * b < dim ? __ldg(src[r] + d + 32 * b) : 0.f;
    };
    float v[R][B];
    load(v, lane);
    for (uint32_t d = lane; d < dim; d += 32 * B) {
      float w[R][B];
      load(w, d + 32 * B);
#pragma unroll
      for (int b = 0; b < B; ++b) {
        if (b && d + 32 * b >= dim) break;
#pragma unroll
        for (int r = 0; r < R; ++r) neumaier_add(sum[r], comp[r], __fmul_rn(v[r][b], v[r][b]));
      }
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int b = 0; b < B; ++b) v[r][b] = w[r][b];
    }
    __syncwarp();
    if constexpr (R == 8) {
      neumaier_halve<4>(sum, comp, 16, lane);
      neumaier_halve<2>(sum, comp, 8, lane);
      neumaier_halve<1>(sum, comp, 4, lane);
    } else {
      static_assert(R <= 2, "eight rows, two or one");
      if constexpr (R == 2) neumaier_halve<1>(sum, comp, 16, lane);
    }
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) {
      const float os = __shfl_xor_sync(0xffffffffu, sum[0], o);
      const float oc = __shfl_xor_sync(0xffffffffu, comp[0], o);
      neumaier_add(sum[0], comp[0], os);
      comp[0] += oc;
    }
    // row r's sum is lane LPR r's
    const uint64_t row = row0 + lane / LPR;
    if (lane % LPR == 0 && row < n) {
      const float nrm = sum[0] + comp[0];
      norms[row] = nrm;
      if (nrm > 0.f) top = max(top, __float_as_uint(nrm));
    }
  }
  top = __reduce_max_sync(0xffffffffu, top);
  if (lane == 0 && top) atomicMax(max_bits, top);
}

// The table's scale exponent b from the largest norm (written over the
// same word, which from here on holds the scale 2^b as a float).
__global__ void fp8_table_scale_kernel(uint32_t* __restrict__ word) {
  const float mx = __uint_as_float(*word);
  *word = __float_as_uint(ldexpf(1.0f, fp8_table_exponent(mx)));
}

// e4m3 code of v (round to nearest even, saturating) and its value.
__device__ __forceinline__ uint8_t e4m3_code(float v) {
  return (uint8_t)__nv_cvt_float_to_fp8(v, __NV_SATFINITE, __NV_E4M3);
}
__device__ __forceinline__ float e4m3_value(uint8_t c) {
  const uint32_t e = (c >> 3) & 15u, m = c & 7u;
  const float mag = e ? ldexpf((float)(8u + m), (int)e - 10) : ldexpf((float)m, -9);
  return (c & 0x80u) ? -mag : mag;
}

// A warp encodes its rows (as many as in the norms' pass) as one run of 4-byte
// words (rows are stored one after the other), so that no lane is idle at any
// width; lane r makes row r's norm digits. Bound by the read of the rows: the
// grid goes from the last row to the first, as the norms' pass has just left
// the last ones in L2 (66 us for 328,756 x 157).
template <bool VEC, int F8_ROWS>
__global__ void __launch_bounds__(256) encode_fp8_kernel(const float* __restrict__ x, uint32_t n, uint32_t dim,
                                                         uint32_t pd, uint8_t* __restrict__ out,
                                                         float* __restrict__ scales,
                                                         const float* __restrict__ norms) {
  const uint64_t groups = ((uint64_t)n + F8_ROWS - 1) / F8_ROWS;
  const uint64_t g = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (g >= groups) return;
  const uint64_t row0 = (groups - 1 - g) * F8_ROWS;
  const uint32_t rows = (uint32_t)min((uint64_t)F8_ROWS, n - row0);
  // scales[0] holds the table scale (row 0 rewrites it with the same value)
  const float s = scales[0];
  const int b = ilogbf(s);
  const float inv = ldexpf(1.0f, -b);  // (b in [-62, 62]: the product is what ldexpf gives)
  uint32_t digits = 0;                 // lane r: row r's
  if (lane < (int)rows) {
    float r = ldexpf(norms[row0 + lane], -1 - 2 * b);
    for (int i = 0; i < 3; ++i) {
      const uint8_t c = e4m3_code(r);
      digits |= (uint32_t)c << (8 * i);
      r -= e4m3_value(c);
    }
    scales[row0 + lane] = s;
  }
  const uint32_t wpr = pd / 4, total = rows * wpr;
  const float* src = x + row0 * dim;
  uint8_t* dst = out + row0 * pd;
  const bool words = (uintptr_t)out % 4 == 0;
  constexpr uint32_t U = 4;
  for (uint32_t e0 = 0; e0 < total; e0 += 32 * U) {
    float v[U][4];
    uint32_t r[U], d[U];
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) {
      const uint32_t e = min(e0 + 32 * u + lane, total - 1);
      r[u] = e / wpr;
      d[u] = (e - r[u] * wpr) * 4;
      const float* p = src + (size_t)r[u] * dim + d[u];
      if constexpr (VEC) {
        // dim is a multiple of 4: four columns in or out together
        const float4 w = d[u] < dim ? __ldg(reinterpret_cast<const float4*>(p)) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[u][0] = w.x, v[u][1] = w.y, v[u][2] = w.z, v[u][3] = w.w;
      } else {
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) v[u][i] = d[u] + i < dim ? __ldg(p + i) : 0.f;
      }
    }
#pragma unroll
    for (uint32_t u = 0; u < U; ++u) {
      const uint32_t dg = __shfl_sync(0xffffffffu, digits, r[u]);
      uint32_t w = 0;
#pragma unroll
      for (uint32_t i = 0; i < 4; ++i) {
        // (a column past the row's digits: 0, as a shift by 24 leaves it)
        const uint32_t col = d[u] + i, dgt = (dg >> min(8 * (col - dim), 24u)) & 255u;
        w |= (col < dim ? (uint32_t)e4m3_code(__fmul_rn(v[u][i], inv)) : dgt) << (8 * i);
      }
      if (e0 + 32 * u + lane < total) {
        uint8_t* o = dst + (size_t)r[u] * pd + d[u];
        if (words) {
          *reinterpret_cast<uint32_t*>(o) = w;
        } else {
#pragma unroll
          for (uint32_t i = 0; i < 4; ++i) o[i] = (uint8_t)(w >> (8 * i));
        }
      }
    }
  }
}

// Per-row-scale table (the other fp8 layout): s_v = max|x_v| / 448 (1 for a
// zero row), codes e4m3(x / s_v) round-to-nearest-even with saturation, zero
// padding, ||x||^2 by compensated fp32 summation.
__global__ void __launch_bounds__(256) encode_fp8_per_vector_kernel(const float* __restrict__ x, uint32_t n,
                                                                    uint32_t dim, uint32_t pd, uint8_t* __restrict__ out,
                                                                    float* __restrict__ scales,
                                                                    float* __restrict__ norms) {
  const uint64_t row = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= n) return;
  const float* src = x + row * dim;
  float amax = 0.f, sum = 0.f, comp = 0.f;
  for (uint32_t d = lane; d < dim; d += 32) {
    const float v = __ldg(src + d);
    amax = fmaxf(amax, fabsf(v));
    neumaier_add(sum, comp, __fmul_rn(v, v));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const float os = __shfl_xor_sync(0xffffffffu, sum, o);
    const float oc = __shfl_xor_sync(0xffffffffu, comp, o);
    neumaier_add(sum, comp, os);
    comp += oc;
  }
  const float scale = amax > 0.f ? amax / 448.0f : 1.0f;
  uint8_t* dst = out + row * pd;
  for (uint32_t d = lane; d < pd; d += 32) dst[d] = d < dim ? e4m3_code(__ldg(src + d) / scale) : (uint8_t)0;
  if (lane == 0) {
    scales[row] = scale;
    norms[row] = sum + comp;
  }
}

}  // namespace

int launch_encode_fp16(const float* x, uint32_t n, uint32_t dim, uint32_t pd, uint16_t* out, float* norms,
                       cudaStream_t stream) {
  if (n == 0) return 0;
  // 16-byte loads and 8-byte stores where every row starts on such a boundary
  const bool vec = dim % 4 == 0 && pd % 4 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)out % 8 == 0;
  auto go = [&](auto kern, uint64_t rows) {
    const uint64_t blocks = ((uint64_t)n + rows * E16_WARPS - 1) / (rows * E16_WARPS);
    kern<<<(unsigned)blocks, 32 * E16_WARPS, 0, stream>>>(x, n, dim, pd, out, norms);
  };
  // two rows a warp for a few long ones, whose warps of eight would leave most of
  // the GPU idle (1,000 x 4,096: 63 us with eight, 30 with two; 10,000 x 1,024: 26
  // and 24; 20,000 x 1,536: 45 and 52)
  if (dim >= 512 && n < 64 * (uint32_t)device_sm_count())
    vec ? go(encode_fp16_kernel<true, 2>, 2) : go(encode_fp16_kernel<false, 2>, 2);
  else
    vec ? go(encode_fp16_kernel<true, 8>, 8) : go(encode_fp16_kernel<false, 8>, 8);
  note_launch();
  return (int)cudaGetLastError();
}

int launch_encode_fp8(const float* x, uint32_t n, uint32_t dim, uint32_t pd, uint8_t* out, float* scales,
                      float* norms, cudaStream_t stream) {
  if (n == 0) return 0;
  uint32_t* word = reinterpret_cast<uint32_t*>(scales);
  cudaError_t e = cudaMemsetAsync(word, 0, sizeof(uint32_t), stream);
  if (e != cudaSuccess) return (int)e;
  const bool vec = dim % 4 == 0 && (uintptr_t)x % 16 == 0;
  const uint64_t sms = (uint64_t)device_sm_count();
  auto go = [&](auto norms_kern, auto kern, uint64_t rows) {
    // eight warps a block; the norms' blocks stay and go on to further rows
    const uint64_t blocks = ((uint64_t)n + 8 * rows - 1) / (8 * rows);
    norms_kern<<<(unsigned)(blocks < 8 * sms ? blocks : 8 * sms), 256, 0, stream>>>(x, n, dim, norms, word);
    fp8_table_scale_kernel<<<1, 1, 0, stream>>>(word);
    kern<<<(unsigned)blocks, 256, 0, stream>>>(x, n, dim, pd, out, scales, norms);
  };
  // Eight rows a warp for short rows, which have the fewest steps to share the
  // sums over, and for tables that fill the GPU so (80,000 x 96: 35 us, 46 with
  // two a warp; 160,000 x 384: 125 and 136). Else two (40,000 x 768: 85 and 72 us;
  // 20,000 x 1,536: 91 and 68; 10,000 x 1,024: 44 and 36), and one for a few rows
  // (1,000 x 4,096: 93 us with eight, 36 with two, 29 with one).
  if (dim < 256 || n >= 640 * sms)
    vec ? go(fp8_norms_kernel<8>, encode_fp8_kernel<true, 8>, 8) : go(fp8_norms_kernel<8>, encode_fp8_kernel<false, 8>, 8);
  else if (n >= 32 * sms)
    vec ? go(fp8_norms_kernel<2>, encode_fp8_kernel<true, 2>, 2) : go(fp8_norms_kernel<2>, encode_fp8_kernel<false, 2>, 2);
  else
    vec ? go(fp8_norms_kernel<1>, encode_fp8_kernel<true, 1>, 1) : go(fp8_norms_kernel<1>, encode_fp8_kernel<false, 1>, 1);
  note_launch(3);
  return (int)cudaGetLastError();
}

}  // namespace fv

namespace fv {

int launch_encode_fp8_per_vector(const float* x, uint32_t n, uint32_t dim, uint32_t pd, uint8_t* out, float* scales,
                                 float* norms, cudaStream_t stream) {
  if (n == 0) return 0;
  const uint64_t blocks = ((uint64_t)n * 32 + 255) / 256;
  encode_fp8_per_vector_kernel<<<(unsigned)blocks, 256, 0, stream>>>(x, n, dim, pd, out, scales, norms);
  note_launch();
  return (int)cudaGetLastError();
}

}  // namespace fv
