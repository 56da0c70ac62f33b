// topk.cuh -- selection / sorting building blocks on 64-bit (distance,
// slot) keys (see common.cuh for the key encoding).
#pragma once

#include "common.cuh"

namespace fv {

// ---------------------------------------------------------------------------
// Bitonic sort of shared-memory keys. Strides below 128 never touch shared
// memory: a warp holds 128 consecutive keys in registers (four a lane) and
// exchanges them by shuffles, so a block barrier is paid only for the strides
// of 128 and above, two of which share a pass. 2,048 keys take 11 barriers
// instead of 66 (one per stride).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void key_order(uint64_t& lo, uint64_t& hi, bool up) {
  if ((lo > hi) == up) {
    const uint64_t t = lo;
    lo = hi;
    hi = t;
  }
}

// Element e of a lane is key 64 (e >> 1) + 2 lane + (e & 1) of the warp's 128
// (16-byte shared accesses without bank conflicts). One compare-exchange step
// of stride STRIDE; up0 / up1: the direction of elements 0, 1 / 2, 3.
template <int STRIDE>
__device__ __forceinline__ void warp128_step(uint64_t (&k)[4], bool up0, bool up1) {
  if constexpr (STRIDE == 64) {
    key_order(k[0], k[2], up0);
    key_order(k[1], k[3], up1);
  } else if constexpr (STRIDE == 1) {
    key_order(k[0], k[1], up0);
    key_order(k[2], k[3], up1);
  } else {
    const bool lower = (threadIdx.x & (STRIDE / 2)) == 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const uint64_t o = __shfl_xor_sync(0xffffffffu, k[e], STRIDE / 2);
      const bool keep_min = lower == (e < 2 ? up0 : up1);
      if ((o < k[e]) == keep_min) k[e] = o;
    }
  }
}
template <int STRIDE>
__device__ __forceinline__ void warp128_merge(uint64_t (&k)[4], bool up0, bool up1) {
  warp128_step<STRIDE>(k, up0, up1);
  if constexpr (STRIDE > 1) warp128_merge<STRIDE / 2>(k, up0, up1);
}
// Sorts the warp's 128 keys, ascending or descending.
__device__ __forceinline__ void warp128_sort(uint64_t (&k)[4], bool up) {
  const uint32_t lane = threadIdx.x & 31u;
  bool d = (lane & 1u) == 0;
  warp128_merge<1>(k, d, d);
  d = (lane & 2u) == 0;
  warp128_merge<2>(k, d, d);
  d = (lane & 4u) == 0;
  warp128_merge<4>(k, d, d);
  d = (lane & 8u) == 0;
  warp128_merge<8>(k, d, d);
  d = (lane & 16u) == 0;
  warp128_merge<16>(k, d, d);
  warp128_merge<32>(k, true, false);
  warp128_merge<64>(k, up, up);
}
__device__ __forceinline__ void warp128_load(uint64_t (&k)[4], const uint64_t* chunk) {
  const int lane = threadIdx.x & 31;
  const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(chunk + 2 * lane);
  const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(chunk + 64 + 2 * lane);
  k[0] = a.x;
  k[1] = a.y;
  k[2] = b.x;
  k[3] = b.y;
}
__device__ __forceinline__ void warp128_store(uint64_t* chunk, const uint64_t (&k)[4]) {
  const int lane = threadIdx.x & 31;
  *reinterpret_cast<ulonglong2*>(chunk + 2 * lane) = make_ulonglong2(k[0], k[1]);
  *reinterpret_cast<ulonglong2*>(chunk + 64 + 2 * lane) = make_ulonglong2(k[2], k[3]);
}

// Ascending sort of n (power of two) keys in shared memory by all threads of
// the block (whole warps); keys 16-byte aligned; returns after a block barrier.
__device__ __forceinline__ void block_bitonic_sort(uint64_t* keys, uint32_t n) {
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, nwarps = blockDim.x >> 5;
  uint64_t k[4];
  if (n < 128) {
    // one warp, the missing keys as sentinels (which sort last)
    if (warp == 0 && n > 1) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t i = 64u * (e >> 1) + 2 * lane + (e & 1);
        k[e] = i < n ? keys[i] : kSentinelKey;
      }
      warp128_sort(k, true);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t i = 64u * (e >> 1) + 2 * lane + (e & 1);
        if (i < n) keys[i] = k[e];
      }
    }
    __syncthreads();
    return;
  }
  const uint32_t chunks = n / 128;
  for (uint32_t c = warp; c < chunks; c += nwarps) {
    warp128_load(k, keys + c * 128);
    warp128_sort(k, (c & 1u) == 0);
    warp128_store(keys + c * 128, k);
  }
  __syncthreads();
  for (uint32_t size = 256; size <= n; size <<= 1) {
    uint32_t stride = size >> 1;
    for (; stride >= 256; stride >>= 2) {
      // strides `stride` and `stride / 2` on the four keys i + {0, 1, 2, 3} h
      const uint32_t h = stride >> 1;
      for (uint32_t p = threadIdx.x; p < n / 4; p += blockDim.x) {
        const uint32_t i = 4 * p - 3 * (p & (h - 1));  // (p / h) * 4 h + p % h
        const bool up = (i & size) == 0;
        uint64_t a = keys[i], b = keys[i + h], c = keys[i + 2 * h], d = keys[i + 3 * h];
        key_order(a, c, up);
        key_order(b, d, up);
        key_order(a, b, up);
        key_order(c, d, up);
        keys[i] = a;
        keys[i + h] = b;
        keys[i + 2 * h] = c;
        keys[i + 3 * h] = d;
      }
      __syncthreads();
    }
    if (stride == 128) {
      for (uint32_t p = threadIdx.x; p < n / 2; p += blockDim.x) {
        const uint32_t i = 2 * p - (p & 127u);
        uint64_t a = keys[i], b = keys[i + 128];
        key_order(a, b, (i & size) == 0);
        keys[i] = a;
        keys[i + 128] = b;
      }
      __syncthreads();
    }
    for (uint32_t c = warp; c < chunks; c += nwarps) {
      const bool up = ((c * 128) & size) == 0;
      warp128_load(k, keys + c * 128);
      warp128_merge<64>(k, up, up);
      warp128_store(keys + c * 128, k);
    }
    __syncthreads();
  }
}

// Gathers the keys src[0, total) that are <= limit (kSentinelKey - 1: every
// key that is not the sentinel) into keys (in no particular order) and
// returns their number; those past `cap` are counted but not stored.
// Block-collective (warp ballots and one shared counter, a word that the
// caller owns).
__device__ __forceinline__ uint32_t block_compact_keys(const uint64_t* __restrict__ src, uint32_t total,
                                                       uint64_t* keys, uint32_t* counter, uint32_t cap,
                                                       uint64_t limit = kSentinelKey - 1) {
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) *counter = 0;
  __syncthreads();
  // eight loads in flight per thread before any of them is compacted
  constexpr int B = 8;
  for (uint32_t i0 = 0; i0 < total; i0 += blockDim.x * B) {
    uint64_t kb[B];
#pragma unroll
    for (int b = 0; b < B; ++b) {
      const uint32_t i = i0 + (uint32_t)b * blockDim.x + threadIdx.x;
      kb[b] = i < total ? src[i] : kSentinelKey;
    }
#pragma unroll
    for (int b = 0; b < B; ++b) {
      const bool keep = kb[b] <= limit;
      const uint32_t m = __ballot_sync(0xffffffffu, keep);
      uint32_t base = 0;
      if (lane == 0 && m) base = atomicAdd(counter, (uint32_t)__popc(m));
      base = __shfl_sync(0xffffffffu, base, 0);
      const uint32_t at = base + __popc(m & ((1u << lane) - 1u));
      if (keep && at < cap) keys[at] = kb[b];
    }
  }
  __syncthreads();
  return *counter;
}

// The k-th smallest of the keys src[0, total) (distinct apart from
// sentinels, at least k of them not sentinels), built from the top bit by
// counting: no storage, 64 passes over src. Block-collective.
__device__ __forceinline__ uint64_t block_kth_key(const uint64_t* __restrict__ src, uint32_t total, uint32_t k) {
  uint64_t ans = 0;
  __shared__ uint32_t s_count;
  for (int bit = 63; bit >= 0; --bit) {
    const uint64_t test = ans | ((1ull << bit) - 1ull);
    if (threadIdx.x == 0) s_count = 0;
    __syncthreads();
    uint32_t c = 0;
    for (uint32_t i = threadIdx.x; i < total; i += blockDim.x) c += __ldcg(src + i) <= test;
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(&s_count, c);
    __syncthreads();
    if (s_count < k) ans |= 1ull << bit;
    __syncthreads();
  }
  return ans;
}

// Keeps the k smallest of the keys[0, total) in shared memory: packed to the
// front in no particular order, sentinels behind them up to k; returns a key
// that is >= all kept and that no dropped key is below (the sentinel when
// fewer than k keys are not sentinels). total <= NT * NV, k <= total. The k-th
// key is found by counting into 256 equal bins of the keys' range and again
// inside the bin that holds it, until a bin's border separates exactly k keys:
// two rounds of a few barriers as a rule, a tenth of the instructions of
// sorting 2,048 keys. Block-collective (NT threads); returns after a barrier.
struct KeepScratch {
  uint64_t lo[32], hi[32];
  uint32_t hist[256], real[32];
  uint32_t bin, below, in, kept, equal;
};
template <int NT, int NV>
__device__ __forceinline__ uint64_t block_keep_smallest(uint64_t* keys, uint32_t total, uint32_t k, KeepScratch& sc) {
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  uint64_t kv[NV], lo = kSentinelKey, hi = 0;
  uint32_t real = 0;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const uint32_t e = (uint32_t)i * NT + tid;
    kv[i] = e < total ? keys[e] : kSentinelKey;
    if (kv[i] != kSentinelKey) {
      lo = lo < kv[i] ? lo : kv[i];
      hi = hi > kv[i] ? hi : kv[i];
      ++real;
    }
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const uint64_t a = __shfl_xor_sync(0xffffffffu, lo, o), b = __shfl_xor_sync(0xffffffffu, hi, o);
    lo = lo < a ? lo : a;
    hi = hi > b ? hi : b;
  }
  real = __reduce_add_sync(0xffffffffu, real);
  if (lane == 0) {
    sc.lo[warp] = lo;
    sc.hi[warp] = hi;
    sc.real[warp] = real;
  }
  if (tid == 0) sc.kept = sc.equal = 0;
  __syncthreads();
  real = 0;
#pragma unroll
  for (int w = 0; w < NT / 32; ++w) {
    lo = lo < sc.lo[w] ? lo : sc.lo[w];
    hi = hi > sc.hi[w] ? hi : sc.hi[w];
    real += sc.real[w];
  }
  uint64_t last = hi;                // keys up to here are kept,
  uint32_t equal = 0xFFFFFFFFu;      // of those equal to it this many
  if (real > k) {
    uint64_t span = hi - lo;  // the k-th key lies in [lo, lo + span]
    uint32_t need = k;        // its rank there
    while (true) {
      const int shift = span < 256 ? 0 : 56 - __clzll((long long)span);
      for (uint32_t b = tid; b < 256; b += NT) sc.hist[b] = 0;
      __syncthreads();
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const uint64_t off = kv[i] - lo;
        if (kv[i] >= lo && off <= span) atomicAdd(&sc.hist[(uint32_t)(off >> shift)], 1u);
      }
      __syncthreads();
      if (warp == 0) {
        uint32_t own = 0;
#pragma unroll
        for (int b = 0; b < 8; ++b) own += sc.hist[8 * lane + b];
        uint32_t upto = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(0xffffffffu, upto, o);
          if (lane >= (uint32_t)o) upto += y;
        }
        uint32_t below = upto - own;
        if (below < need && upto >= need) {  // one lane: the bin is among its eight
          uint32_t b = 0;
          while (below + sc.hist[8 * lane + b] < need) below += sc.hist[8 * lane + b++];
          sc.bin = 8 * lane + b;
          sc.below = below;
          sc.in = sc.hist[8 * lane + b];
        }
      }
      __syncthreads();
      const uint64_t first = lo + ((uint64_t)sc.bin << shift);
      const uint64_t width = (1ull << shift) - 1;
      need -= sc.below;
      if (need == sc.in || shift == 0) {
        last = first + width;  // exactly the k smallest are up to here, or
        if (need != sc.in) equal = need;  // with need of the keys that equal it
        break;
      }
      lo = first;
      span = width;
      __syncthreads();  // the bins are cleared again
    }
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    bool keep = kv[i] <= last && kv[i] != kSentinelKey;
    if (keep && kv[i] == last && equal != 0xFFFFFFFFu) keep = atomicAdd(&sc.equal, 1u) < equal;
    const uint32_t m = __ballot_sync(0xffffffffu, keep);
    uint32_t base = 0;
    if (lane == 0 && m) base = atomicAdd(&sc.kept, (uint32_t)__popc(m));
    base = __shfl_sync(0xffffffffu, base, 0) + __popc(m & ((1u << lane) - 1u));
    if (keep) keys[base] = kv[i];
  }
  __syncthreads();
  for (uint32_t i = sc.kept + tid; i < k; i += NT) keys[i] = kSentinelKey;
  __syncthreads();
  return real < k ? kSentinelKey : last;
}

// Ascending bitonic sort of 32 keys held one per lane.
__device__ __forceinline__ uint64_t warp_bitonic_sort32(uint64_t key) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      uint64_t other = __shfl_xor_sync(0xffffffffu, key, stride);
      bool up = (lane & size) == 0;
      bool lower = (lane & stride) == 0;
      // the lower lane of a pair keeps min when sorting up, max otherwise
      bool keep_min = (lower == up);
      key = keep_min ? (key < other ? key : other) : (key < other ? other : key);
    }
  }
  return key;
}

}  // namespace fv
