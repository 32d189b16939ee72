// Pieces shared by the two cluster-block map kernels (the probability map of blockmap.cu and the
// error-aware one of ear.cu): fixed-order fp32 exp, per-head limits, the warp-wide bitonic sort.
#pragma once

#include "common.cuh"

namespace svoo {

__device__ __forceinline__ float exp_f32_fixed(float x) {
  // exp(x), x <= 0, from fp32 mul/add only; mirrored operation by operation on the CPU side
  if (x < -87.0f) return 0.0f;
  const float n = rintf(__fmul_rn(x, (float)1.4426950408889634));
  float r = __fsub_rn(x, __fmul_rn(n, 0.693145751953125f));
  r = __fsub_rn(r, __fmul_rn(n, (float)1.428606765330187e-06));
  float p = (float)(1.0 / 720);
  p = __fadd_rn(__fmul_rn(p, r), (float)(1.0 / 120));
  p = __fadd_rn(__fmul_rn(p, r), (float)(1.0 / 24));
  p = __fadd_rn(__fmul_rn(p, r), (float)(1.0 / 6));
  p = __fadd_rn(__fmul_rn(p, r), 0.5f);
  p = __fadd_rn(__fmul_rn(p, r), 1.0f);
  p = __fadd_rn(__fmul_rn(p, r), 1.0f);
  int ni = (int)n;
  ni = ni < -126 ? -126 : ni;
  return __fmul_rn(p, __int_as_float((ni + 127) << 23));
}

// The `bytes` (at most 32) map bytes at `at` as aligned 32-bit words, first byte at byte `skew` (returned) of w[0]; the
// other bytes of the words hold whatever lies there, or zeros.  [lo, hi) is the whole map: words that reach over its
// start or end are put together from the bytes inside.  Load: how memory is read (the host test records it).
struct MapLoad {
  __host__ __device__ __forceinline__ uint32_t word(const uint8_t* p) const { return *reinterpret_cast<const uint32_t*>(p); }
  __host__ __device__ __forceinline__ uint32_t byte(const uint8_t* p) const { return *p; }
};
template <class Load>
__host__ __device__ __forceinline__ int map_words(uint32_t (&w)[9], const uint8_t* at, int bytes, const uint8_t* lo,
                                                  const uint8_t* hi, const Load& load) {
  const int skew = (int)(reinterpret_cast<uintptr_t>(at) & 3);
  const int n = bytes > 0 ? (skew + bytes + 3) / 4 : 0;
  const uint8_t* first = at - skew;
  if (first >= lo && first + 4 * n <= hi) {
#pragma unroll
    for (int i = 0; i < 9; ++i) w[i] = i < n ? load.word(first + 4 * i) : 0;
  } else {
#pragma unroll 1
    for (int i = 0; i < 9; ++i) w[i] = 0;
#pragma unroll 1
    for (int b = skew; b < skew + bytes; ++b) w[b >> 2] |= load.byte(first + b) << (8 * (b & 3));
  }
  return skew;
}

struct HeadLimits {
  int32_t preserve[SVOO_MAX_HEADS];
  int32_t cap[SVOO_MAX_HEADS];
};

// Bitonic sort (descending) of 32 * M keys held by one warp, element t in register t / 32 of lane
// t % 32: partners at distance >= 32 are other registers of the same lane, closer ones come by
// shuffle.  Keys are unique (the cluster index is part of the key) except for the zero padding.
template <int M, typename Key = uint32_t>
__device__ __forceinline__ void warp_sort_desc(Key (&v)[M], int lane) {
#pragma unroll
  for (int k = 2; k <= 32 * M; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j >= 32) {
#pragma unroll
        for (int m = 0; m < M; ++m) {
          const int pm = m ^ (j >> 5);
          if (pm > m) {
            const bool desc = ((lane + 32 * m) & k) == 0;
            const Key a = v[m], b = v[pm];
            if (desc ? (a < b) : (a > b)) { v[m] = b; v[pm] = a; }
          }
        }
      } else {
#pragma unroll
        for (int m = 0; m < M; ++m) {
          const Key a = v[m];
          const Key b = __shfl_xor_sync(0xffffffffu, a, j);
          const bool lower = (lane & j) == 0;                      // this lane holds the smaller index of the pair
          const bool desc = ((lane + 32 * m) & k) == 0;
          v[m] = (lower == desc) ? max(a, b) : min(a, b);
        }
      }
    }
  }
}

}  // namespace svoo
