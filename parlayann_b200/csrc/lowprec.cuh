// Low-precision copies of float32 points and their approximate distances
// (the precision form of the search).
//
//   BF16: each value rounded to nearest-even bfloat16; 2 bytes per value.
//   FP8 : E4M3 with one scale per dimension, s_t = max_i |x_it| / 448 (the
//         largest finite E4M3 value); stored value = E4M3(x_it / s_t); 1 byte.
//
// Approximate distances dequantize to float32 and accumulate in float32 with
// fused multiply-adds in any order: they only steer the traversal. The
// search re-ranks its best candidates with the exact float32 distance (the
// reference's sequential sum, common.cuh) before reporting.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include "common.cuh"

namespace pann {

enum Precision { PREC_F32 = 0, PREC_BF16 = 1, PREC_FP8 = 2 };

// bf16 pair (packed in a uint32) -> two floats, exactly
__device__ __forceinline__ float2 bf16x2_to_f2(uint32_t v) {
  return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xFFFF0000u));
}
// e4m3 pair (low 16 bits of v) -> two floats, exactly
__device__ __forceinline__ float2 e4m3x2_to_f2(uint32_t v) {
  __half2_raw h = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(v & 0xFFFFu), __NV_E4M3);
  return __half22float2(*reinterpret_cast<__half2*>(&h));
}

// Adds chunk c (16 bytes) of a low-precision row to the two partial sums of its approximate distance to the query
// staged in shared memory as float32 (negated for L2, as the exact path stores it). FP8 values are dequantized with
// the per-dimension scales.
template <int MT, int PREC>
__device__ __forceinline__ void lp_chunk(const uint4& v, int c, const float* qs, const float* __restrict__ scales, int d,
                                         float& a0, float& a1) {
  constexpr int VPC = PREC == PREC_BF16 ? 8 : 16;  // values per chunk
  const uint32_t wa[4] = {v.x, v.y, v.z, v.w};
  const int e0 = c * VPC;
#pragma unroll
  for (int w = 0; w < 4; w++) {
#pragma unroll
    for (int h = 0; h < (PREC == PREC_BF16 ? 1 : 2); h++) {
      const int e = e0 + w * (VPC / 4) + 2 * h;
      if (e >= d) break;
      float2 x;
      if (PREC == PREC_BF16) {
        x = bf16x2_to_f2(wa[w]);
      } else {
        x = e4m3x2_to_f2(wa[w] >> (16 * h));
        x.x *= scales[e]; x.y *= scales[e + 1];
      }
      const float q0 = qs[e], q1 = qs[e + 1];
      if (MT == MT_L2) {
        float t;
        t = x.x + q0; a0 = fmaf(t, t, a0);
        t = x.y + q1; a1 = fmaf(t, t, a1);
      } else {
        a0 = fmaf(q0, x.x, a0); a1 = fmaf(q1, x.y, a1);
      }
    }
  }
}

// Approximate distance of one low-precision row, eight chunks of it in flight.
template <int MT, int PREC>
__device__ __forceinline__ float lp_dist(const uint8_t* __restrict__ row, const float* qs, const float* scales, int d,
                                         int lp_chunks) {
  const uint4* ra = reinterpret_cast<const uint4*>(row);
  float a0 = 0.0f, a1 = 0.0f;
  for (int c0 = 0; c0 < lp_chunks; c0 += 8) {
    uint4 b[8];
#pragma unroll
    for (int c = 0; c < 8; c++)
      if (c0 + c < lp_chunks) b[c] = __ldg(ra + c0 + c);
#pragma unroll
    for (int c = 0; c < 8; c++)
      if (c0 + c < lp_chunks) lp_chunk<MT, PREC>(b[c], c0 + c, qs, scales, d, a0, a1);
  }
  return MT == MT_L2 ? a0 + a1 : -(a0 + a1);
}

}  // namespace pann
