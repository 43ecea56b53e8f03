// Distances of up to 32 scattered rows to one staged query, a row per lane.
//
// Reading one row per lane costs the L1 a pass per lane and 16-byte chunk (32
// rows of 384 bytes: 768 passes; tier 0 spent 85 % of its L1 pipe on them).
// Here eight neighbouring lanes read the 128 contiguous bytes of a row, four
// rows a load instruction, so the same rows cost 96 passes.
//   8-bit: each lane multiplies its own chunks (integer sums are exact in any
//          order) and eight partial sums are folded across the eight lanes
//          with 7 shuffles, which leaves each lane one row's distance.
//   float: the sum must run through a row in dimension order, so 32 rows x 128
//          bytes pass through a 4 KB shared buffer per warp (cp.async, no
//          registers held), chunk c of row r at slot c ^ (r % 8): both the
//          8-lane writes and the per-lane reads of a row touch every bank
//          once a quarter warp. Two such column blocks are in flight.
#pragma once
#include "common.cuh"

namespace pann {

// Bytes of shared scratch a warp needs (16-byte aligned).
template <int DT>
__host__ __device__ constexpr uint32_t row_score_scratch() { return DT == DT_F32 ? 8192u : 0u; }
__host__ __device__ inline uint32_t row_score_scratch_rt(int dtype) { return dtype == DT_F32 ? 8192u : 0u; }

__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// Lane l < n returns the distance of row `id` (its own) to the query staged at
// qs (stage_query); n <= 32 rows, held by the first n lanes. Every lane of the
// warp takes part; qs and stg are the warp's own.
template <int DT, int MT>
__device__ __forceinline__ float warp_score_rows(const uint8_t* __restrict__ points, uint64_t stride, int nchunks,
                                                 uint32_t id, int n, const uint8_t* qs, uint8_t* stg, int32_t qq,
                                                 int lane) {
  const unsigned FULL = 0xFFFFFFFFu;
  const int g = lane >> 3, sub = lane & 7;
  uint32_t rid[8];  // the rows this lane reads a part of: 4 j + g
#pragma unroll
  for (int j = 0; j < 8; j++) {
    rid[j] = __shfl_sync(FULL, id, 4 * j + g);
    if (4 * j + g >= n) rid[j] = 0u;
  }
  const uint8_t* const base = points + 16 * sub;
  if (DT == DT_F32) {
    const float4* q = reinterpret_cast<const float4*>(qs);
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(stg);
    auto issue = [&](int c0, int slot) {
      if (c0 + sub < nchunks) {
#pragma unroll
        for (int j = 0; j < 8; j++)
          if (4 * j < n) {
            const int r = 4 * j + g;
            cp_async_16(sbase + 4096u * slot + 16u * (r * 8 + (sub ^ (r & 7))), base + rid[j] * stride + 16 * c0);
          }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float r = 0.0f;
    issue(0, 0);
    issue(8, 1);
    for (int c0 = 0, slot = 0; c0 < nchunks; c0 += 8, slot ^= 1) {
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncwarp();
      const float4* s4 = reinterpret_cast<const float4*>(stg) + 256 * slot + lane * 8;
      const int sw = lane & 7;
      if (c0 + 8 <= nchunks) {
#pragma unroll
        for (int c = 0; c < 8; c++) r = f32_chunk<MT>(r, s4[c ^ sw], q[c0 + c]);
      } else {
        for (int c = 0; c < nchunks - c0; c++) r = f32_chunk<MT>(r, s4[c ^ sw], q[c0 + c]);
      }
      __syncwarp();
      issue(c0 + 16, slot);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    return MT == MT_L2 ? r : -r;
  } else {
    const uint4* q = reinterpret_cast<const uint4*>(qs);
    int32_t s[8];  // |p|^2 - 2 p.q (Euclidean) or p.q, this lane's chunks
#pragma unroll
    for (int j = 0; j < 8; j++) s[j] = 0;
    for (int c0 = 0; c0 < nchunks; c0 += 8) {
      if (c0 + sub < nchunks) {
        const uint4 qc = q[c0 + sub];
        uint4 v[8];
#pragma unroll
        for (int j = 0; j < 8; j++)
          if (4 * j < n) v[j] = __ldg(reinterpret_cast<const uint4*>(base + rid[j] * stride + 16 * c0));
#pragma unroll
        for (int j = 0; j < 8; j++)
          if (4 * j < n) {
            int32_t pq = 0, pp = 0;
            int_chunk<DT, MT>(v[j], qc, pq, pp);
            s[j] += MT == MT_L2 ? pp - 2 * pq : pq;
          }
      }
    }
    // fold across the eight lanes of a group: lane sub keeps row 4 sub + g
    const bool h4 = sub & 4, h2 = sub & 2, h1 = sub & 1;
    int32_t t4[4], t2[2];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int32_t mine = h4 ? s[j + 4] : s[j], other = h4 ? s[j] : s[j + 4];
      t4[j] = mine + __shfl_xor_sync(FULL, other, 4);
    }
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int32_t mine = h2 ? t4[j + 2] : t4[j], other = h2 ? t4[j] : t4[j + 2];
      t2[j] = mine + __shfl_xor_sync(FULL, other, 2);
    }
    const int32_t mine = h1 ? t2[1] : t2[0], other = h1 ? t2[0] : t2[1];
    int32_t tot = mine + __shfl_xor_sync(FULL, other, 1);
    // row l = 4 sub' + g' sits at lane 8 g' + sub'
    tot = __shfl_sync(FULL, tot, ((lane & 3) << 3) | (lane >> 2));
    return MT == MT_L2 ? __int2float_rn(qq + tot) : -__int2float_rn(tot);
  }
}

}  // namespace pann
