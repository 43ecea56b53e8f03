// Distances of up to 32 scattered rows to one staged query, a row per lane.
//
// Reading one row per lane costs the L1 a pass per lane and 16-byte chunk (32
// rows of 384 bytes: 768 passes; tier 0 spent 85 % of its L1 pipe on them).
//   8-bit: four neighbouring lanes read 64 contiguous bytes of a row, eight
//          rows a load instruction (a quarter of the passes); each lane
//          multiplies its own chunks (integer sums are exact in any order) and
//          four partial sums are folded across the four lanes with 3 shuffles,
//          which leaves each lane one row's distance. Eight lanes a row halve
//          the passes again but cost 30 more instructions, which a search
//          waits for more than for the L1.
//   float: eight lanes read 128 contiguous bytes, four rows an instruction (96
//          passes for those 32 rows). The sum must run through a row in
//          dimension order, so 32 rows x 128
//          bytes pass through a 4 KB shared buffer per warp (cp.async, no
//          registers held), chunk c of row r at slot c ^ (r % 8): both the
//          8-lane writes and the per-lane reads of a row touch every bank
//          once a quarter warp. Two such column blocks are in flight.
#pragma once
#include "common.cuh"
#include "lowprec.cuh"

namespace pann {

// Bytes of shared scratch a warp needs (16-byte aligned).
template <int DT>
__host__ __device__ constexpr uint32_t row_score_scratch() { return DT == DT_F32 ? 8192u : 0u; }
__host__ __device__ inline uint32_t row_score_scratch_rt(int dtype) { return dtype == DT_F32 ? 8192u : 0u; }

__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// Streams rows of nchunks 16-byte chunks through the warp's scratch: use(c, v) is called in every lane with chunk c of
// row `id` of that lane, c ascending. Every lane's id is a row; loads past the first n lanes' rows are left out.
template <class Use>
__device__ __forceinline__ void warp_stream_rows(const uint8_t* __restrict__ points, uint32_t stride, int nchunks,
                                                 uint32_t id, int n, uint8_t* stg, int lane, Use&& use) {
  const unsigned FULL = 0xFFFFFFFFu;
  const int g = lane >> 3, sub = lane & 7;
  uint32_t rid[8];  // the rows this lane reads a part of: 4 j + g
#pragma unroll
  for (int j = 0; j < 8; j++) rid[j] = __shfl_sync(FULL, id, 4 * j + g);
  // row 4 j + g's chunk goes to slot sub ^ (row % 8): two address patterns, j even and odd
  const uint32_t s0 = (uint32_t)__cvta_generic_to_shared(stg) + 128u * g;
  const uint32_t even = s0 + 16u * (sub ^ g), odd = s0 + 512u + 16u * (sub ^ (g + 4));
  auto issue = [&](int c0, int slot) {
    if (c0 + sub < nchunks) {
      const uint8_t* const base = points + 16 * (c0 + sub);
      const uint32_t de = even + 4096u * slot, dd = odd + 4096u * slot;
#pragma unroll
      for (int j = 0; j < 8; j += 2)
        if (4 * j < n) {
          cp_async_16(de + 512u * j, base + (uint64_t)rid[j] * stride);
          cp_async_16(dd + 512u * j, base + (uint64_t)rid[j + 1] * stride);
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  issue(0, 0);
  issue(8, 1);
  for (int c0 = 0, slot = 0; c0 < nchunks; c0 += 8, slot ^= 1) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    const uint4* s4 = reinterpret_cast<const uint4*>(stg) + 256 * slot + lane * 8;
    const int sw = lane & 7;
    if (c0 + 8 <= nchunks) {
#pragma unroll
      for (int c = 0; c < 8; c++) use(c0 + c, s4[c ^ sw]);
    } else {
      for (int c = 0; c < nchunks - c0; c++) use(c0 + c, s4[c ^ sw]);
    }
    __syncwarp();
    issue(c0 + 16, slot);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Lane l < n returns the distance of row `id` (its own) to the query staged at
// qs (stage_query); 1 <= n <= 32 rows, held by the first n lanes (the other
// lanes' ids are not used). Every lane of the warp takes part; qs and stg are the warp's own. Rows are at most 32 KB
// (stride fits 32 bits).
template <int DT, int MT>
__device__ __forceinline__ float warp_score_rows(const uint8_t* __restrict__ points, uint64_t stride64, int nchunks,
                                                 uint32_t id, int n, const uint8_t* qs, uint8_t* stg, int32_t qq,
                                                 int lane) {
  const unsigned FULL = 0xFFFFFFFFu;
  const uint32_t stride = (uint32_t)stride64;
  // loads that cover lanes past n repeat the first row (one fixed row instead, row 0, makes its L2 lines a hot spot
  // for the whole device: tier 0 of 10K queries on 1M x 96 floats 1.91 -> 2.55 ms)
  const uint32_t id0 = __shfl_sync(FULL, id, 0);
  if (lane >= n) id = id0;
  if (DT == DT_F32) {
    const float4* q = reinterpret_cast<const float4*>(qs);
    float r = 0.0f;
    warp_stream_rows(points, stride, nchunks, id, n, stg, lane, [&](int c, const uint4& v) {
      r = f32_chunk<MT>(r, make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z),
                                       __uint_as_float(v.w)), q[c]);
    });
    return MT == MT_L2 ? r : -r;
  } else {
    const int g = lane >> 2, sub = lane & 3;
    const uint4* q = reinterpret_cast<const uint4*>(qs);
    const uint4* row[4];  // this lane's part of row 8 j + g
    int32_t s[4];         // |p|^2 - 2 p.q (Euclidean) or p.q, this lane's chunks
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const uint32_t rid = __shfl_sync(FULL, id, 8 * j + g);
      row[j] = reinterpret_cast<const uint4*>(points + (uint64_t)rid * stride) + sub;
      s[j] = 0;
    }
    for (int c0 = 0; c0 < nchunks; c0 += 8) {
      const bool h0 = c0 + sub < nchunks, h1 = c0 + 4 + sub < nchunks;
      const uint4 z = make_uint4(0, 0, 0, 0);
      uint4 v[8];
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (8 * j < n) {
          v[2 * j] = h0 ? __ldg(row[j] + c0) : z;
          v[2 * j + 1] = h1 ? __ldg(row[j] + c0 + 4) : z;
        }
      const uint4 q0 = h0 ? q[c0 + sub] : z, q1 = h1 ? q[c0 + 4 + sub] : z;
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (8 * j < n) {
          int32_t pq = 0, pp = 0;
          int_chunk<DT, MT>(v[2 * j], q0, pq, pp);
          int_chunk<DT, MT>(v[2 * j + 1], q1, pq, pp);
          s[j] += MT == MT_L2 ? pp - 2 * pq : pq;
        }
    }
    // fold across the four lanes of a group: lane sub keeps row 8 sub + g
    const bool b1 = sub & 2, b0 = sub & 1;
    const int32_t x0 = (b1 ? s[2] : s[0]) + __shfl_xor_sync(FULL, b1 ? s[0] : s[2], 2);
    const int32_t x1 = (b1 ? s[3] : s[1]) + __shfl_xor_sync(FULL, b1 ? s[1] : s[3], 2);
    int32_t tot = (b0 ? x1 : x0) + __shfl_xor_sync(FULL, b0 ? x0 : x1, 1);
    // row l = 8 sub' + g' sits at lane 4 g' + sub'
    tot = __shfl_sync(FULL, tot, ((lane & 7) << 2) | (lane >> 3));
    return MT == MT_L2 ? __int2float_rn(qq + tot) : -__int2float_rn(tot);
  }
}

// Lane l < n returns the approximate distance of row `id` of the low-precision copy (lowprec.cuh) to the query staged
// at qs; as warp_score_rows, whose bound it shares. Two rows a lane in registers (eight chunks of each in flight)
// spilled 300 bytes and read each 128-byte line in eight passes: 10,000 queries at beam 45, 200K x 96 random graph,
// 6.85 -> 3.57 ms in bf16 and 6.48 -> 3.88 ms in fp8; 60K x 900, 42.7 -> 19.4 and 38.7 -> 21.8 ms.
template <int MT, int PREC>
__device__ __forceinline__ float warp_score_lp(const uint8_t* __restrict__ rows, uint64_t stride, int chunks, uint32_t id,
                                               int n, const float* qs, const float* __restrict__ scales, int d,
                                               uint8_t* stg, int lane) {
  const uint32_t id0 = __shfl_sync(0xFFFFFFFFu, id, 0);
  if (lane >= n) id = id0;
  float a0 = 0.0f, a1 = 0.0f;
  warp_stream_rows(rows, (uint32_t)stride, chunks, id, n, stg, lane,
                   [&](int c, const uint4& v) { lp_chunk<MT, PREC>(v, c, qs, scales, d, a0, a1); });
  return MT == MT_L2 ? a0 + a1 : -(a0 + a1);
}

}  // namespace pann
