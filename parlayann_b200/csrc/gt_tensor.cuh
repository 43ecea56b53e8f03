// Brute-force groundtruth: the pieces shared by the plain kernel
// (bruteforce.cu) and the tensor-core path (gt_tensor.cu).
#pragma once
#include <vector>
#include "common.cuh"
#include "index.cuh"

namespace pann {

// FP64 (float) or exact integer distance of one pair.
template <int DT, int MT>
__device__ __forceinline__ double exact_dist(const uint8_t* __restrict__ row, const uint8_t* q, int d) {
  if (DT == DT_F32) {
    const float* x = reinterpret_cast<const float*>(row);
    const float* y = reinterpret_cast<const float*>(q);
    double r = 0.0;
    for (int i = 0; i < d; i++) {
      double a = (double)y[i], b = (double)__ldg(x + i);
      r = MT == MT_L2 ? __dadd_rn(r, __dmul_rn(__dsub_rn(a, b), __dsub_rn(a, b))) : __dadd_rn(r, __dmul_rn(a, b));
    }
    return MT == MT_L2 ? r : -r;
  } else {
    long long r = 0;
    for (int i = 0; i < d; i++) {
      int a = DT == DT_U8 ? (int)q[i] : (int)(int8_t)q[i];
      int b = DT == DT_U8 ? (int)__ldg(row + i) : (int)(int8_t)__ldg(row + i);
      r += MT == MT_L2 ? (long long)(a - b) * (a - b) : (long long)a * b;
    }
    return MT == MT_L2 ? (double)r : -(double)r;
  }
}

__device__ __forceinline__ bool dless(double a, uint32_t ia, double b, uint32_t ib) {
  return a < b || (a == b && ia < ib);
}

// Bytes of each groundtruth buffer that an index keeps between calls. 10K queries on 1M x 96 floats use 201 MB of images
// and candidate buffers; freeing and allocating them would add to every call.
constexpr size_t GT_KEEP = 384ull << 20;

int groundtruth_tensor(pann_index* idx, const uint8_t* dq, uint32_t nq, uint32_t k, uint32_t* dids, double* dd,
                       std::vector<uint32_t>* fallback, cudaStream_t st);

}  // namespace pann
