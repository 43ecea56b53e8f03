// Exact brute-force top-k on the tensor cores (compute_groundtruth,
// data_tools/compute_groundtruth.cpp:22-60): the scores of every (query,
// point) pair are one matrix product, computed by tcgen05.mma, and only the
// pairs below a per-query threshold leave the tensor memory.
//
//   gt_centre_kernel  (float) a centre c for data far from the origin, else
//                     zero: distances and the order of dot products with one
//                     query do not change when c is taken off every point
//                     (and, Euclidean, off the queries), the norms that the
//                     error margin grows with do
//   gt_absmax_kernel  (float) the largest |value - c|, which fixes a
//                     power-of-two scale into half precision's range
//   gt_image_kernel   operand images: tiles of rows laid out in global memory
//                     exactly as the MMA reads them from shared memory (8-row
//                     x 16-byte core matrices, 64 bytes of K at a time), so a
//                     tile is fetched with plain bulk copies. 8-bit rows are
//                     copied; a float row x (less c) is split into two
//                     half-precision planes, hi = fp16(x s) and lo =
//                     fp16(x s - hi), which hold x s to 2^-23 relative (one
//                     float32 ulp: the rest after hi has up to 13 bits, lo 11).
//   gt_mma_kernel     one block per (N queries, slice of the points): the
//                     queries' image stays in shared memory, point tiles of
//                     128 rows stream through a ring of bulk copies, one
//                     thread issues the MMAs (8-bit: one product, exact int32
//                     sums; float: hi.hi + hi.lo + lo.hi, float32 sums) into
//                     two alternating accumulators, and sixteen warps read
//                     the finished one: score = |b|^2 - 2 q.b (or -q.b), kept if
//                     below the query's threshold. A kept pair goes to the
//                     (query, slice) buffer; a buffer of more than C + GT_CUT keys
//                     is cut to about C, the last of whose scores is a
//                     threshold for every slice of that query.
//   gt_final_kernel   a block per query: the surviving keys of all slices;
//                     8-bit: the k smallest (score, id) keys are the answer;
//                     float: FP64 distances of the candidates within the
//                     scores' error margin decide, ties by id.
//
// Float margin: |score - exact| <= bound with u = 2^-24, b and q the rows less
// c, B = max |b|; first-order sums:
//   centre       b and q are rounded differences, u |b| and u |q| off: moves
//                |b|^2 - 2 q.b by 2 u B^2 + 4 u |q| B (q.b by u |q| B)
//   split        hi + lo misses x s by at most 2 u |x s|, or 2^-25 (half of the
//                smallest step) where lo is below half precision's normal range,
//                which moves a dot product by at most 2^-38 sqrt(d) B (|q| + the
//                batch's largest value); lo.lo <= 4 u |q||b| is left out: 8 u |q||b|
//   accumulation 3 d products, each addition off by at most 2 u |q||b| (the
//                tensor core may truncate): 6 d u |q||b|
//   |b|^2 and the final FMA: u B^2 and u of the result, u (B^2 + 2 |q| B) or u |q| B
// The sums are 4 u B^2 + 2 (6 d + 11) u |q| B for Euclidean distance and
// (6 d + 10) u |q| B for mips (plus the step term); bound is twice that. A true
// top-k point has score <= s_k + 2 bound (s_k: the k-th smallest score); if the
// query's threshold is above that, no slice dropped such a point. A query
// that fails the test (or whose survivors do not fit) is left to the plain
// kernel, which is about 80 times slower: without a centre that were all
// queries of unit-variance data 32 from the origin in each of 96 dimensions
// (100K points, 1,000 queries: 51 ms; 0.62 ms with it, as at the origin).
//
// What bounds it (10K queries x 1M x 96 floats, k 20; 120 ms with float32
// FMAs on the CUDA cores, 8.4 ms here): the three products are 5.8 TFLOP of
// half-precision MMA, 3.4 ms at the measured 1676 TFLOP/s; the epilogue's 1e10
// scores cost about 2.3 instructions each and run beside the MMAs; the rest is
// the falling thresholds, about 800 appends per query and slice, most of them
// in the first segment (4.0 ms of it, the last 1.6). 8-bit scores need one
// product (100K x 128, 1,000 queries, k 100: 55.6 -> 0.80 ms).
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>

#include "common.cuh"
#include "gt_tensor.cuh"
#include "index.cuh"
#include "umma.cuh"

namespace pann {

constexpr int GT_ROWS = 128;           // points per tile: the MMA's M
constexpr int GT_KB = 64;              // bytes of K per chunk and plane
constexpr int GT_EPI_WARPS = 16;         // four a scheduler: with two the epilogue's latencies show
constexpr int GT_THREADS = 32 * (GT_EPI_WARPS + 2);
constexpr int GT_COLS = 256 / GT_EPI_WARPS;    // thresholds a warp keeps
constexpr uint64_t GT_WAIT_NS = 4000000000ull;  // a wait this long means a lost arrival
constexpr uint32_t GT_CUT = 64;        // a buffer of more than C + GT_CUT keys is cut
constexpr uint32_t GT_CAP = 12288;     // slices x C, at most: the final kernel's scores take up to twice as many words
constexpr uint32_t GT_FCAP = 1024;     // float candidates scored in FP64
// scores above this could overflow float32 on the way: the plain kernel takes over
constexpr double GT_HUGE = 1e15;

struct GtScale {
  uint32_t pt_max, q_max;            // bits of the largest |value - c| (float)
  unsigned long long bmax;           // bits of the largest |b| (double)
  uint32_t centre_done;              // blocks of gt_centre_kernel that have finished
};

__device__ __forceinline__ int gt_exp(uint32_t max_bits) {
  // scale 2^e brings the largest value into [2^13, 2^14)
  const float m = __uint_as_float(max_bits);
  if (!(m > 0.0f) || !(m < 1e30f)) return 0;
  int e;
  frexpf(m, &e);
  return min(14 - e, 120);
}

// The centre: the mean of a sample of the points (any centre is valid; 512
// rows bring it within a 22nd of the spread), taken where it holds at least
// three quarters of the sample's mean square, so that B falls to about half or
// less; nearer the origin the points' spread sets B and zero costs no rounding.
// A block per 32 columns and 32 rows, four loads a thread in flight; the last
// one to finish adds the partial sums (always in the same order) and decides.
constexpr uint32_t GT_CEN_ROWS = 512, GT_CEN_PARTS = 16;
struct GtCentre {
  double *sum, *sq;  // GT_CEN_PARTS rows of cols
  uint32_t* cnt;
  float* centre;     // cols
  uint32_t cols;
};
__global__ void __launch_bounds__(256) gt_centre_kernel(const uint8_t* __restrict__ points, uint64_t stride, uint64_t n,
                                                        GtCentre g, GtScale* sc) {
  __shared__ double s_a[8][32], s_b[8][32];
  __shared__ uint32_t s_c[8][32];
  __shared__ bool s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t col = blockIdx.x * 32 + lane;
  const uint32_t m = (uint32_t)min(n, (uint64_t)GT_CEN_ROWS);
  const uint64_t step = n / m * stride;
  constexpr int PER = GT_CEN_ROWS / GT_CEN_PARTS / 8;
  float x[PER];
#pragma unroll
  for (int t = 0; t < PER; t++) {
    const uint32_t r = (blockIdx.y * PER + t) * 8 + warp;
    x[t] = r < m && col < g.cols ? __ldg(reinterpret_cast<const float*>(points + r * step) + col) : __int_as_float(0x7fffffff);
  }
  double sum = 0.0, sq = 0.0;
  uint32_t cnt = 0;
#pragma unroll
  for (int t = 0; t < PER; t++)
    if (fabsf(x[t]) < __int_as_float(0x7f800000)) {  // finite values only
      sum += (double)x[t];
      sq += (double)x[t] * (double)x[t];
      cnt++;
    }
  s_a[warp][lane] = sum;
  s_b[warp][lane] = sq;
  s_c[warp][lane] = cnt;
  __syncthreads();
  if (warp == 0) {
    for (int w = 1; w < 8; w++) {
      sum += s_a[w][lane];
      sq += s_b[w][lane];
      cnt += s_c[w][lane];
    }
    if (col < g.cols) {
      const uint32_t at = blockIdx.y * g.cols + col;
      g.sum[at] = sum;
      g.sq[at] = sq;
      g.cnt[at] = cnt;
    }
    __threadfence();
    __syncwarp();
    if (lane == 0) s_last = atomicAdd(&sc->centre_done, 1u) == gridDim.x * gridDim.y - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  double c2 = 0.0, m2 = 0.0;  // squared norm of the mean, mean squared norm
  for (uint32_t j = threadIdx.x; j < g.cols; j += blockDim.x) {
    double a = 0.0, b = 0.0;
    uint32_t c = 0;
#pragma unroll
    for (uint32_t p = 0; p < GT_CEN_PARTS; p++) {
      a += __ldcg(g.sum + p * g.cols + j);
      b += __ldcg(g.sq + p * g.cols + j);
      c += __ldcg(g.cnt + p * g.cols + j);
    }
    const float mean = c ? (float)(a / c) : 0.0f;
    g.centre[j] = mean;
    c2 += (double)mean * (double)mean;
    m2 += c ? b / c : 0.0;
  }
  for (int o = 16; o; o >>= 1) {
    c2 += __shfl_xor_sync(0xFFFFFFFFu, c2, o);
    m2 += __shfl_xor_sync(0xFFFFFFFFu, m2, o);
  }
  if (lane == 0) {
    s_a[0][warp] = c2;
    s_b[0][warp] = m2;
  }
  __syncthreads();
  c2 = m2 = 0.0;
  for (int w = 0; w < 8; w++) {
    c2 += s_a[0][w];
    m2 += s_b[0][w];
  }
  if (c2 >= 0.75 * m2) return;
  for (uint32_t j = threadIdx.x; j < g.cols; j += blockDim.x) g.centre[j] = 0.0f;
}

// Rows of rowchunks 16-byte chunks each; centre: a row of the same length, or NULL.
__global__ void gt_absmax_kernel(const float4* __restrict__ rows, uint64_t nchunks, uint32_t rowchunks,
                                 const float4* __restrict__ centre, uint32_t* out) {
  uint32_t m = 0;
  const uint64_t first = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (uint64_t)gridDim.x * blockDim.x;
  uint32_t j = (uint32_t)(first % rowchunks);
  const uint32_t jstep = (uint32_t)(step % rowchunks);
  for (uint64_t i = first; i < nchunks; i += step) {
    const float4 v = __ldg(rows + i);
    const float4 c = centre ? __ldg(centre + j) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float x[4] = {__fsub_rn(v.x, c.x), __fsub_rn(v.y, c.y), __fsub_rn(v.z, c.z), __fsub_rn(v.w, c.w)};
#pragma unroll
    for (int t = 0; t < 4; t++) {
      const uint32_t w = __float_as_uint(x[t]) & 0x7FFFFFFFu;
      m = w < 0x7F800000u && w > m ? w : m;  // finite values only
    }
    j += jstep;
    if (j >= rowchunks) j -= rowchunks;
  }
  m = __reduce_max_sync(0xFFFFFFFFu, m);
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// One warp per 8 rows and all of K: lane (r, c) = (lane / 4, lane % 4) takes
// the chunk c of row r, so a float row's 128 bytes are read by four lanes and
// the 512 bytes of a plane's eight rows are written whole. Rows at and past
// nrows, and K past the row, are zero.
template <int DT>
__global__ void __launch_bounds__(256) gt_image_kernel(const uint8_t* __restrict__ rows, uint64_t stride, uint32_t d,
                                                       uint64_t nrows, uint64_t rows_total, uint32_t tile_rows,
                                                       uint32_t kch, const GtScale* sc, const float4* __restrict__ centre,
                                                       int is_query, uint8_t* img, void* norms,
                                                       unsigned long long* bmax) {
  const int lane = threadIdx.x & 31;
  const int r8 = lane >> 2, c = lane & 3;
  const uint32_t planes = DT == DT_F32 ? 2 : 1;
  const float s = DT == DT_F32 ? ldexpf(1.0f, gt_exp(is_query ? sc->q_max : sc->pt_max)) : 1.0f;
  const uint64_t groups = rows_total / 8;
  double mx = 0.0;
  for (uint64_t g = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < groups;
       g += ((uint64_t)gridDim.x * blockDim.x) >> 5) {
    const uint64_t row = g * 8 + r8;
    const uint64_t tile = g * 8 / tile_rows;
    const uint32_t rt = (uint32_t)(g * 8 - tile * tile_rows);
    const uint8_t* src = rows + row * stride;
    uint8_t* dst = img + tile * ((uint64_t)kch * planes * tile_rows * GT_KB) + (rt >> 3) * 512u + c * 128u + r8 * 16u;
    double n2 = 0.0;
    int32_t ni = 0;
    for (uint32_t kc = 0; kc < kch; kc++) {
      if (DT == DT_F32) {
        uint32_t h[4] = {0, 0, 0, 0}, l[4] = {0, 0, 0, 0};
#pragma unroll
        for (int q = 0; q < 2; q++) {
          const uint32_t b = kc * 128 + c * 32 + q * 16;  // byte of the row
          if (row < nrows && b < stride) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(src + b));
            const float4 c4 = centre ? __ldg(centre + b / 16) : make_float4(0.f, 0.f, 0.f, 0.f);
            const float x[4] = {__fsub_rn(v.x, c4.x), __fsub_rn(v.y, c4.y), __fsub_rn(v.z, c4.z), __fsub_rn(v.w, c4.w)};
#pragma unroll
            for (int j = 0; j < 4; j++) {
              n2 += (double)x[j] * (double)x[j];
              const float xs = x[j] * s;
              const __half hh = __float2half_rn(xs);
              const __half ll = __float2half_rn(xs - __half2float(hh));
              h[q * 2 + j / 2] |= (uint32_t)__half_as_ushort(hh) << (16 * (j & 1));
              l[q * 2 + j / 2] |= (uint32_t)__half_as_ushort(ll) << (16 * (j & 1));
            }
          }
        }
        uint8_t* o = dst + (uint64_t)kc * planes * tile_rows * GT_KB;
        *reinterpret_cast<uint4*>(o) = make_uint4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<uint4*>(o + (uint64_t)tile_rows * GT_KB) = make_uint4(l[0], l[1], l[2], l[3]);
      } else {
        uint4 v = make_uint4(0, 0, 0, 0);
        const uint32_t b = kc * GT_KB + c * 16;
        if (row < nrows && b < stride) v = __ldg(reinterpret_cast<const uint4*>(src + b));
        if (DT == DT_U8) {
          ni = dp4u(v.x, v.x, ni); ni = dp4u(v.y, v.y, ni); ni = dp4u(v.z, v.z, ni); ni = dp4u(v.w, v.w, ni);
        } else {
          ni = dp4s(v.x, v.x, ni); ni = dp4s(v.y, v.y, ni); ni = dp4s(v.z, v.z, ni); ni = dp4s(v.w, v.w, ni);
        }
        *reinterpret_cast<uint4*>(dst + (uint64_t)kc * tile_rows * GT_KB) = v;
      }
    }
    if (DT == DT_F32) {
      n2 += __shfl_xor_sync(0xFFFFFFFFu, n2, 1);
      n2 += __shfl_xor_sync(0xFFFFFFFFu, n2, 2);
      if (c == 0) reinterpret_cast<float*>(norms)[row] = (float)n2;
      if (row < nrows) mx = fmax(mx, n2);  // a NaN row scores NaN: below no threshold
    } else {
      ni += __shfl_xor_sync(0xFFFFFFFFu, ni, 1);
      ni += __shfl_xor_sync(0xFFFFFFFFu, ni, 2);
      if (c == 0) reinterpret_cast<int32_t*>(norms)[row] = ni;
    }
  }
  if (DT == DT_F32 && bmax) {
    // non-negative doubles order as their bits
    unsigned long long m = (unsigned long long)__double_as_longlong(sqrt(mx));
    for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
    if (lane == 0) atomicMax(bmax, m);
  }
}

struct GtMma {
  const uint8_t* a_img;  // point tiles of this segment
  const void* pnorm;     // |b|^2 per row of the segment (float / int32)
  uint32_t n_seg;        // rows of the segment
  uint32_t ntiles;
  uint32_t id0;          // id of its first row
  const uint8_t* b_img;  // query tiles of N rows
  uint32_t nq, N, kch, ksteps, slices, stages;
  uint32_t C, CB;
  uint64_t* cand;        // per (query, slice): CB keys
  uint32_t* count;       // per (query, slice)
  uint32_t* thr;         // per query, order-preserving bits
  const GtScale* scale;
  uint32_t* err;
};

struct GtLayout {
  uint32_t b, ring, thr, own, cnt, bars, misc, total;
};
__host__ __device__ inline GtLayout gt_layout(uint32_t N, uint32_t kch, uint32_t planes, uint32_t stages) {
  GtLayout y;
  uint32_t o = 0;
  y.b = o;    o += N * kch * planes * GT_KB;
  y.ring = o; o += stages * planes * GT_ROWS * GT_KB;
  y.thr = o;  o += 4 * 256;
  y.own = o;  o += 4 * 256;
  y.cnt = o;  o += 4 * 256;
  y.bars = o; o += 8 * (1 + 4 + 2 * stages);
  o = (o + 15) & ~15u;
  y.misc = o; o += 16;
  y.total = o;
  return y;
}

// tcgen05.mma with 8-bit integer operands (kind::i8, int32 accumulator).
__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Untiled bulk copy global -> shared (addresses and size multiples of 16).
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void epi_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(32 * GT_EPI_WARPS) : "memory"); }

// int32 scores as order-preserving bits
__device__ __forceinline__ uint32_t ord_of_int(int32_t v) { return (uint32_t)v ^ 0x80000000u; }

// One warp: cut the cnt keys of buf to at least the C and at most the
// C + GT_SLACK smallest (by score, then id); *kept gets their number. Returns
// the last kept score's bits: a later key of this buffer (its id is larger) at
// or above it is not among the C best. The keys stay in registers (KPL a lane); the cut is found by
// bisecting the scores' differing bits with warp counts, which ends as soon as
// a count falls in the slack (about five rounds of KPL compares; a rank sort
// would take cnt^2 / 32). Only where equal scores leave no such count the
// bisection runs to the C-th score itself and its smallest ids are kept.
constexpr uint32_t GT_SLACK = 16;
template <int KPL>
__device__ __forceinline__ uint32_t gt_cut(uint64_t* buf, uint32_t cnt, uint32_t C, int lane, uint32_t* kept) {
  const unsigned FULL = 0xFFFFFFFFu;
  uint32_t hi[KPL], id[KPL];
  uint32_t mn = 0xFFFFFFFFu, mx = 0;
#pragma unroll
  for (int j = 0; j < KPL; j++) {
    const uint32_t i = (uint32_t)j * 32 + lane;
    const uint64_t k = i < cnt ? buf[i] : ~0ull;
    hi[j] = (uint32_t)(k >> 32);
    id[j] = (uint32_t)k;
    mn = min(mn, hi[j]);
    if (i < cnt) mx = max(mx, hi[j]);
  }
  mn = __reduce_min_sync(FULL, mn);
  mx = __reduce_max_sync(FULL, mx);
  const int top = 31 - __clz(mn ^ mx);  // -1: all scores equal
  uint32_t v = top < 0 ? mn : mn & ~((2u << top) - 1u);
  uint32_t idmax = 0x7FFFFFFFu;
  bool ties = true;
  for (int b = top; b >= 0; b--) {
    const uint32_t t = v | ((1u << b) - 1u);
    uint32_t n = 0;
#pragma unroll
    for (int j = 0; j < KPL; j++) n += hi[j] <= t;
    n = __reduce_add_sync(FULL, n);
    if (n < C) {
      v |= 1u << b;
    } else if (n <= C + GT_SLACK) {
      v = t;
      ties = false;
      break;
    }
  }
  if (ties) {
    uint32_t less = 0, eq = 0;
#pragma unroll
    for (int j = 0; j < KPL; j++) {
      less += hi[j] < v;
      eq += hi[j] == v && id[j] != 0xFFFFFFFFu;
    }
    less = __reduce_add_sync(FULL, less);
    eq = __reduce_add_sync(FULL, eq);
    if (less + eq > C) {
      idmax = 0;
      for (int b = 30; b >= 0; b--) {
        const uint32_t t = idmax | ((1u << b) - 1u);
        uint32_t n = 0;
#pragma unroll
        for (int j = 0; j < KPL; j++) n += hi[j] == v && id[j] <= t;
        if (__reduce_add_sync(FULL, n) < C - less) idmax |= 1u << b;
      }
    }
  }
  uint32_t at = 0;
#pragma unroll
  for (int j = 0; j < KPL; j++) {
    const bool keep = id[j] != 0xFFFFFFFFu && (hi[j] < v || (hi[j] == v && id[j] <= idmax));
    const unsigned m = __ballot_sync(FULL, keep);
    if (keep) buf[at + __popc(m & ((1u << lane) - 1u))] = ((uint64_t)hi[j] << 32) | id[j];
    at += __popc(m);
  }
  *kept = at;
  return v;
}

template <int DT, int MT, int KPL>
__global__ void __launch_bounds__(GT_THREADS, 1) gt_mma_kernel(GtMma g) {
  extern __shared__ __align__(128) uint8_t smem[];
  constexpr bool F = DT == DT_F32;
  constexpr uint32_t PL = F ? 2 : 1;
  using T = typename std::conditional<F, float, int32_t>::type;
  const GtLayout y = gt_layout(g.N, g.kch, PL, g.stages);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned FULL = 0xFFFFFFFFu;
  T* thr_s = reinterpret_cast<T*>(smem + y.thr);  // a score enters the buffer if it is below this
  T* own_s = reinterpret_cast<T*>(smem + y.own);  // this slice's own C-th score
  uint32_t* cnt_s = reinterpret_cast<uint32_t*>(smem + y.cnt);
  volatile uint32_t* misc = reinterpret_cast<volatile uint32_t*>(smem + y.misc);  // [0] tensor memory, [1] abort
  const uint32_t bar0 = smem_u32(smem + y.bars);
  const uint32_t b_full = bar0, acc_full = bar0 + 8, acc_empty = bar0 + 24, full = bar0 + 40,
                 empty = full + 8 * g.stages;
  const uint32_t q0 = blockIdx.x * g.N, slice = blockIdx.y;
  const T T_MAX = F ? (T)__int_as_float(0x7f800000) : (T)0x7FFFFFFF;
  const T T_MIN = F ? (T)__int_as_float(0xff800000) : (T)(-2147483647 - 1);

  if (tid < 256) {
    const uint32_t q = q0 + tid;
    const bool live = tid < (int)g.N && q < g.nq;
    cnt_s[tid] = live ? g.count[(uint64_t)q * g.slices + slice] : 0u;
    own_s[tid] = live ? T_MAX : T_MIN;
    thr_s[tid] = own_s[tid];
  }
  if (tid == 0) {
    mbar_init(b_full, 1);
    for (int i = 0; i < 2; i++) {
      mbar_init(acc_full + 8 * i, 1);
      mbar_init(acc_empty + 8 * i, GT_EPI_WARPS);
    }
    for (uint32_t i = 0; i < g.stages; i++) {
      mbar_init(full + 8 * i, 1);
      mbar_init(empty + 8 * i, 1);
    }
    misc[1] = 0;
  }
  if (warp == GT_EPI_WARPS + 1) tmem_alloc(smem_u32(smem + y.misc), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = misc[0];
  const uint32_t stage_bytes = PL * GT_ROWS * GT_KB;
  // this slice's tiles: slice, slice + slices, ...
  const uint32_t my_tiles = g.ntiles > slice ? (g.ntiles - slice + g.slices - 1) / g.slices : 0;

  if (warp == GT_EPI_WARPS) {
    // ---- producer: the queries' image once, then the point tiles
    if (lane == 0 && my_tiles > 0) {
      const uint32_t bbytes = g.N * GT_KB * PL;
      mbar_expect(b_full, bbytes * g.kch);
      for (uint32_t kc = 0; kc < g.kch; kc++)
        bulk_load(smem_u32(smem + y.b) + kc * bbytes, g.b_img + ((uint64_t)blockIdx.x * g.kch + kc) * bbytes, bbytes,
                  b_full);
      uint32_t s = 0, ph = 0;
      bool ok = true;
      uint64_t issued = 0;
      for (uint32_t t = 0; t < my_tiles && ok; t++) {
        const uint8_t* src = g.a_img + (uint64_t)(slice + t * g.slices) * g.kch * stage_bytes;
        for (uint32_t kc = 0; kc < g.kch; kc++) {
          if (!mbar_wait(empty + 8 * s, ph ^ 1u, GT_WAIT_NS) || misc[1]) { ok = false; break; }
          mbar_expect(full + 8 * s, stage_bytes);
          bulk_load(smem_u32(smem + y.ring) + s * stage_bytes, src + (uint64_t)kc * stage_bytes, stage_bytes,
                    full + 8 * s);
          issued++;
          if (++s == g.stages) { s = 0; ph ^= 1u; }
        }
      }
      if (!ok) misc[1] = 1;
      // no copy of this block is in flight when it leaves: wait for the last use of every stage
      mbar_wait(b_full, 0, GT_WAIT_NS);
      for (uint32_t i = 0; i < g.stages && i < issued; i++) {
        const uint64_t last = (issued - 1 - i) / g.stages;  // the stage's last fill
        const uint32_t st = (uint32_t)((issued - 1 - i) % g.stages);
        mbar_wait(full + 8 * st, (uint32_t)(last & 1), GT_WAIT_NS);
      }
    }
  } else if (warp == GT_EPI_WARPS + 1) {
    // ---- MMA issuer
    if (lane == 0 && my_tiles > 0) {
      // instruction descriptor: float: fp16 operands (format 0), float32 sums; 8-bit: unsigned 0 / signed 1, int32 sums (2)
      const uint32_t fmt = DT == DT_I8 ? 1u : 0u;
      const uint32_t idesc = ((F ? 1u : 2u) << 4) | (fmt << 7) | (fmt << 10) | ((g.N >> 3) << 17) | ((GT_ROWS >> 4) << 24);
      const uint32_t bplane = g.N * GT_KB, aplane = GT_ROWS * GT_KB;
      bool ok = mbar_wait(b_full, 0, GT_WAIT_NS);
      uint32_t s = 0, ph = 0;
      for (uint32_t t = 0; t < my_tiles && ok; t++) {
        const uint32_t buf = t & 1u;
        if (!mbar_wait(acc_empty + 8 * buf, ((t >> 1) & 1u) ^ 1u, GT_WAIT_NS)) { ok = false; break; }
        tc_fence_after();
        const uint32_t acc = tmem + buf * g.N;
        for (uint32_t kc = 0; kc < g.kch; kc++) {
          if (!mbar_wait(full + 8 * s, ph, GT_WAIT_NS) || misc[1]) { ok = false; break; }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + y.ring) + s * stage_bytes;
          const uint32_t sb = smem_u32(smem + y.b) + kc * PL * bplane;
          const uint32_t ks = min(2u, g.ksteps - 2 * kc);
          for (uint32_t k = 0; k < ks; k++) {
            const uint64_t ah = umma_desc(sa + k * 256u, 128u, 512u), bh = umma_desc(sb + k * 256u, 128u, 512u);
            const uint32_t acc_on = (kc | k) != 0;
            if (F) {
              const uint64_t al = umma_desc(sa + aplane + k * 256u, 128u, 512u);
              const uint64_t bl = umma_desc(sb + bplane + k * 256u, 128u, 512u);
              umma_bf16(acc, al, bh, idesc, acc_on);  // kind::f16; the descriptor names the operand format
              umma_bf16(acc, ah, bl, idesc, 1u);
              umma_bf16(acc, ah, bh, idesc, 1u);
            } else {
              umma_i8(acc, ah, bh, idesc, acc_on);
            }
          }
          umma_commit(empty + 8 * s);
          if (++s == g.stages) { s = 0; ph ^= 1u; }
        }
        if (ok) umma_commit(acc_full + 8 * buf);
      }
      if (!ok) {
        misc[1] = 1;
        umma_commit(b_full);  // its MMAs leave the tensor memory before it is given back
        mbar_wait(b_full, 1, GT_WAIT_NS);
      }
    }
  } else {
    // ---- epilogue: warp w reads tensor-memory lanes 32 (w % 4).. and quarter w / 4 of the columns
    const int quad = warp & 3;
    const uint32_t part_n = g.N / (GT_EPI_WARPS / 4), c0 = (uint32_t)(warp >> 2) * part_n;
    float mul_f = 0.0f;
    if (F) mul_f = ldexpf(MT == MT_L2 ? -2.0f : -1.0f, -(gt_exp(g.scale->pt_max) + gt_exp(g.scale->q_max)));
    const uint32_t mycol = (uint32_t)(warp * GT_COLS + (lane & (GT_COLS - 1)));  // the query this thread keeps the threshold of
    const bool col_live = lane < GT_COLS && mycol < g.N && q0 + mycol < g.nq;
    uint64_t* const cbase = g.cand + ((uint64_t)q0 * g.slices + slice) * g.CB;
    const uint64_t cstep = (uint64_t)g.slices * g.CB;
    const volatile uint32_t* gthr = g.thr + q0 + mycol;
    bool ok = true;
    for (uint32_t t = 0; t < my_tiles; t++) {
      const uint32_t buf = t & 1u;
      const uint32_t tile = slice + t * g.slices;
      const uint32_t prow = tile * GT_ROWS + quad * 32 + lane;
      const bool pvalid = prow < g.n_seg;
      const uint32_t pid = g.id0 + prow;
      T pn;
      if (F) {
        pn = MT == MT_L2 ? (pvalid ? (T)reinterpret_cast<const float*>(g.pnorm)[prow] : (T)0) : (T)0;
        if (!pvalid) pn = (T)__int_as_float(0x7fffffff);  // NaN: below no threshold
      } else {
        pn = MT == MT_L2 && pvalid ? (T) reinterpret_cast<const int32_t*>(g.pnorm)[prow] : (T)0;
        if (!pvalid) pn = (T)0x7FFFFFFF;  // its dot products are 0: never below a threshold
      }
      uint32_t gb = 0xFFFFFFFFu;
      if (col_live) gb = *gthr;  // the other slices' thresholds, used after this tile
      if (ok && !mbar_wait(acc_full + 8 * buf, (t >> 1) & 1u, GT_WAIT_NS)) { ok = false; misc[1] = 1; }
      if (__any_sync(FULL, !ok)) ok = false;
      tc_fence_after();
      if (ok) {
        const uint32_t tb = tmem + buf * g.N + ((uint32_t)(quad * 32) << 16);
        uint32_t v[16];
        tmem_ld16(tb + c0, v);
        for (uint32_t c = 0; c < part_n; c += 16) {
          tmem_ld_wait();
          T s[16];
          bool any = false;
#pragma unroll
          for (int j = 0; j < 16; j++) {
            if (F) s[j] = (T)__fmaf_rn(mul_f, __uint_as_float(v[j]), (float)pn);
            else s[j] = (T)((int32_t)pn - (MT == MT_L2 ? 2 : 1) * (int32_t)v[j]);
          }
          if (c + 16 < part_n) tmem_ld16(tb + c0 + c + 16, v);
          const T* th = thr_s + c0 + c;
#pragma unroll
          for (int j = 0; j < 16; j++) any |= s[j] < th[j];
          if (__any_sync(FULL, any)) {
#pragma unroll
            for (int j4 = 0; j4 < 16; j4 += 4) {
              bool any4 = false;
#pragma unroll
              for (int j = j4; j < j4 + 4; j++) any4 |= s[j] < th[j];
              if (!__any_sync(FULL, any4)) continue;
#pragma unroll
              for (int j = j4; j < j4 + 4; j++)
                if (s[j] < th[j]) {
                  const uint32_t col = c0 + c + j;
                  const uint32_t pos = atomicAdd(cnt_s + col, 1u);
                  const uint32_t o = F ? ord_of((float)s[j]) : ord_of_int((int32_t)s[j]);
                  if (pos < g.CB) cbase[col * cstep + pos] = ((uint64_t)o << 32) | pid;
                }
            }
          }
        }
        tc_fence_before();
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty + 8 * buf);
      __syncwarp();
      epi_barrier();  // every append of this tile is in its buffer
      // a buffer is cut at C + GT_CUT keys (so it can take a whole tile: CB is at least C + GT_CUT + GT_ROWS): a cut
      // costs about as much as eight appends, and the sooner the threshold falls the fewer there are
      unsigned cut = __ballot_sync(FULL, col_live && cnt_s[mycol] > g.C + GT_CUT);
      while (cut) {
        const int j = __ffs(cut) - 1;
        cut &= cut - 1;
        const uint32_t col = (uint32_t)(warp * GT_COLS + j);
        uint32_t kept = 0;
        const uint32_t v = gt_cut<KPL>(cbase + col * cstep, min(cnt_s[col], g.CB), g.C, lane, &kept);
        __syncwarp();
        if (lane == 0) {
          cnt_s[col] = kept;
          own_s[col] = F ? (T)float_of(v) : (T)(int32_t)(v ^ 0x80000000u);
          atomicMin(g.thr + q0 + col, v);
        }
        __syncwarp();
      }
      if (col_live) {
        // another slice's C-th score v: strictly above v is out; equal scores may still win by id (8-bit only)
        T th = min(thr_s[mycol], own_s[mycol]);
        if (gb != 0xFFFFFFFFu) {
          const T o = F ? (T)float_of(gb) : (T)(int32_t)(gb ^ 0x80000000u);
          th = min(th, F ? o : (T)(o + 1));
        }
        thr_s[mycol] = th;
      }
      __syncwarp();
      epi_barrier();
    }
    if (col_live) g.count[(uint64_t)(q0 + mycol) * g.slices + slice] = min(cnt_s[mycol], g.CB);
  }
  __syncthreads();
  tc_fence_after();
  if (tid == 0 && misc[1]) atomicOr(g.err, 1u);
  if (warp == GT_EPI_WARPS + 1) tmem_dealloc(tmem, 512);
}

struct GtFinal {
  const uint64_t* cand;
  const uint32_t* count;
  const uint32_t* thr;
  uint32_t slices, CB, cap, k;
  const uint8_t* points;
  uint64_t stride;
  uint32_t d;
  const uint8_t* queries;
  const void* qnorm;
  const GtScale* scale;
  uint32_t* out_ids;
  double* out_d;
  uint32_t* fallback;
  uint32_t* nfallback;
};

constexpr int GT_FT = 128;  // threads of the final kernel

// Block-wide sum of n (every thread gets it); red holds one word per warp.
__device__ __forceinline__ uint32_t gt_block_sum(uint32_t n, uint32_t* red) {
  n = __reduce_add_sync(0xFFFFFFFFu, n);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = n;
  __syncthreads();
  uint32_t s = 0;
#pragma unroll
  for (int w = 0; w < GT_FT / 32; w++) s += red[w];
  return s;
}

// Survivors are the keys at or below the query's threshold, the smallest of
// the slices' own; a slice holds at most C + GT_CUT keys when its last tile is
// done, so their scores (a word each) fit in `cap` = slices x (C + GT_CUT)
// words whatever the data. The k-th smallest score is found on those words and
// the keys it selects are read again from the buffers (in L2). Whole keys in a
// block of GT_CAP overflowed with many slices, by the order of the appends: 100
// queries on 300K x 96 floats, k 100, 0.9 or 68 ms; 0.84 ms always now.
template <int DT, int MT>
__global__ void __launch_bounds__(GT_FT) gt_final_kernel(GtFinal g) {
  extern __shared__ __align__(16) uint8_t fsm[];
  __shared__ uint32_t s_n, s_red[GT_FT / 32], s_m;
  constexpr bool F = DT == DT_F32;
  uint32_t* words = reinterpret_cast<uint32_t*>(fsm + (F ? 12u * GT_FCAP : 8u * g.k));
  const uint32_t qi = blockIdx.x, tid = threadIdx.x;
  const uint32_t thr = g.thr[qi];
  if (tid == 0) { s_n = 0; s_m = 0; }
  __syncthreads();
  // every key of the query's buffers: a warp takes every fourth slice, four keys a lane in flight (the passes wait for
  // L2; slice after slice on the whole block they took 43 us at 148 slices)
  auto each_key = [&](auto&& use) {
    constexpr uint32_t NW = GT_FT / 32;
    const uint32_t lane = tid & 31, warp = tid >> 5;
    const uint32_t* cq = g.count + (uint64_t)qi * g.slices;
    for (uint32_t s0 = 0; s0 < g.slices; s0 += GT_FT) {
      const uint32_t mine = s0 + NW * lane + warp;
      const uint32_t cnt = mine < g.slices ? cq[mine] : 0u;
      for (uint32_t l = 0; l < 32 && s0 + NW * l + warp < g.slices; l++) {
        const uint32_t c = __shfl_sync(0xFFFFFFFFu, cnt, l);
        const uint64_t* keys = g.cand + ((uint64_t)qi * g.slices + s0 + NW * l + warp) * g.CB;
        for (uint32_t i = lane; i < c; i += 128) {
          uint64_t k[4];
#pragma unroll
          for (uint32_t j = 0; j < 4; j++) k[j] = i + 32 * j < c ? keys[i + 32 * j] : ~0ull;
#pragma unroll
          for (uint32_t j = 0; j < 4; j++)
            if (i + 32 * j < c) use(k[j]);
        }
      }
    }
  };
  each_key([&](uint64_t key) {
    if ((uint32_t)(key >> 32) <= thr) {
      const uint32_t p = atomicAdd(&s_n, 1u);
      if (p < g.cap) words[p] = (uint32_t)(key >> 32);
    }
  });
  __syncthreads();
  const uint32_t m = s_n;
  bool bad = m > g.cap || m < g.k;
  uint32_t v = 0;
  if (!bad) {  // the k-th smallest score, bit by bit
    for (int b = 31; b >= 0; b--) {
      const uint32_t t = v | ((1u << b) - 1u);
      uint32_t n = 0;
      for (uint32_t i = tid; i < m; i += GT_FT) n += words[i] <= t;
      if (gt_block_sum(n, s_red) < g.k) v |= 1u << b;
    }
  }
  if (!F) {
    // exact scores: the k smallest (score, id) keys
    if (!bad) {
      uint32_t less = 0, eq = 0;
      for (uint32_t i = tid; i < m; i += GT_FT) {
        less += words[i] < v;
        eq += words[i] == v;
      }
      less = gt_block_sum(less, s_red);
      eq = gt_block_sum(eq, s_red);
      uint32_t idmax = 0x7FFFFFFFu;
      if (less + eq > g.k) {  // the ids at that score, in place of the scores
        if (tid == 0) s_n = 0;
        __syncthreads();
        each_key([&](uint64_t key) {
          if ((uint32_t)(key >> 32) == v) words[atomicAdd(&s_n, 1u)] = (uint32_t)key;
        });
        __syncthreads();
        idmax = 0;
        for (int b = 30; b >= 0; b--) {
          const uint32_t t = idmax | ((1u << b) - 1u);
          uint32_t n = 0;
          for (uint32_t i = tid; i < eq; i += GT_FT) n += words[i] <= t;
          if (gt_block_sum(n, s_red) < g.k - less) idmax |= 1u << b;
        }
      }
      uint64_t* best = reinterpret_cast<uint64_t*>(fsm);
      each_key([&](uint64_t key) {
        const uint32_t h = (uint32_t)(key >> 32);
        if (h < v || (h == v && (uint32_t)key <= idmax)) {
          const uint32_t p = atomicAdd(&s_m, 1u);
          if (p < g.k) best[p] = key;
        }
      });
      __syncthreads();
      const long long qn = MT == MT_L2 ? (long long)reinterpret_cast<const int32_t*>(g.qnorm)[qi] : 0ll;
      for (uint32_t i = tid; i < g.k; i += GT_FT) {
        const uint64_t ki = best[i];
        uint32_t r = 0;
        for (uint32_t j = 0; j < g.k; j++) r += best[j] < ki;
        g.out_ids[(uint64_t)qi * g.k + r] = (uint32_t)ki;
        g.out_d[(uint64_t)qi * g.k + r] = (double)((long long)(int32_t)((uint32_t)(ki >> 32) ^ 0x80000000u) + qn);
      }
    }
  } else {
    const float* q = reinterpret_cast<const float*>(g.queries + (uint64_t)qi * g.stride);
    double lim = 0.0;
    if (!bad) {
      const double u = 5.9604644775390625e-08;  // 2^-24
      const double qn = sqrt((double)reinterpret_cast<const float*>(g.qnorm)[qi]) * (1.0 + 1e-6);
      const double B = __longlong_as_double((long long)g.scale->bmax) * (1.0 + 1e-6);
      // 2^-37 sqrt(d): half precision's smallest step below the batch's (the points') largest value, twice
      const double step = 7.275957614183426e-12 * sqrt((double)g.d);
      const double acc = ((6.0 * g.d + (MT == MT_L2 ? 11.0 : 10.0)) * u * qn +
                          step * ((double)__uint_as_float(g.scale->q_max) + qn)) * B;
      const double bound = MT == MT_L2 ? 2.0 * (4.0 * u * B * B + 2.0 * acc) + 1e-12 : 2.0 * acc + 1e-12;
      lim = (double)float_of(v) + 2.0 * bound;
      const bool cut = thr != 0xFFFFFFFFu;  // no slice dropped anything otherwise
      bad = !(qn < GT_HUGE && B < GT_HUGE) || (cut && !((double)float_of(thr) > lim)) || !(lim == lim);
    }
    double* d64 = reinterpret_cast<double*>(fsm);
    uint32_t* idv = reinterpret_cast<uint32_t*>(d64 + GT_FCAP);
    if (!bad)
      each_key([&](uint64_t key) {
        const uint32_t h = (uint32_t)(key >> 32);
        if (h <= thr && (double)float_of(h) <= lim) {
          const uint32_t p = atomicAdd(&s_m, 1u);
          if (p < GT_FCAP) idv[p] = (uint32_t)key;
        }
      });
    __syncthreads();
    const uint32_t nc = s_m;
    bad = bad || nc > GT_FCAP;
    if (!bad) {
      for (uint32_t i = tid; i < nc; i += GT_FT)
        d64[i] = exact_dist<DT_F32, MT>(g.points + (uint64_t)idv[i] * g.stride, reinterpret_cast<const uint8_t*>(q), (int)g.d);
      __syncthreads();
      for (uint32_t i = tid; i < nc; i += GT_FT) {
        uint32_t r = 0;
        for (uint32_t j = 0; j < nc; j++) r += dless(d64[j], idv[j], d64[i], idv[i]);
        if (r < g.k) {
          g.out_ids[(uint64_t)qi * g.k + r] = idv[i];
          g.out_d[(uint64_t)qi * g.k + r] = d64[i];
        }
      }
    }
  }
  if (bad && tid == 0) g.fallback[atomicAdd(g.nfallback, 1u)] = qi;
}

// ------------------------------------------------------------ host side

static uint32_t gt_kch(const pann_index* idx) {
  return (uint32_t)((idx->d * (idx->dtype == DT_F32 ? 2ull : 1ull) + GT_KB - 1) / GT_KB);
}

// Queries per block (N), slices of the points and ring stages: N is at most
// 256 (two accumulators fill the tensor memory) and what shared memory holds
// beside a ring of at least three stages; among the N (multiples of 64) and
// slice counts the pair with the shortest schedule on the SMs is taken, the
// work of a block being its tiles x N. For 10K queries on 148 SMs that is
// N = 256, 40 x 3 blocks. Returns false if not even 64 queries fit.
static bool gt_shape(const pann_index* idx, uint32_t nq, uint32_t tiles, uint32_t C, uint32_t* N, uint32_t* slices,
                     uint32_t* stages) {
  const uint32_t PL = idx->dtype == DT_F32 ? 2 : 1, kch = gt_kch(idx);
  const uint32_t smax = std::max<uint32_t>(1, std::min<uint32_t>({(uint32_t)idx->sm_count, GT_CAP / C, tiles}));
  double best = 1e300;
  for (uint32_t n = 64; n <= 256; n += 64) {
    if (n > 64 && n >= nq + 64) break;
    if (gt_layout(n, kch, PL, 3).total > idx->smem_optin) break;
    const uint64_t qt = (nq + n - 1) / n;
    for (uint32_t s = 1; s <= smax; s++) {
      const uint64_t waves = (qt * s + idx->sm_count - 1) / idx->sm_count;
      // a tile costs its columns plus a fixed part (barriers, the accumulator's hand-over); every query's threshold
      // falls anew in each slice, about 800 appends at the price of one to two scores of the tile's 128 each
      const double t = (double)waves * ((double)((tiles + s - 1) / s) * (n + 32.0) + 1000.0 * n);
      if (t < best) {
        best = t;
        *N = n;
        *slices = s;
      }
    }
  }
  if (best >= 1e300) return false;
  *stages = 3;
  while (*stages < 8 && gt_layout(*N, kch, PL, *stages + 1).total <= idx->smem_optin) (*stages)++;
  return true;
}

template <int DT, int MT, int KPL>
static cudaError_t gt_launch_mma(const GtMma& g, uint32_t qtiles, size_t smem, cudaStream_t st) {
  auto k = gt_mma_kernel<DT, MT, KPL>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_attr_max());
  if (e != cudaSuccess) return e;
  k<<<dim3(qtiles, g.slices), GT_THREADS, smem, st>>>(g);
  return cudaGetLastError();
}

template <int DT, int MT>
static cudaError_t gt_run_dm(const pann_index* idx, GtMma m, GtFinal f, uint32_t qtiles, uint64_t seg_rows,
                             uint8_t* a_img, void* pnorm, GtScale* sc, const float4* centre, size_t smem_mma,
                             size_t smem_fin, cudaStream_t st) {
  for (uint64_t r0 = 0; r0 < idx->n; r0 += seg_rows) {
    const uint64_t rows = std::min<uint64_t>(seg_rows, idx->n - r0);
    const uint64_t total = (rows + GT_ROWS - 1) / GT_ROWS * GT_ROWS;
    gt_image_kernel<DT><<<(int)std::min<uint64_t>((total / 8 + 7) / 8, 16ull * idx->sm_count), 256, 0, st>>>(
        idx->d_points + r0 * idx->stride, idx->stride, idx->d, rows, total, GT_ROWS, m.kch, sc, centre, 0, a_img,
        pnorm, &sc->bmax);
    m.n_seg = (uint32_t)rows;
    m.ntiles = (uint32_t)(total / GT_ROWS);
    m.id0 = (uint32_t)r0;
    cudaError_t e;
    if (m.CB == 256) e = gt_launch_mma<DT, MT, 8>(m, qtiles, smem_mma, st);
    else if (m.CB == 448) e = gt_launch_mma<DT, MT, 14>(m, qtiles, smem_mma, st);
    else e = gt_launch_mma<DT, MT, 22>(m, qtiles, smem_mma, st);
    if (e != cudaSuccess) return e;
  }
  auto k = gt_final_kernel<DT, MT>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_attr_max() - 1024);
  if (e != cudaSuccess) return e;
  k<<<m.nq, GT_FT, smem_fin, st>>>(f);
  return cudaGetLastError();
}

// Exact top-k of the nq queries at dq (device rows of idx->stride bytes);
// fallback lists the queries left to the plain kernel (their count in
// *nfallback). PANN_EINVAL (and nothing done) if the shape does not fit.
int groundtruth_tensor(pann_index* idx, const uint8_t* dq, uint32_t nq, uint32_t k, uint32_t* dids, double* dd,
                       std::vector<uint32_t>* fallback, cudaStream_t st) {
  const bool F = idx->dtype == DT_F32;
  const uint32_t PL = F ? 2 : 1, kch = gt_kch(idx);
  // float: the margin test needs room above the k-th score; 8-bit scores are exact
  const uint32_t need = F ? std::max<uint32_t>(64, 2 * k) : std::max<uint32_t>(64, k);
  if (need > 512 || idx->n > 0x7FFFFFFFull - GT_ROWS) return PANN_EINVAL;
  const uint32_t CB = need <= 64 ? 256 : need <= 256 ? 448 : 704;  // C + GT_CUT + a tile
  const uint32_t C = need;
  // point images in segments of at most 128 MB, queries in chunks whose buffers stay within 128 MB
  const uint64_t row_img = (uint64_t)kch * PL * GT_KB;
  const uint64_t seg_rows = std::max<uint64_t>(GT_ROWS, (128ull << 20) / row_img / GT_ROWS * GT_ROWS);
  const uint64_t seg = std::min<uint64_t>(seg_rows, (idx->n + GT_ROWS - 1) / GT_ROWS * GT_ROWS);
  uint32_t N = 0, slices = 0, stages = 0;
  uint32_t qc = nq;
  const uint32_t tiles = (uint32_t)((idx->n + GT_ROWS - 1) / GT_ROWS);
  for (;;) {
    if (!gt_shape(idx, qc, tiles, C, &N, &slices, &stages)) return PANN_EINVAL;
    if (qc <= 1024 || (uint64_t)qc * slices * CB * 8 <= (128ull << 20)) break;
    qc = (qc + 1) / 2;
  }
  const uint32_t qtiles = (qc + N - 1) / N;
  const size_t smem_mma = gt_layout(N, kch, PL, stages).total;
  const uint32_t cap = slices * (C + GT_CUT);
  const size_t smem_fin = 4ull * cap + (F ? 12ull * GT_FCAP : 8ull * k);
  // workspace
  size_t o = 0;
  auto take = [&](size_t b) {
    const size_t at = o;
    o += (b + 255) & ~size_t(255);
    return at;
  };
  const size_t o_sc = take(sizeof(GtScale) + 64), o_a = take(seg * row_img), o_pn = take(4 * seg),
               o_b = take((size_t)qtiles * N * row_img), o_qn = take(4ull * qtiles * N),
               o_cand = take(8ull * qc * slices * CB), o_cnt = take(4ull * qc * slices), o_thr = take(4ull * qc),
               o_fb = take(4ull * qc), o_cen = take(F ? idx->stride : 0),
               o_part = take(F ? 5ull * GT_CEN_PARTS * idx->stride : 0);
  PANN_CUDA(idx->gt.ensure(o));
  uint8_t* w = idx->gt.as<uint8_t>();
  GtScale* sc = reinterpret_cast<GtScale*>(w + o_sc);
  uint32_t* flags = reinterpret_cast<uint32_t*>(w + o_sc + sizeof(GtScale));  // [0] error, [1] fallbacks
  for (uint32_t c0 = 0; c0 < nq; c0 += qc) {
    const uint32_t nc = std::min(qc, nq - c0);
    const uint8_t* q = dq + (uint64_t)c0 * idx->stride;
    PANN_CUDA(cudaMemsetAsync(w + o_sc, 0, sizeof(GtScale) + 64, st));
    PANN_CUDA(cudaMemsetAsync(w + o_cnt, 0, 4ull * qc * slices, st));
    PANN_CUDA(cudaMemsetAsync(w + o_thr, 0xFF, 4ull * qc, st));
    const float4* centre = F ? reinterpret_cast<const float4*>(w + o_cen) : nullptr;
    const float4* qcentre = idx->metric == MT_L2 ? centre : nullptr;
    if (F) {
      GtCentre gc;
      gc.cols = (uint32_t)(idx->stride / 4);
      gc.sum = reinterpret_cast<double*>(w + o_part);
      gc.sq = gc.sum + (size_t)GT_CEN_PARTS * gc.cols;
      gc.cnt = reinterpret_cast<uint32_t*>(gc.sq + (size_t)GT_CEN_PARTS * gc.cols);
      gc.centre = reinterpret_cast<float*>(w + o_cen);
      gt_centre_kernel<<<dim3((gc.cols + 31) / 32, GT_CEN_PARTS), 256, 0, st>>>(idx->d_points, idx->stride, idx->n, gc, sc);
      gt_absmax_kernel<<<4 * idx->sm_count, 256, 0, st>>>(reinterpret_cast<const float4*>(idx->d_points),
                                                          idx->n * idx->nchunks, idx->nchunks, centre, &sc->pt_max);
      gt_absmax_kernel<<<idx->sm_count, 256, 0, st>>>(reinterpret_cast<const float4*>(q), (uint64_t)nc * idx->nchunks,
                                                      idx->nchunks, qcentre, &sc->q_max);
    }
    const uint64_t qtotal = (uint64_t)qtiles * N;
    const int qb = (int)std::min<uint64_t>((qtotal / 8 + 7) / 8, 16ull * idx->sm_count);
    if (F)
      gt_image_kernel<DT_F32><<<qb, 256, 0, st>>>(q, idx->stride, idx->d, nc, qtotal, N, kch, sc, qcentre, 1, w + o_b,
                                                  w + o_qn, nullptr);
    else if (idx->dtype == DT_U8)
      gt_image_kernel<DT_U8><<<qb, 256, 0, st>>>(q, idx->stride, idx->d, nc, qtotal, N, kch, sc, nullptr, 1, w + o_b,
                                                 w + o_qn, nullptr);
    else
      gt_image_kernel<DT_I8><<<qb, 256, 0, st>>>(q, idx->stride, idx->d, nc, qtotal, N, kch, sc, nullptr, 1, w + o_b,
                                                 w + o_qn, nullptr);
    PANN_CUDA(cudaGetLastError());
    GtMma m{};
    m.a_img = w + o_a;
    m.pnorm = w + o_pn;
    m.b_img = w + o_b;
    m.nq = nc;
    m.N = N;
    m.kch = kch;
    m.ksteps = (uint32_t)((idx->d * (F ? 2ull : 1ull) + 31) / 32);
    m.slices = slices;
    m.stages = stages;
    m.C = C;
    m.CB = CB;
    m.cand = reinterpret_cast<uint64_t*>(w + o_cand);
    m.count = reinterpret_cast<uint32_t*>(w + o_cnt);
    m.thr = reinterpret_cast<uint32_t*>(w + o_thr);
    m.scale = sc;
    m.err = flags;
    GtFinal f{};
    f.cand = m.cand;
    f.count = m.count;
    f.thr = m.thr;
    f.slices = slices;
    f.CB = CB;
    f.cap = cap;
    f.k = k;
    f.points = idx->d_points;
    f.stride = idx->stride;
    f.d = idx->d;
    f.queries = q;
    f.qnorm = w + o_qn;
    f.scale = sc;
    f.out_ids = dids + (uint64_t)c0 * k;
    f.out_d = dd + (uint64_t)c0 * k;
    f.fallback = reinterpret_cast<uint32_t*>(w + o_fb);
    f.nfallback = flags + 1;
    cudaError_t e = cudaErrorInvalidValue;
    const uint32_t qt = (nc + N - 1) / N;
#define PANN_GT_CASE(DT, MT)                                                                                       \
    if (idx->dtype == DT && idx->metric == MT)                                                                     \
      e = gt_run_dm<DT, MT>(idx, m, f, qt, seg, w + o_a, w + o_pn, sc, centre, smem_mma, smem_fin, st);
    PANN_GT_CASE(DT_U8, MT_L2)
    PANN_GT_CASE(DT_U8, MT_IP)
    PANN_GT_CASE(DT_I8, MT_L2)
    PANN_GT_CASE(DT_I8, MT_IP)
    PANN_GT_CASE(DT_F32, MT_L2)
    PANN_GT_CASE(DT_F32, MT_IP)
#undef PANN_GT_CASE
    if (e != cudaSuccess) return cuda_fail(e, "groundtruth kernels");
    uint32_t hf[2] = {0, 0};
    PANN_CUDA(cudaMemcpyAsync(hf, flags, 8, cudaMemcpyDeviceToHost, st));
    PANN_CUDA(cudaStreamSynchronize(st));
    if (hf[0]) return fail(PANN_ETIMEOUT, "a wait of the groundtruth kernel ran out");
    if (hf[1]) {
      const size_t at = fallback->size();
      fallback->resize(at + hf[1]);
      PANN_CUDA(cudaMemcpyAsync(fallback->data() + at, w + o_fb, 4ull * hf[1], cudaMemcpyDeviceToHost, st));
      PANN_CUDA(cudaStreamSynchronize(st));
      for (size_t i = at; i < fallback->size(); i++) (*fallback)[i] += c0;
    }
  }
  return PANN_OK;
}

}  // namespace pann
