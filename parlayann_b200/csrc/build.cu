// Vamana batch-insertion build on the device: knn_index::build_index and
// batch_insert (algorithms/vamana/index.h:150-319).
//
// Per batch [floor, ceiling) of the insertion order, against the pre-batch graph:
//   1. search      beam search from point 0 for every inserted point (build
//                  mode of the search kernel: the query is the point itself,
//                  which is skipped as a neighbour; the visited list is kept)
//                                                        (index.h:247-264)
//   2. prune       candidates = visited list + current out-neighbours with
//                  their distances, sorted by (dist, id), then the greedy
//                  alpha-pruning of robustPrune (index.h:63-120; prune.cuh),
//                  written straight into the graph rows (index.h:265-273)
//   3. reverse     (new neighbour, inserted point) pairs, stable radix sort by
//                  neighbour = group_by_key (index.h:281-285); per target,
//                  append without repeats when it fits, else robustPrune of
//                  the grouped candidates + current neighbours (index.h:292-303)
// The batch schedule is the reference's prefix doubling (index.h:206-240).
#include <cuda_runtime.h>
#include <cub/cub.cuh>
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "index.cuh"
#include "prune.cuh"
#include "rowscore.cuh"
#include "tiers.cuh"

namespace pann {

// Insertion order: indices sorted by splitmix64(seed + i) (the same keys the
// oracle's ParlayLib shim uses for parlay::random_permutation, index.h:212).
__host__ __device__ inline uint64_t splitmix64(uint64_t x) {
  x += 0x9e3779b97f4a7c15ULL;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
  return x ^ (x >> 31);
}

__global__ void perm_keys_kernel(uint64_t* keys, uint32_t* idx, uint64_t n, uint64_t seed) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    keys[i] = splitmix64(seed + i);
    idx[i] = (uint32_t)i;
  }
}

// Job i assembles candidate keys for point pts[i] into keys[begin[i] ..):
//   provided (dist,id) keys (src_keys, src_n) or ids (src_ids, src_n) whose
//   distance to the point is computed here, then the point's current
//   out-neighbours with their distances (robustPrune add = true, index.h:72-77).
template <int DT, int MT>
__global__ void __launch_bounds__(128) assemble_kernel(const uint8_t* __restrict__ points, uint64_t stride, int d,
                                                       int nchunks, const uint32_t* __restrict__ graph, uint32_t R,
                                                       uint32_t njobs, const uint32_t* __restrict__ pts,
                                                       const uint64_t* __restrict__ src_keys, uint32_t src_keys_stride,
                                                       const uint32_t* __restrict__ src_ids,
                                                       const uint32_t* __restrict__ src_off,
                                                       const uint32_t* __restrict__ src_n,
                                                       const uint32_t* __restrict__ seg_begin, uint32_t* seg_end,
                                                       uint64_t* keys, unsigned long long* dist_cmps) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  uint8_t* qs = smem + (size_t)warp * stride;
  for (uint32_t job = blockIdx.x * wpb + warp; job < njobs; job += gridDim.x * wpb) {
    const uint32_t p = pts[job];
    stage_query<DT, MT>(qs, points + (uint64_t)p * stride, nchunks, lane);
    __syncwarp();
    int32_t qq = 0;
    if (DT != DT_F32 && MT == MT_L2) qq = sq_norm_int<DT>(reinterpret_cast<const uint4*>(qs), nchunks);
    uint64_t* out = keys + seg_begin[job];
    uint32_t m = src_n[job];
    uint32_t cmps = 0;
    if (src_keys) {
      const uint64_t* sk = src_keys + (uint64_t)job * src_keys_stride;
      for (uint32_t t = lane; t < m; t += 32) out[t] = sk[t];
    } else {
      const uint32_t* si = src_ids + src_off[job];
      for (uint32_t t = lane; t < m; t += 32) {
        uint32_t c = si[t];
        float dd = point_dist<DT, MT>(points + (uint64_t)c * stride, qs, d, nchunks, qq);
        out[t] = make_key(dd, c);
      }
      cmps += m;  // robustPrune id overload (index.h:131-134)
    }
    const uint32_t* g = graph + (uint64_t)p * R;
    uint32_t deg = 0;
    for (uint32_t b = 0; b < R; b += 32) {
      uint32_t j = b + lane;
      uint32_t v = j < R ? __ldg(g + j) : PANN_PAD;
      bool ok = v != PANN_PAD;
      unsigned msk = __ballot_sync(0xFFFFFFFFu, ok);
      if (ok) {
        float dd = point_dist<DT, MT>(points + (uint64_t)v * stride, qs, d, nchunks, qq);
        out[m + b + __popc(msk & ((1u << lane) - 1))] = make_key(dd, v);
      }
      deg += __popc(msk);
    }
    cmps += deg;
    if (lane == 0) {
      seg_end[job] = seg_begin[job] + m + deg;
      atomicAdd(dist_cmps, (unsigned long long)cmps);
    }
    __syncwarp();
  }
}

// Reverse-edge pairs: key = new neighbour (n for empty slots, so that the sort
// needs only n's bits), value = inserted point.
__global__ void reverse_pairs_kernel(const uint32_t* __restrict__ graph, uint32_t R, const uint32_t* __restrict__ pts,
                                     uint32_t B, uint32_t n, uint32_t* kout, uint32_t* vout) {
  uint64_t total = (uint64_t)B * R;
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t i = (uint32_t)(t / R), j = (uint32_t)(t - (uint64_t)i * R);
    uint32_t p = pts[i];
    kout[t] = min(graph[(uint64_t)p * R + j], n);
    vout[t] = p;
  }
}

// Per group (target j with m new in-edges): append without repeats when
// m + deg(j) <= R (add_neighbors_without_repeats, index.h:140-146,294-297),
// else a robustPrune job (index.h:298-301) of one of four classes:
//   0 few fresh candidates (the new ones and the row's entries since its last
//     prune): their distance table fits reprune_kernel's dcap
//   1 up to cap1 candidates: prune_lazy_kernel, a warp per job
//   2 up to cap2: prune_block_kernel, a block per job
//   3 more: assembled and sorted in global memory first
// Classes 0 and 1 share one job array, filled from its two ends (jobs_cap
// entries); classes 2 and 3 have big_cap entries each. One warp per group.
struct ClassifyArgs {
  uint32_t* graph;
  uint32_t R, n;
  uint32_t* nclean;
  const uint32_t *uniq, *counts, *offs, *num_runs, *vals;
  uint32_t *job_pts, *job_off, *job_n;  // classes 0 and 1
  uint32_t jobs_cap;
  uint32_t *big_pts, *big_off, *big_n;  // classes 2, then 3 at big_cap
  uint32_t big_cap;
  uint32_t* big_begin;                  // class 3: segment starts
  uint32_t* njobs;                      // four counts
  unsigned long long *seg_total, *cands_total;
  uint32_t cap0, dcap, cap1, cap2;
};
__global__ void reverse_classify_kernel(ClassifyArgs a) {
  const int lane = threadIdx.x & 31;
  const unsigned FULL = 0xFFFFFFFFu;
  const uint32_t runs = *a.num_runs;
  const uint32_t R = a.R;
  for (uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < runs; r += (gridDim.x * blockDim.x) >> 5) {
    const uint32_t tgt = a.uniq[r];
    if (tgt >= a.n) continue;
    const uint32_t m = a.counts[r], off = a.offs[r];
    uint32_t* row = a.graph + (uint64_t)tgt * R;
    uint32_t deg = 0;
    for (uint32_t b = 0; b < R; b += 32) {
      uint32_t j = b + lane;
      deg += __popc(__ballot_sync(FULL, j < R && row[j] != PANN_PAD));
    }
    const uint32_t clean = min(deg, a.nclean[tgt]);
    if (m + deg <= R) {
      // old neighbours not among the new candidates, in order
      uint32_t keep_cnt = 0, kept_clean = 0;
      uint32_t oldv[32];  // up to 1024 / 32 per lane
      bool keepv[32];
      int nslot = (int)((R + 31) / 32);
      for (int s = 0; s < nslot; s++) {
        uint32_t j = s * 32 + lane;
        uint32_t v = (j < deg) ? row[j] : PANN_PAD;
        bool keep = v != PANN_PAD;
        if (keep)
          for (uint32_t t = 0; t < m; t++)
            if (a.vals[off + t] == v) { keep = false; break; }
        oldv[s] = v;
        keepv[s] = keep;
        kept_clean += __popc(__ballot_sync(FULL, keep && j >= deg - clean));
      }
      __syncwarp();
      for (uint32_t t = lane; t < m; t += 32) row[t] = a.vals[off + t];
      for (int s = 0; s < nslot; s++) {
        unsigned msk = __ballot_sync(FULL, keepv[s]);
        if (keepv[s]) row[m + keep_cnt + __popc(msk & ((1u << lane) - 1))] = oldv[s];
        keep_cnt += __popc(msk);
      }
      for (uint32_t j = m + keep_cnt + lane; j < R; j += 32) row[j] = PANN_PAD;
      if (lane == 0) a.nclean[tgt] = kept_clean;
      __syncwarp();
    } else if (lane == 0) {
      const uint32_t tot = m + deg;
      const uint64_t table = (uint64_t)(tot - clean) * tot;
      const int c = tot <= a.cap0 && table <= a.dcap ? 0 : tot <= a.cap1 ? 1 : tot <= a.cap2 ? 2 : 3;
      const uint32_t t = atomicAdd(a.njobs + c, 1u);
      atomicAdd(a.cands_total, (unsigned long long)tot);
      if (c < 2) {
        const uint32_t at = c == 0 ? t : a.jobs_cap - 1 - t;
        a.job_pts[at] = tgt;
        a.job_off[at] = off;
        a.job_n[at] = m;
      } else {
        const uint32_t at = c == 2 ? t : a.big_cap + t;
        a.big_pts[at] = tgt;
        a.big_off[at] = off;
        a.big_n[at] = m;
        // a segment of exactly m candidates + deg current neighbours, packed by an atomic cursor
        if (c == 3) a.big_begin[t] = (uint32_t)atomicAdd(a.seg_total, (unsigned long long)tot);
      }
    }
  }
}

// Final per-vertex sort by distance (index.h:180-185); ties by id.
template <int DT, int MT>
__global__ void __launch_bounds__(128) sort_neighbors_kernel(const uint8_t* __restrict__ points, uint64_t stride, int d,
                                                             int nchunks, uint32_t* graph, uint32_t R, uint64_t n) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  constexpr uint32_t SCR = row_score_scratch<DT>();
  uint8_t* qs = smem + (size_t)warp * (stride + SCR + 16ull * R);
  uint8_t* stg = qs + stride;
  uint64_t* kin = reinterpret_cast<uint64_t*>(stg + SCR);
  uint64_t* kout = kin + R;
  for (uint64_t v = (uint64_t)blockIdx.x * wpb + warp; v < n; v += (uint64_t)gridDim.x * wpb) {
    stage_query<DT, MT>(qs, points + v * stride, nchunks, lane);
    __syncwarp();
    int32_t qq = 0;
    if (DT != DT_F32 && MT == MT_L2) qq = sq_norm_int<DT>(reinterpret_cast<const uint4*>(qs), nchunks);
    uint32_t* row = graph + v * R;
    uint32_t deg = 0;
    for (uint32_t b = 0; b < R; b += 32) {  // a row's live entries are a prefix
      const uint32_t j = b + lane;
      const uint32_t u = j < R ? row[j] : PANN_PAD;
      const unsigned msk = __ballot_sync(0xFFFFFFFFu, u != PANN_PAD);
      if (!msk) break;
      // Points[i].distance(Points[j]): the same float whichever of the two is the staged operand
      const float dd = warp_score_rows<DT, MT>(points, stride, nchunks, u, __popc(msk), qs, stg, qq, lane);
      if (u != PANN_PAD) kin[j] = make_key(dd, u);
      deg += __popc(msk);
    }
    __syncwarp();
    for (uint32_t i = lane; i < deg; i += 32) {
      uint64_t ki = kin[i];
      uint32_t r = 0;
      for (uint32_t j = 0; j < deg; j++) r += kin[j] < ki;
      kout[r] = ki;
    }
    __syncwarp();
    for (uint32_t i = lane; i < deg; i += 32) row[i] = key_id(kout[i]);
    __syncwarp();
  }
}

// ------------------------------------------------------------ host side

// Batch schedule of batch_insert (index.h:206-240), same double arithmetic.
static void batch_schedule(uint64_t n, uint64_t m, std::vector<uint64_t>& fl, std::vector<uint64_t>& ce) {
  const double base = 2.0, max_fraction = 0.02;
  uint64_t max_batch = std::min<uint64_t>((uint64_t)(max_fraction * (double)(float)n), 1000000ull);
  if (max_batch == 0) max_batch = n;
  uint64_t count = 0, inc = 0;
  while (count < m) {
    uint64_t f, c;
    if (std::pow(base, (double)inc) <= (double)max_batch) {
      f = (uint64_t)std::pow(base, (double)inc) - 1;
      c = std::min<uint64_t>((uint64_t)std::pow(base, (double)(inc + 1)) - 1, m);
      count = c;
    } else {
      f = count;
      c = std::min<uint64_t>(count + max_batch, m);
      count += max_batch;
    }
    fl.push_back(f);
    ce.push_back(c);
    inc++;
  }
}

// PANN_PRUNE_KERNEL=block: every prune on prune_block_kernel, a block per job
// (the class of jobs with many candidates; the same graph).
static bool prune_all_blocks() {
  static const bool block = [] {
    const char* e = std::getenv("PANN_PRUNE_KERNEL");
    return e && !std::strcmp(e, "block");
  }();
  return block;
}

// Blocks of a grid that fills the device once, at most `want`.
template <typename K>
static int fill_grid(const pann_index* idx, K k, int threads, size_t smem, uint64_t want) {
  int occ = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, threads, smem) != cudaSuccess || occ <= 0) occ = 1;
  return (int)std::max<uint64_t>(1, std::min<uint64_t>(want, (uint64_t)occ * idx->sm_count));
}

// Warps per block of a warp-per-job kernel needing `per_warp` shared bytes a warp; 0 if not even one fits.
static int prune_wpb(const pann_index* idx, size_t per_warp) {
  for (int w = 4; w >= 1; w >>= 1)
    if (per_warp * w <= idx->smem_optin) return w;
  return 0;
}

template <int DT, int MT>
static cudaError_t launch_lazy(const pann_index* idx, const PruneArgs& a, uint64_t max_jobs, cudaStream_t st) {
  auto k = prune_lazy_kernel<DT, MT>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_attr_max());
  if (e != cudaSuccess) return e;
  const size_t pw = prune_warp_bytes(idx->stride, a.cap, row_score_scratch<DT>());
  const int wpb = prune_wpb(idx, pw);
  if (wpb == 0) return cudaErrorInvalidValue;
  k<<<fill_grid(idx, k, 32 * wpb, pw * wpb, (max_jobs + wpb - 1) / wpb), 32 * wpb, pw * wpb, st>>>(a);
  return cudaGetLastError();
}

template <int DT, int MT>
static cudaError_t launch_reprune(const pann_index* idx, const PruneArgs& a, uint64_t max_jobs, cudaStream_t st) {
  auto k = reprune_kernel<DT, MT>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_attr_max());
  if (e != cudaSuccess) return e;
  const size_t pw = prune_warp_bytes(idx->stride, a.cap, row_score_scratch<DT>()) + 4ull * a.dcap;
  const int wpb = prune_wpb(idx, pw);
  if (wpb == 0) return cudaErrorInvalidValue;
  k<<<fill_grid(idx, k, 32 * wpb, pw * wpb, (max_jobs + wpb - 1) / wpb), 32 * wpb, pw * wpb, st>>>(a);
  return cudaGetLastError();
}

template <int DT, int MT, bool GATHERED>
static cudaError_t launch_block(const pann_index* idx, const PruneArgs& a, const PruneSegs& sg, uint64_t max_jobs,
                                cudaStream_t st) {
  auto k = prune_block_kernel<DT, MT, GATHERED>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_attr_max() - 256);
  if (e != cudaSuccess) return e;
  const size_t sm = prune_block_bytes(idx->stride, GATHERED ? 0 : a.cap, row_score_scratch<DT>());
  if (sm > (size_t)smem_attr_max() - 256) return cudaErrorInvalidValue;
  k<<<fill_grid(idx, k, PRUNE_BLOCK, sm, max_jobs), PRUNE_BLOCK, sm, st>>>(a, sg);
  return cudaGetLastError();
}

template <typename F>
static cudaError_t dispatch_dm(int dtype, int metric, F&& f) {
  if (dtype == DT_U8 && metric == MT_L2) return f(std::integral_constant<int, DT_U8>(), std::integral_constant<int, MT_L2>());
  if (dtype == DT_U8 && metric == MT_IP) return f(std::integral_constant<int, DT_U8>(), std::integral_constant<int, MT_IP>());
  if (dtype == DT_I8 && metric == MT_L2) return f(std::integral_constant<int, DT_I8>(), std::integral_constant<int, MT_L2>());
  if (dtype == DT_I8 && metric == MT_IP) return f(std::integral_constant<int, DT_I8>(), std::integral_constant<int, MT_IP>());
  if (dtype == DT_F32 && metric == MT_L2) return f(std::integral_constant<int, DT_F32>(), std::integral_constant<int, MT_L2>());
  if (dtype == DT_F32 && metric == MT_IP) return f(std::integral_constant<int, DT_F32>(), std::integral_constant<int, MT_IP>());
  return cudaErrorInvalidValue;
}

// Device memory of one build: the fixed arrays carved out of one allocation
// (23 allocations cost milliseconds, and on a busy host far more), the visited
// lists (regrown if a search visits more), and the segment buffers of the rare
// prunes that are sorted in global memory.
struct BuildBufs {
  DevBuf fixed, vis_keys, seg_a, seg_b, seg_tmp, seg_se;
  void release() {
    for (DevBuf* b : {&fixed, &vis_keys, &seg_a, &seg_b, &seg_tmp, &seg_se}) b->release();
  }
};

__global__ void iota_begin_kernel(uint32_t* begin, uint32_t n, uint32_t cap) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) begin[i] = i * cap;
}

__global__ void status_or_kernel(const uint32_t* status, uint32_t n, uint32_t* out) {
  uint32_t acc = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) acc |= status[i];
  for (int o = 16; o; o >>= 1) acc |= __shfl_xor_sync(0xFFFFFFFFu, acc, o);
  if ((threadIdx.x & 31) == 0 && acc) atomicOr(out, acc);
}
// One batch's search counters: queries whose status has `flag`, comparisons (into c64[0] and c64[3]) and visits (c64[1]).
__global__ void batch_sums_kernel(const uint32_t* status, uint32_t flag, const uint32_t* cmps, const uint32_t* vis,
                                  uint32_t n, uint32_t* flagged, unsigned long long* c64) {
  unsigned long long c = 0, v = 0;
  uint32_t f = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    f += (status[i] & flag) ? 1u : 0u;
    c += cmps[i];
    v += vis[i];
  }
  for (int o = 16; o; o >>= 1) {
    f += __shfl_xor_sync(0xFFFFFFFFu, f, o);
    c += __shfl_xor_sync(0xFFFFFFFFu, c, o);
    v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (f) atomicAdd(flagged, f);
    if (c) { atomicAdd(c64, c); atomicAdd(c64 + 3, c); }
    if (v) atomicAdd(c64 + 1, v);
  }
}
// Sum of end[i] - begin[i] (segment lengths).
__global__ void seg_len_sum_kernel(const uint32_t* begin, const uint32_t* end, uint32_t n, unsigned long long* out) {
  unsigned long long acc = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) acc += end[i] - begin[i];
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
  if ((threadIdx.x & 31) == 0 && acc) atomicAdd(out, acc);
}
// Live degrees of the rows rows[i], summed.
__global__ void degree_sum_kernel(const uint32_t* graph, uint32_t R, const uint32_t* rows, uint32_t n,
                                  unsigned long long* out) {
  unsigned long long acc = 0;
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < (uint64_t)n * R;
       e += (uint64_t)gridDim.x * blockDim.x)
    acc += graph[(uint64_t)rows[e / R] * R + e % R] != PANN_PAD;
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
  if ((threadIdx.x & 31) == 0 && acc) atomicAdd(out, acc);
}

}  // namespace pann

using namespace pann;

extern "C" int pann_build(pann_index* idx, const pann_build_params* bp, const uint32_t* perm, pann_build_stats* stats) {
  if (!idx || !bp) return fail(PANN_EINVAL, "index or build params is NULL");
  if (!idx->points_set) return fail(PANN_EINVAL, "index has no points");
  if (bp->R != idx->R) return fail(PANN_EINVAL, "build R must equal the index's max degree");
  if (bp->L == 0 || bp->num_passes < 1 || !(bp->alpha > 0.0))
    return fail(PANN_EINVAL, "build needs L > 0, num_passes >= 1, alpha > 0");
  const uint64_t n = idx->n;
  const uint32_t R = idx->R;
  cudaStream_t st = idx->stream;
  if (perm)
    for (uint64_t i = 0; i < n; i++)
      if ((uint64_t)perm[i] >= n)
        return fail(PANN_EINVAL, "ERROR: invalid point " + std::to_string(perm[i]) + " given to batch_insert");

  BuildBufs bb;
  auto cleanup = [&]() { bb.release(); };
  auto cu = [&](cudaError_t e, const char* what) -> int {
    if (e == cudaSuccess) return PANN_OK;
    cleanup();
    return cuda_fail(e, what);
  };
#define BCUDA(call) do { int _rc = cu((call), #call); if (_rc) return _rc; } while (0)

  cudaEvent_t ev0, ev1, ea, eb, ec, ed;
  cudaEventCreate(&ev0); cudaEventCreate(&ev1);
  cudaEventCreate(&ea); cudaEventCreate(&eb); cudaEventCreate(&ec); cudaEventCreate(&ed);
  double t_search = 0, t_prune = 0, t_rev = 0;
  BCUDA(cudaEventRecord(ev0, st));

  // empty graph (Graph(maxDeg, n) is zeroed: every degree 0)
  BCUDA(cudaMemsetAsync(idx->d_graph, 0xFF, sizeof(uint32_t) * R * n, st));

  std::vector<uint64_t> fl, ce;
  batch_schedule(n, n, fl, ce);
  uint64_t maxB = 0;
  for (size_t b = 0; b < fl.size(); b++) maxB = std::max(maxB, ce[b] - fl[b]);
  const uint64_t pairs_cap = maxB * R;
  uint32_t vis_cap = std::max<uint32_t>(2 * bp->L + 64, 128);
  const int dtype = idx->dtype, metric = idx->metric;
  const uint64_t stride = idx->stride;
  const int d = (int)idx->d, nch = (int)idx->nchunks;
  const int wpb = 4;
  const uint32_t scratch = row_score_scratch_rt(dtype);

  // Classes of the reverse-edge prunes (ClassifyArgs). The distance table of
  // class 0 is 6 KB a warp (R 64: 20 fresh candidates), which leaves 12 warps
  // an SM; class 1 ends at three rows' worth of candidates, where one warp
  // starts to outlast the rest of the batch.
  const bool blocks_only = prune_all_blocks();
  const uint32_t cap0 = (R + 32 + 3) & ~3u, dcap = 1536;
  uint32_t cap1 = std::max<uint32_t>(3 * R, 192), cap2 = 4096;
  while (cap2 > 64 && prune_block_bytes(stride, cap2, scratch) > (size_t)smem_attr_max() - 256) cap2 >>= 1;
  const bool reprune_ok = !blocks_only && prune_wpb(idx, prune_warp_bytes(stride, cap0, scratch) + 4ull * dcap) > 0;
  const bool lazy_ok = !blocks_only && prune_wpb(idx, prune_warp_bytes(stride, cap1, scratch)) > 0;
  if (!lazy_ok) cap1 = 0;
  const uint64_t big_cap = lazy_ok ? pairs_cap / 64 + 16 : pairs_cap;

  // sorts and scans of the reverse edges: keys are point ids and n
  int key_bits = 1;
  while (key_bits < 32 && (1ull << key_bits) <= n) key_bits++;
  size_t cub_bytes = 0;
  {
    size_t t[4] = {0, 0, 0, 0};
    uint32_t* u = nullptr;
    cub::DeviceRadixSort::SortPairs(nullptr, t[0], u, u, u, u, (int)pairs_cap, 0, key_bits, st);
    cub::DeviceRunLengthEncode::Encode(nullptr, t[1], u, u, u, u, (int)pairs_cap, st);
    cub::DeviceScan::ExclusiveSum(nullptr, t[2], u, u, (int)pairs_cap, st);
    uint64_t* k = nullptr;
    if (!perm) cub::DeviceRadixSort::SortPairs(nullptr, t[3], k, k, u, u, (int)n, 0, 64, st);
    cub_bytes = *std::max_element(t, t + 4) + 256;
  }
  size_t fixed_bytes = 0;
  auto take = [&](size_t bytes) {
    const size_t at = fixed_bytes;
    fixed_bytes += (bytes + 255) & ~size_t(255);
    return at;
  };
  const size_t o_perm = take(4 * n), o_clean = take(4 * n), o_start = take(16), o_cnt = take(256),
               o_visn = take(4 * maxB), o_cmps = take(4 * maxB), o_status = take(4 * maxB),
               o_pka = take(4 * pairs_cap), o_pkb = take(4 * pairs_cap), o_pva = take(4 * pairs_cap),
               o_pvb = take(4 * pairs_cap), o_uniq = take(4 * pairs_cap), o_counts = take(4 * pairs_cap),
               o_offs = take(4 * pairs_cap), o_nruns = take(16), o_jobs = take(12 * pairs_cap),
               o_big = take(32 * big_cap), o_cub = take(cub_bytes);
  BCUDA(bb.fixed.ensure(fixed_bytes));
  uint8_t* const fb = bb.fixed.as<uint8_t>();
  auto u32 = [&](size_t at) { return reinterpret_cast<uint32_t*>(fb + at); };
  uint32_t* d_perm = u32(o_perm);
  uint32_t *pk_a = u32(o_pka), *pk_b = u32(o_pkb), *pv_a = u32(o_pva), *pv_b = u32(o_pvb);
  BCUDA(bb.vis_keys.ensure(8 * maxB * vis_cap));

  // insertion order
  if (perm) {
    BCUDA(cudaMemcpyAsync(d_perm, perm, 4 * n, cudaMemcpyHostToDevice, st));
  } else {
    DevBuf kk;
    BCUDA(kk.ensure(20 * n));
    uint64_t *k1 = kk.as<uint64_t>(), *k2 = k1 + n;
    uint32_t* i1 = reinterpret_cast<uint32_t*>(k2 + n);
    perm_keys_kernel<<<(int)std::min<uint64_t>((n + 255) / 256, 65535), 256, 0, st>>>(k1, i1, n, bp->perm_seed);
    size_t tb = cub_bytes;
    const cudaError_t e = cub::DeviceRadixSort::SortPairs(fb + o_cub, tb, k1, k2, i1, d_perm, (int)n, 0, 64, st);
    cudaStreamSynchronize(st);
    kk.release();
    BCUDA(e);
  }

  const uint32_t start0 = 0;
  BCUDA(cudaMemcpyAsync(fb + o_start, &start0, 4, cudaMemcpyHostToDevice, st));
  uint32_t* c32 = u32(o_cnt);  // [0] status or, [2] flagged count, [4..7] reverse-edge prunes per class
  // [0] dist cmps, [1] visited, [2] class 3 segment cursor, [3] search cmps,
  // [4] insertion prune candidates, [5] reverse-edge pairs, [6] reverse-edge prune candidates
  unsigned long long* c64 = reinterpret_cast<unsigned long long*>(c32 + 8);
  BCUDA(cudaMemsetAsync(fb + o_cnt, 0, 256, st));
  BCUDA(cudaMemsetAsync(fb + o_clean, 0, 4 * n, st));

  // the searches' buffers at the largest batch, so that they are not regrown batch by batch
  pann_query_params qp{0, bp->L, n, R, bp->batch_factor};
  SearchPlan plan;
  {
    int rc = make_plan(idx, &qp, 1, &plan);
    TierSizes z;
    TierBufs tb;
    if (!rc) rc = size_tiers(idx, plan, maxB, PREC_F32, 0, 0, &z);
    if (!rc) rc = index_tier_buffers(idx, z, (uint32_t)maxB, PREC_F32, &tb);
    if (rc) { cleanup(); return rc; }
  }

  PruneArgs pa{};
  pa.points = idx->d_points;
  pa.stride = stride;
  pa.nchunks = nch;
  pa.graph = idx->d_graph;
  pa.R = R;
  pa.nclean = u32(o_clean);
  pa.dist_cmps = c64;

  // Jobs sorted in global memory: assemble their keys into segments, sort, prune a block per job. begin: segment
  // starts (device); total: keys of all segments.
  auto prune_segments = [&](uint32_t njobs, const uint32_t* jpts, const uint64_t* skeys, uint32_t sstride,
                            const uint32_t* sids, const uint32_t* soff, const uint32_t* sn, uint32_t* begin,
                            uint32_t* end, uint64_t total, double alpha) -> int {
    BCUDA(bb.seg_a.ensure_grow(8 * total + 8));
    BCUDA(bb.seg_b.ensure_grow(8 * total + 8));
    uint64_t *sa = bb.seg_a.as<uint64_t>(), *sb = bb.seg_b.as<uint64_t>();
    size_t need = 0;
    cub::DeviceSegmentedSort::SortKeys(nullptr, need, sa, sb, (int)total, (int)njobs, begin, end, st);
    BCUDA(bb.seg_tmp.ensure_grow(need + 256));
    BCUDA(dispatch_dm(dtype, metric, [&](auto DTc, auto MTc) {
      constexpr int DT = decltype(DTc)::value, MT = decltype(MTc)::value;
      const int blocks = (int)std::min<uint32_t>((njobs + wpb - 1) / wpb, 65535);
      assemble_kernel<DT, MT><<<blocks, 32 * wpb, wpb * stride, st>>>(idx->d_points, stride, d, nch, idx->d_graph, R,
                                                                     njobs, jpts, skeys, sstride, sids, soff, sn, begin,
                                                                     end, sa, c64);
      return cudaGetLastError();
    }));
    BCUDA(cub::DeviceSegmentedSort::SortKeys(bb.seg_tmp.p, need, sa, sb, (int)total, (int)njobs, begin, end, st));
    BCUDA(dispatch_dm(dtype, metric, [&](auto DTc, auto MTc) {
      constexpr int DT = decltype(DTc)::value, MT = decltype(MTc)::value;
      PruneArgs a = pa;
      a.alpha = alpha;
      a.pts = jpts;
      a.njobs_host = njobs;
      return launch_block<DT, MT, true>(idx, a, PruneSegs{begin, end, sb}, njobs, st);
    }));
    return PANN_OK;
  };

  uint32_t batches = 0;
  uint64_t reprunes = 0, inserted = 0;
  double clean_alpha = 0.0;  // the alpha of the rows' clean entries

  for (int pass = 0; pass < bp->num_passes; pass++) {
    const double alpha = (pass == bp->num_passes - 1) ? bp->alpha : 1.0;  // index.h:173-178
    // clean entries stay so at the same alpha; at a larger one only where distances are not negative
    if (pass > 0 && !(alpha == clean_alpha || (metric == MT_L2 && alpha > clean_alpha)))
      BCUDA(cudaMemsetAsync(fb + o_clean, 0, 4 * n, st));
    clean_alpha = alpha;
    pa.alpha = alpha;
    for (size_t b = 0; b < fl.size(); b++) {
      const uint32_t B = (uint32_t)(ce[b] - fl[b]);
      const uint32_t* pts = d_perm + fl[b];
      batches++;
      // ---- 1. search (QueryParams(0, L, n, maxDeg, rerank, batch_factor), index.h:251-252)
      uint32_t sor = 0;
      for (;;) {
        BCUDA(cudaEventRecord(ea, st));
        BCUDA(cudaMemsetAsync(c32, 0, 4, st));
        int rc = run_search(idx, plan, nullptr, pts, B, u32(o_start), nullptr, nullptr, u32(o_visn), u32(o_cmps),
                            u32(o_status), bb.vis_keys.as<uint64_t>(), vis_cap, st);
        if (rc) { cleanup(); return rc; }
        status_or_kernel<<<64, 256, 0, st>>>(u32(o_status), B, c32);
        BCUDA(cudaMemcpyAsync(&sor, c32, 4, cudaMemcpyDeviceToHost, st));
        BCUDA(cudaEventRecord(eb, st));
        BCUDA(cudaStreamSynchronize(st));
        if (sor & (QS_TABLE_FULL | QS_INTERNAL)) {
          cleanup();
          return fail(PANN_EOVERFLOW, "build search: a seen-set outgrew the largest table");
        }
        if (sor & QS_VISIT_OVERFLOW) {
          vis_cap *= 2;
          BCUDA(bb.vis_keys.ensure(8 * maxB * vis_cap));
          continue;
        }
        break;
      }
      {
        float ms = 0;
        cudaEventElapsedTime(&ms, ea, eb);
        t_search += ms * 1e-3;
      }
      BCUDA(cudaEventRecord(ea, st));
      batch_sums_kernel<<<64, 256, 0, st>>>(u32(o_status), QS_REF_WOULD_GROW, u32(o_cmps), u32(o_visn), B, c32 + 2, c64);
      // ---- 2. robustPrune of the inserted points
      const uint32_t segcap = vis_cap + R;
      if (!blocks_only && prune_wpb(idx, prune_warp_bytes(stride, segcap, scratch)) > 0) {
        BCUDA(dispatch_dm(dtype, metric, [&](auto DTc, auto MTc) {
          constexpr int DT = decltype(DTc)::value, MT = decltype(MTc)::value;
          PruneArgs a = pa;
          a.pts = pts;
          a.njobs_host = B;
          a.src_keys = bb.vis_keys.as<uint64_t>();
          a.src_keys_stride = vis_cap;
          a.src_n = u32(o_visn);
          a.cap = segcap;
          a.cands = c64 + 4;
          return launch_lazy<DT, MT>(idx, a, B, st);
        }));
      } else {
        // candidate lists too long for a warp's shared memory
        BCUDA(bb.seg_se.ensure(8 * maxB));
        uint32_t *sbeg = bb.seg_se.as<uint32_t>(), *send = sbeg + maxB;
        iota_begin_kernel<<<(B + 255) / 256, 256, 0, st>>>(sbeg, B, segcap);
        int rc = prune_segments(B, pts, bb.vis_keys.as<uint64_t>(), vis_cap, nullptr, nullptr, u32(o_visn), sbeg, send,
                                (uint64_t)B * segcap, alpha);
        if (rc) return rc;
        seg_len_sum_kernel<<<64, 256, 0, st>>>(sbeg, send, B, c64 + 4);
      }
      BCUDA(cudaEventRecord(eb, st));
      degree_sum_kernel<<<128, 256, 0, st>>>(idx->d_graph, R, pts, B, c64 + 5);
      // ---- 3. reverse edges
      const uint64_t np = (uint64_t)B * R;
      reverse_pairs_kernel<<<(int)std::min<uint64_t>((np + 255) / 256, 65535), 256, 0, st>>>(idx->d_graph, R, pts, B,
                                                                                             (uint32_t)n, pk_a, pv_a);
      {
        size_t tb = cub_bytes;
        BCUDA(cub::DeviceRadixSort::SortPairs(fb + o_cub, tb, pk_a, pk_b, pv_a, pv_b, (int)np, 0, key_bits, st));
        tb = cub_bytes;
        BCUDA(cub::DeviceRunLengthEncode::Encode(fb + o_cub, tb, pk_b, u32(o_uniq), u32(o_counts), u32(o_nruns), (int)np,
                                                 st));
        tb = cub_bytes;
        BCUDA(cub::DeviceScan::ExclusiveSum(fb + o_cub, tb, u32(o_counts), u32(o_offs), (int)np, st));
      }
      BCUDA(cudaMemsetAsync(c32 + 4, 0, 16, st));
      BCUDA(cudaMemsetAsync(c64 + 2, 0, 8, st));
      ClassifyArgs ca{};
      ca.graph = idx->d_graph;
      ca.R = R;
      ca.n = (uint32_t)n;
      ca.nclean = pa.nclean;
      ca.uniq = u32(o_uniq);
      ca.counts = u32(o_counts);
      ca.offs = u32(o_offs);
      ca.num_runs = u32(o_nruns);
      ca.vals = pv_b;
      ca.job_pts = u32(o_jobs);
      ca.job_off = ca.job_pts + pairs_cap;
      ca.job_n = ca.job_off + pairs_cap;
      ca.jobs_cap = (uint32_t)pairs_cap;
      ca.big_pts = u32(o_big);
      ca.big_off = ca.big_pts + 2 * big_cap;
      ca.big_n = ca.big_off + 2 * big_cap;
      ca.big_begin = ca.big_n + 2 * big_cap;
      ca.big_cap = (uint32_t)big_cap;
      ca.njobs = c32 + 4;
      ca.seg_total = c64 + 2;
      ca.cands_total = c64 + 6;
      ca.cap0 = reprune_ok ? cap0 : 0;
      ca.dcap = dcap;
      ca.cap1 = cap1;
      ca.cap2 = cap2;
      reverse_classify_kernel<<<(int)std::min<uint64_t>((np * 32 + 255) / 256, 65535), 256, 0, st>>>(ca);
      BCUDA(cudaGetLastError());
      const uint64_t max_jobs = std::min<uint64_t>(np, n);
      BCUDA(dispatch_dm(dtype, metric, [&](auto DTc, auto MTc) {
        constexpr int DT = decltype(DTc)::value, MT = decltype(MTc)::value;
        PruneArgs a = pa;
        a.src_ids = pv_b;
        a.pts = ca.job_pts;
        a.src_off = ca.job_off;
        a.src_n = ca.job_n;
        cudaError_t e = cudaSuccess;
        // the long jobs first
        if ((uint64_t)B + R > cap1) {
          PruneArgs c = a;
          c.pts = ca.big_pts;
          c.src_off = ca.big_off;
          c.src_n = ca.big_n;
          c.njobs = c32 + 6;
          c.cap = cap2;
          e = launch_block<DT, MT, false>(idx, c, PruneSegs{}, lazy_ok ? max_jobs / 64 + 1 : max_jobs, st);
          if (e != cudaSuccess) return e;
        }
        if (lazy_ok) {
          PruneArgs c = a;
          c.njobs = c32 + 5;
          c.flip = (uint32_t)pairs_cap - 1;
          c.cap = cap1;
          e = launch_lazy<DT, MT>(idx, c, max_jobs, st);
          if (e != cudaSuccess) return e;
        }
        if (reprune_ok) {
          a.njobs = c32 + 4;
          a.cap = cap0;
          a.dcap = dcap;
          e = launch_reprune<DT, MT>(idx, a, max_jobs, st);
        }
        return e;
      }));
      uint32_t nj[4] = {0, 0, 0, 0};
      unsigned long long seg_total = 0;
      BCUDA(cudaMemcpyAsync(nj, c32 + 4, 16, cudaMemcpyDeviceToHost, st));
      BCUDA(cudaMemcpyAsync(&seg_total, c64 + 2, 8, cudaMemcpyDeviceToHost, st));
      BCUDA(cudaEventRecord(ec, st));
      BCUDA(cudaEventSynchronize(ec));
      if (nj[3]) {
        if (seg_total >= 0x7FFFFFFFull) {
          cleanup();
          return fail(PANN_ENOMEM, "reverse-edge prune segments exceed 2^31 keys");
        }
        int rc = prune_segments(nj[3], ca.big_pts + big_cap, nullptr, 0, pv_b, ca.big_off + big_cap, ca.big_n + big_cap,
                                ca.big_begin, ca.big_begin + big_cap, seg_total, alpha);
        if (rc) return rc;
        BCUDA(cudaEventRecord(ec, st));
        BCUDA(cudaEventSynchronize(ec));
      }
      reprunes += (uint64_t)nj[0] + nj[1] + nj[2] + nj[3];
      inserted += B;
      {
        float ms = 0;
        cudaEventElapsedTime(&ms, ea, eb);
        t_prune += ms * 1e-3;
        cudaEventElapsedTime(&ms, eb, ec);
        t_rev += ms * 1e-3;
      }
    }
  }
  if (bp->sort_neighbors) {
    BCUDA(dispatch_dm(dtype, metric, [&](auto DTc, auto MTc) {
      constexpr int DT = decltype(DTc)::value, MT = decltype(MTc)::value;
      size_t sm = wpb * (stride + scratch + 16ull * R);
      auto kern = sort_neighbors_kernel<DT, MT>;
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_attr_max());
      int blocks = (int)std::min<uint64_t>((n + wpb - 1) / wpb, 65535ull * 8);
      kern<<<blocks, 32 * wpb, sm, st>>>(idx->d_points, stride, d, nch, idx->d_graph, R, n);
      return cudaGetLastError();
    }));
  }
  BCUDA(cudaEventRecord(ev1, st));
  BCUDA(cudaEventSynchronize(ev1));
  if (stats) {
    float ms = 0;
    cudaEventElapsedTime(&ms, ev0, ev1);
    std::memset(stats, 0, sizeof(*stats));
    stats->seconds = ms * 1e-3;
    stats->search_seconds = t_search;
    stats->prune_seconds = t_prune;
    stats->reverse_seconds = t_rev;
    unsigned long long h64[7] = {0, 0, 0, 0, 0, 0, 0};
    uint32_t h32[4] = {0, 0, 0, 0};
    cudaMemcpy(h64, c64, 56, cudaMemcpyDeviceToHost);
    cudaMemcpy(h32, c32, 16, cudaMemcpyDeviceToHost);
    stats->dist_cmps = h64[0];
    stats->visited_total = h64[1];
    stats->batches = batches;
    stats->flagged = h32[2];
    stats->search_cmps = h64[3];
    stats->prune_candidates = h64[4] + h64[6];
    stats->edge_pairs = h64[5];
    stats->reprunes = reprunes;
    stats->inserted = inserted;
  }
  cudaEventDestroy(ev0); cudaEventDestroy(ev1);
  cudaEventDestroy(ea); cudaEventDestroy(eb); cudaEventDestroy(ec); cudaEventDestroy(ed);
  cleanup();
  return PANN_OK;
#undef BCUDA
}
