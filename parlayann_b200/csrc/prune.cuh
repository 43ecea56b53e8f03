// robustPrune on the device (algorithms/vamana/index.h:63-137), the kernels of
// build.cu's prune steps. All give the reference's selections in its order and
// count its distance comparisons.
//
// Pairs known not to kill. A row written by robustPrune holds points of which
// no earlier one kills a later one at the alpha used (alpha d(a, b) > d(p, b)).
// Re-pruning that row with further candidates at the same alpha (or, for
// Euclidean distance, a larger one: products with a larger alpha are no
// smaller) asks those pairs again with the same floats and gets the same
// answer. So the build keeps per point how many entries at the end of its row
// are such (`nclean`; appended in-edges go to the front), and only pairs with
// at least one other candidate are evaluated. The comparisons the reference
// would have made are still counted.
#pragma once
#include "common.cuh"
#include "rowscore.cuh"

namespace pann {

// Keys carry PANN_VFLAG while a candidate is not one of the row's clean
// entries ("fresh").

// Bitonic sort of 32 KPL keys in registers, key i = lane * KPL + j.
template <int KPL>
__device__ __forceinline__ void warp_bitonic(uint64_t (&k)[KPL], int lane) {
#pragma unroll
  for (int size = 2; size <= 32 * KPL; size <<= 1) {
#pragma unroll
    for (int st = size >> 1; st > 0; st >>= 1) {
      if (st >= KPL) {  // partner in another lane
        const int ls = st / KPL;
        const bool up = size >= 32 * KPL || ((lane * KPL) & size) == 0;
        const bool low = (lane & ls) == 0;
#pragma unroll
        for (int j = 0; j < KPL; j++) {
          const uint64_t o = __shfl_xor_sync(0xFFFFFFFFu, k[j], ls);
          k[j] = ((o < k[j]) == (low == up)) ? o : k[j];
        }
      } else {
#pragma unroll
        for (int j = 0; j < KPL; j++)
          if ((j & st) == 0) {
            const bool up = size >= KPL ? (size >= 32 * KPL || ((lane * KPL) & size) == 0) : (j & size) == 0;
            const uint64_t x = k[j], y = k[j | st];
            const bool sw = (y < x) == up;
            k[j] = sw ? y : x;
            k[j | st] = sw ? x : y;
          }
      }
    }
  }
}

// Sort the n <= 32 KPL keys of kin by (distance, id) in registers (1,300
// instructions for 256 keys, a rank sort of 200 keys 6,800), drop repeated ids
// (index.h:86-88; a repeat is fresh only if all copies are) and leave the
// distinct keys in kin.
template <int KPL>
__device__ __forceinline__ uint32_t prune_sort_regs(uint64_t* kin, uint32_t n, int lane) {
  const unsigned FULL = 0xFFFFFFFFu;
  uint64_t k[KPL];
  // the flag below the id: copies of an id end up next to each other, a clean one first
#pragma unroll
  for (int j = 0; j < KPL; j++) {
    const uint32_t i = 32 * j + lane;
    const uint64_t v = i < n ? kin[i] : ~0ull;
    k[j] = i < n ? (v & 0xFFFFFFFF00000000ull) | ((uint32_t)v << 1) | (uint32_t)((v >> 31) & 1u) : ~0ull;
  }
  __syncwarp();
  warp_bitonic<KPL>(k, lane);
  // the first of each id stays
  const uint64_t prev = __shfl_up_sync(FULL, k[KPL - 1], 1);
  bool keep[KPL];
  uint32_t c = 0;
#pragma unroll
  for (int j = 0; j < KPL; j++) {
    const uint64_t before = j ? k[j - 1] : prev;
    const uint32_t i = lane * KPL + j;
    keep[j] = i < n && (i == 0 || (uint32_t)(before >> 1) << 1 != (uint32_t)(k[j] >> 1) << 1);
    c += keep[j];
  }
  uint32_t at = c;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(FULL, at, d);
    if (lane >= d) at += t;
  }
  const uint32_t u = __shfl_sync(FULL, at, 31);
  at -= c;
#pragma unroll
  for (int j = 0; j < KPL; j++)
    if (keep[j]) {
      const uint32_t lo = (uint32_t)k[j];
      kin[at++] = (k[j] & 0xFFFFFFFF00000000ull) | (lo >> 1) | ((lo & 1u) << 31);
    }
  __syncwarp();
  return u;
}

// As prune_sort_regs for any n, through `tmp` (n keys) past 512 keys.
__device__ __forceinline__ uint32_t prune_sort_unique(uint64_t* kin, uint32_t n, uint64_t* tmp, int lane) {
  if (n <= 128) return prune_sort_regs<4>(kin, n, lane);
  if (n <= 256) return prune_sort_regs<8>(kin, n, lane);
  if (n <= 512) return prune_sort_regs<16>(kin, n, lane);
  const unsigned FULL = 0xFFFFFFFFu;
  for (uint32_t i = lane; i < n; i += 32) {
    const uint64_t ki = kin[i] & PANN_KEYMASK;
    uint32_t r = 0;
    for (uint32_t j = 0; j < n; j++) {
      const uint64_t kj = kin[j] & PANN_KEYMASK;
      r += (kj < ki) | ((kj == ki) & (j < i));
    }
    tmp[r] = kin[i];
  }
  __syncwarp();
  uint32_t u = 0;
  for (uint32_t b = 0; b < n; b += 32) {
    const uint32_t i = b + lane;
    uint64_t k = 0;
    bool first = false;
    if (i < n) {
      k = tmp[i];
      first = i == 0 || key_id(tmp[i - 1]) != key_id(k);
      if (first)
        for (uint32_t j = i + 1; j < n && key_id(tmp[j]) == key_id(k); j++) k &= tmp[j] | PANN_KEYMASK;
    }
    const unsigned m = __ballot_sync(FULL, first);
    __syncwarp();
    if (first) kin[u + __popc(m & ((1u << lane) - 1u))] = k;
    u += __popc(m);
  }
  __syncwarp();
  return u;
}

__device__ __forceinline__ bool prune_kills(double alpha, float dsp, uint64_t key) {
  return __dmul_rn(alpha, (double)dsp) <= (double)key_dist(key);
}

// Stage row `id` of the points as the query of the distances that follow.
template <int DT, int MT>
__device__ __forceinline__ int32_t prune_stage(const uint8_t* points, uint64_t stride, int nchunks, uint32_t id,
                                               uint8_t* qs, int lane) {
  __syncwarp();
  stage_query<DT, MT>(qs, points + (uint64_t)id * stride, nchunks, lane);
  __syncwarp();
  return DT != DT_F32 && MT == MT_L2 ? sq_norm_int<DT>(reinterpret_cast<const uint4*>(qs), nchunks) : 0;
}

struct PruneArgs {
  const uint8_t* points;
  uint64_t stride;
  int nchunks;
  uint32_t* graph;
  uint32_t R;
  uint32_t* nclean;  // per point: clean entries at the end of its row
  double alpha;
  unsigned long long* dist_cmps;
  const uint32_t* pts;      // per job: the point
  const uint32_t* njobs;    // device count (or njobs_host)
  uint32_t njobs_host;
  uint32_t flip;            // 0, or the index of job 0 in arrays filled from their end
  // candidates besides the row: keys (insertions) or ids (reverse edges)
  const uint64_t* src_keys;
  uint32_t src_keys_stride;
  const uint32_t* src_ids;
  const uint32_t* src_off;
  const uint32_t* src_n;
  uint32_t cap;             // keys a job can hold
  uint32_t dcap;            // reprune: floats of its distance table
  unsigned long long* cands;  // insertion: candidates seen (build statistics)
};

// Gather a job's keys into kin: the given candidates, then the row's entries;
// float distances to p (staged at qs) for ids. Returns their number.
template <int DT, int MT>
__device__ __forceinline__ uint32_t prune_gather(const PruneArgs& a, uint32_t job, uint32_t p, uint64_t* kin,
                                                 const uint8_t* qs, uint8_t* stg, int32_t qq, uint32_t* deg_out,
                                                 int lane) {
  const unsigned FULL = 0xFFFFFFFFu;
  const uint32_t at = a.flip ? a.flip - job : job;
  const uint32_t m = a.src_n[at];
  const uint32_t* grow = a.graph + (uint64_t)p * a.R;
  const uint32_t* si = a.src_keys ? nullptr : a.src_ids + a.src_off[at];
  if (a.src_keys) {
    const uint64_t* sk = a.src_keys + (uint64_t)job * a.src_keys_stride;
    for (uint32_t t = lane; t < m; t += 32) kin[t] = sk[t] | PANN_VFLAG;
  }
  uint32_t deg = 0;
  for (uint32_t b = 0; b < a.R; b += 32) {
    const uint32_t v = b + lane < a.R ? __ldg(grow + b + lane) : PANN_PAD;
    deg += __popc(__ballot_sync(FULL, v != PANN_PAD));
  }
  const uint32_t fresh = deg - min(deg, a.nclean[p]);  // entries appended since the row was pruned
  const uint32_t pre = a.src_keys ? 0u : m;            // ids to score before the row's
  for (uint32_t b = 0; b < pre + deg; b += 32) {
    const uint32_t t = b + lane;
    const bool ok = t < pre + deg;
    const uint32_t id = !ok ? 0u : t < pre ? __ldg(si + t) : __ldg(grow + (t - pre));
    const float dd = warp_score_rows<DT, MT>(a.points, a.stride, a.nchunks, id, (int)min(32u, pre + deg - b), qs, stg,
                                             qq, lane);
    if (ok) kin[(a.src_keys ? m : 0u) + t] = make_key(dd, id) | (t < pre + fresh ? PANN_VFLAG : 0ull);
  }
  *deg_out = deg;
  __syncwarp();
  return m + deg;
}

__host__ __device__ inline uint32_t prune_warp_bytes(uint64_t stride, uint32_t cap, uint32_t scratch) {
  return (uint32_t)(((stride + scratch + 16ull * cap + 4ull * cap + 8ull * ((cap + 31) / 32) + 15) & ~15ull));
}

// robustPrune of the inserted points (and any job whose fresh candidates are
// many): one warp per job, its candidates in shared memory. Per selection the
// live later candidates that a pair test still needs are listed and scored 32
// at a time. With the rows read by eight lanes each, the live candidates
// packed and no separate sort, the insertion prunes of the 100K x 96 float
// build (R 64, L 128, two passes, 2,000 distances a job) went from 109 ms to
// 56 ms. What bounds it: per selection one dependent chain of a row to stage,
// the candidates' rows and their sums, at 12 to 16 warps an SM.
template <int DT, int MT>
__global__ void __launch_bounds__(128, 4) prune_lazy_kernel(PruneArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  const unsigned FULL = 0xFFFFFFFFu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  const uint32_t nwords = (a.cap + 31) / 32;
  uint8_t* qs = smem + (size_t)warp * prune_warp_bytes(a.stride, a.cap, row_score_scratch<DT>());
  uint8_t* stg = qs + a.stride;
  uint64_t* uk = reinterpret_cast<uint64_t*>(stg + row_score_scratch<DT>());
  uint64_t* tmp = uk + a.cap;
  uint32_t* list = reinterpret_cast<uint32_t*>(tmp + a.cap);
  uint32_t* alive = list + a.cap;
  uint32_t* freshm = alive + nwords;
  const uint32_t njobs = a.njobs ? *a.njobs : a.njobs_host;
  unsigned long long cmps = 0, cands = 0;
  for (uint32_t job = blockIdx.x * wpb + warp; job < njobs; job += gridDim.x * wpb) {
    const uint32_t p = a.pts[a.flip ? a.flip - job : job];
    int32_t qq = prune_stage<DT, MT>(a.points, a.stride, a.nchunks, p, qs, lane);
    uint32_t deg;
    const uint32_t m = prune_gather<DT, MT>(a, job, p, uk, qs, stg, qq, &deg, lane);
    cmps += deg + (a.src_keys ? 0u : m - deg);  // robustPrune's own distances (index.h:72-77,131-134)
    cands += m;
    const uint32_t u = prune_sort_unique(uk, m, tmp, lane);
    const uint32_t nw = (u + 31) / 32;
    for (uint32_t w = 0; w < nw; w++) {
      const uint32_t i = 32 * w + lane;
      const unsigned al = __ballot_sync(FULL, i < u), fm = __ballot_sync(FULL, i < u && (uk[i] & PANN_VFLAG));
      if (lane == 0) { alive[w] = al; freshm[w] = fm; }
    }
    __syncwarp();
    uint32_t* row = a.graph + (uint64_t)p * a.R;
    uint32_t nsel = 0, idx = 0;
    while (nsel < a.R && idx < u) {
      uint32_t w = idx >> 5;
      unsigned word = alive[w] & (0xFFFFFFFFu << (idx & 31));
      while (!word && ++w < nw) word = alive[w];
      if (!word) break;
      const uint32_t sel = 32 * w + __ffs(word) - 1;
      idx = sel + 1;
      const uint64_t ks = uk[sel];
      if (key_id(ks) == p) continue;  // index.h:99-101
      if (lane == 0) row[nsel] = key_id(ks);
      nsel++;
      if (idx >= u) break;
      const bool sfresh = (ks & PANN_VFLAG) != 0;
      // the live later candidates; those whose pair with sel is still open
      uint32_t live = 0, n = 0;
      for (uint32_t v = idx >> 5; v < nw; v++) {
        unsigned al = alive[v];
        if (v == idx >> 5) al &= 0xFFFFFFFFu << (idx & 31);
        live += __popc(al);
        const unsigned ev = sfresh ? al : al & freshm[v];
        if ((ev >> lane) & 1u) list[n + __popc(ev & ((1u << lane) - 1u))] = 32 * v + lane;
        n += __popc(ev);
      }
      cmps += live;
      if (n == 0) continue;
      qq = prune_stage<DT, MT>(a.points, a.stride, a.nchunks, key_id(ks), qs, lane);
      for (uint32_t b = 0; b < n; b += 32) {
        const bool ok = b + lane < n;
        const uint32_t i = ok ? list[b + lane] : 0u;
        const uint64_t k = uk[i];
        const float dd = warp_score_rows<DT, MT>(a.points, a.stride, a.nchunks, key_id(k), (int)min(32u, n - b), qs,
                                                 stg, qq, lane);
        if (ok && prune_kills(a.alpha, dd, k)) atomicAnd(alive + (i >> 5), ~(1u << (i & 31)));
      }
      __syncwarp();
    }
    for (uint32_t j = nsel + lane; j < a.R; j += 32) row[j] = PANN_PAD;
    if (lane == 0) a.nclean[p] = nsel;
    __syncwarp();
  }
  if (lane == 0) {
    if (cmps) atomicAdd(a.dist_cmps, cmps);
    if (a.cands && cands) atomicAdd(a.cands, cands);
  }
}

// Re-prune of a row and its new in-edges, with few fresh candidates: one warp
// per job. The distances of every fresh candidate to all others are computed
// first, in full rounds of 32 rows; the greedy selection then needs no more
// memory traffic. Fresh candidates are taken in order: a fresh candidate that
// no earlier selected clean one and no earlier selected fresh one kills is
// selected and kills later ones; a clean candidate can only be killed by a
// selected fresh one. `killer` holds the index of the first selection that
// kills a candidate, which also gives the reference's comparison count: a
// candidate is compared with every selection before it, up to its killer.
// With the skipped pairs about 300 of a job's 2,100 distances are left (100K x
// 96 float, R 64): reverse edges and re-prunes went from 540 ms to 75 ms, and
// the 100K x 128 uint8 build (R 32) from 85 ms to 37 ms for the same steps.
template <int DT, int MT>
__global__ void __launch_bounds__(128, 4) reprune_kernel(PruneArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  const unsigned FULL = 0xFFFFFFFFu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  const uint32_t per_warp = prune_warp_bytes(a.stride, a.cap, row_score_scratch<DT>()) + 4 * a.dcap;
  uint8_t* qs = smem + (size_t)warp * per_warp;
  uint8_t* stg = qs + a.stride;
  uint64_t* uk = reinterpret_cast<uint64_t*>(stg + row_score_scratch<DT>());
  uint64_t* tmp = uk + a.cap;
  uint32_t* flist = reinterpret_cast<uint32_t*>(tmp + a.cap);  // positions of the fresh candidates
  float* dtab = reinterpret_cast<float*>(smem + (size_t)warp * per_warp + per_warp - 4 * a.dcap);
  uint32_t* killer = reinterpret_cast<uint32_t*>(tmp);  // tmp is free once the keys are sorted
  uint32_t* rank = killer + a.cap;                      // selections before a candidate
  const uint32_t njobs = a.njobs ? *a.njobs : a.njobs_host;
  unsigned long long cmps = 0;
  for (uint32_t job = blockIdx.x * wpb + warp; job < njobs; job += gridDim.x * wpb) {
    const uint32_t p = a.pts[job];
    int32_t qq = prune_stage<DT, MT>(a.points, a.stride, a.nchunks, p, qs, lane);
    uint32_t deg;
    const uint32_t m = prune_gather<DT, MT>(a, job, p, uk, qs, stg, qq, &deg, lane);
    const uint32_t u = prune_sort_unique(uk, m, tmp, lane);
    // the fresh candidates, in order
    uint32_t nf = 0;
    for (uint32_t b = 0; b < u; b += 32) {
      const bool f = b + lane < u && (uk[b + lane] & PANN_VFLAG);
      const unsigned fm = __ballot_sync(FULL, f);
      if (f) flist[nf + __popc(fm & ((1u << lane) - 1u))] = b + lane;
      nf += __popc(fm);
      if (b + lane < u) killer[b + lane] = 0xFFFFFFFFu;
    }
    __syncwarp();
    for (uint32_t f = 0; f < nf; f++) {  // nf * u <= dcap: the host sends larger jobs elsewhere
      qq = prune_stage<DT, MT>(a.points, a.stride, a.nchunks, key_id(uk[flist[f]]), qs, lane);
      for (uint32_t b = 0; b < u; b += 32) {
        const bool ok = b + lane < u;
        const float dd = warp_score_rows<DT, MT>(a.points, a.stride, a.nchunks, ok ? key_id(uk[b + lane]) : 0u,
                                                 (int)min(32u, u - b), qs, stg, qq, lane);
        if (ok) dtab[f * u + b + lane] = dd;
      }
    }
    __syncwarp();
    for (uint32_t f = 0; f < nf; f++) {
      const uint32_t x = flist[f];
      const uint64_t kx = uk[x];
      // the first selected clean candidate before x that kills it
      uint32_t kill = killer[x];
      for (uint32_t b = 0; b < x && b < kill; b += 32) {
        const uint32_t i = b + lane;
        bool hit = false;
        if (i < x) {
          const uint64_t k = uk[i];
          hit = !(k & PANN_VFLAG) && key_id(k) != p && killer[i] == 0xFFFFFFFFu && prune_kills(a.alpha, dtab[f * u + i], kx);
        }
        const unsigned hm = __ballot_sync(FULL, hit);
        if (hm) {
          kill = min(kill, b + (uint32_t)__ffs(hm) - 1u);
          break;
        }
      }
      __syncwarp();
      if (kill != 0xFFFFFFFFu) {
        if (lane == 0) killer[x] = kill;
      } else if (key_id(kx) != p) {
        // x is selected: it kills later candidates not killed by an earlier selection
        for (uint32_t b = x + 1; b < u; b += 32) {
          const uint32_t i = b + lane;
          if (i < u && killer[i] == 0xFFFFFFFFu && prune_kills(a.alpha, dtab[f * u + i], uk[i])) killer[i] = x;
        }
      }
      __syncwarp();
    }
    // the first R live candidates other than p, in order; comparisons
    uint32_t* row = a.graph + (uint64_t)p * a.R;
    uint32_t nsel = 0;
    uint32_t comp = 0;
    for (uint32_t b = 0; b < u; b += 32) {
      const uint32_t i = b + lane;
      bool s = false;
      uint64_t k = 0;
      if (i < u) {
        k = uk[i];
        s = killer[i] == 0xFFFFFFFFu && key_id(k) != p;
      }
      const unsigned sm = __ballot_sync(FULL, s);
      const uint32_t before = nsel + __popc(sm & ((1u << lane) - 1u));  // selections before i
      if (s && before < a.R) row[before] = key_id(k);
      if (i < u) rank[i] = before;
      nsel += __popc(sm);
      __syncwarp();
      if (i < u) {
        const uint32_t kl = killer[i];
        const uint32_t upto = kl == 0xFFFFFFFFu ? before : rank[kl] + 1u;
        comp += min(upto, a.R);
      }
    }
    nsel = min(nsel, a.R);
    for (uint32_t j = nsel + lane; j < a.R; j += 32) row[j] = PANN_PAD;
    if (lane == 0) a.nclean[p] = nsel;
    cmps += __reduce_add_sync(FULL, comp) + m;
    __syncwarp();
  }
  if (lane == 0 && cmps) atomicAdd(a.dist_cmps, cmps);
}

// Jobs of many candidates (targets of hundreds of new in-edges, which would
// leave one warp working long after the others): one block of PRUNE_BLOCK
// threads per job. GATHERED = false: the candidates are gathered, scored and
// sorted (bitonic) in shared memory, `cap` (a power of two) of them at most;
// true: the segment keys[begin[job], end[job]) holds them sorted. A killed or
// repeated candidate carries PANN_VFLAG. Per selection each warp packs the
// live later candidates of its part 32 at a time and scores them.
constexpr int PRUNE_BLOCK = 256;
struct PruneSegs {
  const uint32_t* begin;
  const uint32_t* end;
  uint64_t* keys;
};

__host__ __device__ inline uint32_t prune_block_bytes(uint64_t stride, uint32_t cap, uint32_t scratch) {
  return (uint32_t)(((stride + 15) & ~15ull) + 8ull * cap + (PRUNE_BLOCK / 32) * (scratch + 4ull * 64));
}

template <int DT, int MT, bool GATHERED>
__global__ void __launch_bounds__(PRUNE_BLOCK, 2) prune_block_kernel(PruneArgs a, PruneSegs sg) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ uint32_t s_next, s_deg;
  const unsigned FULL = 0xFFFFFFFFu;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int NW = PRUNE_BLOCK / 32;
  constexpr uint32_t SCR = row_score_scratch<DT>();
  uint8_t* qs = smem;
  uint64_t* skeys = reinterpret_cast<uint64_t*>(smem + a.stride);
  uint8_t* wbuf = reinterpret_cast<uint8_t*>(skeys + (GATHERED ? 0 : a.cap)) + (size_t)warp * (SCR + 4 * 64);
  uint8_t* stg = wbuf;
  uint32_t* list = reinterpret_cast<uint32_t*>(wbuf + SCR);
  const uint32_t njobs = a.njobs ? *a.njobs : a.njobs_host;
  unsigned long long cmps = 0;
  for (uint32_t job = blockIdx.x; job < njobs; job += gridDim.x) {
    const uint32_t p = a.pts[job];
    uint32_t* row = a.graph + (uint64_t)p * a.R;
    uint64_t* K;
    uint32_t m;
    auto stage = [&](uint32_t id) -> int32_t {
      __syncthreads();
      if (warp == 0) stage_query<DT, MT>(qs, a.points + (uint64_t)id * a.stride, a.nchunks, lane);
      __syncthreads();
      return DT != DT_F32 && MT == MT_L2 ? sq_norm_int<DT>(reinterpret_cast<const uint4*>(qs), a.nchunks) : 0;
    };
    if (GATHERED) {
      K = sg.keys + sg.begin[job];
      m = sg.end[job] - sg.begin[job];
    } else {
      K = skeys;
      int32_t qq = stage(p);
      if (warp == 0) {
        uint32_t deg = 0;
        for (uint32_t b = 0; b < a.R; b += 32)
          deg += __popc(__ballot_sync(FULL, b + lane < a.R && row[b + lane] != PANN_PAD));
        if (lane == 0) s_deg = deg;
      }
      __syncthreads();
      const uint32_t mn = a.src_n[job], deg = s_deg;
      m = mn + deg;
      const uint32_t* si = a.src_ids + a.src_off[job];
      for (uint32_t b = 32 * warp; b < m; b += 32 * NW) {
        const uint32_t t = b + lane;
        const uint32_t id = t >= m ? 0u : t < mn ? __ldg(si + t) : row[t - mn];
        const float dd = warp_score_rows<DT, MT>(a.points, a.stride, a.nchunks, id, (int)min(32u, m - b), qs, stg, qq, lane);
        if (t < m) K[t] = make_key(dd, id);
      }
      cmps += warp == 0 ? m : 0u;
      uint32_t size = 32;
      while (size < m) size <<= 1;
      for (uint32_t i = m + tid; i < size; i += PRUNE_BLOCK) K[i] = ~0ull;
      for (uint32_t k = 2; k <= size; k <<= 1)
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
          __syncthreads();
          for (uint32_t t = tid; t < size / 2; t += PRUNE_BLOCK) {
            const uint32_t lo = 2 * t - (t & (j - 1)), hi = lo + j;  // pairs j apart
            const uint64_t x = K[lo], y = K[hi];
            if ((x > y) == ((lo & k) == 0)) { K[lo] = y; K[hi] = x; }
          }
        }
    }
    __syncthreads();
    // repeats by id (index.h:86-88), read before any is marked
    for (uint32_t b = 0; b < m; b += PRUNE_BLOCK) {
      const uint32_t i = b + tid;
      const bool dup = i < m && i > 0 && key_id(K[i]) == key_id(K[i - 1]);
      __syncthreads();
      if (dup) K[i] |= PANN_VFLAG;
      __syncthreads();
    }
    uint32_t nsel = 0, idx = 0;
    while (nsel < a.R && idx < m) {
      if (warp == 0) {
        uint32_t found = PANN_PAD;
        for (uint32_t b = idx; b < m && found == PANN_PAD; b += 32) {
          const unsigned msk = __ballot_sync(FULL, b + lane < m && !(K[b + lane] & PANN_VFLAG));
          if (msk) found = b + __ffs(msk) - 1;
        }
        if (lane == 0) s_next = found;
      }
      __syncthreads();
      const uint32_t found = s_next;
      if (found == PANN_PAD) break;
      const uint32_t sel = key_id(K[found]);
      idx = found + 1;
      if (sel == p) {  // index.h:99-101
        __syncthreads();
        continue;
      }
      if (tid == 0) row[nsel] = sel;
      nsel++;
      const int32_t qq = stage(sel);
      uint32_t n = 0;
      auto score = [&](uint32_t cnt) {  // the first cnt entries of the list
        const bool ok = (uint32_t)lane < cnt;
        const uint32_t i = ok ? list[lane] : 0u;
        const uint64_t k = ok ? K[i] : 0ull;
        const float dd = warp_score_rows<DT, MT>(a.points, a.stride, a.nchunks, key_id(k), (int)cnt, qs, stg, qq, lane);
        if (ok && prune_kills(a.alpha, dd, k)) K[i] = k | PANN_VFLAG;
      };
      for (uint32_t b = idx + 32 * warp; b < m; b += 32 * NW) {
        const bool live = b + lane < m && !(K[b + lane] & PANN_VFLAG);
        const unsigned msk = __ballot_sync(FULL, live);
        if (live) list[n + __popc(msk & ((1u << lane) - 1u))] = b + lane;
        n += __popc(msk);
        if (lane == 0) cmps += __popc(msk);
        __syncwarp();
        if (n >= 32) {
          score(32);
          __syncwarp();
          const uint32_t rest = (uint32_t)lane < n - 32 ? list[32 + lane] : 0u;
          __syncwarp();
          if ((uint32_t)lane < n - 32) list[lane] = rest;
          n -= 32;
          __syncwarp();
        }
      }
      if (n) score(n);
      __syncthreads();
    }
    __syncthreads();
    for (uint32_t j = nsel + tid; j < a.R; j += PRUNE_BLOCK) row[j] = PANN_PAD;
    if (tid == 0) a.nclean[p] = nsel;
    __syncthreads();
  }
  if (lane == 0 && cmps) atomicAdd(a.dist_cmps, cmps);
}

}  // namespace pann
