// Warp-per-query beam search: the device form of ParlayANN's
// filtered_beam_search with use_filtering = false and no early stopping
// (algorithms/utils/beamSearch.h:33-228).
//
// One warp owns one query at a time and keeps all of its search state in
// shared memory:
//   qs    the query vector (row stride bytes)
//   fr    the frontier, <= L 64-bit (dist, id) keys, sorted; bit 31 of the id
//         word marks a visited entry. The reference's separate sorted
//         `visited` list and `unvisited_frontier` (set_difference, :217-222)
//         are represented by that flag: the next node to expand is the first
//         unflagged frontier entry, exactly unvisited_frontier[offset] (:119),
//         because between merges the frontier is unchanged and the flagged
//         entries are precisely unvisited_frontier[0..offset).
//   cand  candidates accumulated since the last merge (deferred batching,
//         :185-192); sorted by rank and merged into the frontier (set_union +
//         trim to L, :197-214).
//   scr   scratch: the rows being scored (rowscore.cuh), and between scorings
//         the sorted candidates and the merged frontier.
//   table the seen-set (:66, hashset.h). The reference's hashset is exact
//         until it grows; this table is exact, and the kernel counts inserts
//         against the reference's growth threshold (capacity/2) to flag
//         queries on which the reference's growth could change its result.
// Lanes split the adjacency row (one id per lane), test-and-insert the ids,
// compact the new ones, and score them 32 rows at a time (float sums keep the
// reference's sequential order).
#pragma once
#include "common.cuh"
#include "lowprec.cuh"
#include "rowscore.cuh"

namespace pann {

struct SearchArgs {
  // index
  const uint8_t* points;
  uint64_t stride;  // bytes per row (multiple of 16)
  uint32_t d;
  uint32_t nchunks;  // stride / 16
  const uint32_t* graph;
  uint32_t R;
  // queries
  const uint8_t* queries;  // nq rows of `stride` bytes; null in build mode
  const uint32_t* self_ids;  // build mode: query j is point self_ids[j] and skips itself
  uint32_t nq;
  const uint32_t* job_list;   // optional: job j is query job_list[j]
  const uint32_t* njobs_dev;  // optional: number of jobs read from device memory
  uint32_t* job_counter;      // dynamic work distribution (zeroed before launch)
  // query parameters (QueryParams, types.h:233-252); k and L are the maxima
  // when qk / qL give per-query values (the batched form)
  uint32_t k, L, dl;
  const uint32_t* qk;  // optional per-query k
  const uint32_t* qL;  // optional per-query beam
  uint32_t kstride;    // output row stride (>= every k)
  uint64_t limit;
  double batch_factor;
  uint32_t ref_half;  // the reference hashset's growth threshold: capacity/2
  const uint32_t* starts;
  uint32_t n_start;
  // per-warp shared-memory layout
  uint32_t Ccap;  // candidate buffer capacity
  uint32_t S;     // seen-table slots (power of two)
  uint32_t id_bits;    // 16-bit shared table (SEEN16): bits of an id, at least log2 S
  uint32_t scr_bytes;  // scratch region
  uint32_t warp_bytes;
  uint32_t* gtables;  // global seen tables (TABLE_GLOBAL form), S slots per resident warp
  uint32_t* gspill;   // shared-memory form: per resident warp, Sg-slot table taking inserts
  uint32_t Sg;        // once the shared table is 3/4 full (0 = no spill: re-run instead)
  // outputs
  uint32_t* out_ids;
  float* out_dists;
  uint32_t* out_visited;
  uint32_t* out_cmps;
  uint32_t* out_status;
  uint64_t* vis_keys;  // build mode: visited (dist,id) keys, vis_cap per query
  uint32_t vis_cap;
  uint32_t* redo_list;  // queries whose seen table filled up
  uint32_t* redo_count;
  uint32_t* emu_list;   // queries on which the reference's hashset would grow
  uint32_t* emu_rec;    // per emu_list entry: resume record index, or PAD to re-run from scratch
  uint32_t* emu_count;
  uint64_t opaque_zero;  // always 0; see f32_chunk2
  // Hand-off to the emulation tier. Before the visit in which a query could
  // push the reference's seen-set past its growth threshold, tier 0 stops the
  // query and saves its exact state in a resume record; the emulation tier
  // rebuilds the reference's table from the insertion log and continues.
  uint32_t* inslog;     // per resident warp: logcap ids, inserted in call order
  uint32_t logcap;
  uint32_t* vislog;     // per resident warp: viscap visited ids, in visit order
  uint32_t viscap;
  uint32_t* rec_pool;   // rec_cap records of rec_words words (layout: resume_layout)
  uint32_t rec_cap;
  uint32_t rec_words;
  uint32_t* rec_count;
  // precision form (float32 indexes): low-precision rows steer the search,
  // the best `rerank` frontier entries are re-scored exactly at the end
  const uint8_t* lp_rows;
  uint64_t lp_stride;
  uint32_t lp_chunks;
  const float* lp_scales;
  const float* lp_norms;  // squared norm of every low-precision row (tensor-core tile scoring)
  uint32_t rerank;
  // early stopping of range search (earlyStopping.h:19-29); es_count == 0 disables it
  double es_count;   // QP.early_stopping_count
  double es_radius;  // QP.radius as the rule sees it
  double es_esr;     // QP.early_stopping_radius
};

// The reference's seen-set capacity for beam L and degree limit dl is
// 2^ceil(log2(2 (10 + L) dl)) (beamSearch.h:66, hashset.h:50-54); it grows
// above half of that.
__host__ __device__ inline uint32_t ref_bits(uint32_t L, uint32_t dl) {
  const uint64_t n = 2ull * (10ull + L) * dl;
  uint32_t b = 0;
  while ((1ull << b) < n) b++;
  return b;
}

// Resume record: 8-word header (query, fn, cn, visits, cmps, entries), the
// frontier (2L words), the candidates (2 Ccap words), the insertion log
// (logcap words) and the visited ids (viscap words).
struct ResumeLayout {
  uint32_t fr, cand, log, vis, words;
};
__host__ __device__ inline ResumeLayout resume_layout(uint32_t L, uint32_t Ccap, uint32_t logcap, uint32_t viscap) {
  ResumeLayout r;
  r.fr = 8;
  r.cand = r.fr + 2 * L;
  r.log = r.cand + 2 * Ccap;
  r.vis = r.log + logcap;
  r.words = (r.vis + viscap + 3) & ~3u;
  return r;
}

// Where a query's seen-set lives.
enum SeenTable {
  SEEN16 = 0,    // shared memory, 16 bits an entry (ids of up to log2 S + SEEN16_REM bits: two buckets past home)
  SEEN32 = 1,    // shared memory, 32 bits an entry
  SEEN_GLOBAL = 2,
};
constexpr uint32_t SEEN16_REM = 11;

__host__ __device__ inline uint32_t search_scr_bytes(uint32_t L, uint32_t Ccap, uint32_t score_scratch) {
  const uint32_t m = (8 * L + 8 * Ccap + 15) & ~15u;
  return m > score_scratch ? m : score_scratch;
}
// Shared bytes of one query: query, frontier, candidates, compacted new ids, scratch, seen table.
__host__ __device__ inline uint32_t search_warp_bytes(uint64_t stride, uint32_t L, uint32_t Ccap, uint32_t R,
                                                      uint32_t S, int seen, uint32_t score_scratch) {
  uint64_t b = stride;
  b += (8ull * L + 15) & ~15ull;
  b += (8ull * Ccap + 15) & ~15ull;
  b += 4ull * ((R + 3) & ~3u);
  b += search_scr_bytes(L, Ccap, score_scratch);
  if (seen != SEEN_GLOBAL) b += (seen == SEEN16 ? 2ull : 4ull) * S;
  return (uint32_t)((b + 15) & ~15ull);
}
// Shared bytes of the single-warp emulation's state before its tables (search_emu.cuh).
__host__ __device__ inline uint32_t emu_state_bytes(uint64_t stride, uint32_t L, uint32_t Ccap, uint32_t R) {
  uint64_t b = stride;                 // query
  b += 16ull * L;                      // fr + fr2
  b += 16ull * Ccap;                   // cand + cand2
  b += 4ull * ((R + 3) & ~3u);         // compacted new ids
  return (uint32_t)((b + 15) & ~15ull);
}

// Sort n keys from `in` into `out` by rank (warp-cooperative; equal keys keep
// their order).
__device__ __forceinline__ void warp_rank_sort(const uint64_t* in, uint64_t* out, int n, int lane) {
  for (int i = lane; i < n; i += 32) {
    uint64_t ki = in[i] & PANN_KEYMASK;
    int r = 0;
    for (int j = 0; j < n; j++) {
      uint64_t kj = in[j] & PANN_KEYMASK;
      r += (kj < ki) | ((kj == ki) & (j < i));
    }
    out[r] = in[i];
  }
}

// Merge sorted frontier fr[0..fn) with sorted candidates c[0..cn) into out,
// keeping the first L (std::set_union then trim, beamSearch.h:202-214). Keys
// of the two inputs are disjoint (the seen-set admits each id once).
__device__ __forceinline__ int warp_merge(const uint64_t* fr, int fn, const uint64_t* c, int cn, uint64_t* out,
                                          int L, int lane) {
  for (int i = lane; i < fn; i += 32) {
    uint64_t k = fr[i] & PANN_KEYMASK;
    int lo = 0, hi = cn;
    while (lo < hi) { int mid = (lo + hi) >> 1; if ((c[mid] & PANN_KEYMASK) < k) lo = mid + 1; else hi = mid; }
    int pos = i + lo;
    if (pos < L) out[pos] = fr[i];
  }
  for (int j = lane; j < cn; j += 32) {
    uint64_t k = c[j] & PANN_KEYMASK;
    int lo = 0, hi = fn;
    while (lo < hi) { int mid = (lo + hi) >> 1; if ((fr[mid] & PANN_KEYMASK) < k) lo = mid + 1; else hi = mid; }
    int pos = j + lo;
    if (pos < L) out[pos] = c[j];
  }
  int t = fn + cn;
  return t < L ? t : L;
}

// Sort n distinct unflagged keys from `in` into `out` by rank.
__device__ __forceinline__ void warp_sort_distinct(const uint64_t* in, uint64_t* out, int n, int lane) {
  for (int b = 0; b < n; b += 32) {
    const uint64_t k = b + lane < n ? in[b + lane] : ~0ull;
    int r = 0;
#pragma unroll 4
    for (int j = 0; j < n; j++) r += in[j] < k;
    if (b + lane < n) out[r] = k;
  }
}

// Insert m <= 32 sorted unflagged keys c, one a lane, into the sorted frontier
// fr[0..fn) in place, keeping the first L (std::set_union then trim,
// beamSearch.h:202-214; the keys are new to it, the seen-set admits each id
// once). A lane finds its key's place by bisection; the places taken make a
// bit mask per 32 outputs, from which every output knows its source, so an
// output costs one read and one write whatever L is, and outputs before the
// first new key are left alone. From the last 32 outputs down: a block reads
// only at or before itself. *uword gets lane w's unvisited flags of the blocks
// w rewritten. A visit of the 100K x 128 uint8 search at beam 50 takes about
// 100 instructions here against 200 for merging both lists by bisection; one
// warp alone runs at 7 cycles an instruction, so they are what it waits for.
__device__ __forceinline__ int warp_insert(uint64_t* fr, int fn, const uint64_t* c, int m, int L, uint32_t* uword,
                                           int lane) {
  const unsigned FULL = 0xFFFFFFFFu;
  const uint64_t k = lane < m ? c[lane] : ~0ull;
  int p = 0;
  for (int step = 1 << (31 - __clz(fn)); step; step >>= 1) {
    const int t = p + step;
    if (t <= fn && (fr[t - 1] & PANN_KEYMASK) < k) p = t;
  }
  p += lane;
  const bool in = lane < m && p < L;
  int before = __popc(__ballot_sync(FULL, in));  // new keys before the block at hand
  if (before == 0) return fn;
  const int nfn = min(fn + m, L);
  const int w0 = __shfl_sync(FULL, p, 0) >> 5;
  for (int w = (nfn - 1) >> 5; w >= w0; w--) {
    const unsigned occ = __reduce_or_sync(FULL, in && (p >> 5) == w ? 1u << (p & 31) : 0u);
    before -= __popc(occ);
    const int t = 32 * w + lane;
    const int nb = before + __popc(occ & ((1u << lane) - 1u));
    const uint64_t* src = (occ >> lane) & 1u ? c + nb : fr + (t - nb);
    const uint64_t v = t < nfn ? *src : PANN_VFLAG;
    __syncwarp();
    if (t < nfn) fr[t] = v;
    const unsigned um = __ballot_sync(FULL, !(v & PANN_VFLAG));
    if (lane == w) *uword = um;
  }
  __syncwarp();
  return nfn;
}

// 16 bytes of shared memory as they are now (other lanes may have written).
__device__ __forceinline__ uint4 ld_shared_fresh(const uint32_t* p) {
  uint4 v;
  asm volatile("ld.volatile.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"((uint32_t)__cvta_generic_to_shared(p))
               : "memory");
  return v;
}

// The 16-bit seen-set: buckets of eight entries (16 bytes, one read). An id of
// id_bits bits is scrambled by a multiplication modulo 2^id_bits (a bijection);
// its top bits are its home bucket and the rest, `rem` (r bits), goes into the
// entry together with the bucket's distance from home: (distance << r) | rem.
// Bucket, distance and rem give back the id, so the set is exact in half the
// memory of 32-bit ids: a 4,096-entry table is 8 KB, which is what lets a
// query's row buffers fit beside it without fewer queries an SM. The all-ones
// entry is empty; a bucket fills in order, and an id goes to the next bucket
// only when its own is full, so a lookup ends at the first bucket with room.
struct Seen16 {
  uint32_t* words;
  uint32_t bmask, r, shift, mul, dmax;
  __device__ __forceinline__ void init(uint32_t* w, uint32_t S, uint32_t id_bits) {
    words = w;
    bmask = S / 8 - 1;
    r = id_bits - (28u - __clz(S));
    shift = 32u - id_bits;
    mul = (0x9E3779B1u >> shift) | 1u;
    dmax = (1u << (16u - r)) - 2u;
  }
  static __device__ __forceinline__ uint32_t zero_halves(uint32_t x) {  // lowest zero half marked exactly
    return (x - 0x00010001u) & ~x & 0x80008000u;
  }
  // INSERT: 1 inserted, 0 already present, -1 no room within reach; lookup: 1 present, 0 not
  template <bool INSERT>
  __device__ __forceinline__ int probe(uint32_t id) {
    const uint32_t x = (id * mul) & (0xFFFFFFFFu >> shift);
    uint32_t b = x >> r, code = x & ((1u << r) - 1u);
    for (uint32_t d = 0;;) {
      uint32_t* const bw = words + 4 * b;
      const uint4 w = ld_shared_fresh(bw);
      const uint32_t pat = code * 0x00010001u;
      if (zero_halves(w.x ^ pat) | zero_halves(w.y ^ pat) | zero_halves(w.z ^ pat) | zero_halves(w.w ^ pat))
        return INSERT ? 0 : 1;
      const uint32_t ex = zero_halves(~w.x), ey = zero_halves(~w.y), ez = zero_halves(~w.z), ew = zero_halves(~w.w);
      if (ex | ey | ez | ew) {
        if (!INSERT) return 0;
        const uint32_t i = ex ? 0u : ey ? 1u : ez ? 2u : 3u;
        const uint32_t old = ex ? w.x : ey ? w.y : ez ? w.z : w.w;
        const uint32_t e = ex ? ex : ey ? ey : ez ? ez : ew;
        const uint32_t put = old ^ ((0xFFFFu ^ code) << ((e & 0x8000u) ? 0 : 16));
        if (atomicCAS(bw + i, old, put) == old) return 1;
        continue;  // another lane changed the word: look at the bucket again
      }
      if (++d > dmax) return INSERT ? -1 : 0;
      code += 1u << r;
      b = (b + 1) & bmask;
    }
  }
};

// 32-bit ids in buckets of four (16 bytes, one read), by the same rules.
struct Seen32 {
  uint32_t* words;
  uint32_t bmask;
  __device__ __forceinline__ void init(uint32_t* w, uint32_t S) {
    words = w;
    bmask = S / 4 - 1;
  }
  template <bool INSERT>
  __device__ __forceinline__ int probe(uint32_t id) {
    uint32_t b = hash_slot(id, bmask);
    for (uint32_t d = 0; d <= bmask;) {
      uint32_t* const bw = words + 4 * b;
      const uint4 w = ld_shared_fresh(bw);
      if (w.x == id || w.y == id || w.z == id || w.w == id) return INSERT ? 0 : 1;
      if (w.w == PANN_PAD) {  // filled in order: room iff the last entry is empty
        if (!INSERT) return 0;
        const uint32_t i = w.x == PANN_PAD ? 0u : w.y == PANN_PAD ? 1u : w.z == PANN_PAD ? 2u : 3u;
        if (atomicCAS(bw + i, PANN_PAD, id) == PANN_PAD) return 1;
        continue;
      }
      d++;
      b = (b + 1) & bmask;
    }
    return 0;
  }
};

// Test-and-insert into an open-addressing table (linear probing). Returns 1 if
// id was inserted (first sighting), 0 if it was already present. The caller
// keeps the load below 1 so the probe always ends.
__device__ __forceinline__ int table_insert(uint32_t* table, uint32_t mask, uint32_t id) {
  uint32_t h = hash_slot(id, mask);
  for (uint32_t probe = 0; probe <= mask; probe++) {
    uint32_t old = atomicCAS(table + h, PANN_PAD, id);
    if (old == PANN_PAD) return 1;
    if (old == id) return 0;
    h = (h + 1) & mask;
  }
  return 0;
}

// MINB: blocks of 128 threads the register budget is fitted to (4: 128
// registers a thread; 6: 80).
template <int DT, int MT, int SEEN, int PREC = PREC_F32, int MINB = 4>
__global__ void __launch_bounds__(128, MINB) search_kernel(SearchArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int wpb = blockDim.x >> 5;
  const unsigned FULL = 0xFFFFFFFFu;

  uint8_t* wbase = smem + (size_t)warp * a.warp_bytes;
  uint8_t* qs = wbase;
  uint64_t* fr = reinterpret_cast<uint64_t*>(wbase + a.stride);
  uint64_t* cand = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(fr) + ((8u * a.L + 15u) & ~15u));
  uint32_t* nbuf = reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(cand) + ((8u * a.Ccap + 15u) & ~15u));
  uint8_t* scr = reinterpret_cast<uint8_t*>(nbuf + ((a.R + 3) & ~3u));
  uint64_t* cand2 = reinterpret_cast<uint64_t*>(scr);
  uint64_t* fr2 = cand2 + a.Ccap;
  uint32_t* table;
  if (SEEN == SEEN_GLOBAL) {
    table = a.gtables + ((size_t)blockIdx.x * wpb + warp) * a.S;
  } else {
    table = reinterpret_cast<uint32_t*>(scr + a.scr_bytes);
  }
  Seen16 seen16;
  Seen32 seen32;
  if (SEEN == SEEN16) seen16.init(table, a.S, a.id_bits);
  if (SEEN == SEEN32) seen32.init(table, a.S);
  const uint32_t table_words = SEEN == SEEN16 ? a.S / 2 : a.S;
  const uint32_t mask = a.S - 1;
  const uint32_t table_limit = (a.S >> 2) * 3;  // abort above 3/4 load
  uint32_t* spill =
      (SEEN != SEEN_GLOBAL && a.gspill) ? a.gspill + ((size_t)blockIdx.x * wpb + warp) * a.Sg : nullptr;
  const uint32_t smask = a.Sg - 1;
  const uint32_t spill_limit = (a.Sg >> 2) * 3;
  const uint32_t njobs = a.njobs_dev ? *a.njobs_dev : a.nq;
  const bool handoff = PREC == PREC_F32 && a.inslog != nullptr && a.emu_list != nullptr;
  uint32_t* const wlog = handoff ? a.inslog + ((size_t)blockIdx.x * wpb + warp) * a.logcap : nullptr;
  uint32_t* const wvis = handoff ? a.vislog + ((size_t)blockIdx.x * wpb + warp) * a.viscap : nullptr;
  // up to 1,024 frontier entries, lane w keeps the unvisited flags of entries 32 w .. 32 w + 31 in a register
  const bool flags_in_regs = a.L <= 1024;
  const bool es_on = a.es_count > 0.0;
  const uint32_t limit = (uint32_t)min((uint64_t)0xFFFFFFFFu, a.limit);

  for (;;) {
    uint32_t job = 0;
    if (lane == 0) job = atomicAdd(a.job_counter, 1u);
    job = __shfl_sync(FULL, job, 0);
    if (job >= njobs) break;
    const uint32_t qi = a.job_list ? a.job_list[job] : job;
    const uint32_t self = a.self_ids ? a.self_ids[qi] : PANN_PAD;
    const uint8_t* qsrc = a.self_ids ? a.points + (uint64_t)self * a.stride : a.queries + (uint64_t)qi * a.stride;
    const uint32_t L = a.qL ? a.qL[qi] : a.L;  // this query's beam (<= a.L, the buffer size)
    const uint32_t kq = a.qk ? a.qk[qi] : a.k;
    const uint32_t ref_half = a.qL ? (1u << ref_bits(L, a.dl)) / 2 : a.ref_half;
    // fewer candidates than this wait for the next visit (:185-192)
    const int defer_below = a.limit >= 2ull * L ? (int)ceil(a.batch_factor * (double)L) : 0;

    // stage the query, clear the seen table
    stage_query<DT, MT>(qs, qsrc, (int)a.nchunks, lane);
    {
      uint4 e = make_uint4(PANN_PAD, PANN_PAD, PANN_PAD, PANN_PAD);
      for (uint32_t c = lane; c < (table_words >> 2); c += 32) reinterpret_cast<uint4*>(table)[c] = e;
    }
    if (SEEN == SEEN_GLOBAL) __threadfence_block();
    __syncwarp();
    int32_t qq = 0;
    if (DT != DT_F32 && MT == MT_L2) qq = sq_norm_int<DT>(reinterpret_cast<const uint4*>(qs), a.nchunks);

    // starting points (:73-77); n_start <= L
    uint32_t entries_sh = a.n_start;  // ids in the shared-memory table
    bool spilled = false;
    uint32_t status = 0;
    auto start_spill = [&]() {
      // the shared table is frozen from here on; new ids go to the global spill table
      spilled = true;
      const uint4 e4 = make_uint4(PANN_PAD, PANN_PAD, PANN_PAD, PANN_PAD);
      for (uint32_t c = lane; c < (a.Sg >> 2); c += 32) reinterpret_cast<uint4*>(spill)[c] = e4;
      __threadfence_block();
      __syncwarp();
    };
    // Test-and-insert of one id a lane (PAD: none), every lane of the warp; true if the lane's id was new.
    auto seen_insert = [&](uint32_t v) -> bool {
      const bool has = v != PANN_PAD;
      if (SEEN == SEEN_GLOBAL) return has && table_insert(table, mask, v) != 0;
      int got = 0;
      if (has) {
        if (spilled) got = (SEEN == SEEN16 ? seen16.probe<false>(v) : seen32.probe<false>(v)) ? 0 : -1;
        else got = SEEN == SEEN16 ? seen16.probe<true>(v) : seen32.probe<true>(v);
      }
      if (SEEN == SEEN16 && !spilled && __any_sync(FULL, got < 0)) {  // no room within reach: the rest goes to the spill table
        if (!spill) {
          status |= QS_TABLE_FULL;
          return false;
        }
        start_spill();
      }
      if (got < 0) got = table_insert(spill, smask, v);
      return got > 0;
    };
    // the distance of each of the first n lanes' rows
    auto score = [&](uint32_t id, int n) -> float {
      if constexpr (PREC == PREC_F32)
        return warp_score_rows<DT, MT>(a.points, a.stride, (int)a.nchunks, id, n, qs, scr, qq, lane);
      else
        return warp_score_lp<MT, PREC>(a.lp_rows, a.lp_stride, (int)a.lp_chunks, id, n,
                                       reinterpret_cast<const float*>(qs), a.lp_scales, (int)a.d, scr, lane);
    };
    for (uint32_t b = 0; b < a.n_start; b += 32) {
      const uint32_t s = b + lane;
      const bool ok = s < a.n_start;
      const uint32_t id = ok ? a.starts[s] : PANN_PAD;
      const float dd = score(ok ? id : 0u, (int)min(32u, a.n_start - b));
      if (ok) fr[s] = make_key(dd, id);
      seen_insert(id);
      if (handoff && ok) wlog[s] = id;
    }
    __syncwarp();
    warp_rank_sort(fr, fr2, (int)a.n_start, lane);
    __syncwarp();
    for (uint32_t s = lane; s < a.n_start; s += 32) fr[s] = fr2[s];
    __syncwarp();
    int fn = (int)a.n_start;
    int cn = 0;
    uint32_t entries = a.n_start;    // distinct ids inserted (the reference's num_entries)
    uint32_t cmps = a.n_start;
    uint32_t nvis = 0;
    bool hand_over = false;
    const uint32_t nel = a.dl < a.R ? a.dl : a.R;
    // the reference's early-stopping rule reads unvisited_frontier[0], which is
    // refreshed only at a merge: its distance, taken at the first scan after one
    float u0 = 0.0f;
    bool u0_fresh = true;
    // unvisited entries, counted (and flagged in registers) anew after each merge
    uint32_t uword = 0;
    int cnt = 0;
    auto scan_frontier = [&]() {
      uword = 0;
      cnt = 0;
      for (int b = 0; b < fn; b += 32) {
        const int i = b + lane;
        const unsigned m = __ballot_sync(FULL, i < fn && !(fr[i] & PANN_VFLAG));
        if (lane == b >> 5) uword = m;
        cnt += __popc(m);
      }
    };
    scan_frontier();

    for (;;) {
      if (status & QS_TABLE_FULL) break;
      __syncwarp();
      // the first two unvisited frontier entries
      int first = -1, second = -1;
      if (flags_in_regs) {
        unsigned m = __ballot_sync(FULL, uword != 0);
        if (m) {
          const int w = __ffs(m) - 1;
          unsigned word = __shfl_sync(FULL, uword, w);
          first = 32 * w + __ffs(word) - 1;
          word &= word - 1;
          m &= m - 1;
          const int w2 = word ? w : __ffs(m) - 1;
          if (!word && m) word = __shfl_sync(FULL, uword, w2);
          if (word) second = 32 * w2 + __ffs(word) - 1;
        }
      } else {
        for (int b = 0; b < fn && second < 0; b += 32) {
          const int i = b + lane;
          unsigned m = __ballot_sync(FULL, i < fn && !(fr[i] & PANN_VFLAG));
          if (first < 0 && m) {
            first = b + __ffs(m) - 1;
            m &= m - 1;
          }
          if (first >= 0 && m) second = b + __ffs(m) - 1;
        }
      }
      if (first < 0 || nvis >= limit) break;  // :116
      if (u0_fresh) {
        u0 = key_dist(fr[first]);
        u0_fresh = false;
      }
      if (es_on && (double)nvis >= a.es_count && !((double)key_dist(fr[0]) <= a.es_radius) &&
          !((double)u0 <= a.es_esr))
        break;  // early_stopping (earlyStopping.h:19-29), checked at beamSearch.h:120-121
      if (handoff && entries + nel > ref_half) {
        // this visit could cross the reference's growth threshold
        status |= QS_REF_WOULD_GROW;
        hand_over = true;
        break;
      }
      const uint64_t cur = fr[first];
      const uint32_t cid = key_id(cur);
      const uint32_t* grow = a.graph + (uint64_t)cid * a.R;
      // the adjacency row on its way while the frontier is updated
      uint32_t vnext = (uint32_t)lane < nel ? __ldg(grow + lane) : PANN_PAD;
      // the next node to expand is most often the following unvisited entry:
      // start its adjacency row on its way to L2
      if (second >= 0 && lane == 0)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(a.graph + (uint64_t)key_id(fr[second]) * a.R));
      const bool full = (fn == (int)L);
      const float cutoff = full ? key_dist(fr[fn - 1]) : 3.40282346638528859812e+38F;  // :173-175
      __syncwarp();
      if (lane == 0) fr[first] = cur | PANN_VFLAG;
      if (lane == first >> 5) uword &= ~(1u << (first & 31));
      const int cnt_after = --cnt;  // unvisited entries after this one
      nvis++;
      if (a.vis_keys && lane == 0) {
        if (nvis <= a.vis_cap) a.vis_keys[(uint64_t)qi * a.vis_cap + (nvis - 1)] = cur & PANN_KEYMASK;
      }
      if (nvis > a.vis_cap && a.vis_keys) status |= QS_VISIT_OVERFLOW;
      if (handoff && lane == 0 && nvis <= a.viscap) wvis[nvis - 1] = cid;

      // neighbours not seen before (:151-160), compacted into nbuf
      if (!spilled && entries_sh + nel > table_limit) {
        if (!spill) { status |= QS_TABLE_FULL; break; }
        start_spill();
      }
      if (spilled && entries - entries_sh + nel > spill_limit) { status |= QS_TABLE_FULL; break; }
      int nnew = 0;
      uint32_t ins = 0;
      // the next 32 ids are loaded before this chunk's seen-set work, so a
      // row longer than one warp costs one round trip, not one per chunk
      for (uint32_t b = 0; b < nel; b += 32) {
        const uint32_t v = vnext;
        vnext = (b + 32 + lane < nel) ? __ldg(grow + b + 32 + lane) : PANN_PAD;
        const bool inserted = seen_insert(v);
        const bool isnew = inserted && (v != self);
        const unsigned mi = __ballot_sync(FULL, inserted);
        const unsigned mn = __ballot_sync(FULL, isnew);
        if (handoff && inserted) wlog[entries + ins + __popc(mi & ((1u << lane) - 1))] = v;  // call order
        ins += __popc(mi);
        if (isnew) nbuf[nnew + __popc(mn & ((1u << lane) - 1))] = v;
        nnew += __popc(mn);
      }
      if (status & QS_TABLE_FULL) break;
      entries += ins;
      if (!spilled) entries_sh += ins;
      if (entries > ref_half) status |= QS_REF_WOULD_GROW;
      __syncwarp();

      // distances; keep those below the cutoff (:176-182)
      cmps += (uint32_t)nnew;
      if ((uint32_t)(cn + nnew) > a.Ccap) { status |= QS_INTERNAL; break; }
      for (int b = 0; b < nnew; b += 32) {
        const int i0 = b + lane;
        const uint32_t v0 = i0 < nnew ? nbuf[i0] : 0u;
        const float d0 = score(v0, min(32, nnew - b));
        const bool keep0 = i0 < nnew && !(d0 >= cutoff);
        const unsigned m0 = __ballot_sync(FULL, keep0);
        if (keep0) cand[cn + __popc(m0 & ((1u << lane) - 1))] = make_key(d0, v0);
        cn += __popc(m0);
      }
      // deferred batching (:185-192)
      if (cn == 0 || (cn < defer_below && cnt_after >= 1)) continue;
      __syncwarp();
      warp_sort_distinct(cand, cand2, cn, lane);
      __syncwarp();
      for (int b = 0; b < cn; b += 32) fn = warp_insert(fr, fn, cand2 + b, min(32, cn - b), (int)L, &uword, lane);
      u0_fresh = true;
      cn = 0;
      if (flags_in_regs) cnt = (int)__reduce_add_sync(FULL, (unsigned)__popc(uword));
      else scan_frontier();
    }

    if (status & (QS_TABLE_FULL | QS_INTERNAL)) {
      if (status & QS_INTERNAL) {
        if (lane == 0 && a.out_status) a.out_status[qi] = status;
        __syncwarp();
        continue;
      }
      if (lane == 0 && a.redo_list) a.redo_list[atomicAdd(a.redo_count, 1u)] = qi;
      if (lane == 0 && a.out_status) a.out_status[qi] = status;
      __syncwarp();
      continue;
    }
    if ((status & QS_REF_WOULD_GROW) && a.emu_list) {
      // continued (or re-run) by the exact-emulation tier, which writes this query's outputs
      uint32_t r = PANN_PAD;
      if (hand_over) {
        if (lane == 0) r = atomicAdd(a.rec_count, 1u);
        r = __shfl_sync(FULL, r, 0);
        if (r < a.rec_cap && nvis <= a.viscap) {
          const ResumeLayout ly = resume_layout(a.L, a.Ccap, a.logcap, a.viscap);
          uint32_t* rec = a.rec_pool + (size_t)r * a.rec_words;
          if (lane == 0) {
            rec[0] = qi; rec[1] = (uint32_t)fn; rec[2] = (uint32_t)cn; rec[3] = (uint32_t)nvis;
            rec[4] = cmps; rec[5] = entries; rec[6] = __float_as_uint(u0);
          }
          uint64_t* rfr = reinterpret_cast<uint64_t*>(rec + ly.fr);
          uint64_t* rcand = reinterpret_cast<uint64_t*>(rec + ly.cand);
          for (int i = lane; i < fn; i += 32) rfr[i] = fr[i];
          for (int i = lane; i < cn; i += 32) rcand[i] = cand[i];
          __syncwarp();
          for (uint32_t i = lane; i < entries; i += 32) rec[ly.log + i] = wlog[i];
          for (uint32_t i = lane; i < (uint32_t)nvis; i += 32) rec[ly.vis + i] = wvis[i];
        } else {
          r = PANN_PAD;  // no room: the emulation re-runs the query from the start
        }
      }
      // publish: the record and the list entry before the record index, which
      // an emulation pass running beside this kernel reads as "ready"
      __threadfence();
      __syncwarp();
      if (lane == 0) {
        uint32_t pos = atomicAdd(a.emu_count, 1u);
        a.emu_list[pos] = qi;
        __threadfence();
        atomicExch(a.emu_rec + pos, r);
      }
      __syncwarp();
      continue;
    }
    if ((uint32_t)fn < kq) status |= QS_SHORT;
    uint32_t* const oid = a.out_ids + (uint64_t)qi * a.kstride;
    float* const odist = a.out_dists ? a.out_dists + (uint64_t)qi * a.kstride : nullptr;
    if (PREC != PREC_F32) {
      // re-rank the best min(rerank, fn) entries by exact float32 distance
      // (beam_search_rerank's full-precision pass, beamSearch.h:569-587)
      const uint32_t rr = a.rerank ? a.rerank : 4 * kq;  // 0: 4k of this query
      const int nr = (int)min((uint32_t)fn, rr > kq ? rr : kq);
      for (int b = 0; b < nr; b += 32) {
        const int i0 = b + lane;
        const uint32_t v0 = i0 < nr ? key_id(fr[i0]) : 0u;
        const float d0 = warp_score_rows<DT, MT>(a.points, a.stride, (int)a.nchunks, v0, min(32, nr - b), qs, scr, qq, lane);
        if (i0 < nr) fr[i0] = make_key(d0, v0);
      }
      __syncwarp();
      for (int i = lane; i < nr; i += 32) {
        const uint64_t ki = fr[i];
        int r = 0;
        for (int j = 0; j < nr; j++) r += fr[j] < ki;
        if ((uint32_t)r < kq) {
          oid[r] = key_id(ki);
          if (odist) odist[r] = key_dist(ki);
        }
      }
      for (uint32_t j = min((uint32_t)nr, kq) + lane; j < a.kstride; j += 32) {
        oid[j] = PANN_PAD;
        if (odist) odist[j] = 0.0f;
      }
    } else {
      for (uint32_t j = lane; j < a.kstride; j += 32) {
        bool ok = j < (uint32_t)fn && j < kq;
        oid[j] = ok ? key_id(fr[j]) : PANN_PAD;
        if (odist) odist[j] = ok ? key_dist(fr[j]) : 0.0f;
      }
    }
    if (lane == 0) {
      if (a.out_visited) a.out_visited[qi] = (uint32_t)nvis;
      if (a.out_cmps) a.out_cmps[qi] = cmps;
      if (a.out_status) a.out_status[qi] = status;
    }
    __syncwarp();
  }
}

}  // namespace pann
