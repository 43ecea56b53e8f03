// Shared memory of the tile search (tile.cu): sizes and offsets, on the host for
// the launch and on the device for the kernel.
#pragma once
#include <cstddef>
#include <cstdint>

#if defined(__CUDACC__)
#define PANN_HD __host__ __device__
#else
#define PANN_HD
#endif

namespace pann {

struct TileLayout {
  size_t q, sc, fr, fr2, cand, cid, table, stage, misc, qb, nrm, tcw, total;
  uint32_t sstride;  // staged row stride (bytes; CUDA-core scoring)
};

// Rows a tensor-core scoring round takes: the MMA's M.
constexpr uint32_t TC_ROWS = 128;

// CW: candidates a step can produce (parents x degree); CWs: rows staged at
// once (a step with more candidates stages and scores them in rounds). With
// tensor-core scoring (tc) the rows are staged TC_ROWS at a time in the
// core-matrix layout (umma.cuh), beside the query operand (16 rows: the
// query's split terms, the rest zero), the staged rows' squared norms and the
// MMA barrier and tensor-memory address.
PANN_HD inline TileLayout tile_layout(uint32_t d, uint32_t L, uint32_t CW, uint32_t S, uint64_t lp_stride,
                                      uint32_t CWs, bool tc = false) {
  TileLayout t{};
  size_t o = 0;
  const size_t dpad = (d + 15) & ~15u;  // whole 16-byte chunks of the low-precision row, of either type
  // rows at an odd multiple of 16 bytes apart: conflict-free 16-byte reads
  t.sstride = (uint32_t)(((lp_stride / 16) % 2 == 0) ? lp_stride + 16 : lp_stride);
  // every region starts on a 16-byte boundary (cp.async destinations and MMA operands need it)
#define PANN_TILE_TAKE(field, bytes) \
  t.field = o;                        \
  o += ((size_t)(bytes) + 15) & ~(size_t)15;
  PANN_TILE_TAKE(q, 4 * dpad)
  PANN_TILE_TAKE(sc, 4 * dpad)
  PANN_TILE_TAKE(fr, 8ull * L)
  PANN_TILE_TAKE(fr2, 8ull * L)
  PANN_TILE_TAKE(cand, 8ull * (CW > L ? CW : L))
  PANN_TILE_TAKE(cid, 4ull * CW)
  PANN_TILE_TAKE(table, 4ull * S)
  if (tc) {
    PANN_TILE_TAKE(stage, (size_t)TC_ROWS * lp_stride)
    PANN_TILE_TAKE(qb, 16 * lp_stride)
    PANN_TILE_TAKE(nrm, 4ull * TC_ROWS)
    PANN_TILE_TAKE(tcw, 16)
  } else {
    PANN_TILE_TAKE(stage, (size_t)CWs * t.sstride)
  }
  PANN_TILE_TAKE(misc, 64)
#undef PANN_TILE_TAKE
  t.total = o;
  return t;
}

// Where the exact re-rank keeps what it needs. The query stays in `q`, whose 4 * dpad bytes hold the padded float row
// whatever the tile is (table and stage of a thin tile hold less: one neighbour a step and long rows). Row buffers of
// `scratch` bytes a warp lie over table and stage, for up to four warps; with room for none, each thread scores a row.
struct TileRerank {
  size_t q, scratch;
  uint32_t warps;
};
PANN_HD inline TileRerank tile_rerank(const TileLayout& ly, bool tc, uint32_t scratch) {
  TileRerank r{};
  r.q = ly.q;
  r.scratch = ly.table;
  const size_t fit = ((tc ? ly.qb : ly.misc) - ly.table) / scratch;
  r.warps = fit < 4 ? (uint32_t)fit : 4u;
  return r;
}

// Seen-set slots of a query with beam L: (L + 16) * nel * 1.35 rounded up to
// a multiple of 32, within [4 (R + 1), 16384] (not a power of two: slots are
// chosen by multiplicative range reduction); a query stops early (flagged) when
// its set reaches 15/16 of that. Per query, so a batch answers each query as a
// search with that query's beam alone would.
PANN_HD inline uint32_t tile_seen_slots(uint32_t L, uint32_t nel, uint32_t R) {
  uint64_t s = ((uint64_t)(L + 16) * nel * 135 / 100 + 31) & ~31ull;
  const uint64_t lo = 4ull * (R + 1);
  if (s < lo) s = (lo + 31) & ~31ull;
  if (s > 16384) s = 16384;
  return (uint32_t)s;
}

}  // namespace pann
