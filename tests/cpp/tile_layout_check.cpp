// The tile search's shared-memory layout (csrc/tile_layout.cuh) over the shapes
// the library accepts, on the host: regions in order inside the block's
// allocation, and everything the exact re-rank writes or reads inside a region
// that is free or holds the query. Prints the shapes checked; exit code 1 and
// the first bad shape otherwise.
#include <algorithm>
#include <cstdio>
#include <vector>

#include "tile_layout.cuh"

using namespace pann;

int main() {
  const uint32_t scratch = 8192;  // a warp's row buffers for float rows
  const uint32_t degrees[] = {1, 2, 3, 4, 8, 31, 64, 1024}, beams[] = {1, 2, 10, 45, 200, 1000};
  std::vector<uint32_t> dims;
  for (uint32_t d = 1; d <= 80; d++) dims.push_back(d);
  for (uint32_t d : {96, 127, 128, 200, 256, 512, 1000, 1024, 1536, 3000, 4096, 8191, 8192}) dims.push_back(d);
  unsigned long long shapes = 0;
  for (uint32_t d : dims)
    for (int fp8 = 0; fp8 < 2; fp8++)
      for (uint32_t R : degrees)
        for (uint32_t nel : degrees)
          for (uint32_t L : beams)
            for (uint32_t W = 1; W <= 4; W++)
              for (uint32_t part = 0; part <= 4; part++) {  // 0: tensor-core scoring, else quarters of the tile staged
                if (nel > R) continue;
                const bool tc = part == 0;
                const uint64_t lp_stride = ((uint64_t)d * (fp8 ? 1 : 2) + 15) & ~15ull;
                if (tc && (lp_stride / 16) % 2) continue;
                const uint32_t CW = W * nel, S = tile_seen_slots(L, nel, R);
                const uint32_t CWs = tc ? TC_ROWS : std::max<uint32_t>(1, CW * part / 4);
                const TileLayout y = tile_layout(d, L, CW, S, lp_stride, CWs, tc);
                const TileRerank r = tile_rerank(y, tc, scratch);
                const size_t row = ((size_t)4 * d + 15) & ~size_t(15);  // a float row as stored
                const size_t free_end = tc ? y.qb : y.misc;             // table and stage
                const bool in_query = r.q >= y.q && r.q + row <= y.sc;
                const bool in_free = r.q >= y.table && r.q + row <= std::min(free_end, r.warps ? r.scratch : free_end);
                const bool ok = y.q + row <= y.sc && y.sc + row <= y.fr && y.fr + 8ull * L <= y.fr2 &&
                                y.fr2 + 8ull * L <= y.cand && y.cand + 8ull * std::max(CW, L) <= y.cid &&
                                y.cid + 4ull * CW <= y.table && y.table + 4ull * S <= y.stage && y.stage <= free_end &&
                                y.misc + 64 <= y.total && (in_query || in_free) && r.q % 16 == 0 &&
                                r.scratch % 16 == 0 && r.scratch >= y.table &&
                                r.scratch + (size_t)scratch * r.warps <= free_end && r.warps <= 4;
                if (!ok) {
                  std::printf("d %u fp8 %d R %u degree limit %u beam %u parents %u staged %u tensor %d\n", d, fp8, R, nel,
                              L, W, CWs, (int)tc);
                  return 1;
                }
                shapes++;
              }
  std::printf("%llu shapes\n", shapes);
  return 0;
}
