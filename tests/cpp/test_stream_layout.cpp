// Host-side check of the decode kernel's weight-stream bookkeeping (csrc/kernels.h): the tile order of the packed
// stream is a permutation in which every CTA's tiles are consecutive, the warps' shares cover a CTA's units and a split's
// cache rows exactly once, in order, and the reduction asks the warps that hold a tile's sums. No GPU involved.
#include <cstdio>
#include <vector>

#include "kernels.h"

using namespace vkl;

static int check(uint32_t tiles, uint32_t grid, uint32_t blocks) {
  std::vector<int> seen(tiles, 0);
  for (uint32_t t = 0; t < tiles; ++t) {
    const uint32_t pos = mega_stream_tile(t, tiles, grid);
    if (pos >= tiles || seen[pos]++) return 1;  // a permutation
  }
  for (uint32_t tile0 = 0; tile0 < grid && tile0 < tiles; ++tile0) {
    const uint32_t tl = (tiles - tile0 + grid - 1) / grid;
    for (uint32_t lt = 1; lt < tl; ++lt)  // a CTA's tiles follow each other
      if (mega_stream_tile(tile0 + lt * grid, tiles, grid) != mega_stream_tile(tile0, tiles, grid) + lt) return 2;
    // the warps' shares: every unit once, in order, and as many places for its tiles as a warp needs
    const uint32_t units = tl * blocks, slots = mega_red_slots(tiles, blocks, grid);
    std::vector<uint32_t> owner(units, MEGA_NCW);
    for (uint32_t w = 0; w < MEGA_NCW; ++w) {
      const uint32_t u0 = mega_share_begin(units, w), u1 = mega_share_begin(units, w + 1);
      if (u0 > u1 || u1 > units) return 3;
      for (uint32_t u = u0; u < u1; ++u) owner[u] = w;
      if (u0 < u1 && (u1 - 1) / blocks - u0 / blocks + 1 > slots) return 4;
    }
    if (slots < 1 || mega_share_begin(units, 0) != 0 || mega_share_begin(units, MEGA_NCW) != units) return 5;
    // the warps that the reduction of a tile asks are those with units of it, and it finds the tile's place
    for (uint32_t lt = 0; lt < tl; ++lt) {
      const MegaTileShares ts = mega_tile_shares(units, blocks, lt);
      if (ts.first != owner[lt * blocks] || ts.first + ts.more != owner[lt * blocks + blocks - 1]) return 6;
      if (ts.place != lt - mega_share_begin(units, ts.first) / blocks || ts.place >= slots) return 7;
      for (uint32_t w = ts.first + 1; w <= ts.first + ts.more; ++w) {
        const uint32_t u0 = mega_share_begin(units, w), u1 = mega_share_begin(units, w + 1);
        if (u0 < u1 && u0 / blocks != lt) return 8;  // their first place is this tile's
      }
    }
  }
  return 0;
}

int main() {
  const uint32_t grids[] = {1, 2, 7, 132, 148};
  const uint32_t tile_counts[] = {1, 3, 128, 147, 148, 149, 160, 384, 480, 688, 864, 1000, 1907};
  const uint32_t block_counts[] = {1, 2, 3, 5, 10, 11, 12, 29, 30, 31, 40, 128, 160, 344, 432, 864};
  for (uint32_t g : grids)
    for (uint32_t t : tile_counts)
      for (uint32_t b : block_counts)
        if (int rc = check(t, g, b)) {
          std::printf("FAIL tiles=%u grid=%u blocks=%u code=%d\n", t, g, b, rc);
          return 1;
        }
  // attention split helpers: the splits of a KV length cover it exactly
  for (uint32_t L = 1; L <= 4096; L += (L < 700 ? 1 : 97))
    for (uint32_t splits : {1u, 3u, 4u, 8u, 29u})
      for (uint32_t split_rows : {0u, 128u, 384u}) {
        const uint32_t S = mega_splits(L, splits, split_rows);
        if (S < 1 || S > splits) {
          std::printf("FAIL splits L=%u\n", L);
          return 1;
        }
        uint32_t at = 0;
        for (uint32_t s = 0; s < S; ++s) {
          uint32_t c0, c1;
          mega_kv_range(L, S, s, c0, c1);
          if (c0 != at || c1 < c0) {
            std::printf("FAIL kv range L=%u S=%u s=%u\n", L, S, s);
            return 1;
          }
          uint32_t row = c0;
          for (uint32_t w = 0; w < MEGA_NCW; ++w) {
            uint32_t r0, rows;
            mega_kv_share(c0, c1, w, r0, rows);
            if (rows && r0 != row) {
              std::printf("FAIL kv share L=%u S=%u s=%u w=%u\n", L, S, s, w);
              return 1;
            }
            row += rows;
          }
          if (row != c1) {
            std::printf("FAIL kv shares L=%u S=%u s=%u\n", L, S, s);
            return 1;
          }
          at = c1;
        }
        if (at != L) {
          std::printf("FAIL kv cover L=%u S=%u\n", L, S);
          return 1;
        }
      }
  std::printf("OK\n");
  return 0;
}
