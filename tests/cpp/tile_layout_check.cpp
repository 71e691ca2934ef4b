// Prints layout facts of the tile kernel's buffers, read by tests/test_tile_layout.py.
#include <algorithm>
#include <cstdio>

#include "wfg_internal.h"

using namespace wfg;

int main() {
  // the offset of each row of the widest ring, in 64 bits
  const int pitch = (1 << 27) + WFG_TILE_PAD;
  for (int row = 0; row < 3 * WFG_TILE_BUFS; ++row) std::printf("row\t%d\t%lld\n", row, (long long)wfg_tile_row(row, pitch));
  // the leaf store's blocks: kind (0 gap-affine), rows back to the gap source, block, place, diagonals
  for (int lo = 0; lo <= 4; ++lo)
    for (int b = 0; b < 220; ++b) {
      const int q = lo ? b / lo : b;
      std::printf("leaf\t%d\t%d\t%d\t%d\n", lo, b, wfg_tile_leaf_at(lo > 0, b, q, lo), wfg_tile_leaf_n(lo > 0, q));
    }
  // words planned for a leaf up to score 520 and more, by rows back to the mismatch and gap, the spacing
  // and plen + tlen; gap-affine: x 2g, o 3g, e g
  for (int g : {1, 2, 7})
    for (int lo = 0; lo <= 4; ++lo)
      for (int lx = 1; lx <= (lo ? 4 : 1); ++lx)
        for (int sum : {2, 10, 50, 101, 120, 200, 300, 500, 1000}) {
          const int x = lo ? lx * g : 2 * g, o = lo ? lo * g : 3 * g, e = lo ? 0 : g, scope = std::max(x, o + e) + 1;
          const int smax = std::max(520, x * 100 + o + std::max(e, o) * 100 + scope) + 8;
          const int64_t reach = (int64_t)std::max((x + 1) / 2, lo ? o : e) * sum + o + e + 4 * scope + 16;
          std::printf("plan\t%d\t%d\t%d\t%d\t%lld\n", g, lo, lx, sum,
                      (long long)wfg_leaf_words(smax, sum, g, lo ? std::max(o, 1) : e, 3, true, lo > 0, lo ? lo : 1, reach));
        }
  return 0;
}
