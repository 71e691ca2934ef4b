// Prints layout facts of the tile kernel's buffers, read by tests/test_tile_layout.py.
#include <cstdio>

#include "wfg_internal.h"

using namespace wfg;

int main() {
  // the offset of each row of the widest ring, in 64 bits
  const int pitch = (1 << 27) + WFG_TILE_PAD;
  for (int row = 0; row < 3 * WFG_TILE_BUFS; ++row) std::printf("row\t%d\t%lld\n", row, (long long)wfg_tile_row(row, pitch));
  return 0;
}
