// Test driver (CPU): the update tiles of the diagonal-block kernel.  For every block width
// and every place of the eight columns: each element that a tile's warp touches (its 16 x 8
// result, the 16 and the 8 rows' operands) lies in the shared block's rows and columns, and
// the tiles hold every element of the lower triangle right of the columns exactly once.
// Prints "ok <elements touched>".
#include <cstdio>
#include <cstring>

#include "diag_tiles.h"
using namespace tdem;

int main() {
  long touched = 0;
  static int seen[kDiagRows][kDiagLd];
  for (int wp = kDiagQ; wp <= kDiagPanel; wp += kDiagQ)
    for (int o = 0; o < wp; o += kDiagCols) {
      std::memset(seen, 0, sizeof seen);
      bool in = true;
      auto touch = [&](int r, int c) {
        ++touched;
        if (r < 0 || r >= kDiagRows || c < 0 || c >= kDiagLd) {
          if (in) printf("wp %d o %d: row %d column %d is outside %d x %d\n", wp, o, r, c, kDiagRows, kDiagLd);
          in = false;
        }
      };
      for (int tile = 0; tile < diag_tiles(wp, o); ++tile) {
        const DiagTile t = diag_tile(o, tile);
        for (int r = 0; r < kDiagQ; ++r) {
          for (int c = 0; c < kDiagCols; ++c) {
            touch(t.r0 + r, t.c0 + c);  // read, and written where it is in the lower triangle
            touch(t.r0 + r, o + c);     // operand: the tile's rows of the eight columns
            touch(t.c0 + c, o + c);     // operand: the columns' rows of them
            if (in && t.r0 + r < wp && t.r0 + r >= t.c0 + c) ++seen[t.r0 + r][t.c0 + c];
          }
        }
      }
      if (!in) return 1;
      for (int r = 0; r < kDiagRows; ++r)
        for (int c = 0; c < kDiagLd; ++c) {
          const int want = r < wp && c >= o + kDiagCols && c <= r ? 1 : 0;
          if (seen[r][c] != want) {
            printf("wp %d o %d: element (%d, %d) is updated %d times\n", wp, o, r, c, seen[r][c]);
            return 1;
          }
        }
    }
  if (diag_tiles(kDiagPanel, 0) != kDiagTilesMax) return 1;
  printf("ok %ld\n", touched);
  return 0;
}
