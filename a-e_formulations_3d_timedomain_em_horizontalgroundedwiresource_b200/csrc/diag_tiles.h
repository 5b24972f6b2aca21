// Index arithmetic of the diagonal-block kernel (k_potrf): the tiles of the rank-8
// update that follows every eight columns, for the kernel and for host checks of the
// elements they touch.
#pragma once

#ifdef __CUDACC__
#define TDEM_HD __host__ __device__
#else
#define TDEM_HD
#endif

namespace tdem {

constexpr int kDiagPanel = 64;           // widest diagonal block
constexpr int kDiagCols = 8;             // columns factored at a time
constexpr int kDiagQ = 16;               // rows of an update tile, and of a block row of the inverse
constexpr int kDiagLd = kDiagPanel + 2;  // leading dimension of the shared block
// The block's rows in shared memory, and one more tile half: where the rows right of the
// columns are not a multiple of 16, the last row tile reaches eight rows past the block.
// No tile reaches past its columns.
constexpr int kDiagRows = kDiagPanel + kDiagCols;

struct DiagTile {
  int r0, c0;  // 16 rows from r0, 8 columns from c0
};

// Tiles of the lower triangle of a wp-wide block (wp a multiple of 16) right of the
// columns [o, o + 8): row tile i has 2 (i + 1) column tiles, of which the last row tile's
// last starts at wp, past the block, where the rows left are an odd number of eights.
TDEM_HD constexpr int diag_tiles(int wp, int o) {
  const int left = wp - o - kDiagCols, n = (left + kDiagQ - 1) / kDiagQ;
  return n * (n + 1) - (left % kDiagQ != 0 ? 1 : 0);
}
TDEM_HD constexpr DiagTile diag_tile(int o, int tile) {
  const int i = tile < 2 ? 0 : (tile < 6 ? 1 : (tile < 12 ? 2 : 3)), h = tile - i * (i + 1);
  return {o + kDiagCols + kDiagQ * i, o + kDiagCols + kDiagCols * h};
}
constexpr int kDiagTilesMax = diag_tiles(kDiagPanel, 0);

}  // namespace tdem
