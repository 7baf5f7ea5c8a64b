// pip_rows.cuh -- the rows of tiles of a split stage: those with the rows that a y-halo exchange
// sends (the first tile row, and the last one or two), launched first, and the rows between them.
// No CUDA header, so that the host can check the partition.
#pragma once

#if defined(__CUDACC__)
#define PIP_ROWS_HD __host__ __device__ __forceinline__
#else
#define PIP_ROWS_HD inline
#endif

namespace pip {

// Tile rows of `rows` (0: the whole stage, 1: those the exchange sends, 2: the others) for ny rows
// of cells in tiles of ty >= margin rows.  The last tile row may hold fewer than the margin rows
// that are sent; then the one before it is sent too.
PIP_ROWS_HD int tile_rows(int rows, int ny, int ty, int margin) {
  const int nby = (ny + ty - 1) / ty;
  if (rows == 0) return nby;
  const int tail = ny - (nby - 1) * ty;
  const int want = tail < margin ? 3 : 2, sent = nby < want ? nby : want;
  return rows == 1 ? sent : nby - sent;
}

// The tile row of block row k of n = tile_rows(rows, ...) of nby.
PIP_ROWS_HD int tile_row(int rows, int k, int n, int nby) {
  if (rows == 0) return k;
  if (rows == 2) return k + 1;
  return k == 0 ? 0 : nby - n + k;
}

}  // namespace pip
