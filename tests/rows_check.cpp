// The partition of a split stage's tile rows (pip_rows.cuh): for every grid height, tile height and
// margin, the two launches take each tile row once, and the first one holds every row of cells
// that the halo exchange sends.
#include <cstdio>
#include <vector>

#include "../pip_b200/csrc/pip_rows.cuh"

int main() {
  long grids = 0, wrong = 0;
  for (int ty : {4, 7, 14})
    for (int margin : {2, 3})
      for (int ny = 4; ny <= 300; ++ny) {
        const int nby = (ny + ty - 1) / ty;
        std::vector<int> seen(nby, 0), sent(ny, 0);
        for (int rows : {1, 2}) {
          const int n = pip::tile_rows(rows, ny, ty, margin);
          for (int k = 0; k < n; ++k) {
            const int r = pip::tile_row(rows, k, n, nby);
            if (r < 0 || r >= nby) { ++wrong; continue; }
            ++seen[r];
            if (rows == 1)
              for (int j = r * ty; j < ny && j < (r + 1) * ty; ++j) sent[j] = 1;
          }
        }
        for (int c : seen) wrong += c != 1;
        for (int j = 0; j < margin; ++j) wrong += !sent[j] || !sent[ny - 1 - j];
        const int n = pip::tile_rows(0, ny, ty, margin);
        wrong += n != nby;
        for (int k = 0; k < n; ++k) wrong += pip::tile_row(0, k, n, nby) != k;
        ++grids;
      }
  std::printf("grids %ld wrong %ld\n", grids, wrong);
  return wrong != 0;
}
