// Checks of the bands that share a lens shading table (csrc/isp_bands.hpp): down
// a strip, each band's grid rows fit the table unless one tile's do not, and no
// band could be a tile longer. The rows are counted one by one. Prints the failed
// cases; exits 0 when there is none.
#include <cstdio>

#include "isp_bands.hpp"

namespace {

constexpr int kTable = 8;

// Grid rows that image rows [y0, y1) lie between.
int rows_of(int y0, int y1, float scale, int height) {
  int lo = 1 << 30, hi = -1;
  for (int y = y0; y < y1; ++y) {
    int cell = static_cast<int>(static_cast<float>(y) * scale);
    if (cell > height - 2) cell = height - 2;
    if (cell < lo) lo = cell;
    if (cell > hi) hi = cell;
  }
  return hi - lo + 2;
}

}  // namespace

int main() {
  int failures = 0;
  for (const int image : {48, 480, 719, 1080, 2160, 3072, 8192}) {
    for (const int grid : {2, 3, 13, 17, 33, 129, 1000}) {
      const float scale = static_cast<float>(grid - 1) / static_cast<float>(image - 1);
      const int tiles = (image / 2 * 2 + 63) / 64;
      for (const int longest : {1, 2, 5, 16}) {
        for (int t = 0; t < tiles;) {
          const int most = tiles - t < longest ? tiles - t : longest;
          const int n = isp_b200::lsc_band_tiles(64 * t, most, scale, grid, kTable);
          const bool ok = n >= 1 && n <= most && (n == 1 || rows_of(64 * t, 64 * (t + n), scale, grid) <= kTable) &&
                          (n == most || rows_of(64 * t, 64 * (t + n + 1), scale, grid) > kTable);
          if (!ok) {
            std::printf("image %d grid %d longest %d tile %d: %d\n", image, grid, longest, t, n);
            ++failures;
          }
          t += n > 0 ? n : 1;
        }
      }
    }
  }
  return failures == 0 ? 0 : 1;
}
