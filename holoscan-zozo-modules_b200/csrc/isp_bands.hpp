// isp_bands.hpp - how many tiles of a strip share one lens shading table in the
// statistics pass of a batch: host and device code, without other headers of
// this library.
#pragma once

#include <cuda_runtime.h>

namespace isp_b200 {

// The grid row whose cell holds image row y (isp_math.hpp:121-140); scale: grid
// rows per image row, height: the grid's rows.
__host__ __device__ inline int lsc_row_cell(int y, float scale, int height) {
  const int cell = static_cast<int>(static_cast<float>(y) * scale);
  return cell > height - 2 ? height - 2 : cell;
}

// The tiles of 64 rows, at most `most`, from image row y0 on that a table of
// `table_rows` grid rows serves; at least one (a grid too dense for one tile's
// table is read sample by sample). Sixteen tiles span 13 rows of a 17x13 grid at
// 1080 image rows, and a band that overran its table read every sample's gain
// from the grid.
__host__ __device__ inline int lsc_band_tiles(int y0, int most, float scale, int height, int table_rows) {
  const int first = lsc_row_cell(y0, scale, height);
  int tiles = most;
  while (tiles > 1 && lsc_row_cell(y0 + 64 * tiles - 1, scale, height) - first + 2 > table_rows) --tiles;
  return tiles;
}

}  // namespace isp_b200
