// tensor_map.h — TMA tensor maps over operand planes.
#pragma once

#include <cuda.h>

namespace mb {

// 3-D map over 16-bit planes [planes][rows][kp]; box = {bk, box_rows, 1}; swizzle span = bk * 2 bytes (bk = 32 or 64).
int make_plane_map(CUtensorMap* map, const void* base, int planes, long long rows, int kp, int bk, int box_rows);
// 5-D map over zero-padded NHWC planes [planes][n][hp][wp][c]; box = {bc channels, bx pixels, by rows, 1, 1}.
int make_image_map(CUtensorMap* map, const void* base, int planes, int n, int hp, int wp, int c, int bc, int bx, int by);

}  // namespace mb
