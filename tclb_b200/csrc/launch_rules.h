// Rules of the launches that need no device: plain C++.
#pragma once
#include <algorithm>

namespace tclb {

constexpr int GRID_ROWS = 65535;  // limit of a grid's y (and z)

struct BlockShape {
  int bx, by;
};

// Block of the one-node kernel: in 3D the widest multiple of 32 that divides
// the row (a block of whole rows touches the fewest HBM pages, and none of its
// threads is idle), more rows while it has 64 threads or fewer; in
// 2D, where the lattices of this kernel live in L2, 32 x 4. Measured (us an
// iteration, 128 x 2 before and the shape chosen now): d3q19 192 x 96 x 96 FP32
// 49.7/44.6, 160^3 FP32 108.4/100.8, 256^3 FP32 399/392; d3q27 256^3 FP32
// 580/566, 192 x 64 x 64 FP32 31.4/29.0; d2q9 1024 x 256 FP64 4.82/4.67.
// Where that gives more rows of blocks than a grid holds, 32 x 8.
inline BlockShape block_shape(int nx, int ny, int nz) {
  int bx = 32;
  if (nz > 1)
    for (int b = 64; b <= 256; b += 32)
      if (nx % b == 0) bx = b;
  const int by = std::max(1, 128 / bx);
  if ((ny - 1) / by + 1 > GRID_ROWS) return {32, 8};
  return {bx, by};
}

}  // namespace tclb
