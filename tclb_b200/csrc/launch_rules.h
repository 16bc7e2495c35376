// Rules of the launches that need no device: plain C++.
#pragma once
#include <algorithm>
#include <cstddef>

namespace tclb {

constexpr int GRID_ROWS = 65535;  // limit of a grid's y (and z)

struct BlockShape {
  int bx, by;
};

// Block of the one-node kernel of a model of q populations stored in `elem`
// bytes. In 3D the widest multiple of 32 that divides
// the row (a block of whole rows touches the fewest HBM pages, and none of its
// threads is idle), more rows while it has 64 threads or fewer; in
// 2D, where the lattices of this kernel live in L2, 32 x 4. Measured (us an
// iteration, 128 x 2 before and the shape chosen now): d3q19 192 x 96 x 96 FP32
// 49.7/44.6, 160^3 FP32 108.4/100.8, 256^3 FP32 399/392; d3q27 256^3 FP32
// 580/566, 192 x 64 x 64 FP32 31.4/29.0; d2q9 1024 x 256 FP64 4.82/4.67.
// Two exceptions, found by measuring and not by a model of the hardware:
// d2q9 in FP32 takes 32 x 8 while 32 x 4 would give 4 to 8 blocks per SM (384 x
// 256 2.12 against 2.61, 512 x 256 2.63 against 3.22, 576 x 256 2.63 against
// 3.42; outside, 256 x 256 1.86 against 1.80, 512 x 320 3.68 against 3.56), and
// d3q19 in FP32 no blocks of 224 (224 x 64 x 64 24.7 against 24.0 with 32 x 4,
// 448 x 64 x 64 50.8 against 47.2 with 64 x 2; d3q27 is slower without them, 224
// x 112 x 112 99.1 against 102.1).
// Where that gives more rows of blocks than a grid holds, 32 x 8.
inline BlockShape block_shape(int q, int elem, int nx, int ny, int nz) {
  constexpr long long SMS = 148, BLOCK = 128;
  const long long nodes = (long long)nx * ny;
  int bx = 32, by = 0;
  if (nz > 1) {
    for (int b = 64; b <= 256; b += 32)
      if (nx % b == 0 && !(b == 224 && q == 19 && elem == 4)) bx = b;
    by = std::max(1, 128 / bx);
  } else {
    by = elem == 4 && nodes >= 4 * SMS * BLOCK && nodes < 8 * SMS * BLOCK ? 8 : 4;
  }
  if ((ny - 1) / by + 1 > GRID_ROWS) return {32, 8};
  return {bx, by};
}

// Single launches of d2q9 in 16 bits: whether in pairs of nodes rather than staged
// in tiles of `tile` nodes. Pairs are faster while two snapshots and the node
// types take less than two thirds of the L2, and always where the tiles are too
// small. Us an iteration, pairs / staged: 256 x 1024 in tiles of 512 3.3/4.3, 256 x
// 4096 8.7/9.2, 256 x 7800 15.1/15.0, 256 x 9400 19.7/17.8, 256 x 23400 55.7/40.5; in
// tiles of 256 256 x 8600 19.7/20.5, 256 x 10200 24.7/24.3, 256 x 23400 55.6/49.2;
// 192 x 31200 of 192 55.8/49.2, 160 x 37500 of 160 61.5/57.4, 96 x 62500 of 96 61.5/82.7,
// 32 x 187500 of 32 61.5/184.4; with 10% of the nodes solid 256 x 23400 of 512
// 64.2/53.4, of 256 63.8/61.5, 192 of 192 64.0/65.5, 160 of 160 71.3/77.9.
inline bool pairs_pay_2d(std::size_t nodes, int tile) {
  return tile < 192 || nodes < (tile >= 320 ? 2100000u : 2600000u);
}

}  // namespace tclb
