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

// k_iterate_rows: the columns of a strip (PAIR: two nodes per lane), and those
// lost at either edge. One node per lane pulls
// its first row from the neighbouring columns directly; two nodes per lane
// load aligned pairs and shift them by shuffles in the first stage too, and
// store aligned pairs (an even count lost).
constexpr int rows_lost(bool pair, int T) { return pair ? (T + 1) / 2 * 2 : T - 1; }
constexpr int rows_lanes(bool pair) { return pair ? 64 : 32; }
constexpr int rows_columns(bool pair, int T) { return rows_lanes(pair) - 2 * rows_lost(pair, T); }

// Nodes from which two iterations per launch are faster than two launches of
// the one-iteration kernels, which have one warp per 32 or 64 nodes to hide
// latency with and live in L2 at these sizes. Measured at 1024 x 256, 2048 x
// 512 and 4096 x 1024 (us an iteration, one launch each against this kernel):
// FP64 4.8/5.6, 22.5/17.4, 92.7/57.9; FP32 3.9/5.2, 10.2/10.4, 50.0/33.3;
// 16 bits 3.7/5.2, 8.1/10.8, 35.9/29.1.
inline std::size_t rows_min_nodes(std::size_t elem) { return elem == 8 ? 700000 : (elem == 4 ? 1500000 : 2500000); }

// Whether a lattice of `nodes` nodes, nx wide, takes them. Above rows_min_nodes
// it is the share of the strips' columns that are nodes of the lattice (94% of a
// width that strips divide, 50% of 64 in pairs) that decides, and whether 1% of
// the node pairs or more are `mixed`, one node colliding and the other not: with
// two nodes per lane that of the other is parked across the collision, twice a
// launch, and the one-node kernels hardly slow down. Single launches
// against this kernel, us an iteration, clean and with 10% of the nodes solid:
// FP32 pairs 1024 x 1560 19.1/11.9 and 19.9/17.3, 1024 x 1660 20.4/14.0 and
// 21.2/22.9, 1024 x 2150 28.2/17.6 and 28.8/27.2; 192 x 11460 28.2/18.6 and
// 28.9/28.8; 128 x 32800 49.7/35.2 and 51.0/54.4; 64 x 25000 18.5/18.3 and
// 19.6/28.4, 62 x 25800 18.9/18.6, 30 x 53300 18.8/20.0.
// FP32, one node per lane, 255 x 6270 19.0/15.3 and 19.7/17.6, 99 x 16200 19.0/16.9
// and 19.8/20.1, 91 x 17600 18.9/17.8 and 19.9/21.2, 61 x 26200 19.0/19.8.
// FP64 96 x 7400 13.4/11.7 and 13.9/13.9, 64 x 11700 14.4/13.3 and 14.9/15.7, 64 x
// 18750 27.9/20.3 and 28.2/23.7, 32 x 23400 13.8/15.8, 32 x 62500 45.2/40.2 and
// 45.3/47.8.
// 16 bits, single launches in pairs: 1024 x 2460 24.2/17.8 and 28.6/26.7, 190 x
// 13700 26.1/20.9, 40 x 65000 26.0/24.1 and 30.8/35.5, 66 x 39400 25.9/28.7. Staged
// in tiles of `tile` nodes (0: not staged) they are faster, the more so the
// fuller the tile (of 512): 512 x 11700 40.4/38.5 and 53.5/57.8, 256 x 23400 in
// tiles of 512 40.5/41.7 and 53.4/62.7, of 256 49.2/41.7 and 61.5/62.8; 192 x
// 31200 of 384 41.5/44.6, of 192 49.2/44.6; 352 x 17000 47.2/37.2 and 63.5/55.8; 128
// x 46900 of 256 49.2/49.3 and 61.5/74.1.
inline bool rows_pay(std::size_t elem, int nx, std::size_t nodes, bool mixed, int tile) {
  const bool pair = elem < 8 && nx % 2 == 0;
  if (nodes < rows_min_nodes(elem) || (elem == 2 && !pair)) return false;
  const long long strips = (nx - 1) / rows_columns(pair, 2) + 1;
  const int share = (int)(100LL * nx / (strips * rows_lanes(pair)));  // percent
  if (elem == 8) return nodes >= 1100000 ? share >= (mixed ? 60 : 48) : share >= (mixed ? 75 : 60);
  if (elem == 4 && pair) return mixed ? share >= 75 && nodes >= 2200000 : share >= 48;
  if (elem == 4) return share >= (mixed ? 77 : 65);
  if (tile == 0) return share >= (mixed ? 80 : 60);
  return share >= (tile >= 384 || mixed ? 83 : 70) && !(mixed && tile >= 512);
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

// Whether the cases nx wide of a batch with tiles `tile` columns wide take them
// (with rows_min_nodes nodes in such cases together: FP32 cases of 256^2, 10%
// solid, 15.0/16.7 us an iteration of the batch at 1.0 M nodes, 25.6/25.7 at
// 1.6 M, 60.7/51.3 at 4.0 M). FP64: every width (the least gain, 32 wide on
// tiles of 32: 1.0 M nodes 36.3/27.6, 10% solid 39.0/32.8). FP32: even
// widths whose strips have at most 1.5 times the lanes of the tiles, which have
// idle lanes too (clean and 10% solid, tiles of 64, 1.6 M nodes: 48 wide
// 32.2/18.7 and 34.3/26.4, 96 28.0/18.5 and 29.2/26.2, 128 24.9/18.4 and
// 25.9/27.7, 256 24.9/16.7 and 25.6/25.7; 64 wide, twice the lanes, 25.1/23.3
// and 26.0/33.8), or every even width (tile = ROWS_ALL) where those left over
// have fewer than rows_min_nodes nodes: launches of their own, two for each of
// the others, would cost the batch more (three each of 64 x 16 to 2048 x 512,
// 2% solid: 49.8/43.8).
constexpr int ROWS_ALL = 1 << 20;
constexpr bool rows_case(bool pair, int nx, int tile) {
  if (!pair) return true;
  const long long strips = (nx - 1) / rows_columns(true, 2) + 1, tiles = (nx - 1) / tile + 1;
  return nx % 2 == 0 && 2 * strips * rows_lanes(true) <= 3 * tiles * tile;
}

}  // namespace tclb
