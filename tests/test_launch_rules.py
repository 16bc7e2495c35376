"""The rules that choose a launch, compiled for the host from the header the library includes."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from tclb_b200 import models as M
from tclb_b200.lattice import Lattice

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tclb_b200", "csrc")
SOURCE = """
#include "launch_rules.h"
extern "C" void shape(int q, int elem, int nx, int ny, int nz, int* out) {
  const tclb::BlockShape s = tclb::block_shape(q, elem, nx, ny, nz);
  out[0] = s.bx;
  out[1] = s.by;
}
extern "C" int rows_pay(int elem, int nx, long long nodes, int mixed, int tile) {
  return tclb::rows_pay(elem, nx, nodes, mixed != 0, tile);
}
extern "C" int pairs_pay_2d(long long nodes, int tile) { return tclb::pairs_pay_2d(nodes, tile); }
extern "C" int rows_case(int pair, int nx, int tile) { return tclb::rows_case(pair != 0, nx, tile); }
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "rules.cpp").write_text(SOURCE)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-shared", "-fPIC", "-I", CSRC,
                           "-o", str(d / "rules.so"), str(d / "rules.cpp")])
    return ctypes.CDLL(str(d / "rules.so"))


# rows a launch has always taken: blocks of 128 x 2, 64 x 4 and 32 x 8 threads by the width
@pytest.mark.parametrize("nz", [1, 2])
@pytest.mark.parametrize("nx,rows", [(17, 524280), (32, 524280), (64, 262140), (96, 262140), (128, 131070),
                                     (160, 131070), (192, 131070), (224, 131070), (256, 131070), (300, 131070)])
def test_every_height_fits_the_grid(rules, nx, rows, nz):
    out = (ctypes.c_int * 2)()
    for q, elem in [(9, 4), (9, 8)] if nz == 1 else [(19, 4), (19, 8), (27, 4)]:
        for ny in (1, 2, 65535, 65536, 70000, 131070, 131071, 262140, 262141, rows):
            if ny > rows:
                continue
            rules.shape(q, elem, nx, ny, nz, out)
            bx, by = out
            assert bx % 32 == 0 and by >= 1 and bx * by <= 256
            assert (ny + by - 1) // by <= 65535, (nx, ny, bx, by)


# both sides of the node counts (4 and 8 blocks of 128 for each of 148 SMs) and of the width that have a shape of
# their own
@pytest.mark.parametrize("q,elem,size,shape", [
    (9, 4, (256, 295, 1), (32, 4)), (9, 4, (256, 296, 1), (32, 8)), (9, 4, (512, 256, 1), (32, 8)),
    (9, 4, (256, 591, 1), (32, 8)), (9, 4, (256, 592, 1), (32, 4)), (9, 8, (512, 256, 1), (32, 4)),
    (19, 4, (224, 64, 64), (32, 4)), (19, 4, (448, 64, 64), (64, 2)), (19, 8, (224, 64, 64), (224, 1)),
    (27, 4, (224, 64, 64), (224, 1)), (19, 4, (192, 64, 64), (192, 1)), (19, 4, (256, 64, 64), (256, 1)),
    (27, 4, (128, 64, 64), (128, 1)), (19, 4, (64, 64, 64), (64, 2)), (19, 4, (33, 64, 64), (32, 4))])
def test_block_of_the_one_node_kernel(rules, q, elem, size, shape):
    out = (ctypes.c_int * 2)()
    rules.shape(q, elem, *size, out)
    assert tuple(out) == shape


# (bytes per value, width, nodes): taken when clean, when mixed; and the same where single launches are staged
@pytest.mark.parametrize("elem,nx,nodes,taken", [
    (4, 1024, 1_499_999, "00"), (4, 1024, 1_500_000, "10"), (4, 1024, 2_200_000, "11"), (4, 60, 2_200_000, "11"),
    (4, 192, 2_199_999, "10"), (4, 192, 2_200_000, "11"), (4, 128, 9_000_000, "10"), (4, 64, 1_500_000, "10"),
    (4, 62, 9_000_000, "10"), (4, 30, 9_000_000, "00"), (4, 8, 9_000_000, "00"), (4, 2, 9_000_000, "00"),
    (4, 255, 1_499_999, "00"), (4, 255, 1_500_000, "11"), (4, 99, 1_500_000, "11"), (4, 91, 1_500_000, "10"),
    (4, 61, 9_000_000, "00"), (4, 31, 9_000_000, "00"), (4, 1, 9_000_000, "00"),
    (8, 1024, 699_999, "00"), (8, 1024, 700_000, "11"), (8, 30, 700_000, "11"), (8, 96, 700_000, "11"),
    (8, 64, 700_000, "10"), (8, 64, 1_100_000, "11"), (8, 32, 1_099_999, "00"), (8, 32, 1_100_000, "10"),
    (8, 31, 1_100_000, "10"), (8, 8, 9_000_000, "00"), (8, 1, 9_000_000, "00"),
    (2, 1024, 2_499_999, "00"), (2, 1024, 2_500_000, "11"), (2, 600, 2_500_000, "11"), (2, 190, 2_500_000, "10"),
    (2, 40, 2_500_000, "10"), (2, 66, 9_000_000, "00"), (2, 30, 9_000_000, "00"), (2, 1025, 9_000_000, "00")])
def test_where_two_iterations_per_launch_pay(rules, elem, nx, nodes, taken):
    rules.rows_pay.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_longlong, ctypes.c_int, ctypes.c_int]
    assert "".join(str(rules.rows_pay(elem, nx, nodes, mixed, 0)) for mixed in (0, 1)) == taken


@pytest.mark.parametrize("nx,tile,nodes,taken", [
    (512, 512, 2_499_999, "00"), (512, 512, 2_500_000, "10"), (480, 480, 2_500_000, "11"), (384, 384, 9_000_000, "11"),
    (256, 512, 9_000_000, "00"), (256, 256, 9_000_000, "10"), (192, 384, 9_000_000, "00"), (192, 192, 9_000_000, "10"),
    (128, 512, 9_000_000, "00"), (128, 256, 9_000_000, "00"), (64, 512, 9_000_000, "00")])
def test_where_they_pay_against_staged_launches(rules, nx, tile, nodes, taken):
    rules.rows_pay.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_longlong, ctypes.c_int, ctypes.c_int]
    assert "".join(str(rules.rows_pay(2, nx, nodes, mixed, tile)) for mixed in (0, 1)) == taken


@pytest.mark.parametrize("tile,nodes,pairs", [
    (512, 2_099_999, 1), (512, 2_100_000, 0), (320, 2_100_000, 0), (256, 2_100_000, 1), (256, 2_599_999, 1),
    (256, 2_600_000, 0), (192, 2_600_000, 0), (160, 9_000_000, 1), (32, 9_000_000, 1)])
def test_pairs_or_staged_single_launches(rules, tile, nodes, pairs):
    rules.pairs_pay_2d.argtypes = [ctypes.c_longlong, ctypes.c_int]
    assert rules.pairs_pay_2d(nodes, tile) == pairs


# widths at which the tiles have 1, 1.5 and 2 times fewer lanes than the strips, or more
@pytest.mark.parametrize("nx,tile,pairs", [
    (32, 32, 0), (32, 64, 1), (48, 64, 1), (60, 64, 1), (62, 64, 0), (64, 64, 0), (64, 128, 1), (66, 64, 1),
    (96, 32, 1), (128, 64, 1), (128, 128, 1), (192, 64, 1), (1024, 64, 1), (63, 64, 0), (1, 32, 0), (2, 32, 0),
    (2, 1 << 20, 1), (64, 1 << 20, 1), (63, 1 << 20, 0), (1 << 21, 1 << 20, 1), ((1 << 31) - 2, 1 << 20, 1)])
def test_cases_of_a_batch_with_two_iterations_per_launch(rules, nx, tile, pairs):
    assert rules.rows_case(1, nx, tile) == pairs and rules.rows_case(0, nx, tile) == 1


@pytest.mark.gpu
def test_more_rows_than_a_grid_of_one_row_blocks():
    """160 wide, whole-row blocks while they fit: the height does not, and the result is that of blocks of 64 x 4."""
    nx, ny, nz = 160, 65540, 2
    m = M.get("d3q19")
    flags = np.full((nz, ny, nx), m.flag("MRT"), np.uint16)
    flags[np.random.default_rng(1).random(flags.shape) < 0.05] = m.flag("Wall")
    out = []
    for shape in (None, (64, 4)):
        g = Lattice("d3q19", nx, ny, nz, precision="fp32")
        if shape:
            g.set_launch(*shape)
        g.set_flags(flags)
        g.SetSetting("nu", 0.05)
        g.SetSetting("InletVelocity", 0.02)
        g.Init()
        g.Iterate(3, M.ITER_NORM)
        out.append(g.GetQuantity("U"))
        g.close()
    assert np.isfinite(out[0]).all() and np.abs(out[0]).max() > 1e-3
    assert np.array_equal(out[0], out[1])
