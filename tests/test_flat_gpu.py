"""Widths that are not a multiple of 32: kernels over the flat node index."""
import numpy as np
import pytest

import oracle
from tclb_b200 import models as M
from tclb_b200.lattice import Lattice

from helpers import apply_params, perturbed_equilibrium, random_flags, rel_l2

pytestmark = pytest.mark.gpu

TYPES = {
    "d2q9": ["Wall", "Solid", "WVelocity", "EPressure", "NSymmetry"],
    "d3q19": ["Wall", "Solid", "WVelocity", "EPressure", "WPressure"],
    "d3q27_cumulant": ["Wall", "Solid", "WVelocity", "EPressure", "NVelocity"],
}
PARAMS = {
    "d2q9": [("setting", "Viscosity", 0.05), ("zone", "VelocityX", 0.02, 1)],
    "d3q19": [("setting", "nu", 0.05), ("setting", "InletVelocity", 0.02), ("setting", "ForceX", 1e-5)],
    "d3q27_cumulant": [("setting", "nu", 0.02), ("setting", "nubuffer", 0.05), ("zone", "Velocity", 0.02, 1)],
}


def run(model, fl, f0, precision, storage, niter, **launch):
    nz, ny, nx = fl.shape
    g = Lattice(model, nx, ny, nz, precision=precision, storage=storage)
    if launch:
        g.set_launch(128, 2, **launch)
    g.set_flags(fl)
    apply_params(g, PARAMS[model])
    g.set_densities(f0)
    g.Iterate(niter)
    g.sync()
    path, f = g.launch_path(), g.densities()
    g.close()
    return path, f


# rows shorter than a warp, rows that end anywhere in one, and a node count that
# fills neither the last warp nor the last block
@pytest.mark.parametrize("width", [2, 6, 50, 98])
@pytest.mark.parametrize("storage", ["fp16s", "bf16"])
@pytest.mark.parametrize("model", ["d2q9", "d3q19", "d3q27_cumulant"])
def test_flat_pairs_match_row_pairs_bit_for_bit(model, storage, width):
    """A lattice `width` wide and one of 32 or 64 periodic copies of it side by
    side, whose rows are whole warps of pairs, hold the same values."""
    copies = 32 if width * 32 > 512 and width * 32 % 64 == 0 else 64 * (1 + 512 // (64 * width))
    shape = (1, 13, width) if model == "d2q9" else (3, 5, width)
    fl = random_flags(model, shape, TYPES[model], zones=2, seed=width, p_type=0.15)
    f0 = perturbed_equilibrium(model, shape, seed=3)
    path, f = run(model, fl, f0, "fp32", storage, 5)
    assert path["pairs"] and not path["tma"]
    wide, fw = run(model, np.tile(fl, copies), np.tile(f0, copies), "fp32", storage, 5)
    assert wide["pairs"] and not wide["tma"] and (width * copies) % 64 == 0
    assert np.isfinite(f).all()
    assert np.array_equal(fw[..., :width], f) and np.array_equal(fw[..., -width:], f)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("model,shape", [
    ("d2q9", (1, 9, 33)), ("d2q9", (1, 31, 131)), ("d3q19", (5, 7, 131)), ("d3q19", (3, 11, 45)),
    ("d3q27_cumulant", (4, 6, 77)), ("d3q27_cumulant", (7, 3, 130))])
def test_flat_nodes_and_globals_match_the_oracle(model, shape, precision):
    """One node per thread of the flat index, and the Globals summed over it
    (blocks that are not full, more nodes than one block)."""
    fl = random_flags(model, shape, TYPES[model], zones=2, seed=7, p_type=0.2)
    f0 = perturbed_equilibrium(model, shape, seed=4)
    nz, ny, nx = shape
    g = Lattice(model, nx, ny, nz, precision=precision)
    o = oracle.OracleLattice(model, nx, ny, nz, precision=precision)
    for lat in (g, o):
        lat.set_flags(fl)
        apply_params(lat, PARAMS[model])
        lat.set_densities(f0)
    g.Iterate(6, M.ITER_NORM | M.ITER_LASTGLOB)
    o.iterate(6, M.ITER_NORM | M.ITER_LASTGLOB)
    # FP32: 6 iterations of about 100 roundings of 6e-8, on values of one size
    assert rel_l2(g.densities(), o.densities()) < {"fp64": 1e-13, "fp32": 2e-6}[precision]
    got, ref = np.asarray(g.globals), np.asarray(o.globals() if callable(o.globals) else o.globals)
    scale = np.abs(ref) + nx * ny * nz * 1e-2  # sums of N signed values of that size
    assert (np.abs(got - ref) / scale).max() < {"fp64": 1e-11, "fp32": 3e-4}[precision], (got, ref)
    g.close()
