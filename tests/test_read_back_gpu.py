"""Results copied into pageable memory by several host threads equal those in
pinned memory: sizes below and above the split, and ones that fill neither the
last part nor the last chunk."""
import numpy as np
import pytest
import torch

from tclb_b200 import models as M
from tclb_b200.batch import Batch, CaseSpec
from tclb_b200.lattice import Lattice

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(64, 64, 64), (131, 97, 230), (128, 128, 192)])
def test_quantity_and_snapshot_in_pageable_and_pinned_memory(nx, ny, nz):
    g = Lattice("d3q19", nx, ny, nz, precision="fp32")
    g.set_flags(np.full((nz, ny, nx), M.get("d3q19").flag("MRT"), np.uint16))
    g.SetSetting("nu", 0.05)
    rng = np.random.default_rng(nx)
    g.init_equilibrium(1 + 0.01 * rng.standard_normal(nx * ny * nz), 0.01 * rng.standard_normal((nx * ny * nz, 3)))
    g.Iterate(2)
    n = g.snapshot_bytes()
    buf = torch.empty(n, dtype=torch.uint8, pin_memory=True).numpy()
    g.save(buf)
    assert np.array_equal(g.save(), buf)
    pinned = torch.empty((nz, ny, nx, 3), dtype=torch.float32, pin_memory=True).numpy()
    g.GetQuantity("U", out=pinned)
    for _ in range(2):
        assert np.array_equal(g.GetQuantity("U"), pinned)
    g.close()


def test_batch_quantity():
    flags = np.full((120, 160, 160), M.get("d3q19").flag("MRT"), np.uint16)
    b = Batch("d3q19", "fp32", budget_bytes=2 << 30)
    lat = Lattice("d3q19", 160, 160, 120, precision="fp32")
    c = b.add_case(CaseSpec(flags, {"nu": 0.05, "InletVelocity": 0.02, "ForceX": 1e-4}, {}, 6))
    b.run_to_completion()
    lat.set_flags(flags)
    for k, v in (("nu", 0.05), ("InletVelocity", 0.02), ("ForceX", 1e-4)):
        lat.SetSetting(k, v)
    lat.Init()
    lat.Iterate(6)
    pinned = torch.empty((120, 160, 160, 3), dtype=torch.float32, pin_memory=True).numpy()
    lat.GetQuantity("U", out=pinned)
    assert np.abs(b.quantity(c, "U") - pinned).max() < 1e-6
    b.close()
    lat.close()
