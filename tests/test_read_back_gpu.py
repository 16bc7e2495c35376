"""Results copied into pageable memory by several host threads equal those in
pinned memory: sizes below and above the split, and ones that fill neither the
last part nor the last chunk."""
import ctypes
import threading

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


def flow(nx, ny, nz, seed):
    """A lattice with a field of its own, and its velocity in pinned memory (a direct copy)."""
    g = Lattice("d3q19", nx, ny, nz, precision="fp32")
    g.set_flags(np.full((nz, ny, nx), M.get("d3q19").flag("MRT"), np.uint16))
    rng = np.random.default_rng(seed)
    g.init_equilibrium(1 + 0.01 * rng.standard_normal(nx * ny * nz), 0.01 * rng.standard_normal((nx * ny * nz, 3)))
    pinned = torch.empty((nz, ny, nx, 3), dtype=torch.float32, pin_memory=True).numpy()
    return g, g.GetQuantity("U", out=pinned)


def test_two_threads_and_two_lattices():
    """One copy at a time takes the lanes, the other goes directly; each result is its own lattice's."""
    made = [flow(120 + 8 * k, 128, 140, k) for k in range(2)]
    wrong = []

    def read(g, ref):
        try:
            for _ in range(12):
                if not np.array_equal(g.GetQuantity("U"), ref):
                    wrong.append("differs")
        except Exception as e:  # a thread's exception would be lost
            wrong.append(repr(e))

    threads = [threading.Thread(target=read, args=m) for m in made]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong
    for g, _ in made:
        g.close()


def test_lanes_given_back_and_made_again():
    for k in range(3):  # the only object each time: its end gives the lanes back
        g, ref = flow(128, 128, 100 + k, k)
        assert ref.nbytes >= 16 << 20
        for _ in range(2):
            assert np.array_equal(g.GetQuantity("U"), ref)
        g.close()


def test_batch_quantity_in_pageable_and_pinned_memory():
    b = Batch("d3q19", "fp32", budget_bytes=2 << 30)
    flags = np.full((120, 160, 160), M.get("d3q19").flag("MRT"), np.uint16)
    flags[np.random.default_rng(2).random(flags.shape) < 0.05] = M.get("d3q19").flag("Wall")
    c = b.add_case(CaseSpec(flags, {"nu": 0.05, "InletVelocity": 0.02, "ForceX": 1e-4}, {}, 6))
    b.run_to_completion()
    pinned = torch.empty((120, 160, 160, 3), dtype=torch.float32, pin_memory=True).numpy()
    q = M.get("d3q19").quantity_index("U")
    assert b.lib.tclb_batch_get_quantity(b._h, c, q, pinned.ctypes.data_as(ctypes.c_void_p), 1.0) == 0
    assert np.abs(pinned).max() > 1e-3
    for _ in range(2):
        assert b.quantity(c, "U").tobytes() == pinned.tobytes()
    b.close()
