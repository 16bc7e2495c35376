"""Two plain iterations per launch (2D lattices above a size): the same bits as
one iteration per launch, whose kernels the other tests hold to the oracle."""
import numpy as np
import pytest
import torch

from tclb_b200 import models as M
from tclb_b200.batch import Batch, CaseSpec
from tclb_b200.lattice import Lattice

from helpers import apply_params, random_flags

pytestmark = pytest.mark.gpu

TYPES = ["Wall", "Solid", "WVelocity", "EPressure", "NSymmetry", "EVelocity", "WPressure", "SVelocity"]
PARAMS = [("setting", "Viscosity", 0.05), ("setting", "S3", 0.3), ("setting", "S4", 0.2),
          ("setting", "GravitationX", 1e-6), ("setting", "GravitationY", -2e-6),
          ("zone", "VelocityX", 0.02, 1), ("zone", "Pressure", 0.01, 1)]
BOUNDARY, SOLID = M.get("d2q9").groups["BOUNDARY"][0], M.get("d2q9").flag("Solid")


def kernels(run):
    """Names of the kernels that run() launches (graph replays included)."""
    torch.zeros(1, device="cuda")
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        run()
    return " ".join(e.key for e in p.key_averages())


def start(nx, ny, precision, storage, flags, seed):
    """A lattice from a perturbed flow, with forces and boundary values of its own."""
    rng = np.random.default_rng(seed)
    real = np.float64 if precision == "fp64" else np.float32
    g = Lattice("d2q9", nx, ny, precision=precision, storage=storage)
    g.set_flags(flags)
    apply_params(g, PARAMS)
    g.init_equilibrium((1 + 0.01 * rng.standard_normal(nx * ny)).astype(real),
                       (0.02 * rng.standard_normal((nx * ny, 3))).astype(real))
    return g


# widths that do and do not divide into strips (60 columns in pairs, 30 one per
# lane), odd widths (one node per lane), heights below, at and off the 8 rows of
# a segment; the narrowest lattice that wraps inside one strip
@pytest.mark.parametrize("precision,storage,nx,ny", [
    ("fp32", "same", 1500, 1000), ("fp32", "same", 1498, 1003), ("fp32", "same", 1449, 1051),
    ("fp32", "same", 300000, 7), ("fp32", "same", 34, 45001), ("fp64", "same", 1024, 700), ("fp64", "same", 899, 801),
    ("fp64", "same", 250000, 3), ("fp32", "fp16s", 1920, 1304), ("fp32", "bf16s", 256, 10001),
    ("fp32", "fp16", 2560, 999)])
def test_two_iterations_per_launch_match_single_ones(precision, storage, nx, ny):
    fl = random_flags("d2q9", (1, ny, nx), TYPES, zones=2, seed=nx + ny, p_type=0.1)
    rng = np.random.default_rng(ny)
    real = np.float64 if precision == "fp64" else np.float32
    rho = (1 + 0.01 * rng.standard_normal(nx * ny)).astype(real)
    u = (0.02 * rng.standard_normal((nx * ny, 3))).astype(real)
    out = []
    for cuts in ([1] * 9, [9], [4, 5]):
        g = Lattice("d2q9", nx, ny, precision=precision, storage=storage)
        g.set_flags(fl)
        apply_params(g, PARAMS)
        g.init_equilibrium(rho, u)
        for n in cuts:
            g.Iterate(n, M.ITER_NORM)
        g.sync()
        assert g.iteration == 9
        out.append(g.save())
        g.close()
    assert np.isfinite(out[0].view({"fp64": np.float64}.get(precision, np.float32))).all() or storage != "same"
    assert out[0].tobytes() == out[1].tobytes()
    assert out[0].tobytes() == out[2].tobytes()


def test_graph_replays_of_two_iterations():
    """More iterations than a graph holds, in one call and one by one."""
    nx, ny = 1500, 1000
    fl = random_flags("d2q9", (1, ny, nx), TYPES[:2], seed=5, p_type=0.05)
    out = []
    for cuts in ([1] * 75, [75]):
        g = Lattice("d2q9", nx, ny, precision="fp32")
        g.set_flags(fl)
        apply_params(g, PARAMS)
        g.Init()
        for n in cuts:
            g.Iterate(n, M.ITER_NORM | M.ITER_LASTGLOB if n == cuts[-1] and len(cuts) == 1 else M.ITER_NORM)
        out.append(g.GetQuantity("U"))
        g.close()
    assert np.allclose(out[0], out[1], rtol=0, atol=1e-6)


# both sides of the rule, on flows with 0.2% and 10% of the nodes of another type (below and above 1% of the pairs
# with one node that collides): the kernel that ran, and single launches' bits from both
@pytest.mark.parametrize("precision,storage,nx,ny,p,two", [
    ("fp32", "same", 1500, 1000, 0.002, True), ("fp32", "same", 1500, 1000, 0.1, False),
    ("fp32", "same", 1450, 1531, 0.1, True), ("fp32", "same", 62, 24203, 0.002, True),
    ("fp32", "same", 62, 40001, 0.1, False), ("fp32", "same", 30, 52001, 0.002, False),
    ("fp32", "same", 192, 11461, 0.1, True), ("fp32", "same", 255, 5891, 0.1, True),
    ("fp32", "same", 91, 17001, 0.1, False), ("fp64", "same", 1025, 684, 0.1, True),
    ("fp64", "same", 64, 11001, 0.1, False), ("fp64", "same", 64, 17191, 0.1, True),
    ("fp64", "same", 31, 40001, 0.002, True), ("fp64", "same", 31, 40001, 0.1, False),
    ("fp32", "fp16s", 1922, 1302, 0.1, True), ("fp32", "bf16", 190, 13201, 0.002, True),
    ("fp32", "bf16s", 190, 13201, 0.1, False), ("fp32", "fp16", 66, 38001, 0.002, False),
    ("fp32", "bf16", 512, 4901, 0.002, True), ("fp32", "fp16s", 512, 4901, 0.1, False),
    ("fp32", "fp16s", 256, 10000, 0.002, False), ("fp32", "fp16s", 256, 10301, 0.002, True)])
def test_where_two_iterations_run(precision, storage, nx, ny, p, two):
    fl = random_flags("d2q9", (1, ny, nx), TYPES[:4], zones=2, seed=nx, p_type=p)
    fl[(fl & BOUNDARY) == SOLID] = SOLID  # no collision there
    out = []
    for cuts in ([1] * 5, [5]):
        g = start(nx, ny, precision, storage, fl, ny)

        def run():
            for n in cuts:
                g.Iterate(n, M.ITER_NORM)
            g.sync()

        assert ("k_iterate_rows" in kernels(run)) == (two and cuts == [5])
        out.append(g.save().tobytes())
        g.close()
    assert out[0] == out[1]


# 16-bit rows that can be staged: in pairs while the lattice stays in L2, staged beyond, the same bits
@pytest.mark.parametrize("nx,ny,kernel", [(256, 8202, "k_iterate_pair"), (256, 8204, "k_iterate_tma"),
                                          (256, 10155, "k_iterate_pair"), (256, 10157, "k_iterate_tma"),
                                          (96, 40001, "k_iterate_pair")])
def test_single_launches_of_staged_widths(nx, ny, kernel):
    fl = random_flags("d2q9", (1, ny, nx), TYPES[:4], zones=2, seed=4, p_type=0.05)
    out = []
    for launch in ({}, {"tma_always": True}, {"use_tma": False}):
        g = start(nx, ny, "fp32", "fp16s", fl, 6)
        if launch:
            g.set_launch(32, 4, **launch)
        assert (kernel in kernels(lambda: ([g.Iterate(1, M.ITER_NORM) for _ in range(3)], g.sync()))) or launch
        out.append(g.save().tobytes())
        g.close()
    assert out[0] == out[1] == out[2]


# the choice follows the node types: captured launches of the other kernel are dropped
def test_node_types_that_change_the_choice():
    nx, ny = 1500, 1010
    clean, porous = (random_flags("d2q9", (1, ny, nx), ["Solid"], seed=3, p_type=p) for p in (0.0, 0.1))
    porous[(porous & BOUNDARY) == SOLID] = SOLID
    out = []
    for cuts in ([40], [1] * 40):
        g = start(nx, ny, "fp32", "same", clean, 1)
        ran = []
        for fl in (clean, porous, clean):
            g.set_flags(fl)
            ran.append("k_iterate_rows" in kernels(lambda: ([g.Iterate(n, M.ITER_NORM) for n in cuts], g.sync())))
        assert ran == ([True, False, True] if cuts == [40] else [False] * 3)
        out.append(g.save().tobytes())
        g.close()
    assert out[0] == out[1]


@pytest.mark.parametrize("precision,storage,nx,ny", [
    ("fp32", "same", 1500, 1010), ("fp64", "same", 1024, 700), ("fp32", "fp16s", 1920, 1304)])
def test_graph_replays_equal_single_launches(precision, storage, nx, ny):
    """More iterations than a graph holds, in one call and one by one, bit for bit from a flow."""
    fl = random_flags("d2q9", (1, ny, nx), TYPES[:4], zones=2, seed=5, p_type=0.002)
    out = []
    for cuts in ([1] * 75, [75]):
        g = start(nx, ny, precision, storage, fl, 2)
        for n in cuts:
            g.Iterate(n, M.ITER_NORM)
        u = g.GetQuantity("U")
        assert np.isfinite(u).all() and np.abs(u).max() > 1e-3
        out.append(g.save().tobytes())
        g.close()
    assert out[0] == out[1]


# iterations per replay even, odd and one; iteration counts that end anywhere in
# a replay; a case of odd width (one iteration per launch among the others in
# FP32); Globals in every replay and at the end
@pytest.mark.parametrize("at_end", [True, False])
@pytest.mark.parametrize("K", [1, 5, 8])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_batch_of_two_iterations_per_launch(precision, K, at_end):
    shapes = [(1000, 1600), (45, 301), (64, 128), (257, 640)]
    iters = [13, 10, 3, 16]
    b = Batch("d2q9", precision, budget_bytes=8 << 30)
    b.set_paths(globals_at_end=at_end)
    b.set_launch(64, 16, K)
    specs = [CaseSpec(random_flags("d2q9", (1,) + sh, TYPES[:2] + ["WVelocity"], zones=2, seed=k, p_type=0.05),
                      {"Viscosity": 0.05, "GravitationX": 1e-6}, {0: {"VelocityX": 0.02}, 1: {"VelocityX": 0.01}}, n)
             for k, (sh, n) in enumerate(zip(shapes, iters))]
    ids = [b.add_case(s) for s in specs]
    b.run_to_completion()
    for cid, s in zip(ids, specs):
        assert b.poll(cid) == (s.niter, 0)
        ny, nx = s.flags.shape[1:]
        g = Lattice("d2q9", nx, ny, precision=precision)
        g.set_flags(s.flags)
        apply_params(g, [("setting", k, v) for k, v in s.settings.items()])
        for z, d in s.zone_settings.items():
            g.set_zone_setting("VelocityX", d["VelocityX"], z)
        g.Init()
        g.Iterate(s.niter, M.ITER_NORM | M.ITER_LASTGLOB)
        assert np.array_equal(b.quantity(cid, "U"), g.GetQuantity("U")), (nx, ny)
        # FP64 sums in another order
        assert np.allclose(b.globals(cid), g.globals, rtol=1e-6 if precision == "fp32" else 1e-9, atol=1e-9)
        g.close()
    b.close()


# widths that strips fit and that they do not, even and odd, in one batch; nodes enough for two iterations per launch,
# and not enough; in FP32 the narrow cases with nodes enough for launches of their own, and without
@pytest.mark.parametrize("precision,shapes,two,one", [
    ("fp32", [(1000, 1500), (97, 64), (41, 128), (33, 32), (40, 66)], True, False),
    ("fp32", [(1000, 1500), (97, 64), (41, 128), (55, 301), (33, 32), (40, 66)], True, True),
    ("fp32", [(1000, 1500), (23500, 64), (41, 128)], True, True),
    ("fp32", [(1000, 1300), (23500, 64), (41, 128)], False, True),
    ("fp64", [(1000, 700), (97, 64), (55, 301), (33, 32)], True, False),
    ("fp64", [(1000, 640), (97, 64), (55, 301)], False, True)])
def test_which_cases_of_a_batch_take_two_iterations(precision, shapes, two, one):
    b = Batch("d2q9", precision, budget_bytes=8 << 30)
    b.set_launch(64, 16, 5)
    specs = [CaseSpec(random_flags("d2q9", (1,) + sh, TYPES[:2], seed=k, p_type=0.05),
                      {"Viscosity": 0.05, "GravitationX": 1e-5}, {0: {"VelocityX": 0.02}}, 12)
             for k, sh in enumerate(shapes)]
    ids = [b.add_case(s) for s in specs]
    ran = kernels(b.step)
    assert ("k_iterate_batch_rows" in ran) == two
    assert ("BatchRole)0" in ran) == one, ran  # ROLE_PLAIN: one iteration per launch
    b.run_to_completion()
    for cid, s in zip(ids, specs):
        assert b.poll(cid) == (s.niter, 0)
        ny, nx = s.flags.shape[1:]
        g = Lattice("d2q9", nx, ny, precision=precision)
        g.set_flags(s.flags)
        apply_params(g, [("setting", "Viscosity", 0.05), ("setting", "GravitationX", 1e-5), ("zone", "VelocityX", 0.02, 0)])
        g.Init()
        g.Iterate(s.niter, M.ITER_NORM | M.ITER_LASTGLOB)
        assert np.array_equal(b.quantity(cid, "U"), g.GetQuantity("U")), (nx, ny)
        g.close()
    b.close()
