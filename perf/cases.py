"""Timed cases of the lattice-Boltzmann engine: the runs a user's program makes.

Each case is one pass of a program that holds a lattice (or a batch of them)
on the GPU: ``Lattice.Iterate`` over some logging intervals with the Globals
integrated on the last iteration of each (TCLB's ``<Solve>`` with ``<Log>``),
then the velocity field read back into the program's own pinned buffer
(``<VTK>`` / ``<BIN>``). The Taylor-Green cases also read the kinetic energy
and the enstrophy at each interval. The batch cases take a set of requests
through admission, ``Batch.run_to_completion``, the read-back of each result
and the retirement of the case, as the serving loop does.

``listed`` are the sizes of the repository's configurations and tests, from
one iteration on a small channel to the 256^3 vortex; ``draw`` gives others of
the same families: any size between, widths that are and are not multiples of
32 (the case-file reader pads to 32, the lattice API takes any width), each
precision and the shifted 16-bit storages.

``exact`` restates the three models in FP64 torch operations (dense moment
matrices and index lists, no code of the package): what ``run`` returns from
the same inputs.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from tclb_b200 import cases as C
from tclb_b200 import models as M
from tclb_b200.batch import Batch, CaseSpec
from tclb_b200.lattice import Lattice

LOG = M.ITER_NORM | M.ITER_LASTGLOB
MODEL = {"channel": "d2q9", "vortex19": "d3q19", "vortex27": "d3q27_cumulant", "porous": "d3q19",
         "duct": "d3q27_cumulant", "batch-channel": "d2q9", "batch-porous": "d3q19"}
QS = {"d2q9": 9, "d3q19": 19, "d3q27_cumulant": 27}
# floating-point operations of one node update (moments, relaxation, populations)
FLOPS = {"d2q9": 150, "d3q19": 250, "d3q27_cumulant": 480}


def _one(name, family, nx, ny, nz, precision, storage, every, logs):
    c = {"family": family, "nx": nx, "ny": ny, "nz": nz, "precision": precision, "storage": storage,
         "every": every, "logs": logs}
    return dict(c, name=name) if name else c


def _batch(name, family, count, smin, smax, precision, storage, iters):
    c = {"family": family, "count": count, "smin": smin, "smax": smax, "precision": precision, "storage": storage,
         "iters": iters}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a program that couples to the flow (PID, Sample): one iteration of a
        # small channel, its Globals and its velocity field, at every step
        _one("channel-step", "channel", 128, 48, 1, "fp32", "same", 1, 1),
        # configuration 1: the double-precision channel with a disc, logged every 100
        _one("channel-fp64", "channel", 1024, 256, 1, "fp64", "same", 100, 5),
        # the large d2q9 channel the batched rates are compared with
        _one("channel-large", "channel", 4096, 1024, 1, "fp32", "same", 50, 4),
        # configuration 2, the headline: d3q27 Taylor-Green vortex, energy and enstrophy every 50
        _one("vortex27-fp32", "vortex27", 256, 256, 256, "fp32", "same", 50, 2),
        # the same vortex in shifted 16-bit storage
        _one("vortex27-fp16s", "vortex27", 256, 256, 256, "fp32", "fp16s", 50, 2),
        # and in double precision, at half the edge
        _one("vortex27-fp64", "vortex27", 128, 128, 128, "fp64", "same", 50, 2),
        # configuration 3 at half the edge: d3q19 body-force flow through porous solids
        _one("porous-fp32", "porous", 192, 96, 96, "fp32", "same", 100, 2),
        # configuration 3 at its size in shifted 16-bit storage
        _one("porous-fp16s", "porous", 384, 192, 192, "fp32", "fp16s", 100, 1),
        # a porous sample as scanned, not padded: odd widths
        _one("porous-odd", "porous", 131, 93, 77, "fp32", "same", 100, 1),
        # flow past a sphere in a duct, drag logged every 10 iterations
        _one("duct-fp32", "duct", 192, 64, 64, "fp32", "same", 10, 20),
        # configuration 4's mix of d2q9 channels as one batch, admission to read-back
        _batch("batch-channel-fp32", "batch-channel", 24, 64, 2048, "fp32", "same", 500),
        # configuration 5's d3q19 porous boxes as one batch in 16-bit storage
        _batch("batch-porous-fp16s", "batch-porous", 6, 64, 192, "fp32", "fp16s", 400),
    ]


def _size(rng, lo, hi):
    """Log-uniform in [lo, hi]; a multiple of 32 half of the time."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, (n + 31) // 32 * 32)) if rng.random() < 0.5 else n


def draw(rng):
    # the work of a drawn case: at most that of the 256^3 vortex over 100 iterations
    family = rng.choice(["channel", "channel", "vortex19", "vortex27", "porous", "porous", "duct", "batch-channel",
                         "batch-porous"])
    precision, storage = rng.choice([("fp64", "same"), ("fp32", "same"), ("fp32", "same"), ("fp32", "fp16s"),
                                     ("fp32", "fp16s"), ("fp32", "bf16s")])
    if family == "batch-channel":
        return _batch(None, family, rng.randint(4, 24), 64, rng.choice([512, 1024, 2048]), "fp32",
                      rng.choice(["same", "fp16s"]), rng.randint(100, 500))
    if family == "batch-porous":
        return _batch(None, family, rng.randint(2, 6), 64, rng.choice([96, 128, 192]), "fp32",
                      rng.choice(["same", "fp16s"]), rng.randint(50, 400))
    if family == "channel":
        nx = _size(rng, 96, 4096)
        ny, nz, logs = max(32, int(nx * rng.uniform(0.15, 0.5))), 1, rng.randint(1, 5)
    elif family == "duct":
        nx = _size(rng, 96, 256)
        ny = max(32, int(nx * rng.uniform(0.3, 0.5)))
        nz, logs = ny, rng.randint(1, 10)
    else:
        nx, ny, nz = _size(rng, 48, 256), _size(rng, 40, 200), _size(rng, 40, 200)
        logs = rng.randint(1, 3)
    every = rng.choice([1, 10, 50, 100])
    budget = 3e8 if precision == "fp64" else 6e8  # node updates
    every = max(1, min(every, int(budget / (nx * ny * nz * logs))))
    return _one(None, family, nx, ny, nz, precision, storage, every, logs)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _vortex(nx, ny, nz, rng, dtype):
    """rho and u of a Taylor-Green vortex with a phase and an amplitude of its own, in `dtype`."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    px, py, pz = rng.uniform(0, 2 * math.pi, 3)
    u0 = rng.uniform(0.035, 0.05)
    x = 2 * math.pi * (torch.arange(nx, dtype=torch.float64, device=dev) + 0.5) / nx + px
    y = 2 * math.pi * (torch.arange(ny, dtype=torch.float64, device=dev) + 0.5) / ny + py
    z = (2 * math.pi * (torch.arange(nz, dtype=torch.float64, device=dev) + 0.5) / nz + pz)[:, None, None]
    x, y = x[None, None, :], y[None, :, None]
    u = torch.zeros(nz, ny, nx, 3, dtype=torch.float64, device=dev)
    u[..., 0] = u0 * torch.sin(x) * torch.cos(y) * torch.cos(z)
    u[..., 1] = -u0 * torch.cos(x) * torch.sin(y) * torch.cos(z)
    rho = 1 + 3 * u0 * u0 / 16 * (torch.cos(2 * x) + torch.cos(2 * y)) * (torch.cos(2 * z) + 2)
    t = torch.float64 if dtype == np.float64 else torch.float32
    return rho.to(t).cpu().numpy(), u.to(t).cpu().numpy()


def _inputs(case, seed):
    """Node types, settings, zonal settings and initial fields (or None) of a single lattice."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    fam = case["family"]
    fields = None
    if fam == "channel":
        nu = rng.uniform(0.018, 0.025)
        flags = C.channel_disc_d2q9(nx, ny, r=max(2, ny // 16), cx=int(nx * rng.uniform(0.2, 0.3)),
                                    cy=int(ny * rng.uniform(0.4, 0.6)))
        keep = 1 - 1 / (3 * nu + 0.5)
        settings = {"Viscosity": nu, "S3": keep, "S4": keep}
        zones = {"VelocityX": rng.uniform(0.008, 0.02)}
    elif fam in ("vortex19", "vortex27"):
        flags = np.full((nz, ny, nx), M.get(MODEL[fam]).flag("MRT"), np.uint16)
        settings = {"nu": 1e-2 if fam == "vortex19" else 1e-3}
        zones = {}
        fields = _vortex(nx, ny, nz, rng, np.float64 if case["precision"] == "fp64" else np.float32)
    elif fam == "porous":
        flags = C.porous_channel_d3q19(nx, ny, nz, p=0.08, band=4, seed=int(seed))
        settings = {"nu": 0.01, "ForceX": 1e-5, "InletVelocity": rng.uniform(0.008, 0.012)}  # initial velocity
        zones = {}
    else:  # duct
        flags, _ = C.sphere_channel_d3q27(nx, ny, nz, r=max(3, ny // 8), cx=int(nx * rng.uniform(0.22, 0.3)))
        settings = {"nu": rng.uniform(0.018, 0.025), "nubuffer": 0.02}
        zones = {"Velocity": rng.uniform(0.015, 0.02)}
    return flags, settings, zones, fields


def _sizes(case):
    """(nz, ny, nx) of each lattice of a case: a batch's are spread over the logarithm of its range."""
    if "count" not in case:
        return [(case["nz"], case["ny"], case["nx"])]
    n, lo, hi = case["count"], case["smin"], case["smax"]
    out = []
    for k in range(n):
        s = C.pad_nx(int(round(lo * (hi / lo) ** ((k + 0.5) / n))))
        out.append((1, max(32, s // 4), s) if case["family"] == "batch-channel" else (s, s, s))
    return out


def _specs(case, seed):
    rng = np.random.default_rng(seed)
    specs = []
    for k, (nz, ny, nx) in enumerate(_sizes(case)):
        if case["family"] == "batch-channel":
            r = rng.uniform(ny / 16, ny / 6)
            flags = C.channel_disc_d2q9(nx, ny, int(r), int(rng.uniform(r + 1, max(r + 2, nx / 3))),
                                        int(rng.uniform(r + 1, ny - r - 2)))
            nu = max(0.02 * 2 * r / rng.uniform(20.0, 200.0), 0.0026)
            specs.append(CaseSpec(flags, {"Viscosity": nu}, {z: {"VelocityX": 0.02} for z in range(3)},
                                  case["iters"]))
        else:
            flags = C.porous_channel_d3q19(nx, ny, nz, p=float(rng.uniform(0.02, 0.15)), band=2,
                                           seed=int(seed) * 1000 + k)
            specs.append(CaseSpec(flags, {"nu": 0.02, "ForceX": 1e-5, "InletVelocity": 0.01}, {}, case["iters"]))
    return specs


def prepare(case, seed):
    model, fam = MODEL[case["family"]], case["family"]
    if "count" in case:
        b = Batch(model, case["precision"], case["storage"], budget_bytes=16 << 30, max_cases=64)
        b.set_paths(globals_at_end=True)  # a result's Globals are read when it is done
        b.set_launch(64, 64 if fam == "batch-porous" else 32, 16)
        b.reserve(4 << 30)
        return {"batch": b, "specs": _specs(case, seed)}
    flags, settings, zones, fields = _inputs(case, seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    lat = Lattice(model, nx, ny, nz, precision=case["precision"], storage=case["storage"])
    lat.FlagOverwrite(flags)
    for k, v in settings.items():
        lat.SetSetting(k, v)
    for k, v in zones.items():
        lat.set_zone_setting(k, v)
    lat.Init()
    if fields is not None:
        lat.init_equilibrium(*fields)
    dt = torch.float64 if case["precision"] == "fp64" else torch.float32
    u = torch.empty((nz, ny, nx, 3), dtype=dt, pin_memory=True).numpy()
    return {"lattice": lat, "u": u, "every": case["every"], "logs": case["logs"], "energy": fields is not None}


def run(state):
    if "batch" in state:
        b = state["batch"]
        ids = [b.add_case(s) for s in state["specs"]]
        b.run_to_completion()
        out = {"globals": [b.globals(i) for i in ids], "u": [b.quantity(i, "U") for i in ids]}
        for i in ids:
            b.remove_case(i)
        out["globals"] = np.array(out["globals"])
        return out
    lat = state["lattice"]
    out = {"globals": [], "energy": []}
    for _ in range(state["logs"]):
        lat.Iterate(state["every"], LOG)
        out["globals"].append(lat.globals)
        if state["energy"]:
            out["energy"].append(lat.energy_enstrophy())
    out["globals"] = np.array(out["globals"])
    out["energy"] = np.array(out["energy"]) if state["energy"] else None
    out["u"] = lat.GetQuantity("U", out=state["u"])
    return out


def work(case):
    """The state and node types read once, the state and the results written once; every iteration's arithmetic."""
    q, model = QS[MODEL[case["family"]]], MODEL[case["family"]]
    real = 8 if case["precision"] == "fp64" else 4
    elem = real if case["storage"] == "same" else 2
    nodes = sum(a * b * c for a, b, c in _sizes(case))
    iters = case["iters"] if "count" in case else case["every"] * case["logs"]
    return {"bytes": nodes * (2 * q * elem + 2 + 3 * real), "flops": float(nodes) * iters * FLOPS[model]}


def tolerance(case):
    # About four times the largest error against exact() seen on B200, whatever
    # kernel ran. A velocity is a small difference of populations, so FP32 shows
    # 2.6e-5 on the porous flows and the vortices, 1.6e-4 on small channels and
    # porous boxes started from rest, and 6.1e-4 on the batched channels, which
    # run close to the smallest stable viscosity (FP16-shift there: 2.9e-2).
    # FP64 5.8e-13, FP16-shift 8e-4, BF16-shift 7e-3.
    fam = case["family"]
    if case["precision"] == "fp64":
        return {"rel": 2.5e-12}
    if case["storage"] == "same":
        return {"rel": {"batch-channel": 2.5e-3, "channel": 7e-4, "batch-porous": 6e-4}.get(fam, 1e-4)}
    if case["storage"] == "bf16s" or fam == "batch-channel":
        return {"rel": 3e-2, "max": 0.5}
    return {"rel": 4e-3, "max": 0.1}


# ---------------------------------------------------------------------------
# FP64 restatement of the models
# ---------------------------------------------------------------------------
_D = (0, 1, -1)
VELOCITIES = {
    "d2q9": [(0, 0, 0), (1, 0, 0), (0, 1, 0), (-1, 0, 0), (0, -1, 0), (1, 1, 0), (-1, 1, 0), (-1, -1, 0), (1, -1, 0)],
    "d3q19": [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, 1, 0),
              (1, -1, 0), (-1, -1, 0), (1, 0, 1), (-1, 0, 1), (1, 0, -1), (-1, 0, -1), (0, 1, 1), (0, -1, 1),
              (0, 1, -1), (0, -1, -1)],
    "d3q27_cumulant": [(a, b, c) for c in _D for b in _D for a in _D],
}
# lattice weights by the number of non-zero components
WEIGHTS = {"d2q9": [4 / 9, 1 / 9, 1 / 36], "d3q19": [1 / 3, 1 / 18, 1 / 36],
           "d3q27_cumulant": [8 / 27, 2 / 27, 1 / 54, 1 / 216]}


class _Flow:
    """One lattice in FP64: f[q, z, y, x], pulled with periodic wrap. The package gives only the inputs' encoding
    (the node-type bits)."""

    def __init__(self, model, flags, settings, zones):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.m = M.get(model)
        self.ev = VELOCITIES[model]
        self.e = torch.tensor(self.ev, dtype=torch.float64, device=self.dev)
        self.w = torch.tensor([WEIGHTS[model][sum(c != 0 for c in v)] for v in self.ev], dtype=torch.float64,
                              device=self.dev)
        self.opp = [self.ev.index(tuple(-c for c in v)) for v in self.ev]
        self.shape = flags.shape
        self.fl = torch.from_numpy(flags.astype(np.int64)).reshape(-1).to(self.dev)
        self.s = {"nu": 0.0, "nubuffer": 0.01, "InletVelocity": 0.0, "ForceX": 0.0, "ForceY": 0.0, "ForceZ": 0.0,
                  "GalileanCorrection": 1.0, "S3": 0.0, "S4": 0.0}  # the settings' defaults
        self.s.update(settings)
        self.omega = 1 / (3 * self.s.get("Viscosity", self.s["nu"]) + 0.5)
        self.z = zones
        group, _ = self.m.groups["BOUNDARY"]
        self.sites = {}
        for name, (v, mask, grp) in self.m.node_types.items():
            if grp == "BOUNDARY":
                at = torch.nonzero((self.fl & group) == v).reshape(-1)
                if at.numel():
                    self.sites[name] = at
        self.wall = (self.fl & group) == self.m.node_types["Wall"][0]
        self.mrt = (self.fl & self.m.groups["COLLISION"][0]) == self.m.node_types["MRT"][0]

    def pull(self):
        f = self.f.reshape((-1,) + self.shape)
        return torch.stack([torch.roll(f[i], (v[2], v[1], v[0]), (0, 1, 2)) for i, v in enumerate(self.ev)]).reshape(
            len(self.ev), -1)

    def zouhe(self, g, axis, inward, velocity=None, rho=None):
        """Zou-He at the sites g[q, n]: a face whose unknowns point `inward` (+1 / -1) along `axis`."""
        ea = self.e[:, axis] * inward
        s = g[ea == 0].sum(0) + 2 * g[ea < 0].sum(0)
        j = torch.zeros(3, g.shape[1], dtype=g.dtype, device=g.device)
        if velocity is not None:
            j[axis] = velocity * s / (1 - inward * velocity)
        else:
            j[axis] = inward * (rho - s)
        for t in range(3):
            if t != axis:
                j[t] = -3 * (self.e[:, t][ea == 0, None] * g[ea == 0]).sum(0)
        new = g.clone()
        for i in range(len(self.ev)):
            if float(ea[i]) > 0:
                new[i] = g[self.opp[i]] + 6 * self.w[i] * (self.e[i][:, None] * j).sum(0)
        return new

    def moments(self, f):
        return f.sum(0), self.e.t() @ f

    def start(self, fields):
        n = self.fl.numel()
        if fields is None:
            rho, u = self.initial()
            rho = torch.full((n,), rho, dtype=torch.float64, device=self.dev)
            v = torch.zeros(3, n, dtype=torch.float64, device=self.dev)
            v[0] = u
            if self.m.name != "d3q19":  # walls start at rest
                v[:, self.wall] = 0
        else:
            rho = torch.from_numpy(fields[0].astype(np.float64)).reshape(-1).to(self.dev)
            v = torch.from_numpy(fields[1].astype(np.float64)).reshape(-1, 3).t().to(self.dev)
        self.f = self.feq(rho, rho * v)

    def initial(self):
        return 1.0, self.s["InletVelocity"] if self.m.name == "d3q19" else self.z.get(
            "VelocityX", self.z.get("Velocity", 0.0))

    def feq(self, rho, j):
        """Second-order equilibrium."""
        eu = self.e @ j
        return self.w[:, None] * (rho + 3 * eu + 4.5 * eu * eu / rho - 1.5 * (j * j).sum(0) / rho)

    def iterate(self, n, last_globals):
        for k in range(n):
            want = last_globals and k == n - 1
            p = self.pull()
            extra = self.boundaries(p)
            g = self.globals(p, extra) if want else None
            self.f = torch.where(self.mrt, self.collide(p), p)
        return g

    def velocity(self):
        p = self.pull()
        u = self.read(p)
        return u.t().reshape(self.shape + (3,))

    def energy(self):
        u = self.velocity()

        def d(c, axis):
            return 0.5 * (torch.roll(u[..., c], -1, axis) - torch.roll(u[..., c], 1, axis))

        curl = (d(2, 1) - d(1, 0), d(0, 0) - d(2, 2), d(1, 2) - d(0, 1))
        return [0.5 * float((u * u).sum()), 0.5 * float(sum((c * c).sum() for c in curl))]


class _D2Q9(_Flow):
    def __init__(self, *a):
        super().__init__(*a)
        x, y = self.e[:, 0], self.e[:, 1]
        b = torch.stack([x * 0 + 1, x, y, 3 * x * x - 1, 3 * y * y - 1, 3 * x * y, 3 * x * x * y - y, 3 * x * y * y - x,
                         9 * x * x * y * y - 3 * x * x - 3 * y * y + 1])
        keep = torch.tensor([1.0] * 3 + [1 - self.omega] * 3 + [self.s["S3"]] * 2 + [self.s["S4"]], dtype=torch.float64,
                            device=self.dev)
        back = (b / (b * b * self.w).sum(1, keepdim=True) * self.w).t()
        self.relax = back @ (keep[:, None] * b)

    def boundaries(self, p):
        for name, at in self.sites.items():
            g = p[:, at]
            if name in ("Wall", "Solid"):
                p[:, at] = g[self.opp]
            elif name == "WVelocity":
                p[:, at] = self.zouhe(g, 0, 1, velocity=self.z["VelocityX"])
            elif name == "EPressure":
                p[:, at] = self.zouhe(g, 0, -1, rho=1.0)

    def collide(self, p):
        rho, j = self.moments(p)
        eq = self.feq(rho, j)
        return eq + self.relax @ (p - eq)

    def globals(self, p, _):
        rho, j = self.moments(p)
        flux = j[0] / rho / rho
        loss = flux * ((rho - 1) / 3 + (j[0] ** 2 + j[1] ** 2) / rho ** 2 / rho / 2)
        obj = self.fl & self.m.groups["OBJECTIVE"][0]
        out = self.mrt & (obj == self.m.node_types["Outlet"][0])
        inl = self.mrt & (obj == self.m.node_types["Inlet"][0])
        return [float(loss[inl].sum() - loss[out].sum()), float(flux[out].sum()), float(flux[inl].sum()), 0.0]

    def read(self, p):
        rho, j = self.moments(p)
        return j / rho


class _D3Q19(_Flow):
    """Two rates: gamma1 on the part even under e -> -e, gamma2 on the odd part."""

    def feq(self, rho, j):
        """Equilibrium of the d'Humieres moment basis."""
        out = []
        q = j * j / rho
        for i, v in enumerate(self.ev):
            nz = [a for a in range(3) if v[a]]
            odd = sum(v[a] * j[a] for a in nz) if nz else 0
            if not nz:
                out.append((rho - q.sum(0)) / 3)
            elif len(nz) == 1:
                out.append(rho / 18 + (2 * q[nz[0]] - q.sum(0)) / 6 + odd / 6)
            else:
                a, b = nz
                out.append(rho / 36 + (q[a] + q[b]) / 12 + v[a] * v[b] * j[a] * j[b] / rho / 4 + odd / 12)
        return torch.stack(out)

    def boundaries(self, p):
        for name, at in self.sites.items():
            if name in ("Wall", "Solid"):
                p[:, at] = p[:, at][self.opp]

    def force(self):
        return torch.tensor([[self.s["ForceX"]], [self.s["ForceY"]], [self.s["ForceZ"]]], dtype=torch.float64,
                            device=self.dev)

    def collide(self, p):
        om = self.omega
        g1, g2 = 1 - om, 1 - 8 * (2 - om) / (8 - om)
        rho, j = self.moments(p)
        d = p - self.feq(rho, j)
        r = d[self.opp]
        return self.feq(rho, j + rho * self.force()) + 0.5 * (g1 + g2) * d + 0.5 * (g1 - g2) * r

    def globals(self, p, _):
        # density and momentum divided by their squared column norms, as the model's moments are
        rho, j = self.moments(p)
        rs, js = rho / 19, (j + rho * self.force()) / 10
        u = js / rs
        names = [g[0] for g in self.m.globals]
        out = [0.0] * len(names)
        at = self.mrt
        for k, a in enumerate("xyz"):
            out[names.index("VOLv" + a)] = float(u[k][at].sum())
            out[names.index("VOLp" + a)] = float(js[k][at].sum())
        out[names.index("VOLrho")] = float(rs[at].sum())
        out[names.index("VOLvolume")] = float(at.sum())
        out[names.index("MaxV")] = float((u * u).sum(0)[at].max().sqrt())
        return out

    def read(self, p):
        rho, j = self.moments(p)
        return torch.where(self.wall, torch.zeros_like(j), j / rho)


class _D3Q27(_Flow):
    """Cumulant collision with Galilean correction; cumulants above order 2 are zero (Omega = 1)."""

    def __init__(self, *a):
        super().__init__(*a)
        t = np.array([[1.0, 1, 1], [0, 1, -1], [0, 1, 1]])  # moments 0, 1, 2 of the directions (0, +1, -1)
        k = np.kron(t, np.kron(t, t))
        self.to_raw = torch.tensor(k, device=self.dev)
        self.from_raw = torch.tensor(np.linalg.inv(k), device=self.dev)

    def boundaries(self, p):
        drag = torch.zeros(3, dtype=torch.float64, device=self.dev)
        body, _ = self.m.groups["BODY"]
        for name, at in self.sites.items():
            g = p[:, at]
            if name == "Wall":
                on = (self.fl[at] & body) == self.m.node_types["Body"][0]
                drag = 2 * (self.e.t() @ g[:, on]).sum(1)
                p[:, at] = g[self.opp]
            elif name == "WVelocity":
                p[:, at] = self.zouhe(g, 0, 1, velocity=self.z["Velocity"])
            elif name == "EPressure":
                p[:, at] = self.zouhe(g, 0, -1, rho=1.0)
        return drag

    def collide(self, p):
        s, w = self.s, self.omega
        wb = 1 / (3 * s["nubuffer"] + 0.5)
        b = (self.fl & self.m.groups["BOUNDARY"][0]) != 0
        w = torch.where(b, torch.full_like(p[0], wb), torch.full_like(p[0], w))
        m = self.to_raw @ p
        rho = m[0]
        u = [m[1] / rho, m[3] / rho, m[9] / rho]
        c = {}
        for k, (a, i) in enumerate(((0, 1), (1, 3), (2, 9))):
            c[i] = u[a]
        for i, (a, j) in ((2, (0, 0)), (6, (1, 1)), (18, (2, 2)), (4, (0, 1)), (10, (0, 2)), (12, (1, 2))):
            c[i] = m[i] / rho - u[a] * u[j]
        F = [s["ForceX"], s["ForceY"], s["ForceZ"]]
        v2 = [(u[a] + F[a] / (2 * rho)) ** 2 for a in range(3)]
        sxy, sxz, tr = c[2] - c[6], c[2] - c[18], c[2] + c[6] + c[18]
        dx = -w / 2 * (sxy + sxz) - (tr - 1) / 2
        dy, dz = dx + 1.5 * w * sxy, dx + 1.5 * w * sxz
        gc = s["GalileanCorrection"]
        A = (1 - w) * sxy - 3 * (1 - w / 2) * (v2[0] * dx - v2[1] * dy) * gc
        B = (1 - w) * sxz - 3 * (1 - w / 2) * (v2[0] * dx - v2[2] * dz) * gc
        T = 1 - 1.5 * (v2[0] * dx + v2[1] * dy + v2[2] * dz) * gc
        n = {1: c[1] + F[0], 3: c[3] + F[1], 9: c[9] + F[2], 2: (A + B + T) / 3, 6: (T - 2 * A + B) / 3,
             18: (T - 2 * B + A) / 3, 4: (1 - w) * c[4], 10: (1 - w) * c[10], 12: (1 - w) * c[12]}
        # moments from cumulants: m_{n+e} = sum_k binom(n, k) c_{k+e} m_{n-k}
        out = [rho]
        for i in range(1, 27):
            d = [i % 3, (i // 3) % 3, i // 9]
            ax = next(a for a in range(3) if d[a])
            d[ax] -= 1
            total = 0
            for kx in range(d[0] + 1):
                for ky in range(d[1] + 1):
                    for kz in range(d[2] + 1):
                        k = [kx, ky, kz]
                        j = [d[a] - k[a] for a in range(3)]
                        coef = math.prod(math.comb(d[a], k[a]) for a in range(3))
                        k[ax] += 1
                        if sum(k) <= 2:
                            total = total + coef * n[k[0] + 3 * k[1] + 9 * k[2]] * out[j[0] + 3 * j[1] + 9 * j[2]]
            out.append(total)
        return self.from_raw @ torch.stack(out)

    def globals(self, p, drag):
        rho, j = self.moments(p)
        at = self.mrt
        u = j[:, at] / rho[at]
        mass = float(rho[at].sum())
        mom = [float((rho[at] * u[k]).sum()) for k in range(3)]
        # Density, Flux, Drag, Lift, Lateral, Mass, momenta, Objective
        return [mass, float(u[0].sum()), float(drag[0]), float(drag[2]), float(drag[1]), mass] + mom + [0.0]

    def read(self, p):
        self.boundaries(p)
        rho, j = self.moments(p)
        return torch.where(self.wall, torch.zeros_like(j), j / rho)


_FLOWS = {"d2q9": _D2Q9, "d3q19": _D3Q19, "d3q27_cumulant": _D3Q27}


def _seconds(model, nodes, iters):
    """Rough time of the FP64 restatement on a GPU."""
    ops = {"d2q9": 90, "d3q19": 260, "d3q27_cumulant": 420}[model]
    return iters * ops * max(1.2e-5, nodes * 24 / 4e12)


def exact(case, seed):
    model = MODEL[case["family"]]
    iters = case["iters"] if "count" in case else case["every"] * case["logs"]
    if sum(_seconds(model, a * b * c, iters) for a, b, c in _sizes(case)) > 20:
        return None
    if "count" in case:
        out = {"globals": [], "u": []}
        for spec in _specs(case, seed):
            flags = spec.flags if spec.flags.ndim == 3 else spec.flags[None]
            flow = _FLOWS[model](model, flags, spec.settings, spec.zone_settings.get(0, {}))
            flow.start(None)
            out["globals"].append(flow.iterate(spec.niter, True))
            out["u"].append(flow.velocity().cpu().numpy())
        out["globals"] = np.array(out["globals"])
        return out
    flags, settings, zones, fields = _inputs(case, seed)
    flow = _FLOWS[model](model, flags, settings, zones)
    flow.start(fields)
    out = {"globals": [], "energy": []}
    for _ in range(case["logs"]):
        out["globals"].append(flow.iterate(case["every"], True))
        if fields is not None:
            out["energy"].append(flow.energy())
    out["globals"] = np.array(out["globals"])
    out["energy"] = np.array(out["energy"]) if fields is not None else None
    out["u"] = flow.velocity().cpu().numpy()
    return out
