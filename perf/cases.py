"""Workloads of the Godunov step that are timed and checked on a GPU.

Every case is work a user of the library has it do, through its public Python
entry points: whole coarse steps of a resident uniform or AMR mesh
(``GodunovGPU.coarse_step``, and the reference's leaf calls one by one), a step
of a state kept on the host (``coarse_step_host``), an ensemble of problems
advanced together (``Batch``) and a burst of solve requests (``HydroServer``).

The library holds one mesh and one batch per process.  ``prepare`` therefore
opens the mesh (or the batch) of a case once and makes only the state anew for
each seed; ``run`` puts that state where the step reads it (device to device
through ``rh_state_ptrs`` for resident meshes) and steps it.
"""
import ctypes as C
import math

import numpy as np
import torch

from ramses2_b200 import autotune
from ramses2_b200._abi import HydroParams
from ramses2_b200._lib import check, lib
from ramses2_b200.batch import Batch, ic_blast, ic_split, problem
from ramses2_b200.hydro import GodunovGPU, amr_coarse_step
from ramses2_b200.mesh import sedov_amr_mesh, uniform_mesh
from ramses2_b200.serve import HydroServer, Request

COURANT, SMALLR, SMALLC = 0.8, 1e-10, 1e-10
OUTFLOW = "outflow"
BYTES = {"fp64": 80, "fp32_bulk": 48}  # of one cell's five values, read once and written once
FLOPS = {2: 620, 3: 950}               # of one cell update: conversion, slopes, predictor, Riemann solves, CFL


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _grid(name, prec, level, steps, box="1,1,1", bc=OUTFLOW, ic="sedov", gamma=1.4, slope=2, riemann="hllc",
          gravity=0.0, tuned=False):
    return {"name": name, "kind": "grid", "prec": prec, "level": level, "box": box, "bc": bc, "ic": ic,
            "gamma": gamma, "slope": slope, "riemann": riemann, "gravity": gravity, "tuned": tuned, "steps": steps}


def _amr(name, prec, lmin, lmax, radius, steps, leaf, bc=OUTFLOW, slope=2, riemann="hllc"):
    return {"name": name, "kind": "amr", "prec": prec, "lmin": lmin, "lmax": lmax, "radius": radius, "bc": bc,
            "gamma": 1.4, "slope": slope, "riemann": riemann, "leaf": leaf, "steps": steps}


def _batch(name, prec, count, side_max, mix, steps, slope=2, riemann="hllc"):
    return {"name": name, "kind": "batch", "prec": prec, "count": count, "side_max": side_max, "mix": mix,
            "slope": slope, "riemann": riemann, "steps": steps}


def _serve(name, prec, count, side2d_max, side3d_max, steps_max, mix):
    return {"name": name, "kind": "serve", "prec": prec, "count": count, "side2d_max": side2d_max,
            "side3d_max": side3d_max, "steps_max": steps_max, "mix": mix, "slope": 2, "riemann": "hllc"}


def _host(name, prec, level, bc=OUTFLOW, ic="sedov"):
    return {"name": name, "kind": "host", "prec": prec, "level": level, "box": "1,1,1", "bc": bc, "ic": ic,
            "gamma": 1.4, "slope": 2, "riemann": "hllc", "gravity": 0.0, "tuned": False, "steps": 1}


def listed():
    return [
        # a run of the repository's smallest Sedov configuration, start to end: 64^3, 100 steps
        _grid("sedov64_fp64", "fp64", 6, 100),
        # the headline workload in both precisions, on tiles chosen by the autotuner as the benchmark does
        _grid("sedov256_fp64", "fp64", 8, 6, tuned=True),
        _grid("sedov256_fp32", "fp32_bulk", 8, 12, tuned=True),
        # decaying supersonic turbulence (near-vacuum, high Mach), minmod, as a user who never tunes runs it
        _grid("turb256_fp32", "fp32_bulk", 8, 12, bc="periodic", ic="turb", gamma=1.001, slope=1),
        # a box of unequal sides (160 x 96 x 64) with mixed boundaries and gravity
        _grid("ragged160_fp64", "fp64", 5, 20, box="5,3,2", bc="reflexive,outflow,periodic,periodic,outflow,reflexive",
              ic="waves", slope=1, riemann="hll", gravity=0.05),
        # the smallest mesh: latency of the calls
        _grid("small16_fp32", "fp32_bulk", 4, 20, ic="waves", riemann="llf"),
        # AMR Sedov of 2.7 M leaf cells, whole coarse steps
        _amr("amr9_fp32", "fp32_bulk", 6, 9, 0.16, 10, False),
        # the reference's own call sequence, level by level
        _amr("amr8_leaf_fp64", "fp64", 6, 8, 0.16, 6, True),
        # an ensemble of uneven Riemann and blast problems, 50 steps, states read back
        _batch("ensemble_fp32", "fp32_bulk", 24, 128, 1, 50),
        _batch("ensemble_fp64", "fp64", 12, 64, 2, 50),
        # a burst of mixed 2D and 3D solve requests
        _serve("serve_fp32", "fp32_bulk", 12, 512, 96, 200, 3),
        # a host that keeps its own state and hands it over every step (PCIe both ways)
        _host("host256_fp32", "fp32_bulk", 8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    prec = rng.choice(["fp64", "fp32_bulk"])
    slope, riemann = rng.choice([1, 2, 2]), rng.choice(["llf", "hll", "hllc", "hllc"])
    kind = rng.choice(["grid", "grid", "grid", "amr", "batch", "serve", "host"])
    if kind == "grid":
        # 16^3 to 256^3 cells, sides (1..7) x 2^level
        while True:
            level = rng.randint(3, 7)
            box = [rng.randint(1, 7) for _ in range(3)]
            cells = np.prod([float(b << level) for b in box])
            if 16 ** 3 <= cells <= 256 ** 3 and rng.random() < 0.3:
                break
        steps = max(1, min(100, int(rng.uniform(0.3, 1.0) * 1.0e8 / cells)))
        bc = []
        for _ in range(3):
            bc += ["periodic"] * 2 if rng.random() < 0.3 else [rng.choice([OUTFLOW, "reflexive"]) for _ in range(2)]
        c = _grid("", prec, level, steps, box=",".join(map(str, box)), bc=",".join(bc),
                  ic=rng.choice(["sedov", "waves"]), gamma=round(rng.uniform(1.1, 1.67), 3), slope=slope,
                  riemann=riemann, gravity=rng.choice([0.0, 0.0, 0.05]))
        if c["ic"] == "sedov":  # while the blast stays in its box: reflected on itself it turns chaotic
            c["steps"] = min(c["steps"], min(_cells(c)))
    elif kind == "amr":
        lmin = rng.randint(4, 6)
        c = _amr("", prec, lmin, lmin + rng.randint(1, 9 - lmin if lmin == 6 else 3),
                 round(rng.uniform(0.1, 0.16), 3), rng.randint(2, 8), rng.random() < 0.5,
                 bc=rng.choice([OUTFLOW, "periodic"]), slope=slope, riemann=riemann)
    elif kind == "batch":
        c = _batch("", prec, _log_int(rng, 2, 24), rng.choice([32, 64, 96]), rng.randint(10, 10 ** 6),
                   rng.randint(10, 50), slope, riemann)
    elif kind == "serve":
        c = _serve("", prec, _log_int(rng, 2, 12), rng.choice([128, 256, 512]), rng.choice([32, 64, 96]),
                   rng.randint(50, 200), rng.randint(10, 10 ** 6))
    else:
        c = _host("", prec, rng.randint(5, 7), bc=rng.choice([OUTFLOW, "periodic", "reflexive"]),
                  ic=rng.choice(["sedov", "waves"]))
        c["slope"], c["riemann"] = slope, riemann
    del c["name"]
    return c


def _box(case):
    return [int(b) for b in case["box"].split(",")]


def _bcs(case):
    b = case["bc"].split(",")
    return b * 6 if len(b) == 1 else b


def _cells(case):
    """(nx, ny, nz) of a grid or host case."""
    return [b << case["level"] for b in _box(case)]


def _problems(case):
    """(cells per edge, steps) of each problem of a batch or serve case: the
    same for every seed, so that the work depends on the case alone."""
    r = np.random.default_rng(case["mix"])
    out = []
    for _ in range(case["count"]):
        if case["kind"] == "batch":
            s = int(r.choice([s for s in (16, 32, 48, 64, 96, 128) if s <= case["side_max"]]))
            out.append(((s, s, s), case["steps"]))
        elif r.uniform() < 0.5:
            s = int(round(math.exp(r.uniform(math.log(64), math.log(case["side2d_max"]))) / 16)) * 16
            out.append(((s, s, 2), int(r.integers(20, case["steps_max"] + 1))))
        else:
            s = int(r.integers(2, case["side3d_max"] // 16 + 1)) * 16
            out.append(((s, s, s), int(r.integers(20, case["steps_max"] + 1))))
    return out


def work(case):
    b = BYTES[case["prec"]]
    if case["kind"] in ("grid", "host"):
        n = float(np.prod(_cells(case))) * case["steps"]
        if case["kind"] == "host":
            b = 80  # the host's state is FP64 in either precision
        return {"bytes": n * b, "flops": n * FLOPS[3]}
    if case["kind"] == "amr":
        n = float(_amr_mesh(case).ncells_leaf()) * case["steps"]
        return {"bytes": n * b, "flops": n * FLOPS[3]}
    byts = flops = 0.0
    for n, steps in _problems(case):
        ndim = 2 if n[2] == 2 else 3
        cells = float(n[0]) * n[1] * (n[2] if ndim == 3 else 1) * steps
        byts += cells * b
        flops += cells * FLOPS[ndim]
    return {"bytes": byts, "flops": flops}


def tolerance(case):
    # whole runs amplify a rounding through shocks and limiters; four times the
    # largest distance from exact() seen over the listed and drawn cases
    return {"rel": 2e-14} if case["prec"] == "fp64" else {"rel": 4e-6}


# ---------------------------------------------------------------------------
# meshes and batches: one open at a time
# ---------------------------------------------------------------------------
class _View:
    """A device array at a raw address, for torch.as_tensor."""

    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3}


class _MeshHandle:
    def __init__(self, case):
        self.case = case
        if case["kind"] == "amr":
            self.mesh = _amr_mesh(case)
        else:
            self.mesh = uniform_mesh(case["level"], bc=_bcs(case), box_nx=tuple(_box(case)), boxlen=1.0,
                                     gravity=(0.0, 0.0, -case["gravity"]))
            self.mesh.uold[:] = np.array([1.0, 0.0, 0.0, 0.0, 2.5])[None, :, None]
        self.params = HydroParams.make(gamma=case["gamma"], smallr=SMALLR, smallc=SMALLC, courant_factor=COURANT,
                                       slope_type=case["slope"], riemann=case["riemann"], interpol_type=1)
        self.gpu = GodunovGPU(self.mesh, self.params, precision=case["prec"], deterministic=True)
        m = self.mesh
        if case.get("tuned"):
            autotune.tune(self.gpu, m.levelmin, 0.2 * m.dx(m.levelmin))
        for l in range(m.levelmin, m.levelmax + 1):
            if m.noct[l]:
                self.gpu.courant_fine(l)  # the parameters of the run's time step
        self.order = None
        if case["kind"] != "amr":
            self.order = _oct_order(_cells(case))
        self.host_out = None
        if case["kind"] == "host":
            self.host_out = torch.empty(m.uold.shape, dtype=torch.float64, pin_memory=True)
        self.views = {}

    def state(self):
        """Views of the resident state in the library's device layout."""
        p = [C.c_void_p() for _ in range(4)]
        check(lib().rh_state_ptrs(*[C.byref(x) for x in p]), "rh_state_ptrs")
        n = self.mesh.ngridmax
        key = p[0].value
        if key not in self.views:
            if self.case["prec"] == "fp64":
                self.views[key] = torch.as_tensor(_View(p[0].value, (n, 40), "<f8"), device="cuda")
            else:
                self.views[key] = torch.as_tensor(_View(p[1].value, (n, 48), "<f4"), device="cuda")
        return self.views[key]

    def close(self):
        self.views = {}
        self.gpu.close()


class _BatchHandle:
    def __init__(self, case):
        octs = sum(n[0] * n[1] * n[2] // 8 for n, _ in _problems(case)) + 64
        if case["kind"] == "serve":
            per = 640 if case["prec"] == "fp64" else 384
            self.server = HydroServer(case["prec"], pool_bytes=octs * per, slope_type=case["slope"],
                                      riemann=case["riemann"])
            self.batch = self.server.batch
        else:
            self.batch = Batch(case["prec"], slope_type=case["slope"], riemann=case["riemann"], pool_octs=octs)

    def close(self):
        self.batch.close()


_held = {"key": None, "handle": None}
_meshes = {}


def _amr_mesh(case):
    key = (case["lmin"], case["lmax"], case["radius"], case["bc"])
    if key not in _meshes:
        _meshes.clear()
        _meshes[key] = sedov_amr_mesh(case["lmin"], case["lmax"], radius=case["radius"], bc=case["bc"])[0]
    return _meshes[key]


def _handle(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if _held["key"] != key:
        if _held["handle"] is not None:
            _held["key"] = None
            _held.pop("handle").close()
            _held["handle"] = None
        _held["handle"] = (_BatchHandle if case["kind"] in ("batch", "serve") else _MeshHandle)(case)
        _held["key"] = key
    return _held["handle"]


# ---------------------------------------------------------------------------
# states
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _centres(n, dx):
    """Cell-centre coordinates, each broadcastable to (nz, ny, nx)."""
    dev = _device()
    x, y, z = ((torch.arange(k, device=dev, dtype=torch.float64) + 0.5) * dx for k in n)
    return x[None, None, :], y[None, :, None], z[:, None, None]


def _smooth(n, dx, r, amp):
    """1 + a few waves of random phase, a smooth positive factor."""
    x, y, z = _centres(n, dx)
    box = [k * dx for k in n]
    f = 1.0
    for _ in range(3):
        k = 2 * math.pi * r.integers(1, 4, 3)
        ph = r.uniform(0, 2 * math.pi, 3)
        f = f + amp / 3 * (torch.sin(k[0] * x / box[0] + ph[0]) * torch.sin(k[1] * y / box[1] + ph[1])
                           * torch.sin(k[2] * z / box[2] + ph[2]))
    return f


def _conserved(rho, v, p, gamma):
    ek = 0.5 * rho * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2)
    return torch.stack([rho, rho * v[0], rho * v[1], rho * v[2], p / (gamma - 1.0) + ek])


def _dense(case, seed):
    """Conserved state (5, nz, ny, nx) in FP64 of a grid or host case."""
    n, dx, g = _cells(case), 1.0 / 2 ** case["level"], case["gamma"]
    r = np.random.default_rng(seed)
    shape = (n[2], n[1], n[0])
    if case["ic"] == "sedov":
        # energy E into the cells within two cells of a point near the centre, ambient at rest
        c = [(k / 2 + r.integers(-k // 8, k // 8 + 1)) * dx for k in n]
        x, y, z = _centres(n, dx)
        near = (x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2 <= (2.0 * dx) ** 2 * (1 + 1e-12)
        p_in = (g - 1.0) * r.uniform(0.5, 2.0) / (float(near.sum()) * dx ** 3)
        rho = torch.ones(shape, dtype=torch.float64, device=_device()) * _smooth(n, dx, r, 0.1)
        p = torch.where(near, p_in, 1e-5)
        v = [torch.zeros_like(rho)] * 3
    elif case["ic"] == "turb":
        # solenoidal Gaussian velocities with power k^-2 on 1 <= k <= 4, rms Mach 5; lognormal density
        gen = torch.Generator(device=_device()).manual_seed(seed)
        k = [torch.fft.fftfreq(m, d=1.0 / m, device=_device(), dtype=torch.float64) for m in n]
        kx, ky, kz = k[0][None, None, :], k[1][None, :, None], k[2][:, None, None]
        kk2 = kx ** 2 + ky ** 2 + kz ** 2
        band = (kk2 >= 1) & (kk2 <= 16)
        safe = torch.where(kk2 > 0, kk2, 1.0)

        def noise():
            a = torch.randn(shape, generator=gen, device=_device(), dtype=torch.float64)
            return torch.fft.fftn(a) * band

        w = [noise() / torch.sqrt(safe) for _ in range(3)]
        dot = (kx * w[0] + ky * w[1] + kz * w[2]) / safe
        v = [torch.fft.ifftn(a - b * dot).real for a, b in zip(w, (kx, ky, kz))]
        rms = torch.sqrt((v[0] ** 2 + v[1] ** 2 + v[2] ** 2).mean())
        v = [a * (5.0 / rms) for a in v]
        a = torch.fft.ifftn(noise()).real
        rho = torch.exp(0.1 * a / a.std() - 0.005)
        p = torch.full(shape, 1.0, dtype=torch.float64, device=_device()) * (float(rho.mean()) / g)
    else:
        # two states split along an axis under smooth waves: shocks, contacts and rarefactions everywhere
        axis = int(r.integers(0, 3))
        coord = _centres(n, dx)[axis]
        left = coord < n[axis] * dx / 2
        rho = torch.where(left, r.uniform(0.5, 2.0), r.uniform(0.1, 1.0)) * _smooth(n, dx, r, 0.3)
        p = torch.where(left, r.uniform(0.5, 2.0), r.uniform(0.05, 0.5)) * _smooth(n, dx, r, 0.3)
        v = [(_smooth(n, dx, r, 0.6) - 1.0) * 2.0 for _ in range(3)]
    return _conserved(rho, [a.expand(shape) for a in v], p.expand(shape), g).contiguous()


def _oct_order(n):
    """Rows of (oz, oy, ox) in the Morton order a mesh stores its octs in (x fastest)."""
    o = [k // 2 for k in n]
    dev = _device()
    z, y, x = torch.meshgrid(*(torch.arange(k, device=dev) for k in (o[2], o[1], o[0])), indexing="ij")
    key = torch.zeros_like(x)
    for b in range(12):
        key |= ((x >> b & 1) << (3 * b)) | ((y >> b & 1) << (3 * b + 1)) | ((z >> b & 1) << (3 * b + 2))
    return torch.argsort(key.reshape(-1))


def _octs(dense, order=None):
    """(5, nz, ny, nx) -> (noct, 40) oct records, row-major or in ``order``."""
    v, nz, ny, nx = dense.shape
    a = dense.reshape(v, nz // 2, 2, ny // 2, 2, nx // 2, 2).permute(1, 3, 5, 0, 2, 4, 6).reshape(-1, 40)
    return a[order] if order is not None else a.contiguous()


def _records(u, prec):
    """Oct records in the library's device layout of a precision (FP32-bulk: 32 floats, then 8 doubles)."""
    if prec == "fp64":
        return u
    out = torch.empty(len(u), 48, dtype=torch.float32, device=u.device)
    out[:, :32] = u[:, :32]
    out[:, 32:].view(torch.float64).copy_(u[:, 32:])
    return out


def _split(rec, prec):
    """The values of device records: FP64 (n, 5, 8), or the FP32 and the FP64 parts."""
    if prec == "fp64":
        return {"u": rec.view(-1, 5, 8)}
    return {"u": rec[:, :32], "e": rec[:, 32:].view(torch.float64)}


def _cfl(u, gamma, dx, ndim, grav):
    """courant_fine's time step of conserved values u[5, ...] in FP64 (hydro/godunov_utils.f90:228-333)."""
    r = u[0].clamp(min=SMALLR)
    v = [u[1 + d] / r for d in range(3)]
    e = u[4] - 0.5 * r * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2)
    p = torch.maximum((gamma - 1.0) * e, r * SMALLC ** 2 / gamma)
    c = torch.sqrt(gamma * p / r)
    ctot = sum(v[d].abs() + c for d in range(ndim))
    gr = (grav * dx / ctot ** 2).clamp(min=1e-4)
    dt = 2.0 * COURANT * dx / (ctot * (1.0 + torch.sqrt(1.0 + 2.0 * COURANT * gr)))
    return min(float(dt.min()), COURANT * dx / SMALLC)


def _ics(case, seed):
    """[(problem, initial condition, primitive description)] of a batch or serve case."""
    r = np.random.default_rng(seed)
    out = []
    for n, steps in _problems(case):
        ndim = 2 if n[2] == 2 else 3
        dx, g = 1.0 / n[0], float(r.uniform(1.1, 1.67))
        bc = ["outflow"] * 4 + ["periodic"] * 2 if ndim == 2 else ["outflow"] * 6
        st = []
        for _ in range(2):  # rho, p log-uniform, |v| up to three sound speeds, any direction
            rho, p = 10 ** r.uniform(-3, 3), 10 ** r.uniform(-4, 2)
            d = r.standard_normal(3) * ([1, 1, 0] if ndim == 2 else [1, 1, 1])
            d *= r.uniform(0, 3) * math.sqrt(g * p / rho) / np.linalg.norm(d)
            st.append([rho, *map(float, d), p])
        if r.uniform() < (0.25 if case["kind"] == "batch" else 0.75):
            c = [float(v) for v in r.uniform(0.3, 0.7, 3)]
            if case["kind"] == "serve":
                st[0] = [1.0, 0.0, 0.0, 0.0, 1e-5]
            ic = ("blast", st[0], 100.0 * max(st[0][4], st[1][4]), float(r.uniform(0.05, 0.15)), c)
            ric = ic_blast(*ic[1:])
        else:
            ic = ("split", int(r.integers(0, ndim)), st[0], st[1])
            ric = ic_split(*ic[1:])
        out.append((problem(n, dx=dx, ndim=ndim, bc=bc, gamma=g, courant_factor=COURANT, max_steps=steps), ric, ic))
    return out


def prepare(case, seed):
    h = _handle(case)
    s = {"h": h, "case": case}
    if case["kind"] in ("batch", "serve"):
        s["ics"] = _ics(case, seed)
    elif case["kind"] == "amr":
        # the mesh's blast under a smooth factor that is one function of position on every level
        m = h.mesh
        u = torch.from_numpy(m.uold).reshape(-1, 5, 8)
        r = np.random.default_rng(seed)
        k, ph = 2 * math.pi * r.integers(1, 4, 3), r.uniform(0, 2 * math.pi, 3)
        f = np.empty((m.ngridmax, 1, 8))
        dt = math.inf
        for l in range(m.levelmin, m.levelmax + 1):
            x = m.cell_centres(l)
            f[m.level_slice(l), 0] = 1.0 + 0.2 * np.prod(np.sin(k * x + ph), axis=-1)
        u = (u * torch.from_numpy(f)).to(_device())
        for l in range(m.levelmin, m.levelmax + 1):
            dt = min(dt, _cfl(u[m.level_slice(l)].transpose(0, 1), case["gamma"], m.dx(l), 3, 0.0))
        s["dt"] = dt
        s["u"] = _records(u.reshape(-1, 40), case["prec"])
    else:
        d = _dense(case, seed)
        s["dt"] = _cfl(d, case["gamma"], 1.0 / 2 ** case["level"], 3, case["gravity"])
        u = _octs(d, h.order)
        if case["kind"] == "host":
            s["u"] = torch.empty(h.host_out.shape, dtype=torch.float64, pin_memory=True)
            s["u"].copy_(u.view(-1, 5, 8))
        else:
            s["u"] = _records(u, case["prec"])
    return s


def run(s):
    h, case = s["h"], s["case"]
    if case["kind"] == "batch":
        b = h.batch
        pids = [b.add(p, ic) for p, ic, _ in s["ics"]]
        b.step(case["steps"])
        out = [b.fetch(i) for i in pids]
        for i in pids:
            b.remove(i)
        return out
    if case["kind"] == "serve":
        req = [Request(i, 0.0, p, ic) for i, (p, ic, _) in enumerate(s["ics"])]
        h.server.run(req, realtime=False)
        return [r.result for r in req]
    gpu = h.gpu
    if case["kind"] == "host":
        out = h.host_out.numpy()
        _, nxt = gpu.coarse_step_host(s["u"].numpy(), out, s["dt"])
        return {"u": out, "dt_next": nxt}
    h.state().copy_(s["u"])
    torch.cuda.current_stream().synchronize()  # the library works on its own stream
    t = 0.0
    for k in range(case["steps"]):
        dt = s["dt"] if k == 0 else None
        t += amr_coarse_step(gpu, h.mesh, dt) if case.get("leaf") else gpu.coarse_step(dt)
    gpu.sync()
    return dict(_split(h.state(), case["prec"]), t=t)


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits (hydro/umuscl.f90, hydro/godunov_utils.f90)
# ---------------------------------------------------------------------------
def _pad(u, bcs, ndim):
    """Two ghost cells on each side of every direction; u[5, z, y, x]."""
    for d in range(ndim):
        ax = 3 - d
        n = u.shape[ax]
        lo, hi = bcs[2 * d], bcs[2 * d + 1]

        def side(bc, edge, mirror, wrap):
            if bc == "periodic":
                return u.narrow(ax, wrap, 2)
            if bc == "reflexive":
                g = u.narrow(ax, mirror, 2).flip(ax).clone()
                g[1 + d] = -g[1 + d]
                return g
            return u.narrow(ax, edge, 1).repeat([2 if a == ax else 1 for a in range(4)])

        u = torch.cat([side(lo, 0, 0, n - 2), u, side(hi, n - 1, n - 2, 0)], dim=ax)
    return u


def _at(q, off, ndim):
    """q without its outermost layer, shifted by off (x, y, z)."""
    for d in range(ndim):
        ax = q.dim() - 1 - d
        q = q.narrow(ax, 1 + off[d], q.shape[ax] - 2)
    return q


def _slopes(q, slope, ndim):
    """q[5] on the padded box -> half slopes d[dir][var] without the outermost layer."""
    out = []
    for d in range(ndim):
        e = [1 if k == d else 0 for k in range(3)]
        lo, mid, hi = ([_at(v, [s * k for k in e], ndim) for v in q] for s in (-1, 0, 1))
        ds = []
        for n in range(5):
            a, b = mid[n] - lo[n], hi[n] - mid[n]
            same = a * b > 0
            if slope == 1:
                s = torch.where(a > 0, torch.minimum(a, b), torch.maximum(a, b))
                s = torch.where(same, s, 0.0)
            else:
                cen = 0.5 * (a + b)
                lim = torch.where(same, 2.0 * torch.minimum(a.abs(), b.abs()), 0.0)
                s = torch.copysign(torch.minimum(lim, cen.abs()), cen)
            if n == 1 + d:  # rho |dq| / 2 of the normal velocity bounded by the neighbours' jumps
                lim = 2.0 * torch.minimum(lo[0] * a.abs(), hi[0] * b.abs()) / mid[0]
                s = torch.copysign(torch.minimum(s.abs(), lim), s)
            ds.append(0.5 * s)
        out.append(ds)
    return out


def _flux(ql, qr, g, riemann, cap):
    """Godunov flux of states (rho, un, ut1, ut2, p)."""
    rl, rr = ql[0].clamp(min=SMALLR), qr[0].clamp(min=SMALLR)
    pl, pr = torch.maximum(ql[4], rl * SMALLC ** 2 / g), torch.maximum(qr[4], rr * SMALLC ** 2 / g)
    cl, cr = torch.sqrt(g * pl / rl), torch.sqrt(g * pr / rr)
    if riemann == "hllc":
        el = pl / (g - 1) + 0.5 * rl * (ql[1] ** 2 + ql[2] ** 2 + ql[3] ** 2)
        er = pr / (g - 1) + 0.5 * rr * (qr[1] ** 2 + qr[2] ** 2 + qr[3] ** 2)
        c = torch.maximum(cl.clamp(min=SMALLC), cr.clamp(min=SMALLC))
        sl, sr = torch.minimum(ql[1], qr[1]) - c, torch.maximum(ql[1], qr[1]) + c
        al, ar = rl * (ql[1] - sl), rr * (sr - qr[1])
        us = (ar * qr[1] + al * ql[1] + pl - pr) / (ar + al)
        ps = (ar * pl + al * pr + al * ar * (ql[1] - qr[1])) / (ar + al)
        left = (sl > 0) | (us > 0)
        star = torch.where(left, sl <= 0, sr > 0)

        def pick(a, b):
            return torch.where(left, a, b)

        r, u, p, e, s = pick(rl, rr), pick(ql[1], qr[1]), pick(pl, pr), pick(el, er), pick(sl, sr)
        ro = torch.where(star, r * (s - u) / (s - us), r)
        eo = torch.where(star, ((s - u) * e - p * u + ps * us) / (s - us), e)
        uo, po = torch.where(star, us, u), torch.where(star, ps, p)
        m = ro * uo
        return [m, m * uo + po, m * pick(ql[2], qr[2]), m * pick(ql[3], qr[3]), (eo + po) * uo]

    def cons(q):
        u = [q[0], q[0] * q[1], q[0] * q[2], q[0] * q[3],
             q[4] / (g - 1) + 0.5 * q[0] * (q[1] ** 2 + q[2] ** 2 + q[3] ** 2)]
        return u, [u[1], q[1] * u[1] + q[4], q[1] * u[2], q[1] * u[3], q[1] * (u[4] + q[4])]

    (ul, fl), (ur, fr) = cons(ql), cons(qr)
    if riemann == "llf":
        c = torch.maximum(ql[1].abs() + cl, qr[1].abs() + cr).clamp(max=cap)
        return [0.5 * (fl[n] + fr[n] - c * (ur[n] - ul[n])) for n in range(5)]
    c = torch.maximum(cl, cr)
    sl = (torch.minimum(ql[1], qr[1]) - c).clamp(min=-cap, max=0.0)
    sr = (torch.maximum(ql[1], qr[1]) + c).clamp(min=0.0, max=cap)
    return [(sr * fl[n] - sl * fr[n] + sr * sl * (ur[n] - ul[n])) / (sr - sl) for n in range(5)]


def _step64(u, dt, dx, g, slope, riemann, bcs, ndim, grav):
    """One MUSCL-Hancock step of a dense box u[5, z, y, x] in FP64."""
    U = _pad(u, bcs, ndim)
    r = U[0].clamp(min=SMALLR)
    v = [U[1 + d] / r for d in range(3)]
    e = U[4] - 0.5 * r * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2)
    p = (g - 1.0) * torch.maximum(e, r * (SMALLC ** 2 / g / (g - 1.0)))
    del e, U
    q = [r, v[0] + 0.5 * dt * grav[0], v[1] + 0.5 * dt * grav[1], v[2] + 0.5 * dt * grav[2], p]
    d = _slopes(q, slope, ndim)
    r, u1, v1, w1, p = (_at(a, (0, 0, 0), ndim) for a in q)
    vel, c = (u1, v1, w1), dt / dx
    div = sum(d[a][1 + a] for a in range(ndim))

    def adv(n):
        return sum(vel[a] * d[a][n] for a in range(ndim))

    pred = [r - c * (adv(0) + div * r)]
    for a in range(3):
        pred.append(vel[a] - c * (adv(1 + a) + (d[a][4] / r if a < ndim else 0.0)))
    pred.append(p - c * (adv(4) + div * g * p))
    del q, vel
    new = list(u.clone())
    for a in range(ndim):
        states = []
        for sgn in (1.0, -1.0):
            s = [pred[n] + sgn * d[a][n] for n in range(5)]
            s[0] = torch.where(s[0] < SMALLR, r, s[0])
            s[4] = torch.where(s[4] < SMALLR * SMALLC ** 2, p, s[4])
            rot = [0] + [1 + (a + k) % 3 for k in range(3)] + [4]
            states.append([s[n] for n in rot])
        ax = 2 - a

        def inner(t, k):  # every other direction without its ring layer; face range along ax
            for b in range(ndim):
                if b != a:
                    t = t.narrow(2 - b, 1, t.shape[2 - b] - 2)
            return t.narrow(ax, k, t.shape[ax] - 1)

        ql, qr = [inner(t, 0) for t in states[0]], [inner(t, 1) for t in states[1]]
        f = _flux(ql, qr, g, riemann, COURANT * dx / dt)
        var = [0] + [1 + (a + k) % 3 for k in range(3)] + [4]
        for k, n in enumerate(var):
            m = f[k].shape[ax] - 1
            new[n] = new[n] + c * (f[k].narrow(ax, 0, m) - f[k].narrow(ax, 1, m))
    return torch.stack(new)


def _initial(n, dx, g, ic, ndim):
    """Dense state of a batch problem's initial condition."""
    n = (n[0], n[1], 1) if ndim == 2 else n
    shape = (n[2], n[1], n[0])
    x, y, z = _centres(n, dx)
    one = torch.ones(shape, dtype=torch.float64, device=_device())
    if ic[0] == "split":
        left = ((x, y, z)[ic[1]] < n[ic[1]] * dx / 2).expand(shape)
        q = [torch.where(left, a * one, b * one) for a, b in zip(ic[2], ic[3])]
    else:
        c = ic[4]
        r2 = (x - c[0]) ** 2 + (y - c[1]) ** 2 + ((z - c[2]) ** 2 if ndim == 3 else 0.0 * z)
        q = [a * one for a in ic[1]]
        q[4] = torch.where(r2 <= ic[3] ** 2 * (1 + 1e-12), ic[2] * one, q[4])
    return _conserved(q[0], q[1:4], q[4], g)


def exact(case, seed):
    if case["kind"] == "amr":
        return None  # coarse-fine levels: no plain statement short enough to be one
    if case["kind"] in ("grid", "host"):
        if float(np.prod(_cells(case))) * case["steps"] > 3e8:
            return None
        dx, g, grav = 1.0 / 2 ** case["level"], case["gamma"], (0.0, 0.0, -case["gravity"])
        u = _dense(case, seed)
        dt = _cfl(u, g, dx, 3, case["gravity"])
        if case["prec"] != "fp64":
            u[:4] = u[:4].float().double()
        t = 0.0
        for k in range(case["steps"]):
            if k:
                dt = _cfl(u, g, dx, 3, case["gravity"])
            u = _step64(u, dt, dx, g, case["slope"], case["riemann"], _bcs(case), 3, grav)
            t += dt
        rec = _octs(u, _oct_order(_cells(case)))
        if case["kind"] == "host":
            return {"u": rec.view(-1, 5, 8), "dt_next": _cfl(u, g, dx, 3, 0.0)}
        out = {"u": rec.view(-1, 5, 8)} if case["prec"] == "fp64" else {"u": rec[:, :32], "e": rec[:, 32:]}
        return dict(out, t=t)
    out = []
    for (n, steps), (p, _, ic) in zip(_problems(case), _ics(case, seed)):
        ndim = 2 if n[2] == 2 else 3
        if float(n[0]) * n[1] * n[2] * steps > 1.5e8:
            out.append(None)
            continue
        u = _initial(n, p.dx, p.gamma, ic, ndim)
        if case["prec"] != "fp64":
            u[:4] = u[:4].float().double()
        for _ in range(steps):
            dt = _cfl(u, p.gamma, p.dx, ndim, 0.0)
            u = _step64(u, dt, p.dx, p.gamma, case["slope"], case["riemann"], list(_case_bc(ndim)), ndim, (0, 0, 0))
        if ndim == 2:
            u = u.repeat(1, 2, 1, 1)
        out.append(_octs(u).view(-1, 5, 8))
    return out


def _case_bc(ndim):
    return ("outflow",) * (4 if ndim == 2 else 6)
