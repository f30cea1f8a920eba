"""The rules that cut levels and batches into pencils: whatever tile and depth
they take, the states equal those of an explicitly chosen tile bit for bit (a
cell's update does not depend on where pencils end), dt too, and the
conserved totals to the rounding of another summation order."""
import ctypes as C

import numpy as np
import pytest

from ramses2_b200._abi import HydroParams
from ramses2_b200.batch import Batch, ic_blast, problem
from ramses2_b200.hydro import GodunovGPU
from ramses2_b200.mesh import amr_mesh, fill_amr_prim, prim_to_cons, sedov_amr_mesh, uniform_mesh

pytestmark = pytest.mark.gpu


def waves(m, seed):
    lev = m.levelmin
    n = [b << lev for b in m.box_nx]
    r = np.random.default_rng(seed)
    shape = (n[2], n[1], n[0])
    rho, p = r.uniform(0.5, 1.5, shape), r.uniform(0.5, 1.5, shape)
    m.from_dense(prim_to_cons(rho, *r.uniform(-0.5, 0.5, (3,) + shape), p, 1.4), lev)


def tile_of(gpu):
    v = [C.c_int() for _ in range(4)]
    assert gpu.L.rh_get_tile(*[C.byref(x) for x in v]) == 0
    return [x.value for x in v]


# one CTA, a few, thin and flat boxes, a last pencil shorter than the others, several waves of CTAs
BOXES = [(1, (1, 1, 1)), (2, (1, 1, 1)), (4, (1, 1, 1)), (3, (5, 1, 3)), (2, (1, 1, 17)), (2, (31, 2, 1)), (6, (1, 1, 1)),
         (5, (3, 2, 5))]


@pytest.mark.parametrize("level,box", BOXES)
@pytest.mark.parametrize("prec", ["fp64", "fp32_bulk"])
def test_default_tile_steps_like_an_explicit_one(prec, level, box):
    m = uniform_mesh(level, bc="periodic", box_nx=box)
    waves(m, 7)
    P = HydroParams.make(gamma=1.4)
    got = []
    for tile in (None, (8, 4, 3, 2)):
        g = GodunovGPU(m, P, precision=prec, tile=tile)
        try:
            if tile is None:
                auto = tile_of(g)
                assert (auto[0], auto[1], auto[2]) in g.tiles() and 1 <= auto[3] <= max(1, (box[2] << level) // 2)
            first = g.courant_fine(level)
            dts = [g.coarse_step() for _ in range(3)]
            fused, u = g.courant_fine(level), g.fetch_uold()
            g.push_uold(u)
            alone = g.courant_fine(level)
        finally:
            g.close()
        assert fused[4] == alone[4]
        assert fused[:3] == pytest.approx(alone[:3], rel=1e-12)
        got.append((first[4], dts, u))
    assert got[0][0] == got[1][0] and got[0][1] == got[1][1]
    assert np.array_equal(got[0][2], got[1][2])


@pytest.mark.parametrize("prec", ["fp64", "fp32_bulk"])
def test_a_chosen_tile_is_kept(prec):
    m = uniform_mesh(4, bc="outflow")
    waves(m, 1)
    g = GodunovGPU(m, HydroParams.make(), precision=prec, tile=(8, 4, 5, 2))
    try:
        assert tile_of(g) == [8, 4, 2, 5]
    finally:
        g.close()


@pytest.mark.parametrize("lmin,lmax", [(3, 5), (5, 6)])
@pytest.mark.parametrize("prec,tile", [("fp64", (7, 11, 1, 32)), ("fp64", (8, 4, 2, 3)), ("fp32_bulk", (7, 7, 2, 32))])
def test_default_coarse_fine_tile_steps_like_an_explicit_one(prec, tile, lmin, lmax):
    m, gamma = sedov_amr_mesh(lmin, lmax, radius=0.2)
    P = HydroParams.make(gamma=gamma, interpol_type=1)
    got = []
    for t in (None, tile):
        g = GodunovGPU(m, P, precision=prec, amr_tile=t)
        try:
            got.append(([g.coarse_step() for _ in range(3)], g.fetch_uold()))
        finally:
            g.close()
    assert got[0][0] == got[1][0]
    assert np.array_equal(got[0][1], got[1][1])


@pytest.mark.parametrize("prec,tile", [("fp64", (8, 4, 2, 32)), ("fp32_bulk", (7, 7, 2, 32))])
def test_default_batch_depth_steps_like_an_explicit_one(prec, tile):
    sizes = [(16, 16, 16), (64, 32, 96), (8, 8, 128), (2, 2, 2), (64, 64, 2)]
    got = []
    for t in (None, tile):
        b = Batch(prec, pool_octs=1 << 17, tile=t)
        try:
            ids = []
            for k, n in enumerate(sizes):
                ndim = 2 if n == (64, 64, 2) else 3
                bc = ["outflow"] * 4 + ["periodic"] * 2 if ndim == 2 else "outflow"
                ids.append(b.add(problem(n, dx=1 / 64, ndim=ndim, bc=bc, max_steps=4 + k),
                                 ic_blast([1.0, 0.1, 0.2, 0.0, 0.1], 5.0, 0.06, [0.06, 0.06, 0.06])))
            b.step(10)
            got.append([(b.status(i), b.fetch(i)) for i in ids])
        finally:
            b.close()
    for (sa, ua), (sb, ub) in zip(*got):
        assert (sa["t"], sa["dt"], sa["nstep"]) == (sb["t"], sb["dt"], sb["nstep"])
        assert sa["totals"] == pytest.approx(sb["totals"], rel=1e-12)
        assert np.array_equal(ua, ub)


@pytest.mark.parametrize("tile", [(8, 4, 2, 32), None])
@pytest.mark.parametrize("prec", ["fp64", "fp32_bulk"])
def test_totals_and_the_neighbours(prec, tile):
    """A problem alone and among others that change the default depth and (in
    FP32-bulk, as 2D ones) tile, arriving in mid-run: its sums are the same with a
    chosen tile and equal to rounding without."""
    p = problem((48, 32, 64), dx=1 / 64, bc="outflow", max_steps=6)
    ic = ic_blast([1.0, 0.1, 0.2, 0.0, 0.1], 5.0, 0.1, [0.3, 0.2, 0.5])
    plane = problem((512, 512, 2), dx=1 / 512, ndim=2, bc=["outflow"] * 4 + ["periodic"] * 2, max_steps=20)
    cube = problem((64, 64, 64), dx=1 / 64, bc="periodic", max_steps=20)
    got = []
    for others in ([], [plane, cube, cube]):
        b = Batch(prec, pool_octs=1 << 19, tile=tile)
        try:
            pid = b.add(p, ic)
            b.step(3)
            for o in others:
                b.add(o, ic)
            b.step(3)
            got.append((b.status(pid), b.fetch(pid)))
        finally:
            b.close()
    (sa, ua), (sb, ub) = got
    assert sa["nstep"] == sb["nstep"] == 6
    assert (sa["t"], sa["dt"]) == (sb["t"], sb["dt"]) and np.array_equal(ua, ub)
    if tile:
        assert list(sa["totals"]) == list(sb["totals"])
    else:  # another order of 98,304 positive terms
        assert sa["totals"] == pytest.approx(sb["totals"], rel=1e-13)


def scattered(lmin, lmax, every, nexpand):
    """Clusters of (2 nexpand + 1)^3 octs around every so many-th cell."""
    def refine(x, l):
        k = (x * 2 ** l).astype(np.int64)
        return ((k[:, 0] * 73856093) ^ (k[:, 1] * 19349663) ^ (k[:, 2] * 83492791)) % every == 0

    m = amr_mesh(lmin, lmax, refine, nexpand=nexpand)
    r = np.random.default_rng(2)
    fill_amr_prim(m, lambda x, l: (r.uniform(0.5, 1.5, x.shape[:-1]), *r.uniform(-0.3, 0.3, (3,) + x.shape[:-1]),
                                   r.uniform(0.5, 1.5, x.shape[:-1])), 1.4)
    return m


@pytest.mark.parametrize("which,tile", [("scattered", (8, 4, 2, 32)), ("a few clusters", (7, 11, 1, 32)),
                                        ("blast", (7, 11, 1, 32))])
def test_fp64_coarse_fine_tile_by_how_full_its_columns_are(which, tile):
    """The chosen tile shows in the partial levels' pencils and ghost octs; the
    states equal those of either tile bit for bit.  (The few clusters in a large
    box are counted in a hashed bitmap, the others in a dense one.)"""
    m = {"scattered": lambda: scattered(6, 8, 4001, 2), "a few clusters": lambda: scattered(7, 8, 400001, 2),
         "blast": lambda: sedov_amr_mesh(6, 8, radius=0.16)[0]}[which]()
    P = HydroParams.make(gamma=1.4, interpol_type=1)
    dt = 0.1 * m.dx(m.levelmax)
    partial = [l for l in range(m.levelmin + 1, m.levelmax + 1) if m.noct[l]]
    got = []
    for t in (None, tile, (7, 11, 1, 32) if tile[0] == 8 else (8, 4, 2, 32)):
        g = GodunovGPU(m, P, precision="fp64", amr_tile=t)
        try:
            n = C.c_int()
            cut = []
            for l in partial:
                assert g.L.rh_level_info(l, C.byref(n), None) == 0
                cut.append((n.value, g.L.rh_level_ghosts(l, None, None, None, 0)))
            got.append((cut, [g.coarse_step(dt), g.coarse_step()], g.fetch_uold()))
        finally:
            g.close()
    assert got[0][0] == got[1][0] != got[2][0]
    for other in got[1:]:
        assert got[0][1] == other[1] and np.array_equal(got[0][2], other[2])


# fewer items than SMs, than slots, a few more than slots, several a slot; 3D and with a 2D problem
BATCHES = [[(32, 32, 32)] * 3, [(96, 96, 96)], [(16, 16, 16)] * 100, [(32, 32, 32)] * 40,
           [(128, 32, 64)] * 6 + [(256, 256, 2)], [(48, 80, 72), (16, 16, 128), (96, 64, 32)]]


@pytest.mark.parametrize("sizes", BATCHES)
@pytest.mark.parametrize("prec", ["fp64", "fp32_bulk"])
def test_default_depth_of_few_and_of_many_work_items(prec, sizes):
    got = []
    for tile in (None, (8, 4, 2, 32)):
        b = Batch(prec, pool_octs=sum(n[0] * n[1] * n[2] // 8 for n in sizes) + 8, tile=tile)
        try:
            ids = []
            for k, n in enumerate(sizes):
                plane = n[2] == 2
                ids.append(b.add(problem(n, dx=1 / 32, ndim=2 if plane else 3, max_steps=3 + k % 2,
                                         bc=["outflow"] * 4 + ["periodic"] * 2 if plane else "reflexive"),
                                 ic_blast([1.0, 0.1, 0.05 * (k % 5), 0.0, 0.1], 5.0, 0.1, [0.3, 0.2, 0.03])))
            b.step(4)
            got.append([(b.status(i), b.fetch(i)) for i in (ids[0], ids[len(ids) // 2], ids[-1])])
        finally:
            b.close()
    for (sa, ua), (sb, ub) in zip(*got):
        assert (sa["t"], sa["dt"], sa["nstep"]) == (sb["t"], sb["dt"], sb["nstep"])
        assert sa["totals"] == pytest.approx(sb["totals"], rel=1e-12)
        assert np.array_equal(ua, ub)
