"""Every compiled tile of the uniform kernels, at depths of one, two and an odd
number of layers, on a box no side of which the tiles divide and whose x extent
is wider than the widest tile: the states of two steps and the next dt equal
those of the 8x4 tile bit for bit, for every slope type and Riemann solver and
mixed boundaries, and those of the 8x4 tile the FP64 oracle's."""
import os

import numpy as np
import pytest

import oracle
from ramses2_b200._abi import HydroParams
from ramses2_b200.hydro import GodunovGPU
from ramses2_b200.mesh import prim_to_cons, uniform_mesh

pytestmark = pytest.mark.gpu

BOX, LEVEL = (17, 13, 5), 2  # 34 x 26 x 10 octs
BCS = [["outflow"] * 4 + ["periodic"] * 2, ["periodic"] * 2 + ["reflexive", "outflow"] + ["reflexive"] * 2,
       ["reflexive", "outflow"] + ["periodic"] * 2 + ["outflow", "reflexive"]]


def waves(m):
    n = [b << m.levelmin for b in m.box_nx]
    r = np.random.default_rng(12)
    shape = (n[2], n[1], n[0])
    rho, p = r.uniform(0.5, 1.5, shape), r.uniform(0.5, 1.5, shape)
    m.from_dense(prim_to_cons(rho, *r.uniform(-0.5, 0.5, (3,) + shape), p, 1.4), m.levelmin)


@pytest.mark.parametrize("riemann", ["llf", "hll", "hllc"])
@pytest.mark.parametrize("slope", [0, 1, 2, 3])
@pytest.mark.parametrize("prec", ["fp64", "fp32_bulk"])
def test_tiles_agree_bit_for_bit(prec, slope, riemann):
    bc = BCS[(slope + ["llf", "hll", "hllc"].index(riemann)) % 3]
    m = uniform_mesh(LEVEL, bc=bc, box_nx=BOX, gravity=(0.0, 0.05, -0.1))
    waves(m)
    P = HydroParams.make(gamma=1.4, slope_type=slope, riemann=riemann)
    u0 = m.uold.copy()
    dt = 0.1 * m.dx(LEVEL)
    o = oracle.OracleHydro(m, P, nthreads=os.cpu_count() or 1)
    o.step_uniform(dt)
    one = m.uold.copy()
    m.uold[:] = u0
    g = GodunovGPU(m, P, precision=prec)
    try:
        def steps():
            g.push_uold(u0)
            g.courant_fine(LEVEL)
            g.coarse_step(dt)
            first = g.fetch_uold()
            return first, g.coarse_step(), g.fetch_uold(), g.courant_fine(LEVEL)

        g.set_tile(8, 4, 32, 2)
        ref = steps()
        num, den = np.abs(ref[0] - one).sum(axis=(0, 2)), np.abs(one).sum(axis=(0, 2))
        # FP64: the parity bar; FP32: a handful of roundings of 6e-8 per update term
        assert np.all(num <= (1e-12 if prec == "fp64" else 2e-6) * den), num / den
        seen = 0
        for tx, ty, mb in g.tiles():
            for lz in (1, 2, 7):
                g.set_tile(tx, ty, lz, mb)
                got = steps()
                key = (tx, ty, mb, lz)
                assert np.array_equal(got[0], ref[0]) and np.array_equal(got[2], ref[2]), key
                assert got[1] == ref[1] and got[3][4] == ref[3][4], key
                assert got[3][:3] == pytest.approx(ref[3][:3], rel=1e-12), key
                seen += 1
        assert seen >= 3 * 6
    finally:
        g.close()
