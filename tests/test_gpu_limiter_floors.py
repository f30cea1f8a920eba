"""The predictor's floors and the limiters at the values where their short
forms branch, against the FP64 oracle.

The floors (smallr on the density, smallr*smallc**2 on the pressure of an
interface state) sit behind one test per cell in the kernels; here they act in
part of the cells (a floor inside the range of the states), in none, and next
to zero.  The limiters see equal neighbours, differences of opposite sign and
differences whose product underflows FP32."""
import os

import numpy as np
import pytest

import oracle
from ramses2_b200._abi import HydroParams
from ramses2_b200.hydro import GodunovGPU
from ramses2_b200.mesh import prim_to_cons, uniform_mesh

pytestmark = pytest.mark.gpu

NTHREADS = os.cpu_count() or 1


def steep_state(m, seed, amp):
    """Densities and pressures over decades with plateaus, on a 16^3 level."""
    r = np.random.default_rng(seed)
    n = 16
    rho = 10.0 ** np.round(r.uniform(-2, 0, (n, n, n)), 1)
    p = 10.0 ** np.round(r.uniform(-2, 0, (n, n, n)), 1)
    rho[4:8], p[4:8] = 0.5, 0.25
    v = amp * r.choice([-1.0, 0.0, 0.0, 1.0], (3, n, n, n))
    m.from_dense(prim_to_cons(rho, *v, p, 1.4), m.levelmin)


def one_step(m, P, prec, tile, dt):
    u0 = m.uold.copy()
    o = oracle.OracleHydro(m, P, nthreads=NTHREADS)
    o.step_uniform(dt)
    ref = m.uold.copy()
    m.uold[:] = u0
    g = GodunovGPU(m, P, precision=prec, tile=tile)
    try:
        g.step_uniform(dt)
        return ref, g.fetch_uold()
    finally:
        g.close()


@pytest.mark.parametrize("slope", [1, 2])
@pytest.mark.parametrize("smallr,smallc", [(1e-10, 1e-10), (0.03, 0.3), (0.9, 0.9)])
@pytest.mark.parametrize("prec,tile", [("fp64", (8, 8, 2)), ("fp64", (6, 4, 8)), ("fp32_bulk", (7, 7, 4)),
                                       ("fp32_bulk", (8, 4, 8))])
def test_floors_act_where_the_reference_applies_them(prec, tile, smallr, smallc, slope):
    m = uniform_mesh(4, bc="periodic")
    steep_state(m, 3, 0.3)
    P = HydroParams.make(gamma=1.4, smallr=smallr, smallc=smallc, slope_type=slope, riemann="hllc")
    dt = 0.2 * m.dx(4) / 12.0
    ref, out = one_step(m, P, prec, tile, dt)
    num = np.abs(out - ref).sum(axis=(0, 2))
    den = np.abs(ref).sum(axis=(0, 2))
    # FP64: the parity bar; FP32: a handful of roundings of 6e-8 per update term
    assert np.all(num <= (1e-12 if prec == "fp64" else 2e-6) * den), num / den


@pytest.mark.parametrize("amp", [1e-20, 1e-3])
@pytest.mark.parametrize("prec", ["fp64", "fp32_bulk"])
def test_plateaus_and_tiny_differences(prec, amp):
    m = uniform_mesh(4, bc="outflow")
    r = np.random.default_rng(5)
    one = np.ones((16, 16, 16))
    v = amp * r.choice([-1.0, 0.0, 1.0], (3, 16, 16, 16))
    m.from_dense(prim_to_cons(one, *v, one, 1.4), 4)
    P = HydroParams.make(gamma=1.4, slope_type=2, riemann="hllc")
    ref, out = one_step(m, P, prec, (8, 4, 4), 0.1 * m.dx(4))
    # the momenta are sums of pressure differences of O(1) terms rounded at eps
    eps = 2.3e-16 if prec == "fp64" else 1.2e-7
    assert np.abs(out - ref).max() <= 8 * eps
    assert np.all(np.isfinite(out))
