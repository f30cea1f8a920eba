"""The predictor's floors and the limiters at the values where their short
forms branch, against the FP64 oracle.

The floors (smallr on the density, smallr*smallc**2 on the pressure of an
interface state) sit behind one test per cell in the kernels; here they act in
part of the cells (a floor inside the range of the states), in none, and next
to zero.  The limiters see equal neighbours, differences of opposite sign and
(on a state whose momenta are compared on their own scale) differences whose
product underflows FP32."""
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


@pytest.mark.parametrize("slope", [1, 2])
@pytest.mark.parametrize("prec", ["fp64", "fp32_bulk"])
def test_differences_whose_product_underflows(prec, slope):
    """Velocities of some 1e-20 in a gas whose sound speed is 1e-18: every term
    of the step is a normal FP32 number, but the product of two velocity
    differences (1e-40) is not, so a limiter that tests its sign takes no slope.
    The momenta change by 2 %, and by a third of that less without slopes."""
    m = uniform_mesh(4, bc="periodic")
    r = np.random.default_rng(8)
    n, rho, p = 16, 1e15, 1e-21
    x = 2 * np.pi * (np.arange(n) + 0.5) / n
    wave = np.sin(x)[None, None, :] + np.sin(x)[None, :, None] + np.sin(x)[:, None, None]
    v = 1e-20 * (wave + 0.3 * r.uniform(-1, 1, (3, n, n, n)))
    one = np.ones((n, n, n))
    u = prim_to_cons(rho * one, *v, p * one, 1.4)
    m.from_dense(u, 4)
    P = HydroParams.make(gamma=1.4, smallr=1e-10, smallc=1e-30, slope_type=slope, riemann="hllc")
    dt = 0.1 * m.dx(4) / np.sqrt(1.4 * p / rho)
    u0 = m.uold.copy()
    ref, out = one_step(m, P, prec, (8, 4, 4), dt)
    change = np.abs(ref - u0)[:, 1:4].max()
    eps = 2.3e-16 if prec == "fp64" else 1.2e-7
    # the momentum update is dt/dx times differences of fluxes p + rho u du of
    # which p is the largest term: a few roundings of it, and of the momenta
    bound = 8 * eps * (p * dt / m.dx(4) + np.abs(ref[:, 1:4]).max())
    assert change > 1e3 * bound
    assert np.abs(out - ref)[:, 1:4].max() <= bound
