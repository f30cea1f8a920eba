"""courant_fine of states whose sound-speed argument or density is no normal
number: zero or subnormal pressures (smallc**2 below the smallest normal), a
density as small, an energy that overflowed; against cmpdt
(godunov_utils.f90:228-333) in numpy, whose square roots and divisions are
IEEE's.  (The oracle squares the sound speed's square as the reference does, and
the square of such a number underflows.)"""
import numpy as np
import pytest

from ramses2_b200._abi import HydroParams
from ramses2_b200.hydro import GodunovGPU
from ramses2_b200.mesh import uniform_mesh

pytestmark = pytest.mark.gpu

GAMMA, COURANT = 1.4, 0.8


def smallest_dt(u, dx, smallr, smallc, gravity):
    """min over the cells of u (octs, 5, 8) of cmpdt; a cell without a number
    for its step takes the longest one."""
    r = np.maximum(u[:, 0], smallr)
    with np.errstate(all="ignore"):
        e = u[:, 4] - 0.5 * (u[:, 1] ** 2 + u[:, 2] ** 2 + u[:, 3] ** 2) / r
        p = np.maximum((GAMMA - 1.0) * e, r * (smallc * smallc / GAMMA))
        c = np.sqrt(GAMMA * p / r)
        ctot = sum(np.abs(u[:, d]) / r + c for d in (1, 2, 3))
        grav = np.maximum(gravity * dx / ctot ** 2, 1e-4)
        dt = dx / ctot * (np.sqrt(1.0 + 2.0 * COURANT * grav) - 1.0) / grav
    longest = COURANT * dx / smallc
    return float(np.where(dt < longest, dt, longest).min())


def compare(m, prec, smallr=1e-10, smallc=1e-10, gravity=0.0, rel=1e-13):
    # the closed form of the step cancels in (sqrt(1 + 2 courant g) - 1) / g
    want = smallest_dt(m.uold, m.dx(m.levelmin), smallr, smallc, gravity)
    gpu = GodunovGPU(m, HydroParams.make(gamma=GAMMA, courant_factor=COURANT, smallr=smallr, smallc=smallc),
                     precision=prec)
    try:
        got = gpu.courant_fine(m.levelmin)[4]
    finally:
        gpu.close()
    assert got == pytest.approx(want, rel=max(rel, 1e-11))


# (rho, velocity, E - kinetic energy) of one cell among cells of half its speed
CELLS = [(1.0, 0.0, 0.0), (1.0, 0.5, -1.0), (1.0, 0.0, 1e-312), (1.0, 0.25, 0.0), (1.0, 0.5, 2.0)]


# (with gravity the step divides by the square of the speed, which underflows at
# the two small values in any form)
@pytest.mark.parametrize("smallc,gravity", [(1e-170, 0.0), (1e-160, 0.0), (1e-10, 0.0), (1e-10, 0.3)])
@pytest.mark.parametrize("prec", ["fp64", "fp32_bulk"])
def test_zero_and_subnormal_pressure(prec, smallc, gravity):
    for rho, v, eint in CELLS:
        m = uniform_mesh(2, bc="periodic", gravity=(0.0, 0.0, -gravity))
        m.uold[:] = np.array([1.0, 0.5 * v, 0.0, 0.0, 0.125 * v * v])[None, :, None]
        m.uold[3, :, 5] = [rho, rho * v, 0.0, 0.0, 0.5 * rho * v * v + eint]
        # the square of 1e-160 is subnormal: 2,024 units of the smallest number,
        # so each rounding of the sound speed's square is up to 1/4048 of it
        compare(m, prec, smallc=smallc, gravity=gravity, rel=1e-3 if smallc == 1e-160 else 1e-11)


@pytest.mark.parametrize("rho", [1e-308, 1e-300])
def test_subnormal_density(rho):
    m = uniform_mesh(2, bc="periodic")
    m.uold[:] = np.array([rho, 0.0, 0.0, 0.0, 2.5 * rho])[None, :, None]
    compare(m, "fp64", smallr=1e-308)


def test_an_infinite_energy_gives_no_step():
    m = uniform_mesh(2, bc="periodic")
    m.uold[:] = np.array([1.0, 0.0, 0.0, 0.0, 2.5])[None, :, None]
    m.uold[1, 4, 2] = np.inf
    compare(m, "fp64")
