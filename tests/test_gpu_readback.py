"""Reading states back to the host (rh_batch_fetch, rh_transfer_grid_host) at
the sizes where the copy changes its form: one oct, the threshold below which
a plain copy is made, whole pieces of the pinned slots and one oct more."""
import ctypes as C

import numpy as np
import pytest

from ramses2_b200._abi import HydroParams, dptr
from ramses2_b200._lib import check, lib
from ramses2_b200.batch import Batch, ic_host, problem
from ramses2_b200.hydro import GodunovGPU
from ramses2_b200.mesh import uniform_mesh

pytestmark = pytest.mark.gpu


def octs(n, seed):
    u = np.random.default_rng(seed).uniform(1.0, 2.0, (n, 5, 8))
    u[:, 4] += 10.0
    return u


def as_stored(u, prec):
    """What the device holds of u: FP32-bulk keeps all but E in FP32."""
    out = u.copy()
    if prec != "fp64":
        out[:, :4] = u[:, :4].astype(np.float32)
    return out


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("prec", ["fp64", "fp32_bulk"])
def test_batch_fetch_returns_the_state_at_every_copy_size(prec, pinned):
    import torch

    sizes = (1, 1631, 1632, 1633, 16 * 1632, 16 * 1632 + 17, 17 * 13056 + 5)
    b = Batch(prec, pool_octs=sum(sizes))
    try:
        want = {}
        for k, n in enumerate(sizes):
            u = octs(n, k)
            pid = b.add(problem((2, 2, 2 * n), dx=1.0, max_steps=1), ic_host(u))
            want[pid] = as_stored(u, prec)
        for pid, u in want.items():
            if pinned:
                out = torch.empty(u.shape, dtype=torch.float64, pin_memory=True).numpy()
                check(lib().rh_batch_fetch(pid, dptr(out)), "rh_batch_fetch")
            else:
                out = b.fetch(pid)
            assert np.array_equal(out, u)
    finally:
        b.close()


@pytest.mark.parametrize("prec", ["fp64", "fp32_bulk"])
def test_mesh_state_to_pageable_and_pinned_memory(prec):
    import torch

    m = uniform_mesh(5, box_nx=(3, 2, 1))
    m.uold[:] = octs(m.ngridmax, 9)
    g = GodunovGPU(m, HydroParams.make(), precision=prec)
    try:
        want = as_stored(m.uold, prec)
        assert np.array_equal(g.fetch_uold(), want)
        out = torch.empty(want.shape, dtype=torch.float64, pin_memory=True).numpy()
        check(lib().rh_transfer_grid_host(dptr(out), m.ngridmax, 5, 8), "rh_transfer_grid_host")
        assert np.array_equal(out, want)
    finally:
        g.close()


def resident_mb():
    with open("/proc/self/status") as f:
        return next(int(l.split()[1]) for l in f if l.startswith("VmRSS")) / 1024.0


@pytest.mark.parametrize("prec", ["fp64", "fp32_bulk"])
def test_small_read_backs_pin_little_memory(prec):
    """The pinned slots (4.2 MB each, kept until the library is closed) come with
    the first transfer that needs them, as many as it has workers for; a small
    FP32-bulk one has a slot of 0.5 MB."""
    b = Batch(prec, pool_octs=1 << 16)
    try:
        small = b.add(problem((2, 2, 2), dx=1.0, max_steps=1), ic_host(octs(1, 0)))
        two = b.add(problem((2, 2, 2 * 3264), dx=1.0, max_steps=1), ic_host(octs(3264, 1)))
        b.status(small)
        before = resident_mb()
        assert np.array_equal(b.fetch(small), as_stored(octs(1, 0), prec))
        assert resident_mb() - before < 4.0  # less than one slot
        assert np.array_equal(b.fetch(two), as_stored(octs(3264, 1), prec))
        assert resident_mb() - before < 4.0 + 3 * 4.2  # two pieces of 1,632 octs: two slots and the result
    finally:
        b.close()
