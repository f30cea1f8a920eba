"""courant_fine values reach the host two ways: a launch stores a level's own
values (then its number) in pinned memory, and a coarse step of several levels
copies all levels' values on a stream no launch waits for.  The two never share
an array: a copy that lands late would replace values a later launch stored,
under that launch's number."""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ramses2_b200", "csrc")


def test_launches_and_copies_store_to_different_arrays():
    src = ""
    for f in sorted(os.listdir(CSRC)):
        if f.endswith(".cu"):
            src += re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
    stored = set(re.findall(r"\.cfl_host\s*=\s*c\.(\w+)", src))
    assert len(stored) == 1
    copied = set(re.findall(r"cudaMemcpyAsync\(\s*c\.(\w+)", src))
    assert "h_cfl_next" in copied
    assert not stored & copied
    # values under a launch's number are read from where that launch stored them
    for fn in ("int rh_cmpdt(", "int rh_coarse_step("):
        body = src[src.index(fn):]
        at = body.index("cfl_seq_of[l")
        read = re.search(r"c\.(h_cfl_\w+) \+ 5", body[at:]).group(1)
        assert {read} == stored, fn


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp32_bulk"])
def test_values_follow_the_state_after_a_step_of_given_dt(precision):
    """Coarse steps that choose dt (and copy all levels' values), each followed
    by one of given dt and by leaf calls: every level's values equal those of a
    pass over the same state, while other read-backs keep the copy engine
    busy."""
    import torch

    from ramses2_b200._abi import HydroParams
    from ramses2_b200.hydro import GodunovGPU, amr_coarse_step
    from ramses2_b200.mesh import sedov_amr_mesh

    m, gamma = sedov_amr_mesh(4, 6, radius=0.2)
    P = HydroParams.make(gamma=gamma, interpol_type=1)
    g = GodunovGPU(m, P, precision=precision)
    levels = range(m.levelmin, m.levelmax + 1)
    busy = torch.cuda.Stream()
    dev = torch.zeros(1 << 25, device="cuda")
    host = torch.empty(1 << 25, pin_memory=True)
    try:
        def compare():
            got = {l: g.courant_fine(l) for l in levels}
            g.push_uold(g.fetch_uold())
            for l in levels:
                fresh = g.courant_fine(l)
                assert got[l][4] == fresh[4]
                assert got[l][:3] == pytest.approx(fresh[:3], rel=1e-12)

        for l in levels:
            g.courant_fine(l)
        for _ in range(6):
            dt = g.coarse_step()
            with torch.cuda.stream(busy):
                host.copy_(dev, non_blocking=True)
            g.coarse_step(dt)
            compare()
            dt = g.coarse_step()
            with torch.cuda.stream(busy):
                host.copy_(dev, non_blocking=True)
            amr_coarse_step(g, m, dt)
            compare()
    finally:
        g.close()
        busy.synchronize()
