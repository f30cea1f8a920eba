"""Tables the library makes on first use are on the device before a kernel
reads them: the library's streams do not wait for the default stream, where
cudaMemcpy and cudaMemset run and which cudaMemcpy from pageable memory may
leave before its bytes arrive (a restriction right after its father table's
copy read what the memory held before)."""
import glob
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ramses2_b200", "csrc")


def test_no_upload_on_the_default_stream():
    files = [f for e in ("cu", "cuh", "h", "inc") for f in glob.glob(os.path.join(CSRC, "*." + e))]
    assert files
    for f in files:
        src = re.sub(r"//[^\n]*", "", open(f).read())
        assert not re.search(r"\bcudaMemset\s*\(", src), f
        for m in re.finditer(r"\bcudaMemcpy\s*\([^;]*;", src):
            assert "cudaMemcpyHostToDevice" not in m.group(0), (f, m.group(0))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp32_bulk"])
def test_first_restriction_reads_its_father_table(precision):
    """Refined cells after one coarse step are the means of their children, in
    a fresh context each time (its memory holds what the one before left)."""
    from ramses2_b200._abi import HydroParams
    from ramses2_b200.hydro import GodunovGPU
    from ramses2_b200.mesh import sedov_amr_mesh

    m, _ = sedov_amr_mesh(4, 6, radius=0.2, bc="reflexive")
    first = None
    for _ in range(6):
        g = GodunovGPU(m, HydroParams.make(gamma=1.4, interpol_type=1, interpol_var=0), precision)
        try:
            g.coarse_step()
            u = g.fetch_uold()
        finally:
            g.close()
        for l in range(m.levelmin + 1, m.levelmax + 1):
            at = {tuple(k): i for i, k in enumerate(m.grid["ckey"][m.level_slice(l - 1)].tolist())}
            ck = m.grid["ckey"][m.level_slice(l)].astype(np.int64)
            father = np.array([at[tuple(k)] for k in (ck >> 1).tolist()]) + m.level_slice(l - 1).start
            cell = (ck & 1) @ np.array([1, 2, 4])
            mean = u[m.level_slice(l)].mean(axis=2)
            got = u[father, :, cell]
            scale = np.abs(u[m.level_slice(l)]).max(axis=2)
            # eight roundings of the sum, and one to 32 bits of the stored mean
            eps = 8 * 2.0 ** -53 + (2.0 ** -24 if precision != "fp64" else 0.0)
            assert np.all(np.abs(got - mean) <= 2 * eps * scale)
        first = u if first is None else first
        assert np.array_equal(u, first)
