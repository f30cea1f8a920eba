"""The pencil kernels' FP64 reciprocal and square root (vrcp, vsqrt in
ramses2_b200/csrc/rh_vec.cuh: hardware estimates refined by a Newton-Raphson
and a Goldschmidt-Heron iteration) against correctly rounded results, on the
device: CUDA's 1.0/x and sqrt(x) (which equal IEEE's, checked against numpy)
over a million positive normal doubles spanning 2^-1000 .. 2^1000, the range of
every density, pressure and sound-speed argument of the hydro step."""
import ctypes as C

import numpy as np
import pytest

from ramses2_b200._lib import check, lib

pytestmark = pytest.mark.gpu


def ulps(a, b):
    """Distance in units in the last place between positive doubles."""
    return np.abs(a.view(np.int64) - b.view(np.int64))


def test_vrcp_vsqrt_within_two_ulp_of_correct_rounding():
    import torch

    L = lib()
    check(L.rh_init(0), "rh_init")
    rng = np.random.default_rng(2026)
    n = 1 << 20
    x = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-1000, 1000, n))
    x[:64] = np.ldexp(1.0, np.arange(-32, 32))              # exact powers of two
    x[64:128] = 1.0 + np.arange(64) * np.finfo(np.float64).eps  # just above 1
    x[128:192] = np.nextafter(np.ldexp(1.0, np.arange(-32, 32)), 0)  # just below powers of two
    dx = torch.from_numpy(x).to("cuda")
    out = torch.empty(4 * n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    check(L.rh_selftest_vmath(C.c_void_p(dx.data_ptr()), n, C.c_void_p(out.data_ptr())), "rh_selftest_vmath")
    o = out.cpu().numpy().reshape(4, n)
    rcp_ieee, sqrt_ieee = 1.0 / x, np.sqrt(x)
    assert np.array_equal(o[2], rcp_ieee) and np.array_equal(o[3], sqrt_ieee)  # CUDA's are correctly rounded
    ur, us = ulps(o[0], o[2]), ulps(o[1], o[3])
    assert ur.max() <= 2, (ur.max(), x[ur.argmax()])
    assert us.max() <= 2, (us.max(), x[us.argmax()])
    # The error left before the last rounding is at most that of the estimate (20
    # bits or more) to the fourth power for 1/x, and about the square of s's
    # error after one step (3/8 of the estimate's squared, 2^-41) for the root:
    # below 2^-78, so a result differs from the correctly rounded one where the
    # exact value lies within 2^-25 ulp of a tie, some 0.1 of a million values.
    # (The first 192 are made: 1/x of a number just below a power of two lies
    # 2^-53 ulp from a tie, and either neighbour may come.)
    assert ur.max() <= 1 and (ur[192:] > 0).sum() <= 4, (ur.max(), (ur[192:] > 0).sum())
    assert us.max() <= 1 and (us[192:] > 0).sum() <= 4, (us.max(), (us[192:] > 0).sum())
