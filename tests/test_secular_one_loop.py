"""Sweeps that take both sides of a root's bracket in one loop
(sec_accum_any, csrc/brdc_secular.cuh) find the roots that two-sided sweeps
find, on the host."""
import ctypes

import numpy as np
import pytest


@pytest.fixture(scope="module")
def hostlib(built_lib):
    import build as b

    return ctypes.CDLL(b.HOSTLIB)


@pytest.mark.parametrize("lanes", [1, 2, 32])
@pytest.mark.parametrize("K", [2, 3, 31, 32, 33, 64, 65, 200])
def test_same_roots(hostlib, K, lanes):
    rng = np.random.default_rng(K)
    dp, ci, cd = ctypes.POINTER(ctypes.c_double), ctypes.c_int, ctypes.c_double
    for tiny in (False, True):
        d = np.sort(rng.standard_normal(K))
        z = rng.standard_normal(K)
        z[::2] *= 1e-7 if tiny else 1.0
        z /= np.linalg.norm(z)
        rho, zn = 1.5, float(z @ z)
        for i in range(K):
            got = []
            for one in (False, True):
                org, tau, bad = ci(), cd(), ci()
                tail = (ctypes.byref(org), ctypes.byref(tau), ctypes.byref(bad))
                head = (ci(K), d.ctypes.data_as(dp), z.ctypes.data_as(dp), cd(rho), cd(zn), ci(i))
                if one:
                    hostlib.brdc_host_secular_root_any(*head, ci(lanes), *tail)
                else:
                    hostlib.brdc_host_secular_root(*head, *tail)
                assert bad.value == 0
                got.append((org.value, tau.value))
            # each stops with |f| within its error bound, so a root may move
            # by the rounding of d + tau and of the sums (8 eps a pole)
            lam = [d[o] + t for o, t in got]
            assert abs(lam[0] - lam[1]) <= 8 * K * np.finfo(float).eps * max(1.0, np.abs(d).max())
