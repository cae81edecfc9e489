"""A stop belongs to the call that found it: the error word is cleared in the order
of the calls.  Time steps alternate, with nothing between them, on a level whose
state stops each one (a negative density, timestep.f90:45-48) and on a good one:
every call on the bad level stops, no call on the good level does.  The same after
mge_cycle_poll has returned a stop.
"""
import ctypes as C

import pytest

from code_mge_gb300 import _abi as A
from code_mge_gb300.runtime import Cycle
from tests.parity import small_sphere

pytestmark = pytest.mark.gpu


def _contexts():
    case = small_sphere(nlevel=2, n=16, mcyc_fine=3)
    g = Cycle(case)
    bad = g.field("w", 2).copy()
    bad[0, 4, 4, 4] = -abs(bad[0, 4, 4, 4])
    return g, bad


def test_alternating_stops(gpulib):
    g, bad = _contexts()
    g.upload(bad, 2)
    for _ in range(300):
        assert gpulib.mge_timestep(g.ctx, 2, 1) == A.MGE_ENEGPRESS
        assert gpulib.mge_timestep(g.ctx, 1, 1) == A.MGE_OK
    g.close()


def test_after_a_poll(gpulib):
    g, bad = _contexts()
    good = [g.field("w", lv) for lv in (1, 2)]
    out = C.c_double()
    for n in range(20):
        g.upload(bad, 2)
        assert gpulib.mge_cycle_async(g.ctx, 2) == A.MGE_OK
        rc = 1
        while rc == 1:
            rc = gpulib.mge_cycle_poll(g.ctx, 1, C.byref(out))
        assert rc == A.MGE_ENEGPRESS
        for lv in (1, 2):
            g.upload(good[lv - 1], lv)
        assert gpulib.mge_timestep(g.ctx, 2, 1) == A.MGE_OK
    g.close()
