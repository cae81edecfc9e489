"""An update between mge_cycle_async and mge_cycle_poll: the poll returns the
residual of the cycle it belongs to, and each level records its own.  Both runs
make the same launches in the same order, so the numbers are equal.
"""
import ctypes as C

import pytest

from code_mge_gb300 import _abi as A
from code_mge_gb300.runtime import Cycle
from tests.parity import small_sphere

pytestmark = pytest.mark.gpu


def test_update_of_another_level_before_the_poll(gpulib, monkeypatch):
    monkeypatch.setenv("MGE_TUNE_PLAN", "1:0000,2:0000")
    case = small_sphere(nlevel=2, n=16, mcyc_fine=3)
    f, g = Cycle(case), Cycle(case)
    r = f.cycle(2, ncyc=1)
    f.euler(1, ncyc=4, mgl=1, mlvl=1)

    assert gpulib.mge_cycle_async(g.ctx, 2) == A.MGE_OK
    g.euler(1, ncyc=4, mgl=1, mlvl=1)
    out = C.c_double()
    rc = 1
    while rc == 1:
        rc = gpulib.mge_cycle_poll(g.ctx, 1, C.byref(out))
    assert rc == A.MGE_OK
    assert f.rtrms(1, 4) != r
    assert out.value == r == g.rtrms(2, 1) == f.rtrms(2, 1)
    assert g.rtrms(1, 4) == f.rtrms(1, 4)
    f.close()
    g.close()
