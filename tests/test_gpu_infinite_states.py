"""The time step's stop (timestep.f90:45-48) where gamma*p/rho is not a finite
number: an infinite density, an infinite energy, a quotient beyond the largest
double, and a density of zero.  The quotient by the density is formed as
q = a*(1/rho) and corrected by its remainder, which is NaN for each of them, and a
NaN stops the run: on blocks that take the FP64 pipe's own operations (up to
32,768 cells), on larger ones, which take the integer pipes, and in FP32.
"""
import numpy as np
import pytest

from code_mge_gb300 import _abi as A
from code_mge_gb300 import cases as K
from code_mge_gb300.runtime import Cycle

pytestmark = pytest.mark.gpu

# (variable, value) written into one cell
STATES = {
    "infinite_density": [(0, np.inf)],
    "infinite_energy": [(4, np.inf)],
    "overflow": [(0, 1e-3), (1, 0.0), (2, 0.0), (3, 0.0), (4, 1.7e308)],
    "zero_density": [(0, 0.0)],
}


@pytest.mark.parametrize("n", [(32, 32, 32), (33, 32, 32)], ids=["plain", "integer_pipes"])
@pytest.mark.parametrize("precision", [A.MGE_PREC_FP64, A.MGE_PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("state", sorted(STATES))
def test_time_step_stops(gpulib, state, precision, n, monkeypatch):
    monkeypatch.setenv("MGE_TUNE_PLAN", "1:0000")
    monkeypatch.setenv("MGE_COOP_MAX_CELLS", "0")
    g = Cycle(K.free_stream_box(n=n, nlevel=1, precision=precision))
    good = g.field("w", 1)
    assert gpulib.mge_timestep(g.ctx, 1, 1) == A.MGE_OK
    w = good.copy()
    for v, x in STATES[state]:
        w[v, 9, 8, 7] = x
    g.upload(w, 1)
    assert gpulib.mge_timestep(g.ctx, 1, 1) == A.MGE_ENEGPRESS
    g.upload(good, 1)
    assert gpulib.mge_timestep(g.ctx, 1, 1) == A.MGE_OK
    g.close()
