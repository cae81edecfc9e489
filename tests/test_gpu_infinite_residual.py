"""The stop on the residual norm (solver.f90:180) where a smoothed residual is
infinite: the line sweeps form quotients whose remainder is then NaN, and the norm
with it, whatever form a sweep takes.  A single-stage update in the unsteady mode,
whose source term of one cell overflows (4 w1 with a density of 1e308 in the old
time level), with one cell an access and with pairs, on the FP64 pipe and on the
integer pipes.  The cell lies beyond the rows in which the pivots still change.
"""
import numpy as np
import pytest

from code_mge_gb300 import _abi as A
from code_mge_gb300 import cases as K
from code_mge_gb300.runtime import Cycle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(24, 24, 24), (25, 42, 40), (26, 42, 40), (24, 174, 174)],
                         ids=lambda n: "x".join(map(str, n)))
@pytest.mark.parametrize("plan", ["1:0000", "1:0111"], ids=["lines", "tiles"])
def test_the_norm_stops(gpulib, plan, n, monkeypatch):
    monkeypatch.setenv("MGE_TUNE_PLAN", plan)
    monkeypatch.setenv("MGE_COOP_MAX_CELLS", "0")
    g = Cycle(K.free_stream_box(n=n, nlevel=1, cstp=(0.25,), cdis=(1.0,), execmode=1, dtstep=0.1))
    good = g.field("w", 1)
    w = good.copy()
    w[0, 21, 21, 21] = 1e308
    g.upload(w, 1)
    g.time_advance()
    g.upload(good, 1)
    assert gpulib.mge_timestep(g.ctx, 1, 1) == A.MGE_OK
    assert gpulib.mge_euler(g.ctx, 1, 1, 2, 1, 1, 1, 0, 0) == A.MGE_ENAN
    assert not np.isfinite(g.field("dw", 1)[0]).all()
    # the old levels good again: the update runs
    g.upload(good, 1)
    g.time_advance()
    g.time_advance()
    assert gpulib.mge_timestep(g.ctx, 1, 1) == A.MGE_OK
    assert gpulib.mge_euler(g.ctx, 1, 1, 2, 1, 1, 1, 0, 0) == A.MGE_OK
    g.close()
