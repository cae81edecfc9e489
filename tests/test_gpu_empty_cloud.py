"""A record whose cloud is empty, on the GPU: bc_cutcell.f90:65-70 zeroes that
record and leaves the routine, so the records after it keep the solid state they
had.  Against the oracle, with the empty cloud at the first, a middle and the last
record and with none, and with cells outside the block in every entry of ijkdex
past a record's npoint: those entries are not part of any cloud and nothing may
form an address from them.

The weights and the state are the same numbers on both sides and the operations
round alike: 1e-12.
"""
import numpy as np
import pytest

from code_mge_gb300 import _abi as A
from code_mge_gb300.runtime import Cycle, MgeError
from oracle.oracle import OracleCycle
from tests.parity import RTOL, rel_err, small_sphere

pytestmark = pytest.mark.gpu


def _case(empty):
    case = small_sphere(nlevel=1, n=16, mcyc_fine=2)
    a = case.levels[0][0].arrays
    nm = a["nmir"]
    ncl, ijk, coef = (np.array(a[k]) for k in ("npoint", "ijkdex", "coef"))
    ncl[1::3] = 1  # clouds of one cell among the full ones
    coef[1::3] = 0.0
    coef[1::3, 0] = 1.0
    if empty is not None:
        ncl[int(empty * (nm - 1))] = 0
    outside = np.array([100000, -70000, 2000000], dtype=np.int32)
    for m in range(nm):
        ijk[m, ncl[m]:] = outside
    a.update(npoint=ncl, ijkdex=ijk, coef=coef)
    return case


@pytest.mark.parametrize("path", ["coop", "phases"])
@pytest.mark.parametrize("empty", [None, 0.0, 0.5, 1.0])
def test_solid_states(empty, path, monkeypatch):
    monkeypatch.setenv("MGE_COOP_MAX_CELLS", "0" if path == "phases" else str(10 ** 9))
    monkeypatch.setenv("MGE_TUNE_PLAN", "1:0000" if path == "phases" else "1:1000")
    case = _case(empty)
    o, g = OracleCycle(case), Cycle(case)
    r = np.random.default_rng(5)
    w = o.field("w", 1)
    w = w * (1.0 + 0.02 * r.uniform(-1, 1, w.shape))

    def same():
        for f in ("wsol", "psol"):
            assert rel_err(g.field(f, 1), o.field(f, 1)) <= RTOL, f

    for c in (o, g):
        c.upload(w, 1)
    same()
    # an update: the solid states of its stages share a launch with the boundaries
    if empty is None:
        for c in (o, g):
            c.timestep(1)
            c.euler(1)
        same()
        assert rel_err(g.field("w", 1), o.field("w", 1)) <= RTOL
        return
    # a wall state of zeros divides by its density: the run stops, and goes on
    # from a good state
    g.timestep(1)
    with pytest.raises(MgeError) as e:
        g.euler(1)
    assert e.value.code == A.MGE_ENAN
    g.upload(w, 1)
    m0 = int(empty * (case.levels[0][0].arrays["nmir"] - 1))
    for f in ("wsol", "psol"):  # the records up to the empty one; those after it are not formed again
        assert rel_err(g.field(f, 1)[:m0 + 1], o.field(f, 1)[:m0 + 1]) <= RTOL, f
