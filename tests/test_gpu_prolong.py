"""The prolongation (movfin.f90, addw.f90:83-188) against the oracle on the grids
where its items meet their edges: the smallest block that has octets of fine
cells, blocks without (a ratio of one, fewer than four cells), unequal axes, and a
fine block inside its parent (an offset, no clamped stencil).

FP64 rounds like the reference: 1e-12.  The mixed form interpolates FP32
corrections under an FP64 level: each is eight products and sums of values
rounded to 6e-8, so 1e-6 of the field's largest value bounds the difference.
"""
import numpy as np
import pytest

from code_mge_gb300 import _abi as A
from code_mge_gb300 import cases as K
from code_mge_gb300.runtime import Cycle
from oracle.oracle import OracleCycle
from tests.parity import RTOL, rel_err

pytestmark = pytest.mark.gpu

GRIDS = {
    "smallest": dict(n=(4, 4, 4)),
    "unequal": dict(n=(12, 4, 34)),
    "odd_parent": dict(n=(10, 6, 14)),
    "slab": dict(n=(16, 12, 2), coarsen=(True, True, False)),
    "inside": dict(n=(8, 12, 16), inside=True),
}


def _case(grid, precision):
    g = GRIDS[grid]
    body = K.Body("sphere", center=(0.1, 0.05, 0.02), radius=0.4)
    n = g["n"]
    if g.get("inside"):
        levels = K.embedded_hierarchy(body, (0.0, 0.0, 0.0), (0.25,) * 3, n, 2, coarsen=(True, True, True))
    else:
        hi = tuple(0.1 * v for v in n)
        levels = K.same_domain_hierarchy(body, tuple(-v for v in hi), hi, n, 2, coarsen=g.get("coarsen", (True,) * 3))
    return K.Case("prolong", K.params(0.4, nlevel=2, mcyc=[1, 1], precision=precision), levels, body)


@pytest.mark.parametrize("fmg", [False, True])
@pytest.mark.parametrize("grid", sorted(GRIDS))
def test_prolongation(grid, fmg):
    case = _case(grid, A.MGE_PREC_FP64)
    o, g, m = OracleCycle(case), Cycle(case), Cycle(_case(grid, A.MGE_PREC_MIXED))
    r = np.random.default_rng(7)
    for L in (1, 2):
        w = o.field("w", L)
        w = w * (1.0 + 0.02 * r.uniform(-1, 1, w.shape))
        for c in (o, g, m):
            c.upload(w, L)
    for c in (o, g, m):
        c.movfin(2, 1 if fmg else 2)
    for f in ("w", "p"):
        assert rel_err(g.field(f, 2), o.field(f, 2)) <= RTOL, f
    assert rel_err(m.field("w", 2), o.field("w", 2)) <= 1e-6
