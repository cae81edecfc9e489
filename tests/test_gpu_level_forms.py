"""One update on blocks either side of the sizes at which the stage passes change
their form: plain FP64 operations or the integer pipes (32,768 cells), one thread
per cell or per cell and direction (300,000 and 1,000,000 cells).

FP64 against the oracle: every form rounds like the reference, so the field and
the residual history agree to 1e-12.  The mixed form's finest level differs from
FP64 by its FP32 time step and smoothing: at most a few hundred roundings of 6e-8
of an update that is below the state itself, so 1e-4 bounds it, and an index gone
wrong in a form does not stay below that.
"""
import numpy as np
import pytest

from code_mge_gb300 import _abi as A
from code_mge_gb300 import cases as K
from code_mge_gb300.runtime import Cycle, physical
from oracle.oracle import OracleCycle
from tests.parity import RTOL, rel_err

pytestmark = pytest.mark.gpu

SIZES = [(32, 32, 32), (33, 32, 32), (100, 60, 50), (101, 61, 50), (101, 100, 99), (101, 101, 99)]


def _case(n, precision):
    body = K.Body("ellipsoid", center=(0.03, 0.02, 0.01), semi=(0.6, 0.5, 0.7))
    h = 8.0 / max(n)
    hi = tuple(0.5 * v * h for v in n)
    levels = K.same_domain_hierarchy(body, tuple(-v for v in hi), hi, n, 1)
    return K.Case("forms", K.params(0.5, alpha_deg=2.0, nlevel=1, mcyc=[1], precision=precision), levels, body)


@pytest.mark.parametrize("n", SIZES)
def test_update_either_side_of_a_form(n):
    case = _case(n, A.MGE_PREC_FP64)
    o, g, m = OracleCycle(case), Cycle(case), Cycle(_case(n, A.MGE_PREC_MIXED))
    r = np.random.default_rng(3)
    w = o.field("w", 1) * (1.0 + 0.01 * r.uniform(-1, 1, o.field("w", 1).shape))
    for c in (o, g, m):
        c.upload(w, 1)
        c.timestep(1)
        c.euler(1, ncyc=1)
    sp = case.levels[0][0]
    for f in ("w", "p"):
        assert rel_err(g.field(f, 1), o.field(f, 1)) <= RTOL, f
    assert rel_err(physical(g.field("dw", 1), sp), physical(o.field("dw", 1), sp)) <= RTOL
    assert abs(g.rtrms(1, 1) - o.rtrms(1, 1)) <= RTOL * o.rtrms(1, 1)
    assert rel_err(m.field("w", 1), o.field("w", 1)) <= 1e-4
