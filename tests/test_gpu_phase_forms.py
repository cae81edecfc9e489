"""One update by a launch per phase on blocks either side of the sizes at which the
passes change their form (32,768, 300,000 and 1,000,000 cells), with the launch form
fixed, so that the size alone decides: the central scheme in FP64 and in the mixed
form, and the Roe and MUSCL schemes of the Euler and Navier-Stokes equations.

FP64 against the oracle: every form rounds like the reference, 1e-12.  The mixed
form's FP32 time step and smoothing differ from FP64 by a few hundred roundings of
6e-8 of an update that is below the state itself: 1e-4.
"""
import numpy as np
import pytest

from code_mge_gb300 import _abi as A
from code_mge_gb300 import cases as K
from code_mge_gb300.runtime import Cycle, physical
from oracle.oracle import OracleCycle
from tests.parity import RTOL, rel_err

pytestmark = pytest.mark.gpu

JST = dict()
ROE = dict(distype=A.MGE_DIS_ROE1)
MUSCL = dict(distype=A.MGE_DIS_ROE2)
NS = dict(distype=A.MGE_DIS_ROE2, eqntype=A.MGE_EQN_NS, reynolds=200.0)
CASES = [(n, "jst", JST) for n in ((32, 32, 32), (33, 32, 32), (100, 60, 50), (101, 61, 50), (101, 100, 99),
                                   (101, 101, 99))]
CASES += [(n, name, kw) for n in ((32, 32, 32), (33, 32, 32)) for name, kw in (("roe", ROE), ("muscl", MUSCL), ("ns", NS))]


def _case(n, precision, kw):
    body = K.Body("ellipsoid", center=(0.03, 0.02, 0.01), semi=(0.6, 0.5, 0.7))
    h = 8.0 / max(n)
    hi = tuple(0.5 * v * h for v in n)
    levels = K.same_domain_hierarchy(body, tuple(-v for v in hi), hi, n, 1)
    return K.Case("forms", K.params(0.5, alpha_deg=2.0, nlevel=1, mcyc=[1], precision=precision, **kw), levels, body)


@pytest.mark.parametrize("n,scheme,kw", CASES, ids=["%s-%dx%dx%d" % ((s,) + n) for n, s, _ in CASES])
def test_update_by_phases(n, scheme, kw, monkeypatch):
    monkeypatch.setenv("MGE_TUNE_PLAN", "1:0000")
    monkeypatch.setenv("MGE_COOP_MAX_CELLS", "0")
    case = _case(n, A.MGE_PREC_FP64, kw)
    o, g, m = OracleCycle(case), Cycle(case), Cycle(_case(n, A.MGE_PREC_MIXED, kw))
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
