"""The i line sweeps (psmoo.f90:171-237) that move two cells an access, against the
oracle where their chunks meet their ends: the shortest lines, one chunk of pairs and
a remainder of every length, an odd row (which takes the single cells), blanked cells
at both places of a pair, and enough lines for the integer-pipe form.

The sweeps round like the reference: 1e-12.
"""
import numpy as np
import pytest

from code_mge_gb300 import cases as K
from code_mge_gb300.runtime import Cycle
from oracle.oracle import OracleCycle
from tests.parity import RTOL, rel_err

pytestmark = pytest.mark.gpu

SIZES = [(2, 42, 40), (4, 42, 40), (8, 42, 40), (10, 42, 40), (11, 42, 40), (12, 42, 40), (14, 42, 40), (16, 42, 40),
         (26, 42, 40), (26, 6, 4), (28, 42, 39), (30, 42, 41), (10, 174, 174), (12, 174, 174)]


@pytest.mark.parametrize("n", SIZES, ids=lambda n: "x".join(map(str, n)))
def test_i_sweep(n, monkeypatch):
    monkeypatch.setenv("MGE_TUNE_PLAN", "1:0000")
    monkeypatch.setenv("MGE_COOP_MAX_CELLS", "0")
    body = K.Body("sphere", center=(0.013, 0.021, 0.017), radius=0.22)
    h = 2.0 / max(n[0], 8)
    hi = tuple(0.5 * h * v for v in n)
    levels = K.same_domain_hierarchy(body, tuple(-v for v in hi), hi, n, 1)
    case = K.Case("line_pairs", K.params(0.5, nlevel=1, mcyc=[1]), levels, body)
    o, g = OracleCycle(case), Cycle(case)
    r = np.random.default_rng(3)
    w = o.field("w", 1)
    w = w * (1.0 + 0.01 * r.uniform(-1, 1, w.shape))
    for c in (o, g):
        c.upload(w, 1)
        c.timestep(1)
        c.euler(1)
    for f in ("w", "p", "dw"):
        assert rel_err(g.field(f, 1), o.field(f, 1)) <= RTOL, f
