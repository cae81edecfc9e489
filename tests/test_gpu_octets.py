"""The 2:1 prolongation by octets of fine cells (more than 200,000 cells, movfin.f90,
addw.f90:83-188) against the oracle: unequal axes, an axis of four cells (one octet
between its two shells), a fine block inside its parent, and an FP32 level under an
FP32 one.  The sizes lie just above the one from which a level runs so.

The cells compared are the physical ones, which the prolongation writes (a corner
ghost is an extrapolation, and its pressure a quotient by a density that may be near
zero).  FP64 rounds like the reference: 1e-12.  An FP32 level holds states and corrections
rounded to 6e-8 of the state: the fine state, two coarse ones and the sum, so 1e-6 of
the field's largest value bounds the difference.
"""
import numpy as np
import pytest

from code_mge_gb300 import _abi as A
from code_mge_gb300 import cases as K
from code_mge_gb300.runtime import Cycle, physical
from oracle.oracle import OracleCycle
from tests.parity import RTOL, rel_err

pytestmark = pytest.mark.gpu

GRIDS = {
    "unequal": dict(n=(44, 62, 76)),
    "four_cells": dict(n=(4, 226, 224)),
    "four_cells_along_k": dict(n=(228, 222, 4)),
    "inside": dict(n=(76, 44, 62), inside=True),
}


def _case(grid, precision, nlevel):
    g = GRIDS[grid]
    n = g["n"]
    assert n[0] * n[1] * n[2] > 200000
    body = K.Body("sphere", center=(0.1, 0.05, 0.02), radius=0.4)
    if g.get("inside"):
        levels = K.embedded_hierarchy(body, (0.0, 0.0, 0.0), (0.05,) * 3, n, nlevel, coarsen=(True, True, True))
    else:
        hi = tuple(0.1 * v for v in n)
        levels = K.same_domain_hierarchy(body, tuple(-v for v in hi), hi, n, nlevel)
    return K.Case("octets", K.params(0.4, nlevel=nlevel, mcyc=[1] * nlevel, precision=precision), levels, body)


def _prolonged(c, w, fmg):
    for L in (1, 2):
        c.upload(w[L - 1], L)
    c.movfin(2, 1 if fmg else 2)


def _states(o):
    r = np.random.default_rng(7)
    return [w * (1.0 + 0.02 * r.uniform(-1, 1, w.shape)) for w in (o.field("w", 1), o.field("w", 2))]


@pytest.mark.parametrize("fmg", [False, True])
@pytest.mark.parametrize("grid", sorted(GRIDS))
def test_fp64(grid, fmg, monkeypatch):
    monkeypatch.setenv("MGE_AUTOTUNE", "0")
    case = _case(grid, A.MGE_PREC_FP64, 2)
    o, g = OracleCycle(case), Cycle(case)
    w = _states(o)
    for c in (o, g):
        _prolonged(c, w, fmg)
    sp = case.levels[1][0]
    for f in ("w", "p"):
        assert rel_err(physical(g.field(f, 2), sp), physical(o.field(f, 2), sp)) <= RTOL, f


@pytest.mark.parametrize("fmg", [False, True])
def test_fp32_level(fmg, monkeypatch):
    """Level 2 of three: FP32 in the mixed form, inside its FP32 parent."""
    monkeypatch.setenv("MGE_AUTOTUNE", "0")
    o = OracleCycle(_case("inside", A.MGE_PREC_FP64, 3))
    g = Cycle(_case("inside", A.MGE_PREC_MIXED, 3))
    w = _states(o)
    for c in (o, g):
        _prolonged(c, w, fmg)
    sp = g.spec(2)
    assert rel_err(physical(g.field("w", 2), sp), physical(o.field("w", 2), sp)) <= 1e-6
