"""Which fine ghost cells the parent fills (bc_embed.f90:47-143), against the oracle
with the child's ends on the parent's or inside them, axis by axis: only a child whose
ends are all the parent's has no such cell, and no launch over its cells.

FP64 rounds like the reference: 1e-12.  Every ghost cell is compared, and the group's
form (which asks the same of its cases together) bit for bit with the case alone.
"""
import numpy as np
import pytest

from code_mge_gb300 import cases as K
from code_mge_gb300.runtime import Cycle
from oracle.oracle import OracleCycle
from tests.parity import RTOL, rel_err
from tests.test_gpu_group import _fmg_group, _fmg_single

pytestmark = pytest.mark.gpu

# offset and extent of the child in the parent's 8 x 8 x 8 cells, ratio
ENDS = {
    "all_on": ((0, 0, 0), (8, 8, 8), (2, 2, 2)),
    "all_on_ratio_one": ((0, 0, 0), (8, 8, 8), (2, 1, 2)),
    "above_inside": ((0, 0, 0), (8, 8, 6), (2, 2, 2)),
    "below_inside": ((0, 2, 0), (8, 6, 8), (2, 2, 2)),
    "one_axis": ((2, 0, 0), (4, 8, 8), (2, 2, 1)),
    "inside": ((2, 2, 2), (4, 4, 4), (2, 2, 2)),
}


def _case(ends):
    off, ext, ratio = ENDS[ends]
    body = K.Body("sphere", center=(0.05, 0.02, -0.03), radius=0.25)
    h = 0.2
    coarse = K.BlockSpec(n=(8, 8, 8), h=(h,) * 3, origin=(-0.8,) * 3, bctype=(-20,) * 6)
    bct = [0] * 6
    for d in range(3):
        if off[d] == 0:
            bct[d] = -20
        if off[d] + ext[d] == 8:
            bct[3 + d] = -20
    fine = K.BlockSpec(n=tuple(e * r for e, r in zip(ext, ratio)), h=tuple(h / r for r in ratio),
                       origin=tuple(-0.8 + h * o for o in off), bctype=tuple(bct), parent=1, ratio=ratio, offset=off)
    levels = [[K.make_block_arrays(coarse, body)], [K.make_block_arrays(fine, body)]]
    return K.Case("ends", K.params(0.4, nlevel=2, mcyc=[1, 1]), levels, body)


@pytest.mark.parametrize("ends", sorted(ENDS))
def test_embed_ends(ends):
    case = _case(ends)
    o, g = OracleCycle(case), Cycle(case)
    r = np.random.default_rng(11)
    for L in (1, 2):
        w = o.field("w", L)
        w = w * (1.0 + 0.02 * r.uniform(-1, 1, w.shape))
        for c in (o, g):
            c.upload(w, L)
    for step in ("movco", "movfin"):
        for c in (o, g):
            c.movco(1) if step == "movco" else c.movfin(2, 2)
        for L in (1, 2):
            for f in ("w", "p", "wn"):
                if f == "wn" and (L == 2 or step == "movfin"):
                    continue
                assert rel_err(g.field(f, L), o.field(f, L)) <= RTOL, (step, f, L)


def test_group_asks_all_its_cases(gpulib, monkeypatch):
    cases = [_case("all_on"), _case("inside")]
    monkeypatch.setenv("MGE_TUNE_PLAN", "1:0000,2:0000")
    monkeypatch.setenv("MGE_COOP_MAX_CELLS", "0")
    single, group = [Cycle(c) for c in cases], [Cycle(c) for c in cases]
    hs = [_fmg_single(gpulib, c, k) for c, k in zip(single, cases)]
    hg = _fmg_group(gpulib, group, cases)
    for q in range(len(cases)):
        assert hg[q] == hs[q], q
        for L in (1, 2):
            assert np.array_equal(group[q].field("w", L), single[q].field("w", L)), (q, L)
    for c in single + group:
        c.close()
