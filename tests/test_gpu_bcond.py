"""The ghost cells of every kind of boundary against the oracle's sequential
faces and corners (bcond.f90:16-42, bc_corner.f90:23-157): all of w and p,
ghosts and edges included, after a state upload.

The blocks are the sizes where the items of the boundary launch meet its
edges: the smallest block, lengths around a warp, no two axes alike; the
boundary kinds mix, with walls (whose pressure follows the inner layer) above
and below far-field faces, and faces without a condition, whose ghosts keep
what the upload put there and whose corner cells run as a second launch.

Tolerance: the far field's powers are CUDA's against glibc's (at most 3 ulp
each, and a ghost takes at most three of them in turn), everything else is the
same arithmetic, so 1e-12 of the field's largest value is well above both.
"""
import numpy as np
import pytest

from code_mge_gb300 import cases as K
from code_mge_gb300.runtime import Cycle
from oracle.oracle import OracleCycle
from tests.parity import RTOL, rel_err

pytestmark = pytest.mark.gpu

BC = {
    "far": (-20,) * 6,
    "periodic_k": (-20, -20, -60, -20, -20, -60),
    "walls": (-80, -20, -80, -80, -80, -20),
    "wall_symm": (-50, -80, -20, -80, -50, -80),
    "open": (0, 0, -60, 0, 0, -60),
    "open_far": (-20, 0, -80, 0, -50, 0),
    "none": (0,) * 6,
}


def _state(n, prm, seed):
    """A positive state with inflow and outflow on every face."""
    r = np.random.default_rng(seed)
    shape = (n[2] + 4, n[1] + 4, n[0] + 4)
    rho = 1.0 + 0.2 * r.uniform(-1, 1, shape)
    u = 0.8 * r.uniform(-1, 1, (3,) + shape)
    p = prm.p0 * (1.0 + 0.2 * r.uniform(-1, 1, shape))
    return np.stack([rho, rho * u[0], rho * u[1], rho * u[2],
                     p / (prm.gamma - 1.0) + 0.5 * rho * (u * u).sum(0)])


@pytest.mark.parametrize("gamma", [1.4, 1.3])
@pytest.mark.parametrize("n", [(2, 2, 2), (3, 2, 5), (9, 31, 4), (33, 8, 17)])
@pytest.mark.parametrize("bc", sorted(BC))
def test_ghosts_against_oracle(bc, n, gamma):
    case = K.free_stream_box(n=n, nlevel=1, mach=0.5, bctype=BC[bc], gamma=gamma)
    g, o = Cycle(case), OracleCycle(case)
    for seed in (1, 2):
        w = _state(n, case.prm, seed)
        g.upload(w, 1)
        o.upload(w, 1)
        for f in ("w", "p"):
            assert rel_err(g.field(f, 1), o.field(f, 1)) <= RTOL, (bc, n, f)
