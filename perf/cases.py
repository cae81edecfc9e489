"""Workloads of the multigrid cycle, timed through the library's public entry points.

A case is a flow past a body on a hierarchy of Cartesian blocks, a start state and a
number of cycles (or single Runge-Kutta updates).  One pass is what a host program does
with a resident case: it uploads the finest level's state from pinned host memory, runs the
cycles, and downloads the new state (w, p) into pinned host memory beside the residual of
every cycle.  ``mge_solve`` is timed as a whole from the free stream.

The kinds of work:

* ``update``  mge_timestep + mge_euler per update: the per-call drop-in of solver.f90:154-155
* ``cycles``  mge_cycle: one V- or W-cycle per call, replayed from a CUDA graph
* ``group``   mge_group_cycle_async / _poll: many cases of different sizes in lockstep
* ``solve``   mge_init_flow + mge_solve: the whole full-multigrid solve with its forces

``exact`` restates the same computation in plain torch in float64.
"""
import ctypes as C
import math
import os
import random

import numpy as np
import torch

from code_mge_gb300 import _abi as A
from code_mge_gb300 import cases as K
from code_mge_gb300.runtime import Cycle, load_library

GAMMA = 1.4


# ----------------------------------------------------------------- the cases
def _case(kind, grid, nx, ny, nz, levels, scheme="jst", precision="fp64", mgtype=2, cycles=2, extent=4.0, members=1,
          unsteady=False, body="ellipsoid", name=None):
    c = dict(kind=kind, grid=grid, nx=nx, ny=ny, nz=nz, levels=levels, scheme=scheme, precision=precision,
             mgtype=mgtype, cycles=cycles, extent=extent, members=members, unsteady=unsteady,
             body=body if grid == "box" else "cylinder")
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest calls: a coarse block driven update by update, the host
        # reading the error word after every call; latency and launches count
        _case("update", "box", 24, 24, 24, 1, cycles=4, body="sphere", name="update_box24"),
        # the same calls on one large odd-sized block of a multi-block grid file
        _case("update", "box", 131, 97, 75, 1, cycles=2, name="update_box_odd"),
        # the circular cylinder in a 256x256x2 slab, 3-level V-cycle
        _case("cycles", "slab", 256, 256, 2, 3, mgtype=1, cycles=8, extent=20.0, name="slab256_v"),
        # a small 3-D case, as the tests and the sweep's smaller members run it
        _case("cycles", "box", 48, 48, 48, 3, cycles=4, name="box48_w"),
        # a grid that is no cube: each direction of the sweeps has its own length
        _case("cycles", "box", 120, 88, 56, 3, cycles=4, name="box120x88x56_w"),
        # the 192^3 sphere, 4-level W-cycle: the largest, in FP64 ...
        _case("cycles", "box", 192, 192, 192, 4, cycles=2, extent=10.0, body="sphere", name="sphere192_w"),
        # ... and with FP32 coarse levels, time step and smoothing
        _case("cycles", "box", 192, 192, 192, 4, cycles=2, extent=10.0, body="sphere", precision="mixed",
              name="sphere192_w_mixed"),
        # laminar Navier-Stokes past a cylinder (Roe MUSCL and viscous fluxes), four
        # embedded levels of 512x512x2 cells, V-cycle, in FP64 ...
        _case("cycles", "embedded", 512, 512, 2, 4, scheme="roe_ns", mgtype=1, cycles=2, name="ns512_v"),
        # ... and on a smaller grid in the mixed form
        _case("cycles", "embedded", 256, 256, 2, 4, scheme="roe_ns", mgtype=1, cycles=3, precision="mixed",
              name="ns256_v_mixed"),
        # the batched sweep: ellipsoids on grids of several sizes, mixed form, in lockstep
        _case("group", "box", 64, 64, 64, 3, cycles=3, precision="mixed", members=8, extent=3.0,
              name="group8_mixed"),
        # the cylinder in physical time: one dual-time step's inner cycles
        _case("cycles", "slab", 128, 128, 2, 3, mgtype=1, cycles=6, extent=8.0, unsteady=True, name="slab128_unsteady"),
        # a whole solve from the free stream: full multigrid, then cycles on the finest level
        _case("solve", "box", 64, 64, 64, 3, cycles=6, name="solve_box64"),
    ]


def draw(rng):
    """One more case of the same kinds; sizes spread over the logarithm of their range."""
    def size(lo, hi, mult=1):
        return max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / mult)) * mult)

    def wide(nx, ny, nz, lo, hi):
        """Half the length along x, with room for the body across the shortest axis."""
        return max(rng.uniform(lo, hi), 1.4 * nx / min(ny, nz))

    def coarsest(lv, n, extent):
        """As many of lv levels as leave a cell of the coarsest no larger than the body."""
        while lv > 2 and 2.0 * extent / n * (1 << (lv - 1)) > 1.0:
            lv -= 1
        return lv

    kind = rng.choice(["update", "slab", "box", "box", "box_mixed", "ns", "ns_mixed", "group", "unsteady", "solve"])
    if kind == "update":
        nx, ny, nz = size(17, 150), size(17, 150), size(9, 110)
        return _case("update", "box", nx, ny, nz, 1, cycles=rng.randint(1, 4), extent=wide(nx, ny, nz, 3.0, 6.0),
                     body=rng.choice(["sphere", "ellipsoid"]))
    if kind in ("slab", "unsteady"):
        nx, ny, extent = size(48, 320, 4), size(48, 320, 4), rng.uniform(6.0, 20.0)
        return _case("cycles", "slab", nx, ny, rng.choice([2, 3, 4]), coarsest(3, nx, extent), mgtype=1,
                     cycles=rng.randint(2, 8), extent=extent, unsteady=kind == "unsteady")
    if kind in ("box", "box_mixed", "solve"):
        nx, ny, nz = size(32, 160, 8), size(32, 160, 8), size(24, 128, 8)
        extent = wide(nx, ny, nz, 3.0, 8.0)
        return _case("solve" if kind == "solve" else "cycles", "box", nx, ny, nz,
                     coarsest(rng.choice([2, 3, 4]), nx, extent), mgtype=rng.choice([1, 2]),
                     cycles=rng.randint(1, 4), extent=extent, precision="mixed" if kind == "box_mixed" else "fp64")
    if kind == "group":
        return _case("group", "box", size(32, 88, 4), 0, 0, 3, cycles=rng.randint(1, 3), precision="mixed",
                     members=rng.randint(3, 10), extent=rng.uniform(2.5, 3.5))
    return _case("cycles", "embedded", size(96, 384, 4), size(96, 384, 4), 2, rng.choice([2, 3, 4]), scheme="roe_ns",
                 mgtype=1, cycles=rng.randint(1, 3), precision="mixed" if kind == "ns_mixed" else "fp64")


def _flow(case, seed, member):
    """What the seed decides: the free stream, the body and the start state's waves."""
    r = random.Random(1000003 * int(seed) + member)
    f = {"mach": 0.2 if case["scheme"] == "roe_ns" else (0.3 if case["grid"] == "slab" else r.uniform(0.3, 0.6)),
         "alpha": 0.0 if case["grid"] != "box" else r.uniform(-2.0, 5.0), "semi": None}
    if case["body"] == "ellipsoid":
        f["semi"] = tuple(r.uniform(0.5, 1.0) for _ in range(3))
    f["waves"] = [[(r.uniform(0.2, 1.5), r.uniform(0.2, 1.5), r.uniform(0.2, 1.5), r.uniform(0, 2 * math.pi))
                   for _ in range(2)] for _ in range(5)]
    return f


def _sizes(case, member):
    """The grid of one member; a group's grids run from half to one and a half times its size."""
    if case["kind"] != "group":
        return case["nx"], case["ny"], case["nz"]
    m = max(1, case["members"] - 1)
    n = max(16, int(round(case["nx"] * (0.5 + member / m) / 4)) * 4)
    return n, n, n


def _build(case, seed, member=0):
    """The case's blocks, cut-cell records and solver parameters."""
    f = _flow(case, seed, member)
    nx, ny, nz = _sizes(case, member)
    nl = case["levels"]
    if case["grid"] == "embedded":
        body = K.Body("cylinder", radius=0.5)
        h = 512.0 / 96.0 / case["nx"]  # D/96 on 512 cells
        levels = K.embedded_hierarchy(body, (0.0, 0.0, 0.0), (h, h, h), (nx, ny, nz), nl)
        area = nz * h
    elif case["grid"] == "slab":
        body = K.Body("cylinder", radius=0.5)
        h = 2.0 * case["extent"] / nx
        hi = (case["extent"], 0.5 * ny * h, 0.5 * nz * h)
        levels = K.same_domain_hierarchy(body, tuple(-v for v in hi), hi, (nx, ny, nz), nl,
                                         coarsen=(True, True, False), bctype=(-20, -20, -60, -20, -20, -60))
        area = nz * h
    else:
        off = (0.03, 0.02, 0.01)  # off the cell centres of every level
        body = K.Body("ellipsoid", center=off, semi=f["semi"]) if f["semi"] else K.Body("sphere", center=off, radius=0.5)
        h = 2.0 * case["extent"] / nx
        hi = (case["extent"], 0.5 * ny * h, 0.5 * nz * h)
        levels = K.same_domain_hierarchy(body, tuple(-v for v in hi), hi, (nx, ny, nz), nl)
        area = math.pi * 0.25
    kw = {}
    if case["scheme"] == "roe_ns":
        kw.update(eqntype=A.MGE_EQN_NS, distype=A.MGE_DIS_ROE2, reynolds=40.0)
    if case["unsteady"]:
        kw.update(execmode=1, dtstep=0.2)
    mcyc = [2] * (nl - 1) + [case["cycles"]]
    prm = K.params(f["mach"], alpha_deg=f["alpha"], nlevel=nl, mcyc=mcyc, mgtype=case["mgtype"], conv_drop=1e30,
                   precision=A.MGE_PREC_MIXED if case["precision"] == "mixed" else A.MGE_PREC_FP64, **kw)
    return K.Case("perf", prm, levels, body, ref_area=area), f


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _start(kc, f, dev):
    """The finest level's start state w (5, k, j, i), ghosts included: the potential flow
    past the body, isentropic, with waves of one per cent on every variable."""
    sp, P = kc.levels[-1][0], kc.prm
    x, y, z = (sp.origin[d] + (torch.arange(sp.n[d] + 4, dtype=torch.float64, device=dev) - 1.5) * sp.h[d]
               for d in range(3))
    x, y, z = x[None, None, :], y[None, :, None], z[:, None, None]
    U = (P.u0, P.v0, P.w0)
    flat = kc.body.kind == "cylinder"
    r2 = x * x + y * y + (0.0 if flat else z * z)
    R2 = 0.25
    r2 = torch.clamp(r2, min=R2)
    dot = U[0] * x + U[1] * y + (0.0 if flat else U[2] * z)
    g = R2 / r2 if flat else 0.5 * (R2 / r2) ** 1.5
    m = 2.0 if flat else 3.0
    u = [U[d] + g * (U[d] - m * dot * (x, y, z)[d] / r2) for d in range(3)]
    if flat:
        u[2] = torch.full_like(u[0], U[2])
    size = max(sp.n[d] * sp.h[d] for d in range(3))
    wave = []
    for v in range(5):
        s = 0.0
        for a, b, c, ph in f["waves"][v]:
            kz = 0.0 if flat else c
            s = s + torch.sin(2.0 * math.pi / size * (4.0 * a * x + 4.0 * b * y + 4.0 * kz * z) + ph)
        wave.append(0.005 * s)
    un = math.sqrt(sum(q * q for q in U))
    for d in range(3):
        u[d] = (u[d] + un * wave[1 + d]).expand(r2.shape[0] if not flat else sp.n[2] + 4, sp.n[1] + 4, sp.n[0] + 4)
    q2 = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
    T = 1.0 + 0.5 * (GAMMA - 1.0) * P.rm ** 2 * (1.0 - q2 / un ** 2)
    rho = P.rho0 * T ** (1.0 / (GAMMA - 1.0)) * (1.0 + wave[0])
    p = P.p0 * T ** (GAMMA / (GAMMA - 1.0)) * (1.0 + wave[4])
    return torch.stack([rho, rho * u[0], rho * u[1], rho * u[2], p / (GAMMA - 1.0) + 0.5 * rho * q2]).contiguous()


# ----------------------------------------------------------------- the library's side
def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())


def _ptr(t):
    return C.cast(C.c_void_p(t.data_ptr()), C.POINTER(C.c_double))


def prepare(case, seed):
    """Resident cases, their start states and result buffers in pinned host memory."""
    lib = load_library()
    members = []
    for q in range(case["members"]):
        kc, f = _build(case, seed, q)
        # the mixed form's FP32 sweeps round by their launch form: a fixed plan
        # gives every run of a case the same bits
        plan = os.environ.get("MGE_TUNE_PLAN")
        if case["precision"] == "mixed" and case["kind"] != "group":
            os.environ["MGE_TUNE_PLAN"] = ",".join("%d:0200" % (L + 1) for L in range(case["levels"]))
        try:
            cyc = Cycle(kc)
        finally:
            if plan is None:
                os.environ.pop("MGE_TUNE_PLAN", None)
            else:
                os.environ["MGE_TUNE_PLAN"] = plan
        w0 = _start(kc, f, _device())
        start, w, p = _pinned(w0.shape), _pinned(w0.shape), _pinned(w0.shape[1:])
        start.copy_(w0)
        members.append({"cycle": cyc, "start": start, "start_np": start.numpy(), "w": w, "p": p})
    if case["unsteady"]:  # one physical step in, so that the transient source is on
        members[0]["cycle"].time_advance()
    st = {"lib": lib, "case": dict(case), "members": members}
    if case["kind"] == "group":
        n = len(members)
        st["ctxs"] = (C.c_void_p * n)(*[m["cycle"].ctx.value for m in members])
        st["res"], st["rcs"] = (C.c_double * n)(), (C.c_int * n)()
    return st


def run(state):
    """One pass; the state's buffers hold the new state (w, p) of every member."""
    case, lib, members = state["case"], state["lib"], state["members"]
    L, kind, out = case["levels"], case["kind"], {}
    if kind == "solve":
        cyc = members[0]["cycle"]
        cyc.init_flow()
        hist, _, fo = cyc.solve()
        out = {"residual": hist, "force": list(fo.force), "cd": fo.cd, "cl": fo.cl}
    else:
        for m in members:
            m["cycle"].upload(m["start_np"], L)
    if kind == "update":
        cyc = members[0]["cycle"]
        out["residual"] = []
        for n in range(1, case["cycles"] + 1):
            cyc.timestep(L)
            cyc.euler(L, ncyc=n)
            out["residual"].append(cyc.rtrms(L, n))
    elif kind == "cycles":
        cyc = members[0]["cycle"]
        out["residual"] = [cyc.cycle(L) for _ in range(case["cycles"])]
    elif kind == "group":
        n, out["residual"] = len(members), []
        for _ in range(case["cycles"]):
            rc = lib.mge_group_cycle_async(state["ctxs"], n, L)
            if rc != 0:
                raise RuntimeError("group cycle: %s" % A.error_name(rc))
            while lib.mge_group_cycle_poll(state["ctxs"], n, -1, state["res"], state["rcs"]) == 1:
                pass
            out["residual"].append(list(state["res"]))
    for m in members:
        rc = lib.mge_download_state(m["cycle"].ctx, L, 1, _ptr(m["w"]), _ptr(m["p"]))
        if rc != 0:
            raise RuntimeError("download: %s" % A.error_name(rc))
    out["w"] = [m["w"] for m in members]
    out["p"] = [m["p"] for m in members]
    return out


def _level_cells(case, member):
    nx, ny, nz = _sizes(case, member)
    out = []
    for L in range(case["levels"]):
        f = 1 << (case["levels"] - 1 - L)
        if case["grid"] == "embedded":
            out.append(nx * ny * nz)
        else:
            out.append((nx // f) * (ny // f) * (nz if case["grid"] == "slab" else nz // f))
    return out


def _updates(levels, top, mgtype):
    """Updates and residual evaluations per level of one cycle at FMG level `top` (1-based)."""
    up, res, icyc = [0] * (levels + 1), [0] * (levels + 1), [0] * (levels + 2)
    mgl = top
    while True:
        while True:
            icyc[mgl] += 1
            up[mgl] += 1
            if top == 1:
                return up, res
            res[mgl] += 1
            mgl -= 1
            if mgl == 1:
                break
        while True:
            up[mgl] += 1
            mgl += 1
            if mgl == top:
                return up, res
            if icyc[mgl] != mgtype:
                break
            icyc[mgl] = 0


def work(case):
    """The state in and out once, and about 1,800 operations for a cell's update (half of
    them again for the Roe and viscous fluxes) with a fifth of that for a residual alone."""
    per = 2700.0 if case["scheme"] == "roe_ns" else 1800.0
    nbytes = flops = 0.0
    for q in range(case["members"]):
        cells = _level_cells(case, q)
        tops = [(case["levels"], case["cycles"])]
        if case["kind"] == "solve":
            tops += [(L, 2) for L in range(1, case["levels"])]
        for top, count in tops:
            up, res = _updates(case["levels"], top, case["mgtype"]) if case["kind"] != "update" else ([0, 1], [0, 0])
            flops += count * per * sum((up[L + 1] + 0.2 * res[L + 1]) * cells[L] for L in range(case["levels"]))
        nx, ny, nz = _sizes(case, q)
        nbytes += (5 + 6) * 8.0 * (nx + 4) * (ny + 4) * (nz + 4)
    return {"bytes": nbytes, "flops": flops}


# ----------------------------------------------------------------- the same in plain torch, float64
class _Block:
    """One block: fields shaped (variable, k, j, i) with two ghost layers on every face."""

    def __init__(self, sp, dev):
        self.n, self.h = sp.n, sp.h
        self.dims = (sp.n[2] + 4, sp.n[1] + 4, sp.n[0] + 4)
        self.bc, self.ratio, self.offset = sp.bctype, sp.ratio, sp.offset
        self.s = [-(sp.h[1] * sp.h[2]), -(sp.h[0] * sp.h[2]), -(sp.h[0] * sp.h[1])]
        self.vol = sp.h[0] * sp.h[1] * sp.h[2]
        a = sp.arrays
        self.fluid = torch.as_tensor(a["blank"].reshape(self.dims) != 0, device=dev)
        z = lambda *s: torch.zeros(s + self.dims, dtype=torch.float64, device=dev)  # noqa: E731
        self.w, self.wn, self.ws, self.dw, self.fw, self.wr, self.qf = (z(5) for _ in range(7))
        self.p, self.vd, self.lam = z(), z(), z()
        self.marker = torch.zeros(self.dims, dtype=torch.bool, device=dev)
        self.st = (1, self.dims[2], self.dims[2] * self.dims[1])
        self.nm = int(a["nmir"])
        self.w1 = self.w2 = None
        if self.nm:
            t = lambda v, dt=torch.float64: torch.as_tensor(np.array(v), dtype=dt, device=dev)  # noqa: E731
            cc = t(a["ccid"], torch.int64)
            self.ax = t(a["zz"], torch.int64) - 1
            self.plus = t(a["faceid"], torch.int64) >= 4
            self.rc = cc[:, 0] + self.st[1] * cc[:, 1] + self.st[2] * cc[:, 2]
            self.rs = torch.tensor(self.st, device=dev)[self.ax]
            self.pos = cc.gather(1, self.ax[:, None])[:, 0]
            self.lq = torch.tensor([sp.n[d] + 1 for d in range(3)], device=dev)[self.ax]
            nb = self.pos + torch.where(self.plus, -1, 1)
            self.nb_in = (nb >= 2) & (nb <= self.lq)
            ij = t(a["ijkdex"], torch.int64)
            self.cloud = ij[..., 0] + self.st[1] * ij[..., 1] + self.st[2] * ij[..., 2]
            use = torch.arange(ij.shape[1], device=dev)[None, :] < t(a["npoint"], torch.int64)[:, None]
            self.coef = torch.where(use, t(a["coef"]), torch.zeros((), dtype=torch.float64, device=dev))
            self.cloud = torch.where(use, self.cloud, self.rc[:, None])
            nv = t(a["nvec"])
            self.nv = nv / nv.square().sum(1, keepdim=True).sqrt()
            self.qb, self.area = t(a["qb"]), t(a["area"])
            self.rsf = torch.tensor(self.s, dtype=torch.float64, device=dev)[self.ax]
            self.rh = torch.tensor(self.h, dtype=torch.float64, device=dev)[self.ax]
            self.wsol = torch.zeros((5, self.nm), dtype=torch.float64, device=dev)
            self.psol = torch.zeros(self.nm, dtype=torch.float64, device=dev)

    def phys(self, f):
        return f[..., 2:-2, 2:-2, 2:-2]


def _along(f, d, lo, hi):
    """f restricted to indices lo..hi of direction d (0 = i) and physical elsewhere."""
    sl = [slice(2, -2)] * 3
    sl[2 - d] = slice(lo, hi + 1)
    return f[(Ellipsis,) + tuple(sl)]


def _albada(a, b, e2):
    return ((b * b + e2) * a + (a * a + e2) * b) / (a * a + b * b + 2.0 * e2)


class _Solver:
    """The multigrid Runge-Kutta cycle of one case in float64."""

    def __init__(self, kc, dev):
        self.P, self.kc = kc.prm, kc
        P = kc.prm
        self.roe, self.ns, self.unsteady = P.distype == A.MGE_DIS_ROE2, P.eqntype == A.MGE_EQN_NS, P.execmode == 1
        self.lv = [_Block(L[0], dev) for L in kc.levels]
        self.itime = 0
        for b in self.lv:
            U = (P.u0, P.v0, P.w0)
            b.w[0] = P.rho0
            for d in range(3):
                b.w[1 + d] = P.rho0 * U[d]
            b.w[4] = P.rho0 * P.h0 - P.p0
            self.settle(b)
            if self.unsteady:
                b.w1, b.w2 = b.w.clone(), b.w.clone()

    def depvars(self, w):
        q = 0.5 * (w[1] * w[1] + w[2] * w[2] + w[3] * w[3]) / w[0]
        return (self.P.gamma - 1.0) * torch.clamp(w[4] - q, min=0.0)

    def settle(self, b):
        b.p = self.depvars(b.w)
        self.cutcell(b)
        self.bcond(b)

    # ---- time step
    def timestep(self, b):
        P, c = self.P, b.phys
        w, p = c(b.w), c(b.p)
        cc = torch.sqrt(torch.clamp(P.gamma * p / w[0], min=0.0))
        lsum = sum(torch.abs(w[1 + d] / w[0] * b.s[d]) + cc * abs(b.s[d]) for d in range(3))
        if self.ns:
            cfac = 1.0 if self.roe else 4.0
            fac = torch.maximum(4.0 / w[0] / 3.0, P.gamma / w[0]) * (P.viscl / P.prlmean) / b.vol
            fict = b.vol / (lsum + cfac * fac * sum(s * s for s in b.s))
        else:
            fict = b.vol / lsum
        dp = 0.0
        for d in range(3):
            n = b.n[d] + 1
            lo, hi = _along(b.p, d, 1, n - 1), _along(b.p, d, 3, n + 1)
            dp = dp + torch.abs((hi - 2.0 * p + lo) / (hi + 2.0 * p + lo + 0.001))
        r = 1.0 / (1.0 + torch.clamp(2.0 * dp, max=max(P.cfl - 1.0, 0.0)))
        if self.unsteady:
            fict = torch.clamp(fict, max=2.0 * P.dtstep / (3.0 * P.cfl))
        zero = torch.zeros_like(fict)
        c(b.vd).copy_(torch.where(c(b.fluid), fict * r, zero))
        c(b.lam).copy_(torch.where(c(b.fluid), lsum, zero))

    def flux(self, w, p, d, s):
        f0 = w[1 + d] * s
        f = [f0, f0 * w[1] / w[0], f0 * w[2] / w[0], f0 * w[3] / w[0], f0 * (w[4] + p) / w[0]]
        f[1 + d] = f[1 + d] + p * s
        return torch.stack(f)

    def roe_diss(self, d, S, wl, pl, wr, pr):
        P = self.P
        ul, ur = wl[1:4] / wl[0], wr[1:4] / wr[0]
        hl, hr = (wl[4] + pl) / wl[0], (wr[4] + pr) / wr[0]
        rt = torch.sqrt(wr[0] / wl[0])
        rh = rt * wl[0]
        uh, hh = (ul + rt * ur) / (1.0 + rt), (hl + rt * hr) / (1.0 + rt)
        q2 = (uh * uh).sum(0)
        c2 = (P.gamma - 1.0) * (hh - 0.5 * q2)
        ch = torch.sqrt(torch.clamp(c2, min=1e-300))
        if isinstance(d, int):
            on = torch.zeros(3, dtype=torch.float64, device=wl.device)
            on[d] = 1.0
            on = on.reshape((3,) + (1,) * (wl.dim() - 1))
        else:  # one axis per record
            on = torch.nn.functional.one_hot(d, 3).T.to(torch.float64)
        un, du = (uh * on).sum(0), ur - ul
        dun = (du * on).sum(0)
        dr, dp = wr[0] - wl[0], pr - pl
        delta = P.epsentr * (torch.abs(un) + ch)

        def fix(lam):
            a = torch.abs(lam)
            return torch.where((a < delta) & (delta > 0.0), (lam * lam + delta * delta) / (2.0 * delta), a)

        l1, l2, l5 = fix(un - ch), fix(un), fix(un + ch)
        a1 = l1 * (dp - rh * ch * dun) / (2.0 * c2)
        a2 = dr - dp / c2
        a5 = l5 * (dp + rh * ch * dun) / (2.0 * c2)
        sh = rh * (du - on * dun)
        mom = a1 * (uh - on * ch) + l2 * (a2 * uh + sh) + a5 * (uh + on * ch)
        en = a1 * (hh - ch * un) + l2 * (a2 * 0.5 * q2 + (uh * sh).sum(0)) + a5 * (hh + ch * un)
        return 0.5 * S * torch.cat([(a1 + l2 * a2 + a5)[None], mom, en[None]])

    # ---- the faces q = 2..n+2 of direction d: convective, dissipative and viscous fluxes
    def faces(self, b, d, dissip, cd):
        P, n, s = self.P, b.n[d], b.s[d]
        lo, hi = 1, n + 2
        at = lambda f, a: _along(f, d, 2 + a, n + 2 + a)  # noqa: E731  (cells q+a of faces q = 2..n+2)
        E = D = V = None
        if self.roe:
            wl, wr, pl, pr = at(b.w, -1), at(b.w, 0), at(b.p, -1), at(b.p, 0)
            prim = torch.cat([b.w[:1], b.w[1:4] / b.w[0], b.p[None]])
            u0n = math.sqrt(P.u0 ** 2 + P.v0 ** 2 + P.w0 ** 2)
            e2 = torch.tensor([1e-6 * r * r / P.limfac for r in (P.rho0, u0n, u0n, u0n, P.p0)], dtype=torch.float64,
                              device=b.w.device).reshape(5, 1, 1, 1)
            q = [at(prim, a) for a in (-2, -1, 0, 1)]
            L = q[1] + 0.5 * _albada(q[1] - q[0], q[2] - q[1], e2)
            R = q[2] - 0.5 * _albada(q[2] - q[1], q[3] - q[2], e2)
            ok = at(b.fluid, -2) & at(b.fluid, -1) & at(b.fluid, 0) & at(b.fluid, 1)
            ok = ok & (L[0] > 0) & (R[0] > 0) & (L[4] > 0) & (R[4] > 0)

            def cons(X):
                return torch.cat([X[:1], X[0] * X[1:4],
                                  (X[4] / (P.gamma - 1.0) + 0.5 * X[0] * (X[1:4] ** 2).sum(0))[None]])

            wl, wr = torch.where(ok, cons(L), wl), torch.where(ok, cons(R), wr)
            pl, pr = torch.where(ok, L[4], pl), torch.where(ok, R[4], pr)
            E = 0.5 * (self.flux(wr, pr, d, s) + self.flux(wl, pl, d, s))
            if dissip:
                D = cd * self.roe_diss(d, abs(s), wl, pl, wr, pr)
        else:
            F = self.flux(_along(b.w, d, lo, hi), _along(b.p, d, lo, hi), d, s)
            ax = 3 - d
            E = 0.5 * (F.narrow(ax, 1, n + 1) + F.narrow(ax, 0, n + 1))
            if dissip:
                pc, pm, pp = _along(b.p, d, 1, n + 2), _along(b.p, d, 0, n + 1), _along(b.p, d, 2, n + 3)
                bot = torch.abs(pm + 2.0 * pc + pp)
                fp = torch.where(bot > 0.0, torch.abs(pm - 2.0 * pc + pp) / bot, torch.zeros_like(bot))
                pad = [0, 0] * (d) + [1, 1]
                fp = torch.nn.functional.pad(fp, pad)      # zero at indices 0 and n+3
                cut = lambda a: fp.narrow(2 - d, 2 + a, n + 1)  # noqa: E731
                ep = torch.maximum(torch.maximum(cut(-2), cut(-1)), torch.maximum(cut(0), cut(1)))
                lam = _along(b.lam, d, 2, n + 1)
                first, last = lam.narrow(2 - d, 0, 1), lam.narrow(2 - d, n - 1, 1)
                lam = torch.cat([first, lam, last], 2 - d)
                lam = 0.5 * (lam.narrow(2 - d, 0, n + 1) + lam.narrow(2 - d, 1, n + 1))
                d2 = P.vis2 * ep
                d4 = torch.clamp(P.vis4 - d2, min=0.0)
                W = torch.cat([b.w[:4], (b.w[4] + b.p)[None]])
                df = at(W, 0) - at(W, -1)
                dm = torch.cat([df.narrow(ax, 0, 1), df.narrow(ax, 0, n)], ax)
                dn = torch.cat([df.narrow(ax, 1, n), df.narrow(ax, n, 1)], ax)
                D = (cd * d2 * df - cd * d4 * (dn - 2.0 * df + dm)) * lam
        if self.ns and dissip:
            V = cd * self.viscous(b, d)
        return E, D, V

    def viscous(self, b, d):
        P, n = self.P, b.n[d]
        zero = torch.zeros((), dtype=torch.float64, device=b.w.device)
        vt = torch.cat([b.w[1:4] / b.w[0], (b.p / (b.w[0] * P.gas_const))[None]])
        vt = torch.where(b.fluid, vt, zero)

        def at(a, t=None, e=0):  # cells q+a, moved by e along the tangential direction t
            sl = [slice(2, -2)] * 3
            sl[2 - d] = slice(2 + a, n + 3 + a)
            if t is not None:
                sl[2 - t] = slice(2 + e, b.n[t] + 2 + e)
            return vt[(slice(None),) + tuple(sl)]

        g = []
        for t in range(3):
            if t == d:
                g.append((at(0) - at(-1)) / b.h[t])
            else:
                g.append(((at(0, t, 1) - at(0, t, -1)) + (at(-1, t, 1) - at(-1, t, -1))) / (4.0 * b.h[t]))
        S, mu = abs(b.s[d]), P.viscl
        kt = P.viscl * P.gamma * P.gas_const / ((P.gamma - 1.0) * P.prlmean)
        div = g[0][0] + g[1][1] + g[2][2]
        tau = [mu * (g[d][a] + g[a][d]) - ((2.0 / 3.0) * mu * div if a == d else 0.0) for a in range(3)]
        uf = 0.5 * (at(-1) + at(0))
        heat = uf[0] * tau[0] + uf[1] * tau[1] + uf[2] * tau[2] + kt * g[d][3]
        return S * torch.stack([torch.zeros_like(heat)] + tau + [heat])

    # ---- a stage: dw (convective + fw), fw blended; cut-cell walls replace the faces they cut
    def residual(self, b, m):
        P = self.P
        cd = P.cdis[m - 1]
        dissip = cd > 0.0
        dims = b.dims
        dw, fw = torch.zeros_like(b.w), torch.zeros_like(b.w)
        fw_old = b.fw * (1.0 - cd) if m > 1 else torch.zeros_like(b.w)
        full = {}
        for d in range(3):
            E, D, V = self.faces(b, d, dissip, cd)
            n, ax = b.n[d], 3 - d
            diff = lambda X: X.narrow(ax, 0, n) - X.narrow(ax, 1, n)  # noqa: E731
            b.phys(dw).add_(diff(E))
            if dissip:
                b.phys(fw).add_(diff(D))
                if V is not None:
                    b.phys(fw).add_(diff(V))
            if b.nm:
                for key, X in (("E", E), ("D", D), ("V", V)):
                    if X is None:
                        continue
                    f = torch.zeros((5,) + dims, dtype=torch.float64, device=b.w.device)
                    _along(f, d, 2, n + 2).copy_(X)
                    full.setdefault(key, []).append(f.reshape(5, -1))
        fw = fw + fw_old
        if b.nm:
            self.records(b, full, dissip, cd, dw.view(5, -1), fw.view(5, -1))
        b.phys(b.fw).copy_(b.phys(fw))
        return dw + fw

    def records(self, b, full, dissip, cd, dw, fw):
        P, c, st, plus, D = self.P, b.rc, b.rs, b.plus, b.ax
        w, p = b.w.reshape(5, -1), b.p.reshape(-1)
        sgn = torch.where(plus, 1.0, -1.0).to(torch.float64)

        every = torch.arange(b.nm, device=c.device)

        def pick(name, a):  # the face flux along each record's axis at cell c + a*st
            return torch.stack([X[:, c + a * st] for X in full[name]])[D, :, every].T

        def cef(x, px):
            f0 = x[1:4].gather(0, D[None])[0] * b.rsf
            f = torch.stack([f0, f0 * x[1] / x[0], f0 * x[2] / x[0], f0 * x[3] / x[0], f0 * (x[4] + px) / x[0]])
            return f.scatter_add(0, (1 + D)[None], (px * b.rsf)[None])

        wc, pc = w[:, c], p[c]
        cn = torch.where(plus, c - st, c + st)
        f1, f2, f3 = cef(wc, pc), cef(b.wsol, b.psol), cef(w[:, cn], p[cn])
        fs, fa = 0.5 * (f1 + f2), 0.5 * (f1 + f3)
        dw.index_add_(1, c, sgn * (fa - fs) - (pick("E", 0) - pick("E", 1)))
        if not dissip:
            return

        def wall_face(name):
            return torch.where(plus, pick(name, 1), pick(name, 0))

        if self.ns:
            u = wc[1:4] / wc[0]
            ug = 2.0 * b.qb.T - u
            gn = sgn * (ug - u) / b.rh
            tau = P.viscl * gn
            on = torch.nn.functional.one_hot(D, 3).T.to(torch.float64)
            tau = tau * (1.0 + on / 3.0)
            S = torch.abs(b.rsf)
            o = S * torch.cat([torch.zeros_like(tau[:1]), tau, (b.qb.T * tau).sum(0)[None]])
            fw.index_add_(1, c, sgn * wall_face("V") - sgn * cd * o)
        if self.roe:
            S = torch.abs(b.rsf)
            L = torch.where(plus, wc, b.wsol)
            R = torch.where(plus, b.wsol, wc)
            o = self.roe_diss(D, S, L, torch.where(plus, pc, b.psol), R, torch.where(plus, b.psol, pc))
            fw.index_add_(1, c, sgn * wall_face("D") - sgn * cd * o)
            return
        # scalar dissipation next to the wall; e points into the fluid
        e = torch.where(plus, -1, 1) * st
        W = torch.cat([w[:4], (w[4] + p)[None]])
        ws = torch.cat([b.wsol[:4], (b.wsol[4] + b.psol)[None]])
        lamf = b.lam.reshape(-1)
        estep = torch.where(plus, -1, 1)

        def lam(a):
            q = b.pos + a * estep
            qq = torch.minimum(torch.clamp(q, min=2), b.lq)
            return lamf[c + (qq - b.pos) * st]

        def sensor(x, y, z):
            return torch.abs(x - 2.0 * y + z) / torch.abs(x + 2.0 * y + z)

        p1, p2 = p[c + e], p[c + 2 * e]
        far = b.pos + 3 * estep
        inside = (far >= 0) & (far <= b.lq + 2)
        p3 = p[torch.where(inside, c + 3 * e, c)]
        s0, s1 = sensor(b.psol, pc, p1), sensor(pc, p1, p2)
        s2 = torch.where(inside, sensor(p1, p2, p3), torch.zeros_like(p1))

        def coefs(ep):
            d2 = P.vis2 * ep
            return cd * d2, cd * torch.clamp(P.vis4 - d2, min=0.0)

        # differences pointing away from the wall, then with the axis' sign
        d0, d1, d2_ = W[:, c] - ws, W[:, c + e] - W[:, c], W[:, c + 2 * e] - W[:, c + e]
        a2, a4 = coefs(torch.maximum(s0, s1))
        wallf = (a2 * d0 - a4 * (d1 - 2.0 * d0 + d0)) * lam(0)
        a2, a4 = coefs(torch.maximum(torch.maximum(s0, s1), s2))
        nextf = (a2 * d1 - a4 * (d2_ - 2.0 * d1 + d0)) * (0.5 * (lam(0) + lam(1)))
        ax = -sgn  # +1 where the axis runs from the wall into the fluid
        wallf, nextf = ax * wallf, ax * nextf
        z0 = torch.where(plus, nextf - wallf, wallf - nextf)
        fw.index_add_(1, c, z0 - (pick("D", 0) - pick("D", 1)))
        nb = (c + e)[b.nb_in]
        dense = torch.where(plus, pick("D", 0), pick("D", 1))  # the face between the cut cell and its neighbour
        corr = torch.where(plus, dense - nextf, nextf - dense)
        fw.index_add_(1, nb, corr[:, b.nb_in])

    # ---- implicit residual smoothing along i, j, k; blanked cells keep their value
    def smooth(self, b):
        eps = self.P.smoo
        aa, bb = 1.0 + 2.0 * eps, -eps
        dw = b.phys(b.dw)
        fluid = b.phys(b.fluid)
        for d in range(3):
            n, ax = b.n[d], 3 - d
            e1, e2 = [aa], [bb / aa]
            for q in range(1, n):
                e1.append(aa - bb * e2[q - 1])
                e2.append(bb / e1[q])
            x = dw.movedim(ax, 0).contiguous()
            on = fluid.movedim(2 - d, 0).contiguous()[:, None]
            for q in range(n):
                new = (x[q] - bb * x[q - 1]) / e1[q] if q else x[q] / e1[q]
                x[q] = torch.where(on[q], new, x[q])
            for q in range(n - 2, -1, -1):
                x[q] = torch.where(on[q], x[q] - e2[q] * x[q + 1], x[q])
            dw.copy_(x.movedim(0, ax))

    def euler(self, b, mgl, top, lres, lfir, want):
        P, c = self.P, b.phys
        if lfir:
            b.ws = b.w.clone()
        c(b.wn).copy_(c(b.w))
        b.dw.zero_()
        b.fw.zero_()
        for m in range(1, P.mstage + 1):
            r = self.residual(b, m)
            if self.unsteady and self.itime >= 1:
                f = 0.5 * b.vol / P.dtstep
                r = r + f * (b.w - b.w1 if self.itime == 1 else (3.0 * b.w - 4.0 * b.w1) + b.w2)
            lam = 1.0
            if self.unsteady:
                lam = 1.0 + P.cstp[m - 1] * P.cfl * b.vd * 3.0 / 2.0 / P.dtstep
            if mgl < top:
                if lfir and m == 1:
                    b.qf = torch.where(b.marker, b.wr - r, torch.zeros_like(r))
                r = r + b.qf
                if self.unsteady:
                    r = r / lam
            r = torch.where(b.fluid, r, torch.zeros_like(r))
            if lres:
                c(b.dw).copy_(c(r))
                return None
            c(b.dw).copy_(c((P.cstp[m - 1] * P.cfl * b.vd / b.vol) * r))
            if m % 2 and P.smoo > 0.0:
                self.smooth(b)
            step = b.dw / lam if self.unsteady and mgl == top else b.dw
            c(b.w).copy_(c(b.wn) - c(step))
            c(b.p).copy_(self.depvars(c(b.w)))
            self.cutcell(b)
            self.bcond(b)
        if not want:
            return None
        rt = torch.where(c(b.fluid), c(b.dw)[0] / (P.cfl * c(b.vd)), torch.zeros_like(c(b.vd)))
        return float(torch.sqrt((rt * rt).sum() / rt.numel()))

    # ---- boundaries
    def cutcell(self, b):
        if not b.nm:
            return
        w, p = b.w.reshape(5, -1), b.p.reshape(-1)
        vr = (w[:, b.cloud] * b.coef).sum(-1)
        psol = (p[b.cloud] * b.coef).sum(-1)
        mom = vr[1:4]
        if self.ns:
            mom = 2.0 * b.qb.T * vr[0] - mom
        else:
            qn = 2.0 * (b.nv.T * (mom - vr[0] * b.qb.T)).sum(0)
            mom = mom - qn * b.nv.T
        en = psol / (self.P.gamma - 1.0) + 0.5 * (mom * mom).sum(0) / vr[0]
        b.wsol, b.psol = torch.cat([vr[:1], mom, en[None]]), psol

    def bcond(self, b):
        P, g = self.P, self.P.gamma
        gm = 1.0 / (g - 1.0)
        U = (P.u0, P.v0, P.w0)
        for face in range(6):
            kind, d, low = b.bc[face], face % 3, face < 3
            if kind == 0:
                continue
            l = b.n[d] + 1  # noqa: E741
            g1, g2, c1, c2 = (1, 0, 2, 3) if low else (l + 1, l + 2, l, l - 1)
            if kind == -60:
                c1, c2 = (l, l - 1) if low else (2, 3)
            w, p = b.w.movedim(3 - d, 1), b.p.movedim(2 - d, 0)
            wc, pc = w[:, c1].clone(), p[c1].clone()
            if kind == -60:
                w2, p2 = w[:, c2].clone(), p[c2].clone()
                w[:, g1], w[:, g2], p[g1], p[g2] = wc, w2, pc, p2
                continue
            if kind != -20:
                raise NotImplementedError("bctype %d" % kind)
            fn = -1.0 if low else 1.0
            vel = wc[1:4] / wc[0]
            vn = vel[d] * fn
            rmi = U[d] * fn - 2.0 * P.c0 * gm
            rpo = vn + 2.0 * torch.sqrt(g * pc / wc[0]) * gm
            ci = 0.25 * (g - 1.0) * (rpo - rmi)
            inflow = vn <= 0.0
            s = torch.where(inflow, torch.full_like(pc, P.rho0 ** g / P.p0), wc[0] ** g / pc)
            cc = ci * ci / g
            rho = (s * cc) ** gm
            pr = rho * cc
            vv = [torch.where(inflow, torch.full_like(pc, U[a]), vel[a]) for a in range(3)]
            vv[d] = 0.5 * (rpo + rmi) * fn
            new = torch.stack([rho, rho * vv[0], rho * vv[1], rho * vv[2],
                               pr * gm + 0.5 * rho * (vv[0] ** 2 + vv[1] ** 2 + vv[2] ** 2)])
            w[:, g1], w[:, g2], p[g1], p[g2] = new, new, pr, pr
        self.corners(b)

    def corners(self, b):
        w, p = b.w, b.p
        il, jl, kl = (b.n[d] + 1 for d in range(3))
        ie, je, ke = il + 1, jl + 1, kl + 1

        def put(dst, v):
            w[(slice(None),) + dst] = v
            p[dst] = self.depvars(v)

        def at(k, j, i):
            return w[:, k, j, i]

        ks, js, every = slice(2, kl + 1), slice(2, jl + 1), slice(None)
        for i, ii in ((1, 2), (ie, il)):
            for j, jj in ((1, 2), (je, jl)):
                put((ks, j, i), at(ks, j, ii) + at(ks, jj, i) - at(ks, jj, ii))
        for i, ii in ((1, 2), (ie, il)):
            for k, kk in ((1, 2), (ke, kl)):
                put((k, js, i), at(k, js, ii) + at(kk, js, i) - at(kk, js, ii))
        old = w.clone()
        a = lambda k, j: old[:, k, j, every]  # noqa: E731
        put((1, 1, every), a(2, 1) + a(1, 2) - a(2, 2))
        put((ke, 1, every), a(ke, 2) + a(kl, 1) - a(kl, 2))
        # bc_corner.f90:120 as written: the cell keeps its value
        put((1, je, every), a(1, je) + a(2, jl) - a(2, jl))
        put((ke, je, every), a(ke, jl) + a(kl, je) - a(kl, jl))
        old = w.clone()
        for i, ii in ((1, 2), (ie, il)):
            for j, jj in ((1, 2), (je, jl)):
                for k, kk in ((1, 2), (ke, kl)):
                    q = old[:, k, j, ii] + old[:, k, jj, i] + old[:, kk, j, i]
                    put((k, j, i), q * 2.0 / 3.0 - old[:, kk, jj, ii])

    # ---- transfers
    def stencil(self, fine, coarse, d, idx):
        """Base index and weight in `coarse` of the fine cells idx along d; whether they lie inside it."""
        r, o, n = fine.ratio[d], fine.offset[d], coarse.n[d]
        u = o + (idx.to(torch.float64) - 1.5) / r
        s = torch.clamp(torch.floor(u + 1.5).to(torch.int64), 2, n)
        return s, u + 1.5 - s, (u >= 0.0) & (u < n)

    def interpolate(self, X, s, x):
        """X (v, k, j, i) at the tensor product of the stencils s, weights x (per direction)."""
        for d in range(3):
            ax = 3 - d
            shape = [1, 1, 1, 1]
            shape[ax] = -1
            t = x[d].reshape(shape)
            X = (1.0 - t) * X.index_select(ax, s[d]) + t * X.index_select(ax, s[d] + 1)
        return X

    def movco(self, L):
        c, f = self.lv[L], self.lv[L + 1]
        dev = c.w.device
        s, x, sl = [], [], []
        for d in range(3):
            m = f.n[d] // f.ratio[d]
            ic = torch.arange(m, device=dev) + f.offset[d] + 2
            t = (ic.to(torch.float64) - 1.5 - f.offset[d]) * f.ratio[d]
            q = torch.clamp(torch.floor(t + 1.5).to(torch.int64), 2, f.n[d])
            s.append(q)
            x.append(t + 1.5 - q)
            sl.append(slice(f.offset[d] + 2, f.offset[d] + 2 + m))
        at = (slice(None), sl[2], sl[1], sl[0])
        c.wr[at] = self.interpolate(f.dw / f.vol, s, x) * c.vol
        c.w[at] = self.interpolate(f.w, s, x)
        c.marker.zero_()
        c.marker[at[1:]] = True
        c.p = self.depvars(c.w)
        c.phys(c.wn).copy_(c.phys(c.w))
        self.bcond(c)

    def movfin(self, L, fmg):
        f, c = self.lv[L], self.lv[L - 1]
        dev = f.w.device
        s, x, inside = zip(*(self.stencil(f, c, d, torch.arange(f.n[d] + 4, device=dev)) for d in range(3)))
        ok = inside[2][:, None, None] & inside[1][None, :, None] & inside[0][None, None, :] & f.fluid
        phys = torch.zeros_like(ok)
        f.phys(phys).fill_(True)
        X = self.interpolate(c.w if fmg else c.w - c.ws, s, x)
        f.w = torch.where(ok & phys, X if fmg else f.w + X, f.w)
        f.p = self.depvars(f.w)
        X = self.interpolate(c.w, s, x)
        f.w = torch.where(ok & ~phys, X, f.w)
        f.p = self.depvars(f.w) if bool((ok & ~phys).any()) else f.p
        self.bcond(f)

    def cycle(self, top):
        P, res = self.P, None
        icyc = [0] * (len(self.lv) + 2)
        mgl = top
        while True:
            while True:
                icyc[mgl] += 1
                b = self.lv[mgl - 1]
                self.timestep(b)
                r = self.euler(b, mgl, top, False, mgl != top, mgl == top)
                res = r if mgl == top else res
                if top == 1:
                    return res
                self.euler(b, mgl, top, True, False, False)
                mgl -= 1
                self.movco(mgl - 1)
                if mgl == 1:
                    break
            lfir = True
            while True:
                b = self.lv[mgl - 1]
                self.timestep(b)
                self.euler(b, mgl, top, False, lfir, False)
                lfir = False
                mgl += 1
                self.movfin(mgl - 1, False)
                if mgl == top:
                    return res
                if icyc[mgl] != P.mgtype:
                    break
                icyc[mgl] = 0

    def forces(self):
        P, b = self.P, self.lv[-1]
        F = torch.zeros(3, dtype=torch.float64, device=b.w.device)
        if b.nm:
            pw = 0.5 * (b.p.reshape(-1)[b.rc] + b.psol) * b.area * torch.where(b.plus, 1.0, -1.0).to(torch.float64)
            F.index_add_(0, b.ax, pw)
        F = [float(v) for v in F]
        q = 0.5 * P.rho0 * (P.u0 ** 2 + P.v0 ** 2 + P.w0 ** 2) * self.kc.ref_area
        ca, sa, cb, sb = math.cos(P.alpha), math.sin(P.alpha), math.cos(P.beta), math.sin(P.beta)
        return F, (F[0] * ca * cb + F[1] * sa * cb + F[2] * sb) / q, (-F[0] * sa + F[1] * ca) / q


def exact(case, seed):
    """run()'s outputs in float64 by the restatement above."""
    dev = _device()
    out = {"residual": [], "w": [], "p": []}
    for q in range(case["members"]):
        kc, f = _build(case, seed, q)
        S = _Solver(kc, dev)
        b, L, res = S.lv[-1], case["levels"], []
        if case["unsteady"]:
            S.itime = 1
        if case["kind"] == "solve":
            for top in range(1, L + 1):
                hist = [S.cycle(top) for _ in range(kc.prm.mcyc[top - 1])]
                if top < L:
                    S.movfin(top, True)
            res = np.array(hist)
            F, cd, cl = S.forces()
            out.update(force=F, cd=cd, cl=cl)
        else:
            b.w = _start(kc, f, dev)
            S.settle(b)
            for _ in range(case["cycles"]):
                if case["kind"] == "update":
                    S.timestep(b)
                    res.append(S.euler(b, 1, 1, False, False, True))
                else:
                    res.append(S.cycle(L))
        out["residual"].append(res)
        out["w"].append(b.w)
        out["p"].append(b.p)
    if case["kind"] == "group":  # one list per cycle, as run() gives them
        out["residual"] = [list(r) for r in zip(*out["residual"])]
    else:
        out["residual"] = out["residual"][0]
    return out
