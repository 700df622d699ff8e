"""Timed workloads of the solver library: the calls a Heat3ds user makes, over the sizes this
repository is used at.

Every case is the reference's 3-die IC stack (h2_b200.model: Mode-3 boundary set, Z grid of 30
planes or its refinement) with a heat map of 4-16 hotspots per die (the batched workload's
distribution, h2_b200.batch) and conductivities perturbed by +-20 % per layer band (the adjoint's
parameters), all drawn from the seed.  A pass is one public call with what it needs around it:
theta restored to its start, the solve, theta copied to a pinned host array.

  residual   h2g_calcrk_noalloc on the caller's own device arrays (latency of a single call)
  solve      Solver.solve on a resident handle: PBiCGSTAB + RB-GS, or CG
  oneshot    h2_b200.PBiCGSTAB, the reference's call with its host arrays in and out
  transient  Solver.transient: steps of main()'s time loop
  sor        Solver.sor: a fixed number of solveSOR! passes
  batch      BatchSolver.solve: members of uneven size in one call
  adjoint    steady_gradient: forward and adjoint solve, two gradient fields
"""
import ctypes
import math

import numpy as np
import torch

import h2_b200
from h2_b200 import _lib, adjoint, batch, model

MAXITR = 20_000


def listed():
    return [
        # the residual norm a stepping loop checks between solves, on arrays it owns: one launch
        dict(name="residual_240", kind="residual", nx=240, ny=240, nz=30, steady=True),
        # the reference's own small test grid: a solve bound by latency and launches
        dict(name="solve_40", kind="solve", method="pbicgstab", precision="fp64", nx=40, ny=40, nz=30, tol=1e-8),
        # an odd, ragged plan (no multiple of the warp or the block in x or y)
        dict(name="solve_121x117", kind="solve", method="pbicgstab", precision="fp64", nx=121, ny=117, nz=30,
             tol=1e-8),
        # the headline: 240 x 240 x 30 to 1e-8
        dict(name="solve_240", kind="solve", method="pbicgstab", precision="fp64", nx=240, ny=240, nz=30, tol=1e-8),
        # the reference's published case as its user calls it: host arrays, epsilon = 1e-4
        dict(name="oneshot_240", kind="oneshot", nx=240, ny=240, nz=30, tol=1e-4),
        # the refined grid of the scaling study (13.8 M cells: vectors stream from memory)
        dict(name="solve_480x60", kind="solve", method="pbicgstab", precision="fp64", nx=480, ny=480, nz=60,
             tol=1e-4),
        # CG, the reference's other Krylov driver, on the stack with adiabatic faces
        dict(name="cg_240", kind="solve", method="cg", precision="fp64", nx=240, ny=240, nz=30, tol=1e-4),
        # the mixed-precision option: FP32 smoother inside FP64 Krylov
        dict(name="mixed_180", kind="solve", method="pbicgstab", precision="mixed", nx=180, ny=180, nz=30, tol=1e-8),
        # the time loop (a_p0 on the diagonal, b rebuilt per step)
        dict(name="transient_181x179", kind="transient", nx=181, ny=179, nz=30, dt=1e-4, nt=4, tol=1e-6),
        # solveSOR!, a fixed number of passes
        dict(name="sor_200", kind="sor", nx=200, ny=200, nz=30, omega=1.0, passes=200),
        # the batched workload: members of 120^2, 180^2 and 240^2 together
        dict(name="batch_6", kind="batch", members=6, lo=120, hi=240, nz=30, tol=1e-8),
        # a gradient step: forward solve, adjoint solve, two gradient fields to the host
        dict(name="adjoint_120", kind="adjoint", nx=120, ny=120, nz=30, tol=1e-8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["residual", "solve", "solve", "solve", "oneshot", "transient", "sor", "batch", "adjoint",
                       "refined"])
    nx = _log_int(rng, 40, 300)
    ny = nx if rng.random() < 0.4 else max(33, nx + rng.randint(-9, 9))
    tol = rng.choice([1e-4, 1e-6, 1e-8])
    if kind == "residual":
        return dict(kind=kind, nx=nx, ny=ny, nz=30, steady=rng.random() < 0.5)
    if kind == "solve":
        precision = rng.choice(["fp64", "fp64", "mixed"])
        method = rng.choice(["pbicgstab", "pbicgstab", "cg"])
        if precision == "mixed":
            nx, ny = min(nx, 180), min(ny, 180)
        return dict(kind=kind, method=method, precision=precision, nx=nx, ny=ny, nz=30,
                    tol=1e-4 if method == "cg" else tol)
    if kind == "refined":
        nx = _log_int(rng, 120, 400)
        return dict(kind="solve", method="pbicgstab", precision="fp64", nx=nx, ny=nx + rng.randint(-5, 5), nz=60,
                    tol=1e-4)
    if kind == "oneshot":
        return dict(kind=kind, nx=nx, ny=ny, nz=30, tol=tol)
    if kind == "transient":
        return dict(kind=kind, nx=nx, ny=ny, nz=30, dt=rng.choice([1e-4, 1e-3]), nt=rng.randint(2, 6), tol=1e-6)
    if kind == "sor":
        return dict(kind=kind, nx=nx, ny=ny, nz=30, omega=rng.choice([1.0, 1.5]), passes=rng.randint(50, 300))
    if kind == "batch":
        lo = rng.choice([40, 60, 120])
        return dict(kind=kind, members=rng.randint(3, 8), lo=lo, hi=min(240, 2 * lo), nz=30, tol=tol)
    return dict(kind=kind, nx=min(nx, 240), ny=min(ny, 240), nz=30, tol=1e-8)


# ---- inputs ------------------------------------------------------------------------------------

def _band_scale(seed, ZC):
    return adjoint.lam_scale(adjoint.draw_beta(seed), ZC)


def _model(case, seed, nx=None, member=None, pinned=False):
    """The stack with the seed's conductivities and heat map; b = -(hsrc V) (theta starts at the
    ambient temperature, so calRHS!'s convective terms vanish)."""
    nx = case["nx"] if nx is None else nx
    ny = case.get("ny", nx)
    nz = case["nz"]
    steady = case["kind"] != "transient" and case.get("steady", True)
    _, ZC, _ = model.zgrid(nz)
    m = model.build_mode3(nx, ny, nz, is_steady=steady, dt=case.get("dt", 1e-4),
                          symmetric=case.get("method") == "cg", lam_scale=_band_scale(seed, ZC), calrhs=False)
    mem = batch.draw_member(member or 0, 10_000 + 64 * seed)
    m.wk.hsrc[...] = batch.heat_map(mem, m.ID, m.ZC, m.dx, m.dy)
    m.wk.b[...] = -(m.wk.hsrc * (m.dx * m.dy) * m.dZ[None, None, :])
    if case["kind"] == "residual":
        # a field part of the way to its solution: hot near the top of the stack
        z = np.linspace(0.0, 1.0, m.shape[2])[None, None, :]
        rng = np.random.default_rng(seed)
        m.wk.theta[1:-1, 1:-1, 1:-1] += (30.0 * z + rng.uniform(0.0, 5.0, m.shape))[1:-1, 1:-1, 1:-1]
    if pinned:
        for n in ("theta", "b", "lam", "mask", "rho", "cp"):
            setattr(m.wk, n, _pinned(getattr(m.wk, n)))
    return m


def _pinned(a):
    out = torch.empty(a.size, dtype=torch.float64, pin_memory=True).numpy().reshape(a.shape, order="F")
    out[...] = a
    return out


def _solver(m, precision="fp64"):
    s = h2_b200.Solver(*m.shape, precision=precision)
    w = m.wk
    s.set_grid(m.ZC, m.dZ, m.dx, m.dy, m.dt, m.HC, m.is_steady)
    s.set_fields(w.lam, w.mask, None if m.is_steady else w.rho, None if m.is_steady else w.cp)
    s.set_rhs(w.b)
    s.set_theta(w.theta)
    s.set_hsrc(w.hsrc)
    s.snapshot()
    return s


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _prepare_batch(case, seed)
    m = _model(case, seed, pinned=kind == "oneshot")
    st = dict(case=case, shape=m.shape)
    if kind == "residual":
        w = m.wk
        dev = {n: torch.from_numpy(np.ascontiguousarray(getattr(w, n).ravel(order="F"))).cuda()
               for n in ("theta", "b", "lam", "mask", "rho", "cp")}
        dev["ZC"], dev["dZ"] = torch.from_numpy(m.ZC.copy()).cuda(), torch.from_numpy(m.dZ.copy()).cuda()
        st.update(dev=dev, r=torch.zeros_like(dev["theta"]), HC=np.ascontiguousarray(m.HC), m=m,
                  res=ctypes.c_double(0.0))
        torch.cuda.synchronize()
        return st
    if kind == "oneshot":
        st.update(m=m, theta0=m.wk.theta.copy(order="F"))
        return st
    st["solver"] = _solver(m, case.get("precision", "fp64"))
    st["out"] = _pinned(np.zeros(m.shape, order="F"))
    if kind == "transient":
        st["bcs"] = m.bcs
    if kind == "adjoint":
        st["weights"] = adjoint.silicon_weights(m.ID, m.dx, m.dy, m.dZ)
    return st


def _members(case, seed):
    """Sizes and heat maps of a batch: the three sizes lo, (lo + hi) / 2, hi in turn."""
    sizes = (case["lo"], (case["lo"] + case["hi"]) // 2, case["hi"])
    return [batch.draw_member(q, 10_000 + 64 * seed, sizes=(sizes[q % 3],)) for q in range(case["members"])]


def _prepare_batch(case, seed):
    bs = batch.BatchSolver(_members(case, seed))
    outs = [_pinned(np.zeros(s.shape, order="F")) for s in bs.solvers]
    return dict(case=case, batch=bs, outs=outs)


# ---- one pass ----------------------------------------------------------------------------------

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "residual":
        m, d = state["m"], state["dev"]
        ptr = {n: ctypes.c_void_p(t.data_ptr()) for n, t in d.items()}
        st = _lib.load().h2g_calcrk_noalloc(
            *m.shape, ptr["theta"], ptr["b"], ptr["lam"], ptr["mask"], ptr["rho"], ptr["cp"], ptr["ZC"], ptr["dZ"],
            m.dx, m.dy, m.dt, state["HC"].ctypes.data_as(ctypes.POINTER(ctypes.c_double)), int(m.is_steady),
            ctypes.c_void_p(state["r"].data_ptr()), ctypes.byref(state["res"]), None)
        _lib.check(st)
        return dict(r=state["r"], norm=state["res"].value)
    if kind == "oneshot":
        m, w = state["m"], state["m"].wk
        w.theta[...] = state["theta0"]
        conv, itr, res0 = h2_b200.PBiCGSTAB(w, (m.dx, m.dy), m.dt, m.ZC, m.dZ, m.HC, tol=case["tol"], maxItr=MAXITR,
                                            smoother="gs", par="gpu", is_steady=True)
        return dict(theta=w.theta, converged=conv, itr=itr, res0=res0)
    if kind == "batch":
        bs = state["batch"]
        bs.restore()
        _, res = bs.solve(tol=case["tol"], maxItr=MAXITR)
        for s, o in zip(bs.solvers, state["outs"]):
            s.get_theta(o)
        return dict(theta=state["outs"], itr=[r.itr for r in res], converged=[bool(r.isconverged) for r in res])
    s = state["solver"]
    s.snapshot(restore=True)
    if kind == "solve":
        _, res = s.solve(case["method"], tol=case["tol"], maxItr=MAXITR, smoother="gs")
        return dict(theta=s.get_theta(state["out"]), converged=bool(res.isconverged), itr=res.itr, res0=res.res0)
    if kind == "transient":
        _, res, stats = s.transient(state["bcs"], case["nt"], tol=case["tol"], maxItr=MAXITR)
        return dict(theta=s.get_theta(state["out"]), itr=res.itr, stats=stats[:, :3])
    if kind == "sor":
        s.sor(omega=case["omega"], tol=0.0, maxItr=case["passes"])
        return dict(theta=s.get_theta(state["out"]))
    J, gh, gl, fwd, adj = adjoint.steady_gradient(s, state["weights"], p=8.0, tol=case["tol"], maxItr=MAXITR)
    return dict(J=J, dJ_dhsrc=gh, dJ_dlnlam=gl, itr=[fwd.itr, adj.itr])


# ---- what a pass cannot do without -------------------------------------------------------------

def _iterations(nx, nz, tol):
    """Krylov iterations of the stack, about: proportional to the cells per side and to the digits
    asked for (319 at 240 x 240 x 30 to 1e-8)."""
    return max(10.0, 1.33 * nx * (nz / 30.0) ** 0.35 * (0.25 + 0.75 * math.log10(1.0 / tol) / 8.0))


# operations per cell: one Gauss-Seidel update (6 products, 5 sums, 2 differences, a division and
# the relaxation), CalcAX, and the vector updates and inner products of one iteration
_F_GS, _F_AX = 16, 13
_F_PBICG = 2 * (5 * _F_GS + _F_AX) + 6 + 2 + 2 + 4 + 6 + 4
_F_CG = 5 * _F_GS + _F_AX + 2 + 4 + 2 + 2 + 2


def work(case):
    """bytes: fields, right-hand side and start read once, the field written once (the Krylov
    vectors of a solve need not leave the chip, so they are not counted)."""
    kind, nz = case["kind"], case["nz"]
    if kind == "batch":
        tot = dict(bytes=0, flops=0)
        for m in _members(case, 0):
            n = m.nx * m.nx * nz
            tot["bytes"] += n * 8 * 3
            tot["flops"] += int(n * _F_PBICG * _iterations(m.nx, nz, case["tol"]))
        return tot
    n = case["nx"] * case["ny"] * nz
    if kind == "residual":  # theta, b, lambda, mask (rho, cp) read, r written
        return dict(bytes=n * 8 * (5 if case["steady"] else 7), flops=n * 80)
    it = _iterations(max(case["nx"], case["ny"]), nz, case.get("tol", 1e-8))
    if kind == "oneshot":  # six host arrays in, one out
        return dict(bytes=n * 8 * 7, flops=int(n * _F_PBICG * it))
    if kind == "solve":
        f = _F_PBICG * it if case["method"] == "pbicgstab" else _F_CG * 4.0 * it
        return dict(bytes=n * 8 * 3, flops=int(n * f))
    if kind == "transient":
        return dict(bytes=n * 8 * 3 * case["nt"], flops=int(n * _F_PBICG * 0.2 * it * case["nt"]))
    if kind == "sor":
        return dict(bytes=n * 8 * 3, flops=n * (_F_GS + 6) * case["passes"])
    return dict(bytes=n * 8 * 6, flops=int(n * (2 * _F_PBICG * it + 60)))


# ---- the same quantities in 64 bits by plain torch ---------------------------------------------

class _Plain:
    """The 7-point operator of the stack as torch arrays (z, y, x)."""

    def __init__(self, m):
        t = lambda a: torch.from_numpy(np.ascontiguousarray(np.asarray(a).transpose(2, 1, 0))).cuda()  # noqa: E731
        w = m.wk
        lam, mask = t(w.lam), t(w.mask)
        dz = torch.from_numpy(m.dZ.copy()).cuda()[1:-1].view(-1, 1, 1)
        zc = torch.from_numpy(m.ZC.copy()).cuda()
        zm, zp = (zc[1:-1] - zc[:-2]).view(-1, 1, 1), (zc[2:] - zc[1:-1]).view(-1, 1, 1)
        self.sl = [(slice(1, -1), slice(1, -1), slice(0, -2)), (slice(1, -1), slice(1, -1), slice(2, None)),
                   (slice(1, -1), slice(0, -2), slice(1, -1)), (slice(1, -1), slice(2, None), slice(1, -1)),
                   (slice(0, -2), slice(1, -1), slice(1, -1)), (slice(2, None), slice(1, -1), slice(1, -1))]
        self.inner = (slice(1, -1),) * 3
        l0, m0 = lam[self.inner], mask[self.inner]
        geo = [m.dy * dz / m.dx] * 2 + [m.dx * dz / m.dy] * 2 + [m.dx * m.dy / zm, m.dx * m.dy / zp]
        area = [m.dy * dz] * 2 + [m.dx * dz] * 2 + [torch.full_like(dz, m.dx * m.dy)] * 2
        self.c, self.cv, self.wf = [], [], []
        for f in range(6):
            lq, mq = lam[self.sl[f]], mask[self.sl[f]]
            self.c.append(2.0 * lq * l0 / (lq + l0) * (2.0 - torch.trunc((mq + m0) / 2.0)) * geo[f])
            self.cv.append(float(m.HC[f]) * area[f] * (1.0 - mq))
            self.wf.append(torch.where(mq == 0.0, torch.ones_like(lq), lq / (lq + l0)))
        self.vol = m.dx * m.dy * dz
        self.ap = 0.0
        if not m.is_steady:
            self.ap = (t(w.rho) * t(w.cp))[self.inner] * self.vol / m.dt
        self.dd = sum(self.c) + sum(self.cv) + self.ap
        self.h = [float(m.HC[f]) * area[f] for f in range(6)]
        self.theta, self.b, self.hsrc = t(w.theta), t(w.b), t(w.hsrc)
        self.t = t

    def nb(self, x):
        return sum(self.c[f] * x[self.sl[f]] for f in range(6))

    def residual(self, x, b):
        return b[self.inner] - (self.nb(x) - self.dd * x[self.inner])

    def solve(self, x, b, tol=1e-13, cap=30_000):
        """Jacobi-preconditioned CG on -A, restarted once on the recomputed residual."""
        x = x.clone()
        p = torch.zeros_like(x)
        for _ in range(2):
            r = -self.residual(x, b)
            n0 = float(r.norm())
            if n0 == 0.0:
                return x
            z = r / self.dd
            p[self.inner] = z
            rz = (r * z).sum()
            for k in range(cap):
                pi = p[self.inner]
                q = self.dd * pi - self.nb(p)
                alpha = rz / (pi * q).sum()
                x[self.inner] += alpha * pi
                r -= alpha * q
                if k % 50 == 49 and float(r.norm()) < tol * n0:
                    break
                z = r / self.dd
                new = (r * z).sum()
                p[self.inner] = z + (new / rz) * pi
                rz = new
        return x

    def host(self, x):
        return np.asfortranarray(x.cpu().numpy().transpose(2, 1, 0))


def _exact_theta(m, case):
    op = _Plain(m)
    return op.host(op.solve(op.theta, op.b))


def exact(case, seed):
    """The converged quantities (a direct evaluation for the residual and solveSOR!); iteration
    counts have no such value, and the largest grids would take too long."""
    kind = case["kind"]
    none = dict(converged=None, itr=None, res0=None)
    if kind == "batch":
        sizes = [m.nx for m in _members(case, seed)]
        if sum(s * s for s in sizes) * case["nz"] > 2_500_000:
            return None
        out = []
        for mem in _members(case, seed):
            m = model.build_mode3(mem.nx, mem.nx, case["nz"], calrhs=False)
            m.wk.hsrc[...] = batch.heat_map(mem, m.ID, m.ZC, m.dx, m.dy)
            m.wk.b[...] = -(m.wk.hsrc * (m.dx * m.dy) * m.dZ[None, None, :])
            out.append(_exact_theta(m, case))
        return dict(theta=out, itr=[None] * len(out), converged=[None] * len(out))
    if case["nx"] * case["ny"] * case["nz"] > 2_500_000:
        return None
    m = _model(case, seed)
    op = _Plain(m)
    if kind in ("solve", "oneshot"):
        return dict(theta=op.host(op.solve(op.theta, op.b)), **none)
    if kind == "residual":
        r = torch.zeros_like(op.theta)
        r[op.inner] = op.residual(op.theta, op.b)
        return dict(r=r.flatten(), norm=float(r.norm()))
    if kind == "transient":
        x, stats = op.theta, []
        # calRHS!: convective faces add -h A (ta - theta) on the minus sides, + on the plus sides
        n = [op.dd.shape[2], op.dd.shape[1], op.dd.shape[0]]
        for _ in range(case["nt"]):
            b = torch.zeros_like(x)
            xi = x[op.inner]
            rhs = torch.zeros_like(xi)
            for f in range(6):
                if m.bcs[f][0] != model.CONVECTION:
                    continue
                edge = [slice(None)] * 3
                ax = 2 - f // 2
                edge[ax] = slice(0, 1) if f % 2 == 0 else slice(n[f // 2] - 1, n[f // 2])
                edge = tuple(edge)
                h = op.h[f].expand(xi.shape[0], 1, 1)[edge[0]]
                term = h * (float(m.bcs[f][4]) - xi[edge])
                rhs[edge] += term if f % 2 else -term
            b[op.inner] = -(op.ap * xi + op.hsrc[op.inner] * op.vol + rhs)
            x = op.solve(x, b)
            xi = x[op.inner]
            stats.append([float(xi.min()), float(xi.max()), float(xi.norm())])
        return dict(theta=op.host(x), itr=None, stats=np.array(stats))
    if kind == "sor":
        x = op.theta.clone()
        shp = op.dd.shape
        k, j, i = torch.meshgrid(*[torch.arange(1, q + 1, device="cuda") for q in shp], indexing="ij")
        col = ((i + j + k) % 2) ^ 1
        bi = op.b[op.inner]
        for _ in range(case["passes"]):
            for c in (0, 1):
                xi = x[op.inner]
                new = xi + case["omega"] * ((op.nb(x) - bi) / op.dd - xi)
                x[op.inner] = torch.where(col == c, new, xi)
        return dict(theta=op.host(x))
    # adjoint: A theta = b, J = (sum w theta^8)^(1/8), A la = dJ/dtheta (zero guards)
    th = op.solve(op.theta, op.b)
    w = op.t(adjoint.silicon_weights(m.ID, m.dx, m.dy, m.dZ))
    J = float((w * th ** 8).sum() ** 0.125)
    g = w * th ** 7 * J ** -7
    la = op.solve(torch.zeros_like(th), g)
    gh, gl = torch.zeros_like(th), torch.zeros_like(th)
    gh[op.inner] = -op.vol * la[op.inner]
    tp, ap = th[op.inner], la[op.inner]
    gl[op.inner] = -sum(op.c[f] * op.wf[f] * (th[op.sl[f]] - tp) * (ap - la[op.sl[f]]) for f in range(6))
    return dict(J=J, dJ_dhsrc=op.host(gh), dJ_dlnlam=op.host(gl), itr=[None, None])
