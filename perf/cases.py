"""Performance cases of the framework: what its users run, through the public
entry points, over the range of grids and options they run it with.

A case is a dict of plain values; its "kind" is the way of use:

* ``unsteady``: BDF2 steps (Newton to convergence) of a developing flow
  through ``Solver``, with the state handed in and taken out through host
  buffers, and the force coefficients of every step, as a time loop with
  output does it.  Where factors are kept across steps, a pass takes several.
* ``steady``: a whole steady solve from the free stream through ``Solver``.
* ``core``: one call each of the kernel seam's host-array functions.
* ``mumps``: the replicated Newton loop of a reference-style program: COO
  assembly on host arrays, ``MumpsSolver`` for the linear systems.
* ``sweep``: a batch of steady solves of uneven grids (``v2d_batch_*``).
* ``adjoint``: gradients of a force objective with respect to the angle of
  attack, the Reynolds number and the wall shape at a steady state.

``exact`` gives the same results in 64 bits without this package: the metric,
residual and Jacobian expressions written out on torch tensors, and Newton
with a direct solver over the grid's radial rows (block tridiagonal).
"""
from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import torch

F64 = torch.float64
FF_CODES = {"dirichlet": 0, "outflow": 1, "outflow_psi": 2}


# ------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest grids users start from (smoke tests, teaching): launches and host time
        dict(name="step_25x17", kind="unsteady", body="cylinder", imax=25, jmax=17, dt=0.2,
             farfield="outflow", precision="fp64", reuse=0, warm=2),
        # a coarse steady solve, the quick look before a production run
        dict(name="steady_65x49", kind="steady", body="cylinder", imax=65, jmax=49,
             precision="fp64"),
        # the steady validation grid
        dict(name="steady_129x129", kind="steady", body="cylinder", imax=129, jmax=129,
             precision="fp64"),
        # the headline: unsteady cylinder, mixed precision, factors kept over Newton and time steps
        dict(name="step_181x181_mixed", kind="unsteady", body="cylinder", imax=181, jmax=181,
             dt=0.2, farfield="outflow", precision="mixed", reuse=8, warm=3, steps=4),
        # the same with the default configuration: FP64, every Jacobian factored
        dict(name="step_181x181_fp64", kind="unsteady", body="cylinder", imax=181, jmax=181,
             dt=0.2, farfield="outflow", precision="fp64", reuse=0, warm=3),
        # an airfoil O-grid (uneven sides) at an angle of attack, default configuration
        dict(name="step_naca_257x129", kind="unsteady", body="naca0012", imax=257, jmax=129,
             dt=0.05, farfield="dirichlet", precision="fp64", reuse=0, warm=2),
        # a fine grid the way long runs take it: FP64, factors kept while GMRES stays short
        dict(name="step_513x513_reuse", kind="unsteady", body="cylinder", imax=513, jmax=513,
             dt=0.05, farfield="outflow", precision="fp64", reuse=12, warm=2,
             steps=3),
        # the largest: a million nodes, every Jacobian factored
        dict(name="step_1025x1025", kind="unsteady", body="cylinder", imax=1025, jmax=1025,
             dt=0.05, farfield="outflow", precision="fp64", reuse=0, warm=1),
        # drop-in kernels on host arrays, as a reference-style program calls them
        dict(name="core_181x181", kind="core", body="cylinder", imax=181, jmax=181),
        # the linear-solver drop-in inside the replicated Newton loop
        dict(name="mumps_129x129", kind="mumps", body="cylinder", imax=129, jmax=129, dt=0.2,
             farfield="dirichlet", warm=1),
        # a parameter sweep of uneven grids solved together
        dict(name="sweep_9", kind="sweep", count=9, imax=129, jmax=129),
        # gradients for design: reverse direction
        dict(name="adjoint_129x97", kind="adjoint", body="cylinder", imax=129, jmax=97),
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["unsteady"] * 5 + ["steady"] * 2 + ["core", "mumps", "sweep", "adjoint"])
    body = rng.choice(["cylinder", "cylinder", "naca0012"]) if kind == "unsteady" else "cylinder"
    if kind == "unsteady":
        # the largest grids are square-ish cylinders in FP64; the mixed form's range ends at 257
        precision = rng.choice(["fp64", "fp64", "mixed"])
        hi = 257 if precision == "mixed" or body == "naca0012" else 641
        imax = _log_int(rng, 33 if body == "naca0012" else 25, hi)
        jmax = max(17, min(hi, int(round(imax * rng.uniform(0.5, 1.1)))))
        reuse = rng.choice([0, 8, 12])
        return dict(kind=kind, body=body, imax=imax, jmax=jmax,
                    dt=0.05 if body == "naca0012" else rng.choice([0.05, 0.1, 0.2]),
                    farfield="dirichlet" if body == "naca0012"
                    else rng.choice(["dirichlet", "outflow"]),
                    precision=precision, reuse=reuse, warm=2, steps=3 if reuse else 1)
    # steady Newton from the free stream converges from about 49 columns on at these Re
    hi = {"steady": 193, "core": 513, "mumps": 181, "sweep": 145, "adjoint": 161}[kind]
    imax = _log_int(rng, 33 if kind in ("core", "mumps") else 65, hi)
    jmax = max(33, int(round(imax * rng.uniform(0.6, 1.1))))
    if kind == "steady":
        return dict(kind=kind, body=body, imax=imax, jmax=jmax,
                    precision=rng.choice(["fp64", "fp64", "mixed"]))
    if kind == "mumps":
        return dict(kind=kind, body=body, imax=imax, jmax=jmax, dt=rng.choice([0.1, 0.2]),
                    farfield="dirichlet", warm=1)
    if kind == "sweep":
        return dict(kind=kind, count=rng.choice([3, 6, 9]), imax=imax, jmax=jmax)
    return dict(kind=kind, body=body, imax=imax, jmax=jmax)


# ------------------------------------------------------------------ inputs
def _physics(case, seed):
    """What the seed decides: the flow's parameters and the body's size."""
    rng = random.Random(1000003 * int(seed) + 17)
    if case["kind"] == "unsteady" or case["kind"] == "mumps":
        naca = case["body"] == "naca0012"
        return dict(re=rng.uniform(90.0, 210.0), alpha=rng.uniform(1.0, 4.0) if naca else 0.0,
                    rot=0.0 if naca else rng.uniform(0.3, 0.6),
                    outer=rng.uniform(40.0, 60.0))
    return dict(re=rng.uniform(20.0, 40.0), alpha=rng.uniform(1.0, 6.0), rot=0.0,
                outer=rng.uniform(40.0, 60.0))


def _mesh(body, imax, jmax, outer):
    """The O-grid (xg, yg), an input like any other: the package's generators."""
    from vorti2d_b200 import mesh
    if body == "naca0012":
        return mesh.generate_naca0012(imax, jmax)
    return mesh.generate_cylinder(imax, jmax, outer_rad=outer)


def _sweep_instances(case, seed):
    """The batch: cylinders on three grids, each instance with its own Reynolds
    number and angle."""
    rng = random.Random(7919 * int(seed) + 5)
    imax, jmax = case["imax"], case["jmax"]
    shapes = [(imax, jmax), (max(49, (3 * imax) // 4), max(33, (3 * jmax) // 4)),
              (imax, max(33, jmax // 2))]
    return [dict(imax=shapes[k % 3][0], jmax=shapes[k % 3][1], re=rng.uniform(15.0, 35.0),
                 alpha=rng.uniform(1.0, 6.0)) for k in range(case["count"])]


def _smooth_fields(imax, jmax, xg, yg, seed):
    """psi, ome and two earlier vorticity levels of a smooth seeded flow."""
    rng = np.random.default_rng(int(seed))
    x, y = (np.asarray(a).T.ravel() for a in (xg, yg))
    r = np.hypot(x, y)
    a, b, c = rng.uniform(0.1, 0.4, 3)
    psi = y * (1.0 - 0.25 / np.maximum(r, 0.5) ** 2) + 0.1 * np.sin(a * x) * np.cos(b * y)
    ome = np.cos(c * x) * np.sin(a * y) * np.exp(-0.02 * r)
    return psi, ome, 0.9 * ome, 0.8 * ome


def _config(case, ph):
    from vorti2d_b200 import Config
    steady = case["kind"] in ("steady", "adjoint")
    kw = dict(re=ph["re"], steady=steady, alpha_deg=ph["alpha"], verbose=False, write_csv=False,
              write_xdmf=False, precision=case.get("precision", "fp64"),
              ref_length=1.0 if case["body"] == "naca0012" else None)
    if not steady:
        kw.update(dt_phys=case["dt"], rot_speed=ph["rot"], rot_until=2.0,
                  farfield_bc=case["farfield"], max_pseudo_iter=20)
    if case["kind"] == "adjoint":
        kw.update(pseudo_tol=1e-13, max_pseudo_iter=40)
    if case.get("reuse"):
        kw.update(lu_reuse_its=case["reuse"], lu_reuse_steps=True, ksp_restart=30)
    return Config(**kw)


def _host_buffers(n):
    pin = torch.cuda.is_available()
    return [torch.zeros(n, dtype=F64, pin_memory=pin).numpy() for _ in range(4)]


def prepare(case, seed):
    import vorti2d_b200 as v
    kind = case["kind"]
    if kind == "sweep":
        return _prepare_sweep(case, seed)
    ph = _physics(case, seed)
    imax, jmax = case["imax"], case["jmax"]
    xg, yg = _mesh(case["body"], imax, jmax, ph["outer"])
    st = dict(case=case, ph=ph, mesh=(xg, yg))
    if kind == "core":
        st["fields"] = _smooth_fields(imax, jmax, xg, yg, seed)
        return st
    if kind == "mumps":
        N = imax * jmax
        st["met"] = v.core.compute_metrics(1.0 / (imax - 1), 1.0 / (jmax - 1), xg, yg)
        st["lin"] = v.MumpsSolver(2 * N, grid=(imax, jmax))
        psi = np.zeros(N)
        psi[imax * (jmax - 1):] = st["met"][9][imax * (jmax - 1):]
        q = [psi, np.zeros(N), np.zeros(N), np.zeros(N)]
        for _ in range(case["warm"]):
            q = _mumps_step(st, q)
        st["start"] = q
        return st
    s = v.Solver(_config(case, ph), mesh=(xg, yg))
    st["solver"] = s
    if kind == "unsteady":
        for k in range(case["warm"]):
            s.advance(k * case["dt"])
        st["t"] = case["warm"] * case["dt"]
    elif kind == "adjoint":
        s.advance(0.0)
        rng = random.Random(31 * int(seed) + 3)
        st["weights"] = [rng.uniform(0.5, 1.5) for _ in range(3)]
    st["start"] = _host_buffers(s.ndof)
    s.get_state(st["start"])
    st["out"] = _host_buffers(s.ndof)
    return st


class _Batch:
    """A batch handle of the C ABI and its instances' solver handles."""

    def __init__(self, insts, meshes):
        from vorti2d_b200 import Config, _lib
        from vorti2d_b200.solver import solver_params
        self.lib, n = _lib, len(insts)
        cfgs = [Config(re=i["re"], alpha_deg=i["alpha"], steady=True, ksp_restart=30)
                for i in insts]
        prm = (_lib.SolverParams * n)(*[solver_params(c) for c in cfgs])
        xs = [np.asfortranarray(m[0]) for m in meshes]
        ys = [np.asfortranarray(m[1]) for m in meshes]
        im = np.array([i["imax"] for i in insts], dtype=np.intc)
        jm = np.array([i["jmax"] for i in insts], dtype=np.intc)
        self.h = ctypes.c_void_p()
        _lib.check(_lib.lib().v2d_batch_create(
            n, _lib.iptr(im), _lib.iptr(jm), (_lib._dp * n)(*[_lib.dptr(x) for x in xs]),
            (_lib._dp * n)(*[_lib.dptr(y) for y in ys]), prm, ctypes.byref(self.h)))
        self.inst = []
        for k in range(n):
            p = ctypes.c_void_p()
            _lib.check(_lib.lib().v2d_batch_instance(self.h, k, ctypes.byref(p)))
            self.inst.append(p)

    def set_active(self, active):
        self.lib.check(self.lib.lib().v2d_batch_set_active(self.h, self.lib.iptr(active)))

    def set_state(self, k, q):
        self.lib.check(self.lib.lib().v2d_solver_set_state(self.inst[k],
                                                           *[self.lib.dptr(a) for a in q]))

    def get_state(self, k, psi, ome):
        self.lib.check(self.lib.lib().v2d_solver_get_state(
            self.inst[k], self.lib.dptr(psi), self.lib.dptr(ome), None, None))

    def newton(self, res):
        st = self.lib.LinStats()
        self.lib.check(self.lib.lib().v2d_batch_newton(self.h, self.lib.dptr(res), None,
                                                       ctypes.byref(st)))

    def __del__(self):
        if self.h:
            self.lib.lib().v2d_batch_destroy(self.h)
            self.h = None


def _free_stream(inst, mesh):
    imax, jmax = inst["imax"], inst["jmax"]
    N, a = imax * jmax, math.radians(inst["alpha"])
    psi = np.zeros(N)
    ff = math.cos(a) * mesh[1] - math.sin(a) * mesh[0]
    psi[imax * (jmax - 1):] = ff[:, jmax - 1]
    return [psi, np.zeros(N), np.zeros(N), np.zeros(N)]


def _prepare_sweep(case, seed):
    insts = _sweep_instances(case, seed)
    meshes = [_mesh("cylinder", i["imax"], i["jmax"], 50.0) for i in insts]
    return dict(case=case, batch=_Batch(insts, meshes),
                start=[_free_stream(i, m) for i, m in zip(insts, meshes)],
                out=[(np.zeros(i["imax"] * i["jmax"]), np.zeros(i["imax"] * i["jmax"]))
                     for i in insts])


# --------------------------------------------------------------------- run
def _mumps_step(st, q):
    """One BDF2 step: assemble the COO system, solve, update, until converged."""
    import vorti2d_b200 as v
    case, ph = st["case"], st["ph"]
    imax, jmax = case["imax"], case["jmax"]
    N = imax * jmax
    psi, ome, old, oldold = (a.copy() for a in q)
    for _ in range(20):
        ci, cj, cv, nnz, b = v.core.assemble_coo(
            imax, jmax, ph["re"], 0.0, 0.5 / case["dt"], ph["rot"], 1.0 / (imax - 1),
            1.0 / (jmax - 1), *st["met"], psi, ome, old, oldold, 0, 2 * N, 26 * N,
            FF_CODES[case["farfield"]], 1.0, 0.0)
        st["lin"].assemble(ci[:nnz], cj[:nnz], cv[:nnz], b)
        dq = st["lin"].solve()
        psi += dq[:N]
        ome += dq[N:]
        if np.linalg.norm(dq) / (2.0 * N) <= 1e-10:
            break
    return [psi, ome, ome.copy(), old]


def _forces(fc):
    return np.array([fc.cd, fc.cl, fc.cm])


def run(state):
    import vorti2d_b200 as v
    kind = state["case"]["kind"]
    if kind == "core":
        case = state["case"]
        imax, jmax = case["imax"], case["jmax"]
        N, dk, de = imax * jmax, 1.0 / (imax - 1), 1.0 / (jmax - 1)
        met = v.core.compute_metrics(dk, de, *state["mesh"])
        coo = v.core.assemble_coo(imax, jmax, state["ph"]["re"], 0.0, 2.5, 0.0, dk, de, *met,
                                  *state["fields"], 0, 2 * N, 26 * N, 1, 1.0, 0.0)
        jac, _, beta, gama, _, _, ex, ey, xp, yp = met
        vel = v.compute_velocity(imax, jmax, dk, de, jac, beta, gama, ex, ey,
                                 state["fields"][0], want_mag=True)
        fc = v.compute_force_coeffs(imax, jmax, state["ph"]["re"], dk, de, beta, gama, ex, ey,
                                    xp, yp, state["fields"][1])
        return [list(met), list(coo), list(vel), _forces(fc)]
    if kind == "mumps":
        return _mumps_step(state, state["start"])
    if kind == "sweep":
        B, n = state["batch"], state["case"]["count"]
        for k in range(n):
            B.set_state(k, state["start"][k])
        active, res = np.ones(n, dtype=np.intc), np.zeros(n)
        B.set_active(active)
        for _ in range(20):
            B.newton(res)
            active[(active != 0) & (res <= 1e-10)] = 0
            if not active.any():
                break
            B.set_active(active)
        for k in range(n):
            B.get_state(k, *state["out"][k])
        return state["out"]
    s = state["solver"]
    s.set_state(*state["start"])
    if kind == "adjoint":
        from vorti2d_b200.adjoint import force_vjp, shape_vjp
        d_alpha, d_re, _ = force_vjp(s, state["weights"])
        shape, _ = shape_vjp(s, state["weights"], state["mesh"])
        return [np.array([d_alpha, d_re]), shape]
    hist = []
    for k in range(state["case"].get("steps", 1)):
        s.advance(state["t"] + k * state["case"]["dt"] if kind == "unsteady" else 0.0)
        hist.append(_forces(s.force_coeffs()))
    s.get_state(state["out"])
    return [state["out"], np.array(hist)]


# -------------------------------------------------------------------- work
def _newton_work(N, its, es):
    """Factorization flops and factor bytes of `its` Newton iterations on N
    nodes: about 1000 N^1.5 flops by nested dissection, and 40 log2(N) factor
    entries a node written once and read once, besides the 264-byte system."""
    entries = 40.0 * math.log2(N) * N
    return its * (264.0 * N + 2.0 * es * entries), its * 1000.0 * N ** 1.5


def work(case):
    N = case["imax"] * case["jmax"]
    kind = case["kind"]
    if kind == "core":
        return dict(bytes=float(N * (2 + 10 + 14 + 20 + 6 + 3 + 7 + 2) * 8 + 26 * N * 8),
                    flops=900.0 * N)
    if kind == "sweep":
        b = f = 0.0
        for i in _sweep_instances(case, 0):
            bi, fi = _newton_work(i["imax"] * i["jmax"], 7, 8)
            b, f = b + bi, f + fi
        return dict(bytes=b, flops=f)
    its = {"unsteady": 4 * case.get("steps", 1), "steady": 7, "mumps": 4, "adjoint": 1}[kind]
    b, f = _newton_work(N, its, 4 if case.get("precision") == "mixed" else 8)
    if case.get("reuse"):
        f /= 4.0      # the factors of about one Jacobian a step serve its Newton iterations
    return dict(bytes=b + 12.0 * 8 * N, flops=f)


# ------------------------------------------------------------------- exact
class _Grid:
    """Metrics, residual and Jacobian of one O-grid on torch tensors of shape
    (jmax, imax), 64 bits."""

    def __init__(self, xg, yg, device):
        self.imax, self.jmax = xg.shape
        self.dev = device
        self.dk, self.de = 1.0 / (self.imax - 1), 1.0 / (self.jmax - 1)
        i = torch.arange(self.imax, device=device)
        self.e, self.w = i + 1, i - 1
        self.e[-1], self.w[0] = 1, self.imax - 2
        self.metrics(*(torch.as_tensor(np.ascontiguousarray(a.T), dtype=F64, device=device)
                       for a in (xg, yg)))

    def metrics(self, x, y):
        dk, de = self.dk, self.de

        def xi(a):
            return (a[:, self.e] - a[:, self.w]) / (2 * dk)

        def xixi(a):
            return (a[:, self.e] - 2 * a + a[:, self.w]) / dk ** 2

        def eta(a):
            return torch.cat([(-3 * a[:1] + 4 * a[1:2] - a[2:3]) / (2 * de),
                              (a[2:] - a[:-2]) / (2 * de),
                              (3 * a[-1:] - 4 * a[-2:-1] + a[-3:-2]) / (2 * de)])

        def etaeta(a):
            return torch.cat([(2 * a[:1] - 5 * a[1:2] + 4 * a[2:3] - a[3:4]) / de ** 2,
                              (a[2:] - 2 * a[1:-1] + a[:-2]) / de ** 2,
                              (2 * a[-1:] - 5 * a[-2:-1] + 4 * a[-3:-2] - a[-4:-3]) / de ** 2])

        xe, ye = eta(x), eta(y)
        J = 1.0 / (xi(x) * ye - xe * xi(y))
        kx, ky, ex, ey = J * ye, -J * xe, -J * xi(y), J * xi(x)
        a, b, g = kx * kx + ky * ky, ex * ex + ey * ey, kx * ex + ky * ey
        xx, yy = (xixi(x), etaeta(x), xi(xe)), (xixi(y), etaeta(y), xi(ye))

        def conv(cx, cy):
            return -(a * (xx[0] * cx + yy[0] * cy) + 2 * g * (xx[2] * cx + yy[2] * cy)
                     + b * (xx[1] * cx + yy[1] * cy))

        self.x, self.y, self.J, self.a, self.b, self.g = x, y, J, a, b, g
        self.p, self.q, self.ex, self.ey = conv(kx, ky), conv(ex, ey), ex, ey
        return [J, a, b, g, self.p, self.q, ex, ey, x, y]

    def _parts(self, f):
        """The stencil differences of a field on the interior rows: xi, eta,
        xi-xi, eta-eta, cross."""
        c, n, s = f[1:-1], f[2:], f[:-2]
        e, w = self.e, self.w
        return ((c[:, e] - c[:, w]) / (2 * self.dk), (n - s) / (2 * self.de),
                (c[:, e] - 2 * c + c[:, w]) / self.dk ** 2, (n - 2 * c + s) / self.de ** 2,
                (n[:, e] - n[:, w] - s[:, e] + s[:, w]) / (4 * self.dk * self.de))

    def _laplace(self, d):
        i = slice(1, -1)
        return (self.a[i] * d[2] + 2 * self.g[i] * d[4] + self.b[i] * d[3] + self.p[i] * d[0]
                + self.q[i] * d[1])

    def out_mask(self, prm):
        return (prm["ca"] * self.ex[-1] + prm["sa"] * self.ey[-1]) > 0

    def rhs(self, psi, ome, old, oldold, prm):
        """b = -R: the psi rows and the vorticity rows."""
        re, i2, ca, sa = prm["re"], prm["inv2dt"], prm["ca"], prm["sa"]
        dp, do = self._parts(psi), self._parts(ome)
        i = slice(1, -1)
        bp = self._laplace(dp) / re + ome[i] / re
        bo = (self.J[i] * (dp[0] * do[1] - dp[1] * do[0]) + self._laplace(do) / re
              - (3 * ome[i] - 4 * old[i] + oldold[i]) * i2)
        bw = self.b[0] / self.de ** 2
        rad = torch.sqrt(self.x[0] ** 2 + self.y[0] ** 2)
        slip = prm["rot"] / ((self.ex[0] * self.x[0] + self.ey[0] * self.y[0]) / rad)
        wall = (ome[0] - 3.5 * bw * psi[0] + 4 * bw * psi[1] - 0.5 * bw * psi[2]
                - (self.q[0] - 3 * self.b[0] / self.de) * slip)
        far_p = ca * self.y[-1] - sa * self.x[-1] - psi[-1]
        far_o = -ome[-1]
        out = self.out_mask(prm)
        if prm["ff"] >= 2:
            far_p = torch.where(out, -(psi[-1] - 2 * psi[-2] + psi[-3]), far_p)
        if prm["ff"] >= 1:
            far_o = torch.where(out, (4 * ome[-2] - ome[-3]) / 3 - ome[-1], far_o)
        return (torch.cat([-psi[:1], bp, far_p[None]]), torch.cat([wall[None], bo, far_o[None]]))

    def table(self, psi, ome, prm):
        """The Jacobian of R row by row: (columns, values), each 2N x 14 in
        the order a row's entries are written, column -1 where there is none."""
        im, jm, dev = self.imax, self.jmax, self.dev
        N, re = im * jm, prm["re"]
        col = torch.full((2, jm, im, 14), -1, dtype=torch.int64, device=dev)
        val = torch.zeros((2, jm, im, 14), dtype=F64, device=dev)
        k = torch.arange(N, device=dev).reshape(jm, im)
        i = slice(1, -1)
        c, n, s = k[1:-1], k[2:], k[:-2]
        nine = [c, c[:, self.e], c[:, self.w], n, s, n[:, self.e], n[:, self.w], s[:, self.e],
                s[:, self.w]]
        A, B = self.a[i] / (re * self.dk ** 2), self.b[i] / (re * self.de ** 2)
        P, Q = self.p[i] / (2 * re * self.dk), self.q[i] / (2 * re * self.de)
        G = 2 * self.g[i] / (4 * re * self.dk * self.de)
        diff = [2 * A + 2 * B, -A - P, -A + P, -B - Q, -B + Q, -G, G, G, -G]
        dp, do = self._parts(psi), self._parts(ome)
        Jk, Je = self.J[i] / (2 * self.dk), self.J[i] / (2 * self.de)
        conv = [3 * prm["inv2dt"], Jk * dp[1], -Jk * dp[1], -Je * dp[0], Je * dp[0], 0, 0, 0, 0]
        for q in range(9):
            col[0, i, :, q], val[0, i, :, q] = nine[q], diff[q]
            col[1, i, :, q], val[1, i, :, q] = nine[q] + N, diff[q] + conv[q]
        col[0, i, :, 9], val[0, i, :, 9] = c + N, -1.0 / re
        for q, (at, v) in enumerate([(3, Je * do[0]), (4, -Je * do[0]), (1, -Jk * do[1]),
                                     (2, Jk * do[1])]):
            col[1, i, :, 9 + q], val[1, i, :, 9 + q] = nine[at], v
        col[0, 0, :, 0], val[0, 0, :, 0] = k[0], 1.0
        bw = self.b[0] / self.de ** 2
        for q, (at, v) in enumerate([(k[0] + N, -torch.ones_like(bw)), (k[0], 3.5 * bw),
                                     (k[1], -4 * bw), (k[2], 0.5 * bw)]):
            col[1, 0, :, q], val[1, 0, :, q] = at, v
        out = self.out_mask(prm)
        for f, (off, least, three) in enumerate([(0, 2, (1.0, -2.0, 1.0)),
                                                 (N, 1, (1.0, -4 / 3, 1 / 3))]):
            col[f, -1, :, 0], val[f, -1, :, 0] = k[-1] + off, 1.0
            if prm["ff"] >= least:
                for q in (1, 2):
                    col[f, -1, :, q] = torch.where(out, k[-1 - q] + off, -1)
                    val[f, -1, :, q] = three[q] * out.to(F64)
        return col.reshape(2 * N, 14), val.reshape(2 * N, 14)

    def force_terms(self, ome, re, ref_length):
        """(cd, cl, cm) of the wall integrals."""
        P = self.imax - 1
        r = [t[0, :P] for t in (self.x, self.y, self.ex, self.ey, self.b, self.g)]
        xw, yw, ex, ey, b, g = r
        ow = ome[0, :P]
        inv = 1.0 / torch.sqrt(b)
        tx, ty = ey * inv, -ex * inv
        oxi = (torch.roll(ow, -1) - torch.roll(ow, 1)) / (2 * self.dk)
        oeta = (-3 * ow + 4 * ome[1, :P] - ome[2, :P]) / (2 * self.de)
        dn = (g * oxi + b * oeta) * inv
        seg = torch.sqrt((torch.roll(xw, -1) - xw) ** 2 + (torch.roll(yw, -1) - yw) ** 2)
        ds = 0.5 * (seg + torch.roll(seg, 1))
        if ref_length is None:
            cx, cy = (xw * ds).sum() / ds.sum(), (yw * ds).sum() / ds.sum()
            d = 2 * (torch.sqrt((xw - cx) ** 2 + (yw - cy) ** 2) * ds).sum() / ds.sum()
        else:
            d = ref_length
        fr = ow / re
        fx = (yw * dn * ds).sum() / re - (fr * tx * ds).sum()
        fy = -(xw * dn * ds).sum() / re - (fr * ty * ds).sum()
        m = (-((xw ** 2 + yw ** 2) * dn * ds).sum() / (2 * re)
             - ((xw * ty - yw * tx) * fr * ds).sum())
        return torch.stack([2 * fx / d, 2 * fy / d, 2 * m / d ** 2])


class _RowLU:
    """Block tridiagonal LU of the 2N system over radial rows (the two rows
    next to each boundary together: the boundary rows reach two rows away)."""

    def __init__(self, grid, col, val, transpose=False):
        im, jm, dev = grid.imax, grid.jmax, grid.dev
        N = im * jm
        r = torch.arange(2 * N, device=dev)[:, None].expand_as(col)
        keep = col >= 0
        r, c, v = r[keep], col[keep], val[keep]
        if transpose:
            r, c = c, r
        self.csr = torch.sparse_coo_tensor(torch.stack([r, c]), v, (2 * N, 2 * N),
                                           check_invariants=False).coalesce()
        self.n, self.im, self.jm = N, im, jm
        # group of each radial row, and the place of an unknown in its group
        grp = torch.clamp(torch.arange(jm, device=dev) - 1, 0, jm - 3)
        first = torch.zeros(jm - 2, dtype=torch.int64, device=dev)
        first[1:] = torch.arange(2, jm - 1, device=dev)
        size = torch.full((jm - 2,), 1, dtype=torch.int64, device=dev)
        size[0] = size[-1] = 2

        def place(u):
            node, fld = u % N, u // N
            j, i = node // im, node % im
            return grp[j], ((j - first[grp[j]]) * 2 + fld) * im + i

        gr, pr = place(r)
        gc, pc = place(c)
        order = torch.argsort(gr, stable=True)
        gr, pr, gc, pc, v = (t[order] for t in (gr, pr, gc, pc, v))
        cut = torch.searchsorted(gr, torch.arange(jm - 1, device=dev)).tolist()
        u = torch.arange(2 * N, device=dev)
        gu, pu = place(u)
        self.perm = torch.argsort(gu * (4 * im) + pu)
        self.size = (size * 2 * im).tolist()
        self.fac, self.up, self.low = [], [], []
        prev = None
        for q in range(jm - 2):
            s = slice(cut[q], cut[q + 1])

            def block(other):
                m = gc[s] == other
                B = torch.zeros(self.size[q], self.size[other], dtype=F64, device=dev)
                B.index_put_((pr[s][m], pc[s][m]), v[s][m], accumulate=True)
                return B

            D = block(q)
            if q > 0:
                low = block(q - 1)
                D -= low @ prev
                self.low.append(low.to_sparse())
            lu = torch.linalg.lu_factor(D)
            self.fac.append(lu)
            if q < jm - 3:
                prev = torch.linalg.lu_solve(*lu, block(q + 1))
                self.up.append(prev)

    def solve(self, b):
        parts = list(torch.split(b[self.perm], self.size))
        z = []
        for q, p in enumerate(parts):
            if q > 0:
                p = p - torch.mv(self.low[q - 1], z[-1])
            z.append(torch.linalg.lu_solve(*self.fac[q], p[:, None])[:, 0])
        for q in range(len(z) - 2, -1, -1):
            z[q] = z[q] - self.up[q] @ z[q + 1]
        x = torch.empty_like(b)
        x[self.perm] = torch.cat(z)
        return x


def _converge(grid, q, prm, chord):
    """Newton on (psi, ome) until the update is at rounding level; chord: a
    factorization serves while its iterations contract quickly."""
    psi, ome, old, oldold = q
    lu, last = None, math.inf
    for _ in range(60):
        b = torch.cat([t.reshape(-1) for t in grid.rhs(psi, ome, old, oldold, prm)])
        if lu is None:
            lu = _RowLU(grid, *grid.table(psi, ome, prm))
        dq = lu.solve(b).reshape(2, grid.jmax, grid.imax)
        psi, ome = psi + dq[0], ome + dq[1]
        size = float(torch.linalg.norm(dq) / torch.linalg.norm(torch.stack([psi, ome])))
        if size < 1e-13 or (size < 1e-11 and size > 0.5 * last):
            return psi, ome
        if not chord or size > 0.05 * last:
            lu = None
        last = size
    return psi, ome


def _params(re, alpha, ff=0, inv2dt=0.0, rot=0.0):
    a = math.radians(alpha)
    return dict(re=re, ca=math.cos(a), sa=math.sin(a), ff=ff, inv2dt=inv2dt, rot=rot)


def _free_stream_state(grid, prm):
    z = torch.zeros_like(grid.x)
    psi = z.clone()
    psi[-1] = prm["ca"] * grid.y[-1] - prm["sa"] * grid.x[-1]
    return [psi, z.clone(), z.clone(), z.clone()]


def _flat(t):
    return t.reshape(-1).cpu().numpy()


def _exact_unsteady(case, ph, grid, ref):
    prm = _params(ph["re"], ph["alpha"], FF_CODES[case["farfield"]], 0.5 / case["dt"], ph["rot"])
    q, forces = _free_stream_state(grid, prm), []
    for _ in range(case["warm"] + case.get("steps", 1)):
        psi, ome = _converge(grid, q, prm, True)
        q = [psi, ome, ome, q[2]]
        forces.append(_flat(grid.force_terms(ome, ph["re"], ref)))
    return [_flat(t) for t in q], np.array(forces[case["warm"]:])


def exact(case, seed):
    kind = case["kind"]
    # a million nodes take minutes here
    if kind != "core" and case["imax"] * case["jmax"] > 500 * 500:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "sweep":
        out = []
        for i in _sweep_instances(case, seed):
            grid = _Grid(*_mesh("cylinder", i["imax"], i["jmax"], 50.0), dev)
            prm = _params(i["re"], i["alpha"])
            out.append(tuple(_flat(t) for t in _converge(grid, _free_stream_state(grid, prm),
                                                         prm, False)))
        return out
    ph = _physics(case, seed)
    grid = _Grid(*_mesh(case["body"], case["imax"], case["jmax"], ph["outer"]), dev)
    ref = 1.0 if case["body"] == "naca0012" else None
    if kind == "core":
        return _exact_core(case, seed, ph, grid)
    if kind in ("unsteady", "mumps"):
        state, forces = _exact_unsteady(case, ph, grid, ref)
        return state if kind == "mumps" else [state, forces]
    prm = _params(ph["re"], ph["alpha"])
    q = _free_stream_state(grid, prm)
    psi, ome = _converge(grid, q, prm, False)
    if kind == "steady":
        return [[_flat(t) for t in (psi, ome, q[2], q[3])],
                _flat(grid.force_terms(ome, ph["re"], ref))[None]]
    return _exact_adjoint(case, seed, ph, grid, psi, ome)


def _exact_core(case, seed, ph, grid):
    N = case["imax"] * case["jmax"]
    xg, yg = _mesh(case["body"], case["imax"], case["jmax"], ph["outer"])
    fields = [torch.as_tensor(f, dtype=F64, device=grid.dev).reshape(grid.jmax, grid.imax)
              for f in _smooth_fields(case["imax"], case["jmax"], xg, yg, seed)]
    prm = _params(ph["re"], 0.0, 1, 2.5, 0.0)
    met = [_flat(t) for t in (grid.J, grid.a, grid.b, grid.g, grid.p, grid.q, grid.ex, grid.ey,
                              grid.x, grid.y)]
    col, val = grid.table(fields[0], fields[1], prm)
    cv = np.zeros(26 * N)
    got = val[col >= 0].cpu().numpy()
    cv[:got.size] = got
    b = np.concatenate([_flat(t) for t in grid.rhs(*fields, prm)])
    psi = fields[0]
    pxi = (psi[:, grid.e] - psi[:, grid.w]) / (2 * grid.dk)
    pe = torch.cat([(-3 * psi[:1] + 4 * psi[1:2] - psi[2:3]), psi[2:] - psi[:-2],
                    (3 * psi[-1:] - 4 * psi[-2:-1] + psi[-3:-2])]) / (2 * grid.de)
    kx = (grid.g * grid.ex + grid.J * grid.ey) / grid.b
    ky = (grid.g * grid.ey - grid.J * grid.ex) / grid.b
    u, w = pxi * ky + pe * grid.ey, -(pxi * kx + pe * grid.ex)
    vel = [_flat(t) for t in (u, w, torch.sqrt(u * u + w * w))]
    fc = grid.force_terms(fields[1], ph["re"], None).cpu().numpy()
    return [met, [None, None, cv, None, b], vel, fc]


def _exact_adjoint(case, seed, ph, grid, psi, ome):
    """Gradients of w . (Cl, Cd, Cm): one solve with J^T, then the derivatives
    of the objective plus lambda . b at the fixed state."""
    rng = random.Random(31 * int(seed) + 3)
    w = [rng.uniform(0.5, 1.5) for _ in range(3)]
    wt = torch.tensor([w[1], w[0], w[2]], dtype=F64, device=grid.dev)
    prm = _params(ph["re"], ph["alpha"])
    o = ome.clone().requires_grad_(True)
    (gome,) = torch.autograd.grad((grid.force_terms(o, ph["re"], None) * wt).sum(), o)
    g = torch.cat([torch.zeros_like(gome).reshape(-1), gome.reshape(-1)])
    lu = _RowLU(grid, *grid.table(psi, ome, prm), transpose=True)
    lam = lu.solve(g)
    for _ in range(3):
        lam = lam + lu.solve(g - torch.mv(lu.csr, lam))
    # wall displacement along the outward normals, decaying to the far field
    x0, y0 = grid.x, grid.y
    P = grid.imax - 1
    tx = torch.roll(x0[0, :P], -1) - torch.roll(x0[0, :P], 1)
    ty = torch.roll(y0[0, :P], -1) - torch.roll(y0[0, :P], 1)
    tn = torch.hypot(tx, ty)
    nx, ny = ty / tn, -tx / tn
    sgn = torch.where(nx * (x0[1, :P] - x0[0, :P]) + ny * (y0[1, :P] - y0[0, :P]) < 0, -1.0, 1.0)
    nx, ny = nx * sgn, ny * sgn
    cum = torch.cat([torch.zeros_like(x0[:1]),
                     torch.cumsum(torch.hypot(x0[1:] - x0[:-1], y0[1:] - y0[:-1]), 0)])
    phi = (1 - cum / cum[-1:]) ** 2
    d = torch.zeros(P, dtype=F64, device=grid.dev, requires_grad=True)
    re = torch.tensor(ph["re"], dtype=F64, device=grid.dev, requires_grad=True)
    al = torch.tensor(ph["alpha"], dtype=F64, device=grid.dev, requires_grad=True)
    full = torch.cat([d * nx, (d * nx)[:1]]), torch.cat([d * ny, (d * ny)[:1]])
    grid.metrics(x0 + full[0] * phi, y0 + full[1] * phi)
    p = dict(prm, re=re, ca=torch.cos(al * math.pi / 180), sa=torch.sin(al * math.pi / 180))
    z = torch.zeros_like(psi)
    b = torch.cat([t.reshape(-1) for t in grid.rhs(psi, ome, z, z, p)])
    total = (grid.force_terms(ome, re, None) * wt).sum() + (lam * b).sum()
    gd, gr, ga = torch.autograd.grad(total, (d, re, al))
    return [np.array([float(ga), float(gr)]), gd.cpu().numpy()]
