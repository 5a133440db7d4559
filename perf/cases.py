"""Performance cases: what a program that uses this framework has it compute.

Most of them are a time loop between two field outputs: `tg_step` over a fixed
number of steps, then the solution fields copied into the program's own
(pinned) host arrays. One is the drop-in call with host state in and out on
every step (`tg_step_host`), one the gradient of a functional through the
discrete adjoint. Grids, schemes and tolerances are those of the framework's
own workloads (`tosca_b200.cases`, `bench.py`): the pressure solve stops on the
divergence bound, time steps are those of the workloads.

    kind    domain
    tgv     Taylor-Green vortex, all-periodic, central, no LES (the vortex is
            restarted on every pass, as in a parameter study)
    abl     neutral boundary layer: periodic x and y, Schumann wall function,
            slip top, Smagorinsky, stretched z
    host    abl, advanced by tg_step_host
    sabl    stratified abl: transported temperature, buoyancy, thermal wall
            function
    hill    terrain-following curvilinear mesh, QUICK, transported temperature
    farm    abl opened in x (inflow and outflow patches) with actuator disks
    abcn    abl with the implicit-explicit ABCN scheme (GMRES)
    adj     abl with a body force: forward steps and their adjoint
"""
import ctypes
import math

import numpy as np
import torch

import tosca_b200
from tosca_b200 import api, cases

DIV_TOL = 5e-9            # divergence bound at which the pressure solve stops


def listed():
    def c(name, kind, nx, ny, nz, steps, prec="fp64"):
        return {"name": name, "kind": kind, "nx": nx, "ny": ny, "nz": nz, "steps": steps, "prec": prec}

    return [
        # the smallest runs: regression and convergence studies, bound by launches and latency
        c("tgv_32", "tgv", 32, 32, 32, 20),
        # the published Taylor-Green configuration
        c("tgv_64_mixed", "tgv", 64, 64, 64, 20, "mixed"),
        # the horizontal shape of TOSCA's boundary-layer decks: odd in every direction
        c("abl_75x75x25", "abl", 75, 75, 25, 20),
        # a production boundary layer in double precision
        c("abl_192x192x96", "abl", 192, 192, 96, 20),
        # the headline configuration
        c("abl_256x256x128_mixed", "abl", 256, 256, 128, 20, "mixed"),
        # TOSCA's loop calling this library as a drop-in step on host arrays
        c("host_128x128x64_mixed", "host", 128, 128, 64, 10, "mixed"),
        # night-time (stable) boundary layer
        c("sabl_128x128x64", "sabl", 128, 128, 64, 20),
        # flow over terrain, the curvilinear path
        c("hill_192x96x96_mixed", "hill", 192, 96, 96, 10, "mixed"),
        # turbines behind an inflow
        c("farm_192x128x64_mixed", "farm", 192, 128, 64, 20, "mixed"),
        # larger time steps through the implicit-explicit scheme
        c("abcn_96x96x48", "abcn", 96, 96, 48, 10),
        # data assimilation: gradient of a velocity misfit with respect to the body force
        c("adj_128x64x64", "adj", 128, 64, 64, 10),
    ]


def _span(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tgv", "abl", "abl", "abl", "host", "sabl", "hill", "farm", "abcn", "adj"])
    prec = rng.choice(["fp64", "mixed"])
    steps = 20
    if kind == "tgv":
        nx = ny = nz = _span(rng, 16, 96)
    elif kind == "abl":
        nx, ny, nz = _span(rng, 24, 256), _span(rng, 24, 256), _span(rng, 16, 128)
    elif kind == "hill":
        nx, ny, nz, steps = 2 * _span(rng, 24, 96), _span(rng, 16, 96), _span(rng, 16, 96), 10
    elif kind == "abcn":
        nx, ny, nz, steps, prec = _span(rng, 32, 128), _span(rng, 32, 128), _span(rng, 16, 64), 10, "fp64"
    elif kind == "adj":
        nx, ny, nz, steps, prec = 2 * _span(rng, 16, 64), _span(rng, 24, 64), _span(rng, 16, 64), 10, "fp64"
    elif kind == "farm":
        nx, ny, nz = _span(rng, 96, 256), _span(rng, 64, 160), _span(rng, 24, 96)
    else:
        nx, ny, nz = _span(rng, 24, 192), _span(rng, 24, 192), _span(rng, 16, 96)
    if kind == "host":
        steps = 10
    return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "steps": steps, "prec": prec}


# ------------------------------------------------------------------ inputs
def _inputs(case, seed):
    """(config, nodes, Ucat, P, T or None, turbines or None) of a case."""
    kind, nx, ny, nz = case["kind"], case["nx"], case["ny"], case["nz"]
    box = dict(nx=nx, ny=ny, nz=nz, Lx=10.0 * nx, Ly=10.0 * ny, H=1000.0 * nz / 128.0)
    T = turbines = None
    if kind == "tgv":
        cfg, nodes, u, p = cases.tgv_case(nx, ddt=api.DDT_RK4)
        # a solenoidal perturbation of the vortex: one mode per direction, seeded
        a, b = np.random.default_rng(seed).uniform(-0.05, 0.05, (2, 3))
        x, y, z = (cases.cell_centres(nodes)[1:-1, 1:-1, 1:-1, q] for q in range(3))
        w = u[1:-1, 1:-1, 1:-1]
        w[..., 0] += a[0] * np.sin(2 * z) + b[0] * np.cos(y)
        w[..., 1] += a[1] * np.sin(2 * x) + b[1] * np.cos(z)
        w[..., 2] += a[2] * np.sin(2 * y) + b[2] * np.cos(x)
    elif kind == "sabl":
        cfg, nodes, u, p, T = cases.stratified_abl_case(ddt=api.DDT_RK4, seed=seed + 1, **box)
        # the generator seeds the velocity by its own default: perturb it too
        u[1:-1, 1:-1, 1:-1] *= 1.0 + np.random.default_rng(seed).uniform(-0.01, 0.01, (nx, nz, ny, 1))
    elif kind == "hill":
        cfg, nodes, u, p, T = cases.hill_case(nx=nx, ny=ny, nz=nz, ddt=api.DDT_RK4, teqn=True, t_amp=0.05, seed=seed + 1)
    elif kind == "farm":
        cfg, nodes, u, p, turbines = cases.farm_case(rows=2, cols=2, D=63.0, hub=60.0, ddt=api.DDT_RK4, seed=seed + 1, **box)
        cases.open_x(cfg, 8.0, None)
    else:
        cfg, nodes, u, p = cases.abl_case(ddt=api.DDT_ABCN if kind == "abcn" else api.DDT_RK4, seed=seed + 1, **box)
    if kind == "abcn":
        cfg.snes_atol, cfg.snes_rtol, cfg.gmres_restart = 1e-5, 1e-30, 30
    if kind == "adj":
        cfg.source = 1
    cfg.poisson_rtol, cfg.poisson_div_tol, cfg.poisson_maxit = 1e-30, DIV_TOL, 400
    cfg.precision = api.PREC_MIXED if case["prec"] == "mixed" else api.PREC_FP64
    return cfg, nodes, u, p, T, turbines


def _pinned(shape, values=None):
    """A page-locked host array (numpy), as a program keeps for its fields."""
    a = torch.zeros(tuple(shape), dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()
    if values is not None:
        a[...] = values
    return a


class _State:
    """A solver with the host arrays of the program that drives it."""

    def __init__(self, solver, case):
        self.solver, self.case, self.out, self.start = solver, case, {}, {}

    def array(self, field):
        if field not in self.out:
            self.out[field] = _pinned(self.solver.field_shape(field))
        return self.out[field]

    def get(self, field):
        """tg_get_field into the program's own array."""
        a = self.array(field)
        s = self.solver
        s._check(s.fns["get_field"](s.h, api.F[field], a.ctypes.data_as(ctypes.c_void_p), 0), "get_field " + field)
        return a

    def __del__(self):
        self.solver.close()


def prepare(case, seed):
    cfg, nodes, u, p, T, turbines = _inputs(case, seed)
    s = tosca_b200.gpu_solver(cfg)
    cases.setup(s, nodes, u, p, T)
    if turbines:
        s.set_turbines(turbines, 1.225)
    st = _State(s, case)
    kind = case["kind"]
    for f in ("UCONT", "UCAT", "P") + (("TMPRT",) if T is not None else ()):
        st.array(f)
    if kind == "host":
        st.array("NUT")
        for f in ("UCONT", "UCAT", "P"):
            st.get(f)                     # the program's state lives in its own arrays
    if kind in ("tgv", "adj"):
        st.start = {f: _pinned(s.field_shape(f), s.get(f)) for f in ("UCONT", "UCAT", "P")}
    if kind == "adj":
        rng = np.random.default_rng(seed + 7)
        st.start["SOURCE"] = _pinned(s.field_shape("SOURCE"), rng.standard_normal(s.field_shape("SOURCE")) * 1e-3)
        # misfit gradient on the horizontal plane of cells at mid height, every
        # second cell along x; every other adjoint field starts at zero
        st.adjoint = {f: _pinned(s.field_shape(f)) for f in ("UCAT_ADJ", "UCONT_ADJ", "P_ADJ", "SOURCE_ADJ", "WALL_ADJ")}
        probe = st.adjoint["UCAT_ADJ"][1:-1:2, cfg.my // 2, 1:-1, 0]
        probe[...] = rng.standard_normal(probe.shape)
        for f in ("SOURCE_ADJ", "UCAT_ADJ", "UCONT_ADJ"):
            st.array(f)
    return st


def run(st):
    s, kind, n = st.solver, st.case["kind"], st.case["steps"]
    if kind == "host":
        for _ in range(n):
            s.step_host(st.out["UCONT"], st.out["UCAT"], st.out["P"], st.out["NUT"])
        return dict(st.out)
    if kind == "adj":
        for f, a in st.start.items():
            s.set(f, a)
        s.adjoint_forward(n, n)
        ucat = st.get("UCAT")
        for f, a in st.adjoint.items():
            s.set(f, a)
        s.adjoint_reverse()
        return {"UCAT": ucat, "SOURCE_ADJ": st.get("SOURCE_ADJ"), "UCONT_ADJ": st.get("UCONT_ADJ"), "UCAT_ADJ": st.get("UCAT_ADJ")}
    for f, a in st.start.items():
        s.set(f, a)
    s.step(n)
    return {f: st.get(f) for f in st.out}


# ------------------------------------------------------- necessary work
def work(case):
    """Bytes and FP64/FP32 operations that the steps of one pass cannot do
    without on their grid: per momentum stage the velocity and flux fields, the
    pressure gradient, the old and the running state read and the new state
    written, once each; per step the eddy viscosity, the pressure solve (right-
    hand side in, solution out, two passes over the unknowns per direction of
    a direct solve), the projection and the final conversion; the mesh metrics
    of a curvilinear grid once per stage; and the fields handed to and from
    the host."""
    kind, cells, n = case["kind"], case["nx"] * case["ny"] * case["nz"], case["steps"]
    stages = 1 if kind == "abcn" else 4
    values = stages * (3 + 3 + 1 + 3 + 3 + 3 + 3)          # U, Ucat, nut, dP, U_o, running sum, new U
    values += (3 + 1) + (1 + 3) + (3 + 1) + (1 + 3 + 3) + (3 + 3) + 12
    flops = stages * 300 + 250
    if kind == "tgv":
        values -= stages + 4
    if kind in ("sabl", "hill"):
        values += 4 * 8
        flops += 4 * 200
    if kind == "hill":
        met = 4 if case["prec"] == "mixed" else 8
        return {"bytes": cells * n * (8.0 * values + (stages + 1) * 30 * met + 8 * 30), "flops": cells * n * (flops + stages * 500.0)}
    if kind == "abcn":
        values += 5 * 10
        flops += 5 * 250
    if kind == "adj":
        values *= 3
        flops *= 3
    moved = 8 * ({"host": 15 * n, "adj": 9}.get(kind, 7))
    return {"bytes": cells * (8.0 * values * n + moved), "flops": float(cells) * n * flops}


def tolerance(case):
    """The pressure solve stops at a divergence of 5e-9 per step, which leaves
    the pressure uncertain far above the rounding of the arithmetic. Measured
    against the same steps with the solve carried to a relative residual of
    1e-12 (20 and 40 steps, these sizes and drawn ones): neutral boundary
    layers and farms, whose pressure is small, up to 8.3e-6 in P (2.1e-5 at
    the worst point) and 1e-9 in the velocities; the vortex 9e-9; stratified
    and hill cases 1.4e-8, to which mixed precision adds about 1e-7; adjoint
    fields 1.6e-7 (2.8e-6)."""
    kind = case["kind"]
    if kind == "tgv":
        return {"rel": 2e-7, "max": 2e-6}
    if kind in ("sabl", "hill"):
        return {"rel": 1e-6, "max": 1e-5}
    if kind == "adj":
        return {"rel": 1e-6, "max": 2e-5}
    return {"rel": 3e-5, "max": 1e-4}


# ------------------------------------------------- the same steps in torch
def exact(case, seed):
    """The fields of `run` from a plain torch float64 evaluation of the scheme
    on Cartesian meshes with uniform x and y spacing (kinds tgv, abl and
    host), with the pressure equation solved directly. The curvilinear,
    stratified, open, implicit and adjoint cases have no such value."""
    if case["kind"] not in ("tgv", "abl", "host"):
        return None
    cfg, nodes, u0, p0, _, _ = _inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    ref = _Cartesian(cfg, nodes, dev)
    ref.start(torch.as_tensor(u0, device=dev), torch.as_tensor(p0, device=dev))
    for _ in range(case["steps"]):
        ref.step()
    out = {"UCONT": ref.V.movedim(0, -1), "UCAT": ref.U.movedim(0, -1), "P": ref.p}
    if case["kind"] == "host":
        out["NUT"] = ref.nut
    return {k: v.contiguous().cpu().numpy() for k, v in out.items()}


class _Cartesian:
    """TOSCA's RK4 step with central convection on (k, j, i) arrays with one
    ghost layer; i and k periodic and uniform, j periodic, or a Schumann wall
    below and a slip plane above. Physical axes: i -> y, j -> z, k -> x."""

    def __init__(self, cfg, nodes, dev):
        self.cfg = c = cfg
        self.pj = c.bc[2] == api.BC_PERIODIC
        N = torch.as_tensor(nodes, device=dev)
        z = N[0, : c.my - 1, 0, 2]
        self.dx, self.dy = float(N[1, 0, 0, 0] - N[0, 0, 0, 0]), float(N[0, 0, 1, 1] - N[0, 0, 0, 1])
        dz = z[1:] - z[:-1]                                            # cells j = 1 .. my-2
        self.dz = torch.cat([dz[:1], dz, dz[-1:]])                     # with ghosts
        # distance across the j faces 0 .. my-2
        inner = 0.5 * (z[2:] - z[:-2])
        last = 0.5 * (dz[:1] + dz[-1:]) if self.pj else dz[-1:]
        self.dzf = torch.cat([dz[:1], inner, last])
        col = lambda v: v[None, :, None]                               # noqa: E731
        self.col = col
        self.A = (self.dx * col(self.dz), self.dx * self.dy, self.dy * col(self.dz))   # i, j, k face areas
        self.aj = 1.0 / (self.dx * self.dy * col(self.dz))
        # Jacobians of the i, j, k faces (j faces 0 .. my-2, padded)
        self.jaj = 1.0 / (self.dx * self.dy * col(torch.cat([self.dzf, self.dzf[-1:]])))
        self.shape = (c.mz, c.my, c.mx)
        self.zeros = lambda *s: torch.zeros(*s, *self.shape, dtype=torch.float64, device=dev)   # noqa: E731
        self.it = c.it_start
        self._poisson_setup(dev)

    # ---- boundary and ghost updates
    def _periodic(self, a):
        a[..., 0], a[..., -1] = a[..., -2].clone(), a[..., 1].clone()
        if self.pj:
            a[..., 0, :], a[..., -1, :] = a[..., -2, :].clone(), a[..., 1, :].clone()
        a[..., 0, :, :], a[..., -1, :, :] = a[..., -2, :, :].clone(), a[..., 1, :, :].clone()

    def _face_periodic(self, V):
        V[..., 0] = V[..., -2].clone()
        if self.pj:
            V[..., 0, :] = V[..., -2, :].clone()
        V[..., 0, :, :] = V[..., -2, :, :].clone()

    def _no_penetration(self):
        if not self.pj:
            self.V[1, :-1, 0, :-1] = 0.0
            self.V[1, :-1, -2, :-1] = 0.0

    def _cartesian_bcs(self):
        U, s = self.U, slice(1, -1)
        U[:, s, s, 0], U[:, s, s, -1] = U[:, s, s, -2].clone(), U[:, s, s, 1].clone()
        if self.pj:
            U[:, s, 0, s], U[:, s, -1, s] = U[:, s, -2, s].clone(), U[:, s, 1, s].clone()
        else:
            for q in (0, 1):                                           # wall-parallel, extrapolated
                U[q, s, 0, s] = 2 * U[q, s, 1, s] - U[q, s, 2, s]
            U[2, s, 0, s] = -U[2, s, 1, s]
            U[0, s, -1, s], U[1, s, -1, s], U[2, s, -1, s] = U[0, s, -2, s], U[1, s, -2, s], -U[2, s, -2, s]
        U[:, 0, s, s], U[:, -1, s, s] = U[:, -2, s, s].clone(), U[:, 1, s, s].clone()

    def _contravariant_bcs(self):
        V, U, m = self.V, self.U, slice(0, -1)
        V[0, m, m, 0] = V[0, m, m, -2].clone()
        V[0, m, m, -2] = self._edge0(0.5 * (U[1, m, m, -1] + U[1, m, m, -2]) * self.A[0][0, m, 0])
        if self.pj:
            V[1, m, 0, m] = V[1, m, -2, m].clone()
            V[1, m, -2, m] = self._edge0(0.5 * (U[2, m, -1, m] + U[2, m, -2, m]) * self.A[1])
        else:
            V[1, m, 0, m] = 0.0
            V[1, m, -2, m] = 0.0
        V[2, 0, m, m] = V[2, -2, m, m].clone()
        V[2, -2, m, m] = self._edge0(0.5 * (U[0, -1, m, m] + U[0, -2, m, m]) * self.A[2][0, m, :])

    @staticmethod
    def _edge0(a):
        """Face metrics vanish on the faces outside the interior rows."""
        a[0], a[:, 0] = 0.0, 0.0
        return a

    def _scalar_ghosts(self, a):
        a[..., 0], a[..., -1] = a[..., -2].clone(), a[..., 1].clone()
        if self.pj:
            a[:, 0], a[:, -1] = a[:, -2].clone(), a[:, 1].clone()
        else:
            a[:, 0], a[:, -1] = a[:, 1].clone(), a[:, -2].clone()
        a[0], a[-1] = a[-2].clone(), a[1].clone()

    # ---- stencils on interior cells
    def _to_cart(self, U):
        V, s = self.V, slice(1, -1)
        U[1, s, s, s] = 0.5 * (V[0, s, s, :-2] + V[0, s, s, 1:-1]) / self.A[0][:, s]
        U[2, s, s, s] = 0.5 * (V[1, s, :-2, s] + V[1, s, 1:-1, s]) / self.A[1]
        U[0, s, s, s] = 0.5 * (V[2, :-2, s, s] + V[2, 1:-1, s, s]) / self.A[2][:, s]

    def start(self, u, p):
        self.U, self.V, self.nut = self.zeros(3), self.zeros(3), self.zeros()
        s = slice(1, -1)
        self.U[:, s, s, s] = u.movedim(-1, 0)[:, s, s, s]
        self._cartesian_bcs()
        U, V, m = self.U, self.V, slice(0, -1)
        V[0, 1:-1, 1:-1, m] = (0.5 * (U[1, 1:-1, 1:-1, :-1] + U[1, 1:-1, 1:-1, 1:])) * self.A[0][:, 1:-1]
        V[1, 1:-1, m, 1:-1] = (0.5 * (U[2, 1:-1, :-1, 1:-1] + U[2, 1:-1, 1:, 1:-1])) * self.A[1]
        V[2, m, 1:-1, 1:-1] = (0.5 * (U[0, :-1, 1:-1, 1:-1] + U[0, 1:, 1:-1, 1:-1])) * self.A[2][:, 1:-1]
        self._contravariant_bcs()
        self.p = p.clone()
        self.filt = self.um = None
        self.tau = None

    def _grad_cell(self):
        """Velocity gradients dU_a/dx_b of the interior cells, [a][b]."""
        U, s = self.U, slice(1, -1)
        di = 0.5 * (U[:, s, s, 2:] - U[:, s, s, :-2])
        dj = 0.5 * (U[:, s, 2:, s] - U[:, s, :-2, s])
        if not self.pj:
            dj[:, :, 0] = U[:, s, 2, s] - U[:, s, 1, s]
            dj[:, :, -1] = U[:, s, -2, s] - U[:, s, -3, s]
        dk = 0.5 * (U[:, 2:, s, s] - U[:, :-2, s, s])
        return dk / self.dx, di / self.dy, dj / self.col(self.dz[1:-1])

    def _nut(self):
        gx, gy, gz = self._grad_cell()
        g = (gx, gy, gz)                                               # g[b][a]
        s2 = sum((0.5 * (g[b][a] + g[a][b])) ** 2 for a in range(3) for b in range(3))
        width2 = (self.dx * self.dy * self.col(self.dz[1:-1])) ** (2.0 / 3.0)
        nut = self.zeros()
        s = slice(1, -1)
        nut[s, s, s] = self.cfg.cs * width2 * torch.sqrt(2.0 * s2)
        nut[s, s, 0], nut[s, s, -1] = nut[s, s, -2], nut[s, s, 1]
        nut[0, s, s], nut[-1, s, s] = nut[-2, s, s], nut[1, s, s]
        self.nut = nut

    def _wall(self):
        c, s = self.cfg, slice(1, -1)
        up = self.U[:2, s, 1, s]
        mag = torch.sqrt(up[0] ** 2 + up[1] ** 2)
        mean = mag.mean()
        dist = 0.5 * self.dz[1]
        us = mean * c.wall_kappa / torch.log(dist / c.wall_roughness)
        if self.filt is None:
            self.filt, self.um = up.clone(), torch.zeros_like(mag)
        a = self.it / (self.it + 1.0)
        self.um = a * self.um + (1 - a) * mag
        T = torch.clamp(math.hypot(self.dx, self.dy) / self.um, min=c.dt)
        self.filt = (1 - c.dt / T) * self.filt + (c.dt / T) * up
        self.tau = -us * us * self.filt / torch.clamp(mean, min=1e-5) * self.A[1]

    def _rhs(self):
        """FormU and the pressure gradient at the + faces of interior cells."""
        c, U, V, s = self.cfg, self.U, self.V, slice(1, -1)
        les = bool(c.les)
        nt = self.nut
        dzc, A = self.col(self.dz), self.A
        last_j = self.shape[1] - 2
        # --- i faces 0 .. mx-2 of the interior (k, j) rows
        L, R = U[:, :, :, :-1], U[:, :, :, 1:]
        S2 = L + R
        dc = (R - L)[:, s, s]
        dzk = 0.25 * (S2[:, 2:, s] - S2[:, :-2, s])
        dej = 0.25 * (S2[:, s, 2:] - S2[:, s, :-2])
        if not self.pj:
            # the periodic seam face next to the wall and the top: one-sided
            dej[:, :, 0, -1] = 0.5 * (S2[:, s, 2, -1] - S2[:, s, 1, -1])
            dej[:, :, -1, -1] = 0.5 * (S2[:, s, -2, -1] - S2[:, s, -3, -1])
        nu = c.nu + (0.5 * (nt[s, s, :-1] + nt[s, s, 1:]) if les else 0.0)
        a = A[0][:, s]
        faj = self.aj[:, s]
        ze, et = A[2][:, s], A[1]
        visc = torch.stack([a * a * dc[0] + dzk[1] * ze * a, 2 * a * a * dc[1], a * a * dc[2] + dej[1] * et * a]) * faj * nu
        F1 = -V[0, s, s, :-1] * 0.5 * S2[:, s, s] + visc
        # --- j faces 0 .. my-2
        L, R = U[:, :, :-1], U[:, :, 1:]
        S2 = L + R
        de = (R - L)[:, s, :, s]
        dci = 0.25 * (S2[:, s, :, 2:] - S2[:, s, :, :-2])
        dzk = 0.25 * (S2[:, 2:, :, s] - S2[:, :-2, :, s])
        if not self.pj:
            for f in (0, last_j):
                dci[:, :, f, 0] = 0.5 * (S2[:, s, f, 2] - S2[:, s, f, 1])
                dci[:, :, f, -1] = 0.5 * (S2[:, s, f, -2] - S2[:, s, f, -3])
                dzk[:, 0, f] = 0.5 * (S2[:, 2, f, s] - S2[:, 1, f, s])
                dzk[:, -1, f] = 0.5 * (S2[:, -2, f, s] - S2[:, -3, f, s])
        nu = c.nu + (0.5 * (nt[s, :-1, s] + nt[s, 1:, s]) if les else torch.zeros_like(de[0]))
        if not self.pj:
            nu[:, 0] = c.nu
            nu[:, -1] = 0.0
        a = A[1]
        # areas of the i and k faces at a j face: with the distance across it
        cs, ze = self.dx * self.col(self.dzf), self.dy * self.col(self.dzf)
        visc = torch.stack([a * a * de[0] + dzk[2] * ze * a, a * a * de[1] + dci[2] * cs * a, 2 * a * a * de[2]])
        visc = visc * self.jaj[:, :-1] * nu
        if not self.pj and les:
            visc[0, :, 0] -= self.tau[0]
            visc[1, :, 0] -= self.tau[1]
        F2 = -V[1, s, :-1, s] * 0.5 * S2[:, s, :, s] + visc
        # --- k faces 0 .. mz-2
        L, R = U[:, :-1], U[:, 1:]
        S2 = L + R
        dz = (R - L)[:, :, s, s]
        dci = 0.25 * (S2[:, :, s, 2:] - S2[:, :, s, :-2])
        dej = 0.25 * (S2[:, :, 2:, s] - S2[:, :, :-2, s])
        if not self.pj:
            dej[:, -1, 0] = 0.5 * (S2[:, -1, 2, s] - S2[:, -1, 1, s])
            dej[:, -1, -1] = 0.5 * (S2[:, -1, -2, s] - S2[:, -1, -3, s])
        nu = c.nu + (0.5 * (nt[:-1, s, s] + nt[1:, s, s]) if les else 0.0)
        a, cs, et = A[2][:, s], A[0][:, s], A[1]
        visc = torch.stack([2 * a * a * dz[0], a * a * dz[1] + dci[0] * cs * a, a * a * dz[2] + dej[0] * et * a]) * faj * nu
        F3 = -V[2, :-1, s, s] * 0.5 * S2[:, :, s, s] + visc
        # a periodic direction takes its first face from its last
        F1[..., 0] = F1[..., -1]
        F3[:, 0] = F3[:, -1]
        if self.pj:
            F2[:, :, 0] = F2[:, :, -1]
        fp = (F1[..., 1:] - F1[..., :-1]) + (F2[:, :, 1:] - F2[:, :, :-1]) + (F3[:, 1:] - F3[:, :-1])
        nxt_j = torch.roll(fp[2], -1, 1)
        if not self.pj:
            nxt_j[:, -1] = fp[2][:, -1]
        r = torch.stack([
            faj * 0.5 * A[0][:, s] * (fp[1] + torch.roll(fp[1], -1, 2)),
            self.jaj[:, 1:-1] * 0.5 * A[1] * (fp[2] + nxt_j),
            faj * 0.5 * A[2][:, s] * (fp[0] + torch.roll(fp[0], -1, 0))]) - self.dp
        if c.mean_grad_p:
            g = c.mean_grad_p_value
            r[0] += g[1] * A[0][:, s]
            r[1] += g[2] * A[1]
            r[2] += g[0] * A[2][:, s]
        if not self.pj:
            r[1][:, -1] = torch.where(self.Vo[1, s, -2, s] > 0, r[1][:, -1], torch.zeros_like(r[1][:, -1]))
        return r

    def _grad_p(self):
        p, s = self.p, slice(1, -1)
        q = p.clone()
        self._scalar_wrap(q)
        a, faj = self.A, self.aj[:, s]
        dp = torch.stack([(q[s, s, 2:] - q[s, s, s]) * a[0][:, s] ** 2 * faj,
                          (q[s, 2:, s] - q[s, s, s]) * a[1] ** 2 * self.jaj[:, 1:-1],
                          (q[2:, s, s] - q[s, s, s]) * a[2][:, s] ** 2 * faj])
        if not self.pj:
            dp[1][:, -1] = 0.0
        self.dp = dp

    def _scalar_wrap(self, q):
        q[:, :, -1] = q[:, :, 1].clone()
        if self.pj:
            q[:, -1] = q[:, 1].clone()
        q[-1] = q[1].clone()

    def _poisson_setup(self, dev):
        c = self.cfg
        nx, ny, nz = c.mx - 2, c.my - 2, c.mz - 2
        dz = self.dz[1:-1]
        ke, kn = self.dx * dz / self.dy, self.dx * self.dy / self.dzf[1:]
        kt = self.dy * dz / self.dx
        K = torch.zeros(ny, ny, dtype=torch.float64, device=dev)
        for j in range(ny if self.pj else ny - 1):
            e = (j + 1) % ny
            K[j, j] += kn[j]
            K[e, e] += kn[j]
            K[j, e] -= kn[j]
            K[e, j] -= kn[j]
        # divide by the cell height (ke and kt share it) to a standard eigenproblem
        w = dz.rsqrt()
        mu, E = torch.linalg.eigh(w[:, None] * K * w[None, :])
        self.E, self.w = E, w
        li = 2 - 2 * torch.cos(2 * math.pi * torch.arange(nx, dtype=torch.float64, device=dev) / nx)
        lk = 2 - 2 * torch.cos(2 * math.pi * torch.arange(nz, dtype=torch.float64, device=dev) / nz)
        lam = (lk[:, None, None] * (self.dy / self.dx) + mu.clamp(min=0.0)[None, :, None]) + li[None, None, :] * (self.dx / self.dy)
        lam[0, 0, 0] = math.inf
        self.lam = lam[:, :, : nx // 2 + 1]
        self.kk = (ke, kn, kt)

    def _laplace(self, x):
        """(L x)_c = sum over the faces of a_f (x_c - x_nb)."""
        ke, kn, kt = (self.col(v) for v in self.kk)
        y = ke * (2 * x - torch.roll(x, 1, 2) - torch.roll(x, -1, 2)) + kt * (2 * x - torch.roll(x, 1, 0) - torch.roll(x, -1, 0))
        d = kn * (torch.roll(x, -1, 1) - x)
        if not self.pj:
            d[:, -1] = 0.0
        return y - d + torch.roll(d, 1, 1)

    def _direct(self, b):
        h = torch.fft.rfft2(b * self.col(self.w), dim=(0, 2))
        h = torch.einsum("jm,kji->kmi", self.E.to(h.dtype), h) / self.lam
        h = torch.einsum("jm,kmi->kji", self.E.to(h.dtype), h)
        return torch.fft.irfft2(h, s=(b.shape[0], b.shape[2]), dim=(0, 2)) * self.col(self.w)

    def step(self):
        c, s = self.cfg, slice(1, -1)
        self.Vo = self.V.clone()
        if c.les:
            self._nut()
            self._wall()
        self._grad_p()
        b, a = (1 / 6, 1 / 3, 1 / 3, 1 / 6), (0.0, 0.5, 0.5, 1.0)
        acc = self.Vo.clone()
        for st in range(4):
            self._no_penetration()
            self._face_periodic(self.V)
            self._to_cart(self.U)
            self._periodic(self.U)
            r = self._rhs()
            acc[:, s, s, s] += c.dt * b[st] * r
            if st < 3:
                self.V = self.Vo.clone()
                self.V[:, s, s, s] += a[st + 1] * c.dt * r
        self.V = acc
        self._no_penetration()
        self._face_periodic(self.V)
        self._to_cart(self.U)
        self._periodic(self.U)
        # pressure correction
        V = self.V
        div = (V[0, s, s, s] - V[0, s, s, :-2]) + (V[1, s, s, s] - V[1, s, :-2, s]) + (V[2, s, s, s] - V[2, :-2, s, s])
        rhs = -div / c.dt
        x = self._direct(rhs)
        x = x + self._direct(rhs - self._laplace(x))                   # one refinement
        x = x - x[0, 0, 0]
        phi = self.zeros()
        phi[s, s, s] = x
        self._scalar_ghosts(phi)
        self.p[s, s, s] += x
        self._scalar_ghosts(self.p)
        ar, aj = self.A, self.aj[:, s]
        V[0, s, s, :-1] -= (phi[s, s, 1:] - phi[s, s, :-1]) * ar[0][:, s] ** 2 * aj * c.dt
        if self.pj:
            V[1, s, :-1, s] -= (phi[s, 1:, s] - phi[s, :-1, s]) * ar[1] ** 2 * self.jaj[:, :-1] * c.dt
        else:
            V[1, s, 1:-2, s] -= (phi[s, 2:-1, s] - phi[s, 1:-2, s]) * ar[1] ** 2 * self.jaj[:, 1:-2] * c.dt
        V[2, :-1, s, s] -= (phi[1:, s, s] - phi[:-1, s, s]) * ar[2][:, s] ** 2 * aj * c.dt
        self._to_cart(self.U)
        self._cartesian_bcs()
        self._contravariant_bcs()
        self.p = self.p - self.p[1, 1, 1]
        self.it += 1
