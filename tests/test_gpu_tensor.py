"""The stage kernels for meshes of planes (tg_tensor.cu) against the general
curvilinear kernels on the same mesh and against the oracle, at sizes around
their tiles (32 x 8 columns, 2 or 4 cells along k, 32-lane rows), with every
kind of boundary patch, stretched spacings, LES on and off, and each momentum
scheme that shares them. A caller that writes a metric field gets the general
kernels, which is how the second solver here is made.

Bounds: both paths evaluate the same products in another order, some tens of
operations per face and stage at 1.1e-16 each; 1e-12 in the velocities and
fluxes leaves two orders for the cancellation in the budgets. Pressure 1e-9:
the solve stops at a relative residual of 1e-13 on either side."""
import numpy as np
import pytest

import oracle
import tosca_b200
from tosca_b200 import api, cases
from tests.common import rel_l2
from tests.test_gpu_fdm import stretch

pytestmark = pytest.mark.gpu


def make(kind, nx, ny, nz, ddt=api.DDT_RK4, stretched=False, **over):
    box = dict(nx=nx, ny=ny, nz=nz, Lx=10.0 * nx, Ly=10.0 * ny, H=8.0 * nz)
    T = None
    if kind == "tgv":
        cfg, nodes, u, p = cases.tgv_case(nx, ddt=ddt)
        u[1:-1, 1:-1, 1:-1] += 0.1 * np.random.default_rng(nx).standard_normal((nx, nx, nx, 3))
    elif kind == "channel":
        cfg, nodes, u, p = cases.channel_case(ddt=ddt, dt=0.1, **box)
    elif kind == "sabl":
        cfg, nodes, u, p, T = cases.stratified_abl_case(**box)
    elif kind == "box":                                    # closed: noSlip and slip patches in every direction
        cfg, nodes, u, p = cases.abl_case(ddt=ddt, dt=0.05, wall=api.BC_NOSLIP, **box)
        cfg.bc = (api.BC_NOSLIP, api.BC_SLIP, api.BC_NOSLIP, api.BC_SLIP, api.BC_SLIP, api.BC_NOSLIP)
        cfg.nut_bc = (api.NUTBC_FIXEDVALUE, api.NUTBC_ZEROGRADIENT, api.NUTBC_FIXEDVALUE, api.NUTBC_FIXEDVALUE,
                      api.NUTBC_ZEROGRADIENT, api.NUTBC_FIXEDVALUE)
        cfg.mean_grad_p = 0
        u *= 0.1
    else:
        cfg, nodes, u, p = cases.abl_case(ddt=ddt, **box)
    if stretched:
        stretch(nodes, 0, 0.2)
        stretch(nodes, 1, 0.2)
    cfg.poisson_rtol = 1e-13
    for k, v in over.items():
        setattr(cfg, k, v)
    return cfg, nodes, u, p, T


def pair(cfg, nodes, u, p, T):
    """(solver on the kernels for meshes of planes, solver on the general ones)."""
    out = []
    for general in (False, True):
        s = tosca_b200.gpu_solver(cfg)
        cases.setup(s, nodes, u, p, T)
        assert s.mesh_info() == (True, True)
        if general:
            s.set("AJ", s.get("AJ"))
            assert s.mesh_info() == (True, False)
        out.append(s)
    return out


CASES = [("abl", 4, 4, 4, {}), ("abl", 5, 31, 8, {}), ("abl", 9, 33, 10, {}), ("abl", 8, 35, 11, dict(stretched=True)),
         ("abl", 37, 66, 18, {}), ("abl", 7, 12, 9, dict(les=0, nu=0.5)), ("abl", 12, 9, 7, dict(div_scheme=api.DIV_QUICK)),
         ("abl", 10, 34, 12, dict(ddt=api.DDT_FE, dt=0.02)), ("tgv", 4, 4, 4, {}), ("tgv", 13, 13, 13, {}), ("tgv", 34, 34, 34, {}),
         ("channel", 13, 33, 9, {}), ("channel", 9, 12, 10, dict(stretched=True)), ("box", 6, 9, 8, {}), ("box", 12, 34, 7, dict(les=0, nu=0.5)),
         ("box", 7, 8, 12, dict(stretched=True)), ("sabl", 12, 34, 10, {}), ("abl", 12, 16, 9, dict(precision=api.PREC_MIXED)),
         ("abl", 12, 10, 9, dict(ddt=api.DDT_ABCN, snes_atol=1e-12)), ("abl", 8, 10, 9, dict(ddt=api.DDT_CN, snes_atol=1e-11)),
         ("tgv", 10, 10, 10, dict(ddt=api.DDT_RK3WCN, snes_atol=1e-12))]


@pytest.mark.parametrize("kind,nx,ny,nz,over", CASES)
def test_against_general_kernels(kind, nx, ny, nz, over):
    case = make(kind, nx, ny, nz, **over)
    a, b = pair(*case)
    mixed = case[0].precision == api.PREC_MIXED           # the general kernels read FP32 metrics there
    for s in (a, b):
        s.FormU(0.7, True)
    tol = 1e-6 if mixed else 1e-12
    assert rel_l2(a.get("RHS"), b.get("RHS")) <= (1e-4 if mixed else tol)
    # P is the sum of the steps' phi, each solved to a relative residual: where
    # the first step's impulse cancels afterwards the error scales with the
    # largest P, not the last
    big = 0.0
    for _ in range(3):
        for s in (a, b):
            s.step(1)
        big = max(big, np.linalg.norm(b.get("P")))
    implicit = case[0].ddt_scheme not in (api.DDT_FE, api.DDT_RK4)
    for f in ("UCAT", "UCONT", "NUT"):
        whole = lambda x: x                               # noqa: E731  ghost layers too
        assert rel_l2(a.get(f), b.get(f), whole) <= (1e-9 if implicit else tol), f
    assert np.linalg.norm(a.get("P") - b.get("P")) <= (1e-5 if mixed else 1e-8 if implicit else 1e-9) * big
    a.close(); b.close()


@pytest.mark.parametrize("kind,nx,ny,nz,over", [c for c in CASES if c[4].get("precision") is None and c[0] != "sabl"][:16])
def test_against_oracle(kind, nx, ny, nz, over):
    cfg, nodes, u, p, T = make(kind, nx, ny, nz, **over)
    g, o = tosca_b200.gpu_solver(cfg), oracle.solver(cfg)
    for s in (g, o):
        cases.setup(s, nodes, u, p, T)
        s.FormU(1.0, True)
    assert rel_l2(g.get("RHS"), o.get("RHS")) <= 1e-12
    big = 0.0                                              # see above
    for _ in range(3):
        for s in (g, o):
            s.step(1)
        big = max(big, np.linalg.norm(o.get("P")))
    for f in ("UCAT", "UCONT"):
        assert rel_l2(g.get(f), o.get(f)) <= 1e-11, f
    assert np.linalg.norm(g.get("P") - o.get("P")) <= 1e-9 * big
    g.close(); o.close()


# 79 x 65 x 64 cells away from the boundary give 480 tiles of 32 x 8 x 4 cells,
# above the three per SM from which the tile kernel takes four cells along k; 79
# and 65 leave remainders
@pytest.mark.parametrize("over", [{}, dict(les=0, nu=0.5), dict(ddt=api.DDT_ABCN, snes_atol=1e-12)])
def test_deep_tiles(over):
    case = make("abl", 80, 66, 66, **over)
    a, b = pair(*case)
    o = oracle.solver(case[0])
    cases.setup(o, *case[1:])
    for s in (a, b, o):
        s.FormU(1.0, True)
    assert rel_l2(a.get("RHS"), o.get("RHS")) <= 1e-12
    assert rel_l2(a.get("RHS"), b.get("RHS")) <= 1e-12
    if case[0].ddt_scheme == api.DDT_ABCN:                 # the convective and the viscous part by themselves
        for s in (a, b):
            s.step(1)
        assert rel_l2(a.get("UCAT"), b.get("UCAT")) <= 1e-9
    for s in (a, b, o):
        s.close()


def test_metric_write_rebuilds_the_step():
    """A metric written between replayed steps takes effect on the next one."""
    a, b = pair(*make("abl", 12, 16, 9))
    a.step(3); b.step(3)
    a.set("AJ", a.get("AJ"))
    assert a.mesh_info() == (True, False)
    a.step(3); b.step(3)
    assert rel_l2(a.get("UCAT"), b.get("UCAT")) <= 1e-12
    assert not a.graph_info()[1] and a.graph_info()[0] > 2
    a.close(); b.close()


@pytest.mark.parametrize("nx,ny,nz", [(13, 11, 9), (33, 8, 5)])
def test_metric_write_reaches_the_metric_products(nx, ny, nz):
    """The curvilinear kernels read products of the face metrics that are formed
    once: doubling a face Jacobian doubles its component of GradP, exactly."""
    cfg, nodes, u, p, T = cases.hill_case(nx=nx, ny=ny, nz=nz, ddt=api.DDT_RK4, teqn=True, t_amp=0.05, seed=3)
    s = tosca_b200.gpu_solver(cfg)
    cases.setup(s, nodes, u, p, T)
    s.step(2)
    s.GradP()
    d = s.get("DP")
    assert np.abs(d).max(axis=(0, 1, 2)).min() > 0.0
    for f, q in (("IAJ", 0), ("JAJ", 1), ("KAJ", 2)):
        s.set(f, 2.0 * s.get(f))
        s.GradP()
        d[..., q] *= 2.0
        assert np.array_equal(s.get("DP"), d)
    s.close()


@pytest.mark.parametrize("nx,ny,nz,kind,over", [
    (7, 7, 7, "abl", {}), (6, 9, 8, "abl", {}), (9, 38, 11, "abl", dict(stretched=True)), (12, 36, 8, "abl", dict(les=0, nu=0.5)),
    (13, 13, 13, "tgv", {}), (10, 37, 9, "box", {}), (9, 12, 10, "abl", dict(ddt=api.DDT_FE, dt=0.02))])
def test_adjoint_against_general_kernels(nx, ny, nz, kind, over):
    """The reverse step's kernels for meshes of planes, around their tile of
    32 x 4 x 2 cells and the two cells to an end that the scatter keeps. Same
    products in another order, as above; the transposed pressure solve stops at
    the context's relative tolerance of 1e-13. The adjoint of P is bounded
    against its seed: with one stage per step (forward Euler) the projection takes
    out all that an old P puts in, and what is left is rounding."""
    cfg, nodes, u, p, T = make(kind, nx, ny, nz, **over)
    cfg.source = 1
    rng = np.random.default_rng(nx + ny)
    a, b = pair(cfg, nodes, u, p, T)
    seeds = {f: rng.standard_normal(a.field_shape(f)) for f in ("UCAT_ADJ", "UCONT_ADJ", "P_ADJ")}
    for s in (a, b):
        s.step(2)
        for f, v in seeds.items():
            w = np.zeros_like(v)
            w[1:-1, 1:-1, 1:-1] = v[1:-1, 1:-1, 1:-1]
            s.set(f, w)
        s.adjoint_step()
    for f in ("UCONT_ADJ", "UCAT_ADJ", "SOURCE_ADJ"):
        assert rel_l2(a.get(f), b.get(f)) <= 1e-11, f
    assert np.linalg.norm(a.get("P_ADJ") - b.get("P_ADJ")) <= 1e-9 * np.linalg.norm(seeds["P_ADJ"])
    a.close(); b.close()
