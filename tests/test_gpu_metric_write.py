"""A program that writes the metrics of another mesh gets the steps of that
mesh: what is derived from the metrics (pressure operator and its solver, filter
widths, the kernels' choice of operator) follows them. The second context has its
mesh from nodes; both run the general kernels (a metric write withdraws the
kernels for meshes of planes), so the same products in the same order. The two
pressure solves stop at a relative residual of 1e-13."""
import numpy as np
import pytest

import tosca_b200
from tosca_b200 import api, cases
from tests.common import div_roundoff_floor, rel_l2
from tests.test_gpu_fdm import stretch

pytestmark = pytest.mark.gpu

METRICS = ("CSI", "ETA", "ZET", "ICSI", "IETA", "IZET", "JCSI", "JETA", "JZET", "KCSI", "KETA", "KZET", "AJ", "IAJ", "JAJ", "KAJ")


def case(scaled, stretched=False, precision=api.PREC_FP64):
    cfg, nodes, u, p = cases.abl_case(nx=14, ny=11, nz=9, Lx=140.0, Ly=110.0, H=72.0, ddt=api.DDT_RK4, dt=0.1, wall=api.BC_NOSLIP)
    cfg.poisson_rtol = 1e-13
    cfg.precision = precision
    if stretched:
        stretch(nodes, 1, 0.2)
    nodes = nodes * scaled
    return cfg, nodes, u, p


@pytest.mark.parametrize("when", ["before the first step", "between steps"])
@pytest.mark.parametrize("stretched,precision", [(False, api.PREC_FP64), (True, api.PREC_FP64), (False, api.PREC_MIXED)])
def test_metrics_of_another_mesh(when, stretched, precision):
    cfg, nodes, u, p = case(1.0, False, precision)
    a, b = tosca_b200.gpu_solver(cfg), tosca_b200.gpu_solver(cfg)
    a.set_mesh_nodes(nodes)
    if when == "between steps":
        a.init_from_cartesian(u)
        a.set("P", p)
        a.step(3)
    b.set_mesh_nodes(case(1.7, stretched)[1])
    for f in METRICS:
        a.set(f, b.get(f))
    b.set("AJ", b.get("AJ"))                       # onto the general kernels too
    assert a.mesh_info() == b.mesh_info() == (True, False)
    for s in (a, b):
        for f in ("RHS", "DP", "PHI"):
            s.set(f, np.zeros(s.field_shape(f)))
        s.set("UCAT", np.zeros(s.field_shape("UCAT")))
        s.init_from_cartesian(u)
        s.set("P", p)
    for _ in range(3):
        st = a.step(1)
        b.step(1)
        assert st.max_divergence <= max(1e-12, div_roundoff_floor(a.get("UCONT"), a.get("AJ")))
    for f, tol in (("NUT", 1e-12), ("UCAT", 1e-11), ("P", 1e-9)):
        assert rel_l2(a.get(f), b.get(f)) <= tol, f
    a.close(); b.close()


def test_cross_metrics_change_the_operator():
    """Metrics of a hill written over a mesh of planes: the 7-point operator is no
    longer the one to solve."""
    cfg, nodes, u, p, T = cases.hill_case(nx=16, ny=10, nz=10, ddt=api.DDT_RK4)
    cfg.poisson_rtol = 1e-13
    cfg.buoyancy = 0
    flat = cases.cartesian_nodes(nodes[:-1, 0, 0, 0], nodes[0, 0, :-1, 1], nodes[0, :-1, 0, 2])
    a, b = tosca_b200.gpu_solver(cfg), tosca_b200.gpu_solver(cfg)
    a.set_mesh_nodes(flat)
    b.set_mesh_nodes(nodes)
    assert a.mesh_info() == (True, True) and b.mesh_info() == (False, False)
    for f in METRICS + ("CENT",):
        a.set(f, b.get(f))
    assert a.mesh_info() == (False, False)
    for s in (a, b):
        s.init_from_cartesian(u)
        s.set("P", p)
        s.step(1)
    for f, tol in (("UCONT", 1e-10), ("P", 1e-9)):
        assert rel_l2(a.get(f), b.get(f)) <= tol, f
    a.close(); b.close()
