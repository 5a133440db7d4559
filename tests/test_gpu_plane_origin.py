"""Meshes of planes whose coordinates are rounded: an origin far from zero, or
many cells of a spacing that is no binary fraction. The metrics of such a mesh
differ from the products of its spacings by some units of rounding of the
coordinates over the spacing, and it is a mesh of planes all the same
(tg_mesh_info). The step agrees with the oracle, which forms its metrics from the
rounded coordinates.

Bounds. r = eps max|coordinate| / smallest spacing. A cell size by the sums of
eight nodes that the metrics use is off by up to 3.5 r, a face distance by 1.5 r,
a Jacobian by the sum over three directions; a flux has up to three such
factors on top of the area, some 30 r in all, and three steps of four stages
change a velocity by less than its own size: 100 r beside the 1e-11 that the
oracle comparisons of these kernels have at the origin. The pressure is solved
from a divergence in which the fluxes cancel to about a tenth, and the solve of
a perturbed operator carries the perturbation over: 1000 r beside 1e-9."""
import numpy as np
import pytest

import oracle
import tosca_b200
from tosca_b200 import api, cases
from tests.common import div_roundoff_floor, rel_l2

pytestmark = pytest.mark.gpu
EPS = float(np.finfo(np.float64).eps)


def shifted(nx, ny, nz, origin, h=7.3, **kw):
    """A neutral boundary layer with spacing h along x and y whose corner is at
    (origin, origin, 0), and r of the bounds."""
    cfg, nodes, u, p = cases.abl_case(nx=nx, ny=ny, nz=nz, Lx=h * nx, Ly=h * ny, H=8.0 * nz, ddt=api.DDT_RK4, dt=0.1, **kw)
    nodes[:-1, :-1, :-1, 0] = (origin + h * np.arange(nx + 1))[:, None, None]
    nodes[:-1, :-1, :-1, 1] = (origin + h * np.arange(ny + 1))[None, None, :]
    cfg.poisson_rtol = 1e-13
    return cfg, nodes, u, p, EPS * np.abs(nodes).max() / min(h, np.diff(nodes[0, :-1, 0, 2]).min())


@pytest.mark.parametrize("nx,ny,nz,origin", [(24, 16, 10, 0.0), (24, 16, 10, 10000.1), (24, 16, 10, 500000.3), (1500, 8, 8, 0.0)])
def test_planes_by_their_coordinates(nx, ny, nz, origin):
    cfg, nodes, u, p, r = shifted(nx, ny, nz, origin)
    g, o = tosca_b200.gpu_solver(cfg), oracle.solver(cfg)
    for s in (g, o):
        cases.setup(s, nodes, u, p)
    assert g.mesh_info() == (True, True)
    st = g.step(3)
    o.step(3)
    assert st.poisson_total_iterations <= 6
    # the projection inverts the operator it is solved with, however the
    # coordinates are rounded
    assert st.max_divergence <= max(1e-12, div_roundoff_floor(g.get("UCONT"), g.get("AJ")))
    for f in ("UCAT", "UCONT"):
        assert rel_l2(g.get(f), o.get(f)) <= 1e-11 + 100 * r, f
    assert rel_l2(g.get("P"), o.get("P")) <= 1e-9 + 1000 * r
    g.close(); o.close()


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_a_bent_plane_is_not_one(axis):
    """One node off its plane by a millionth of the spacing."""
    cfg, nodes, u, p, r = shifted(12, 10, 8, 10000.1)
    nodes[5, 4, 3, axis] += 7.3e-6
    g = tosca_b200.gpu_solver(cfg)
    g.set_mesh_nodes(nodes)
    assert not g.mesh_info()[1]
    g.close()


@pytest.mark.parametrize("nx,ny,nz,origin", [(24, 16, 10, 0.0), (13, 33, 9, 10000.1)])
def test_nodes_off_their_planes_by_rounding(nx, ny, nz, origin):
    """Nodes that were computed point by point: each is off its plane by up to two
    units of rounding. The mesh counts as one of planes, though its cross metrics no
    longer vanish exactly, so the pressure solve is the general one; the step runs
    on the kernels for planes and agrees with the oracle, which sees every node, and
    with the general kernels. The jitter adds four units to the difference of two
    nodes: 2 r for r of the bounds."""
    cfg, nodes, u, p, r = shifted(nx, ny, nz, origin)
    rng = np.random.default_rng(nx)
    nodes *= 1.0 + EPS * rng.integers(-2, 3, nodes.shape)
    g, b, o = tosca_b200.gpu_solver(cfg), tosca_b200.gpu_solver(cfg), oracle.solver(cfg)
    for s in (g, b, o):
        cases.setup(s, nodes, u, p)
    assert g.mesh_info()[1]
    b.set("AJ", b.get("AJ"))
    assert not b.mesh_info()[1]
    for s in (g, b, o):
        s.step(3)
    for other in (b, o):
        for f in ("UCAT", "UCONT"):
            assert rel_l2(g.get(f), other.get(f)) <= 1e-11 + 300 * r, f
        assert rel_l2(g.get("P"), other.get("P")) <= 1e-9 + 3000 * r
    for s in (g, b, o):
        s.close()
