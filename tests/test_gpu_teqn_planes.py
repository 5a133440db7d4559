"""The marching temperature flux kernel around its block of 32 x 8 columns and its
chunks of planes, against the oracle: sizes of one column, one block, one more
than a block, and few and many planes, on the curvilinear hill and on a mesh of
planes, with and without Smagorinsky. One RK4 step of transported T: both sides
evaluate the same stencils in FP64 from the same state, and the pressure solve
stops at 1e-13, so 1e-10 leaves room for its round-off in the velocities."""
import pytest

import oracle
import tosca_b200
from tosca_b200 import api, cases
from tests.common import rel_l2

pytestmark = pytest.mark.gpu


SIZES = [("hill", 4, 4, 4), ("hill", 5, 33, 9), ("hill", 23, 32, 8), ("hill", 9, 31, 17),
         ("sabl", 4, 4, 4), ("sabl", 6, 33, 9), ("sabl", 41, 34, 8)]


# the stratified boundary layer's wall functions need Smagorinsky
@pytest.mark.parametrize("kind,nx,ny,nz,les", [c + (1,) for c in SIZES] + [c + (0,) for c in SIZES if c[0] == "hill"])
def test_planes(kind, nx, ny, nz, les):
    if kind == "hill":
        cfg, nodes, u, p, T = cases.hill_case(nx=nx, ny=ny, nz=nz, ddt=api.DDT_RK4, teqn=True, t_amp=0.5)
    else:
        cfg, nodes, u, p, T = cases.stratified_abl_case(nx=nx, ny=ny, nz=nz, ddt=api.DDT_RK4, Lx=10.0 * nx, Ly=10.0 * ny, H=8.0 * nz)
    cfg.les = les
    cfg.poisson_rtol = 1e-13
    out = []
    for make in (tosca_b200.gpu_solver, oracle.solver):
        s = make(cfg)
        cases.setup(s, nodes, u, p, T)
        s.step(1)
        out.append((s.get("TMPRT"), s.get("UCAT")))
        s.close()
    assert rel_l2(out[0][0], out[1][0]) <= 1e-12
    assert rel_l2(out[0][1], out[1][1]) <= 1e-10
