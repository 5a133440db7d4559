"""The direct pressure solve on meshes of planes (tg_fdm.cu) against the oracle
on whole steps, at the sizes where its transforms change form: directions of 4
cells, odd, even and multiples of 4 (one, two and four groups of modes), row
counts around the 8-row tiles, stretched (unfolded) directions, panels of 32,
16 and 8 columns, and a periodic wall-normal direction. The solve must reach
rtol 1e-13 within two iterations, which the multigrid preconditioner does not.

Bounds: velocities as in test_gpu_parity; the pressure to 1e-9 as in
test_gpu_odd_sizes, and on long directions to the bound that the stopping test
gives: both solvers stop at a relative residual of 1e-13, which leaves a
relative error of up to 1e-13 times the condition number of the operator, whose
part of an equidistant direction of n cells is 1 / sin^2(pi / (2 n)), about
(2 n / pi)^2."""
import numpy as np
import pytest

import oracle
import tosca_b200
from tosca_b200 import api, cases
from tests.common import rel_l2

pytestmark = pytest.mark.gpu


def stretch(nodes, axis, amp=0.3):
    """Smoothly non-uniform nodes along physical x (axis 0) or y (axis 1)."""
    d = 0 if axis == 0 else 2
    idx = [0, 0, 0]
    idx[d] = slice(0, -1)
    X = nodes[tuple(idx) + (axis,)].copy()
    L = X[-1]
    Y = X + amp * L / (2 * np.pi) * np.sin(2 * np.pi * X / L)
    shape = [1, 1, 1]
    shape[d] = -1
    nodes[:-1, :-1, :-1, axis] = Y.reshape(shape)


def compare(cfg, nodes, u, p, steps=3):
    cfg.poisson_rtol = 1e-13
    g, o = tosca_b200.gpu_solver(cfg), oracle.solver(cfg)
    for s in (g, o):
        cases.setup(s, nodes, u, p)
    for _ in range(steps):
        st = g.step(1)
        assert st.poisson_iterations <= 2
    o.step(steps)
    p_tol = max(1e-9, 1e-13 * (2 * max(cfg.mx, cfg.my, cfg.mz) / np.pi) ** 2)
    for f, tol in (("UCAT", 1e-10), ("UCONT", 1e-10), ("P", p_tol)):
        assert rel_l2(g.get(f), o.get(f)) <= tol, f
    g.close(); o.close()


@pytest.mark.parametrize("nx,ny,nz", [(4, 4, 4), (5, 7, 5), (6, 9, 8), (8, 16, 7), (33, 10, 6), (36, 66, 5), (63, 65, 4),
                                      (300, 6, 4), (4, 301, 4), (6, 1100, 4)])
def test_periodic_channel_sizes(nx, ny, nz):
    cfg, nodes, u, p = cases.abl_case(nx=nx, ny=ny, nz=nz, Lx=10.0 * nx, Ly=10.0 * ny, H=8.0 * nz, ddt=api.DDT_RK4)
    compare(cfg, nodes, u, p)


@pytest.mark.parametrize("nz", [32, 33, 61, 64, 65, 113, 255, 256, 257, 300])
def test_line_lengths(nz):
    """The solver of the j lines has four forms: chunks of 4, 8 and 16 cells per
    warp (up to 32, 64 and 256 cells) and one thread per line, each with its
    remainders. A line solve that is off shows in the bound on the iterations."""
    cfg, nodes, u, p = cases.abl_case(nx=5, ny=5, nz=nz, Lx=50.0, Ly=50.0, H=8.0 * nz, ddt=api.DDT_RK4, dt=0.1)
    compare(cfg, nodes, u, p)


@pytest.mark.parametrize("nx,ny,nz,axis", [(12, 6, 5, None), (13, 8, 5, None), (9, 6, 5, 0), (16, 8, 6, 0), (42, 5, 4, 0)])
def test_open_channel_sizes(nx, ny, nz, axis):
    cfg, nodes, u, p = cases.channel_case(nx=nx, ny=ny, nz=nz, Lx=10.0 * nx, Ly=10.0 * ny, H=8.0 * nz, ddt=api.DDT_RK4, dt=0.1)
    if axis is not None:
        stretch(nodes, axis)
    compare(cfg, nodes, u, p)


@pytest.mark.parametrize("n", [4, 6, 7, 9, 12])
def test_periodic_box(n):
    cfg, nodes, u, p = cases.tgv_case(n, ddt=api.DDT_RK4)
    rng = np.random.default_rng(n)
    u[1:-1, 1:-1, 1:-1] += 0.1 * rng.standard_normal((n, n, n, 3))
    compare(cfg, nodes, u, p)


@pytest.mark.parametrize("nx,ny,nz,direct", [(2032, 4, 5, True), (2048, 4, 5, False)])
def test_longest_directions(nx, ny, nz, direct):
    """508 + 1 rows per group of modes run the direct solve, 512 + 1 the multigrid;
    the step conserves the discrete divergence either way."""
    cfg, nodes, u, p = cases.abl_case(nx=nx, ny=ny, nz=nz, Lx=10.0 * nx, Ly=10.0 * ny, H=8.0 * nz, ddt=api.DDT_RK4)
    cfg.poisson_rtol = 1e-10
    s = tosca_b200.gpu_solver(cfg)
    cases.setup(s, nodes, u, p)
    st = s.step(1)
    assert (st.poisson_iterations <= 2) == direct
    assert st.max_divergence <= 1e-9
    s.close()


def test_stretched_periodic_direction_keeps_multigrid():
    """A periodic direction that is not equidistant is outside the direct
    solver's range: the step runs on the multigrid and agrees all the same."""
    cfg, nodes, u, p = cases.abl_case(nx=16, ny=12, nz=8, Lx=160.0, Ly=120.0, H=64.0, ddt=api.DDT_RK4)
    stretch(nodes, 0, amp=0.1)
    cfg.poisson_rtol = 1e-13
    g, o = tosca_b200.gpu_solver(cfg), oracle.solver(cfg)
    for s in (g, o):
        cases.setup(s, nodes, u, p)
    assert g.step(1).poisson_iterations > 2
    g.step(2)
    o.step(3)
    for f, tol in (("UCAT", 1e-10), ("P", 1e-9)):
        assert rel_l2(g.get(f), o.get(f)) <= tol, f
    g.close(); o.close()


def test_a_refused_mesh_pays_for_no_eigenvectors():
    """An open mesh of 500 x 500 cells stretched both ways is beyond the direct
    solver's rows. Its set-up must cost what that of 500 x 513 cells costs, where one
    direction alone is beyond them: both set up the multigrid. The two eigenproblems
    of 500 cells take 0.1 to 0.25 s."""
    import time
    seconds = []
    for ny in (500, 513):
        cfg, nodes, u, p = cases.abl_case(nx=500, ny=ny, nz=4, Lx=5000.0, Ly=10.0 * ny, H=40.0)
        cfg.bc = (api.BC_SLIP, api.BC_SLIP, api.BC_NOSLIP, api.BC_SLIP, api.BC_SLIP, api.BC_SLIP)
        cfg.nut_bc = (api.NUTBC_ZEROGRADIENT,) * 6
        stretch(nodes, 0, 0.2)
        stretch(nodes, 1, 0.2)
        s = tosca_b200.gpu_solver(cfg)
        t = []
        for _ in range(6):
            t0 = time.perf_counter()
            s.set_mesh_nodes(nodes)
            t.append(time.perf_counter() - t0)
        seconds.append(min(t))
        s.close()
    assert seconds[0] <= 1.25 * seconds[1], seconds
