"""Device memory of a context whose mesh is set again."""
import pytest
import torch

import tosca_b200
from tosca_b200 import cases
from tests.test_gpu_fdm import stretch

pytestmark = pytest.mark.gpu


def test_replaced_meshes_give_their_memory_back():
    """Setting a mesh again and writing metrics again does not grow the context:
    the pressure solver's arrays belong to the mesh they were made for, and the
    mesh's own temporaries to the call."""
    cfg, nodes, u, p = cases.abl_case(nx=96, ny=96, nz=64, Lx=960.0, Ly=960.0, H=512.0)
    s = tosca_b200.gpu_solver(cfg)
    bent = nodes.copy()
    stretch(bent, 0, 0.1)                           # a periodic direction that the direct solver refuses
    used = []
    for _ in range(4):
        for n in (nodes, bent):
            s.set_mesh_nodes(n)
            s.init_from_cartesian(u)
            s.step(1)
            s.set("AJ", s.get("AJ"))
            s.step(1)
        free, total = torch.cuda.mem_get_info()
        used.append(total - free)
    # one vector of the grid is 5 MB; a solver has some 20, a mesh's temporaries are 12
    assert used[-1] - used[0] <= 16 << 20, used
    s.close()
