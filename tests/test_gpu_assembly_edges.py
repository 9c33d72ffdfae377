"""Assembly around nodes that are not ordinary: a fan of tets about one centre, which has every other node as its
neighbour (more ring nodes, tets and rows than the kernels take in one go). Against the CPU oracle, with the tolerances of test_gpu_3d.py: fields
that are summed in the reference's order are equal, values agree to a few ulps of pow()."""
import dataclasses

import numpy as np
import pytest
from scipy.spatial import ConvexHull

from impressionfea_b200.config import Forging3DConfig
from impressionfea_b200.forging3d import Forging3DSolver
from impressionfea_b200.meshes import upset_case_3d
from oracle import Oracle3D
from test_gpu_3d import RTOL_ELEM, RTOL_ENERGY, _close

pytestmark = pytest.mark.gpu


def _fan(points, like):
    """Tets from the centre of a ball (on the lower die, clear of the symmetry planes) to its hull's triangles."""
    i = np.arange(points)
    z = 1 - 2 * i / (points - 1)
    r, phi = np.sqrt(np.maximum(0, 1 - z * z)), i * np.pi * (3 - np.sqrt(5))
    ball = np.stack([r * np.cos(phi), r * np.sin(phi), z], 1)
    tri = ConvexHull(ball).simplices + 1
    x = np.vstack([[0, 0, 0], ball]) * 5 + [12, 12, 5]
    t = np.hstack([np.zeros((len(tri), 1), int), tri])
    det = np.einsum("ij,ij->i", x[t[:, 1]] - x[t[:, 0]], np.cross(x[t[:, 2]] - x[t[:, 0]], x[t[:, 3]] - x[t[:, 0]]))
    t[det < 0] = t[det < 0][:, [0, 2, 1, 3]]
    zeros = np.zeros(len(x), np.uint8)
    return dataclasses.replace(like, x=np.ascontiguousarray(x), tets=np.ascontiguousarray(t.astype(np.int32)), on_x0=zeros, on_y0=zeros, gap0=0.0)


@pytest.mark.parametrize("points", [12, 33, 120, 420])
def test_a_fan_assembles_like_the_oracle(points):
    like, dies = upset_case_3d(10.0, 10.0, 2.0, 10.0)
    mesh = _fan(points, like)
    cfg = Forging3DConfig(C=150, N=0.1, M=0.12, eps0=0.01, friction=0.3, ram=10, h=2.0, ds=0.4, size=10.0, tol=1e-6)
    gpu, ora = Forging3DSolver(cfg, mesh, dies), Oracle3D(cfg, mesh, dies)
    gpu.prepare_step()
    ora.prepare_step()
    for name in ("v_node", "g_coef", "kvol"):
        np.testing.assert_array_equal(gpu.array(name), ora.array(name))
    n = len(ora.array("v"))
    v = ora.array("v") + 0.1 * np.sin(np.arange(n))
    for newton in (0, 1):
        eg, pg = gpu.assemble(1, newton, v)
        eo, po = ora.assemble(1, newton, v)
        assert abs(eg / eo - 1) < RTOL_ENERGY and abs(pg / po - 1) < RTOL_ENERGY
        _close(gpu.array("val"), ora.array("val"), RTOL_ELEM, "assembled values")
        _close(gpu.array("r"), ora.array("r"), 1e-11, "residual")
        assert abs(gpu.apply_bc() / ora.apply_bc() - 1) < 1e-12
        _close(gpu.array("val"), ora.array("val"), RTOL_ELEM, "values after BC")
        _close(gpu.array("r"), ora.array("r"), 1e-11, "residual after BC")
    gpu.close()
