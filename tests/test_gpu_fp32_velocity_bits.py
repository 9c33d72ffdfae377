"""A single-precision form's whole velocity solution keeps its bits: assembly (energies among it), factor, sweeps and
conjugate gradients in the order of sums that the digests were taken with (level-by-level sweeps, dot products and
energies by launches of their own). On meshes small enough that a reused factor's budget is the reference's 15
iterations, so that no measured time is in the result."""
import hashlib

import numpy as np
import pytest

from impressionfea_b200.config import Forging3DConfig
from impressionfea_b200.forging3d import Forging3DSolver
from impressionfea_b200.meshes import gear_blank_case_3d, h_for_tets, upset_case_3d

pytestmark = pytest.mark.gpu


def solution(die, tets, seed):
    """Digests: the assembled system's energy and power; the velocities of the first increment and of the second."""
    if die == "gear":
        h = h_for_tets(20.0, 50.0, tets)
        mesh, dies = gear_blank_case_3d(h, R=20.0, H=50.0, ramp=4.0, seed=seed)
        ds, size = mesh.gap0 / 200, 50.0
    else:
        h = h_for_tets(15.0, 45.0, tets)
        mesh, dies = upset_case_3d(15.0, 45.0, h, shut=27.0, seed=seed)
        ds, size = 0.2, 45.0
    cfg = Forging3DConfig(C=120, N=0.1, M=0.12, eps0=0.01, friction=0.3, ram=50, h=h, ds=ds, size=size, tol=1e-6)
    s = Forging3DSolver(cfg, mesh, dies)
    s.set_scalar("factor_fp32", 1)
    s.prepare_step()
    out = [np.array(s.assemble(1, 1))]
    for _ in range(2):
        s.step()
        out.append(s.array("vg"))
    assert s.scalar("pcg_budget_now") == 15
    s.close()
    return tuple(hashlib.sha256(a.tobytes()).hexdigest()[:16] for a in out)


CASES = [
    ("flat", 2000, 1, ("38f648b9770d8902", "24b83de9b195cd2f", "705d804f56849b28")),
    ("gear", 2500, 2, ("9b554a59af2b54e7", "7855b6e16d5c8079", "f22c5442738819b7")),
    ("flat", 3000, 3, ("e8eda8deaa16020c", "de1bbb257ff51aea", "7bbf84101fab19ee")),
]


@pytest.mark.parametrize("die,tets,seed,digests", CASES)
def test_fp32_velocity_bits(die, tets, seed, digests):
    assert solution(die, tets, seed) == digests
