"""The single-precision factor's solutions keep their bits. The factor is a preconditioner: what its conjugate gradients
return within their tolerance follows its last bits, and an unconverged Newton iteration carries that on (velocities of
60k tets moved by 4e-8 when the sweeps summed in another order). The digests are those of the level-by-level
sweeps that the order of sums comes from, on the same assembled systems: one-CTA fronts of every size, wide fronts,
super-panels on the tensor cores, and fronts of several panels kept on one CTA."""
import ctypes as C
import hashlib

import pytest

from impressionfea_b200.config import Forging3DConfig
from impressionfea_b200.forging3d import Forging3DSolver
from impressionfea_b200.meshes import h_for_tets, upset_case_3d

pytestmark = pytest.mark.gpu


def _digest(a):
    return hashlib.sha256(a.tobytes()).hexdigest()[:16]


def solution(tets, seed, options):
    """Digests of an assembled upsetting system and of its plain FP32 solution (factorise, solve, no refinement)."""
    h = h_for_tets(15.0, 45.0, tets)
    mesh, dies = upset_case_3d(15.0, 45.0, h, shut=27.0, seed=seed)
    cfg = Forging3DConfig(C=120, N=0.1, M=0.12, eps0=0.01, friction=0.3, ram=50, h=h, ds=0.2, size=45.0, tol=1e-6)
    s = Forging3DSolver(cfg, mesh, dies)
    s.set_scalar("factor_fp32", 1)
    for name, value in options.items():
        s.set_scalar(name, value)
    s.prepare_step()
    s.assemble(1, 1)
    s.apply_bc()
    ms = C.c_double()
    s._check(s._L.ifea3d_time_factor_solve(s._h, C.byref(ms)))
    out = _digest(s.array("val")), _digest(s.array("dv"))
    s.close()
    return out


CASES = [
    (2000, 1, {}, "06ef07013876ca2c", "66bb0ffc1f6fed18"),
    (9000, 2, {"tc_rows": 256}, "8e2a69a3eabb7241", "70f671f169ef694d"),
    (9000, 2, {"wide_front_rows": 500}, "8e2a69a3eabb7241", "00e5d1b15dfc6a96"),
    (24000, 3, {}, "c24895eda334d415", "26607f5cc525cfd1"),
]


@pytest.mark.parametrize("tets,seed,options,system,digest", CASES)
def test_fp32_solution_bits(tets, seed, options, system, digest):
    val, dv = solution(tets, seed, options)
    assert val == system, "another system than the digests were taken on"
    assert dv == digest
