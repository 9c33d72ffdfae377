"""A solve whose waits run out (limit zero: a tile that is not ready when it is looked at gives up) ends, is reported as
what it is in both precisions, and leaves the solver usable: the next solve has the bits of one that never gave up."""
import ctypes as C

import numpy as np
import pytest

from impressionfea_b200._lib import EngineUnavailableError
from impressionfea_b200.config import Forging3DConfig
from impressionfea_b200.forging3d import Forging3DSolver
from impressionfea_b200.meshes import h_for_tets, upset_case_3d

pytestmark = pytest.mark.gpu


def _solver(fp32):
    h = h_for_tets(15.0, 45.0, 4000)
    mesh, dies = upset_case_3d(15.0, 45.0, h, shut=27.0, seed=8)
    cfg = Forging3DConfig(C=120, N=0.1, M=0.12, eps0=0.01, friction=0.3, ram=50, h=h, ds=0.2, size=45.0, tol=1e-6)
    s = Forging3DSolver(cfg, mesh, dies)
    s.set_scalar("factor_fp32", fp32)
    s.prepare_step()
    return s


def _factor_solve(s):
    ms = C.c_double()
    s._check(s._L.ifea3d_time_factor_solve(s._h, C.byref(ms)))
    return s.array("dv")


@pytest.mark.parametrize("fp32", [0, 1])
def test_the_solve_after_one_that_gave_up(fp32):
    s = _solver(fp32)
    s.assemble(1, 1)
    s.apply_bc()
    want = _factor_solve(s)
    for _ in range(2):
        s.set_scalar("solve_wait_ms", 0)
        with pytest.raises(EngineUnavailableError, match="timed out"):
            _factor_solve(s)
        s.set_scalar("solve_wait_ms", 2000)
        np.testing.assert_array_equal(_factor_solve(s), want)
    s.close()


@pytest.mark.parametrize("fp32", [0, 1])
def test_a_velocity_solution_reports_the_wait(fp32):
    clean, s = _solver(fp32), _solver(fp32)
    clean.solve_velocity()
    for reused in (0, 1):  # with a new factor, then (the second time round) with a kept one
        if reused:
            s.prepare_step()
            s.solve_velocity()
            s.prepare_step()
        s.set_scalar("solve_wait_ms", 0)
        with pytest.raises(EngineUnavailableError, match="timed out"):
            s.solve_velocity()
        s.set_scalar("solve_wait_ms", 2000)
    s.prepare_step()
    s.solve_velocity()
    v, want = s.array("v"), clean.array("v")
    assert np.linalg.norm(v - want) <= 1e-4 * np.linalg.norm(want)  # (both converged to 1e-6 in the update's norm)
    s.step()  # and an increment runs
    s.close()
    clean.close()
