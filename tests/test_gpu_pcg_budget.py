"""How long the single-precision form tries a reused factor (pcg_budget_now) follows from the mesh, the factorisations'
device time and the counts of PCG calls and iterations, not from the host's clock: a host that waits for every solve
(profile_solves) comes to the same budget. The rates are the solver's own (milliseconds a level of the elimination
tree, and a million matrix entries); two solvers' factorisations differ in device time by a few per cent, so their
budgets may by one in twenty and a rounding."""
import pytest

from impressionfea_b200.config import Forging3DConfig
from impressionfea_b200.forging3d import Forging3DSolver
from impressionfea_b200.meshes import h_for_tets, upset_case_3d

pytestmark = pytest.mark.gpu
LEVEL_MS, ENTRY_MS, SCALE = 0.0193, 0.0424, 2.0


def _solver(tets, waits):
    h = h_for_tets(15.0, 45.0, tets)
    mesh, dies = upset_case_3d(15.0, 45.0, h, shut=27.0, seed=6)
    cfg = Forging3DConfig(C=120, N=0.1, M=0.12, eps0=0.01, friction=0.3, ram=50, h=h, ds=0.2, size=45.0, tol=1e-6)
    s = Forging3DSolver(cfg, mesh, dies)
    s.set_scalar("factor_fp32", 1)
    s.set_scalar("profile_solves", waits)
    return s


@pytest.mark.parametrize("tets", [4000, 16000, 40000])
def test_budget_does_not_follow_the_hosts_clock(tets):
    budgets = []
    for waits in (0, 1):
        s = _solver(tets, waits)
        for _ in range(2):
            s.step()
            its, calls, facts = s.scalar("lin_its"), s.scalar("pcg_calls"), s.scalar("n_fact")
            assert its > 0 and facts > 0 and calls >= facts  # (every factorisation here is refined)
            solve_ms = LEVEL_MS * s.scalar("levels") + ENTRY_MS * 1e-6 * s.scalar("nnz")
            want = SCALE * (s.scalar("factor_gpu_ms") / facts) / (solve_ms * (its + 2 * calls) / its)
            assert abs(s.scalar("pcg_budget_now") - min(120, max(15, int(want)))) <= (abs(want - round(want)) < 1e-9)
        budgets.append(s.scalar("pcg_budget_now"))
        s.close()
    assert abs(budgets[0] - budgets[1]) <= 1 + 0.05 * budgets[0]
