"""How long the single-precision form tries a reused factor (pcg_budget_now) follows from the mesh, the factorisations'
device time and the counts of PCG calls and iterations, not from the host's clock: the rule gives the budget as well
on a host that waits for every solve (profile_solves). The rates are the solver's own (milliseconds a level of the
elimination tree, the more the less of the factor stays in L2, a factor entry, and once for a context's first solve)."""
import pytest

from impressionfea_b200.config import Forging3DConfig
from impressionfea_b200.forging3d import Forging3DSolver
from impressionfea_b200.meshes import h_for_tets, upset_case_3d

pytestmark = pytest.mark.gpu
LEVEL_MS, COLD_MS, ENTRY_MS, FIRST_MS, SCALE = 0.0209, 0.0091, 2.25e-9, 0.25, 2.0


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
    for waits in (0, 1):
        s = _solver(tets, waits)
        for _ in range(2):
            s.step()
            its, calls, facts = s.scalar("lin_its"), s.scalar("pcg_calls"), s.scalar("n_fact")
            assert its > 0 and facts > 0 and calls >= facts  # (every factorisation here is refined)
            entries = s.scalar("factor_nnz")
            cold = min(1, max(0, (entries - 5e6) / 7e6))
            solve_ms = s.scalar("levels") * (LEVEL_MS + cold * COLD_MS) + entries * ENTRY_MS
            want = SCALE * (s.scalar("factor_gpu_ms") / facts) / ((solve_ms * (its + 2 * calls) + FIRST_MS) / its)
            assert abs(s.scalar("pcg_budget_now") - min(120, max(15, int(want)))) <= (abs(want - round(want)) < 1e-9)
        s.close()
