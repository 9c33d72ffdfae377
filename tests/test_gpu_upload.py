"""The SPD solver's values from host arrays either side of the size from which threads stage them (8 MiB), with a last
chunk that is not full, and an array that changes as soon as the call returns. Tolerance as in test_gpu_sweep.py."""
import numpy as np
import pytest

from impressionfea_b200.forging3d import GpuSpdSolver
from test_gpu_sweep import _dense

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1023, 1024, 1025, 1449])
def test_factorize_takes_the_whole_array(n):
    a = _dense(n, n)
    assert np.all(a != 0)
    s = GpuSpdSolver()
    s.analyze(n, np.arange(n + 1) * n, np.tile(np.arange(n), n))
    b = np.random.default_rng(n).standard_normal(n)
    for k in range(3):
        m = a + k * np.eye(n)
        values = m.reshape(-1).copy()  # symmetric: row-major order is its CSC order
        s.factorize(values)
        values[:] = 0.0
        assert np.linalg.norm(m @ s.solve(b) - b) <= 3e-12 * np.linalg.norm(b)
    s.close()
