"""The factorisation's tiles where they end: fronts either side of a panel (64), of a half block (32), of a super-panel
(256) and of the next one's columns; several unequal fronts in one sequence of tiles; and a front whose trailing update
runs beside the next super-panel's panels (more than 512 pivot columns).

The matrices are diagonally dominant (condition below 10): a backward-stable factorisation's residual is within
n eps * 10 of the right-hand side, 3e-12 at the largest n here.
"""
import numpy as np
import pytest

from impressionfea_b200.forging3d import GpuSpdSolver
from test_gpu_sweep import _dense, _matrix

pytestmark = pytest.mark.gpu


def _solve(a):
    n = len(a)
    cols, rows = np.nonzero(a)
    s = GpuSpdSolver()
    s.analyze(n, np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=n))]), rows)
    s.factorize(a[cols, rows])
    b = np.random.default_rng(n).standard_normal(n)
    x = s.solve(b)
    s.factorize(a[cols, rows])
    again = s.solve(b)
    s.close()
    return b, x, again


@pytest.mark.parametrize("shape", [("dense", n) for n in (1, 7, 8, 9, 31, 33, 63, 64, 65, 95, 128, 255, 256, 257, 319, 321, 513, 577, 900)]
                         + [("forest", 700), ("star", 300)])
def test_factor_solves_and_repeats_bit_for_bit(shape):
    a = _matrix(shape)
    b, x, again = _solve(a)
    assert np.linalg.norm(a @ x - b) <= 3e-12 * np.linalg.norm(b)
    assert np.array_equal(x, again)


@pytest.mark.parametrize("n,bad", [(64, 0), (64, 63), (65, 64), (300, 7), (300, 8), (300, 299)])
def test_a_pivot_that_is_not_positive_is_found(n, bad):
    a = _dense(n, n)
    a[bad, bad] = -1.0
    with pytest.raises(Exception, match="not positive definite"):
        _solve(a)
