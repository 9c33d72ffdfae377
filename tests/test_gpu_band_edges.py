"""The band kernel at the edges of its plan: bands narrower than its eight-column block, either side of a warp of rows,
the widest one whose triangle fits shared memory and the first that does not, systems that end inside a block or are
smaller than the window; and values outside the range of its corrected quotients (tiny and huge scales, exact powers of
two, zeros of either sign), which take plain divisions. Bit for bit against the reference's loop."""
import numpy as np
import pytest

from impressionfea_b200 import _lib
from impressionfea_b200.forging2d import band_factor_solve
from oracle import OracleBand

pytestmark = pytest.mark.gpu


def _spd_band(n, b, seed):
    rng = np.random.default_rng(seed)
    a = np.zeros((n, b + 1))
    for i in range(n):
        lo = max(0, i - b)
        a[i, lo - i + b:b] = rng.random(i - lo) - 0.5
        a[i, b] = 2.0 * b + 1.0 + rng.random()
    return a, rng.standard_normal(n)


def _check(a, rhs, b):
    n = len(rhs)
    ob = OracleBand(n, b)
    ob.set_data(a.ravel())
    assert ob.factorize()[0] == -1
    x_ref = ob.solve(rhs)
    low, x = band_factor_solve(a.ravel(), b, rhs)
    np.testing.assert_array_equal(low, ob.data())
    np.testing.assert_array_equal(x, x_ref)


@pytest.mark.parametrize("n,b", [(1, 0), (9, 0), (64, 2), (77, 6), (77, 7), (200, 8), (201, 14), (202, 23), (203, 24), (301, 38),
                                 (303, 39), (20, 19), (150, 149), (190, 186), (700, 185), (701, 187), (702, 188), (703, 189)])
def test_band_shapes(n, b):
    _check(*_spd_band(n, b, 7 * n + b), b)


@pytest.mark.parametrize("values", ["tiny", "huge", "powers", "zeros", "mixed"])
def test_band_values_outside_the_corrected_quotients(values):
    n, b = 300, 40
    a, rhs = _spd_band(n, b, 3)
    rng = np.random.default_rng(4)
    if values == "tiny":
        a *= 1e-200
    elif values == "huge":
        a *= 1e200
    elif values == "powers":  # diagonal 4^k, so that roots are powers of two
        a[:, :b] *= 1e-3
        a[:, b] = 4.0 ** rng.integers(3, 6, n)
    elif values == "zeros":
        a[:, :b][rng.random((n, b)) < 0.7] = 0.0
        a[50, :] = 0.0
        a[50, b] = 1.0
        rhs[rng.random(n) < 0.5] = -0.0
    else:
        a[:, :b][rng.random((n, b)) < 0.2] *= 1e-280
    _check(a, rhs, b)


@pytest.mark.parametrize("row,value", [(0, -1.0), (7, 0.0), (8, np.nan), (123, -5.0), (299, -1e9)])
def test_band_reports_the_first_failing_row(row, value):
    n, b = 300, 40
    a, rhs = _spd_band(n, b, 5)
    a[row, b] = value
    with pytest.raises(_lib.MatrixNotPositiveDefiniteError, match=f"equation {row} "):
        band_factor_solve(a.ravel(), b, rhs)
