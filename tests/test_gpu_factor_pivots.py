"""Pivots at the edges of the panel kernels: a factorisation names the equation whose pivot is not positive (columns either
side of eight, of a panel and of a super-panel; several trees; both precisions, whose panels are kernels of their
own), takes valid pivots that lie outside the range of its fast reciprocals, and a trailing update of more tiles than
its CTAs take in one go leaves the residual of a backward-stable factorisation.

The matrices are diagonally dominant (condition below 10): the residual is within n eps * 10 of the right-hand side,
6e-12 at the largest n here. A power of two scales every step exactly but the reciprocals, so it keeps that bound.
"""
import ctypes as C
import re

import numpy as np
import pytest

from impressionfea_b200._lib import MatrixNotPositiveDefiniteError
from impressionfea_b200.config import Forging3DConfig
from impressionfea_b200.forging3d import Forging3DSolver, GpuSpdSolver
from impressionfea_b200.meshes import h_for_tets, upset_case_3d
from test_gpu_sweep import _dense, _matrix

pytestmark = pytest.mark.gpu


def _analysed(a):
    n = len(a)
    cols, rows = np.nonzero(a)
    s = GpuSpdSolver()
    s.analyze(n, np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=n))]), rows)
    return s, a[cols, rows]


@pytest.mark.parametrize("shape,bad", [(("dense", 64), b) for b in (0, 7, 8, 62, 63)] + [(("dense", 65), 64), (("dense", 300), 255),
                                       (("dense", 300), 256), (("dense", 300), 299), (("forest", 230), 0), (("forest", 230), 233),
                                       (("forest", 230), 303), (("star", 40), 17), (("star", 40), 330), (("star", 150), 1399)])
@pytest.mark.parametrize("value", [-1.0, 0.0, np.nan])
def test_the_failing_equation_is_named(shape, bad, value):
    a = _matrix(shape)
    if value == 0.0:  # a pivot of zero exactly: nothing else in its row and column, but entries that are stored
        a[bad, a[bad] != 0] = 1e-300
        a[a[:, bad] != 0, bad] = 1e-300
    a[bad, bad] = 1.0
    s, values = _analysed(a)
    a[bad, bad] = value
    cols, rows = np.nonzero(_matrix(shape))
    with pytest.raises(MatrixNotPositiveDefiniteError, match=rf"equation {bad}\."):
        s.factorize(a[cols, rows])
    s.factorize(values)  # and the solver is usable again
    s.close()


@pytest.mark.parametrize("node", [0, 200, 700])
def test_both_precisions_name_the_same_equation(node):
    """A velocity that is not a number at one node: the equations around it have no pivots."""
    h = h_for_tets(15.0, 45.0, 4000)
    mesh, dies = upset_case_3d(15.0, 45.0, h, shut=27.0, seed=9)
    cfg = Forging3DConfig(C=120, N=0.1, M=0.12, eps0=0.01, friction=0.3, ram=50, h=h, ds=0.2, size=45.0, tol=1e-6)
    named = []
    for fp32 in (0, 1):
        s = Forging3DSolver(cfg, mesh, dies)
        s.set_scalar("factor_fp32", fp32)
        s.prepare_step()
        v = s.array("v")
        v[3 * node:3 * node + 3] = np.nan
        s.assemble(1, 1, v)
        s.apply_bc()
        cp, ri = s.pattern()
        diag = s.array("val")[[c0 + int(np.searchsorted(ri[c0:c1], k)) for k, (c0, c1) in enumerate(zip(cp, cp[1:]))]]
        ms = C.c_double()
        with pytest.raises(MatrixNotPositiveDefiniteError) as e:
            s._check(s._L.ifea3d_time_factor_solve(s._h, C.byref(ms)))
        named.append(int(re.search(r"equation (\d+)\.", str(e.value))[1]))
        assert np.isnan(diag[named[-1]])
        s.close()
    assert named[0] == named[1]


@pytest.mark.parametrize("power", [-990, -970, 0, 970, 990])
@pytest.mark.parametrize("n", [7, 64, 200, 700])
def test_pivots_outside_the_fast_reciprocals(n, power):
    a = np.ldexp(_dense(n, n), power)
    s, values = _analysed(a)
    s.factorize(values)
    b = np.random.default_rng(n).standard_normal(n)
    x = s.solve(np.ldexp(b, power))
    s.close()
    assert np.linalg.norm(np.ldexp(a, -power) @ x - b) <= 3e-12 * np.linalg.norm(b)


def test_a_trailing_update_of_several_tiles_a_group():
    n = 2600  # right of the second super-panel 33 x 33 lower tiles: 561, and 128 CTAs take 384 at a time
    a = _dense(n, 3)
    s, values = _analysed(a)
    b = np.random.default_rng(n).standard_normal(n)
    x = []
    for _ in range(2):
        s.factorize(values)
        x.append(s.solve(b))
    s.close()
    assert np.linalg.norm(a @ x[0] - b) <= 6e-12 * np.linalg.norm(b)
    assert np.array_equal(x[0], x[1])
