"""The solve's persistent sweep at the shapes where its task list changes form: a single small front, a single wide one
either side of the row where its right-hand side is assembled separately, several trees, and a parent that many
children update. Compared with a dense FP64 solve; the matrices are diagonally dominant (condition below 10), so a
backward-stable solve is within n * eps * 10 < 3e-12 of it in norm."""
import numpy as np
import pytest

from impressionfea_b200.forging3d import GpuSpdSolver

pytestmark = pytest.mark.gpu


def _dense(n, seed):
    a = np.random.default_rng(seed).uniform(-1, 1, (n, n))
    a = (a + a.T) / 2
    return a / np.abs(a).sum(1).max() + np.diag(np.full(n, 1.5))


def _matrix(shape):
    kind, n = shape
    if kind == "dense":
        return _dense(n, n)
    if kind == "forest":  # independent dense blocks of unequal size
        sizes = [n, 3, 70, 1, n // 2]
        a = np.zeros((sum(sizes),) * 2)
        k = 0
        for q, s in enumerate(sizes):
            a[k:k + s, k:k + s] = _dense(s, q)
            k += s
        return a
    # star: eight dense leaves, each coupled to the same separator (a front row with updates of many children)
    leaf, sep, m = n, 200, 8
    a = np.diag(np.full(m * leaf + sep, 3.0))
    rng = np.random.default_rng(n)
    for q in range(m):
        k = q * leaf
        a[k:k + leaf, k:k + leaf] += _dense(leaf, q)
        c = rng.uniform(-1, 1, (leaf, sep)) / (m * leaf)
        a[k:k + leaf, -sep:] = c
        a[-sep:, k:k + leaf] = c.T
    a[-sep:, -sep:] += _dense(sep, 99)
    return a


@pytest.mark.parametrize("shape", [("dense", 1), ("dense", 64), ("dense", 65), ("dense", 191), ("dense", 192), ("dense", 257),
                                   ("dense", 1024), ("dense", 1025), ("dense", 1300), ("forest", 230), ("star", 40), ("star", 150)])
def test_sweep_matches_a_dense_solve_and_repeats_bit_for_bit(shape):
    a = _matrix(shape)
    n = len(a)
    cols, rows = np.nonzero(a)  # symmetric: row-major order of a is its CSC order
    ptr = np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=n))])
    s = GpuSpdSolver()
    s.analyze(n, ptr, rows)
    s.factorize(a[cols, rows])
    rng = np.random.default_rng(7)
    for _ in range(3):
        b = rng.standard_normal(n)
        x = s.solve(b)
        ref = np.linalg.solve(a, b)
        assert np.linalg.norm(x - ref) <= 3e-12 * np.linalg.norm(ref)
        assert np.array_equal(x, s.solve(b))
    s.close()
