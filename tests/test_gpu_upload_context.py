"""The staged upload in a host's own CUDA context (cuCtxCreate): its copying threads work in that context, and the
caller's thread is left in it. In a process of its own, whose only context that is. And from a thread that has made no
CUDA call before."""
import subprocess
import sys
import threading

import numpy as np
import pytest

from impressionfea_b200.forging3d import GpuSpdSolver
from test_gpu_sweep import _dense

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes as C
import numpy as np
cu = C.CDLL("libcuda.so.1")
def ok(status):
    assert status == 0, status
ok(cu.cuInit(0))
dev, ctx, now = C.c_int(), C.c_void_p(), C.c_void_p()
ok(cu.cuDeviceGet(C.byref(dev), 0))
ok(cu.cuCtxCreate_v2(C.byref(ctx), 0, dev))
from impressionfea_b200.forging3d import GpuSpdSolver
n = {n}
rng = np.random.default_rng(1)
a = rng.uniform(-1, 1, (n, n))
a = (a + a.T) / (4 * n) + 1.5 * np.eye(n)
s = GpuSpdSolver()
s.analyze(n, np.arange(n + 1) * n, np.tile(np.arange(n), n))
b = rng.standard_normal(n)
for _ in range(2):
    s.factorize(a.reshape(-1))
    ok(cu.cuCtxGetCurrent(C.byref(now)))
    assert now.value == ctx.value, "the caller's thread was left in another context"
    assert np.linalg.norm(a @ s.solve(b) - b) <= 3e-12 * np.linalg.norm(b)
s.close()
"""


@pytest.mark.parametrize("n", [600, 1200])  # 2.9 and 11.5 MB of values: below and above the staged upload's least size
def test_factorize_keeps_the_callers_context(n):
    p = subprocess.run([sys.executable, "-c", CHILD.format(n=n)], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]


def test_factorize_from_a_new_thread():
    n = 1200
    a, b, x = _dense(n, n), np.random.default_rng(2).standard_normal(n), []
    s = GpuSpdSolver()
    s.analyze(n, np.arange(n + 1) * n, np.tile(np.arange(n), n))

    def work():
        s.factorize(a.reshape(-1))
        x.append(s.solve(b))

    t = threading.Thread(target=work)
    t.start()
    t.join()
    s.close()
    assert np.linalg.norm(a @ x[0] - b) <= 3e-12 * np.linalg.norm(b)
