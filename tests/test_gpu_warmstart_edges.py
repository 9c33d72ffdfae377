"""The network's fused passes where their tiles end: one row, a row on either side of a 128-row tile, one slice of the
weight gradients (512 rows), a slice that is not full, the largest batch; and training that shuffles ahead.

Tolerances as in test_gpu_warmstart.py: against the CPU network that rounds to bfloat16 where the GPU stores it only
the order of FP32 sums differs (relative 2e-3 in outputs and gradients).
"""
import numpy as np
import pytest

import mlp_ref
from impressionfea_b200.warmstart import WarmStartNetwork
from test_gpu_warmstart import _net, _random_params, _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 19000])
def test_inference_rows(rows):
    p = _random_params(21)
    x = np.random.default_rng(rows).standard_normal((rows, mlp_ref.NIN)).astype(np.float32)
    net = _net(params=p)
    y = net.forward(x)
    net.close()
    want, _ = mlp_ref.forward(p.astype(np.float64), x.astype(np.float64), bf16=True)
    assert y.shape == want.shape and _rel(y, want) < 2e-3


@pytest.mark.parametrize("rows", [128, 512, 640, 8192])
def test_gradient_rows(rows):
    rng = np.random.default_rng(rows)
    p = _random_params(22)
    x = rng.standard_normal((rows, mlp_ref.NIN)).astype(np.float32)
    t = rng.standard_normal((rows, mlp_ref.NOUT)).astype(np.float32)
    net = _net(params=p)
    loss, g = net.gradients(x, t)
    net.close()
    want_loss, want = mlp_ref.loss_and_gradients(p.astype(np.float64), x.astype(np.float64), t.astype(np.float64), bf16=True)
    assert abs(loss / want_loss - 1) < 1e-3
    k = 0
    for name, shape in mlp_ref.SHAPES:
        n = int(np.prod(shape))
        assert _rel(g[k:k + n], want[k:k + n]) < 2e-3, name
        k += n


@pytest.mark.parametrize("samples,batch", [(100, 128), (4095, 640), (4096, 640), (9000, 8192)])
def test_training_is_reproducible(samples, batch):
    """Below and above the size from which the next order is made on a second thread; batches larger than the set."""
    rng = np.random.default_rng(samples)
    x = rng.standard_normal((samples, mlp_ref.NIN)).astype(np.float32)
    t = np.sin(x[:, :mlp_ref.NOUT]).astype(np.float32)
    runs = []
    for _ in range(2):
        net = WarmStartNetwork(23)
        net.add_samples(x, t)
        net.fit_normalisation()
        loss = net.train(steps=30, batch=batch, lr=1e-3, seed=3)
        runs.append((loss, net.params()))
        net.close()
    assert runs[0][0] == runs[1][0] and np.isfinite(runs[0][0])
    np.testing.assert_array_equal(runs[0][1], runs[1][1])
