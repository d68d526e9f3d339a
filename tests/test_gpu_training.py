"""The training kernels at batch sizes that leave their splits uneven (32
samples per block, four row sets of 64-row steps), and the standardisation,
against the FP64 CPU restatement."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_learned import he_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 31, 33, 127, 255, 256, 257, 1021, 4099])
def test_gradient_at_uneven_batches(bh, n):
    from oracle import mlp
    rng = np.random.default_rng(n)
    p = he_params(rng)
    X = rng.normal(0, 1, (n, 8)).astype(np.float32)
    T = rng.normal(0, 1, n).astype(np.float32)
    loss_gpu, g_gpu = bh.mlp_gradient(p, X, T)
    loss_cpu, g_cpu = mlp.loss_and_grad(p, X, T)
    # FP32 against FP64 accumulation with the same BF16 roundings; a rounding
    # that falls the other way (one in 2^15 activations) moves one sample's
    # terms by 2^-8, so few samples get the widest bound: 1e-4 on the loss and
    # 2e-3 on the gradient from 2,000 samples on, 2^-8 and 2e-2 for one.
    few = n < 2000
    assert abs(loss_gpu - loss_cpu) <= (2.0 ** -8 if few else 1e-4) * loss_cpu + 1e-7
    assert np.linalg.norm(g_gpu - g_cpu) <= (2e-2 if few else 2e-3) * np.linalg.norm(g_cpu)


@pytest.mark.parametrize("n,batch", [(16, 16), (100, 33), (1000, 4096), (5003, 257)])
def test_training_is_repeatable_and_scales(bh, n, batch):
    rng = np.random.default_rng(n)
    F = (rng.normal(0, 1, (n, 8)) * np.arange(1, 9) + 3).astype(np.float32)
    L = (F[:, 0] - 0.5 * F[:, 1]).astype(np.float32)
    a = bh.mlp_train(F, L, epochs=2, batch=batch, seed=5)
    b = bh.mlp_train(F, L, epochs=2, batch=batch, seed=5)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
    F64 = F.astype(np.float64)
    mean, std = F64.mean(0), np.sqrt(np.maximum((F64 ** 2).mean(0) - F64.mean(0) ** 2, 1e-12))
    scale = a[1]
    np.testing.assert_allclose(scale[:8], mean, rtol=2e-7, atol=1e-6)
    np.testing.assert_allclose(scale[8:16], 1.0 / std, rtol=1e-6)
    z = (F - scale[:8]) * scale[8:16]
    assert np.array_equal(scale[16:24], z.min(0)) and np.array_equal(scale[24:32], z.max(0))
    np.testing.assert_allclose(scale[32:], [L.astype(np.float64).mean(), L.astype(np.float64).std()], rtol=2e-6,
                               atol=1e-6)
    assert np.all(np.isfinite(a[2]))
