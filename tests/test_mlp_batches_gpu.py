"""Gradients of the stop network at batch sizes around the 32-sample tiles, against the NumPy oracle."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import mlp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 31, 32, 33, 296 * 32, 296 * 32 + 1, 20_001])
def test_gradients_at_tile_edges(batch: int) -> None:
    import torch

    from hnsw_engine_b200.learned_stop import StopNetwork

    rng = np.random.default_rng(batch)
    X = rng.standard_normal((batch, 12)).astype(np.float32)
    y = rng.standard_normal(batch).astype(np.float32)
    net = StopNetwork("cuda")
    net.params = torch.from_numpy(mlp.init_params(2)).cuda()
    g, loss = net.gradients(X, y)
    p = net.params.cpu().numpy()
    # the tolerance of the training kernels' gradient test (float32 passes over BF16 weights)
    np.testing.assert_allclose(g, mlp.gradients(p, X, y), rtol=2e-3, atol=2e-5)
    assert loss == pytest.approx(mlp.loss(p, X, y), rel=1e-4)
    again, _ = net.gradients(X, y)
    np.testing.assert_array_equal(g, again)  # fixed summation order
