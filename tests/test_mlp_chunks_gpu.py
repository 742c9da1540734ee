"""The stop network's training at the edges of its gradient kernel (chunks of 64 samples, four in flight) and of
its gathers, against the NumPy oracle."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import mlp

pytestmark = pytest.mark.gpu


def test_gathers_in_parts_leave_the_weights_and_the_memory(monkeypatch: pytest.MonkeyPatch) -> None:
    """An epoch gathered in parts takes the same steps; the parts, not the epoch, are what it holds beside
    the samples."""
    import torch

    from hnsw_engine_b200 import learned_stop
    from hnsw_engine_b200.learned_stop import StopNetwork

    n, batch = 1_000_037, 4_096
    rng = np.random.default_rng(8)
    X = rng.standard_normal((n, 12), dtype=np.float32)
    y = rng.standard_normal(n, dtype=np.float32)
    weights, peaks = [], []
    for samples in (1 << 22, 3 * batch, 5_000, 1):
        monkeypatch.setattr(learned_stop, "GATHER_SAMPLES", samples, raising=False)
        net = StopNetwork("cuda")
        net.params = torch.from_numpy(mlp.init_params(2)).cuda()
        torch.cuda.empty_cache()
        base = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        net.fit(X, y, epochs=2, batch=batch)
        peaks.append(torch.cuda.max_memory_allocated() - base)
        weights.append(net.params.cpu().numpy())
    for w in weights[1:]:
        np.testing.assert_array_equal(w, weights[0])
    # features, targets and order are 60 bytes a sample, the last epoch's order 8, the kernels' scratch 4; a copy
    # of the features would be 48 more
    assert max(peaks[1:]) < 90 * n
