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


@pytest.mark.parametrize("batch", [63, 64, 65, 128, 192, 193, 256, 257, 320])
def test_gradients_at_chunk_edges(batch: int) -> None:
    """Around the first whole chunk, and where a chunk's place in shared memory is used again; rows on
    16-byte boundaries and on 4-byte ones give the same bits, in scratch of just the stated size."""
    import torch

    from hnsw_engine_b200 import _lib

    rng = np.random.default_rng(batch)
    X = rng.standard_normal((batch, 12)).astype(np.float32)
    y = rng.standard_normal(batch).astype(np.float32)
    p = mlp.init_params(2)
    lib = _lib.load()
    floats = int(lib.hnsw_b200_mlp_scratch_bytes(batch)) // 4
    assert floats == batch * (4 * 64 + 1)
    got = []
    for shift in (0, 1, 3):
        rows = torch.zeros(batch * 12 + 4, device="cuda")
        rows[shift : shift + batch * 12] = torch.from_numpy(X.ravel()).cuda()
        params = torch.from_numpy(p).cuda()
        targets = torch.from_numpy(y).cuda()
        scratch = torch.full((shift + floats + 8,), 7.0, device="cuda")
        grads, loss = torch.empty(p.size, device="cuda"), torch.zeros(1, device="cuda")
        stream = torch.cuda.current_stream().cuda_stream
        _lib.check(lib.hnsw_b200_mlp_gradients(
            params.data_ptr(), rows[shift:].data_ptr(), targets.data_ptr(), batch, scratch[shift:].data_ptr(),
            grads.data_ptr(), loss.data_ptr(), stream))
        got.append(grads.cpu().numpy())
        assert loss.item() == pytest.approx(mlp.loss(p, X, y), rel=1e-4)
        assert (scratch[shift + floats :] == 7.0).all() and (scratch[:shift] == 7.0).all()
    # the tolerance of the training kernels' gradient test (float32 passes over BF16 weights)
    np.testing.assert_allclose(got[0], mlp.gradients(p, X, y), rtol=2e-3, atol=2e-5)
    np.testing.assert_array_equal(got[1], got[0])
    np.testing.assert_array_equal(got[2], got[0])
