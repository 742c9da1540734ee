"""Query statistics and filter bitmaps computed on the GPU against NumPy."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(n: int, locality: bool):
    from hnsw_engine_b200.engine import DeviceGraph

    rng = np.random.default_rng(n)
    arrays = {
        "vectors": rng.standard_normal((n, 8)).astype(np.float32), "levels": np.zeros(n, np.int64),
        "links0": rng.integers(0, n, (n, 33)).astype(np.int32), "count0": np.full(n, 8, np.int32),
        "upper_offset": np.full(n, -1, np.int64), "links_up": np.zeros((0, 17), np.int32),
        "count_up": np.zeros(0, np.int32),
    }
    return DeviceGraph(arrays, 0, 0, "l2", locality=locality)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 1000, 65_537])
@pytest.mark.parametrize("locality", [False, True])
def test_bitmap_of_a_mask(n: int, locality: bool) -> None:
    from hnsw_engine_b200.engine import pack_mask

    g = _graph(n, locality)
    rng = np.random.default_rng(1)
    for mask in (rng.random(n) < 0.3, np.ones(n, bool), np.zeros(n, bool)):
        np.testing.assert_array_equal(g._device_bitmap(mask).cpu().numpy().view(np.uint32),
                                      pack_mask(g.internal_mask(mask)))
    strided = np.zeros(2 * n, bool)[::2]  # not contiguous
    strided[: n // 2 + 1] = True
    strided.setflags(write=False)
    np.testing.assert_array_equal(g._device_bitmap(strided).cpu().numpy().view(np.uint32),
                                  pack_mask(g.internal_mask(strided)))


@pytest.mark.parametrize("count", [1, 31, 257, 4096, 100_003, 3_000_001])
def test_device_stats(count: int) -> None:
    import torch

    from hnsw_engine_b200 import _lib

    g = _graph(4, False)
    rng = np.random.default_rng(count)
    values = rng.integers(-300, 70_000, count).astype(np.float64)
    for dtype in (torch.float32, torch.float64):
        flags, st = g.device_stats(torch.from_numpy(values).to("cuda", dtype))
        assert (flags, st.finite, st.integer, st.min, st.max) == (0, 1, 1, values.min(), values.max())
    at = int(rng.integers(count))
    x = values.copy()
    x[at] += 0.5
    flags, st = g.device_stats(torch.from_numpy(x).cuda())
    assert flags == _lib.NOT_INTEGER and st.finite and not st.integer
    for bad in (np.nan, np.inf, -np.inf):
        x[at] = bad
        flags, st = g.device_stats(torch.from_numpy(x.astype(np.float32)).cuda())
        assert flags & _lib.NOT_FINITE and not st.finite
    # float64 values beyond float32, and a zero norm
    x[at] = 1e300
    rows = torch.from_numpy(x).cuda().to(torch.float32)
    norms = torch.ones(count, dtype=torch.float64, device="cuda")
    norms[at] = 0.0
    flags, _ = g.device_stats(torch.from_numpy(x).cuda(), rows, norms)
    assert flags == _lib.ROWS_NOT_FINITE | _lib.ZERO_NORM


@pytest.mark.parametrize("metric", ["l2", "ip", "cosine"])
def test_code_space_queries(metric: str) -> None:
    import torch

    from hnsw_engine_b200.quantization import QuantizedIndex, ScalarQuantizer

    rng = np.random.default_rng(7)
    for nq, dim in ((0, 5), (1, 1), (3, 33), (70, 127), (1000, 100)):
        q = rng.standard_normal((nq, dim)).astype(np.float32)
        qi = QuantizedIndex.__new__(QuantizedIndex)
        qi.quantizer = ScalarQuantizer(rng.standard_normal(dim), 0.037)
        got = qi.transform_device(torch.from_numpy(q).cuda(), metric)
        np.testing.assert_array_equal(got.cpu().numpy(), qi.quantizer.transform_queries(q, metric))


def test_counters_of_mixed_searches() -> None:
    """The running counters over host, device, filtered and code-space batches and single queries are
    the sums of the same batches' per-query counters."""
    import torch

    from conftest import load_golden, mix10k_arrays
    from hnsw_engine_b200 import HNSWIndex, QuantizedIndex

    arrays, ep, ml = mix10k_arrays()
    index = HNSWIndex.from_arrays(arrays, ep, ml, dim=128, metric="l2", M=16)
    g = index.device_graph
    q = load_golden("search_mix10k")["queries"][:300]
    mask = np.random.default_rng(3).random(10_000) < 0.4
    want = np.zeros(2, np.int64)
    for ef in (10, 64):
        for kw in ({}, {"allowed": mask}):
            ids, dists, ctr = g.search(q, 10, ef, **kw)
            want += ctr.sum(0).cpu().numpy()
            got = index.batch_search(q, 10, ef, filter=kw.get("allowed"))
            np.testing.assert_array_equal(got[0], ids.cpu().numpy())
            np.testing.assert_array_equal(got[1], dists.cpu().numpy())
    dev = index.batch_search(torch.from_numpy(q).cuda(), 10, 64)
    want += g.search(q, 10, 64)[2].sum(0).cpu().numpy()
    assert dev[0].is_cuda and dev[1].is_cuda
    one = index.search(q[0], 10, 64)
    ids, dists, ctr = g.search(q[:1], 10, 64)
    np.testing.assert_array_equal(one[0], ids[0].cpu().numpy())
    np.testing.assert_array_equal(one[1], dists[0].cpu().numpy())
    want += ctr.sum(0).cpu().numpy()
    assert (index.distance_computations, index.hops) == tuple(want)
    index.reset_counters()
    assert (index.distance_computations, index.hops) == (0, 0)
    qi = QuantizedIndex(index)
    qi.batch_search(q, 10, 64, rerank=32)
    code_q = qi.quantizer.transform_queries(q, "l2")
    ctr = g.search(code_q, 10, 64, use_codes=True, k_search=32, rerank_queries=q)[2]
    assert (index.distance_computations, index.hops) == tuple(ctr.sum(0).cpu().numpy())
