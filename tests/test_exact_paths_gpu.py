"""The exact k-NN's branches by size, against the NumPy oracle: query operand resident or streamed
with the rows, row and query counts around the tiles, results gathered and sorted or inserted, and
a sampled threshold that turns out too low."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import exact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nq,dim,k", [
    (255, 1, 16, 3),        # less than a tile of rows, one query
    (257, 129, 64, 1),      # one row and one query past a tile
    (20_000, 130, 896, 7),  # seven chunks of K: the last size with the query operand resident
    (6_000, 33, 897, 7),    # eight: streamed
    (5_000, 5, 20, 2_000),  # too many results to gather in shared memory: inserted
])
def test_byte_rows_by_size(n: int, nq: int, dim: int, k: int) -> None:
    from hnsw_engine_b200.exact_knn import exact_search

    rng = np.random.default_rng(n + dim)
    data = rng.integers(0, 256, (n, dim)).astype(np.uint8)
    queries = rng.integers(0, 256, (nq, dim)).astype(np.uint8)
    for metric in ("l2", "ip"):
        ids, dists = exact_search(data, queries, k, metric)
        o_ids, o_d = exact.exact_search(data, queries, k, metric)
        np.testing.assert_array_equal(ids, o_ids, err_msg=metric)
        np.testing.assert_array_equal(dists, o_d, err_msg=metric)


@pytest.mark.parametrize("n,nq,dim,k", [
    (300, 3, 5, 300),         # every row a result
    (9_000, 140, 129, 10),    # nine chunks of K: streamed; values beyond a lane's registers
    (4_000, 20, 255, 10),     # products of a partial block of dimensions
    (4_000, 20, 256, 10),     # the first width scored by the whole warp
    (3_000, 2, 24, 2_500),    # inserted
])
def test_float_rows_by_size(n: int, nq: int, dim: int, k: int) -> None:
    from hnsw_engine_b200.exact_knn import exact_search

    rng = np.random.default_rng(n + dim)
    data = rng.standard_normal((n, dim)).astype(np.float32)
    queries = rng.standard_normal((nq, dim)).astype(np.float32)
    for metric in ("l2", "ip", "cosine"):
        ids, dists, st = exact_search(data, queries, k, metric, return_stats=True)
        o_ids, o_d = exact.exact_search(data, queries, k, metric)
        # float64 sums of dim terms in another order: dim roundings of the largest partial sum
        scale = 1.0 if metric == "cosine" else float(np.abs(o_d).max())
        np.testing.assert_allclose(dists, o_d, rtol=0, atol=dim * 2.0**-52 * scale, err_msg=metric)
        assert (ids == o_ids).mean() > 0.999
        assert 0.0 <= st.filter_max_error <= st.filter_error_bound


@pytest.mark.parametrize("as_bytes", [True, False])
def test_sampled_threshold_too_low_is_repeated(as_bytes: bool) -> None:
    """The nearest rows lie one in each sampled tile and nowhere else, fewer than k of them: the
    threshold taken from the sample then admits too few rows, and the call runs again with a safe one."""
    from hnsw_engine_b200.exact_knn import exact_search

    n, dim, k, tile = 128 * 1024, 16, 100, 256
    tiles = n // tile
    sample_rows = max(64 * k, int(np.sqrt(75.0 * k * n)))
    stride = tiles // -(-sample_rows // tile)
    rng = np.random.default_rng(5)
    data = rng.integers(100, 256, (n, dim)).astype(np.float32)
    # 80 of them, in different blocks of the sample (two tiles' columns share a block)
    near = (np.arange(0, tiles, stride) * tile + np.resize([3, 40], -(-tiles // stride)))[:80]
    assert near.size == 80 and stride > 1
    data[near] = rng.integers(0, 8, (near.size, dim))
    queries = rng.integers(0, 8, (6, dim)).astype(np.float32)
    if not as_bytes:
        data += rng.random(data.shape, dtype=np.float32) * 0.5
    ids, dists, st = exact_search(data, queries, k, "l2", return_stats=True)
    o_ids, o_d = exact.exact_search(data, queries, k, "l2")
    np.testing.assert_array_equal(ids, o_ids)
    np.testing.assert_allclose(dists, o_d, rtol=dim * 2.0**-52)
    plain = exact_search(data[rng.permutation(n)], queries, k, "l2", return_stats=True)[2]
    assert st.launches > plain.launches  # the passes ran twice
