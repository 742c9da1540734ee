"""The exact k-NN where lanes, distances or rows are uneven, against NumPy."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import exact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("as_bytes", [True, False])
@pytest.mark.parametrize("n,nq,k", [(4_096, 128, 400), (4_099, 77, 1), (65_536, 200, 100)])
def test_neighbouring_queries_with_unlike_candidates(as_bytes: bool, n: int, nq: int, k: int) -> None:
    """Candidates of each query of a warp in other columns than its neighbours': the rows near a query
    are those whose index is congruent to its own modulo 37, so in most groups of four columns some
    lanes append and the others do not."""
    from hnsw_engine_b200.exact_knn import exact_search

    rng = np.random.default_rng(n + k)
    centres = rng.integers(40, 216, (37, 24))
    data = (centres[np.arange(n) % 37] + rng.integers(-40, 40, (n, 24))).astype(np.float32)
    queries = (centres[np.arange(nq) % 37] + rng.integers(-40, 40, (nq, 24))).astype(np.float32)
    if not as_bytes:
        data += rng.random(data.shape, dtype=np.float32)
    ids, dists = exact_search(data, queries, k, "l2")
    o_ids, o_d = exact.exact_search(data, queries, k, "l2")
    np.testing.assert_array_equal(ids, o_ids)
    np.testing.assert_allclose(dists, o_d, rtol=0 if as_bytes else 24 * 2.0**-52)


@pytest.mark.parametrize("n,dim,nq,run,k", [
    (20_000, 64, 1_000, 20, 10),    # runs within a tile
    (60_000, 64, 2_000, 20, 10),
    (50_000, 32, 300, 100, 50),     # runs across tiles
])
@pytest.mark.parametrize("as_bytes", [True, False])
def test_rows_stored_by_cluster_fit_the_first_lists(n: int, dim: int, nq: int, run: int, k: int,
                                                    as_bytes: bool) -> None:
    """Rows in runs of similar ones, as a data set sorted by cluster has them: a query's near rows fall
    into one segment or two of its candidate list, and the call need not run again for longer lists."""
    import torch

    from hnsw_engine_b200 import _lib
    from hnsw_engine_b200.exact_knn import exact_search

    rng = np.random.default_rng(n + k)
    centres = rng.random((n // run, dim)) * 128 + 30
    data = centres[np.sort(rng.integers(0, n // run, n))] + 20 * rng.standard_normal((n, dim))
    queries = centres[rng.integers(0, n // run, nq)] + 20 * rng.standard_normal((nq, dim))
    if as_bytes:
        data, queries = np.rint(data).clip(0, 255), np.rint(queries).clip(0, 255)
    data, queries = data.astype(np.float32), queries.astype(np.float32)
    lib = _lib.load()
    with pytest.raises(_lib.HnswB200Error):
        _lib.check(lib.hnsw_b200_pack_mask(None, None, 1, None, None))  # the thread's last failure
    before = lib.hnsw_b200_last_error()
    ids, dists = exact_search(torch.from_numpy(data).cuda(), torch.from_numpy(queries).cuda(), k, "l2")
    assert lib.hnsw_b200_last_error() == before  # an overflow would have been recorded
    o_ids, o_d = exact.exact_search(data, queries[:64], k, "l2")
    np.testing.assert_array_equal(ids[:64].cpu().numpy(), o_ids)
    np.testing.assert_allclose(dists[:64].cpu().numpy(), o_d, rtol=0 if as_bytes else dim * 2.0**-52)


def _cosine_nan_last(data: np.ndarray, queries: np.ndarray, k: int) -> tuple[np.ndarray, np.ndarray]:
    """Exact cosine order by (distance, id) with undefined distances (zero rows or queries) last."""
    x, q = data.astype(np.float64), queries.astype(np.float64)
    with np.errstate(invalid="ignore", divide="ignore"):
        x, q = x / np.linalg.norm(x, axis=1)[:, None], q / np.linalg.norm(q, axis=1)[:, None]
    d = 1.0 - q @ x.T
    ids = np.argsort(d, axis=1, kind="stable")[:, :k]  # NumPy sorts NaN last
    return ids, np.take_along_axis(d, ids, axis=1)


@pytest.mark.parametrize("dim", [24, 300])        # a lane's sums, the warp's sums
@pytest.mark.parametrize("n,k", [
    (1, 1), (33, 33), (300, 300),  # every row a result
    (300, 40),                     # some
    (5_000, 3_000),                # too many to gather: inserted
])
def test_zero_rows_and_queries_under_cosine_come_last(dim: int, n: int, k: int) -> None:
    """Rows on the GPU are taken as they are: a zero row's distance is NaN, and it comes after every
    other result, by id among its like; a zero query's results are the first rows."""
    import torch

    from hnsw_engine_b200.exact_knn import exact_search

    rng = np.random.default_rng(n + dim)
    data = rng.standard_normal((n, dim)).astype(np.float32)
    # in the second half of the directions every distance of the first queries is above 1, the filter
    # value of a zero row, so zero rows are within the threshold
    data[:, 0] = -np.abs(data[:, 0]) - 4.0
    data[rng.permutation(n)[: max(1, n // 50)]] = 0.0
    queries = rng.standard_normal((5, dim)).astype(np.float32)
    queries[:, 0] = 8.0
    queries[3] = 0.0
    ids, dists = exact_search(torch.from_numpy(data).cuda(), torch.from_numpy(queries).cuda(), k, "cosine")
    ids, dists = ids.cpu().numpy(), dists.cpu().numpy()
    if k == n:
        w_ids, w_d = _cosine_nan_last(data, queries, k)
        np.testing.assert_allclose(dists, w_d, rtol=0, atol=dim * 2.0**-52)
        np.testing.assert_array_equal(ids, w_ids)
        return
    norms = np.linalg.norm(data, axis=1)
    for i in range(len(queries)):
        assert np.unique(ids[i]).size == k and (ids[i] >= 0).all() and (ids[i] < n).all()
        nan = np.isnan(dists[i])
        m = int((~nan).sum())
        assert not nan[:m].any() and (np.diff(dists[i, :m]) >= 0).all()
        assert (np.diff(ids[i, m:]) > 0).all()
        if i == 3:
            assert m == 0
            continue
        assert (norms[ids[i, m:]] == 0).all() and (norms[ids[i, :m]] > 0).all()
        _, w_d = _cosine_nan_last(data[norms > 0], queries[i : i + 1], max(m, 1))
        np.testing.assert_allclose(dists[i, :m], w_d[0, :m], rtol=0, atol=dim * 2.0**-52)


@pytest.mark.parametrize("dim", [24, 300])
@pytest.mark.parametrize("k", [1, 40, 3_000])
def test_more_ties_than_are_gathered(dim: int, k: int) -> None:
    """All rows but a few zero ones at one distance from the query, some just below it: results are inserted,
    and rows at the last result's distance stay out unless their id is lower."""
    import torch

    from hnsw_engine_b200.exact_knn import exact_search

    n = 6_000
    rng = np.random.default_rng(dim)
    data = np.zeros((n, dim), dtype=np.float32)
    data[:, 0], data[:, 1] = 3.0, 4.0
    near = rng.permutation(n)[:25]  # in no order of ids
    data[near, 1] = np.linspace(3.0, 3.9, 25).astype(np.float32)
    zero = rng.permutation(np.setdiff1d(np.arange(n), near))[:50]
    data[zero] = 0.0
    queries = np.zeros((2, dim), dtype=np.float32)
    queries[0, 0] = 1.0
    queries[1, 1] = 2.0
    ids, dists = exact_search(torch.from_numpy(data).cuda(), torch.from_numpy(queries).cuda(), k, "cosine")
    w_ids, w_d = _cosine_nan_last(data, queries, k)
    np.testing.assert_array_equal(ids.cpu().numpy(), w_ids)
    np.testing.assert_allclose(dists.cpu().numpy(), w_d, rtol=0, atol=dim * 2.0**-52)


@pytest.mark.parametrize("as_bytes", [True, False])
@pytest.mark.parametrize("run,k", [(1_000, 10), (10_000, 10), (10_000, 300)])
def test_lists_that_overflow_are_collected_again(as_bytes: bool, run: int, k: int) -> None:
    """Rows in runs longer than a segment has room for: the first attempt is thrown away, and the next one's
    results are whole."""
    import torch

    from hnsw_engine_b200.exact_knn import exact_search

    rng = np.random.default_rng(run + k)
    n, dim, nq = 100_000, 24, 140
    centres = rng.random((n // run, dim)) * 128 + 30
    data = centres[np.sort(rng.integers(0, n // run, n))] + 20 * rng.standard_normal((n, dim))
    queries = centres[rng.integers(0, n // run, nq)] + 20 * rng.standard_normal((nq, dim))
    if as_bytes:
        data, queries = np.rint(data).clip(0, 255), np.rint(queries).clip(0, 255)
    data, queries = data.astype(np.float32), queries.astype(np.float32)
    ids, dists = exact_search(torch.from_numpy(data).cuda(), torch.from_numpy(queries).cuda(), k, "l2")
    o_ids, o_d = exact.exact_search(data, queries, k, "l2")
    np.testing.assert_array_equal(ids.cpu().numpy(), o_ids)
    np.testing.assert_allclose(dists.cpu().numpy(), o_d, rtol=0 if as_bytes else dim * 2.0**-52)


# k and n over the blocks of the threshold pass (groups of four columns over 16 tiles to one, single groups, every row)
# and k over the sizes at which survivors are gathered (cosine about 220, else about 1,040).
@pytest.mark.parametrize("n,k", [(2_000, k) for k in (1, 10, 20, 50, 100, 200, 213, 222, 400, 600, 1_030, 1_060)]
                         + [(30_011, k) for k in (1, 7, 70, 150, 400)])
@pytest.mark.parametrize("kind", ["bytes", "l2", "ip", "cosine"])
def test_results_at_every_size_of_block(kind: str, n: int, k: int) -> None:
    import torch

    from hnsw_engine_b200.exact_knn import exact_search

    dim, nq = 24, 70
    rng = np.random.default_rng(n + k)
    data = rng.integers(0, 256, (n, dim)).astype(np.float32)
    queries = rng.integers(0, 256, (nq, dim)).astype(np.float32)
    if kind != "bytes":
        data, queries = data + rng.random(data.shape, dtype=np.float32), queries - rng.random(queries.shape, dtype=np.float32)
    metric = "l2" if kind == "bytes" else kind
    ids, dists = exact_search(torch.from_numpy(data).cuda(), torch.from_numpy(queries).cuda(), k, metric)
    o_ids, o_d = exact.exact_search(data, queries, k, metric)
    np.testing.assert_array_equal(ids.cpu().numpy(), o_ids)
    tol = {"bytes": 0.0, "cosine": 0.0}.get(kind, dim * 2.0**-52)
    np.testing.assert_allclose(dists.cpu().numpy(), o_d, rtol=tol, atol=dim * 2.0**-52 if kind == "cosine" else 0.0)


def test_lists_beyond_their_room_are_collected_again() -> None:
    """Every row at one distance of every query, and more queries than lists as long as the rows have room for: the
    first attempt overflows, and the next ones take fewer queries at a time."""
    import torch

    from hnsw_engine_b200 import _lib
    from hnsw_engine_b200.exact_knn import exact_search

    n, nq, k = 200_000, 4_000, 7
    lib = _lib.load()
    with pytest.raises(_lib.HnswB200Error):
        _lib.check(lib.hnsw_b200_pack_mask(None, None, 1, None, None))  # the thread's last failure
    before = lib.hnsw_b200_last_error()
    data = torch.full((n, 8), 3.0, device="cuda")
    data[n - 5] = 4.0  # one row nearer than the rest
    queries = torch.full((nq, 8), 6.0, device="cuda")
    ids, dists = exact_search(data, queries, k, "l2")
    assert lib.hnsw_b200_last_error() != before  # the overflow
    np.testing.assert_array_equal(ids.cpu().numpy(), np.tile([n - 5, 0, 1, 2, 3, 4, 5], (nq, 1)))
    np.testing.assert_array_equal(dists.cpu().numpy(), np.tile([32.0] + [72.0] * 6, (nq, 1)))


def test_long_runs_fit_where_there_is_room() -> None:
    """Rows in runs of 1,000 similar ones and 200 queries: no overflow, as lists may be longer than expected."""
    import torch

    from hnsw_engine_b200 import _lib
    from hnsw_engine_b200.exact_knn import exact_search

    rng = np.random.default_rng(3)
    n, dim, nq, k = 150_000, 32, 200, 10
    centres = rng.random((n // 1_000, dim)) * 128 + 30
    data = (centres[np.sort(rng.integers(0, n // 1_000, n))] + 10 * rng.standard_normal((n, dim))).astype(np.float32)
    queries = (centres[rng.integers(0, n // 1_000, nq)] + 10 * rng.standard_normal((nq, dim))).astype(np.float32)
    lib = _lib.load()
    with pytest.raises(_lib.HnswB200Error):
        _lib.check(lib.hnsw_b200_pack_mask(None, None, 1, None, None))
    before = lib.hnsw_b200_last_error()
    ids, dists = exact_search(torch.from_numpy(data).cuda(), torch.from_numpy(queries).cuda(), k, "l2")
    assert lib.hnsw_b200_last_error() == before
    o_ids, o_d = exact.exact_search(data, queries, k, "l2")
    np.testing.assert_array_equal(ids.cpu().numpy(), o_ids)
    np.testing.assert_allclose(dists.cpu().numpy(), o_d, rtol=dim * 2.0**-52)


@pytest.mark.parametrize("as_bytes", [True, False])
def test_a_loose_threshold_costs_a_pass_not_the_call(as_bytes: bool) -> None:
    """Rows in runs far longer than lists have room for: what overflowing segments kept tightens the threshold, and
    no call with longer lists is needed."""
    import torch

    from hnsw_engine_b200 import _lib
    from hnsw_engine_b200.exact_knn import exact_search

    g = torch.Generator("cuda").manual_seed(5)
    n, dim, nq, run, k = 400_000, 24, 2_000, 20_000, 10
    centres = torch.rand((n // run, dim), generator=g, device="cuda") * 128 + 30
    label = torch.randint(0, n // run, (n,), generator=g, device="cuda").sort().values
    data = centres[label] + 20 * torch.randn((n, dim), generator=g, device="cuda")
    queries = centres[torch.randint(0, n // run, (nq,), generator=g, device="cuda")]
    queries = queries + 20 * torch.randn((nq, dim), generator=g, device="cuda")
    if as_bytes:
        data, queries = data.round().clamp(0, 255), queries.round().clamp(0, 255)
    lib = _lib.load()
    with pytest.raises(_lib.HnswB200Error):
        _lib.check(lib.hnsw_b200_pack_mask(None, None, 1, None, None))  # the thread's last failure
    before = lib.hnsw_b200_last_error()
    ids, dists = exact_search(data, queries, k, "l2")
    assert lib.hnsw_b200_last_error() == before  # an overflow that ends the attempt would have been recorded
    o_ids, o_d = exact.exact_search(data.cpu().numpy(), queries[:48].cpu().numpy(), k, "l2")
    np.testing.assert_array_equal(ids[:48].cpu().numpy(), o_ids)
    np.testing.assert_allclose(dists[:48].cpu().numpy(), o_d, rtol=0 if as_bytes else dim * 2.0**-52)
