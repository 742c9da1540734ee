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
