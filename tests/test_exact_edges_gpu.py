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
