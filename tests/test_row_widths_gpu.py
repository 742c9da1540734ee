"""Code and byte rows over the widths and result capacities that choose their path."""

from __future__ import annotations

from functools import lru_cache

import numpy as np
import pytest
from conftest import mix10k_arrays

pytestmark = pytest.mark.gpu


@lru_cache(maxsize=None)
def _codes_case(dim: int, metric: str):
    from hnsw_engine_b200 import HNSWIndex

    arrays, ep, ml = mix10k_arrays()
    n = arrays["vectors"].shape[0]
    rng = np.random.default_rng(dim)
    arrays = dict(arrays, vectors=rng.standard_normal((n, dim)).astype(np.float32))
    codes = rng.integers(0, 256, (n, dim)).astype(np.uint8)
    index = HNSWIndex.from_arrays(arrays, ep, ml, dim=dim, metric=metric, M=16)
    index.device_graph.attach_codes(codes)
    return index, arrays, ep, ml, codes


# Widths: one word, part of a 128-byte piece, exactly one, one word more, several with a remainder; and rows
# off 4-byte boundaries, which a lane reads by itself. ef: the largest tile, smaller ones and none.
@pytest.mark.parametrize("dim,ef", [(4, 24), (36, 24), (128, 24), (132, 24), (260, 24), (6, 24), (33, 24),
                                    (64, 400), (64, 900), (64, 2500)])
@pytest.mark.parametrize("metric", ["l2", "ip", "cosine"])
@pytest.mark.parametrize("filtered", [False, True])
def test_code_rows_match_the_oracle(dim: int, ef: int, metric: str, filtered: bool) -> None:
    from oracle import cpu

    index, arrays, ep, ml, codes = _codes_case(dim, metric)
    rng = np.random.default_rng(1)
    queries = rng.standard_normal((12, dim)) * 100 + 120
    mask = rng.random(codes.shape[0]) < 0.4 if filtered else None
    ids, dists, ctr = index.device_graph.search(queries, 10, ef, allowed=mask, use_codes=True)
    o_ids, o_d, o_c = cpu.search_batch(arrays, ep, ml, queries, 10, ef, metric, allowed=mask, codes=codes, threads=8)
    np.testing.assert_array_equal(ids.cpu().numpy(), o_ids)
    np.testing.assert_array_equal(dists.cpu().numpy(), o_d)
    np.testing.assert_array_equal(ctr.cpu().numpy(), o_c)


# Byte rows of one word to several words a lane, those with words for some lanes only in the last round
# (132, 200, 784) among them. Values to 99 keep every sum within a float32's whole numbers.
@pytest.mark.parametrize("dim", [4, 96, 128, 132, 144, 200, 256, 260, 784])
@pytest.mark.parametrize("metric", ["l2", "ip"])
def test_byte_rows_match_the_oracle(dim: int, metric: str) -> None:
    from hnsw_engine_b200 import HNSWIndex
    from oracle import cpu

    arrays, ep, ml = mix10k_arrays()
    n = arrays["vectors"].shape[0]
    rng = np.random.default_rng(dim)
    arrays = dict(arrays, vectors=rng.integers(0, 100, (n, dim)).astype(np.float32))
    index = HNSWIndex.from_arrays(arrays, ep, ml, dim=dim, metric=metric, M=16)
    queries = rng.integers(0, 100, (40, dim)).astype(np.float32)
    for mask in (None, rng.random(n) < 0.4):
        ids, dists, ctr = index.device_graph.search(queries, 10, 48, allowed=mask, dist_mode=2)
        o_ids, o_d, o_c = cpu.search_batch(arrays, ep, ml, queries, 10, 48, metric, allowed=mask, threads=8)
        np.testing.assert_array_equal(ids.cpu().numpy(), o_ids)
        np.testing.assert_array_equal(dists.cpu().numpy(), o_d)
        np.testing.assert_array_equal(ctr.cpu().numpy(), o_c)


# Around the widths and result capacities at which code rows go through tiles of 24 rows, of 16, or none: up to 32
# codes and multiples of 32 that fill no whole pieces (none), others (by the room that ef leaves).
@pytest.mark.parametrize("dim,ef", [(28, 24), (32, 24), (36, 350), (64, 24), (96, 60), (100, 24), (100, 350), (100, 550),
                                    (128, 350), (160, 24), (256, 24), (256, 200), (384, 24)])
@pytest.mark.parametrize("metric", ["l2", "cosine"])
def test_code_rows_match_the_oracle_where_tiles_change(dim: int, ef: int, metric: str) -> None:
    from oracle import cpu

    index, arrays, ep, ml, codes = _codes_case(dim, metric)
    queries = np.random.default_rng(2).standard_normal((12, dim)) * 100 + 120
    ids, dists, ctr = index.device_graph.search(queries, 10, ef, use_codes=True)
    o_ids, o_d, o_c = cpu.search_batch(arrays, ep, ml, queries, 10, ef, metric, codes=codes, threads=8)
    np.testing.assert_array_equal(ids.cpu().numpy(), o_ids)
    np.testing.assert_array_equal(dists.cpu().numpy(), o_d)
    np.testing.assert_array_equal(ctr.cpu().numpy(), o_c)
