"""One graph used by several threads: the buffers that its calls share, with the library replaced by
functions that do its copies on the host, slowly, while other threads run."""

from __future__ import annotations

import ctypes
import threading
import time
from contextlib import nullcontext
from types import SimpleNamespace

import numpy as np
import pytest


@pytest.fixture
def host_graph(monkeypatch: pytest.MonkeyPatch):
    """A DeviceGraph without a GPU: its device is the host, and nothing of its graph is set."""
    import torch

    from hnsw_engine_b200.engine import DeviceGraph

    monkeypatch.setattr(torch.cuda, "device", lambda dev: nullcontext())
    stream = SimpleNamespace(cuda_stream=0, synchronize=lambda: None)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: stream)
    empty = torch.empty
    monkeypatch.setattr(torch, "empty", lambda *a, pin_memory=False, **kw: empty(*a, **kw))
    g = DeviceGraph.__new__(DeviceGraph)
    g.device = torch.device("cpu")
    g.dim = 8
    g._stage = None
    g._stage_done = SimpleNamespace(synchronize=lambda: None, record=lambda stream: None)
    g._stage_lock = threading.Lock()
    g.counters_lock = threading.Lock()
    g._one = None
    g._one_lock = threading.Lock()
    g._handle = ctypes.c_void_p()
    g.choose_mode = lambda q, codes: 0
    return g


def _together(work, count: int) -> None:
    """work(0) .. work(count - 1) on a thread each; the first error is raised here."""
    errors: list[BaseException] = []
    gate = threading.Barrier(count)

    def body(i: int) -> None:
        try:
            gate.wait()
            work(i)
        except BaseException as e:  # noqa: BLE001 - reported below
            errors.append(e)

    threads = [threading.Thread(target=body, args=(i,)) for i in range(count)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]


def test_threads_upload_their_own_rows(host_graph) -> None:
    """Every upload of a graph goes through one staging buffer."""
    import torch

    def upload(src, dst, count, threads, stats, stage, stream):
        ctypes.memmove(stage, src, count * 4)
        time.sleep(0.05)  # another thread runs here, as it does while the library stages rows
        ctypes.memmove(dst, stage, count * 4)
        return 0

    g = host_graph
    g.lib = SimpleNamespace(hnsw_b200_upload_queries=upload)
    rows = [np.full((64 + i, 8), float(i), dtype=np.float32) for i in range(6)]
    out = [torch.full(r.shape, -1.0) for r in rows]
    g.upload_queries(rows[0], out[0])  # the buffer is there before the threads are
    _together(lambda i: g.upload_queries(rows[i], out[i]), len(rows))
    for r, o in zip(rows, out):
        np.testing.assert_array_equal(o.numpy(), r)


def test_counters_read_during_a_search_keep_its_share(host_graph) -> None:
    """A search in flight adds to the sums that it was given; reading or resetting the counters meanwhile
    takes what is there and leaves the rest to the next reading."""
    from hnsw_engine_b200 import HNSWIndex

    index = HNSWIndex(8, "l2")
    index._graph = host_graph
    sums = index._totals()
    sums += 5
    assert (index.distance_computations, index.hops) == (5, 5)
    sums += 7  # the search that began before the reading ends after it
    assert (index.distance_computations, index.hops) == (12, 12)
    assert (index.distance_computations, index.hops) == (12, 12)
    index.reset_counters()
    assert (index.distance_computations, index.hops) == (0, 0)
    sums += 3
    assert (index.distance_computations, index.hops) == (3, 3)
    got: list[int] = []
    _together(lambda i: got.append(index._totals().data_ptr()), 8)
    assert set(got) == {sums.data_ptr()}


@pytest.mark.parametrize("ks", [[4] * 6, [3, 4, 5, 3, 4, 5]])
def test_threads_get_their_own_single_results(host_graph, ks: list[int]) -> None:
    """Single searches of a graph share the page-locked query and results."""
    g = host_graph

    def values(address, ctype, count):
        return np.ctypeslib.as_array(ctypes.cast(address, ctypes.POINTER(ctype)), (count,))

    def search(handle, args_ref, stream):
        args = args_ref._obj
        q, k = values(args.queries, ctypes.c_float, g.dim)[0], args.k
        ef = values(args.ef, ctypes.c_int32, 1)[0]
        values(args.out_ids, ctypes.c_int64, k)[:] = int(q)
        time.sleep(0.02)  # another thread runs here, as it does while the library searches
        values(args.out_dists, ctypes.c_double, k)[:] = values(args.queries, ctypes.c_float, g.dim)[0]
        values(args.out_counters, ctypes.c_int64, 2)[:] = ef
        return 0

    g.lib = SimpleNamespace(hnsw_b200_search=search)
    got = {}

    def work(i: int) -> None:
        got[i] = g.search_one(np.full(8, float(i), dtype=np.float32), ks[i], 10 + i)

    g.search_one(np.zeros(8, dtype=np.float32), 4, 10)  # the buffers are there before the threads are
    _together(work, len(ks))
    for i, (ids, dists, ctr) in got.items():
        np.testing.assert_array_equal(ids, np.full(ks[i], i))
        np.testing.assert_array_equal(dists, np.full(ks[i], float(i)))
        np.testing.assert_array_equal(ctr, np.full(2, 10 + i))
