"""The work that users of this framework have it do, as cases that can be timed and compared.

Each case is one call (or one short run of calls) through the public entry points: batched and
single searches of an opened graph, filtered and code-space searches, the learned stop, exact k-NN
and the training of the stop network. Sizes are those of this repository's workloads
(``hnsw_engine_b200/graphs.py``, ``bench.py``, ``hnsw_engine_b200/suite.py``) and of its tests.

The workloads' graphs come from a host build that a checkout does not have, so the graphs here are
made on the GPU at the same degrees (at most 32, and 16 above layer 0): the near neighbours that a
diversity heuristic keeps, linked both ways, and a few random nodes, on each layer. An index is opened once and serves every batch of its process, as in a user's program; a seed makes
the queries, filters and training samples.
"""

from __future__ import annotations

import heapq
import math
from functools import lru_cache
from typing import Any

import numpy as np
import torch

from hnsw_engine_b200 import HNSWIndex, QuantizedIndex
from hnsw_engine_b200.exact_knn import exact_search
from hnsw_engine_b200.learned_stop import FEATURES, HIDDEN, StopNetwork
from hnsw_engine_b200.train_stop import SHIPPED

M = 16  # links per node: the workloads' value
DEVICE = "cuda"


def listed() -> list[dict[str, Any]]:
    big = {"data": "mixture", "n": 1_000_000, "dim": 128, "metric": "l2"}
    unit = {"data": "student_t", "n": 1_000_000, "dim": 100, "metric": "cosine"}
    search = {"do": "search", "k": 10, "host": False, "allowed": 1.0, "stop": False}
    return [
        # requests answered one at a time: a service's latency path
        {"name": "single-requests", "do": "single", **big, "nq": 16, "ef": 64, "k": 10},
        # a web service's collected requests: too few queries to fill the GPU, host arrays
        {"name": "batch-100-host", **search, **big, "nq": 100, "ef": 128, "host": True},
        # the smallest workload of the repository: everything stays in L2
        {"name": "small-graph", **search, **big, "n": 10_000, "nq": 1_000, "ef": 50, "host": True},
        # the headline: 10K queries already on the GPU, at the ef of recall 0.95
        {"name": "bytes-10k", **search, **big, "nq": 10_000, "ef": 192},
        # the same batch from host arrays under the learned stop (ef is then the cap)
        {"name": "learned-stop-host", **search, **big, "nq": 10_000, "ef": 192, "host": True, "stop": True},
        # word-embedding-like float rows, cosine: float64 sums
        {"name": "cosine-10k", **search, **unit, "nq": 10_000, "ef": 128},
        # ragged sizes: float rows that no vector load divides, few queries, one result or a few
        {"name": "ragged-float", **search, "data": "normal", "n": 50_021, "dim": 33, "metric": "l2",
         "nq": 777, "ef": 40, "k": 3, "host": True},
        # a metadata filter that one node in ten passes
        {"name": "filtered", **search, **big, "nq": 10_000, "ef": 64, "allowed": 0.1},
        # int8 codes with the exact re-rank, host arrays (the memory-saving configuration)
        {"name": "codes-rerank", "do": "codes", **unit, "nq": 5_000, "ef": 128, "k": 10, "rerank": 128},
        # ground truth of the byte workload: every query against every row
        {"name": "exact-bytes", "do": "exact", **big, "nq": 10_000, "k": 100},
        # exact answers over float rows, as the selectivity planner and audits ask for them
        {"name": "exact-float", "do": "exact", **unit, "n": 200_000, "nq": 1_000, "k": 10},
        # one epoch of the stop network: forward, backward and Adam
        {"name": "train-stop", "do": "train", "samples": 65_536, "batch": 4_096},
    ]


def draw(rng: Any) -> dict[str, Any]:
    """One more case of the same kinds: sizes over their ranges, none above the listed ones."""
    def log(lo: float, hi: float) -> int:
        return max(int(lo), min(int(hi), round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))

    do = rng.choice(["single", "search", "search", "search", "search", "codes", "exact", "exact", "train"])
    if do == "train":
        batch = log(512, 4096)
        return {"do": do, "samples": batch * rng.randint(2, 16) + rng.randint(0, batch - 1), "batch": batch}
    data = rng.choice(["mixture", "mixture", "student_t", "normal"])
    dim = rng.choice([128, 128, 96, 64, 48, 200]) if data == "mixture" else rng.choice([100, 25, 33, 50, 64, 128, 200])
    metric = {"mixture": rng.choice(["l2", "l2", "ip"]), "student_t": "cosine",
              "normal": rng.choice(["l2", "ip"])}[data]
    c: dict[str, Any] = {"do": do, "data": data, "n": log(3_000, 128e6 / max(dim, 128)), "dim": dim,
                         "metric": metric}
    if do == "exact":
        c |= {"nq": log(1, 10_000), "k": log(1, 100)}
        if data != "mixture":  # three BF16 terms a value: keep the cost below the listed byte case
            c["nq"] = min(c["nq"], max(1, int(10_000 * 1e6 * 128 / (6 * c["n"] * max(64, dim)))))
        return c
    c |= {"ef": log(10, 512), "nq": rng.randint(4, 24) if do == "single" else log(1, 10_000)}
    c["k"] = log(1, min(100, c["ef"]))
    # the work of a batch stays below the listed batches'
    weight = dim / 100 if data != "mixture" else max(1.0, dim / 128)
    c["nq"] = max(1, min(c["nq"], int(1_280_000 / (c["ef"] * weight))))
    if do == "search":
        c |= {"host": rng.random() < 0.5, "allowed": 1.0, "stop": False}
        kind = rng.random()
        if kind < 0.3:
            c["allowed"] = round(rng.uniform(0.1, 0.9), 3)
            c["nq"] = max(1, min(c["nq"], int(640_000 * c["allowed"] * 10 / c["ef"])))
        elif kind < 0.45 and data == "mixture" and dim == 128:
            c["stop"] = True
    if do == "codes":
        c["rerank"] = rng.choice([0, c["k"], c["ef"]])
        c["nq"] = max(1, min(c["nq"], int(640_000 / (max(c["ef"], c["rerank"]) * weight))))
    return c


# ------------------------------------------------------------------------------------------- data
def _rows(data: str, n: int, dim: int, gen: torch.Generator) -> torch.Tensor:
    """Float32 rows: a mixture of 100 clusters of byte values, unit rows with heavy tails, or normal."""
    if data == "mixture":
        fixed = torch.Generator(DEVICE).manual_seed(dim)
        centres = torch.rand((100, dim), generator=fixed, device=DEVICE) * 128
        label = torch.randint(0, 100, (n,), generator=gen, device=DEVICE)
        x = centres[label] + 20 * torch.randn((n, dim), generator=gen, device=DEVICE)
        return x.round_().clamp_(0, 255)
    x = torch.randn((n, dim), generator=gen, device=DEVICE)
    if data == "student_t":
        chi = sum(torch.randn((n, dim), generator=gen, device=DEVICE) ** 2 for _ in range(3))
        x = x / (chi / 3).sqrt()
        x = x / x.norm(dim=1, keepdim=True)
    return x


def _chosen(x: torch.Tensor, near: torch.Tensor, most: int) -> tuple[torch.Tensor, torch.Tensor]:
    """Which of each row's neighbours (nearest first) a diversity heuristic keeps, at most ``most``:
    those nearer to the row than to any neighbour kept before; and their squared distances."""
    keep, far = [], []
    for at in torch.arange(x.shape[0], device=DEVICE).split(1 << 14):
        c = x[near[at]]
        d = ((c - x[at][:, None]) ** 2).sum(2)
        cc = (c * c).sum(2)
        between = cc[:, :, None] + cc[:, None, :] - 2 * c @ c.transpose(1, 2)
        least = torch.full_like(d, math.inf)  # from each candidate to the nearest one kept
        kept = torch.zeros_like(d, dtype=torch.bool)
        for j in range(d.shape[1]):
            take = (d[:, j] < least[:, j]) & (kept.sum(1) < most)
            kept[:, j] = take
            least = torch.where(take[:, None], torch.minimum(least, between[:, :, j]), least)
        keep.append(kept)
        far.append(d)
    return torch.cat(keep), torch.cat(far)


def _links(x: torch.Tensor, ids: torch.Tensor, width: int, some: int, gen: torch.Generator
           ) -> tuple[torch.Tensor, torch.Tensor]:
    """Link rows (``width`` + 1 slots, as the native layout has them) and counts of one layer:
    ``some`` random nodes, the chosen near neighbours of each node and the nodes that chose it."""
    n = x.shape[0]
    links = torch.zeros((n, width + 1), dtype=torch.int32, device=DEVICE)
    if n < 2:
        return links, torch.zeros(n, dtype=torch.int32, device=DEVICE)
    own = torch.arange(n, device=DEVICE)
    near, _ = exact_search(x, x, min(n, 2 * M + 1), "l2")
    near = near.gather(1, (near == own[:, None]).sort(stable=True, dim=1).indices)[:, :-1]
    keep, d = _chosen(x, near, M)
    u, v, d = own[:, None].expand_as(near)[keep], near[keep], d[keep]
    far = torch.randint(0, n - 1, (n, some), generator=gen, device=DEVICE)
    far += far >= own[:, None]
    src = torch.cat([own[:, None].expand_as(far).flatten(), u, v])
    dst = torch.cat([far.flatten(), v, u])
    d = torch.cat([torch.full((far.numel(),), -1.0, device=DEVICE), d, d])
    key, order = torch.sort(src * n + dst, stable=True)  # a pair once
    once = order[torch.cat([torch.ones_like(key[:1], dtype=torch.bool), key[1:] != key[:-1]])]
    once = once[torch.sort(d[once], stable=True).indices]
    once = once[torch.sort(src[once], stable=True).indices]  # by node, nearest first
    src, dst = src[once], dst[once]
    rank = torch.arange(src.numel(), device=DEVICE) - torch.searchsorted(src, src)
    use = rank < width
    links[src[use], rank[use]] = ids[dst[use]].to(torch.int32)
    return links, torch.bincount(src, minlength=n).clamp(max=width).to(torch.int32)


@lru_cache(maxsize=8)
def _graph(data: str, n: int, dim: int, metric: str) -> tuple[dict[str, np.ndarray], int, int]:
    """Native arrays, entry point and top level of a graph over ``n`` rows."""
    gen = torch.Generator(DEVICE).manual_seed(n + dim)
    x = _rows(data, n, dim, gen)
    if metric == "cosine":
        x = (x.double() / x.double().norm(dim=1, keepdim=True)).float()
    u = torch.rand(n, generator=gen, device=DEVICE, dtype=torch.float64).clamp(min=1e-12)
    levels = (-u.log() / math.log(M)).floor().to(torch.int64)
    all_ids = torch.arange(n, device=DEVICE)
    links0, count0 = _links(x, all_ids, 2 * M, 2, gen)
    offset = torch.where(levels > 0, levels.cumsum(0) - levels, -1)
    rows, top = int(levels.sum()), int(levels.max())
    links_up = torch.zeros((rows, M + 1), dtype=torch.int32, device=DEVICE)
    count_up = torch.zeros(rows, dtype=torch.int32, device=DEVICE)
    for layer in range(1, top + 1):
        ids = all_ids[levels >= layer]
        at = offset[ids] + layer - 1
        links_up[at], count_up[at] = _links(x[ids].contiguous(), ids, M, 4, gen)
    arrays = {"vectors": x, "levels": levels, "links0": links0, "count0": count0,
              "upper_offset": offset, "links_up": links_up, "count_up": count_up}
    return {k: v.cpu().numpy() for k, v in arrays.items()}, int(all_ids[levels == top][0]), top


@lru_cache(maxsize=8)
def _index(data: str, n: int, dim: int, metric: str) -> HNSWIndex:
    arrays, entry, top = _graph(data, n, dim, metric)
    return HNSWIndex.from_arrays(arrays, entry, top, dim=dim, metric=metric, M=M)


@lru_cache(maxsize=8)
def _quantized(data: str, n: int, dim: int, metric: str) -> QuantizedIndex:
    return QuantizedIndex(_index(data, n, dim, metric))


@lru_cache(maxsize=4)
def _base(data: str, n: int, dim: int) -> torch.Tensor:
    return _rows(data, n, dim, torch.Generator(DEVICE).manual_seed(n + dim))


@lru_cache(maxsize=1)
def _stop_network() -> StopNetwork:
    return StopNetwork.load(SHIPPED / "mix1m", DEVICE)


def _samples(case: dict[str, Any], seed: int) -> tuple[np.ndarray, np.ndarray]:
    """Stop features and labels: correlated features at different scales, few further hits."""
    rng = np.random.default_rng(seed)
    mix = np.random.default_rng(0).standard_normal((FEATURES, FEATURES)) * np.linspace(0.1, 3.0, FEATURES)
    x = (rng.standard_normal((case["samples"], FEATURES)) @ mix + 2.0).astype(np.float32)
    return x, rng.poisson(np.exp(np.clip(0.2 * x[:, 0], -2, 2))).clip(0, 10).astype(np.float32)


# ------------------------------------------------------------------------------------------ cases
def prepare(case: dict[str, Any], seed: int) -> dict[str, Any]:
    do = case["do"]
    if do == "train":
        x, y = _samples(case, seed)
        return {"case": case, "x": x, "y": y}
    spec = (case["data"], case["n"], case["dim"])
    gen = torch.Generator(DEVICE).manual_seed(1_000_003 + seed)
    q = _rows(case["data"], case["nq"], case["dim"], gen)
    state: dict[str, Any] = {"case": case, "queries": q, "mask": None, "stop": None}
    if do == "exact":
        bytes_ = case["data"] == "mixture"
        state["rows"] = _base(*spec).to(torch.uint8) if bytes_ else _base(*spec)
        state["queries"] = q.to(torch.uint8) if bytes_ else q
        return state
    if do in ("single", "codes") or case["host"]:
        state["queries"] = q.cpu().numpy()
    if do == "codes":
        state["quantized"] = _quantized(*spec, case["metric"])
        return state
    state["index"] = _index(*spec, case["metric"])
    if do == "search":
        if case["allowed"] < 1.0:
            state["mask"] = np.random.default_rng(seed).random(case["n"]) < case["allowed"]
        if case["stop"]:
            state["stop"] = _stop_network()
    return state


def run(state: dict[str, Any]) -> dict[str, Any]:
    c = state["case"]
    if c["do"] == "train":
        net = StopNetwork(DEVICE)
        net.fit(state["x"], state["y"], epochs=1, batch=c["batch"])
        return {"params": net.params, "m": net.m, "v": net.v}
    q = state["queries"]
    if c["do"] == "exact":
        ids, dists = exact_search(state["rows"], q, c["k"], c["metric"])
    elif c["do"] == "codes":
        ids, dists = state["quantized"].batch_search(q, k=c["k"], ef=c["ef"], rerank=c["rerank"])
    elif c["do"] == "single":
        got = [state["index"].search(row, k=c["k"], ef=c["ef"]) for row in q]
        ids, dists = np.stack([g[0] for g in got]), np.stack([g[1] for g in got])
    else:
        ids, dists = state["index"].batch_search(q, k=c["k"], ef=c["ef"], filter=state["mask"],
                                                 stop=state["stop"])
    return {"ids": ids, "dists": dists}


def work(case: dict[str, Any]) -> dict[str, float]:
    if case["do"] == "train":
        weights = FEATURES * HIDDEN + HIDDEN * HIDDEN + HIDDEN
        steps = case["samples"] // case["batch"]
        return {"bytes": case["samples"] * (FEATURES + 1) * 4.0 + steps * 6 * 4 * weights,
                "flops": steps * case["batch"] * 6.0 * weights}
    n, dim, nq, k = case["n"], case["dim"], case["nq"], case["k"]
    byte = case["data"] == "mixture"
    if case["do"] == "exact":
        return {"bytes": (n + nq) * dim * (1.0 if byte else 4.0) + nq * k * 16.0,
                "flops": 2.0 * n * nq * dim}
    # a beam search expands about ef nodes (over the allowed share under a filter), reads a link row
    # of each and, once, the rows of the neighbours it has not seen: about eighteen a node, fewer
    # where a filter makes it walk on in one region
    share = case.get("allowed", 1.0)
    hops = min(n, 1.03 * max(case["ef"], case.get("rerank", 0), k) / share + 14)
    rows = min(n, 18 * hops * share**0.2)
    row = dim * (1 if byte or case["do"] == "codes" else 4)
    again = case.get("rerank", 0) * dim * (1 if byte else 4)
    return {"bytes": nq * (hops * 84 + rows * row + again + dim * 4 + k * 16.0),
            "flops": nq * rows * 3.0 * dim}


# ------------------------------------------------------------------------- the same in 64 bits
def exact(case: dict[str, Any], seed: int) -> dict[str, Any] | None:
    if case["do"] == "train":
        return _exact_train(case, seed)
    if case["do"] == "exact":
        return _exact_knn(case, seed)
    if case["do"] == "codes" or case.get("stop") or case["nq"] * case["ef"] > 60_000 * case.get("allowed", 1.0):
        return None  # codes round and the stop predicts; a walk of every query would take minutes
    return _exact_walk(case, seed)


def _exact_knn(case: dict[str, Any], seed: int) -> dict[str, Any]:
    s = prepare(case, seed)
    x, q = s["rows"].double(), s["queries"].double()
    if case["metric"] == "cosine":
        x, q = x / x.norm(dim=1, keepdim=True), q / q.norm(dim=1, keepdim=True)
    xx, out = (x * x).sum(1), []
    for part in q.split(512):
        dot = part @ x.T
        d = {"l2": lambda: (part * part).sum(1, keepdim=True) + xx - 2 * dot, "ip": lambda: -dot,
             "cosine": lambda: 1 - dot}[case["metric"]]()
        best = d.topk(case["k"], largest=False, sorted=True).indices
        if case["metric"] == "l2":  # of the best, without the cancellation
            d = torch.cat([((x[i] - p[:, None]) ** 2).sum(2) for i, p in zip(best.split(64), part.split(64))])
        else:
            d = d.gather(1, best)
        out.append(d.sort(1).values)
    return {"ids": None, "dists": torch.cat(out)}


def _exact_walk(case: dict[str, Any], seed: int) -> dict[str, Any]:
    """The beam search itself, one query at a time over the native arrays."""
    s = prepare(case, seed)
    a, entry, top = _graph(case["data"], case["n"], case["dim"], case["metric"])
    q = s["queries"] if isinstance(s["queries"], np.ndarray) else s["queries"].cpu().numpy()
    q64 = q.astype(np.float64)
    if case["metric"] == "cosine":
        q64 = (q64 / np.linalg.norm(q64, axis=1)[:, None]).astype(np.float32).astype(np.float64)
    mask = s["mask"]
    dists = np.full((case["nq"], case["k"]), np.inf)
    for j, query in enumerate(q64):

        def far(ids: np.ndarray, query: np.ndarray = query) -> np.ndarray:
            x = a["vectors"][ids].astype(np.float64)
            if case["metric"] == "l2":
                return ((x - query) ** 2).sum(1)
            return (0.0 if case["metric"] == "ip" else 1.0) - x @ query

        at = [(float(far(np.array([entry]))[0]), entry)]
        for layer in range(top, -1, -1):
            ef = max(case["ef"], case["k"]) if layer == 0 else 1
            ok = mask if layer == 0 else None
            d0, i0 = at[0]
            seen, todo = {i0}, [(d0, i0)]
            best = [(-d0, -i0)] if ok is None or ok[i0] else []
            while todo:
                d, c = heapq.heappop(todo)
                if len(best) == ef and d > -best[0][0]:
                    break
                if layer == 0:
                    row = a["links0"][c, : a["count0"][c]]
                else:
                    up = a["upper_offset"][c] + layer - 1
                    row = a["links_up"][up, : a["count_up"][up]]
                new = [i for i in dict.fromkeys(row.tolist()) if i not in seen]
                seen.update(new)
                for e, i in zip(far(np.array(new, dtype=np.int64)).tolist() if new else [], new):
                    if len(best) < ef or e < -best[0][0]:
                        heapq.heappush(todo, (e, i))
                        if ok is None or ok[i]:
                            heapq.heappush(best, (-e, -i))
                            if len(best) > ef:
                                heapq.heappop(best)
            at = sorted((-d, -i) for d, i in best)
        got = [d for d, _ in at[: case["k"]]]
        dists[j, : len(got)] = got
    return {"ids": None, "dists": dists}


def _exact_train(case: dict[str, Any], seed: int) -> dict[str, Any]:
    """The same epoch in float64: weights rounded to BF16 in the passes (straight through in the
    backward), mean squared error, Adam (0.9, 0.999, 1e-8)."""
    from hnsw_engine_b200.learned_stop import init_params

    x, y = _samples(case, seed)
    mean, std = x.mean(axis=0), np.maximum(x.std(axis=0), 1e-6)
    xd = torch.from_numpy((x.astype(np.float64) - mean) / std).to(DEVICE)
    yd = torch.from_numpy(y.astype(np.float64)).to(DEVICE)
    p = torch.from_numpy(init_params(0).astype(np.float64)).to(DEVICE).requires_grad_()
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    sizes = [HIDDEN * FEATURES, HIDDEN, HIDDEN * HIDDEN, HIDDEN, HIDDEN, 1]
    order = torch.randperm(len(x), generator=torch.Generator().manual_seed(0)).to(DEVICE)

    def rounded(w: torch.Tensor) -> torch.Tensor:
        return w + (w.detach().float().bfloat16().double() - w.detach())

    for step, s in enumerate(range(0, len(x) - case["batch"] + 1, case["batch"]), 1):
        at = order[s : s + case["batch"]]
        w1, b1, w2, b2, w3, b3 = p.split(sizes)
        h = torch.relu(xd[at] @ rounded(w1).view(HIDDEN, FEATURES).T + b1)
        h = torch.relu(h @ rounded(w2).view(HIDDEN, HIDDEN).T + b2)
        loss = ((h @ rounded(w3) + b3 - yd[at]) ** 2).mean()
        (g,) = torch.autograd.grad(loss, p)
        with torch.no_grad():
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g * g
            p -= 2e-3 * (m / (1 - 0.9**step)) / ((v / (1 - 0.999**step)).sqrt() + 1e-8)
    return {"params": p.detach(), "m": m, "v": v}
