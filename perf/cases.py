"""Performance cases of the query path: batched hierarchical graph search and exact brute force.

Each case names an index (vectors drawn from the benchmark stand-ins' Gaussian mixtures, plus
a hierarchical proximity graph over them), a batch of queries and the call a user makes:
``GpuRouter.batch_query`` on host arrays, ``GpuRouter.batch_query_device`` on device tensors,
``DeviceIndex.bruteforce`` / ``bruteforce_device`` for ground truth, and
``DeviceIndex.centroid_entry`` for the compactor's entry point. Index and router are created in
``prepare`` (a program keeps them for many batches), with one call that lets the router settle
its launch parameters, as a program does at start-up.

The graphs stand in for the reference builder's, which needs minutes of CPU time: level 0 holds
in-cluster nearest neighbours (the near ones all, the farther ones thinned, as pruning leaves
them), some random members of the cluster and some links to nearby clusters, at most 64 distinct
ids a row, nearest first; levels 1 and 2 hold a 32nd and a 1024th of the vertices.
"""

import math

import numpy as np
import torch

from artea_b200 import datasets as ds
from artea_b200.graph import INVALID_VID, CompactHierarchicalGraph
from artea_b200.router import DeviceIndex, GpuRouter

_DEV = "cuda" if torch.cuda.is_available() else "cpu"
_BL, _UL = 64, 32
_NEAR, _FAR, _RANDOM = 24, 56, 8   # ranks kept whole, last rank of the thinned ones, random members
# Vectors a cluster and links between clusters for each mixture. The cluster sizes are those of
# the 1M x 128, 10M x 96 and 1M x 960 stand-ins.
_PER_CLUSTER = {"sift": 977, "deep": 2439, "gist": 1953}
_CROSS = {"sift": 8, "deep": 2, "gist": 4}


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def _search(name, **kw):
    case = dict(name=name, call="device", kind="sift", n=100_000, dim=128, metric="euclidean_sqr", nq=1000, topk=100,
                queue=200, mode="exact", uneven="", graphs=False, early_stop=False, l0_only=False)
    case.update(kw)
    return case


def _exact(name, **kw):
    case = dict(name=name, call="ground_truth_device", kind="sift", n=100_000, dim=128, metric="euclidean_sqr",
                nq=1000, topk=100, subset=0)
    case.update(kw)
    return case


def listed():
    return [
        # One interactive lookup on host arrays: latency of a whole call.
        _search("lookup", call="host", n=100_000, nq=1, topk=10, queue=64),
        # A request of a serving process, its queries already on the device.
        _search("request", kind="deep", n=200_000, dim=96, metric="cosine", nq=16, topk=10, queue=128),
        # A larger serving request with its own topk and queue per query, from host arrays.
        _search("request_uneven", call="host", kind="deep", n=200_000, dim=96, metric="cosine", nq=256, queue=400,
                uneven="serving"),
        # Ragged sizes, inner product, the FAST mode.
        _search("ragged_dot", call="host", kind="deep", n=50_001, dim=40, metric="dot", nq=333, topk=17, queue=50,
                mode="fast"),
        # The 100k x 128 batch at queue 200, from host arrays.
        _search("sift100k", call="host", n=100_000, nq=1000, topk=100, queue=200),
        # The 1M x 128 sweep's ends in use: queue 100 and queue 400, replayed from CUDA graphs.
        _search("sift1m_q100", n=1_000_000, nq=10_000, topk=100, queue=100, graphs=True),
        _search("sift1m_q400", n=1_000_000, nq=10_000, topk=100, queue=400, graphs=True),
        # The cosine batch with topk in {10, 100} and queue in {64, ..., 512} per query.
        _search("deep1m_uneven", kind="deep", n=1_000_000, dim=96, metric="cosine", nq=10_000, queue=512,
                uneven="batch", graphs=True),
        # Wide vectors, L2, few long searches.
        _search("gist200k", kind="gist", n=200_000, dim=960, metric="euclidean", nq=1000, topk=100, queue=400),
        # Ground truth for recall@100 of the 1M x 128 index.
        _exact("truth1m", n=1_000_000, nq=1000, topk=100),
        # Exact search restricted to a few vectors (a filtered lookup), host arrays.
        _exact("truth_subset", call="ground_truth_host", kind="deep", n=123_457, dim=96, metric="cosine", nq=37,
               topk=10, subset=40_001),
        # The compactor's entry point over an index's vectors.
        dict(name="centroid", call="centroid", kind="deep", n=200_000, dim=96, metric="cosine", nq=1, topk=1),
    ]


def _spread(rng, lo, hi):
    """An odd-looking whole number in [lo, hi], even over the logarithm."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, v))


def draw(rng):
    kind = rng.choice(["sift", "sift", "deep", "deep", "gist"])
    dim = {"sift": rng.choice([64, 100, 128, 128, 192, 256]), "deep": rng.choice([32, 40, 96, 96, 200]),
           "gist": rng.choice([480, 784, 960])}[kind]
    n = _spread(rng, 5_000, min(1_000_000, 192_000_000 // dim))
    what = rng.choice(["search"] * 7 + ["truth"] * 2 + ["centroid"])
    if what == "centroid":
        return dict(call="centroid", kind=kind, n=n, dim=dim, nq=1, topk=1,
                    metric="cosine" if kind == "deep" else "euclidean")
    if kind == "deep":
        metric = rng.choice(["cosine", "cosine", "cosine", "dot"])
    else:
        metric = rng.choice(["euclidean_sqr", "euclidean_sqr", "euclidean_sqr", "euclidean"])
    topk = rng.choice([1, 10, 10, 17, 64, 100, 100])
    if what == "truth":
        nq = _spread(rng, 1, min(1000, max(1, 128_000_000_000 // (n * dim))))
        return dict(call=rng.choice(["ground_truth_host", "ground_truth_device"]), kind=kind, n=n, dim=dim,
                    metric=metric, nq=nq, topk=topk, subset=rng.choice([0, 0, _spread(rng, 100, n)]))
    nq = _spread(rng, 1, 10_000 if kind != "gist" else 1_000)
    queue = max(topk, _spread(rng, 20, 800 if nq <= 2000 else 400))
    call = rng.choice(["host", "device"])
    uneven = rng.choice(["", "", "batch", "serving"])
    if uneven:
        topk, queue = 100, {"batch": 512, "serving": 400}[uneven]
    l0_only = call == "host" and not uneven and rng.random() < 0.15
    return dict(call=call, kind=kind, n=n, dim=dim, metric=metric, nq=nq, topk=topk, queue=queue,
                mode=rng.choice(["exact", "exact", "exact", "fast"]), uneven=uneven,
                graphs=call == "device" and rng.random() < 0.5, early_stop=rng.random() < 0.15, l0_only=l0_only)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
class _Mixture:
    """A stand-in's Gaussian mixture (the distributions of artea_b200.datasets), drawn on the device."""

    def __init__(self, kind, n, dim, gen):
        self.kind, self.dim, self.gen = kind, dim, gen
        self.clusters = max(1, n // _PER_CLUSTER[kind])
        shape = (self.clusters, dim)
        if kind == "deep":
            self.centres = torch.randn(shape, device=_DEV, generator=gen)
        else:
            self.centres = torch.rand(shape, device=_DEV, generator=gen) * (128.0 if kind == "sift" else 0.3)

    def draw(self, n):
        labels = torch.randint(self.clusters, (n,), device=_DEV, generator=self.gen)
        sigma = {"sift": 20.0, "deep": 0.35, "gist": 0.05}[self.kind]
        x = torch.randn((n, self.dim), device=_DEV, generator=self.gen).mul_(sigma).add_(self.centres[labels])
        if self.kind == "sift":
            x.round_().clamp_(0.0, 218.0)
        elif self.kind == "deep":
            x /= x.norm(dim=1, keepdim=True)
        else:
            x.clamp_(min=0.0)
        out = torch.zeros((n, ds.padded_dim(self.dim)), device=_DEV)
        out[:, :self.dim] = x
        return out, labels


def _nearest(x, rows, pool, k):
    """Per row of x[rows], the k nearest of pool (vids) other than itself; -1 where there are fewer."""
    k_in = min(k, pool.numel() - 1)
    out = torch.full((rows.numel(), k), -1, dtype=torch.int64, device=_DEV)
    if k_in <= 0:
        return out
    p = x[pool]
    sq = (p * p).sum(1)
    step = max(1, (1 << 27) // pool.numel())
    for lo in range(0, rows.numel(), step):
        r = rows[lo:lo + step]
        d = sq[None, :] - 2.0 * (x[r] @ p.T)
        d.masked_fill_(r[:, None] == pool[None, :], math.inf)
        out[lo:lo + step, :k_in] = pool[d.topk(k_in, dim=1, largest=False).indices]
    return out


def _distinct(rows):
    """Row entries that repeat an earlier one replaced by -1."""
    s, at = rows.sort(dim=1, stable=True)
    again = torch.zeros_like(rows, dtype=torch.bool)
    again[:, 1:] = s[:, 1:] == s[:, :-1]
    return rows.masked_fill(torch.zeros_like(again).scatter_(1, at, again), -1)


def _level0(x, labels, mix):
    n, gen = x.shape[0], mix.gen
    order = labels.argsort(stable=True)
    counts = torch.bincount(labels, minlength=mix.clusters)
    first = counts.cumsum(0) - counts
    most = int(counts.max())
    member = torch.arange(most, device=_DEV)
    cross = _CROSS[mix.kind] if mix.clusters > 1 else 0
    rows = torch.full((n, _BL), -1, dtype=torch.int64, device=_DEV)
    step = max(1, (1 << 28) // (most * most))
    k = min(_FAR, most - 1)
    for lo in range(0, mix.clusters, step):
        c = torch.arange(lo, min(mix.clusters, lo + step), device=_DEV)
        inside = member[None, :] < counts[c][:, None]
        vids = order[(first[c][:, None] + member[None, :]).clamp(max=n - 1)]
        p = x[vids]
        sq = (p * p).sum(2).masked_fill(~inside, math.inf)
        d = torch.baddbmm(sq[:, None, :], p, p.transpose(1, 2), alpha=-2.0)
        d.diagonal(dim1=1, dim2=2).fill_(math.inf)
        d, at = d.topk(k, dim=2, largest=False)
        near = torch.gather(vids[:, None, :].expand(-1, most, -1), 2, at).masked_fill(torch.isinf(d), -1)
        # The near ranks whole, every second of the farther ones.
        near = torch.cat([near[:, :, :_NEAR], near[:, :, _NEAR:_FAR:2]], 2)
        rows[vids[inside], :near.shape[2]] = near[inside]
    used = _NEAR + (_FAR - _NEAR) // 2
    if n > 1:
        pick = torch.rand((n, _RANDOM), device=_DEV, generator=gen)
        rows[:, used:used + _RANDOM] = order[first[labels][:, None] + (pick * counts[labels][:, None]).long()]
        used += _RANDOM
    if cross:
        # Links to random members of the clusters nearest to the vertex's own.
        near = _nearest(mix.centres, torch.arange(mix.clusters, device=_DEV),
                        torch.arange(mix.clusters, device=_DEV), 2 * cross)[:, :min(2 * cross, mix.clusters - 1)]
        which = torch.randint(near.shape[1], (n, cross), device=_DEV, generator=gen)
        to = torch.gather(near[labels], 1, which)
        pick = torch.rand((n, cross), device=_DEV, generator=gen) * counts[to]
        rows[:, used:used + cross] = order[(first[to] + pick.long()).clamp(max=n - 1)].masked_fill(counts[to] == 0, -1)
    # Ragged rows: some of the farther links are not there.
    gone = torch.rand((n, _BL - _NEAR), device=_DEV, generator=gen) < 0.15
    rows[:, _NEAR:].masked_fill_(gone, -1)
    rows.masked_fill_(rows == torch.arange(n, device=_DEV)[:, None], -1)
    return _distinct(rows)


def _upper(x, members, above, gen):
    """Rows of an upper level: its nearest members, the nearest of the level above, some random ones."""
    m = members.numel()
    parts = [_nearest(x, members, members, 12)]
    if above is not None:
        parts.append(_nearest(x, members, above, 10))
    else:
        parts.append(_nearest(x, members, members, 24)[:, 12:])
    parts.append(members[torch.randint(m, (m, 6), device=_DEV, generator=gen)])
    rows = torch.cat(parts, 1)
    rows.masked_fill_(rows == members[:, None], -1)
    return _distinct(rows)[:, :_UL]


def _graph(x, labels, mix):
    n = x.shape[0]
    top = 2 if n >= 32_768 else 1 if n >= 1024 else 0
    perm = torch.randperm(n, device=_DEV, generator=mix.gen)
    highest = torch.zeros(n, dtype=torch.int64, device=_DEV)
    if top >= 1:
        highest[perm[:n // 32]] = 1
    if top >= 2:
        highest[perm[:n // 1024]] = 2
    level_rows = [_level0(x, labels, mix)]
    above = None
    for h in range(top, 0, -1):
        members = (highest >= h).nonzero()[:, 0]
        rows = torch.full((n, _UL), -1, dtype=torch.int64, device=_DEV)
        r = _upper(x, members, above, mix.gen)
        rows[members, :r.shape[1]] = r
        level_rows.insert(1, rows)
        above = members
    vinfo = torch.zeros((n, 2), dtype=torch.int64, device=_DEV)
    vinfo[:, 0] = highest
    offsets, ids, at = [], [], 0
    for h in range(top + 1):
        group = (highest == h).nonzero()[:, 0]
        vinfo[group, 1] = torch.arange(group.numel(), device=_DEV)
        wide = torch.full((group.numel(), h + 1, _BL), -1, dtype=torch.int64, device=_DEV)
        for level in range(h + 1):
            wide[:, h - level, :level_rows[level].shape[1]] = level_rows[level][group]
        wide = wide.reshape(-1, _BL)
        there = wide >= 0
        off = torch.zeros(wide.shape[0] + 1, dtype=torch.int64, device=_DEV)
        off[1:] = there.sum(1).cumsum(0)
        offsets.append((off + at).cpu().numpy().astype(np.uint64))
        at = int(offsets[-1][-1])
        ids.append(wide[there].to(torch.int32))
    entry = int((highest == top).nonzero()[0, 0]) if n else INVALID_VID
    return CompactHierarchicalGraph(n, top, _UL, _BL, entry, vinfo.to(torch.int32).cpu().numpy().view(np.uint32),
                                    offsets, torch.cat(ids).cpu().numpy().view(np.uint32))


def _per_query(case, seed):
    """Per-query topk and queue: the uneven batch's draws, or one request's of the serving mix."""
    rng = np.random.default_rng([seed, 7])
    queues = (64, 128, 256, 512) if case["uneven"] == "batch" else (100, 200, 400)
    topk = rng.choice(np.array([10, 100], dtype=np.uint32), size=case["nq"])
    queue = np.maximum(rng.choice(np.array(queues, dtype=np.uint32), size=case["nq"]), topk)
    return topk, queue


def prepare(case, seed):
    gen = torch.Generator(device=_DEV)
    gen.manual_seed(int(seed))
    mix = _Mixture(case["kind"], case["n"], case["dim"], gen)
    x, labels = mix.draw(case["n"])
    queries, _ = mix.draw(case["nq"])
    search = case["call"] in ("host", "device")
    if search:
        graph = _graph(x, labels, mix)
    else:
        graph = CompactHierarchicalGraph(0, 0, 4, 4, INVALID_VID, np.zeros((0, 2), np.uint32),
                                         [np.zeros(1, np.uint64)], np.zeros(0, np.uint32))
    state = {"case": case, "index": DeviceIndex(graph, x.cpu().numpy())}
    host = not case["call"].endswith("device")
    state["queries"] = queries.cpu().numpy() if host else queries
    if search:
        state["router"] = router = GpuRouter(state["index"], case["metric"], case["topk"], case["queue"],
                                             mode=case["mode"], use_graphs=case["graphs"])
        if case["early_stop"]:
            # A distance that a walk reaches once it is inside the query's cluster.
            unit = {"sift": 20.0, "deep": 0.35, "gist": 0.05}[case["kind"]] * math.sqrt(2.0 * case["dim"])
            reach = {"cosine": 0.15, "dot": 0.15}.get(case["metric"], unit)
            router.set_early_stop([reach] * 3)
        if case["uneven"]:
            topk, queue = _per_query(case, int(seed))
            if host:
                state["per_query"] = (topk, queue)
            else:
                state["per_query"] = tuple(torch.from_numpy(a.view(np.int32)).to(_DEV) for a in (topk, queue))
    elif case.get("subset"):
        ids = torch.randperm(case["n"], device=_DEV, generator=gen)[:case["subset"]].to(torch.int32)
        state["subset"] = ids.cpu().numpy().view(np.uint32) if host else ids
    if not host:
        state["out"] = torch.empty((case["nq"], case["topk"]), dtype=torch.int64, device=_DEV)
    if search:
        run(state)   # the router settles its launch parameters
    return state


# ---------------------------------------------------------------------------
# The calls
# ---------------------------------------------------------------------------
def run(state):
    case, call = state["case"], state["case"]["call"]
    if call == "host":
        topk, queue = state.get("per_query", (None, None))
        words = state["router"].batch_query(state["queries"], topk=topk, queue=queue, k_stride=case["topk"],
                                            l0_only=case["l0_only"])
        return words.view(np.int64)
    stream = torch.cuda.current_stream().cuda_stream
    if call == "device":
        topk, queue = state.get("per_query", (None, None))
        state["router"].batch_query_device(state["queries"], case["nq"], case["topk"], state["out"], d_topk=topk,
                                           d_queue=queue, stream=stream)
        return state["out"]
    if call == "ground_truth_device":
        sub = state.get("subset")
        state["index"].bruteforce_device(state["queries"], case["nq"], case["topk"], case["metric"], state["out"],
                                         d_subset=sub, n_subset=0 if sub is None else sub.numel(), stream=stream)
        return state["out"]
    if call == "ground_truth_host":
        return state["index"].bruteforce(state["queries"], case["topk"], case["metric"],
                                         state.get("subset")).view(np.int64)
    return state["index"].centroid_entry(case["metric"])


def work(case):
    """Bytes and operations of one pass: for a search, the rows of its distance evaluations (each
    vector of the index at most once for the batch), the ids of its expansions and the results."""
    row = 4 * ds.padded_dim(case["dim"])
    ends = case["nq"] * (row + 8 * case["topk"])
    if case["call"] in ("host", "device"):
        queue = {"batch": 260, "serving": 245}.get(case["uneven"], case["queue"])
        # Counted on these graphs: about one expansion per queue entry, 1000 + 6.5 a queue entry evaluations.
        expansions = case["nq"] * (queue + 2.0)
        evals = case["nq"] * min(case["n"], 1000.0 + 6.5 * queue)
        ids = min(expansions, case["n"]) * 50 * 4
        return {"bytes": ends + min(evals, case["n"]) * row + ids, "flops": evals * 3 * case["dim"]}
    rows = case.get("subset") or case["n"]
    if case["call"] == "centroid":
        return {"bytes": rows * row, "flops": rows * case["dim"] * 4.0}
    return {"bytes": rows * row + ends, "flops": float(rows) * case["nq"] * 3 * case["dim"]}


def exact(case, seed):
    """Every output is a whole number: packed (id, distance bits) words or an id. They stay equal."""
    return None
