"""The workloads this engine's speed is judged on.

Every case is a program a user of the engine has: it loads a data graph,
registers queries, and then streams update batches through the public API
(`dsm_b200.Engine`, or the C ABI entry that takes device buffers).  A pass
applies a batch (or a burst of requests) and then the batch that undoes it, so
the graph is the same before every pass and both directions count: inserts and
deletes, each with its positive or negative embeddings.

Sizes and shapes are those of the five seeded workloads of
`dsm_workload_generate` (R-MAT and Chung-Lu graphs, random-walk queries,
withheld edges re-inserted, live edges deleted), scaled so that a graph is
generated and loaded in a second or two.  Graphs, queries and updates are
drawn here from the case's seed, except where a case says `screened`: those
come from `dsm_b200.Workload`, whose queries are tested for selectivity and can
therefore be counted without a work limit.

All outputs are whole numbers: counts (-1 where the search went over the work
limit, whose partial count depends on scheduling), signs, tuples, bitmaps.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

import dsm_b200 as d

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # One update per call on a small graph, its embeddings listed: the
        # interactive form of the command line tool (one cyclic 5-vertex query);
        # ten such calls, then the ten that undo them.  Latency and launches
        # are all there is.
        dict(name="one_update", kind="stream", workload=1, scale=0, updates=1, calls=10, list=1,
             work_limit=1 << 13),
        # The same stream in batches of about five hundred: up to a million
        # tuples listed and canonically sorted per batch.
        dict(name="stream_listed", kind="stream", workload=1, scale=0, updates=509, calls=1, list=1,
             work_limit=1 << 13),
        # Three screened 8-vertex queries (a tree, one cycle, dense) on a
        # power-law graph, 4096-update batches, exact counts and no work limit.
        dict(name="count_screened", kind="stream", workload=2, scale=-6, updates=4096, calls=1, list=0,
             work_limit=0),
        # The same shapes unscreened on the full-size power-law graph (2^20
        # vertices, 2^24 edges: runs and slot offsets exceed L2), counts, each
        # search bounded by a work limit.
        dict(name="count_full_size", kind="batch", graph="chung_lu", log2_v=20, edges=1 << 24, labels=16, zipf=1.2,
             queries=3, q_min=8, q_max=8, extra=0.75, updates=4096, inserts=0.5, list=0, work_limit=1 << 18,
             filter=0, replay=0),
        # 256 registered queries of 4 to 12 vertices matched in one launch that
        # is replayed from a captured graph, counts.
        dict(name="many_queries", kind="batch", graph="chung_lu", log2_v=18, edges=1 << 22, labels=16, zipf=1.2,
             queries=256, q_min=4, q_max=12, extra=0.5, updates=1021, inserts=0.5, list=0, work_limit=1 << 14,
             filter=0, replay=1),
        # One serving request of median size against 64 queries on a graph far
        # larger than L2, 32 labels, listed and sorted.
        dict(name="request_listed", kind="batch", graph="rmat", log2_v=20, edges=1 << 24, labels=32, zipf=0.0,
             queries=64, q_min=4, q_max=10, extra=0.5, updates=512, inserts=0.6, list=1, work_limit=1 << 16,
             filter=0, replay=0),
        # A burst of requests of uneven size through the serving loop, with a
        # query retired and another registered in the middle: continuous
        # batching, host assembly beside the device, graph replay.
        dict(name="served_burst", kind="served", graph="rmat", log2_v=18, edges=1 << 22, labels=32, zipf=0.0,
             queries=64, q_min=4, q_max=10, extra=0.5, requests=9, median=512, inserts=0.6, work_limit=1 << 12),
        # Hub-heavy graph, 12-vertex cyclic queries, one large batch of mostly
        # deletions: skew, donation between warps, long ranges.
        dict(name="skewed_deletes", kind="batch", graph="rmat_hubs", log2_v=17, edges=1 << 22, labels=8, zipf=0.0,
             queries=64, q_min=12, q_max=12, extra=0.27, updates=32768, inserts=0.2, list=0, work_limit=1 << 10,
             filter=0, replay=0),
        # The candidate filter of one 8-vertex query over the whole graph, as a
        # program that wants candidate sets asks for it.
        dict(name="filter_whole_graph", kind="filter", graph="rmat", log2_v=20, edges=1 << 24, labels=16, zipf=0.0,
             q_min=8, q_max=8, extra=0.3),
        # Small batches with the cluster-encoding filter on, kept resident and
        # recomputed only around the updates.
        dict(name="filtered_updates", kind="batch", graph="chung_lu", log2_v=18, edges=1 << 20, labels=16, zipf=1.2,
             queries=8, q_min=6, q_max=8, extra=0.5, updates=61, inserts=0.5, list=0, work_limit=1 << 16,
             filter=2, replay=0),
        # Counting on device buffers the caller owns, without allocating: plain
        # id-sorted runs, one cyclic 5-vertex query.
        dict(name="device_buffers", kind="device", graph="rmat", log2_v=17, edges=1 << 20, labels=16, zipf=0.0,
             q_min=5, q_max=5, extra=0.25, updates=1024),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["stream", "stream", "batch", "batch", "batch", "batch", "served", "filter", "device"])
    if kind == "stream":
        workload = rng.choice([1, 2])
        updates = _log(rng, 1, 1000) if workload == 1 else _log(rng, 64, 4096)
        return dict(kind=kind, workload=workload, scale=0 if workload == 1 else rng.choice([-7, -6]),
                    updates=updates, calls=max(1, min(10, 100 // updates)),
                    list=rng.choice([0, 1]) if workload == 1 else 0,
                    work_limit=1 << rng.randint(8, 13) if workload == 1 else 0)
    graph = rng.choice(["chung_lu", "rmat", "rmat_hubs"])
    log2_v = rng.randint(12, 19)
    edges = int((1 << log2_v) * rng.uniform(4, 16))
    case = dict(kind=kind, graph=graph, log2_v=log2_v, edges=edges, labels=rng.choice([4, 7, 8, 16, 32]),
                zipf=1.2 if graph == "chung_lu" else 0.0)
    q_min = rng.randint(3, 8)
    case.update(q_min=q_min, q_max=min(12, q_min + rng.randint(0, 4)), extra=round(rng.uniform(0.0, 0.6), 2))
    if kind == "filter":
        return dict(case, q_max=q_min)
    if kind == "device":
        case.update(labels=16, q_min=rng.randint(3, 4), graph="rmat", updates=_log(rng, 128, 4096))
        case["q_max"] = case["q_min"]
        return case
    if kind == "served":
        case.update(queries=_log(rng, 2, 64), requests=rng.randint(3, 10), median=_log(rng, 16, 512),
                    inserts=round(rng.uniform(0.2, 0.8), 2), work_limit=1 << rng.randint(6, 11))
        return case
    queries = _log(rng, 1, 256)
    case.update(queries=queries, updates=_log(rng, 16, 8192 if queries < 64 else 1024),
                inserts=round(rng.uniform(0.2, 0.8), 2), list=rng.choice([0, 0, 1]),
                work_limit=1 << rng.randint(6, 14 if queries < 64 else 12), filter=rng.choice([0, 0, 0, 1, 2]),
                replay=rng.choice([0, 1]))
    if case["filter"] == 2:
        case["queries"] = min(queries, 16)
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _quadrants(kind):
    return (0.70, 0.12, 0.12) if kind == "rmat_hubs" else (0.57, 0.19, 0.19)


class _Graph:
    """An undirected graph without loops or repeats: labels, live edges, and
    a tenth of the edges withheld to be inserted.  Vertex ids are permuted."""

    def __init__(self, case, seed):
        gen = torch.Generator(device=DEVICE)
        gen.manual_seed(seed)

        def rand(n, dtype=torch.float32):
            return torch.rand(n, generator=gen, device=DEVICE, dtype=dtype)

        nv, m = 1 << case["log2_v"], case["edges"]
        n = m + m // 3
        if case["graph"] == "chung_lu":  # exponent 2.1, weights capped at the admissibility bound
            w = torch.arange(1, nv + 1, device=DEVICE, dtype=torch.float64) ** (-1.0 / 1.1)
            w = torch.clamp(w * (2.0 * m / float(w.sum())), max=math.sqrt(2.0 * m))
            cdf = torch.cumsum(w, 0)
            cdf /= float(cdf[-1])
            s = torch.searchsorted(cdf, rand(n, torch.float64)).clamp_(max=nv - 1)
            t = torch.searchsorted(cdf, rand(n, torch.float64)).clamp_(max=nv - 1)
        else:
            a, b, c = _quadrants(case["graph"])
            s = torch.zeros(n, dtype=torch.int64, device=DEVICE)
            t = torch.zeros(n, dtype=torch.int64, device=DEVICE)
            for _ in range(case["log2_v"]):
                x = rand(n)
                s = 2 * s + (x >= a + b).long()
                t = 2 * t + (((x >= a) & (x < a + b)) | (x >= a + b + c)).long()
        perm = torch.randperm(nv, generator=gen, device=DEVICE)
        s, t = perm[s], perm[t]
        keys = torch.unique(torch.minimum(s, t)[s != t] * nv + torch.maximum(s, t)[s != t])
        keys = keys[torch.randperm(len(keys), generator=gen, device=DEVICE)[:m]]
        self.nv = nv
        nl = case["labels"]
        p = torch.arange(1, nl + 1, device=DEVICE, dtype=torch.float64) ** -case["zipf"]
        p = torch.cumsum(p / p.sum(), 0)
        self.labels_t = torch.searchsorted(p, rand(nv, torch.float64)).clamp_(max=nl - 1)
        self.labels = self.labels_t.cpu().numpy().astype(np.uint32)
        held = len(keys) // 10
        self.live_t = keys[held:]
        self.pool = self._pairs(keys[:held])
        self.live = self._pairs(self.live_t)

    def _pairs(self, keys):
        return torch.stack([keys // self.nv, keys % self.nv], 1).cpu().numpy().astype(np.uint32)

    def csr(self):
        """(offsets, neighbours) of the live edges on the device, ids ascending."""
        x, y = self.live_t // self.nv, self.live_t % self.nv
        k = torch.sort(torch.cat([x * self.nv + y, y * self.nv + x])).values
        deg = torch.bincount(k // self.nv, minlength=self.nv)
        off = torch.zeros(self.nv + 1, dtype=torch.int64, device=DEVICE)
        off[1:] = torch.cumsum(deg, 0)
        return off, k % self.nv


def _random_walk_queries(off, nbr, labels, case, count, rng):
    """Queries of q_min..q_max vertices: the tree of a random walk plus up to
    extra * (nq - 1) further data edges between its vertices, labels copied."""
    out = []
    nv = len(labels)
    while len(out) < count:
        nq = rng.randint(case["q_min"], case["q_max"])
        extra = int(case["extra"] * (nq - 1) * (rng.random() if count > 3 else 1.0) + 0.5)
        best = None
        for _ in range(40):
            # dense shapes start at the end of a random edge, others anywhere
            v = int(nbr[rng.randrange(len(nbr))]) if extra * 2 > nq else rng.randrange(nv)
            vs, edges = [v], []
            for _ in range(32 * nq):
                lo, hi = int(off[v]), int(off[v + 1])
                if hi == lo or len(vs) == nq:
                    break
                w = int(nbr[rng.randrange(lo, hi)])
                if w not in vs:
                    edges.append((vs.index(v), len(vs)))
                    vs.append(w)
                v = w
            if len(vs) < nq:
                continue
            more = []
            for i in range(nq):
                run = nbr[int(off[vs[i]]):int(off[vs[i] + 1])]
                for j in range(i + 1, nq):
                    if (i, j) not in edges and (j, i) not in edges:
                        k = int(np.searchsorted(run, vs[j]))
                        if k < len(run) and run[k] == vs[j]:
                            more.append((i, j))
            rng.shuffle(more)
            more = more[:extra]
            if best is None or len(more) > len(best[1]):
                best = (vs, more, edges)
            if len(more) == extra:
                break
        if best is not None:
            vs, more, edges = best
            edges = sorted((min(e), max(e)) for e in edges + more)
            out.append(d.Query.from_edges([int(labels[x]) for x in vs], edges))
    return out


def _updates(graph, edges, n, inserts, rng):
    """About n updates (fewer where they would be most of the graph): withheld
    edges inserted and live edges deleted, interleaved, each edge named once;
    one more in sixty-four repeats an earlier insert and changes nothing.
    With them the updates that undo them, newest first."""
    n_ins = min(int(n * inserts + 0.5), edges // 40)
    n_del = min(n - n_ins, edges // 8)
    ins = graph.pool[rng.choice(len(graph.pool), n_ins, replace=False)]
    dele = graph.live[rng.choice(len(graph.live), n_del, replace=False)]
    ups = np.zeros((n_ins + n_del, 4), np.uint32)
    ups[:n_ins, 0] = 1
    ups[:n_ins, 1:3] = ins
    ups[n_ins:, 1:3] = dele
    ups = ups[rng.permutation(len(ups))]
    flip = rng.random(len(ups)) < 0.5
    ups[flip] = ups[flip][:, [0, 2, 1, 3]]
    ups[:, 3] = graph.labels[ups[:, 1]]
    undo = ups[::-1].copy()
    undo[:, 0] ^= 1
    seen = np.nonzero(ups[:, 0])[0]
    repeats = len(ups) // 64
    if repeats and len(seen):
        ups = np.concatenate([ups, ups[rng.choice(seen, repeats)]])
    return ups, undo


ROOM = 1 << 24  # words of tuples a program keeps room for, per batch


def _list_limit(case):
    """Tuples a query may list per device batch: its share of that room.  The
    serving loop merges requests into device batches as they come, so there
    the limit is one that no query meets."""
    if case["kind"] == "served":
        return 1 << 22
    return min(1 << 22, ROOM // (case.get("queries", 1) * case.get("q_max", 5)))


def _engine(case, nv, labels, edges, queries):
    e = d.Engine(0)
    e.set_option(d.OPT_LIST, case.get("list", 1))
    e.set_option(d.OPT_WORK_LIMIT, case.get("work_limit", 0))
    e.set_option(d.OPT_QUERY_LIST_LIMIT, _list_limit(case) if case.get("list", 1) else 0)
    e.set_option(d.OPT_FILTER, case.get("filter", 0))
    e.set_option(d.OPT_GRAPH, case.get("replay", 0))
    e.load_graph_edges(nv, labels, edges)
    return e, [e.register(q) for q in queries]


def prepare(case, seed):
    kind = case["kind"]
    rng = random.Random(seed * 7919 + 17)
    nrng = np.random.default_rng(seed + 1)
    if kind == "stream":
        n = case["updates"]
        w = d.Workload(case["workload"], seed=seed % (1 << 31) + 1, scale_log2=case["scale"],
                       num_batches=0 if case["workload"] == 1 else 1)
        ups = w.updates[:n * case["calls"]].copy()
        undo = ups[::-1].copy()  # each update of these streams takes effect
        undo[:, 0] ^= 1
        e, _ = _engine(case, w.nv, w.labels, w.edges, w.queries)
        batches = np.split(ups, case["calls"]) + np.split(undo, case["calls"])
        return {"kind": kind, "engine": e, "batches": batches, "room": _rooms(case, len(batches))}
    g = _Graph(case, seed)
    off_t, nbr_t = g.csr()
    off, nbr = off_t.cpu().numpy(), nbr_t.to(torch.int32).cpu().numpy()
    count = case.get("queries", 1)
    queries = _random_walk_queries(off, nbr, g.labels, case, count + (kind == "served"), rng)
    if kind == "batch":
        ups, undo = _updates(g, case["edges"], case["updates"], case["inserts"], nrng)
        e, _ = _engine(case, g.nv, g.labels, g.live, queries)
        return {"kind": kind, "engine": e, "batches": [ups, undo], "room": _rooms(case, 2)}
    if kind == "served":
        sizes = np.exp(np.random.default_rng(case["requests"]).standard_normal(case["requests"]))  # lognormal
        sizes = np.clip(case["median"] * sizes, 1, 16 * case["median"])
        ups, undo = _updates(g, case["edges"], int(sizes.sum()), case["inserts"], nrng)
        cut = np.minimum(np.cumsum(sizes).astype(int)[:-1], len(ups))
        cut_undo = np.minimum(np.cumsum(sizes[::-1]).astype(int)[:-1], len(undo))
        e, ids = _engine(dict(case, list=1, replay=1), g.nv, g.labels, g.live, queries[:count])
        e.serve_start()
        return {"kind": kind, "engine": e, "forward": np.split(ups, cut), "back": np.split(undo, cut_undo),
                "query": ids[count // 2], "first": queries[count // 2], "second": queries[count],
                "room": _rooms(case, 2 * case["requests"])}
    if kind == "filter":
        e, ids = _engine(case, g.nv, g.labels, g.live, queries)
        return {"kind": kind, "engine": e, "query": ids[0], "nq": queries[0].nv, "nv": g.nv}
    # device: {run start in 16-byte units, degree} per vertex, runs padded to 4 entries
    deg = off_t[1:] - off_t[:-1]
    units = (deg + 3) // 4
    start = torch.cumsum(units, 0) - units
    owner = torch.repeat_interleave(torch.arange(g.nv, device=DEVICE), deg)
    arena = torch.full((int(units.sum()) * 4 + 4,), -1, dtype=torch.int32, device=DEVICE)
    arena[start[owner] * 4 + torch.arange(len(nbr_t), device=DEVICE) - off_t[owner]] = nbr_t.to(torch.int32)
    ups, _ = _updates(g, case["edges"], case["updates"], 0.5, nrng)
    ups = ups[:case["updates"]]
    return {"kind": kind, "nv": g.nv, "adj": torch.stack([start, deg], 1).to(torch.int32).contiguous(),
            "arena": arena, "labels": g.labels_t.to(torch.int32), "query": queries[0], "n": len(ups),
            "updates": torch.from_numpy(ups.view(np.int32).copy()).to(DEVICE)}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _rooms(case, n):
    """The buffers a program keeps its results in (zero beyond the tuples of
    the pass; a batch with more than fits is answered by its own array)."""
    if not case.get("list", 1):
        return [None] * n
    words = 1 << 18 if case.get("calls", 1) > 1 else ROOM
    return [np.zeros(words, np.uint32) for _ in range(n)]


def _answer(r, room):
    counts = r.counts.astype(np.int64)
    counts[counts < 0] = -1  # over the work limit
    if room is None:
        return [r.signs, counts]
    if len(r.tuples) > len(room):
        return [r.signs, counts, r.tuples]
    room[:len(r.tuples)] = r.tuples
    return [r.signs, counts, room]


def _count_on_device(s):
    f = d.lib.dsm_count_edge_embeddings_noalloc
    q = s["query"]
    counts = torch.empty(s["n"], dtype=torch.int64, device=DEVICE)
    rc = f(C.c_int(0), C.c_uint32(s["nv"]), C.c_void_p(s["adj"].data_ptr()), C.c_void_p(s["arena"].data_ptr()),
           C.c_void_p(s["labels"].data_ptr()), C.c_void_p(q.offsets.ctypes.data), C.c_void_p(q.nbrs.ctypes.data),
           C.c_void_p(q.labels.ctypes.data), C.c_uint32(q.nv), C.c_void_p(s["updates"].data_ptr()),
           C.c_uint32(s["n"]), C.c_void_p(counts.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    if rc:
        raise RuntimeError("dsm_count_edge_embeddings_noalloc: %d" % rc)
    return counts


def _serve(s):
    e, out = s["engine"], []
    for requests, query in ((s["forward"], s["second"]), (s["back"], s["first"])):
        ids, tickets = [], []
        for k, r in enumerate(requests):
            if k == len(requests) // 2:  # one query leaves, another takes its place
                tickets = [e.retire_async(s["query"]), e.register_async(query)]
            ids.append(e.submit(r))
        for bid in ids:
            out.append(_answer(e.results(bid), s["room"][len(out)]))
        for t in tickets:
            e.admission(t)
    return out


def run(state):
    kind = state["kind"]
    if kind == "device":
        return _count_on_device(state)
    if kind == "filter":
        return list(state["engine"].filter(state["query"], state["nq"], state["nv"]))
    if kind == "served":
        return _serve(state)
    return [_answer(state["engine"].run_batch(b), room) for b, room in zip(state["batches"], state["room"])]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: updates in, signs and counts out, and the two endpoints' runs of
    every update read once (and written once); for the filter the graph's
    entries and labels read once and its bitmaps and masks written once.  The
    search itself has no size that is known before it ran.  Operations: one
    comparison per byte pair of those runs is negligible; none are counted."""
    if case["kind"] == "stream":
        nq, deg = (1, 16) if case["workload"] == 1 else (3, 32)
        n, passes = case["updates"] * case["calls"], 2
    else:
        nv = 1 << case["log2_v"]
        deg = 2 * case["edges"] / nv
        if case["kind"] == "filter":
            return {"bytes": 8.0 * case["edges"] + 12.0 * nv + case["q_max"] * nv / 8 + 4.0 * nv, "flops": 0}
        if case["kind"] == "device":
            return {"bytes": case["updates"] * (16.0 + 8 + 2 * 4 * deg), "flops": 0}
        nq, passes = case["queries"], 2
        n = case["requests"] * case["median"] if case["kind"] == "served" else case["updates"]
    return {"bytes": passes * n * (16.0 + 1 + 8 * nq + 2 * 2 * 4 * deg), "flops": 0}


def exact(case, seed):
    """No output is a computed real number: all are whole and compared for equality."""
    return None
