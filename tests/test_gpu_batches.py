"""The matcher's batches of partial embeddings (match.cu): levels that leave
around 31, 32, 33, 63, 64, 65 and many survivors, queries whose vertices have
more backward neighbours than the stored ranges (cliques up to 7 vertices) and
the widest query (16 vertices), donated pieces of every kind (long ranges,
many partials, waiting survivors), each listed and counted.  All results are
whole numbers and must equal the oracle's."""
import numpy as np
import pytest

import dsm_b200 as d
from tests.helpers import oracle_stream

pytestmark = pytest.mark.gpu


def _layers(m, r, seed):
    """Vertex 0 (label 0) joins a hub (label 1) of m middles (label 2), each
    with r leaves (label 3); half of the leaves also neighbour the hub."""
    rng = np.random.default_rng(seed)
    labels, edges = [0, 1], []
    for _ in range(m):
        mid = len(labels)
        labels.append(2)
        edges.append((1, mid))
        for _ in range(r):
            edges.append((mid, len(labels)))
            if rng.random() < 0.5:
                edges.append((1, len(labels)))
            labels.append(3)
    perm = rng.permutation(len(labels))
    out = np.zeros(len(labels), np.uint32)
    out[perm] = labels
    e = perm[np.array(edges, np.int64)].astype(np.uint32)
    return len(labels), out, e, np.array([[1, perm[0], perm[1], 0], [0, perm[0], perm[1], 0]], np.uint32)


PATH = d.Query.from_edges([0, 1, 2, 3], [(0, 1), (1, 2), (2, 3)])
CLOSED = d.Query.from_edges([0, 1, 2, 3], [(0, 1), (1, 2), (2, 3), (1, 3)])
TWO = d.Query.from_edges([0, 1, 2, 3, 2], [(0, 1), (1, 2), (2, 3), (1, 4)])


def _check(nv, labels, edges, batches, queries, listed, **opts):
    e = d.Engine(0)
    e.set_option(d.OPT_LIST, listed)
    for k, v in opts.items():
        e.set_option(getattr(d, k), v)
    e.load_graph_edges(nv, labels, edges)
    ids = [e.register(q) for q in queries]
    sts = [oracle_stream(nv, labels, edges, q) for q in queries]
    total = 0
    for b in batches:
        r = e.run_batch(b)
        for qid, st in zip(ids, sts):
            s, c, t = st.apply(b, listed=bool(listed))
            assert np.array_equal(r.signs, s)
            assert np.array_equal(r.counts[r.query_index(qid)], c)
            total += int(c.sum())
            for i in range(len(b) if listed else 0):
                assert np.array_equal(r.tuples_of(qid, i), t[i])
    stats = e.stats()
    e.close()
    return total, stats


@pytest.mark.parametrize("listed", [0, 1])
@pytest.mark.parametrize("m,r", [(1, 1), (1, 33), (31, 1), (32, 2), (33, 1), (63, 3), (64, 1), (65, 2), (7, 40), (200, 9)])
def test_levels_around_a_batch(m, r, listed):
    nv, labels, edges, ups = _layers(m, r, m * 100 + r)
    for opts in ({}, {"OPT_PACK_MAX": 0}, {"OPT_BFS_LEVELS": 1}, {"OPT_BFS_LEVELS": 2, "OPT_BFS_ROWS": 64}):
        total, _ = _check(nv, labels, edges, [ups], [PATH, CLOSED, TWO], listed, **opts)
        assert total > 0


@pytest.mark.parametrize("nq", [3, 4, 5, 6, 7])
def test_cliques_have_more_backward_neighbours_than_stored_ranges(nq):
    rng = np.random.default_rng(nq)
    nv = 26
    pairs = [(a, b) for a in range(nv) for b in range(a)]
    edges = np.array([p for p in pairs if rng.random() < 0.6], np.uint32)
    labels = (rng.random(nv) < 0.3).astype(np.uint32)
    q = d.Query.from_edges(labels[:nq], [(a, b) for a in range(nq) for b in range(a)])
    pick = rng.choice(len(pairs), 40)
    ups = np.array([[rng.integers(2), *pairs[k], 0] for k in pick], np.uint32)
    total, _ = _check(nv, labels, edges, [ups, ups[::-1].copy()], [q], 1)
    assert total > 0 or nq == 7


def test_sixteen_vertices():
    """Paths and cycles of 16 vertices around a ring with chords."""
    nv = 40
    edges = [(k, (k + 1) % nv) for k in range(nv)] + [(k, k + 7) for k in range(0, nv - 7, 5)]
    labels = np.array([k % 4 for k in range(nv)], np.uint32)
    path = d.Query.from_edges([k % 4 for k in range(16)], [(k, k + 1) for k in range(15)])
    cycle = d.Query.from_edges([k % 4 for k in range(16)], [(k, (k + 1) % 16) for k in range(16)])
    ups = np.array([[0, 3, 4, 0], [1, 4, 3, 0], [1, 0, 15, 0], [0, 10, 11, 0], [1, 10, 11, 0], [1, 21, 36, 0]], np.uint32)
    total, _ = _check(nv, labels, np.array(edges, np.uint32), [ups], [path, cycle], 1)
    assert total > 0


@pytest.mark.parametrize("split,dd", [(0, 0), (64, 1), (512, 4)])
@pytest.mark.parametrize("m,r", [(3, 4000), (900, 12), (2500, 1)])
def test_donated_pieces(m, r, split, dd):
    """One update feeds every warp: a few long ranges, many partials, one
    range of many short ones."""
    nv, labels, edges, ups = _layers(m, r, 5)
    total, s = _check(nv, labels, edges, [ups], [PATH, CLOSED, TWO], 0, OPT_SPLIT_MIN=split, OPT_DONATE_DEPTH=dd)
    assert total > 0 and s["donations"] > 0
    _check(nv, labels, edges, [ups], [PATH, CLOSED, TWO], 0, OPT_DONATE=0)


@pytest.mark.parametrize("nlab", [1, 2])
@pytest.mark.parametrize("limit", [0, 300, 5000])
@pytest.mark.parametrize("listed", [0, 1])
def test_leaves_counted_without_a_scan(nlab, limit, listed):
    """Leaves on hubs of 700 neighbours: their ranges are counted, not read
    (with a listing, once the query is over its budget).  The batch toggles
    the hubs' edges, so ranges hold entries that are not live, and with one or
    two labels they hold images of earlier vertices."""
    rng = np.random.default_rng(nlab * 7 + limit)
    nv = 1600
    edges = {(0, 1)}
    for h, deg in ((0, 700), (1, 650)):
        edges |= {(h, int(w)) for w in rng.choice(np.arange(2, nv), deg, replace=False)}
    while len(edges) < 1700:
        a, b = sorted(int(x) for x in rng.integers(2, nv, 2))
        if a != b:
            edges.add((a, b))
    edges = np.array(sorted(edges), np.uint32)
    labels = rng.integers(0, nlab, nv).astype(np.uint32)
    pairs = edges[rng.choice(np.nonzero(edges[:, 0] < 2)[0], 24)].tolist() + [[0, 1]]
    pairs += [[int(rng.integers(2)), int(w)] for w in rng.integers(2, nv, 6)]
    ups = np.array([[rng.integers(2), *pairs[rng.integers(len(pairs))], 0] for _ in range(70)], np.uint32)
    shapes = [(3, [(0, 1), (1, 2)]), (4, [(0, 1), (1, 2), (2, 3)]), (4, [(0, 1), (1, 2), (0, 2), (0, 3)])]
    queries = [d.Query.from_edges(rng.integers(0, nlab, n), es) for n, es in shapes]
    e = d.Engine(0)
    e.set_option(d.OPT_LIST, listed)
    e.set_option(d.OPT_WORK_LIMIT, limit)
    e.set_option(d.OPT_QUERY_LIST_LIMIT, 500 if listed else 0)
    e.load_graph_edges(nv, labels, edges)
    ids = [e.register(q) for q in queries]
    for b in (ups, ups[::-1].copy()):
        r = e.run_batch(b)
        for k, (qid, q) in enumerate(zip(ids, queries)):
            st = oracle_stream(nv, labels, edges, q)
            st.set_work_limit(limit)
            if b is not ups:
                st.apply_graph(ups)
            s, c, t = st.apply(b, listed=False)
            got, over = r.counts[r.query_index(qid)], (c & d.INCOMPLETE) != 0
            assert np.array_equal((got & d.INCOMPLETE) != 0, over)
            assert np.array_equal(got[~over], c[~over])
            if listed and not over.any():
                assert r.query_listed[r.query_index(qid)] == (int(c.sum()) <= 500)
    e.close()


def _dense(nv, m, seed):
    rng = np.random.default_rng(seed)
    edges = set()
    while len(edges) < m:
        a, b = sorted(int(x) for x in rng.integers(0, nv, 2))
        if a != b:
            edges.add((a, b))
    return rng, np.array(sorted(edges), np.uint32), rng.integers(0, 3, nv).astype(np.uint32)


def test_edge_filter_is_built_anew():
    """More deletes, then more inserts, than the edge filter's words: it is
    built anew between batches, grows, and every batch equals the oracle."""
    rng, edges, labels = _dense(300, 4000, 3)
    q = [d.Query.from_edges(labels[:4], [(0, 1), (1, 2), (2, 3), (0, 3), (0, 2)]),
         d.Query.from_edges(labels[4:7], [(0, 1), (1, 2), (0, 2)])]
    batches = []
    for k in range(6):
        op = k % 2
        pick = edges[rng.permutation(len(edges))[:3000]] if k < 4 else rng.integers(0, 300, (3000, 2))
        batches.append(np.concatenate([np.full((3000, 1), op), pick, np.zeros((3000, 1))], 1).astype(np.uint32))
    batches[4][:, 0] = 1  # a random graph on top, denser than the one loaded
    total, _ = _check(300, labels, edges, batches, q, 0)
    assert total > 0


def test_without_room_for_the_edge_filter():
    """An engine whose budget ends before the filter searches every run."""
    rng, edges, labels = _dense(300, 4000, 4)
    q = d.Query.from_edges(labels[:4], [(0, 1), (1, 2), (2, 3), (0, 3), (0, 2)])
    e = d.Engine(0)
    e.load_graph_edges(300, labels, edges)
    full = e.stats()["device_bytes_in_use"]
    e.close()
    pick = edges[rng.permutation(len(edges))[:200]]
    ups = np.concatenate([np.zeros((200, 1)), pick, np.zeros((200, 1))], 1).astype(np.uint32)
    want = oracle_stream(300, labels, edges, q).apply(ups)
    for budget in (full - 1, 0):
        e = d.Engine(0, budget)
        e.load_graph_edges(300, labels, edges)
        assert (e.stats()["device_bytes_in_use"] < full) == (budget > 0)
        e.set_option(d.OPT_MEM_BUDGET, 8 << 30)
        qid = e.register(q)
        r = e.run_batch(ups)
        assert np.array_equal(r.counts[0], want[1])
        for i in range(len(ups)):
            assert np.array_equal(r.tuples_of(qid, i), want[2][i])
        e.close()


@pytest.mark.parametrize("m,r", [(1, 1), (31, 1), (33, 2), (64, 1), (65, 3), (900, 12), (3, 4000)])
def test_plain_runs_count_alike(m, r):
    """The allocation-free entry point on plain id-sorted runs: the same levels
    around a batch, counted on the graph that has the edge."""
    import ctypes as C

    torch = pytest.importorskip("torch")
    nv, labels, edges, ups = _layers(m, r, m * 100 + r)
    both = np.concatenate([edges, edges[:, ::-1], ups[:1, 1:3], ups[:1, 2:0:-1]])
    both = np.unique(both, axis=0)  # sorted by vertex, then neighbour
    deg = np.bincount(both[:, 0], minlength=nv)
    start = np.concatenate([[0], np.cumsum((deg + 3) // 4)])
    arena = np.full(4 * int(start[-1]), 0xFFFFFFFF, np.uint32)
    first = np.concatenate([[0], np.cumsum(deg)])
    for v in range(nv):
        arena[4 * start[v]:4 * start[v] + deg[v]] = both[first[v]:first[v + 1], 1]
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x.astype(np.uint32)).view(np.int32)).cuda()
    t_adj, t_arena = dev(np.stack([start[:-1], deg], 1)), dev(arena)
    t_lab, t_ups = dev(labels), dev(ups[:1])
    total = 0
    for q in (PATH, CLOSED, TWO):
        want = int(oracle_stream(nv, labels, edges, q).apply(ups[:1], listed=False)[1][0])
        cnt = torch.full((1,), -1, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        rc = d.lib.dsm_count_edge_embeddings_noalloc(
            C.c_int(0), C.c_uint32(nv), C.c_void_p(t_adj.data_ptr()), C.c_void_p(t_arena.data_ptr()),
            C.c_void_p(t_lab.data_ptr()), C.c_void_p(q.offsets.ctypes.data), C.c_void_p(q.nbrs.ctypes.data),
            C.c_void_p(q.labels.ctypes.data), C.c_uint32(q.nv), C.c_void_p(t_ups.data_ptr()), C.c_uint32(1),
            C.c_void_p(cnt.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0
        assert int(cnt[0]) == want
        total += want
    assert total > 0


@pytest.mark.parametrize("fill", [(1 << 27) - 200, (1 << 27) + 5])
def test_plain_runs_of_more_entries_than_32_bits_count(fill):
    """A hub whose run, 32 times over, holds just under and just over 2^32
    entries: 40 partials at the hub, each with the hub's run as its pivot.
    The fillers' label is in no query, so the count is that of the graph
    without them."""
    import ctypes as C

    torch = pytest.importorskip("torch")
    q = d.Query.from_edges([0, 5, 1, 2], [(0, 1), (0, 2), (0, 3)])
    small = np.array([0, 5] + [1] * 40 + [2] * 40, np.uint32)
    spokes = np.array([(0, k) for k in range(2, 82)], np.uint32)
    want = int(oracle_stream(82, small, spokes, q).apply(np.array([[1, 0, 1, 0]], np.uint32), listed=False)[1][0])
    assert want == 1600
    # ids: fillers, 40 + 40 + 1 neighbours that count, the hub; runs: the hub's, then {hub}, which all others share
    nv = fill + 82
    hub, deg = nv - 1, nv - 1
    i32 = dict(dtype=torch.int32, device="cuda")
    t_lab = torch.full((nv,), 3, **i32)
    t_lab[fill:] = torch.tensor([1] * 40 + [2] * 40 + [5, 0], **i32)
    unit = (deg + 3) // 4
    t_arena = torch.zeros(4 * unit + 4, **i32)
    t_arena[:deg] = torch.arange(deg, **i32)
    t_arena[4 * unit] = hub
    t_adj = torch.empty((nv, 2), **i32)
    t_adj[:, 0], t_adj[:, 1] = unit, 1
    t_adj[hub, 0], t_adj[hub, 1] = 0, deg
    t_ups = torch.tensor([[1, hub, nv - 2, 0]], **i32)
    cnt = torch.full((1,), -1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    rc = d.lib.dsm_count_edge_embeddings_noalloc(
        C.c_int(0), C.c_uint32(nv), C.c_void_p(t_adj.data_ptr()), C.c_void_p(t_arena.data_ptr()),
        C.c_void_p(t_lab.data_ptr()), C.c_void_p(q.offsets.ctypes.data), C.c_void_p(q.nbrs.ctypes.data),
        C.c_void_p(q.labels.ctypes.data), C.c_uint32(q.nv), C.c_void_p(t_ups.data_ptr()), C.c_uint32(1),
        C.c_void_p(cnt.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    assert int(cnt[0]) == want


def test_edge_filter_keeps_to_the_graph_size():
    """Edges deleted and inserted again and again, and inserts of edges that
    are there: the graph stays the size it is, and so does the memory in use."""
    rng, edges, labels = _dense(300, 4000, 6)
    q = d.Query.from_edges(labels[:4], [(0, 1), (1, 2), (2, 3), (0, 3), (0, 2)])
    e = d.Engine(0)
    e.set_option(d.OPT_LIST, 0)
    e.load_graph_edges(300, labels, edges)
    e.register(q)
    st = oracle_stream(300, labels, edges, q)
    used = []
    for k in range(24):
        pick = edges[rng.permutation(len(edges))[:3000]]
        ups = np.concatenate([np.full((3000, 1), k & 1), pick, np.zeros((3000, 1))], 1).astype(np.uint32)
        r = e.run_batch(ups)
        assert np.array_equal(r.counts[0], st.apply(ups, listed=False)[1])
        used.append(e.stats()["device_bytes_in_use"])
    assert used[-1] == used[0], used
    e.close()


def _budgeted(**opts):
    """An engine on a graph whose edge filter takes 512 KiB, the memory in use
    without that filter, and one query's footprint."""
    rng, edges, labels = _dense(2000, 200_000, 7)
    q = d.Query.from_edges(labels[:4], [(0, 1), (1, 2), (2, 3), (0, 3), (0, 2)])
    e = d.Engine(0)
    for k, v in opts.items():
        e.set_option(getattr(d, k), v)
    e.load_graph_edges(2000, labels, edges)
    full = e.stats()["device_bytes_in_use"]
    lean = d.Engine(0, full - 1)
    lean.load_graph_edges(2000, labels, edges)
    bare = lean.stats()["device_bytes_in_use"]
    lean.register(q)
    foot = lean.stats()["query_bytes"]
    lean.close()
    assert full - bare == 512 << 10 and foot < 100_000
    return e, q, rng, edges, labels, bare, foot


def _toggles(rng, edges, n):
    pick = edges[rng.permutation(len(edges))[:n]]
    return np.concatenate([rng.integers(0, 2, (n, 1)), pick, np.zeros((n, 1))], 1).astype(np.uint32)


@pytest.mark.parametrize("queries", [3, 30])
@pytest.mark.parametrize("when", ["created", "loaded"])
def test_the_edge_filter_makes_room_for_queries(queries, when):
    """A budget for the graph and some queries, less than the filter takes or
    more, given at creation or (less) after loading: as many are admitted as if
    there were no filter, and not one more."""
    e, q, rng, edges, labels, bare, foot = _budgeted()
    budget = bare + queries * foot
    if when == "created":
        e.close()
        e = d.Engine(0, budget)
        e.load_graph_edges(2000, labels, edges)
        assert e.stats()["device_bytes_in_use"] == bare + (512 << 10) * (queries == 30)
    elif queries == 30:  # set against the bytes in use, which count the filter
        budget += 512 << 10
        e.set_option(d.OPT_MEM_BUDGET, budget)
    else:
        e.set_option(d.OPT_MEM_BUDGET, budget)
    ids = [e.register(q) for _ in range(queries)]
    with pytest.raises(d.DSMError) as x:
        e.register(q)
    assert x.value.code == 2  # DSM_ERR_OOM
    e.set_option(d.OPT_MEM_BUDGET, 8 << 30)
    ups = _toggles(rng, edges, 40)
    want = oracle_stream(2000, labels, edges, q).apply(ups, listed=False)[1]
    r = e.run_batch(ups)
    for qid in ids:
        assert np.array_equal(r.counts[r.query_index(qid)], want)
    e.close()


def test_the_edge_filter_stays_while_queries_fit():
    e, q, rng, edges, labels, bare, foot = _budgeted()
    full = e.stats()["device_bytes_in_use"]
    e.set_option(d.OPT_MEM_BUDGET, full + 2 * foot)
    e.register(q)
    e.register(q)
    assert e.stats()["device_bytes_in_use"] == full
    e.close()


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("n,cap", [(600, 1 << 20), (40, 1200)])
def test_the_edge_filter_makes_room_for_a_batch(n, cap, graph):
    """A batch that needs more scratch, and one whose result table has to grow,
    with the budget at the bytes in use: the filter's go to them."""
    e, q, rng, edges, labels, bare, foot = _budgeted(OPT_RESULT_CAP=cap, OPT_GRAPH=graph)
    e.register(q)
    st = oracle_stream(2000, labels, edges, q)
    none = np.array([[1, *edges[0], 0]] * 40, np.uint32)  # there already
    e.run_batch(none)
    e.set_option(d.OPT_MEM_BUDGET, e.stats()["device_bytes_in_use"])
    st.apply(none, listed=False)
    for _ in range(2):
        ups = _toggles(rng, edges, n)
        r = e.run_batch(ups)
        _, c, t = st.apply(ups)
        assert r.listed and np.array_equal(r.counts[0], c)
        assert np.array_equal(r.tuples.reshape(-1, 4), np.concatenate(t))
    assert e.stats()["result_regrows"] == (cap == 1200) or n == 600
    e.close()


def test_a_batch_takes_little_beside_the_ring():
    """The upload and the packed download lie in the donation ring (64 MiB of
    records, 4 MiB of slots): a batch of one update takes 64 KiB more at most,
    one of 4,096 up to 256 bytes an update."""
    rng, edges, labels = _dense(2000, 200_000, 7)
    e = d.Engine(0)
    e.set_option(d.OPT_LIST, 0)
    e.load_graph_edges(2000, labels, edges)
    e.register(d.Query.from_edges([0, 1, 2], [(0, 1), (1, 2)]))
    before = e.stats()["device_bytes_in_use"]
    e.run_batch(_toggles(rng, edges, 1))
    one = e.stats()["device_bytes_in_use"] - before
    assert one <= (68 << 20) + (64 << 10)
    e.run_batch(_toggles(rng, edges, 4096))
    assert e.stats()["device_bytes_in_use"] - before - one <= 256 * 4096
    e.close()


def test_a_ring_refused_by_halves():
    """A budget with room for the ring's records and not for its slots: the
    batch is refused; with room it runs, and equals the oracle."""
    rng, edges, labels = _dense(2000, 200_000, 7)
    q = d.Query.from_edges([0, 1, 2], [(0, 1), (1, 2)])
    e = d.Engine(0)
    e.set_option(d.OPT_LIST, 0)
    e.load_graph_edges(2000, labels, edges)
    qid = e.register(q)
    ups = _toggles(rng, edges, 20)
    e.set_option(d.OPT_MEM_BUDGET, e.stats()["device_bytes_in_use"] + (66 << 20))
    with pytest.raises(d.DSMError) as x:
        e.run_batch(ups)
    assert x.value.code == 2  # DSM_ERR_OOM
    e.set_option(d.OPT_MEM_BUDGET, 8 << 30)
    r = e.run_batch(ups)
    assert np.array_equal(r.counts[0], oracle_stream(2000, labels, edges, q).apply(ups, listed=False)[1])
    e.close()
