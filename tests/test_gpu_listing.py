"""Listed tuples placed and sorted on the device (list.cu) at the segment
sizes where the sort changes hands: none, one, a warp's 32, one chunk of 1024,
several chunks and their merges; tuple widths from 2 to 16 words; with
searches over the work limit and queries over their listing budget beside
them; and the host's placing, when the device has no room.  All results are
whole numbers and must equal the oracle's."""
import numpy as np
import pytest

import dsm_b200 as d
from tests.helpers import oracle_stream

pytestmark = pytest.mark.gpu

SIZES = [0, 1, 2, 3, 31, 32, 33, 63, 64, 65, 1023, 1024, 1025, 2047, 2049, 3100, 4096, 4097, 9000]


def _hubs(sizes, tail):
    """One hub (label 1) per size with that many leaves (label 2), a chain of
    `tail` vertices (labels 3, 4, ...) behind it, and one update that joins
    vertex 0 (label 0) to the hub."""
    labels, edges, ups = [0], [], []
    for m in sizes:
        h = len(labels)
        labels.append(1)
        for k in range(m):
            edges.append((h, len(labels)))
            labels.append(2)
        last = h
        for k in range(tail):
            edges.append((last, len(labels)))
            last = len(labels)
            labels.append(3 + k)
        ups.append((1, 0, h, 0))
    perm = np.random.default_rng(len(labels)).permutation(len(labels))
    out = np.zeros(len(labels), np.uint32)
    out[perm] = labels
    e = perm[np.array(edges, np.int64).reshape(-1, 2)].astype(np.uint32)
    u = np.array(ups, np.uint32)
    u[:, 1:3] = perm[u[:, 1:3]]
    return len(labels), out, e, u


def _query(tail, leaf_first):
    labels, edges = [0, 1, 2], [(0, 1), (1, 2)]
    last = 1
    for k in range(tail):
        edges.append((last, len(labels)))
        last = len(labels)
        labels.append(3 + k)
    if leaf_first:  # the column that differs is the first, not the third
        swap = {0: 2, 2: 0}
        labels[0], labels[2] = labels[2], labels[0]
        edges = [tuple(swap.get(x, x) for x in e) for e in edges]
    return d.Query.from_edges(labels, edges)


def _run(nv, labels, edges, ups, queries, **opts):
    e = d.Engine(0)
    for k, v in opts.items():
        e.set_option(getattr(d, k), v)
    e.load_graph_edges(nv, labels, edges)
    ids = [e.register(q) for q in queries]
    out = [e.run_batch(ups)]
    undo = ups[::-1].copy()
    undo[:, 0] ^= 1
    out.append(e.run_batch(undo))
    return e, ids, out, undo


@pytest.mark.parametrize("graph,cap", [(0, 1 << 20), (1, 1 << 20), (0, 1024)])
@pytest.mark.parametrize("tail", [0, 1, 6, 13])
def test_segments_of_every_size(tail, graph, cap):
    nv, labels, edges, ups = _hubs(SIZES, tail)
    queries = [_query(tail, False), _query(tail, True), d.Query.from_edges([0, 1], [(0, 1)])]
    e, ids, (ra, rb), undo = _run(nv, labels, edges, ups, queries, OPT_GRAPH=graph,
                                  OPT_RESULT_CAP=cap)
    for qid, q in zip(ids, queries):
        st = oracle_stream(nv, labels, edges, q)
        for r, b in ((ra, ups), (rb, undo)):
            s, c, t = st.apply(b)
            assert np.array_equal(r.counts[r.query_index(qid)], c)
            for i in range(len(b)):
                assert np.array_equal(r.tuples_of(qid, i), t[i]), (tail, i)
    e.close()


@pytest.mark.parametrize("plain", [0, 1])
def test_limits_leave_the_other_segments_whole(plain):
    """Two leaves per hub: m (m - 1) tuples.  A work limit flags the large
    segments, a listing budget drops the query that lists too much."""
    nv, labels, edges, ups = _hubs([1, 2, 6, 7, 33, 40, 70, 0, 25], 0)
    two = d.Query.from_edges([0, 1, 2, 2], [(0, 1), (1, 2), (1, 3)])
    one = _query(0, False)
    lim, budget = 1500, 3000
    e, ids, (ra, rb), undo = _run(nv, labels, edges, ups, [two, one, two], OPT_WORK_LIMIT=lim, OPT_PLAIN=plain)
    for qid, q in zip(ids, (two, one, two)):
        st = oracle_stream(nv, labels, edges, q)
        st.set_work_limit(lim)
        for r, b in ((ra, ups), (rb, undo)):
            s, c, t = st.apply(b)
            got, over = r.counts[r.query_index(qid)], (c & d.INCOMPLETE) != 0
            assert np.array_equal((got & d.INCOMPLETE) != 0, over)
            assert np.array_equal(got[~over], c[~over])
            for i in range(len(b)):
                assert np.array_equal(r.tuples_of(qid, i), t[i])
    assert (ra.counts[0] & d.INCOMPLETE).any() and not (ra.counts[1] & d.INCOMPLETE).any()
    e.close()
    e, ids, (ra, _), _ = _run(nv, labels, edges, ups, [two, one], OPT_QUERY_LIST_LIMIT=budget, OPT_PLAIN=plain)
    assert ra.query_listed.tolist() == [False, True]
    st = oracle_stream(nv, labels, edges, one)
    _, c, t = st.apply(ups)
    assert np.array_equal(ra.counts[1], c)
    for i in range(len(ups)):
        assert len(ra.tuples_of(ids[0], i)) == 0
        assert np.array_equal(ra.tuples_of(ids[1], i), t[i])
    e.close()


def test_unsorted_results_are_the_same_tuples():
    nv, labels, edges, ups = _hubs([40, 1100, 2], 2)
    q = _query(2, True)
    e, ids, (ra, _), _ = _run(nv, labels, edges, ups, [q], OPT_SORT=0)
    t = oracle_stream(nv, labels, edges, q).apply(ups)[2]
    for i in range(len(ups)):
        got = ra.tuples_of(ids[0], i)
        assert np.array_equal(got[np.lexsort(got.T[::-1])], t[i])
    e.close()


def test_without_room_the_host_places_and_sorts():
    """A result table with room for the rows only and the memory budget pinned
    to the bytes in use: the placed tuples have no room, and the table crosses
    to the host instead."""
    nv, labels, edges, ups = _hubs([40, 1100, 2], 2)
    q = _query(2, True)
    e = d.Engine(0)
    e.set_option(d.OPT_RESULT_CAP, 1200)
    e.load_graph_edges(nv, labels, edges)
    qid = e.register(q)
    none = np.array([[0, 0, 1, 0]] * len(ups), np.uint32)  # as many updates, no tuples
    e.run_batch(none)
    e.set_option(d.OPT_MEM_BUDGET, e.stats()["device_bytes_in_use"])
    r = e.run_batch(ups)
    t = oracle_stream(nv, labels, edges, q).apply(ups)[2]
    for i in range(len(ups)):
        assert np.array_equal(r.tuples_of(qid, i), t[i])
    e.close()


@pytest.mark.parametrize("n", [2047, 2048, 2049, 40000])
def test_batches_around_the_scan_and_the_packed_download(n):
    """As many (query, update) segments as one block scans, one more, and more
    counts than the packed download holds."""
    nv, labels, edges, ups = _hubs([5, 40, 1], 0)
    q = _query(0, False)
    # toggles of the three hub edges and edges that change nothing
    rng = np.random.default_rng(n)
    pick = ups[rng.integers(0, len(ups), n)].copy()
    pick[:, 0] = rng.integers(0, 2, n)
    e = d.Engine(0)
    e.load_graph_edges(nv, labels, edges)
    qid = e.register(q)
    st = oracle_stream(nv, labels, edges, q)
    for b in (pick, pick[:3], pick[::-1].copy()):
        r = e.run_batch(b)
        s, c, t = st.apply(b)
        assert np.array_equal(r.signs, s)
        assert np.array_equal(r.counts[0], c)
        assert np.array_equal(r.tuples.reshape(-1, 3), np.concatenate(t))
    e.close()
