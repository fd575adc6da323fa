"""Edges that are not live at an update's view time (match.cu edge_live behind
the changed-edge filter): batches that name the same few edges around two hubs
again and again, so most ranges hold entries the view must leave out.  Batch
sizes lie around the filter's smallest size and its doublings; all results are
whole numbers and must equal the oracle's."""
import numpy as np
import pytest

import dsm_b200 as d
from tests.helpers import oracle_stream

pytestmark = pytest.mark.gpu

SHAPES = {
    "star": (4, [(0, 1), (0, 2), (0, 3)]),
    "path": (4, [(0, 1), (1, 2), (2, 3)]),
    "triangle with a tail": (4, [(0, 1), (1, 2), (0, 2), (0, 3)]),
    "square": (4, [(0, 1), (1, 2), (2, 3), (0, 3)]),
    "clique": (4, [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]),
}


def hub_graph(nlab, n, seed):
    """Two hubs in a sparse graph, and n updates that toggle 28 edges, most of
    them at the hubs (no-ops and a self loop among them)."""
    rng = np.random.default_rng(seed)
    nv = 72
    edges = {(0, 1)}
    for h, deg in ((0, 26), (1, 20)):
        edges |= {(h, int(w)) for w in rng.choice(np.arange(2, nv), deg, replace=False)}
    while len(edges) < 150:
        a, b = (int(x) for x in rng.integers(2, nv, 2))
        if a != b:
            edges.add((min(a, b), max(a, b)))
    labels = rng.integers(0, nlab, nv).astype(np.uint32)
    pairs = [(0, int(w)) for w in rng.choice(np.arange(2, nv), 10, replace=False)]
    pairs += [(1, int(w)) for w in rng.choice(np.arange(2, nv), 8, replace=False)] + [(0, 1), (5, 5)]
    pairs += [tuple(int(x) for x in rng.integers(2, nv, 2)) for _ in range(8)]
    ups = np.zeros((n, 4), np.uint32)
    for i in range(n):
        a, b = pairs[rng.integers(len(pairs))]
        ups[i] = (rng.integers(2), a, b, labels[a]) if rng.random() < 0.5 else (rng.integers(2), b, a, labels[b])
    return nv, labels, np.array(sorted(edges), np.uint32), ups


@pytest.mark.parametrize("n", [1, 63, 64, 65, 130, 300])
@pytest.mark.parametrize("pack", [0, 1024])
def test_views_of_toggled_edges_equal_oracle(n, pack):
    nv, labels, edges, ups = hub_graph(2, n, 60 + n)
    rng = np.random.default_rng(3)
    queries = [d.Query.from_edges(rng.integers(0, 2, nq), es) for nq, es in SHAPES.values()]
    e = d.Engine(0)
    e.set_option(d.OPT_PACK_MAX, pack)
    e.load_graph_edges(nv, labels, edges)
    ids = [e.register(q) for q in queries]
    sts = [oracle_stream(nv, labels, edges, q) for q in queries]
    for part in (ups, ups[::-1].copy()):  # the second batch starts from the first one's graph
        r = e.run_batch(part)
        for qid, st in zip(ids, sts):
            s, c, t = st.apply(part)
            assert np.array_equal(r.signs, s)
            assert np.array_equal(r.counts[r.query_index(qid)], c)
            for i in range(n):
                assert np.array_equal(r.tuples_of(qid, i), t[i])
    e.close()


@pytest.mark.parametrize("timeout", [10, 40])
def test_a_hub_with_many_changed_edges_keeps_the_waits_going(timeout):
    """200,000 edges of one hub deleted and inserted in a batch that counts
    leaves on that hub: the search through the changed edges takes longer than
    the matcher's bounded waits and counts as progress."""
    n, m = 200_000, 8
    hub, first = 0, 1 + m
    nv = first + n
    labels = np.zeros(nv, np.uint32)
    labels[1:first] = 2
    labels[first:] = 1
    spokes = np.stack([np.zeros(nv - 1, np.int64), np.arange(1, nv)], 1).astype(np.uint32)
    half = np.arange(first, nv)[::2]
    flip = lambda op: np.stack([np.full(len(half), op), np.zeros(len(half), np.int64), half, 0 * half], 1)
    ends = lambda: np.array([[op, hub, 1 + k, 0] for k in range(m) for op in (0, 1)])
    # the hub with its leaves, half of them, all of them again: seen by the
    # updates of its edges to the m ends
    ups = np.concatenate([ends(), flip(0), ends(), flip(1), ends()]).astype(np.uint32)
    q = d.Query.from_edges([2, 0, 1], [(0, 1), (1, 2)])
    e = d.Engine(0)
    e.set_option(d.OPT_LIST, 0)
    e.set_option(d.OPT_TIMEOUT_MS, timeout)
    e.load_graph_edges(nv, labels, spokes)
    qid = e.register(q)
    r = e.run_batch(ups)
    got = r.counts[r.query_index(qid)]
    a, b = 2 * m, 2 * m + len(half)
    assert (got[:a] == n).all()
    assert (got[b:b + a] == n - len(half)).all()
    assert (got[b + a + len(half):] == n).all()
    assert (got[a:b] == m).all() and (got[b + a:b + a + len(half)] == m).all()
    e.close()
