"""The in-place merge and removal of adjacency runs (kernels.cu) at the sizes
where they change hands: runs around a warp's and a block's tile (128, 1024
entries) and around the length from which a block takes a run (2048), changes
at the front, the back and everywhere, in place and past the run's capacity,
and a run emptied and filled again.  Graph and counts (which read the slot
offsets) must equal the oracle's."""
import numpy as np
import pytest

import dsm_b200 as d
from tests.helpers import oracle_stream

pytestmark = pytest.mark.gpu


def _updates(op, vs):
    u = np.zeros((len(vs), 4), np.uint32)
    u[:, 0] = op
    u[:, 2] = vs
    return u


@pytest.mark.parametrize("nlab", [1, 5])
@pytest.mark.parametrize("deg", [0, 1, 3, 4, 127, 128, 129, 1023, 1025, 2046, 2047, 2048, 2049, 4097, 9001])
def test_hub_run_grows_and_shrinks(deg, nlab):
    rng = np.random.default_rng(deg * 10 + nlab)
    nv = deg + 600
    labels = rng.integers(0, nlab, nv).astype(np.uint32)
    others = rng.permutation(np.arange(1, nv))
    edges = [(0, int(v)) for v in others[:deg]]
    edges += [(int(a), int(b)) for a, b in rng.integers(1, nv, (300, 2)) if a != b]
    q = d.Query.from_edges([labels[0], 0, nlab - 1], [(0, 1), (1, 2)])
    e = d.Engine(0)
    e.set_option(d.OPT_LIST, 0)
    e.load_graph_edges(nv, labels, np.array(edges, np.uint32).reshape(-1, 2))
    qid = e.register(q)
    st = oracle_stream(nv, labels, np.array(edges, np.uint32).reshape(-1, 2), q)
    there, absent = np.sort(others[:deg]), np.sort(others[deg:])
    steps = [
        _updates(1, absent[:1]),  # one at the front of its label's range
        _updates(1, absent[-2:]),
        _updates(1, absent[1:80:3]),
        _updates(0, there[:1]),
        _updates(0, there[-3:]),
        _updates(1, absent),  # past the capacity: the run moves
        np.concatenate([_updates(0, absent[5:200]), _updates(1, there[:1])]),
        _updates(0, np.arange(1, nv)),  # empties it
        _updates(1, others[:deg + 1]),
    ]
    for k, b in enumerate(steps):
        r = e.run_batch(b)
        s, c, _ = st.apply(b, listed=False)
        assert np.array_equal(r.signs, s), k
        assert np.array_equal(r.counts[r.query_index(qid)], c), k
        for x, y in zip(e.export_graph(), st.export()):
            assert np.array_equal(x, y), k
    e.close()


@pytest.mark.parametrize("n", [511, 512, 513, 3000])
@pytest.mark.parametrize("nv,nlab", [(1024, 3), (1025, 31), (70_000, 40)])
def test_batches_around_the_counting_sort(n, nv, nlab):
    """Batches of as many updates as are sorted by counting, and fewer; vertex
    ids of 10, 11 and 17 bits; labels on both sides of the shared slot; each
    edge named several times.  Graph, signs and counts equal the oracle's."""
    rng = np.random.default_rng(n + nv)
    labels = rng.integers(0, nlab, nv).astype(np.uint32)
    edges = rng.integers(0, nv, (2000, 2)).astype(np.uint32)
    edges = edges[edges[:, 0] != edges[:, 1]]
    pool = np.concatenate([edges[:200], rng.integers(0, nv, (200, 2)), [[0, nv - 1], [nv - 1, nv - 2], [4, 4]]])
    q = d.Query.from_edges([labels[edges[0, 0]] % 32, labels[edges[0, 1]] % 32], [(0, 1)])
    e = d.Engine(0)
    e.set_option(d.OPT_LIST, 0)
    e.load_graph_edges(nv, labels, edges)
    qid = e.register(q)
    st = oracle_stream(nv, labels, edges, q)
    for _ in range(2):
        pick = pool[rng.integers(0, len(pool), n)]
        b = np.concatenate([rng.integers(0, 2, (n, 1)), pick, np.zeros((n, 1))], 1).astype(np.uint32)
        r = e.run_batch(b)
        s, c, _t = st.apply(b, listed=False)
        assert np.array_equal(r.signs, s)
        assert np.array_equal(r.counts[r.query_index(qid)], c)
        for x, y in zip(e.export_graph(), st.export()):
            assert np.array_equal(x, y)
    e.close()


@pytest.mark.parametrize("deg", [0, 1, 3, 5, 2047, 2049])
@pytest.mark.parametrize("where", ["below", "above", "between", "everywhere"])
def test_many_more_neighbours_than_there_were(deg, where):
    """A run that moves with 6,000 new entries: all in one gap, or in every."""
    rng = np.random.default_rng(deg)
    n = 6000
    nv = 1 + deg + n
    there = {"below": np.arange(1 + n, nv), "above": np.arange(1, 1 + deg),
             "between": np.concatenate([np.arange(1, 1 + deg // 2), np.arange(1 + deg // 2 + n, nv)]),
             "everywhere": np.sort(rng.permutation(np.arange(1, nv))[:deg])}[where]
    new = np.setdiff1d(np.arange(1, nv), there)
    for nlab in (1, 3):
        labels = rng.integers(0, nlab, nv).astype(np.uint32)
        edges = np.stack([np.zeros_like(there), there], 1).astype(np.uint32).reshape(-1, 2)
        q = d.Query.from_edges([labels[0], nlab - 1], [(0, 1)])
        e = d.Engine(0)
        e.set_option(d.OPT_LIST, 0)
        e.load_graph_edges(nv, labels, edges)
        qid = e.register(q)
        st = oracle_stream(nv, labels, edges, q)
        for b in (_updates(1, rng.permutation(new)), _updates(0, new[::2])):
            r = e.run_batch(b)
            assert np.array_equal(r.counts[r.query_index(qid)], st.apply(b, listed=False)[1])
            for x, y in zip(e.export_graph(), st.export()):
                assert np.array_equal(x, y)
        e.close()
