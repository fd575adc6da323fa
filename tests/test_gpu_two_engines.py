"""Engines of different query widths on one GPU, each in a host thread of its
own, beside the allocation-free entry point: launch limits belong to a kernel
and a device, so no caller may lower them for another.  Listed tuples and
counts equal the oracle's in every batch."""
import ctypes as C
import threading

import numpy as np
import pytest

import dsm_b200 as d
from tests.helpers import oracle_stream

pytestmark = pytest.mark.gpu


def _graph():
    """A hub of 60 middles with three leaves each, and a tail of eight
    vertices behind the updates' edge {8, 9}."""
    labels = list(range(4, 12)) + [0, 1]  # the tail 0..7, the ends 8 and 9
    edges = [(k, k + 1) for k in range(8)]
    for _ in range(60):
        mid = len(labels)
        labels += [2, 3, 3, 3]
        edges += [(9, mid)] + [(mid, mid + k) for k in (1, 2, 3)]
    return len(labels), np.array(labels, np.uint32), np.array(edges, np.uint32)


NARROW = d.Query.from_edges([0, 1, 2, 3], [(0, 1), (1, 2), (2, 3)])
WIDE = d.Query.from_edges(list(range(4, 12)) + [0, 1, 2, 3], [(k, k + 1) for k in range(11)])
UPS = np.array([[1, 8, 9, 0], [0, 9, 8, 0]], np.uint32)


def _engine(q, rounds, errors, **opts):
    try:
        nv, labels, edges = _graph()
        _, want, tuples = oracle_stream(nv, labels, edges, q).apply(UPS)
        assert int(want.sum()) == 360
        for _ in range(4):
            e = d.Engine(0)
            for k, v in opts.items():
                e.set_option(getattr(d, k), v)
            e.load_graph_edges(nv, labels, edges)
            qid = e.register(q)
            for _ in range(rounds // 4):
                r = e.run_batch(UPS)
                assert np.array_equal(r.counts[0], want)
                for i in range(len(UPS)):
                    assert np.array_equal(r.tuples_of(qid, i), tuples[i])
            e.close()
    except BaseException as x:  # noqa: BLE001 - reported by the test
        errors.append(x)


def _plain_runs(q, rounds, errors):
    import torch
    try:
        nv, labels, edges = _graph()
        both = np.unique(np.concatenate([edges, edges[:, ::-1], UPS[:1, 1:3], UPS[:1, 2:0:-1]]), axis=0)
        deg = np.bincount(both[:, 0], minlength=nv)
        start = np.concatenate([[0], np.cumsum((deg + 3) // 4)])
        first = np.concatenate([[0], np.cumsum(deg)])
        arena = np.full(4 * int(start[-1]), 0xFFFFFFFF, np.uint32)
        for v in range(nv):
            arena[4 * start[v]:4 * start[v] + deg[v]] = both[first[v]:first[v + 1], 1]
        stream = torch.cuda.Stream()
        dev = lambda x: torch.from_numpy(np.ascontiguousarray(x.astype(np.uint32)).view(np.int32)).cuda()
        t = [dev(x) for x in (np.stack([start[:-1], deg], 1), arena, labels, UPS[:1])]
        cnt = torch.zeros(1, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        for _ in range(rounds):
            rc = d.lib.dsm_count_edge_embeddings_noalloc(
                C.c_int(0), C.c_uint32(nv), C.c_void_p(t[0].data_ptr()), C.c_void_p(t[1].data_ptr()),
                C.c_void_p(t[2].data_ptr()), C.c_void_p(q.offsets.ctypes.data), C.c_void_p(q.nbrs.ctypes.data),
                C.c_void_p(q.labels.ctypes.data), C.c_uint32(q.nv), C.c_void_p(t[3].data_ptr()), C.c_uint32(1),
                C.c_void_p(cnt.data_ptr()), C.c_void_p(stream.cuda_stream))
            assert rc == 0
            with torch.cuda.stream(stream):
                assert int(cnt[0]) == 180
    except BaseException as x:  # noqa: BLE001
        errors.append(x)


@pytest.mark.parametrize("opts", [{}, {"OPT_GRAPH": 1}])
def test_widths_side_by_side(opts):
    errors = []
    threads = [threading.Thread(target=_engine, args=(WIDE, 1200, errors), kwargs=opts),
               threading.Thread(target=_engine, args=(NARROW, 1200, errors), kwargs=opts),
               threading.Thread(target=_plain_runs, args=(NARROW, 1200, errors))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]
