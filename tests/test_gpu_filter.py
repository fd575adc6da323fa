"""The GPU cluster-encoding candidate filter against the oracle's restatement
of the reference filter (filter.cu): per-u candidate bitmaps and the LDF+NLF
masks must be identical; with the filter pruning the matcher, every update's
embeddings must still equal the oracle's (which matches without a filter)."""
import numpy as np
import pytest

import dsm_b200 as d
from oracle import oracle as orc
from tests.helpers import oracle_stream, run_stream, workload

pytestmark = pytest.mark.gpu


def _filter_case(nv, labels, edges, queries):
    e = d.Engine(0)
    e.load_graph_edges(nv, labels, edges)
    qids = [e.register(q) for q in queries]
    off, nb = e.export_graph()
    checked = 0
    for qid, q in zip(qids, queries):
        bm, vc = e.filter(qid, q.nv, nv)
        obm, ovc, pos, plan = orc.cluster_filter(q.labels, q.offsets, q.nbrs, nv, labels, off, nb)
        assert np.array_equal(vc, ovc), f"query {qid}: LDF+NLF masks differ"
        assert np.array_equal(bm, obm), f"query {qid}: bitmaps differ at u {np.nonzero((bm != obm).any(1))[0]}"
        checked += len(plan)
    e.close()
    return checked


def test_filter_reference_fixture():
    import os
    gold = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")
    q = d.TextGraph(os.path.join(gold, "example_q_01.in"), True).query()
    g = d.TextGraph(os.path.join(gold, "example_g_01.in"), False)
    _filter_case(g.nv, g.labels, g.edges, [q])


@pytest.mark.parametrize("cfg", [1, 2, 3])
def test_filter_bitmaps_match_oracle(cfg):
    w = workload(cfg, scale_log2=-6 if cfg > 1 else 0, num_batches=1)
    queries = w.queries[:48]
    ops = _filter_case(w.nv, w.labels, w.edges, queries)
    assert ops >= len(queries)  # every query ran at least one op


def test_filter_random_queries_with_merges_and_combines():
    """Random trees and cyclic queries of 5-12 vertices exercise the merge
    and combine ops of the clustering plan."""
    rng = np.random.default_rng(3)
    w = workload(1)
    qs = []
    for _ in range(24):
        nq = int(rng.integers(5, 13))
        edges = {(int(rng.integers(0, v)), v) for v in range(1, nq)}
        while len(edges) < nq - 1 + int(rng.integers(0, 3)):
            a, b = sorted(int(x) for x in rng.integers(0, nq, 2))
            if a != b:
                edges.add((a, b))
        qs.append(d.Query.from_edges(rng.integers(0, 4, nq), sorted(edges)))
    _filter_case(w.nv, w.labels, w.edges, qs)


@pytest.mark.parametrize("mode", [1, 2])
def test_matching_with_filter_c1(mode):
    w = workload(1)
    q = w.queries[0]
    e = d.Engine(0)
    e.set_option(d.OPT_FILTER, mode)
    e.load_graph_edges(w.nv, w.labels, w.edges)
    qid = e.register(q)
    st = oracle_stream(w.nv, w.labels, w.edges, q)
    ups = w.updates
    run_stream(e, [qid], [st], [ups[i:i + 512] for i in range(0, len(ups), 512)], check_graph_every=1)
    e.close()


def test_matching_with_filter_multi_query():
    w = workload(3, scale_log2=-6, num_batches=2)
    bs = [b[:1024] for b in w.batches()]
    qs = w.queries[:32]
    e = d.Engine(0)
    e.set_option(d.OPT_FILTER, 2)
    e.load_graph_edges(w.nv, w.labels, w.edges)
    qids = [e.register(q) for q in qs]
    streams = [oracle_stream(w.nv, w.labels, w.edges, q) for q in qs]
    total, checked = run_stream(e, qids, streams, bs, check_graph_every=1, limit=200_000)
    assert checked >= 32 * 512
    e.close()


@pytest.mark.parametrize("qi", [0, 1, 2])
def test_matching_with_filter_c2_counts(qi):
    w = workload(2, scale_log2=-6, num_batches=2)
    q = w.queries[qi]
    e = d.Engine(0)
    e.set_option(d.OPT_FILTER, 2)
    e.set_option(d.OPT_LIST, 0)
    e.load_graph_edges(w.nv, w.labels, w.edges)
    qid = e.register(q)
    st = oracle_stream(w.nv, w.labels, w.edges, q)
    total, checked = run_stream(e, [qid], [st], list(w.batches()), check_graph_every=1, listed=False,
                                limit=150_000)
    assert checked >= 1024
    e.close()


def _inc_pair(w, queries, mode=2, **opts):
    engines = []
    for inc in (1, 0):
        e = d.Engine(0)
        e.set_option(d.OPT_FILTER, mode)
        e.set_option(d.OPT_FILTER_INCREMENTAL, inc)
        for k, v in opts.items():
            e.set_option(getattr(d, k), v)
        e.load_graph_edges(w.nv, w.labels, w.edges)
        engines.append((e, [e.register(q) for q in queries]))
    return engines


def _same_state(inc, full, queries, nv, tag):
    """Resident filter state of the incremental engine == the full one's;
    returns the runs that were incremental and their vertex counts."""
    (ei, qi), (ef, qf) = inc, full
    runs = []
    for a, b, q in zip(qi, qf, queries):
        bi, vi, (fi, ni) = ei.filter_state(a, q.nv, nv)
        bf, vf, (ff, nf) = ef.filter_state(b, q.nv, nv)
        assert ff and nf == nv, tag
        assert np.array_equal(vi, vf), f"{tag} query {a}: LDF+NLF masks differ at {np.nonzero(vi != vf)[0][:8]}"
        assert np.array_equal(bi, bf), f"{tag} query {a}: bitmaps differ (u {np.nonzero((bi != bf).any(1))[0]})"
        if not fi:
            runs.append(ni)
    return runs


@pytest.mark.parametrize("cfg,scale,nqs,bsz,nb", [(1, 0, 1, 32, 10), (2, -4, 3, 8, 10), (3, -6, 16, 64, 6),
                                                  (4, -10, 8, 16, 8)])
def test_incremental_filter_equals_full(cfg, scale, nqs, bsz, nb):
    """DSM_OPT_FILTER_INCREMENTAL: after every batch the resident bitmaps and
    LDF+NLF masks of the incremental filter (region of the batch's and the
    previous batch's endpoints, validity replay outside it) equal those of a
    full recompute on the same union graph; the matches are identical; later
    batches ran incrementally on regions smaller than the graph."""
    w = workload(cfg, scale_log2=scale, num_batches=1)
    qs = w.queries[:nqs]
    inc, full = _inc_pair(w, qs)
    ups = next(w.batches())
    region_runs = []
    for k in range(nb):
        b = ups[k * bsz:(k + 1) * bsz]
        ri, rf = inc[0].run_batch(b), full[0].run_batch(b)
        assert np.array_equal(ri.counts, rf.counts) and np.array_equal(ri.tuples, rf.tuples)
        region_runs += _same_state(inc, full, qs, w.nv, f"batch {k}")
    assert len(region_runs) >= (nb - 1) * len(qs) // 2, region_runs
    assert min(region_runs) < w.nv
    for e, _ in (inc, full):
        e.close()


def test_incremental_filter_ldf_only_and_graph_changes():
    """Mode 1 (LDF+NLF, a region of the endpoints alone), a graph-only apply
    between batches (the next run recomputes every vertex), and CUDA-graph
    replay: the state still equals a full recompute after every batch."""
    w = workload(2, scale_log2=-4, num_batches=1)
    qs = w.queries[:3]
    ups = next(w.batches())
    for mode, opts in ((1, {}), (2, {"OPT_GRAPH": 1})):
        inc, full = _inc_pair(w, qs, mode=mode, **opts)
        fulls = 0
        for k in range(8):
            b = ups[k * 16:(k + 1) * 16]
            if k == 4:  # graph-only apply: not filtered
                for e, _ in (inc, full):
                    e.apply_graph(ups[200:232])
            ri, rf = inc[0].run_batch(b), full[0].run_batch(b)
            assert np.array_equal(ri.counts, rf.counts)
            runs = _same_state(inc, full, qs, w.nv, f"mode {mode} batch {k}")
            if k == 4:
                assert runs == [], "the run after a graph-only apply must be full"
            fulls += len(qs) - len(runs)
        assert fulls < 8 * len(qs)
        for e, _ in (inc, full):
            e.close()


@pytest.mark.parametrize("nv", [31, 32, 33, 255, 256, 257, 700])
@pytest.mark.parametrize("labels_to", [3, 31, 32, 40])
def test_filter_at_the_edges_of_its_tiles(nv, labels_to):
    """Vertex counts around the tiles of 32 and 256, labels up to and beyond
    the slot they share (31), one hub that neighbours every vertex, vertices
    without neighbours: masks and bitmaps equal the oracle's."""
    rng = np.random.default_rng(nv * 100 + labels_to)
    # labels from the top of the range down, so that slot 31 is crowded where there is one
    labels = (labels_to - 1 - rng.integers(0, min(labels_to, 10), nv)).astype(np.uint32)
    edges = {(0, v) for v in range(1, nv - 2)}
    while len(edges) < 3 * nv:
        a, b = sorted(int(x) for x in rng.integers(0, nv - 2, 2))
        if a != b:
            edges.add((a, b))
    qs = []
    for k in range(4):
        nq = 4 + k
        tree = {(int(rng.integers(0, v)), v) for v in range(1, nq)} | {(0, nq - 1)}
        ql = np.minimum(labels[rng.integers(0, nv, nq)], 31)
        qs.append(d.Query.from_edges(ql, sorted(tree)))
    _filter_case(nv, labels, np.array(sorted(edges), np.uint32), qs)


@pytest.mark.parametrize("first,fan", [(64_000, 4), (65_530, 4), (65_537, 1), (70_000, 1), (30_000, 3)])
def test_region_list_fills_within_a_hop(first, fan):
    """The region's list (65,536 vertices here) fills while a hop is being
    expanded: by the hub's own neighbours, or by theirs with the list nearly
    full before; the last case fits.  The state equals a full recompute."""
    rng = np.random.default_rng(first + fan)
    nv = 100_000
    labels = rng.integers(0, 3, nv).astype(np.uint32)
    labels[0] = 0
    near = 1 + rng.permutation(nv - 1)[:first]
    rest = np.setdiff1d(np.arange(1, nv), near)
    out = np.repeat(near, fan)
    edges = np.concatenate([np.stack([np.zeros_like(near), near], 1),
                            np.stack([out, rest[rng.integers(0, len(rest), len(out))]], 1)]).astype(np.uint32)
    qs = [d.Query.from_edges([0, 1, 2, 1, 2], [(0, 1), (1, 2), (2, 3), (0, 4), (0, 2)]),
          d.Query.from_edges([1, 0, 2], [(0, 1), (1, 2)])]

    class W:
        pass

    w = W()
    w.nv, w.labels, w.edges = nv, labels, edges
    inc, full = _inc_pair(w, qs)
    for e, _ in (inc, full):
        e.set_option(d.OPT_LIST, 0)
        e.set_option(d.OPT_WORK_LIMIT, 1000)
    for k in range(4):
        b = np.array([[k & 1, 0, near[0], 0], [1, 0, rest[k], 0]], np.uint32)
        for e, _ in (inc, full):
            e.run_batch(b)
        _same_state(inc, full, qs, nv, f"batch {k}")
    for e, _ in (inc, full):
        e.close()


@pytest.mark.parametrize("tiles,extra", [(1, 0), (1, 1), (1, 1025), (2, 300)])
def test_filter_ops_carry_candidates_from_tile_to_tile(tiles, extra):
    """16 queries leave an SM's worth of blocks for each, so a block looks
    through several tiles of 1024 vertices and carries fewer than 256
    candidates from one to the next: tiles of 0 to 1024 candidates, around 256
    of them in sum, against the oracle."""
    torch = pytest.importorskip("torch")
    stride = 1024 * torch.cuda.get_device_properties(0).multi_processor_count
    nv = tiles * stride + extra
    rng = np.random.default_rng(nv)
    per_tile = np.array([0, 1, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1024])
    v = np.arange(nv)
    core = v % 1024 < per_tile[(v // 1024 + v // stride * 5) % len(per_tile)]
    labels = np.where(core, 0, 1 + rng.integers(0, 2, nv)).astype(np.uint32)
    of = [np.nonzero(labels == k)[0] for k in range(3)]
    ends = lambda a, k: np.stack([a, of[k][rng.integers(0, len(of[k]), len(a))]], 1)
    keep = rng.random(len(of[0])) < 0.9  # the others are no candidates of a vertex with both neighbours
    edges = np.concatenate([ends(of[0], 1), ends(of[0][keep], 2), ends(of[1], 2), ends(of[0][::3], 0)])
    edges = edges[edges[:, 0] != edges[:, 1]].astype(np.uint32)
    shapes = [(3, [(0, 1), (0, 2)]), (4, [(0, 1), (0, 2), (1, 3)]), (4, [(0, 1), (1, 2), (2, 3), (0, 3)]),
              (5, [(0, 1), (0, 2), (1, 3), (2, 4)])]
    qs = [d.Query.from_edges([0, 1, 2, 0, 1][:n] if k % 4 == 0 else rng.permutation([0, 0, 1, 1, 2])[:n], es)
          for k in range(4) for n, es in shapes]
    e = d.Engine(0)
    e.set_option(d.OPT_FILTER, 2)
    e.set_option(d.OPT_LIST, 0)
    e.set_option(d.OPT_WORK_LIMIT, 100)
    e.load_graph_edges(nv, labels, edges)
    qids = [e.register(q) for q in qs]
    e.run_batch(np.array([[1, *edges[0], 0]], np.uint32))  # there already: the filter's graph is the one loaded
    off, nb = e.export_graph()
    for qid, q in zip(qids, qs):
        bm, vc, (full, _) = e.filter_state(qid, q.nv, nv)
        obm, ovc, _, _ = orc.cluster_filter(q.labels, q.offsets, q.nbrs, nv, labels, off, nb)
        assert full and np.array_equal(vc, ovc)
        assert np.array_equal(bm, obm), f"query {qid}: bitmaps differ at u {np.nonzero((bm != obm).any(1))[0]}"
    assert any(b.any() for b in obm)
    e.close()


def test_ranges_laid_in_several_rounds(tmp_path):
    """The filter's block-wide ranges with rounds of 5 entries a vertex, in a
    library built for the purpose: bitmaps, masks and regions as ever."""
    import os
    import shutil
    import subprocess
    import sys

    from dsm_b200 import build as b
    pkg = tmp_path / "dsm_b200"
    pkg.mkdir()
    shutil.copy(os.path.join(b.HERE, "__init__.py"), pkg)
    objs = []
    for src in b.LIB_SOURCES:  # the build's objects, but for the filter's (and any that is not there)
        obj = os.path.join(b.BUILD, src.replace("/", "_") + ".o")
        if src == "engine/filter.cu" or not os.path.exists(obj):
            obj = str(tmp_path / os.path.basename(obj))
            flags = [*b.CU_FLAGS, "-DDSM_RANGE_SPAN=5"] if src.endswith(".cu") else b.CXX_FLAGS
            subprocess.run([b.NVCC, *flags, "-c", os.path.join(b.CSRC, src), "-o", obj], check=True)
        objs.append(obj)
    subprocess.run([b.NVCC, *b.ARCH, "-shared", "-o", str(pkg / "libdsm.so"), *objs, "-lcudart"], check=True)
    script = """
import dsm_b200, tests.test_gpu_filter as t
assert dsm_b200.__file__.startswith({tmp!r})
for nv, labels in ((257, 32), (700, 3)):
    t.test_filter_at_the_edges_of_its_tiles(nv, labels)
t.test_region_list_fills_within_a_hop(30_000, 3)
t.test_region_list_fills_within_a_hop(65_530, 4)
t.test_incremental_filter_equals_full(1, 0, 1, 32, 10)
""".format(tmp=str(tmp_path))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([str(tmp_path), b.ROOT]))
    r = subprocess.run([sys.executable, "-c", script], env=env, cwd=str(tmp_path), capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("first,second", [(40, 3000), (3000, 40)])
def test_another_graph_under_registered_queries(first, second):
    """A graph of another size loaded while queries stay registered and
    filtered: the bitmaps' rows are the new graph's."""
    rng = np.random.default_rng(first)
    q = d.Query.from_edges([0, 1, 2, 1], [(0, 1), (1, 2), (2, 3)])
    e = d.Engine(0)
    e.set_option(d.OPT_FILTER, 2)
    qid = None
    for nv in (first, second, first):
        labels = rng.integers(0, 3, nv).astype(np.uint32)
        edges = rng.integers(0, nv, (8 * nv, 2)).astype(np.uint32)
        edges = edges[edges[:, 0] != edges[:, 1]]
        e.load_graph_edges(nv, labels, edges)
        if qid is None:
            qid = e.register(q)
        st = oracle_stream(nv, labels, edges, q)
        a = rng.integers(0, nv, 24)
        ups = np.stack([rng.integers(0, 2, 24), a, (a + 1 + rng.integers(0, nv - 1, 24)) % nv, 0 * a], 1).astype(np.uint32)
        total, _ = run_stream(e, [qid], [st], [ups, ups[::-1].copy()], check_graph_every=1)
        assert total > 0
    e.close()


def test_a_query_s_filter_between_captured_batches():
    """dsm_query_filter between filtered batches: bitmaps as the oracle's, the
    batches' captured segments replayed, not captured again."""
    w = workload(2, scale_log2=-4, num_batches=1)
    ups, qs = next(w.batches()), w.queries[:3]
    inc, full = _inc_pair(w, qs, OPT_GRAPH=1)
    captures = []
    for k in range(8):
        b = ups[k * 16:(k + 1) * 16]
        ri, rf = inc[0].run_batch(b), full[0].run_batch(b)
        assert np.array_equal(ri.counts, rf.counts)
        _same_state(inc, full, qs, w.nv, f"batch {k}")
        q = qs[k % 3]
        bm, vc = inc[0].filter(inc[1][k % 3], q.nv, w.nv)
        obm, ovc, _, _ = orc.cluster_filter(q.labels, q.offsets, q.nbrs, w.nv, w.labels, *inc[0].export_graph())
        assert np.array_equal(vc, ovc) and np.array_equal(bm, obm)
        captures.append(inc[0].stats()["graph_captures"])
    assert captures[-1] == captures[2], captures
    for e, _ in (inc, full):
        e.close()
