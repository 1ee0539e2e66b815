"""Pre-count by sums (count mode, one back edge at each of the last two depths):
counts and the per-level work counters equal the oracle's enumeration on
graphs where the two lists meet in every way -- pairs joined by two labels (a
vertex's lists of two labels share neighbours), hubs longer than a piece and
than the block limit of the vertex sums, lists of every kind, graphs whose
e-lines lack their reverse or loop (where the rule must not be used), and level
buffers small enough to drain.  Integer work: no tolerance."""
import numpy as np
import pytest

import forkmatch_gb300 as fm
from forkmatch_gb300 import synth as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from forkmatch_gb300 import build
    build.build()
    c = fm.Context(prealloc_bytes=2 << 30, soln_prealloc_bytes=512 << 20, output_prealloc_bytes=64 << 20,
                   bank_rows=256)
    yield c
    c.close()


def _edges(kind):
    """Directed e-lines (src, dst, label), no duplicates."""
    rng = np.random.default_rng(17)
    n, m = 6000, 27000                               # over 4096 lists of each label: the rule's least
    a, b = rng.integers(0, n, m), rng.integers(0, n, m)
    lab = rng.integers(1, 4, m)
    if kind == "hub":                                # label 1: two hubs of 1500 common neighbours
        x = np.arange(2, 1502)
        a = np.concatenate([a, np.zeros(1500, int), np.ones(1500, int)])
        b = np.concatenate([b, x, x])
        lab = np.concatenate([lab, np.ones(1500, int), np.where(x % 3 == 0, 1, 2)])
    if kind == "two_labels":                         # every third edge carries a second label
        a, b, lab = np.concatenate([a, a[::3]]), np.concatenate([b, b[::3]]), np.concatenate([lab, lab[::3] % 3 + 1])
    keep = a != b
    a, b, lab = a[keep], b[keep], lab[keep]
    e = np.stack([np.concatenate([a, b]), np.concatenate([b, a]), np.concatenate([lab, lab])], 1)
    if kind == "one_way":
        e = e[rng.random(len(e)) < 0.8]
    if kind == "loops":
        v = np.arange(0, n, 5)
        e = np.concatenate([e, np.stack([v, v, np.ones(len(v), int)], 1)])
    e = np.unique(e, axis=0).astype(np.uint32)
    return n, [np.ascontiguousarray(e[:, i]) for i in range(3)]


def _queries():
    """Paths, stars, and trees whose last two vertices hang on different ancestors, labels equal and mixed."""
    qs = [S.query_path(4, [1, 2, 3]), S.query_path(4, [1, 1, 1]), S.query_path(4, [2, 1, 2]),
          S.query_path(5, [1, 2, 1, 2]), S.query_path(5, [3, 1, 2, 3]), S.query_star(4, [1, 2, 3]),
          S.query_star(4, [1, 1, 2]), S.query_star(4, [2, 2, 2]),
          S.Query(5, [(0, 1, 1), (0, 2, 2), (1, 3, 3), (2, 4, 1)]), S.Query(5, [(0, 1, 2), (1, 2, 1), (1, 3, 2), (0, 4, 1)]),
          S.Query(5, [(0, 1, 1), (1, 2, 2), (0, 2, 3), (2, 3, 1), (3, 4, 2)])]
    return [q.to_g_text() for q in qs]


@pytest.mark.parametrize("bitmaps", ["default", "none", "short"])
@pytest.mark.parametrize("kind", ["plain", "two_labels", "hub", "one_way", "loops"])
def test_sums_equal_enumeration(ctx, monkeypatch, kind, bitmaps):
    if bitmaps == "none":
        monkeypatch.setenv("FM_BITMAP_BYTES", "0")
    if bitmaps == "short":
        monkeypatch.setenv("FM_BITMAP_MIN_LEN", "4")
    V, (src, dst, lab) = _edges(kind)
    g = fm.Graph.from_edges(ctx, V, 4, src, dst, lab)
    og = O.Graph.from_edges(V, 4, src, dst, lab)
    small = fm.Context(prealloc_bytes=256 << 20, soln_prealloc_bytes=8 * 4 * 7 * (32 * g.info().max_list + 64) + 128 * V,
                       output_prealloc_bytes=1 << 20, bank_rows=1)
    for text in _queries():
        p = O.plan(text, enumerate_aut=0)
        want, _, st = O.match(og, p, count_rule=True, limit=1 << 40)
        q = fm.Query.from_text(text)
        # an e-line is read from the vertex matched first, so without its
        # reverse the count belongs to one order: the oracle's is the reference's
        for order in (fm.ORDER_REFERENCE,) if kind == "one_way" else (fm.ORDER_REFERENCE, fm.ORDER_AUTO):
            assert fm.match(ctx, g, q, mode=fm.MODE_COUNT, order=order).count == want
            assert fm.match(small, g, q, mode=fm.MODE_COUNT, order=order).count == want
        r = fm.match(ctx, g, q, mode=fm.MODE_COUNT, order=fm.ORDER_REFERENCE)
        assert r.count == want
        for d in range(2, p.q):
            assert r.level[d].lookups == st.lookups[d], ("lookups", d)
            assert r.level[d].list_words == st.list_words[d], ("list_words", d)
            assert r.level[d].parents == st.partials[d - 1], ("parents", d)
        for d in range(1, p.q - 1):
            assert r.level[d].produced == st.partials[d], ("produced", d)
    # the same queries in shared launches, counting and as count-only ones of a table batch
    queries = [fm.Query.from_text(t) for t in _queries()]
    want = [fm.match(ctx, g, q, mode=fm.MODE_COUNT).count for q in queries]
    for mode, engine in ((fm.MODE_COUNT, fm.ENGINE_LEVELS), (fm.MODE_COUNT, fm.ENGINE_PERSISTENT),
                         (fm.MODE_TABLE, fm.ENGINE_LEVELS)):
        for c in (ctx, small):
            b = fm.Batch(c, g, queries, mode=mode)
            b.set_engine(engine)
            for i in range(len(queries)):
                b.set_query_mode(i, fm.MODE_COUNT)
            assert b.run()[0] == want and b.run()[0] == want
            b.close()
    small.close()
    g.close()


def _uneven(n, m):
    """n vertices, about m edges; one edge in 50 carries label 1, the others 2 to 4 (fewer than 4096 lists of each)."""
    rng = np.random.default_rng(3)
    a, b = rng.integers(0, n, m), rng.integers(0, n, m)
    lab = np.where(rng.random(m) < 0.02, 1, rng.integers(2, 5, m))
    keep = a != b
    e = np.unique(np.stack([np.minimum(a, b)[keep], np.maximum(a, b)[keep]], 1), axis=0, return_index=True)[1]
    a, b, lab = a[keep][e], b[keep][e], lab[keep][e]
    return [np.concatenate(x).astype(np.uint32) for x in ((a, b), (b, a), (lab, lab))]


@pytest.mark.parametrize("edges,labels", [(20000, [2, 3, 4, 2]), (60000, [2, 3, 4, 2]), (60000, [1, 2, 1, 3]),
                                          (400000, [3, 1, 2, 1])])
def test_fork_orders_come_with_sums(ctx, edges, labels):
    """A fork order is not costed for candidates of its last two depths, so a count that takes one counts those by
    sums, on few lists too; the count is the one of the table's order."""
    g = fm.Graph.from_edges(ctx, 3000, 5, *_uneven(3000, edges))
    q = fm.Query.from_text(S.query_path(5, labels).to_g_text())
    t = fm.match(ctx, g, q, mode=fm.MODE_TABLE, allow_truncation=True)
    c = fm.match(ctx, g, q, mode=fm.MODE_COUNT)
    assert c.count == t.count and c.routes in (0, fm.ROUTE_SUMS, fm.ROUTE_SUMS | fm.ROUTE_FORK)
    if labels == [2, 3, 4, 2]:                       # equally frequent: a fork's other vertices cost the same
        assert c.routes & fm.ROUTE_FORK
    # no fork order where nothing is counted by sums
    assert fm.match(ctx, g, q, mode=fm.MODE_COUNT, work_limit=1 << 62).routes == 0
    g.close()


def test_no_fork_order_is_planned_for_few_candidates(ctx):
    """A 24-vertex path on a graph with half a neighbour a label: nothing to spare, no plan."""
    g = fm.Graph.from_edges(ctx, 3000, 5, *_uneven(3000, 3000))
    q = fm.Query.from_text(S.query_path(24, [2 + i % 3 for i in range(23)]).to_g_text())
    t = fm.match(ctx, g, q, mode=fm.MODE_TABLE, allow_truncation=True)
    c = fm.match(ctx, g, q, mode=fm.MODE_COUNT)
    assert c.count == t.count and not c.routes & fm.ROUTE_FORK
    g.close()


def _long_lists(ctx):
    """5000 vertices, 100000 edges of labels 2 and 3 and 40 of label 1."""
    rng = np.random.default_rng(4)
    n = 5000
    e = np.unique(np.sort(rng.integers(0, n, (100000, 2)), axis=1), axis=0)
    e = e[e[:, 0] != e[:, 1]]
    lab = rng.integers(2, 4, len(e))
    lab[:40] = 1
    src, dst, lab = [np.concatenate(x).astype(np.uint32) for x in ((e[:, 0], e[:, 1]), (e[:, 1], e[:, 0]), (lab, lab))]
    return fm.Graph.from_edges(ctx, n, 4, src, dst, lab)


def test_batches_compute_vertex_sums_only_where_they_pay(ctx):
    """A table of vertex sums reads every e-line of its label.  Paths whose first label is rare meet few of them: no
    table; paths over frequent labels of a graph with long lists: one a pair of labels, shared by its queries."""
    g = _long_lists(ctx)
    per = 2 if g.info().max_list > 16 else 1
    for labels, shared in (([[1, 2, 3], [1, 3, 2], [1, 2, 2]], None), ([[2, 3, 2], [2, 3, 2]], 1),
                           ([[2, 3, 2], [2, 2, 2], [3, 3, 3]], 0)):
        qs = [fm.Query.from_text(S.query_path(4, l).to_g_text()) for l in labels]
        b = fm.Batch(ctx, g, qs, mode=fm.MODE_COUNT)
        want = [fm.match(ctx, g, q, mode=fm.MODE_COUNT, order=fm.ORDER_REFERENCE).count for q in qs]
        # a count of its own launches the vertex sums if its order needs them
        alone = [fm.match(ctx, g, q, mode=fm.MODE_COUNT) for q in qs]
        tables = 0 if shared is None else sum(r.launches - per * r.passes for r in alone) - shared
        assert shared is None or tables >= 1
        for _ in range(2):
            counts, st = b.run()
            assert counts == want and st.launches == 3 * per + tables
        b.close()
    g.close()


def test_table_batches_keep_their_level_memory(ctx):
    """A table batch counts every query once, to size the tables; after that the level region has no tables of vertex
    sums but those of its count-only queries, and its level buffers take the rest."""
    g = _long_lists(ctx)
    qs = [fm.Query.from_text(S.query_path(4, l).to_g_text()) for l in ([2, 3, 2], [2, 2, 2])] + \
        [fm.Query.from_text(S.query_cycle(3, [1, 2, 3]).to_g_text())]
    want = [fm.match(ctx, g, q, mode=fm.MODE_COUNT, order=fm.ORDER_REFERENCE).count for q in qs]
    full = (512 << 20) // (4 * (3 + 4))              # rows of 3 and 4 words at depths 2 and 3
    c = fm.Batch(ctx, g, qs, mode=fm.MODE_COUNT)
    counted, st = c.run()
    assert counted == want and st.level_rows < full
    c.close()
    b = fm.Batch(ctx, g, qs, mode=fm.MODE_TABLE)
    for engine in (fm.ENGINE_LEVELS, fm.ENGINE_PERSISTENT):
        b.set_engine(engine)
        for _ in range(3):                           # sizing, captured and replayed
            counted, st = b.run(allow_truncation=True)
            assert counted == want and st.level_rows == full
    b.set_query_mode(0, fm.MODE_COUNT)               # sized again, then one query counted by sums
    for _ in range(3):
        counted, st = b.run(allow_truncation=True)
        assert counted == want and st.level_rows < full
    b.set_solo(0, True)                              # matched alone: its table goes
    for _ in range(2):
        counted, st = b.run(allow_truncation=True)
        assert counted == want and st.level_rows == full
    b.set_solo(0, False)
    b.set_query_mode(0, fm.MODE_TABLE)
    for _ in range(2):
        counted, st = b.run(allow_truncation=True)
        assert counted == want and st.level_rows == full
    assert len(b.rows(2, want[2])) == want[2]
    b.close()
    g.close()
