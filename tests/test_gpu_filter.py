"""The e-line filter and the queue of candidates it lets pass: graphs where every
candidate passes (complete graphs: full queues, remainders at every chunk's
end), and labels whose slice is one word.  Closed forms; no tolerance."""
import math

import numpy as np
import pytest

import forkmatch_gb300 as fm
from forkmatch_gb300 import synth as S
from oracle import oracle as O
from tests.helpers import complete_graph, table_sha

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from forkmatch_gb300 import build
    build.build()
    c = fm.Context(prealloc_bytes=1 << 30, soln_prealloc_bytes=512 << 20, output_prealloc_bytes=256 << 20,
                   bank_rows=256)
    yield c
    c.close()


# 17 and 18: the longest list (16, 17) without and with a heavy pass
@pytest.mark.parametrize("n", [3, 4, 17, 18, 31, 32, 33, 34, 65])
def test_every_candidate_passes(ctx, n):
    V, s, d, l = complete_graph(n)
    g = fm.Graph.from_edges(ctx, V, 2, s, d, l)
    for q in (S.query_cycle(3, [1] * 3), S.query_cycle(4, [1] * 4), S.query_clique(4, [1])):
        query = fm.Query.from_text(q.to_g_text())
        want = math.perm(n, q.k)
        assert fm.match(ctx, g, query, mode=fm.MODE_COUNT).count == want
        cnt, rows, _ = fm.match_table(ctx, g, query, max_rows=max(1, want))
        assert cnt == want == len(rows) == len(np.unique(rows, axis=0))
        assert all(len(set(r)) == q.k for r in rows[:100].tolist())
    g.close()


@pytest.mark.parametrize("labels", [1, 3, 255])
def test_one_edge_per_label(ctx, labels):
    """A triangle whose edges carry labels of their own, among other single edges."""
    e = [(0, 1, 1), (1, 2, min(2, labels)), (2, 0, min(3, labels))] + [(0, 10 + i, 1 + i) for i in range(3, labels)]
    src = np.array([a for a, _, _ in e] + [b for _, b, _ in e], dtype=np.uint32)
    dst = np.array([b for _, b, _ in e] + [a for a, _, _ in e], dtype=np.uint32)
    lab = np.array([x for _, _, x in e] * 2, dtype=np.uint32)
    g = fm.Graph.from_edges(ctx, 300, labels + 1, src, dst, lab)
    q = fm.Query.from_text(S.query_cycle(3, [1, min(2, labels), min(3, labels)]).to_g_text())
    assert fm.match(ctx, g, q, mode=fm.MODE_COUNT).count == (6 if labels == 1 else 1)
    g.close()


def test_shared_intersections(ctx):
    """Levels with enough chunks to share the intersection of their two oldest lists: it fits the buffer (complete
    graph), it does not for pairs of hubs and does for a hub and a leaf (hubs joined to everything), and it is the
    whole candidate list (a vertex on two old ones, the newest column free)."""
    V, s, d, l = complete_graph(104)
    g = fm.Graph.from_edges(ctx, V, 2, s, d, l)
    k4 = fm.Query.from_text(S.query_clique(4, [1]).to_g_text())
    assert fm.match(ctx, g, k4, mode=fm.MODE_COUNT).count == math.perm(104, 4)
    g.close()
    hubs, leaves = 40, 1100
    e = np.array([(a, b) for a in range(hubs) for b in range(a)] +
                 [(a, hubs + b) for a in range(hubs) for b in range(leaves)], dtype=np.uint32)
    src, dst = np.concatenate([e[:, 0], e[:, 1]]), np.concatenate([e[:, 1], e[:, 0]])
    g = fm.Graph.from_edges(ctx, hubs + leaves, 2, src, dst, np.ones(len(src), dtype=np.uint32))
    for order in (fm.ORDER_AUTO, fm.ORDER_REFERENCE):
        r = fm.match(ctx, g, k4, mode=fm.MODE_COUNT, order=order)
        assert r.count == math.perm(hubs, 4) + 4 * math.perm(hubs, 3) * leaves
    g.close()
    V, s, d, l = complete_graph(40)
    g = fm.Graph.from_edges(ctx, V, 2, s, d, l)
    q = S.Query(5, [(0, 1, 1), (0, 2, 1), (1, 2, 1), (2, 3, 1), (0, 4, 1), (1, 4, 1)])
    query = fm.Query.from_text(q.to_g_text())
    for order in (fm.ORDER_AUTO, fm.ORDER_REFERENCE):
        assert fm.match(ctx, g, query, mode=fm.MODE_COUNT, order=order).count == math.perm(40, 5)
    g.close()


@pytest.mark.parametrize("n", [2, 45, 46, 64])
def test_tables_around_the_first_read_back(ctx, n):
    """Tables just below, at and above the 16 KiB that are read back with the totals, and host buffers smaller than
    the table: 2-vertex rows of a complete graph (45 * 44 * 8 bytes is 15840, 46 * 45 * 8 is 16560)."""
    V, s, d, l = complete_graph(n)
    g = fm.Graph.from_edges(ctx, V, 2, s, d, l)
    q = fm.Query.from_text(S.query_path(2, [1]).to_g_text())
    want = sorted((int(a), int(b)) for a in range(n) for b in range(n) if a != b)
    for cap in {1, len(want) - 1, len(want), len(want) + 7}:
        buf = np.full((cap + 1) * 2, 7, dtype=np.uint32)
        r = fm.match(ctx, g, q, host_rows=buf[:cap * 2])
        assert r.count == len(want) and r.rows_copied == min(cap, len(want))
        rows = list(map(tuple, buf[:2 * r.rows_copied].reshape(-1, 2).tolist()))
        assert len(set(rows)) == len(rows) and set(rows) <= set(want)
        assert (buf[2 * r.rows_copied:] == 7).all()
    g.close()


def test_shared_intersections_of_tables_and_middle_levels(ctx):
    """A dense random graph with 1.1e6 ordered triangles: the table level of 4-cliques and the middle level of 5-cliques
    share; the rows are the oracle's."""
    rng = np.random.default_rng(11)
    n = 420
    a, b = np.nonzero(np.triu(rng.random((n, n)) < 0.25, 1))
    src, dst = [np.concatenate(x).astype(np.uint32) for x in ((a, b), (b, a))]
    lab = np.ones(len(src), dtype=np.uint32)
    g = fm.Graph.from_edges(ctx, n, 2, src, dst, lab)
    og = O.Graph.from_edges(n, 2, src, dst, lab)
    t4, t5 = [S.query_clique(k, [1]).to_g_text() for k in (4, 5)]
    want, rows, _ = O.match(og, O.plan(t4, enumerate_aut=0), table=True, table_cap=1 << 23)
    assert want == len(rows) > 1 << 22
    buf = np.zeros(want * 4, dtype=np.uint32)
    r = fm.match(ctx, g, fm.Query.from_text(t4), host_rows=buf)
    assert r.count == want == r.rows_copied and r.routes == fm.ROUTE_SHARED
    assert table_sha(buf.reshape(-1, 4)) == table_sha(rows)
    r = fm.match(ctx, g, fm.Query.from_text(t5), mode=fm.MODE_COUNT)
    assert r.count == O.match(og, O.plan(t5, enumerate_aut=0), count_rule=True)[0] and r.routes & fm.ROUTE_SHARED
    g.close()


def test_shared_intersections_in_pieces(ctx):
    """Two groups of 20 hubs, all hubs joined, each group joined to 1400 leaves of its own.  Two hubs of one group have
    1438 common neighbours, which do not fit the buffer, and the rows of such a pair with a third hub have about 1439
    candidates each; hubs of different groups have 38, which fit.  Rows of both kinds meet in chunks of more than
    32768 candidates, which the heavy pass loads again, piece by piece."""
    hubs, leaves = 40, 1400
    a, b = np.triu_indices(hubs, 1)
    h, x = [v.ravel() for v in np.meshgrid(np.arange(hubs), np.arange(leaves))]
    a, b = np.concatenate([a, h]), np.concatenate([b, hubs + (h % 2) * leaves + x])
    src, dst = [np.concatenate(v).astype(np.uint32) for v in ((a, b), (b, a))]
    g = fm.Graph.from_edges(ctx, hubs + 2 * leaves, 2, src, dst, np.ones(len(src), dtype=np.uint32))
    want = math.perm(hubs, 4) + 2 * 4 * math.perm(hubs // 2, 3) * leaves
    k4 = fm.Query.from_text(S.query_clique(4, [1]).to_g_text())
    for mode in (fm.MODE_COUNT, fm.MODE_TABLE):
        for order in (fm.ORDER_AUTO, fm.ORDER_REFERENCE):
            r = fm.match(ctx, g, k4, mode=mode, order=order, allow_truncation=True)
            assert r.count == want and r.routes == fm.ROUTE_SHARED | fm.ROUTE_SHARED_PIECES
    g.close()
