"""The e-line filter and the queue of candidates it lets pass: graphs where every
candidate passes (complete graphs: full queues, remainders at every chunk's
end), and labels whose slice is one word.  Closed forms; no tolerance."""
import math

import numpy as np
import pytest

import forkmatch_gb300 as fm
from forkmatch_gb300 import synth as S
from tests.helpers import complete_graph

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
