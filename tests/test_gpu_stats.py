"""What a match reports about itself: the kernels it launched, the bytes it read
back, the device bytes of a graph, and the ways its level passes took (counting
by sums, shared intersections) -- which counts and work counters cannot show,
since every way gives the same ones.  Integer work: no tolerance."""
import ctypes

import numpy as np
import pytest

import forkmatch_gb300 as fm
from forkmatch_gb300 import synth as S
from tests.helpers import complete_graph, star_graph
from tests.test_gpu_sums import _edges, _queries

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from forkmatch_gb300 import build
    build.build()
    c = fm.Context(prealloc_bytes=2 << 30, soln_prealloc_bytes=512 << 20, output_prealloc_bytes=256 << 20,
                   bank_rows=256)
    yield c
    c.close()


@pytest.mark.parametrize("dup", [0, 7])
@pytest.mark.parametrize("V,L,E", [(50, 2, 0), (300, 4, 900), (5000, 33, 40001)])
def test_device_bytes(ctx, V, L, E, dup):
    rng = np.random.default_rng(V)
    key = np.unique(np.stack([rng.integers(1, L, E), rng.integers(0, V, E), rng.integers(0, V, E)], 1), axis=0)
    key = np.concatenate([key, key[:dup]]).astype(np.uint32)
    g = fm.Graph.from_edges(ctx, V, L, key[:, 1], key[:, 2], key[:, 0])
    i = g.info()
    per_label = np.bincount(key[:, 0], minlength=L)
    filt = 0 if i.has_duplicates else 4 * int((per_label // 2 + 1).sum()) + 4 * (L + 1)
    assert bool(i.has_duplicates) == (E > 0 and dup > 0)
    assert i.device_bytes == 16 * L * V + 4 * i.nbr_words + 4 * i.segments + i.bitmap_bytes + filt
    g.close()


@pytest.mark.parametrize("n", [17, 18])
def test_launches_are_kernels(ctx, n):
    """Complete graphs whose longest list is 16 (main passes only) and 17 (main and heavy)."""
    V, s, d, l = complete_graph(n)
    g = fm.Graph.from_edges(ctx, V, 2, s, d, l)
    per = 1 if n == 17 else 2
    qs = [fm.Query.from_text(q.to_g_text()) for q in (S.query_cycle(3, [1] * 3), S.query_clique(4, [1]))]
    for q in qs:
        for mode in (fm.MODE_COUNT, fm.MODE_TABLE):
            r = fm.match(ctx, g, q, mode=mode)
            assert (r.passes, r.launches) == (q.q - 1, per * (q.q - 1))
            assert sum(r.level[i].launches for i in range(q.q)) == r.passes
    b = fm.Batch(ctx, g, qs, mode=fm.MODE_COUNT)
    for _ in range(2):                               # the captured run and its replay
        assert b.run()[1].launches == per * 3
    b.close()
    g.close()


def test_bytes_read_back(ctx):
    """Control blocks and totals, the first rows of a table that a host buffer asks for, and the rows copied later."""
    V, s, d, l = star_graph(300)
    g = fm.Graph.from_edges(ctx, V, 2, s, d, l)
    q = fm.Query.from_text(S.query_path(3, [1, 1]).to_g_text())
    base = fm.match(ctx, g, q, mode=fm.MODE_COUNT).d2h_bytes
    assert 32 * 48 < base < 4096                     # 32 control blocks and the totals
    assert fm.match(ctx, g, q, mode=fm.MODE_TABLE).d2h_bytes == base
    n = 300 * 299
    for cap, more in ((10, 10 * 12), (1365, 1365 * 12), (1366, 16384 + 1366 * 12), (n, 16384 + n * 12)):
        r = fm.match(ctx, g, q, host_rows=np.zeros(cap * 3, dtype=np.uint32))
        assert r.rows_copied == cap and r.d2h_bytes == base + more
    rows = fm.PinnedRows(n, 3)
    assert fm.match(ctx, g, q, host_rows=rows, host_direct=True).d2h_bytes == base + n * 12
    g.close()


@pytest.mark.parametrize("kind", ["plain", "two_labels", "hub", "one_way", "loops"])
def test_sums_are_taken_where_they_may(ctx, kind):
    V, (src, dst, lab) = _edges(kind)
    g = fm.Graph.from_edges(ctx, V, 4, src, dst, lab)
    taken, per = 0, 2 if g.info().max_list > 16 else 1
    for i, text in enumerate(_queries()):
        q = fm.Query.from_text(text)
        qi = q.info()
        r = fm.match(ctx, g, q, mode=fm.MODE_COUNT, order=fm.ORDER_REFERENCE)
        two = qi.nreq[q.q - 2] == qi.nreq[q.q - 1] == 1
        chain = two and qi.req_climb[q.q - 1][0] == 1
        may = two and kind != "loops" and not (chain and kind == "one_way")
        vertex = may and (chain or (qi.req_climb[q.q - 1][0] == qi.req_climb[q.q - 2][0] + 1 and
                                    qi.req_label[q.q - 2][0] != qi.req_label[q.q - 1][0]))
        if vertex:
            # a quarter as many parents as the vertex sums read lists, at least: decided on the device, after the launch
            lists = len(np.unique(src[lab == qi.req_label[q.q - 2][0]]))
            assert lists >= 4096
            may = 4 * r.level[q.q - 2].parents >= lists
        assert bool(r.routes & fm.ROUTE_SUMS) == may, i
        assert r.launches == per * r.passes + vertex, i
        taken += may
        # neither a table, nor the persistent engine, nor a work limit takes it
        for kw in (dict(mode=fm.MODE_TABLE, allow_truncation=True), dict(mode=fm.MODE_COUNT, engine=fm.ENGINE_PERSISTENT),
                   dict(mode=fm.MODE_COUNT, work_limit=1 << 40)):
            assert fm.match(ctx, g, q, order=fm.ORDER_REFERENCE, **kw).routes == 0
        a = fm.match(ctx, g, q, mode=fm.MODE_COUNT)
        assert not a.routes & fm.ROUTE_FORK or a.routes & fm.ROUTE_SUMS
    assert taken >= 6 if kind in ("plain", "two_labels", "hub") else taken == 0 if kind == "loops" else taken >= 2
    g.close()


def test_result_layout():
    assert ctypes.sizeof(fm.Result) % 8 == 0 and fm.Result.routes.offset + 4 == ctypes.sizeof(fm.Result)
