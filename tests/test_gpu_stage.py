"""Levels whose every candidate survives (one back edge a query): their survivors
are staged in blocks of 256 rows, two slots a lane before each look at the
stage.  Lists around the block's bounds, alone and in shared launches, with and
without duplicate e-lines: the table's rows are the oracle's, as a multiset.
Integer work: no tolerance."""
import numpy as np
import pytest

import forkmatch_gb300 as fm
from forkmatch_gb300 import synth as S
from oracle import oracle as O
from tests.helpers import star_graph, table_sha

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from forkmatch_gb300 import build
    build.build()
    c = fm.Context(prealloc_bytes=1 << 30, soln_prealloc_bytes=256 << 20, output_prealloc_bytes=512 << 20,
                   bank_rows=256)
    yield c
    c.close()


@pytest.mark.parametrize("dup", [0, 5])
@pytest.mark.parametrize("leaves", [31, 33, 64, 65, 191, 193, 224, 225, 256, 257])
def test_every_candidate_is_staged(ctx, leaves, dup):
    V, src, dst, lab = star_graph(leaves)
    src, dst, lab = [np.concatenate([x, x[:dup]]) for x in (src, dst, lab)]
    g = fm.Graph.from_edges(ctx, V, 2, src, dst, lab)
    og = O.Graph.from_edges(V, 2, src, dst, lab)
    queries = [S.query_path(2, [1]).to_g_text(), S.query_path(3, [1, 1]).to_g_text()]
    if leaves < 70:
        queries.append(S.query_star(4, [1, 1, 1]).to_g_text())
    want = [O.match(og, O.plan(t, enumerate_aut=0), table=True) for t in queries]
    for t, (n, rows, _) in zip(queries, want):
        q = fm.Query.from_text(t)
        for engine in (fm.ENGINE_LEVELS, fm.ENGINE_PERSISTENT):
            buf = np.zeros(max(1, n) * q.q, dtype=np.uint32)
            r = fm.match(ctx, g, q, host_rows=buf, engine=engine)
            assert r.count == n == r.rows_copied
            assert table_sha(buf.reshape(-1, q.q)[:n]) == table_sha(rows)
        assert fm.match(ctx, g, q, mode=fm.MODE_COUNT).count == n
    b = fm.Batch(ctx, g, [fm.Query.from_text(t) for t in queries], mode=fm.MODE_TABLE)
    for engine in (fm.ENGINE_LEVELS, fm.ENGINE_PERSISTENT):
        b.set_engine(engine)
        assert b.run()[0] == [n for n, _, _ in want]
        if not dup:                      # with duplicates a batch only counts
            for i, (n, rows, _) in enumerate(want):
                assert table_sha(b.rows(i, n)) == table_sha(rows)
    b.close()
    g.close()


@pytest.mark.parametrize("n", [7, 33, 48])
def test_a_batch_mixes_levels_with_one_and_two_back_edges(ctx, n):
    """Shared levels that take both ways at once: chunks whose parents have one back edge go straight on, chunks of a
    triangle's last depth through the filter, into one stage."""
    src, dst = np.nonzero(~np.eye(n, dtype=bool))
    lab = 1 + (src + dst) % 2
    g = fm.Graph.from_edges(ctx, n, 3, *[x.astype(np.uint32) for x in (src, dst, lab)])
    og = O.Graph.from_edges(n, 3, *[x.astype(np.uint32) for x in (src, dst, lab)])
    texts = [q.to_g_text() for q in (S.query_path(4, [1, 2, 1]), S.query_cycle(3, [1, 1, 2]), S.query_path(3, [1, 1]),
                                     S.Query(4, [(0, 1, 1), (1, 2, 2), (0, 2, 1), (2, 3, 1)]))]
    want = [O.match(og, O.plan(t, enumerate_aut=0), table=True) for t in texts]
    for mode in (fm.MODE_TABLE, fm.MODE_COUNT):
        b = fm.Batch(ctx, g, [fm.Query.from_text(t) for t in texts], mode=mode)
        for engine in (fm.ENGINE_LEVELS, fm.ENGINE_PERSISTENT):
            b.set_engine(engine)
            assert b.run()[0] == [c for c, _, _ in want] and b.run()[0] == [c for c, _, _ in want]
            if mode == fm.MODE_TABLE:
                for i, (c, rows, _) in enumerate(want):
                    assert table_sha(b.rows(i, c)) == table_sha(rows)
        b.close()
    g.close()
