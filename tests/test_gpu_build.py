"""Device graph build and text parse at the edges of their tiles (512 keys a
warp, 4096 keys a block, 1024 segments a block, 4096 bytes of text a block):
the graph's totals equal numpy's on the same e-lines and the 2-vertex path of
every label lists exactly that label's e-lines.  Integer work: no tolerance."""
import numpy as np
import pytest

import forkmatch_gb300 as fm
from forkmatch_gb300 import synth as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from forkmatch_gb300 import build
    build.build()
    c = fm.Context(prealloc_bytes=1 << 30, soln_prealloc_bytes=256 << 20, output_prealloc_bytes=256 << 20,
                   bank_rows=256)
    yield c
    c.close()


def _lines(E, V, L, hub, dup, seed):
    """E distinct e-lines (plus repeats of the first with `dup`), vertex 0's label-1 list holding `hub` of them."""
    rng = np.random.default_rng(seed)
    key = set()
    while len(key) < min(hub, E):
        key.add((1, 0, int(rng.integers(0, V))))
    while len(key) < E:
        key.add((int(rng.integers(1, L)), int(rng.integers(0, V)), int(rng.integers(0, V))))
    a = np.array(sorted(key), dtype=np.uint32).reshape(-1, 3)
    a = a[rng.permutation(len(a))]
    if dup and E:
        a = np.concatenate([a, a[:dup]])
    return np.ascontiguousarray(a[:, 1]), np.ascontiguousarray(a[:, 2]), np.ascontiguousarray(a[:, 0])


@pytest.mark.parametrize("form", ["edges", "text"])
@pytest.mark.parametrize("E,V,L,hub,dup", [
    (0, 5, 2, 0, 0), (1, 1, 2, 0, 0), (511, 40, 3, 0, 0), (512, 3000, 3, 0, 0), (513, 3000, 2, 513, 0),
    (1024, 5000, 3, 4, 0), (1025, 1 << 20, 3, 0, 0), (4095, 65, 4, 60, 0), (4096, 70000, 256, 0, 0),
    (4097, 9000, 3, 4000, 3), (8193, 20000, 2, 8000, 0), (70001, 30011, 5, 9001, 1)])
def test_build_totals_and_lists(ctx, form, E, V, L, hub, dup):
    src, dst, lab = _lines(E, V, L, hub, dup, seed=E + V)
    if form == "edges":
        g = fm.Graph.from_edges(ctx, V, L, src, dst, lab)
    else:
        g = fm.Graph.from_text(ctx, S.g_text(V, np.ones(V, dtype=np.uint32), src, dst, lab, 1, L - 1))
    gi = g.info()
    seg = np.unique(lab.astype(np.uint64) * V + src, return_counts=True)[1] if len(src) else np.zeros(0, np.int64)
    assert (gi.vertices, gi.label_slots, gi.edges, gi.segments) == (V, L, len(src), len(seg))
    assert gi.long_segments == int((seg > 3).sum()) and gi.max_list == (int(seg.max()) if len(seg) else 0)
    assert gi.nbr_words == int(((seg[seg > 3] + 3) // 4 * 4).sum()) and bool(gi.has_duplicates) == bool(dup)
    for l in sorted(set(lab.tolist()))[:6]:
        q = fm.Query.from_text(S.query_path(2, [l]).to_g_text())
        n, rows, _ = fm.match_table(ctx, g, q, max_rows=1 << 17, columns=fm.COLUMNS_QUERY_ID)
        m = (lab == l) & (src != dst)         # a path's vertices are distinct
        assert n == int(m.sum())
        # one of the two directions of the pattern: (vertex 0, vertex 1) or (vertex 1, vertex 0)
        got = sorted(map(tuple, rows.tolist()))
        want = list(zip(src[m].tolist(), dst[m].tolist()))
        assert got == sorted(want) or got == sorted((b, a) for a, b in want)
    g.close()


@pytest.mark.parametrize("E,V,L,hub,dup", [(0, 5, 2, 0, 0), (1, 1, 2, 0, 0), (513, 3000, 2, 513, 0), (4095, 65, 4, 60, 0),
                                           (4097, 9000, 3, 4000, 3), (70001, 30011, 5, 9001, 1)])
def test_texts_whose_lines_are_counted_first(ctx, monkeypatch, E, V, L, hub, dup):
    """The way of texts above the size limit, where the lines are counted before the build's arrays are sized."""
    monkeypatch.setenv("FM_INGEST_BOUND_BYTES", "0")
    test_build_totals_and_lists(ctx, "text", E, V, L, hub, dup)


@pytest.mark.parametrize("body,status", [
    ("", 0), ("\n" * 5000, 6), ("v 0 1\n" * 3 + "\n" * 900, 6), ("e 0 1 1\ne 1 0 1\n", 0), ("e 0 1 1\n" * 4, 6),
    ("v 0 1\ne 0 1 1\ne 0 4 1\ne 1 0 1\n", 6), ("e 0 1 1\nx 1 0 1\n", 6), ("e 0 1 1\ne 1 0 4294967296\n", 6),
    ("e 0 1 1\ne 1 0 1", 6), ("v 4 1\n" * 700, 6), ("v 3 1\n" * 700 + "v 3\n" + "v 4 1\n" * 700, 6)])
def test_both_ways_of_texts_refuse_the_same_lines(ctx, monkeypatch, body, status):
    """4 vertices, a header of 2 e-lines; FM_ERR_DATA_LINE is 6."""
    text = "t # 0\n4 2 1 2\n" + body + "t # -1"
    got = []
    for limit in (str(1 << 30), "0"):
        monkeypatch.setenv("FM_INGEST_BOUND_BYTES", limit)
        try:
            g = fm.Graph.from_text(ctx, text)
            got.append((0, g.info().edges, ""))
            g.close()
        except fm.FMError as e:
            got.append((e.status, 0, str(e)))
    assert got[0] == got[1] and got[0][0] == status
