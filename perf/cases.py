"""Performance cases: the matching work this library is used for, one pass per call of its public API.

Data graphs are the shapes of the library's own configurations (``forkmatch_gb300/workloads.py`` and the test
suite): Erdos-Renyi, R-MAT(0.57, 0.19, 0.19, 0.05) and Chung-Lu with exponent 2.1, generated on the device from the
seed.  A case names a graph (kind, vertices, undirected edges, edge labels), a set of queries and what a pass does with
them.  Matches return whole numbers; a table's row order is unspecified, so tables come back as row sets in a fixed
order, in buffers as large as a query's table may get.
"""
import numpy as np
import torch

import forkmatch_gb300 as fm
from forkmatch_gb300 import synth as S

MB, GB = 1 << 20, 1 << 30
WALK_PARTIALS = 1 << 23       # partial matches and embeddings that a walk query of these cases may have
WALK_ROWS = 1 << 17
CYCLE_ROWS = 1 << 22
HOST_ROWS = 1 << 14


def listed():
    return [
        # the smallest call: one count on a graph of a few kilobytes, where launches and latency are everything
        dict(name="small_count", task="count", graph="er", vertices=300, edges=1500, labels=2, shape="path", k=4,
             queries=1),
        # the small plain configuration: queries of 2 to 4 vertices one after another, their tables read on the host
        dict(name="small_tables", task="host_table", graph="er", vertices=1000, edges=2000, labels=87, shape="mixed",
             k=4, queries=8),
        # the plain-at-scale configuration: walk-induced queries of 8 vertices, their tables kept on the device
        dict(name="walk8_tables", task="table", graph="rmat", vertices=1 << 20, edges=16_000_000, labels=32,
             shape="walk", k=8, queries=4),
        # long walk queries on a graph of odd size: many levels, each with little work
        dict(name="walk13_tables", task="table", graph="rmat", vertices=300_007, edges=4_700_001, labels=48,
             shape="walk", k=13, queries=3),
        # count-only 5-vertex path on the batched configuration's graph: most of its embeddings come from these
        dict(name="path5_count", task="count", graph="rmat", vertices=1 << 22, edges=64_000_000, labels=64,
             shape="path", k=5, queries=1),
        # 4-cycle with its table: the closing intersection of two lists over many two-paths
        dict(name="cycle4_table", task="table", graph="rmat", vertices=1 << 20, edges=16_000_000, labels=64,
             shape="cycle", k=4, queries=1),
        # the skew configuration: cliques on a power-law graph with two labels, where hubs hold most of the work
        dict(name="skew_clique4", task="count", graph="chung_lu", vertices=1 << 18, edges=4_000_000, labels=2,
             shape="clique", k=4, queries=1),
        # the batched configuration in shared launches: paths, stars, cycles and walks of 4 to 16 vertices
        dict(name="batch_mixed", task="batch", graph="rmat", vertices=1 << 20, edges=16_000_000, labels=64,
             shape="mixed", k=16, queries=48),
        # the serving configuration: queued count requests of interactive walk queries, several slots
        dict(name="serve_walks", task="serve", graph="rmat", vertices=1 << 18, edges=4_000_000, labels=64,
             shape="walk", k=7, queries=32),
        # what the command line does: a `.g` text is parsed and built, then one query is counted
        dict(name="load_text", task="load_text", graph="rmat", vertices=50_021, edges=400_000, labels=16,
             shape="cycle", k=3, queries=1),
        # a resident graph built from edge arrays, then one query counted on it
        dict(name="build_edges", task="build", graph="rmat", vertices=1 << 20, edges=8_000_000, labels=64,
             shape="cycle", k=3, queries=1),
    ]


def _log_int(rng, lo, hi):
    """An integer spread evenly over the logarithm of [lo, hi]; mostly odd sizes."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["small", "small_tables", "walks", "path", "cycle", "star", "skew", "batch", "serve", "load",
                       "build"])
    if kind == "small":
        v = _log_int(rng, 100, 4000)
        return dict(task="count", graph="er", vertices=v, edges=int(v * rng.uniform(2, 5)),
                    labels=rng.randint(1, 4), shape=rng.choice(["path", "star", "cycle"]), k=rng.randint(3, 5),
                    queries=1)
    if kind == "small_tables":
        v = _log_int(rng, 200, 8000)
        return dict(task="host_table", graph="er", vertices=v, edges=int(v * rng.uniform(1.5, 4)),
                    labels=rng.randint(20, 120), shape="mixed", k=rng.randint(3, 5), queries=rng.randint(2, 8))
    if kind == "walks":
        v = _log_int(rng, 1 << 14, 1 << 20)
        return dict(task="table", graph="rmat", vertices=v, edges=int(v * rng.uniform(10, 16)),
                    labels=rng.randint(32, 64), shape="walk", k=rng.randint(6, 14), queries=rng.randint(1, 4))
    if kind == "path":
        v = _log_int(rng, 1 << 12, 1 << 20)
        return dict(task="count", graph="rmat", vertices=v, edges=int(v * rng.uniform(6, 15)),
                    labels=rng.randint(64, 120), shape="path", k=rng.randint(3, 5), queries=1)
    if kind == "cycle":
        v = _log_int(rng, 1 << 12, 1 << 20)
        return dict(task="table", graph="rmat", vertices=v, edges=int(v * rng.uniform(6, 15)),
                    labels=rng.randint(64, 120), shape="cycle", k=rng.randint(3, 4), queries=1)
    if kind == "star":
        v = _log_int(rng, 1 << 12, 1 << 20)
        return dict(task="count", graph="rmat", vertices=v, edges=int(v * rng.uniform(6, 15)),
                    labels=rng.randint(64, 120), shape="star", k=4, queries=1)
    if kind == "skew":
        v = _log_int(rng, 1 << 12, 1 << 16)
        return dict(task="count", graph="chung_lu", vertices=v, edges=int(v * rng.uniform(3, 7)), labels=2,
                    shape=rng.choice(["clique", "cycle"]), k=rng.choice([3, 4]), queries=1)
    if kind == "batch":
        v = _log_int(rng, 1 << 14, 1 << 19)
        return dict(task="batch", graph="rmat", vertices=v, edges=int(v * rng.uniform(8, 15)),
                    labels=rng.randint(64, 96), shape="mixed", k=rng.randint(6, 16), queries=rng.randint(8, 48))
    if kind == "serve":
        v = _log_int(rng, 1 << 14, 1 << 18)
        return dict(task="serve", graph="rmat", vertices=v, edges=int(v * rng.uniform(8, 15)),
                    labels=rng.randint(48, 96), shape="walk", k=rng.randint(5, 10), queries=rng.randint(8, 32))
    if kind == "load":
        v = _log_int(rng, 1000, 50_000)
        return dict(task="load_text", graph="rmat", vertices=v, edges=int(v * rng.uniform(3, 7)),
                    labels=rng.randint(4, 64), shape="cycle", k=3, queries=1)
    v = _log_int(rng, 1 << 12, 1 << 19)
    return dict(task="build", graph="rmat", vertices=v, edges=int(v * rng.uniform(4, 15)), labels=rng.randint(16, 96),
                shape="cycle", k=3, queries=1)


# ------------------------------------------------------------------ graphs

def _pairs(case, n, gen):
    """n random endpoint pairs of the case's graph model (before duplicates and self loops are dropped)."""
    v = case["vertices"]
    if case["graph"] == "er":
        return (torch.randint(0, v, (n,), generator=gen, device="cuda"),
                torch.randint(0, v, (n,), generator=gen, device="cuda"))
    if case["graph"] == "chung_lu":
        w = torch.arange(1, v + 1, dtype=torch.float64, device="cuda") ** (-1.0 / 1.1)
        w = torch.clamp(w * (2.0 * case["edges"] / w.sum()), max=float(1 << 20))
        cdf = torch.cumsum(w / w.sum(), 0)
        pick = [torch.searchsorted(cdf, torch.rand(n, generator=gen, device="cuda", dtype=torch.float64))
                for _ in range(2)]
        return pick[0].clamp(max=v - 1), pick[1].clamp(max=v - 1)
    s = torch.zeros(n, dtype=torch.int64, device="cuda")
    t = torch.zeros(n, dtype=torch.int64, device="cuda")
    for _ in range((v - 1).bit_length()):
        r = torch.rand(n, generator=gen, device="cuda")
        s = s * 2 + (r >= 0.76)
        t = t * 2 + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    keep = (s < v) & (t < v)
    return s[keep], t[keep]


def _edges(case, gen):
    """Distinct undirected edges u < v with labels 1..labels, vertex ids scrambled; sorted by (u, v)."""
    v, m = case["vertices"], case["edges"]
    keys = torch.zeros(0, dtype=torch.int64, device="cuda")
    for _ in range(40):
        if len(keys) >= m:
            break
        a, b = _pairs(case, int((m - len(keys)) * 1.3) + 1024, gen)
        lo, hi = torch.minimum(a, b), torch.maximum(a, b)
        keys = torch.unique(torch.cat([keys, (lo * v + hi)[lo != hi]]))
    if len(keys) > m:
        keys = keys[torch.randperm(len(keys), generator=gen, device="cuda")[:m]]
    perm = torch.randperm(v, generator=gen, device="cuda")
    a, b = perm[keys // v], perm[keys % v]
    keys = torch.sort(torch.minimum(a, b) * v + torch.maximum(a, b)).values
    lab = torch.randint(1, case["labels"] + 1, (len(keys),), generator=gen, device="cuda")
    return keys // v, keys % v, lab


def _e_lines(u, w, lab):
    """Host arrays of the directed e-lines (both directions), as a user passes them."""
    def host(a, b):
        return torch.cat([a, b]).to(torch.int32).cpu().numpy().view(np.uint32)
    return host(u, w), host(w, u), host(lab, lab)


class _Adjacency:
    """Device adjacency of a generated graph, to draw queries from it."""

    def __init__(self, case, u, w, lab):
        self.v = case["vertices"]
        key = torch.cat([u * self.v + w, w * self.v + u])
        self.key, order = torch.sort(key)
        self.lab = torch.cat([lab, lab])[order]
        ends = torch.arange(self.v + 1, device="cuda") * self.v
        self.ptr = torch.searchsorted(self.key, ends)

    def step(self, at, gen):
        """A uniform random neighbour of each vertex."""
        n = self.ptr[at + 1] - self.ptr[at]
        i = (torch.rand(at.shape, generator=gen, device="cuda", dtype=torch.float64) * n).long()
        return self.key[torch.clamp(self.ptr[at] + torch.minimum(i, n - 1), min=0, max=len(self.key) - 1)] % self.v

    def labels(self, a, b):
        """Label of the edge {a, b}, 0 where there is none."""
        k = a * self.v + b
        i = torch.searchsorted(self.key, k).clamp(max=len(self.key) - 1)
        return torch.where(self.key[i] == k, self.lab[i], torch.zeros_like(k))

    def walks(self, k, count, gen):
        """Vertex sets of `count` random walks that found k distinct vertices (fewer walks may come back), and the
        labels of the edges they induce."""
        deg = self.ptr[1:] - self.ptr[:-1]
        start = torch.nonzero(deg > 0).flatten()
        cur = start[torch.randint(0, len(start), (count,), generator=gen, device="cuda")]
        seen = torch.full((count, k), -1, dtype=torch.int64, device="cuda")
        seen[:, 0] = cur
        n = torch.ones(count, dtype=torch.int64, device="cuda")
        rows = torch.arange(count, device="cuda")
        for _ in range(6 * k):
            cur = self.step(cur, gen)
            new = (n < k) & ~(seen == cur[:, None]).any(1)
            seen[rows[new], n[new]] = cur[new]
            n = n + new
        seen = seen[n == k]
        return seen.cpu().numpy(), self.labels(seen[:, :, None], seen[:, None, :]).cpu().numpy()


# ------------------------------------------------------------------ queries

def _shape_query(shape, k, rng, labels):
    if shape == "clique":
        lab = rng.integers(1, labels + 1, size=k * (k - 1) // 2)
        return S.query_clique(k, [int(x) for x in lab])
    lab = [int(x) for x in rng.integers(1, labels + 1, size=k)]
    return {"path": S.query_path, "star": S.query_star, "cycle": S.query_cycle}[shape](k, lab)


def _walk_queries(case, adj, ctx, graph, k, count, rng, gen):
    """Induced subgraphs of random walks, of edge density 0.3 to 0.8, kept when they are interactive: few enough
    partial matches and embeddings to be enumerated."""
    out = []
    lo = 0.25 if k >= 10 else 0.3
    for _ in range(6):
        seen, lab = adj.walks(k, 2048, gen)
        dens = np.count_nonzero(lab, axis=(1, 2)) / (k * (k - 1))
        for i in np.nonzero((dens >= lo) & (dens <= 0.8))[0][:64]:
            q = S.Query(k, [(a, b, int(lab[i, a, b])) for a in range(k) for b in range(a + 1, k) if lab[i, a, b]])
            text = q.to_g_text()
            r = fm.match(ctx, graph, fm.Query.from_text(text), mode=fm.MODE_COUNT, work_limit=WALK_PARTIALS, allow_limit=True)
            rows = sum(r.level[d].produced for d in range(1, k))
            if r.status == fm.FM_OK and 0 < r.count <= WALK_ROWS and rows <= WALK_PARTIALS:
                out.append(text)
                if len(out) == count:
                    return out
    # a graph too small for more of them: triangles
    return out + [_shape_query("cycle", 3, rng, case["labels"]).to_g_text() for _ in range(count - len(out))]


def _small_walks(case, adj, count, rng, gen):
    """Random walk paths and induced subgraphs of 2 to k vertices, at least one embedding each."""
    out = []
    while len(out) < count:
        k = 2 + len(out) % (case["k"] - 1)
        seen, lab = adj.walks(k, 64, gen)
        if not len(seen):
            continue
        out.append(S.Query(k, [(a, b, int(lab[0, a, b])) for a in range(k) for b in range(a + 1, k)
                               if lab[0, a, b]]).to_g_text())
    return out


def _mixed(case, adj, ctx, graph, rng, gen):
    """The batched configuration's mix: a quarter paths, stars and cycles of 4 vertices, the rest walks of 5 to k."""
    n, out = case["queries"], []
    for i in range(n // 4):
        out.append(_shape_query(["path", "star", "cycle"][i % 3], 4, rng, case["labels"]).to_g_text())
    sizes = [5 + (i % max(1, case["k"] - 4)) for i in range(n - len(out))]
    for k in sorted(set(sizes)):
        out += _walk_queries(case, adj, ctx, graph, k, sizes.count(k), rng, gen)
    return out


# ------------------------------------------------------------------ prepare, run

def _context(case):
    if case["graph"] == "er":
        return fm.Context(prealloc_bytes=512 * MB, soln_prealloc_bytes=256 * MB, output_prealloc_bytes=64 * MB,
                          bank_rows=256)
    soln = 16 * GB if case["task"] in ("batch", "serve") else 8 * GB
    return fm.Context(prealloc_bytes=soln + 5 * GB, soln_prealloc_bytes=soln, output_prealloc_bytes=4 * GB,
                      bank_rows=1024)


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    rng = np.random.default_rng(seed)
    u, w, lab = _edges(case, gen)
    lines = _e_lines(u, w, lab)
    st = {"task": case["task"], "case": case, "ctx": _context(case)}
    ctx, task = st["ctx"], case["task"]
    if task in ("load_text", "build"):
        st["texts"] = [_shape_query(case["shape"], case["k"], rng, case["labels"]).to_g_text()]
        if task == "load_text":
            vlab = np.ones(case["vertices"], dtype=np.uint32)
            st["text"] = S.g_text(case["vertices"], vlab, *lines, 1, case["labels"])
        else:
            st["lines"] = lines
        return st
    graph = st["graph"] = fm.Graph.from_edges(ctx, case["vertices"], case["labels"] + 1, *lines)
    if case["shape"] in ("walk", "mixed"):
        adj = _Adjacency(case, u, w, lab)
        if case["graph"] == "er":
            texts = _small_walks(case, adj, case["queries"], rng, gen)
        elif case["shape"] == "mixed":
            texts = _mixed(case, adj, ctx, graph, rng, gen)
        else:
            texts = _walk_queries(case, adj, ctx, graph, case["k"], case["queries"], rng, gen)
    else:
        texts = [_shape_query(case["shape"], case["k"], rng, case["labels"]).to_g_text()
                 for _ in range(case["queries"])]
    queries = st["queries"] = [fm.Query.from_text(t) for t in texts]
    if task == "host_table":
        st["rows"] = [fm.PinnedRows(HOST_ROWS, q.q) for q in queries]
        st["tables"] = [np.zeros((HOST_ROWS, q.q), dtype=np.int32) for q in queries]
    elif task == "table":
        st["stream"] = torch.cuda.Stream()
        cap = WALK_ROWS if case["shape"] == "walk" else CYCLE_ROWS
        st["tables"] = [torch.zeros(cap, q.q, dtype=torch.int32, device="cuda") for q in queries]
        st["mix"] = torch.tensor([pow(0x5851F42D4C957F2D, i + 1, 1 << 63) for i in range(16)], device="cuda")
    elif task == "batch":
        st["batch"] = fm.Batch(ctx, graph, queries, mode=fm.MODE_COUNT)
    elif task == "serve":
        st["server"] = fm.Server(ctx, graph, slots=4, max_batch=8)
    return st


class _DeviceRows:
    def __init__(self, ptr, n, q):
        self.__cuda_array_interface__ = {"shape": (n, q), "typestr": "<i4", "data": (ptr, False), "version": 3}


def _row_set(r, mix, out):
    """The rows of a device table, put into `out` in an order that depends on their values alone."""
    rows = torch.as_tensor(_DeviceRows(r.rows_device, r.rows, r.q), device="cuda")
    torch.index_select(rows, 0, torch.argsort((rows * mix).sum(1)), out=out[:r.rows])


def run(state):
    task, ctx = state["task"], state["ctx"]
    if task == "count":
        return [fm.match(ctx, state["graph"], q, mode=fm.MODE_COUNT).count for q in state["queries"]]
    if task == "host_table":
        out = []
        for q, buf, table in zip(state["queries"], state["rows"], state["tables"]):
            r = fm.match(ctx, state["graph"], q, host_rows=buf)
            rows = buf.view(r.rows_copied)
            table[:r.rows_copied] = rows[np.lexsort(rows.T[::-1])]
            out += [r.count, table]
        return out
    if task == "table":
        out = []
        with torch.cuda.stream(state["stream"]):
            for q, table in zip(state["queries"], state["tables"]):
                r = fm.match(ctx, state["graph"], q, stream=state["stream"].cuda_stream)
                if r.rows:
                    _row_set(r, state["mix"][:r.q], table)
                out += [r.count, table]
        return out
    if task == "batch":
        return np.array(state["batch"].run()[0], dtype=np.int64)
    if task == "serve":
        server = state["server"]
        tickets = [server.submit(q) for q in state["queries"]]
        counts = [server.poll(t).count for t in tickets]
        for t in tickets:
            server.release(t)
        return np.array(counts, dtype=np.int64)
    case = state["case"]
    if task == "load_text":
        graph = fm.Graph.from_text(ctx, state["text"])
    else:
        graph = fm.Graph.from_edges(ctx, case["vertices"], case["labels"] + 1, *state["lines"])
    info = graph.info()
    count = fm.match(ctx, graph, fm.Query.from_text(state["texts"][0]), mode=fm.MODE_COUNT).count
    graph.close()
    return [count, info.vertices, info.edges, info.segments, info.long_segments, info.max_list, info.has_duplicates]


def work(case):
    """Each e-line of a query's labels is read once (4 bytes) with its vertex's list head (8 bytes a vertex that has
    one), and a result written per query; building a graph reads every e-line (12 bytes, or its text) and writes it.
    One comparison per e-line that is read: counts and tables that need more are not known from the sizes."""
    lines = 2 * case["edges"]
    if case["task"] in ("load_text", "build"):
        read = lines * (18 if case["task"] == "load_text" else 12)
        return {"bytes": read + 4 * lines, "flops": lines}
    per_label = lines / case["labels"]
    edges = {"path": case["k"] - 1, "star": case["k"] - 1, "cycle": case["k"], "clique": case["k"] * (case["k"] - 1) / 2,
             "walk": case["k"] * (case["k"] - 1) / 5, "mixed": case["k"]}[case["shape"]]
    used = min(edges, case["labels"])
    heads = 8 * min(case["vertices"], per_label)
    per_query = used * (4 * per_label + heads) + 8
    return {"bytes": case["queries"] * per_query, "flops": case["queries"] * used * per_label}
