"""The work that users of this framework have it do, as measurable cases.

Every case goes through the package's public entry points (Graph, Server).  A
case is a dict of plain values:

  kind    what is called (see `run`): "query", "query_host", "batch", "bc",
          "bc_batch", "centrality", "serve" or "build"
  graph   "rmat" (power law, a=0.57 b=c=0.19, permuted ids), "rmat_ids" (the
          same with the generator's own ids), "uniform" (uniform random edges)
          or "mesh" (a 2-D street grid with a tenth of its streets closed, both
          directions of each: many levels, small frontiers)
  n, m    vertices and directed edges (mesh: m follows from n and the seed)
  w, s    tile width and stripe length of the layout
  k       sources (batch, bc_batch, centrality) or queries (serve)
  rule    direction rule of the single-source traversal: "reference" (the
          default) or "unvisited" (Beamer's, which the autotuner usually picks)
  layout  "tiles" (the caller's ids) or "degree" (the degree-ordered layout)

Graphs are seeded: another seed is another graph and other sources.
"""
import numpy as np
import torch

import bfs_simd_benchmarks_gb300 as B

POKEC = dict(n=1_632_803, m=30_622_564, w=1024, s=16)
TWITTER = dict(n=41_652_230, m=1_468_365_182, w=1024, s=16)
BFS_DST_DEVICE = 2  # the C ABI's constant: a query's levels go to device memory
SERVE_SCALES = (14, 16, 18, 19, 20)


def _case(name, kind, graph, n, m, w=1024, s=16, k=1, rule="reference", layout="tiles"):
    return dict(name=name, kind=kind, graph=graph, n=n, m=m, w=w, s=s, k=k, rule=rule, layout=layout)


def listed():
    return [
        # One query on a tiny graph, levels and parents to host arrays: what a call costs by itself.
        _case("query_host_s10", "query_host", "rmat_ids", 1 << 10, 1 << 14, 64, 4),
        # The reference's own CPU configuration (scale 16, edge factor 16): levels and parents to host arrays.
        _case("query_host_s16", "query_host", "rmat_ids", 1 << 16, 1 << 20),
        # A street grid of odd size: hundreds of levels of a few hundred vertices each.
        _case("query_mesh", "query", "mesh", 301 * 287, 0, 512, 8),
        # The Pokec shape, one source, levels left on the device, with the direction rule that tuning picks.
        _case("query_pokec", "query", "rmat", **POKEC, rule="unvisited"),
        # The Twitter shape, one source: the largest graph that is run.
        _case("query_twitter", "query", "rmat", **TWITTER),
        # 64 sources of the Pokec shape in one batch: one bit-sliced word per vertex.
        _case("batch_pokec_64", "batch", "rmat", **POKEC, k=64),
        # The full batch: 4096 sources at scale 22.
        _case("batch_s22_4096", "batch", "rmat_ids", 1 << 22, 1 << 26, k=4096),
        # Betweenness dependencies and path counts of one source.
        _case("bc_pokec", "bc", "rmat", **POKEC),
        # The same for 64 sources in one call, every (source, vertex) pair written.
        _case("bc_batch_pokec_64", "bc_batch", "rmat", **POKEC, k=64),
        # Centrality over an odd number of sources of a small graph, the sum copied to the host.
        _case("centrality_s16_201", "centrality", "rmat_ids", 1 << 16, 1 << 20, k=201),
        # A burst of queries over several resident graphs through the server, levels to device buffers.
        _case("serve_burst_256", "serve", "rmat_ids", 1 << 20, 1 << 24, k=256),
        # A graph that has just arrived: the layout built from an edge list in device memory, and a first query.
        _case("build_pokec", "build", "rmat", **POKEC),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["query_host", "query", "query", "batch", "batch", "bc", "bc_batch", "centrality", "serve", "build"])
    graph = rng.choice(["rmat", "rmat", "rmat_ids", "uniform"] + (["mesh"] if kind in ("query", "query_host") else []))
    w, s = rng.choice([64, 256, 512, 1024, 2048, 4096]), rng.choice([4, 8, 16, 32])
    rule, layout, k = "reference", "tiles", 1
    if kind in ("query", "query_host"):
        n = _log_int(rng, 1 << 10, 1 << 17 if graph == "mesh" else 1 << 20 if kind == "query_host" else 1 << 24)
        rule = rng.choice(["reference", "unvisited"])
        if n <= 1 << 16:
            layout = rng.choice(["tiles", "degree"])
    elif kind == "batch":
        n = _log_int(rng, 1 << 12, 1 << 22)
        k = _log_int(rng, 2, min(4096, (1 << 32) // n))
    elif kind == "bc":
        n = _log_int(rng, 1 << 12, 1 << 22)
    elif kind == "bc_batch":
        n = _log_int(rng, 1 << 12, 1 << 20)
        k = _log_int(rng, 16, 256)
    elif kind == "centrality":
        n = _log_int(rng, 1 << 12, 1 << 20)
        k = _log_int(rng, 16, 400)
    elif kind == "serve":
        n = _log_int(rng, 1 << 14, 1 << 20)
        k = _log_int(rng, 16, 1024)
    else:
        n = _log_int(rng, 1 << 14, 1 << 22)
    m = 0 if graph == "mesh" else min(int(n * (4 + 28 * rng.random())), n * 40, 1 << 28)
    while w > 64 and w * 8 > n:
        w //= 2
    c = _case("", kind, graph, n, m, w, s, k, rule, layout)
    del c["name"]
    return c


def _mesh(n, seed):
    """Rows x columns vertices (about n), every street kept with probability 0.9, both ways."""
    rows = int(n ** 0.5)
    cols = n // rows
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 7 + 3)
    ids = torch.arange(rows * cols, device="cuda", dtype=torch.int32).view(rows, cols)
    a = torch.cat([ids[:, :-1].reshape(-1), ids[:-1].reshape(-1)])
    b = torch.cat([ids[:, 1:].reshape(-1), ids[1:].reshape(-1)])
    keep = torch.rand(a.numel(), device="cuda", generator=g) < 0.9
    a, b = a[keep], b[keep]
    return torch.cat([a, b]), torch.cat([b, a])


def _edges(graph, n, m, seed):
    """The directed edge list as int32 device tensors."""
    if graph == "mesh":
        return _mesh(n, seed)
    p = dict(a=0.25, b=0.25, c=0.25) if graph == "uniform" else {}
    return B.gen_rmat_device(n, m, seed=seed * 16 + 1, permute=graph == "rmat", **p)


def _graph(case, src, dst):
    if case["layout"] == "degree":
        g = B.Graph.from_edges(case["n"], src.cpu().numpy(), dst.cpu().numpy(), case["w"], case["s"], degree_order=True)
    else:
        g = B.Graph.from_device_edges(case["n"], src.data_ptr(), dst.data_ptr(), src.numel(), case["w"], case["s"])
    if case["rule"] == "unvisited":
        g.set_options(switch_rule=1)
    return g


def _widest():
    """Builds and drops a graph whose layout needs the most shared memory of any here.

    Every build sets the traversal kernel's shared-memory limit to what its own
    graph needs, and a graph that needs more is then refused: a program that
    holds several graphs builds its widest layout last.
    """
    edge = torch.tensor([0, (1 << 15) - 1], dtype=torch.int32, device="cuda")
    B.Graph.from_device_edges(1 << 15, edge.data_ptr(), edge.data_ptr() + 4, 1, 1024, 16).close()


def _sources(src, n, k, seed):
    """Seeded vertices with an out-edge: a mesh's from its crossings, others uniformly."""
    has_out = torch.zeros(n, dtype=torch.bool, device="cuda")
    has_out[src.long()] = True
    cand = torch.nonzero(has_out).view(-1)
    at = np.random.default_rng(seed * 31 + 5).integers(0, cand.numel(), size=k)
    return cand[torch.from_numpy(at).cuda()].cpu().numpy().astype(np.uint32)


def _serve_graphs(case, seed):
    """(n, src, dst) of the resident graphs: the serving scales up to the case's size, same edge factor."""
    sizes = [1 << x for x in SERVE_SCALES if 1 << x < case["n"]] + [case["n"]]
    return [(n, *_edges(case["graph"], n, n * (case["m"] // case["n"]), seed * 8 + i)) for i, n in enumerate(sizes)]


def prepare(case, seed):
    kind, k = case["kind"], case["k"]
    st = {"kind": kind, "case": case}
    if kind == "serve":
        graphs = _serve_graphs(case, seed)
        srv = B.Server(budget_bytes=24 << 30, slot_bytes=256 << 20, max_batch=256)
        ids = [srv.add_graph(_graph(dict(case, n=n), s, d)) for n, s, d in graphs]
        _widest()
        pick = np.random.default_rng(seed * 13 + 1).permutation(np.arange(k) % len(graphs))
        pools = [_sources(s, n, k, seed + i) for i, (n, s, _) in enumerate(graphs)]
        st["server"] = srv
        st["queries"] = [(ids[gi], int(pools[gi][j])) for j, gi in enumerate(pick)]
        # one result buffer, a query's levels at a 256-byte boundary of it
        ends = np.cumsum([-(-graphs[gi][0] // 256) * 256 for gi in pick])
        st["levels"] = torch.zeros(int(ends[-1]), dtype=torch.uint8, device="cuda")
        st["at"] = [st["levels"].data_ptr() + int(e) for e in np.concatenate([[0], ends[:-1]])]
        return st
    src, dst = _edges(case["graph"], case["n"], case["m"], seed)
    n = case["n"]
    st["sources"] = _sources(src, n, k, seed)
    if kind == "build":
        st["src"], st["dst"] = src, dst
        st["levels"] = torch.empty(n, dtype=torch.int32, device="cuda")
        return st
    st["graph"] = _graph(case, src, dst)
    _widest()
    if kind == "query":
        st["levels"] = torch.empty(n, dtype=torch.int32, device="cuda")
    elif kind == "batch":
        st["levels"] = torch.empty((k, n), dtype=torch.uint8, device="cuda")
    elif kind in ("bc", "bc_batch"):
        shape = (n,) if kind == "bc" else (k, n)
        st["dependencies"] = torch.empty(shape, dtype=torch.float32, device="cuda")
        st["paths"] = torch.empty(shape, dtype=torch.int32, device="cuda")
    return st


def run(st):
    kind = st["kind"]
    if kind == "query_host":
        # parents come back too; any valid tree may, so only the levels are the same from run to run
        levels, _, stats = st["graph"].run(int(st["sources"][0]))
        return {"levels": levels, "reached": stats["reached"]}
    if kind == "query":
        st["graph"].run_device(int(st["sources"][0]), st["levels"].data_ptr())
        return {"levels": st["levels"]}
    if kind == "batch":
        st["graph"].run_batch_device(st["sources"], st["levels"].data_ptr())
        return {"levels": st["levels"]}
    if kind == "bc":
        st["graph"].bc_device(int(st["sources"][0]), st["dependencies"].data_ptr(), st["paths"].data_ptr())
        return {"dependencies": st["dependencies"], "paths": st["paths"]}
    if kind == "bc_batch":
        st["graph"].bc_batch_device(st["sources"], st["dependencies"].data_ptr(), st["paths"].data_ptr())
        return {"dependencies": st["dependencies"], "paths": st["paths"]}
    if kind == "centrality":
        centrality, _ = st["graph"].betweenness(st["sources"])
        return {"centrality": centrality}
    if kind == "serve":
        srv = st["server"]
        tickets = [srv.submit(g, s, at, BFS_DST_DEVICE) for (g, s), at in zip(st["queries"], st["at"])]
        for t in tickets:
            srv.wait(t)
        return {"levels": st["levels"]}
    case = st["case"]
    with _graph(case, st["src"], st["dst"]) as g:
        g.run_device(int(st["sources"][0]), st["levels"].data_ptr())
        degrees = g.degrees()
    return {"levels": st["levels"], "degrees": degrees.astype(np.int64)}


def work(case):
    n, k, kind = case["n"], case["k"], case["kind"]
    m = case["m"] or int(3.6 * n)
    graph = 4 * (n + 1) + 4 * m  # the CSR, read once
    if kind == "serve":
        sizes = [1 << x for x in SERVE_SCALES if 1 << x < n] + [n]
        return {"bytes": sum(4 * (x + 1) + 4 * x * (m // n) for x in sizes) + 2 * k * sum(sizes) // len(sizes), "flops": 0}
    out = {"query": 4 * n, "query_host": 8 * n, "batch": k * n, "bc": 8 * n, "bc_batch": 8 * n * k, "centrality": 4 * n,
           "build": 8 * n + 8 * m}[kind]
    if kind == "build":
        return {"bytes": out + 2 * graph, "flops": 0}
    flops = 4 * m * k if kind in ("bc", "bc_batch", "centrality") else 0  # an add each way per shortest-path edge
    return {"bytes": graph + out, "flops": flops}


def _exact_bc(n, src, dst, source, far=1 << 30):
    """Dependencies of one source in 64 bits: path counts modulo 2^32 (read as signed, as the inverses are), sums from the deepest level."""
    level = torch.full((n,), far, dtype=torch.int64, device="cuda")
    sigma = torch.zeros(n, dtype=torch.int64, device="cuda")
    level[source], sigma[source] = 0, 1
    steps, d = [], 0
    while True:
        e = torch.nonzero(level[src] == d).view(-1)
        e = e[level[dst[e]] > d]
        if not e.numel():
            break
        u, v = src[e], dst[e]
        level[v] = d + 1
        sigma.index_add_(0, v, sigma[u])
        sigma &= 0xFFFFFFFF
        steps.append((u, v))
        d += 1
    signed = torch.where(sigma >= 1 << 31, sigma - (1 << 32), sigma).double()
    inverse = torch.where(sigma != 0, 1.0 / signed, torch.zeros_like(signed))
    total = inverse.clone()
    for u, v in reversed(steps):
        total.index_add_(0, u, total[v])
    return torch.where(inverse != 0, (total - inverse) / inverse, torch.zeros_like(total))


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("bc", "bc_batch", "centrality"):
        return None  # levels and degrees are whole numbers
    if case["m"] * case["k"] > 1 << 31:
        return None
    n = case["n"]
    src, dst = _edges(case["graph"], n, case["m"], seed)
    sources = _sources(src, n, case["k"], seed)
    src, dst = src.long(), dst.long()
    rows = (_exact_bc(n, src, dst, int(s)) for s in sources)
    if kind == "bc":
        return {"dependencies": next(rows), "paths": None}
    if kind == "bc_batch":
        return {"dependencies": torch.stack(list(rows)), "paths": None}
    total = torch.zeros(n, dtype=torch.float64, device="cuda")
    for s, row in zip(sources, rows):
        row[int(s)] = 0
        total += row
    return {"centrality": total}
