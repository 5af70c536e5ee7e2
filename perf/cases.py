"""The work that users of this library have it do, as cases that can be timed.

A case names a call (``call``), the graph it runs on (``graph`` and its sizes)
and the call's options.  Graphs are the shapes of the library's benchmark and
test configurations -- R-MAT, road-like grids, web-like directed graphs,
Chung-Lu power-law graphs and the star -- drawn on the GPU from the seed.

call
  bfs      one traversal, depths in host memory: GpuBfs.run
  many     up to 64 sources in one call: GpuBfs.run_many.  "host": every
           source's depths in a host array of its own; otherwise the result
           stays on the GPU (the last source's depths and every level count)
  pagerank GpuPageRank.run for a fixed number of iterations, or to a tolerance,
           then the ranks in host memory
  build    from_edges_gpu: an edge list to a sorted, duplicate-free CSR
"""
import math

import numpy as np
import torch

import graph_analytics_applesilicon_b200 as gb

TOL_ITERS = 200  # cap of the runs to a tolerance


def listed():
    return [
        # the smallest graph that users start with (the reference's own star):
        # latency of one call, two levels
        dict(name="bfs_star100k_hybrid", call="bfs", graph="star", n=100_001, variant="hybrid", selector="rule", hub_first=False),
        # the host-driven direction-optimizing form, one synchronisation per level
        dict(name="bfs_rmat16_do", call="bfs", graph="rmat", n=1 << 16, edges=16 << 16, variant="gpu_do", selector="rule",
             hub_first=False),
        # the benchmark graph (soc-LiveJournal1's shape), one source, default options
        dict(name="bfs_rmat22_hybrid", call="bfs", graph="rmat", n=1 << 22, edges=17 << 21, variant="hybrid", selector="rule",
             hub_first=False),
        # a road network (roadNet-CA's shape): 1,800 small levels, the shipped selector
        dict(name="bfs_road1400_learned", call="bfs", graph="road", n=1400 * 1400, cols=1400, variant="hybrid",
             selector="learned", hub_first=False),
        # the headline: 64 sources of the benchmark graph in one call, hub-first lists
        dict(name="many_rmat22_batch64", call="many", graph="rmat", n=1 << 22, edges=17 << 21, variant="batch", sources=64,
             selector="rule", hub_first=True, host=False),
        # 64 sources of the road network in one call
        dict(name="many_road1400_batch64", call="many", graph="road", n=1400 * 1400, cols=1400, variant="batch", sources=64,
             selector="rule", hub_first=False, host=False),
        # a mid-size power-law graph, every source's depths returned to the host
        dict(name="many_chunglu300k_host", call="many", graph="chung_lu", n=300_000, mean=30.0, variant="batch", sources=64,
             selector="rule", hub_first=True, host=True),
        # 8 sources side by side through the single-source kernel, odd sizes
        dict(name="many_rmat18_inflight", call="many", graph="rmat", n=(1 << 18) - 77, edges=(16 << 18) + 13,
             variant="gpu_do_persistent", sources=24, selector="rule", hub_first=False, host=True, in_flight=8),
        # web-Google's shape to the usual tolerance
        dict(name="pr_web875k_tol", call="pagerank", graph="web", n=875_000, mean=5.8, variant="gpu_pull_adaptive", iters=TOL_ITERS,
             tol=1e-6),
        # com-Orkut's shape, 20 iterations: the largest in-CSR
        dict(name="pr_chunglu3m_20", call="pagerank", graph="chung_lu", n=3_070_000, mean=76.0, variant="gpu_pull_adaptive",
             iters=20, tol=0.0),
        # the warp-per-vertex pull, the reference's fastest form on social graphs
        dict(name="pr_rmat18_vector_20", call="pagerank", graph="rmat_directed", n=1 << 18, edges=16 << 18,
             variant="gpu_pull_vector", iters=20, tol=0.0),
        # building a graph from a drawn edge list (host arrays in and out)
        dict(name="build_rmat20", call="build", graph="rmat", n=1 << 20, edges=8 << 20, directed=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["bfs", "bfs", "many", "many", "pagerank", "pagerank", "build"])
    if call == "build":
        n = _log(rng, 20_000, 1_000_000)
        return dict(call=call, graph="rmat", n=n, edges=n * rng.randint(3, 8) + rng.randint(0, 99), directed=rng.random() < 0.5)
    if call == "pagerank":
        graph = rng.choice(["web", "rmat_directed", "chung_lu"])
        n = _log(rng, 10_000, 1_500_000)
        tol = rng.random() < 0.4
        c = dict(call=call, graph=graph, n=n, variant=rng.choice(["gpu_pull_adaptive", "gpu_pull_adaptive", "gpu_pull_vector"]),
                 iters=TOL_ITERS if tol else 20, tol=1e-6 if tol else 0.0)
        if graph == "rmat_directed":
            c["edges"] = n * rng.randint(4, 16) + rng.randint(0, 99)
        else:
            c["mean"] = round(rng.uniform(4.0, 8.0) if graph == "web" else rng.uniform(10.0, 60.0), 2)
        return c
    graph = rng.choice(["rmat", "chung_lu", "road", "star"] if call == "bfs" else ["rmat", "chung_lu", "road"])
    c = dict(call=call, graph=graph)
    if graph == "star":
        c["n"] = _log(rng, 10_000, 1_000_000)
    elif graph == "road":
        rows = _log(rng, 120, 1300)
        c["cols"] = min(1400, max(100, int(rows * rng.uniform(0.8, 1.25))))
        c["n"] = rows * c["cols"]
    else:
        c["n"] = _log(rng, 20_000, 3_000_000)
        if graph == "rmat":
            c["edges"] = c["n"] * rng.randint(6, 10) + rng.randint(0, 99)
        else:
            c["mean"] = round(rng.uniform(8.0, 40.0), 2)
    if call == "bfs":
        c["variant"] = rng.choice(["hybrid", "hybrid", "hybrid", "gpu_do"])
        # the shipped selector where it is used in earnest: on road networks
        c["selector"] = "learned" if graph == "road" and c["variant"] == "hybrid" and rng.random() < 0.7 else "rule"
        c["hub_first"] = graph != "road" and c["variant"] == "hybrid" and rng.random() < 0.3
        return c
    c["variant"] = rng.choice(["batch", "batch", "gpu_do_persistent"])
    c["sources"] = rng.randint(5, 64) if c["variant"] == "batch" else rng.randint(4, 24)
    c["selector"] = "learned" if graph == "road" and c["variant"] != "batch" else "rule"
    c["hub_first"] = graph != "road" and rng.random() < 0.5
    c["host"] = c["n"] * c["sources"] < 20_000_000 and rng.random() < 0.5
    if c["variant"] != "batch":
        c["in_flight"] = rng.choice([1, 2, 4, 8])
    return c


# ------------------------------------------------------------------- graphs

def _rng(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1_000_003 + salt) & 0x7FFFFFFFFFFFFFFF)
    return g


def _rmat(n, edges, g):
    """Quadrant draws (0.57, 0.19, 0.19, 0.05), ids permuted; for n below the
    next power of two the ids are taken modulo n."""
    scale = max(1, (n - 1).bit_length())
    u = torch.zeros(edges, dtype=torch.int64, device="cuda")
    v = torch.zeros(edges, dtype=torch.int64, device="cuda")
    for _ in range(scale):
        r = torch.rand(edges, generator=g, device="cuda")
        u = u * 2 + (r >= 0.76)
        v = v * 2 + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    perm = torch.randperm(n, generator=g, device="cuda")
    return perm[u % n], perm[v % n]


def _road(n, cols, g):
    """4-neighbour grid, 4% of the edges dropped, 0.5% n diagonal links."""
    v = torch.arange(n, device="cuda")
    right = v[(v % cols) != cols - 1]
    down = v[v < n - cols]
    u = torch.cat([right, down])
    w = torch.cat([right + 1, down + cols])
    keep = torch.rand(u.numel(), generator=g, device="cuda") >= 0.04
    k = max(1, int(round(0.005 * n)))
    d = torch.randint(0, n, (k,), generator=g, device="cuda")
    d = d[((d % cols) != cols - 1) & (d < n - cols)]
    return torch.cat([u[keep], d]), torch.cat([w[keep], d + cols + 1])


def _web(n, mean, g):
    """Geometric out-degrees, Zipf-popular targets (s = 2.1), ids permuted."""
    lq = math.log1p(-1.0 / (1.0 + mean))
    od = torch.floor(torch.log1p(-torch.rand(n, generator=g, device="cuda", dtype=torch.float64)) / lq).clamp(max=1e6).long()
    u = torch.repeat_interleave(torch.arange(n, device="cuda"), od)
    e1 = 1.0 - 1.0 / 1.1
    x = torch.rand(u.numel(), generator=g, device="cuda", dtype=torch.float64)
    r = ((1.0 + x * ((n + 1.0) ** e1 - 1.0)) ** (1.0 / e1)).floor().long().clamp(1, n) - 1
    return u, torch.randperm(n, generator=g, device="cuda")[r]


def _chung_lu(n, mean, g):
    """Weights ~ (i + i0)^(-1/1.2), largest weight sqrt(sum), ids permuted."""
    a = 1.0 / 1.2
    total = mean * n
    lo, hi = 1e-3, float(n)
    for _ in range(100):
        mid = math.sqrt(lo * hi)
        s = ((n + mid) ** (1 - a) - mid ** (1 - a)) / (1 - a) + 0.5 * (mid ** -a - (n + mid) ** -a)
        lo, hi = (mid, hi) if mid ** -a * total / s > math.sqrt(total) else (lo, mid)
    w = (torch.arange(n, device="cuda", dtype=torch.float64) + hi) ** -a
    cdf = torch.cumsum((w * (2.0 ** 40 / float(w[0]))).long() + 1, 0)  # whole numbers: the same sums in every run
    top = int(cdf[-1])
    perm = torch.randperm(n, generator=g, device="cuda")

    def ends(k):
        return perm[torch.searchsorted(cdf, torch.randint(0, top, (k,), generator=g, device="cuda"), right=True)]
    k = int(round(total / 2))
    return ends(k), ends(k)


def _edges(case, seed):
    g = _rng(seed, 17)
    n, kind = case["n"], case["graph"]
    if kind == "star":
        hub = int(torch.randint(0, n, (1,), generator=g, device="cuda"))
        v = torch.arange(n, device="cuda")
        v = v[v != hub]
        return torch.full_like(v, hub), v
    if kind == "road":
        return _road(n, case["cols"], g)
    if kind == "web":
        return _web(n, case["mean"], g)
    if kind == "chung_lu":
        return _chung_lu(n, case["mean"], g)
    return _rmat(n, case["edges"], g)


def _csr(n, u, v, both):
    """Sorted, duplicate- and loop-free CSR on the GPU: (row_ptr, col_idx)."""
    if both:
        u, v = torch.cat([u, v]), torch.cat([v, u])
    keys = torch.unique((u * n + v)[u != v])
    row = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    row[1:] = torch.cumsum(torch.bincount(keys // n, minlength=n), 0)
    return row, (keys % n).to(torch.int32)


def _host(row, col, n, directed):
    flags = gb.FLAG_SORTED | gb.FLAG_DEDUP | (gb.FLAG_DIRECTED if directed else 0)
    return gb.Graph(n, int(col.numel()), flags, row.to(torch.int32).cpu().numpy().view(np.uint32),
                    col.cpu().numpy().view(np.uint32))


def _edge_list(case, seed):
    """case["edges"] distinct edges in random order and direction, one in 20
    of them listed twice."""
    n, want = case["n"], case["edges"]
    u, v = _edges(dict(case, edges=2 * want), seed)
    if not case["directed"]:
        u, v = torch.minimum(u, v), torch.maximum(u, v)
    keys = torch.unique((u * n + v)[u != v])
    g = _rng(seed, 29)
    keys = keys[torch.randperm(keys.numel(), generator=g, device="cuda")[:want]]
    assert keys.numel() == want
    keys = torch.cat([keys, keys[: want // 20]])
    keys = keys[torch.randperm(keys.numel(), generator=g, device="cuda")]
    u, v = keys // n, keys % n
    if not case["directed"]:
        flip = torch.rand(keys.numel(), generator=g, device="cuda") < 0.5
        u, v = torch.where(flip, v, u), torch.where(flip, u, v)
    return u, v


def _directed(case):
    return case["graph"] in ("web", "rmat_directed")


def _pagerank_csrs(case, seed):
    """In-CSR and out-degrees of the case's graph, on the GPU."""
    n = case["n"]
    u, v = _edges(case, seed)
    row, col = _csr(n, v, u, not _directed(case))
    deg = torch.bincount(col, minlength=n) if _directed(case) else row[1:] - row[:-1]
    return row, col, deg


# --------------------------------------------------------------------- calls

class _Device:
    """A handle's device array for torch, which keeps this object and so the handle."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<i4", "data": (int(ptr), False), "version": 3, "strides": None}


def prepare(case, seed):
    n, call = case["n"], case["call"]
    if call == "build":
        u, v = _edge_list(case, seed)
        return dict(case=case, u=u.to(torch.int32).cpu().numpy().view(np.uint32), v=v.to(torch.int32).cpu().numpy().view(np.uint32))
    if call == "pagerank":
        row, col, deg = _pagerank_csrs(case, seed)
        gin = _host(row, col, n, _directed(case))
        pr = gb.GpuPageRank(n, None, gin, deg.to(torch.int32).cpu().numpy().view(np.uint32))
        if case["variant"] == "gpu_pull_adaptive":
            pr.prepareAdaptive()
        return dict(case=case, pr=pr, opts=gb.PrOptions(iters=case["iters"], tol=case["tol"]))
    u, v = _edges(case, seed)
    row, col = _csr(n, u, v, True)
    g = _host(row, col, n, False)
    del u, v, row, col
    k = case.get("sources", 1)
    src = gb.pick_sources_gpu(g, k, 1 + int(seed))
    src = np.resize(src, k).astype(np.uint32)
    bfs = gb.GpuBfs(g)
    if case["hub_first"]:
        bfs.hub_first()
    if case["selector"] == "learned":
        bfs.set_selector(gb.default_selector_params("single"), 0)
    opts = gb.BfsOptions(selector=case["selector"], in_flight=case.get("in_flight", 1))
    out = np.zeros((k, n) if call == "many" else n, np.uint32) if case.get("host", True) else None
    return dict(case=case, bfs=bfs, src=src, opts=opts, out=out)


def run(state):
    c = state["case"]
    if c["call"] == "bfs":
        return state["bfs"].run(c["variant"], int(state["src"][0]), out=state["out"], opts=state["opts"]).view(np.int32)
    if c["call"] == "many":
        b = state["bfs"]
        if state["out"] is not None:
            out, _, levels = b.run_many(c["variant"], state["src"], out=state["out"], opts=state["opts"])
            return {"depths": out.view(np.int32), "levels": levels.astype(np.int64)}
        _, _, levels = b.run_many(c["variant"], state["src"], opts=state["opts"], device=True)
        last = torch.as_tensor(_Device(b, gb.lib().gb_bfs_device_dist(b._h), c["n"]), device="cuda")
        return {"depths": last, "levels": levels.astype(np.int64)}
    if c["call"] == "pagerank":
        state["pr"].run(c["variant"], state["opts"])
        return state["pr"].ranks()
    g = gb.from_edges_gpu(c["n"], state["u"], state["v"], c["directed"])
    return {"row_ptr": g.row_ptr.view(np.int32), "col_idx": g.col_idx.view(np.int32)}


def _entries(case):
    """About how many adjacency entries the case's graph has."""
    n, kind = case["n"], case["graph"]
    both = 1 if case.get("directed") or _directed(case) else 2
    if kind == "star":
        return 2 * (n - 1)
    if kind == "road":
        return 3.85 * n
    if kind in ("web", "chung_lu"):
        return case["mean"] * n
    return both * case["edges"]


def work(case):
    n, m, call = case["n"], _entries(case), case["call"]
    if call == "build":  # the edge list in, the CSR out
        return {"bytes": 8 * case["edges"] + 4 * m + 4 * n, "flops": 0}
    if call == "pagerank":  # per sweep: the in-CSR, the ranks in and out
        sweeps = 20
        return {"bytes": sweeps * (4 * n + 4 * m + 8 * n), "flops": sweeps * (2 * m + 4 * n)}
    # the CSR in, every source's depths out
    return {"bytes": 4 * n + 4 * m + 4 * n * case.get("sources", 1), "flops": 0}


def exact(case, seed):
    """PageRank in 64 bits with the library's definition and stop rule."""
    if case["call"] != "pagerank":
        return None
    n = case["n"]
    row, col, deg = _pagerank_csrs(case, seed)
    a = torch.sparse_csr_tensor(row.to(torch.int32), col, torch.ones(col.numel(), dtype=torch.float64, device="cuda"), size=(n, n))
    od = deg.to(torch.float64)
    inv = torch.where(od > 0, 1.0 / od.clamp(min=1.0), torch.zeros_like(od))
    r = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    best, since = 1e300, 0
    for _ in range(case["iters"]):
        new = 0.15 / n + 0.85 * (a @ (r * inv) + r[od == 0].sum() / n)
        delta = float((new - r).abs().sum()) if case["tol"] > 0 else 0.0
        r = new
        if case["tol"] > 0:
            if delta < case["tol"]:
                break
            best, since = (delta, 0) if delta < best else (best, since + 1)
            if since >= 5:
                break
    return r.cpu().numpy()
