"""The timed cases: what a program asks of this library, through its public
entry points, over the sizes it asks them at.

The listed cases follow the benchmark's configurations: plain BFS and
PageRank on R-MAT 16, iterated products on R-MAT and G(n, m), the batched
searches (BFS, min-plus, personalised PageRank), Lanczos on a symmetrised
graph's largest component and the PageRank adjoint.  draw() gives others of
the same paths: sizes from a few thousand nodes up, node counts that are no
multiple of anything, both orientations, each element type and option those
paths take.  Graphs are synthetic (seeded R-MAT with (a, b, c, d) = (.57,
.19, .19, .05), or uniform G(n, m)), without self-loops or duplicates, node
ids in random order; `degree` is the edges drawn per node, before duplicates
go.
"""

import math

import numpy as np
import torch

import pg_warren_b200 as W

DEVICE = "cuda"


def listed():
    return [
        # The smallest call: one search, a handful of levels, launches and
        # the wait dominate (a program asks this per query).
        {"name": "bfs rmat16 cap8", "path": "bfs", "graph": "rmat", "nodes": 1 << 16,
         "degree": 16, "weights": "none", "depth": 8, "direction": "out"},
        # Rank a small graph: a dozen iterations, each a few microseconds of work.
        {"name": "pagerank rmat16", "path": "pagerank", "graph": "rmat", "nodes": 1 << 16,
         "degree": 16, "weights": "none", "weighted": False, "seeded": False, "tol": 1e-10},
        # Rank a large graph.
        {"name": "pagerank rmat22", "path": "pagerank", "graph": "rmat", "nodes": 1 << 22,
         "degree": 16, "weights": "none", "weighted": False, "seeded": False, "tol": 1e-10},
        # One step of a user's own float iteration over a large weighted graph.
        {"name": "spmv plus_times f64 rmat22", "path": "spmv", "graph": "rmat",
         "nodes": 1 << 22, "degree": 16, "weights": "uniform", "semiring": "plus_times",
         "dtype": "f64", "transpose": True, "mask": False},
        # One relaxation of a shortest-path loop, integer weights, even rows.
        {"name": "spmv min_plus i64 gnm", "path": "spmv", "graph": "gnm", "nodes": 1000003,
         "degree": 16, "weights": "int", "semiring": "min_plus", "dtype": "i64",
         "transpose": True, "mask": False},
        # Features spread over edges: a narrow float matrix, a ragged node count.
        {"name": "spmm plus_times f32 x16", "path": "spmm", "graph": "rmat", "nodes": 300007,
         "degree": 16, "weights": "uniform", "semiring": "plus_times", "dtype": "f32",
         "transpose": False, "width": 16},
        # The headline: 1,024 searches at once.
        {"name": "bfs_batched rmat22 x1024", "path": "bfs_batched", "graph": "rmat",
         "nodes": 1 << 22, "degree": 16, "weights": "none", "sources": 1024},
        # A modest batch on a graph of no particular size.
        {"name": "bfs_batched 150k x100", "path": "bfs_batched", "graph": "rmat",
         "nodes": 150001, "degree": 16, "weights": "none", "sources": 100},
        # Hop-bounded shortest paths from many sources.
        {"name": "minplus_batched rmat20 x128", "path": "minplus_batched", "graph": "rmat",
         "nodes": 1 << 20, "degree": 16, "weights": "int", "sources": 128},
        # Personalised ranks of many seed sets.
        {"name": "ppr_batched rmat20 x64", "path": "ppr_batched", "graph": "rmat",
         "nodes": 1 << 20, "degree": 16, "weights": "none", "sets": 64},
        # Edge gradients of losses over the ranks.
        {"name": "adjoint rmat18 x32", "path": "adjoint", "graph": "rmat", "nodes": 1 << 18,
         "degree": 16, "weights": "lognormal", "losses": 32},
        # The smallest eigenpairs of a component's normalised Laplacian.
        {"name": "eigen rmat18 k8", "path": "eigen", "graph": "rmat", "nodes": 1 << 18,
         "degree": 16, "weights": "none", "k": 8, "which": "smallest",
         "operator": "normalized_laplacian"},
    ]


def draw(rng):
    """One more case: a path, and sizes spread over its range's logarithm."""

    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    path = rng.choice(["bfs", "pagerank", "spmv", "spmm", "bfs_batched", "minplus_batched",
                       "ppr_batched", "adjoint", "eigen"])
    c = {"path": path, "graph": rng.choice(["rmat", "rmat", "gnm"]), "weights": "none"}
    if path == "bfs":
        c.update(nodes=size(1 << 12, 1 << 22), degree=rng.randint(4, 16),
                 depth=rng.choice([3, 8, 64]), direction=rng.choice(["out", "in", "both"]))
    elif path == "pagerank":
        weighted = rng.random() < 0.4
        c.update(nodes=size(1 << 12, 1 << 22), degree=rng.randint(4, 16),
                 weights="uniform" if weighted else "none", weighted=weighted,
                 seeded=rng.random() < 0.3, tol=rng.choice([1e-6, 1e-10]))
    elif path in ("spmv", "spmm"):
        semiring, dtype, weights = rng.choice([
            ("plus_times", "f64", "uniform"), ("plus_times", "f32", "uniform"),
            ("plus_times", "f64", "none"), ("min_plus", "i64", "int"),
            ("min_plus", "f64", "uniform"), ("lor_land", "bool", "none")])
        c.update(nodes=size(1 << 12, 1 << (22 if path == "spmv" else 18)),
                 degree=rng.randint(4, 16), weights=weights, semiring=semiring, dtype=dtype,
                 transpose=rng.random() < 0.5)
        if path == "spmv":
            c["mask"] = rng.random() < 0.2
        else:
            c["width"] = rng.choice([2, 3, 4, 8, 16, 24, 32, 64])
    elif path == "bfs_batched":
        c.update(nodes=size(1 << 12, 1 << 21), degree=rng.randint(4, 16), sources=size(32, 1024))
    elif path == "minplus_batched":
        c.update(nodes=size(1 << 12, 1 << 19), degree=rng.randint(4, 16), weights="int",
                 sources=size(8, 128))
    elif path == "ppr_batched":
        c.update(nodes=size(1 << 12, 1 << 19), degree=rng.randint(4, 16), sets=size(8, 64))
    elif path == "adjoint":
        c.update(nodes=size(1 << 12, 1 << 17), degree=rng.randint(4, 16), weights="lognormal",
                 losses=size(4, 48))
    else:
        which, operator = rng.choice([("smallest", "normalized_laplacian"),
                                      ("largest", "adjacency")])
        c.update(graph="rmat", nodes=size(1 << 12, 1 << 18), degree=rng.randint(8, 16),
                 k=rng.randint(2, 8), which=which, operator=operator)
    return c


# ------------------------------------------------------------------ graphs


def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    return g


def _unique_edges(key, n):
    """(sources, targets) of the sorted distinct keys source·n + target."""
    key = torch.unique(key)
    src = torch.div(key, n, rounding_mode="floor")
    return src, key - src * n


def _edges(case, seed):
    """The case's edges on the device, in CSR order: (n, sources, targets).
    Where the outputs' shape depends on the topology (one gradient an edge,
    one vector over a component) the seed only numbers its nodes."""
    n = case["nodes"]
    order = _generator(seed)
    gen = _generator(n) if case["path"] in ("adjoint", "eigen") else order
    m = n * case["degree"]
    if case["graph"] == "gnm":
        src = torch.randint(0, n, (m,), generator=gen, device=DEVICE)
        dst = torch.randint(0, n, (m,), generator=gen, device=DEVICE)
    else:
        src = torch.zeros(m, dtype=torch.int64, device=DEVICE)
        dst = torch.zeros(m, dtype=torch.int64, device=DEVICE)
        for _ in range((n - 1).bit_length()):
            r = torch.rand(m, generator=gen, device=DEVICE)
            src.mul_(2).add_(r >= 0.76)
            dst.mul_(2).add_(((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
        del r
    keep = (src != dst) & (src < n) & (dst < n)
    src, dst = src[keep], dst[keep]
    if case["path"] == "eigen":
        src, dst = torch.cat([src, dst]), torch.cat([dst, src])
        n, src, dst = _largest_component(n, *_unique_edges(src * n + dst, n))
    relabel = torch.randperm(n, generator=order, device=DEVICE)
    key = relabel[src] * n + relabel[dst]
    del src, dst
    return n, *_unique_edges(key, n)


def _largest_component(n, src, dst):
    """A symmetric graph's largest component, its nodes renumbered in order."""
    label = torch.arange(n, device=DEVICE)
    while True:
        low = label.scatter_reduce(0, dst, label[src], "amin")
        low = torch.minimum(low, low[low])
        if torch.equal(low, label):
            break
        label = low
    inside = label == torch.bincount(label, minlength=n).argmax()
    number = torch.cumsum(inside, 0) - 1
    keep = inside[src]
    return int(inside.sum()), number[src[keep]], number[dst[keep]]


def _weights(case, n, src, seed):
    """Per-edge weights (host float64): U(0, 1], U{1..100}, or exp(N(0, 1))
    normalised so that each row sums to 1."""
    rng = np.random.default_rng(seed)
    m = len(src)
    if case["weights"] == "none":
        return None
    if case["weights"] == "uniform":
        return 1.0 - rng.random(m)
    if case["weights"] == "int":
        return rng.integers(1, 101, m).astype(np.float64)
    w = np.exp(rng.standard_normal(m))
    rows = src.cpu().numpy()
    return w / np.bincount(rows, weights=w, minlength=n)[rows]


def _inputs(case, seed):
    """The graph and the path's inputs, from the seed alone."""
    n, src, dst = _edges(case, seed)
    w = _weights(case, n, src, seed)
    rng = np.random.default_rng(seed + 1)
    path, s = case["path"], {"n": n, "src": src, "dst": dst, "w": w}
    if path == "bfs":
        # A node that has edges in the searched direction.
        ends = dst if case["direction"] == "in" else src
        s["starts"] = [int(ends[int(rng.integers(0, len(ends)))])]
    elif path == "pagerank":
        s["seed"] = None
        if case["seeded"]:
            seeds = np.zeros(n)
            seeds[rng.choice(n, max(1, n // 1000), replace=False)] = 1.0
            s["seed"] = torch.as_tensor(seeds, device=DEVICE)
    elif path in ("spmv", "spmm"):
        gen = _generator(seed + 2)
        shape = (n,) if path == "spmv" else (n, case["width"])
        dtype = case["dtype"]
        if dtype in ("f64", "f32") and case["semiring"] == "plus_times":
            s["x"] = torch.rand(shape, generator=gen, device=DEVICE, dtype=torch.float64).to(
                torch.float64 if dtype == "f64" else torch.float32)
        else:
            # A frontier: one node in a hundred holds a value, the others
            # the additive identity.
            hot = torch.rand(shape, generator=gen, device=DEVICE) < 0.01
            if dtype == "bool":
                s["x"] = hot.to(torch.uint8)
            elif dtype == "i64":
                d = torch.randint(0, 1000, shape, generator=gen, device=DEVICE)
                s["x"] = torch.where(hot, d, torch.full_like(d, np.iinfo(np.int64).max))
            else:
                d = torch.rand(shape, generator=gen, device=DEVICE, dtype=torch.float64)
                s["x"] = torch.where(hot, d, torch.full_like(d, math.inf))
        s["y"] = torch.zeros_like(s["x"])
        s["mask"] = None
        if case.get("mask"):
            s["mask"] = (torch.rand(n, generator=gen, device=DEVICE) < 0.5).to(torch.uint8)
    elif path in ("bfs_batched", "minplus_batched"):
        k = case["sources"]
        s["sources"] = rng.integers(0, n, k).astype(np.uint64)
        s["caps"] = rng.integers(1, 17, k).astype(np.uint32)
    elif path == "ppr_batched":
        sizes = np.exp(rng.uniform(0, np.log(1000), case["sets"])).astype(np.int64)
        s["sets"] = [rng.choice(n, int(q), replace=False) for q in sizes]
    elif path == "adjoint":
        s["losses"] = [rng.choice(n, 1000, replace=False) for _ in range(case["losses"])]
    return s


# ---------------------------------------------------------------- the calls


def prepare(case, seed):
    s = _inputs(case, seed)
    n, src, dst, w = s["n"], s.pop("src"), s.pop("dst"), s.pop("w")
    offsets = torch.zeros(n + 1, dtype=torch.int64, device=DEVICE)
    offsets[1:] = torch.cumsum(torch.bincount(src, minlength=n), 0)
    m = len(src)
    graph = W.GraphVersion(offsets.cpu().numpy().view(np.uint64),
                           dst.to(torch.int32).cpu().numpy().view(np.uint32), w)
    del src, dst, offsets
    s.update(case=case, graph=graph)

    def empty(shape, dtype):
        return torch.zeros(shape, dtype=dtype, device=DEVICE)

    path = case["path"]
    if path == "bfs":
        s.update(depth=empty(n, torch.int32), via=empty(n, torch.int64))
    elif path == "pagerank":
        s["out"] = empty(n, torch.float64)
    elif path == "bfs_batched":
        s.update(depth=empty((case["sources"], n), torch.uint8),
                 edges=empty(case["sources"], torch.int64))
    elif path == "minplus_batched":
        s.update(dist=empty((case["sources"], n), torch.int64),
                 iterations=empty(case["sources"], torch.int32))
    elif path == "ppr_batched":
        s.update(ranks=empty((case["sets"], n), torch.float64),
                 iterations=empty(case["sets"], torch.int32))
    elif path == "adjoint":
        s["grad"] = empty((case["losses"], m), torch.float64)
    return s


def run(s):
    c, g = s["case"], s["graph"]
    path = c["path"]
    if path == "bfs":
        _, _, stats = W.bfs_depths(g, s["starts"], max_depth=c["depth"], direction=c["direction"],
                                   depth_out=s["depth"], via_out=s["via"])
        return [s["depth"], s["via"], stats.nodes_visited, stats.edges_traversed]
    if path == "pagerank":
        opts = W.PageRank(0.85, c["tol"], 100, c["weighted"], s["seed"])
        r = W.pagerank(g, None, opts, out=s["out"])
        return [r.values, r.iterations]
    if path in ("spmv", "spmm"):
        call = W.spmv if path == "spmv" else W.spmm
        call(g, W.Product(c["semiring"], transpose=c["transpose"], mask=s["mask"]), s["x"], s["y"])
        return [s["y"]]
    if path == "bfs_batched":
        return list(W.bfs_batched(g, s["sources"], s["caps"], depth_out=s["depth"],
                                  edges_out=s["edges"]))
    if path == "minplus_batched":
        return list(W.minplus_batched(g, s["sources"], s["caps"], dist_out=s["dist"],
                                      iterations_out=s["iterations"]))
    if path == "ppr_batched":
        return list(W.ppr_batched(g, s["sets"], W.PageRank(0.85, 1e-10, 100),
                                  ranks_out=s["ranks"], iterations_out=s["iterations"]))
    if path == "adjoint":
        grad, ranks, iterations = W.pagerank_adjoint(
            g, s["losses"], W.PageRank(0.85, None, 100), adjoint_tol=1e-14, grad_out=s["grad"])
        return [grad, ranks, iterations]
    e = W.eigen(g, W.EigenOptions(c["k"], which=c["which"], operator=c["operator"], tol=1e-10,
                                  max_iter=1000, seed=7))
    return [e.values, e.vectors]


def work(case):
    """What one pass cannot do without: the graph (u32 offsets and targets,
    the weights the path reads) and the path's inputs read once, its outputs
    written once; the multiply-adds over the edges, with the iterations such
    a solve takes on these graphs.  Edges as drawn, duplicates among them."""
    n, path = case["nodes"], case["path"]
    m = n * case["degree"]
    graph = 4 * (n + 1) + 4 * m
    if path == "bfs":
        return {"bytes": graph + 12 * n, "flops": 0}
    if path == "pagerank":
        return {"bytes": graph + (8 * m if case["weighted"] else 0) + 8 * n,
                "flops": 2.0 * m * (10 if case["tol"] < 1e-8 else 5)}
    if path in ("spmv", "spmm"):
        element = {"f64": 8, "f32": 4, "i64": 8, "bool": 1}[case["dtype"]]
        weight = {"none": 0, "int": 4, "uniform": 8}[case["weights"]]
        width = case.get("width", 1)
        return {"bytes": graph + weight * m + 2 * element * width * n, "flops": 2.0 * m * width}
    if path == "bfs_batched":
        return {"bytes": graph + n * case["sources"], "flops": 0}
    if path == "minplus_batched":
        return {"bytes": graph + 4 * m + 8 * n * case["sources"], "flops": 0}
    if path == "ppr_batched":
        return {"bytes": graph + 8 * n * case["sets"], "flops": 2.0 * m * case["sets"] * 13}
    if path == "adjoint":
        return {"bytes": graph + 8 * m + 8 * m * case["losses"],
                "flops": 2.0 * m * (case["losses"] * 101 + 100)}
    return {"bytes": 2 * graph + 8 * n * case["k"], "flops": 4.0 * m * 150}


# ------------------------------------------------------------ in 64 bits


def _pull(src, dst, w, x, n):
    """y[dst] += w · x[src] over the edges; x: n or n × k."""
    v = x[src]
    if w is not None:
        v = v * (w if x.dim() == 1 else w[:, None])
    return torch.zeros_like(x).index_add_(0, dst, v)


def _pagerank(n, src, dst, w, shares, tol, max_iter, columns=None):
    """The ranks as the iteration leaves them: start 1/n, shares the
    personalisation (1/n, or one column per seed set), each column stopping
    when its L1 change falls below n · tol."""
    ones = torch.ones(len(src), dtype=torch.float64, device=DEVICE)
    out = torch.zeros(n, dtype=torch.float64, device=DEVICE).index_add_(
        0, src, ones if w is None else w)
    some = out > 0
    k = columns or 1
    x = torch.full((n, k), 1.0 / n, dtype=torch.float64, device=DEVICE)
    p = shares if columns else shares[:, None] if torch.is_tensor(shares) else shares
    scale = torch.where(some, out, torch.ones_like(out))[:, None]
    going = torch.ones(k, dtype=torch.bool, device=DEVICE)
    for _ in range(max_iter):
        msg = torch.where(some[:, None], x / scale, torch.zeros_like(x))
        dangling = torch.where(some[:, None], torch.zeros_like(x), x).sum(0)
        nxt = 0.85 * (_pull(src, dst, w, msg, n) + dangling * p) + (1.0 - 0.85) * p
        change = (nxt - x).abs().sum(0)
        x = torch.where(going, nxt, x)
        if tol is not None:
            going = going & ~(change < n * tol)
            if not bool(going.any()):
                break
    return (x if columns else x[:, 0]), out


def _smallest_or_largest(n, src, dst, case):
    """Eigenvalues by Lanczos with full reorthogonalisation, far past the
    steps the wanted end of the spectrum needs."""
    one = torch.ones(len(src), dtype=torch.float64, device=DEVICE)
    degree = torch.zeros(n, dtype=torch.float64, device=DEVICE).index_add_(0, src, one)
    laplacian = case["operator"] == "normalized_laplacian"
    inv = degree.rsqrt()

    def apply(v):
        if laplacian:
            return v - inv * _pull(src, dst, None, inv * v, n)
        return _pull(src, dst, None, v, n)

    steps = min(n, 500)
    q = torch.zeros(steps + 1, n, dtype=torch.float64, device=DEVICE)
    q[0] = torch.randn(n, generator=_generator(5), device=DEVICE, dtype=torch.float64)
    q[0] /= q[0].norm()
    alpha, beta = [], []
    for j in range(steps):
        v = apply(q[j])
        alpha.append(float(q[j] @ v))
        for _ in range(2):
            v = v - q[: j + 1].T @ (q[: j + 1] @ v)
        beta.append(float(v.norm()))
        if beta[-1] < 1e-12:
            break
        q[j + 1] = v / beta[-1]
    t = torch.diag(torch.tensor(alpha, dtype=torch.float64))
    if len(alpha) > 1:
        off = torch.tensor(beta[: len(alpha) - 1], dtype=torch.float64)
        t = t + torch.diag(off, 1) + torch.diag(off, -1)
    values = torch.linalg.eigvalsh(t)
    if case["which"] == "largest":  # in magnitude
        values = values[values.abs().argsort(descending=True)]
    return values[: case["k"]]


def exact(case, seed):
    path = case["path"]
    if path in ("bfs", "bfs_batched", "minplus_batched"):
        return None  # whole numbers
    if path in ("spmv", "spmm") and case["dtype"] in ("i64", "bool"):
        return None
    s = _inputs(case, seed)
    n, src, dst = s["n"], s["src"], s["dst"]
    w = None if s["w"] is None else torch.as_tensor(s["w"], device=DEVICE)
    if path == "pagerank":
        shares = 1.0 / n if s["seed"] is None else s["seed"] / s["seed"].sum()
        ranks, _ = _pagerank(n, src, dst, w if case["weighted"] else None, shares, case["tol"], 100)
        return [ranks, None]
    if path in ("spmv", "spmm"):
        frm, to = (src, dst) if case["transpose"] else (dst, src)
        x = s["x"].to(torch.float64)
        columns = []
        for c in (x[:, None] if x.dim() == 1 else x).unbind(1):
            c = c.contiguous()
            if case["semiring"] == "plus_times":
                columns.append(_pull(frm, to, w, c, n))
            else:
                y = torch.full_like(c, math.inf)
                columns.append(y.scatter_reduce_(0, to, c[frm] + w, "amin"))
        y = columns[0] if x.dim() == 1 else torch.stack(columns, 1)
        if s["mask"] is not None:
            y = torch.where(s["mask"] != 0, y, torch.zeros_like(y))
        return [y]
    if path == "ppr_batched":
        ranks = torch.empty(case["sets"], n, dtype=torch.float64, device=DEVICE)
        for a in range(0, case["sets"], 8):
            some = s["sets"][a:a + 8]
            shares = torch.zeros(n, len(some), dtype=torch.float64, device=DEVICE)
            for q, nodes in enumerate(some):
                shares[torch.as_tensor(nodes, device=DEVICE), q] = 1.0 / len(nodes)
            ranks[a:a + len(some)] = _pagerank(n, src, dst, None, shares, 1e-10, 100,
                                               len(some))[0].T
        return [ranks, None]
    if path == "adjoint":
        x, out = _pagerank(n, src, dst, w, 1.0 / n, None, 100)
        grad = torch.empty(case["losses"], len(src), dtype=torch.float64, device=DEVICE)
        some = (out > 0)[:, None]
        scale = torch.where(out > 0, out, torch.ones_like(out))[:, None]
        for a in range(0, case["losses"], 8):
            losses = s["losses"][a:a + 8]
            c = torch.zeros(n, len(losses), dtype=torch.float64, device=DEVICE)
            for q, nodes in enumerate(losses):
                c[torch.as_tensor(nodes, device=DEVICE), q] = 1.0
            lam, zero = c, torch.zeros_like(c)
            for _ in range(100):
                mean = torch.where(some, zero, lam.sum(0) / n)
                lam = 0.85 * (torch.where(some, _pull(dst, src, w, lam, n) / scale, mean)) + c
            rows = torch.where(some, _pull(dst, src, w, lam, n) / scale, zero)
            coef = (0.85 * x / scale[:, 0])[src]
            for q in range(len(losses)):
                grad[a + q] = coef * (lam[dst, q] - rows[src, q])
        return [grad, x, None]
    return [_smallest_or_largest(n, src, dst, case).numpy(), None]
