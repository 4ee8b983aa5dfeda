"""Performance cases: the work a program has this engine do, over its range.

A case names a vertex program, the graph it runs on and the options it is called
with. Graphs are made on the GPU from the seed: R-MAT (0.57, 0.19, 0.19, 0.05) for
skewed degrees, uniform random (Erdos-Renyi) and the 4-neighbour lattice with 0.1%
long-range pairs for long diameters; the listed sizes are the ones of bench.py and
of the tests. Every pass goes through ``mirrorofmapgraph_b200.Graph``.
"""
from __future__ import annotations

import math

import torch

import mirrorofmapgraph_b200 as mg

ALPHA = 0.85
# Sweeps of a PageRank case: about what L1 < 1e-6 takes on the R-MAT graphs; a fixed
# number, so that a result does not hang on which side of the tolerance a sum rounds.
SWEEPS = 16
NEVER = 1e-30  # a tolerance no iterate reaches
# Iterations of the adjoint to its 1e-7 (R-MAT, alpha 0.85); only work() uses it.
ADJOINT_SWEEPS = 65


def listed():
    return [
        # The smallest call: one BFS on 4,096 vertices, depths back on the host (launches and latency).
        dict(name="bfs_er4k", kind="bfs", graph="er", n=4096, deg=16, sym=False, host=True),
        # The four programs on a resident graph of 4.2 M vertices and 134 M edges, results left on the device.
        dict(name="bfs_rmat22", kind="bfs", graph="rmat", n=1 << 22, deg=16, sym=True, host=False),
        dict(name="sssp_rmat22", kind="sssp", graph="rmat", n=1 << 22, deg=16, sym=True, host=False),
        dict(name="cc_rmat22", kind="cc", graph="rmat", n=1 << 22, deg=16, sym=True, host=False),
        # PageRank solved again and again on one graph, its gather tuned once for that graph.
        dict(name="pagerank_rmat22", kind="pagerank", graph="rmat", n=1 << 22, deg=16, sym=True, weighted=False,
             gather="auto"),
        # Hundreds of rounds of small frontiers: shortest paths over a 4096 x 4096 grid.
        dict(name="sssp_lattice4096", kind="sssp", graph="lattice", n=4096 * 4096, deg=4, sym=True, host=False),
        # Many sources or teleport vectors on one graph in one call.
        dict(name="bfs64_rmat20", kind="bfs_batch", graph="rmat", n=1 << 20, deg=16, sym=True, k=64),
        dict(name="sssp64_rmat20", kind="sssp_batch", graph="rmat", n=1 << 20, deg=16, sym=True, k=64),
        dict(name="ppr256_rmat20", kind="ppr", graph="rmat", n=1 << 20, deg=16, sym=True, weighted=False, k=256),
        # Training the edge weights: gradients of a loss on the ranks by every weight and the teleport vector.
        dict(name="adjoint_rmat22", kind="adjoint", graph="rmat", n=1 << 22, deg=16, sym=False, weighted=True),
        # A new weighted digraph each time: upload (device CSR), transpose, one solve, release.
        dict(name="oneshot_rmat20", kind="oneshot", graph="rmat", n=1 << 20, deg=16, sym=False, weighted=True),
        # The reference's own PageRank (delta frontier, 0.01) on a digraph, ranks back on the host.
        dict(name="refcompat_rmat18", kind="refcompat", graph="rmat", n=1 << 18, deg=16, sym=False),
    ]


def _between(rng, lo, hi):
    """A whole number between lo and hi, spread over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["bfs", "bfs", "sssp", "sssp", "cc", "pagerank", "bfs_batch", "sssp_batch", "ppr", "adjoint",
                       "oneshot", "refcompat"])
    graph = rng.choice(["rmat", "rmat", "er"])
    sym = rng.random() < 0.6
    most = {"bfs": 4 << 20, "sssp": 4 << 20, "cc": 4 << 20, "pagerank": 4 << 20, "bfs_batch": 1 << 20,
            "sssp_batch": 1 << 18, "ppr": 1 << 17, "adjoint": 1 << 20, "oneshot": 1 << 20, "refcompat": 1 << 18}[kind]
    n = _between(rng, 1000, most)
    c = dict(kind=kind, graph=graph, n=n, deg=_between(rng, 3, 24), sym=sym)
    if kind in ("bfs", "sssp"):
        if rng.random() < 0.3:
            side = _between(rng, 60, 2500)
            c.update(graph="lattice", n=side * side, deg=4, sym=True)
        c["host"] = c["n"] < 100000
    elif kind == "cc":
        c["host"] = n < 100000
        if graph == "er":
            c["deg"] = rng.randint(1, 3)  # more than one component
    elif kind == "pagerank":
        c.update(weighted=rng.random() < 0.4, gather=rng.choice(["auto", "default"]))
    elif kind in ("bfs_batch", "sssp_batch"):
        c["k"] = rng.randint(3, 100)
    elif kind == "ppr":
        c.update(weighted=rng.random() < 0.4, k=rng.randint(5, 256))
    elif kind in ("adjoint", "oneshot"):
        c["weighted"] = rng.random() < 0.7
    return c


# ---------------------------------------------------------------------------
# Graphs: int32 CSR on the GPU, duplicates kept, a self-loop turned to the next vertex.
def _rmat(n, m, gen):
    """R-MAT endpoints, skewed towards low ids (no relabelling), scaled to n vertices."""
    scale = max(1, math.ceil(math.log2(n)))
    src = torch.zeros(m, dtype=torch.int32, device="cuda")
    dst = torch.zeros(m, dtype=torch.int32, device="cuda")
    for _ in range(scale):
        r = torch.rand(m, device="cuda", generator=gen)
        src.mul_(2).add_(r >= 0.76)
        dst.mul_(2).add_(((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
    if n != 1 << scale:
        src = ((src.long() * n) >> scale).int()
        dst = ((dst.long() * n) >> scale).int()
    return src, dst


def _lattice(side, gen):
    v = torch.arange(side * side, dtype=torch.int32, device="cuda")
    right, down = v[v % side != side - 1], v[: side * (side - 1)]
    far = torch.randint(0, side * side, (2, side * side // 1000), device="cuda", generator=gen, dtype=torch.int32)
    return torch.cat([right, down, far[0]]), torch.cat([right + 1, down + side, far[1]])


def _csr(case, gen):
    """(row offsets, column indices, edge values or None) of the case's graph."""
    n = case["n"]
    if case["graph"] == "lattice":
        src, dst = _lattice(math.isqrt(n), gen)
    elif case["graph"] == "rmat":
        src, dst = _rmat(n, n * case["deg"], gen)
    else:
        src, dst = torch.randint(0, n, (2, n * case["deg"]), device="cuda", generator=gen, dtype=torch.int32)
    dst = torch.where(src == dst, (dst + 1) % n, dst)
    w = None
    if case["kind"] in ("sssp", "sssp_batch"):
        w = torch.randint(1, 1001 if case["graph"] == "lattice" else 256, src.shape, device="cuda", generator=gen,
                          dtype=torch.int32)
    elif case.get("weighted"):
        w = torch.empty(src.shape, device="cuda").log_normal_(0.0, 1.0, generator=gen)
    if case["sym"]:
        src, dst = torch.cat([src, dst]), torch.cat([dst, src])
        w = None if w is None else torch.cat([w, w])
    src, order = torch.sort(src, stable=True)
    ro = torch.searchsorted(src, torch.arange(n + 1, dtype=torch.int32, device="cuda"), out_int32=True)
    return ro, dst[order], None if w is None else w[order]


def _sources(ro, k, gen):
    """k vertices that have out-edges (a search from any other ends at once)."""
    cand = torch.nonzero(ro[1:] > ro[:-1]).view(-1)
    return cand[torch.randint(0, cand.numel(), (k,), device="cuda", generator=gen)].int().cpu().numpy()


def _teleports(n, k, gen):
    """k sparse teleport vectors: 1 to 32 vertices each, uniform mass on them."""
    t = torch.zeros(k, n, device="cuda")
    at = torch.randint(0, n, (k, 32), device="cuda", generator=gen)
    cnt = torch.randint(1, 33, (k, 1), device="cuda", generator=gen)
    on = torch.arange(32, device="cuda").view(1, 32) < cnt
    t.scatter_add_(1, at, on.float() / cnt)
    return t.view(-1)


# ---------------------------------------------------------------------------
def _inputs(case, seed):
    """Everything random of a case, from the seed: the CSR, then sources, teleports or loss weights."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    ro, ci, w = _csr(case, gen)
    kind, n = case["kind"], case["n"]
    more = None
    if kind in ("bfs", "sssp"):
        more = [0] if case["graph"] != "rmat" else _sources(ro, 1, gen)
    elif kind in ("bfs_batch", "sssp_batch"):
        more = _sources(ro, case["k"], gen)
    elif kind == "ppr":
        more = _teleports(n, case["k"], gen)
    elif kind == "adjoint":
        more = torch.randn(n, device="cuda", generator=gen)
    return ro, ci, w, more


def _pr_keys(case):
    return dict(mode="normalized", alpha=ALPHA, tol=NEVER, max_iter=SWEEPS, weighted=bool(case.get("weighted")))


def prepare(case, seed):
    ro, ci, w, more = _inputs(case, seed)
    kind, n, m = case["kind"], case["n"], ci.numel()
    s = dict(case=case, more=more)
    torch.cuda.synchronize()  # the engine copies on its own stream
    if kind == "oneshot":
        s.update(ro=ro, ci=ci, w=w, out=torch.empty(n, device="cuda"))
        return s
    g = s["g"] = mg.Graph(ro, ci, w, symmetric=case["sym"])
    if kind in ("bfs", "sssp", "cc"):
        s["out"] = None if case["host"] else torch.empty(n, dtype=torch.int32, device="cuda")
    elif kind in ("bfs_batch", "sssp_batch"):
        s["out"] = torch.empty(case["k"] * n, dtype=torch.int32, device="cuda")
    elif kind == "ppr":
        s["out"] = torch.empty(case["k"] * n, device="cuda")
        # tuned once for the graph, as a program that keeps it does
        g.pagerank(teleport=more, nvec=case["k"], out=s["out"], autotune=True, **_pr_keys(case))
    elif kind == "pagerank":
        s["out"] = torch.empty(n, device="cuda")
        if case["gather"] == "auto":
            g.pagerank(out=s["out"], autotune=True, **_pr_keys(case))
    elif kind == "adjoint":
        s["x"] = g.pagerank(out=torch.empty(n, device="cuda"), **_pr_keys(case))[0]
        s["out"] = torch.empty(m, device="cuda"), torch.empty(n, device="cuda")
    return s


def run(s):
    case, g, more, out = s["case"], s.get("g"), s["more"], s.get("out")
    kind = case["kind"]
    if kind == "bfs":
        return g.bfs(more, out=out)[0]
    if kind == "sssp":
        return g.sssp(more, out=out)[0]
    if kind == "cc":
        return g.cc(out=out)[0]
    if kind == "bfs_batch":
        return g.bfs_batch(more, out=out)[0]
    if kind == "sssp_batch":
        return g.sssp_batch(more, out=out)[0]
    if kind == "pagerank":
        return g.pagerank(out=out, autotune=case["gather"] == "auto", **_pr_keys(case))[0]
    if kind == "ppr":
        return g.pagerank(teleport=more, nvec=case["k"], out=out, autotune=True, **_pr_keys(case))[0]
    if kind == "adjoint":
        gw, gt, _ = g.pagerank_backward(s["x"], more, alpha=ALPHA, tol=1e-7, max_iter=200,
                                        weighted=bool(case["weighted"]), out_weights=out[0], out_teleport=out[1])
        return gw, gt
    if kind == "oneshot":
        with mg.Graph(s["ro"], s["ci"], s["w"], symmetric=case["sym"]) as once:
            return once.pagerank(out=out, **_pr_keys(case))[0]
    return g.pagerank(mode="refcompat")[0]


def work(case):
    """Each array of the graph read once per sweep (a traversal is one sweep), the results written once."""
    n, kind = case["n"], case["kind"]
    m = n * case["deg"] * (2 if case["sym"] and case["graph"] != "lattice" else 1)
    graph = 4 * (n + 1) + 4 * m
    if kind in ("bfs", "cc"):
        return dict(bytes=graph + 4 * n, flops=0)
    if kind == "sssp":
        return dict(bytes=graph + 4 * m + 4 * n, flops=0)
    if kind in ("bfs_batch", "sssp_batch"):
        return dict(bytes=graph + (4 * m if kind == "sssp_batch" else 0) + 4 * n * case["k"], flops=0)
    if case.get("weighted"):
        graph += 4 * m
    if kind == "ppr":
        k = case["k"]
        return dict(bytes=SWEEPS * (graph + 12 * n * k), flops=SWEEPS * 2 * m * k)
    if kind == "adjoint":
        return dict(bytes=ADJOINT_SWEEPS * (graph + 12 * n) + 2 * graph + 4 * m, flops=ADJOINT_SWEEPS * 2 * m)
    if kind == "oneshot":
        return dict(bytes=SWEEPS * (graph + 12 * n) + 3 * graph, flops=SWEEPS * 2 * m)
    return dict(bytes=SWEEPS * (graph + 12 * n), flops=SWEEPS * 2 * m)


def tolerance(case):
    kind = case["kind"]
    if kind in ("bfs", "sssp", "cc", "bfs_batch", "sssp_batch"):
        return "exact"
    if kind == "refcompat":
        # a vertex whose change rounds to the other side of 0.01 stops or goes on one sweep earlier
        return {"rel": 1e-6, "max": 1e-2}
    if kind == "adjoint":
        # stopped at a relative change of 1e-7, one sweep earlier or later (4e-7 off the 64-bit solution)
        return {"rel": 2e-6, "max": 1e-4}
    return {"rel": 2e-7, "max": 1e-5}  # 3e-8 off the 64-bit sweeps


# ---------------------------------------------------------------------------
# The results in 64 bits, by sparse products of plain torch.
def _sparse(ro, ci, w, n):
    return torch.sparse_csr_tensor(ro.long(), ci.long(),
                                   torch.ones(ci.shape, dtype=torch.float64, device=ci.device) if w is None
                                   else w.double(), size=(n, n))


def _rows_of(ro, m):
    return torch.repeat_interleave(torch.arange(ro.numel() - 1, device=ro.device), (ro[1:] - ro[:-1]).long(),
                                   output_size=m)


def _transposed(ro, ci, w):
    rows = _rows_of(ro, ci.numel())
    col, order = torch.sort(ci, stable=True)
    co = torch.searchsorted(col, torch.arange(ro.numel(), dtype=torch.int32, device="cuda"), out_int32=True)
    return co, rows[order].int(), None if w is None else w[order]


def _power(at, s, t, sweeps):
    """x <- alpha (A^T (x / s) + d t) + (1 - alpha) t from x = t; s, t and x have a column per vector."""
    x, live = t.clone(), s > 0
    for _ in range(sweeps):
        g = torch.where(live, x / s, torch.zeros_like(x))
        d = torch.where(live, torch.zeros_like(x), x).sum(0, keepdim=True)
        x = ALPHA * (at @ g + d * t) + (1 - ALPHA) * t
    return x


def _refcompat(ro, ci, n):
    """x = 0.15 + 0.85 sum x_u / deg_u on the frontier; next: the heads of those that moved by 0.01 or more."""
    co, ri, _ = _transposed(ro, ci, None)
    at = _sparse(co, ri, None, n)
    deg = (ro[1:] - ro[:-1]).double().view(-1, 1).clamp(min=1)
    x = torch.full((n, 1), 0.15, dtype=torch.float64, device="cuda")
    front = torch.ones(n, 1, dtype=torch.bool, device="cuda")
    while bool(front.any()):
        new = 0.15 + 0.85 * (at @ (x / deg))
        moved = front & ((new - x).abs() >= 0.01)
        x = torch.where(front, new, x)
        front = (at @ moved.double()) > 0
    return x


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if tolerance(case) == "exact":
        return None  # whole numbers: depths, distances, labels
    ro, ci, w, more = _inputs(case, seed)
    if kind == "refcompat":
        return _refcompat(ro, ci, n).view(-1).cpu().numpy()
    m = ci.numel()
    a = _sparse(ro, ci, w, n)
    s = a @ torch.ones(n, 1, dtype=torch.float64, device="cuda")
    at = _sparse(*_transposed(ro, ci, w), n)
    u = torch.full((n, 1), 1.0 / n, dtype=torch.float64, device="cuda")
    if kind in ("pagerank", "oneshot"):
        return _power(at, s, u, SWEEPS).view(-1)
    if kind == "ppr":
        t = more.view(case["k"], n).t()
        cols = [_power(at, s, t[:, c:c + 32].double().contiguous(), SWEEPS) for c in range(0, case["k"], 32)]
        return torch.cat([c.t() for c in cols]).reshape(-1)
    # adjoint: lambda = w + alpha (P lambda + [dangling] (t . lambda)), then the two gradients. The ranks are
    # an input of the call; their 64-bit values stand for them.
    x = _power(at, s, u, SWEEPS)
    del at
    live = s > 0
    wv = more.double().view(-1, 1)
    lam = wv.clone()
    for _ in range(400):
        pl = torch.where(live, (a @ lam) / s, torch.zeros_like(lam))
        new = wv + ALPHA * (pl + torch.where(live, 0.0, 1.0) * lam.mean())
        change = float((new - lam).abs().sum() / new.abs().sum())
        lam = new
        if change < 1e-14:
            break
    pl = torch.where(live, (a @ lam) / s, torch.zeros_like(lam))
    rows = _rows_of(ro, m)
    coef = torch.where(live, ALPHA * x / s, torch.zeros_like(s)).view(-1)
    gw = coef[rows] * (lam.view(-1)[ci.long()] - pl.view(-1)[rows])
    d = x[~live].sum()
    return gw, lam.view(-1) * (1 - ALPHA + ALPHA * d)
