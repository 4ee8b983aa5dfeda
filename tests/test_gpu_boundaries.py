"""Kernels at the sizes where their tiles, bins and limits end, against the oracle:
the degree bins of the PageRank gather and of its adjoint, the radix sort behind the
CSC, the sampled forest of the components, the reference-compatible sweep in its
three forms, the near-far rounds in one launch and the cluster BFS of small graphs."""
import numpy as np
import pytest

import oracle
import mirrorofmapgraph_b200 as mg
from mirrorofmapgraph_b200 import _lib as L

pytestmark = pytest.mark.gpu

L1_TOL = 1e-6  # FP32 compensated sums against the FP64 oracle, same iterations


def _csr(n, src, dst, w=None):
    order = np.argsort(src, kind="stable")
    ro = np.searchsorted(src[order], np.arange(n + 1)).astype(np.int32)
    return ro, dst[order].astype(np.int32), None if w is None else w[order]


def _device_array(ptr, n, dtype):
    import torch

    class View:
        __cuda_array_interface__ = {"data": (ptr, False), "shape": (n,), "typestr": np.dtype(dtype).str, "version": 2}
    return torch.as_tensor(View(), device="cuda").cpu().numpy()


def _in_degrees(degs, seed):
    """A digraph whose vertex i has degs[i] in-edges from random vertices."""
    rng = np.random.default_rng(seed)
    n = max(len(degs), 64)
    dst = np.repeat(np.arange(len(degs)), degs)
    src = rng.integers(0, n, dst.size)
    p = rng.permutation(dst.size)
    return (n,) + _csr(n, src[p], dst[p], rng.lognormal(0, 1, dst.size).astype(np.float32))


# every bin's first and last degree, one or several rows of each
BIN_DEGREES = [0, 1, 2, 3, 4, 5, 8, 9, 12, 13, 16, 17, 24, 25, 32, 33, 48, 49, 64, 65, 255, 256, 257, 2047, 2048, 4097]


@pytest.mark.parametrize("rep", [1, 9, 33])
@pytest.mark.parametrize("weighted", [False, True])
def test_gather_bins(rep, weighted):
    n, ro, ci, w = _in_degrees(BIN_DEGREES * rep, rep)
    with mg.Graph(ro, ci, w) as g:
        for gather in ("binned", "cached"):
            x, st = g.pagerank(mode="normalized", weighted=weighted, max_iter=12, tol=1e-30, gather=gather)
            xr, _, _ = oracle.pr_normalized(ro, ci, w if weighted else None, 0.85, 0.0, 12)
            assert np.abs(x - xr).sum() <= L1_TOL
    # the adjoint gathers over the rows: the same degrees on the out-side
    co, ri, _ = mg.csr_to_csc(mg.HostCsr(ro, ci))
    wt = np.random.default_rng(1).lognormal(0, 1, ci.size).astype(np.float32)
    dl = np.random.default_rng(2).standard_normal(n).astype(np.float32)
    with mg.Graph(co, ri, wt) as g:
        x, _ = g.pagerank(mode="normalized", weighted=weighted, max_iter=300, tol=1e-9)
        gw, gt, _ = g.pagerank_backward(x, dl, weighted=weighted, tol=1e-7, max_iter=300)
        rw, rt, _, _ = oracle.pr_adjoint(co, ri, wt if weighted else None, x.astype(np.float64), dl, 0.85, 1e-12, 1000)
        assert np.linalg.norm(gw - rw) <= 1e-5 * np.linalg.norm(rw)
        assert np.linalg.norm(gt - rt) <= 1e-5 * np.linalg.norm(rt)


def test_edge_gradients_unaligned_output():
    import torch
    n, ro, ci, w = _in_degrees(BIN_DEGREES, 5)
    dl = torch.randn(n, device="cuda")
    with mg.Graph(torch.from_numpy(ro).cuda(), torch.from_numpy(ci).cuda(), torch.from_numpy(w).cuda()) as g:
        x = g.pagerank(mode="normalized", weighted=True, out=torch.empty(n, device="cuda"))[0]
        a = g.pagerank_backward(x, dl, weighted=True, out_weights=torch.empty(ci.size, device="cuda"),
                                out_teleport=torch.empty(n, device="cuda"))[0]
        buf = torch.full((ci.size + 2,), 7.0, device="cuda")
        b = g.pagerank_backward(x, dl, weighted=True, out_weights=buf[1:-1],
                                out_teleport=torch.empty(n, device="cuda"))[0]
        # two solves agree to an ulp or so (their FP64 sums follow the work schedule)
        assert torch.allclose(a, b, rtol=1e-5, atol=1e-7 * float(a.abs().max()))
        assert buf[0] == 7.0 and buf[-1] == 7.0


@pytest.mark.parametrize("n,m", [(1, 0), (1, 5), (2, 1), (3, 31), (255, 4095), (256, 4096), (257, 4097), (65536, 9000),
                                 (65537, 70001), (300000, 5)])
@pytest.mark.parametrize("vals", [None, np.int32, np.float32])
@pytest.mark.parametrize("hot", [False, True])
def test_csc_build(n, m, vals, hot):
    rng = np.random.default_rng(n + m)
    src, dst = rng.integers(0, n, m), rng.integers(0, n, m)
    if hot:  # half of the edges into one column, from one row
        dst[: m // 2] = n - 1
        src[m // 3:] = n // 2
    w = None if vals is None else rng.integers(1, 1000, m).astype(vals)
    ro, ci, w = _csr(n, src, dst, w)
    co, ri, perm = mg.csr_to_csc(mg.HostCsr(ro, ci))
    with mg.Graph(ro, ci, w) as g:
        d = g.device_arrays()
        np.testing.assert_array_equal(_device_array(d["col_offsets"], n + 1, np.int32), co)
        if m:
            np.testing.assert_array_equal(_device_array(d["row_idx"], m, np.int32), ri)
            np.testing.assert_array_equal(_device_array(d["csc_perm"], m, np.int32), perm)
        if m and vals is not None:  # in-edge values: the undirected run reads them
            if vals is np.int32:
                np.testing.assert_array_equal(g.sssp([n // 2], directed=0)[0],
                                              oracle.sssp(ro, ci, w, [n // 2], directed=0))
            else:
                x, _ = g.pagerank(mode="normalized", weighted=True, max_iter=5, tol=1e-30)
                assert np.abs(x - oracle.pr_normalized(ro, ci, w, 0.85, 0.0, 5)[0]).sum() <= L1_TOL


@pytest.mark.parametrize("shape", ["lattice", "path", "star", "pairs", "er1", "rmat", "isolated"])
@pytest.mark.parametrize("sym", [False, True])
def test_cc_forest(shape, sym):
    rng = np.random.default_rng(3)
    n = 5000
    if shape == "lattice":
        h = mg.gen_lattice(61, 83, 0.0, 1)
        n, ro, ci = h.n, h.row_offsets, h.col_idx
    elif shape == "rmat":
        h = mg.gen_rmat(13, 3, 4, symmetrize=True)
        n, ro, ci = h.n, h.row_offsets, h.col_idx
    else:
        src, dst = {"path": (np.arange(n - 1, 0, -1), np.arange(n - 2, -1, -1)),
                    "star": (np.full(n - 1, n - 1), np.arange(n - 1)),
                    "pairs": (np.arange(0, n, 2), np.arange(1, n, 2)),
                    "er1": (rng.integers(0, n, n), rng.integers(0, n, n)),
                    "isolated": (np.array([n - 1]), np.array([n - 1]))}[shape]
        if sym:
            src, dst = np.concatenate([src, dst]), np.concatenate([dst, src])
        ro, ci, _ = _csr(n, src, dst)
    with mg.Graph(ro, ci, symmetric=sym or shape in ("lattice", "rmat")) as g:
        for rounds in (0, 1, 3):
            g.set_tuning(cc_rounds=rounds)
            np.testing.assert_array_equal(g.cc()[0], oracle.cc(ro, ci))


@pytest.mark.parametrize("clique,alone,passes", [(12, 3, 2), (40, 5, 2), (3, 50, 3), (2, 1, 3)])
def test_cc_edges_inspected(clique, alone, passes):
    """One clique that the first forest joins, and vertices without edges: the edges read are the first four
    of a row and two per hooking pass (one pass more up to 4 edges per vertex)."""
    src, dst = np.nonzero(~np.eye(clique, dtype=bool))
    n = clique + alone
    ro, ci, _ = _csr(n, src, dst)
    with mg.Graph(ro, ci, symmetric=True) as g:
        for rounds in (0, 1, 4):
            g.set_tuning(cc_rounds=rounds)
            label, st = g.cc()
            np.testing.assert_array_equal(label, oracle.cc(ro, ci))
            reads = min(clique - 1, 4) + 2 * (rounds + passes - 1)
            assert st["edges_inspected"] == clique * reads


@pytest.mark.parametrize("directed", [0, 1])
@pytest.mark.parametrize("sym", [False, True])
def test_refcompat_sweep(directed, sym):
    n, ro, ci, _ = _in_degrees(BIN_DEGREES * 3, 8)
    if sym:
        src = np.repeat(np.arange(n), np.diff(ro))
        ro, ci, _ = _csr(n, np.concatenate([src, ci]), np.concatenate([ci, src]))
    with mg.Graph(ro, ci, symmetric=sym) as g:
        for cap in (0, 1, 3):
            x, st = g.pagerank(mode="refcompat", directed=directed, max_iter=cap)
            xr, it = oracle.pr_refcompat(ro, ci, directed, cap or 2**31 - 1)
            assert st["iterations"] == it
            assert np.abs(x - xr).max() <= 1e-5 * max(1.0, np.abs(xr).max())


@pytest.mark.parametrize("directed,sym", [(1, False), (0, False), (0, True)])
def test_refcompat_plain_sums(directed, sym):
    """compensated=False: plain FP32 sums, in the sweep's three forms."""
    n, ro, ci, _ = _in_degrees(BIN_DEGREES * 9, 8)
    if sym:
        src = np.repeat(np.arange(n), np.diff(ro))
        ro, ci, _ = _csr(n, np.concatenate([src, ci]), np.concatenate([ci, src]))
    with mg.Graph(ro, ci, symmetric=sym) as g:
        a, _ = g.pagerank(mode="refcompat", directed=directed, max_iter=1)
        b, _ = g.pagerank(mode="refcompat", directed=directed, max_iter=1, compensated=False)
    xr, _ = oracle.pr_refcompat(ro, ci, directed, 1)
    # ranks, terms and degrees in FP32: a few roundings; a lane adds at most 64 terms in a row
    assert np.abs(a / xr - 1).max() <= 8 * 2.0**-24
    assert np.abs(b / xr - 1).max() <= 72 * 2.0**-24
    assert (a != b).any()  # some of the 234 rows round otherwise


@pytest.mark.parametrize("kind", ["lattice", "hubs", "path", "one"])
@pytest.mark.parametrize("directed", [0, 1])
def test_near_far_rounds(kind, directed):
    if kind == "lattice":
        h = mg.gen_lattice(90, 70, 0.01, 2, weights="int", p0=1, p1=1000)
    elif kind == "hubs":  # mean degree 6, some vertices of thousands of edges: chunks
        h = mg.gen_rmat(15, 3, 6, symmetrize=True, weights="int", p0=1, p1=50)
    elif kind == "path":
        n = 700
        ro, ci, w = _csr(n, np.arange(n - 1), np.arange(1, n), np.arange(1, n, dtype=np.int32))
        h = mg.HostCsr(ro, ci, w)
    else:
        h = mg.HostCsr(np.array([0, 1], dtype=np.int32), np.array([0], dtype=np.int32), np.array([3], dtype=np.int32))
    with mg.Graph(h.row_offsets, h.col_idx, h.weights_i32) as g:
        ref = oracle.sssp(h.row_offsets, h.col_idx, h.weights_i32, [0], directed=directed)
        for delta in (0, 1, 37, 1 << 28):
            d, st = g.sssp([0], directed=directed, delta=delta)
            np.testing.assert_array_equal(d, ref)
            assert st["edges_traversed"] == int(np.diff(h.row_offsets)[ref != 2**31 - 1].sum())
        rows = g.sssp_batch([0, 0], directed=directed, delta=5)[0]
        np.testing.assert_array_equal(rows[1], ref)


@pytest.mark.parametrize("n,m", [(1, 0), (1, 3), (31, 60), (32, 64), (33, 40), (8193, 40000), (131072, 300000),
                                 (131073, 300000), (500, 1 << 20), (500, (1 << 20) + 1)])
@pytest.mark.parametrize("directed", [0, 1])
def test_small_bfs(n, m, directed):
    rng = np.random.default_rng(n + m)
    src, dst = rng.integers(0, n, m), rng.integers(0, n, m)
    src[: m // 3] = n // 2  # a hub: chunks
    ro, ci, _ = _csr(n, src, dst)
    deg = np.diff(ro)
    with mg.Graph(ro, ci) as g:
        for srcs in ([n // 2], [0, n - 1, 0], [int(v) for v in rng.integers(0, n, 11)]):
            ref = oracle.bfs(ro, ci, srcs, directed=directed)
            d, st = g.bfs(srcs, directed=directed)
            np.testing.assert_array_equal(d, ref)
            assert st["iterations"] == ref.max() + 1
            assert st["edges_traversed"] == int(deg[ref >= 0].sum())
            d, st = g.bfs(srcs, directed=directed, iter_num=1)
            np.testing.assert_array_equal(d, np.where(ref <= 1, ref, -1))
            assert st["edges_traversed"] == int(deg[(ref >= 0) & (ref <= 1)].sum())
        if n >= 33:
            with pytest.raises(mg.MapGraphError):
                g.bfs(list(range(33)), queue_sizing=2 / n)
            np.testing.assert_array_equal(g.bfs([0])[0], oracle.bfs(ro, ci, [0]))


def test_loop_modes_agree():
    """Launches ahead of the device (the default), the CUDA-graph loop and the host-driven one."""
    h = mg.gen_rmat(17, 16, 9, symmetrize=True, weights="int", p0=1, p1=255)
    modes = (True, "graph", False)
    with mg.Graph(h.row_offsets, h.col_idx, h.weights_i32, symmetric=True) as g:
        runs = [(g.bfs([5], use_graph=m), g.sssp([5], use_graph=m), g.sssp([5], delta=20, use_graph=m),
                 g.bfs_batch([5, 9, 70000], use_graph=m), g.sssp_batch([5, 9], use_graph=m),
                 g.bfs([5], iter_num=2, use_graph=m)) for m in modes]
        for other in runs[1:]:
            for (a, sa), (b, sb) in zip(runs[0], other):
                np.testing.assert_array_equal(a, b)
                assert sa["edges_traversed"] == sb["edges_traversed"]
        for kw in (dict(mode="refcompat"), dict(mode="normalized"), dict(mode="normalized", gather="segmented"),
                   dict(mode="normalized", gather="tma"), dict(mode="normalized", max_iter=1)):
            res = [g.pagerank(use_graph=m, **kw) for m in modes]
            assert len({r[1]["iterations"] for r in res}) == 1
            for r in res[1:]:
                assert np.abs(r[0] - res[0][0]).sum() <= 1e-9 * max(1.0, float(np.abs(res[0][0]).sum()))


@pytest.mark.parametrize("n,m", [(300, 100), (300, 1200), (300, 1201), (20000, 10000), (20000, 20000), (20000, 60000),
                                 (700000, 700000)])
@pytest.mark.parametrize("sym", [False, True])
def test_cc_sparse(n, m, sym):
    """Trees and small cycles, on both sides of 4 edges per vertex."""
    rng = np.random.default_rng(m)
    src, dst = rng.integers(0, n, m), rng.integers(0, n, m)
    if sym:
        src, dst = np.concatenate([src, dst[: m // 2]])[:m], np.concatenate([dst, src[: m // 2]])[:m]
        src, dst = np.concatenate([src[: m // 2], dst[: m // 2]]), np.concatenate([dst[: m // 2], src[: m // 2]])
    ro, ci, _ = _csr(n, src, dst)
    with mg.Graph(ro, ci, symmetric=sym) as g:
        np.testing.assert_array_equal(g.cc()[0], oracle.cc(ro, ci))


@pytest.mark.parametrize("depth", [1, 30, 31, 32, 33, 34, 70])
@pytest.mark.parametrize("k", [1, 9, 33, 64, 65])
@pytest.mark.parametrize("directed", [0, 1])
def test_bfs_batch_levels(depth, k, directed):
    """The level at which the depth rows are written, with sources that are done by then and some beyond it."""
    rng = np.random.default_rng(depth)
    n = depth + 1 + 90
    src = np.concatenate([np.arange(depth), rng.integers(depth + 1, n, 150)])
    dst = np.concatenate([np.arange(1, depth + 1), rng.integers(depth + 1, n, 150)])
    ro, ci, w = _csr(n, src, dst, np.ones(src.size, dtype=np.int32))
    srcs = [0] + [int(v) for v in rng.integers(0, n, k - 1)]
    ref = np.stack([oracle.bfs(ro, ci, [s], directed=directed) for s in srcs])
    with mg.Graph(ro, ci) as g:
        for direction in ("auto", "push", "pull"):
            d, st = g.bfs_batch(srcs, directed=directed, direction=direction)
            np.testing.assert_array_equal(d, ref)
            assert st["edges_traversed"] == int((np.diff(ro)[None] * (ref >= 0)).sum())
        for cap in (1, 31, 32, 33):
            d, _ = g.bfs_batch(srcs, directed=directed, iter_num=cap)
            np.testing.assert_array_equal(d, np.where(ref <= cap, ref, -1))


@pytest.mark.parametrize("wide,deg", [(37, 9000), (5000, 40), (5000, 200), (40000, 20)])
def test_bfs_skewed_frontier(wide, deg):
    """A sparse graph whose second level holds most of the edges: few vertices per warp,
    hubs beyond the deferral list's 4096, and full tiles."""
    rng = np.random.default_rng(wide)
    n = max(1 << 18, wide * deg // 6)
    src = np.concatenate([np.zeros(wide, np.int64), np.repeat(np.arange(1, wide + 1), deg)])
    dst = np.concatenate([np.arange(1, wide + 1), rng.integers(0, n, wide * deg)])
    ro, ci, _ = _csr(n, src, dst)
    ref = oracle.bfs(ro, ci, [0])
    with mg.Graph(ro, ci) as g:
        for mode in (True, False):
            d, st = g.bfs([0], use_graph=mode)
            np.testing.assert_array_equal(d, ref)
            assert st["edges_traversed"] == int(np.diff(ro)[ref >= 0].sum())
        np.testing.assert_array_equal(g.bfs([0], direction="push")[0], ref)
        np.testing.assert_array_equal(g.bfs_batch([0, 1], direction="push")[0][0], ref)


@pytest.mark.parametrize("n", [33, 8191, 140001])
def test_bottom_up_degrees(n):
    """In-degrees at the ends of the shares of a bottom-up level: one lane, four, the warp; with and
    without a parent in the last edge."""
    rng = np.random.default_rng(n)
    degs = np.array([0, 1, 7, 8, 9, 10, 263, 264, 265, 266, 511, 512, 4097])
    rows = np.arange(min(n - 2, 16 * degs.size)) + 1
    indeg = degs[rng.integers(0, degs.size, rows.size)]
    dst = np.repeat(rows, indeg)
    src = np.full(dst.size, n - 1)  # a vertex nothing reaches
    last = np.cumsum(indeg)[(indeg > 0) & (rng.random(rows.size) < 0.7)] - 1
    src[last] = rng.integers(0, rows.size, last.size)  # its parent, in the row's last edge
    pos = np.arange(dst.size)
    order = np.lexsort((pos, src))
    ro = np.searchsorted(src[order], np.arange(n + 1)).astype(np.int32)
    ci = dst[order].astype(np.int32)
    with mg.Graph(ro, ci) as g:
        for srcs in ([0], [0, 5, n - 2], [n - 1]):
            ref = oracle.bfs(ro, ci, srcs)
            for kw in (dict(direction="pull"), dict(direction="pull", use_graph=False), dict()):
                np.testing.assert_array_equal(g.bfs(srcs, **kw)[0], ref)
        np.testing.assert_array_equal(g.bfs_batch([0, 5], direction="pull")[0][1], oracle.bfs(ro, ci, [5]))


@pytest.mark.parametrize("m", [(1 << 22) - 1, 1 << 22, (1 << 22) + 1])
def test_plain_sssp_one_launch_limit(m):
    rng = np.random.default_rng(m & 7)
    n = 300001
    src, dst = rng.integers(0, n, m), rng.integers(0, n, m)
    ro, ci, w = _csr(n, src, dst, rng.integers(0, 100, m).astype(np.int32))
    ref = oracle.sssp(ro, ci, w, [3, 70000])
    with mg.Graph(ro, ci, w) as g:
        for kw in (dict(), dict(use_graph=False), dict(use_graph="graph"), dict(delta=64)):
            np.testing.assert_array_equal(g.sssp([3, 70000], **kw)[0], ref)


@pytest.mark.parametrize("shape", ["cut", "sinks", "cycle2"])
@pytest.mark.parametrize("teleport", [False, True])
def test_adjoint_settles(shape, teleport):
    """The adjoint solve where the constant is not the slowest part of its error, or not the only one: closed
    parts, rows without edges, a slow alternating mode, each with a loss on five vertices, whose tolerance
    FP32 rounding hides."""
    rng = np.random.default_rng(5)
    n = 1500
    if shape == "cut":  # two halves without an edge between them
        src = rng.integers(0, n // 2, 9000)
        dst = rng.integers(0, n // 2, 9000)
        src[::2] += n // 2
        dst[::2] += n // 2
    elif shape == "sinks":  # a third of the vertices without out-edges
        src, dst = rng.integers(0, 2 * n // 3, 6000), rng.integers(0, n, 6000)
    else:  # bipartite
        src, dst = rng.integers(0, n // 2, 4000), rng.integers(n // 2, n, 4000)
        src, dst = np.concatenate([src, dst]), np.concatenate([dst, src])
    ro, ci, w = _csr(n, src, dst, rng.lognormal(0, 1, src.size).astype(np.float32))
    t = None
    if teleport:
        t = np.zeros(n)
        t[rng.integers(0, n, 7)] = 1.0
        t /= t.sum()
    dl = np.zeros(n)
    dl[rng.integers(0, n, 5)] = rng.standard_normal(5) + 3
    x, _, _ = oracle.pr_normalized(ro, ci, w, 0.85, 1e-15, 5000, t)
    rw, rt, _, _ = oracle.pr_adjoint(ro, ci, w, x, dl, teleport=t)
    with mg.Graph(ro, ci, w) as g:
        for gather in ("binned", "cached"):
            gw, gt, st = g.pagerank_backward(x.astype(np.float32), dl.astype(np.float32),
                                             teleport=None if t is None else t.astype(np.float32), weighted=True,
                                             tol=1e-8, max_iter=400, gather=gather)
            assert st["iterations"] < 400
            # 1e-8 relative over 1 - alpha, with FP32 ranks, iterates and results
            assert np.linalg.norm(gt - rt) <= 2e-6 * np.linalg.norm(rt)
            assert np.linalg.norm(gw - rw) <= 2e-6 * np.linalg.norm(rw) + 1e-12


@pytest.mark.parametrize("nvec", [2, 32, 33, 70])
def test_batched_ranks_sparse_rows(nvec):
    """Rows with and without in-edges, with and without teleport entries, in every pairing."""
    rng = np.random.default_rng(nvec)
    n, m = 3001, 9000
    src, dst = rng.integers(0, n, m), rng.integers(0, n // 3, m)  # two thirds of the rows have no in-edge
    ro, ci, w = _csr(n, src, dst, rng.lognormal(0, 1, m).astype(np.float32))
    tele = np.zeros((nvec, n), dtype=np.float32)
    for k in range(nvec):
        s = rng.integers(0, n, 1 + k % 5)
        np.add.at(tele[k], s, np.float32(1.0 / s.size))
    tele[0] = 1.0 / n
    with mg.Graph(ro, ci, w) as g:
        xs, st = g.pagerank(teleport=tele, nvec=nvec, mode="normalized", weighted=True)
        ys, _ = g.pagerank(teleport=tele, nvec=nvec, mode="normalized", weighted=True)  # over the first run's state
        for k in range(nvec):
            xr, _, _ = oracle.pr_normalized(ro, ci, w, 0.85, 0.0, st["iterations"], tele[k].astype(np.float64))
            assert np.abs(xs[k] - xr).sum() <= L1_TOL
            assert np.abs(ys[k] - xr).sum() <= L1_TOL
        tele[1, n - 1] = np.inf
        zs, st = g.pagerank(teleport=tele, nvec=nvec, mode="normalized", weighted=True, max_iter=5)
        assert np.isfinite(zs[0]).all() and not np.isfinite(zs[1]).all()


def _capacities(run, ref, widths, n):
    """Runs with queues of just the widest frontier, and of one less than every frontier."""
    def sized(cap):
        return run(queue_sizing=(cap - 0.5) / n)  # rounded up

    for _ in range(20):
        np.testing.assert_array_equal(sized(int(widths.max())), ref)
        for cap in sorted({int(w) - 1 for w in widths if w > 1}):
            with pytest.raises(mg.MapGraphError) as e:
                sized(cap)
            assert e.value.status == L.MG_ERR_QUEUE_OVERFLOW
        np.testing.assert_array_equal(run(), ref)


@pytest.mark.parametrize("directed", [0, 1])
def test_small_bfs_queue_capacity(directed):
    """The run ends in every CTA alike, at any level, and the next one is right."""
    rng = np.random.default_rng(2)
    n, m = 20000, 50000
    ro, ci, _ = _csr(n, rng.integers(0, n, m), rng.integers(0, n, m))
    ref = oracle.bfs(ro, ci, [0], directed=directed)
    with mg.Graph(ro, ci) as g:
        _capacities(lambda **kw: g.bfs([0], directed=directed, **kw)[0], ref, np.bincount(ref[ref >= 0]), n)


def test_persistent_bfs_queue_capacity():
    h = mg.gen_lattice(400, 500, 0.001, 4)  # past the cluster BFS; every level within the one-launch limits
    ref = oracle.bfs(h.row_offsets, h.col_idx, [0])
    widths = np.bincount(ref)
    with mg.Graph(h.row_offsets, h.col_idx, symmetric=True) as g:
        _capacities(lambda **kw: g.bfs([0], **kw)[0], ref, widths[np.argsort(widths)[-3:]], h.n)


@pytest.mark.parametrize("kind", ["near_far", "plain", "per_round", "batch"])
def test_sssp_queue_capacity(kind):
    """Queues too small for a round: in the one-launch rounds, near-far and plain (near frontier, far pile),
    in the per-round kernels, and with several instances per run. Each is followed by a correct run."""
    if kind == "plain":
        h = mg.gen_rmat(14, 16, 6, symmetrize=True, weights="int", p0=1, p1=50)
    else:
        h = mg.gen_lattice(300, 200, 0.001, 4, weights="int", p0=1, p1=1000)
    srcs = [0, 7] if kind == "batch" else [0]
    kw = dict(use_graph="graph") if kind == "per_round" else {}
    if kind == "batch":
        kw["delta"] = 500
    ref = np.stack([oracle.sssp(h.row_offsets, h.col_idx, h.weights_i32, [s]) for s in srcs])
    with mg.Graph(h.row_offsets, h.col_idx, h.weights_i32, symmetric=True) as g:
        for _ in range(10):
            for size in (0.5 / h.n, 3.5 / h.n, 20.5 / h.n, 0.002):
                with pytest.raises(mg.MapGraphError) as e:
                    if kind == "batch":
                        g.sssp_batch(srcs, queue_sizing=size, **kw)
                    else:
                        g.sssp(srcs, queue_sizing=size, **kw)
                assert e.value.status == L.MG_ERR_QUEUE_OVERFLOW
            d = g.sssp_batch(srcs, **kw)[0] if kind == "batch" else g.sssp(srcs, **kw)[0][None]
            np.testing.assert_array_equal(d, ref)
