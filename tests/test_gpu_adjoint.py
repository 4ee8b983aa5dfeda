"""PageRank adjoint on the GPU (mg_pagerank_backward) against the FP64 CPU adjoint
and central finite differences of the FP64 forward solve.

Tolerance: gradient errors are measured norm-wise over the checked entries,
||g_gpu - g_ref|| / ||g_ref|| <= 1e-4."""
import concurrent.futures as cf

import numpy as np
import pytest

import oracle
import mirrorofmapgraph_b200 as mg

pytestmark = pytest.mark.gpu

REL = 1e-4


def _problem(scale, seed, weighted=True, teleport=False):
    h = mg.gen_rmat(scale, 16, seed, symmetrize=False, weights="lognormal" if weighted else None, p0=0, p1=1)
    rng = np.random.default_rng(seed)
    w = rng.standard_normal(h.n)
    t = None
    if teleport:
        t = rng.random(h.n)
        t /= t.sum()
    a = h.weights_f32 if weighted else None
    x, _, _ = oracle.pr_normalized(h.row_offsets, h.col_idx, a, 0.85, 1e-15, 5000, t)
    return h, a, w, t, x


def _rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


@pytest.mark.parametrize("weighted", [True, False])
@pytest.mark.parametrize("teleport", [False, True])
def test_adjoint_matches_fp64_adjoint(weighted, teleport):
    h, a, w, t, x = _problem(12, 5 + weighted + 2 * teleport, weighted, teleport)
    ga, gt, lam, _ = oracle.pr_adjoint(h.row_offsets, h.col_idx, a, x, w, teleport=t)
    with mg.Graph(h.row_offsets, h.col_idx, a) as g:
        gw, gtt, st = g.pagerank_backward(x.astype(np.float32), w.astype(np.float32),
                                          teleport=None if t is None else t.astype(np.float32),
                                          weighted=weighted, tol=1e-9, max_iter=400)
        assert _rel(gw, ga) <= REL and _rel(gtt, gt) <= REL
        for gather in ("tma",):
            gw2, gt2, _ = g.pagerank_backward(x.astype(np.float32), w.astype(np.float32),
                                              teleport=None if t is None else t.astype(np.float32),
                                              weighted=weighted, tol=1e-9, max_iter=400, gather=gather)
            assert _rel(gw2, ga) <= REL and _rel(gt2, gt) <= REL


def test_adjoint_finite_differences_1000_edges():
    """Forward and backward both on the GPU; central differences of L = w . x at
    1,000 seeded edges with h = 1e-3 |a_uv| in FP64 forward solves."""
    h, a, w, t, x64 = _problem(12, 17, True, False)
    with mg.Graph(h.row_offsets, h.col_idx, a) as g:
        x, st = g.pagerank(mode="normalized", weighted=True, tol=1e-9, max_iter=400)
        gw, gt, _ = g.pagerank_backward(x, w.astype(np.float32), weighted=True, tol=1e-9, max_iter=400)
    rng = np.random.default_rng(99)
    edges = rng.choice(h.m, size=1000, replace=False)
    a64 = a.astype(np.float64)

    def fd(e):
        step = 1e-3 * a64[e]
        ap, am = a64.copy(), a64.copy()
        ap[e] += step
        am[e] -= step
        ap32, am32 = ap.astype(np.float32), am.astype(np.float32)
        lp = oracle.pr_loss(h.row_offsets, h.col_idx, ap32, w, x64, tol=1e-15, max_iter=5000)
        lm = oracle.pr_loss(h.row_offsets, h.col_idx, am32, w, x64, tol=1e-15, max_iter=5000)
        return (lp - lm) / (float(ap32[e]) - float(am32[e]))

    with cf.ThreadPoolExecutor(max_workers=16) as ex:
        ref = np.array(list(ex.map(fd, edges)))
    assert _rel(gw[edges], ref) <= REL


def test_adjoint_device_arrays_and_determinism():
    torch = pytest.importorskip("torch")
    h, a, w, t, x = _problem(11, 3, True, False)
    with mg.Graph(h.row_offsets, h.col_idx, a) as g:
        xd = torch.from_numpy(x.astype(np.float32)).cuda()
        wd = torch.from_numpy(w.astype(np.float32)).cuda()
        ow = torch.empty(h.m, dtype=torch.float32, device="cuda")
        ot = torch.empty(h.n, dtype=torch.float32, device="cuda")
        g.pagerank_backward(xd, wd, weighted=True, out_weights=ow, out_teleport=ot, tol=1e-9, max_iter=400)
        gw, gt, _ = g.pagerank_backward(x.astype(np.float32), w.astype(np.float32), weighted=True, tol=1e-9,
                                        max_iter=400)
        assert np.abs(ow.cpu().numpy() - gw).max() <= 1e-6 * max(1.0, np.abs(gw).max())
        assert np.abs(ot.cpu().numpy() - gt).max() <= 1e-6 * max(1.0, np.abs(gt).max())


def test_adjoint_rejects_refcompat_mode():
    h, a, w, t, x = _problem(8, 1, True, False)
    with mg.Graph(h.row_offsets, h.col_idx, a) as g:
        with pytest.raises(mg.MapGraphError):
            g.pagerank_backward(x.astype(np.float32), w.astype(np.float32), mode="refcompat")


# ---------------------------------------------------------------------------
# The solve itself, against a dense FP64 solve and the plain FP32 iteration.
def _csr(n, src, dst, w):
    order = np.argsort(src, kind="stable")
    ro = np.searchsorted(src[order], np.arange(n + 1)).astype(np.int32)
    return ro, dst[order].astype(np.int32), w[order].astype(np.float32)


def _dense(ro, ci, w, t):
    """M of lambda = dl + alpha M lambda."""
    n = ro.size - 1
    a = np.zeros((n, n))
    np.add.at(a, (np.repeat(np.arange(n), np.diff(ro)), ci), w.astype(np.float64))
    s = a.sum(1, keepdims=True)
    return np.where(s > 0, a / np.where(s > 0, s, 1), t[None, :])


def _plain(mat, dl, alpha, tol, max_iter):
    """The plain iteration on FP32 iterates until the change is below tol |dl|_1 in the L1 norm and 0.6 tol
    |dl|_2 in the 2-norm: (lambda, iterations)."""
    v, wn, w2 = dl.astype(np.float32), np.abs(dl).sum(), np.linalg.norm(dl)
    for k in range(1, max_iter + 1):
        new = (dl + alpha * (mat @ v.astype(np.float64))).astype(np.float32)
        change = new.astype(np.float64) - v
        v = new
        if np.abs(change).sum() < tol * wn and np.linalg.norm(change) < 0.6 * tol * w2:
            break
    return v.astype(np.float64), k


def _check_solve(ro, ci, w, t, dl, alpha, tol=1e-7, max_iter=400, gathers=("binned",)):
    n = dl.size
    t = np.full(n, 1.0 / n) if t is None else t.astype(np.float32).astype(np.float64)
    dl = dl.astype(np.float32).astype(np.float64)
    mat = _dense(ro, ci, w, t)
    lam = np.linalg.solve(np.eye(n) - alpha * mat, dl)
    plain, iters = _plain(mat, dl, alpha, tol, max_iter)
    ref_err = np.linalg.norm(plain - lam) / np.linalg.norm(lam)
    # ranks that leave no mass on dangling rows: dL/dt = (1 - alpha) lambda
    x = np.where(np.diff(ro) > 0, 1.0 / n, 0.0).astype(np.float32)
    # the changes at which the other two rules stop, over 1 - alpha (taken twice: M is no
    # contraction in the 2-norm), and the FP32 result
    bound = 2 * ref_err + alpha / (1 - alpha) * 2 * (2.0**-24 + 0.6 * tol * np.linalg.norm(dl) / np.linalg.norm(lam)) + 6e-8
    with mg.Graph(ro, ci, w) as g:
        for gather in gathers:
            _, gt, st = g.pagerank_backward(x, dl.astype(np.float32), teleport=t.astype(np.float32), alpha=alpha,
                                            weighted=True, tol=tol, max_iter=max_iter, gather=gather)
            err = np.linalg.norm(gt / (1 - alpha) - lam) / np.linalg.norm(lam)
            assert err <= bound, (err, ref_err, st["iterations"], iters)
            # the iteration in which FP32 iterates settle depends on the rounding of their sums
            assert st["iterations"] <= min(1.1 * iters + 2, max_iter), (st["iterations"], iters)


_SUMS = [0.0, 0.5, 0.8, 0.9, 0.999, 1.0, 1.0 + 1e-5]


@pytest.mark.parametrize("tau,dangling", [(t, d) for t in _SUMS for d in (False, True)] +
                         [(1.3, False), (2.0, False), (500.0, False)])
def test_adjoint_teleport_of_any_sum(tau, dangling):
    """The linear system has no need of a teleport vector that sums to 1, and gradient steps on one
    leave that sum; with rows without edges a larger sum may leave it without a solution that the
    iteration reaches."""
    rng = np.random.default_rng(11)
    n = 500
    src, dst = rng.integers(0, n - n // 10 if dangling else n, 8000), rng.integers(0, n, 8000)
    if not dangling:
        src[:n] = np.arange(n)
    ro, ci, w = _csr(n, src, dst, rng.lognormal(0, 1, src.size))
    t = rng.random(n)
    if tau == 500.0:
        t = np.ones(n)
    elif tau == 0.0:
        t -= t.mean()
        t /= np.abs(t).sum()
    else:
        t *= tau / t.sum()
    _check_solve(ro, ci, w, t, rng.standard_normal(n), 0.85, gathers=("binned", "tma"))


@pytest.mark.parametrize("alpha", [0.5, 0.85, 0.95, 0.99])
@pytest.mark.parametrize("shape", ["rmat", "rmat_sym", "star", "two_sided", "sinks", "cut"])
def test_adjoint_loss_on_few_vertices(shape, alpha):
    """|lambda| far above |dL/dx|: FP32 rounding hides the tolerance. Never more iterations than the
    plain iteration."""
    rng = np.random.default_rng(3)
    n = 900
    if shape.startswith("rmat"):
        h = mg.gen_rmat(10, 8, 4, symmetrize=shape == "rmat_sym")
        n, src, dst = h.n, np.repeat(np.arange(h.n), np.diff(h.row_offsets)), h.col_idx.astype(np.int64)
    elif shape == "star":
        src, dst = np.zeros(n - 1, dtype=np.int64), np.arange(1, n)
    elif shape == "two_sided":  # 20 hubs against the others, edges both ways
        src, dst = rng.integers(0, 20, 4000), rng.integers(20, n, 4000)
    elif shape == "sinks":
        src, dst = rng.integers(0, 2 * n // 3, 5000), rng.integers(0, n, 5000)
    else:
        src, dst = rng.integers(0, n // 2, 6000), rng.integers(0, n // 2, 6000)
        src[::2] += n // 2
        dst[::2] += n // 2
    if shape in ("star", "two_sided"):
        src, dst = np.concatenate([src, dst]), np.concatenate([dst, src])
    ro, ci, w = _csr(n, src, dst, rng.lognormal(0, 1, src.size))
    hub = int(np.bincount(dst, minlength=n).argmax())
    few = np.zeros(n)
    few[rng.integers(0, n, 5)] = 3 + rng.standard_normal(5)
    for dl in (np.eye(1, n, hub)[0], few, rng.standard_normal(n)):
        for t in (None, np.eye(1, n, 7)[0]):
            _check_solve(ro, ci, w, t, dl, alpha, max_iter=2500)
