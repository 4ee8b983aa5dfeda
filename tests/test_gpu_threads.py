"""Several threads, each with its own graph (and so its own stream, control block, mailbox
and workspaces), running every program at the same time: one-launch kernels that fill the
GPU, launches ahead of the device, CUDA-graph loops and the batched programs side by side."""
import threading

import numpy as np
import pytest

import oracle
import mirrorofmapgraph_b200 as mg

pytestmark = pytest.mark.gpu


def _work(seed, rounds, errors):
    try:
        lat = mg.gen_lattice(150 + 3 * seed, 140, 0.001, seed, weights="int", p0=1, p1=1000)
        rm = mg.gen_rmat(13, 16, seed, symmetrize=True, weights="int", p0=1, p1=255)
        big = mg.gen_rmat(17, 8, seed, symmetrize=False)
        srcs = [1, 5, 9 + seed]
        ref_lat = oracle.sssp(lat.row_offsets, lat.col_idx, lat.weights_i32, [seed])
        ref_rm = oracle.sssp(rm.row_offsets, rm.col_idx, rm.weights_i32, [seed])
        ref_bfs = [oracle.bfs(big.row_offsets, big.col_idx, [s]) for s in srcs]
        ref_small = oracle.bfs(rm.row_offsets, rm.col_idx, [seed])
        ref_pr = oracle.pr_normalized(big.row_offsets, big.col_idx, None, 0.85, 0.0, 12)[0]
        ref_cc = oracle.cc(rm.row_offsets, rm.col_idx)
        ref_rc = oracle.pr_refcompat(big.row_offsets, big.col_idx, 1, 5)[0]
        dl = np.random.default_rng(seed).standard_normal(big.n).astype(np.float32)
        ref_gt = oracle.pr_adjoint(big.row_offsets, big.col_idx, None, ref_pr, dl.astype(np.float64))[1]
        with mg.Graph(lat.row_offsets, lat.col_idx, lat.weights_i32, symmetric=True) as g1, \
                mg.Graph(rm.row_offsets, rm.col_idx, rm.weights_i32, symmetric=True) as g2, \
                mg.Graph(big.row_offsets, big.col_idx) as g3:
            for _ in range(rounds):
                np.testing.assert_array_equal(g1.sssp([seed])[0], ref_lat)
                np.testing.assert_array_equal(g2.sssp([seed])[0], ref_rm)
                np.testing.assert_array_equal(g2.bfs([seed])[0], ref_small)
                np.testing.assert_array_equal(g3.bfs([srcs[0]])[0], ref_bfs[0])
                np.testing.assert_array_equal(g3.bfs_batch(srcs)[0], np.stack(ref_bfs))
                np.testing.assert_array_equal(g2.cc()[0], ref_cc)
                for gather in ("binned", "cached", "segmented"):
                    x = g3.pagerank(mode="normalized", gather=gather, max_iter=12, tol=1e-30)[0]
                    assert np.abs(x - ref_pr).sum() <= 1e-6  # FP32 sums against FP64
                x = g3.pagerank(mode="refcompat", max_iter=5)[0]
                assert np.abs(x / ref_rc - 1).max() <= 1e-5
                gt = g3.pagerank_backward(ref_pr.astype(np.float32), dl, max_iter=400)[1]
                assert np.linalg.norm(gt - ref_gt) <= 1e-5 * np.linalg.norm(ref_gt)
                rows = g1.sssp_batch([seed, 3])[0]
                np.testing.assert_array_equal(rows[0], ref_lat)
                with mg.Graph(big.row_offsets, big.col_idx) as once:
                    x = once.pagerank(mode="normalized", max_iter=12, tol=1e-30)[0]
                    assert np.abs(x - ref_pr).sum() <= 1e-6
    except BaseException as e:  # noqa: BLE001 - reported by the test
        errors.append(e)


@pytest.mark.parametrize("threads", [2, 4])
def test_programs_on_several_threads(threads):
    errors = []
    ts = [threading.Thread(target=_work, args=(k, 6, errors)) for k in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    if errors:
        raise errors[0]
