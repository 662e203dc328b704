"""GPU tests of the dense-vector SpMV and PageRank against float64 restatements
(tolerances in each test: float32 accumulation only). PageRank stops at an L1 change of
1e-6, above what float32 ranks resolve (a tol near 1e-9 would run to max_iter)."""
import numpy as np
import pytest

import apspie_b200 as ap
import oracle

pytestmark = pytest.mark.gpu


def _t(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()


@pytest.mark.parametrize("shape,dens", [((1, 1), 1.0), ((300, 500), 0.01), ((4000, 4000), 0.002),
                                        ((2000, 3000), 0.05)])
def test_spmv_matches_float64(ctx, shape, dens):
    import scipy.sparse as sp

    m, n = shape
    A = sp.random(m, n, density=dens, format="csr", dtype=np.float32, random_state=np.random.RandomState(m))
    g = ap.HostGraph(m, n, A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data.astype(np.float32))
    x = np.random.default_rng(1).uniform(-1, 1, n).astype(np.float32)
    y0 = np.random.default_rng(2).uniform(-1, 1, m).astype(np.float32)
    y = _t(y0)
    ctx.spmv_into(ap.DeviceGraph(g), _t(x), y, 2.0, 0.5)
    ref = 2.0 * oracle.spmv(A.indptr, A.indices, A.data, x) + 0.5 * y0.astype(np.float64)
    bound = 2.0 * oracle.spmv(A.indptr, A.indices, np.abs(A.data), np.abs(x)) + 0.5 * np.abs(y0)
    assert np.all(np.abs(y.cpu().numpy() - ref) <= 1e-5 * bound + 1e-6)


def test_spmv_pattern_counts_degrees(ctx):
    g = ap.gen_rmat(12, 16, 1, 3, weights=False)
    y = _t(np.zeros(g.m))
    ctx.spmv_into(ap.DeviceGraph(g), _t(np.ones(g.m)), y)
    np.testing.assert_array_equal(y.cpu().numpy(), np.diff(g.row_ptr).astype(np.float32))


@pytest.mark.parametrize("key", ["test_pr_d", "test_pr_u", "test_cc_d", "chesapeake_u"])
def test_pagerank_fixtures(ctx, golden, key):
    rp, ci = golden[key + "_row_ptr"], golden[key + "_col_ind"]
    m = rp.shape[0] - 1
    g = ap.HostGraph(m, m, rp, ci, None, key.endswith("_u"))
    r, it = ctx.pagerank(ap.DeviceGraph(g), 0.85, 1e-6, 200)
    ref, rit = oracle.pagerank(rp, ci, 0.85, 1e-6, 200)
    np.testing.assert_allclose(r.cpu().numpy(), ref, rtol=1e-4, atol=1e-7)
    assert abs(it - rit) <= 2
    assert abs(float(r.sum().item()) - 1.0) < 1e-4


@pytest.mark.parametrize("symmetric", [True, False])
def test_pagerank_rmat(ctx, symmetric):
    g = ap.gen_rmat(14, 16, 1, 3, weights=False)
    if not symmetric:
        keep = np.repeat(np.arange(g.m), np.diff(g.row_ptr)) < g.col_ind  # upper triangle: a DAG
        rows = np.repeat(np.arange(g.m), np.diff(g.row_ptr))[keep]
        rp = np.zeros(g.m + 1, dtype=np.int32)
        rp[1:] = np.cumsum(np.bincount(rows, minlength=g.m))
        g = ap.HostGraph(g.m, g.m, rp, g.col_ind[keep].astype(np.int32), None, False)
    r, it = ctx.pagerank(ap.DeviceGraph(g), 0.85, 1e-6, 100)
    ref, _ = oracle.pagerank(g.row_ptr, g.col_ind, 0.85, 1e-6, 100)
    np.testing.assert_allclose(r.cpu().numpy(), ref, rtol=2e-4, atol=1e-8)


@pytest.mark.parametrize("n,hub", [(1, 0), (2, 3), (9000, 2047), (9000, 2048), (9000, 8999), (70001, 30000)])
@pytest.mark.parametrize("symmetric", [True, False])
def test_pagerank_rows_across_entry_chunks(ctx, n, hub, symmetric):
    """In-edge rows that end at, cross and cover whole 2,048-entry chunks, between runs of
    vertices without in-edges and without out-edges. Bound: a float32 sum of d positive terms
    is off by at most d * 2^-24 relative, and an iteration damps earlier errors by 0.85, so the
    ranks are off by at most (2 + the longest partial sum) * 2^-24 / 0.15; sums inside a chunk
    are at most 8 + 5 + 8 terms deep, a row's chunks at most 15."""
    import torch

    rng = np.random.default_rng(n + hub)
    src = np.concatenate((rng.choice(n, min(hub, n), replace=False), rng.integers(0, n, n // 3)))
    dst = np.concatenate((np.full(min(hub, n), n // 2), rng.integers(n // 4, max(n // 4 + 1, n // 2), n // 3)))
    if symmetric:
        src, dst = np.concatenate((src, dst)), np.concatenate((dst, src))
    key = np.unique(src.astype(np.int64) * n + dst)
    rp = np.concatenate(([0], np.cumsum(np.bincount(key // n, minlength=n)))).astype(np.int32)
    ci = (key % n).astype(np.int32)
    # an odd number of entries in front makes col_ind's address no multiple of 16
    cols = torch.from_numpy(np.concatenate((np.zeros(3, dtype=np.int32), ci))).cuda()[3:]
    g = ap.DeviceGraph.from_tensors(n, n, torch.from_numpy(rp).cuda(), cols, symmetric=symmetric)
    for iters in (1, 7):  # 7: no multiple of the iterations enqueued at a time
        r, it = ctx.pagerank(g, 0.85, 0.0, iters)
        ref, _ = oracle.pagerank(rp, ci, 0.85, 0.0, iters)
        assert it == iters
        np.testing.assert_allclose(r.cpu().numpy(), ref, rtol=(2 + 21 + 15) * 2.0 ** -24 / 0.15, atol=0)
        again, _ = ctx.pagerank(g, 0.85, 0.0, iters)
        assert torch.allclose(r, again, rtol=2.0 ** -23, atol=0)  # the double sums' order may turn a last bit
