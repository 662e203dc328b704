"""GPU tests of device graph construction: COO -> CSR with the generator's symmetrise /
dedup rules (identical to the host R-MAT CSR), plain COO -> CSR against a numpy
restatement, and CSR transpose against scipy."""
import numpy as np
import pytest

import apspie_b200 as ap

pytestmark = pytest.mark.gpu

SYM, DROP, DEDUP = ap.BUILD_SYMMETRIZE, ap.BUILD_DROP_SELF_LOOPS, ap.BUILD_DEDUP


def _dev(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("scale", [10, 14, 17])
def test_rmat_edge_list_builds_the_host_generator_csr(ctx, scale):
    src, dst, w = ap.gen_rmat_coo(scale, 16, 1, 3)
    g = ap.gen_rmat(scale, 16, 1, 3)
    C = ctx.build_csr(g.m, _dev(src), _dev(dst), _dev(w), SYM | DROP | DEDUP)
    rp, ci, val = C.to_numpy()
    np.testing.assert_array_equal(rp, g.row_ptr)
    np.testing.assert_array_equal(ci, g.col_ind)
    np.testing.assert_array_equal(val, g.val)


def _ref_build(m, src, dst, val, flags):
    a, b = src.astype(np.int64), dst.astype(np.int64)
    order_in = np.arange(a.shape[0])
    if flags & SYM:
        a, b = np.minimum(a, b), np.maximum(a, b)
    keep = np.ones(a.shape[0], dtype=bool)
    if flags & DROP:
        keep &= a != b
    a, b, val, order_in = a[keep], b[keep], val[keep], order_in[keep]
    o = np.lexsort((order_in, b, a))
    a, b, val, order_in = a[o], b[o], val[o], order_in[o]
    if flags & DEDUP and a.shape[0]:
        first = np.concatenate(([True], (a[1:] != a[:-1]) | (b[1:] != b[:-1])))
        a, b, val, order_in = a[first], b[first], val[first], order_in[first]
    if flags & SYM:
        rows = np.concatenate((b, a))
        cols = np.concatenate((a, b))
        val = np.concatenate((val, val))
        tie = np.concatenate((order_in, order_in))
        o = np.lexsort((tie, cols, rows))
        rows, cols, val = rows[o], cols[o], val[o]
    else:
        rows, cols = a, b
    rp = np.zeros(m + 1, dtype=np.int64)
    rp[1:] = np.cumsum(np.bincount(rows, minlength=m))
    return rp.astype(np.int32), cols.astype(np.int32), val


@pytest.mark.parametrize("flags", [0, DROP, DEDUP, DROP | DEDUP, SYM | DROP, SYM | DROP | DEDUP])
@pytest.mark.parametrize("m", [1, 7, 300, 4096])
def test_coo_build_matches_numpy(ctx, flags, m):
    rng = np.random.default_rng(m * 31 + flags)
    ne = 5 * m + 3
    src = rng.integers(0, m, ne).astype(np.int32)
    dst = rng.integers(0, m, ne).astype(np.int32)
    dup = rng.integers(0, ne, ne // 4)
    src[dup[: len(dup) // 2]] = src[dup[len(dup) // 2:][: len(dup) // 2]]
    dst[dup[: len(dup) // 2]] = dst[dup[len(dup) // 2:][: len(dup) // 2]]
    val = rng.uniform(-1, 1, ne).astype(np.float32)
    C = ctx.build_csr(m, _dev(src), _dev(dst), _dev(val), flags)
    rp, ci, v = C.to_numpy()
    erp, eci, ev = _ref_build(m, src, dst, val, flags)
    np.testing.assert_array_equal(rp, erp)
    np.testing.assert_array_equal(ci, eci)
    np.testing.assert_array_equal(v, ev)


def test_coo_build_without_values_and_empty(ctx):
    import torch

    C = ctx.build_csr(5, torch.empty(0, dtype=torch.int32, device="cuda"),
                      torch.empty(0, dtype=torch.int32, device="cuda"), None, SYM | DROP | DEDUP)
    rp, ci, v = C.to_numpy()
    assert rp.tolist() == [0] * 6 and ci.shape[0] == 0 and v is None
    src = np.array([0, 1, 1, 2], dtype=np.int32)
    dst = np.array([1, 0, 2, 2], dtype=np.int32)
    rp, ci, _ = ctx.build_csr(3, _dev(src), _dev(dst), None, SYM | DROP | DEDUP).to_numpy()
    assert rp.tolist() == [0, 1, 3, 4] and ci.tolist() == [1, 0, 2, 1]


def test_coo_build_rejects_out_of_range_ids(ctx):
    src = np.array([0, 5], dtype=np.int32)
    dst = np.array([1, 1], dtype=np.int32)
    with pytest.raises(ap.ApspieError):
        ctx.build_csr(4, _dev(src), _dev(dst))
    # the context stays usable
    rp, ci, _ = ctx.build_csr(4, _dev(src[:1]), _dev(dst[:1])).to_numpy()
    assert rp.tolist() == [0, 1, 1, 1, 1] and ci.tolist() == [1]


@pytest.mark.parametrize("shape", [(1, 1), (50, 300), (3000, 700), (1 << 14, 1 << 14)])
def test_transpose_matches_scipy(ctx, shape):
    import scipy.sparse as sp

    m, n = shape
    A = sp.random(m, n, density=min(1.0, 8.0 / n), format="csr", dtype=np.float32,
                  random_state=np.random.RandomState(m + n))
    A.sort_indices()
    g = ap.HostGraph(m, n, A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data.astype(np.float32))
    T = ctx.transpose(ap.DeviceGraph(g))
    rp, ci, v = T.to_numpy()
    AT = A.T.tocsr()
    AT.sort_indices()
    np.testing.assert_array_equal(rp, AT.indptr)
    np.testing.assert_array_equal(ci, AT.indices)
    np.testing.assert_array_equal(v, AT.data)
    # transposing twice gives A back
    rp2, ci2, v2 = ctx.transpose(T).to_numpy()
    np.testing.assert_array_equal(rp2, A.indptr)
    np.testing.assert_array_equal(ci2, A.indices)
    np.testing.assert_array_equal(v2, A.data)


@pytest.mark.parametrize("ne", [1, 6143, 6144, 6145, 8191, 8192, 8193, 49153])
def test_build_at_the_edges_of_sort_and_compaction_tiles(ctx, ne):
    """Edge counts around the sort's tiles (6,144 pairs) and the compaction's (8,192); half of
    the edges repeat others, a few are self-loops, and the last vertices have no edges."""
    rng = np.random.default_rng(ne)
    m = 70001  # 17 bits an id: two passes of 8 and more of fewer bits
    src = rng.integers(0, m // 2, ne).astype(np.int32)
    dst = rng.integers(0, m // 2, ne).astype(np.int32)
    src[ne // 2:], dst[ne // 2:] = src[: ne - ne // 2], dst[: ne - ne // 2]
    dst[::17] = src[::17]
    val = rng.integers(1, 256, ne).astype(np.int32)
    for flags in (SYM | DROP | DEDUP, SYM | DROP, DROP, 0):
        got = ctx.build_csr(m, _dev(src), _dev(dst), _dev(val), flags).to_numpy()
        for a, b in zip(got, _ref_build(m, src, dst, val, flags)):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("valued", [True, False])
@pytest.mark.parametrize("lengths", ["one long row", "short rows", "tile ends"])
def test_transpose_of_uneven_rows(ctx, valued, lengths):
    """Rows longer than the 4,096-entry tiles in which entries find their rows, runs of empty
    rows before, between and after them, rows that end at a tile's end; columns in any order
    and repeated, so that the order of equal columns shows (it is the entries' order)."""
    n = 333
    deg = np.zeros(3000, dtype=np.int64)
    if lengths == "one long row":
        deg[[700, 701, 2500]] = [9000, 3, 1]
    elif lengths == "short rows":
        deg[100:2900] = np.arange(2800) % 7
    else:
        deg[[5, 600, 601, 602]] = [4095, 1, 4096, 4096]
    rp = np.concatenate(([0], np.cumsum(deg))).astype(np.int32)
    rng = np.random.default_rng(int(deg.sum()))
    ci = rng.integers(0, n, rp[-1]).astype(np.int32)
    val = rng.integers(-99, 99, rp[-1]).astype(np.int32) if valued else None
    T = ctx.transpose(ap.DeviceGraph(ap.HostGraph(3000, n, rp, ci, val)))
    trp, tci, tval = T.to_numpy()
    order = np.argsort(ci, kind="stable")
    rows = np.repeat(np.arange(3000), deg)
    np.testing.assert_array_equal(trp, np.concatenate(([0], np.cumsum(np.bincount(ci, minlength=n)))))
    np.testing.assert_array_equal(tci, rows[order])
    if valued:
        np.testing.assert_array_equal(tval, val[order])
    else:
        assert tval is None


def test_matrices_from_reused_memory_in_two_threads(ctx):
    """Memory of freed matrices is handed out again, across threads and streams: two threads
    with contexts and streams of their own build, check and free matrices of changing sizes."""
    import threading

    import torch

    torch.cuda.synchronize()
    errors = []

    def work(seed):
        try:
            rng = np.random.default_rng(seed)
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream), ap.Context(0, stream) as c:
                for k in range(12):
                    m = int(rng.integers(2, 3000))
                    src, dst = rng.integers(0, m, (2, 4 * m)).astype(np.int32)
                    val = rng.integers(0, 99, 4 * m).astype(np.int32)
                    d = [torch.from_numpy(x).cuda() for x in (src, dst, val)]
                    A = c.build_csr(m, *d, DROP)
                    T = c.transpose(A)
                    A.free()  # its memory may come back for the next transpose
                    B = c.transpose(T)
                    got, T = B.to_numpy(), T.free()
                    for x, y in zip(got, _ref_build(m, src, dst, val, DROP)):
                        np.testing.assert_array_equal(x, y)
                    B.free()
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in (1, 2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_memory_kept_from_freed_matrices_is_bounded(ctx):
    import torch

    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    n = 60_000_000  # 240 MB a matrix
    src = torch.zeros(1, dtype=torch.int32, device="cuda")
    made = [ctx.build_csr(n + 20_000_000 * k, src, src) for k in range(8)]
    assert sum(4 * c.m for c in made) > 3 << 30
    scratch = ctx.scratch_bytes()
    for c in made:
        c.free()
    torch.cuda.synchronize()
    # at most 1 GiB of blocks, the context's scratch, and what the driver rounds up
    assert before - torch.cuda.mem_get_info()[0] <= (1 << 30) + scratch + (64 << 20)


def test_matrix_freed_during_a_stream_capture(ctx):
    """Freeing a matrix leaves a capture under way alone, and its memory is reused afterwards."""
    import torch

    src = torch.arange(300000, dtype=torch.int32, device="cuda") % 3000
    A = ctx.build_csr(3000, src, src.flip(0).contiguous())
    x = torch.arange(1000, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="relaxed"):
        y = x + 1
        A.free()
        z = y * 2
    graph.replay()
    assert torch.equal(z, (x + 1) * 2)
    B = ctx.build_csr(3000, src, src.flip(0).contiguous())
    rp, ci, _ = B.to_numpy()
    assert rp[-1] == 300000 and np.array_equal(np.sort(ci), np.sort(src.cpu().numpy()))
    B.free()


def test_kept_memory_makes_room(ctx):
    """What is kept of freed matrices is given to the library's other allocations when memory
    is short, and back to CUDA on demand."""
    import torch

    one = torch.zeros(1, dtype=torch.int32, device="cuda")
    g = ap.gen_rmat(16, 8, 1, 3, weights=False)
    dg = ap.DeviceGraph(g)
    nq = 1024  # the tuner's output: 268 MB
    with ap.Context(0) as c:
        c.autotune(ap.TUNE_BFS_BATCH, dg, sources=[1] * 32, reps=1)  # scratch
        c.bfs_batch(dg, torch.ones(512, dtype=torch.int32, device="cuda"))
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        kept = [c.build_csr(100_000_000, one, one) for _ in range(2)]  # 400 MB each, and scratch
        for k in kept:
            k.free()
        free = torch.cuda.mem_get_info()[0]
        rest = torch.empty(free - (160 << 20), dtype=torch.uint8, device="cuda")
        assert torch.cuda.mem_get_info()[0] < 200 << 20
        best, _ = c.autotune(ap.TUNE_BFS_BATCH, dg, sources=[1] * nq, reps=1)
        assert best["batch_push_frac"] > 0
        kept = c.build_csr(100_000_000, one, one)
        kept.free()
        low = torch.cuda.mem_get_info()[0]
        c.trim()
        assert torch.cuda.mem_get_info()[0] >= low + (380 << 20)
        del rest
    torch.cuda.empty_cache()


def _few_entries(m, n):
    """n entries between vertices spread over all of 0 .. m - 1, the first and the last among them."""
    rng = np.random.default_rng(n)
    u, v = rng.integers(0, m, (2, n))
    u[0], v[0] = m - 1, 0
    return u.astype(np.int32), v.astype(np.int32)


@pytest.mark.parametrize("m,n", [(20000, 3), (17000, 4096), (3_000_000, 70), (3_000_000, 9000), (3_000_000, 2_999_999),
                                 (200_000, 200_000)])
@pytest.mark.parametrize("flags", [0, DROP])
def test_build_and_transpose_of_mostly_empty_rows(ctx, m, n, flags):
    """Fewer entries than rows, and entries of a block in rows far apart."""
    import torch

    u, v = _few_entries(m, n)
    if n > 5000:  # a part in neighbouring rows, a part in rows far apart
        u[: n // 2] = 77 + np.arange(n // 2) % 4000
    val = np.arange(n, dtype=np.int32)
    d = [torch.from_numpy(x).cuda() for x in (u, v, val)]
    A = ctx.build_csr(m, *d, flags)
    rp, ci, va = A.to_numpy()
    if flags:
        for x, y in zip((rp, ci, va), _ref_build(m, u, v, val, flags)):
            np.testing.assert_array_equal(x, y)
    else:
        order = np.lexsort((np.arange(n), v, u))
        np.testing.assert_array_equal(rp, np.concatenate(([0], np.cumsum(np.bincount(u, minlength=m)))))
        np.testing.assert_array_equal(ci, v[order])
        np.testing.assert_array_equal(va, val[order])
    rows = np.repeat(np.arange(m), np.diff(rp))
    back = np.argsort(ci, kind="stable")
    want = np.concatenate(([0], np.cumsum(np.bincount(ci, minlength=m))))
    host = ap.HostGraph(m, m, rp, ci, None)
    for T, vals in ((ctx.transpose(A), True), (ctx.transpose(ap.DeviceGraph(host)), False)):
        trp, tci, tva = T.to_numpy()
        np.testing.assert_array_equal(trp, want)
        np.testing.assert_array_equal(tci, rows[back])
        if vals:
            np.testing.assert_array_equal(tva, va[back])
        T.free()
    A.free()


def test_few_entries_in_many_rows_take_little_time(ctx):
    """The empty rows are filled by all of the device: 64 entries in 2^25 rows."""
    import time

    import torch

    m = 1 << 25
    u, v = _few_entries(m, 64)
    d = [torch.from_numpy(x).cuda() for x in (u, v, np.arange(64, dtype=np.int32))]
    seconds = []
    for _ in range(4):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        A = ctx.build_csr(m, *d, 0)
        T = ctx.transpose(A)
        torch.cuda.synchronize()
        seconds.append(time.perf_counter() - t0)
        T.free()
        A.free()
    # writing the two 134 MB arrays of row starts takes 0.05 ms; a thread or a block that fills or
    # walks the rows alone 10 ms and more
    assert min(seconds) < 8e-3, seconds
