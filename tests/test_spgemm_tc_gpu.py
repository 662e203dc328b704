"""GPU parity tests of the row-binned hash SpGEMM and the masked-SpGEMM triangle count.

int32 values and structures are compared bit-exact with the oracle (row-wise Gustavson).
FP32: rows with at most 128 products (the warp tier: every ER row of the benchmark) are
summed in the oracle's order and compared bit-exact; longer rows accumulate in any order
and are compared within |got - ref| <= 1e-5 * sum(|a_ik * b_kj|) + 1e-30."""
import numpy as np
import pytest

import apspie_b200 as ap
import oracle

pytestmark = pytest.mark.gpu


def _abs_bound(Ah, Bh, crp, cci):
    """sum over products of |a*b| for every output entry (float64)."""
    m = Ah.m
    out = np.zeros(cci.shape[0], dtype=np.float64)
    for i in range(m):
        acc = {}
        for ea in range(Ah.row_ptr[i], Ah.row_ptr[i + 1]):
            k = Ah.col_ind[ea]
            for eb in range(Bh.row_ptr[k], Bh.row_ptr[k + 1]):
                j = int(Bh.col_ind[eb])
                acc[j] = acc.get(j, 0.0) + abs(float(Ah.val[ea]) * float(Bh.val[eb]))
        for p in range(crp[i], crp[i + 1]):
            out[p] = acc[int(cci[p])]
    return out


def _check(ctx, Ah, Bh, exact_f32=True):
    A, B = ap.DeviceGraph(Ah), ap.DeviceGraph(Bh)
    rp, ci, cv = ctx.spgemm(A, B)
    orp, oci, ocv = oracle.spgemm(Ah.m, Bh.n, Ah.row_ptr, Ah.col_ind, Ah.val, Bh.row_ptr, Bh.col_ind, Bh.val)
    np.testing.assert_array_equal(rp, orp)
    np.testing.assert_array_equal(ci, oci)
    if Ah.val.dtype == np.int32 or exact_f32:
        np.testing.assert_array_equal(cv, ocv)
    else:
        bound = _abs_bound(Ah, Bh, orp, oci)
        assert np.all(np.abs(cv.astype(np.float64) - ocv) <= 1e-5 * bound + 1e-30)
    return rp, ci, cv


def test_spgemm_golden_fixture(ctx, golden):
    rp, ci = golden["test_spgemm_d_row_ptr"], golden["test_spgemm_d_col_ind"]
    g = ap.HostGraph(rp.shape[0] - 1, rp.shape[0] - 1, rp, ci, np.ones(ci.shape[0], dtype=np.float32))
    crp, cci, cv = ctx.spgemm(ap.DeviceGraph(g), ap.DeviceGraph(g))
    np.testing.assert_array_equal(crp, golden["spgemm_fixture_row_ptr"])
    np.testing.assert_array_equal(cci, golden["spgemm_fixture_col_ind"])
    np.testing.assert_array_equal(cv, golden["spgemm_fixture_val"])


@pytest.mark.parametrize("vt", [ap.VAL_F32, ap.VAL_I32])
def test_spgemm_er64_golden(ctx, golden, vt):
    e = ap.gen_er(64, 4, 5, vt)
    tag = "f32" if vt == ap.VAL_F32 else "i32"
    rp, ci, cv = ctx.spgemm(ap.DeviceGraph(e), ap.DeviceGraph(e))
    np.testing.assert_array_equal(rp, golden[f"spgemm_er64_{tag}_row_ptr"])
    np.testing.assert_array_equal(ci, golden[f"spgemm_er64_{tag}_col_ind"])
    np.testing.assert_array_equal(cv, golden[f"spgemm_er64_{tag}_val"])


@pytest.mark.parametrize("vt", [ap.VAL_F32, ap.VAL_I32])
def test_spgemm_er_exact(ctx, vt):
    e = ap.gen_er(1 << 14, 8, 5, vt)  # every row: 64 products -> warp tier
    _check(ctx, e, e, exact_f32=True)


def _skewed(n, seed, vt, scale_rows=True):
    """Rows of very different lengths so every bin (warp/block/global) is exercised."""
    rng = np.random.default_rng(seed)
    lens = rng.integers(0, 4, n)
    lens[rng.choice(n, 8, replace=False)] = rng.integers(40, 300, 8)
    lens[rng.choice(n, 3, replace=False)] = [1500, 2200, 3000]
    rp = np.zeros(n + 1, dtype=np.int32)
    rp[1:] = np.cumsum(lens)
    ci = np.concatenate([np.sort(rng.choice(n, int(l), replace=False)) for l in lens]).astype(np.int32)
    if vt == ap.VAL_F32:
        val = rng.uniform(-1, 1, ci.shape[0]).astype(np.float32)
    else:
        val = rng.integers(1, 9, ci.shape[0]).astype(np.int32)
    return ap.HostGraph(n, n, rp, ci, val)


@pytest.mark.parametrize("vt", [ap.VAL_F32, ap.VAL_I32])
def test_spgemm_all_bins(ctx, vt):
    A = _skewed(6000, 1, vt)
    B = _skewed(6000, 2, vt)
    _check(ctx, A, B, exact_f32=False)
    _check(ctx, B, A, exact_f32=False)


def test_spgemm_rectangular_and_empty(ctx):
    rng = np.random.default_rng(3)
    m, k, n = 300, 50, 700
    ra = np.sort(rng.integers(0, 4, m))
    rpa = np.zeros(m + 1, dtype=np.int32)
    rpa[1:] = np.cumsum(ra)
    cia = np.concatenate([np.sort(rng.choice(k, int(x), replace=False)) for x in ra]).astype(np.int32)
    rb = rng.integers(0, 9, k)
    rb[:5] = 0  # empty rows of B
    rpb = np.zeros(k + 1, dtype=np.int32)
    rpb[1:] = np.cumsum(rb)
    cib = np.concatenate([np.sort(rng.choice(n, int(x), replace=False)) for x in rb]).astype(np.int32)
    A = ap.HostGraph(m, k, rpa, cia, rng.integers(1, 9, cia.shape[0]).astype(np.int32))
    B = ap.HostGraph(k, n, rpb, cib, rng.integers(1, 9, cib.shape[0]).astype(np.int32))
    _check(ctx, A, B)


def test_spgemm_two_step_matches(ctx):
    e = ap.gen_er(4096, 8, 7, ap.VAL_I32)
    A = ap.DeviceGraph(e)
    rp, ci, cv = ctx.spgemm_two_step(A, A)
    orp, oci, ocv = oracle.spgemm(e.m, e.n, e.row_ptr, e.col_ind, e.val, e.row_ptr, e.col_ind, e.val)
    np.testing.assert_array_equal(rp.cpu().numpy(), orp)
    np.testing.assert_array_equal(ci.cpu().numpy(), oci)
    np.testing.assert_array_equal(cv.cpu().numpy(), ocv)


def test_spgemm_er_full_size_properties(ctx):
    """ER n=2^20, 8/row, C = A*A (the benchmark size): structure vs the oracle, f32 exact."""
    e = ap.gen_er(1 << 20, 8, 5, ap.VAL_F32)
    _check(ctx, e, e, exact_f32=True)


@pytest.mark.parametrize("vt", [ap.VAL_F32, ap.VAL_I32])
@pytest.mark.parametrize("n", [1, 9, 200, 1 << 24])
def test_spgemm_register_tier_edges(ctx, n, vt):
    """Rows of as many products as a register tier takes, one fewer and one more, from few
    columns (runs of equal columns that cross lanes, one run a row, a run up to the last
    product) to the most columns that the keys hold; more entries than products, rows of B
    that are empty, and numbers of rows that leave groups of a warp without one. Sums are in
    the oracle's order up to 128 products, so FP32 is compared exactly."""
    rng = np.random.default_rng(n)
    k = 400
    lb = rng.integers(0, 9, k)
    lb[:60] = 0
    lb[60:64] = 1
    rpb = np.concatenate(([0], np.cumsum(lb))).astype(np.int32)
    # columns of a row may repeat: both sides treat every entry as one product
    cib = (np.sort(rng.integers(0, n, lb.sum())) if n < 1000 else rng.integers(0, n, lb.sum())).astype(np.int32)
    if n == 1 << 24:
        cib[:: 7] = n - 1
    rows = []
    for want in (1, 2, 31, 32, 33, 63, 64, 65, 127, 128) * 3 + (5,):
        row, left = [], want
        while left:
            c = int(rng.integers(60, k))
            if lb[c] and lb[c] <= left:
                row.append(c)
                left -= lb[c]
        row += [int(x) for x in rng.integers(0, 60, rng.integers(0, 20))]  # empty rows of B
        rows.append(rng.permutation(row))
    rpa = np.concatenate(([0], np.cumsum([len(r) for r in rows]))).astype(np.int32)
    cia = np.concatenate(rows).astype(np.int32)
    f32 = vt == ap.VAL_F32
    va, vb = (rng.uniform(-1, 1, s).astype(np.float32) if f32 else rng.integers(-8, 9, s).astype(np.int32)
              for s in (cia.shape[0], cib.shape[0]))
    _check(ctx, ap.HostGraph(len(rows), k, rpa, cia, va), ap.HostGraph(k, n, rpb, cib, vb))


@pytest.mark.parametrize("vt", [ap.VAL_F32, ap.VAL_I32])
@pytest.mark.parametrize("n", [1, 31, 33, 1000, 32768, 32769, 49152, 49153])
def test_spgemm_rows_of_many_products(ctx, n, vt):
    """Rows past the shared-table tier over few columns (dense accumulators: up to 49,152
    columns, one and two bitmap words a thread) and over one more (global tables); rows of the
    three size classes, repeated columns, rows of B from empty to longer than a warp's step."""
    rng = np.random.default_rng(n)
    k, m = 2500, 40
    lb = np.minimum(rng.choice([0, 1, 3, 31, 40, 130, 300], k), n)
    rpb = np.concatenate(([0], np.cumsum(lb))).astype(np.int32)
    cib = np.concatenate([np.sort(rng.choice(n, int(x), replace=False)) for x in lb]).astype(np.int32)
    la = np.concatenate(([2500, 2000, 0, 1500, 1200], rng.integers(0, 60, m - 5)))
    rpa = np.concatenate(([0], np.cumsum(la))).astype(np.int32)
    cia = np.concatenate([np.sort(rng.choice(k, int(x), replace=False)) for x in la]).astype(np.int32)
    f32 = vt == ap.VAL_F32
    va, vb = (rng.uniform(-1, 1, s).astype(np.float32) if f32 else rng.integers(-8, 9, s).astype(np.int32)
              for s in (cia.shape[0], cib.shape[0]))
    _check(ctx, ap.HostGraph(m, k, rpa, cia, va), ap.HostGraph(k, n, rpb, cib, vb), exact_f32=False)


def test_spgemm_rejects_mismatch(ctx):
    e = ap.gen_er(64, 4, 5, ap.VAL_F32)
    f = ap.gen_er(64, 4, 5, ap.VAL_I32)
    with pytest.raises(ap.ApspieError):
        ctx.spgemm(ap.DeviceGraph(e), ap.DeviceGraph(f))


# --------------------------------------------------------------------------- TC
def test_tc_fixtures(ctx, golden, fixture_keys):
    for key in fixture_keys:
        if key + "_tc" not in golden:
            continue
        rp, ci = golden[key + "_row_ptr"], golden[key + "_col_ind"]
        A = ap.DeviceGraph(ap.HostGraph(rp.shape[0] - 1, rp.shape[0] - 1, rp, ci, None, True))
        Lg = ctx.strict_lower(A)
        assert ctx.tc(Lg) == int(golden[key + "_tc"][0]), key
        Lg.free()


@pytest.mark.parametrize("scale,ef", [(10, 16), (14, 16)])
def test_tc_rmat_vs_oracle(ctx, scale, ef):
    g = ap.gen_rmat(scale, ef, 1, 3, weights=False)
    Lh = ap.strict_lower(g)
    ref = oracle.tc(Lh.row_ptr, Lh.col_ind)
    assert ctx.tc(ap.DeviceGraph(Lh)) == ref
    Ld = ctx.strict_lower(ap.DeviceGraph(g))
    lrp, lci, _ = Ld.to_numpy()
    np.testing.assert_array_equal(lrp, Lh.row_ptr)
    np.testing.assert_array_equal(lci, Lh.col_ind)
    assert ctx.tc(Ld) == ref


def test_tc_rmat18_full_size(ctx):
    g = ap.gen_rmat(18, 16, 1, 3, weights=False)
    Lh = ap.strict_lower(g)
    assert ctx.tc(ap.DeviceGraph(Lh)) == oracle.tc(Lh.row_ptr, Lh.col_ind)


def test_tc_dense_clique_uses_block_and_global_tiers(ctx):
    # a 3000-clique: every row of L up to 2999 long -> block and global tiers
    n = 3000
    rows = [np.arange(i, dtype=np.int32) for i in range(n)]
    rp = np.zeros(n + 1, dtype=np.int32)
    rp[1:] = np.cumsum([len(r) for r in rows])
    ci = np.concatenate(rows)
    assert ctx.tc(ap.DeviceGraph(ap.HostGraph(n, n, rp, ci))) == n * (n - 1) * (n - 2) // 6


@pytest.mark.parametrize("m", [2, 31, 33, 257, 5000, 1638400, 1638401])
def test_tc_bitmap_and_hash_paths(ctx, m):
    """Vertices around a bitmap word, the most whose bitmap fits an SM and one more; a vertex
    with more partners than the first class begins at, lists from empty to longer than a
    warp's step, beside a random part."""
    rng = np.random.default_rng(m)
    core = min(m, 700)
    ids = np.sort(rng.choice(m, core, replace=False))
    u, v = rng.integers(0, core, (2, 12 * core))
    u[: core // 2], v[: core // 2] = 0, rng.integers(0, core, core // 2)  # one vertex meets half of them
    u, v = ids[u], ids[v]
    key = np.unique(np.maximum(u, v)[u != v].astype(np.int64) * m + np.minimum(u, v)[u != v])
    rp = np.concatenate(([0], np.cumsum(np.bincount(key // m, minlength=m)))).astype(np.int32)
    Lh = ap.HostGraph(m, m, rp, (key % m).astype(np.int32))
    assert ctx.tc(ap.DeviceGraph(Lh)) == oracle.tc(Lh.row_ptr, Lh.col_ind)


@pytest.mark.parametrize("what", ["equal neighbours", "a diagonal entry", "an upper entry"])
def test_tc_of_what_is_no_set_of_lower_entries(ctx, what):
    """sum((L*L) .* L) as given: what the bitmap path cannot count (rows that repeat an entry,
    entries on or above the diagonal) is counted as it was before there was one."""
    rng = np.random.default_rng(7)
    m = 400
    d = np.tril(rng.random((m, m)) < 0.1, -1).astype(np.int64)
    if what == "a diagonal entry":
        d[200, 200] = 1
    elif what == "an upper entry":
        d[100, 300] = 1
    rows, cols = np.nonzero(d)
    if what == "equal neighbours":
        again = rng.choice(rows.size, 50, replace=False)
        rows, cols = np.concatenate((rows, rows[again])), np.concatenate((cols, cols[again]))
        order = np.lexsort((cols, rows))
        rows, cols = rows[order], cols[order]
    rp = np.concatenate(([0], np.cumsum(np.bincount(rows, minlength=m)))).astype(np.int32)
    got = ctx.tc(ap.DeviceGraph(ap.HostGraph(m, m, rp, cols.astype(np.int32))))
    if what == "equal neighbours":
        # oriented by (degree, id), then every wedge's end looked up in the first vertex's set
        deg = np.bincount(rows, minlength=m) + np.bincount(cols, minlength=m)
        fwd = (deg[rows] < deg[cols]) | ((deg[rows] == deg[cols]) & (rows < cols))
        a, b = np.where(fwd, rows, cols), np.where(fwd, cols, rows)
        D = np.zeros((m, m), dtype=np.int64)
        np.add.at(D, (a, b), 1)
        assert got == int(((D @ D) * (D > 0)).sum())
    else:
        assert got == int(((d @ d) * d).sum())


@pytest.mark.parametrize("m,p", [(60, 0.5), (400, 0.1)])
def test_tc_of_rows_out_of_order(ctx, m, p):
    """Rows whose entries don't ascend: as many triangles as in order without repeated entries;
    with entries repeated at the end of their row (never beside each other), the wedges of the
    oriented edges whose end is in the first vertex's set, each as often as its edges are given."""
    rng = np.random.default_rng(m)
    rows, cols = np.nonzero(np.tril(rng.random((m, m)) < p, -1))
    for repeats in (0, rows.size // 3):
        largest = np.append(rows[1:] != rows[:-1], True)
        again = rng.choice(np.nonzero(~largest)[0], repeats, replace=False)
        r, c = np.concatenate((rows, rows[again])), np.concatenate((cols, cols[again]))
        order = np.lexsort((c if repeats else -c, np.arange(r.size) >= rows.size, r))
        r, c = r[order], c[order]
        assert not np.any((r[1:] == r[:-1]) & (c[1:] == c[:-1]))
        deg = np.bincount(r, minlength=m) + np.bincount(c, minlength=m)
        fwd = (deg[r] < deg[c]) | ((deg[r] == deg[c]) & (r < c))
        D = np.zeros((m, m), dtype=np.int64)
        np.add.at(D, (np.where(fwd, r, c), np.where(fwd, c, r)), 1)
        rp = np.concatenate(([0], np.cumsum(np.bincount(r, minlength=m)))).astype(np.int32)
        got = ctx.tc(ap.DeviceGraph(ap.HostGraph(m, m, rp, c.astype(np.int32))))
        assert got == int(((D @ D) * (D > 0)).sum()), repeats


def test_sizes_of_threads_do_not_meet(ctx):
    """Contexts are independent: threads with contexts of their own and small or large operands,
    whose kernels take shared memory by the operands' size (five seconds of calls, since a call
    has to fall between two steps of another)."""
    import threading
    import time

    import torch

    n = 60
    rng = np.random.default_rng(5)
    d = (rng.random((n, n)) < 0.6).astype(np.int32)
    low = np.tril(d, -1)

    def operand(a, m, val):
        rp = np.full(m + 1, np.count_nonzero(a), dtype=np.int32)
        rp[: n + 1] = np.concatenate(([0], np.cumsum(a.sum(1))))
        ci = np.nonzero(a)[1].astype(np.int32)
        return ap.HostGraph(m, m, rp, ci, np.ones(ci.size, dtype=np.int32) if val else None)

    want, triangles = d @ d, int(((low @ low) * low).sum())
    errors = []

    def work(kind, m):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream), ap.Context(0, stream) as c:
                g = ap.DeviceGraph(operand(d if kind == "spgemm" else low, m, kind == "spgemm"))
                stream.synchronize()
                end, k = time.monotonic() + 5.0, 0
                while time.monotonic() < end and not errors:
                    if kind == "tc":
                        assert c.tc(g) == triangles
                        continue
                    rp, ci, v = c.spgemm_two_step(g, g)
                    if k % 64 == 0:
                        rows = np.repeat(np.arange(m), np.diff(rp.cpu().numpy()))
                        got = np.zeros((n, n), dtype=np.int64)
                        got[rows, ci.cpu().numpy()] = v.cpu().numpy()
                        np.testing.assert_array_equal(got, want)
                    k += 1
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=a)
               for a in (("tc", 100), ("tc", 600000), ("spgemm", 100), ("spgemm", 49000))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


@pytest.mark.parametrize("uneven", [False, True])
@pytest.mark.parametrize("m", [8192, 8193, 131072, 140000, 600000])
def test_tc_lists_of_every_size(ctx, m, uneven):
    """Lists around the limits of what a warp counts (17 entries, or 64), beside many vertices of
    degree one and two: of about even degrees, and with a vertex that meets half of them."""
    rng = np.random.default_rng(m)
    at = m // 3
    edges = [np.stack((np.arange(1, at), np.arange(at - 1)))]  # a path
    if uneven:
        edges.append(np.stack((np.arange(2, at), np.zeros(at - 2, dtype=np.int64))))
        i, j = np.tril_indices(200, -1)
        edges.append(np.stack((i, j)))
    for c in (3, 8, 9, 10, 17, 18, 19, 33, 34, 64, 65, 66, 67):  # cliques: lists up to c - 1
        i, j = np.tril_indices(c, -1)
        edges.append(np.stack((i + at, j + at)))
        at += c
    for hubs, leaves in ((2, 31), (2, 32), (2, 33), (5, 40), (9, 33), (20, 300)):  # hubs joined, all to every leaf
        i, j = np.tril_indices(hubs, -1)
        edges.append(np.stack((i + at, j + at)))
        a, b = np.meshgrid(np.arange(hubs), np.arange(leaves))
        edges.append(np.stack((b.ravel() + at + hubs, a.ravel() + at)))
        at += hubs + leaves
    e = np.concatenate(edges, axis=1)
    e = rng.permutation(m)[e]  # ids in no order
    key = np.unique(np.maximum(*e).astype(np.int64) * m + np.minimum(*e))
    rp = np.concatenate(([0], np.cumsum(np.bincount(key // m, minlength=m)))).astype(np.int32)
    ci = (key % m).astype(np.int32)
    assert ctx.tc(ap.DeviceGraph(ap.HostGraph(m, m, rp, ci))) == oracle.tc(rp, ci)


def test_tc_of_low_degrees_takes_little_time(ctx):
    """A grid of a million vertices: two entries a row, no triangles."""
    import time

    n = 1024
    i = np.arange(n * n)
    key = np.sort(np.concatenate((i[i % n > 0] * (n * n + 1) - 1, i[n:] * (n * n + 1) - n)))
    rp = np.concatenate(([0], np.cumsum(np.bincount(key // (n * n), minlength=n * n)))).astype(np.int32)
    g = ap.DeviceGraph(ap.HostGraph(n * n, n * n, rp, (key % (n * n)).astype(np.int32)))
    seconds = []
    for _ in range(4):
        t0 = time.perf_counter()
        assert ctx.tc(g) == 0
        seconds.append(time.perf_counter() - t0)
    # 0.7 ms, where a block's round for each vertex made it 13
    assert min(seconds) < 4e-3, seconds


def _joined_halves(rows, cols):
    """`rows` vertices that meet all of the first `cols`, of which the first two meet: rows triangles."""
    m = rows + cols
    deg = np.zeros(m, dtype=np.int64)
    deg[1] = 1
    deg[cols:] = cols
    rp = np.concatenate(([0], np.cumsum(deg))).astype(np.int32)
    ci = np.concatenate(([0], np.tile(np.arange(cols), rows))).astype(np.int32)
    return ap.HostGraph(m, m, rp, ci)


def test_tc_when_memory_is_short(ctx):
    """Where the bitmap path's scratch (16 bytes an entry) does not fit, the hash path's (4) does."""
    import torch

    g = ap.DeviceGraph(_joined_halves(8000, 2000))
    with ap.Context(0) as c:
        ctx.trim()
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        rest = torch.empty(free - (200 << 20), dtype=torch.uint8, device="cuda")
        assert torch.cuda.mem_get_info()[0] < 230 << 20
        assert c.tc(g) == 8000
        assert c.scratch_bytes() < 200 << 20
        del rest
    torch.cuda.empty_cache()
    assert ctx.tc(g) == 8000


@pytest.mark.parametrize("rows,cols", [(2100, 4000), (9000, 1865)])
def test_tc_hash_path_in_parts(ctx, rows, cols):
    """More vertices than the bitmaps take, and more entries than a part of the hash path (2^24):
    the orientation is made part by part."""
    g = _joined_halves(rows, cols)
    m = 1_700_000
    rp = np.concatenate((g.row_ptr, np.full(m - g.m, g.row_ptr[-1], dtype=np.int32)))
    assert (g.nnz > 1 << 24) == (rows == 9000)
    assert ctx.tc(ap.DeviceGraph(ap.HostGraph(m, m, rp, g.col_ind))) == rows
