"""GPU parity tests of the SpMSpV traversals (BFS, SSSP, MIS) through the C ABI.

Bit-exact against golden vectors from the reference's own CPU code (small fixtures, all
sources) and against the oracle on generated R-MAT graphs up to the benchmark's full
size (scale 20)."""
import numpy as np
import pytest

import apspie_b200 as ap
import oracle

pytestmark = pytest.mark.gpu


def _dev(golden, key, with_w=False):
    rp, ci = golden[key + "_row_ptr"], golden[key + "_col_ind"]
    val = golden[key + "_w"] if with_w else None
    g = ap.HostGraph(rp.shape[0] - 1, rp.shape[0] - 1, rp, ci, val, symmetric=key.endswith("_u"))
    return g, ap.DeviceGraph(g)


@pytest.fixture(scope="module")
def rmat14():
    g = ap.gen_rmat(14, 16, 1, 3)
    return g, ap.DeviceGraph(g), ap.max_degree_vertex(g)


@pytest.fixture(scope="module")
def rmat20():
    g = ap.gen_rmat(20, 16, 2, 3)
    return g, ap.DeviceGraph(g), ap.max_degree_vertex(g)


# ------------------------------------------------------------------------------- BFS
def test_bfs_fixtures_all_sources(ctx, golden, fixture_keys):
    for key in fixture_keys:
        g, dg = _dev(golden, key)
        for s in range(g.m):
            got = ctx.bfs(dg, s).cpu().numpy()
            np.testing.assert_array_equal(got, golden[key + "_bfs"][s], err_msg=f"{key} src {s}")


@pytest.mark.parametrize("alpha", [0.0, 14.0, 1e6])
def test_bfs_rmat12_golden_all_directions(ctx, golden, alpha):
    g = ap.gen_rmat(12, 16, 1, 3)
    src = int(golden["rmat12_meta"][2])
    dg = ap.DeviceGraph(g)
    ctx.set_bfs_tuning(alpha, 24.0)
    try:
        d = ctx.bfs(dg, src).cpu().numpy()
    finally:
        ctx.set_bfs_tuning(14.0, 24.0)
    np.testing.assert_array_equal(d, golden["rmat12_bfs"])


def test_bfs_rmat14_many_sources_vs_oracle(ctx, rmat14):
    g, dg, src = rmat14
    rng = np.random.default_rng(0)
    for s in [src] + rng.integers(0, g.m, 12).tolist():
        np.testing.assert_array_equal(ctx.bfs(dg, int(s)).cpu().numpy(), oracle.bfs(g.row_ptr, g.col_ind, int(s)))


def test_bfs_push_and_pull_paths_both_taken(ctx, rmat14):
    import torch

    g, dg, src = rmat14
    out = torch.empty(g.m, dtype=torch.int32, device="cuda")
    st = ctx.bfs_into(dg, src, out, stats=True)
    assert st["push_iterations"] >= 1 and st["pull_iterations"] >= 1, st
    ref = oracle.bfs(g.row_ptr, g.col_ind, src)
    np.testing.assert_array_equal(out.cpu().numpy(), ref)
    reached = ref >= 0
    assert st["vertices_reached"] == int(reached.sum())
    assert st["edges_component"] == int(g.degrees()[reached].sum())
    assert st["iterations"] == int(ref.max()) + 1


def test_bfs_depth_cap(ctx, rmat14):
    g, dg, src = rmat14
    full = oracle.bfs(g.row_ptr, g.col_ind, src)
    for cap in (1, 2, 3):
        got = ctx.bfs(dg, src, depth_cap=cap).cpu().numpy()
        np.testing.assert_array_equal(got, np.where((full >= 0) & (full < cap), full, -1))


def test_bfs_rmat20_full_size(ctx, rmat20):
    g, dg, src = rmat20
    np.testing.assert_array_equal(ctx.bfs(dg, src).cpu().numpy(), oracle.bfs(g.row_ptr, g.col_ind, src))


def test_bfs_isolated_source_and_empty_rows(ctx):
    # vertices 0..3 isolated, a path 4-5-6, vertex 7 isolated
    rp = np.array([0, 0, 0, 0, 0, 1, 3, 4, 4], dtype=np.int32)
    ci = np.array([5, 4, 6, 5], dtype=np.int32)
    g = ap.HostGraph(8, 8, rp, ci, symmetric=True)
    dg = ap.DeviceGraph(g)
    for s in range(8):
        np.testing.assert_array_equal(ctx.bfs(dg, s).cpu().numpy(), oracle.bfs(rp, ci, s))


# ------------------------------------------------------------------------------ SSSP
def test_sssp_fixtures_all_sources(ctx, golden, fixture_keys):
    for key in fixture_keys:
        if key + "_sssp" not in golden:
            continue
        g, dg = _dev(golden, key, with_w=True)
        for s in range(g.m):
            np.testing.assert_array_equal(ctx.sssp(dg, s).cpu().numpy(), golden[key + "_sssp"][s], err_msg=f"{key} {s}")


def test_sssp_rmat12_golden(ctx, golden):
    g = ap.gen_rmat(12, 16, 1, 3)
    np.testing.assert_array_equal(ctx.sssp(ap.DeviceGraph(g), int(golden["rmat12_meta"][2])).cpu().numpy(),
                                  golden["rmat12_sssp"])


def test_sssp_rmat14_vs_oracle(ctx, rmat14):
    import torch

    g, dg, src = rmat14
    out = torch.empty(g.m, dtype=torch.int32, device="cuda")
    st = ctx.sssp_into(dg, src, out, stats=True)
    ref = oracle.sssp(g.row_ptr, g.col_ind, g.val, src)
    np.testing.assert_array_equal(out.cpu().numpy(), ref)
    assert st["vertices_reached"] == int((ref >= 0).sum())


def test_sssp_rmat20_full_size(ctx, rmat20):
    g, dg, src = rmat20
    np.testing.assert_array_equal(ctx.sssp(dg, src).cpu().numpy(), oracle.sssp(g.row_ptr, g.col_ind, g.val, src))


def test_sssp_zero_weights_and_repeated_calls(ctx, rmat14):
    g, _, src = rmat14
    w = g.val.copy()
    w[::3] = 0
    h = ap.HostGraph(g.m, g.n, g.row_ptr, g.col_ind, w, symmetric=True)
    dg = ap.DeviceGraph(h)
    ref = oracle.sssp(h.row_ptr, h.col_ind, h.val, src)
    for _ in range(3):
        np.testing.assert_array_equal(ctx.sssp(dg, src).cpu().numpy(), ref)


# ------------------------------------------------------------------------------- MIS
def test_mis_fixtures(ctx, golden, fixture_keys):
    import torch

    for key in fixture_keys:
        if key + "_mis" not in golden:
            continue
        g, dg = _dev(golden, key)
        prio = torch.from_numpy(golden["mt19937_seed4"][: g.m].astype(np.uint32).view(np.int32)).cuda()
        got = ctx.mis(dg, prio).cpu().numpy()
        np.testing.assert_array_equal(got, golden[key + "_mis"], err_msg=key)


def _prio(m):
    import torch

    return torch.from_numpy(ap.mt19937_u32(4, m).view(np.int32)).cuda()


def test_mis_rmat12_golden(ctx, golden):
    g = ap.gen_rmat(12, 16, 1, 3)
    got = ctx.mis(ap.DeviceGraph(g), _prio(g.m)).cpu().numpy()
    np.testing.assert_array_equal(got, golden["rmat12_mis"])


def test_mis_rmat20_full_size(ctx, rmat20):
    g, dg, _ = rmat20
    pr = ap.mt19937_u32(4, g.m)
    got = ctx.mis(dg, _prio(g.m)).cpu().numpy()
    ref = oracle.mis_greedy(g.row_ptr, g.col_ind, pr)
    np.testing.assert_array_equal(got, ref)
    assert oracle.mis_check(g.row_ptr, g.col_ind, got) == 0


def test_mis_priority_ties_broken_by_id(ctx, rmat14):
    import torch

    g, dg, _ = rmat14
    pr = (ap.mt19937_u32(9, g.m) % 4).astype(np.uint32)  # heavy ties
    got = ctx.mis(dg, torch.from_numpy(pr.view(np.int32)).cuda()).cpu().numpy()
    np.testing.assert_array_equal(got, oracle.mis_greedy(g.row_ptr, g.col_ind, pr))


# ----------------------------------------------------------------- SpMSpV (one hop)
def test_spmspv_bool_matches_mis_check_semantics(ctx, rmat14):
    import torch

    g, dg, _ = rmat14
    x = (np.arange(g.m) % 7 == 0).astype(np.int32)
    y = torch.empty(g.m, dtype=torch.int32, device="cuda")
    ctx.spmspv_bool_into(dg, torch.from_numpy(x).cuda(), y)
    exp = np.zeros(g.m, dtype=np.int32)
    for u in np.flatnonzero(x):
        exp[g.col_ind[g.row_ptr[u]:g.row_ptr[u + 1]]] = 1
    np.testing.assert_array_equal(y.cpu().numpy(), exp)


# ------------------------------------------------------------------------ errors
def test_invalid_arguments_rejected(ctx, rmat14):
    import torch

    g, dg, src = rmat14
    out = torch.empty(g.m, dtype=torch.int32, device="cuda")
    with pytest.raises(ap.ApspieError) as e:
        ctx.bfs_into(dg, g.m, out)
    assert e.value.name == "APSPIE_ERR_INVALID_ARG"
    with pytest.raises(ap.ApspieError):
        ctx.bfs_into(dg, -1, out)
    with pytest.raises(ap.ApspieError):  # SSSP needs int32 weights
        ctx.sssp_into(ap.DeviceGraph(ap.HostGraph(g.m, g.n, g.row_ptr, g.col_ind, None)), src, out)
    # the context stays usable
    np.testing.assert_array_equal(ctx.bfs(dg, src).cpu().numpy(), oracle.bfs(g.row_ptr, g.col_ind, src))


def test_poisoned_csr_caught_by_validation(ctx, rmat14):
    g, _, src = rmat14
    bad = g.col_ind.copy()
    bad[123] = g.m + 5  # column out of range
    dg = ap.DeviceGraph(ap.HostGraph(g.m, g.n, g.row_ptr, bad, g.val, symmetric=True))
    with pytest.raises(ap.ApspieError):
        ctx.validate(dg)
    ctx.set_validate(True)
    try:
        with pytest.raises(ap.ApspieError) as e:
            ctx.bfs(dg, src)
        assert "column index out of range" in str(e.value)
        rp = g.row_ptr.copy()
        rp[5], rp[6] = rp[6], rp[5]
        dg2 = ap.DeviceGraph(ap.HostGraph(g.m, g.n, rp, g.col_ind, g.val))
        with pytest.raises(ap.ApspieError):
            ctx.sssp(dg2, src)
    finally:
        ctx.set_validate(False)
    good = ap.DeviceGraph(g)
    np.testing.assert_array_equal(ctx.bfs(good, src).cpu().numpy(), oracle.bfs(g.row_ptr, g.col_ind, src))


def test_negative_weight_reported_not_hung(ctx):
    rp = np.array([0, 1, 2], dtype=np.int32)
    ci = np.array([1, 0], dtype=np.int32)
    w = np.array([-3, -3], dtype=np.int32)
    dg = ap.DeviceGraph(ap.HostGraph(2, 2, rp, ci, w))
    import torch

    out = torch.empty(2, dtype=torch.int32, device="cuda")
    with pytest.raises(ap.ApspieError):
        ctx.sssp_into(dg, 0, out, stats=True)


def test_bfs_directed_graph_never_pulls(ctx, golden):
    """A directed pattern must be expanded top-down only: pull would follow in-edges."""
    import torch

    g, dg = _dev(golden, "chesapeake_d")
    assert not dg.symmetric
    out = torch.empty(g.m, dtype=torch.int32, device="cuda")
    for s in range(g.m):
        st = ctx.bfs_into(dg, s, out, stats=True)
        assert st["pull_iterations"] == 0
        np.testing.assert_array_equal(out.cpu().numpy(), golden["chesapeake_d_bfs"][s])


@pytest.mark.parametrize("delta", [1, 7, 64, 100000])
def test_sssp_bucket_width_does_not_change_result(ctx, rmat14, delta):
    g, dg, src = rmat14
    ref = oracle.sssp(g.row_ptr, g.col_ind, g.val, src)
    ctx.set_sssp_delta(delta)
    try:
        np.testing.assert_array_equal(ctx.sssp(dg, src).cpu().numpy(), ref)
    finally:
        ctx.set_sssp_delta(0)


@pytest.mark.parametrize("band", [-1, 1, 4096, 0, 1 << 40])
@pytest.mark.parametrize("delta", [0, 64])
def test_sssp_band_does_not_change_result(ctx, rmat14, band, delta):
    """The distance band only orders the work: band 1 expands one histogram bin per
    iteration (deferring almost the whole frontier every time), -1 and 2^40 never defer."""
    g, dg, src = rmat14
    ref = oracle.sssp(g.row_ptr, g.col_ind, g.val, src)
    ctx.set_sssp_band(band)
    ctx.set_sssp_delta(delta)
    try:
        out = ctx.sssp(dg, src)
        st = ctx.sssp_into(dg, src, out, stats=True)
        np.testing.assert_array_equal(out.cpu().numpy(), ref)
        assert st["edges_expanded"] >= st["edges_component"]
    finally:
        ctx.set_sssp_band(0)
        ctx.set_sssp_delta(0)


def test_sssp_band_cuts_rework(ctx, rmat14):
    """With the default band, re-expansion stays near one pass over the component's edges
    (a whole-frontier Bellman-Ford pass expands several times more)."""
    g, dg, src = rmat14
    out = ctx.sssp(dg, src)
    banded = ctx.sssp_into(dg, src, out, stats=True)
    ctx.set_sssp_band(-1)
    ctx.set_sssp_delta(1 << 20)
    try:
        whole = ctx.sssp_into(dg, src, out, stats=True)
    finally:
        ctx.set_sssp_band(0)
        ctx.set_sssp_delta(0)
    assert banded["edges_expanded"] < whole["edges_expanded"]


@pytest.mark.skipif(not oracle.ref_available(), reason="reference CPU driver not built")
@pytest.mark.parametrize("band", [1, 0, -1])
def test_sssp_f32_band_matches_reference_ssspCPU(ctx, rmat14, band):
    import torch

    g, _, src = rmat14
    rows = np.repeat(np.arange(g.m), np.diff(g.row_ptr))
    lo, hi = np.minimum(rows, g.col_ind), np.maximum(rows, g.col_ind)
    w = (((lo * 7919 + hi * 104729) % 1000) / 9700.0 + 0.0001).astype(np.float32)
    dg = ap.DeviceGraph(ap.HostGraph(g.m, g.n, g.row_ptr, g.col_ind, w, True))
    out = torch.empty(g.m, dtype=torch.float32, device="cuda")
    ctx.set_sssp_band(band)
    try:
        ctx.sssp_f32_into(dg, src, out, unreached=-1.0)
    finally:
        ctx.set_sssp_band(0)
    ref, _ = oracle.ref_sssp_f32(g.row_ptr, g.col_ind, w, src)
    np.testing.assert_array_equal(out.cpu().numpy(), ref)


@pytest.mark.parametrize("blocks", [1, 3, 148])
def test_grid_size_does_not_change_results(ctx, rmat14, blocks):
    import torch

    g, dg, src = rmat14
    ctx.set_max_grid(blocks)
    try:
        np.testing.assert_array_equal(ctx.bfs(dg, src).cpu().numpy(), oracle.bfs(g.row_ptr, g.col_ind, src))
        np.testing.assert_array_equal(ctx.sssp(dg, src).cpu().numpy(), oracle.sssp(g.row_ptr, g.col_ind, g.val, src))
        pr = ap.mt19937_u32(4, g.m)
        got = ctx.mis(dg, torch.from_numpy(pr.view(np.int32)).cuda()).cpu().numpy()
        np.testing.assert_array_equal(got, oracle.mis_greedy(g.row_ptr, g.col_ind, pr))
    finally:
        ctx.set_max_grid(0)


# ------------------------------------------------------------ float SSSP / int32 MIS
def test_sssp_f32_integral_weights_match_golden(ctx, golden):
    import torch

    for key in ("chesapeake_u", "test_mesh_u", "test_cc_u"):
        rp, ci = golden[key + "_row_ptr"], golden[key + "_col_ind"]
        w = golden[key + "_w"].astype(np.float32)
        dg = ap.DeviceGraph(ap.HostGraph(rp.shape[0] - 1, rp.shape[0] - 1, rp, ci, w, True))
        out = torch.empty(rp.shape[0] - 1, dtype=torch.float32, device="cuda")
        for s in range(rp.shape[0] - 1):
            ctx.sssp_f32_into(dg, s, out, unreached=-1.0)
            np.testing.assert_array_equal(out.cpu().numpy(), golden[key + "_sssp"][s].astype(np.float32))


@pytest.mark.skipif(not oracle.ref_available(), reason="reference CPU driver not built")
def test_sssp_f32_fractional_weights_match_reference_ssspCPU(ctx, rmat14):
    """Non-integral float weights: the fixed point of float min-plus relaxation does not
    depend on the order relaxations land, so the GPU result equals the reference's own
    ssspCPU (label-correcting priority queue, src/testSssp.cpp:33-115) bit for bit."""
    import torch

    g, _, src = rmat14
    rows = np.repeat(np.arange(g.m), np.diff(g.row_ptr))
    lo, hi = np.minimum(rows, g.col_ind), np.maximum(rows, g.col_ind)
    w = (((lo * 7919 + hi * 104729) % 1000) / 97.0 + 0.01).astype(np.float32)  # symmetric
    dg = ap.DeviceGraph(ap.HostGraph(g.m, g.n, g.row_ptr, g.col_ind, w, True))
    out = torch.empty(g.m, dtype=torch.float32, device="cuda")
    ctx.sssp_f32_into(dg, src, out, unreached=-1.0)
    ref, _ = oracle.ref_sssp_f32(g.row_ptr, g.col_ind, w, src)
    np.testing.assert_array_equal(out.cpu().numpy(), ref)


def test_sssp_f32_unreached_value(ctx):
    import torch

    rp = np.array([0, 1, 2, 2], dtype=np.int32)
    ci = np.array([1, 0], dtype=np.int32)
    w = np.array([0.5, 0.5], dtype=np.float32)
    dg = ap.DeviceGraph(ap.HostGraph(3, 3, rp, ci, w, True))
    out = torch.empty(3, dtype=torch.float32, device="cuda")
    ctx.sssp_f32_into(dg, 0, out, unreached=1.70141e38)
    np.testing.assert_array_equal(out.cpu().numpy(), np.array([0.0, 0.5, 1.70141e38], dtype=np.float32))


def test_mis_int32_layout(ctx, rmat14):
    import torch

    g, dg, _ = rmat14
    pr = ap.mt19937_u32(4, g.m)
    out = torch.empty(g.m, dtype=torch.int32, device="cuda")
    ctx.mis_int32_into(dg, torch.from_numpy(pr.view(np.int32)).cuda(), out)
    np.testing.assert_array_equal(out.cpu().numpy(), oracle.mis_greedy(g.row_ptr, g.col_ind, pr).astype(np.int32))


@pytest.mark.parametrize("prio", ["up", "down", "random"])
@pytest.mark.parametrize("shape", ["complete 2", "complete 33", "complete 140", "complete 1030", "complete 2100",
                                   "even 4735", "even 4737", "even 23679", "even 47361", "even 94721"])
def test_mis_dense_graphs_and_small_tiles(ctx, shape, prio):
    """Vertices that a push puts out while a warp or the block still scans their rows (complete graphs: a
    warp's step and more, more than a warp takes), and vertices around the sizes at which tiles shrink."""
    import torch

    kind, _, size = shape.partition(" ")
    m = int(size)
    if kind == "complete":
        src, dst = np.repeat(np.arange(m), m), np.tile(np.arange(m), m)
    else:
        rng = np.random.default_rng(6)
        src, dst = rng.integers(0, m, 5 * m), rng.integers(0, m, 5 * m)
    edges = np.unique(np.concatenate((src * m + dst, dst * m + src))[np.concatenate((src, src)) != np.concatenate((dst, dst))])
    rp = np.concatenate(([0], np.cumsum(np.bincount(edges // m, minlength=m)))).astype(np.int32)
    ci = (edges % m).astype(np.int32)
    pr = {"up": np.arange(m), "down": np.arange(m)[::-1], "random": ap.mt19937_u32(7, m)}[prio].astype(np.uint32)
    dg = ap.DeviceGraph(ap.HostGraph(m, m, rp, ci, None, True))
    ref = oracle.mis_greedy(rp, ci, pr)
    dpr = torch.from_numpy(pr.view(np.int32)).cuda()
    for _ in range(3):
        np.testing.assert_array_equal(ctx.mis(dg, dpr).cpu().numpy(), ref)


@pytest.mark.parametrize("prio", ["up", "down", "random", "equal"])
@pytest.mark.parametrize("shape", ["path 700", "star 8", "star 9", "star 1024", "star 1025", "star 40000",
                                   "hubs 300", "loops", "m 255", "m 256", "m 257", "one vertex", "no edges"])
@pytest.mark.parametrize("grid", [1, 0])
def test_mis_scans_and_pushes(ctx, shape, prio, grid):
    """Scans and pushes that end in a thread, go on in a warp and in the block, and in several passes of
    the block; more of each in one block than its lists hold (a grid of one block); chains as long as the
    graph; ties; self-loops; vertices around a whole tile. The set is unique."""
    import torch

    kind, _, size = shape.partition(" ")
    rng = np.random.default_rng(5)
    if kind == "path":
        m = int(size)
        src, dst = np.arange(m - 1), np.arange(1, m)
    elif kind == "star":
        m = int(size) + 1
        src, dst = np.zeros(m - 1, np.int64), np.arange(1, m)
    elif kind == "hubs":
        k, m = int(size), 3000 + int(size)
        src, dst = np.repeat(np.arange(k), 3000), np.tile(np.arange(k, m), k)
    elif kind == "m":
        m = int(size)
        src, dst = rng.integers(0, m, 4 * m), rng.integers(0, m, 4 * m)
    elif kind == "loops":
        m = 600
        src = np.concatenate((np.arange(m), rng.integers(0, m, 2 * m)))
        dst = np.concatenate((np.arange(m), rng.integers(0, m, 2 * m)))
    else:
        m = 1 if kind == "one" else 300
        src = dst = np.zeros(0, np.int64)
    g = _csr(m, src, dst, True)
    pr = {"up": np.arange(m), "down": np.arange(m)[::-1], "random": rng.integers(0, 2**32, m),
          "equal": np.full(m, 7)}[prio].astype(np.uint32)
    out = torch.empty(m, dtype=torch.int32, device="cuda")
    ctx.set_max_grid(grid)
    try:
        ctx.mis_int32_into(ap.DeviceGraph(g), torch.from_numpy(pr.view(np.int32)).cuda(), out)
    finally:
        ctx.set_max_grid(0)
    np.testing.assert_array_equal(out.cpu().numpy(), oracle.mis_greedy(g.row_ptr, g.col_ind, pr).astype(np.int32))


def _csr(m, src, dst, symmetric):
    if symmetric:
        src, dst = np.concatenate((src, dst)), np.concatenate((dst, src))
    key = np.unique(src.astype(np.int64) * m + dst)
    rp = np.concatenate(([0], np.cumsum(np.bincount(key // m, minlength=m)))).astype(np.int32)
    return ap.HostGraph(m, m, rp, (key % m).astype(np.int32), None, symmetric)


@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("shape", ["star 127", "star 128", "star 129", "star 20000", "path", "dense", "hubs in a row",
                                   "comb", "one vertex", "no edges"])
def test_bfs_edge_queue_shapes(ctx, shape, symmetric):
    """Rows that fill, just miss and cross an edge queue's 128-edge units and a warp's staging
    buffer; a row of many units shared among lanes; a frontier of one entry per level; units of
    more than a tile (mean degree above 128); rows without entries in the frontier; rows that a
    pull level's lanes hand over to their warp. Push only, pull wherever allowed, and both."""
    rng = np.random.default_rng(11)
    if shape.startswith("star"):
        k = int(shape.split()[1])
        m, src, dst = k + 40, np.zeros(k, dtype=np.int64), np.arange(1, k + 1)
    elif shape == "path":
        m = 150
        src, dst = np.arange(m - 1), np.arange(1, m)
    elif shape == "dense":
        m = 300
        src, dst = np.nonzero(~np.eye(m, dtype=bool))
    elif shape == "hubs in a row":  # vertex 0 leads to 200 vertices of 900 to 1,100 edges each
        m = 6000
        deg = rng.integers(900, 1100, 200)
        src = np.concatenate((np.zeros(200, dtype=np.int64), np.repeat(np.arange(1, 201), deg)))
        dst = np.concatenate((np.arange(1, 201), rng.integers(0, m, deg.sum())))
    elif shape == "comb":  # long rows whose only visited vertex comes last
        m = 3000
        src = np.concatenate((np.full(40, m - 1), np.repeat(np.arange(40), 70)))
        dst = np.concatenate((np.arange(40), 40 + rng.integers(0, 2000, 2800)))
    else:
        m = 1 if shape == "one vertex" else 70
        src = dst = np.zeros(0, dtype=np.int64)
    g = _csr(m, src[src != dst], dst[src != dst], symmetric)
    dg = ap.DeviceGraph(g)
    sources = {0, m - 1, m // 2}
    try:
        for alpha, beta in ((14.0, 24.0), (0.0, 24.0), (1e9, 1e9), (1e9, 2.0)):
            ctx.set_bfs_tuning(alpha, beta)
            for s in sources:
                np.testing.assert_array_equal(ctx.bfs(dg, s).cpu().numpy(), oracle.bfs(g.row_ptr, g.col_ind, s),
                                              err_msg=f"alpha {alpha} beta {beta} source {s}")
    finally:
        ctx.set_bfs_tuning(14.0, 24.0)


@pytest.mark.parametrize("kind", ["i32", "f32"])
@pytest.mark.parametrize("shape", ["star 127", "star 128", "star 129", "star 20000", "path", "dense", "hubs in a row",
                                   "largest distances", "zero weights"])
def test_sssp_edge_queue_shapes(ctx, shape, kind):
    """Rows that fill, just miss and cross the edge queue's units, a row of many units, one
    entry an iteration, units of more than a tile; with the default band, narrow bands (most
    entries deferred), no band, and far piles; weights of 0 and distances up to 2^31 - 2."""
    rng = np.random.default_rng(5)
    if shape.startswith("star"):
        k = int(shape.split()[1])
        m, src, dst = k + 40, np.zeros(k, dtype=np.int64), np.arange(1, k + 1)
    elif shape in ("path", "largest distances"):
        m = 150
        src, dst = np.arange(m - 1), np.arange(1, m)
    elif shape == "dense":
        m = 300
        src, dst = np.nonzero(~np.eye(m, dtype=bool))
    elif shape == "hubs in a row":
        m = 6000
        deg = rng.integers(900, 1100, 200)
        src = np.concatenate((np.zeros(200, dtype=np.int64), np.repeat(np.arange(1, 201), deg)))
        dst = np.concatenate((np.arange(1, 201), rng.integers(0, m, deg.sum())))
    else:
        m = 2000
        src, dst = rng.integers(0, m, (2, 16000))
    g = _csr(m, src[src != dst], dst[src != dst], False)
    w = rng.integers(1, 256, g.nnz)
    if shape == "zero weights":
        w = rng.choice([0, 0, 1, 250], g.nnz)
    elif shape == "largest distances" and kind == "i32":
        w = np.full(g.nnz, (2 ** 31 - 2) // g.nnz)
        w[-1] += (2 ** 31 - 2) - w.sum()
    val = w.astype(np.int32) if kind == "i32" else (w / np.float32(7)).astype(np.float32)
    g = ap.HostGraph(m, m, g.row_ptr, g.col_ind, np.ascontiguousarray(val))
    dg = ap.DeviceGraph(g)
    import torch

    out = torch.empty(m, dtype=torch.int32 if kind == "i32" else torch.float32, device="cuda")
    run = ctx.sssp_into if kind == "i32" else ctx.sssp_f32_into
    if kind == "i32":
        ref = oracle.sssp(g.row_ptr, g.col_ind, g.val, 0)
    else:  # the least float32 sum over paths: relaxed to the fixed point, in any order
        rows = np.repeat(np.arange(m), np.diff(g.row_ptr))
        ref, old = np.full(m, np.inf, dtype=np.float32), None
        ref[0] = 0
        while old is None or not np.array_equal(ref, old):
            old = ref.copy()
            np.minimum.at(ref, g.col_ind, old[rows] + g.val)
        ref[np.isinf(ref)] = -1
    try:
        for band, delta in ((0, 0), (1, 0), (500, 0), (-1, 0), (-1, 50), (300, 40)):
            if delta and shape == "largest distances":
                continue  # 40 million advances of the far threshold: past the 4 m + 4096 steps a call may take
            ctx.set_sssp_band(band)
            ctx.set_sssp_delta(delta)
            run(dg, 0, out)
            np.testing.assert_array_equal(out.cpu().numpy(), ref, err_msg=f"band {band} delta {delta}")
    finally:
        ctx.set_sssp_band(0)
        ctx.set_sssp_delta(0)


def test_a_first_call_reserves_what_it_uses(ctx):
    """A new context's scratch: int arrays of m + 1 entries and two bitmaps, an eighth more as
    headroom. Six arrays for a BFS, seven for an SSSP, nine with far piles."""
    import torch

    m = 1 << 18
    rp = np.zeros(m + 1, dtype=np.int32)
    rp[1:] = 1
    g = ap.DeviceGraph(ap.HostGraph(m, m, rp, np.array([1], dtype=np.int32), np.array([3], dtype=np.int32)))

    def bound(lists):
        return (lists * 4 * (m + 1 + 64) + 2 * (m // 8 + 256)) * 9 // 8 + 4096

    for lists, call in ((6, lambda c: c.bfs(g, 0)), (7, lambda c: c.sssp(g, 0)),
                        (9, lambda c: (c.set_sssp_delta(5), c.sssp(g, 0))[1]),
                        (9, lambda c: (c.set_sssp_band(-1), c.sssp(g, 0))[1])):
        with ap.Context(0) as c:
            out = call(c).cpu().numpy()
            assert bound(lists - 1) < c.scratch_bytes() <= bound(lists), lists
            assert out[0] == 0 and out[1] in (1, 3) and (out[2:] == -1).all()


def _complete(m):
    ci = np.tile(np.arange(m, dtype=np.int32), m)
    rows = np.repeat(np.arange(m), m)
    keep = rows != ci
    rp = np.arange(m + 1, dtype=np.int32) * (m - 1)
    return rp, ci[keep], rows[keep]


@pytest.mark.parametrize("m", [2, 130, 1500])
def test_complete_graphs(ctx, m):
    """Many tiles of edges for each entry of a queue: hop counts, distances of one and of 40
    sources, by far piles too."""
    import torch

    rp, ci, rows = _complete(m)
    rng = np.random.default_rng(m)
    sym = rng.integers(1, 1000, (m, m))
    w = np.minimum(sym, sym.T)[rows, ci].astype(np.int32)
    g = ap.DeviceGraph(ap.HostGraph(m, m, rp, ci, w, True))
    assert (ctx.bfs(g, m // 2).cpu().numpy() == (np.arange(m) != m // 2)).all()
    want = oracle.sssp(rp, ci, w, m // 2)
    np.testing.assert_array_equal(ctx.sssp(g, m // 2).cpu().numpy(), want)
    with ap.Context(0) as c:
        c.set_sssp_delta(7)
        np.testing.assert_array_equal(c.sssp(g, m // 2).cpu().numpy(), want)
    src = rng.integers(0, m, 40).astype(np.int32)
    src[3] = m // 2
    got = ctx.sssp_batch(g, torch.from_numpy(src).cuda()).cpu().numpy()
    np.testing.assert_array_equal(got[3], want)
    np.testing.assert_array_equal(got[11], oracle.sssp(rp, ci, w, int(src[11])))


def test_complete_graph_takes_little_time(ctx):
    """The edges of a dense graph's frontier are shared out among all warps, however few vertices
    there are: 9M entries of 3,000 vertices."""
    import torch

    m = 3000
    rp, ci, _ = _complete(m)
    g = ap.DeviceGraph(ap.HostGraph(m, m, rp, ci, np.ones(ci.size, dtype=np.int32), True))
    out = torch.empty(m, dtype=torch.int32, device="cuda")
    for call, limit in ((ctx.bfs_into, 65.0), (ctx.sssp_into, 320.0)):
        us = []
        for _ in range(12):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            call(g, 1, out)
            b.record()
            torch.cuda.synchronize()
            us.append(a.elapsed_time(b) * 1e3)
        # 31 and 176 us; 97 and 457 with a unit of edges for each vertex
        assert min(us) < limit, us
