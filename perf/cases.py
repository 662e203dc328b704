"""Performance cases: the calls a program makes on this library, over the sizes it makes them at.

Every case is one public entry point on a graph that is resident in device memory. Graphs
are R-MAT (a, b, c, d = 0.57, 0.19, 0.19, 0.05: few rows of very high degree, many short
ones) or Erdos-Renyi with a fixed number of entries per row; `m` vertices (any number, not
only powers of two) and `ef` generated edges per vertex. The serving loop is not timed as
such: the launches it makes are the single-source and the batched calls listed here.
"""
import math

import numpy as np
import torch

import apspie_b200 as ap

RMAT_A, RMAT_B, RMAT_C = 0.57, 0.19, 0.19
DAMPING, TOL, MAX_ITER = 0.85, 1e-6, 100


def listed():
    return [
        # one hop-count query on a small graph: launch and level latency, nothing else
        {"name": "bfs_rmat14", "op": "bfs", "m": 1 << 14, "ef": 16},
        # one hop-count query on an ordinary graph
        {"name": "bfs_rmat20", "op": "bfs", "m": 1 << 20, "ef": 16},
        # one shortest-path query, int32 weights: the library's headline workload
        {"name": "sssp_rmat20_i32", "op": "sssp", "dtype": "i32", "m": 1 << 20, "ef": 16},
        # the same with float weights, on a smaller graph of ragged size
        {"name": "sssp_rmat300k_f32", "op": "sssp", "dtype": "f32", "m": 300007, "ef": 12},
        # maximal independent set under random priorities
        {"name": "mis_rmat20", "op": "mis", "m": 1 << 20, "ef": 16},
        # C = A * A of uniformly short rows (64 products each), caller-owned C
        {"name": "spgemm_er20_f32", "op": "spgemm", "kind": "er", "dtype": "f32", "m": 1 << 20, "ef": 8},
        # C = A * A of very uneven rows (every row length class), integer values, ragged size
        {"name": "spgemm_rmat9k_i32", "op": "spgemm", "kind": "rmat", "dtype": "i32", "m": 9001, "ef": 8},
        # triangles of a graph given as its strict lower triangle
        {"name": "tc_rmat18", "op": "tc", "m": 1 << 18, "ef": 16},
        # hop counts from many sources at once: few sources on a large graph
        {"name": "bfs_batch_rmat22_q32", "op": "bfs_batch", "m": 1 << 22, "ef": 16, "nq": 32},
        # distances from many sources at once: a batch that is no multiple of 32
        {"name": "sssp_batch_rmat19_q100", "op": "sssp_batch", "m": 1 << 19, "ef": 16, "nq": 100},
        # edge list -> deduplicated symmetric CSR with weights (loading a graph)
        {"name": "csr_build_rmat20", "op": "csr_build", "m": 1 << 20, "ef": 16},
        # PageRank of a directed graph (transpose, then dense-vector products), ragged size
        {"name": "pagerank_rmat700k", "op": "pagerank", "m": 700001, "ef": 16},
    ]


def _log_uniform(rng, lo, hi):
    """An integer between lo and hi, spread over its logarithm; mostly odd."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return v | 1 if rng.random() < 0.75 else v


def draw(rng):
    op = rng.choice(["bfs", "bfs", "sssp", "sssp", "mis", "spgemm", "spgemm", "tc", "bfs_batch", "sssp_batch",
                     "csr_build", "pagerank"])
    case = {"op": op}
    if op in ("bfs", "sssp", "mis", "csr_build"):
        case["m"] = _log_uniform(rng, 3000, 1 << 21)
        case["ef"] = rng.randint(6, 20)
    elif op == "tc":
        case["m"] = _log_uniform(rng, 3000, 1 << 19)
        case["ef"] = rng.randint(6, 20)
    elif op == "pagerank":
        case["m"] = _log_uniform(rng, 3000, 700000)
        case["ef"] = rng.randint(6, 16)
    elif op == "bfs_batch":
        case["nq"] = rng.randint(2, 512)
        case["m"] = _log_uniform(rng, 3000, min(1 << 22, (1 << 27) // case["nq"]))
        case["ef"] = rng.randint(6, 16)
    elif op == "sssp_batch":
        case["nq"] = rng.randint(2, 512)
        case["m"] = _log_uniform(rng, 3000, min(1 << 20, (1 << 25) // case["nq"]))
        case["ef"] = rng.randint(6, 16)
    else:
        case["kind"] = rng.choice(["er", "rmat"])
        er = case["kind"] == "er"
        case["m"] = _log_uniform(rng, 1000, (1 << 20) if er else 12000)
        case["ef"] = rng.randint(3, 9)
    if op in ("sssp", "spgemm"):
        case["dtype"] = rng.choice(["i32", "f32"])
    return case


# ---------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _rmat_edges(m, ef, gen):
    """m * ef R-MAT edges (int64 endpoints below m), repeats and self-loops included."""
    ne, bits = m * ef, max(1, (m - 1).bit_length())
    u = torch.zeros(ne, dtype=torch.int64, device="cuda")
    v = torch.zeros(ne, dtype=torch.int64, device="cuda")
    for _ in range(bits):
        r = torch.rand(ne, generator=gen, device="cuda")
        down = r >= RMAT_A + RMAT_B
        right = ((r >= RMAT_A) & ~down) | (r >= RMAT_A + RMAT_B + RMAT_C)
        u.mul_(2).add_(down)
        v.mul_(2).add_(right)
    if m != 1 << bits:
        u, v = (u * m) >> bits, (v * m) >> bits
    return u, v


def _relabelled(m, seed, *ids):
    """The vertices' numbers turned by an amount that the seed gives: another graph with the
    same number of entries, in the operand as in what is computed from it."""
    shift = (seed * 2654435761 + 12345) % m
    return [(x + shift) % m for x in ids]


def _row_ptr(rows, m):
    rp = torch.zeros(m + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(rows, minlength=m), 0, out=rp[1:])
    return rp.to(torch.int32)


def _values(dtype, n, gen, lo, hi):
    if dtype == "f32":
        return torch.rand(n, generator=gen, device="cuda") * (hi - lo) + lo
    return torch.randint(lo, hi + 1, (n,), generator=gen, device="cuda", dtype=torch.int32)


def _graph(m, rows, cols, val=None, symmetric=False):
    """Device CSR of entries sorted by (row, column)."""
    vt = ap.VAL_NONE if val is None else ap.VAL_F32 if val.dtype == torch.float32 else ap.VAL_I32
    return ap.DeviceGraph.from_tensors(m, m, _row_ptr(rows, m), cols.to(torch.int32), val, vt, symmetric)


def _row_of(g):
    """The row of each entry."""
    return torch.repeat_interleave(torch.arange(g.m, device="cuda"), torch.diff(g.row_ptr).long())


def _undirected(m, ef, gen, dtype=None):
    """Symmetric, deduplicated, loop-free R-MAT graph; edge weights (1..255) symmetric too."""
    u, v = _rmat_edges(m, ef, gen)
    key = torch.unique((torch.minimum(u, v) * m + torch.maximum(u, v))[u != v])
    del u, v
    lo, hi = key // m, key % m
    both, order = torch.sort(torch.cat([key, hi * m + lo]))
    w = None
    if dtype is not None:
        w = _values(dtype, lo.numel(), gen, 1, 255).repeat(2)[order]
    return _graph(m, both // m, both % m, w, symmetric=True)


def _directed(m, ef, gen):
    u, v = _rmat_edges(m, ef, gen)
    key = torch.unique((u * m + v)[u != v])
    return _graph(m, key // m, key % m)


def _lower(g):
    rows = _row_of(g)
    keep = g.col_ind < rows
    return _graph(g.m, rows[keep], g.col_ind[keep])


def _matrix(case, seed):
    """The operand of the matrix product: values in [-1, 1] or 1..8. The pattern is one per
    case, relabelled by the seed, so that C has as many entries whatever the seed."""
    m, ef, gen = case["m"], case["ef"], _generator(5)
    if case["kind"] == "er":
        rows = torch.arange(m, device="cuda").repeat_interleave(ef)
        cols = torch.randint(0, m, (m * ef,), generator=gen, device="cuda")
    else:
        g = _undirected(m, ef, gen)
        rows, cols = _row_of(g), g.col_ind.long()
    rows, cols = _relabelled(m, seed, rows, cols)
    key = torch.unique(rows * m + cols)
    val = _values(case["dtype"], key.numel(), _generator(seed), *((-1, 1) if case["dtype"] == "f32" else (1, 8)))
    return _graph(m, key // m, key % m, val)


def _sources(g, nq, gen):
    """nq vertices with edges (almost all of them in the largest component)."""
    some = torch.nonzero(torch.diff(g.row_ptr)).flatten()
    return some[torch.randint(0, some.numel(), (nq,), generator=gen, device="cuda")].to(torch.int32)


def prepare(case, seed):
    """Graph, sources, output buffers and the context that a program keeps for its calls."""
    op, m, ef, gen = case["op"], case["m"], case["ef"], _generator(seed)
    s = {"op": op, "ctx": ap.Context(0)}
    if op == "bfs":
        s["g"] = _undirected(m, ef, gen)
    elif op == "sssp":
        s["g"] = _undirected(m, ef, gen, case["dtype"])
        s["run"] = s["ctx"].sssp_into if case["dtype"] == "i32" else s["ctx"].sssp_f32_into
    elif op == "mis":
        s["g"] = _undirected(m, ef, gen)
        s["prio"] = torch.randint(-(1 << 31), 1 << 31, (m,), generator=gen, device="cuda", dtype=torch.int64).to(torch.int32)
        s["out"] = torch.empty(m, dtype=torch.uint8, device="cuda")
    elif op == "spgemm":
        s["g"] = _matrix(case, seed)
    elif op == "tc":
        s["g"] = _lower(_undirected(m, ef, gen))
    elif op in ("bfs_batch", "sssp_batch"):
        s["g"] = _undirected(m, ef, gen, None if op == "bfs_batch" else "i32")
        s["sources"] = _sources(s["g"], case["nq"], gen)
        s["out"] = torch.empty((case["nq"], m), dtype=torch.int32, device="cuda")
    elif op == "csr_build":
        # one edge set per case, relabelled and reordered by the seed: as many entries each time
        u, v = _relabelled(m, seed, *_rmat_edges(m, ef, _generator(2)))
        order = torch.randperm(m * ef, generator=gen, device="cuda")
        s["m"], s["src"], s["dst"] = m, u[order].to(torch.int32), v[order].to(torch.int32)
        s["w"] = _values("i32", m * ef, gen, 1, 255)
    elif op == "pagerank":
        s["g"] = _directed(m, ef, gen)
    if op in ("bfs", "sssp"):
        s["source"] = int(torch.argmax(torch.diff(s["g"].row_ptr)))
        s["out"] = torch.empty(m, dtype=torch.float32 if case.get("dtype") == "f32" else torch.int32, device="cuda")
    return s


class _Array:
    """Zero-copy view of an array that the library owns; keeps its owner alive."""

    def __init__(self, owner, ptr, n, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 3}


def run(s):
    op, ctx = s["op"], s["ctx"]
    if op == "bfs":
        ctx.bfs_into(s["g"], s["source"], s["out"])
        return s["out"]
    if op == "sssp":
        s["run"](s["g"], s["source"], s["out"])
        return s["out"]
    if op == "mis":
        ctx.mis_into(s["g"], s["prio"], s["out"])
        return s["out"]
    if op == "spgemm":
        return ctx.spgemm_two_step(s["g"], s["g"])
    if op == "tc":
        return ctx.tc(s["g"])
    if op == "bfs_batch":
        ctx.bfs_batch_into(s["g"], s["sources"], s["out"])
        return s["out"]
    if op == "sssp_batch":
        ctx.sssp_batch_into(s["g"], s["sources"], s["out"])
        return s["out"]
    if op == "csr_build":
        c = ctx.build_csr(s["m"], s["src"], s["dst"], s["w"],
                          ap.BUILD_SYMMETRIZE | ap.BUILD_DROP_SELF_LOOPS | ap.BUILD_DEDUP)
        return [torch.as_tensor(_Array(c, p, n, "<i4"), device="cuda")
                for p, n in ((c.C.row_ptr, c.m + 1), (c.C.col_ind, c.nnz), (c.C.val, c.nnz))]
    rank, _ = ctx.pagerank(s["g"], DAMPING, TOL, MAX_ITER)
    return rank


# ---------------------------------------------------------------- what a pass needs
def _entries(case):
    """Expected entries of the symmetric, deduplicated R-MAT graph."""
    m, ef = case["m"], case["ef"]
    return 2 * m * ef * (1 - min(0.6, 0.012 * ef * 2 ** (-(math.log2(m) - 14) / 4)))


def work(case):
    op, m, ef = case["op"], case["m"], case["ef"]
    if op == "bfs":
        return {"bytes": 4 * (m + 1) + 4 * _entries(case) + 4 * m, "flops": 0}
    if op == "sssp":
        return {"bytes": 4 * (m + 1) + 8 * _entries(case) + 4 * m, "flops": 0}
    if op == "mis":
        return {"bytes": 4 * (m + 1) + 4 * _entries(case) + 5 * m, "flops": 0}
    if op == "tc":
        return {"bytes": 4 * (m + 1) + 2 * _entries(case), "flops": 0}
    if op == "bfs_batch":
        return {"bytes": 4 * (m + 1) + 4 * _entries(case) + 4 * case["nq"] * (m + 1), "flops": 0}
    if op == "sssp_batch":
        return {"bytes": 4 * (m + 1) + 8 * _entries(case) + 4 * case["nq"] * (m + 1), "flops": 0}
    if op == "csr_build":
        return {"bytes": 12 * m * ef + 4 * (m + 1) + 8 * _entries(case), "flops": 0}
    if op == "pagerank":
        return {"bytes": 4 * (m + 1) + 4 * m * ef + 4 * m, "flops": 2 * m * ef}
    if case["kind"] == "er":
        return {"bytes": 2 * (4 * (m + 1) + 8 * m * ef) + 4 * (m + 1) + 8 * m * ef * ef, "flops": 2 * m * ef * ef}
    # sum of squared degrees of an R-MAT graph, and how full that leaves C
    nnz, products = _entries(case), 2.5 * (m * ef) ** 2 * 0.6352 ** math.log2(m)
    full = m * m * (1 - math.exp(-0.35 * products / (m * m)))
    return {"bytes": 2 * (4 * (m + 1) + 8 * nnz) + 4 * (m + 1) + 8 * full, "flops": 2 * products}


# ---------------------------------------------------------------- what a pass returns, in 64 bits
def _exact_sssp(s):
    g = s["g"]
    rows, cols, w = _row_of(g), g.col_ind.long(), g.val.double()
    dist = torch.full((g.m,), math.inf, dtype=torch.float64, device="cuda")
    dist[s["source"]] = 0
    while True:
        new = torch.scatter_reduce(dist, 0, cols, dist[rows] + w, "amin")
        if torch.equal(new, dist):
            return torch.where(torch.isinf(dist), -1.0, dist)
        dist = new


def _exact_spgemm(s):
    g = s["g"]
    rp, rows, cols, val = g.row_ptr.long(), _row_of(g), g.col_ind.long(), g.val.double()
    found = []
    for r0 in range(0, g.m, 1 << 17):  # rows of C, a part at a time
        e = slice(int(rp[r0]), int(rp[min(g.m, r0 + (1 << 17))]))
        n = (rp[1:] - rp[:-1])[cols[e]]
        entry = torch.repeat_interleave(torch.arange(e.start, e.stop, device="cuda"), n)
        first = torch.repeat_interleave(rp[cols[e]] - (torch.cumsum(n, 0) - n), n)
        other = first + torch.arange(entry.numel(), device="cuda")
        _, at = torch.unique(rows[entry] * g.n + cols[other], return_inverse=True)
        out = torch.zeros(int(at.max()) + 1 if at.numel() else 0, dtype=torch.float64, device="cuda")
        found.append(out.index_add_(0, at, val[entry] * val[other]))
    return [None, None, torch.cat(found)]


def _exact_pagerank(s):
    g = s["g"]
    rows, cols, n = _row_of(g), g.col_ind.long(), g.m
    deg = torch.diff(g.row_ptr).double()
    r = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    for _ in range(MAX_ITER):
        share = torch.where(deg > 0, r / deg.clamp(min=1), 0.0)
        pulled = torch.zeros_like(r).index_add_(0, cols, share[rows])
        new = (1 - DAMPING) / n + DAMPING * (pulled + r[deg == 0].sum() / n)
        change = float((new - r).abs().sum())
        r = new
        if change < TOL:
            break
    return r


def exact(case, seed):
    """The floating outputs in 64 bits (whole numbers have to be equal anyway)."""
    if case["op"] == "pagerank":
        found = _exact_pagerank(prepare(case, seed))
    elif case["op"] == "sssp" and case["dtype"] == "f32":
        found = _exact_sssp(prepare(case, seed))
    elif case["op"] == "spgemm" and case["dtype"] == "f32":
        found = _exact_spgemm(prepare(case, seed))
    else:
        return None
    if isinstance(found, list):
        return [None if x is None else np.asarray(x.cpu()) for x in found]
    return np.asarray(found.cpu())
