// Batched multi-source SSSP: many sources on one resident graph in ONE persistent launch.
//
// By default apspie_sssp_batch runs the multi-query kernel below: it reads each frontier
// row once for all of its changed queries and relaxes in label-correcting (Bellman-Ford)
// order. apspie_ctx_set_sssp_batch_groups(ctx, g > 0) runs the query groups of traverse.cu
// instead (g groups of blocks, each running the banded single-source SSSP on its share of
// the sources).
//
// Labels are vertex-major: the distances of one vertex for the 32 queries of word w sit in
// one 128-byte line, lab[(v * W + w) * 32 + q % 32]. Frontier entries are (vertex u, query
// word w) pairs whose "changed" bits (the queries whose distance at u dropped in the
// previous iteration) are non-zero. An iteration puts them on an edge queue (frontier.cuh)
// with their changed word, so that the edges are shared out evenly. A warp keeps its tile's
// edges as 16-byte records in shared memory and walks them four at a time, eight lanes to an
// edge, four queries to a lane: a lane reads 16 bytes of u's and of v's label line, relaxes
// nd = dist[q][u] + w(u,v) where q changed at u, and atomicMin's the label; the improved
// queries go into the record, a byte per lane, and at the end of the tile each lane ORs its
// own edges' into v's next changed word, enqueueing (v, w) on the first bit.
//
// What bounds it: instruction issue (half of the slots; 16 instructions a visit) and the
// latency of the label reads. 100 queries on R-MAT of 2^19 vertices (345M visits of a row's
// entry for a word): one edge at a time, a lane per query, 18.9 ms; four edges a step with
// their fields as records 12.9 ms (26.6 instructions a visit, half of them in the merge-path
// searches that shared out the edges); edge queue and improved queries as bytes instead of
// shuffles 10.3 ms; no branch around the label reads 9.3 ms; five blocks per SM instead of
// four 8.9 ms; warps taking their block's units in turn 8.0 ms. With a fixed share: one step in flight instead of two 10.0, four 9.5 ms; tiles of 32, 64 and 96
// edges 9.8, 8.9 and 9.4 ms. Bands of distances per query, also counted from each query's
// distance to the highest-degree vertex, and bounds by way of up to 32 such vertices spare
// relaxations but hardly any visits (5.5 to 18 a row's entry instead of 6.4): a visit serves
// all 32 queries of a word, and some of them want it in each iteration.
// Every query reaches the same label-correcting fixed point as apspie_sssp computes alone
// (exact shortest distances for non-negative integer weights). A last pass transposes the
// labels into the query-major output out[q * m + v] (0xFFFFFFFF, -1 as int32, unreached).
// Each launch serves at most 32 * W queries with (nnz + m) * W < 2^31 (int32 item counts).
#include <algorithm>
#include <cstring>

#include "frontier.cuh"

namespace apspie {
namespace {

constexpr int kSbBlock = 256;
constexpr int kSbVT = 4;
constexpr int kSbTile = 32 * kSbVT;
constexpr int kSbSteps = 2;  // steps of four edges whose label reads a warp issues together
constexpr int kSbPA = 4;  // entries a thread takes off the queue together
constexpr int kSbQCap = 128;
// every edge of a tile is visited exactly once
static_assert(kSbTile % (4 * kSbSteps) == 0, "the steps must divide the tile");
using SbWQ = WarpQueue<kSbQCap>;

enum : int { kSiteSb = 500, kSiteSbNeg = 501, kSiteSbOverflow = 502, kSiteSbCap = 503, kSiteSbBadSource = 504 };

// Bit of a query in the words that say which queries changed: its label's place in the 128-byte
// line is 4 l + c (lane l of the eight at an edge, component c), and the lanes' four bits are
// stored as bytes and folded, l and l + 4 into the same byte.
__device__ __forceinline__ int sb_shift(int l) { return ((l & 3) << 3) | ((l >> 2) << 2); }
__device__ __forceinline__ unsigned sb_bit(int q) { return 1u << (sb_shift((q & 31) >> 2) + (q & 3)); }

struct SbArgs {
    int m, nnz, nq, W, shift;
    const int *__restrict__ row_ptr;
    const int *__restrict__ col_ind;
    const int *__restrict__ wt;
    const int *__restrict__ srcs;
    unsigned *lab;         // m x W x 32 labels, vertex-major, pre-filled with 0xFFFFFFFF
    unsigned *chg;         // m x W changed-query words
    int *q;                // frontier: u * W + w of the non-zero ones
    uint2 *ent;            // the edge queue's entries: u * W + w and its changed word
    int *off, *delta, *owner;
    TravCtl *ctl;
    int *sticky;
};

struct SbShared {
    union {
        int slice[kSbBlock / 32][3 * kSbTile];  // edge_expand's
        unsigned long long scan[33];            // phase A's
    };
    uint4 rec[kSbBlock / 32][kSbTile];
    int qbuf[kSbBlock / 32][kSbQCap];
    unsigned long long abase;
    int claim[2];  // units taken, by iteration parity
};

__global__ void __launch_bounds__(kSbBlock, 5) sssp_batch_kernel(SbArgs a) {
    __shared__ __align__(16) SbShared sh;
    grid_begin(a.ctl);
    const int G = gridDim.x;
    const int gtid = blockIdx.x * kSbBlock + threadIdx.x;
    const int gstride = G * kSbBlock;
    const int m = a.m, W = a.W;
    const long long mw = static_cast<long long>(m) * W;
    const int wid = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    for (long long i = gtid; i < mw; i += gstride) a.chg[i] = 0u;
    if (threadIdx.x < 2) sh.claim[threadIdx.x] = 0;
    if (gtid == 0) {
        a.ctl->qlen[0] = a.ctl->qlen[1] = 0;
        a.ctl->rcnt64[0] = a.ctl->rcnt64[1] = 0ull;
    }
    if (!grid_barrier(a.ctl, a.sticky, kSiteSb)) return;
    {
        SbWQ wq(sh.qbuf[wid], a.q, &a.ctl->qlen[0]);
        for (int base = blockIdx.x * kSbBlock; base < a.nq; base += gstride) {
            const int qi = base + threadIdx.x;
            bool fresh = false;
            int e = 0;
            if (qi < a.nq) {
                const int v = a.srcs[qi];
                if (v < 0 || v >= m) {  // reported; the barrier below then ends the launch
                    raise_error(a.ctl, a.sticky, APSPIE_ERR_INVALID_ARG, kSiteSbBadSource);
                } else {
                    e = v * W + (qi >> 5);
                    a.lab[static_cast<size_t>(e) * 32 + (qi & 31)] = 0u;
                    fresh = atomicOr(a.chg + e, sb_bit(qi)) == 0u;
                }
            }
            wq.push(fresh, e);
        }
        wq.flush();
    }
    if (!grid_barrier(a.ctl, a.sticky, kSiteSb + 10)) return;

    int cur = 0, iters = 0;
    long long relaxed = 0;
    for (;;) {
        const int nf = ld_volatile_i32(&a.ctl->qlen[cur]);
        if (nf == 0) break;
        if (iters > m + 1) {
            if (gtid == 0) raise_error(a.ctl, a.sticky, APSPIE_ERR_NOT_CONVERGED, kSiteSbCap);
            break;
        }
        // phase A: take each entry's changed word (and clear it for reuse) and put the entry on
        // the iteration's edge queue
        unsigned long long *asize = a.ctl->rcnt64 + (iters & 1);
        {
            const int C = (nf + G - 1) / G;
            const int c0 = min(static_cast<int>(blockIdx.x) * C, nf);
            const int c1 = min(c0 + C, nf);
            for (int base = c0; base < c1; base += kSbBlock * kSbPA) {
                int e[kSbPA], r0[kSbPA], deg[kSbPA];
                unsigned bits[kSbPA];
#pragma unroll
                for (int k = 0; k < kSbPA; ++k) {
                    const int i = base + k * kSbBlock + threadIdx.x;
                    e[k] = i < c1 ? __ldcg(a.q + i) : -1;
                }
                int sum = 0, cnt = 0;
#pragma unroll
                for (int k = 0; k < kSbPA; ++k) {
                    r0[k] = deg[k] = 0;
                    bits[k] = 0u;
                    if (e[k] >= 0) {
                        const int u = e[k] / W;
                        bits[k] = __ldcg(a.chg + e[k]);
                        r0[k] = __ldg(a.row_ptr + u);
                        deg[k] = __ldg(a.row_ptr + u + 1) - r0[k];
                    }
                }
#pragma unroll
                for (int k = 0; k < kSbPA; ++k) {
                    if (e[k] >= 0) a.chg[e[k]] = 0u;
                    sum += deg[k];
                    cnt += deg[k] > 0;
                }
                const unsigned long long mine = (static_cast<unsigned long long>(cnt) << 32) | static_cast<unsigned>(sum);
                const unsigned long long incl = block_inclusive_scan_u64<kSbBlock>(mine, sh.scan);
                if (threadIdx.x == 0 && sh.scan[32]) sh.abase = atomicAdd(asize, sh.scan[32]);
                __syncthreads();
                const unsigned long long at = sh.abase + incl - mine;
                int idx = static_cast<int>(at >> 32), off = static_cast<int>(at & 0xffffffffull);
#pragma unroll
                for (int k = 0; k < kSbPA; ++k) {
                    const bool some = deg[k] > 0;
                    eq_write(a.off, a.delta, a.owner, a.shift, some, idx, off, r0[k], deg[k]);
                    if (some) a.ent[idx] = make_uint2(static_cast<unsigned>(e[k]), bits[k]);
                    idx += some;
                    off += deg[k];
                }
                __syncthreads();  // the scan's words and the base are reused by the next step
            }
        }
        if (!grid_barrier(a.ctl, a.sticky, kSiteSb + 1)) return;
        // the queue has been read: phase B fills it again, and counts in the other length
        const unsigned long long asz = __ldcg(asize);
        const int ne = static_cast<int>(asz >> 32), E = static_cast<int>(asz & 0xffffffffull);
        if (gtid == 0) {
            a.ctl->qlen[cur] = 0;
            a.ctl->rcnt64[(iters & 1) ^ 1] = 0ull;
        }
        ++iters;
        relaxed += E;
        if (threadIdx.x == 0) sh.claim[(iters & 1) ^ 1] = 0;
        SbWQ wq(sh.qbuf[wid], a.q, &a.ctl->qlen[cur ^ 1]);
        const int *col = a.col_ind;
        const int *wt = a.wt;
        unsigned *lab = a.lab;
        unsigned *chg = a.chg;
        uint4 *rec = sh.rec[wid];
        TravCtl *ctl = a.ctl;
        int *sticky = a.sticky;
        EdgeQueue qe{a.off, a.delta, a.owner, nullptr, nullptr};
        edge_expand<kSbVT, true>(
            qe, a.ent, ne, E, a.shift, sh.slice[wid], &sh.claim[iters & 1], blockIdx.x, G,
            [&](const bool (&valid)[kSbVT], const uint2 (&src)[kSbVT], const int (&idx)[kSbVT]) {
                // the tile's edges as records: target entry (v, w), weight + 1, source entry and
                // its changed queries; the improved queries replace the last two, a byte per lane
                int ned = 0, tv[kSbVT];
                int v[kSbVT], we[kSbVT];
#pragma unroll
                for (int r = 0; r < kSbVT; ++r) {
                    v[r] = valid[r] ? __ldg(col + idx[r]) : 0;
                    we[r] = valid[r] ? __ldg(wt + idx[r]) : 0;
                }
#pragma unroll
                for (int r = 0; r < kSbVT; ++r) {
                    const unsigned e = src[r].x;
                    unsigned bits = src[r].y;
                    tv[r] = v[r] * W + static_cast<int>(e - (e / static_cast<unsigned>(W)) * static_cast<unsigned>(W));
                    if (we[r] < 0) {  // reported once here; the edge is then left out
                        raise_error(ctl, sticky, APSPIE_ERR_INVALID_ARG, kSiteSbNeg);
                        bits = 0u;
                    }
                    rec[r * 32 + lane] =
                        make_uint4(static_cast<unsigned>(tv[r]), static_cast<unsigned>(we[r]) + 1u, e, bits);
                    ned += __popc(__ballot_sync(0xffffffffu, valid[r]));
                }
                __syncwarp();
                // four edges a step, eight lanes each, four queries (16 bytes of the label line) a lane
                const int sub = lane & 7, grp = lane >> 3, sub4 = 4 * sub, shift = sb_shift(sub);
                bool over = false;
#pragma unroll 1
                for (int l0 = 0; l0 < ned; l0 += 4 * kSbSteps) {
                    uint4 du[kSbSteps], dv[kSbSteps];
                    unsigned *lv[kSbSteps];
                    unsigned act[kSbSteps], w1[kSbSteps];
#pragma unroll
                    for (int t = 0; t < kSbSteps; ++t) {
                        const uint4 e = rec[l0 + 4 * t + grp];
                        act[t] = (e.w >> shift) & 15u;
                        w1[t] = e.y;
                        lv[t] = lab + static_cast<size_t>(e.x) * 32 + sub4;
                        // through L1 (a row's edges all read the same source line, and many edges the
                        // lines of high-degree targets), by all lanes (of the lanes with no query to
                        // relax, one in twelve, a branch costs more than the reads). u's labels: one
                        // lowered in this iteration has its change bit set for the next, so any value
                        // since the barrier will do. v's: a stale, larger value only costs an atomic
                        // and one more expansion of v's query
                        du[t] = *reinterpret_cast<const uint4 *>(lab + static_cast<size_t>(e.z) * 32 + sub4);
                        dv[t] = *reinterpret_cast<const uint4 *>(lv[t]);
                    }
                    __syncwarp();  // the records are read: their last halves take the results
                    // an improvement over the label just read is reported without waiting for the
                    // atomic's old value: if another edge lowered the label further meanwhile, v's
                    // query is only re-expanded once more (same values)
#pragma unroll
                    for (int t = 0; t < kSbSteps; ++t) {
                        // s = candidate + 1. An active label is finite (< 2^31 - 1) and the weight
                        // non-negative, so s does not wrap, and s > 2^31 - 1 is an overflow; an
                        // inactive, unreached label wraps to the weight, below that
                        const unsigned s0 = du[t].x + w1[t], s1 = du[t].y + w1[t];
                        const unsigned s2 = du[t].z + w1[t], s3 = du[t].w + w1[t];
                        if (static_cast<int>(s0 | s1 | s2 | s3) < 0) {
                            const unsigned big = (s0 >> 31) | ((s1 >> 31) << 1) | ((s2 >> 31) << 2) | ((s3 >> 31) << 3);
                            over |= (big & act[t]) != 0u;
                            act[t] &= ~big;
                        }
                        const unsigned imp = ((s0 <= dv[t].x ? 1u : 0u) | (s1 <= dv[t].y ? 2u : 0u) |
                                              (s2 <= dv[t].z ? 4u : 0u) | (s3 <= dv[t].w ? 8u : 0u)) &
                                             act[t];
                        if (imp) {
                            if (imp & 1u) atomicMin(lv[t], s0 - 1u);
                            if (imp & 2u) atomicMin(lv[t] + 1, s1 - 1u);
                            if (imp & 4u) atomicMin(lv[t] + 2, s2 - 1u);
                            if (imp & 8u) atomicMin(lv[t] + 3, s3 - 1u);
                        }
                        reinterpret_cast<unsigned char *>(&rec[l0 + 4 * t + grp].z)[sub] = static_cast<unsigned char>(imp);
                    }
                }
                if (over) raise_error(ctl, sticky, APSPIE_ERR_INVALID_ARG, kSiteSbOverflow);
                __syncwarp();
#pragma unroll
                for (int r = 0; r < kSbVT; ++r) {
                    // improved queries of this lane's edge r (a slot without an edge was either not
                    // visited or has none)
                    const uint4 e = rec[r * 32 + lane];
                    const unsigned mine = valid[r] ? e.z | (e.w << 4) : 0u;
                    bool fresh = false;
                    if (mine) fresh = atomicOr(chg + tv[r], mine) == 0u;
                    wq.push(fresh, tv[r]);
                }
            });
        wq.flush();
        if (!grid_barrier(a.ctl, a.sticky, kSiteSb + 2)) return;
        cur ^= 1;
    }
    if (gtid == 0) {
        a.ctl->iterations = iters;
        a.ctl->push_iterations = iters;
        a.ctl->edges_expanded = relaxed;
    }
}

// Labels (vertex-major, 32 queries per line) -> query-major rows out[q * m + v], one
// 32-vertex x 32-query tile at a time through shared memory (both sides coalesced).
__global__ void __launch_bounds__(256) sb_unpack(const unsigned *__restrict__ lab, int m, int W, int nq,
                                                 unsigned *out) {
    __shared__ unsigned t[32][33];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const long long ntiles = static_cast<long long>((m + 31) / 32) * W;
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int vb = static_cast<int>(tile / W) * 32;
        const int w = static_cast<int>(tile % W);
        for (int i = wid; i < 32; i += 8) {
            const int v = vb + i;
            t[i][lane] = v < m ? __ldcs(lab + (static_cast<size_t>(v) * W + w) * 32 + lane) : 0u;
        }
        __syncthreads();
        for (int i = wid; i < 32; i += 8) {
            const int q = w * 32 + i;
            if (q < nq && vb + lane < m) out[static_cast<size_t>(q) * m + vb + lane] = t[lane][i];
        }
        __syncthreads();
    }
}

}  // namespace

// Scratch of a launch on mw (vertex, query word) pairs and so many entries of their rows.
static size_t multi_need(size_t mw, long long edges) {
    return Carver::need({mw * 128, mw * 4, mw * 4, mw * 8, mw * 4, mw * 4,
                         static_cast<size_t>(edge_owner_slots(static_cast<long long>(mw) + 1, edges)) * 4});
}

size_t sssp_batch_scratch_need(int m, long long nnz, int nq) {
    const int W = ((nq < 512 ? nq : 512) + 31) / 32;
    const size_t mw = static_cast<size_t>(m) * (W > 0 ? W : 1);
    const size_t multi =
        multi_need(mw, nnz * (W > 0 ? W : 1));
    // the grouped form (groups > 0): at most 4 groups are costed here
    const size_t grouped = sssp_group_scratch_need(m, nnz, std::max(1, std::min(nq, 4)));
    return std::max(multi, grouped);
}

}  // namespace apspie

using namespace apspie;

extern "C" apspie_status apspie_sssp_batch(apspie_ctx *ctx, const apspie_csr *A, const int32_t *d_sources,
                                           int32_t num_sources, int32_t *d_dists, apspie_run_stats *stats) {
    if (!ctx) return APSPIE_ERR_INVALID_ARG;
    cudaSetDevice(ctx->device);
    apspie_status st = check_csr_view(ctx, A, "apspie_sssp_batch");
    if (st != APSPIE_OK) return st;
    if (A->m != A->n || A->m <= 0)
        return set_error(ctx, APSPIE_ERR_INVALID_ARG, "apspie_sssp_batch: square, non-empty graph required");
    if (A->val_type != APSPIE_VAL_I32 || (A->nnz > 0 && !A->val))
        return set_error(ctx, APSPIE_ERR_INVALID_ARG, "apspie_sssp_batch: int32 edge weights required");
    if (num_sources < 0 || (num_sources > 0 && (!d_sources || !d_dists)))
        return set_error(ctx, APSPIE_ERR_INVALID_ARG, "apspie_sssp_batch: bad sources/output");
    if (ctx->validate && (st = validate_csr(ctx, A, true)) != APSPIE_OK) return st;
    if (ctx->sssp_batch_groups > 0) return sssp_batch_grouped(ctx, A, d_sources, num_sources, d_dists, stats);
    const int m = A->m;
    // queries per launch: W words with (nnz + m) * W below 2^31 (int32 item counts)
    long long wmax = 0x7fffffffLL / (static_cast<long long>(A->nnz) + m + 1);
    if (wmax > 16) wmax = 16;
    if (wmax < 1) return set_error(ctx, APSPIE_ERR_UNSUPPORTED, "apspie_sssp_batch: graph too large");
    const int per_launch = static_cast<int>(32 * wmax);
    if (stats) std::memset(stats, 0, sizeof(*stats));
    for (int q0 = 0; q0 < num_sources; q0 += per_launch) {
        const int nq = std::min(per_launch, num_sources - q0);
        const int W = (nq + 31) / 32;
        const size_t mw = static_cast<size_t>(m) * W;
        void *base;
        st = scratch_reserve(
            ctx, multi_need(mw, static_cast<long long>(A->nnz) * W),
            &base);
        if (st != APSPIE_OK) return st;
        Carver c(base);
        SbArgs a;
        a.lab = c.take<unsigned>(mw * 32);
        a.chg = c.take<unsigned>(mw);
        a.q = c.take<int>(mw);
        a.ent = c.take<uint2>(mw);
        a.off = c.take<int>(mw);
        a.delta = c.take<int>(mw);
        const long long slots = edge_owner_slots(static_cast<long long>(mw) + 1, static_cast<long long>(A->nnz) * W);
        a.owner = c.take<int>(static_cast<size_t>(slots));
        a.shift = edge_unit_shift(static_cast<long long>(A->nnz) * W, slots, kSbTile);
        a.m = m;
        a.nnz = A->nnz;
        a.nq = nq;
        a.W = W;
        a.row_ptr = A->row_ptr;
        a.col_ind = A->col_ind;
        a.wt = static_cast<const int *>(A->val);
        a.srcs = d_sources + q0;
        a.ctl = ctx->d_ctl;
        a.sticky = ctx->d_sticky_err;
        cudaError_t e = cudaMemsetAsync(a.lab, 0xff, mw * 32 * sizeof(unsigned), ctx->stream);
        if (e != cudaSuccess) return cuda_error(ctx, e, "apspie_sssp_batch reset");
        if ((st = reset_ctl(ctx)) != APSPIE_OK) return st;
        void *args[] = {&a};
        st = launch_persistent(ctx, reinterpret_cast<const void *>(sssp_batch_kernel), kSbBlock, args, 1LL << 40);
        if (st != APSPIE_OK) return st;
        const long long tiles = static_cast<long long>((m + 31) / 32) * W;
        const int ublocks = static_cast<int>(std::min<long long>(tiles, ctx->num_sms * 16LL));
        sb_unpack<<<ublocks, 256, 0, ctx->stream>>>(
            a.lab, m, W, nq, reinterpret_cast<unsigned *>(d_dists + static_cast<size_t>(q0) * m));
        if ((e = cudaGetLastError()) != cudaSuccess) return cuda_error(ctx, e, "apspie_sssp_batch unpack");
        if (stats) {
            apspie_run_stats part;
            if ((st = finish_call(ctx, &part, "apspie_sssp_batch")) != APSPIE_OK) return st;
            stats->iterations += part.iterations;
            stats->push_iterations += part.push_iterations;
            stats->edges_expanded += part.edges_expanded;
        }
    }
    return APSPIE_OK;
}
