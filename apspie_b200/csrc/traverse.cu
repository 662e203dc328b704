// Persistent SpMSpV traversal kernels: BFS (boolean OR-AND), SSSP (min-plus), MIS
// (priority max), and the one-hop boolean SpMSpV.
//
// Each algorithm is ONE cooperative launch whose blocks loop over levels/iterations with
// a bounded grid barrier between phases; the host never reads a count mid-run. This
// replaces the reference's host-driven level loops (src/bfs.cuh:87-110,
// src/spmspvBfs.cuh:174-222, src/sssp.cuh:79-98, src/spmspvMis.cuh:232-318), which issue
// ~10-14 launches, up to 3 device->host syncs and a cudaMalloc/cudaFree per level, and
// which stop after a caller-supplied `depth` taken from the CPU BFS.
#include <cstdio>
#include <cstring>
#include <mutex>

#include "frontier.cuh"

namespace apspie {

namespace {

constexpr int kBlock = 256;
constexpr int kSsspVT = 4;  // edges per lane of a tile
constexpr int kSsspPA = 4;  // frontier entries per thread per phase-A step
constexpr int kQCap = 128;  // per-warp queue staging (see WarpQueue)
using WQ = WarpQueue<kQCap>;

constexpr int kInf = 0x7fffffff;

// device error sites (reported as err_where)
enum : int {
    kSiteBfs = 100,
    kSiteSssp = 200,
    kSiteSsspNegWeight = 201,
    kSiteSsspOverflow = 202,
    kSiteSsspIterCap = 203,
    kSiteSsspBarA = 210,
    kSiteSsspBarB = 211,
    kSiteSsspBarF0 = 212,
    kSiteSsspBarF1 = 213,
    kSiteSsspGroup = 214,  // and 215
    kSiteSsspBadSource = 216,
    kSiteMis = 300,
    kSiteMisRoundCap = 301,
};

struct TravBuffers {
    int *q0, *q1, *q2, *q3, *rs, *loc_off, *aux, *aux2, *aux3;
    unsigned *bits0, *bits1;
};

size_t trav_scratch_bytes(int m) {
    const size_t words = (static_cast<size_t>(m) + 31) / 32;
    const size_t mi = static_cast<size_t>(m) + 1;
    return Carver::need({mi * 4, mi * 4, mi * 4, mi * 4, mi * 4, mi * 4, mi * 4, mi * 4, mi * 4, words * 4, words * 4});
}

TravBuffers carve_trav(void *base, int m) {
    const size_t words = (static_cast<size_t>(m) + 31) / 32;
    const size_t mi = static_cast<size_t>(m) + 1;
    Carver c(base);
    TravBuffers b;
    b.q0 = c.take<int>(mi);
    b.q1 = c.take<int>(mi);
    b.q2 = c.take<int>(mi);
    b.q3 = c.take<int>(mi);
    b.rs = c.take<int>(mi);
    b.loc_off = c.take<int>(mi);
    b.aux = c.take<int>(mi);
    b.aux2 = c.take<int>(mi);
    b.aux3 = c.take<int>(mi);
    b.bits0 = c.take<unsigned>(words);
    b.bits1 = c.take<unsigned>(words);
    return b;
}

// BFS's view of the buffers: edge queues in q0-q3, rs and loc_off, visited bitmaps in bits0-1.
struct BfsArgs;
void set_bfs_buffers(BfsArgs &a, const TravBuffers &b, int m, int nnz);

// ================================================================================
// BFS
// ================================================================================
constexpr int kBfsBlock = 256;
constexpr int kPullSteps = 4;  // steps of four neighbours a lane scans alone in a pull level

struct BfsArgs {
    int m, nnz, src, depth_cap;
    const int *__restrict__ row_ptr;
    const int *__restrict__ col_ind;
    int *depth;
    EdgeQueue q[2];     // by level parity (size and empty are slots of the control block)
    unsigned *vis[2];   // visited bitmap; a pull level reads one and writes the other
    int shift;          // edges per queue unit: 1 << shift
    TravCtl *ctl;
    int *sticky;
    float alpha, beta;
    int allow_pull;  // pattern declared symmetric
};

// Level-synchronous BFS, one grid barrier per level. Level L discovers the vertices at hop
// distance L.
//  push (top-down): the frontier is an edge queue; a neighbour is claimed by an atomicOr
//      test-and-set on the visited bitmap (the dedup that replaces the reference's radix
//      sort, src/spmspvBfs.cuh:195-197), its depth written, and it is appended to the next
//      queue.
//  pull (bottom-up): one warp per 32-vertex bitmap word; each unvisited vertex scans its
//      row until it meets a visited vertex. That vertex is in the frontier: had it been
//      visited a level earlier, its neighbour here would be visited too. So the visited
//      bitmap as it was at the level's start is all that a pull level reads (through L1; it
//      writes the next bitmap into the other buffer), and no frontier bitmap is kept. A lane
//      scans its row alone for kPullSteps steps of four neighbours; what is left of longer
//      rows the warp scans together.
// The direction follows Beamer's rule on the edges out of the frontier (m_f) against the
// edges still unexplored (m_u): push->pull when m_f > m_u/alpha, pull->push when the
// frontier holds fewer than m/beta vertices; and m_f > nnz/(8 alpha), so that the last small
// frontiers, when hardly any edge is left unexplored, don't read every row that is left (a
// pull level of 9 us in place of a push level of 6 us at scale 20). Depth results do not
// depend on the choice.
//
// What bounds it: at scale 14 the chain of dependent L2 reads in a level (queue, entry,
// column, visited word, claim, row length, reservation) and its barrier; at scale 20 the pull
// levels' gathers. Kernel time at scale 14 / 20 with a phase that scanned the frontier's row
// lengths, two barriers a level and frontier bitmaps: 43.9 / 113 us; now 31 / 63 us. Blocks
// of 256 threads, three an SM: four an SM 36 / 65 us, 512 threads 38 / 65 us, 128 threads
// 34 / 68 us (fewer blocks make the barrier cheaper, more warps the pull levels).
__global__ void __launch_bounds__(kBfsBlock, 3) bfs_kernel(BfsArgs a) {
    __shared__ int s_buf[kBfsBlock / 32][kEqCap];
    __shared__ int s_slice[kBfsBlock / 32][kEqTile];
    __shared__ EqBlock<kBfsBlock> s_blk;
    grid_begin(a.ctl);
    if (threadIdx.x == 0) s_blk.empty = 0;
    const int gtid = blockIdx.x * kBfsBlock + threadIdx.x;
    const int gstride = gridDim.x * kBfsBlock;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned before = (1u << lane) - 1u;
    // warps of one block are far apart in the order in which work is handed out
    const int gwarp = wid * gridDim.x + blockIdx.x, nwarps = gstride >> 5;
    const int m = a.m;
    const int words = (m + 31) >> 5;
    const int *col = a.col_ind;
    int *depth = a.depth;
    // three slots: a level reads one, fills the next and clears the third
    unsigned long long *size = a.ctl->rcnt64;
    int *empty = a.ctl->rcnt;

    const int sr0 = __ldg(a.row_ptr + a.src), sdeg = __ldg(a.row_ptr + a.src + 1) - sr0;
    for (int i = gtid; i < m; i += gstride) depth[i] = (i == a.src) ? 0 : -1;
    for (int w = gtid; w < words; w += gstride) a.vis[0][w] = (w == (a.src >> 5)) ? (1u << (a.src & 31)) : 0u;
    for (int c = gtid; sdeg > 0 && c <= (sdeg - 1) >> a.shift; c += gstride) a.q[0].owner[c] = 0;
    if (gtid == 0) {
        a.q[0].off[0] = 0;
        a.q[0].delta[0] = sr0;
        size[0] = sdeg > 0 ? (1ull << 32) | static_cast<unsigned>(sdeg) : 0ull;
        empty[0] = sdeg > 0 ? 0 : 1;
    }
    if (!grid_barrier(a.ctl, a.sticky, kSiteBfs)) return;

    bool pull = false;
    long long visited_edges = 0, reached = 0;
    int levels = 0, npush = 0, npull = 0, vc = 0;
    const double limit = static_cast<double>(m) / a.beta;  // fewer frontier vertices than this: push
    const double tail = 0.125 * static_cast<double>(a.nnz);
    for (int L = 1;; ++L) {
        const int s0 = (L - 1) % 3, s1 = L % 3, s2 = (L + 1) % 3;
        const unsigned long long sz = __ldcg(size + s0);
        const int nq = static_cast<int>(sz >> 32), E = static_cast<int>(sz & 0xffffffffull);
        const int nf = nq + ld_volatile_i32(empty + s0);
        if (nf == 0) break;
        if (a.depth_cap > 0 && L >= a.depth_cap) break;
        visited_edges += E;
        reached += nf;
        const long long m_u = static_cast<long long>(a.nnz) - visited_edges;
        if (!pull) {
            if (a.allow_pull && a.alpha > 0.0f &&
                static_cast<double>(E) > fmax(static_cast<double>(m_u), tail) / a.alpha)
                pull = true;
        } else if (static_cast<double>(nf) < limit) {
            pull = false;
        }
        ++levels;
        if (gtid == 0) {
            size[s2] = 0ull;
            empty[s2] = 0;
        }
        EdgeQueue qc = a.q[(L - 1) & 1], qn = a.q[L & 1];
        qn.size = size + s1;
        qn.empty = empty + s1;
        unsigned *vis = a.vis[vc];
        int *buf = s_buf[wid];
        int staged = 0;
        // how long a next queue may get before the next level is known to pull
        int enough_n = 0x7fffffff, enough_e = 0x7fffffff;
        if (pull) {
            if (limit < 2e9) enough_n = static_cast<int>(limit) + 1;
        } else if (a.allow_pull && a.alpha > 0.0f) {
            const double al = static_cast<double>(a.alpha);
            const double e = fmax(static_cast<double>(m_u) / (al + 1.0), tail / al) + 1.0;
            if (e < 2e9) enough_e = static_cast<int>(e) + 1;
        }
        auto append = [&](EqBlock<kBfsBlock> *blk) {
            eq_append<kBfsBlock>(buf, staged, blk, qn, a.row_ptr, a.shift, enough_n, enough_e);
            __syncwarp();
            staged = 0;
        };
        if (!pull) {
            ++npush;
            // while few vertices are visited, claiming at once saves a trip to L2 per level; later
            // most neighbours are visited and a look spares the atomic
            const bool look = reached * 16 > m;
            edge_expand<4, false>(qc, nullptr, nq, E, a.shift, s_slice[wid], gwarp, nwarps,
                        [&](const bool (&valid)[4], const int (&)[4], const int (&idx)[4]) {
                            int v[4];
                            unsigned word[4];
                            bool fresh[4];
#pragma unroll
                            for (int r = 0; r < 4; ++r) v[r] = valid[r] ? __ldg(col + idx[r]) : 0;
#pragma unroll
                            for (int r = 0; r < 4; ++r)
                                word[r] = valid[r] ? (look ? __ldcg(vis + (v[r] >> 5)) : 0u) : ~0u;
#pragma unroll
                            for (int r = 0; r < 4; ++r) {
                                const unsigned bit = 1u << (v[r] & 31);
                                fresh[r] = false;
                                if (!(word[r] & bit)) fresh[r] = !(atomicOr(vis + (v[r] >> 5), bit) & bit);
                            }
                            if (staged > kEqCap - kEqTile) append(nullptr);
#pragma unroll
                            for (int r = 0; r < 4; ++r) {
                                if (fresh[r]) depth[v[r]] = L;
                                const unsigned mask = __ballot_sync(0xffffffffu, fresh[r]);
                                if (fresh[r]) buf[staged + __popc(mask & before)] = v[r];
                                staged += __popc(mask);
                            }
                        });
        } else {
            ++npull;
            unsigned *visn = a.vis[vc ^ 1];
            for (int w = gwarp; w < words; w += nwarps) {
                const unsigned vw = vis[w];
                const int v = (w << 5) + lane;
                bool found = false;
                int e = 0, r1 = 0;
                if (v < m && !(vw & (1u << lane))) {
                    e = __ldg(a.row_ptr + v);
                    r1 = __ldg(a.row_ptr + v + 1);
                }
#pragma unroll 1
                for (int step = 0; step < kPullSteps && __any_sync(0xffffffffu, e < r1); ++step) {
                    if (e < r1) {
                        int u[4];
                        unsigned uw[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k) u[k] = __ldg(col + min(e + k, r1 - 1));
#pragma unroll
                        for (int k = 0; k < 4; ++k) uw[k] = vis[u[k] >> 5];
#pragma unroll
                        for (int k = 0; k < 4; ++k) found |= (uw[k] >> (u[k] & 31)) & 1u;
                        e = found ? r1 : e + 4;
                    }
                }
                for (unsigned rest = __ballot_sync(0xffffffffu, e < r1); rest; rest &= rest - 1) {
                    const int l = __ffs(rest) - 1;
                    const int l1 = __shfl_sync(0xffffffffu, r1, l);
                    bool hit = false;
                    for (int b = __shfl_sync(0xffffffffu, e, l); b < l1 && !hit; b += 64) {
                        const int u0 = __ldg(col + min(b + lane, l1 - 1)), u1 = __ldg(col + min(b + 32 + lane, l1 - 1));
                        const unsigned w0 = vis[u0 >> 5], w1 = vis[u1 >> 5];
                        hit = __any_sync(0xffffffffu, ((w0 >> (u0 & 31)) | (w1 >> (u1 & 31))) & 1u);
                    }
                    if (lane == l) found = hit;
                }
                const unsigned fm = __ballot_sync(0xffffffffu, found);
                if (lane == 0) visn[w] = vw | fm;
                if (found) depth[v] = L;
                if (staged > kEqCap - 32) append(nullptr);
                if (found) buf[staged + __popc(fm & before)] = v;
                staged += __popc(fm);
            }
            vc ^= 1;
        }
        append(&s_blk);
        if (!grid_barrier(a.ctl, a.sticky, kSiteBfs + 2)) return;
    }
    if (gtid == 0) {
        a.ctl->iterations = levels;
        a.ctl->push_iterations = npush;
        a.ctl->pull_iterations = npull;
        a.ctl->edges_expanded = visited_edges;
        a.ctl->edges_component = visited_edges;
        a.ctl->vertices_reached = reached;
    }
}

// ================================================================================
// SSSP
// ================================================================================
struct SsspArgs {
    int m, nnz, src, delta_hint;
    int unreached_bits;  // written for unreached vertices (int -1, or a float's bits)
    long long band;      // edges per iteration of the distance band; <= 0: whole frontier
    const int *__restrict__ row_ptr;
    const int *__restrict__ col_ind;
    const int *__restrict__ w;
    int *dist;
    // bits0 = queued in the near frontier, bits1 = held in the far pile;
    // q0/q1 near queues (vertices), q2/q3 far piles; rs, loc_off, aux3 = the edge queue of the
    // entries expanded this iteration (off, delta, owner), aux = their distances;
    // aux2 = distance each vertex was last expanded with
    TravBuffers buf;
    int shift;  // edges per queue unit: 1 << shift
    TravCtl *ctl;
    int *sticky;
};

// Histogram bin of distance d above the band base hb: 8 linear bins, then 8 bins per
// octave (three mantissa bits), 256 in all. Integer distances count in units of 1; float
// distances in units of 1/inv_unit.
__device__ __forceinline__ int band_bin(int d, int hb, int is_float, float inv_unit) {
    if (d <= hb) return 0;
    if (!is_float) {
        const unsigned x = static_cast<unsigned>(d) - static_cast<unsigned>(hb);
        if (x < 8u) return static_cast<int>(x);
        const int e = 31 - __clz(x);
        return 8 * (e - 2) + static_cast<int>((x >> (e - 3)) & 7u);
    }
    const float x = (__int_as_float(d) - __int_as_float(hb)) * inv_unit;
    if (x < 8.0f) return static_cast<int>(x);
    const unsigned b = __float_as_uint(x);
    const int e = static_cast<int>(b >> 23) - 127;
    const int bin = 8 * (e - 2) + static_cast<int>((b >> 20) & 7u);
    return bin < kBandBins - 1 ? bin : kBandBins - 1;
}

// The band histogram takes one vertex in kSampleOf, by a hash, with kSampleOf times its
// degree: it only decides how much work an iteration takes on.
constexpr int kSampleOf = 4;
__device__ __forceinline__ bool sampled(int v) { return (static_cast<unsigned>(v) * 2654435761u) >> 30 == 0u; }

struct SsspShared {
    int slice[kBlock / 32][64 * kSsspVT];  // edge_expand's
    int near[kBlock / 32][32 * kSsspVT + 32];  // vertices on their way to the next queue,
    int far[kBlock / 32][kQCap];          // to the far pile
    unsigned long long hist[kBandBins];   // this block's share of the next band histogram
    unsigned long long scan[33];
    int hmin;                             // least distance this block queued
    int dbase;                            // where this block's deferred entries go
    unsigned long long abase;             // and its expanded entries and their edges
    int sent[kBlock / 32];                // per warp: vertices it queues at the end, then where
};

// Min-plus SpMSpV iterated to the fixed point with near/far buckets (delta-stepping in
// the near-far form): the frontier holds the vertices whose distance dropped below the
// current threshold T; a relaxation that lands at or above T parks the vertex on the far
// pile instead. When the near frontier empties, T advances by delta and the far pile is
// split into the new near frontier and what stays far. A vertex is expanded again only
// if its distance changed since its last expansion. Within the near frontier only the band
// of lowest distances carrying about a.band edges is expanded per iteration; the rest wait
// in the queue. The band's cut comes from a degree-weighted histogram of the distances
// queued during the previous iteration, taken relative to that queue's least distance,
// which is tracked exactly, and the vertices at that least distance always expand, so
// every iteration makes progress. The reference expands every finite
// vertex each iteration (src/spmspvSssp.cuh:31-36, sort + ReduceByKey(min) :220-232) and
// stops after the CPU BFS depth; here a relaxation is a plain read of dist[v] and, only
// if it improves, an atomicMin, and the loop ends when both piles are empty. The result is
// the exact fixed point for non-negative integer weights, independent of relaxation order.
//
// An iteration is two phases with a grid barrier each: phase A goes through the queue (what
// is above the band it only reads the distance of) and puts what is expanded on an edge queue;
// phase B relaxes that queue's edges, a warp per 128. What bounds it (scale 20, 12 iterations):
// phase B at 90-140G relaxations/s with 40 warps on an SM each waiting for a chain of queue
// entry, column, distance (27 % of the issue slots, 28 % of L2); phase A and the barriers
// about 14 us an iteration. Measured: merge-path tiles found by searches with block barriers
// between batches, and every entry read in full each iteration, 709 us; edge queues 619 us;
// reading only the distance of deferred entries and queueing per block 571 us; five blocks
// per SM 553 us. Two, six or eight edges per lane instead of four: 596 / 623 / 580 us.
template <bool F>
__device__ __forceinline__ void sssp_body(SsspArgs a, VGrid vg) {
    static_assert(kBlock == kBandBins, "one histogram bin per thread");
    __shared__ SsspShared sh;
    const int G = vg.n;
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gtid = vg.id * kBlock + threadIdx.x;
    const int gstride = G * kBlock;
    const int m = a.m;
    const int words = (m + 31) >> 5;
    unsigned *inq = a.buf.bits0;
    unsigned *infar = a.buf.bits1;
    int *last = a.buf.aux2;

    // non-negative float32 values order like their int bit patterns, so one integer
    // atomicMin serves both weight types; +inf is the float "infinity"
    const int INF = F ? 0x7f800000 : kInf;
    for (int i = gtid; i < m; i += gstride) {
        a.dist[i] = (i == a.src) ? 0 : INF;
        last[i] = -1;
    }
    for (int w = gtid; w < words; w += gstride) {
        inq[w] = (w == (a.src >> 5)) ? (1u << (a.src & 31)) : 0u;
        infar[w] = 0u;
    }
    // sample the weights for the default bucket width
    constexpr int kSample = 1 << 16;
    const int nsamp = a.nnz < kSample ? a.nnz : kSample;
    {
        double ws = 0.0;
        for (int k = gtid; k < nsamp; k += gstride) {
            const int wb = __ldg(a.w + static_cast<long long>(k) * a.nnz / nsamp);
            ws += F ? static_cast<double>(__int_as_float(wb)) : static_cast<double>(wb);
        }
        for (int o = 16; o; o >>= 1) ws += __shfl_down_sync(0xffffffffu, ws, o);
        if ((threadIdx.x & 31) == 0 && ws != 0.0) atomicAdd(reinterpret_cast<double *>(&a.ctl->aux[0]), ws);
    }
    if (gtid == 0) {
        a.buf.q0[0] = a.src;
        a.ctl->qlen[0] = 1;
        a.ctl->qlen[1] = 0;
        a.ctl->flen[0] = 0;
        a.ctl->flen[1] = 0;
        a.ctl->sbase[0] = 0;  // the source's distance
        a.ctl->sbase[1] = INF;
        a.ctl->rcnt64[0] = a.ctl->rcnt64[1] = 0ull;
    }
    sh.hist[threadIdx.x] = 0ull;
    if (threadIdx.x == 0) sh.hmin = INF;
    if (!grid_barrier(a.ctl, a.sticky, kSiteSssp, vg)) return;

    const bool banded = a.band > 0;
    const double sum_w = __longlong_as_double(__ldcg(&a.ctl->aux[0]));
    const double mean_w = nsamp ? sum_w / nsamp : 1.0;
    // float distances are binned in units of mean weight / 256
    const float inv_unit = (F && mean_w > 0.0) ? static_cast<float>(256.0 / mean_w) : 1.0f;
    double delta = a.delta_hint;
    if (delta <= 0 && banded) {
        delta = 1e300;  // the band orders the work: no far pile
    } else if (delta <= 0) {
        const double mean_deg = m ? static_cast<double>(a.nnz) / m : 1.0;
        delta = 32.0 * mean_w / (mean_deg > 1.0 ? mean_deg : 1.0);
        if (!F) delta = floor(delta);
        if (!(delta >= 1.0)) delta = F ? (delta > 0.0 ? delta : 1.0) : 1.0;
    }
    double thresh = delta;
    const bool piles = delta < 1e300;
    int hb = 0;  // base of the histogram in ctl->shist[cur] (the previous iteration's base)
    int cur = 0, fc = 0;
    long long expanded = 0;
    int iters = 0, steps = 0;
    const long long step_cap = 4LL * m + 4096;
    for (;;) {
        if (++steps > step_cap) {
            if (gtid == 0) raise_error(a.ctl, a.sticky, APSPIE_ERR_NOT_CONVERGED, kSiteSsspIterCap);
            break;
        }
        const int nf = ld_volatile_i32(&a.ctl->qlen[cur]);
        int *qc = cur ? a.buf.q1 : a.buf.q0;
        int *qn = cur ? a.buf.q0 : a.buf.q1;
        int *fcur = fc ? a.buf.q3 : a.buf.q2;
        int *fnext = fc ? a.buf.q2 : a.buf.q3;
        int *dist = a.dist;
        if (nf == 0) {
            // near frontier empty: advance the threshold and split the far pile
            const int nfar = ld_volatile_i32(&a.ctl->flen[fc]);
            if (nfar == 0) break;
            thresh += delta;
            // every block must have read qlen[cur] (== 0) before any block appends to it
            if (!grid_barrier(a.ctl, a.sticky, kSiteSsspBarF0, vg)) return;
            WQ wn(sh.near[wid], qc, &a.ctl->qlen[cur]);
            WQ wf(sh.far[wid], fnext, &a.ctl->flen[fc ^ 1]);
            for (int base = vg.id * kBlock; base < nfar; base += gstride) {
                const int i = base + threadIdx.x;
                bool to_near = false, stay = false;
                int v = 0;
                if (i < nfar) {
                    v = __ldcg(fcur + i);
                    const int d = __ldcg(dist + v);
                    const double dv = F ? static_cast<double>(__int_as_float(d)) : static_cast<double>(d);
                    if (dv < thresh) {
                        atomicAnd(infar + (v >> 5), ~(1u << (v & 31)));
                        const unsigned bit = 1u << (v & 31);
                        to_near = !(atomicOr(inq + (v >> 5), bit) & bit);
                        atomicMin(&a.ctl->sbase[cur], d);
                    } else {
                        stay = true;
                    }
                }
                wn.push(to_near, v);
                wf.push(stay, v);
            }
            wn.flush();
            wf.flush();
            if (!grid_barrier(a.ctl, a.sticky, kSiteSsspBarF1, vg)) return;
            if (gtid == 0) a.ctl->flen[fc] = 0;  // drained; every block read nfar above
            fc ^= 1;
            continue;
        }
        int *qlen_next = &a.ctl->qlen[cur ^ 1];  // zero: reset when that queue was last read
        int *snap = a.buf.aux;

        // the band: histogram bins up to the first where the running edge count reaches
        // a.band (kBandBins = every bin: band off, or too little queued work to cut)
        const int base_i = ld_volatile_i32(&a.ctl->sbase[cur]);
        int cut = kBandBins;
        if (banded) {
            const unsigned long long h = __ldcg(&a.ctl->shist[cur][threadIdx.x]);
            const unsigned long long incl = block_inclusive_scan_u64<kBlock>(h, sh.scan);
            const unsigned long long S = static_cast<unsigned long long>(a.band);
            const bool reach = sh.scan[32] >= S;
            const int below = __syncthreads_count(incl < S);
            if (reach && below < kBandBins - 1) cut = below;
        }
        const int hb_prev = hb;
        hb = base_i;
        // phase A: dequeue (clear queued bit), skip vertices whose distance is the one they were
        // expanded with, put the others on the iteration's edge queue with their distance;
        // vertices above the band stay queued (re-appended to the next queue, bit kept)
        unsigned long long *asize = a.ctl->rcnt64 + (iters & 1);
        {
            // kSsspPA entries per thread per step, their loads issued together
            constexpr int PA = kSsspPA;
            const int C = (nf + G - 1) / G;
            const int c0 = min(vg.id * C, nf);
            const int c1 = min(c0 + C, nf);
            const int *rpa = a.row_ptr;
            for (int base = c0; base < c1; base += kBlock * PA) {
                const int i0 = base + static_cast<int>(threadIdx.x) * PA;
                int v[PA], r0[PA], r1[PA], d[PA], lst[PA], out[PA];
                bool valid[PA], defer[PA];
#pragma unroll
                for (int k = 0; k < PA; ++k) {
                    valid[k] = i0 + k < c1;
                    v[k] = valid[k] ? __ldcg(qc + i0 + k) : 0;
                }
#pragma unroll
                for (int k = 0; k < PA; ++k) d[k] = valid[k] ? __ldcg(dist + v[k]) : 0;
                // most of a long queue is deferred: only what is expanded, and the sample of the
                // deferred that the histogram takes, needs more than its distance
#pragma unroll
                for (int k = 0; k < PA; ++k) {
                    defer[k] = valid[k] && cut < kBandBins && d[k] != base_i &&
                               band_bin(d[k], hb_prev, F, inv_unit) > cut;
                    const bool row = valid[k] && (!defer[k] || sampled(v[k]));
                    r0[k] = row ? __ldg(rpa + v[k]) : 0;
                    r1[k] = row ? __ldg(rpa + v[k] + 1) : 0;
                    lst[k] = valid[k] && !defer[k] ? __ldcg(last + v[k]) : 0;
                }
                int sum = 0, nact = 0, ndef = 0;
#pragma unroll
                for (int k = 0; k < PA; ++k) {
                    out[k] = 0;
                    if (valid[k] && !defer[k]) {
                        atomicAnd(inq + (v[k] >> 5), ~(1u << (v[k] & 31)));
                        if (lst[k] != d[k]) {
                            last[v[k]] = d[k];
                            out[k] = r1[k] - r0[k];
                        }
                    }
                    sum += out[k];
                    nact += out[k] > 0;
                }
#pragma unroll
                for (int k = 0; k < PA; ++k) {
                    if (defer[k] && r1[k] > r0[k])
                        atomicAdd(&sh.hist[band_bin(d[k], base_i, F, inv_unit)],
                                  static_cast<unsigned long long>(kSampleOf) * static_cast<unsigned>(r1[k] - r0[k]));
                    const int mn = __reduce_min_sync(0xffffffffu, defer[k] ? d[k] : 0x7fffffff);
                    if (mn != 0x7fffffff && lane == 0) atomicMin(&sh.hmin, mn);
                    ndef += defer[k] ? 1 : 0;
                }
                // one scan carries the edges, the expanded entries and the deferred ones (the
                // counts at most kBlock * PA = 1024 per step, so neither carries over)
                static_assert(kBlock * PA <= 1024, "counts fit 11 bits");
                const unsigned long long packed = (static_cast<unsigned long long>(sum) << 22) |
                                                  (static_cast<unsigned>(nact) << 11) | static_cast<unsigned>(ndef);
                const unsigned long long incl = block_inclusive_scan_u64<kBlock>(packed, sh.scan);
                const unsigned long long excl = incl - packed;
                if (threadIdx.x == 0) {
                    const unsigned long long total = sh.scan[32];
                    const unsigned td = static_cast<unsigned>(total) & 2047u, ta = static_cast<unsigned>(total >> 11) & 2047u;
                    if (td) sh.dbase = atomicAdd(qlen_next, static_cast<int>(td));
                    if (ta) sh.abase = atomicAdd(asize, (static_cast<unsigned long long>(ta) << 32) | (total >> 22));
                }
                __syncthreads();
                const unsigned long long ab = sh.abase;
                int idx = static_cast<int>(ab >> 32) + static_cast<int>(static_cast<unsigned>(excl >> 11) & 2047u);
                int off = static_cast<int>(ab & 0xffffffffull) + static_cast<int>(excl >> 22);
                int dpos = sh.dbase + static_cast<int>(static_cast<unsigned>(excl) & 2047u);
#pragma unroll
                for (int k = 0; k < PA; ++k) {
                    const bool some = out[k] > 0;
                    eq_write(a.buf.rs, a.buf.loc_off, a.buf.aux3, a.shift, some, idx, off, r0[k], out[k]);
                    if (some) snap[idx] = d[k];
                    idx += some;
                    off += out[k];
                    if (defer[k]) qn[dpos++] = v[k];
                }
                __syncthreads();  // sh.scan and the bases are reused by the next step
            }
        }
        if (!grid_barrier(a.ctl, a.sticky, kSiteSsspBarA, vg)) return;
        // every block has read this queue's length, base and histogram, and the last iteration's
        // edge queue: reset them for the iteration that fills them next
        if (gtid < kBandBins) a.ctl->shist[cur][gtid] = 0ull;
        if (gtid == 0) {
            a.ctl->qlen[cur] = 0;
            a.ctl->sbase[cur] = INF;
            a.ctl->rcnt64[(iters & 1) ^ 1] = 0ull;
        }
        const unsigned long long asz = __ldcg(asize);
        const int nact = static_cast<int>(asz >> 32), E = static_cast<int>(asz & 0xffffffffull);
        expanded += E;
        ++iters;
        const int *col = a.col_ind;
        const int *wt = a.w;
        const int *rp = a.row_ptr;
        // nd < Tkey exactly when the distance nd (bits, if float) is below thresh
        const int Tkey = F ? __float_as_int(__double2float_ru(thresh))
                           : thresh < 2147483647.0 ? static_cast<int>(ceil(thresh)) : kInf;
        int *near = sh.near[wid];
        int staged = 0;
        const unsigned before = (1u << lane) - 1u;
        auto send = [&]() {  // staged vertices -> next queue
            __syncwarp();
            int at = 0;
            if (lane == 0) at = atomicAdd(qlen_next, staged);
            at = __shfl_sync(0xffffffffu, at, 0);
            for (int i = lane; i < staged; i += 32) qn[at + i] = near[i];
            __syncwarp();
            staged = 0;
        };
        WQ wf(sh.far[wid], fcur, &a.ctl->flen[fc]);
        bool bad = false, over = false;
        EdgeQueue qa{a.buf.rs, a.buf.loc_off, a.buf.aux3, nullptr, nullptr};
        edge_expand<kSsspVT, true>(
            qa, snap, nact, E, a.shift, sh.slice[wid], wid * G + vg.id, G * (kBlock / 32),
            [&](const bool (&valid)[kSsspVT], const int (&du)[kSsspVT], const int (&idx)[kSsspVT]) {
                int v[kSsspVT], we[kSsspVT], cd[kSsspVT], nd[kSsspVT];
                bool got[kSsspVT], queue[kSsspVT];
#pragma unroll
                for (int r = 0; r < kSsspVT; ++r) {
                    v[r] = valid[r] ? __ldg(col + idx[r]) : 0;
                    we[r] = valid[r] ? __ldg(wt + idx[r]) : 0;
                }
                // coherent reads; a slot without an edge relaxes 0 + 0 against 0
#pragma unroll
                for (int r = 0; r < kSsspVT; ++r) cd[r] = valid[r] ? __ldcg(dist + v[r]) : 0;
#pragma unroll
                for (int r = 0; r < kSsspVT; ++r) {
                    if (F) {
                        const float wf32 = __int_as_float(we[r]);
                        const bool ok = wf32 >= 0.0f;  // neither negative nor NaN
                        bad |= !ok;
                        nd[r] = __float_as_int(__fadd_rn(__int_as_float(du[r]), wf32));
                        got[r] = ok && nd[r] < cd[r];
                    } else {
                        // both below 2^31, so the sum does not wrap; a sum past INT_MAX - 1 is
                        // never below cd
                        const unsigned s = static_cast<unsigned>(du[r]) + static_cast<unsigned>(we[r]);
                        bad |= we[r] < 0;
                        over |= s >= 0x7fffffffu;
                        nd[r] = static_cast<int>(s);
                        got[r] = we[r] >= 0 && s < static_cast<unsigned>(cd[r]);
                    }
                }
#pragma unroll
                for (int r = 0; r < kSsspVT; ++r)
                    if (got[r]) atomicMin(dist + v[r], nd[r]);
#pragma unroll
                for (int r = 0; r < kSsspVT; ++r) {
                    queue[r] = false;
                    if (got[r] && nd[r] < Tkey) {
                        const unsigned bit = 1u << (v[r] & 31);
                        queue[r] = !(atomicOr(inq + (v[r] >> 5), bit) & bit);
                    }
                }
                if (banded) {
                    // improvements below T (queued now or already): a sample enters the next band
                    // histogram at their new distance; the least distance is exact
#pragma unroll
                    for (int r = 0; r < kSsspVT; ++r) {
                        if (!(got[r] && nd[r] < Tkey)) continue;
                        if (nd[r] < *static_cast<volatile int *>(&sh.hmin)) atomicMin(&sh.hmin, nd[r]);
                        if (sampled(v[r]))
                            atomicAdd(&sh.hist[band_bin(nd[r], base_i, F, inv_unit)],
                                      static_cast<unsigned long long>(kSampleOf) *
                                          static_cast<unsigned>(__ldg(rp + v[r] + 1) - __ldg(rp + v[r])));
                    }
                }
                if (staged > 32) send();
#pragma unroll
                for (int r = 0; r < kSsspVT; ++r) {
                    const unsigned mask = __ballot_sync(0xffffffffu, queue[r]);
                    if (queue[r]) near[staged + __popc(mask & before)] = v[r];
                    staged += __popc(mask);
                }
                if (piles) {
#pragma unroll
                    for (int r = 0; r < kSsspVT; ++r) {
                        bool far = false;
                        if (got[r] && nd[r] >= Tkey) {
                            const unsigned bit = 1u << (v[r] & 31);
                            far = !(atomicOr(infar + (v[r] >> 5), bit) & bit);
                        }
                        wf.push(far, v[r]);
                    }
                }
            });
        // what is still staged goes out for the whole block at once (4,736 reservations on one
        // word, one after the other, took most of the 10 us at the end of an iteration)
        if (lane == 0) sh.sent[wid] = staged;
        __syncthreads();
        if (threadIdx.x == 0) {
            int all = 0;
            for (int w = 0; w < kBlock / 32; ++w) {
                const int c = sh.sent[w];
                sh.sent[w] = all;
                all += c;
            }
            const int at = all ? atomicAdd(qlen_next, all) : 0;
            for (int w = 0; w < kBlock / 32; ++w) sh.sent[w] += at;
        }
        __syncthreads();
        for (int i = lane; i < staged; i += 32) qn[sh.sent[wid] + i] = near[i];
        wf.flush();
        if (bad) raise_error(a.ctl, a.sticky, APSPIE_ERR_INVALID_ARG, kSiteSsspNegWeight);
        if (over) raise_error(a.ctl, a.sticky, APSPIE_ERR_INVALID_ARG, kSiteSsspOverflow);
        if (banded) {
            __syncthreads();
            const unsigned long long hv = sh.hist[threadIdx.x];
            if (hv) {
                atomicAdd(&a.ctl->shist[cur ^ 1][threadIdx.x], hv);
                sh.hist[threadIdx.x] = 0ull;
            }
            if (threadIdx.x == 0 && sh.hmin != INF) {
                atomicMin(&a.ctl->sbase[cur ^ 1], sh.hmin);
                sh.hmin = INF;
            }
        }
        if (!grid_barrier(a.ctl, a.sticky, kSiteSsspBarB, vg)) return;
        cur ^= 1;
    }
    // unreached -> -1, and the component statistics
    long long comp = 0, reached = 0;
    for (int i = gtid; i < m; i += gstride) {
        const int d = a.dist[i];
        if (d == INF) {
            a.dist[i] = a.unreached_bits;
        } else {
            comp += __ldg(a.row_ptr + i + 1) - __ldg(a.row_ptr + i);
            ++reached;
        }
    }
    for (int o = 16; o; o >>= 1) {
        comp += __shfl_down_sync(0xffffffffu, comp, o);
        reached += __shfl_down_sync(0xffffffffu, reached, o);
    }
    if ((threadIdx.x & 31) == 0 && (comp || reached)) {
        atomicAdd(reinterpret_cast<unsigned long long *>(&a.ctl->edges_component),
                  static_cast<unsigned long long>(comp));
        atomicAdd(reinterpret_cast<unsigned long long *>(&a.ctl->vertices_reached),
                  static_cast<unsigned long long>(reached));
    }
    if (gtid == 0) {
        a.ctl->iterations = iters;
        a.ctl->push_iterations = iters;
        a.ctl->pull_iterations = steps - 1 - iters;  // threshold advances
        a.ctl->edges_expanded = expanded;
        a.ctl->delta = delta < 2147483647.0 ? static_cast<int>(delta) : 0;  // 0: no far pile
    }
}

template <bool F>
__global__ void __launch_bounds__(kBlock, 5) sssp_kernel(SsspArgs a) {
    grid_begin(a.ctl);
    sssp_body<F>(a, hw_grid());
}

// Many sources in one launch: the grid splits into `groups` equal groups of blocks, each
// with its own control block and scratch, and each group runs the single-source SSSP
// above on queries grp, grp + groups, ... in turn, synchronising only among its own
// blocks. Every answer is the single-source kernel's answer; the queries of different
// groups run side by side, which pays because one query alone keeps the device
// latency-bound (few warps issue at a time).
struct SsspGroupArgs {
    SsspArgs base;       // graph, weights, band, sticky word; per query: src, dist, ctl, buf
    const int *srcs;
    int *out;            // nq x m, query-major
    int nq, groups, m;
    TravCtl *ctls;       // one control block per group
    size_t buf_stride;   // bytes between consecutive groups' scratch (base.buf is group 0's)
    TravCtl *main;       // the context's control block: errors and summed statistics
};

__device__ __forceinline__ TravBuffers shift_buffers(TravBuffers b, size_t off) {
    auto sh = [off](auto *p) { return reinterpret_cast<decltype(p)>(reinterpret_cast<char *>(p) + off); };
    b.q0 = sh(b.q0);
    b.q1 = sh(b.q1);
    b.q2 = sh(b.q2);
    b.q3 = sh(b.q3);
    b.rs = sh(b.rs);
    b.loc_off = sh(b.loc_off);
    b.aux = sh(b.aux);
    b.aux2 = sh(b.aux2);
    b.aux3 = sh(b.aux3);
    b.bits0 = sh(b.bits0);
    b.bits1 = sh(b.bits1);
    return b;
}

__global__ void __launch_bounds__(kBlock, 5) sssp_group_kernel(SsspGroupArgs g) {
    const int bpg = static_cast<int>(gridDim.x) / g.groups;  // the host launches groups * bpg blocks
    const int grp = static_cast<int>(blockIdx.x) / bpg;
    const VGrid vg{static_cast<int>(blockIdx.x) - grp * bpg, bpg};
    TravCtl *ctl = g.ctls + grp;
    grid_begin(ctl);
    SsspArgs a = g.base;
    a.ctl = ctl;
    a.buf = shift_buffers(g.base.buf, g.buf_stride * grp);
    const int tid = vg.id * kBlock + static_cast<int>(threadIdx.x);
    for (int q = grp; q < g.nq; q += g.groups) {
        a.src = __ldg(g.srcs + q);
        if (a.src < 0 || a.src >= g.m) {
            // every block of the group reads the same source and skips the query alike
            if (tid == 0) raise_error(g.main, a.sticky, APSPIE_ERR_INVALID_ARG, kSiteSsspBadSource);
            continue;
        }
        a.dist = g.out + static_cast<size_t>(q) * g.m;
        sssp_body<false>(a, vg);
        // every block of the group is done with the control block before it is reset
        if (!grid_barrier(ctl, a.sticky, kSiteSsspGroup, vg)) break;
        if (tid == 0) {
            atomicAdd(reinterpret_cast<unsigned long long *>(&g.main->edges_expanded),
                      static_cast<unsigned long long>(ctl->edges_expanded));
            atomicAdd(reinterpret_cast<unsigned long long *>(&g.main->edges_component),
                      static_cast<unsigned long long>(ctl->edges_component));
            atomicAdd(reinterpret_cast<unsigned long long *>(&g.main->vertices_reached),
                      static_cast<unsigned long long>(ctl->vertices_reached));
            atomicAdd(&g.main->iterations, ctl->iterations);
            atomicAdd(&g.main->push_iterations, ctl->push_iterations);
            ctl->edges_component = 0;
            ctl->vertices_reached = 0;
            for (int k = 0; k < 4; ++k) ctl->aux[k] = 0;
        }
        for (int k = tid; k < 2 * kBandBins; k += vg.n * kBlock) ctl->shist[k / kBandBins][k % kBandBins] = 0ull;
        if (!grid_barrier(ctl, a.sticky, kSiteSsspGroup + 1, vg)) break;
    }
    if (tid == 0 && ctl->err != 0) raise_error(g.main, a.sticky, ctl->err, ctl->err_where);
}

// ================================================================================
// MIS
// ================================================================================
enum : unsigned char { kUndecided = 0, kIn = 1, kOut = 2 };
#ifndef APSPIE_MIS_THREAD
#define APSPIE_MIS_THREAD 16
#endif
#ifndef APSPIE_MIS_WARP_CHUNKS
#define APSPIE_MIS_WARP_CHUNKS 8
#endif
constexpr int kMisThread = APSPIE_MIS_THREAD;          // neighbours one thread scans (phase S) before handing on
constexpr int kMisWarpChunks = APSPIE_MIS_WARP_CHUNKS;  // chunks of 32 neighbours a warp scans (phase L)
constexpr int kMisLightRow = 64;   // joiners with at most this many neighbours push by one thread

struct MisArgs {
    int m, nnz;
    const int *__restrict__ row_ptr;
    const int *__restrict__ col_ind;
    const unsigned *__restrict__ prio;
    unsigned char *member;
    int *member_i32;  // when set, the set is written here as int32 1/0 instead
    unsigned char *state;
    int *pos;          // CSR index of the outranking neighbour that blocks the vertex (row start - 1: none yet)
    int *queue[2];     // undecided vertices, by round parity
    int *longq;        // scans that go on past a thread's share (one warp each, phase L)
    int *longq2;       // scans that go on past a warp's share (one block each, phase L2)
    int *light;        // vertices that joined with rows of at most kMisLightRow (pushed next round)
    int *heavy_v;      // vertices that joined with longer rows,
    int *heavy_base;   // the offset of each one's row in the next round's flat range of pushes,
    int *heavy_delta;  // and row start - offset (push t of the range is CSR entry t + delta)
    int *unit_owner;   // the heavy entry holding the first push of each unit of the range
    int unit_shift;    // units of 1 << unit_shift pushes (one warp each)
    TravCtl *ctl;
    int *sticky;
};

__device__ __forceinline__ bool outranks(unsigned pu, int u, unsigned pv, int v) {
    return pu > pv || (pu == pv && u > v);
}

// A neighbour's state as a scan reads it: through L1, so the lines of high-degree
// neighbours (read by many scans at once) are not all fetched from L2. A stale value is
// safe: states only move from undecided to in or out, so a stale read can only make a scan
// stop early at a neighbour that is already out, and the next round's blocker check (a
// coherent read) sees it out and resumes the scan behind it.
#ifndef APSPIE_MIS_STATE_STRIDE
#define APSPIE_MIS_STATE_STRIDE 1
#endif
constexpr int kMisStateStride = APSPIE_MIS_STATE_STRIDE;  // bytes between consecutive vertices' states
__device__ __forceinline__ long long sx(int v) { return static_cast<long long>(v) * kMisStateStride; }
__device__ __forceinline__ unsigned char scan_state(const unsigned char *state, int u) { return state[sx(u)]; }

// One neighbour of a scanning vertex v: does it decide anything (an outranking neighbour
// that is not out: v's new blocker, or -- if in -- the vertex that knocks v out)?
__device__ __forceinline__ bool mis_stop(const MisArgs &a, int idx, int v, unsigned pv) {
    const int u = __ldg(a.col_ind + idx);
    const unsigned pu = __ldg(a.prio + u);
    const unsigned char su = scan_state(a.state, u);
    return u != v && su != kOut && outranks(pu, u, pv, v);
}

// Knock out neighbour u of a vertex that joined. Many joiners share their high-degree
// neighbours, and stores from many SMs into one line queue up in L2, so (check) a neighbour
// already seen out (through L1: a stale "undecided" only costs a redundant store) is
// skipped. In the first push round nothing is out yet.
__device__ __forceinline__ void mis_knock(const MisArgs &a, int u, bool check) {
    if (!check || scan_state(a.state, u) != kOut) a.state[sx(u)] = kOut;
}

// v joined with a row [r0, r0 + deg) longer than kMisLightRow: list it for the next
// round's pushes. One atomic on (entries << 32 | pushes) gives the entry index and the
// row's offset in the flat range, so offsets ascend with the index; the units starting
// inside the row record it.
__device__ __forceinline__ void mis_list_heavy(const MisArgs &a, unsigned long long *heavy, int v, int r0, int deg) {
    const unsigned long long old = atomicAdd(heavy, (1ull << 32) | static_cast<unsigned>(deg));
    const int idx = static_cast<int>(old >> 32);
    const int base = static_cast<int>(old & 0xffffffffull);
    a.heavy_v[idx] = v;
    a.heavy_base[idx] = base;
    a.heavy_delta[idx] = r0 - base;
    const int sh = a.unit_shift;
    for (int c = ((base - 1) >> sh) + 1; (c << sh) < base + deg; ++c) a.unit_owner[c] = idx;
}

// Greedy MIS in descending (priority, id) order -- the set spmspvMis converges to
// (src/spmspvMis.cuh:54-78: candidate if rand > threshold, select if rand > every
// candidate neighbour's, knock out the neighbours), with ties broken by id instead of
// left undecided. A vertex joins exactly when every neighbour that outranks it is out;
// it is out as soon as a neighbour joins.
//
// Only outranking neighbours can ever decide a vertex (a lower-ranked neighbour cannot
// join while the vertex is undecided), and a neighbour once seen out or lower-ranked
// stays so. So each undecided vertex keeps a scan position `pos`: every neighbour before
// it is settled, and the neighbour at it is its current blocker (undecided, outranking).
// Each scan stops at the first neighbour that decides anything, so rows are read about
// once over the whole run and mostly not to their end (about 6.8M of R-MAT scale 20's
// 31.4M entries). Round r, over the undecided vertices (round 0: all of them, which also
// sets every state; vertices without neighbours join there) and the vertices that joined
// in round r - 1:
//  phase P  (when anything joined) the joiners write out into their neighbours: rows of at
//           most kMisLightRow one thread each; longer rows, laid end to end in the order
//           they were listed, in equal units of 1 << unit_shift entries, one warp each.
//           Only stores (and L1 reads): on the B200 a phase in which many SMs both store
//           into and read the lines of high-degree vertices' states runs several times
//           slower, so the pushes are not made by the joining threads during the scans;
//  phase S  each undecided vertex, by one thread: out -> leaves; its blocker still
//           undecided (or in: its push comes next round) -> waits; else it scans on, four
//           neighbours a step, and stops at the first neighbour that outranks it and is not
//           out (its new blocker); no such neighbour -> it joins and is listed for the next
//           round's pushes. After kMisThread neighbours without an end the vertex goes to
//           the long list;
//  phase L  (only when that list is not empty) one warp per vertex goes on in chunks of
//           32, for up to kMisWarpChunks chunks; the rest (phase L2) one block each.
// The pushes of a round are complete before its scans start, so a scan sees every vertex
// knocked out so far; scans and joins of the same phase race only safely (a vertex joins
// only if every outranking neighbour was seen out, and out is final). The set is the
// greedy MIS whatever the timing.
//
// The lists a round fills (long lists and joiners in slot r mod 3 of the control block's
// round counters, the next queue in slot r + 1) are cleared by the round before: their
// last readers finished a full round earlier, so no block can still be reading them.
__global__ void __launch_bounds__(kBlock) mis_kernel(MisArgs a) {
    __shared__ int qbuf[kBlock / 32][3][kQCap];
    __shared__ int s_stop;
    grid_begin(a.ctl);
    const int G = gridDim.x;
    const int gtid = blockIdx.x * kBlock + threadIdx.x;
    const int gstride = G * kBlock;
    const int lane = threadIdx.x & 31;
    const int wid = threadIdx.x >> 5;
    const int m = a.m;
    const int *col = a.col_ind;
    unsigned char *state = a.state;
    int *qlen = a.ctl->rcnt;                   // [3] undecided-queue lengths
    int *l1len = a.ctl->rcnt + 3;              // [3] long list (phase L)
    int *l2len = a.ctl->rcnt + 6;              // [3] longest list (phase L2)
    int *nlight = a.ctl->rcnt + 9;             // [3] light joiners
    unsigned long long *heavy = a.ctl->rcnt64;  // [3] (entries << 32) | pushes of heavy joiners
    long long pushed = 0, scanned = 0;
    int r = 0;
    for (;; ++r) {
        const int s0 = r % 3, s1 = (r + 1) % 3, s2 = (r + 2) % 3;
        const int sp = (r + 2) % 3;  // the joiner lists of round r - 1
        const int nf = r == 0 ? m : ld_volatile_i32(qlen + s0);  // round 0: every vertex
        const int nl = ld_volatile_i32(nlight + sp);
        const unsigned long long hh = __ldcg(reinterpret_cast<const unsigned long long *>(heavy + sp));
        const int nh = static_cast<int>(hh >> 32);
        const int H = static_cast<int>(hh & 0xffffffffull);
        const int sh = a.unit_shift;
        const int nu = H > 0 ? ((H - 1) >> sh) + 1 : 0;
        if (nf == 0 && nl == 0 && nu == 0) break;
        if (r > m + 1) {
            if (gtid == 0) raise_error(a.ctl, a.sticky, APSPIE_ERR_NOT_CONVERGED, kSiteMisRoundCap);
            break;
        }
        const int *qc = a.queue[r & 1];
        int *qn = a.queue[(r & 1) ^ 1];

        // phase P: the last round's joiners knock out their neighbours -- short rows one
        // thread each, long rows laid end to end and shared out in equal units, one warp
        // each. Plain byte stores: every neighbour of a vertex in the set is out.
        if (nl > 0 || nu > 0) {
            // skipping known outs pays when many joiners share neighbours; with few of them
            // the read before each store only lengthens the chain
            const bool check = r >= 2 && nl + nh >= 4096;
            // lanes per joiner: 1 when the joiners fill the grid, up to 8 when they are few,
            // so that a short round's rows are not walked one entry at a time by one thread
            int lpj = 1;
            while (lpj < 8 && static_cast<long long>(nl) * lpj * 2 <= gstride) lpj <<= 1;
            const int sub = gtid & (lpj - 1);
            for (int i = gtid / lpj; i < nl; i += gstride / lpj) {
                const int j = __ldcg(a.light + i);
                const int r0 = __ldg(a.row_ptr + j), r1 = __ldg(a.row_ptr + j + 1);
                if (sub == 0) pushed += r1 - r0;
                for (int e = r0 + sub; e < r1; e += 8 * lpj) {
                    int u[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) u[k] = e + k * lpj < r1 ? __ldg(col + e + k * lpj) : j;
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        if (u[k] != j) mis_knock(a, u[k], check);
                }
            }
            const int gw = gtid >> 5, nw = gstride >> 5;
            for (int c = gw; c < nu; c += nw) {
                // a unit spans the end of one row and the start of the next where rows meet in it
                const int t0 = c << sh, t1 = min(H, t0 + (1 << sh));
                int i = __ldcg(a.unit_owner + c);
                int hv = __ldcg(a.heavy_v + i), hd = __ldcg(a.heavy_delta + i);
                int nb = i + 1 < nh ? __ldcg(a.heavy_base + i + 1) : INT_MAX;
                if (lane == 0) pushed += t1 - t0;
                for (int tb = t0; tb < t1; tb += 128) {
                    int e[4], w[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int t = tb + 32 * q + lane;
                        while (t < t1 && t >= nb) {
                            ++i;
                            hv = __ldcg(a.heavy_v + i);
                            hd = __ldcg(a.heavy_delta + i);
                            nb = i + 1 < nh ? __ldcg(a.heavy_base + i + 1) : INT_MAX;
                        }
                        e[q] = t < t1 ? t + hd : -1;
                        w[q] = hv;
                    }
                    int u[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) u[q] = e[q] >= 0 ? __ldg(col + e[q]) : -1;
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (u[q] >= 0 && u[q] != w[q]) mis_knock(a, u[q], check);
                }
            }
            if (!grid_barrier(a.ctl, a.sticky, kSiteMis + 2)) return;
        }
        // the lists this round fills start empty; their slots were last read a round ago
        if (gtid == 0) {
            qlen[s2] = 0;
            l1len[s1] = 0;
            l2len[s1] = 0;
            nlight[s1] = 0;
            heavy[s1] = 0ull;
        }

        // phase S: blocker checks, short scans and decisions, one thread per vertex; each
        // scan step loads four neighbours at once and takes the first that decides anything
        {
            WQ wq(qbuf[wid][0], qn, qlen + s1);
            WQ wj(qbuf[wid][1], a.light, nlight + s0);
            WQ wl(qbuf[wid][2], a.longq, l1len + s0);
            for (int base = blockIdx.x * kBlock; base < nf; base += gstride) {
                const int i = base + threadIdx.x;
                bool keep = false, light = false, along = false;
                int v = 0;
                if (i < nf) {
                    // round 0 takes every vertex and writes every state: vertices without
                    // neighbours join at once, the others start undecided with no blocker
                    v = r == 0 ? i : __ldcg(qc + i);
                    const int r0 = __ldg(a.row_ptr + v), r1 = __ldg(a.row_ptr + v + 1);
                    if (r == 0 && r1 == r0) {
                        state[sx(v)] = kIn;
                    } else if (r == 0 || __ldcg(state + sx(v)) == kUndecided) {
                        const int p = r == 0 ? r0 - 1 : __ldcg(a.pos + v);
                        if (r == 0) state[sx(v)] = kUndecided;
                        if (p >= r0 && __ldcg(state + sx(__ldg(col + p))) != kOut) {
                            keep = true;  // its blocker is undecided (or joined: its push comes next)
                        } else {
                            const unsigned pv = __ldg(a.prio + v);
                            const int start = p + 1, lim = min(r1, start + kMisThread);
                            int stop = -1, e = start;
                            for (; e < lim && stop < 0; e += 4) {
                                int u[4];
                                unsigned pu[4];
                                unsigned char su[4];
#pragma unroll
                                for (int k = 0; k < 4; ++k) u[k] = e + k < lim ? __ldg(col + e + k) : v;
#pragma unroll
                                for (int k = 0; k < 4; ++k) {
                                    pu[k] = __ldg(a.prio + u[k]);
                                    // in the first round every vertex with neighbours is undecided
                                    su[k] = r == 0 ? kUndecided : scan_state(state, u[k]);
                                }
#pragma unroll
                                for (int k = 0; k < 4; ++k)
                                    if (stop < 0 && u[k] != v && su[k] != kOut && outranks(pu[k], u[k], pv, v))
                                        stop = e + k;
                            }
                            scanned += (stop >= 0 ? stop + 1 : lim) - start;
                            if (stop >= 0) {
                                keep = true;
                                a.pos[v] = stop;
                            } else if (lim >= r1) {
                                state[sx(v)] = kIn;
                                light = r1 - r0 <= kMisLightRow;
                                if (!light) mis_list_heavy(a, heavy + s0, v, r0, r1 - r0);
                            } else {  // settled up to lim - 1: a warp goes on
                                a.pos[v] = lim - 1;
                                along = true;
                            }
                        }
                    }
                }
                wq.push(keep, v);
                wj.push(light, v);
                wl.push(along, v);
            }
            wq.flush();
            wj.flush();
            wl.flush();
        }
        if (!grid_barrier(a.ctl, a.sticky, kSiteMis + 3)) return;

        // phase L: longer scans, one warp per vertex (up to kMisWarpChunks chunks of 32)
        const int n1 = ld_volatile_i32(l1len + s0);
        if (n1 > 0) {
            WQ wq(qbuf[wid][0], qn, qlen + s1);
            WQ wj(qbuf[wid][1], a.light, nlight + s0);
            const int gw = gtid >> 5, nw = gstride >> 5;
            for (int k = gw; k < n1; k += nw) {
                const int v = __ldcg(a.longq + k);
                const int r1 = __ldg(a.row_ptr + v + 1);
                const int start = __ldcg(a.pos + v) + 1;
                const unsigned pv = __ldg(a.prio + v);
                int stop = -1, c = 0;
                for (; c < kMisWarpChunks && start + 32 * c < r1; ++c) {
                    const int idx = start + 32 * c + lane;
                    const unsigned b = __ballot_sync(0xffffffffu, idx < r1 && mis_stop(a, idx, v, pv));
                    if (b) {
                        stop = start + 32 * c + __ffs(b) - 1;
                        break;
                    }
                }
                const bool end = stop < 0 && start + 32 * c >= r1;
                bool light = false;
                if (lane == 0) {
                    scanned += min(r1, stop >= 0 ? stop + 1 : start + 32 * c) - start;
                    if (stop >= 0) {
                        a.pos[v] = stop;
                    } else if (end) {
                        state[sx(v)] = kIn;
                        const int r0 = __ldg(a.row_ptr + v);
                        light = r1 - r0 <= kMisLightRow;
                        if (!light) mis_list_heavy(a, heavy + s0, v, r0, r1 - r0);
                    } else {
                        a.pos[v] = start + 32 * kMisWarpChunks - 1;
                        a.longq2[atomicAdd(l2len + s0, 1)] = v;
                    }
                }
                wq.push(stop >= 0 && lane == 0, v);
                wj.push(light, v);
            }
            wq.flush();
            wj.flush();
            if (!grid_barrier(a.ctl, a.sticky, kSiteMis + 4)) return;
        }

        // phase L2: the longest scans, one block per vertex
        const int n2 = n1 > 0 ? ld_volatile_i32(l2len + s0) : 0;
        if (n2 > 0) {
            for (int k = blockIdx.x; k < n2; k += G) {
                const int v = __ldcg(a.longq2 + k);
                const int r1 = __ldg(a.row_ptr + v + 1);
                const int start = __ldcg(a.pos + v) + 1;
                const unsigned pv = __ldg(a.prio + v);
                if (threadIdx.x == 0) s_stop = kInf;
                __syncthreads();
                for (int b0 = start; b0 < r1; b0 += kBlock) {
                    const int idx = b0 + threadIdx.x;
                    const bool st = idx < r1 && mis_stop(a, idx, v, pv);
                    if (st) atomicMin(&s_stop, idx);
                    if (__syncthreads_or(st)) break;
                }
                if (threadIdx.x == 0) {
                    const int spos = s_stop;
                    scanned += (spos != kInf ? spos + 1 : r1) - start;
                    if (spos != kInf) {
                        a.pos[v] = spos;
                        qn[atomicAdd(qlen + s1, 1)] = v;
                    } else {
                        state[sx(v)] = kIn;
                        const int r0 = __ldg(a.row_ptr + v);
                        if (r1 - r0 <= kMisLightRow)
                            a.light[atomicAdd(nlight + s0, 1)] = v;
                        else
                            mis_list_heavy(a, heavy + s0, v, r0, r1 - r0);
                    }
                }
                __syncthreads();
            }
            if (!grid_barrier(a.ctl, a.sticky, kSiteMis + 5)) return;
        }
    }
    long long insz = 0;
    for (int i = gtid; i < m; i += gstride) {
        const unsigned char s = a.state[sx(i)];
        if (a.member_i32)
            a.member_i32[i] = (s == kIn) ? 1 : 0;
        else
            a.member[i] = (s == kIn) ? 1 : 0;
        insz += (s == kIn);
    }
    long long work = scanned + pushed;
    for (int o = 16; o; o >>= 1) {
        insz += __shfl_down_sync(0xffffffffu, insz, o);
        work += __shfl_down_sync(0xffffffffu, work, o);
    }
    if (lane == 0 && insz)
        atomicAdd(reinterpret_cast<unsigned long long *>(&a.ctl->vertices_reached),
                  static_cast<unsigned long long>(insz));
    if (lane == 0 && work)
        atomicAdd(reinterpret_cast<unsigned long long *>(&a.ctl->edges_expanded),
                  static_cast<unsigned long long>(work));
    if (gtid == 0) {
        a.ctl->iterations = r;
        a.ctl->push_iterations = r;
        a.ctl->edges_component = a.nnz;
    }
}

// ================================================================================
// one-hop boolean SpMSpV (MIS validity helper)
// ================================================================================
__global__ void spmspv_bool_kernel(int m, const int *__restrict__ row_ptr,
                                   const int *__restrict__ col_ind, const int *__restrict__ x,
                                   int *y) {
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int u = warp; u < m; u += nwarps) {
        if (__ldg(x + u) == 0) continue;
        const int r0 = __ldg(row_ptr + u), r1 = __ldg(row_ptr + u + 1);
        for (int e = r0 + lane; e < r1; e += 32) y[__ldg(col_ind + e)] = 1;
    }
}

void set_bfs_buffers(BfsArgs &a, const TravBuffers &b, int m, int nnz) {
    a.q[0] = EdgeQueue{b.q0, b.q2, b.rs, nullptr, nullptr};
    a.q[1] = EdgeQueue{b.q1, b.q3, b.loc_off, nullptr, nullptr};
    a.vis[0] = b.bits0;
    a.vis[1] = b.bits1;
    a.shift = edge_unit_shift(nnz, static_cast<long long>(m) + 1, kEqTile);
}

apspie_status prepare_square(apspie_ctx *ctx, const apspie_csr *A, const char *who) {
    apspie_status st = check_csr_view(ctx, A, who);
    if (st != APSPIE_OK) return st;
    if (A->m != A->n)
        return set_error(ctx, APSPIE_ERR_INVALID_ARG, std::string(who) + ": matrix must be square");
    if (A->m <= 0) return set_error(ctx, APSPIE_ERR_INVALID_ARG, std::string(who) + ": empty graph");
    if (ctx->validate) {
        st = validate_csr(ctx, A, true);
        if (st != APSPIE_OK) return st;
    }
    return APSPIE_OK;
}


}  // namespace

// ================================================================================
// Allocation-free BFS: scratch in a file-scope device array
// ================================================================================
namespace {

constexpr size_t align256(size_t x) { return (x + 255) & ~size_t(255); }
constexpr size_t kNaMaxV = APSPIE_NOALLOC_MAX_VERTICES;
constexpr size_t kNaQueueBytes = align256((kNaMaxV + 1) * sizeof(int));
constexpr size_t kNaWordsBytes = align256(((kNaMaxV + 31) / 32) * sizeof(unsigned));
constexpr size_t kNaCtlBytes = align256(sizeof(TravCtl)) + 256;  // control block + sticky error word
constexpr size_t kNaBytes =
    kNaCtlBytes + 6 * kNaQueueBytes + 2 * kNaWordsBytes;

// Shared by every apspie_bfs_noalloc call in the process (one copy per device). It keeps
// the last call's contents; the control block is cleared at the start of each call and the
// kernel initialises every queue and bitmap it reads.
static __device__ __align__(256) unsigned char g_bfs_noalloc_scratch[kNaBytes];

// A __device__ array has one address per CUDA context: the primary context of each device,
// any context a caller made with cuCtxCreate, and a primary context re-created after
// cudaDeviceReset each hold their own copy. The address is therefore looked up once per
// context and cached under the context's process-unique id (cuCtxGetId), never under a
// device number or a context handle, which a re-created context may reuse.
struct NaEntry {
    unsigned long long ctx_id;
    void *addr;
};
std::vector<NaEntry> g_na_cache;
std::mutex g_na_mu;

// Device address of g_bfs_noalloc_scratch in the current context, looked up (with
// cudaGetSymbolAddress, which also loads the library's device code into the context under
// lazy module loading) on the first call in each context.
cudaError_t noalloc_scratch(void **out) {
    std::lock_guard<std::mutex> lock(g_na_mu);
    unsigned long long id = current_ctx_id();
    if (id != 0)
        for (const NaEntry &e : g_na_cache)
            if (e.ctx_id == id) {
                *out = e.addr;
                return cudaSuccess;
            }
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_bfs_noalloc_scratch);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return e;
    }
    if (id == 0) id = current_ctx_id();  // the lookup may have made the primary context current
    if (id != 0) g_na_cache.push_back({id, p});
    *out = p;
    return cudaSuccess;
}

}  // namespace

size_t traversal_scratch_need(int m) { return trav_scratch_bytes(m); }

// what mis_common reserves: the traversal buffers, the state array, the push-unit owners
// and the list of light joiners
size_t mis_scratch_need(int m) {
    const size_t mi = static_cast<size_t>(m) + 1;
    return trav_scratch_bytes(m) + Carver::need({static_cast<size_t>(m) * kMisStateStride, mi * 4, mi * 4});
}

apspie_status trav_reserve(apspie_ctx *ctx, int m) {
    void *base;
    return scratch_reserve(ctx, std::max(trav_scratch_bytes(m) + static_cast<size_t>(m) * 5 + 512, mis_scratch_need(m)),
                           &base);
}

}  // namespace apspie

using namespace apspie;

extern "C" {

apspie_status apspie_ctx_reserve(apspie_ctx *ctx, int32_t m, int64_t nnz) {
    (void)nnz;
    if (!ctx || m < 0) return APSPIE_ERR_INVALID_ARG;
    cudaSetDevice(ctx->device);
    return trav_reserve(ctx, m);
}

apspie_status apspie_bfs(apspie_ctx *ctx, const apspie_csr *A, int32_t source, int32_t depth_cap,
                         int32_t *d_depth, apspie_run_stats *stats) {
    if (!ctx) return APSPIE_ERR_INVALID_ARG;
    cudaSetDevice(ctx->device);
    apspie_status st = prepare_square(ctx, A, "apspie_bfs");
    if (st != APSPIE_OK) return st;
    if (source < 0 || source >= A->m)
        return set_error(ctx, APSPIE_ERR_INVALID_ARG, "apspie_bfs: source out of range");
    if (!d_depth) return set_error(ctx, APSPIE_ERR_INVALID_ARG, "apspie_bfs: NULL output");
    void *base;
    st = scratch_reserve(ctx, trav_scratch_bytes(A->m), &base);
    if (st != APSPIE_OK) return st;
    if ((st = reset_ctl(ctx)) != APSPIE_OK) return st;
    BfsArgs a;
    a.m = A->m;
    a.nnz = A->nnz;
    a.src = source;
    a.depth_cap = depth_cap;
    a.row_ptr = A->row_ptr;
    a.col_ind = A->col_ind;
    a.depth = d_depth;
    set_bfs_buffers(a, carve_trav(base, A->m), A->m, A->nnz);
    a.ctl = ctx->d_ctl;
    a.sticky = ctx->d_sticky_err;
    const apspie_tune_params tp = effective_params(ctx, APSPIE_TUNE_BFS, A);
    a.alpha = tp.bfs_alpha;
    a.beta = tp.bfs_beta;
    a.allow_pull = (A->flags & APSPIE_CSR_SYMMETRIC) ? 1 : 0;
    void *args[] = {&a};
    st = launch_persistent(ctx, reinterpret_cast<const void *>(bfs_kernel), kBfsBlock, args, A->nnz);
    if (st != APSPIE_OK) return st;
    return finish_call(ctx, stats, "apspie_bfs");
}

namespace apspie {
namespace {
apspie_status sssp_common(apspie_ctx *ctx, const apspie_csr *A, int32_t source, void *d_dist,
                          apspie_run_stats *stats, bool is_float, int unreached_bits);
}
}  // namespace apspie

apspie_status apspie_sssp(apspie_ctx *ctx, const apspie_csr *A, int32_t source, int32_t *d_dist,
                          apspie_run_stats *stats) {
    if (!ctx) return APSPIE_ERR_INVALID_ARG;
    if (A && A->val_type != APSPIE_VAL_I32)
        return set_error(ctx, APSPIE_ERR_INVALID_ARG, "apspie_sssp: int32 edge weights required");
    return sssp_common(ctx, A, source, d_dist, stats, false, -1);
}

apspie_status apspie_sssp_f32(apspie_ctx *ctx, const apspie_csr *A, int32_t source, float *d_dist,
                              float unreached, apspie_run_stats *stats) {
    if (!ctx) return APSPIE_ERR_INVALID_ARG;
    if (A && A->val_type != APSPIE_VAL_F32)
        return set_error(ctx, APSPIE_ERR_INVALID_ARG, "apspie_sssp_f32: float32 edge weights required");
    int bits;
    std::memcpy(&bits, &unreached, sizeof bits);
    return sssp_common(ctx, A, source, d_dist, stats, true, bits);
}

}  // extern "C"

namespace apspie {
namespace {
// Blocks of a launch: throughput grows with the warps on an SM (553 us with five blocks an SM
// against 568 us with four and 802 us with two at scale 20), but so do the barriers' times,
// and an iteration of a smaller graph has no more than a tile for each warp (6.7M entries:
// 306 us with three, 315 us with four, 333 us with five).
long long sssp_blocks(const apspie_ctx *ctx, long long nnz) {
    return static_cast<long long>(ctx->num_sms) * (nnz >= 25000000 ? 5 : nnz >= 12000000 ? 4 : 3);
}

// Edges per iteration: an eighth of the graph's where an iteration's edges are most of its
// time (scale 20: 571 us, a fifth 601 us), a fifth of smaller graphs', where its barriers and
// dependent reads are, so that fewer iterations pay for more relaxations (6.7M entries:
// 332 -> 314 us, 0.5M entries: 202 -> 190 us).
long long default_band(long long nnz) {
    const long long b = nnz >= (1LL << 24) ? nnz / 8 : nnz / 5;
    return b < (1LL << 16) ? (1LL << 16) : (b > (1LL << 23) ? (1LL << 23) : b);
}

apspie_status sssp_common(apspie_ctx *ctx, const apspie_csr *A, int32_t source, void *d_dist,
                          apspie_run_stats *stats, bool is_float, int unreached_bits) {
    cudaSetDevice(ctx->device);
    apspie_status st = prepare_square(ctx, A, "apspie_sssp");
    if (st != APSPIE_OK) return st;
    if (A->nnz > 0 && !A->val) return set_error(ctx, APSPIE_ERR_INVALID_ARG, "apspie_sssp: NULL weights");
    if (source < 0 || source >= A->m)
        return set_error(ctx, APSPIE_ERR_INVALID_ARG, "apspie_sssp: source out of range");
    if (!d_dist) return set_error(ctx, APSPIE_ERR_INVALID_ARG, "apspie_sssp: NULL output");
    void *base;
    st = scratch_reserve(ctx, trav_scratch_bytes(A->m), &base);
    if (st != APSPIE_OK) return st;
    if ((st = reset_ctl(ctx)) != APSPIE_OK) return st;
    SsspArgs a;
    a.m = A->m;
    a.nnz = A->nnz;
    a.src = source;
    a.row_ptr = A->row_ptr;
    a.col_ind = A->col_ind;
    a.w = static_cast<const int *>(A->val);
    a.dist = static_cast<int *>(d_dist);
    const apspie_tune_params tp = effective_params(ctx, APSPIE_TUNE_SSSP, A);
    a.delta_hint = tp.sssp_delta;
    if (tp.sssp_band > 0) {
        a.band = tp.sssp_band;
    } else if (tp.sssp_band == 0) {
        a.band = default_band(A->nnz);
    } else {
        a.band = 0;
    }
    a.unreached_bits = unreached_bits;
    a.buf = carve_trav(base, A->m);
    a.shift = edge_unit_shift(A->nnz, static_cast<long long>(A->m) + 1, 32 * kSsspVT);
    a.ctl = ctx->d_ctl;
    a.sticky = ctx->d_sticky_err;
    void *args[] = {&a};
    st = launch_persistent(ctx, is_float ? reinterpret_cast<const void *>(sssp_kernel<true>) : reinterpret_cast<const void *>(sssp_kernel<false>),
                           kBlock, args, sssp_blocks(ctx, A->nnz) * kWorkPerBlock);
    if (st != APSPIE_OK) return st;
    return finish_call(ctx, stats, "apspie_sssp");
}
}  // namespace

size_t sssp_group_scratch_need(int m, int groups) {
    const size_t per = (trav_scratch_bytes(m) + 255) / 256 * 256;
    return per * static_cast<size_t>(groups) + static_cast<size_t>(groups) * ((sizeof(TravCtl) + 255) / 256 * 256);
}

int sssp_group_count(const apspie_ctx *ctx, int nq) {
    int g = ctx->sssp_batch_groups > 0 ? ctx->sssp_batch_groups : 4;
    return std::max(1, std::min(g, nq));
}

apspie_status sssp_batch_grouped(apspie_ctx *ctx, const apspie_csr *A, const int32_t *d_sources, int32_t nq,
                                 int32_t *d_dists, apspie_run_stats *stats) {
    if (stats) std::memset(stats, 0, sizeof(*stats));
    if (nq == 0) return APSPIE_OK;
    const int m = A->m;
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &per_sm, reinterpret_cast<const void *>(sssp_group_kernel), kBlock, 0);
    if (e != cudaSuccess || per_sm < 1) return cuda_error(ctx, e, "occupancy query");
    const int cap = persistent_cap(ctx, per_sm);
    const int groups = std::min(sssp_group_count(ctx, nq), cap);
    const int bpg = std::min(cap / groups, kMaxGrid);
    void *base;
    apspie_status st = scratch_reserve(ctx, sssp_group_scratch_need(m, groups), &base);
    if (st != APSPIE_OK) return st;
    if ((st = reset_ctl(ctx)) != APSPIE_OK) return st;
    const size_t per = (trav_scratch_bytes(m) + 255) / 256 * 256;
    TravCtl *ctls = reinterpret_cast<TravCtl *>(static_cast<char *>(base) + per * groups);
    if ((e = cudaMemsetAsync(ctls, 0, groups * ((sizeof(TravCtl) + 255) / 256 * 256), ctx->stream)) != cudaSuccess)
        return cuda_error(ctx, e, "apspie_sssp_batch reset");
    SsspGroupArgs g;
    SsspArgs &a = g.base;
    std::memset(&a, 0, sizeof(a));
    a.m = m;
    a.nnz = A->nnz;
    a.row_ptr = A->row_ptr;
    a.col_ind = A->col_ind;
    a.w = static_cast<const int *>(A->val);
    const apspie_tune_params tp = effective_params(ctx, APSPIE_TUNE_SSSP, A);
    a.delta_hint = tp.sssp_delta;
    if (tp.sssp_band > 0) {
        a.band = tp.sssp_band;
    } else if (tp.sssp_band == 0) {
        // the single-query default, scaled to the group's share of the device
        const long long b = default_band(A->nnz) * bpg / cap;
        a.band = b < (1LL << 16) ? (1LL << 16) : b;
    } else {
        a.band = 0;
    }
    a.unreached_bits = -1;
    a.buf = carve_trav(base, m);
    a.shift = edge_unit_shift(A->nnz, static_cast<long long>(m) + 1, 32 * kSsspVT);
    a.sticky = ctx->d_sticky_err;
    g.srcs = d_sources;
    g.out = d_dists;
    g.nq = nq;
    g.groups = groups;
    g.m = m;
    g.ctls = ctls;
    g.buf_stride = per;
    g.main = ctx->d_ctl;
    void *args[] = {&g};
    e = cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(sssp_group_kernel), dim3(groups * bpg),
                                    dim3(kBlock), args, 0, ctx->stream);
    if (e != cudaSuccess) return cuda_error(ctx, e, "cooperative launch");
    return finish_call(ctx, stats, "apspie_sssp_batch");
}

}  // namespace apspie

extern "C" {

static apspie_status mis_common(apspie_ctx *ctx, const apspie_csr *A, const uint32_t *d_priority,
                                uint8_t *d_member, int32_t *d_member_i32, apspie_run_stats *stats);

apspie_status apspie_mis(apspie_ctx *ctx, const apspie_csr *A, const uint32_t *d_priority,
                         uint8_t *d_member, apspie_run_stats *stats) {
    if (!ctx) return APSPIE_ERR_INVALID_ARG;
    if (!d_member) return set_error(ctx, APSPIE_ERR_INVALID_ARG, "apspie_mis: NULL output");
    return mis_common(ctx, A, d_priority, d_member, nullptr, stats);
}

apspie_status apspie_mis_int32(apspie_ctx *ctx, const apspie_csr *A, const uint32_t *d_priority,
                               int32_t *d_mis_result, apspie_run_stats *stats) {
    if (!ctx) return APSPIE_ERR_INVALID_ARG;
    if (!d_mis_result) return set_error(ctx, APSPIE_ERR_INVALID_ARG, "apspie_mis_int32: NULL output");
    return mis_common(ctx, A, d_priority, nullptr, d_mis_result, stats);
}

static apspie_status mis_common(apspie_ctx *ctx, const apspie_csr *A, const uint32_t *d_priority,
                                uint8_t *d_member, int32_t *d_member_i32, apspie_run_stats *stats) {
    cudaSetDevice(ctx->device);
    apspie_status st = prepare_square(ctx, A, "apspie_mis");
    if (st != APSPIE_OK) return st;
    if (!d_priority) return set_error(ctx, APSPIE_ERR_INVALID_ARG, "apspie_mis: NULL priority");
    void *base;
    const size_t tb = trav_scratch_bytes(A->m);
    const size_t mi = static_cast<size_t>(A->m) + 1;
    st = scratch_reserve(ctx, mis_scratch_need(A->m), &base);
    if (st != APSPIE_OK) return st;
    if ((st = reset_ctl(ctx)) != APSPIE_OK) return st;
    MisArgs a;
    a.m = A->m;
    a.nnz = A->nnz;
    a.row_ptr = A->row_ptr;
    a.col_ind = A->col_ind;
    a.prio = d_priority;
    a.member = d_member;
    a.member_i32 = d_member_i32;
    const TravBuffers buf = carve_trav(base, A->m);
    a.pos = buf.aux;
    a.queue[0] = buf.q0;
    a.queue[1] = buf.q1;
    a.longq = buf.q2;
    a.longq2 = buf.aux2;
    a.heavy_v = buf.q3;
    a.heavy_base = buf.rs;
    a.heavy_delta = buf.loc_off;
    Carver c(static_cast<char *>(base) + tb);
    a.state = c.take<unsigned char>(static_cast<size_t>(A->m) * kMisStateStride);
    a.unit_owner = c.take<int>(mi);
    a.light = c.take<int>(mi);
    // push units hold at least 128 entries, and few enough that the units of a round's
    // pushes (at most nnz entries) fit the m + 1 slots of unit_owner
    a.unit_shift = 7;
    while ((static_cast<long long>(A->nnz) >> a.unit_shift) + 1 > static_cast<long long>(mi)) ++a.unit_shift;
    a.ctl = ctx->d_ctl;
    a.sticky = ctx->d_sticky_err;
    void *args[] = {&a};
    st = launch_persistent(ctx, reinterpret_cast<const void *>(mis_kernel), kBlock, args, A->nnz);
    if (st != APSPIE_OK) return st;
    return finish_call(ctx, stats, "apspie_mis");
}

apspie_status apspie_bfs_noalloc(const apspie_csr *A, int32_t source, int32_t depth_cap, int32_t *d_depth,
                                 void *cuda_stream, apspie_run_stats *stats) {
    if (!A || !d_depth || !A->row_ptr || (A->nnz > 0 && !A->col_ind) || A->m != A->n || A->m <= 0 ||
        A->nnz < 0)
        return APSPIE_ERR_INVALID_ARG;
    if (A->m > APSPIE_NOALLOC_MAX_VERTICES) return APSPIE_ERR_INVALID_ARG;  // beyond the static scratch
    if (source < 0 || source >= A->m) return APSPIE_ERR_INVALID_ARG;
    cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return APSPIE_ERR_CUDA;
    void *base = nullptr;
    if (noalloc_scratch(&base) != cudaSuccess) return APSPIE_ERR_CUDA;
    char *p = static_cast<char *>(base);
    TravCtl *ctl = reinterpret_cast<TravCtl *>(p);
    int *sticky = reinterpret_cast<int *>(p + align256(sizeof(TravCtl)));
    p += kNaCtlBytes;
    BfsArgs a;
    TravBuffers b{};
    int **queues[] = {&b.q0, &b.q1, &b.q2, &b.q3, &b.rs, &b.loc_off};
    for (int **q : queues) {
        *q = reinterpret_cast<int *>(p);
        p += kNaQueueBytes;
    }
    b.bits0 = reinterpret_cast<unsigned *>(p);
    b.bits1 = reinterpret_cast<unsigned *>(p + kNaWordsBytes);
    set_bfs_buffers(a, b, A->m, A->nnz);
    if (cudaMemsetAsync(ctl, 0, kNaCtlBytes, stream) != cudaSuccess) return APSPIE_ERR_CUDA;
    a.m = A->m;
    a.nnz = A->nnz;
    a.src = source;
    a.depth_cap = depth_cap;
    a.row_ptr = A->row_ptr;
    a.col_ind = A->col_ind;
    a.depth = d_depth;
    a.ctl = ctl;
    a.sticky = sticky;
    a.alpha = 14.0f;
    a.beta = 24.0f;
    a.allow_pull = (A->flags & APSPIE_CSR_SYMMETRIC) ? 1 : 0;
    int sms = 0, per_sm = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bfs_kernel, kBfsBlock, 0) != cudaSuccess ||
        per_sm < 1)
        return APSPIE_ERR_CUDA;
    long long grid = (static_cast<long long>(A->nnz) + kWorkPerBlock - 1) / kWorkPerBlock;
    if (grid < sms) grid = sms;
    if (grid > static_cast<long long>(per_sm) * sms) grid = static_cast<long long>(per_sm) * sms;
    if (grid > kMaxGrid) grid = kMaxGrid;
    void *args[] = {&a};
    if (cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(bfs_kernel), dim3(static_cast<int>(grid)),
                                    dim3(kBfsBlock), args, 0, stream) != cudaSuccess) {
        (void)cudaGetLastError();
        return APSPIE_ERR_CUDA;
    }
    TravCtl h;
    if (cudaMemcpyAsync(&h, ctl, kCtlHostBytes, cudaMemcpyDeviceToHost, stream) != cudaSuccess ||
        cudaStreamSynchronize(stream) != cudaSuccess)
        return APSPIE_ERR_CUDA;
    if (stats) {
        stats->iterations = h.iterations;
        stats->push_iterations = h.push_iterations;
        stats->pull_iterations = h.pull_iterations;
        stats->reserved = 0;
        stats->edges_expanded = h.edges_expanded;
        stats->edges_component = h.edges_component;
        stats->vertices_reached = h.vertices_reached;
    }
    return h.err != 0 ? static_cast<apspie_status>(h.err) : APSPIE_OK;
}

apspie_status apspie_spmspv_bool(apspie_ctx *ctx, const apspie_csr *A, const int32_t *d_x,
                                 int32_t *d_y) {
    if (!ctx) return APSPIE_ERR_INVALID_ARG;
    cudaSetDevice(ctx->device);
    apspie_status st = check_csr_view(ctx, A, "apspie_spmspv_bool");
    if (st != APSPIE_OK) return st;
    if (!d_x || !d_y) return set_error(ctx, APSPIE_ERR_INVALID_ARG, "apspie_spmspv_bool: NULL vector");
    if (ctx->validate && (st = validate_csr(ctx, A, false)) != APSPIE_OK) return st;
    cudaError_t e = cudaMemsetAsync(d_y, 0, static_cast<size_t>(A->n) * sizeof(int32_t), ctx->stream);
    if (e != cudaSuccess) return cuda_error(ctx, e, "spmspv_bool memset");
    if (A->m > 0) {
        spmspv_bool_kernel<<<ctx->num_sms * 8, 256, 0, ctx->stream>>>(A->m, A->row_ptr, A->col_ind,
                                                                      d_x, d_y);
        e = cudaGetLastError();
        if (e != cudaSuccess) return cuda_error(ctx, e, "spmspv_bool launch");
    }
    return APSPIE_OK;
}

}  // extern "C"
