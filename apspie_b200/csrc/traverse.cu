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
    kSiteMis = 300,  // and 301
};

struct TravBuffers {
    int *q0, *q1, *q2, *q3, *rs, *loc_off, *aux, *aux2, *aux3;
    unsigned *bits0, *bits1;
};

// What a call uses of these (a new context's first call is mostly their allocation): int arrays
// of m + 1, the last of them (two of BFS's, one of SSSP's) with room for the owners of an edge
// queue's units.
struct TravLists {
    int arrays, owners;
};
constexpr TravLists kBfsLists{4, 2}, kSsspLists{6, 1}, kSsspPileLists{8, 1};

size_t trav_scratch_bytes(int m, long long nnz, TravLists lists) {
    const size_t words = (static_cast<size_t>(m) + 31) / 32, mi = static_cast<size_t>(m) + 1;
    return Carver::need({words * 4, words * 4}) + lists.arrays * Carver::need({mi * 4}) +
           lists.owners * Carver::need({static_cast<size_t>(edge_owner_slots(m + 1ll, nnz)) * 4});
}

TravBuffers carve_trav(void *base, int m, long long nnz, TravLists lists) {
    const size_t words = (static_cast<size_t>(m) + 31) / 32, mi = static_cast<size_t>(m) + 1;
    const size_t slots = static_cast<size_t>(edge_owner_slots(m + 1ll, nnz));
    Carver c(base);
    TravBuffers b{};
    if (lists.owners == kBfsLists.owners) {
        for (int **p : {&b.q0, &b.q1, &b.q2, &b.q3}) *p = c.take<int>(mi);
        for (int **p : {&b.rs, &b.loc_off}) *p = c.take<int>(slots);
    } else {
        for (int **p : {&b.q0, &b.q1, &b.rs, &b.loc_off, &b.aux, &b.aux2}) *p = c.take<int>(mi);
        b.aux3 = c.take<int>(slots);
        if (lists.arrays == kSsspPileLists.arrays)
            for (int **p : {&b.q2, &b.q3}) *p = c.take<int>(mi);
    }
    b.bits0 = c.take<unsigned>(words);
    b.bits1 = c.take<unsigned>(words);
    return b;
}

// BFS's view of the buffers: edge queues in q0-q3, rs and loc_off, visited bitmaps in bits0-1.
struct BfsArgs;
void set_bfs_buffers(BfsArgs &a, const TravBuffers &b, int nnz, long long slots);

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
// lengths, two barriers a level and frontier bitmaps: 43.9 / 113 us; now 30 / 59 us. Blocks
// of 256 threads, three an SM: four an SM 36 / 65 us, 512 threads 38 / 65 us, 128 threads
// 34 / 68 us (fewer blocks make the barrier cheaper, more warps the pull levels).
template <bool WIDE>
__global__ void __launch_bounds__(kBfsBlock, 3) bfs_kernel(BfsArgs a) {
    __shared__ int s_buf[kBfsBlock / 32][kEqCap];
    __shared__ int s_slice[kBfsBlock / 32][kEqTile];
    __shared__ EqBlock<kBfsBlock> s_blk;
    __shared__ int s_claim[2];  // units taken, by level parity
    grid_begin(a.ctl);
    if (threadIdx.x == 0) s_blk.empty = s_claim[0] = s_claim[1] = 0;
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
        if (threadIdx.x == 0) s_claim[(L & 1) ^ 1] = 0;
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
            edge_expand<4, WIDE>(qc, static_cast<const NoPayload *>(nullptr), nq, E, a.shift, s_slice[wid],
                           &s_claim[L & 1], blockIdx.x, gridDim.x,
                        [&](const bool (&valid)[4], const NoPayload (&)[4], const int (&idx)[4]) {
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
    // q0/q1 near queues (vertices), q2/q3 far piles (if any); rs, loc_off, aux3 = the edge queue of the
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
    int claim[2];                         // units taken, by iteration parity
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
template <bool F, bool WIDE>
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
    if (threadIdx.x == 0) {
        sh.hmin = INF;
        sh.claim[0] = sh.claim[1] = 0;
    }
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
        if (threadIdx.x == 0) sh.claim[(iters & 1) ^ 1] = 0;
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
        edge_expand<kSsspVT, WIDE>(
            qa, snap, nact, E, a.shift, sh.slice[wid], &sh.claim[iters & 1], vg.id, G,
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

template <bool F, bool WIDE>
__global__ void __launch_bounds__(kBlock, 5) sssp_kernel(SsspArgs a) {
    grid_begin(a.ctl);
    sssp_body<F, WIDE>(a, hw_grid());
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
        sssp_body<false, true>(a, vg);
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
constexpr int kMisThread = 8;           // neighbours a thread scans before handing on to a warp
constexpr int kMisWarp = 1024;          // neighbours a warp scans before handing on to the block
constexpr int kMisPart = 16384;         // neighbours a block scans or pushes to in a pass
constexpr int kMisPush = -2;
constexpr int kMisLong = 256, kMisHuge = 32;  // room for scans handed on in a pass

struct MisArgs {
    int m, nnz;
    int tile, tiles;  // vertices that a block takes together (a power of two), and how many such
    const int *__restrict__ row_ptr;
    const int *__restrict__ col_ind;
    const unsigned *__restrict__ prio;
    unsigned char *member;
    int *member_i32;  // when set, the set is written here as int32 1/0 instead
    unsigned char *state;
    // each block's undecided vertices (two lists, by pass parity): the vertex, the CSR index its
    // scan stopped at, and the neighbour there that blocks it (-1: the scan goes on behind it)
    int *v, *pos, *by;
    size_t list;  // entries of one list
    TravCtl *ctl;
    int *sticky;
};

__device__ __forceinline__ bool outranks(unsigned pu, int u, unsigned pv, int v) {
    return pu > pv || (pu == pv && u > v);
}

__device__ __forceinline__ void mis_set(const MisArgs &a, int v, unsigned char s) {
    asm volatile("st.relaxed.gpu.global.u8 [%0], %1;" ::"l"(a.state + v), "r"(static_cast<unsigned>(s)) : "memory");
}

// A state as it is now, past L1.
__device__ __forceinline__ unsigned char mis_now(const MisArgs &a, int v) {
    unsigned s;
    asm volatile("ld.relaxed.gpu.global.u8 %0, [%1];" : "=r"(s) : "l"(a.state + v) : "memory");
    return static_cast<unsigned char>(s);
}

// Does neighbour u, in state su, decide anything for v: is it one that outranks v and is not
// out? Returns kOut for "nothing to stop at", else its state.
__device__ __forceinline__ unsigned char mis_look(int u, unsigned pu, unsigned char su, int v, unsigned pv) {
    return u == v || !outranks(pu, u, pv, v) ? kOut : su;
}

enum : int { kScanBlocked, kScanIn, kScanOut, kScanOn };

// A thread's scan of v from CSR index e to lim: where it stops (pos), at whom (by).
template <bool FIRST>
__device__ __forceinline__ int mis_scan_thread(const MisArgs &a, int v, unsigned pv, Pos e, Pos lim, int r1, int &pos,
                                               int &by) {
    for (; e < lim; e += 4) {
        int u[4];
        unsigned pu[4];
        unsigned char su[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) u[k] = e + k < lim ? __ldg(a.col_ind + e + k) : v;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            pu[k] = __ldg(a.prio + u[k]);
            if (!FIRST) su[k] = a.state[u[k]];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const unsigned char s = mis_look(u[k], pu[k], FIRST ? kUndecided : su[k], v, pv);
            if (s != kOut) {
                pos = static_cast<int>(e) + k;
                by = u[k];
                return s == kIn ? kScanOut : kScanBlocked;
            }
        }
    }
    pos = static_cast<int>(lim) - 1;
    by = -1;
    return lim >= static_cast<Pos>(r1) ? kScanIn : kScanOn;
}

// Greedy MIS in descending (priority, id) order -- the set spmspvMis converges to
// (src/spmspvMis.cuh:54-78: candidate if rand > threshold, select if rand > every
// candidate neighbour's, knock out the neighbours), with ties broken by id instead of
// left undecided. A vertex joins exactly when every neighbour that outranks it is out;
// it is out as soon as one of them has joined.
//
// Only outranking neighbours decide a vertex, and states never change once decided, so the
// kernel has no rounds: every block owns every G-th tile of up to 256 vertices and goes through its
// undecided ones again and again, on its own, until none is left. A vertex keeps the position
// of the first outranking neighbour that is not out (everything before it is settled for
// good): in -> the vertex is out; undecided -> look again in the next pass; out -> scan on
// behind it. The highest-ranked undecided vertex can always be decided, whichever block owns
// it, and all blocks are resident, so every block gets to its end; the set does not depend on
// timing. Scans go on by a warp past kMisThread neighbours and by the block past kMisWarp.
//
// A joiner stores "out" into its undecided neighbours, so that a vertex leaves as soon as any
// outranking neighbour is in, not only the one it waits for: without that, chains of waits
// thousands of passes long form (3,450 us instead of 283 at R-MAT scale 20). The store is kept
// from states already seen as out: without the look, every joiner stores into the lines of the
// same high-degree vertices (3,660 us). The first pass looks at ranks only, when nearly
// every state is still undecided (260 -> 240 us).
//
// Scans and pushes go on by a warp past kMisThread entries and by the block past kMisWarp,
// kMisPart at a time, so that one long row does not keep the block's other vertices waiting. Each
// step of such a scan looks at v's own state, past L1: in dense graphs one joiner's push goes through
// the very vertices that wait for one another, and those whose blocker it had already reached scanned
// thousands of entries that were out by then (a complete graph of 4,000 vertices 204 us,
// now 37, of 1,500 143 and 37).
// States are read through L1, which thread 0's acquire drops once a pass: every look in L2
// had all SMs poll the few lines of the high-degree vertices that most others wait for
// (240 -> 219 us; 418 -> 362 at 2M vertices). A stale state can only be "undecided" where it
// is decided by now, and costs a pass.
//
// What bounds it: the latency of each pass's chain of gathers (column, priority and state,
// mostly out of L2 and DRAM) and the number of decisions that follow one another; most of the
// entries, 7.5M of 31.4M, are looked at in the first two passes. Five blocks an SM (260 us)
// against four (280) and six (279); tiles of 64, 128 and 512 vertices, steps of 2 and 8
// entries and warp limits from 128 to 2,048 are all within 10 % or slower. With rounds (the
// joiners' pushes, then scans, each closed by a grid barrier: 22 barriers at scale 20) 376 us,
// now 219; 248 -> 125 us at 300,007 vertices, 60 -> 35 at 3,001; a path of 20,000 vertices
// in rank order, one decision after the other, 78 -> 15 ms.
//
// A block that decides nothing waits for others. It gives up (APSPIE_ERR_TIMEOUT) when no
// block has decided anything for the context's wait limit: blocks count their passes that did
// in ctl->aux[0].
__global__ void __launch_bounds__(kBlock, 5) mis_kernel(MisArgs a) {
    __shared__ int s_n[2], s_long, s_huge[2], s_decided, s_stop, s_end;
    __shared__ int s_lv[kMisLong], s_lp[kMisLong], s_hv[kMisHuge], s_hp[kMisHuge];
    grid_begin(a.ctl);
    const int G = gridDim.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int m = a.m;
    const int *col = a.col_ind;
    for (int i = blockIdx.x * kBlock + tid; i < m; i += G * kBlock) a.state[i] = kUndecided;
    // the part of the lists that holds this block's vertices
    const int tiles = a.tiles, each = tiles / G, extra = tiles % G, b = blockIdx.x;
    const size_t part = (static_cast<size_t>(b) * each + min(b, extra)) * a.tile;
    if (tid == 0) s_n[0] = s_n[1] = s_long = s_huge[0] = s_huge[1] = s_decided = s_end = 0;
    if (!grid_barrier(a.ctl, a.sticky, kSiteMis)) return;

    long long insz = 0, scanned = 0;
    auto decide = [&](int v, bool in) {
        mis_set(a, v, in ? kIn : kOut);
        if (a.member_i32)
            a.member_i32[v] = in ? 1 : 0;
        else
            a.member[v] = in ? 1 : 0;
        insz += in;
        s_decided = 1;
    };
    auto keep = [&](int to, int v, int pos, int by) {
        const size_t at = part + to * a.list + atomicAdd(&s_n[to], 1);
        a.v[at] = v;
        a.pos[at] = pos;
        a.by[at] = by;
    };
    // hands v's scan behind pos (kMisPush: the push of a joiner) on to a warp; without room it
    // goes on in the next pass
    auto hand_on = [&](int to, int v, int pos, int from) {
        const int at = atomicAdd(&s_long, 1);
        if (at < kMisLong) {
            s_lv[at] = v;
            s_lp[at] = from;
            return true;
        }
        keep(to, v, pos, -1);
        return false;
    };
    auto outcome = [&](int to, int code, int v, int pos, int by) {
        if (code == kScanOut) {
            decide(v, false);
        } else if (code == kScanBlocked) {
            keep(to, v, pos, by);
        } else if (code == kScanOn) {
            hand_on(to, v, pos, pos);
        } else {
            const Pos r0 = __ldg(a.row_ptr + v), r1 = __ldg(a.row_ptr + v + 1);
            if (r1 - r0 > kMisThread) {
                if (hand_on(to, v, static_cast<int>(r1) - 1, kMisPush)) decide(v, true);
            } else {
                decide(v, true);
                scanned += r1 - r0;
                for (Pos e = r0; e < r1; e += 4) {
                    int u[4];
                    unsigned char s[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) u[k] = e + k < r1 ? __ldg(col + e + k) : v;
#pragma unroll
                    for (int k = 0; k < 4; ++k) s[k] = a.state[u[k]];
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (u[k] != v && s[k] == kUndecided) mis_set(a, u[k], kOut);
                }
            }
        }
    };
    unsigned long long t0 = 0, seen = 0;  // thread 0's: when something was last decided anywhere
    int pass = 0, idle = 0;
    for (;; ++pass) {
        const int cur = pass & 1, nxt = cur ^ 1;
        if (pass == 0) {
            for (int t = b; t < tiles; t += G) {
                const int v = t * a.tile + tid;
                if (tid >= a.tile || v >= m) continue;
                const int r0 = __ldg(a.row_ptr + v), r1 = __ldg(a.row_ptr + v + 1);
                int pos = 0, by = -1;
                const int code = mis_scan_thread<true>(a, v, __ldg(a.prio + v), r0, step_end(r0, kMisThread, r1), r1, pos, by);
                scanned += pos + 1 - r0;
                outcome(nxt, code, v, pos, by);
            }
        } else {
            const int n = s_n[cur];
            for (int i = tid; i < n; i += kBlock) {
                const size_t at = part + cur * a.list + i;
                const int v = a.v[at], by = a.by[at];
                int pos = a.pos[at];
                if (by == v) {  // a push that goes on
                    const int h = atomicAdd(&s_huge[cur], 1);
                    if (h < kMisHuge) {
                        s_hv[h] = v;
                        s_hp[h] = pos;
                    } else {
                        keep(nxt, v, pos, v);
                    }
                    continue;
                }
                const int r1 = __ldg(a.row_ptr + v + 1);  // fetched alongside the states
                const unsigned pv = __ldg(a.prio + v);
                const unsigned char own = a.state[v];
                const unsigned char s = by < 0 ? kOut : a.state[by];
                if (own == kOut) {
                    decide(v, false);
                } else if (s == kUndecided) {
                    keep(nxt, v, pos, by);
                } else if (s == kIn) {
                    decide(v, false);
                } else {
                    const int e = pos + 1;
                    int who = -1;
                    const int code =
                        mis_scan_thread<false>(a, v, pv, e, step_end(e, kMisThread, r1), r1, pos, who);
                    scanned += pos + 1 - e;
                    outcome(nxt, code, v, pos, who);
                }
            }
        }
        __syncthreads();
        // longer scans, a warp each, 128 neighbours a step
        const int nlong = min(s_long, kMisLong);
        for (int i = wid; i < nlong; i += kBlock / 32) {
            const int v = s_lv[i];
            const Pos r1 = __ldg(a.row_ptr + v + 1);
            if (s_lp[i] == kMisPush) {
                const Pos r0 = __ldg(a.row_ptr + v);
                if (r1 - r0 > kMisWarp) {
                    if (lane == 0) {
                        const int at = atomicAdd(&s_huge[cur], 1);
                        if (at < kMisHuge) {
                            s_hv[at] = v;
                            s_hp[at] = -2 - static_cast<int>(r0);
                        } else {
                            keep(nxt, v, -2 - static_cast<int>(r0), v);
                        }
                    }
                    continue;
                }
                for (Pos e = r0; e < r1; e += 128) {
                    int u[4];
                    unsigned char s[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) u[k] = e + 32 * k + lane < r1 ? __ldg(col + e + 32 * k + lane) : v;
#pragma unroll
                    for (int k = 0; k < 4; ++k) s[k] = a.state[u[k]];
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (u[k] != v && s[k] == kUndecided) mis_set(a, u[k], kOut);
                }
                if (lane == 0) scanned += r1 - r0;
                continue;
            }
            const int first = s_lp[i] + 1;
            const unsigned pv = __ldg(a.prio + v);
            const Pos lim = step_end(first, kMisWarp, r1);
            int code = lim >= r1 ? kScanIn : kScanOn, pos = static_cast<int>(lim) - 1, by = -1;
            for (Pos e = first; e < lim; e += 128) {
                int u[4];
                unsigned char s[4];
                unsigned pu[4];
                const unsigned char own = e > first ? mis_now(a, v) : static_cast<unsigned char>(kUndecided);
#pragma unroll
                for (int k = 0; k < 4; ++k) u[k] = e + 32 * k + lane < lim ? __ldg(col + e + 32 * k + lane) : v;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    pu[k] = __ldg(a.prio + u[k]);
                    s[k] = a.state[u[k]];
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) s[k] = mis_look(u[k], pu[k], s[k], v, pv);
#pragma unroll
                for (int k = 3; k >= 0; --k) {  // the first stop counts
                    const unsigned stops = __ballot_sync(0xffffffffu, s[k] != kOut);
                    if (stops) {
                        const int l = __ffs(stops) - 1;
                        pos = static_cast<int>(e) + 32 * k + l;
                        by = __shfl_sync(0xffffffffu, u[k], l);
                        code = __shfl_sync(0xffffffffu, static_cast<int>(s[k]), l) == kIn ? kScanOut : kScanBlocked;
                    }
                }
                if (__any_sync(0xffffffffu, own == kOut)) code = kScanOut, by = v;
                if (by >= 0) break;
            }
            if (lane == 0) {
                scanned += pos + 1 - first;
                if (code == kScanIn) {
                    keep(nxt, v, static_cast<int>(r1) - 1, -1);  // joins in the next pass, which hands its push on
                } else if (code != kScanOn) {
                    outcome(nxt, code, v, pos, by);
                } else {
                    const int at = atomicAdd(&s_huge[cur], 1);
                    if (at < kMisHuge) {
                        s_hv[at] = v;
                        s_hp[at] = pos;
                    } else {
                        keep(nxt, v, pos, -1);
                    }
                }
            }
        }
        __syncthreads();
        // the longest, by the block, 1,024 neighbours a step and kMisPart at a time
        const int nhuge = min(s_huge[cur], kMisHuge);
        for (int i = 0; i < nhuge; ++i) {
            const int v = s_hv[i], r1 = __ldg(a.row_ptr + v + 1), p = s_hp[i];
            if (p < -1) {  // a push, from CSR index -2 - p on
                const int first = -2 - p, lim = step_end(first, kMisPart, r1);
                for (Pos e = first + tid; e < static_cast<Pos>(lim); e += 4 * kBlock) {
                    int u[4];
                    unsigned char s[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) u[k] = e + k * kBlock < static_cast<Pos>(lim) ? __ldg(col + e + k * kBlock) : v;
#pragma unroll
                    for (int k = 0; k < 4; ++k) s[k] = a.state[u[k]];
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (u[k] != v && s[k] == kUndecided) mis_set(a, u[k], kOut);
                }
                if (tid == 0) {
                    s_decided = 1;
                    scanned += lim - first;
                    if (lim < r1) keep(nxt, v, -2 - lim, v);
                }
                continue;
            }
            const int first = p + 1, lim = step_end(first, kMisPart, r1);
            const unsigned pv = __ldg(a.prio + v);
            if (tid == 0) s_stop = kInf;
            __syncthreads();
            for (Pos e = first; e < static_cast<Pos>(lim); e += 4 * kBlock) {
                int stop = kInf, u[4];
                unsigned pu[4];
                unsigned char s[4];
                if (tid == 0 && mis_now(a, v) == kOut) stop = -1;
#pragma unroll
                for (int k = 0; k < 4; ++k) u[k] = e + k * kBlock + tid < static_cast<Pos>(lim) ? __ldg(col + e + k * kBlock + tid) : v;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    pu[k] = __ldg(a.prio + u[k]);
                    s[k] = a.state[u[k]];
                }
#pragma unroll
                for (int k = 3; k >= 0; --k)
                    if (stop >= 0 && mis_look(u[k], pu[k], s[k], v, pv) != kOut) stop = static_cast<int>(e) + k * kBlock + tid;
                if (stop != kInf) atomicMin(&s_stop, stop);
                if (__syncthreads_or(stop != kInf)) break;
            }
            if (tid == 0) {
                const int stop = s_stop;
                s_decided = 1;
                scanned += (stop != kInf && stop >= 0 ? stop + 1 : lim) - first;
                if (stop < 0)
                    decide(v, false);
                else if (stop == kInf)
                    keep(nxt, v, lim - 1, -1);  // goes on, or joins, in the next pass
                else
                    keep(nxt, v, stop, __ldg(col + stop));  // whose state may have changed since
            }
            __syncthreads();
        }
        if (tid == 0) {
            // the next pass reads states through L1, which this acquire has dropped
            ld_acquire_u64(&a.ctl->aux[0]);
            s_n[cur] = 0;
            s_long = 0;
            s_huge[nxt] = 0;  // (a warp may still be about to read this pass's)
            if (s_n[nxt] == 0) s_end = 1;
            if (s_decided) {
                s_decided = 0;
                idle = 0;
                t0 = 0;
                if (!s_end) atomicAdd(reinterpret_cast<unsigned long long *>(&a.ctl->aux[0]), 1ull);
            } else if ((++idle & 63) == 0) {
                const unsigned long long now = globaltimer_ns();
                const unsigned long long count = *reinterpret_cast<volatile unsigned long long *>(&a.ctl->aux[0]);
                const unsigned long long limit = a.ctl->wait_limit_ns ? a.ctl->wait_limit_ns : kBarrierTimeoutNs;
                if (ld_volatile_i32(&a.ctl->err) != 0) s_end = 1;
                if (t0 == 0 || count != seen) {
                    t0 = now;
                    seen = count;
                } else if (now - t0 > limit) {
                    raise_error(a.ctl, a.sticky, APSPIE_ERR_TIMEOUT, kSiteMis + 1);
                    s_end = 1;
                }
            }
        }
        __syncthreads();
        if (s_end) break;
    }
    long long work = scanned;
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
    if (tid == 0) {
        atomicMax(&a.ctl->iterations, pass + 1);
        atomicMax(&a.ctl->push_iterations, pass + 1);
        if (blockIdx.x == 0) a.ctl->edges_component = a.nnz;
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

void set_bfs_buffers(BfsArgs &a, const TravBuffers &b, int nnz, long long slots) {
    a.q[0] = EdgeQueue{b.q0, b.q2, b.rs, nullptr, nullptr};
    a.q[1] = EdgeQueue{b.q1, b.q3, b.loc_off, nullptr, nullptr};
    a.vis[0] = b.bits0;
    a.vis[1] = b.bits1;
    a.shift = edge_unit_shift(nnz, slots, kEqTile);
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

size_t traversal_scratch_need(int m, long long nnz) { return trav_scratch_bytes(m, nnz, kSsspLists); }

// Pull levels need a symmetric pattern, and step past a row's end in an int.
int bfs_may_pull(const apspie_csr *A) { return (A->flags & APSPIE_CSR_SYMMETRIC) && A->nnz <= kMaxStepped; }
const void *bfs_fn(const apspie_csr *A) {
    return A->nnz <= kMaxStepped ? reinterpret_cast<const void *>(bfs_kernel<false>)
                                 : reinterpret_cast<const void *>(bfs_kernel<true>);
}

// Blocks of a BFS launch, one to three an SM: more shorten a level's expansion, fewer its barrier
// and its queue (a block's reservations are made one after the other). R-MAT, one / two / three:
// 1.7M entries 32.5 / 34.0 / 37.2 us; 4.3M 37.2 / 36.9 / 41.1; 7.6M 44.7 / 41.4 / 43.6; 11.7M
// 52.2 / 45.8 / 45.8; 31.4M 86 / 64 / 60.
long long bfs_blocks(int num_sms, long long nnz) {
    return static_cast<long long>(num_sms) * (nnz >= 10000000 ? 3 : nnz >= 3000000 ? 2 : 1);
}

// what mis_common reserves: the states and the blocks' lists (whole tiles)
size_t mis_scratch_need(int m) {
    const size_t l = (static_cast<size_t>(m) + kBlock) * 8;
    return Carver::need({static_cast<size_t>(m), l, l, l});
}

apspie_status trav_reserve(apspie_ctx *ctx, int m, long long nnz) {
    void *base;
    return scratch_reserve(ctx, std::max(trav_scratch_bytes(m, nnz, kSsspPileLists) + static_cast<size_t>(m) * 5 + 512, mis_scratch_need(m)),
                           &base);
}

}  // namespace apspie

using namespace apspie;

extern "C" {

apspie_status apspie_ctx_reserve(apspie_ctx *ctx, int32_t m, int64_t nnz) {
    if (!ctx || m < 0) return APSPIE_ERR_INVALID_ARG;
    cudaSetDevice(ctx->device);
    return trav_reserve(ctx, m, std::max<long long>(0, nnz));
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
    st = scratch_reserve(ctx, trav_scratch_bytes(A->m, A->nnz, kBfsLists), &base);
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
    set_bfs_buffers(a, carve_trav(base, A->m, A->nnz, kBfsLists), A->nnz, edge_owner_slots(A->m + 1ll, A->nnz));
    a.ctl = ctx->d_ctl;
    a.sticky = ctx->d_sticky_err;
    const apspie_tune_params tp = effective_params(ctx, APSPIE_TUNE_BFS, A);
    a.alpha = tp.bfs_alpha;
    a.beta = tp.bfs_beta;
    a.allow_pull = bfs_may_pull(A);
    void *args[] = {&a};
    st = launch_persistent(ctx, bfs_fn(A), kBfsBlock, args,
                           bfs_blocks(ctx->num_sms, A->nnz) * kWorkPerBlock);
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
// 306 us with three, 315 us with four, 333 us with five; 3.1M: 247 us with three, 239 with two;
// 0.43M: 190 with three, 177 with one; 0.04M: 168 and 160).
long long sssp_blocks(const apspie_ctx *ctx, long long nnz) {
    return static_cast<long long>(ctx->num_sms) *
           (nnz >= 25000000 ? 5 : nnz >= 12000000 ? 4 : nnz >= 5000000 ? 3 : nnz >= 1200000 ? 2 : 1);
}

// Edges per iteration: an eighth of the graph's where an iteration's edges are most of its
// time (scale 20: 571 us, a fifth 601 us), a fifth of smaller graphs', where its barriers and
// dependent reads are, so that fewer iterations pay for more relaxations (6.7M entries:
// 332 -> 314 us, 0.5M entries: 202 -> 190 us).
long long default_band(long long nnz) {
    const long long b = nnz >= (1LL << 24) ? nnz / 8 : nnz / 5;
    return b < (1LL << 16) ? (1LL << 16) : (b > (1LL << 23) ? (1LL << 23) : b);
}

// A far pile is kept with a step, or without a band (as the kernel decides).
TravLists sssp_lists(const SsspArgs &a) { return a.delta_hint > 0 || a.band <= 0 ? kSsspPileLists : kSsspLists; }

apspie_status sssp_common(apspie_ctx *ctx, const apspie_csr *A, int32_t source, void *d_dist,
                          apspie_run_stats *stats, bool is_float, int unreached_bits) {
    cudaSetDevice(ctx->device);
    apspie_status st = prepare_square(ctx, A, "apspie_sssp");
    if (st != APSPIE_OK) return st;
    if (A->nnz > 0 && !A->val) return set_error(ctx, APSPIE_ERR_INVALID_ARG, "apspie_sssp: NULL weights");
    if (source < 0 || source >= A->m)
        return set_error(ctx, APSPIE_ERR_INVALID_ARG, "apspie_sssp: source out of range");
    if (!d_dist) return set_error(ctx, APSPIE_ERR_INVALID_ARG, "apspie_sssp: NULL output");
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
    void *base;
    const TravLists lists = sssp_lists(a);
    st = scratch_reserve(ctx, trav_scratch_bytes(A->m, A->nnz, lists), &base);
    if (st != APSPIE_OK) return st;
    if ((st = reset_ctl(ctx)) != APSPIE_OK) return st;
    a.unreached_bits = unreached_bits;
    a.buf = carve_trav(base, A->m, A->nnz, lists);
    a.shift = edge_unit_shift(A->nnz, edge_owner_slots(A->m + 1ll, A->nnz), 32 * kSsspVT);
    a.ctl = ctx->d_ctl;
    a.sticky = ctx->d_sticky_err;
    void *args[] = {&a};
    const bool wide = A->nnz > kMaxStepped;
    const void *fn = is_float ? wide ? reinterpret_cast<const void *>(sssp_kernel<true, true>)
                                     : reinterpret_cast<const void *>(sssp_kernel<true, false>)
                     : wide   ? reinterpret_cast<const void *>(sssp_kernel<false, true>)
                              : reinterpret_cast<const void *>(sssp_kernel<false, false>);
    st = launch_persistent(ctx, fn, kBlock, args, sssp_blocks(ctx, A->nnz) * kWorkPerBlock);
    if (st != APSPIE_OK) return st;
    return finish_call(ctx, stats, "apspie_sssp");
}
}  // namespace

size_t sssp_group_scratch_need(int m, long long nnz, int groups) {
    const size_t per = (trav_scratch_bytes(m, nnz, kSsspPileLists) + 255) / 256 * 256;
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
    apspie_status st = scratch_reserve(ctx, sssp_group_scratch_need(m, A->nnz, groups), &base);
    if (st != APSPIE_OK) return st;
    if ((st = reset_ctl(ctx)) != APSPIE_OK) return st;
    const size_t per = (trav_scratch_bytes(m, A->nnz, kSsspPileLists) + 255) / 256 * 256;
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
    a.buf = carve_trav(base, m, A->nnz, kSsspPileLists);
    a.shift = edge_unit_shift(A->nnz, edge_owner_slots(m + 1ll, A->nnz), 32 * kSsspVT);
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
    // First a tile for every block: few vertices of many neighbours are as much work as many of few
    // (5,001 vertices, 0.63M entries: 95 us with tiles of 256, now 81; 65,536 and 1.8M: 118, 108).
    a.tile = kBlock;
    while (a.tile > 32 && a.tile * 5ll * ctx->num_sms > A->m) a.tile >>= 1;
    a.tiles = (A->m - 1) / a.tile + 1;
    Carver c(base);
    a.state = c.take<unsigned char>(static_cast<size_t>(A->m));
    a.list = static_cast<size_t>(A->m) + kBlock;
    a.v = c.take<int>(2 * a.list);
    a.pos = c.take<int>(2 * a.list);
    a.by = c.take<int>(2 * a.list);
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
    set_bfs_buffers(a, b, A->nnz, static_cast<long long>(kNaMaxV) + 1);
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
    a.allow_pull = bfs_may_pull(A);
    int sms = 0, per_sm = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bfs_fn(A), kBfsBlock, 0) != cudaSuccess ||
        per_sm < 1)
        return APSPIE_ERR_CUDA;
    long long grid = bfs_blocks(sms, A->nnz);
    if (grid > static_cast<long long>(per_sm) * sms) grid = static_cast<long long>(per_sm) * sms;
    if (grid > kMaxGrid) grid = kMaxGrid;
    void *args[] = {&a};
    if (cudaLaunchCooperativeKernel(bfs_fn(A), dim3(static_cast<int>(grid)),
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
