// What the persistent traversal kernels share: the merge-path frontier expander (batched BFS) and the
// edge queues (BFS, SSSP and batched SSSP).
//
// It replaces the reference's per-level library chain (src/mXv.cuh:142-176,
// src/spmspvBfs.cuh:178-186, src/spmspvMis.cuh:245-263): Scan -> streamCompact ->
// IntervalGather(row lengths) -> Scan -> IntervalGather(row starts) ->
// IntervalGather/Expand(neighbours), with two D2H count reads per level. Here:
//
//  phase A  every block takes a contiguous chunk of the frontier queue, reads each
//           entry's CSR row start and length, and writes a block-local exclusive scan
//           of the lengths plus one chunk total (no host round trip);
//  barrier
//  phase B  every block loads the chunk totals (the second level of the scan). The merge
//           path of (frontier entries, edges) is cut into warp tiles of 32*VT items; each
//           block owns a contiguous run of them. The block finds the split point of every
//           tile of a batch in parallel (one two-level binary search per thread: chunk
//           bases in shared memory, then the chunk's local offsets), then each warp walks
//           its tiles on its own: it stages the tile's entries in its shared-memory slice,
//           merges them per lane to label every edge slot with its owning entry, and hands
//           each lane VT edges (strided, so a row's neighbour indices are read coalesced)
//           whose loads the operation issues back to back. No block barrier inside the
//           tile loop; the semiring operation runs on every (entry, edge) pair in the same
//           pass (no materialised neighbour list, no sort).
#pragma once

#include <type_traits>

#include "common.cuh"

namespace apspie {

// Per-warp staging slice.
template <int WT>
struct WarpSlice {
    int off[WT + 1];   // global edge offset of each staged entry
    int rs[WT + 1];    // CSR row start of each staged entry
    int aux[WT + 1];   // per-entry payload
    int seg[WT];       // tile edge slot -> staged entry
};

// ROOM: ints that the kernel uses a warp's slice for otherwise, outside the expansion.
template <int BLOCK, int VT, int ROOM = 1>
struct ExpandSmem {
    static constexpr int NWARP = BLOCK / 32;
    static constexpr int WT = 32 * VT;  // items (entries + edges) per warp tile
    static constexpr int BATCH = BLOCK; // warp tiles whose splits are found together
    using Warp = WarpSlice<WT>;
    static constexpr int QCAP = 128;  // per-warp queue staging (see WarpQueue)
    int qbuf[NWARP][2][QCAP];
    int base[kMaxGrid + 1];  // exclusive prefix of chunk totals
    int tsplit[BATCH + 1];   // merge-path split of each warp tile of the current batch
    int next_tile;           // tiles of the batch handed out so far (warps take them in turn)
    int scan_tmp[33];
    union Slice {
        Warp w;
        int room[ROOM];
    } w[NWARP];
};

// Phase A over this block's chunk of queue q[0, nf). hook(i, v, deg) may rewrite the
// degree (e.g. 0 for an entry that needs no expansion) and do per-entry work.
template <int BLOCK, class Hook>
__device__ __forceinline__ void frontier_phase_a(const int *__restrict__ q, int nf,
                                                 const int *__restrict__ row_ptr, int *rs,
                                                 int *loc_off, int *chunk_sum, int *scan_tmp,
                                                 Hook hook) {
    const int G = gridDim.x;
    const int C = (nf + G - 1) / G;
    const int c0 = min(static_cast<int>(blockIdx.x) * C, nf);
    const int c1 = min(c0 + C, nf);
    int carry = 0;
    for (int base = c0; base < c1; base += BLOCK) {
        const int i = base + threadIdx.x;
        int deg = 0;
        if (i < c1) {
            const int v = __ldcg(q + i);
            const int r0 = __ldg(row_ptr + v);
            deg = __ldg(row_ptr + v + 1) - r0;
            deg = hook(i, v, deg);
            rs[i] = r0;
        }
        int tot;
        const int ex = block_exclusive_scan<BLOCK>(deg, tot, scan_tmp);
        if (i < c1) loc_off[i] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0) chunk_sum[blockIdx.x] = carry;
}

// Loads the chunk totals of phase A into base[] as an exclusive prefix; returns the total
// number of edges of the frontier.
template <int BLOCK>
__device__ __forceinline__ int frontier_chunk_bases(const int *__restrict__ chunk_sum, int *base,
                                                    int *scan_tmp) {
    const int G = gridDim.x;
    const int per = (G + BLOCK - 1) / BLOCK;
    const int t0 = threadIdx.x * per;
    int local = 0;
    for (int k = 0; k < per; ++k)
        if (t0 + k < G) local += __ldcg(chunk_sum + t0 + k);
    int tot;
    int run = block_exclusive_scan<BLOCK>(local, tot, scan_tmp);
    for (int k = 0; k < per; ++k)
        if (t0 + k < G) {
            base[t0 + k] = run;
            run += __ldcg(chunk_sum + t0 + k);
        }
    if (threadIdx.x == 0) base[G] = tot;
    __syncthreads();
    return tot;
}

// Number of entries among the first `diag` items of the merge of entry offsets
// (offset(j) = base[j / C] + loc_off[j]) with edge indices 0..E-1, entries first on ties.
// The first entry of every chunk has loc_off 0, so the search first bisects the chunk
// starts in shared memory and then at most one chunk's local offsets in global memory.
__device__ __forceinline__ int frontier_merge_path(long long diag, int nf, int E,
                                                   const int *__restrict__ loc_off,
                                                   const int *base, int C) {
    long long lo = diag - E > 0 ? diag - E : 0;
    long long hi = diag < nf ? diag : nf;
    if (lo >= hi) return static_cast<int>(lo);
    long long clo = (lo + C - 1) / C, chi = (hi - 1) / C;
    while (clo <= chi) {
        const long long c = (clo + chi) >> 1;
        if (base[c] <= diag - 1 - c * C) {
            lo = c * C + 1;
            clo = c + 1;
        } else {
            hi = c * C;
            chi = c - 1;
        }
    }
    if (lo < hi) {
        const int cb = base[lo / C];
        while (lo < hi) {
            const long long mid = (lo + hi) >> 1;
            if (cb + __ldcg(loc_off + mid) <= diag - 1 - mid)
                lo = mid + 1;
            else
                hi = mid;
        }
    }
    return static_cast<int>(lo);
}

// Phase B. load(j, k, ws) stages entry j's payload into the warp slice at k;
// op(valid, k, idx, ws) handles a lane's VT edges (CSR positions idx[], owning staged
// entries k[]). Both are called by every lane of the warp, so they may use warp collectives.
// Warps claim the tiles of their block's batch in turn.
template <int BLOCK, int VT, int ROOM, class Load, class Op>
__device__ __forceinline__ void frontier_expand(int nf, int E, const int *__restrict__ loc_off,
                                                const int *__restrict__ rs,
                                                ExpandSmem<BLOCK, VT, ROOM> &sm, Load load, Op op) {
    using S = ExpandSmem<BLOCK, VT, ROOM>;
    constexpr int WT = S::WT;
    constexpr int NWARP = S::NWARP;
    constexpr int BATCH = S::BATCH;
    const int G = gridDim.x;
    const int C = (nf + G - 1) / G;
    const long long total = static_cast<long long>(nf) + E;
    const long long ntiles = (total + WT - 1) / WT;
    const int lane = threadIdx.x & 31;
    const int wid = threadIdx.x >> 5;
    typename S::Warp &ws = sm.w[wid].w;
    // one warp tile: stage its entries, label its edge slots, run the operation
    auto run_tile = [&](long long tile, long long tb) {
        const long long d0 = tile * WT;
        const long long d1 = d0 + WT < total ? d0 + WT : total;
        const int a0 = sm.tsplit[tile - tb];
        const int a1 = sm.tsplit[tile - tb + 1];
        const int e0 = static_cast<int>(d0 - a0);
        const int e1 = static_cast<int>(d1 - a1);
        const int jb = a0 > 0 ? a0 - 1 : 0;
        const int ne = a1 - jb;
        // the tile's entries lie in chunk jb / C and, with chunks at least as long as a tile, the
        // next one
        const int jc = jb / C, jn = (jc + 1) * C;
        for (int k = lane; k < ne; k += 32) {
            const int j = jb + k;
            const int c = C >= WT ? jc + (j >= jn ? 1 : 0) : j / C;
            ws.off[k] = sm.base[c] + __ldcg(loc_off + j);
            ws.rs[k] = __ldcg(rs + j);
            load(j, k, ws);
        }
        __syncwarp();
        const int tcount = static_cast<int>(d1 - d0);
        const int diag = lane * VT;
        if (diag < tcount) {
            const int acount = a1 - a0, bcount = e1 - e0;
            int lo = diag - bcount > 0 ? diag - bcount : 0;
            int hi = diag < acount ? diag : acount;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (ws.off[a0 + mid - jb] <= e0 + diag - 1 - mid)
                    lo = mid + 1;
                else
                    hi = mid;
            }
            int ja = a0 + lo, eb = e0 + diag - lo;
            int cur = ja - 1 - jb;
            const int end = diag + VT < tcount ? diag + VT : tcount;
            for (int it = diag; it < end; ++it) {
                if (ja < a1 && ws.off[ja - jb] <= eb) {
                    cur = ja - jb;
                    ++ja;
                } else {
                    ws.seg[eb - e0] = cur;
                    ++eb;
                }
            }
        }
        __syncwarp();
        const int ned = e1 - e0;
        bool valid[VT];
        int kk[VT], idx[VT];
#pragma unroll
        for (int r = 0; r < VT; ++r) {
            const int el = r * 32 + lane;
            valid[r] = el < ned;
            kk[r] = 0;
            idx[r] = 0;
            if (valid[r]) {
                kk[r] = ws.seg[el];
                idx[r] = ws.rs[kk[r]] + (e0 + el - ws.off[kk[r]]);
            }
        }
        op(valid, kk, idx, ws);
        __syncwarp();
    };
    // the tiles [tb, te) of one batch: split points found together, then the warps
    auto run_batch = [&](long long tb, long long te) {
        for (int s = threadIdx.x; s <= te - tb; s += BLOCK) {
            long long d = (tb + s) * WT;
            if (d > total) d = total;
            sm.tsplit[s] = frontier_merge_path(d, nf, E, loc_off, sm.base, C);
        }
        if (threadIdx.x == 0) sm.next_tile = NWARP;
        __syncthreads();
        // a warp that finishes its tile takes the next unclaimed one, so tiles of uneven
        // cost (atomics, queue flushes) do not leave warps idle at the batch's barrier
        for (long long tile = tb + wid; tile < te;) {
            run_tile(tile, tb);
            int nt = 0;
            if (lane == 0) nt = atomicAdd(&sm.next_tile, 1);
            tile = tb + __shfl_sync(0xffffffffu, nt, 0);
            __syncwarp();
        }
        __syncthreads();
    };
    const long long per = (ntiles + G - 1) / G;
    const long long t_begin = static_cast<long long>(blockIdx.x) * per;
    const long long t_end = t_begin + per < ntiles ? t_begin + per : ntiles;
    for (long long tb = t_begin; tb < t_end; tb += BATCH) run_batch(tb, tb + BATCH < t_end ? tb + BATCH : t_end);
}

// ---- edge queues ----------------------------------------------------------------------
// A frontier queue whose entries carry the running sum of their row lengths, so that the
// kernel that reads it needs neither a scan nor a search. Whoever appends entries reserves
// room for them and for their edges with one 64-bit atomic on (entries << 32 | edges), which
// makes edge offsets ascend with entry indices; an entry records its offset, its row start
// minus that offset, and, for every unit of 1 << shift edges that begins inside its row, its
// index as that unit's owner. A reader takes a unit per warp: the owner, the entries from it
// on, and the edges, all of them a fixed number of dependent reads.
//
// It replaces phase A, its grid barrier and the merge-path searches above where the entries'
// row lengths are final when they are appended (BFS), and the searches where an iteration takes its
// entries off another queue first (SSSP, batched SSSP); rows of length zero are only counted.
struct EdgeQueue {
    int *off;                  // edge offset of each entry
    int *delta;                // row start - off: edge t of the queue is CSR entry t + delta
    int *owner;                // entry that holds the first edge of each unit
    unsigned long long *size;  // entries << 32 | edges
    int *empty;                // entries without edges (counted, not stored)
};

constexpr int kEqTile = 128;  // edges of a BFS warp at a time: four per lane
constexpr int kEqCap = kEqTile + 32;  // vertices a warp stages before it appends them

// Per block: what its warps append at the end of a phase.
template <int BLOCK>
struct EqBlock {
    unsigned long long size[BLOCK / 32];  // per warp: entries << 32 | edges, then where they go
    int empty;
};

__device__ __forceinline__ void eq_own(int *owner, int shift, int idx, int off, int deg, int first, int step) {
    const int c1 = (off + deg - 1) >> shift;
    for (int c = (off > 0 ? ((off - 1) >> shift) + 1 : 0) + first; c <= c1; c += step) owner[c] = idx;
}

// Writes entry idx (row start r0, deg > 0 edges from offset off on; nothing if !some) and its
// units' owners; all lanes of the warp call it. A row of many units is shared out among the
// lanes.
__device__ __forceinline__ void eq_write(int *q_off, int *q_delta, int *q_owner, int shift, bool some, int idx, int off,
                                         int r0, int deg) {
    if (some) {
        q_off[idx] = off;
        q_delta[idx] = r0 - off;
    }
    const bool wide = some && deg >> shift >= 64;
    if (some && !wide) eq_own(q_owner, shift, idx, off, deg, 0, 1);
    for (unsigned m = __ballot_sync(0xffffffffu, wide); m; m &= m - 1) {
        const int l = __ffs(m) - 1;
        eq_own(q_owner, shift, __shfl_sync(0xffffffffu, idx, l), __shfl_sync(0xffffffffu, off, l),
               __shfl_sync(0xffffffffu, deg, l), threadIdx.x & 31, 32);
    }
}

// Appends the warp's `count` staged vertices. With blk (then every warp of the block calls it)
// room is reserved for the whole block at once: reservations are made one after the other in
// L2. Once a reservation ends past `enough` entries or edges, the reader of the queue is known
// not to need its entries (the next level pulls): they are counted and not written, which
// spares the owners of the highest-degree vertices' rows (a source's first neighbours are
// those: one warp wrote their owners for 8 us of a 15 us level at scale 20).
template <int BLOCK>
__device__ __forceinline__ void eq_append(const int *buf, int count, EqBlock<BLOCK> *blk, const EdgeQueue &q,
                                              const int *__restrict__ row_ptr, int shift, int enough_entries,
                                              int enough_edges) {
    constexpr int PER = kEqCap / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncwarp();
    int r0[PER], deg[PER];
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int i = k * 32 + lane;
        const int v = i < count ? buf[i] : -1;
        r0[k] = v >= 0 ? __ldg(row_ptr + v) : 0;
        deg[k] = v >= 0 ? __ldg(row_ptr + v + 1) : 0;
    }
    int n = 0, d = 0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        deg[k] -= r0[k];
        n += deg[k] > 0;
        d += deg[k];
    }
    int sn = n, sd = d;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int yn = __shfl_up_sync(0xffffffffu, sn, o), yd = __shfl_up_sync(0xffffffffu, sd, o);
        if (lane >= o) {
            sn += yn;
            sd += yd;
        }
    }
    unsigned long long base =
        (static_cast<unsigned long long>(static_cast<unsigned>(sn)) << 32) | static_cast<unsigned>(sd);
    if (blk) {
        if (lane == 31) {
            blk->size[warp] = base;
            if (sn < count) atomicAdd(&blk->empty, count - sn);
        }
        __syncthreads();
        if (warp == 0) {
            const unsigned long long mine = lane < BLOCK / 32 ? blk->size[lane] : 0ull;
            unsigned long long sum = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long y = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += y;
            }
            unsigned long long at = 0ull;
            if (lane == 31) {
                if (sum) at = atomicAdd(q.size, sum);
                if (blk->empty) atomicAdd(q.empty, blk->empty);
                blk->empty = 0;
            }
            at = __shfl_sync(0xffffffffu, at, 31);
            if (lane < BLOCK / 32) blk->size[lane] = at + sum - mine;
        }
        __syncthreads();
        base = blk->size[warp];
    } else {
        if (lane == 31) {
            base = atomicAdd(q.size, base);
            if (sn < count) atomicAdd(q.empty, count - sn);
        }
        base = __shfl_sync(0xffffffffu, base, 31);
    }
    int idx = static_cast<int>(base >> 32) + sn - n;
    int off = static_cast<int>(base & 0xffffffffull) + sd - d;
    const int all_n = __shfl_sync(0xffffffffu, idx + n, 31), all_d = __shfl_sync(0xffffffffu, off + d, 31);
    if (count == 0 || all_n > enough_entries || all_d > enough_edges) return;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const bool some = deg[k] > 0;
        eq_write(q.off, q.delta, q.owner, shift, some, idx, off, r0[k], deg[k]);
        idx += some;
        off += deg[k];
    }
}

// Owners' room for a queue of at most `entries` entries and nnz edges: one for each entry, or for
// each tile where those are more, up to 2^20. Dense graphs of few vertices have many tiles an
// entry: with a unit for each vertex a frontier's edges were a few warps' (hop counts on a complete
// graph of 3,000 vertices 97 us instead of 31, distances 457 instead of 176).
inline long long edge_owner_slots(long long entries, long long nnz) {
    const long long tiles = (nnz >> 7) + 1 < (1 << 20) ? (nnz >> 7) + 1 : 1 << 20;
    return entries > tiles ? entries : tiles;
}

// Smallest unit (a power of two, at least a tile) for which the units of up to nnz edges fit
// `slots` owners.
__host__ __device__ inline int edge_unit_shift(long long nnz, long long slots, int tile) {
    int s = 7;
    while ((1 << s) < tile) ++s;
    while ((nnz >> s) + 1 > slots) ++s;
    return s;
}

struct NoPayload {};
__device__ __forceinline__ NoPayload ld_payload(const NoPayload *) { return NoPayload{}; }
template <class P>
__device__ __forceinline__ P ld_payload(const P *p) {
    return __ldcg(p);
}

// op(valid, pay, idx) on every edge of the queue, VT per lane (CSR positions idx[]; pay[] is the
// `payload` of each edge's entry, unless NoPayload), called by all lanes of the warp. A tile's
// entries are read 32 at a time; where each begins goes into a mask of its edges in registers, so
// an edge finds its entry by counting bits. `slice`: shared memory private to the warp, 32 * VT
// ints and payloads; units are at least a tile. A block has every nblocks-th unit and its warps take
// them in turn (`claim`: in shared memory, zero at first): units differ in their rows and in what
// they improve, and with a fixed share per warp the blocks waited for their slowest warps (SSSP
// scale 20 558 -> 534 us, batched SSSP 8.75 -> 8.03 ms, BFS 60.1 -> 58.9 us). WIDE: E may be more
// than kMaxStepped (a plain step is up to 1 % faster in BFS and SSSP, the other one 4 % in batched
// SSSP). (Fetching the next tile's entries, columns and weights
// while one is worked on made SSSP slower: 650 us against 619 us at scale 20.)
template <int VT, bool WIDE, class P, class Op>
__device__ __forceinline__ void edge_expand(const EdgeQueue &q, const P *payload, int nf, int E, int shift,
                                            int *slice, int *claim, int block, int nblocks, Op op) {
    constexpr int TILE = 32 * VT;
    constexpr bool PAY = !std::is_same<P, NoPayload>::value;
    P *pslice = reinterpret_cast<P *>(slice + TILE);
    const int lane = threadIdx.x & 31;
    const unsigned upto = lane == 31 ? 0xffffffffu : (2u << lane) - 1u;
    const int units = E > 0 ? ((E - 1) >> shift) + 1 : 0;
    auto take = [&]() {
        int i = 0;
        if (lane == 0) i = atomicAdd(claim, 1);
        const long long u = block + static_cast<long long>(__shfl_sync(0xffffffffu, i, 0)) * nblocks;
        return static_cast<int>(u < units ? u : units);
    };
    for (int u = take(); u < units; u = take()) {
        int k = __ldcg(q.owner + u);
        // the next unit's owner, read beside it: when it is the same entry, the unit lies inside
        // that entry's row
        const bool one = u + 1 < units && __ldcg(q.owner + u + 1) == k;
        const long long uend = (static_cast<long long>(u) + 1) << shift;
        const int end = uend < E ? static_cast<int>(uend) : E;
        for (int t0 = u << shift, t1; t0 < end; t0 = WIDE ? t1 : t0 + TILE) {
            t1 = WIDE ? step_end(t0, TILE, end) : min(t0 + TILE, end);
            unsigned begin[VT];
#pragma unroll
            for (int r = 0; r < VT; ++r) begin[r] = 0u;
            int n = 0, next = 0x7fffffff;
            if (one) {
                if (lane == 0) slice[0] = __ldcg(q.delta + k);
                if (PAY && lane == 1) pslice[0] = ld_payload(payload + k);
                begin[0] = 1u;
                n = 1;
            }
            while (!one) {
                const int j = k + n + lane;
                const int o = j < nf ? __ldcg(q.off + j) : 0x7fffffff;
                const int d = j < nf ? __ldcg(q.delta + j) : 0;
                const P p = PAY && j < nf ? ld_payload(payload + j) : P{};
                const bool in = o < t1;
                const int s = o > t0 ? o - t0 : 0;
                if (in) slice[n + lane] = d;
                if (PAY && in) pslice[n + lane] = p;
#pragma unroll
                for (int r = 0; r < VT; ++r)
                    begin[r] |= __reduce_or_sync(0xffffffffu, in && (s >> 5) == r ? 1u << (s & 31) : 0u);
                const int c = __popc(__ballot_sync(0xffffffffu, in));
                n += c;
                if (c < 32) {
                    next = __shfl_sync(0xffffffffu, o, c);
                    break;
                }
            }
            __syncwarp();
            bool valid[VT];
            P pay[VT];
            int idx[VT];
            int before = -1;
#pragma unroll
            for (int r = 0; r < VT; ++r) {
                const int x = r * 32 + lane, t = static_cast<int>(static_cast<Pos>(t0) + x);  // past 2^31: not valid
                const int i = before + __popc(begin[r] & upto);
                before += __popc(begin[r]);
                valid[r] = WIDE ? x < t1 - t0 : t < t1;
                idx[r] = valid[r] ? t + slice[i] : 0;
                pay[r] = PAY && valid[r] ? pslice[i] : P{};
            }
            op(valid, pay, idx);
            k += next == t1 ? n : n - 1;  // the entry that holds the next tile's first edge
            __syncwarp();
        }
    }
}

}  // namespace apspie
