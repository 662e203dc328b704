// Triangle counting as a masked SpGEMM: count = sum((L*L) .* L) for the strict lower
// triangle L of a symmetric graph, without materialising L*L.
//
// The reference builds L and U on the host (buildLower, test/tc/main.cu:39-55), forms
// D = U*L with cuSPARSE csrgemm (tc.cuh:62-165, D is materialised), intersects each
// column of D with the same column of U in one thread per column (ewiseMultTc,
// tc.cuh:168-199) and reduces a float vector (mgpu::Reduce, test/tc/main.cu:249).
//
// Here L's edges are first re-oriented on the device from the endpoint of lower
// (degree, id) rank to the higher one: D is another acyclic orientation of the same
// undirected edge set, so sum((D*D) .* D) is the same count, but every row of D has at
// most about sqrt(2 * nnz) entries and the wedge total drops (R-MAT scale 18: 1.11G wedges
// under L, 0.66G under D, largest row 8,083 -> 411).
//
// On up to 1.6M vertices the count is then taken edge by edge, each as the intersection of
// its endpoints' rows of D, the longer one a bitmap in shared memory (see tc_bits; rows that are
// both short a warp's, see tc_small). Larger
// graphs, and inputs that the bitmaps cannot count, take masks in hash sets: each row i of D
// is loaded into a hash set (its mask); every wedge (k in D(i,:), j in D(k,:)) probes the set, and hits are
// counted in int64. Rows with masks of at most 256 entries are cut into warp tasks of at
// most task_work wedges (4096 unless tuned); each task loads its row's mask into a
// 512-slot shared-memory set, so skewed rows cannot unbalance the warps. Larger masks
// take a block with a 4096-slot shared set, or a block with a global set. An input with
// an entry on or above the diagonal is not a strict lower triangle; it is counted as
// given, sum((L*L) .* L), without re-orientation (also when orientation is tuned off).
#include <algorithm>
#include <cstring>

#include "common.cuh"

namespace apspie {
namespace {

constexpr int kTcBlock = 256;
constexpr int kEmpty = -1;
constexpr int kTcBins = 4;        // 0 nothing to do | 1 warp | 2 block/shared | 3 block/global
constexpr int kWarpSet = 512;     // slots (mask <= 256)
#ifndef APSPIE_TC_CHUNKS
#define APSPIE_TC_CHUNKS 4
#endif
constexpr int kTcChunks = APSPIE_TC_CHUNKS;  // 32-wedge chunks a warp gathers at once
constexpr int kBlockSet = 4096;   // slots (mask <= 2048)

struct TcInfo {
    int bin_count[kTcBins];
    long long global_slots;
    unsigned long long count;
    int overflow;
    int not_lower;  // an entry with column >= row
    int unsorted;   // a row whose entries don't ascend strictly (it may hold an entry twice)
    int ticket;     // owners handed out
    int beyond;     // entries of D far back in their lists (tc_even_limit)
    int owners[3];  // owners with many partners, with few, vertices with short lists (tc_owners)
};

__device__ __forceinline__ unsigned tc_hash(int key, int log2ts) {
    return (static_cast<unsigned>(key) * 2654435761u) >> (32 - log2ts);
}

// 8 lanes per row: mask size d and wedge count; the row's bin goes to row_bin and, for a
// warp-tier row, its number of warp tasks (task_work wedges each) to ntask.
__global__ void tc_rowinfo(int m, const int *__restrict__ rp, const int *__restrict__ ci, int task_work,
                           unsigned char *row_bin, int *ntask, long long *tbl_off, TcInfo *info) {
    const int sub = threadIdx.x & 7;
    const int grp = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
    const int ngrp = (gridDim.x * blockDim.x) >> 3;
    const unsigned gmask = 0xffu << (threadIdx.x & 24);
    for (int i0 = grp - (grp & 3); i0 < m; i0 += ngrp) {  // the warp's 4 groups move together
        const int i = i0 + (grp & 3);
        int r0 = 0, r1 = 0;
        long long work = 0;
        if (i < m) {
            r0 = __ldg(rp + i);
            r1 = __ldg(rp + i + 1);
            if (r1 - r0 >= 2)
                for (int e = r0 + sub; e < r1; e += 8) {
                    const int k = __ldg(ci + e);
                    work += __ldg(rp + k + 1) - __ldg(rp + k);
                }
        }
        for (int o = 4; o; o >>= 1) work += __shfl_down_sync(gmask, work, o, 8);
        if (i < m && sub == 0) {
            const int d = r1 - r0;
            int b;
            if (d < 2 || work == 0)
                b = 0;
            else if (d <= kWarpSet / 2)
                b = 1;
            else if (d <= kBlockSet / 2)
                b = 2;
            else
                b = 3;
            row_bin[i] = static_cast<unsigned char>(b);
            ntask[i] = b == 1 ? static_cast<int>((work + task_work - 1) / task_work) : 0;
            if (b == 3) {
                long long ts = 64;
                while (ts < 2LL * d) ts <<= 1;
                tbl_off[i] = static_cast<long long>(
                    atomicAdd(reinterpret_cast<unsigned long long *>(&info->global_slots),
                              static_cast<unsigned long long>(ts)));
            }
        }
    }
}

// Per-bin row lists (stride m, bin 0 skipped): warp ballots count a block's rows per
// bin, one global atomic per bin reserves their room.
__global__ void tc_binlists(int m, const unsigned char *__restrict__ row_bin, int *bin_rows, TcInfo *info) {
    __shared__ int cnt[kTcBins];
    __shared__ int base[kTcBins];
    const int lane = threadIdx.x & 31;
    for (int c0 = blockIdx.x * blockDim.x; c0 < m; c0 += gridDim.x * blockDim.x) {
        if (threadIdx.x < kTcBins) cnt[threadIdx.x] = 0;
        __syncthreads();
        const int i = c0 + threadIdx.x;
        const int b = i < m ? row_bin[i] : 0;
        int pos = 0;
#pragma unroll
        for (int k = 1; k < kTcBins; ++k) {
            const unsigned mk = __ballot_sync(0xffffffffu, b == k);
            int wbase = 0;
            if (mk && lane == __ffs(mk) - 1) wbase = atomicAdd(&cnt[k], __popc(mk));
            wbase = __shfl_sync(0xffffffffu, wbase, mk ? __ffs(mk) - 1 : 0);
            if (b == k) pos = wbase + __popc(mk & ((1u << lane) - 1u));
        }
        __syncthreads();
        if (threadIdx.x >= 1 && threadIdx.x < kTcBins && cnt[threadIdx.x])
            base[threadIdx.x] = atomicAdd(&info->bin_count[threadIdx.x], cnt[threadIdx.x]);
        __syncthreads();
        if (b > 0) bin_rows[static_cast<long long>(b) * m + base[b] + pos] = i;
        __syncthreads();
    }
}

// ---------------------------------------------------------------- degree orientation
// All passes over L's entries take an entry per thread (a warp per row left rows of 8,000
// entries to one warp), and places are handed out by the atomics that count, so the scatters
// need none: degrees and orientation of R-MAT scale 18 (3.8M entries) take 0.15 ms (0.72 before).

// deg[v] = |L(v,:)| (tc_columns adds the column's entries)
__global__ void tc_row_lengths(int m, const int *__restrict__ rp, int *deg) {
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < m; v += gridDim.x * blockDim.x)
        deg[v] = __ldg(rp + v + 1) - __ldg(rp + v);
}

// deg[j] += 1 for every entry (i, j). The highest-degree columns take tens of thousands of
// additions each, and additions to one word are made one after the other in L2: a block
// first adds up in shared memory, in a slot per column modulo kTcSlots that belongs to the
// first column that uses it (others go straight to L2), and adds each slot once at the end.
constexpr int kTcSlots = 4096;
constexpr int kTcColumnsBlock = 512;
__global__ void __launch_bounds__(kTcColumnsBlock) tc_columns(unsigned nnz, int m, const unsigned *__restrict__ row,
                                                              const int *__restrict__ ci, int *deg, TcInfo *info) {
    __shared__ int s_col[kTcSlots], s_cnt[kTcSlots];
    for (int k = threadIdx.x; k < kTcSlots; k += kTcColumnsBlock) {
        s_col[k] = kEmpty;
        s_cnt[k] = 0;
    }
    __syncthreads();
    bool bad = false, unsorted = false;
    for (unsigned e = blockIdx.x * kTcColumnsBlock + threadIdx.x; e < nnz; e += gridDim.x * kTcColumnsBlock) {
        const int i = static_cast<int>(__ldg(row + e)), j = __ldg(ci + e);
        bad |= j >= i || j < 0;
        unsorted |= e > 0 && __ldg(ci + e - 1) >= j && static_cast<int>(__ldg(row + e - 1)) == i;
        if (j < 0 || j >= m) continue;
        const int k = j & (kTcSlots - 1);
        int of = s_col[k];
        if (of == kEmpty) of = atomicCAS(s_col + k, kEmpty, j);
        if (of == kEmpty || of == j)
            atomicAdd(s_cnt + k, 1);
        else
            atomicAdd(deg + j, 1);
    }
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(&info->not_lower, 1);
    if (__any_sync(0xffffffffu, unsorted) && (threadIdx.x & 31) == 0) atomicOr(&info->unsorted, 1);
    __syncthreads();
    for (int k = threadIdx.x; k < kTcSlots; k += kTcColumnsBlock)
        if (s_cnt[k]) atomicAdd(deg + s_col[k], s_cnt[k]);
}

// The edge of entry (i, j) leaves the endpoint of lower (degree, id) rank; without degrees, i.
__device__ __forceinline__ void tc_edge(const int *deg, int i, int j, int &a, int &b) {
    bool fwd = true;
    if (deg) {
        const int di = __ldg(deg + i), dj = __ldg(deg + j);
        fwd = di < dj || (di == dj && i < j);
    }
    a = fwd ? i : j;
    b = fwd ? j : i;
}

// Edges between vertices with short lists are counted by a warp for each vertex (tc_small), the
// others from the bitmap of the longer list by a block (tc_bits): its round of setting, testing
// and clearing takes 0.4 to 1.8 us, whatever it tests, and the larger the bitmap the fewer blocks
// there are. "Short" is up to 64 entries in graphs of about even degrees (up to 32 edges a vertex,
// and less than 1 in 32 of D's entries past three times the mean list: grids, uniform graphs);
// else it grows with the vertices, and the blocks count everything up to 131,072, and up to 8,192
// in any graph (what a launch takes is more than what it spares). Whole counts in
// us, with hash sets / all by blocks / so: a 1,024 x 1,024 grid 1,440 / 13,340 / 604, uniform 2^19
// (10M edges) 1,226 / 3,380 / 1,082, 2^16 (0.5M) 192 / 227 / 142, 2^16 (2M) 367 / 379 / 350; R-MAT of
// 1.5M (ef 4) 3,270 / 3,560 / 1,526, 2^19 (ef 20) 12,960 / 2,640 / 2,354, 2^18 (ef 16) 3,620 / 866 /
// 850; of 2^16 (ef 6) 339 / 173 / 173 (181 with lists up to 16, 222 with 64).
constexpr int kTcSmallList = 64, kTcNoSmall = 8192;
inline int tc_even_limit(int m, unsigned nnz) {  // past which D's entries are counted
    return m <= kTcNoSmall ? 0x7fffffff : 3 * static_cast<int>(nnz / m + 1);
}
__device__ __forceinline__ int tc_small_list(int m, unsigned nnz, const TcInfo *info) {
    if (m <= kTcNoSmall) return 0;
    if (nnz / m < 32 && static_cast<unsigned>(info->beyond) <= nnz / 32) return kTcSmallList;
    return m <= 131072 ? 0 : min(kTcSmallList, m >> 13);
}

// place[e] = the edge's place in its tail's list; len[a] the list's length
__global__ void tc_out_places(unsigned nnz, const unsigned *__restrict__ row, const int *__restrict__ ci,
                              const int *__restrict__ deg, int *len, int *place, int even_limit, TcInfo *info) {
    __shared__ int s_beyond;
    if (info->not_lower) return;
    if (threadIdx.x == 0) s_beyond = 0;
    __syncthreads();
    int beyond = 0;
    for (unsigned e = blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += gridDim.x * blockDim.x) {
        int a, b;
        tc_edge(deg, static_cast<int>(__ldg(row + e)), __ldg(ci + e), a, b);
        const int at = atomicAdd(len + a, 1);
        place[e] = at;
        beyond += at >= even_limit;
    }
    if (even_limit == 0x7fffffff) return;
    beyond = __reduce_add_sync(0xffffffffu, beyond);
    if ((threadIdx.x & 31) == 0 && beyond) atomicAdd(&s_beyond, beyond);
    __syncthreads();
    if (threadIdx.x == 0 && s_beyond) atomicAdd(&info->beyond, s_beyond);
}

// The same in two passes, for the hash path: the lists' lengths, then D, its places handed out by
// a second count in `cursor`. Nothing is kept per edge between the two.
__global__ void tc_out_lengths(unsigned nnz, const unsigned *__restrict__ row, const int *__restrict__ ci,
                               const int *__restrict__ deg, int *len, const TcInfo *info) {
    if (info->not_lower) return;
    for (unsigned e = blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += gridDim.x * blockDim.x) {
        int a, b;
        tc_edge(deg, static_cast<int>(__ldg(row + e)), __ldg(ci + e), a, b);
        atomicAdd(len + a, 1);
    }
}
__global__ void tc_out_lists(unsigned nnz, const unsigned *__restrict__ row, const int *__restrict__ ci,
                             const int *__restrict__ deg, const int *__restrict__ drp, int *cursor, int *dci,
                             const TcInfo *info) {
    if (info->not_lower) return;
    for (unsigned e = blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += gridDim.x * blockDim.x) {
        int a, b;
        tc_edge(deg, static_cast<int>(__ldg(row + e)), __ldg(ci + e), a, b);
        dci[__ldg(drp + a) + atomicAdd(cursor + a, 1)] = b;
    }
}

// Writes D (unless D is L as it is: dci null) and
// hands out the edge's place in its owner's list of partners; -1 where the shorter list is
// empty or both are short (tc_small).
__global__ void tc_owner_places(unsigned nnz, const unsigned *__restrict__ row, const int *__restrict__ ci,
                                const int *__restrict__ deg, const int *__restrict__ drp, int *dci, int *place,
                                int *partners, int m, const TcInfo *info) {
    if (info->not_lower) return;
    if (info->unsorted) partners = nullptr;  // the hash sets count it
    const int small_list = tc_small_list(m, nnz, info);
    for (unsigned e = blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += gridDim.x * blockDim.x) {
        int a, b;
        tc_edge(deg, static_cast<int>(__ldg(row + e)), __ldg(ci + e), a, b);
        const int a0 = __ldg(drp + a), la = __ldg(drp + a + 1) - a0;
        const int lb = __ldg(drp + b + 1) - __ldg(drp + b);
        if (dci) dci[a0 + place[e]] = b;
        if (!partners) continue;
        // la > 0: it holds this edge
        const int owner = lb <= 0 || max(la, lb) <= small_list ? -1 : la >= lb ? a : b;
        // consecutive entries often have one owner: one atomic for the lanes that share it
        const unsigned active = __activemask();
        if (!__any_sync(active, owner >= 0)) {
            place[e] = -1;
            continue;
        }
        const unsigned peers = __match_any_sync(active, owner);
        const int first = __ffs(peers) - 1, lane = threadIdx.x & 31;
        int base = 0;
        if (lane == first && owner >= 0) base = atomicAdd(partners + owner, __popc(peers));
        base = __shfl_sync(peers, base, first);
        place[e] = owner >= 0 ? base + __popc(peers & ((1u << lane) - 1u)) : -1;
    }
}

__device__ __forceinline__ void set_insert(int *keys, long long ts, int log2ts, int key, TcInfo *info) {
    unsigned long long s = tc_hash(key, log2ts) & (ts - 1);
    for (long long p = 0; p <= ts; ++p) {
        const int old = atomicCAS(keys + s, kEmpty, key);
        if (old == kEmpty || old == key) return;
        s = (s + 1) & (ts - 1);
    }
    atomicOr(&info->overflow, 1);
}

template <bool COHERENT>
__device__ __forceinline__ bool set_find(const int *keys, long long ts, int log2ts, int key) {
    unsigned long long s = tc_hash(key, log2ts) & (ts - 1);
    for (long long p = 0; p <= ts; ++p) {
        const int k = COHERENT ? __ldcg(keys + s) : keys[s];
        if (k == key) return true;
        if (k == kEmpty) return false;
        s = (s + 1) & (ts - 1);
    }
    return false;
}

struct TcWarpSmem {
    int keys[kWarpSet];
    int rs[kWarpSet / 2];
    int soff[kWarpSet / 2 + 1];
};

// Warp tasks: task t belongs to the row r with task_ptr[r] <= t < task_ptr[r + 1] and
// covers wedges [c * task_work, (c + 1) * task_work) of it, c = t - task_ptr[r]. Each task
// loads its row's mask (<= 256 entries) into its warp's set, so tasks are independent and
// of bounded size, and warps stay balanced however skewed the rows are.
__global__ void __launch_bounds__(kTcBlock) tc_warp(const int *__restrict__ task_ptr, int m, int ntasks,
                                                    int task_work, const int *__restrict__ rp,
                                                    const int *__restrict__ ci, TcInfo *info) {
    __shared__ TcWarpSmem smem[kTcBlock / 32];
    const int lane = threadIdx.x & 31;
    TcWarpSmem &sm = smem[threadIdx.x >> 5];
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    constexpr int LOG = kWarpSet == 512 ? 9 : (kWarpSet == 256 ? 8 : 7);  // log2(kWarpSet)
    static_assert((1 << LOG) == kWarpSet, "warp set size");
    unsigned long long hits = 0;
    for (int t = warp; t < ntasks; t += nwarps) {
        int lo = 0, hi = m;  // last row with task_ptr[row] <= t
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (__ldg(task_ptr + mid) <= t)
                lo = mid;
            else
                hi = mid;
        }
        const int i = lo;
        const int w0 = (t - __ldg(task_ptr + i)) * task_work;
        const int r0 = __ldg(rp + i);
        const int d = __ldg(rp + i + 1) - r0;
        for (int s = lane; s < kWarpSet; s += 32) sm.keys[s] = kEmpty;
        __syncwarp();
        // mask into the set; rows k of the mask with entries are listed (row start, offset)
        int carry = 0, nv = 0;
        for (int base = 0; base < d; base += 32) {
            const int tt = base + lane;
            int len = 0, b0 = 0;
            if (tt < d) {
                const int k = __ldg(ci + r0 + tt);
                set_insert(sm.keys, kWarpSet, LOG, k, info);
                b0 = __ldg(rp + k);
                len = __ldg(rp + k + 1) - b0;
            }
            const unsigned nz = __ballot_sync(0xffffffffu, len > 0);
            int incl = len;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            if (len > 0) {
                const int slot = nv + __popc(nz & ((1u << lane) - 1u));
                sm.rs[slot] = b0;
                sm.soff[slot] = carry + incl - len;
            }
            nv += __popc(nz);
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) sm.soff[nv] = carry;
        __syncwarp();
        const int w1 = min(carry, w0 + task_work);
        // o0: the listed row holding wedge w0 (last with soff <= w0)
        int o0 = 0;
        {
            int a = 0, b = nv;
            while (b - a > 1) {
                const int mid = (a + b) >> 1;
                if (sm.soff[mid] <= w0)
                    a = mid;
                else
                    b = mid;
            }
            o0 = a;
        }
        // wedges in chunks of 32: the next 32 listed rows' starts that fall inside the
        // chunk are marked in a 32-bit word (distinct, since every listed row is
        // non-empty); each lane's row is o0 plus the marks at or before its position
        // kTcChunks chunks per step, so that each lane has that many gathers in flight
        const unsigned upto = lane == 31 ? 0xffffffffu : ((2u << lane) - 1u);
        for (int base = w0; base < w1; base += 32 * kTcChunks) {
            int own[kTcChunks], q[kTcChunks];
#pragma unroll
            for (int h = 0; h < kTcChunks; ++h) {
                const int cb = base + 32 * h;
                const int nb = o0 + 1 + lane;
                const int st = nb <= nv ? sm.soff[nb] - cb : 32;
                const unsigned mark = (st >= 0 && st < 32) ? (1u << st) : 0u;
                const unsigned starts = __reduce_or_sync(0xffffffffu, mark);
                own[h] = o0 + __popc(starts & upto);
                q[h] = cb + lane;
                o0 += __popc(starts);
            }
            int j[kTcChunks];
#pragma unroll
            for (int h = 0; h < kTcChunks; ++h)
                j[h] = q[h] < w1 ? __ldg(ci + sm.rs[own[h]] + (q[h] - sm.soff[own[h]])) : -1;
#pragma unroll
            for (int h = 0; h < kTcChunks; ++h)
                if (q[h] < w1) hits += set_find<false>(sm.keys, kWarpSet, LOG, j[h]) ? 1 : 0;
        }
        __syncwarp();
    }
    for (int o = 16; o; o >>= 1) hits += __shfl_down_sync(0xffffffffu, hits, o);
    if (lane == 0 && hits) atomicAdd(&info->count, hits);
}

struct TcBlockSmem {
    int keys[kBlockSet];
    int rs[kTcBlock];
    int soff[kTcBlock + 1];
    int scan_tmp[33];
    unsigned long long bsum;
};

// One block per row; the mask set is in shared memory, or in scratch for GLOBAL rows.
template <bool GLOBAL>
__global__ void __launch_bounds__(kTcBlock) tc_block(const int *__restrict__ rows, int nrows,
                                                     const int *__restrict__ rp, const int *__restrict__ ci,
                                                     const long long *__restrict__ tbl_off, int *gkeys,
                                                     TcInfo *info) {
    __shared__ TcBlockSmem sm;
    const int tid = threadIdx.x;
    if (tid == 0) sm.bsum = 0;
    unsigned long long hits = 0;
    for (int w = blockIdx.x; w < nrows; w += gridDim.x) {
        const int i = rows[w];
        const int r0 = rp[i];
        const int d = rp[i + 1] - r0;
        long long ts = kBlockSet;
        int *keys = sm.keys;
        if (GLOBAL) {
            ts = 64;
            while (ts < 2LL * d) ts <<= 1;
            keys = gkeys + tbl_off[i];
        }
        int log2ts = 0;
        while ((1LL << log2ts) < ts) ++log2ts;
        if (log2ts > 31) log2ts = 31;
        for (long long s = tid; s < ts; s += kTcBlock) keys[s] = kEmpty;
        __syncthreads();
        for (int t = tid; t < d; t += kTcBlock) set_insert(keys, ts, log2ts, ci[r0 + t], info);
        __syncthreads();
        for (int c0 = 0; c0 < d; c0 += kTcBlock) {
            const int t = c0 + tid;
            int deg = 0;
            if (t < d) {
                const int k = ci[r0 + t];
                const int b0 = rp[k];
                sm.rs[tid] = b0;
                deg = rp[k + 1] - b0;
            }
            int tot;
            sm.soff[tid] = block_exclusive_scan<kTcBlock>(deg, tot, sm.scan_tmp);
            __syncthreads();
            const int nt = d - c0 < kTcBlock ? d - c0 : kTcBlock;
            for (int q = tid; q < tot; q += kTcBlock) {
                int lo = 0, hi = nt;
                while (hi - lo > 1) {
                    const int mid = (lo + hi) >> 1;
                    if (sm.soff[mid] <= q)
                        lo = mid;
                    else
                        hi = mid;
                }
                const int j = ci[sm.rs[lo] + (q - sm.soff[lo])];
                hits += set_find<GLOBAL>(keys, ts, log2ts, j) ? 1 : 0;
            }
            __syncthreads();
        }
    }
    for (int o = 16; o; o >>= 1) hits += __shfl_down_sync(0xffffffffu, hits, o);
    if ((tid & 31) == 0 && hits) atomicAdd(&sm.bsum, hits);
    __syncthreads();
    if (tid == 0 && sm.bsum) atomicAdd(&info->count, sm.bsum);
}

// ---------------------------------------------------------------- bitmap path
// count = sum over the edges (a, b) of D of |D(a) ^ D(b)|, and an intersection may be taken
// from either side: each edge goes to its endpoint with the longer list (its owner), whose
// list is held as a bitmap over all vertices in shared memory, and the other endpoint's (the
// partner's) list is read and tested against it. That reads the shorter list of every edge:
// R-MAT scale 18, 321M tests instead of the 660M wedges of sum((D*D) .* D), and a test is one
// shared-memory word instead of a probe chain in a hash set.
//
// Measured at scale 18: counting 2.74 ms with hash sets; 0.51 ms with bitmaps and tc_small (and
// 0.13 ms for the partner lists), tc_bits at 71 % of the issue slots and 83 % of the L1/shared-memory
// pipe.
//
// Needs: L strict lower triangular with strictly ascending rows (both found out on the way: a
// row's list then is a set, so that either side may be the bitmap; in rows out of order an entry
// may be repeated anywhere), and the bitmap to fit an SM's shared memory. Everything else is
// counted by the hash path above.
constexpr int kTcBitmapVertices = 1600 * 1024;  // 200 KB of bits
constexpr int kTcManyPartners = 256;            // owners with at least this many start first
__global__ void tc_partner_lists(int m, unsigned nnz, const unsigned *__restrict__ row, const int *__restrict__ ci,
                                 const int *__restrict__ deg, const int *__restrict__ drp,
                                 const int *__restrict__ place, const int *__restrict__ prp, int *plist,
                                 const TcInfo *info) {
    if (info->not_lower || info->unsorted || __ldg(prp + m) == 0) return;
    for (unsigned e = blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += gridDim.x * blockDim.x) {
        const int at = place[e];
        if (at < 0) continue;
        int a, b;
        tc_edge(deg, static_cast<int>(__ldg(row + e)), __ldg(ci + e), a, b);
        const int la = __ldg(drp + a + 1) - __ldg(drp + a), lb = __ldg(drp + b + 1) - __ldg(drp + b);
        const bool tail = la >= lb;
        plist[__ldg(prp + (tail ? a : b)) + at] = tail ? b : a;
    }
}

// Owners with many partners from the front of `list`, the others from its back; in `small` the
// vertices whose lists are short (and long enough for a triangle).
__global__ void tc_owners(int m, unsigned nnz, const int *__restrict__ drp, const int *__restrict__ prp, int *list,
                          int *small, TcInfo *info) {
    if (info->not_lower || info->unsorted) return;
    const int small_list = tc_small_list(m, nnz, info);
    const int lane = threadIdx.x & 31;
    for (int v0 = blockIdx.x * blockDim.x; v0 < m; v0 += gridDim.x * blockDim.x) {
        const int v = v0 + threadIdx.x;
        const int n = v < m ? __ldg(prp + v + 1) - __ldg(prp + v) : 0;
        const int len = v < m && small_list > 0 ? __ldg(drp + v + 1) - __ldg(drp + v) : 0;
        const int kind = n >= kTcManyPartners ? 0 : n > 0 ? 1 : len >= 2 && len <= small_list ? 2 : -1;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const bool in = k == kind;
            const unsigned mask = __ballot_sync(0xffffffffu, in);
            int base = 0;
            if (lane == 0 && mask) base = atomicAdd(&info->owners[k], __popc(mask));
            base = __shfl_sync(0xffffffffu, base, 0) + __popc(mask & ((1u << lane) - 1u));
            if (in) (k == 2 ? small : list)[k == 1 ? m - 1 - base : base] = v;
        }
    }
}

// One block per owner, taken from a counter: its list's bits are set, its warps read the
// partners' lists (an entry per lane, ranges fetched 32 partners at a time) and test them, the
// bits are cleared again.
__global__ void __launch_bounds__(1024) tc_bits(int m, const int *__restrict__ list, const int *__restrict__ drp,
                                                const int *__restrict__ dci, const int *__restrict__ prp,
                                                const int *__restrict__ plist, TcInfo *info) {
    extern __shared__ unsigned bits[];
    __shared__ int s_next;
    if (info->not_lower || info->unsorted) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nthreads = blockDim.x, nwarps = nthreads >> 5;
    const int nmany = info->owners[0], nall = nmany + info->owners[1];
    if (nall == 0) return;
    for (int w = tid; w < (m + 31) >> 5; w += nthreads) bits[w] = 0u;
    unsigned long long hits = 0;
    for (;;) {
        if (tid == 0) s_next = atomicAdd(&info->ticket, 1);
        __syncthreads();
        const int at = s_next;
        if (at >= nall) break;
        const int v = __ldg(list + (at < nmany ? at : m - 1 - (at - nmany)));
        const int r0 = __ldg(drp + v), r1 = __ldg(drp + v + 1);
        const int p0 = __ldg(prp + v), p1 = __ldg(prp + v + 1);
        for (int e = r0 + tid; e < r1; e += nthreads) {
            const int j = __ldg(dci + e);
            atomicOr(bits + (j >> 5), 1u << (j & 31));
        }
        __syncthreads();
        for (int t0 = p0 + warp; t0 < p1; t0 += 32 * nwarps) {
            const int t = t0 + nwarps * lane;
            int b0 = 0, b1 = 0;
            if (t < p1) {
                const int p = __ldg(plist + t);
                b0 = __ldg(drp + p);
                b1 = __ldg(drp + p + 1);
            }
            const int n = min(32, (p1 - t0 + nwarps - 1) / nwarps);
            unsigned found = 0u;
            for (int k = 0; k < n; ++k) {
                const int e0 = __shfl_sync(0xffffffffu, b0, k), e1 = __shfl_sync(0xffffffffu, b1, k);
                for (int e = e0 + lane; e < e1; e += 128) {
                    int j[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) j[u] = e + 32 * u < e1 ? __ldg(dci + e + 32 * u) : -1;
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (j[u] >= 0) found += (bits[j[u] >> 5] >> (j[u] & 31)) & 1u;
                }
            }
            hits += found;
        }
        __syncthreads();
        for (int e = r0 + tid; e < r1; e += nthreads) bits[__ldg(dci + e) >> 5] = 0u;
    }
    for (int o = 16; o; o >>= 1) hits += __shfl_down_sync(0xffffffffu, hits, o);
    if (lane == 0 && hits) atomicAdd(&info->count, hits);
}

// Vertices with short lists, a warp each: the list goes into a hash set in shared memory, and the
// short ones among the lists of its entries, one after the other, are looked up in it, 128
// entries at a time. What bounds it: the chain of reads (vertex, its list, an entry's list)
// with 64 warps on an SM.
struct TcSmallSmem {
    int keys[4 * kTcSmallList];
    int rs[kTcSmallList];        // of each list looked up: where it begins, minus
    int soff[kTcSmallList + 1];  // the entries before it
};
__global__ void __launch_bounds__(kTcBlock) tc_small(int m, unsigned nnz, const int *__restrict__ small,
                                                     const int *__restrict__ drp, const int *__restrict__ dci,
                                                     TcInfo *info) {
    __shared__ TcSmallSmem smem[kTcBlock / 32];
    const int small_list = tc_small_list(m, nnz, info);
    if (small_list == 0 || info->not_lower || info->unsorted) return;
    TcSmallSmem &sm = smem[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const unsigned upto = lane == 31 ? 0xffffffffu : (2u << lane) - 1u;
    const int n = info->owners[2];
    const int nwarps = (gridDim.x * kTcBlock) >> 5;
    unsigned long long hits = 0;
    for (long long w = (blockIdx.x * kTcBlock + threadIdx.x) >> 5; w < n; w += nwarps) {
        const int v = __ldg(small + w);
        const int r0 = __ldg(drp + v), d = __ldg(drp + v + 1) - r0;
        // a power of two of slots, at least four times the list's
        const int log2ts = max(5, 32 - __clz(4 * d - 1)), ts = 1 << log2ts;
        for (int s = lane; s < ts; s += 32) sm.keys[s] = kEmpty;
        __syncwarp();
        int nv = 0, all = 0;
        for (int t0 = 0; t0 < d; t0 += 32) {
            int b0 = 0, len = 0;
            if (t0 + lane < d) {
                const int k = __ldg(dci + r0 + t0 + lane);
                b0 = __ldg(drp + k);
                len = __ldg(drp + k + 1) - b0;
                set_insert(sm.keys, ts, log2ts, k, info);
                if (len > small_list) len = 0;  // the blocks count it
            }
            const unsigned some = __ballot_sync(0xffffffffu, len > 0);
            int incl = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            if (len > 0) {
                const int at = nv + __popc(some & ((1u << lane) - 1u));
                sm.soff[at] = all + incl - len;
                sm.rs[at] = b0 - (all + incl - len);
            }
            nv += __popc(some);
            all += __shfl_sync(0xffffffffu, incl, 31);
        }
        __syncwarp();
        int o0 = 0;  // the list of the chunk's first entry
        unsigned found = 0u;
        for (int base = 0; base < all; base += 128) {
            int j[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                const int cb = base + 32 * h;
                const int nb = o0 + 1 + lane;
                const int st = nb < nv ? sm.soff[nb] - cb : 32;
                const unsigned starts = __reduce_or_sync(0xffffffffu, st >= 0 && st < 32 ? 1u << st : 0u);
                const int q = cb + lane;
                j[h] = q < all ? __ldg(dci + sm.rs[o0 + __popc(starts & upto)] + q) : -1;
                o0 += __popc(starts);
            }
#pragma unroll
            for (int h = 0; h < 4; ++h)
                if (j[h] >= 0) found += set_find<false>(sm.keys, ts, log2ts, j[h]) ? 1u : 0u;
        }
        hits += found;
        __syncwarp();
    }
    for (int o = 16; o; o >>= 1) hits += __shfl_down_sync(0xffffffffu, hits, o);
    if (lane == 0 && hits) atomicAdd(&info->count, hits);
}

// strict lower triangle extraction: counts, then copy
__global__ void lower_count(int m, const int *__restrict__ rp, const int *__restrict__ ci, int *cnt) {
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int i = warp; i < m; i += nwarps) {
        int c = 0;
        for (int e = rp[i] + lane; e < rp[i + 1]; e += 32) c += ci[e] < i;
        for (int o = 16; o; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
        if (lane == 0) cnt[i] = c;
    }
}

__global__ void lower_copy(int m, const int *__restrict__ rp, const int *__restrict__ ci,
                           const int *__restrict__ lrp, int *lci) {
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int i = warp; i < m; i += nwarps) {
        int out = lrp[i];
        for (int e0 = rp[i]; e0 < rp[i + 1]; e0 += 32) {
            const int e = e0 + lane;
            const bool keep = e < rp[i + 1] && ci[e] < i;
            const unsigned mask = __ballot_sync(0xffffffffu, keep);
            if (keep) lci[out + __popc(mask & ((1u << lane) - 1u))] = ci[e];
            out += __popc(mask);
        }
    }
}

int entry_blocks(const apspie_ctx *ctx, unsigned nnz) {
    return static_cast<int>(std::min<long long>((static_cast<long long>(nnz) + 255) / 256, ctx->num_sms * 16LL));
}

// *info by way of pinned memory (a copy to pageable memory is waited for by itself).
cudaError_t read_info(apspie_ctx *ctx, const TcInfo *info, TcInfo &h) {
    static_assert(sizeof(TcInfo) <= kPinnedBytes, "room");
    cudaError_t e = cudaMemcpyAsync(ctx->h_word, info, sizeof(TcInfo), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e == cudaSuccess) std::memcpy(&h, ctx->h_word, sizeof(TcInfo));
    return e;
}

// What counting by hash sets takes beside D, and a scan's scratch.
struct TcHashBufs {
    int *bin_rows;
    long long *tbl_off;
    unsigned char *row_bin;
    int *ntask, *task_ptr;
    static size_t need(int m) {
        const size_t mi = static_cast<size_t>(m) + 1;
        return Carver::need({kTcBins * mi * 4, mi * 8, mi, mi * 4, mi * 4});
    }
    static TcHashBufs carve(Carver &c, int m) {
        const size_t mi = static_cast<size_t>(m) + 1;
        TcHashBufs b;
        b.bin_rows = c.take<int>(kTcBins * mi);
        b.tbl_off = c.take<long long>(mi);
        b.row_bin = c.take<unsigned char>(mi);
        b.ntask = c.take<int>(mi);
        b.task_ptr = c.take<int>(mi);
        return b;
    }
};

// sum((D*D) .* D) of D = (rp, ci) by hash sets; *info is cleared. With `check`, an L that is not
// strictly lower (info->not_lower, set when D was made from it) is counted as given instead.
apspie_status tc_count_by_hash(apspie_ctx *ctx, const apspie_csr *L, const int *rp, const int *ci, bool check,
                               const TcHashBufs &b, void *stmp, TcInfo *info, int64_t *count) {
    apspie_status st;
    cudaError_t e = cudaSuccess;
    const int m = L->m;
    const int task_work = effective_params(ctx, APSPIE_TUNE_TC, L).tc_task_work;
    const int rblocks = std::max(1, std::min<int>((m * 8LL + 255) / 256, ctx->num_sms * 16));
    const int lblocks = std::max(1, std::min<int>((m + 255LL) / 256, ctx->num_sms * 8));
    TcInfo h;
    int ntasks = 0;
    for (int attempt = 0; attempt < 2; ++attempt) {
        if (m > 0) {
            tc_rowinfo<<<rblocks, 256, 0, ctx->stream>>>(m, rp, ci, task_work, b.row_bin, b.ntask, b.tbl_off, info);
            tc_binlists<<<lblocks, 256, 0, ctx->stream>>>(m, b.row_bin, b.bin_rows, info);
            if ((st = device_exclusive_scan(ctx, b.ntask, m, b.task_ptr, stmp, &info->overflow)) != APSPIE_OK) return st;
            if ((e = cudaMemcpyAsync(&ntasks, b.task_ptr + m, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream)) !=
                cudaSuccess)
                return cuda_error(ctx, e, "tc plan");
        }
        if ((e = read_info(ctx, info, h)) != cudaSuccess)
            return cuda_error(ctx, e, "tc plan");
        if (!h.not_lower || attempt == 1 || !check) break;
        // not a strict lower triangle: count sum((L*L) .* L) on L as given
        rp = L->row_ptr;
        ci = L->col_ind;
        if ((e = cudaMemsetAsync(info, 0, sizeof(TcInfo), ctx->stream)) != cudaSuccess)
            return cuda_error(ctx, e, "tc reset");
    }
    int *gkeys = nullptr;
    if (h.global_slots > 0) {
        void *tb;
        if ((st = scratch2_reserve(ctx, static_cast<size_t>(h.global_slots) * 4 + 256, &tb)) != APSPIE_OK)
            return st;
        gkeys = static_cast<int *>(tb);
    }
    const int cap = ctx->num_sms * 8;
    if (ntasks > 0)
        tc_warp<<<std::min((ntasks + 7) / 8, cap), kTcBlock, 0, ctx->stream>>>(b.task_ptr, m, ntasks, task_work, rp, ci,
                                                                                 info);
    if (h.bin_count[2] > 0)
        tc_block<false><<<std::min(h.bin_count[2], cap), kTcBlock, 0, ctx->stream>>>(
            b.bin_rows + 2 * static_cast<size_t>(m), h.bin_count[2], rp, ci, b.tbl_off, gkeys, info);
    if (h.bin_count[3] > 0)
        tc_block<true><<<std::min(h.bin_count[3], cap), kTcBlock, 0, ctx->stream>>>(
            b.bin_rows + 3 * static_cast<size_t>(m), h.bin_count[3], rp, ci, b.tbl_off, gkeys, info);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_error(ctx, e, "tc launch");
    if ((e = read_info(ctx, info, h)) != cudaSuccess)
        return cuda_error(ctx, e, "tc result");
    if (h.overflow) return set_error(ctx, APSPIE_ERR_HASH_OVERFLOW, "apspie_tc: mask set overflow");
    *count = static_cast<int64_t>(h.count);
    return APSPIE_OK;
}

// By hash sets: any L, any size. Beside D it keeps nothing per entry but the rows of a part of
// them at a time.
constexpr long long kTcPart = 1 << 24;
apspie_status tc_by_hash_sets(apspie_ctx *ctx, const apspie_csr *L, int64_t *count) {
    apspie_status st;
    const int m = L->m;
    const size_t mi = static_cast<size_t>(m) + 1;
    const size_t nz = static_cast<size_t>(L->nnz > 0 ? L->nnz : 1);
    const size_t part = std::min(nz, static_cast<size_t>(kTcPart));
    void *base;
    st = scratch_reserve(ctx,
                         Carver::need({TcHashBufs::need(m), sizeof(TcInfo), mi * 4, mi * 4, mi * 4, nz * 4,
                                       scan_scratch_bytes(m) + 64, part * 4}),
                         &base);
    if (st != APSPIE_OK) return st;
    Carver c(base);
    const TcHashBufs hash = TcHashBufs::carve(c, m);
    TcInfo *info = c.take<TcInfo>(1);
    int *deg = c.take<int>(mi);
    int *len = c.take<int>(mi);
    int *drp = c.take<int>(mi);
    int *dci = c.take<int>(nz);
    void *stmp = c.take<char>(scan_scratch_bytes(m) + 64);
    unsigned *row = c.take<unsigned>(part);
    cudaError_t e = cudaMemsetAsync(info, 0, sizeof(TcInfo), ctx->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(len, 0, mi * 4, ctx->stream);
    if (e != cudaSuccess) return cuda_error(ctx, e, "tc reset");
    const int *rp = L->row_ptr, *ci = L->col_ind;
    const bool orient = effective_params(ctx, APSPIE_TUNE_TC, L).tc_orient != 0;
    if (m > 0 && L->nnz > 0 && orient) {
        // D: L's edges oriented from lower to higher (degree, id) rank
        tc_row_lengths<<<std::min((m + 255) / 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(m, rp, deg);
        for (int pass = 0; pass < 3; ++pass) {
            for (long long first = 0; first < L->nnz; first += kTcPart) {
                const unsigned n = static_cast<unsigned>(std::min<long long>(kTcPart, L->nnz - first));
                const int eb = entry_blocks(ctx, n);
                if ((pass == 0 || L->nnz > kTcPart) && (st = expand_entry_rows(ctx, L, first, n, row)) != APSPIE_OK)
                    return st;
                if (pass == 0)
                    tc_columns<<<std::min(eb, ctx->num_sms * 4), kTcColumnsBlock, 0, ctx->stream>>>(n, m, row, ci + first,
                                                                                                   deg, info);
                else if (pass == 1)
                    tc_out_lengths<<<eb, 256, 0, ctx->stream>>>(n, row, ci + first, deg, len, info);
                else
                    tc_out_lists<<<eb, 256, 0, ctx->stream>>>(n, row, ci + first, deg, drp, len, dci, info);
            }
            if (pass != 1) continue;
            if ((st = device_exclusive_scan(ctx, len, m, drp, stmp, &info->overflow)) != APSPIE_OK) return st;
            if ((e = cudaMemsetAsync(len, 0, mi * 4, ctx->stream)) != cudaSuccess) return cuda_error(ctx, e, "tc reset");
        }
        rp = drp;
        ci = dci;
    }
    return tc_count_by_hash(ctx, L, rp, ci, orient, hash, stmp, info, count);
}

// By bitmaps; an L that turns out not to fit them is counted by hash sets, on the D that was made.
apspie_status tc_by_bitmaps(apspie_ctx *ctx, const apspie_csr *L, int64_t *count) {
    const int m = L->m;
    const unsigned nnz = static_cast<unsigned>(L->nnz);
    const size_t mi = static_cast<size_t>(m) + 1, nz = static_cast<size_t>(nnz);
    void *base;
    apspie_status st = scratch_reserve(ctx,
                                       Carver::need({sizeof(TcInfo), mi * 4, mi * 4, mi * 4, mi * 4, mi * 4, mi * 4,
                                                     nz * 4, nz * 4, nz * 4, nz * 4, scan_scratch_bytes(m) + 64,
                                                     TcHashBufs::need(m)}),
                                       &base);
    if (st == APSPIE_ERR_OOM) return tc_by_hash_sets(ctx, L, count);  // a quarter of that an entry
    if (st != APSPIE_OK) return st;
    Carver c(base);
    TcInfo *info = c.take<TcInfo>(1);
    int *len = c.take<int>(mi);
    int *partners = c.take<int>(mi);
    int *deg = c.take<int>(mi);
    int *drp = c.take<int>(mi);
    int *prp = c.take<int>(mi);
    int *list = c.take<int>(mi);
    unsigned *row = c.take<unsigned>(nz);
    int *place = c.take<int>(nz);
    int *dci = c.take<int>(nz);
    int *plist = c.take<int>(nz);
    void *stmp = c.take<char>(scan_scratch_bytes(m) + 64);
    const TcHashBufs hash = TcHashBufs::carve(c, m);
    const size_t zeroed = static_cast<size_t>(reinterpret_cast<char *>(partners + mi) - reinterpret_cast<char *>(info));
    cudaError_t e = cudaMemsetAsync(info, 0, zeroed, ctx->stream);  // info, len, partners
    if (e != cudaSuccess) return cuda_error(ctx, e, "tc reset");
    const bool orient = effective_params(ctx, APSPIE_TUNE_TC, L).tc_orient != 0;
    const int eb = entry_blocks(ctx, nnz), vb = std::min((m + 255) / 256, ctx->num_sms * 8);
    if ((st = expand_entry_rows(ctx, L, 0, nnz, row)) != APSPIE_OK) return st;
    tc_row_lengths<<<vb, 256, 0, ctx->stream>>>(m, L->row_ptr, deg);
    tc_columns<<<std::min(eb, ctx->num_sms * 4), kTcColumnsBlock, 0, ctx->stream>>>(nnz, m, row, L->col_ind, deg, info);
    const int *rp = L->row_ptr, *ci = L->col_ind, *degree = nullptr;
    if (orient) {
        degree = deg;
        tc_out_places<<<eb, 256, 0, ctx->stream>>>(nnz, row, L->col_ind, degree, len, place, tc_even_limit(m, nnz), info);
        if ((st = device_exclusive_scan(ctx, len, m, drp, stmp, &info->overflow)) != APSPIE_OK) return st;
        rp = drp;
        ci = dci;
    }
    tc_owner_places<<<eb, 256, 0, ctx->stream>>>(nnz, row, L->col_ind, degree, rp, orient ? dci : nullptr, place,
                                                 partners, m, info);
    if ((st = device_exclusive_scan(ctx, partners, m, prp, stmp, &info->overflow)) != APSPIE_OK) return st;
    tc_partner_lists<<<eb, 256, 0, ctx->stream>>>(m, nnz, row, L->col_ind, degree, rp, place, prp, plist, info);
    int *small = partners;  // prp has taken its place
    tc_owners<<<vb, 256, 0, ctx->stream>>>(m, nnz, rp, prp, list, small, info);
    if (m > kTcNoSmall)
        tc_small<<<ctx->num_sms * 8, kTcBlock, 0, ctx->stream>>>(m, nnz, small, rp, ci, info);
    // threads enough to fill an SM beside the bitmaps that fit on it
    const size_t smem = (static_cast<size_t>(m) + 31) / 32 * 4;
    const int threads = smem <= 36 * 1024 ? 256 : smem <= 72 * 1024 ? 512 : 1024;
    int per_sm = 0;
    // the limit belongs to the kernel on the device: the same from every thread's calls
    e = cudaFuncSetAttribute(tc_bits, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcBitmapVertices / 8);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, tc_bits, threads, smem);
    if (e != cudaSuccess) return cuda_error(ctx, e, "tc launch");
    tc_bits<<<std::max(per_sm, 1) * ctx->num_sms, threads, smem, ctx->stream>>>(m, list, rp, ci, prp, plist, info);
    TcInfo h;
    if ((e = cudaGetLastError()) != cudaSuccess ||
        (e = read_info(ctx, info, h)) != cudaSuccess)
        return cuda_error(ctx, e, "tc result");
    if (h.overflow) return set_error(ctx, APSPIE_ERR_HASH_OVERFLOW, "apspie_tc: mask set overflow");
    if (!h.not_lower && !h.unsorted) {
        ctx->tc_by_bitmaps = true;
        *count = static_cast<int64_t>(h.count);
        return APSPIE_OK;
    }
    if (h.not_lower) {
        rp = L->row_ptr;
        ci = L->col_ind;
    }
    if ((e = cudaMemsetAsync(info, 0, sizeof(TcInfo), ctx->stream)) != cudaSuccess) return cuda_error(ctx, e, "tc reset");
    return tc_count_by_hash(ctx, L, rp, ci, false, hash, stmp, info, count);
}

}  // namespace
}  // namespace apspie

using namespace apspie;

extern "C" {

apspie_status apspie_tc(apspie_ctx *ctx, const apspie_csr *L, int64_t *count) {
    if (!ctx || !count) return APSPIE_ERR_INVALID_ARG;
    cudaSetDevice(ctx->device);
    apspie_status st = check_csr_view(ctx, L, "apspie_tc");
    if (st != APSPIE_OK) return st;
    if (L->m != L->n) return set_error(ctx, APSPIE_ERR_INVALID_ARG, "apspie_tc: L must be square");
    if (ctx->validate && (st = validate_csr(ctx, L, true)) != APSPIE_OK) return st;
    ctx->tc_by_bitmaps = false;
    if (L->m > 0 && L->nnz > 0 && L->m <= kTcBitmapVertices && L->nnz <= kMaxStepped)
        return tc_by_bitmaps(ctx, L, count);
    return tc_by_hash_sets(ctx, L, count);
}

apspie_status apspie_csr_strict_lower_device(apspie_ctx *ctx, const apspie_csr *A, apspie_csr_owned *L) {
    if (!ctx || !L) return APSPIE_ERR_INVALID_ARG;
    cudaSetDevice(ctx->device);
    std::memset(L, 0, sizeof(*L));
    apspie_status st = check_csr_view(ctx, A, "apspie_csr_strict_lower_device");
    if (st != APSPIE_OK) return st;
    if (A->m != A->n) return set_error(ctx, APSPIE_ERR_INVALID_ARG, "strict lower: A must be square");
    if (ctx->validate && (st = validate_csr(ctx, A, true)) != APSPIE_OK) return st;
    const int m = A->m;
    const size_t mi = static_cast<size_t>(m) + 1;
    void *base;
    st = scratch_reserve(ctx, Carver::need({mi * 4, scan_scratch_bytes(m) + 64, 64}), &base);
    if (st != APSPIE_OK) return st;
    Carver c(base);
    int *cnt = c.take<int>(mi);
    void *stmp = c.take<char>(scan_scratch_bytes(m) + 64);
    int *ovf = c.take<int>(16);
    cudaError_t e = cudaMemsetAsync(ovf, 0, sizeof(int), ctx->stream);
    int32_t *lrp = nullptr;
    if (e == cudaSuccess) e = owned_alloc(reinterpret_cast<void **>(&lrp), mi * sizeof(int32_t));
    if (e != cudaSuccess) return cuda_error(ctx, e, "strict lower alloc");
    const int blocks = std::max(1, std::min<int>((m * 32LL + 255) / 256, ctx->num_sms * 16));
    lower_count<<<blocks, 256, 0, ctx->stream>>>(m, A->row_ptr, A->col_ind, cnt);
    if ((st = device_exclusive_scan(ctx, cnt, m, lrp, stmp, ovf)) != APSPIE_OK) {
        owned_free(lrp);
        return st;
    }
    int nnz = 0;
    if ((e = cudaMemcpyAsync(&nnz, lrp + m, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream)) != cudaSuccess ||
        (e = cudaStreamSynchronize(ctx->stream)) != cudaSuccess) {
        owned_free(lrp);
        return cuda_error(ctx, e, "strict lower sync");
    }
    int32_t *lci = nullptr;
    if ((e = owned_alloc(reinterpret_cast<void **>(&lci), std::max(nnz, 1) * sizeof(int32_t))) != cudaSuccess) {
        owned_free(lrp);
        return cuda_error(ctx, e, "strict lower alloc");
    }
    lower_copy<<<blocks, 256, 0, ctx->stream>>>(m, A->row_ptr, A->col_ind, lrp, lci);
    if ((e = cudaGetLastError()) != cudaSuccess) {
        owned_free(lrp);
        owned_free(lci);
        return cuda_error(ctx, e, "strict lower launch");
    }
    L->m = L->n = m;
    L->nnz = nnz;
    L->val_type = APSPIE_VAL_NONE;
    L->row_ptr = lrp;
    L->col_ind = lci;
    L->val = nullptr;
    return APSPIE_OK;
}

}  // extern "C"
