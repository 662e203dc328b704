// Device-side graph construction: COO -> CSR (optionally symmetrised and deduplicated with
// the generator's rules) and CSR transpose, on a stable LSD radix sort of this file's own.
//
// The reference builds graphs on the host: readMtx + makeSymmetric (src/util.cuh:371-643,
// a qsort of every edge and its mirror, then a compaction) and buildMatrix
// (src/matrix.cpp:55-111, a COO -> CSR conversion through cuSPARSE), and transposes with
// csr2csc (src/util.cuh:474). Here the same results come from device kernels:
//   * keys (a << B) | b of B = bit length of m bits each; symmetrising canonicalises
//     {u, v} to a = min, b = max; dropped self-loops get a sentinel key that sorts last;
//   * a stable radix sort (sort.cuh), so equal keys keep their input order and deduplication
//     keeps the first occurrence;
//   * symmetric CSR rows: lower neighbours (pairs (lo, r)) then upper ones ((r, hi)), each
//     ascending, so rows come out sorted without a per-row sort: row_ptr[r] is the number
//     of pairs with lo < r plus the number with hi < r, read off the two sorted orders.
#include <algorithm>
#include <climits>
#include <cstring>

#include "sort.cuh"

namespace apspie {
namespace {

// Keys of the edge list (see the head of this file) and the digit counts of their sort.
__global__ void __launch_bounds__(256) coo_keys(long long ne, int m, const int *__restrict__ src,
                                                const int *__restrict__ dst, const unsigned *__restrict__ w, int B,
                                                int symmetrize, int drop_loops, RsPlan pl, unsigned long long *keys,
                                                unsigned *vals, int *ghist, int *bad) {
    __shared__ int h[kRsMaxPasses * kRsDigits];
    rs_count_begin(h, pl);
    const unsigned long long sentinel = (1ull << (2 * B)) - 1ull;
    for (long long k = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; k < ne;
         k += static_cast<long long>(gridDim.x) * blockDim.x) {
        int u = __ldg(src + k), v = __ldg(dst + k);
        if (u < 0 || u >= m || v < 0 || v >= m) {
            atomicOr(bad, 1);
            u = v = 0;
        }
        if (symmetrize && u > v) {
            const int t = u;
            u = v;
            v = t;
        }
        const unsigned long long key = (drop_loops && u == v)
                                           ? sentinel
                                           : ((static_cast<unsigned long long>(u) << B) | static_cast<unsigned>(v));
        keys[k] = key;
        vals[k] = w ? __ldg(w + k) : 0u;
        rs_count(h, key, pl);
    }
    rs_count_end(h, pl, ghist);
}

// Drops sentinels (keys >= `sentinel`, which sort last) and, with dedup, all but the first of
// equal keys, in one pass: tiles are taken in order, a look-back gives each tile's place.
// start[r] becomes the first kept pair whose upper field is >= r, for r up to the last kept
// pair's field (start null: not), and the kept keys' digits are counted for the sort by the lower field
// (pl2.passes = 0: not). One read and one write of the pairs where flags, scan and compaction
// took three.
//
// A tile is 8,192 pairs, counted first (the keep bits stay in a register per lane) and read
// again from L2 when its place is known: with 2,048-pair tiles held in registers the
// look-back, which walks past every tile in flight, took most of 260 us for 16.8M pairs.
constexpr int kCompactTile = 8192;
__global__ void __launch_bounds__(256) compact_pairs(long long n, const unsigned long long *__restrict__ kin,
                                                     const unsigned *__restrict__ vin, unsigned long long sentinel,
                                                     int dedup, int B, RsPlan pl2, int *ghist2,
                                                     unsigned long long *kout, unsigned *vout, int *start,
                                                     unsigned long long *status, int *ticket, int *kept, int *err) {
    __shared__ int h[kRsMaxPasses * kRsDigits];
    __shared__ int s_warp[8];
    __shared__ int s_tile;
    __shared__ long long s_base;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    rs_count_begin(h, pl2);
    const long long ntiles = (n + kCompactTile - 1) / kCompactTile;
    for (;;) {
        if (tid == 0) s_tile = ld_volatile_i32(err) == 0 ? atomicAdd(ticket, 1) : INT_MAX;
        __syncthreads();
        const int tile = s_tile;
        if (tile >= ntiles) break;
        // a warp's 1,024 pairs are consecutive, 32 a step; lane i keeps step i's keep bits
        const long long w0 = static_cast<long long>(tile) * kCompactTile + warp * 1024 + lane;
        unsigned bits = 0u;
        // the key before the step's first one (lane 0's neighbour)
        unsigned long long last = (w0 - lane > 0 && w0 - lane <= n) ? __ldg(kin + w0 - lane - 1) : 0ull;
#pragma unroll
        for (int i0 = 0; i0 < 32; i0 += 8) {
            unsigned long long key[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) key[i] = w0 + 32 * (i0 + i) < n ? __ldg(kin + w0 + 32 * (i0 + i)) : ~0ull;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const long long at = w0 + 32 * (i0 + i);
                unsigned long long prev = __shfl_up_sync(0xffffffffu, key[i], 1);
                if (lane == 0) prev = last;
                last = __shfl_sync(0xffffffffu, key[i], 31);
                const bool keep = at < n && key[i] < sentinel && !(dedup && at > 0 && prev == key[i]);
                const unsigned b = __ballot_sync(0xffffffffu, keep);
                if (lane == i0 + i) bits = b;
            }
        }
        const int mine = __reduce_add_sync(0xffffffffu, __popc(bits));
        if (lane == 0) s_warp[warp] = mine;
        __syncthreads();
        if (warp == 0) {
            const int c = lane < 8 ? s_warp[lane] : 0;
            int incl = c;
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const int tot = __shfl_sync(0xffffffffu, incl, 7);
            if (lane < 8) s_warp[lane] = incl - c;
            if (lane == 0) st_relaxed_u64(status + tile, look_word(kRsOwn, tile == 0, tot));
            long long base = 0;
            if (tile > 0) {
                base = look_back_warp(status, tile, kRsOwn, err);
                if (lane == 0 && base >= 0) st_relaxed_u64(status + tile, look_word(kRsOwn, true, base + tot));
            }
            if (lane == 0) {
                s_base = base;
                if (base >= 0 && tile == ntiles - 1) *kept = static_cast<int>(base) + tot;
            }
        }
        __syncthreads();
        if (s_base < 0) break;
        int p = static_cast<int>(s_base) + s_warp[warp];
        for (int i0 = 0; i0 < 32; i0 += 4) {
            unsigned long long key[4], prev[4];
            unsigned val[4];
            bool keep[4];
            int at[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const unsigned m = __shfl_sync(0xffffffffu, bits, i0 + i);
                keep[i] = (m >> lane) & 1u;
                at[i] = p + __popc(m & ((1u << lane) - 1u));
                p += __popc(m);
                const long long e = w0 + 32 * (i0 + i);
                key[i] = keep[i] ? __ldg(kin + e) : 0ull;
                val[i] = keep[i] ? __ldcs(vin + e) : 0u;
                // the pair before, kept or an equal of a kept one, has the field of the one kept before
                prev[i] = keep[i] && e > 0 ? __ldg(kin + e - 1) : 0ull;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (!keep[i]) continue;
                kout[at[i]] = key[i];
                vout[at[i]] = val[i];
                const int r = static_cast<int>(key[i] >> B);
                const int rp = w0 + 32 * (i0 + i) > 0 ? static_cast<int>(prev[i] >> B) : -1;
                if (start)
                    for (int x = rp + 1; x <= r; ++x) start[x] = at[i];
                rs_count(h, key[i], pl2);
            }
        }
    }
    rs_count_end(h, pl2, ghist2);
}

// start[r] = first index i with field(key[i]) >= r, for r up to the last key's field; keys
// ascending in the field ((key >> shift) & fmask). fill_tail completes it.
template <class K>
__global__ void run_starts(long long n, const K *__restrict__ keys, int shift, K fmask, int *start, const int *err) {
    if (ld_volatile_i32(err) != 0) return;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int r = static_cast<int>((keys[i] >> shift) & fmask);
        const int rp = i > 0 ? static_cast<int>((keys[i - 1] >> shift) & fmask) : -1;
        for (int x = rp + 1; x <= r; ++x) start[x] = static_cast<int>(i);
    }
}

// start[r] = n for every r past the last key's field, up to m (all of them for n = 0): by all
// threads, where one thread used to walk the empty rows at the end.
template <class K>
__global__ void fill_tail(long long n, const K *__restrict__ keys, int shift, K fmask, int m, int *start,
                          const int *err) {
    if (ld_volatile_i32(err) != 0) return;
    const int last = n > 0 ? static_cast<int>((keys[n - 1] >> shift) & fmask) : -1;
    for (int x = last + 1 + blockIdx.x * blockDim.x + threadIdx.x; x <= m; x += gridDim.x * blockDim.x)
        start[x] = static_cast<int>(n);
}

// The same for every r up to m when there are fewer keys than rows, and most rows are gaps that
// one thread would fill: a block takes 1,024 rows, finds the keys that lie in them and looks each
// row up among those. (64 entries in 2^25 rows: the transpose took 91 ms by the two above and a
// scan of all rows for the entries', 21 ms before that; now 0.27 ms.)
template <class K>
__global__ void __launch_bounds__(256) search_starts(long long n, const K *__restrict__ keys, int shift, K fmask, int m,
                                                     int *start, const int *err) {
    if (ld_volatile_i32(err) != 0) return;
    auto bound = [&](long long lo, long long hi, long long r) {  // first of [lo, hi) with a field >= r
        while (lo < hi) {
            const long long mid = (lo + hi) >> 1;
            if (static_cast<long long>((__ldg(keys + mid) >> shift) & fmask) < r)
                lo = mid + 1;
            else
                hi = mid;
        }
        return lo;
    };
    for (long long r0 = blockIdx.x * 1024ll; r0 <= m; r0 += gridDim.x * 1024ll) {
        const long long lo = bound(0, n, r0), hi = bound(lo, n, r0 + 1024);
        for (long long r = r0 + threadIdx.x; r < r0 + 1024 && r <= m; r += 256)
            start[r] = static_cast<int>(bound(lo, hi, r));
    }
}

__global__ void plain_fill(long long n, const unsigned long long *__restrict__ keys, const unsigned *__restrict__ vals,
                           unsigned long long cmask, int *col, unsigned *val) {
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        col[i] = static_cast<int>(keys[i] & cmask);
        if (val) val[i] = vals[i];
    }
}

// Symmetric rows: row r's lower neighbours (pairs (lo, r)), then its upper ones ((r, hi)).
// Pair i of the (lo, hi) order goes to row lo, behind the row's lower neighbours; pair i of
// the (hi, lo) order to row hi's start. Both orders carry the other end and the value, so
// both sides are read and written in runs (an index into the other order, as before, cost a
// random 8- and 4-byte read per pair: 308 us for 15.7M pairs).
__global__ void sym_fill(long long np, const unsigned long long *__restrict__ keys, const unsigned *__restrict__ vals,
                         const unsigned long long *__restrict__ hkeys, const unsigned *__restrict__ hvals, int B,
                         const int *__restrict__ up, const int *__restrict__ low, int *col, unsigned *val,
                         const int *err) {
    if (ld_volatile_i32(err) != 0) return;
    const unsigned long long mask = (1ull << B) - 1ull;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < np;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const unsigned long long k = __ldcs(keys + i), h = __ldcs(hkeys + i);
        const int lo = static_cast<int>(k >> B), hi = static_cast<int>(h & mask);
        // up[x] + low[x] entries lie before row x, and row x begins with its lower neighbours
        const long long pu = static_cast<long long>(__ldg(low + lo + 1)) + i;
        const long long pl = static_cast<long long>(__ldg(up + hi)) + i;
        col[pu] = static_cast<int>(k & mask);
        col[pl] = static_cast<int>(h >> B);
        if (val) {
            val[pu] = __ldcs(vals + i);
            val[pl] = __ldcs(hvals + i);
        }
    }
}

__global__ void sym_row_ptr(int m, const int *__restrict__ up, const int *__restrict__ low, int *row_ptr) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r <= m; r += gridDim.x * blockDim.x)
        row_ptr[r] = up[r] + low[r];
}

// The row of every entry from `first` on: row_of[e - first], or (KEYS) keys[e - first] = column << 32 |
// row, for entries before `nnz`. A block takes
// kExpandTile entries whatever rows they belong to (a warp per row left a row of 50,000
// entries to one warp): it finds the row of its first entry by a 32-way search, marks where
// rows begin and spreads the marks by a running maximum. A block whose entries lie so far apart
// that it has not gone past their rows after kExpandSteps steps of 256 rows looks each entry's
// row up instead: going on would walk through millions of empty rows alone.
constexpr int kExpandSteps = 64;
constexpr int kExpandItems = 16;
constexpr int kExpandTile = 256 * kExpandItems;
template <bool KEYS>
__global__ void __launch_bounds__(256) expand_rows(int m, long long first, long long nnz, const int *__restrict__ rp,
                                                   const int *__restrict__ ci, unsigned *row_of,
                                                   unsigned long long *keys) {
    __shared__ int s_row[kExpandTile + kExpandTile / 32];  // padded: threads walk 16 entries each
    __shared__ int s_max[8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto at = [](int i) { return i + (i >> 5); };
    const long long t0 = first + static_cast<long long>(blockIdx.x) * kExpandTile;
    const long long t1 = t0 + kExpandTile < nnz ? t0 + kExpandTile : nnz;
    row_of -= first;
    keys -= first;
    for (int i = tid; i < kExpandTile; i += 256) s_row[at(i)] = -1;
    // last row that begins at or before t0: rp[lo] <= t0 < rp[hi]
    int lo = 0, hi = m;
    while (hi - lo > 1) {
        const int step = (hi - lo + 31) / 32;
        const long long p = static_cast<long long>(lo) + static_cast<long long>(step) * (lane + 1);
        const bool le = p < hi && __ldg(rp + p) <= t0;
        const int c = __popc(__ballot_sync(0xffffffffu, le));
        const long long nh = static_cast<long long>(lo) + static_cast<long long>(step) * (c + 1);
        lo += step * c;
        hi = nh < hi ? static_cast<int>(nh) : hi;
    }
    __syncthreads();
    bool far = false;  // the same for all threads
    int steps = 0;
    for (long long r0 = lo; r0 < m; r0 += 256) {
        if (steps++ == kExpandSteps) {
            far = true;
            break;
        }
        const long long r = r0 + tid;
        int b = 0, e = 0;
        if (r < m) {
            b = __ldg(rp + r);
            e = __ldg(rp + r + 1);
            if (e > b && b < t1) s_row[at(static_cast<int>((b > t0 ? b : t0) - t0))] = static_cast<int>(r);
        }
        if (__syncthreads_or(r < m && e >= t1)) break;
    }
    if (far) {
        for (int i0 = 0; i0 < kExpandItems; i0 += 4) {
            long long e[4];
            int row[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                e[k] = t0 + (i0 + k) * 256 + tid;
                row[k] = lo;
            }
            for (long long s = 1ll << 30; s > 0; s >>= 1) {  // the last row that begins at or before e
                if (lo + s >= m) continue;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (row[k] + s < m && __ldg(rp + row[k] + s) <= e[k]) row[k] += static_cast<int>(s);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (e[k] >= t1) continue;
                if (KEYS)
                    keys[e[k]] = (static_cast<unsigned long long>(static_cast<unsigned>(__ldg(ci + e[k]))) << 32) |
                                 static_cast<unsigned>(row[k]);
                else
                    row_of[e[k]] = static_cast<unsigned>(row[k]);
            }
        }
        return;
    }
    int run = -1;
#pragma unroll
    for (int i = 0; i < kExpandItems; ++i) run = max(run, s_row[at(tid * kExpandItems + i)]);
    int incl = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl = max(incl, y);
    }
    if (lane == 31) s_max[warp] = incl;
    __syncthreads();
    int cur = __shfl_up_sync(0xffffffffu, incl, 1);
    if (lane == 0) cur = -1;
    for (int w = 0; w < warp; ++w) cur = max(cur, s_max[w]);
#pragma unroll
    for (int i = 0; i < kExpandItems; ++i) {
        int *x = &s_row[at(tid * kExpandItems + i)];
        cur = max(cur, *x);
        *x = cur;
    }
    __syncthreads();
    for (int i = tid; t0 + i < t1; i += 256) {
        const unsigned r = static_cast<unsigned>(s_row[at(i)]);
        if (KEYS)
            keys[t0 + i] = (static_cast<unsigned long long>(static_cast<unsigned>(__ldg(ci + t0 + i))) << 32) | r;
        else
            row_of[t0 + i] = r;
    }
}

template <bool KEYS>
cudaError_t launch_expand_rows(apspie_ctx *ctx, const apspie_csr *A, long long first, long long n, unsigned *row_of,
                               unsigned long long *keys) {
    if (n > 0)
        expand_rows<KEYS><<<static_cast<int>((n + kExpandTile - 1) / kExpandTile), 256, 0, ctx->stream>>>(
            A->m, first, first + n, A->row_ptr, A->col_ind, row_of, keys);
    return cudaGetLastError();
}

// Columns (rows of A) out of the sorted (column, row) keys.
__global__ void low_half(long long n, const unsigned long long *__restrict__ keys, int *col) {
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x)
        col[i] = static_cast<int>(__ldcs(keys + i));
}

// The pair that a sort of `passes` passes, the first into pair 0, ends in.
int last_pair(int passes) { return (passes - 1) & 1; }

int grid_for(const apspie_ctx *ctx, long long n) {
    return static_cast<int>(std::max<long long>(1, std::min<long long>((n + 255) / 256, ctx->num_sms * 16LL)));
}

// Row starts out of n sorted keys.
template <class K>
void launch_starts(apspie_ctx *ctx, long long n, const K *keys, int shift, K fmask, int m, int *start, const int *err) {
    const int gm = grid_for(ctx, m + 1ll);
    if (n < m) {
        search_starts<K><<<gm, 256, 0, ctx->stream>>>(n, keys, shift, fmask, m, start, err);
        return;
    }
    if (n > 0) run_starts<K><<<grid_for(ctx, n), 256, 0, ctx->stream>>>(n, keys, shift, fmask, start, err);
    fill_tail<K><<<gm, 256, 0, ctx->stream>>>(n, keys, shift, fmask, m, start, err);
}

apspie_status alloc_owned(apspie_ctx *ctx, int m, int n, long long nnz, int val_type, apspie_csr_owned *out) {
    std::memset(out, 0, sizeof(*out));
    cudaError_t e = owned_alloc(reinterpret_cast<void **>(&out->row_ptr), (static_cast<size_t>(m) + 1) * 4);
    if (e == cudaSuccess) e = owned_alloc(reinterpret_cast<void **>(&out->col_ind), static_cast<size_t>(std::max(nnz, 1LL)) * 4);
    if (e == cudaSuccess && val_type != APSPIE_VAL_NONE)
        e = owned_alloc(reinterpret_cast<void **>(&out->val), static_cast<size_t>(std::max(nnz, 1LL)) * 4);
    if (e != cudaSuccess) {
        apspie_csr_free(out);
        return cuda_error(ctx, e, "csr allocation");
    }
    out->m = m;
    out->n = n;
    out->nnz = static_cast<int32_t>(nnz);
    out->val_type = val_type;
    return APSPIE_OK;
}

}  // namespace

// A pattern's entries sorted by column, the row as the payload (8 bytes each through a pass);
// row starts in out_rp. The last pass writes the rows to out_col.
static apspie_status sort_pattern(apspie_ctx *ctx, const apspie_csr *A, SortBufs<unsigned> &s, unsigned *row_of,
                                  int *out_rp, int *out_col, const unsigned **keys) {
    const long long nnz = A->nnz;
    const int n = A->n;
    const RsPlan pl = rs_plan(0, bit_length(n));
    s.v[last_pair(pl.passes)] = reinterpret_cast<unsigned *>(out_col);
    cudaError_t e = launch_expand_rows<false>(ctx, A, 0, nnz, row_of, nullptr);
    if (e != cudaSuccess) return cuda_error(ctx, e, "transpose rows");
    int which = 0;
    apspie_status st =
        radix_sort(ctx, s, pl, reinterpret_cast<const unsigned *>(A->col_ind), row_of, nnz, 0, &which);
    if (st != APSPIE_OK) return st;
    launch_starts<unsigned>(ctx, nnz, s.k[which], 0, ~0u, n, out_rp, s.err);
    *keys = s.k[which];
    e = cudaGetLastError();
    return e == cudaSuccess ? APSPIE_OK : cuda_error(ctx, e, "transpose");
}

size_t transpose_pattern_need(int n, long long nnz) {
    const size_t c = static_cast<size_t>(nnz) + 1;
    return sort_need<unsigned>(nnz) + Carver::need({c * 4, c * 4, (static_cast<size_t>(n) + 1) * 4});
}

apspie_status transpose_pattern(apspie_ctx *ctx, const apspie_csr *A, void *scratch, PatternCoo *out) {
    Carver c(scratch);
    SortBufs<unsigned> s = carve_sort<unsigned>(c, A->nnz);
    unsigned *row_of = c.take<unsigned>(static_cast<size_t>(A->nnz) + 1);
    int *col = c.take<int>(static_cast<size_t>(A->nnz) + 1);
    int *rp = c.take<int>(static_cast<size_t>(A->n) + 1);
    const unsigned *keys = nullptr;
    apspie_status st = sort_pattern(ctx, A, s, row_of, rp, col, &keys);
    *out = PatternCoo{rp, keys, col, s.err};
    return st;
}

apspie_status expand_entry_rows(apspie_ctx *ctx, const apspie_csr *A, long long first, long long n, unsigned *row_of) {
    cudaError_t e = launch_expand_rows<false>(ctx, A, first, n, row_of, nullptr);
    return e == cudaSuccess ? APSPIE_OK : cuda_error(ctx, e, "entry rows");
}

}  // namespace apspie

using namespace apspie;

extern "C" {

apspie_status apspie_csr_build(apspie_ctx *ctx, int32_t m, int64_t nedges, const int32_t *d_src,
                               const int32_t *d_dst, const void *d_val, int32_t val_type, int32_t flags,
                               apspie_csr_owned *out) {
    if (!ctx || !out || m < 1 || nedges < 0 || (nedges > 0 && (!d_src || !d_dst))) return APSPIE_ERR_INVALID_ARG;
    if (val_type != APSPIE_VAL_NONE && val_type != APSPIE_VAL_I32 && val_type != APSPIE_VAL_F32)
        return APSPIE_ERR_INVALID_ARG;
    if (val_type != APSPIE_VAL_NONE && nedges > 0 && !d_val) return APSPIE_ERR_INVALID_ARG;
    cudaSetDevice(ctx->device);
    std::memset(out, 0, sizeof(*out));
    const bool sym = (flags & APSPIE_BUILD_SYMMETRIZE) != 0;
    const bool dedup = (flags & APSPIE_BUILD_DEDUP) != 0;
    const bool loops = (flags & APSPIE_BUILD_DROP_SELF_LOOPS) != 0;
    if (nedges > 0x7fffffffLL || (sym && 2 * nedges > 0x7fffffffLL))
        return set_error(ctx, APSPIE_ERR_UNSUPPORTED, "apspie_csr_build: more than 2^31 - 1 entries");
    // the all-ones key is a self-loop, so with self-loops dropped it can stand for them; kept
    // self-loops need no such key
    const int B = bit_length(m);
    const unsigned long long sentinel = loops ? (1ull << (2 * B)) - 1ull : ~0ull;
    const long long n = nedges;
    const size_t mi = static_cast<size_t>(m) + 1;
    void *base;
    const size_t need = sort_need<unsigned long long>(n) +
                        Carver::need({mi * 4, mi * 4, 64, static_cast<size_t>(n + 1) * 8, static_cast<size_t>(n + 1) * 4});
    apspie_status st = scratch_reserve(ctx, need, &base);
    if (st != APSPIE_OK) return st;
    Carver c(base);
    SortBufs<unsigned long long> s = carve_sort<unsigned long long>(c, n);
    int *up = c.take<int>(mi);
    int *low = c.take<int>(mi);
    int *flag = c.take<int>(16);  // [0] an id was out of range, [1] pairs kept
    unsigned long long *k2 = c.take<unsigned long long>(n + 1);  // a third buffer pair (symmetric)
    unsigned *v2 = c.take<unsigned>(n + 1);
    cudaError_t e = cudaMemsetAsync(flag, 0, 64, ctx->stream);
    if (e != cudaSuccess) return cuda_error(ctx, e, "apspie_csr_build reset");
    if ((st = sort_begin(ctx, s)) != APSPIE_OK) return st;
    const RsPlan pl = rs_plan(0, 2 * B);
    RsPlan pl2 = rs_plan(0, B);
    if (!sym) pl2.passes = 0;
    const int gk = static_cast<int>(std::max<long long>(1, std::min<long long>((n + 1023) / 1024, ctx->num_sms * 8LL)));
    if (n > 0)
        coo_keys<<<gk, 256, 0, ctx->stream>>>(n, m, d_src, d_dst, static_cast<const unsigned *>(d_val), B, sym ? 1 : 0,
                                              loops ? 1 : 0, pl, s.k[0], s.v[0], s.hist_of(0), flag);
    int which = 0;
    if ((st = radix_passes(ctx, s, 0, pl, s.k[0], s.v[0], n, 1, &which)) != APSPIE_OK) return st;
    // drop sentinels (and duplicates): compact into the other buffer pair
    const int o = which ^ 1;
    if (n > 0)
        compact_pairs<<<static_cast<int>(std::min<long long>((n + kCompactTile - 1) / kCompactTile, ctx->num_sms * 4LL)),
                        256, 0, ctx->stream>>>(n, s.k[which], s.v[which], sentinel, dedup ? 1 : 0, B, pl2,
                                               s.hist_of(1), s.k[o], s.v[o], n < m ? nullptr : up, s.status, s.ticket + kRsOwn, flag + 1,
                                               s.err);
    int h_flag[2] = {0, 0}, sort_err = 0;
    if ((e = cudaGetLastError()) != cudaSuccess ||
        (e = cudaMemcpyAsync(h_flag, flag, 8, cudaMemcpyDeviceToHost, ctx->stream)) != cudaSuccess ||
        (e = cudaMemcpyAsync(&sort_err, s.err, 4, cudaMemcpyDeviceToHost, ctx->stream)) != cudaSuccess ||
        (e = cudaStreamSynchronize(ctx->stream)) != cudaSuccess)
        return cuda_error(ctx, e, "apspie_csr_build count");
    if (h_flag[0]) return set_error(ctx, APSPIE_ERR_INVALID_ARG, "apspie_csr_build: vertex id out of range");
    if (sort_err) return set_error(ctx, static_cast<apspie_status>(sort_err), "apspie_csr_build: sort");
    const long long np = h_flag[1];
    const long long nnz = sym ? 2 * np : np;
    if ((st = alloc_owned(ctx, m, m, nnz, val_type, out)) != APSPIE_OK) return st;
    unsigned *oval = static_cast<unsigned *>(out->val);
    const int gp = grid_for(ctx, np);
    const int gm = grid_for(ctx, m + 1LL);
    const unsigned long long fmask = (1ull << B) - 1ull;
    if (n < m)
        search_starts<unsigned long long><<<gm, 256, 0, ctx->stream>>>(np, s.k[o], B, fmask, m, up, s.err);
    else
        fill_tail<unsigned long long><<<gm, 256, 0, ctx->stream>>>(np, s.k[o], B, fmask, m, up, s.err);
    if (!sym) {
        e = cudaMemcpyAsync(out->row_ptr, up, mi * 4, cudaMemcpyDeviceToDevice, ctx->stream);
        if (np > 0) plain_fill<<<gp, 256, 0, ctx->stream>>>(np, s.k[o], s.v[o], fmask, out->col_ind, oval);
    } else {
        // the pairs again, ordered by hi (stably, so ascending lo within each hi): sorted from
        // where they are into the pre-compaction buffers and the third pair
        SortBufs<unsigned long long> t = s;
        t.k[0] = s.k[which];
        t.v[0] = s.v[which];
        t.k[1] = k2;
        t.v[1] = v2;
        int hw = 0;
        if ((st = radix_passes(ctx, t, 1, pl2, s.k[o], s.v[o], np, 0, &hw)) != APSPIE_OK) {
            apspie_csr_free(out);
            return st;
        }
        launch_starts<unsigned long long>(ctx, np, t.k[hw], 0, fmask, m, low, s.err);
        sym_row_ptr<<<gm, 256, 0, ctx->stream>>>(m, up, low, out->row_ptr);
        if (np > 0)
            sym_fill<<<gp, 256, 0, ctx->stream>>>(np, s.k[o], s.v[o], t.k[hw], t.v[hw], B, up, low, out->col_ind, oval,
                                                  s.err);
    }
    if (e != cudaSuccess || (e = cudaGetLastError()) != cudaSuccess ||
        (e = cudaMemcpyAsync(&sort_err, s.err, 4, cudaMemcpyDeviceToHost, ctx->stream)) != cudaSuccess ||
        (e = cudaStreamSynchronize(ctx->stream)) != cudaSuccess) {
        apspie_csr_free(out);
        return cuda_error(ctx, e, "apspie_csr_build");
    }
    if (sort_err) {
        apspie_csr_free(out);
        return set_error(ctx, static_cast<apspie_status>(sort_err), "apspie_csr_build: sort");
    }
    return APSPIE_OK;
}

// Entries with values are sorted as (column, row) keys with the value as the payload, 12
// bytes each through a pass (an index as the payload, as before, costs two random reads per
// entry at the end); the last pass writes the payload straight into the output.
apspie_status apspie_csr_transpose(apspie_ctx *ctx, const apspie_csr *A, apspie_csr_owned *out) {
    if (!ctx || !out) return APSPIE_ERR_INVALID_ARG;
    cudaSetDevice(ctx->device);
    std::memset(out, 0, sizeof(*out));
    apspie_status st = check_csr_view(ctx, A, "apspie_csr_transpose");
    if (st != APSPIE_OK) return st;
    if (ctx->validate && (st = validate_csr(ctx, A, false)) != APSPIE_OK) return st;
    const long long nnz = A->nnz;
    const int n = A->n;
    const bool valued = A->val != nullptr && A->val_type != APSPIE_VAL_NONE;
    void *base;
    st = scratch_reserve(ctx, valued ? sort_need<unsigned long long>(nnz)
                                     : sort_need<unsigned>(nnz) + Carver::need({static_cast<size_t>(nnz + 1) * 4}),
                         &base);
    if (st != APSPIE_OK) return st;
    if ((st = alloc_owned(ctx, n, A->m, nnz, A->val ? A->val_type : APSPIE_VAL_NONE, out)) != APSPIE_OK) return st;
    Carver c(base);
    const int *err = nullptr;
    cudaError_t e = cudaSuccess;
    int which = 0;
    if (valued) {
        SortBufs<unsigned long long> s = carve_sort<unsigned long long>(c, nnz);
        const RsPlan pl = rs_plan(32, 32 + bit_length(n));
        s.v[last_pair(pl.passes)] = static_cast<unsigned *>(out->val);
        err = s.err;
        // the keys are made in the pair that the first pass does not write
        e = launch_expand_rows<true>(ctx, A, 0, nnz, nullptr, s.k[1]);
        if (e == cudaSuccess)
            st = radix_sort(ctx, s, pl, s.k[1], static_cast<const unsigned *>(A->val), nnz, 0, &which);
        if (e == cudaSuccess && st == APSPIE_OK) {
            launch_starts<unsigned long long>(ctx, nnz, s.k[which], 32, ~0ull, n, out->row_ptr, err);
            if (nnz > 0) low_half<<<grid_for(ctx, nnz), 256, 0, ctx->stream>>>(nnz, s.k[which], out->col_ind);
        }
    } else {
        SortBufs<unsigned> s = carve_sort<unsigned>(c, nnz);
        unsigned *row_of = c.take<unsigned>(nnz + 1);
        const unsigned *keys = nullptr;
        err = s.err;
        st = sort_pattern(ctx, A, s, row_of, out->row_ptr, out->col_ind, &keys);
    }
    int sort_err = 0;
    if (st == APSPIE_OK &&
        (e != cudaSuccess || (e = cudaGetLastError()) != cudaSuccess ||
         (e = cudaMemcpyAsync(&sort_err, err, 4, cudaMemcpyDeviceToHost, ctx->stream)) != cudaSuccess ||
         (e = cudaStreamSynchronize(ctx->stream)) != cudaSuccess))
        st = cuda_error(ctx, e, "apspie_csr_transpose");
    if (st == APSPIE_OK && sort_err)
        st = set_error(ctx, static_cast<apspie_status>(sort_err), "apspie_csr_transpose: sort");
    if (st != APSPIE_OK) apspie_csr_free(out);
    return st;
}

}  // extern "C"
