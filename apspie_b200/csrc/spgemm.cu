// Row-binned hash SpGEMM  C = A * B  (Gustavson, row by row).
//
// Replaces the reference's 2-D partitioned outer-product hash SpGEMM
// (src/spgemm.cuh:131-342, src/spgemmKernel.cuh:439-738: CSR->DCSC per partition,
// SetOpPairs, cudpp segmented scan, MergePathPartitions, KernelInsert into per-pair global
// tables of 131071 slots with <= 25 double-hash probes, then a segmented radix sort of
// every table and a COO->CSR rebuild) and its cuSPARSE csrgemm wrappers
// (src/spgemm.cuh:344-445, src/tc.cuh:62-165). Results: C's structure is the exact
// union of products; rows are sorted by column; int32 values are exact; FP32 values of a
// register-tier row (at most 128 products) are summed in increasing position of A's row
// (the oracle's order, so bit-identical); block/global-tier rows accumulate with
// atomicAdd (order-dependent rounding only).
//
// Pipeline (all on the context stream):
//  1. rowinfo: per row, ub = sum of deg_B over A's row (products) -> bin; rows appended to
//     per-bin lists; global-tier rows get a hash table carved from scratch. One sync
//     reads the bin sizes.
//  2. symbolic: per bin, count distinct columns per row with a hash set -> cnt[]
//  3. scan cnt -> row_ptr(C); one sync reads nnz(C) (the caller may allocate C here)
//  4. numeric: register tiers sort the products and sum each column's run; hash tiers
//     accumulate values in the table, then emit the row sorted by ranking entries against
//     a 64K-column bitmap window (prefix popcounts).
// Bins: 0 no products | 1-3 ub <= 32 / 64 / 128: 8 or 16 lanes per row, the row's products
// held in registers (4 or 8 per lane) and sorted by (column, product index) with a bitonic
// network; duplicates are then adjacent and summed in product order |
// 4 ub <= 1024: one block, 2048-slot shared table | 5-7 larger: with at most 49,152 columns
// one block and a dense accumulator in shared memory, else (bin 5) one block and a global
// table of >= 2*min(ub, columns) slots (power of two). Tables stay at most half full.
#include <algorithm>
#include <cstring>

#include "common.cuh"

namespace apspie {
namespace {

constexpr int kEmptyKey = -1;
constexpr int kBins = 8;
constexpr int kBinBlock = 4;   // shared-memory hash table tier
constexpr int kBinGlobal = 5;  // global-memory hash table tier, or
constexpr int kBinDense = 5;   // 5-7: dense accumulator tier, by size class (see sg_dense)
// The dense tier serves every row past the shared-table tier when C has at most this many
// columns: an accumulator and a bit per column fit in an SM's shared memory (200 KB).
constexpr int kDenseCols = 48 * 1024;
bool takes_dense(const apspie_csr *A, const apspie_csr *B) {
    return B->n <= kDenseCols && A->nnz <= kMaxStepped && B->nnz <= kMaxStepped;
}
constexpr int kDenseBlock = 1024;
constexpr int kBlockTS = 2048;
constexpr int kSgBlock = 256;
constexpr int kWindowBits = 65536;  // columns per bitmap window
constexpr int kWindowWords = kWindowBits / 32;

struct SgInfo {
    int bin_count[kBins];
    int overflow;  // hash probe overflow or scan overflow
    int ticket;    // rows of the dense tier handed out
    long long global_slots;
};

// Rows of at most reg_max products (0, 32, 64 or 128) go to the register tiers (needs B
// with at most 2^24 columns, so that a key column << 7 | product stays below the padding
// key 0xffffffff; the host passes reg_max 0 otherwise), rows of at most block_max (<= 1024,
// the shared table holds 2048 slots) to the shared-memory table, longer rows to the dense
// tier (in three classes, so that the longest can start first) or a global table.
__device__ __forceinline__ int bin_of(long long ub, int degA, int reg_max, int block_max, int dense) {
    const long long w = ub > degA ? ub : degA;
    if (ub == 0) return 0;
    if (w <= reg_max) return w <= 32 ? 1 : (w <= 64 ? 2 : 3);
    if (w <= block_max) return kBinBlock;
    if (dense) return kBinDense + (w <= 8192 ? 0 : (w <= 65536 ? 1 : 2));
    return kBinGlobal;
}

// Slots of a global table for a row of ub products over n columns: at most half full.
__device__ __forceinline__ long long table_slots(long long ub, int n) {
    const long long most = ub < n ? ub : n;
    long long ts = 64;
    while (ts < 2 * most) ts <<= 1;
    return ts;
}

__device__ __forceinline__ unsigned hash_slot(int col, int log2ts) {
    return (static_cast<unsigned>(col) * 2654435761u) >> (32 - log2ts);
}

template <typename V>
__device__ __forceinline__ V vmul(V a, V b);
template <>
__device__ __forceinline__ float vmul<float>(float a, float b) { return __fmul_rn(a, b); }
template <>
__device__ __forceinline__ int vmul<int>(int a, int b) { return a * b; }
template <typename V>
__device__ __forceinline__ V vadd(V a, V b);
template <>
__device__ __forceinline__ float vadd<float>(float a, float b) { return __fadd_rn(a, b); }
template <>
__device__ __forceinline__ int vadd<int>(int a, int b) { return a + b; }

struct Mat {
    const int *rp;
    const int *ci;
    const void *val;
};

// ---------------------------------------------------------------- 1. row info / bins
// 8 lanes per row: ub = sum of deg_B over A's row, and the row's bin.
__global__ void sg_rowinfo(int m, Mat A, Mat B, int ncols, int reg_max, int block_max, int dense, long long *ub,
                           unsigned char *row_bin, SgInfo *info, long long *tbl_off) {
    const int sub = threadIdx.x & 7;
    const int grp = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
    const int ngrp = (gridDim.x * blockDim.x) >> 3;
    const unsigned gmask = 0xffu << (threadIdx.x & 24);
    for (int i0 = grp - (grp & 3); i0 < m; i0 += ngrp) {  // the warp's 4 groups move together
        const int i = i0 + (grp & 3);
        long long s = 0;
        int r0 = 0, r1 = 0;
        if (i < m) {
            r0 = __ldg(A.rp + i);
            r1 = __ldg(A.rp + i + 1);
            for (int e = r0 + sub; e < r1; e += 8) {
                const int k = __ldg(A.ci + e);
                s += __ldg(B.rp + k + 1) - __ldg(B.rp + k);
            }
        }
        for (int o = 4; o; o >>= 1) s += __shfl_down_sync(gmask, s, o, 8);
        if (i < m && sub == 0) {
            ub[i] = s;
            const int b = bin_of(s, r1 - r0, reg_max, block_max, dense);
            row_bin[i] = static_cast<unsigned char>(b);
            if (b == kBinGlobal && !dense)
                tbl_off[i] = static_cast<long long>(
                    atomicAdd(reinterpret_cast<unsigned long long *>(&info->global_slots),
                              static_cast<unsigned long long>(table_slots(s, ncols))));
        }
    }
}

// Per-bin row lists (stride m): each block counts its rows per bin with warp ballots,
// reserves room with one global atomic per bin, then scatters.
__global__ void sg_binlists(int m, const unsigned char *__restrict__ row_bin, int *bin_rows, SgInfo *info) {
    __shared__ int cnt[kBins];
    __shared__ int base[kBins];
    const int lane = threadIdx.x & 31;
    for (int c0 = blockIdx.x * blockDim.x; c0 < m; c0 += gridDim.x * blockDim.x) {
        if (threadIdx.x < kBins) cnt[threadIdx.x] = 0;
        __syncthreads();
        const int i = c0 + threadIdx.x;
        const int b = i < m ? row_bin[i] : -1;
        int pos = 0;
#pragma unroll
        for (int k = 0; k < kBins; ++k) {
            const unsigned mk = __ballot_sync(0xffffffffu, b == k);
            int wbase = 0;
            if (mk && lane == __ffs(mk) - 1) wbase = atomicAdd(&cnt[k], __popc(mk));
            wbase = __shfl_sync(0xffffffffu, wbase, mk ? __ffs(mk) - 1 : 0);
            if (b == k) pos = wbase + __popc(mk & ((1u << lane) - 1u));
        }
        __syncthreads();
        if (threadIdx.x < kBins && cnt[threadIdx.x])
            base[threadIdx.x] = atomicAdd(&info->bin_count[threadIdx.x], cnt[threadIdx.x]);
        __syncthreads();
        if (b >= 0) bin_rows[static_cast<long long>(b) * m + base[b] + pos] = i;
        __syncthreads();
    }
}

__device__ __forceinline__ void st_stream(float *p, float v) { __stcs(p, v); }
__device__ __forceinline__ void st_stream(int *p, int v) { __stcs(p, v); }

// ---------------------------------------------------------------- register tier
// A group of G lanes per row of at most N = G * K products, K of them in each lane's
// registers: 8 lanes x 4, 8 x 8 or 16 x 8.
template <int G, int K>
struct RegTier {
    static constexpr int N = G * K;
    static constexpr int WORDS = N / 32;
    static constexpr int QB = N == 32 ? 5 : N == 64 ? 6 : 7;
    static constexpr int ROWS = 32 / G;  // rows a warp handles side by side
    // shared-memory words of a row: columns, values (with a word of padding after every 8, so
    // that lanes that write 8 consecutive ranks each use different banks), A entries (two words
    // each); the groups of a warp are 8 (16) words apart modulo the banks. Symbolic: the same
    // words are a table of 4 N columns.
    static constexpr int PADDED = N + N / 8;
    static constexpr int STRIDE = 2 * PADDED + 2 * N + (N == 32 ? 0 : N == 64 ? 8 : 16);
    __device__ static __forceinline__ int padded(int rank) { return rank + (rank >> 3); }
};

// Ascending sort of the group's N keys, element index sub * K + r: bitonic merges whose first
// step compares mirrored elements, so that every comparison puts the smaller key first and no
// direction has to be chosen. Elements of one lane are compared in registers; of the 21
// steps for N = 64, 15 are (one lane per key took a shuffle for each).
template <int G, int K>
__device__ __forceinline__ void group_sort(unsigned (&key)[K], int sub) {
    constexpr unsigned FULL = 0xffffffffu;
#pragma unroll
    for (int k = 2; k <= G * K; k <<= 1) {
        if (k <= K) {
#pragma unroll
            for (int r = 0; r < K; ++r) {
                const int p = r ^ (k - 1);
                if (p > r) {
                    const unsigned a = min(key[r], key[p]), b = max(key[r], key[p]);
                    key[r] = a;
                    key[p] = b;
                }
            }
        } else {
            unsigned other[K];
#pragma unroll
            for (int r = 0; r < K; ++r) other[r] = __shfl_xor_sync(FULL, key[K - 1 - r], k / K - 1, G);
            const bool lower = (sub & (k / K / 2)) == 0;
#pragma unroll
            for (int r = 0; r < K; ++r) key[r] = lower ? min(key[r], other[r]) : max(key[r], other[r]);
        }
#pragma unroll
        for (int j = k >> 2; j > 0; j >>= 1) {
            if (j >= K) {
                const bool lower = (sub & (j / K)) == 0;
#pragma unroll
                for (int r = 0; r < K; ++r) {
                    const unsigned o = __shfl_xor_sync(FULL, key[r], j / K, G);
                    key[r] = lower ? min(key[r], o) : max(key[r], o);
                }
            } else {
#pragma unroll
                for (int r = 0; r < K; ++r) {
                    const int p = r ^ j;
                    if (p > r) {
                        const unsigned a = min(key[r], key[p]), b = max(key[r], key[p]);
                        key[r] = a;
                        key[p] = b;
                    }
                }
            }
        }
    }
}

template <typename V>
__device__ __forceinline__ int as_word(V v);
template <>
__device__ __forceinline__ int as_word<float>(float v) { return __float_as_int(v); }
template <>
__device__ __forceinline__ int as_word<int>(int v) { return v; }
template <typename V>
__device__ __forceinline__ V from_word(int w);
template <>
__device__ __forceinline__ float from_word<float>(int w) { return __int_as_float(w); }
template <>
__device__ __forceinline__ int from_word<int>(int w) { return w; }

// Product q of a row belongs to the last entry of A's row (among those whose row of B is not
// empty) that begins at or before q: where the entries begin is an N-bit mask in every lane's
// registers, and counting its bits gives the entry. The product gets the key
// (column << QB) | q. Numeric: after the sort the products of one output column are adjacent
// and in increasing q, i.e. increasing position in A's row, so a run's head sums them in the
// oracle's order (bit-identical FP32); the row is put together in shared memory and written
// by the whole warp. Symbolic: only the distinct columns are counted, without sorting: every
// lane stores its keys in a table (a slot per hash of the column) and reads them back; the
// key that is found was counted by its owner, an equal column is a repeat, anything else goes
// into the next round with another hash. Nothing has to be cleared, and no atomics are made.
// Requires B->n <= 2^24 (see bin_of).
//
// What bounds it: the shared-memory and shuffle pipe (68 % of its wavefronts in the symbolic
// pass), then issue. C = A * A of 2^20 uniform rows of 8 (64 products each, 67M in all): one
// warp per row, one lane per two keys, numeric 592 us and symbolic 422 us (atomicCAS table);
// now 391 us and 215 us (numeric 515 us with ranks 8 words apart for neighbouring lanes and
// every run looked for in shared memory).
template <int G, int K, bool NUMERIC, typename V>
__global__ void __launch_bounds__(kSgBlock) sg_reg(const int *__restrict__ rows, int nrows, Mat A, Mat B, int *cnt,
                                                   const int *__restrict__ crp, int *cci, V *cval) {
    using T = RegTier<G, K>;
    constexpr int N = T::N, QB = T::QB, ROWS = T::ROWS, WORDS = T::WORDS;
    constexpr unsigned QMASK = (1u << QB) - 1u, PAD = 0xffffffffu, FULL = 0xffffffffu;
    constexpr unsigned GMASK = (1u << G) - 1u;
    __shared__ __align__(16) int smem[kSgBlock / 32 * ROWS * T::STRIDE];
    const int lane = threadIdx.x & 31, sub = lane & (G - 1), grp = lane / G;
    int *row_sm = smem + ((threadIdx.x >> 5) * ROWS + grp) * T::STRIDE;
    int *skey = row_sm, *spv = row_sm + T::PADDED, *sent = row_sm + 2 * T::PADDED;  // sent: (B position - q, A value)
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const V *aval = static_cast<const V *>(A.val);
    const V *bval = static_cast<const V *>(B.val);
    for (int w = warp * ROWS; w < nrows; w += nwarps * ROWS) {
        const bool on = w + grp < nrows;
        const int i = on ? __ldg(rows + w + grp) : 0;
        const int rA = on ? __ldg(A.rp + i) : 0;
        const int degA = on ? __ldg(A.rp + i + 1) - rA : 0;  // <= N by binning
        // A's entries: rows of B that are not empty, their products' offsets
        unsigned begin[WORDS];
#pragma unroll
        for (int x = 0; x < WORDS; ++x) begin[x] = 0u;
        int ub = 0, listed = 0;
#pragma unroll
        for (int r = 0; r < K; ++r) {
            if (!__any_sync(FULL, r * G < degA)) break;
            const int t = r * G + sub;
            int b0 = 0, len = 0;
            V av = V(0);
            if (t < degA) {
                const int k = __ldg(A.ci + rA + t);
                b0 = __ldg(B.rp + k);
                len = __ldg(B.rp + k + 1) - b0;
                if (NUMERIC) av = __ldg(aval + rA + t);
            }
            int incl = len;
#pragma unroll
            for (int o = 1; o < G; o <<= 1) {
                const int y = __shfl_up_sync(FULL, incl, o, G);
                if (sub >= o) incl += y;
            }
            const unsigned some = (__ballot_sync(FULL, len > 0) >> (grp * G)) & GMASK;
            if (len > 0) {
                const int q0 = ub + incl - len;
                const int at = listed + __popc(some & ((1u << sub) - 1u));
                *reinterpret_cast<int2 *>(sent + 2 * at) = make_int2(b0 - q0, NUMERIC ? as_word<V>(av) : 0);
#pragma unroll
                for (int x = 0; x < WORDS; ++x)
                    if ((q0 >> 5) == x) begin[x] |= 1u << (q0 & 31);
            }
            listed += __popc(some);
            ub += __shfl_sync(FULL, incl, G - 1, G);
        }
#pragma unroll
        for (int x = 0; x < WORDS; ++x)
#pragma unroll
            for (int o = 1; o < G; o <<= 1) begin[x] |= __shfl_xor_sync(FULL, begin[x], o, G);
        __syncwarp();
        // the products, G at a time (so that neighbouring lanes read neighbouring entries of B)
        unsigned key[K];
        int e[K], aw[K];
#pragma unroll
        for (int r = 0; r < K; ++r) {
            const int q = r * G + sub;
            int own = -1;
#pragma unroll
            for (int x = 0; x < WORDS; ++x) {
                if (x < (r * G) / 32) own += __popc(begin[x]);
                if (x == (r * G) / 32) own += __popc(begin[x] & (FULL >> (31 - (q & 31))));
            }
            e[r] = -1;
            aw[r] = 0;
            if (q < ub) {
                const int2 en = *reinterpret_cast<const int2 *>(sent + 2 * own);
                e[r] = en.x + q;
                aw[r] = en.y;
            }
        }
#pragma unroll
        for (int r = 0; r < K; ++r)
            key[r] = e[r] >= 0 ? (static_cast<unsigned>(__ldg(B.ci + e[r])) << QB) | static_cast<unsigned>(r * G + sub)
                               : PAD;
        if (!NUMERIC) {
            __syncwarp();  // the entries were read: their words become part of the table
            int fresh = 0;
            unsigned todo = 0u;
#pragma unroll
            for (int r = 0; r < K; ++r) todo |= key[r] != PAD ? 1u << r : 0u;
            for (unsigned mul = 2654435761u; __any_sync(FULL, todo != 0u); mul = mul * 0x9e3779b1u + 2u) {
                constexpr int LOG = QB + 2;  // SLOTS = 4 N
                unsigned slot[K];
#pragma unroll
                for (int r = 0; r < K; ++r) {
                    slot[r] = ((key[r] >> QB) * mul) >> (32 - LOG);
                    if ((todo >> r) & 1u) row_sm[slot[r]] = static_cast<int>(key[r]);
                }
                __syncwarp();
#pragma unroll
                for (int r = 0; r < K; ++r) {
                    if (!((todo >> r) & 1u)) continue;
                    const unsigned got = static_cast<unsigned>(row_sm[slot[r]]);
                    fresh += got == key[r];
                    if ((got ^ key[r]) <= QMASK) todo &= ~(1u << r);
                }
                __syncwarp();
            }
#pragma unroll
            for (int o = 1; o < G; o <<= 1) fresh += __shfl_xor_sync(FULL, fresh, o, G);
            if (on && sub == 0) cnt[i] = fresh;
            continue;
        }
#pragma unroll
        for (int r = 0; r < K; ++r)
            if (e[r] >= 0) spv[r * G + sub] = as_word<V>(vmul<V>(from_word<V>(aw[r]), __ldg(bval + e[r])));
        group_sort<G, K>(key, sub);
        unsigned prev = __shfl_up_sync(FULL, key[K - 1], 1, G);
        if (sub == 0) prev = ~key[0];  // another column, whatever key[0] is
        unsigned heads = 0u, repeats = 0u;
#pragma unroll
        for (int r = 0; r < K; ++r) {
            const unsigned before = r == 0 ? prev : key[r > 0 ? r - 1 : 0];
            if (key[r] != PAD) ((before ^ key[r]) > QMASK ? heads : repeats) |= 1u << r;
        }
        __syncwarp();  // the products are there
        // a run's head sums it; its column and sum go to the run's rank
        V sum[K];
#pragma unroll
        for (int r = 0; r < K; ++r) sum[r] = ((heads >> r) & 1u) ? from_word<V>(spv[key[r] & QMASK]) : V(0);
        if (__any_sync(FULL, repeats != 0u)) {  // some row of the warp has equal columns: runs are walked
#pragma unroll
            for (int r = 0; r < K; r += 4)
                *reinterpret_cast<uint4 *>(skey + sub * K + r) = make_uint4(key[r], key[r + 1], key[r + 2], key[r + 3]);
            __syncwarp();
#pragma unroll
            for (int r = 0; r < K; ++r) {
                if (!((heads >> r) & 1u)) continue;
                if (r + 1 < K && !((repeats >> (r + 1)) & 1u)) continue;
                for (int f = sub * K + r + 1; f < ub; ++f) {
                    const unsigned kf = static_cast<unsigned>(skey[f]);
                    if ((kf ^ key[r]) > QMASK) break;
                    sum[r] = vadd<V>(sum[r], from_word<V>(spv[kf & QMASK]));
                }
            }
        }
        const int mine = __popc(heads);
        int incl = mine;
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
            const int y = __shfl_up_sync(FULL, incl, o, G);
            if (sub >= o) incl += y;
        }
        const int total = __shfl_sync(FULL, incl, G - 1, G);
        const int c0 = on ? __ldg(crp + i) : 0;
        __syncwarp();  // keys and products were read: their words take the row
        int at = incl - mine;
#pragma unroll
        for (int r = 0; r < K; ++r)
            if ((heads >> r) & 1u) {
                skey[T::padded(at)] = static_cast<int>(key[r] >> QB);
                spv[T::padded(at)] = as_word<V>(sum[r]);
                ++at;
            }
        __syncwarp();
        // streaming stores: C is written once and never re-read here, so it should not push B
        // (re-read by every row that names it) out of L2
#pragma unroll
        for (int g = 0; g < ROWS; ++g) {
            const int n = __shfl_sync(FULL, total, g * G), c = __shfl_sync(FULL, c0, g * G);
            const int *rs = row_sm + (g - grp) * T::STRIDE;
            for (int q = lane; q < n; q += 32) {
                __stcs(cci + c + q, rs[T::padded(q)]);
                st_stream(cval + c + q, from_word<V>(rs[T::PADDED + T::padded(q)]));
            }
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------- block / global tiers
template <typename V>
struct BlockTierSmem {
    int keys[kBlockTS];
    V vals[kBlockTS];
    int sk_rs[kSgBlock];
    int soff[kSgBlock + 1];
    V sa[kSgBlock];
    unsigned bits[kWindowWords];
    int wpre[kWindowWords];  // exclusive popcount prefix of the window's words
    int scan_tmp[33];
    int red[2];
};

template <typename V>
__device__ __forceinline__ void atomic_vadd(V *p, V v);
template <>
__device__ __forceinline__ void atomic_vadd<float>(float *p, float v) { atomicAdd(p, v); }
template <>
__device__ __forceinline__ void atomic_vadd<int>(int *p, int v) { atomicAdd(p, v); }

// One block per row. GLOBAL: the table lives in scratch at tbl_off[i] with a per-row size;
// otherwise it is the block's shared-memory table of kBlockTS slots. Products of all A
// entries are inserted concurrently (values by atomicAdd).
template <bool GLOBAL, bool NUMERIC, typename V>
__global__ void __launch_bounds__(kSgBlock) sg_block(const int *__restrict__ rows, int nrows, Mat A, Mat B,
                                                     int ncols, const long long *__restrict__ ub_all,
                                                     const long long *__restrict__ tbl_off, int *gkeys,
                                                     V *gvals, int *cnt, const int *__restrict__ crp, int *cci,
                                                     V *cval, SgInfo *info) {
    __shared__ BlockTierSmem<V> sm;
    const V *aval = static_cast<const V *>(A.val);
    const V *bval = static_cast<const V *>(B.val);
    const int tid = threadIdx.x;
    for (int w = blockIdx.x; w < nrows; w += gridDim.x) {
        const int i = rows[w];
        int *keys = sm.keys;
        V *vals = sm.vals;
        long long ts = kBlockTS;
        if (GLOBAL) {
            ts = table_slots(ub_all[i], ncols);
            keys = gkeys + tbl_off[i];
            vals = gvals + tbl_off[i];
        }
        int log2ts = 0;
        while ((1LL << log2ts) < ts) ++log2ts;
        for (long long s = tid; s < ts; s += kSgBlock) {
            keys[s] = kEmptyKey;
            if (NUMERIC) vals[s] = V(0);
        }
        if (tid == 0) sm.red[0] = 0;
        __syncthreads();
        const int rA = A.rp[i];
        const int degA = A.rp[i + 1] - rA;
        int fresh = 0;
        for (int c0 = 0; c0 < degA; c0 += kSgBlock) {
            const int t = c0 + tid;
            int d = 0;
            if (t < degA) {
                const int k = A.ci[rA + t];
                const int b0 = B.rp[k];
                sm.sk_rs[tid] = b0;
                d = B.rp[k + 1] - b0;
                if (NUMERIC) sm.sa[tid] = aval[rA + t];
            }
            int tot;
            const int ex = block_exclusive_scan<kSgBlock>(d, tot, sm.scan_tmp);
            sm.soff[tid] = ex;
            if (tid == 0) sm.soff[kSgBlock] = tot;
            __syncthreads();
            const int nt = degA - c0 < kSgBlock ? degA - c0 : kSgBlock;
            for (int q = tid; q < tot; q += kSgBlock) {
                int lo = 0, hi = nt;
                while (hi - lo > 1) {
                    const int mid = (lo + hi) >> 1;
                    if (sm.soff[mid] <= q)
                        lo = mid;
                    else
                        hi = mid;
                }
                const int e = sm.sk_rs[lo] + (q - sm.soff[lo]);
                const int col = B.ci[e];
                unsigned long long s = hash_slot(col, log2ts < 32 ? log2ts : 31) & (ts - 1);
                long long probes = 0;
                for (;;) {
                    const int k = GLOBAL ? __ldcg(keys + s) : keys[s];
                    if (k == col) break;
                    if (k == kEmptyKey) {
                        const int old = atomicCAS(keys + s, kEmptyKey, col);
                        if (old == kEmptyKey) {
                            ++fresh;
                            break;
                        }
                        if (old == col) break;
                    }
                    s = (s + 1) & (ts - 1);
                    if (++probes > ts) {
                        atomicOr(&info->overflow, 1);
                        break;
                    }
                }
                if (NUMERIC) atomic_vadd<V>(vals + s, vmul<V>(sm.sa[lo], bval[e]));
            }
            __syncthreads();
        }
        if (!NUMERIC) {
            for (int o = 16; o; o >>= 1) fresh += __shfl_down_sync(0xffffffffu, fresh, o);
            if ((tid & 31) == 0) atomicAdd(&sm.red[0], fresh);
            __syncthreads();
            if (tid == 0) cnt[i] = sm.red[0];
            __syncthreads();
            continue;
        }
        // emit the row sorted by column: rank entries inside 64K-column bitmap windows
        int cmin = 0x7fffffff, cmax = -1;
        for (long long s = tid; s < ts; s += kSgBlock) {
            const int k = GLOBAL ? __ldcg(keys + s) : keys[s];
            if (k != kEmptyKey) {
                cmin = min(cmin, k);
                cmax = max(cmax, k);
            }
        }
        for (int o = 16; o; o >>= 1) {
            cmin = min(cmin, __shfl_down_sync(0xffffffffu, cmin, o));
            cmax = max(cmax, __shfl_down_sync(0xffffffffu, cmax, o));
        }
        if (tid == 0) {
            sm.red[0] = 0x7fffffff;
            sm.red[1] = -1;
        }
        __syncthreads();
        if ((tid & 31) == 0) {
            atomicMin(&sm.red[0], cmin);
            atomicMax(&sm.red[1], cmax);
        }
        __syncthreads();
        cmin = sm.red[0];
        cmax = sm.red[1];
        const int c0 = crp[i];
        int done = 0;
        for (long long w0 = (cmax < 0 ? 1 : (cmin / kWindowBits)) * static_cast<long long>(kWindowBits);
             w0 <= cmax; w0 += kWindowBits) {
            for (int x = tid; x < kWindowWords; x += kSgBlock) sm.bits[x] = 0u;
            __syncthreads();
            for (long long s = tid; s < ts; s += kSgBlock) {
                const int k = GLOBAL ? __ldcg(keys + s) : keys[s];
                if (k != kEmptyKey && k >= w0 && k < w0 + kWindowBits) {
                    const int off = static_cast<int>(k - w0);
                    atomicOr(&sm.bits[off >> 5], 1u << (off & 31));
                }
            }
            __syncthreads();
            // exclusive prefix of popcounts over the window's words (WPT words per thread)
            constexpr int WPT = kWindowWords / kSgBlock;
            int local = 0;
#pragma unroll
            for (int x = 0; x < WPT; ++x) local += __popc(sm.bits[tid * WPT + x]);
            int tot;
            int run = block_exclusive_scan<kSgBlock>(local, tot, sm.scan_tmp);
#pragma unroll
            for (int x = 0; x < WPT; ++x) {
                sm.wpre[tid * WPT + x] = run;
                run += __popc(sm.bits[tid * WPT + x]);
            }
            __syncthreads();
            // every entry of the window lands at its column's rank
            for (long long s = tid; s < ts; s += kSgBlock) {
                const int k = GLOBAL ? __ldcg(keys + s) : keys[s];
                if (k != kEmptyKey && k >= w0 && k < w0 + kWindowBits) {
                    const int off = static_cast<int>(k - w0);
                    const int word = off >> 5;
                    const int rank = sm.wpre[word] + __popc(sm.bits[word] & ((1u << (off & 31)) - 1u));
                    __stcs(cci + c0 + done + rank, k);
                    st_stream(cval + c0 + done + rank, GLOBAL ? __ldcg(vals + s) : vals[s]);
                }
            }
            done += tot;
            __syncthreads();
        }
    }
}

// ---------------------------------------------------------------- dense tier
// Rows of many products over few columns: one block per row, an accumulator and a presence
// bit per column of C in shared memory (no hashing, no probing, no sorting: columns are
// ranked by prefix popcounts). A warp takes an entry of A's row and its lanes walk B's row,
// so neighbouring lanes add to neighbouring columns. Blocks take rows from a counter, the
// size classes from the longest down. The accumulators are cleared as they are written out.
//
// Measured, A * A of an R-MAT matrix of 9,001 rows and 123,180 entries (int32, 8.1M entries in
// C): numeric 2.9 ms and symbolic 0.87 ms with hash tables in global memory (a probe chain
// and two L2 atomics per product, and a table walked three times to sort a row); now 0.19 ms
// and 0.073 ms. FP32 sums are taken in no fixed order, as in the hash tiers.
template <bool NUMERIC, typename V>
size_t dense_smem(int ncols) {
    const size_t nw = (static_cast<size_t>(ncols) + 31) / 32;
    return NUMERIC ? nw * 8 + static_cast<size_t>(ncols) * sizeof(V) : nw * 4;
}

template <bool NUMERIC, typename V>
__global__ void __launch_bounds__(kDenseBlock) sg_dense(const int *__restrict__ rows7, int n7,
                                                        const int *__restrict__ rows6, int n6,
                                                        const int *__restrict__ rows5, int n5, Mat A, Mat B, int ncols,
                                                        int *cnt, const int *__restrict__ crp, int *cci, V *cval,
                                                        int *ticket) {
    extern __shared__ unsigned dyn[];
    __shared__ int scan_tmp[33];
    __shared__ int s_next;
    constexpr int NWARP = kDenseBlock / 32;
    const int nw = (ncols + 31) >> 5;
    unsigned *bits = dyn;
    int *wpre = reinterpret_cast<int *>(dyn + nw);       // numeric only
    V *acc = reinterpret_cast<V *>(dyn + 2 * nw);        // numeric only
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const V *aval = static_cast<const V *>(A.val);
    const V *bval = static_cast<const V *>(B.val);
    for (int w = tid; w < nw; w += kDenseBlock) bits[w] = 0u;
    if (NUMERIC)
        for (int c = tid; c < ncols; c += kDenseBlock) acc[c] = V(0);
    for (;;) {
        if (tid == 0) s_next = atomicAdd(ticket, 1);
        __syncthreads();
        const int at = s_next;
        if (at >= n7 + n6 + n5) break;
        const int i = at < n7 ? rows7[at] : at < n7 + n6 ? rows6[at - n7] : rows5[at - n7 - n6];
        const int rA = __ldg(A.rp + i), degA = __ldg(A.rp + i + 1) - rA;
        // a warp's entries are warp, warp + NWARP, ...; its lanes fetch 32 of them at a time
        for (int t0 = warp; t0 < degA; t0 += 32 * NWARP) {
            const int t = t0 + NWARP * lane;
            int b0 = 0, b1 = 0;
            V av = V(0);
            if (t < degA) {
                const int k = __ldg(A.ci + rA + t);
                b0 = __ldg(B.rp + k);
                b1 = __ldg(B.rp + k + 1);
                if (NUMERIC) av = aval[rA + t];
            }
            const int left = (degA - t0 + NWARP - 1) / NWARP;
            for (int j = 0; j < min(32, left); ++j) {
                const int e0 = __shfl_sync(0xffffffffu, b0, j), e1 = __shfl_sync(0xffffffffu, b1, j);
                const V a = __shfl_sync(0xffffffffu, av, j);
                for (int e = e0 + lane; e < e1; e += 128) {
                    int c[4];
                    V v[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) c[u] = e + 32 * u < e1 ? __ldg(B.ci + e + 32 * u) : -1;
                    if (NUMERIC) {
#pragma unroll
                        for (int u = 0; u < 4; ++u) v[u] = c[u] >= 0 ? __ldg(bval + e + 32 * u) : V(0);
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        if (static_cast<unsigned>(c[u]) >= static_cast<unsigned>(ncols)) continue;  // none, or not a column
                        const unsigned bit = 1u << (c[u] & 31);
                        if (!(bits[c[u] >> 5] & bit)) atomicOr(bits + (c[u] >> 5), bit);
                        if (NUMERIC) atomic_vadd<V>(acc + c[u], vmul<V>(a, v[u]));
                    }
                }
            }
        }
        __syncthreads();
        // presence bits -> each word's first rank
        const int per = (nw + kDenseBlock - 1) / kDenseBlock;
        int local = 0;
        for (int x = 0; x < per; ++x) {
            const int w = tid * per + x;
            if (w < nw) local += __popc(bits[w]);
        }
        int tot;
        int run = block_exclusive_scan<kDenseBlock>(local, tot, scan_tmp);
        if (!NUMERIC) {
            if (tid == 0) cnt[i] = tot;
        } else {
            for (int x = 0; x < per; ++x) {
                const int w = tid * per + x;
                if (w < nw) {
                    wpre[w] = run;
                    run += __popc(bits[w]);
                }
            }
            __syncthreads();
            const int c0 = crp[i];
            for (int c = tid; c < ncols; c += kDenseBlock) {
                const unsigned word = bits[c >> 5], below = (1u << (c & 31)) - 1u;
                if (word & (below + 1u)) {
                    const int at_c = c0 + wpre[c >> 5] + __popc(word & below);
                    __stcs(cci + at_c, c);
                    st_stream(cval + at_c, acc[c]);
                    acc[c] = V(0);
                }
            }
            __syncthreads();
        }
        for (int w = tid; w < nw; w += kDenseBlock) bits[w] = 0u;
    }
}

// ---------------------------------------------------------------- host side
struct SgPlan {
    long long *ub;
    int *bin_rows;
    long long *tbl_off;
    int *cnt;
    void *scan_tmp;
    int *gkeys;
    void *gvals;
    SgInfo *info;
    unsigned char *row_bin;
    bool dense;  // rows past the shared-table tier go to the dense tier
    SgInfo h;
};

apspie_status check_pair(apspie_ctx *ctx, const apspie_csr *A, const apspie_csr *B, const char *who) {
    apspie_status st = check_csr_view(ctx, A, who);
    if (st != APSPIE_OK) return st;
    if ((st = check_csr_view(ctx, B, who)) != APSPIE_OK) return st;
    if (A->n != B->m) return set_error(ctx, APSPIE_ERR_INVALID_ARG, std::string(who) + ": A.n != B.m");
    if (A->val_type != B->val_type)
        return set_error(ctx, APSPIE_ERR_INVALID_ARG, std::string(who) + ": A and B value types differ");
    if (ctx->validate) {
        if ((st = validate_csr(ctx, A, false)) != APSPIE_OK) return st;
        if ((st = validate_csr(ctx, B, false)) != APSPIE_OK) return st;
    }
    return APSPIE_OK;
}

// Runs rowinfo and sizes every buffer; leaves plan.h filled (synchronises once).
apspie_status sg_plan(apspie_ctx *ctx, const apspie_csr *A, const apspie_csr *B, SgPlan &p) {
    const int m = A->m;
    const size_t mi = static_cast<size_t>(m) + 1;
    const size_t base_need =
        Carver::need({mi * 8, static_cast<size_t>(kBins) * mi * 4, mi * 8, mi * 4,
                      scan_scratch_bytes(m) + 64, sizeof(SgInfo), mi});
    void *base;
    apspie_status st = scratch_reserve(ctx, base_need, &base);
    if (st != APSPIE_OK) return st;
    Carver c(base);
    p.ub = c.take<long long>(mi);
    p.bin_rows = c.take<int>(static_cast<size_t>(kBins) * mi);
    p.tbl_off = c.take<long long>(mi);
    p.cnt = c.take<int>(mi);
    p.scan_tmp = c.take<char>(scan_scratch_bytes(m) + 64);
    p.info = c.take<SgInfo>(1);
    p.row_bin = c.take<unsigned char>(mi);
    cudaError_t e = cudaMemsetAsync(p.info, 0, sizeof(SgInfo), ctx->stream);
    if (e != cudaSuccess) return cuda_error(ctx, e, "spgemm info reset");
    Mat a{A->row_ptr, A->col_ind, A->val}, b{B->row_ptr, B->col_ind, B->val};
    p.dense = takes_dense(A, B);
    if (m > 0) {
        const int blocks = std::min<long long>((static_cast<long long>(m) * 8 + 255) / 256, ctx->num_sms * 16LL);
        const apspie_tune_params tp = effective_params(ctx, APSPIE_TUNE_SPGEMM, A);
        const int reg_max = B->n <= (1 << 24) ? tp.spgemm_reg_max : 0;
        sg_rowinfo<<<blocks, 256, 0, ctx->stream>>>(m, a, b, B->n, reg_max, tp.spgemm_block_max, p.dense ? 1 : 0,
                                                    p.ub, p.row_bin, p.info, p.tbl_off);
        const int lblocks = std::min<long long>((static_cast<long long>(m) + 255) / 256, ctx->num_sms * 8LL);
        sg_binlists<<<lblocks, 256, 0, ctx->stream>>>(m, p.row_bin, p.bin_rows, p.info);
        if ((e = cudaGetLastError()) != cudaSuccess) return cuda_error(ctx, e, "spgemm rowinfo");
    }
    // into pinned memory (a copy to pageable memory is waited for by itself)
    static_assert(sizeof(SgInfo) <= kPinnedBytes, "room");
    e = cudaMemcpyAsync(ctx->h_word, p.info, sizeof(SgInfo), cudaMemcpyDeviceToHost, ctx->stream);
    if (e != cudaSuccess) return cuda_error(ctx, e, "spgemm info copy");
    if ((e = cudaStreamSynchronize(ctx->stream)) != cudaSuccess) return cuda_error(ctx, e, "spgemm sync");
    std::memcpy(&p.h, ctx->h_word, sizeof(SgInfo));
    // global-tier hash tables live in the context's secondary arena
    const size_t gslots = static_cast<size_t>(p.h.global_slots);
    p.gkeys = nullptr;
    p.gvals = nullptr;
    if (gslots > 0) {
        void *tb;
        st = scratch2_reserve(ctx, Carver::need({gslots * 4, gslots * 4}), &tb);
        if (st != APSPIE_OK) return st;
        Carver c2(tb);
        p.gkeys = c2.take<int>(gslots);
        p.gvals = c2.take<char>(gslots * 4);
    }
    return APSPIE_OK;
}

template <bool NUMERIC, typename V>
apspie_status sg_run(apspie_ctx *ctx, const apspie_csr *A, const apspie_csr *B, SgPlan &p, const int *crp,
                     int *cci, V *cval) {
    const int m = A->m;
    Mat a{A->row_ptr, A->col_ind, A->val}, b{B->row_ptr, B->col_ind, B->val};
    const long long mi = static_cast<long long>(m) + 1;
    const int grid_cap = ctx->num_sms * 8;
    (void)mi;
    // per-bin lists are laid out with stride m (sg_rowinfo)
    auto rows = [&](int bin) { return p.bin_rows + static_cast<long long>(bin) * m; };
    const int reg_cap = ctx->num_sms * 16;
    auto reg_grid = [&](int n, int rows_per_warp) {
        const int per_block = rows_per_warp * kSgBlock / 32;
        return std::min((n + per_block - 1) / per_block, reg_cap);
    };
    int nb = p.h.bin_count[1];
    if (nb > 0)
        sg_reg<8, 4, NUMERIC, V><<<reg_grid(nb, 4), kSgBlock, 0, ctx->stream>>>(rows(1), nb, a, b, p.cnt, crp, cci, cval);
    nb = p.h.bin_count[2];
    if (nb > 0)
        sg_reg<8, 8, NUMERIC, V><<<reg_grid(nb, 4), kSgBlock, 0, ctx->stream>>>(rows(2), nb, a, b, p.cnt, crp, cci, cval);
    nb = p.h.bin_count[3];
    if (nb > 0)
        sg_reg<16, 8, NUMERIC, V><<<reg_grid(nb, 2), kSgBlock, 0, ctx->stream>>>(rows(3), nb, a, b, p.cnt, crp, cci, cval);
    nb = p.h.bin_count[kBinBlock];
    if (nb > 0) {
        const int g = std::min(nb, grid_cap);
        sg_block<false, NUMERIC, V><<<g, kSgBlock, 0, ctx->stream>>>(rows(kBinBlock), nb, a, b, B->n, p.ub, p.tbl_off,
                                                                      p.gkeys, static_cast<V *>(p.gvals), p.cnt,
                                                                      crp, cci, cval, p.info);
    }
    nb = p.h.bin_count[kBinGlobal];
    const int nd = p.dense ? p.h.bin_count[5] + p.h.bin_count[6] + p.h.bin_count[7] : 0;
    if (nd > 0) {
        const void *fn = reinterpret_cast<const void *>(sg_dense<NUMERIC, V>);
        const size_t smem = dense_smem<NUMERIC, V>(B->n);
        int per_sm = 0;
        // the limit belongs to the kernel on the device, not to this call: always the most it can
        // ask for, so that contexts of other threads that launch it with another size agree on it
        cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(dense_smem<NUMERIC, V>(kDenseCols)));
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kDenseBlock, smem);
        if (e == cudaSuccess) e = cudaMemsetAsync(&p.info->ticket, 0, sizeof(int), ctx->stream);
        if (e != cudaSuccess) return cuda_error(ctx, e, "spgemm dense tier");
        sg_dense<NUMERIC, V><<<std::min(nd, std::max(per_sm, 1) * ctx->num_sms), kDenseBlock, smem, ctx->stream>>>(
            rows(7), p.h.bin_count[7], rows(6), p.h.bin_count[6], rows(5), p.h.bin_count[5], a, b, B->n, p.cnt, crp, cci,
            cval, &p.info->ticket);
    } else if (nb > 0) {
        const int g = std::min(nb, grid_cap);
        sg_block<true, NUMERIC, V><<<g, kSgBlock, 0, ctx->stream>>>(rows(kBinGlobal), nb, a, b, B->n, p.ub, p.tbl_off,
                                                                     p.gkeys, static_cast<V *>(p.gvals), p.cnt,
                                                                     crp, cci, cval, p.info);
    }
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? APSPIE_OK : cuda_error(ctx, e, "spgemm launch");
}

__global__ void zero_empty_rows(const int *rows, int n, int *cnt) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) cnt[rows[k]] = 0;
}

apspie_status sg_symbolic(apspie_ctx *ctx, const apspie_csr *A, const apspie_csr *B, SgPlan &p, int *crp,
                          long long *nnz) {
    apspie_status st;
    const int m = A->m;
    if (p.h.bin_count[0] > 0) {
        const int n0 = p.h.bin_count[0];
        zero_empty_rows<<<std::min((n0 + 255) / 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(p.bin_rows, n0, p.cnt);
    }
    if (A->val_type == APSPIE_VAL_F32)
        st = sg_run<false, float>(ctx, A, B, p, nullptr, nullptr, nullptr);
    else
        st = sg_run<false, int>(ctx, A, B, p, nullptr, nullptr, nullptr);
    if (st != APSPIE_OK) return st;
    if ((st = device_exclusive_scan(ctx, p.cnt, m, crp, p.scan_tmp, &p.info->overflow)) != APSPIE_OK) return st;
    cudaError_t e = cudaMemcpyAsync(ctx->h_word, crp + m, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(ctx->h_word + 1, &p.info->overflow, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_error(ctx, e, "spgemm symbolic sync");
    p.h.overflow = ctx->h_word[1];
    if (p.h.overflow) return set_error(ctx, APSPIE_ERR_HASH_OVERFLOW, "spgemm: hash table or nnz(C) overflow");
    *nnz = ctx->h_word[0];
    return APSPIE_OK;
}

apspie_status sg_numeric(apspie_ctx *ctx, const apspie_csr *A, const apspie_csr *B, SgPlan &p, const int *crp,
                         int *cci, void *cval) {
    apspie_status st;
    if (A->val_type == APSPIE_VAL_I32)
        st = sg_run<true, int>(ctx, A, B, p, crp, cci, static_cast<int *>(cval));
    else if (A->val_type == APSPIE_VAL_F32)
        st = sg_run<true, float>(ctx, A, B, p, crp, cci, static_cast<float *>(cval));
    else {
        // pattern only: reuse the int path with products of 1s written to a scratch sink
        return set_error(ctx, APSPIE_ERR_UNSUPPORTED, "spgemm numeric needs values (use symbolic for patterns)");
    }
    return st;
}

bool same_view(const apspie_csr &x, const apspie_csr *y) {
    return x.m == y->m && x.n == y->n && x.nnz == y->nnz && x.val_type == y->val_type &&
           x.row_ptr == y->row_ptr && x.col_ind == y->col_ind && x.val == y->val;
}

// The validation pass (ctx->validate) reserves no scratch, so it leaves the epoch alone.
void sg_cache_store(apspie_ctx *ctx, const apspie_csr *A, const apspie_csr *B, const SgPlan &p) {
    apspie_spgemm_plan_cache &c = ctx->sg_cache;
    c.a = *A;
    c.b = *B;
    c.dev[0] = p.ub;
    c.dev[1] = p.bin_rows;
    c.dev[2] = p.tbl_off;
    c.dev[3] = p.cnt;
    c.dev[4] = p.scan_tmp;
    c.dev[5] = p.gkeys;
    c.dev[6] = p.gvals;
    c.dev[7] = p.info;
    static_assert(kBins <= 8, "cache layout");
    for (int b = 0; b < kBins; ++b) c.host[b] = p.h.bin_count[b];
    c.host[8] = p.h.global_slots;
    c.host[9] = reinterpret_cast<long long>(p.row_bin);
    c.epoch = ctx->scratch_epoch;
    c.valid = true;
}

bool sg_cache_load(apspie_ctx *ctx, const apspie_csr *A, const apspie_csr *B, SgPlan &p) {
    const apspie_spgemm_plan_cache &c = ctx->sg_cache;
    if (!c.valid || c.epoch != ctx->scratch_epoch || !same_view(c.a, A) || !same_view(c.b, B)) return false;
    p.ub = static_cast<long long *>(c.dev[0]);
    p.bin_rows = static_cast<int *>(c.dev[1]);
    p.tbl_off = static_cast<long long *>(c.dev[2]);
    p.cnt = static_cast<int *>(c.dev[3]);
    p.scan_tmp = c.dev[4];
    p.gkeys = static_cast<int *>(c.dev[5]);
    p.gvals = c.dev[6];
    p.info = static_cast<SgInfo *>(c.dev[7]);
    std::memset(&p.h, 0, sizeof(p.h));
    for (int b = 0; b < kBins; ++b) p.h.bin_count[b] = static_cast<int>(c.host[b]);
    p.h.global_slots = c.host[8];
    p.row_bin = reinterpret_cast<unsigned char *>(c.host[9]);
    p.dense = takes_dense(A, B);
    return true;
}

}  // namespace
}  // namespace apspie

using namespace apspie;

extern "C" {

apspie_status apspie_spgemm_symbolic(apspie_ctx *ctx, const apspie_csr *A, const apspie_csr *B,
                                     int32_t *d_row_ptr_c, int64_t *nnz_c) {
    if (!ctx || !d_row_ptr_c || !nnz_c) return APSPIE_ERR_INVALID_ARG;
    cudaSetDevice(ctx->device);
    ctx->sg_cache.valid = false;
    apspie_status st = check_pair(ctx, A, B, "apspie_spgemm_symbolic");
    if (st != APSPIE_OK) return st;
    SgPlan p;
    if ((st = sg_plan(ctx, A, B, p)) != APSPIE_OK) return st;
    long long nnz = 0;
    if ((st = sg_symbolic(ctx, A, B, p, d_row_ptr_c, &nnz)) != APSPIE_OK) return st;
    *nnz_c = nnz;
    sg_cache_store(ctx, A, B, p);
    return APSPIE_OK;
}

apspie_status apspie_spgemm_numeric(apspie_ctx *ctx, const apspie_csr *A, const apspie_csr *B,
                                    const int32_t *d_row_ptr_c, int32_t *d_col_c, void *d_val_c) {
    if (!ctx || !d_row_ptr_c) return APSPIE_ERR_INVALID_ARG;
    cudaSetDevice(ctx->device);
    apspie_status st = check_pair(ctx, A, B, "apspie_spgemm_numeric");
    if (st != APSPIE_OK) return st;
    SgPlan p;
    if (!sg_cache_load(ctx, A, B, p) && (st = sg_plan(ctx, A, B, p)) != APSPIE_OK) return st;
    return sg_numeric(ctx, A, B, p, d_row_ptr_c, d_col_c, d_val_c);
}

apspie_status apspie_spgemm(apspie_ctx *ctx, const apspie_csr *A, const apspie_csr *B, apspie_csr_owned *C) {
    if (!ctx || !C) return APSPIE_ERR_INVALID_ARG;
    cudaSetDevice(ctx->device);
    std::memset(C, 0, sizeof(*C));
    apspie_status st = check_pair(ctx, A, B, "apspie_spgemm");
    if (st != APSPIE_OK) return st;
    if (A->val_type == APSPIE_VAL_NONE)
        return set_error(ctx, APSPIE_ERR_UNSUPPORTED, "apspie_spgemm: values required (F32 or I32)");
    SgPlan p;
    if ((st = sg_plan(ctx, A, B, p)) != APSPIE_OK) return st;
    int32_t *rp = nullptr;
    cudaError_t e = owned_alloc(reinterpret_cast<void **>(&rp), (static_cast<size_t>(A->m) + 1) * sizeof(int32_t));
    if (e != cudaSuccess) return cuda_error(ctx, e, "apspie_spgemm row_ptr");
    long long nnz = 0;
    if ((st = sg_symbolic(ctx, A, B, p, rp, &nnz)) != APSPIE_OK) {
        owned_free(rp);
        return st;
    }
    int32_t *ci = nullptr;
    void *val = nullptr;
    const size_t n = static_cast<size_t>(nnz > 0 ? nnz : 1);
    if ((e = owned_alloc(reinterpret_cast<void **>(&ci), n * sizeof(int32_t))) != cudaSuccess ||
        (e = owned_alloc(reinterpret_cast<void **>(&val), n * 4)) != cudaSuccess) {
        owned_free(rp);
        if (ci) owned_free(ci);
        return cuda_error(ctx, e, "apspie_spgemm C");
    }
    if ((st = sg_numeric(ctx, A, B, p, rp, ci, val)) != APSPIE_OK) {
        owned_free(rp);
        owned_free(ci);
        owned_free(val);
        return st;
    }
    C->m = A->m;
    C->n = B->n;
    C->nnz = static_cast<int32_t>(nnz);
    C->val_type = A->val_type;
    C->row_ptr = rp;
    C->col_ind = ci;
    C->val = val;
    return APSPIE_OK;
}

void apspie_csr_free(apspie_csr_owned *C) {
    if (!C) return;
    if (C->row_ptr) owned_free(C->row_ptr);
    if (C->col_ind) owned_free(C->col_ind);
    if (C->val) owned_free(C->val);
    std::memset(C, 0, sizeof(*C));
}

}  // extern "C"
