// Stable LSD radix sort of (32- or 64-bit key, 32-bit value) pairs on the device, shared by
// the graph construction (build.cu), the transpose and the sparse-vector product
// (spmspv.cu). One read of the keys counts every pass's digits; a pass then reads and
// writes each pair once: its tiles are taken in order from a ticket, each ranks its keys in
// input order with warp match masks, publishes its digit counts, adds up the counts of the
// tiles before it (decoupled look-back: Merrill and Garland, "Single-pass Parallel Prefix Scan
// with Decoupled Look-back", 2016), reorders the tile by digit in shared memory and
// writes every digit's run with consecutive threads.
//
// Measured over 16.8M pairs of 12 bytes (0.40 GB, 61 us at the copy rate): 138 us a pass;
// a digit count per pass, three scan launches and a scatter straight from registers (a
// 32-byte sector written per pair), as it was before, took 277 us. What bounds a pass now is
// the tile's chain of phases (loads, ranking, block scan, look-back, writes) with two tiles
// on an SM: 42 % of the issue slots and 29 % of the HBM rate are used. Tried: match.any
// instead of eight ballots (160 us), shared-memory OR masks (150 us), 256 threads a tile
// (150 us), 1,024 (169 us), 9 / 16 pairs a thread (149 / 198 us), look-back of 1 / 4 / 8 /
// 16 words a step (141 / 136 / 151 / 174 us; the words' own traffic).
#pragma once

#include "common.cuh"

namespace apspie {
namespace {

constexpr int kRsBlock = 512;
constexpr int kRsWarps = kRsBlock / 32;
constexpr int kRsDigits = 256;   // at most 8 bits a pass; thread t of a block owns digit t
constexpr int kRsMaxPasses = 8;  // 64-bit keys
// Pairs per thread and pass: the longer a tile, the longer the runs that it writes per digit
// and the fewer look-backs; two tiles (74 KB of pairs, 16 KB of digit counts) fit on an SM.
template <class K>
constexpr int kRsItems = sizeof(K) == 8 ? 12 : 16;
template <class K>
constexpr int kRsTile = kRsBlock * kRsItems<K>;

// The digits of a sort on key bits [lo, hi): as few passes as 8-bit digits allow, of
// (nearly) equal width, so that no pass scatters into more runs than it needs to.
struct RsPlan {
    int passes;
    int shift[kRsMaxPasses];
    int bits[kRsMaxPasses];
};

RsPlan rs_plan(int lo, int hi) {
    RsPlan p;
    const int bits = hi > lo ? hi - lo : 0;
    p.passes = (bits + 7) / 8;
    int at = lo;
    for (int i = 0; i < p.passes; ++i) {
        const int w = (hi - at + (p.passes - i) - 1) / (p.passes - i);
        p.shift[i] = at;
        p.bits[i] = w;
        at += w;
    }
    for (int i = p.passes; i < kRsMaxPasses; ++i) p.shift[i] = p.bits[i] = 0;
    return p;
}

// Adds one key's digits to a block's counts h[pass * kRsDigits + digit].
template <class K>
__device__ __forceinline__ void rs_count(int *h, K key, const RsPlan &pl) {
#pragma unroll
    for (int p = 0; p < kRsMaxPasses; ++p)
        if (p < pl.passes)
            atomicAdd(h + p * kRsDigits + (static_cast<int>(key >> pl.shift[p]) & ((1 << pl.bits[p]) - 1)), 1);
}

__device__ __forceinline__ void rs_count_begin(int *h, const RsPlan &pl) {
    for (int i = threadIdx.x; i < pl.passes * kRsDigits; i += blockDim.x) h[i] = 0;
    __syncthreads();
}

__device__ __forceinline__ void rs_count_end(const int *h, const RsPlan &pl, int *ghist) {
    __syncthreads();
    for (int i = threadIdx.x; i < pl.passes * kRsDigits; i += blockDim.x)
        if (h[i]) atomicAdd(ghist + i, h[i]);
}

template <class K>
__global__ void __launch_bounds__(kRsBlock) rs_histograms(const K *__restrict__ keys, long long n, RsPlan pl,
                                                          int *ghist) {
    __shared__ int h[kRsMaxPasses * kRsDigits];
    rs_count_begin(h, pl);
    const long long stride = static_cast<long long>(gridDim.x) * kRsBlock;
    for (long long i = blockIdx.x * static_cast<long long>(kRsBlock) + threadIdx.x; i < n; i += 4 * stride) {
        K k[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) k[j] = i + j * stride < n ? __ldg(keys + i + j * stride) : K(0);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (i + j * stride < n) rs_count(h, k[j], pl);
    }
    rs_count_end(h, pl, ghist);
}

// Each pass's digit counts -> where the digit's pairs begin (one block per pass).
__global__ void __launch_bounds__(kRsDigits) rs_bases(int *ghist) {
    __shared__ int tmp[33];
    int *h = ghist + blockIdx.x * kRsDigits;
    int tot;
    h[threadIdx.x] = block_exclusive_scan<kRsDigits>(h[threadIdx.x], tot, tmp);
}

// A tile's published word: the pass and what the count covers (the tile alone, or it and all
// tiles before it) above 40 bits of count. The words of one pass never pass for those of
// another, so they are cleared once per sort.
__device__ __forceinline__ unsigned long long look_word(int pass, bool all, long long count) {
    return (static_cast<unsigned long long>(2 * pass + (all ? 2 : 1)) << 40) | static_cast<unsigned long long>(count);
}

__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_relaxed_u64(unsigned long long *p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Sum of the counts of the tiles before `tile`, from the words status[t * stride + column]
// (t < tile): walks back over single-tile counts to the nearest running total, kLookAhead
// words a step, read together. Tiles are taken in order, so every earlier tile is running or done;
// the wait is bounded all the same (kBarrierTimeoutNs): it then reports APSPIE_ERR_TIMEOUT
// in *err, which also ends the other tiles' waits, and returns -1.
constexpr int kLookAhead = 2;
__device__ __forceinline__ long long look_back(const unsigned long long *status, int tile, int stride, int column,
                                               int pass, int *err) {
    const unsigned part = 2u * pass + 1u, all = 2u * pass + 2u;
    long long sum = 0;
    unsigned long long t0 = 0;
    unsigned spin = 0;
    for (int t = tile - 1; t >= 0;) {
        unsigned long long w[kLookAhead];
#pragma unroll
        for (int j = 0; j < kLookAhead; ++j)
            w[j] = t - j >= 0 ? ld_relaxed_u64(status + static_cast<long long>(t - j) * stride + column) : 0ull;
        int used = 0;
        bool done = false;
#pragma unroll
        for (int j = 0; j < kLookAhead; ++j) {
            const unsigned tag = static_cast<unsigned>(w[j] >> 40);
            if (!done && used == j && (tag == part || tag == all)) {
                sum += static_cast<long long>(w[j] & ((1ull << 40) - 1ull));
                ++used;
                done = tag == all;
            }
        }
        if (done) break;
        t -= used;
        if (used == 0 && (++spin & 255u) == 0u) {
            if (ld_volatile_i32(err) != 0) return -1;
            const unsigned long long now = globaltimer_ns();
            if (t0 == 0) {
                t0 = now;
            } else if (now - t0 > kBarrierTimeoutNs) {
                atomicExch(err, APSPIE_ERR_TIMEOUT);
                return -1;
            }
        }
    }
    return sum;
}

// The same by a whole warp over words status[t], 32 a step (for passes with one word a tile,
// where a thread's walk would be the longest chain of the tile). All lanes get the sum.
__device__ __forceinline__ long long look_back_warp(const unsigned long long *status, int tile, int pass, int *err) {
    const unsigned part = 2u * pass + 1u, all = 2u * pass + 2u;
    const int lane = threadIdx.x & 31;
    long long sum = 0;
    unsigned long long t0 = 0;
    for (int t = tile - 1; t >= 0; t -= 32) {
        unsigned long long w = 0;
        for (unsigned spin = 1;; ++spin) {
            w = t - lane >= 0 ? ld_relaxed_u64(status + t - lane) : static_cast<unsigned long long>(all) << 40;
            const unsigned tag = static_cast<unsigned>(w >> 40);
            const unsigned ready = __ballot_sync(0xffffffffu, tag == part || tag == all);
            const unsigned total = __ballot_sync(0xffffffffu, tag == all);
            // the words up to the nearest running total (all 32 without one) have to be there
            const unsigned need = total ? ((total & (0u - total)) << 1) - 1u : 0xffffffffu;
            if ((ready & need) == need) {
                long long v = ((need >> lane) & 1u) ? static_cast<long long>(w & ((1ull << 40) - 1ull)) : 0;
#pragma unroll
                for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                sum += v;
                if (total) return sum;
                break;
            }
            if ((spin & 255u) == 0u) {
                int bad = 0;
                if (lane == 0) {
                    const unsigned long long now = globaltimer_ns();
                    bad = ld_volatile_i32(err) != 0;
                    if (t0 == 0) {
                        t0 = now;
                    } else if (!bad && now - t0 > kBarrierTimeoutNs) {
                        atomicExch(err, APSPIE_ERR_TIMEOUT);
                        bad = 1;
                    }
                }
                if (__shfl_sync(0xffffffffu, bad, 0)) return -1;
            }
        }
    }
    return sum;
}

template <class K>
struct RsSmem {
    K keys[kRsTile<K>];
    unsigned vals[kRsTile<K>];
    int wh[kRsWarps][kRsDigits];  // per warp: pairs per digit, then where they begin in the tile
    int goff[kRsDigits];          // where the digit's run goes, minus where it begins in the tile
    int scan_tmp[33];
    int tile;
    int ok;
};

template <class K>
__global__ void __launch_bounds__(kRsBlock, 2) rs_pass(const K *__restrict__ kin, const unsigned *__restrict__ vin,
                                                       K *kout, unsigned *vout, long long n, int pass, int shift,
                                                       int bits, const int *__restrict__ base,
                                                       unsigned long long *status, int *ticket, int *err) {
    constexpr int ITEMS = kRsItems<K>;
    constexpr int TILE = kRsTile<K>;
    extern __shared__ __align__(16) unsigned char rs_smem[];
    RsSmem<K> &sm = *reinterpret_cast<RsSmem<K> *>(rs_smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned dmask = (1u << bits) - 1u;
    if (tid == 0) {
        sm.tile = atomicAdd(ticket, 1);
        sm.ok = ld_volatile_i32(err) == 0;
    }
    for (int i = tid; i < kRsWarps * kRsDigits; i += kRsBlock) (&sm.wh[0][0])[i] = 0;
    __syncthreads();
    if (!sm.ok) return;  // an earlier pass gave up: its output is not a permutation of its input
    const int tile = sm.tile;
    const long long t0 = static_cast<long long>(tile) * TILE;
    const int cnt = static_cast<int>(n - t0 < TILE ? n - t0 : TILE);
    // a warp's pairs are consecutive, 32 a step, so input order is (warp, step, lane);
    // what is past the end takes the largest digit and so stays behind the last pair
    K key[ITEMS];
    unsigned val[ITEMS];
    const int w0 = warp * 32 * ITEMS + lane;
    const K *kt = kin + t0 + w0;
    const unsigned *vt = vin + t0 + w0;
    if (cnt == TILE) {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) key[i] = __ldcs(kt + 32 * i);
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) val[i] = __ldcs(vt + 32 * i);
    } else {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) key[i] = w0 + 32 * i < cnt ? __ldcs(kt + 32 * i) : ~K(0);
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) val[i] = w0 + 32 * i < cnt ? __ldcs(vt + 32 * i) : 0u;
    }
    unsigned place[ITEMS];  // digit << 16 | pairs of that digit before it in the warp
    const unsigned before = (1u << lane) - 1u;
    int *wh = sm.wh[warp];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const unsigned d = static_cast<unsigned>(key[i] >> shift) & dmask;
        unsigned peers = 0xffffffffu;  // lanes with the same digit
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const bool one = (d >> b) & 1u;
            const unsigned m = __ballot_sync(0xffffffffu, one);
            peers &= one ? m : ~m;
        }
        const int old = wh[d];
        __syncwarp();
        const unsigned r = __popc(peers & before);
        if (r == 0) wh[d] = old + __popc(peers);
        __syncwarp();
        place[i] = d << 16 | (old + r);
    }
    __syncthreads();
    int c = 0;
    unsigned long long *mine = status + static_cast<long long>(tile) * kRsDigits + tid;
    if (tid < kRsDigits) {
#pragma unroll
        for (int w = 0; w < kRsWarps; ++w) {
            const int t = sm.wh[w][tid];
            sm.wh[w][tid] = c;
            c += t;
        }
        st_relaxed_u64(mine, look_word(pass, tile == 0, c));
    }
    int tot;
    const int ex = block_exclusive_scan<kRsBlock>(c, tot, sm.scan_tmp);
    if (tid < kRsDigits) {
#pragma unroll
        for (int w = 0; w < kRsWarps; ++w) sm.wh[w][tid] += ex;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const int p = wh[place[i] >> 16] + (place[i] & 0xffffu);
        sm.keys[p] = key[i];
        sm.vals[p] = val[i];
    }
    if (tid < kRsDigits) {
        long long prev = 0;
        if (tile > 0) {
            prev = look_back(status, tile, kRsDigits, tid, pass, err);
            if (prev >= 0)
                st_relaxed_u64(mine, look_word(pass, true, prev + c));
            else
                sm.ok = 0;
        }
        sm.goff[tid] = base[tid] + static_cast<int>(prev) - ex;
    }
    __syncthreads();
    if (!sm.ok) return;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const int p = i * kRsBlock + tid;
        if (cnt == TILE || p < cnt) {
            const K k = sm.keys[p];
            const int g = sm.goff[static_cast<unsigned>(k >> shift) & dmask] + p;
            kout[g] = k;
            vout[g] = sm.vals[p];
        }
    }
}

// Buffers of up to kRsSorts sorts of at most n pairs, one after the other. The state area is
// cleared once, by sort_begin: err, the tickets, the digit counts of every sort's passes, the
// published words. Look-back number t (tickets and tags) is pass p of sort i for
// t = i * kRsMaxPasses + p; callers' own look-backs take numbers from kRsOwn on.
constexpr int kRsSorts = 2;
constexpr int kRsOwn = kRsSorts * kRsMaxPasses;
constexpr int kRsHistBytes = kRsSorts * kRsMaxPasses * kRsDigits * static_cast<int>(sizeof(int));
template <class K>
struct SortBufs {
    K *k[2];
    unsigned *v[2];
    int *err;     // first word of the state area
    int *ticket;  // [kRsOwn + ...], 48 in all
    int *ghist;   // [kRsSorts][kRsMaxPasses * kRsDigits]
    unsigned long long *status;
    size_t state_bytes;
    int *hist_of(int sort) const { return ghist + sort * kRsMaxPasses * kRsDigits; }
};

template <class K>
size_t sort_state_bytes(long long n) {
    const size_t nb = static_cast<size_t>((n + kRsTile<K> - 1) / kRsTile<K>);
    return 256 + kRsHistBytes + (nb > 0 ? nb : 1) * kRsDigits * sizeof(unsigned long long);
}

template <class K>
size_t sort_need(long long n) {
    const size_t c = static_cast<size_t>(n > 0 ? n : 1);
    return Carver::need({c * sizeof(K), c * sizeof(K), c * 4, c * 4, sort_state_bytes<K>(n)});
}

template <class K>
SortBufs<K> carve_sort(Carver &c, long long n) {
    SortBufs<K> s;
    s.k[0] = c.take<K>(n > 0 ? n : 1);
    s.k[1] = c.take<K>(n > 0 ? n : 1);
    s.v[0] = c.take<unsigned>(n > 0 ? n : 1);
    s.v[1] = c.take<unsigned>(n > 0 ? n : 1);
    s.state_bytes = sort_state_bytes<K>(n);
    char *state = c.take<char>(s.state_bytes);
    s.err = reinterpret_cast<int *>(state);
    s.ticket = s.err + 16;
    s.ghist = reinterpret_cast<int *>(state + 256);
    s.status = reinterpret_cast<unsigned long long *>(state + 256 + kRsHistBytes);
    return s;
}

template <class K>
apspie_status sort_begin(apspie_ctx *ctx, const SortBufs<K> &s) {
    cudaError_t e = cudaMemsetAsync(s.err, 0, s.state_bytes, ctx->stream);
    return e == cudaSuccess ? APSPIE_OK : cuda_error(ctx, e, "radix sort reset");
}

// The passes of sort number `sort`, whose digits are counted in s.hist_of(sort) (by
// rs_histograms, or by the kernel that made the keys): reads (kin, vin), which may be
// buffers of the caller's, writes pair `to` of s first and then the two pairs in turn, and
// returns the pair that holds the result. With nothing to do (no pairs, no bits) nothing is
// written and *which is to ^ 1.
template <class K>
apspie_status radix_passes(apspie_ctx *ctx, const SortBufs<K> &s, int sort, const RsPlan &pl, const K *kin,
                           const unsigned *vin, long long n, int to, int *which) {
    *which = to ^ 1;
    if (n <= 0 || pl.passes == 0) return APSPIE_OK;
    const int nb = static_cast<int>((n + kRsTile<K> - 1) / kRsTile<K>);
    // more than 48 KB of shared memory has to be asked for (per device: not kept)
    cudaError_t e = cudaFuncSetAttribute(rs_pass<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(sizeof(RsSmem<K>)));
    if (e != cudaSuccess) return cuda_error(ctx, e, "radix sort");
    rs_bases<<<pl.passes, kRsDigits, 0, ctx->stream>>>(s.hist_of(sort));
    for (int p = 0; p < pl.passes; ++p) {
        const int t = sort * kRsMaxPasses + p;
        rs_pass<K><<<nb, kRsBlock, sizeof(RsSmem<K>), ctx->stream>>>(kin, vin, s.k[to], s.v[to], n, t, pl.shift[p], pl.bits[p],
                                                     s.hist_of(sort) + p * kRsDigits, s.status, s.ticket + t, s.err);
        kin = s.k[to];
        vin = s.v[to];
        *which = to;
        to ^= 1;
    }
    e = cudaGetLastError();
    return e == cudaSuccess ? APSPIE_OK : cuda_error(ctx, e, "radix sort");
}

// A whole sort (number 0) of (kin, vin) into s.
template <class K>
apspie_status radix_sort(apspie_ctx *ctx, const SortBufs<K> &s, const RsPlan &pl, const K *kin, const unsigned *vin,
                         long long n, int to, int *which) {
    apspie_status st = sort_begin(ctx, s);
    if (st != APSPIE_OK) return st;
    if (n > 0 && pl.passes > 0) {
        const long long blocks = (n + 8 * kRsBlock - 1) / (8 * kRsBlock);
        rs_histograms<K><<<static_cast<int>(blocks < ctx->num_sms * 8LL ? blocks : ctx->num_sms * 8LL), kRsBlock, 0,
                           ctx->stream>>>(kin, n, pl, s.hist_of(0));
    }
    return radix_passes(ctx, s, 0, pl, kin, vin, n, to, which);
}

int bit_length(long long x) {  // bits needed for values 0 .. x-1 (at least 1)
    int b = 1;
    while ((1LL << b) < x) ++b;
    return b;
}

}  // namespace
}  // namespace apspie
