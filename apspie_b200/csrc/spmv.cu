// Dense-vector SpMV and PageRank: the dense-frontier end of the push/pull spectrum.
//
// The reference multiplies by a dense vector through moderngpu's SpmvCsrBinary
// (src/bfs.cuh:11-14) and a cuSPARSE csrmv wrapper (cuspmv, src/tc.cuh:17-59); it ships
// test_pr.mtx but no PageRank. Here:
//   * apspie_spmv: y = alpha * A * x + beta * y in FP32, a group of G lanes per row (G from
//     the mean row length: 4, 8, 16 or 32), lane-strided partial sums reduced by shuffles
//     (fixed order, so repeated calls give identical bits);
//   * apspie_pagerank: power iteration r' = (1 - d) / n + d * (A^T (r / outdeg) + dangling
//     mass / n) on the transposed graph (pull: no atomics on the ranks), stopping when the L1
//     change is below tol or after max_iter iterations.
#include <algorithm>
#include <cstring>

#include "common.cuh"

namespace apspie {
namespace {

template <int G>
__global__ void spmv_kernel(int m, const int *__restrict__ rp, const int *__restrict__ ci,
                            const float *__restrict__ val, const float *__restrict__ x, float *y, float alpha,
                            float beta) {
    const int lane = threadIdx.x % G;
    const long long grp = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) / G;
    const long long ngrp = static_cast<long long>(gridDim.x) * blockDim.x / G;
    for (long long r0 = grp - grp % (32 / G); r0 < m; r0 += ngrp) {  // a warp's groups move together
        const long long r = r0 + grp % (32 / G);
        float s = 0.0f;
        if (r < m) {
            const int e1 = __ldg(rp + r + 1);
            for (int e = __ldg(rp + r) + lane; e < e1; e += G) {
                const float a = val ? __ldg(val + e) : 1.0f;
                s = __fmaf_rn(a, __ldg(x + __ldg(ci + e)), s);
            }
        }
#pragma unroll
        for (int o = G / 2; o; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, G);
        if (r < m && lane == 0) y[r] = beta == 0.0f ? alpha * s : alpha * s + beta * y[r];
    }
}

apspie_status launch_spmv(apspie_ctx *ctx, const apspie_csr *A, const float *x, float *y, float alpha,
                          float beta) {
    const float *val = A->val_type == APSPIE_VAL_F32 ? static_cast<const float *>(A->val) : nullptr;
    const double mean = A->m > 0 ? static_cast<double>(A->nnz) / A->m : 0.0;
    const int blocks = static_cast<int>(std::max<long long>(
        1, std::min<long long>((static_cast<long long>(A->m) * 32 + 255) / 256, ctx->num_sms * 16LL)));
    if (mean <= 6)
        spmv_kernel<4><<<blocks, 256, 0, ctx->stream>>>(A->m, A->row_ptr, A->col_ind, val, x, y, alpha, beta);
    else if (mean <= 12)
        spmv_kernel<8><<<blocks, 256, 0, ctx->stream>>>(A->m, A->row_ptr, A->col_ind, val, x, y, alpha, beta);
    else if (mean <= 24)
        spmv_kernel<16><<<blocks, 256, 0, ctx->stream>>>(A->m, A->row_ptr, A->col_ind, val, x, y, alpha, beta);
    else
        spmv_kernel<32><<<blocks, 256, 0, ctx->stream>>>(A->m, A->row_ptr, A->col_ind, val, x, y, alpha, beta);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? APSPIE_OK : cuda_error(ctx, e, "spmv launch");
}

// ---- PageRank -----------------------------------------------------------------------
// An iteration is two launches: pr_gather sums x over every row's in-edges, pr_update turns
// the sums into new ranks, their L1 change, the next x and the next dangling mass. Whether
// to stop is decided on the device; the host looks every kPrBatch iterations (launches
// enqueued past the end return at once).
//
// pr_gather cuts the entries, not the rows, into equal chunks: a thread takes 8 consecutive
// entries (two 128-bit loads), sums the pieces of rows in them, and a segmented scan joins
// pieces across threads. A chunk writes the sums of the rows that begin in it; what it holds
// of a row that began earlier goes to carry[], which pr_update adds in chunk order: a row's sum has
// the same bits in repeated calls (the dangling mass and the change are added up by atomics, so the
// ranks' last bits may differ). Bound: 4 bytes an entry from HBM plus one gather from
// L2. Measured, R-MAT of 700,001 vertices and 10.7M entries, per iteration: 16 lanes per
// row 228 us (the row of 55,000 entries is the last to finish) + 34 us for the two vector
// kernels, whose warps all added doubles to one word; now see pr_update.
constexpr int kPrBlock = 256;
constexpr int kPrItems = 8;
constexpr int kPrChunk = kPrBlock * kPrItems;
constexpr int kPrVec = 256;  // threads a block in the vector kernels, four blocks an SM
constexpr int kPrOwn = 2;    // vertices whose data a thread fetches together
constexpr int kPrBatch = 4;

// Sums over the vertices, each in kPrSlots parts, and the word that every block looks at first, all
// in cache lines of their own: blocks that start while others still write to the line of their
// first look wait for it (with everything in one line the gathers of 700,001 vertices and 10.7M
// entries took 683 us in 16 iterations and the updates 187; 1, 2, 4, 8 and 16 parts: 759, 753, 736, 747 and
// 768 us together).
constexpr int kPrSlots = 4;
struct PrState {
    struct {
        double dang[2];  // rank mass of the vertices without out-edges, by iteration parity
        double diff[2];  // L1 change, by iteration parity
        double pad[12];
    } part[kPrSlots];
    int done;  // iterations after which the change was below tol (0: not yet)
    int pad;

    __host__ __device__ double dang(int i) const {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < kPrSlots; ++k) s += part[k].dang[i];
        return s;
    }
    __host__ __device__ double diff(int i) const {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < kPrSlots; ++k) s += part[k].diff[i];
        return s;
    }
};

__device__ __forceinline__ double block_sum(double v, double *tmp) {
    for (int o = 16; o; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) tmp[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < static_cast<int>(blockDim.x) / 32; ++w) s += tmp[w];
    __syncthreads();
    return s;  // thread 0's
}

// heads[b] bit j: entry 8 b + j is the first of its row
__global__ void pr_heads(long long nnz, const unsigned *__restrict__ row, unsigned char *heads) {
    const long long nb = (nnz + 7) / 8;
    for (long long b = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; b < nb;
         b += static_cast<long long>(gridDim.x) * blockDim.x) {
        unsigned m = 0u;
        unsigned prev = b > 0 ? __ldg(row + 8 * b - 1) : 0u;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const long long e = 8 * b + j;
            if (e < nnz) {
                const unsigned r = __ldg(row + e);
                if (e == 0 || r != prev) m |= 1u << j;
                prev = r;
            }
        }
        heads[b] = static_cast<unsigned char>(m);
    }
}

// The same out of row starts (heads is zero), and of the entries' rows what pr_gather reads: those of
// the last entries of rows and chunks. (Written out for every entry and read again for the heads:
// a call that is done after one iteration took 184 us on a complete graph of 4,000 vertices, 142 on
// 100,000 in cliques of 100, 65 on two vertices; now 160, 126 and 52.)
__global__ void pr_marks(int n, long long nnz, const int *__restrict__ rp, unsigned *heads, unsigned *row) {
    const long long first = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    const long long step = static_cast<long long>(gridDim.x) * blockDim.x;
    for (long long v = first; v < n; v += step) {
        const int a = __ldg(rp + v), b = __ldg(rp + v + 1);
        if (a >= b) continue;
        atomicOr(heads + (a >> 5), 1u << (a & 31));
        row[b - 1] = static_cast<unsigned>(v);
    }
    for (long long c = first; c * kPrChunk < nnz; c += step) {
        const long long last = ((c + 1) * kPrChunk < nnz ? (c + 1) * kPrChunk : nnz) - 1;
        int lo = 0, hi = n;  // rp[lo] <= last < rp[hi]
        while (hi - lo > 1) {
            const int mid = lo + (hi - lo) / 2;
            if (__ldg(rp + mid) <= last)
                lo = mid;
            else
                hi = mid;
        }
        row[last] = static_cast<unsigned>(lo);
    }
}

// r = 1 / n, x[u] = r[u] / outdeg(u), dang[0] = the mass of vertices without out-edges
__global__ void __launch_bounds__(kPrVec) pr_init(int n, const int *__restrict__ out_rp, float *r, float *x,
                                                    PrState *st) {
    __shared__ double tmp[kPrVec / 32];
    const float r0 = 1.0f / n;
    double dang = 0.0;
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const int d = __ldg(out_rp + v + 1) - __ldg(out_rp + v);
        r[v] = r0;
        x[v] = d > 0 ? r0 / static_cast<float>(d) : 0.0f;
        if (d == 0) dang += r0;
    }
    dang = block_sum(dang, tmp);
    if (threadIdx.x == 0 && dang != 0.0) atomicAdd(&st->part[blockIdx.x % kPrSlots].dang[0], dang);
}

// VEC: col is 16-byte aligned
template <bool VEC>
__global__ void __launch_bounds__(kPrBlock) pr_gather(long long nnz, const int *__restrict__ col,
                                                      const unsigned char *__restrict__ heads,
                                                      const unsigned *__restrict__ row, const float *__restrict__ x,
                                                      float *y, float *carry, PrState *st, int it, double tol,
                                                      const int *err) {
    __shared__ float s_val[kPrBlock / 32];
    __shared__ int s_any[kPrBlock / 32];
    // the columns are fetched beside the words that say whether they are to be used (604 -> 580 us
    // in 16 iterations)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long c0 = static_cast<long long>(blockIdx.x) * kPrChunk;
    const long long e0 = c0 + tid * kPrItems;
    int u[kPrItems];
    if (VEC && e0 + kPrItems <= nnz) {
        const int4 a = __ldg(reinterpret_cast<const int4 *>(col + e0));
        const int4 b = __ldg(reinterpret_cast<const int4 *>(col + e0) + 1);
        u[0] = a.x, u[1] = a.y, u[2] = a.z, u[3] = a.w;
        u[4] = b.x, u[5] = b.y, u[6] = b.z, u[7] = b.w;
    } else {
#pragma unroll
        for (int j = 0; j < kPrItems; ++j) u[j] = e0 + j < nnz ? __ldg(col + e0 + j) : -1;
    }
    const unsigned m = e0 < nnz ? __ldg(heads + (e0 >> 3)) : 0u;
    const int bad = err ? ld_volatile_i32(err) : 0;
    const int done = ld_volatile_i32(&st->done);
    const double change = it > 0 ? st->diff((it - 1) & 1) : 0.0;  // the last launch wrote it
    if (bad != 0 || done != 0) return;
    if (it > 0 && change < tol) {  // every block sees the same
        if (blockIdx.x == 0 && tid == 0) st->done = it;
        return;
    }
    if (blockIdx.x == 0 && tid < kPrSlots) {  // read by the last launch, added to by the next
        st->part[tid].dang[(it + 1) & 1] = 0.0;
        st->part[tid].diff[it & 1] = 0.0;
    }
    if (c0 >= nnz) return;
    float v[kPrItems];
#pragma unroll
    for (int j = 0; j < kPrItems; ++j) v[j] = u[j] >= 0 ? __ldg(x + u[j]) : 0.0f;
    // pieces: before the thread's first head (`first`), whole rows, after its last head (`acc`)
    float first = 0.0f, acc = 0.0f;
    bool seen = false;
#pragma unroll
    for (int j = 0; j < kPrItems; ++j) {
        if ((m >> j) & 1u) {
            if (seen)
                y[__ldg(row + e0 + j - 1)] = acc;
            else
                first = acc;
            seen = true;
            acc = 0.0f;
        }
        acc += v[j];
    }
    // inclusive segmented scan of (acc, seen) over the block's threads
    float sv = acc;
    int sf = seen;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float pv = __shfl_up_sync(0xffffffffu, sv, o);
        const int pf = __shfl_up_sync(0xffffffffu, sf, o);
        if (lane >= o) {
            if (!sf) sv += pv;
            sf |= pf;
        }
    }
    if (lane == 31) {
        s_val[warp] = sv;
        s_any[warp] = sf;
    }
    float in = __shfl_up_sync(0xffffffffu, sv, 1);  // what the threads before hold of the open row
    int any = __shfl_up_sync(0xffffffffu, sf, 1);   // and whether it began in this chunk
    if (lane == 0) {
        in = 0.0f;
        any = 0;
    }
    __syncthreads();
    float wv = 0.0f;
    int wf = 0;
    for (int w = 0; w < warp; ++w) {
        wv = s_any[w] ? s_val[w] : wv + s_val[w];
        wf |= s_any[w];
    }
    if (!any) in += wv;
    any |= wf;
    if (seen) {  // the row that is open before this thread ends at its first head
        const float t = in + first;
        if (any)
            y[__ldg(row + e0 + (__ffs(m) - 1) - 1)] = t;
        else
            carry[blockIdx.x] = t;
    }
    if (tid == kPrBlock - 1) {  // the row that is open at the chunk's end
        const long long last = (c0 + kPrChunk < nnz ? c0 + kPrChunk : nnz) - 1;
        const float t = seen ? acc : in + acc;
        if (seen || any)
            y[__ldg(row + last)] = t;
        else
            carry[blockIdx.x] = t;
    }
}

// r'[v] = (1 - d) / n + d * (sum over in-edges + dangling / n), the L1 change, and the next
// iteration's x and dangling mass. 7.0 us for 700,001 vertices (14 MB, 2.1 us at the copy rate:
// launch, the loads' latency and the blocks' sums); with one vertex at a time and the sums beside
// the first look's word 11.7 us; one vertex, four blocks of 512 7.9 us.
__global__ void __launch_bounds__(kPrVec) pr_update(int n, float damping, const int *__restrict__ in_rp,
                                                      const int *__restrict__ out_rp, const float *__restrict__ y,
                                                      const float *__restrict__ carry, float *r, float *x,
                                                      PrState *st, int it, const int *err) {
    __shared__ double tmp[kPrVec / 32];
    const int bad = err ? ld_volatile_i32(err) : 0;
    const int done = ld_volatile_i32(&st->done);
    if (bad != 0 || done != 0) return;
    const float base = static_cast<float>((1.0 - damping) / n + damping * st->dang(it & 1) / n);
    double diff = 0.0, dang = 0.0;
    const int stride = gridDim.x * blockDim.x;
    for (int v0 = blockIdx.x * blockDim.x + threadIdx.x; v0 < n; v0 += kPrOwn * stride) {
        int a[kPrOwn], b[kPrOwn], d[kPrOwn];
        float s[kPrOwn], old[kPrOwn];
#pragma unroll
        for (int k = 0; k < kPrOwn; ++k) {
            const int v = v0 + k * stride;
            const bool in = v < n && v >= v0;
            a[k] = in ? __ldg(in_rp + v) : 0;
            b[k] = in ? __ldg(in_rp + v + 1) : 0;
            d[k] = in ? __ldg(out_rp + v + 1) - __ldg(out_rp + v) : 1;
            s[k] = in ? y[v] : 0.0f;  // rows without entries have none
            old[k] = in ? r[v] : 0.0f;
        }
#pragma unroll
        for (int k = 0; k < kPrOwn; ++k) {
            const int v = v0 + k * stride;
            if (v >= n || v < v0) break;
            if (b[k] > a[k]) {
                const int c1 = (b[k] - 1) / kPrChunk;
#pragma unroll 4
                for (int c = a[k] / kPrChunk + 1; c <= c1; ++c) s[k] += __ldg(carry + c);
            } else {
                s[k] = 0.0f;
            }
            const float nr = __fmaf_rn(damping, s[k], base);
            diff += fabs(static_cast<double>(nr) - static_cast<double>(old[k]));
            r[v] = nr;
            x[v] = d[k] > 0 ? nr / static_cast<float>(d[k]) : 0.0f;
            if (d[k] == 0) dang += nr;
        }
    }
    diff = block_sum(diff, tmp);
    dang = block_sum(dang, tmp);
    if (threadIdx.x == 0) {
        if (diff != 0.0) atomicAdd(&st->part[blockIdx.x % kPrSlots].diff[it & 1], diff);
        if (dang != 0.0) atomicAdd(&st->part[blockIdx.x % kPrSlots].dang[(it + 1) & 1], dang);
    }
}

}  // namespace
}  // namespace apspie

using namespace apspie;

extern "C" {

apspie_status apspie_spmv(apspie_ctx *ctx, const apspie_csr *A, const float *d_x, float *d_y, float alpha,
                          float beta) {
    if (!ctx) return APSPIE_ERR_INVALID_ARG;
    cudaSetDevice(ctx->device);
    apspie_status st = check_csr_view(ctx, A, "apspie_spmv");
    if (st != APSPIE_OK) return st;
    if (A->val_type == APSPIE_VAL_I32)
        return set_error(ctx, APSPIE_ERR_UNSUPPORTED, "apspie_spmv: float32 values or a pattern required");
    if (A->m > 0 && (!d_y || (A->nnz > 0 && !d_x)))
        return set_error(ctx, APSPIE_ERR_INVALID_ARG, "apspie_spmv: NULL vector");
    if (ctx->validate && (st = validate_csr(ctx, A, false)) != APSPIE_OK) return st;
    if (A->m == 0) return APSPIE_OK;
    return launch_spmv(ctx, A, d_x, d_y, alpha, beta);
}

apspie_status apspie_pagerank(apspie_ctx *ctx, const apspie_csr *A, float damping, double tol, int32_t max_iter,
                              float *d_rank, int32_t *iterations) {
    if (!ctx || !d_rank || max_iter < 1 || !(damping >= 0.0f && damping < 1.0f) || !(tol >= 0.0))
        return APSPIE_ERR_INVALID_ARG;
    cudaSetDevice(ctx->device);
    apspie_status st = check_csr_view(ctx, A, "apspie_pagerank");
    if (st != APSPIE_OK) return st;
    if (A->m != A->n || A->m == 0)
        return set_error(ctx, APSPIE_ERR_INVALID_ARG, "apspie_pagerank: square, non-empty graph required");
    if (ctx->validate && (st = validate_csr(ctx, A, true)) != APSPIE_OK) return st;
    const int n = A->m;
    // pull over in-edges: A^T, or A itself when the pattern is symmetric
    const long long nnz = A->nnz;
    const bool sym = (A->flags & APSPIE_CSR_SYMMETRIC) != 0;
    const size_t nn = static_cast<size_t>(n);
    const size_t chunks = static_cast<size_t>(nnz / kPrChunk) + 1;
    const size_t mat = sym ? (static_cast<size_t>(nnz) + 1) * 4 : transpose_pattern_need(A->n, nnz);
    const size_t head_bytes = (static_cast<size_t>(nnz / 32) + 1) * 4;
    void *base;
    st = scratch_reserve(ctx, Carver::need({mat, nn * 4, nn * 4, chunks * 4, head_bytes, sizeof(PrState)}),
                         &base);
    if (st != APSPIE_OK) return st;
    Carver c(base);
    char *mat_base = c.take<char>(mat);
    float *x = c.take<float>(nn);
    float *y = c.take<float>(nn);
    float *carry = c.take<float>(chunks);
    unsigned char *heads = c.take<unsigned char>(head_bytes);
    PrState *state = c.take<PrState>(1);
    cudaError_t e = cudaMemsetAsync(state, 0, sizeof(PrState), ctx->stream);
    if (e == cudaSuccess && sym) e = cudaMemsetAsync(heads, 0, head_bytes, ctx->stream);
    if (e != cudaSuccess) return cuda_error(ctx, e, "apspie_pagerank reset");
    PatternCoo in{A->row_ptr, reinterpret_cast<const unsigned *>(mat_base), A->col_ind, nullptr};
    if (!sym && (st = transpose_pattern(ctx, A, mat_base, &in)) != APSPIE_OK) return st;
    const int vblocks = std::max(1, std::min((n + kPrVec - 1) / kPrVec, ctx->num_sms * 4));
    const int gblocks = static_cast<int>((nnz + kPrChunk - 1) / kPrChunk);
    if (nnz > 0 && sym)
        pr_marks<<<vblocks, kPrVec, 0, ctx->stream>>>(n, nnz, A->row_ptr, reinterpret_cast<unsigned *>(heads),
                                                      reinterpret_cast<unsigned *>(mat_base));
    else if (nnz > 0)
        pr_heads<<<static_cast<int>(std::min<long long>((nnz / 8 + 256) / 256, ctx->num_sms * 8LL)), 256, 0,
                   ctx->stream>>>(nnz, in.row, heads);
    pr_init<<<vblocks, kPrVec, 0, ctx->stream>>>(n, A->row_ptr, d_rank, x, state);
    const bool vec = (reinterpret_cast<uintptr_t>(in.col) & 15u) == 0;
    int it = 0;
    PrState h;
    for (;;) {
        for (int k = 0; k < kPrBatch && it < max_iter; ++k, ++it) {
            (vec ? pr_gather<true> : pr_gather<false>)<<<std::max(gblocks, 1), kPrBlock, 0, ctx->stream>>>(
                nnz, in.col, heads, in.row, x, y, carry, state, it, tol, in.err);
            pr_update<<<vblocks, kPrVec, 0, ctx->stream>>>(n, damping, in.rp, A->row_ptr, y, carry, d_rank, x,
                                                             state, it, in.err);
        }
        int sort_err = 0;
        if ((e = cudaGetLastError()) != cudaSuccess ||
            (e = cudaMemcpyAsync(&h, state, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream)) != cudaSuccess ||
            (in.err &&
             (e = cudaMemcpyAsync(&sort_err, in.err, 4, cudaMemcpyDeviceToHost, ctx->stream)) != cudaSuccess) ||
            (e = cudaStreamSynchronize(ctx->stream)) != cudaSuccess)
            return cuda_error(ctx, e, "apspie_pagerank");
        if (sort_err) return set_error(ctx, static_cast<apspie_status>(sort_err), "apspie_pagerank: transpose");
        if (h.done != 0) {
            it = h.done;
            break;
        }
        if (it >= max_iter || h.diff((it - 1) & 1) < tol) break;
    }
    if (iterations) *iterations = it;
    return APSPIE_OK;
}

}  // extern "C"
