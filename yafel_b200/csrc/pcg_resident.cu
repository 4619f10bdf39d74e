// pcg_resident.cu -- Jacobi-PCG iterations of systems whose matrix fits the
// shared memory of the GPU, as one cooperative kernel.
//
// The three-kernel iteration of krylov.cu costs 12-16 us whatever the size: three
// launches that each wait for the last block of the one before and reduce
// hundreds of partials.  Here every SM takes a contiguous share of the block rows,
// copies its values, columns and vector entries to shared memory once, and
// iterates on them; only the search direction crosses the SMs.  An iteration has
// two grid-wide sums and no other barrier:
//   * p = z + beta p is not formed before the product but in it: each gathered
//     column reads the pair (z, p_old) from global memory and combines them, with
//     the same rounding as the owner does for its own entries;
//   * q = A p, partial p.q                                   -> first sum, alpha
//   * x += alpha p, r -= alpha q, z = D^-1 r, partial r.z and r.r; (z, p) of the own
//     rows to global memory                                  -> second sum, beta
// The sum of iteration k publishes the pairs that iteration k + 1 gathers, and the
// first sum of k + 1 tells that all have read them before they are written again.
//
// A grid-wide sum is one store and one load per SM: a block writes its partials
// with the sum's number in the upper half of each 64-bit word, and one warp of
// every block polls all blocks' words until the numbers are right (no counter, no
// atomics).  All blocks add the partials in the same order, so they agree on
// alpha, beta and the stopping tests bit for bit and a solve is reproducible.
//
// Measured (us an iteration, before -> now): 4,225 unknowns of Q1 Poisson 14.9 -> 5.7;
// 14,884 nodes of order-2 plane elasticity 15.8 -> 9.2; 10,125 unknowns of Q2
// elasticity 17 -> 11.8.  The trips through L2 of the two sums bound it: a matrix
// this size takes 1-4 us from shared memory.
// Polls are bounded: a block that gives up records YG_TIMEOUT and returns, and so
// do the others.
#include "internal.h"
#include "device_common.cuh"

#include <algorithm>
#include <cmath>
#include <mutex>

namespace yg {

enum { FLAG_RUN = 0, FLAG_CONVERGED = 1, FLAG_BREAKDOWN = 2, FLAG_NAN = 3, FLAG_MAXITER = 4 };

constexpr long long kGridSpinLimit = 1ll << 22;  // polls of one grid-wide sum (seconds; a sum takes microseconds)
constexpr int kMaxSumBlocks = 256;

struct alignas(32) SumSlot {
    unsigned long long w[4];  // low and high halves of two doubles, each below the sum's number
};

struct ResidentArgs {
    int nbrows;
    const int32_t *rowptr, *col;
    const void *val;
    const double *corr, *dinv;
    double *x, *r, *p;
    double *zp;              // per block row: B entries of z, B of p
    SumSlot *slots;          // [2][kMaxSumBlocks]
    KrylovScalars *S;
    int32_t *err;
    int64_t block_cost, row_cost, total_cost;  // shared memory bytes per block, per block row, of all
    int lanes;               // lanes per block row
    int max_its, check;      // iterations of this launch at most; residual replacement is looked at every `check`
    double rr_replace;       // leave when r.r < rr_replace at such a point (0: never)
};

__device__ __forceinline__ double warp_sum_all(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sums over all threads of the grid of v0 and v1, the same bits in every block.
// PUBLISH: what the block's threads wrote to global memory before is visible to
// the blocks that return.  False when the poll gave up.
// Release / acquire at GPU scope (__threadfence is the sequentially consistent
// fence, which a pair of blocks that hand data over does not need).
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

__device__ __forceinline__ void put_sums(SumSlot *s, unsigned epoch, double v0, double v1, bool two) {
    const unsigned long long e = (unsigned long long)epoch << 32;
    const unsigned long long b0 = (unsigned long long)__double_as_longlong(v0), b1 = (unsigned long long)__double_as_longlong(v1);
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(s->w), "l"(e | (b0 & 0xffffffffu)), "l"(e | (b0 >> 32)) : "memory");
    if (two)
        asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(s->w + 2), "l"(e | (b1 & 0xffffffffu)), "l"(e | (b1 >> 32)) : "memory");
}
// Whether the slot's words are those of sum `epoch`; then v0 and v1 are its values.
__device__ __forceinline__ bool get_sums(const SumSlot *s, unsigned epoch, double &v0, double &v1, bool two) {
    unsigned long long u[4];
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(u[0]), "=l"(u[1]) : "l"(s->w) : "memory");
    bool ok = (unsigned)(u[0] >> 32) == epoch && (unsigned)(u[1] >> 32) == epoch;
    v0 = __longlong_as_double((long long)((u[0] & 0xffffffffu) | (u[1] << 32)));
    if (two) {
        asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(u[2]), "=l"(u[3]) : "l"(s->w + 2) : "memory");
        ok = ok && (unsigned)(u[2] >> 32) == epoch && (unsigned)(u[3] >> 32) == epoch;
        v1 = __longlong_as_double((long long)((u[2] & 0xffffffffu) | (u[3] << 32)));
    }
    return ok;
}

template <bool TWO, bool PUBLISH>
__device__ bool grid_sum(SumSlot *slots, unsigned epoch, double v0, double v1, double &o0, double &o1) {
    __shared__ double part[2][32];
    __shared__ double total[3];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5, G = gridDim.x;
    v0 = warp_sum_all(v0);
    if (TWO) v1 = warp_sum_all(v1);
    if (lane == 0) {
        part[0][w] = v0;
        if (TWO) part[1][w] = v1;
    }
    __syncthreads();
    if (w == 0) {
        const double s0 = warp_sum_all(lane < nw ? part[0][lane] : 0.0);
        const double s1 = TWO ? warp_sum_all(lane < nw ? part[1][lane] : 0.0) : 0.0;
        if (lane == 0) {
            if (PUBLISH) fence_gpu();
            put_sums(slots + blockIdx.x, epoch, s0, s1, TWO);
        }
        double a0 = 0, a1 = 0;
        bool ok = false;
        __nanosleep(200);  // no word is there sooner; polls before only hold up the stores
        for (long long spins = 0; spins < kGridSpinLimit && !ok; ++spins) {
            ok = true;
            a0 = a1 = 0;
#pragma unroll 5
            for (int s = lane; s < G; s += 32) {
                double b0, b1 = 0;
                ok = get_sums(slots + s, epoch, b0, b1, TWO) && ok;
                a0 += b0;
                a1 += b1;
            }
            ok = __all_sync(0xffffffffu, ok);
        }
        a0 = warp_sum_all(a0);
        if (TWO) a1 = warp_sum_all(a1);
        if (PUBLISH) fence_gpu();
        if (lane == 0) {
            total[0] = a0;
            total[1] = a1;
            total[2] = ok ? 1.0 : 0.0;
        }
    }
    __syncthreads();
    o0 = total[0];
    o1 = total[1];
    return total[2] != 0;
}

// First block row whose cost before it (blocks and rows) reaches `target`, by one warp.
__device__ int first_row(const int32_t *rowptr, int n, int64_t block_cost, int64_t row_cost, int64_t target) {
    const int lane = threadIdx.x & 31;
    int lo = 0, hi = n;  // the answer is in [lo, hi]
    while (lo < hi) {
        const int step = (hi - lo + 31) / 32;
        const int i = min(lo + lane * step, hi);  // probes lo, lo + step, ...
        const bool below = i < hi && (int64_t)__ldg(rowptr + i) * block_cost + i * row_cost < target;
        const unsigned m = __ballot_sync(0xffffffffu, below);
        const int k = __popc(m);  // probes 0 .. k - 1 are below (the cost grows with the row)
        if (k == 0) return lo;
        const int last = lo + (k - 1) * step;
        hi = min(last + step, hi);
        lo = last + 1;
    }
    return lo;
}

template <int B, typename VT>
__global__ void __launch_bounds__(512, 1) k_pcg_resident(ResidentArgs a) {
    constexpr int B2 = B * B;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int bounds[2];
    KrylovScalars *S = a.S;
    if (read_flag(&S->flag)) return;  // set before the launch: the same for every block
    const int tid = threadIdx.x, nt = blockDim.x, G = gridDim.x;
    if (tid < 64) {
        const int64_t t = blockIdx.x + (tid >> 5);
        const int r = t == G ? a.nbrows : first_row(a.rowptr, a.nbrows, a.block_cost, a.row_cost, t * a.total_cost / G);
        if ((tid & 31) == 0) bounds[tid >> 5] = r;
    }
    __syncthreads();
    const int r0 = bounds[0], nr = bounds[1] - r0, nd = nr * B;
    const int e0 = a.rowptr[r0], nb = a.rowptr[bounds[1]] - e0;
    // shared memory: values | columns | row pointers | x, r, p, q (z after the update), dinv, correction
    auto up = [](size_t v) { return (v + 15) & ~(size_t)15; };
    VT *val = reinterpret_cast<VT *>(smem);
    int32_t *col = reinterpret_cast<int32_t *>(smem + up((size_t)nb * B2 * sizeof(VT)));
    int32_t *rp = reinterpret_cast<int32_t *>(reinterpret_cast<unsigned char *>(col) + up((size_t)nb * 4));
    double *x = reinterpret_cast<double *>(reinterpret_cast<unsigned char *>(rp) + up((size_t)(nr + 1) * 4));
    double *r = x + nd, *p = r + nd, *q = p + nd, *dinv = q + nd;
    double *corr = dinv + (a.dinv ? nd : 0);
    const VT *gval = static_cast<const VT *>(a.val) + (int64_t)e0 * B2;
    for (int i = tid; i < nb * B2; i += nt) val[i] = gval[i];
    for (int i = tid; i < nb; i += nt) col[i] = a.col[e0 + i];
    for (int i = tid; i <= nr; i += nt) rp[i] = a.rowptr[r0 + i] - e0;
    if (a.corr)
        for (int i = tid; i < nr * B2; i += nt) corr[i] = a.corr[(int64_t)r0 * B2 + i];
    double *zp = a.zp + (int64_t)r0 * 2 * B;
    for (int i = tid; i < nd; i += nt) {
        const int64_t g = (int64_t)r0 * B + i;
        x[i] = a.x[g];
        r[i] = a.r[g];
        if (a.dinv) dinv[i] = a.dinv[g];
        // the direction of the first iteration, as z with beta = 0
        const double v = a.p[g];
        p[i] = 0;
        q[i] = v;
        const int row = i / B, c = i - row * B;
        zp[row * 2 * B + c] = v;
        zp[row * 2 * B + B + c] = 0;
    }
    const double tol = S->tol, bb = S->bb, rz0 = S->rz0;
    const int criterion = S->criterion;
    const int64_t maxiter = S->maxiter;
    int64_t iter = S->iter;
    double rz = S->rz[0], rr = S->rr, beta = 0;
    unsigned epoch = 1;
    int flag = FLAG_RUN;
    double t0, t1;
    bool ok = grid_sum<false, true>(a.slots + kMaxSumBlocks, epoch, 0, 0, t0, t1);
    const int L = a.lanes, lane = tid & (L - 1), group = tid / L, ngroups = nt / L;
    for (int it = 0; ok; ++it) {
        for (int i = tid; i < nd; i += nt) p[i] = fma(beta, p[i], q[i]);
        __syncthreads();  // p is read and q overwritten by other threads
        double pq = 0;
        for (int rb = 0; rb < nr; rb += ngroups) {  // the lanes of a warp take the same steps
            const int row = rb + group;
            double acc[B];
#pragma unroll
            for (int i = 0; i < B; ++i) acc[i] = 0;
            if (row < nr) {
                const int je = rp[row + 1];
                constexpr int U = B == 1 ? 4 : 2;  // gathers in flight per lane
                for (int j0 = rp[row] + lane; j0 < je; j0 += U * L) {
                    double v[U][2 * B];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int j = j0 + u * L;
                        if (j < je) {
                            const double2 *s = reinterpret_cast<const double2 *>(a.zp + (int64_t)col[j] * 2 * B);
#pragma unroll
                            for (int k = 0; k < B; ++k) {
                                const double2 d = s[k];
                                v[u][2 * k] = d.x;
                                v[u][2 * k + 1] = d.y;
                            }
                        }
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int j = j0 + u * L;
                        if (j < je) {
#pragma unroll
                            for (int c = 0; c < B; ++c) {
                                const double pc = fma(beta, v[u][B + c], v[u][c]);
#pragma unroll
                                for (int i = 0; i < B; ++i) acc[i] = fma((double)val[j * B2 + i * B + c], pc, acc[i]);
                            }
                        }
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < B; ++i)
                for (int o = L >> 1; o > 0; o >>= 1) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
            if (row < nr && lane == 0) {
                if (a.corr) add_corr<B>(corr, p, row, acc);
#pragma unroll
                for (int i = 0; i < B; ++i) {
                    q[row * B + i] = acc[i];
                    pq = fma(acc[i], p[row * B + i], pq);
                }
            }
        }
        ++epoch;
        if (!(ok = grid_sum<false, false>(a.slots, epoch, pq, 0, pq, t1))) break;
        const double alpha = rz / pq;
        if (pq == 0 || !isfinite(alpha)) {
            flag = isfinite(pq) ? FLAG_BREAKDOWN : FLAG_NAN;
            break;
        }
        double srz = 0, srr = 0;
        for (int i = tid; i < nd; i += nt) {
            const double pi = p[i], ri = r[i] + (-alpha) * q[i];
            x[i] += pi * alpha;
            r[i] = ri;
            const double zi = a.dinv ? dinv[i] * ri : ri;
            q[i] = zi;
            srz += ri * zi;
            srr += ri * ri;
            const int row = i / B, c = i - row * B;
            zp[row * 2 * B + c] = zi;
            zp[row * 2 * B + B + c] = pi;
        }
        double rz_new;
        if (!(ok = grid_sum<true, true>(a.slots + kMaxSumBlocks, epoch, srz, srr, rz_new, rr))) break;
        ++iter;
        const bool conv = criterion == YG_CRIT_REFERENCE ? rz_new / rz0 < tol : sqrt(rr) <= tol * sqrt(bb);
        if (conv) flag = FLAG_CONVERGED;
        if (!isfinite(rz_new)) flag = FLAG_NAN;
        if (flag == FLAG_RUN && iter >= maxiter) flag = FLAG_MAXITER;
        beta = rz_new / rz;
        rz = rz_new;
        if (flag != FLAG_RUN || it + 1 >= a.max_its || ((it + 1) % a.check == 0 && rr < a.rr_replace)) break;
    }
    if (!ok) {
        if (tid == 0) atomicExch(a.err, (int32_t)YG_TIMEOUT);
        flag = FLAG_NAN;
    }
    for (int i = tid; i < nd; i += nt) {
        const int64_t g = (int64_t)r0 * B + i;
        a.x[g] = x[i];
        a.r[g] = r[i];
        if (flag == FLAG_RUN) a.p[g] = fma(beta, p[i], q[i]);  // the next direction
    }
    if (blockIdx.x == 0 && tid == 0) {
        S->rz[0] = S->rz[1] = rz;
        S->rr = rr;
        S->iter = S->iter_seen = iter;
        S->flag = flag;
    }
}

// Cooperative kernels of two streams must not hold part of the SMs each: their
// launches on a device follow one another, whatever context they come from.
yg_status launch_cooperative(yg_context ctx, const void *kern, int grid, int threads, size_t smem, void **args) {
    static std::mutex m;
    static cudaEvent_t last[64] = {};
    const int d = ctx->device & 63;
    cudaStreamCaptureStatus cs;
    YG_CUDA(cudaStreamIsCapturing(ctx->stream, &cs));
    if (cs != cudaStreamCaptureStatusNone) {  // (an ILU(0) apply in a captured iteration: small blocks, which fit beside any)
        YG_CUDA(cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(threads), args, smem, ctx->stream));
        YG_LAUNCHED(ctx);
        return YG_OK;
    }
    std::lock_guard<std::mutex> hold(m);
    if (last[d]) YG_CUDA(cudaStreamWaitEvent(ctx->stream, last[d], 0));
    else YG_CUDA(cudaEventCreateWithFlags(&last[d], cudaEventDisableTiming));
    YG_CUDA(cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(threads), args, smem, ctx->stream));
    YG_CUDA(cudaEventRecord(last[d], ctx->stream));
    YG_LAUNCHED(ctx);
    return YG_OK;
}

template <int B, typename VT>
static const void *resident_kernel() { return reinterpret_cast<const void *>(&k_pcg_resident<B, VT>); }
static const void *resident_kernel(int B, bool f32) {
    if (B == 1) return f32 ? resident_kernel<1, float>() : resident_kernel<1, double>();
    if (B == 2) return f32 ? resident_kernel<2, float>() : resident_kernel<2, double>();
    return f32 ? resident_kernel<3, float>() : resident_kernel<3, double>();
}

// Shared memory per block (values, column) and per block row (row pointer, x, r,
// p, q, dinv, correction) of a resident solve.
static void resident_costs(yg_matrix A, bool f32, bool jacobi, int64_t *block, int64_t *row) {
    const int B = A->block;
    *block = (f32 ? 4 : 8) * B * B + 4;
    *row = 4 + 8 * B * (jacobi ? 5 : 4) + (f32 && A->d_corr32 ? 8 * B * B : 0);
}

// Shared memory of the largest share among G blocks: at most the mean and one row more.
static int64_t resident_smem(yg_matrix A, bool f32, bool jacobi, int G) {
    int64_t bc, rc;
    resident_costs(A, f32, jacobi, &bc, &rc);
    return (A->nnzb * bc + A->nbrows * rc + G - 1) / G + A->row_max * bc + rc + 256;
}

// Blocks of a resident solve, one per SM at most.  The two sums cost 4.5 us + 0.028 us
// per block (5.0 us an iteration of 882 unknowns on 32 blocks, 5.4 on 64, 6.6 on 96,
// 8.9 on 148: every block polls every other's words) and the products 0.52 ns per CSR
// entry, 0.27 ns per entry of a block, divided by the blocks (40,401 unknowns, 361,201
// entries: 10.7 us on 32, 8.3 on 64, 8.4 on 96, 10.0 on 148), so the best number grows
// with the square root of the entries; the shared memory sets a lower bound.
static int resident_blocks(yg_matrix A, bool f32, bool jacobi) {
    yg_context ctx = A->ctx;
    const double entries = (double)A->nnzb * A->block * A->block;
    const int most = (int)std::min<int64_t>(ctx->num_sms, A->nbrows);
    int G = (int)std::max(16.0, (A->block == 1 ? 0.136 : 0.098) * std::sqrt(entries));
    while (G < most && resident_smem(A, f32, jacobi, G) > (int64_t)ctx->smem_optin - 2048) G += 4;
    return std::min(G, most);
}

// Whether A's PCG iterations run resident: a block size the kernel has, and each
// SM's share (at most the mean and one row more) within a block's shared memory.
yg_status pcg_resident_fits(yg_matrix A, bool f32, bool jacobi, bool *fits) {
    yg_context ctx = A->ctx;
    *fits = false;
    if (A->block > 3 || A->nbrows < 1 || A->nbrows >= (1 << 24) || ctx->num_sms > kMaxSumBlocks) return YG_OK;
    int64_t bc, rc;
    resident_costs(A, f32, jacobi, &bc, &rc);
    const int64_t total = A->nnzb * bc + A->nbrows * rc, room = (int64_t)ctx->smem_optin - 2048;
    if (total / ctx->num_sms > room) return YG_OK;
    YG_TRY(matrix_row_extent(A));
    *fits = resident_smem(A, f32, jacobi, resident_blocks(A, f32, jacobi)) <= room;
    return YG_OK;
}

// One launch of at most max_its iterations on the state pcg_core keeps (x, r, p and
// the scalars; zp: 2 n doubles of scratch).
yg_status pcg_resident_launch(yg_matrix A, bool f32, const double *dinv, double *x, double *r, double *p, double *zp,
                              int max_its, int check, double rr_replace) {
    yg_context ctx = A->ctx;
    ResidentArgs a;
    a.nbrows = (int)A->nbrows;
    a.rowptr = A->d_rowptr;
    a.col = A->d_col;
    a.val = f32 ? static_cast<const void *>(A->d_val32) : A->d_val;
    a.corr = f32 ? A->d_corr32 : nullptr;
    a.dinv = dinv;
    a.x = x;
    a.r = r;
    a.p = p;
    a.zp = zp;
    a.slots = reinterpret_cast<SumSlot *>(ctx->d_slots);
    a.S = ctx->d_scalars;
    a.err = ctx->d_err;
    resident_costs(A, f32, dinv != nullptr, &a.block_cost, &a.row_cost);
    a.total_cost = A->nnzb * a.block_cost + A->nbrows * a.row_cost;
    a.max_its = max_its;
    a.check = check;
    a.rr_replace = rr_replace;
    const int G = resident_blocks(A, f32, dinv != nullptr);
    // lanes per row: about two blocks (four entries) each, more where the threads allow
    const double mean = (double)A->nnzb / A->nbrows;
    const int64_t rows = (A->nbrows + G - 1) / G;
    const int threads = rows * (mean > 8 ? 8 : 4) > 512 ? 512 : 256;
    int L = 2;
    while (L < 32 && L * (A->block == 1 ? 4 : 2) < mean) L *= 2;
    while (L < 32 && L < mean && rows * 2 * L <= threads) L *= 2;
    a.lanes = L;
    const size_t smem = (size_t)resident_smem(A, f32, dinv != nullptr, G);
    const void *kern = resident_kernel(A->block, f32);
    YG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    YG_CUDA(cudaMemsetAsync(ctx->d_slots, 0, sizeof(SumSlot) * 2 * kMaxSumBlocks, ctx->stream));
    void *args[] = {&a};
    return launch_cooperative(ctx, kern, G, threads, smem, args);
}

}  // namespace yg
