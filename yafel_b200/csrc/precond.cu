// precond.cu -- Jacobi and ILU(0) preconditioners.
//
// Jacobi replaces JacobiPreconditioner (solver/iterative/JacobiPreconditioner.hpp:11-54):
// z_i = r_i / a_ii with the scalar diagonal; a zero diagonal gives inf, as the
// reference computes 1/0 (its warning text says otherwise).  Inside PCG it is
// fused into the vector kernels (krylov.cu) and never launched on its own.
//
// ILU(0) replaces ILUPreconditioner (ILUPreconditioner.hpp:96-329): incomplete
// LU without pivoting on the scalar pattern of A (a BCSR matrix counts with its
// full B*B entries per block), zero pivots skipped.  The reference walks pivots
// (KIJ, O(N^2) row scans); here rows are factored in IKJ order, which applies to
// every entry the same updates in the same order.
//
// A warp takes the B rows of a block row together (they share their columns) and
// waits only for the block rows it reads: the factorization and an apply are one
// cooperative launch each, without grid-wide barriers.  Block rows are handed out
// sorted by dependency level, so what a warp waits for is always at work or done,
// and a level costs one trip through L2 instead of a barrier.  In an apply the
// values themselves are the messages: the vectors are filled with a signalling NaN,
// which no arithmetic produces, and readers poll them.  7^3 Q2 elasticity (10,125
// unknowns, 549 scalar levels each way), barrier per scalar level -> now:
// factorization and levels 497 -> 4.4 ms, apply 5.06 -> 0.46 ms.
#include "internal.h"
#include "device_common.cuh"

#include <algorithm>
#include <cmath>

namespace yg {

int stream_grid(yg_context ctx, int64_t n);

__global__ void k_jacobi_build(int64_t nbrows, int B, const int32_t *__restrict__ diag, const double *__restrict__ val,
                               double *__restrict__ dinv, int *__restrict__ zeros) {
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < nbrows * B; r += (int64_t)gridDim.x * blockDim.x) {
        int64_t I = r / B, i = r % B;
        int32_t d = diag[I];
        double a = d >= 0 ? val[(int64_t)d * B * B + i * B + i] : 0.0;
        dinv[r] = 1.0 / a;
        if (a == 0) atomicAdd(zeros, 1);
    }
}

__global__ void k_jacobi_apply(int64_t n, const double *__restrict__ dinv, const double *__restrict__ r,
                               double *__restrict__ z) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        z[i] = r[i] * dinv[i];
}

// ---------------------------------------------------------------------------
// ILU(0).  Factor values: the scalar rows of block row I start at rowptr[I] * B * B,
// row r of them at r * len * B (len blocks); column e of a row is
// B * col[e / B] + e % B.

// A wait of a launch: polls it may take, the launch's own abort word (a warp that gives
// up sets it and the others follow; the context's error word may still hold an earlier
// launch's) and the context's error word.
struct Waits {
    long long limit;
    int32_t *abort, *err;
};
constexpr unsigned long long kPending = 0x7ff4a11ce0000001ull;  // a signalling NaN: no arithmetic gives it

__device__ __forceinline__ double ld_relaxed(const double *p) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(double *p, double v) {
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
__device__ __forceinline__ int ld_relaxed_i(const int32_t *p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ bool pending(double v) { return (unsigned long long)__double_as_longlong(v) == kPending; }

// One more failed poll of a wait: false when the wait gives up (its limit, or
// another warp's: then the error word is set).
__device__ __forceinline__ bool wait_on(long long &spins, const Waits &w) {
    if (++spins > w.limit) {
        atomicExch(w.err, (int32_t)YG_TIMEOUT);
        atomicExch(w.abort, 1);
        return false;
    }
    return (spins & 1023) || ld_relaxed_i(w.abort) == 0;
}

__global__ void k_fill_pending(int64_t n, double *__restrict__ z, int32_t *__restrict__ abort) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *abort = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        z[i] = __longlong_as_double((long long)kPending);
}

// The factor's starting values: A's, row by row.
__global__ void k_ilu_expand(int64_t nbrows, int B, const int32_t *__restrict__ rowptr, const double *__restrict__ val,
                             double *__restrict__ lu) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t I = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; I < nbrows; I += nw) {
        const int64_t e0 = (int64_t)rowptr[I] * B * B;
        const int n = (rowptr[I + 1] - rowptr[I]) * B * B, row = n / B;
        for (int i = lane; i < n; i += 32) {
            const int blk = i / (B * B), r = i / B - blk * B, c = i % B;
            lu[e0 + r * row + blk * B + c] = val[e0 + i];
        }
    }
}

// First position in the sorted list c[lo, hi) that is not below v.
__device__ __forceinline__ int lower_bound(const int32_t *c, int lo, int hi, int v) {
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (c[mid] < v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Factorization.  rows: block rows by level; done[I] set when I's rows are final.
// room: doubles of shared memory per warp (0: the rows are updated in place).
template <int B>
__global__ void __launch_bounds__(kThreads)
k_ilu_factor(int nbrows, const int32_t *__restrict__ rows, const int32_t *__restrict__ rowptr,
             const int32_t *__restrict__ col, const int32_t *__restrict__ diag, double *lu, int32_t *done,
             int *__restrict__ zero_pivots, int room, Waits waits) {
    extern __shared__ double sm[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, nwb = blockDim.x >> 5;
    for (int t = blockIdx.x * nwb + wib; t < nbrows; t += gridDim.x * nwb) {
        const int I = rows[t], b0 = rowptr[I], len = rowptr[I + 1] - b0, n = len * B;
        const int nl = diag[I] >= 0 ? diag[I] - b0 : lower_bound(col + b0, 0, len, I);
        double *g = lu + (int64_t)b0 * B * B;
        double *a = room ? sm + (size_t)wib * room : g;
        const int32_t *bc = col + b0;
        if (room) {
            int32_t *c = reinterpret_cast<int32_t *>(a + n * B);
            for (int i = lane; i < n * B; i += 32) a[i] = g[i];
            for (int i = lane; i < len; i += 32) c[i] = bc[i];
            bc = c;
        }
        __syncwarp();
        int ready = 0;  // block columns [0, ready) are known to be final
        for (int jj = 0; jj < nl; ++jj) {
            if (jj == ready) {  // look at the next 32
                long long spins = 0;
                for (;;) {
                    const bool ok = jj + lane < nl && ld_relaxed_i(done + bc[jj + lane]) != 0;
                    const unsigned m = __ballot_sync(0xffffffffu, ok);
                    ready = jj + (m == 0xffffffffu ? 32 : __ffs(~m) - 1);
                    if (ready > jj) break;
                    if (!__all_sync(0xffffffffu, wait_on(spins, waits))) return;
                }
                asm volatile("fence.acq_rel.gpu;" ::: "memory");
            }
            const int J = bc[jj], bj = rowptr[J], dj = diag[J], lj = (rowptr[J + 1] - bj) * B;
            // pivot rows of J from their diagonal on
            const double *u = lu + (int64_t)bj * B * B + (int64_t)(dj - bj) * B;
            const int nu = dj >= 0 ? (rowptr[J + 1] - dj - 1) * B : 0;
            double m[B][B];
            bool skip[B];
            {
                double x[B][B], d[B][B];
#pragma unroll
                for (int j = 0; j < B; ++j)
#pragma unroll
                    for (int c = 0; c < B; ++c) {
                        d[j][c] = dj >= 0 && c >= j ? __ldcg(u + (int64_t)j * lj + c) : 0.0;
                        x[j][c] = a[j * n + jj * B + c];
                    }
#pragma unroll
                for (int j = 0; j < B; ++j) {
                    skip[j] = d[j][j] == 0;
                    if (skip[j] && lane == 0) atomicAdd(zero_pivots, B);
#pragma unroll
                    for (int r = 0; r < B; ++r) {
                        m[r][j] = skip[j] ? 0.0 : x[r][j] / d[j][j];
#pragma unroll
                        for (int c = j + 1; c < B; ++c)
                            if (!skip[j]) x[r][c] -= m[r][j] * d[j][c];
                    }
                }
                __syncwarp();  // every lane has read the block
#pragma unroll
                for (int r = 0; r < B; ++r)
#pragma unroll
                    for (int j = 0; j < B; ++j)
                        if (lane == 0) a[r * n + jj * B + j] = skip[j] ? x[r][j] : m[r][j];
            }
            constexpr int U = 3;  // pivot-row entries a lane has in flight
            for (int e0 = 0; e0 < nu; e0 += 32 * U) {
                double v[U][B];
                int at[U];
#pragma unroll
                for (int k = 0; k < U; ++k) {
                    const int e = e0 + 32 * k + lane;
                    at[k] = -1;
                    if (e < nu) {
#pragma unroll
                        for (int j = 0; j < B; ++j) v[k][j] = __ldcg(u + (int64_t)j * lj + B + e);
                        const int K = col[dj + 1 + e / B], pos = lower_bound(bc, jj + 1, len, K);
                        if (pos < len && bc[pos] == K) at[k] = pos * B + e % B;
                    }
                }
#pragma unroll
                for (int k = 0; k < U; ++k)
                    if (at[k] >= 0) {
#pragma unroll
                        for (int r = 0; r < B; ++r) {
                            double w = a[r * n + at[k]];
#pragma unroll
                            for (int j = 0; j < B; ++j)
                                if (!skip[j]) w -= m[r][j] * v[k][j];
                            a[r * n + at[k]] = w;
                        }
                    }
            }
            __syncwarp();
        }
        // the block row's own pivots
        if (diag[I] >= 0) {
#pragma unroll
            for (int r = 1; r < B; ++r)
#pragma unroll
                for (int k = 0; k < r; ++k) {
                    const double piv = a[k * n + nl * B + k], x = a[r * n + nl * B + k];
                    __syncwarp();
                    if (piv == 0) {
                        if (lane == 0) atomicAdd(zero_pivots, 1);
                        continue;
                    }
                    const double q = x / piv;
                    if (lane == 0) a[r * n + nl * B + k] = q;
                    for (int e = nl * B + k + 1 + lane; e < n; e += 32) a[r * n + e] -= q * a[k * n + e];
                    __syncwarp();
                }
        }
        if (room)
            for (int i = lane; i < n * B; i += 32) g[i] = a[i];
        __syncwarp();
        if (lane == 0) {
            asm volatile("fence.acq_rel.gpu;" ::: "memory");
            asm volatile("st.relaxed.gpu.global.s32 [%0], 1;" ::"l"(done + I) : "memory");
        }
        __syncwarp();
    }
}

// Entries [e0, e1) of a block row's B rows (l, n entries each) times z, which is
// polled: sums over the warp in every lane.  False when a wait gave up.
template <int B>
__device__ __forceinline__ bool row_sums(const int32_t *__restrict__ bc, const double *__restrict__ l, int n, int e0,
                                         int e1, const double *z, double (&s)[B], const Waits &waits) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int r = 0; r < B; ++r) s[r] = 0;
    constexpr int U = 4;  // entries a lane has in flight
    for (int e = e0; e < e1; e += 32 * U) {
        double v[U][B], x[U];
        const double *at[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const int i = e + 32 * k + lane;
            at[k] = nullptr;
            x[k] = 0;
            if (i < e1) {
                at[k] = z + (int64_t)bc[i / B] * B + i % B;
#pragma unroll
                for (int r = 0; r < B; ++r) v[k][r] = l[(int64_t)r * n + i];
            }
        }
        long long spins = 0;
        for (bool all = false; !all;) {
            all = true;
#pragma unroll
            for (int k = 0; k < U; ++k)
                if (at[k]) x[k] = ld_relaxed(at[k]);
#pragma unroll
            for (int k = 0; k < U; ++k) all = all && !pending(x[k]);
            all = __all_sync(0xffffffffu, all);
            if (!all && !__all_sync(0xffffffffu, wait_on(spins, waits))) return false;
        }
#pragma unroll
        for (int k = 0; k < U; ++k)
            if (at[k]) {
#pragma unroll
                for (int r = 0; r < B; ++r) s[r] = fma(v[k][r], x[k], s[r]);
            }
    }
#pragma unroll
    for (int r = 0; r < B; ++r)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s[r] += __shfl_xor_sync(0xffffffffu, s[r], o);
    return true;
}

// z = U^-1 L^-1 rin: forward substitution with unit L (f_subst,
// ILUPreconditioner.hpp:201-221) into zf, then backward (b_subst, :226-253) into zb
// and z.  A row without a diagonal divides by its first entry, as the reference does,
// and reads columns below it as the forward substitution left them.
template <int B>
__global__ void __launch_bounds__(kThreads)
k_ilu_apply(int nbrows, const int32_t *__restrict__ lower, const int32_t *__restrict__ upper,
            const int32_t *__restrict__ rowptr, const int32_t *__restrict__ col, const int32_t *__restrict__ diag,
            const double *__restrict__ lu, const double *rin, double *zf, double *zb, double *z,
            const int32_t *__restrict__ flag, Waits waits) {
    if (flag && read_flag(flag)) return;
    const int lane = threadIdx.x & 31;
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    for (int t = w; t < nbrows; t += nw) {
        const int I = lower[t], b0 = rowptr[I], len = rowptr[I + 1] - b0, n = len * B;
        const bool has = diag[I] >= 0;
        const int nl = has ? diag[I] - b0 : lower_bound(col + b0, 0, len, I);
        const double *l = lu + (int64_t)b0 * B * B;
        double x[B], d[B][B], s[B];
#pragma unroll
        for (int r = 0; r < B; ++r) {
            x[r] = rin[(int64_t)I * B + r];
#pragma unroll
            for (int j = 0; j < r; ++j) d[r][j] = has ? l[r * n + nl * B + j] : 0.0;
        }
        if (!row_sums<B>(col + b0, l, n, 0, nl * B, zf, s, waits)) return;
#pragma unroll
        for (int r = 0; r < B; ++r) {
            x[r] -= s[r];
#pragma unroll
            for (int j = 0; j < r; ++j)
                if (has) x[r] -= d[r][j] * x[j];
            if (lane == r) st_relaxed(zf + (int64_t)I * B + r, x[r]);
        }
    }
    for (int t = w; t < nbrows; t += nw) {
        const int I = upper[t], b0 = rowptr[I], len = rowptr[I + 1] - b0, n = len * B;
        const bool has = diag[I] >= 0;
        const int nl = has ? diag[I] - b0 : lower_bound(col + b0, 0, len, I);
        const double *l = lu + (int64_t)b0 * B * B;
        double x[B], d[B][B], s[B];
#pragma unroll
        for (int r = 0; r < B; ++r)
#pragma unroll
            for (int j = r; j < B; ++j) d[r][j] = has ? l[r * n + nl * B + j] : (j == r && n > 0 ? l[r * n] : 0.0);
        // (without a diagonal every entry but the first, the divisor, counts)
        if (!row_sums<B>(col + b0, l, n, has ? (nl + 1) * B : max(nl * B, 1), n, zb, s, waits)) return;
        if (!has) {
            double f[B];
            if (!row_sums<B>(col + b0, l, n, 1, nl * B, zf, f, waits)) return;
#pragma unroll
            for (int r = 0; r < B; ++r) s[r] += f[r];
        }
        long long spins = 0;
        for (bool all = false; !all;) {
            all = true;
#pragma unroll
            for (int r = 0; r < B; ++r) {
                x[r] = ld_relaxed(zf + (int64_t)I * B + r);
                all = all && !pending(x[r]);
            }
            all = __all_sync(0xffffffffu, all);
            if (!all && !__all_sync(0xffffffffu, wait_on(spins, waits))) return;
        }
#pragma unroll
        for (int r = B - 1; r >= 0; --r) {
            double v = x[r] - s[r];
#pragma unroll
            for (int j = r + 1; j < B; ++j)
                if (has) v -= d[r][j] * x[j];
            x[r] = v / d[r][r];
            if (lane == r) {
                st_relaxed(zb + (int64_t)I * B + r, x[r]);
                z[(int64_t)I * B + r] = x[r];
            }
        }
    }
}

// (d_tmp: the factorization's count of zero pivots, then the abort word)
static Waits waits_of(yg_precond M) { return {M->ctx->wait_polls, reinterpret_cast<int32_t *>(M->d_tmp) + 1, M->ctx->d_err}; }

template <int B>
static yg_status ilu_factor(yg_precond M, int32_t *done, int *zeros) {
    yg_matrix A = M->A;
    yg_context ctx = A->ctx;
    YG_TRY(matrix_row_extent(A));
    // the rows in shared memory, as many warps as fit; longer rows are updated in place
    int room = (int)std::min<int64_t>((int64_t)A->row_max * B * B + (A->row_max + 1) / 2, 1 << 20);
    int warps = (int)std::min<int64_t>(kThreads / 32, (int64_t)ctx->smem_optin / std::max(8 * room, 1));
    if (warps < 1) { room = 0; warps = kThreads / 32; }
    const int smem = 8 * room * warps;
    int nb = (int)A->nbrows;
    auto kern = k_ilu_factor<B>;
    YG_TRY(allow_all_smem(ctx, reinterpret_cast<const void *>(kern)));
    Waits waits = waits_of(M);
    void *args[] = {&nb, &M->d_lower_rows, &A->d_rowptr, &A->d_col, &A->d_diag, &M->d_lu, &done, &zeros, &room, &waits};
    return launch_cooperative(ctx, reinterpret_cast<const void *>(kern), std::min(ctx->num_sms, (nb + warps - 1) / warps), 32 * warps,
                              (size_t)smem, args);
}

// (flag: set when the solver that captured the apply has stopped)
static yg_status ilu_apply(yg_precond M, const double *r, double *z, const int32_t *flag) {
    yg_matrix A = M->A;
    yg_context ctx = A->ctx;
    const int64_t n = A->rows();
    if (n == 0) return YG_OK;
    double *zf = M->d_z, *zb = M->d_z + n;
    Waits waits = waits_of(M);
    k_fill_pending<<<stream_grid(ctx, 2 * n), kThreads, 0, ctx->stream>>>(2 * n, M->d_z, waits.abort);
    YG_LAUNCHED(ctx);
    int nb = (int)A->nbrows;
    void *args[] = {&nb, &M->d_lower_rows, &M->d_upper_rows, &A->d_rowptr, &A->d_col, &A->d_diag, &M->d_lu, &r, &zf, &zb, &z,
                    &flag, &waits};
    const void *kern = nullptr;
    switch (A->block) {
    case 1: kern = reinterpret_cast<const void *>(&k_ilu_apply<1>); break;
    case 2: kern = reinterpret_cast<const void *>(&k_ilu_apply<2>); break;
    case 3: kern = reinterpret_cast<const void *>(&k_ilu_apply<3>); break;
    case 4: kern = reinterpret_cast<const void *>(&k_ilu_apply<4>); break;
    case 5: kern = reinterpret_cast<const void *>(&k_ilu_apply<5>); break;
    case 6: kern = reinterpret_cast<const void *>(&k_ilu_apply<6>); break;
    case 7: kern = reinterpret_cast<const void *>(&k_ilu_apply<7>); break;
    default: kern = reinterpret_cast<const void *>(&k_ilu_apply<8>); break;
    }
    const int grid = (int)std::min<int64_t>(ctx->num_sms, (nb + kThreads / 32 - 1) / (kThreads / 32));
    YG_TRY(launch_cooperative(ctx, kern, grid, kThreads, 0, args));
    YG_CUDA(cudaGetLastError());
    return YG_OK;
}

static yg_status build_ilu(yg_precond M) {
    yg_matrix A = M->A;
    yg_context ctx = A->ctx;
    const int B = A->block;
    const int64_t n = A->rows(), nb = A->nbrows;
    const int64_t nnz = A->nnzb * B * B;
    if (nnz >= INT32_MAX) return fail(YG_UNSUPPORTED, "ILU(0): too many entries for 32-bit indices");
    if (nb == 0) return YG_OK;
    cudaStream_t st = ctx->stream;
    YG_TRY(dev_alloc_t(ctx, &M->d_lu, nnz));
    YG_TRY(dev_alloc_t(ctx, &M->d_z, 2 * n));
    YG_TRY(dev_alloc_t(ctx, &M->d_tmp, 1));
    YG_TRY(dev_alloc_t(ctx, &M->d_lower_rows, nb));
    YG_TRY(dev_alloc_t(ctx, &M->d_upper_rows, nb));
    k_ilu_expand<<<stream_grid(ctx, nb * 32), kThreads, 0, st>>>(nb, B, A->d_rowptr, A->d_val, M->d_lu);
    YG_LAUNCHED(ctx);
    YG_CUDA(cudaGetLastError());
    // dependency levels on the host: a block row's first scalar row comes one level
    // after the last of the block rows it reads, its other rows one by one behind
    std::vector<int32_t> rp(nb + 1), col(A->nnzb + 1), diag(nb), lev(nb);
    YG_CUDA(cudaMemcpyAsync(rp.data(), A->d_rowptr, sizeof(int32_t) * (nb + 1), cudaMemcpyDeviceToHost, st));
    YG_CUDA(cudaMemcpyAsync(col.data(), A->d_col, sizeof(int32_t) * A->nnzb, cudaMemcpyDeviceToHost, st));
    YG_CUDA(cudaMemcpyAsync(diag.data(), A->d_diag, sizeof(int32_t) * nb, cudaMemcpyDeviceToHost, st));
    YG_CUDA(cudaStreamSynchronize(st));
    std::vector<int32_t> rows(nb), ptr;
    auto sorted = [&](int64_t levels) {  // block rows by level, then by index
        ptr.assign(levels + 1, 0);
        for (int64_t i = 0; i < nb; ++i) ptr[lev[i] + 1]++;
        for (int64_t l = 0; l < levels; ++l) ptr[l + 1] += ptr[l];
        for (int64_t i = 0; i < nb; ++i) rows[ptr[lev[i]]++] = (int32_t)i;
    };
    auto last = [&](int64_t i) { return lev[i] + (diag[i] >= 0 ? B - 1 : 0); };
    int32_t top = 0;
    for (int64_t i = 0; i < nb; ++i) {
        int32_t l = 0;
        for (int32_t k = rp[i]; k < rp[i + 1] && col[k] < i; ++k) l = std::max(l, last(col[k]) + 1);
        lev[i] = l;
        top = std::max(top, last(i));
    }
    M->lower_levels = top + 1;
    sorted(M->lower_levels);
    YG_CUDA(cudaMemcpyAsync(M->d_lower_rows, rows.data(), sizeof(int32_t) * nb, cudaMemcpyHostToDevice, st));
    YG_CUDA(cudaStreamSynchronize(st));
    // factor while the host sorts the backward levels
    int32_t *done = reinterpret_cast<int32_t *>(M->d_z);
    int *d_zero = reinterpret_cast<int *>(M->d_tmp);
    YG_CUDA(cudaMemsetAsync(done, 0, sizeof(int32_t) * nb, st));
    YG_CUDA(cudaMemsetAsync(d_zero, 0, 2 * sizeof(int), st));  // (and the abort word)
    switch (B) {
    case 1: YG_TRY(ilu_factor<1>(M, done, d_zero)); break;
    case 2: YG_TRY(ilu_factor<2>(M, done, d_zero)); break;
    case 3: YG_TRY(ilu_factor<3>(M, done, d_zero)); break;
    case 4: YG_TRY(ilu_factor<4>(M, done, d_zero)); break;
    case 5: YG_TRY(ilu_factor<5>(M, done, d_zero)); break;
    case 6: YG_TRY(ilu_factor<6>(M, done, d_zero)); break;
    case 7: YG_TRY(ilu_factor<7>(M, done, d_zero)); break;
    default: YG_TRY(ilu_factor<8>(M, done, d_zero)); break;
    }
    top = 0;
    for (int64_t i = nb - 1; i >= 0; --i) {
        int32_t l = 0;
        for (int32_t k = rp[i + 1] - 1; k >= rp[i] && col[k] > i; --k) l = std::max(l, last(col[k]) + 1);
        lev[i] = l;
        top = std::max(top, last(i));
    }
    M->upper_levels = top + 1;
    sorted(M->upper_levels);
    YG_CUDA(cudaMemcpyAsync(M->d_upper_rows, rows.data(), sizeof(int32_t) * nb, cudaMemcpyHostToDevice, st));
    int zeros = 0;
    YG_CUDA(cudaMemcpyAsync(&zeros, d_zero, sizeof(int), cudaMemcpyDeviceToHost, st));
    YG_CUDA(cudaStreamSynchronize(st));
    M->zero_pivots = zeros;
    return check_device_error(ctx);
}

yg_status precond_apply_dev(yg_precond M, const double *r, double *z, const int32_t *flag) {
    yg_context ctx = M->A->ctx;
    cudaStream_t st = ctx->stream;
    const int64_t n = M->A->rows();
    if (M->kind == YG_PRECOND_IDENTITY) {
        if (z != r) YG_CUDA(cudaMemcpyAsync(z, r, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
        return YG_OK;
    }
    if (M->kind == YG_PRECOND_JACOBI) {
        k_jacobi_apply<<<stream_grid(ctx, n), kThreads, 0, st>>>(n, M->d_dinv, r, z);
        YG_LAUNCHED(ctx);
        return YG_OK;
    }
    return ilu_apply(M, r, z, flag);
}

bool precond_fusable(yg_precond M) { return !M || M->kind == YG_PRECOND_IDENTITY || M->kind == YG_PRECOND_JACOBI; }
const double *precond_dinv(yg_precond M) { return (M && M->kind == YG_PRECOND_JACOBI) ? M->d_dinv : nullptr; }

}  // namespace yg

using namespace yg;

extern "C" yg_status yg_precond_create(yg_matrix A, int32_t kind, yg_precond *out) {
    if (!A || !out) return fail(YG_BAD_ARG, "yg_precond_create: NULL argument");
    Beside beside(A->ctx, Beside::kStreams);
    if (A->rows() != A->cols()) return fail(YG_BAD_ARG, "preconditioner needs a square matrix");
    *out = nullptr;
    auto *M = new yg_precond_t();
    M->A = A;
    M->ctx = A->ctx;
    M->kind = kind;
    yg_context ctx = A->ctx;
    yg_status s = YG_OK;
    if (kind == YG_PRECOND_JACOBI) {
        const int64_t n = A->rows();
        if ((s = dev_alloc_t(ctx, &M->d_dinv, n)) == YG_OK && (s = dev_alloc_t(ctx, &M->d_tmp, 1)) == YG_OK) {
            int *d_zero = reinterpret_cast<int *>(M->d_tmp);
            cudaMemsetAsync(d_zero, 0, sizeof(int), ctx->stream);
            k_jacobi_build<<<stream_grid(ctx, n), kThreads, 0, ctx->stream>>>(A->nbrows, A->block, A->d_diag, A->d_val,
                                                                             M->d_dinv, d_zero);
            YG_LAUNCHED(ctx);
            int zeros = 0;
            cudaMemcpyAsync(&zeros, d_zero, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream);
            cudaError_t e = cudaStreamSynchronize(ctx->stream);
            if (e != cudaSuccess) s = fail(YG_CUDA_ERROR, "Jacobi build: %s", cudaGetErrorString(e));
            M->zero_pivots = zeros;
        }
    } else if (kind == YG_PRECOND_ILU0) {
        s = build_ilu(M);
    } else if (kind != YG_PRECOND_IDENTITY) {
        s = fail(YG_BAD_ARG, "unknown preconditioner kind %d", kind);
    }
    if (s != YG_OK) { yg_precond_destroy(M); return s; }
    *out = M;
    return YG_OK;
}

extern "C" yg_status yg_precond_apply(yg_precond M, yg_vector z) {
    if (!M || !z || z->n != M->A->rows()) return fail(YG_BAD_ARG, "yg_precond_apply: size mismatch");
    return precond_apply_dev(M, z->d, z->d, nullptr);
}

extern "C" yg_status yg_precond_destroy(yg_precond M) {
    if (!M) return YG_OK;
    yg_context ctx = M->ctx;
    for (void *p : {(void *)M->d_dinv, (void *)M->d_lu, (void *)M->d_lower_rows, (void *)M->d_upper_rows, (void *)M->d_z,
                    (void *)M->d_tmp})
        dev_free(ctx, p);
    delete M;
    return YG_OK;
}

extern "C" int64_t yg_precond_zero_pivots(yg_precond M) { return M ? M->zero_pivots : -1; }

extern "C" yg_status yg_precond_levels(yg_precond M, int64_t *lower, int64_t *upper) {
    if (!M || !lower || !upper) return fail(YG_BAD_ARG, "yg_precond_levels: NULL argument");
    *lower = M->lower_levels;
    *upper = M->upper_levels;
    return YG_OK;
}
