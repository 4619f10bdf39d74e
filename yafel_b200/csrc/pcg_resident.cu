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
// Measured (us an iteration, before -> now): 4,225 unknowns of Q1 Poisson 14.9 -> 4.8;
// 30,258 unknowns of order-2 plane elasticity 15.8 -> 9.0; 10,125 unknowns of Q2
// elasticity 17 -> 11.8.  The trips through L2 of the two sums bound it: a matrix
// this size takes 1-4 us from shared memory.
// A mixed-precision solve replaces its residual inside the kernel too (4,225 unknowns:
// 1.97 -> 1.66 ms a solve of 295 iterations and 8 replacements).
// Polls are bounded: a block that gives up records YG_TIMEOUT and returns, and so
// do the others.
#include "resident.cuh"

namespace yg {

using namespace resident;

constexpr int kMaxSumBlocks = 256;
constexpr int kStaticSmem = 3072;  // shared memory left to the kernel's static arrays and the runtime

struct ResidentArgs {
    System sys;
    KrylovScalars *S;
    int32_t *err;
    int max_its, check;
    double rr_replace;
    const double *val64, *b;  // what a residual is replaced from
};

template <int B, typename VT, bool LONG>
__global__ void __launch_bounds__(512, 1) k_pcg_resident(ResidentArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    KrylovScalars *S = a.S;
    if (read_flag(&S->flag)) return;  // set before the launch: the same for every block
    State st{S->tol, S->bb, S->rz0, S->maxiter, S->criterion, a.max_its, a.check, a.rr_replace, a.val64, a.b, 0, S->iter, S->rz[0], S->rr, false};
    const int flag = pcg_run<B, VT, false, LONG>(a.sys, blockIdx.x, gridDim.x, st, smem);
    if (threadIdx.x == 0) {
        if (st.timed_out) atomicExch(a.err, (int32_t)YG_TIMEOUT);
        if (blockIdx.x == 0) {
            S->rz[0] = S->rz[1] = st.rz;
            S->rr = st.rr;
            S->iter = S->iter_seen = st.iter;
            S->replaced = st.replaced;
            S->rr_replace = st.rr_replace;
            S->flag = flag;
        }
    }
}

template <int B, typename VT>
static const void *resident_kernel(bool long_rows) {
    return long_rows ? reinterpret_cast<const void *>(&k_pcg_resident<B, VT, true>)
                     : reinterpret_cast<const void *>(&k_pcg_resident<B, VT, false>);
}
static const void *resident_kernel(int B, bool f32, bool long_rows) {
    if (B == 1) return f32 ? resident_kernel<1, float>(long_rows) : resident_kernel<1, double>(long_rows);
    if (B == 2) return f32 ? resident_kernel<2, float>(long_rows) : resident_kernel<2, double>(long_rows);
    return f32 ? resident_kernel<3, float>(long_rows) : resident_kernel<3, double>(long_rows);
}

static void resident_costs(yg_matrix A, bool f32, bool jacobi, int64_t *block, int64_t *row) {
    costs(A->block, f32, f32 && A->d_corr32, jacobi, block, row);
}

// Shared memory of the largest share among G blocks.
static int64_t resident_smem(yg_matrix A, bool f32, bool jacobi, int G) {
    int64_t bc, rc;
    resident_costs(A, f32, jacobi, &bc, &rc);
    return share(A->block, A->nnzb * bc + A->nbrows * rc, A->row_max, bc, rc, G);
}

// Blocks of a resident solve, one per SM at most.  The two sums cost 4.5 us + 0.028 us
// per block (5.0 us an iteration of 882 unknowns on 32 blocks, 5.4 on 64, 6.6 on 96,
// 8.9 on 148: every block polls every other's words) and the products 0.52 ns per CSR
// entry, 0.27 ns per entry of a block, divided by the blocks (40,401 unknowns, 361,201
// entries: 10.7 us on 32, 8.3 on 64, 8.4 on 96, 10.0 on 148), so the best number grows
// with the square root of the entries; the shared memory sets a lower bound.  Solves of
// several contexts run side by side as far as their blocks fit the SMs (solves a second
// with 1, 2, 4, 8 threads, streaming iterations -> these: 4,225 unknowns 201, 322, 458, 490 ->
// 527, 1007, 2000, 2359; 30,258 of order-2 plane elasticity 32, 49, 62, 58 -> 53 whatever the
// threads; 150,000 of order-2 Poisson 15, 22, 27, 26 -> 22).  Half the SMs for the second
// would let two run at once, 102 a second, but a solve alone takes 1.9 % longer.
int pcg_resident_blocks(yg_matrix A, bool f32, bool jacobi) {
    yg_context ctx = A->ctx;
    const double entries = (double)A->nnzb * A->block * A->block;
    const int most = (int)std::min<int64_t>(ctx->num_sms, A->nbrows);
    int G = (int)std::max(16.0, (A->block == 1 ? 0.136 : 0.098) * std::sqrt(entries));
    while (G < most && resident_smem(A, f32, jacobi, G) > (int64_t)ctx->smem_optin - kStaticSmem) G += 4;
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
    const int64_t total = A->nnzb * bc + A->nbrows * rc, room = (int64_t)ctx->smem_optin - kStaticSmem;
    if (total / ctx->num_sms > room) return YG_OK;
    YG_TRY(matrix_row_extent(A));
    *fits = resident_smem(A, f32, jacobi, pcg_resident_blocks(A, f32, jacobi)) <= room;
    return YG_OK;
}

// One launch of at most max_its iterations on the state pcg_core keeps (x, r, p and
// the scalars; zp: 2 n doubles of scratch).
yg_status pcg_resident_launch(yg_matrix A, bool f32, const double *dinv, const double *b, double *x, double *r,
                              double *p, double *zp, int max_its, int check, double rr_replace) {
    yg_context ctx = A->ctx;
    ResidentArgs a;
    System &m = a.sys;
    m.nbrows = (int)A->nbrows;
    m.rowptr = A->d_rowptr;
    m.col = A->d_col;
    m.val = f32 ? static_cast<const void *>(A->d_val32) : A->d_val;
    m.corr = f32 ? A->d_corr32 : nullptr;
    m.dinv = dinv;
    m.x = x;
    m.r = r;
    m.p = p;
    m.zp = zp;
    m.z = nullptr;
    m.slots = reinterpret_cast<SumSlot *>(ctx->d_slots);
    m.stride = kMaxSumBlocks;
    resident_costs(A, f32, dinv != nullptr, &m.block_cost, &m.row_cost);
    m.total_cost = A->nnzb * m.block_cost + A->nbrows * m.row_cost;
    a.S = ctx->d_scalars;
    a.err = ctx->d_err;
    a.max_its = max_its;
    a.check = check;
    a.rr_replace = rr_replace;
    a.val64 = A->d_val;
    a.b = b;
    const int G = pcg_resident_blocks(A, f32, dinv != nullptr);
    const double mean = (double)A->nnzb / A->nbrows;
    const int64_t rows = (A->nbrows + G - 1) / G;
    const int threads = rows * (mean > 8 ? 8 : 4) > 512 ? 512 : 256;
    m.lanes = row_lanes(A->block, mean, rows, threads);
    m.long_row = long_row(A->block, m.lanes);
    const size_t smem = (size_t)resident_smem(A, f32, dinv != nullptr, G);
    const void *kern = resident_kernel(A->block, f32, has_long_rows(A->block, m.lanes, A->row_max));
    YG_TRY(allow_all_smem(ctx, kern, kStaticSmem));
    YG_CUDA(cudaMemsetAsync(ctx->d_slots, 0, sizeof(SumSlot) * 2 * kMaxSumBlocks, ctx->stream));
    void *args[] = {&a};
    return launch_cooperative(ctx, kern, G, threads, smem, args);
}

}  // namespace yg
