// resident.cuh -- Jacobi-PCG iterations of a system held in the shared memory of a
// group of CTAs: the device code shared by the kernel that gives all CTAs to one
// system (pcg_resident.cu) and the one that gives a group of CTAs to each of many
// systems (batch.cu).
#pragma once
#include "internal.h"
#include "device_common.cuh"

#include <algorithm>
#include <cmath>

namespace yg {
namespace resident {

enum { FLAG_RUN = 0, FLAG_CONVERGED = 1, FLAG_BREAKDOWN = 2, FLAG_NAN = 3, FLAG_MAXITER = 4 };

constexpr long long kGridSpinLimit = 1ll << 22;  // polls of one grid-wide sum (seconds; a sum takes microseconds)

struct alignas(32) SumSlot {
    unsigned long long w[4];  // low and high halves of two doubles, each below the sum's number
};

// Blocks of a row that a lane gathers at a time: a round costs a trip to L2 whatever
// their number, and there are rows x lanes / threads rounds.  Against 4, 2 and 2 (us an
// iteration): 40,401 unknowns of Q1 8.2 -> 7.6, of Q2 8.9 -> 9.5, 44,521 of Q3 11.7 -> 11.3,
// 45,602 of order-3 plane elasticity 13.3 -> 12.6; batches of 24 systems 47.7 -> 40.4 and 93.5 -> 88.6 ms (39.8
// and 94.0 with 6, 3 and 2).
constexpr int gathers(int B) { return B == 1 ? 8 : (B == 2 ? 4 : 2); }

// A row of more than kLongRounds rounds of its lanes is left to a whole warp: with the
// 2 lanes that suit a mean of 7 entries, a row of 1,000 took 62 rounds while all others
// waited (us an iteration, streaming kernels / lanes by the mean / a warp for a long row:
// 5,000 unknowns with a row of 1,000 21 / 32 / 12, with one of 4,000 34 / 108 / 19; 40,000 with one of
// 15,000 84 / 406 / 67).  Kernels of their own (LONG) do so: with the second pass, and the
// lanes that change between them, in the loop of all systems a solve of 4,225 unknowns
// without long rows took 1.62 ms instead of 1.54, a batch of 24 systems 43.1 instead of 40.4.
constexpr int kLongRounds = 4;
// Long rows of a CTA at most: a row longer than kLongRounds * lanes * gathers(B) blocks fills 512
// bytes of its shared memory or more.
constexpr int kLongRows = 512;

struct System {
    int nbrows;
    const int32_t *rowptr, *col;
    const void *val;
    const double *corr, *dinv;
    double *x, *r, *p;
    double *zp;              // z and p for the other CTAs: per block row B entries of each
    double *z;               // or (SPLIT) z here and p in p, no memory beside the vectors
    SumSlot *slots;          // two per CTA of the group, `stride` apart
    int stride;
    int64_t block_cost, row_cost, total_cost;  // shared memory bytes per block, per block row, of all
    int lanes;               // lanes per block row
    int long_row;            // LONG: rows of more blocks are long
};
struct State {
    double tol, bb, rz0;
    int64_t maxiter;
    int criterion;
    int max_its, check;      // iterations at most; residual replacement is looked at every `check`
    double rr_replace;       // replace r by b - A x when r.r < rr_replace at such a point (0: never; FP32 values only)
    const double *val64, *b; // from these
    int replaced;            // how often; rr_replace follows the residual
    int64_t iter;            // these three are updated
    double rz, rr;
    bool timed_out;
};

__device__ __forceinline__ double warp_sum_all(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sums over all threads of the group's G CTAs of v0 and v1, the same bits in every block.
// PUBLISH: what the block's threads wrote to global memory before is visible to
// the CTAs that return.  False when the poll gave up.
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
__device__ bool group_sum(SumSlot *slots, int rank, int G, unsigned epoch, double v0, double v1, double &o0, double &o1) {
    __shared__ double part[2][32];
    __shared__ double total[3];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
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
            if (G > 1) put_sums(slots + rank, epoch, s0, s1, TWO);
        }
        double a0 = s0, a1 = s1;
        bool ok = G == 1;
        if (G > 1) {
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
                if (spins > 4096) __nanosleep(1000);  // a CTA of the group is still at another system
            }
            a0 = warp_sum_all(a0);
            if (TWO) a1 = warp_sum_all(a1);
            if (PUBLISH) fence_gpu();
        }
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
__device__ inline int first_row(const int32_t *rowptr, int n, int64_t block_cost, int64_t row_cost, int64_t target) {
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

// Iterations of one system by CTA `rank` of the group's G (the same state in all of
// them; S is one for all threads or one for each, read before the first sum and written
// after the last); x, r and, when the flag returned is FLAG_RUN, p are written back.
template <int B, typename VT, bool SPLIT, bool LONG>
__device__ __forceinline__ int pcg_run(const System &a, int rank, int G, State &S, unsigned char *smem) {
    constexpr int B2 = B * B;
    __shared__ int bounds[2], nlong;
    const int tid = threadIdx.x, nt = blockDim.x;
    if (LONG && tid == 0) nlong = 0;
    if (tid < 64) {
        const int64_t t = rank + (tid >> 5);
        const int r = t == G ? a.nbrows : first_row(a.rowptr, a.nbrows, a.block_cost, a.row_cost, t * a.total_cost / G);
        if ((tid & 31) == 0) bounds[tid >> 5] = r;
    }
    __syncthreads();
    const int r0 = bounds[0], nr = bounds[1] - r0, nd = nr * B;
    const int e0 = a.rowptr[r0], nb = a.rowptr[bounds[1]] - e0;
    // shared memory: values | columns | row pointers | x, r, p, q (z after the update), dinv, correction | long rows
    auto up = [](size_t v) { return (v + 15) & ~(size_t)15; };
    VT *val = reinterpret_cast<VT *>(smem);
    int32_t *col = reinterpret_cast<int32_t *>(smem + up((size_t)nb * B2 * sizeof(VT)));
    int32_t *rp = reinterpret_cast<int32_t *>(reinterpret_cast<unsigned char *>(col) + up((size_t)nb * 4));
    double *x = reinterpret_cast<double *>(reinterpret_cast<unsigned char *>(rp) + up((size_t)(nr + 1) * 4));
    double *r = x + nd, *p = r + nd, *q = p + nd, *dinv = q + nd;
    double *corr = dinv + (a.dinv ? nd : 0);
    unsigned short *longs = reinterpret_cast<unsigned short *>(corr + (a.corr ? nr * B2 : 0));
    const VT *gval = static_cast<const VT *>(a.val) + (int64_t)e0 * B2;
    for (int i = tid; i < nb * B2; i += nt) val[i] = gval[i];
    for (int i = tid; i < nb; i += nt) col[i] = a.col[e0 + i];
    for (int i = tid; i <= nr; i += nt) rp[i] = a.rowptr[r0 + i] - e0;
    if (a.corr)
        for (int i = tid; i < nr * B2; i += nt) corr[i] = a.corr[(int64_t)r0 * B2 + i];
    auto publish = [&](int i, double zi, double pi) {  // entry i of this CTA's
        if (SPLIT) {
            a.z[(int64_t)r0 * B + i] = zi;
            a.p[(int64_t)r0 * B + i] = pi;
        } else {
            const int row = i / B, c = i - row * B;
            double *zp = a.zp + (int64_t)(r0 + row) * 2 * B + c;
            zp[0] = zi;
            zp[B] = pi;
        }
    };
    for (int i = tid; i < nd; i += nt) {
        const int64_t g = (int64_t)r0 * B + i;
        x[i] = a.x[g];
        r[i] = a.r[g];
        if (a.dinv) dinv[i] = a.dinv[g];
        // the direction of the first iteration, as z with beta = 0
        const double v = a.p[g];
        p[i] = 0;
        q[i] = v;
        publish(i, v, 0.0);
    }
    if (LONG) {
        __syncthreads();
        if (tid < 32) {
            int n = 0;
            for (int i0 = 0; i0 < nr; i0 += 32) {
                const bool is = i0 + tid < nr && rp[i0 + tid + 1] - rp[i0 + tid] > a.long_row;
                const unsigned m = __ballot_sync(0xffffffffu, is);
                if (is) longs[n + __popc(m & ((1u << tid) - 1))] = (unsigned short)(i0 + tid);
                n += __popc(m);
            }
            if (tid == 0) nlong = n;
        }
    }
    const double tol = S.tol, bb = S.bb, rz0 = S.rz0;
    int64_t iter = S.iter;
    double rz = S.rz, rr = S.rr, beta = 0, rr_replace = S.rr_replace;
    int replaced = 0;
    unsigned epoch = 1;
    int flag = FLAG_RUN;
    double t0, t1;
    bool ok = group_sum<false, true>(a.slots + a.stride, rank, G, epoch, 0, 0, t0, t1);
    // products: `lanes` lanes a row, then a warp for each long row
    constexpr int passes = LONG ? 2 : 1;
    const int L0 = a.lanes, group0 = tid / L0, ngroups0 = nt / L0;
    for (int it = 0; ok; ++it) {
        for (int i = tid; i < nd; i += nt) p[i] = fma(beta, p[i], q[i]);
        __syncthreads();  // p is read and q overwritten by other threads
        double pq = 0;
#pragma unroll 1
        for (int pass = 0; pass < passes; ++pass) {
            const bool second = LONG && pass;
            const int L = second ? 32 : L0, lane = tid & (L - 1), count = second ? nlong : nr;
            const int group = second ? tid >> 5 : group0, ngroups = second ? nt >> 5 : ngroups0;
            for (int rb = 0; rb < count; rb += ngroups) {  // the lanes of a warp take the same steps
                int row = rb + group;
                bool on = row < count;
                if (second && on) row = longs[row];
                const int js = on ? rp[row] : 0, je = on ? rp[row + 1] : 0;
                if (LONG && !second) on = on && je - js <= a.long_row;
                double acc[B];
#pragma unroll
                for (int i = 0; i < B; ++i) acc[i] = 0;
                if (on) {
                    constexpr int U = gathers(B);
                    for (int j0 = js + lane; j0 < je; j0 += U * L) {
                        double v[U][2 * B];
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            const int j = j0 + u * L;
                            if (j < je) {
                                if (!SPLIT || B == 2) {
                                    const double *z = SPLIT ? a.z + (int64_t)col[j] * B : a.zp + (int64_t)col[j] * 2 * B;
                                    const double *p2 = SPLIT ? a.p + (int64_t)col[j] * B : z + B;
#pragma unroll
                                    for (int k = 0; k < B; ++k) {
                                        const double2 d = reinterpret_cast<const double2 *>(SPLIT && k ? p2 : z)[SPLIT ? 0 : k];
                                        v[u][2 * k] = d.x;
                                        v[u][2 * k + 1] = d.y;
                                    }
                                } else {
#pragma unroll
                                    for (int k = 0; k < B; ++k) {
                                        v[u][k] = a.z[(int64_t)col[j] * B + k];
                                        v[u][B + k] = a.p[(int64_t)col[j] * B + k];
                                    }
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
                if (on && lane == 0) {
                    if (a.corr) add_corr<B>(corr, p, row, acc);
#pragma unroll
                    for (int i = 0; i < B; ++i) {
                        q[row * B + i] = acc[i];
                        pq = fma(acc[i], p[row * B + i], pq);
                    }
                }
            }
        }
        ++epoch;
        if (!(ok = group_sum<false, false>(a.slots, rank, G, epoch, pq, 0, pq, t1))) break;
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
            publish(i, zi, pi);
        }
        double rz_new;
        if (!(ok = group_sum<true, true>(a.slots + a.stride, rank, G, epoch, srz, srr, rz_new, rr))) break;
        ++iter;
        const bool conv = S.criterion == YG_CRIT_REFERENCE ? rz_new / rz0 < tol : sqrt(rr) <= tol * sqrt(bb);
        if (conv) flag = FLAG_CONVERGED;
        if (!isfinite(rz_new)) flag = FLAG_NAN;
        if (flag == FLAG_RUN && iter >= S.maxiter) flag = FLAG_MAXITER;
        beta = rz_new / rz;
        rz = rz_new;
        // (a slot is written again only after a sum in the other half: all have read it)
        const bool due = flag == FLAG_RUN && (it + 1) % S.check == 0 && rr < rr_replace;
        if (sizeof(VT) == 4 && due) {
            // r = b - A x from the FP64 values; the sums keep alternating between the slots
            for (int i = tid; i < nd; i += nt) a.x[(int64_t)r0 * B + i] = x[i];
            ++epoch;
            if (!(ok = group_sum<false, true>(a.slots, rank, G, epoch, 0, 0, t0, t1))) break;
            srz = srr = 0;
#pragma unroll 1
            for (int pass = 0; pass < passes; ++pass) {
                const bool second = LONG && pass;
                const int L = second ? 32 : L0, lane = tid & (L - 1), count = second ? nlong : nr;
                const int group = second ? tid >> 5 : group0, ngroups = second ? nt >> 5 : ngroups0;
                for (int rb = 0; rb < count; rb += ngroups) {
                    int row = rb + group;
                    bool on = row < count;
                    if (second && on) row = longs[row];
                    const int js = on ? rp[row] : 0, je = on ? rp[row + 1] : 0;
                    if (LONG && !second) on = on && je - js <= a.long_row;
                    double acc[B];
#pragma unroll
                    for (int i = 0; i < B; ++i) acc[i] = 0;
                    if (on) {
                        for (int j = js + lane; j < je; j += L) {
                            const double *v = S.val64 + (int64_t)(e0 + j) * B2, *xc = a.x + (int64_t)col[j] * B;
#pragma unroll
                            for (int c = 0; c < B; ++c)
#pragma unroll
                                for (int i = 0; i < B; ++i) acc[i] = fma(v[i * B + c], xc[c], acc[i]);
                        }
                    }
#pragma unroll
                    for (int i = 0; i < B; ++i)
                        for (int o = L >> 1; o > 0; o >>= 1) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
                    if (on && lane == 0) {
#pragma unroll
                        for (int i = 0; i < B; ++i) {
                            const double ri = S.b[(int64_t)(r0 + row) * B + i] - acc[i];
                            r[row * B + i] = ri;
                            srz += ri * (a.dinv ? dinv[row * B + i] * ri : ri);
                            srr += ri * ri;
                        }
                    }
                }
            }
            if (!(ok = group_sum<true, false>(a.slots + a.stride, rank, G, epoch, srz, srr, rz, rr))) break;
            rr_replace = 1e-2 * rr;
            ++replaced;
            if (it + 1 >= S.max_its) break;
        } else if (flag != FLAG_RUN || it + 1 >= S.max_its) {
            break;
        }
    }
    if (!ok) flag = FLAG_NAN;
    for (int i = tid; i < nd; i += nt) {
        const int64_t g = (int64_t)r0 * B + i;
        a.x[g] = x[i];
        a.r[g] = r[i];
        if (flag == FLAG_RUN) a.p[g] = fma(beta, p[i], q[i]);  // the next direction
    }
    S.iter = iter;
    S.rz = rz;
    S.rr = rr;
    S.rr_replace = rr_replace;
    S.replaced = replaced;
    S.timed_out = !ok;
    return flag;
}

// Shared memory per block (values, column) and per block row (row pointer, x, r,
// p, q, dinv, correction) of a resident solve.
inline void costs(int B, bool f32, bool corr, bool jacobi, int64_t *block, int64_t *row) {
    *block = (f32 ? 4 : 8) * B * B + 4;
    *row = 4 + 8 * B * (jacobi ? 5 : 4) + (corr ? 8 * B * B : 0);
}

// Shared memory of the largest share among G CTAs: at most the mean and one row more, and
// the list of long rows where there can be any.
inline int64_t share(int B, int64_t total_cost, int64_t row_max, int64_t block_cost, int64_t row_cost, int G) {
    const int64_t list = row_max > kLongRounds * 2 * gathers(B) ? sizeof(unsigned short) * kLongRows : 0;
    return (total_cost + G - 1) / G + row_max * block_cost + row_cost + 256 + list;
}

// The row length above which a row takes a warp, and whether a system has such rows.
inline int long_row(int B, int lanes) { return kLongRounds * lanes * gathers(B); }
inline bool has_long_rows(int B, int lanes, int64_t row_max) { return lanes < 32 && row_max > long_row(B, lanes); }

// Lanes per block row: one round of gathers each, more where the threads allow.
inline int row_lanes(int B, double mean, int64_t rows, int threads) {
    int L = 2;
    while (L < 32 && L * gathers(B) < mean) L *= 2;
    while (L < 32 && L < mean && rows * 2 * L <= threads) L *= 2;
    return L;
}

}  // namespace resident
}  // namespace yg
