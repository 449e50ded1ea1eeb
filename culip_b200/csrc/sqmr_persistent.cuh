// Persistent SQMR: the whole preconditioned solve in one cooperative launch.
//
// Same recurrence and lagged convergence check as SQMR<T>::solve
// (libs/la/iterative_solvers/sqmr.impl.cuh:109-355) with the block-iLDL^T
// split preconditioner (solve_left / solve_middle / solve_right,
// libs/la/preconditioner/block_ildlt.impl.cuh:183-246).  Where the reference
// issues ~35 launches per iteration (cuBLAS BLAS-1, single-thread scalar
// kernels, per-level sweep kernels, cuSPARSE csrmv), one iteration here is
// three groups of phases separated by grid-wide barriers.  A phase is a set
// of work items, one warp per block row and one lane per fine row, plus
// coalesced loops over whole vectors:
//
//   P1  v+ = Av - alpha v - beta v- (kept unscaled) and ||v+||^2 over all
//       rows; the first U-sweep level (the last level set) on v+.
//       Barrier + reduction: delta and the rotation scalars that need only
//       alpha, beta and delta (rho, tau, epsilon, gamma).
//   P2  the remaining U-sweep levels: D^-1 (k_solve_D), the off-diagonal
//       terms, back substitution with the pivot tile; the result goes
//       straight to its permuted place, ev = P U^-1 D^-1 v+.  One barrier
//       per level.
//   P3  the U'-sweep levels with the SpMV fused into the right-hand side:
//       each block row's warp computes (K ev) for its own rows (the P'
//       permutation is local to a block row), scales by 1/delta and
//       forward-substitutes into Av.  The same warp accumulates, over its
//       rows, beta's numerator v' D^-1 Av and the next alpha's dots
//       v+' D^-1 Av and v+' D^-1 v+; the first level also updates p and x.
//       Barrier + reduction: beta, the next alpha, ||x||, the tests.
//
// That is 2 x (number of levels) barriers per iteration, fewer for a KKT
// system in natural order (two levels, level 0 of simple rows): there the
// level-0 rows also compute their (K ev) in the U sweep (the U' sweep's
// level-0 phase goes away), and instead of a grid barrier between the U
// sweep's two levels every CTA counts its finished level-1 rows on a device
// counter that the level-0 rows wait for (one elected poller per CTA, a
// bounded wait: a wait that gives up ends the solve with CULIPX_TIMEOUT).
// The two reductions are then the iteration's only grid-wide barriers, and
// where every phase is short they are counted and bounded the same way
// (grid_reduce).  Re-associations against the reference, all exact in real
// arithmetic:
//   * v+ is divided by delta after the U sweep instead of before it (the
//     sweep is linear); the division is applied to the SpMV result.
//   * The reference's w_k (sqmr.impl.cuh, solve_middle of v_k scaled by eta
//     and 1/beta) equals eta_k D^-1 v_k at every step, so it is not stored:
//     beta = (w' Av) / (w' v) = (v' D^-1 Av) / (v' D^-1 v), whose
//     denominator is the previous alpha's denominator.  eta is still
//     carried for the reference's breakdown test.
//   * The p / x update runs one phase later than in the reference (it needs
//     only alpha, beta_k and delta).
// Every CTA reduces the per-CTA partials in the same fixed order and its
// thread 0 runs the scalar recurrence in shared memory, so control flow is
// uniform across the grid and the result is deterministic for a given grid
// size.
//
// Data the loop reads: K (CSR), U and U' as fine-row CSR (U's columns mapped
// through P), the non-identity pivot tiles as packed upper triangles (column
// by column for U, row by row for U'), the diagonal of D for block rows with
// 1x1 pivots only (D^-1 y = y / d there, which is what the Givens form
// computes for a 1x1 pivot) and tri / is_piv for the others, and 9 vectors.
#pragma once

#include "sqmr.h"
#include "factor.h"
#include "pattern.h"
#include "kernels_common.cuh"

#include <cooperative_groups.h>


namespace cg = cooperative_groups;

namespace culipx {

namespace persistent {

constexpr int kT = 512;          // threads per CTA
constexpr int kW = kT / 32;      // warps per CTA
constexpr int kCtasPerSm = 2;    // 32 resident warps per SM
constexpr int kMaxNR = 4;        // right-hand sides per launch
constexpr int kMaxNV = 4 * kMaxNR;  // values per grid reduction
constexpr int kBatch = 8;        // loads issued ahead in row sums and tile solves
constexpr int kVecs = 7;         // work vectors of n doubles
constexpr unsigned kFull = 0xffffffffu;

template <class TF>
struct PArgs {
    int n, nl, max_it;
    int fuse_l0;               // level-0 simple rows compute (K ev) in the U sweep
    int count_red;             // the fused iteration's reductions may use the counted barrier
    double tol;
    const int* rowptr;
    const int* colidx;
    const double* kval;
    const TF* pk_col;          // pivot tile upper triangles, column by column
    const TF* pk_row;          // the same, row by row
    const long long* pk_off;   // per block row
    const unsigned* ndmask;    // per block row: non-unit diagonal entries of the pivot tile
    const TF* dg;              // diagonal of D
    const TF* tri;
    const int* is_piv;
    const int* perm;
    const int* lvl_off;
    const int* lvl_rows;
    const int* bs;
    const int2* u_rng;         // per fine row: its entries' [first, end)
    const int* u_colp;         // U columns mapped through P
    const TF* u_val;
    const int2* ut_rng;
    const int* ut_col;
    const TF* ut_val;
    const int* rowflags;
    const int* scan_s;         // simple / other block rows per level (factor.h)
    const int* scan_c;
    const int* simple_rows;
    const int* cplx;
    const CItem* citem;        // per entry of cplx: the block row's metadata
    double* v[2];              // v_k and v_k-1, v_k+1 overwrites v_k-1 in place
    double* p[2];              // p_k-1 and p_k-2, p_k overwrites p_k-2 in place
    double* Av;
    double* ev;    // P U^-1 D^-1 (...)
    double* xt;    // the iterate x~ (interleaved)
    double* x;     // the caller's solutions, column-major n x NR
    const double* b;  // the caller's right-hand sides, column-major n x NR
    double* partials;  // 2 buffers x kMaxNV x gridDim
    double* out;       // [0] gamma/norm_pb, [1] iterations, [2] breakdown, [3] converged, [4] norm_pb, [5] it
    unsigned long long* ts;  // optional phase timestamps: [it * 8 + phase], it < kTsIters
    // Level-completion counter of the fused two-level iteration (grid launches
    // only; NULL: a grid synchronisation instead): every CTA adds 1 once its
    // level-1 rows of an iteration are written, level-0 rows wait for
    // G (it + 1) before they read them.  [1]: set when a wait gave up.
    unsigned long long* lvl_done;  // [2], [3]: the same for the reductions' barrier
    unsigned long long wait_skew;  // added to the wait's target (fault injection in tests; 0)
    unsigned long long red_skew;   // the same for the reductions' counted barrier
};

// Bound of one device wait on a counter, far below a watchdog.  The level
// handoff waits for level-1 tiles, which walk no rows: a few microseconds.
// The reductions wait for whole phases and are counted only where the rows
// keep those well under it (reductions_counted, sqmr_persistent.cu).
constexpr unsigned long long kWaitLimitNs = 200ull * 1000 * 1000;

// Shared state of a CTA's level waits: the iteration (+1) whose count the CTA
// has seen, and the iteration (+1) whose poller was elected.
struct LvlWait {
    int seen;
    int poll;
};

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p)
{
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void red_release_add_u64(unsigned long long* p, unsigned long long v)
{
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// One thread spins (acquire loads, backing off) until *ctr >= target; gives up
// after kWaitLimitNs, or at once if an earlier wait gave up, and records that
// in ctr[1].  Returns false when it gave up.
inline __device__ bool wait_count(unsigned long long* ctr, unsigned long long target)
{
    if (ld_acquire_u64(ctr) >= target) return true;
    volatile unsigned long long* failed = ctr + 1;
    if (*failed) return false;
    unsigned long long t0;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (unsigned k = 0;; ++k) {
        __nanosleep(k < 8 ? 32 : 256);
        if (ld_acquire_u64(ctr) >= target) return true;
        if ((k & 15) == 15) {
            unsigned long long t;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            if (*failed || t - t0 > kWaitLimitNs) {
                *failed = 1;
                return false;
            }
        }
    }
}

constexpr int kTsIters = 64;

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// CTA 0 stamps phase boundaries (right after the barrier that ends a phase)
__device__ __forceinline__ void stamp(unsigned long long* ts, int it, int phase)
{
    if (ts && it < kTsIters && blockIdx.x == 0 && threadIdx.x == 0) ts[it * 8 + phase] = global_ns();
}

// scalar state of the recurrence, in shared memory, written by thread 0 only
struct Scal {
    double alpha, alpha_next, beta[3], delta[3], c[3], s[3];
    double norm_A, epsilon, beta_rr, tau, rho, gamma, norm_pb, norm_x, eta;
    double inv_pb, inv_delta, inv_beta, inv_rho;
    double vdv;  // v_k' D^-1 v_k
    int test0, test1, snap0, snap1, done, iters, breakdown, stop_it;
};

__host__ __device__ __forceinline__ int acc3(int r) { return (r % 3) + ((r < 0) ? 3 : 0); }

// Fixed-order sum over the grid (one barrier).  Thread 0 of every CTA gets
// the totals in v, identical in every CTA.  The caller publishes what thread
// 0 derives from them with a __syncthreads() before the next reduction.
// ctr (counter, gave-up flag): the barrier is one release add per CTA and one
// acquiring poller, a round trip to L2 less than grid.sync's (scale: 1656 ->
// 1621 us for 32 iterations); the wait is bounded (wait_count).  NULL:
// grid.sync.
// Thread 0 gets false when its wait gave up: the totals are then not the
// grid's and may differ between CTAs, so the caller must leave its loop, and
// that loop may hold no grid.sync of its own (the CTAs need not leave at the
// same iteration).  They all leave soon: the first CTA that gave up adds at
// most one more count (the iteration's second reduction), so no later target
// is reached, and with the flag set a wait short of its target gives up at
// once.
template <int NV>
__device__ bool grid_reduce(double (&v)[NV], double* partials, int& red, double (*sh)[kW], cg::grid_group& grid,
                            unsigned long long* ctr, int counted_from, unsigned long long skew)
{
    bool ok = true;
    const int lane = (int)lane_id(), w = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; ++k)
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(kFull, v[k], o);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; ++k) sh[k][w] = v[k];
    __syncthreads();
    double* buf = partials + (size_t)(red & 1) * kMaxNV * gridDim.x;
    ++red;
    if (threadIdx.x < NV) {
        double t = 0.0;
        for (int i = 0; i < kW; ++i) t += sh[threadIdx.x][i];
        buf[threadIdx.x * gridDim.x + blockIdx.x] = t;
    }
    if (ctr) {
        if (w == 0) {
            __syncwarp();
            if (lane == 0) {
                red_release_add_u64(ctr, 1ull);
                const unsigned long long target =
                    (unsigned long long)gridDim.x * (unsigned long long)(red - counted_from) + skew;
                int k = 0;
                while (k < 64 && ld_acquire_u64(ctr) < target) ++k;  // the others are usually close behind
                if (k == 64) ok = wait_count(ctr, target);
            }
        }
        __syncthreads();
    } else {
        grid.sync();
    }
    // the NV partials of a CTA position are loaded together (one round trip
    // to L2 for all NV sums); each sum keeps its order over c
    double t[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) t[k] = 0.0;
    for (int c = threadIdx.x; c < (int)gridDim.x; c += kT)
#pragma unroll
        for (int k = 0; k < NV; ++k) t[k] += __ldcg(buf + k * gridDim.x + c);
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        for (int o = 16; o > 0; o >>= 1) t[k] += __shfl_down_sync(kFull, t[k], o);
        if (lane == 0) sh[k][w] = t[k];
    }
    __syncthreads();
    if (threadIdx.x == 0)
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            double t = 0.0;
            for (int i = 0; i < kW; ++i) t += sh[k][i];
            v[k] = t;
        }
    return ok;
}

// D^-1 of one block row (k_solve_D, helper_kernels.impl.cuh:720-774).  With
// 1x1 pivots only the Givens form reduces to y / d exactly (c = sign(d),
// s = 0, r = |d|); a block row with a 2x2 pivot keeps the Givens form, its
// pairs never straddle block rows.  Every lane of the warp calls apply().
template <class TF>
struct DBlock {
    bool two;
    double d;                       // 1x1: the pivot (1 on lanes >= h)
    double gc, gs, tp12, tp22, gr;  // Givens form
    bool ip;

    __device__ __forceinline__ void load(const PArgs<TF>& a, int fr, int h, int flags)
    {
        const int lane = (int)lane_id();
        two = (flags & kRowHas2x2) != 0;
        d = 1.0;
        gc = gs = tp12 = 0.0;
        tp22 = gr = 1.0;
        ip = true;
        if (lane >= h) return;
        const size_t r = (size_t)(fr + lane);
        if (!two) {
            d = (double)__ldg(a.dg + r);
            return;
        }
        ip = __ldg(a.is_piv + r) != 0;
        const bool np = (lane + 1 < h) ? (__ldg(a.is_piv + r + 1) != 0) : true;
        const double p11 = (double)__ldg(a.tri + 3 * r + 1), p12 = (double)__ldg(a.tri + 3 * r + 2);
        const double p22 = !np ? (double)__ldg(a.tri + 3 * (r + 1) + 1) : 1.0;
        gr = sqrt(fma_rn(p11, p11, p12 * p12));
        gc = p11 / gr;
        gs = p12 / gr;
        tp12 = fma_rn(gc, p12, gs * p22);
        tp22 = fma_rn(gc, p22, -(gs * p12));
    }

    __device__ __forceinline__ double apply(double y, int h) const
    {
        const int lane = (int)lane_id();
        if (!two) return (lane < h) ? y / d : 0.0;
        const double ynext = __shfl_down_sync(kFull, y, 1);
        double g1 = 0.0, g2 = 0.0;
        if (lane < h) {
            const double r2 = (lane + 1 < h) ? ynext : 0.0;
            g1 = fma_rn(gc, y, gs * r2);
            g2 = fma_rn(gc, r2, -(gs * y));
            g2 = g2 / tp22;
            g1 = fma_rn(-tp12, g2, g1) / gr;
        }
        const double from_prev = __shfl_up_sync(kFull, g2, 1);
        return ip ? g1 : from_prev;
    }
};

// acc[j] - sum_k val[k] x[col[k] NR + j] in increasing k for the NR
// interleaved right-hand sides (x is written during the kernel: plain loads);
// index / value loads of a batch, then its gathers (the NR values of one
// column are adjacent: 16-byte loads for even NR).  SC: the gathered values
// are stored unscaled and enter as (TF)(x * xs[j]), the value an earlier
// phase would have stored after scaling.
template <class TF, int NR, bool SC = false>
__device__ __forceinline__ void row_sub(TF (&acc)[NR], int k0, int k1, const int* __restrict__ col,
                                        const TF* __restrict__ val, const double* x,
                                        const double* xs = nullptr)
{
    constexpr int B = (NR == 1) ? kBatch : (NR == 2 ? 4 : 2);
    for (int k = k0; k < k1; k += B) {
        int c[B];
        TF v[B];
#pragma unroll
        for (int j = 0; j < B; ++j) {
            c[j] = (k + j < k1) ? __ldg(col + k + j) : -1;
            v[j] = (k + j < k1) ? __ldg(val + k + j) : TF(0);
        }
        double xv[B][NR];
#pragma unroll
        for (int j = 0; j < B; ++j) {
            if (NR % 2 == 0) {
#pragma unroll
                for (int r = 0; r < NR; r += 2) {
                    double2 q = make_double2(0.0, 0.0);
                    if (c[j] >= 0) q = *reinterpret_cast<const double2*>(x + (size_t)c[j] * NR + r);
                    xv[j][r] = q.x;
                    xv[j][r + 1] = q.y;
                }
            } else {
#pragma unroll
                for (int r = 0; r < NR; ++r) xv[j][r] = (c[j] >= 0) ? x[(size_t)c[j] * NR + r] : 0.0;
            }
        }
#pragma unroll
        for (int j = 0; j < B; ++j)
            if (k + j < k1)
#pragma unroll
                for (int r = 0; r < NR; ++r)
                    acc[r] = fma_rn(-v[j], SC ? (TF)(xv[j][r] * xs[r]) : (TF)xv[j][r], acc[r]);
    }
}

// (K x)_q for the NR interleaved vectors, entries in increasing column order
template <class TF, int NR>
__device__ __forceinline__ void spmv_row(const PArgs<TF>& a, int q, const double* x, double (&acc)[NR])
{
    constexpr int B = (NR == 1) ? kBatch : (NR == 2 ? 4 : 2);
    const int k0 = __ldg(a.rowptr + q), k1 = __ldg(a.rowptr + q + 1);
#pragma unroll
    for (int r = 0; r < NR; ++r) acc[r] = 0.0;
    for (int k = k0; k < k1; k += B) {
        int c[B];
        double v[B];
#pragma unroll
        for (int j = 0; j < B; ++j) {
            c[j] = (k + j < k1) ? __ldg(a.colidx + k + j) : -1;
            v[j] = (k + j < k1) ? __ldg(a.kval + k + j) : 0.0;
        }
        double xv[B][NR];
#pragma unroll
        for (int j = 0; j < B; ++j) {
            if (NR % 2 == 0) {
#pragma unroll
                for (int r = 0; r < NR; r += 2) {
                    double2 q2 = make_double2(0.0, 0.0);
                    if (c[j] >= 0) q2 = *reinterpret_cast<const double2*>(x + (size_t)c[j] * NR + r);
                    xv[j][r] = q2.x;
                    xv[j][r + 1] = q2.y;
                }
            } else {
#pragma unroll
                for (int r = 0; r < NR; ++r) xv[j][r] = (c[j] >= 0) ? x[(size_t)c[j] * NR + r] : 0.0;
            }
        }
#pragma unroll
        for (int j = 0; j < B; ++j)
            if (k + j < k1)
#pragma unroll
                for (int r = 0; r < NR; ++r) acc[r] = fma_rn(v[j], xv[j][r], acc[r]);
    }
}

// Back substitution with the block row's pivot tile, upper triangle packed
// column by column (U sweep; d_left_solve_row_major,
// block_ildlt_kernels.impl.cuh:2087-2113): for c = h-1 .. 0:
// x_c = t_c / U_cc, t_r -= U_rc x_c (r < c), for each right-hand side.  The
// division is taken only where bit c of nd says U_cc != 1 (t / 1 == t
// exactly); with nd == 0 the chain is shuffle + fma per step.
// SM: P is a copy of the column-packed triangle in shared memory
template <bool SM, class TF>
__device__ __forceinline__ TF tile_ld(const TF* p)
{
    if (SM) return *p;
    return __ldg(p);
}

template <class TF, int NR, bool DIV, bool SM>
__device__ __forceinline__ void tile_upper_t(TF (&t)[NR], const TF* __restrict__ P, int h, unsigned nd)
{
    const int lane = (int)lane_id();
    constexpr int B = (NR == 1) ? kBatch : 4;
    for (int c0 = h - 1; c0 >= 0; c0 -= B) {
        TF u[B];
#pragma unroll
        for (int j = 0; j < B; ++j) {
            const int c = c0 - j;
            u[j] = (c >= 0 && lane <= c) ? tile_ld<SM>(P + c * (c + 1) / 2 + lane) : TF(0);
        }
#pragma unroll
        for (int j = 0; j < B; ++j) {
            const int c = c0 - j;
            if (c >= 0) {
                if (DIV && ((nd >> c) & 1u)) {
                    if (lane == c)
#pragma unroll
                        for (int r = 0; r < NR; ++r) t[r] = t[r] / u[j];
                }
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    const TF xc = __shfl_sync(kFull, t[r], c);
                    if (lane < c) t[r] = fma_rn(-u[j], xc, t[r]);
                }
            }
        }
    }
}

// Forward substitution with the upper triangle packed row by row (U'
// sweep): for r = 0 .. h-1: x_r = t_r / U_rr, t_c -= U_rc x_r (r < c < h);
// divisions as in tile_upper_t.  With SM the triangle is the column-packed
// copy in shared memory, read along its rows: lane c reads c(c+1)/2 + r, and
// c(c+1)/2 mod 16 is a permutation of 0..15 on each half-warp, so the
// 8-byte reads of a half-warp hit distinct banks.
template <class TF, int NR, bool DIV, bool SM>
__device__ __forceinline__ void tile_lower_t(TF (&t)[NR], const TF* __restrict__ P, int h, unsigned nd)
{
    const int lane = (int)lane_id();
    constexpr int B = (NR == 1) ? kBatch : 4;
    for (int r0 = 0; r0 < h; r0 += B) {
        TF u[B];
#pragma unroll
        for (int j = 0; j < B; ++j) {
            const int r = r0 + j;
            u[j] = (r < h && lane >= r && lane < h)
                       ? (SM ? P[lane * (lane + 1) / 2 + r] : __ldg(P + r * h - r * (r - 1) / 2 + lane - r))
                       : TF(0);
        }
#pragma unroll
        for (int j = 0; j < B; ++j) {
            const int r = r0 + j;
            if (r < h) {
                if (DIV && ((nd >> r) & 1u)) {
                    if (lane == r)
#pragma unroll
                        for (int q = 0; q < NR; ++q) t[q] = t[q] / u[j];
                }
#pragma unroll
                for (int q = 0; q < NR; ++q) {
                    const TF xr = __shfl_sync(kFull, t[q], r);
                    if (lane > r && lane < h) t[q] = fma_rn(-u[j], xr, t[q]);
                }
            }
        }
    }
}

template <class TF, int NR, bool SM = false>
__device__ __forceinline__ void tile_upper(double (&v)[NR], const TF* P, int h, unsigned nd)
{
    TF t[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) t[r] = (TF)v[r];
    if (nd) tile_upper_t<TF, NR, true, SM>(t, P, h, nd);
    else tile_upper_t<TF, NR, false, SM>(t, P, h, 0u);
#pragma unroll
    for (int r = 0; r < NR; ++r) v[r] = (double)t[r];
}

template <class TF, int NR, bool SM = false>
__device__ __forceinline__ void tile_lower(double (&v)[NR], const TF* P, int h, unsigned nd)
{
    TF t[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) t[r] = (TF)v[r];
    if (nd) tile_lower_t<TF, NR, true, SM>(t, P, h, nd);
    else tile_lower_t<TF, NR, false, SM>(t, P, h, 0u);
#pragma unroll
    for (int r = 0; r < NR; ++r) v[r] = (double)t[r];
}

// A work item's block-row metadata
struct ItemMeta {
    int I, fr, h, flags;
    long long pko;
    unsigned nd;
};

// from the block row (sweeps over every block row of a level)
template <class TF>
__device__ __forceinline__ ItemMeta meta_of_row(const PArgs<TF>& a, int I)
{
    ItemMeta m;
    m.I = I;
    m.fr = __ldg(a.bs + I);
    m.h = __ldg(a.bs + I + 1) - m.fr;
    m.flags = __ldg(a.rowflags + I);
    m.pko = __ldg(a.pk_off + I);
    m.nd = __ldg(a.ndmask + I);
    return m;
}

// from entry t of the pivot-tile block rows: two independent 16-byte loads
// instead of the chain cplx -> (bs, rowflags, pk_off, ndmask)
template <class TF>
__device__ __forceinline__ ItemMeta meta_of_item(const PArgs<TF>& a, int t)
{
    const int4* p = reinterpret_cast<const int4*>(a.citem + t);
    const int4 u = __ldg(p), w = __ldg(p + 1);
    ItemMeta m;
    m.I = u.x;
    m.fr = u.y;
    m.h = u.z;
    m.flags = u.w;
    m.pko = (long long)(((unsigned long long)(unsigned)w.y << 32) | (unsigned)w.x);
    m.nd = (unsigned)w.z;
    return m;
}

// Shared-memory copy of one warp's pivot-tile work item, loaded once per
// solve.  Each warp of the persistent kernel keeps the same item of a level
// for the whole solve (item c0 + wid), so the level with the most such items
// keeps, per warp slot, the item's metadata, its lanes' permuted rows and U /
// U' row ranges, D's diagonal (block rows without 2x2 pivots) and the pivot
// tile's upper triangle (column-packed).  The item's per-iteration chain of
// dependent loads (descriptor, permutation and offsets, four batches of tile
// values, D) becomes shared-memory reads.
constexpr int kResSlots = 12;  // warps per CTA with a resident item
constexpr int kTileMax = 32 * 33 / 2;

template <class TF>
struct ResSlot {
    ItemMeta m;  // m.h == 0: the warp has no item of the resident level
    int q[32];   // perm[fr + lane]
    int u0[32], u1[32], ut0[32], ut1[32];
    double d[32];
    TF tile[kTileMax];
};

// warp-collective: fills the slot with item t of the citem list (has) or marks it empty
template <class TF>
__device__ void res_load(const PArgs<TF>& a, ResSlot<TF>& rs, int t, bool has)
{
    const int lane = (int)lane_id();
    if (!has) {
        if (lane == 0) rs.m.h = 0;
        return;
    }
    const ItemMeta m = meta_of_item(a, t);
    if (lane == 0) rs.m = m;
    const int fr = m.fr, h = m.h;
    if (lane < h) {
        const int g = fr + lane;
        rs.q[lane] = (m.flags & kRowPermIdentity) ? g : __ldg(a.perm + g);
        const int2 ur = __ldg(a.u_rng + g), utr = __ldg(a.ut_rng + g);
        rs.u0[lane] = ur.x;
        rs.u1[lane] = ur.y;
        rs.ut0[lane] = utr.x;
        rs.ut1[lane] = utr.y;
        rs.d[lane] = (m.flags & kRowHas2x2) ? 1.0 : (double)__ldg(a.dg + g);
    }
    if (!(m.flags & kRowIdentity))
        for (int e = lane; e < h * (h + 1) / 2; e += 32) rs.tile[e] = __ldg(a.pk_col + m.pko + e);
}

// D of a resident item: its diagonal from the slot, or the Givens form from
// global memory when the block row has a 2x2 pivot
template <class TF>
__device__ __forceinline__ DBlock<TF> dblock_res(const PArgs<TF>& a, const ResSlot<TF>& rs)
{
    DBlock<TF> D;
    const int flags = rs.m.flags, h = rs.m.h;
    if (flags & kRowHas2x2) {
        D.load(a, rs.m.fr, h, flags);
        return D;
    }
    const int lane = (int)lane_id();
    D.two = false;
    D.d = (lane < h) ? rs.d[lane] : 1.0;
    D.gc = D.gs = D.tp12 = 0.0;
    D.tp22 = D.gr = 1.0;
    D.ip = true;
    return D;
}

// One U-sweep work item: block row I (rows fr .. fr+h-1), lane's right-hand
// sides y: d = D^-1 y; t = U_II^-1 (d - U_I* t); out[perm[r]] = t (NR
// interleaved).  The gathers of the later levels' t read out through the
// permuted columns.  d receives D^-1 y (0 on lanes >= h).
template <class TF, int NR>
__device__ __forceinline__ void u_item(const PArgs<TF>& a, const ItemMeta& m, const double (&y)[NR], double* out,
                                       double (&d)[NR])
{
    const int lane = (int)lane_id();
    const int fr = m.fr, h = m.h, flags = m.flags;
    DBlock<TF> D;
    D.load(a, fr, h, flags);
#pragma unroll
    for (int r = 0; r < NR; ++r) d[r] = D.apply(y[r], h);
    double t[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) t[r] = d[r];
    if (lane < h) {
        TF acc[NR];
#pragma unroll
        for (int r = 0; r < NR; ++r) acc[r] = (TF)d[r];
        const int2 kr = __ldg(a.u_rng + fr + lane);
        row_sub<TF, NR>(acc, kr.x, kr.y, a.u_colp, a.u_val, out);
#pragma unroll
        for (int r = 0; r < NR; ++r) t[r] = (double)acc[r];
    }
    if (!(flags & kRowIdentity)) tile_upper<TF, NR>(t, a.pk_col + m.pko, h, m.nd);
    if (lane < h) {
        const int q = (flags & kRowPermIdentity) ? fr + lane : __ldg(a.perm + fr + lane);
#pragma unroll
        for (int r = 0; r < NR; ++r) out[(size_t)q * NR + r] = t[r];
    }
}

// Where a U'-sweep item's right-hand side comes from
enum RhsFrom {
    kRhsCaller = 0,  // b[r n + perm[row]] of the caller's column-major right-hand sides
    kRhsSpmv = 1,    // sc[r] * (K src)[perm[row]], src interleaved
    kRhsPre = 2,     // dst[perm[row]]: sc (K src) stored there by an earlier phase
};

// One U'-sweep work item: dst[row] = U_II'^-1 (rhs - U'_I* dst) (interleaved)
// with the lane's right-hand sides taken as FROM says.  t receives the
// lane's results (0 for lanes >= h).
template <class TF, int NR, int FROM, bool SCG = false>
__device__ __forceinline__ void ut_item(const PArgs<TF>& a, const ItemMeta& m, const double* src,
                                        const double (&sc)[NR], double* dst, double (&t)[NR])
{
    const int lane = (int)lane_id();
    const int fr = m.fr, h = m.h, flags = m.flags;
#pragma unroll
    for (int r = 0; r < NR; ++r) t[r] = 0.0;
    if (lane < h) {
        const int q = (flags & kRowPermIdentity) ? fr + lane : __ldg(a.perm + fr + lane);
        double y[NR];
        if (FROM == kRhsSpmv) {
            spmv_row<TF, NR>(a, q, src, y);
#pragma unroll
            for (int r = 0; r < NR; ++r) y[r] *= sc[r];
        } else if (FROM == kRhsPre) {
#pragma unroll
            for (int r = 0; r < NR; ++r) y[r] = dst[(size_t)q * NR + r];
        } else {
#pragma unroll
            for (int r = 0; r < NR; ++r) y[r] = src[(size_t)r * a.n + q];
        }
        TF acc[NR];
#pragma unroll
        for (int r = 0; r < NR; ++r) acc[r] = (TF)y[r];
        const int2 kr = __ldg(a.ut_rng + fr + lane);
        row_sub<TF, NR, SCG>(acc, kr.x, kr.y, a.ut_col, a.ut_val, dst, sc);
#pragma unroll
        for (int r = 0; r < NR; ++r) t[r] = (double)acc[r];
    }
    // with kRhsPre the lanes read dst inside this block row: all reads before any write
    if (FROM == kRhsPre) __syncwarp();
    if (!(flags & kRowIdentity)) tile_lower<TF, NR>(t, a.pk_row + m.pko, h, m.nd);
    if (lane < h)
#pragma unroll
        for (int r = 0; r < NR; ++r) dst[(size_t)(fr + lane) * NR + r] = t[r];
}

// u_item / ut_item of a resident item (same arithmetic, data from the slot)
template <class TF, int NR>
__device__ __forceinline__ void u_item_res(const PArgs<TF>& a, const ResSlot<TF>& rs, const double (&y)[NR],
                                           double* out, double (&d)[NR])
{
    const int lane = (int)lane_id();
    const int h = rs.m.h, flags = rs.m.flags;
    const DBlock<TF> D = dblock_res(a, rs);
#pragma unroll
    for (int r = 0; r < NR; ++r) d[r] = D.apply(y[r], h);
    double t[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) t[r] = d[r];
    if (lane < h) {
        TF acc[NR];
#pragma unroll
        for (int r = 0; r < NR; ++r) acc[r] = (TF)d[r];
        row_sub<TF, NR>(acc, rs.u0[lane], rs.u1[lane], a.u_colp, a.u_val, out);
#pragma unroll
        for (int r = 0; r < NR; ++r) t[r] = (double)acc[r];
    }
    if (!(flags & kRowIdentity)) tile_upper<TF, NR, true>(t, rs.tile, h, rs.m.nd);
    if (lane < h) {
        const int q = rs.q[lane];
#pragma unroll
        for (int r = 0; r < NR; ++r) out[(size_t)q * NR + r] = t[r];
    }
}

template <class TF, int NR, int FROM, bool SCG = false>
__device__ __forceinline__ void ut_item_res(const PArgs<TF>& a, const ResSlot<TF>& rs, const double* src,
                                            const double (&sc)[NR], double* dst, double (&t)[NR])
{
    const int lane = (int)lane_id();
    const int fr = rs.m.fr, h = rs.m.h, flags = rs.m.flags;
#pragma unroll
    for (int r = 0; r < NR; ++r) t[r] = 0.0;
    if (lane < h) {
        const int q = rs.q[lane];
        double y[NR];
        if (FROM == kRhsSpmv) {
            spmv_row<TF, NR>(a, q, src, y);
#pragma unroll
            for (int r = 0; r < NR; ++r) y[r] *= sc[r];
        } else if (FROM == kRhsPre) {
#pragma unroll
            for (int r = 0; r < NR; ++r) y[r] = dst[(size_t)q * NR + r];
        } else {
#pragma unroll
            for (int r = 0; r < NR; ++r) y[r] = src[(size_t)r * a.n + q];
        }
        TF acc[NR];
#pragma unroll
        for (int r = 0; r < NR; ++r) acc[r] = (TF)y[r];
        row_sub<TF, NR, SCG>(acc, rs.ut0[lane], rs.ut1[lane], a.ut_col, a.ut_val, dst, sc);
#pragma unroll
        for (int r = 0; r < NR; ++r) t[r] = (double)acc[r];
    }
    if (FROM == kRhsPre) __syncwarp();
    if (!(flags & kRowIdentity)) tile_lower<TF, NR, true>(t, rs.tile, h, rs.m.nd);
    if (lane < h)
#pragma unroll
        for (int r = 0; r < NR; ++r) dst[(size_t)(fr + lane) * NR + r] = t[r];
}

inline __device__ double sgn(double v) { return v < 0 ? -1.0 : 1.0; }

// k_sym_ortho (helper_kernels.impl.cuh:662-700)
inline __device__ void sym_ortho(double a, double b, double& c, double& s, double& r)
{
    if (b == 0) { s = 0; r = fabs(a); c = (a == 0) ? 1 : sgn(a); }
    else if (a == 0) { c = 0; s = sgn(b); r = fabs(b); }
    else if (fabs(b) >= fabs(a)) {
        const double tao = a / b;
        s = sgn(b) / sqrt(fma_rn(tao, tao, 1.0));
        c = s * tao;
        r = b / s;
    } else {
        const double tao = b / a;
        c = sgn(a) / sqrt(fma_rn(tao, tao, 1.0));
        s = c * tao;
        r = a / c;
    }
}

// The recurrence after a U sweep: rr = ||v+||^2 (unscaled) gives delta and the
// rotation of step k (k0, k1, km1: the places of k, k + 1, k - 1).
inline __device__ void scal_after_u(Scal& Q, double rr, int k0, int k1, int km1)
{
    const double alpha = Q.alpha_next;
    Q.alpha = alpha;
    const double bk = Q.beta[k0];
    const double dl = sqrt(rr);
    Q.delta[k1] = dl;
    Q.inv_delta = 1.0 / dl;
    const double nA = sqrt(fma_rn(dl, dl, fma_rn(alpha, alpha, bk * bk)));
    Q.norm_A = fmax(Q.norm_A, nA);
    Q.epsilon = Q.s[km1] * bk;
    const double beta_rot = (-Q.c[km1]) * bk;
    Q.beta_rr = fma_rn(Q.c[k0], beta_rot, Q.s[k0] * alpha);
    const double alpha_rot = fma_rn(Q.s[k0], beta_rot, (-Q.c[k0]) * alpha);
    double c, s, rho;
    sym_ortho(alpha_rot, dl, c, s, rho);
    Q.c[k1] = c;
    Q.s[k1] = s;
    Q.rho = rho;
    Q.inv_rho = 1.0 / rho;
    Q.tau = c * Q.gamma;
    Q.gamma = s * Q.gamma;
}

// The recurrence after a U' sweep: vda = v_k' D^-1 Av, wda = v+' D^-1 Av, wdw
// = v+' D^-1 v+, xx = ||x||^2; beta, the next alpha and the lagged tests.
inline __device__ void scal_after_ut(Scal& Q, double vda, double wda, double wdw, double xx, int it, int k1,
                                     double tol, int max_it)
{
    const double bt = vda / Q.vdv;
    Q.beta[k1] = bt;
    Q.inv_beta = 1.0 / bt;
    Q.eta = (Q.delta[k1] / bt) * Q.eta;
    Q.alpha_next = wda / wdw;
    Q.vdv = wdw;
    Q.norm_x = sqrt(xx);
    Q.test0 |= (fabs(Q.delta[k1]) <= tol);
    Q.test1 |= (Q.gamma / fma_rn(Q.norm_A, Q.norm_x, Q.norm_pb) <= tol);
    bool stop = false;
    if (it > 0 && (it % 4) == 0) {
        if (Q.snap0 || Q.snap1) {
            stop = true;
            Q.iters = it;
        }
    } else if (((it + 1) % 4) == 0) {
        Q.snap0 = Q.test0;
        Q.snap1 = Q.test1;
    }
    if (!isfinite(Q.inv_beta) || !isfinite(Q.inv_rho) || !isfinite(Q.eta) || !isfinite(Q.inv_delta) ||
        !isfinite(Q.alpha)) {
        Q.breakdown = 1;
        stop = true;
        Q.iters = it;
    }
    if (!stop && it + 1 >= max_it) Q.iters = max_it;
    if (stop) {
        Q.done = 1;
        Q.stop_it = it;
    }
}

// A reduction's wait gave up: the solve ends here (its results are marked
// invalid by the counter's flag)
template <int NR>
__device__ __forceinline__ void abandon(Scal (&S)[NR], int it)
{
    for (int j = 0; j < NR; ++j) {
        if (S[j].done) continue;
        S[j].done = 1;
        S[j].iters = it;
        S[j].stop_it = it;
    }
}

// Fixed-order sum over one CTA: thread 0 gets the totals (same protocol as
// grid_reduce).
template <int NV>
__device__ void cta_reduce(double (&v)[NV], double (*sh)[kW])
{
    const int lane = (int)lane_id(), w = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; ++k)
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(kFull, v[k], o);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; ++k) sh[k][w] = v[k];
    __syncthreads();
    if (threadIdx.x == 0)
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            double t = 0.0;
            for (int i = 0; i < kW; ++i) t += sh[k][i];
            v[k] = t;
        }
}

// Where one solve runs: the whole grid of a cooperative launch (one system)
// or one CTA of a batched launch (one system per CTA at a time).  Work items
// go to warps wid, wid + nwarps, ...; vector loops to threads g0, g0 + gstride.
struct GridCtx {
    cg::grid_group grid;
    double* partials;
    int red;
    int wid, nwarps, g0, gstride;
    unsigned long long* ctr;  // the reductions' barrier (grid_reduce); NULL before begin_counted
    int counted_from;         // reductions before it
    unsigned long long skew;  // added to their targets (tests)
    __device__ void sync() { grid.sync(); }
    // from here on the reductions use the counter behind the level counter,
    // zeroed before the initial phases; only for a loop without sync()
    __device__ void begin_counted(unsigned long long* lvl_done, unsigned long long red_skew)
    {
        ctr = lvl_done + 2;
        counted_from = red;  // red goes on: the partials' two buffers keep alternating
        skew = red_skew;
    }
    template <int NV>
    __device__ bool reduce(double (&v)[NV], double (*sh)[kW])
    {
        return grid_reduce<NV>(v, partials, red, sh, grid, ctr, counted_from, skew);
    }
};

struct CtaCtx {
    int wid, nwarps, g0, gstride;
    __device__ void sync() const { __syncthreads(); }
    __device__ void begin_counted(unsigned long long*, unsigned long long) const {}
    template <int NV>
    __device__ bool reduce(double (&v)[NV], double (*sh)[kW])
    {
        cta_reduce<NV>(v, sh);
        return true;
    }
};

// The system a solve works on: its rows [row0, row1) and, for each level L,
// its block rows' positions [qb[L], qe[L]) in the level lists; out receives
// per right-hand side r at out + 8 r: [0] gamma/norm_pb, [1] iterations,
// [2] breakdown, [3] converged, [4] norm_pb, [5] it.
struct SysView {
    int row0, row1;
    const int* qb;
    const int* qe;
    double* out;
};

// Per-RHS coefficients of the p / x update and of the dots' scaling
template <int NR>
struct Coef {
    double sc[NR], nbrr[NR], ne[NR], ir[NR], tau[NR];
    double na[NR], nb[NR];  // the U sweep's -alpha, -beta_k
    const double* vk;       // the iteration's v_k, v_k+1 (= v_k-1 on entry), p_k (= p_k-2 on entry), p_k-1
    double* vk1;
    double* pk;
    const double* pkm1;
    bool act[NR];  // right-hand sides still iterating (x of the others is final)
};

// Per-row tail of the U' sweep for a row of a simple block row (1x1 pivot
// d): v+ scaled in place, beta's numerator v_k' D^-1 Av, the next alpha's
// dots v+' D^-1 Av and v+' D^-1 v+, and p_k = (v_k - beta_rr p_k-1 -
// epsilon p_k-2) / rho, x += tau p_k with ||x||^2 (r[k NR + rhs]).
template <class TF, int NR>
__device__ __forceinline__ void simple_epilogue(const PArgs<TF>& a, int g, const double (&av)[NR], const double* vk,
                                                double* vk1, const double* pkm1, const double* pkm2, double* pk,
                                                const volatile Coef<NR>& cf, double (&r)[4 * NR])
{
    const double dd = (double)__ldg(a.dg + g);
#pragma unroll
    for (int j = 0; j < NR; ++j) {
        const size_t o = (size_t)g * NR + j;
        const double vkr = vk[o];
        const double vs = vk1[o] * cf.sc[j];
        vk1[o] = vs;
        if (cf.act[j]) {
            double p = vkr;
            p = fma_rn(cf.nbrr[j], pkm1[o], p);
            p = fma_rn(cf.ne[j], pkm2[o], p);
            p = p * cf.ir[j];
            pk[o] = p;
            const double xv = fma_rn(cf.tau[j], p, a.xt[o]);
            a.xt[o] = xv;
            r[3 * NR + j] = fma_rn(xv, xv, r[3 * NR + j]);
        }
        const double da = av[j] / dd, dv = vs / dd;
        r[j] = fma_rn(vkr, da, r[j]);
        r[NR + j] = fma_rn(vs, da, r[NR + j]);
        r[2 * NR + j] = fma_rn(vs, dv, r[2 * NR + j]);
    }
}

// The whole preconditioned SQMR solve of one system for NR right-hand sides
// at once (see the top of the file): every work item loads the factor and
// K once for all of them; each right-hand side has its own scalars and stops
// on its own test (its x is final from then on).
// A level's work lists: pivot-tile items [c0, c1) of citem, simple rows
// [s0, s1) of simple_rows.  The first kLvlCache levels' bounds are kept in
// shared memory for the whole solve (each phase starts by reading them).
struct LvlBounds {
    int c0, c1, s0, s1;
};
constexpr int kLvlCache = 32;

template <class TF>
__device__ __forceinline__ LvlBounds level_bounds(const PArgs<TF>& a, const SysView& sv, int L)
{
    const int q0 = __ldg(sv.qb + L), q1 = __ldg(sv.qe + L);
    return LvlBounds{__ldg(a.scan_c + q0), __ldg(a.scan_c + q1), __ldg(a.scan_s + q0), __ldg(a.scan_s + q1)};
}

// REST: a solve that another kernel began (k_sqmr_lockstep), from iteration it0
// on: S and the vectors hold its state, sc0 the scale of its level-0 Av.
template <class TF, int NR, class Ctx, bool REST = false>
__device__ void sqmr_body(const PArgs<TF>& a, Ctx& ctx, const SysView& sv, Scal (&S)[NR], double (*sh)[kW],
                          ResSlot<TF>* slots = nullptr, int it0 = 0, double sc0 = 1.0)
{
    const int tid = threadIdx.x, lane = (int)lane_id();
    const int wid = ctx.wid, nwarps = ctx.nwarps;
    const int row0 = sv.row0, row1 = sv.row1;
    __shared__ Coef<NR> cfs;  // the U' phase's coefficients, written by thread 0
    __shared__ LvlBounds lvb[kLvlCache];
    __shared__ long long npre_s;  // rows of the pivot-tile items of levels >= 1
    if (tid < kLvlCache && tid < a.nl) lvb[tid] = level_bounds(a, sv, tid);
    if (tid == 0) {
        for (int j = 0; j < NR; ++j) {
            if constexpr (!REST) {
                memset(&S[j], 0, sizeof(Scal));
                S[j].c[0] = -1.0;
            }
            cfs.sc[j] = REST ? sc0 : 1.0;  // the scale of the Av that the initial phase leaves
        }
        long long np = 0;
        for (int L = 1; L < a.nl; ++L) {
            const LvlBounds b = level_bounds(a, sv, L);
            np += 32LL * (b.c1 - b.c0);
        }
        npre_s = np;
    }
    __syncthreads();
    auto lvl = [&](int L) -> LvlBounds { return L < kLvlCache ? lvb[L] : level_bounds(a, sv, L); };
    // Two levels, level 0 all simple block rows whose K rows reach only
    // themselves and level-1 rows (a natural-order KKT system): each level-0
    // row computes its (K ev) in the U sweep, right after its ev, and the U'
    // sweep's level-0 phase and its barrier go away.  Level-0 Av is then kept
    // unscaled (the 1/delta it needs is known only after the U sweep's
    // reduction); every reader applies the scale of the iteration that wrote
    // it, at the point where the unfused path rounded it, so the results are
    // the unfused path's bit for bit.
    const bool fused = a.fuse_l0 && a.nl == 2 && lvb[0].c1 == lvb[0].c0;
    // fused grid launches hand level 1 to level 0 through the level counter
    const bool counted = fused && a.lvl_done != nullptr;
    if (a.lvl_done && blockIdx.x == 0 && tid == 0)  // read only after the initial phases' grid synchronisations
        for (int k = 0; k < 4; ++k) a.lvl_done[k] = 0;
    __shared__ LvlWait lw;
    if (tid == 0) {
        lw.seen = 0;
        lw.poll = 0;
    }
    // the calling warp's active lanes wait until the count for iteration it is
    // reached: the first warp of the CTA to get here polls global memory, the
    // others watch the CTA's shared flag; then every lane reads the counter
    // itself with an acquire load and checks it (at once satisfied, or at once
    // given up after a timeout), which orders its own later loads after every
    // CTA's release
    auto level_wait = [&](int it) {
        const unsigned mask = __activemask();
        const int want = it + 1;
        const unsigned long long target = (unsigned long long)gridDim.x * (unsigned long long)want + a.wait_skew;
        const int leader = __ffs(mask) - 1;
        if (*(volatile int*)&lw.seen < want && lane == leader) {
            if (atomicMax(&lw.poll, want) < want) {
                wait_count(a.lvl_done, target);
                __threadfence_block();
                *(volatile int*)&lw.seen = want;
            } else {
                unsigned long long t0, t;
                asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
                for (unsigned k = 0; *(volatile int*)&lw.seen < want; ++k) {
                    __nanosleep(64);
                    if ((k & 15) == 15) {
                        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
                        if (t - t0 > 2 * kWaitLimitNs) {
                            *(volatile unsigned long long*)(a.lvl_done + 1) = 1;
                            break;
                        }
                    }
                }
            }
        }
        __syncwarp(mask);
        wait_count(a.lvl_done, target);
    };

    // the level with the most pivot-tile items keeps its first kResSlots x
    // (grid) items in the warps' shared-memory slots
    __shared__ int res_level_s;
    if (tid == 0) {
        int best = -1, most = 0;
        if (slots)
            for (int L = 0; L < a.nl; ++L) {
                const LvlBounds b = lvl(L);
                if (b.c1 - b.c0 > most) {
                    most = b.c1 - b.c0;
                    best = L;
                }
            }
        res_level_s = best;
    }
    __syncthreads();
    const int res_level = res_level_s;
    ResSlot<TF>* const rs = (res_level >= 0 && (tid >> 5) < kResSlots) ? slots + (tid >> 5) : nullptr;
    int res_t = -1;  // the item of the resident level this warp holds
    if (rs) {
        const LvlBounds rb = lvl(res_level);
        const int t = rb.c0 + wid;
        res_load(a, *rs, t, t < rb.c1);
        if (t < rb.c1) res_t = t;
    }
    __syncthreads();

    // ---- init: v0 = U'^-1 P' b; ||v0|| ----
    if constexpr (!REST) {
        double one[NR];
#pragma unroll
        for (int j = 0; j < NR; ++j) one[j] = 1.0;
        for (int L = 0; L < a.nl; ++L) {
            const int r0 = __ldg(sv.qb + L), nr = __ldg(sv.qe + L) - r0;
            for (int t = wid; t < nr; t += nwarps) {
                const ItemMeta m = meta_of_row(a, __ldg(a.lvl_rows + r0 + t));
                double tt[NR];
                ut_item<TF, NR, kRhsCaller>(a, m, a.b, one, a.v[0], tt);
            }
            ctx.sync();
        }
    }
    if constexpr (!REST) {
        double r[NR];
#pragma unroll
        for (int j = 0; j < NR; ++j) r[j] = 0.0;
        for (int g = row0 + ctx.g0; g < row1; g += ctx.gstride)
#pragma unroll
            for (int j = 0; j < NR; ++j) r[j] = fma_rn(a.v[0][(size_t)g * NR + j], a.v[0][(size_t)g * NR + j], r[j]);
        ctx.template reduce<NR>(r, sh);
        if (tid == 0)
            for (int j = 0; j < NR; ++j) {
                S[j].norm_pb = sqrt(r[j]);
                S[j].gamma = S[j].norm_pb;
                S[j].inv_pb = 1.0 / S[j].norm_pb;
            }
        __syncthreads();
    }
    // v0 /= ||v0|| (in place), ev = P U^-1 D^-1 v0, ||D^-1 v0||^2
    double ww[NR];
#pragma unroll
    for (int j = 0; j < NR; ++j) ww[j] = 0.0;
    if constexpr (!REST) {
        double inv_pb[NR];
#pragma unroll
        for (int j = 0; j < NR; ++j) inv_pb[j] = S[j].inv_pb;
        for (int L = a.nl - 1; L >= 0; --L) {
            const int r0 = __ldg(sv.qb + L), nr = __ldg(sv.qe + L) - r0;
            for (int t = wid; t < nr; t += nwarps) {
                const ItemMeta m = meta_of_row(a, __ldg(a.lvl_rows + r0 + t));
                const int fr = m.fr, h = m.h;
                double y[NR], d[NR];
#pragma unroll
                for (int j = 0; j < NR; ++j) {
                    y[j] = 0.0;
                    if (lane < h) {
                        const size_t o = (size_t)(fr + lane) * NR + j;
                        y[j] = a.v[0][o] * inv_pb[j];
                        a.v[0][o] = y[j];
                    }
                }
                u_item<TF, NR>(a, m, y, a.ev, d);
#pragma unroll
                for (int j = 0; j < NR; ++j) ww[j] = fma_rn(d[j], d[j], ww[j]);
            }
            ctx.sync();
        }
    }
    // Av = U'^-1 P' K ev; alpha's dots for iteration 0; eta_0 = 1/||D^-1 v0||
    if constexpr (!REST) {
        double r[3 * NR];
        double one[NR];
#pragma unroll
        for (int j = 0; j < NR; ++j) {
            r[j] = ww[j];
            r[NR + j] = 0.0;
            r[2 * NR + j] = 0.0;
            one[j] = 1.0;
        }
        for (int L = 0; L < a.nl; ++L) {
            const int r0 = __ldg(sv.qb + L), nr = __ldg(sv.qe + L) - r0;
            for (int t = wid; t < nr; t += nwarps) {
                const ItemMeta m = meta_of_row(a, __ldg(a.lvl_rows + r0 + t));
                const int fr = m.fr, h = m.h, flags = m.flags;
                double av[NR];
                ut_item<TF, NR, kRhsSpmv>(a, m, a.ev, one, a.Av, av);
                DBlock<TF> D;
                D.load(a, fr, h, flags);
#pragma unroll
                for (int j = 0; j < NR; ++j) {
                    const double vs = (lane < h) ? a.v[0][(size_t)(fr + lane) * NR + j] : 0.0;
                    const double da = D.apply(av[j], h), dv = D.apply(vs, h);
                    if (lane < h) {
                        r[NR + j] = fma_rn(vs, da, r[NR + j]);
                        r[2 * NR + j] = fma_rn(vs, dv, r[2 * NR + j]);
                    }
                }
            }
            if (L < a.nl - 1) ctx.sync();
        }
        ctx.template reduce<3 * NR>(r, sh);
        if (tid == 0)
            for (int j = 0; j < NR; ++j) {
                S[j].eta = 1.0 / sqrt(r[j]);
                S[j].alpha_next = r[NR + j] / r[2 * NR + j];
                S[j].vdv = r[2 * NR + j];
                if (!isfinite(S[j].inv_pb) || !isfinite(S[j].eta)) {
                    S[j].breakdown = 1;
                    S[j].done = 1;
                }
            }
        __syncthreads();
    }

    // the counted iteration has no ctx.sync() between here and the loop's end
    if (counted && a.count_red) ctx.begin_counted(a.lvl_done, a.red_skew);
    int it = REST ? it0 : 0;
    for (;;) {
        bool any = false;
#pragma unroll
        for (int j = 0; j < NR; ++j) any |= !S[j].done;
        if (!any || it >= a.max_it) break;
        const int k0 = acc3(it), k1 = acc3(it + 1), km1 = acc3(it - 1);
        if (NR == 1) stamp(a.ts, it, 0);
        // -alpha and -beta_k of each right-hand side, read from shared memory
        // where used (registers are the kernel's scarce resource)
        if (tid == 0) {
            for (int j = 0; j < NR; ++j) {
                cfs.na[j] = -S[j].alpha_next;
                cfs.nb[j] = -S[j].beta[k0];
            }
            cfs.vk = a.v[it & 1];
            cfs.vk1 = a.v[(it + 1) & 1];
            cfs.pk = a.p[it & 1];
            cfs.pkm1 = a.p[(it + 1) & 1];
        }
        __syncthreads();
        const volatile Coef<NR>& cv = cfs;
        const volatile double* const na = cfs.na;
        const volatile double* const nb = cfs.nb;
        // ---- U sweep on v+ = Av - alpha v - beta v- (each item computes and
        //      stores its rows' v+, kept unscaled), ||v+||^2 ----
        {
            double r[NR];
#pragma unroll
            for (int j = 0; j < NR; ++j) r[j] = 0.0;
            for (int L = a.nl - 1; L >= 0; --L) {
                const LvlBounds lb = lvl(L);
                // block rows with a pivot tile, swaps or 2x2 pivots: warp per block row
                const int c1 = lb.c1;
                for (int t = lb.c0 + wid; t < c1; t += nwarps) {
                    const bool res = (t == res_t && L == res_level);
                    const ItemMeta m = res ? rs->m : meta_of_item(a, t);
                    const int fr = m.fr, h = m.h;
                    double y[NR], d[NR];
#pragma unroll
                    for (int j = 0; j < NR; ++j) {
                        y[j] = 0.0;
                        if (lane < h) {
                            const size_t o = (size_t)(fr + lane) * NR + j;
                            double v = a.Av[o];
                            double* const vk1 = cv.vk1;  // vk1 holds v_k-1 until written
                            v = fma_rn(na[j], cv.vk[o], v);
                            v = fma_rn(nb[j], vk1[o], v);
                            vk1[o] = v;
                            r[j] = fma_rn(v, v, r[j]);
                            y[j] = v;
                        }
                    }
                    if (res) u_item_res<TF, NR>(a, *rs, y, a.ev, d);
                    else u_item<TF, NR>(a, m, y, a.ev, d);
                }
                // rows of simple block rows: thread per row (u_item with D = d,
                // an identity tile and no swaps)
                const int s1 = lb.s1;
                const bool fz = fused && L == 0;
                bool ready = !(counted && L == 0);
                for (int i = lb.s0 + ctx.g0; i < s1; i += ctx.gstride) {
                    const int g = __ldg(a.simple_rows + i);
                    const double dd = (double)__ldg(a.dg + g);
                    TF acc[NR];
#pragma unroll
                    for (int j = 0; j < NR; ++j) {
                        const size_t o = (size_t)g * NR + j;
                        // fused level 0: Av holds the last iteration's unscaled (K ev)
                        double v = fz ? (double)(TF)(a.Av[o] * cv.sc[j]) : a.Av[o];
                        double* const vk1 = cv.vk1;
                        v = fma_rn(na[j], cv.vk[o], v);
                        v = fma_rn(nb[j], vk1[o], v);
                        vk1[o] = v;
                        r[j] = fma_rn(v, v, r[j]);
                        acc[j] = (TF)(v / dd);
                    }
                    if (!ready) {
                        // v+ and D^-1 v+ above need no level-1 value; the gathers below do
                        level_wait(it);
                        ready = true;
                    }
                    const int2 kr = __ldg(a.u_rng + g);
                    row_sub<TF, NR>(acc, kr.x, kr.y, a.u_colp, a.u_val, a.ev);
#pragma unroll
                    for (int j = 0; j < NR; ++j) a.ev[(size_t)g * NR + j] = (double)acc[j];
                    if (fz) {
                        // K row g reaches only ev[g] (written just above) and level-1
                        // rows (final since the last barrier)
                        double y[NR];
                        spmv_row<TF, NR>(a, g, a.ev, y);
#pragma unroll
                        for (int j = 0; j < NR; ++j) a.Av[(size_t)g * NR + j] = y[j];
                    }
                }
                if (L > 0) {
                    if (counted) {
                        // this CTA's level-1 rows are written: count it (release);
                        // level-0 rows wait for every CTA's count before reading them
                        __syncthreads();
                        if (tid == 0) red_release_add_u64(a.lvl_done, 1ull);
                    } else {
                        ctx.sync();
                    }
                    if (NR == 1 && L == a.nl - 1) stamp(a.ts, it, 1);
                }
            }
            const bool ok = ctx.template reduce<NR>(r, sh);
            if (tid == 0 && !ok) abandon<NR>(S, it);
            if (tid == 0)
                for (int j = 0; j < NR; ++j) {
                    if (S[j].done) continue;
                    scal_after_u(S[j], r[j], k0, k1, km1);
                }
            if (tid == 0)
                for (int j = 0; j < NR; ++j) {
                    cfs.sc[j] = S[j].inv_delta;
                    cfs.nbrr[j] = -S[j].beta_rr;
                    cfs.ne[j] = -S[j].epsilon;
                    cfs.ir[j] = S[j].inv_rho;
                    cfs.tau[j] = S[j].tau;
                    cfs.act[j] = !S[j].done;
                }
            __syncthreads();
        }
        if (NR == 1) {
            if (a.nl == 1) stamp(a.ts, it, 1);
            stamp(a.ts, it, 2);
        }
        // ---- U' sweep with the fused SpMV; beta's and alpha's dots; p, x ----
        {
            double r[4 * NR];
#pragma unroll
            for (int j = 0; j < 4 * NR; ++j) r[j] = 0.0;
            const volatile Coef<NR>& cf = cfs;
            for (int L = 0; L < a.nl; ++L) {
                // fused: level 0 has no items and its rows' products are done
                if (fused && L == 0) continue;
                const LvlBounds lb = lvl(L);
                const int c1 = lb.c1;
                for (int t = lb.c0 + wid; t < c1; t += nwarps) {
                    const bool res = (t == res_t && L == res_level);
                    const ItemMeta m = res ? rs->m : meta_of_item(a, t);
                    const int fr = m.fr, h = m.h, flags = m.flags;
                    double av[NR];
                    double scv[NR];
#pragma unroll
                    for (int j = 0; j < NR; ++j) scv[j] = cf.sc[j];
                    DBlock<TF> D;
                    if (res) {
                        if (fused) ut_item_res<TF, NR, kRhsSpmv, true>(a, *rs, a.ev, scv, a.Av, av);
                        else if (L == 0) ut_item_res<TF, NR, kRhsSpmv>(a, *rs, a.ev, scv, a.Av, av);
                        else ut_item_res<TF, NR, kRhsPre>(a, *rs, a.ev, scv, a.Av, av);
                        D = dblock_res(a, *rs);
                    } else {
                        if (fused) ut_item<TF, NR, kRhsSpmv, true>(a, m, a.ev, scv, a.Av, av);
                        else if (L == 0) ut_item<TF, NR, kRhsSpmv>(a, m, a.ev, scv, a.Av, av);
                        else ut_item<TF, NR, kRhsPre>(a, m, a.ev, scv, a.Av, av);
                        D.load(a, fr, h, flags);
                    }
#pragma unroll
                    for (int j = 0; j < NR; ++j) {
                        double vkr = 0.0, vs = 0.0;
                        if (lane < h) {
                            const size_t o = (size_t)(fr + lane) * NR + j;
                            double* const vk1 = cv.vk1;
                            vkr = cv.vk[o];
                            vs = vk1[o] * cf.sc[j];
                            vk1[o] = vs;
                            if (cf.act[j]) {
                                // p_k = (v_k - beta_rr p_k-1 - epsilon p_k-2) / rho, x += tau p_k
                                double p = vkr;
                                double* const pk = cv.pk;  // holds p_k-2 until written
                                p = fma_rn(cf.nbrr[j], cv.pkm1[o], p);
                                p = fma_rn(cf.ne[j], pk[o], p);
                                p = p * cf.ir[j];
                                pk[o] = p;
                                const double xv = fma_rn(cf.tau[j], p, a.xt[o]);
                                a.xt[o] = xv;
                                r[3 * NR + j] = fma_rn(xv, xv, r[3 * NR + j]);
                            }
                        }
                        const double da = D.apply(av[j], h), dv = D.apply(vs, h);
                        if (lane < h) {
                            r[j] = fma_rn(vkr, da, r[j]);
                            r[NR + j] = fma_rn(vs, da, r[NR + j]);
                            r[2 * NR + j] = fma_rn(vs, dv, r[2 * NR + j]);
                        }
                    }
                }
                // simple rows of this level: Av; their dots and the p / x
                // update wait for the next level's phase, whose threads are
                // mostly free (the last level does them at once)
                const bool last = (L == a.nl - 1);
                const int s0 = lb.s0, s1 = lb.s1;
                // Level 0 also computes (K ev) / delta for the rows of the later
                // levels' pivot-tile block rows and leaves it in Av at those rows:
                // their items read it there instead of running the product on
                // the critical path of a level of few, long items.  Units
                // [0, npre) are those rows (lane ln of item t), the rest this
                // level's simple rows, both spread over all threads.
                const long long npre = (L == 0) ? npre_s : 0;
                const long long nunits = npre + (s1 - s0);
                for (long long k = ctx.g0; k < nunits; k += ctx.gstride) {
                    if (k < npre) {
                        long long u = k;
                        int L2 = 1;
                        LvlBounds b2 = lvl(L2);
                        for (;;) {
                            const long long len = 32LL * (b2.c1 - b2.c0);
                            if (u < len) break;
                            u -= len;
                            b2 = lvl(++L2);
                        }
                        const ItemMeta m = meta_of_item(a, b2.c0 + (int)(u >> 5));
                        const int ln = (int)(u & 31), fr = m.fr;
                        if (ln < m.h) {
                            double y[NR];
                            spmv_row<TF, NR>(a, fr + ln, a.ev, y);
#pragma unroll
                            for (int j = 0; j < NR; ++j) a.Av[(size_t)(fr + ln) * NR + j] = y[j] * cf.sc[j];
                        }
                        continue;
                    }
                    const int g = __ldg(a.simple_rows + s0 + (int)(k - npre));
                    double y[NR];
                    spmv_row<TF, NR>(a, g, a.ev, y);
                    TF acc[NR];
                    double scv[NR];
#pragma unroll
                    for (int j = 0; j < NR; ++j) {
                        scv[j] = cf.sc[j];
                        acc[j] = (TF)(y[j] * scv[j]);
                    }
                    const int2 kr = __ldg(a.ut_rng + g);
                    if (fused)  // level 1: its U' rows gather the unscaled level-0 Av
                        row_sub<TF, NR, true>(acc, kr.x, kr.y, a.ut_col, a.ut_val, a.Av, scv);
                    else
                        row_sub<TF, NR>(acc, kr.x, kr.y, a.ut_col, a.ut_val, a.Av);
                    double av[NR];
#pragma unroll
                    for (int j = 0; j < NR; ++j) {
                        av[j] = (double)acc[j];
                        a.Av[(size_t)g * NR + j] = av[j];
                    }
                    if (last) simple_epilogue<TF, NR>(a, g, av, cv.vk, cv.vk1, cv.pkm1, cv.pk, cv.pk, cf, r);
                }
                if (L > 0) {
                    // warps without a block row in this level take the tails;
                    // if every warp has one, all threads do, after their items
                    const LvlBounds pb = lvl(L - 1);
                    const int e1 = pb.s1;
                    const int items = c1 - lb.c0;
                    const bool spare = items < nwarps;
                    if (!spare || wid >= items) {
                        const int t0 = spare ? (wid - items) * 32 + lane : ctx.g0;
                        const int ts = spare ? (nwarps - items) * 32 : ctx.gstride;
                        for (int i = pb.s0 + t0; i < e1; i += ts) {
                            const int g = __ldg(a.simple_rows + i);
                            double av[NR];
#pragma unroll
                            for (int j = 0; j < NR; ++j) {
                                const double w = a.Av[(size_t)g * NR + j];
                                av[j] = (fused && L == 1) ? (double)(TF)(w * cf.sc[j]) : w;
                            }
                            simple_epilogue<TF, NR>(a, g, av, cv.vk, cv.vk1, cv.pkm1, cv.pk, cv.pk, cf, r);
                        }
                    }
                }
                if (L < a.nl - 1) {
                    ctx.sync();
                    if (NR == 1 && L == 0) stamp(a.ts, it, 4);
                }
            }
            const bool ok = ctx.template reduce<4 * NR>(r, sh);
            if (tid == 0 && !ok) abandon<NR>(S, it);
            if (tid == 0)
                for (int j = 0; j < NR; ++j) {
                    if (S[j].done) continue;
                    scal_after_ut(S[j], r[j], r[NR + j], r[2 * NR + j], r[3 * NR + j], it, k1, a.tol, a.max_it);
                }
            __syncthreads();
        }
        if (NR == 1) stamp(a.ts, it, 3);
        bool more = false;
#pragma unroll
        for (int j = 0; j < NR; ++j) more |= !S[j].done;
        if (more) ++it;
        else break;
    }
    // ---- x = P U^-1 D^-1 x~ into ev, then x (column-major) ----
    for (int L = a.nl - 1; L >= 0; --L) {
        const int r0 = __ldg(sv.qb + L), nr = __ldg(sv.qe + L) - r0;
        for (int t = wid; t < nr; t += nwarps) {
            const ItemMeta m = meta_of_row(a, __ldg(a.lvl_rows + r0 + t));
            const int fr = m.fr, h = m.h;
            double y[NR], d[NR];
#pragma unroll
            for (int j = 0; j < NR; ++j) y[j] = (lane < h) ? a.xt[(size_t)(fr + lane) * NR + j] : 0.0;
            u_item<TF, NR>(a, m, y, a.ev, d);
        }
        ctx.sync();
    }
    for (int g = row0 + ctx.g0; g < row1; g += ctx.gstride)
#pragma unroll
        for (int j = 0; j < NR; ++j) a.x[(size_t)j * a.n + g] = a.ev[(size_t)g * NR + j];
    if (sv.out && tid == 0)
        for (int j = 0; j < NR; ++j) {
            const Scal& Q = S[j];
            double* o = sv.out + 8 * j;
            o[0] = Q.gamma / Q.norm_pb;
            o[1] = Q.done ? Q.iters : it;
            o[2] = Q.breakdown;
            o[3] = (Q.snap0 || Q.snap1) ? 1 : 0;
            o[4] = Q.norm_pb;
            o[5] = Q.done ? Q.stop_it : it;
            // a bounded wait that gave up: the results are invalid
            o[6] = (a.lvl_done && (*(volatile unsigned long long*)(a.lvl_done + 1) ||
                                   *(volatile unsigned long long*)(a.lvl_done + 3)))
                       ? 1.0
                       : 0.0;
            if (o[6] != 0.0) o[2] = 1.0;
        }
    __syncthreads();
}

// launched with kResSlots ResSlot<TF> of dynamic shared memory
template <class TF, int CTAS, int NR>
__global__ void __launch_bounds__(kT, CTAS) k_sqmr_persistent(PArgs<TF> a)
{
    __shared__ Scal S[NR];
    __shared__ double sh[kMaxNV][kW];
    extern __shared__ __align__(16) unsigned char res_smem[];
    const int G = gridDim.x;
    GridCtx ctx{cg::this_grid(), a.partials, 0, (int)(threadIdx.x >> 5) * G + (int)blockIdx.x,  // items interleaved
                G * kW, (int)(blockIdx.x * kT + threadIdx.x), G * kT, nullptr, 0, 0ull};
    const SysView sv{0, a.n, a.lvl_off, a.lvl_off + 1, blockIdx.x == 0 ? a.out : nullptr};
    sqmr_body<TF, NR>(a, ctx, sv, S, sh, reinterpret_cast<ResSlot<TF>*>(res_smem));
}

template <class TF>
constexpr size_t res_smem_bytes()
{
    return (size_t)kResSlots * sizeof(ResSlot<TF>);
}

// Batched solves of independent systems stored as one block-diagonal union
// (one pattern, one factor): each CTA takes the next unsolved system from a
// counter and runs its whole SQMR with CTA barriers only.  A system's result
// does not depend on the others or on which CTA solves it.
struct BatchArgs {
    int num;
    const int* row_off;  // num + 1
    const int* qb;       // num x nl
    const int* qe;
    double* out;         // num x 8
    int* next;           // counter, 0 at launch
};

template <class TF>
__global__ void __launch_bounds__(kT, kCtasPerSm) k_sqmr_batched(PArgs<TF> a, BatchArgs bt)
{
    __shared__ Scal S[1];
    __shared__ double sh[kMaxNV][kW];
    __shared__ int sys;
    CtaCtx ctx{(int)(threadIdx.x >> 5), kW, (int)threadIdx.x, kT};
    for (;;) {
        if (threadIdx.x == 0) sys = atomicAdd(bt.next, 1);
        __syncthreads();
        const int s = sys;
        __syncthreads();
        if (s >= bt.num) break;
        const SysView sv{__ldg(bt.row_off + s), __ldg(bt.row_off + s + 1), bt.qb + (size_t)s * a.nl,
                         bt.qe + (size_t)s * a.nl, bt.out + (size_t)s * 8};
        sqmr_body<TF, 1>(a, ctx, sv, S, sh);
    }
}

// One system's coefficients in k_sqmr_lockstep, read by the units of the next
// phase
struct alignas(16) LockCoef {
    double na, nb;              // U sweep: -alpha, -beta_k
    double sc;                  // 1 / delta (the scale of level-0 Av)
    double nbrr, ne, ir, tau;   // p / x update
    int act, pad;               // still iterating
};

// The systems that k_sqmr_lockstep left unfinished (small ones, once every
// larger system has stopped), a CTA each from its iteration `at` on.
template <class TF>
__global__ void __launch_bounds__(kT, kCtasPerSm)
    k_sqmr_rest(PArgs<TF> a, BatchArgs bt, const Scal* scal, const LockCoef* coef, const int* at)
{
    __shared__ Scal S[1];
    __shared__ double sh[kMaxNV][kW];
    __shared__ int sys;
    CtaCtx ctx{(int)(threadIdx.x >> 5), kW, (int)threadIdx.x, kT};
    const int it0 = *at;
    if (it0 >= a.max_it) return;
    for (;;) {
        if (threadIdx.x == 0) sys = atomicAdd(bt.next, 1);
        __syncthreads();
        const int s = sys;
        __syncthreads();
        if (s >= bt.num) break;
        if (!coef[s].act) continue;
        if (threadIdx.x == 0) S[0] = scal[s];
        const SysView sv{__ldg(bt.row_off + s), __ldg(bt.row_off + s + 1), bt.qb + (size_t)s * a.nl,
                         bt.qe + (size_t)s * a.nl, bt.out + (size_t)s * 8};
        sqmr_body<TF, 1, CtaCtx, true>(a, ctx, sv, S, sh, nullptr, it0, coef[s].sc);
    }
}

// Batched solves of independent systems that each have their own pattern,
// factor, matrix and vectors (the serving path): the CTA copies system s's
// argument block into shared memory and runs the same body over its rows,
// for nr[s] (1, 2 or 4) right-hand sides of that system at once.  Systems are
// handed out in index order, so the host lists the longest first.  MULTI =
// false compiles the one-right-hand-side body alone (every nr[s] == 1): the
// 2- and 4-wide bodies in the same kernel cost the common case registers.
template <class TF, bool MULTI>
__global__ void __launch_bounds__(kT, kCtasPerSm) k_sqmr_many(const PArgs<TF>* __restrict__ sys_args,
                                                             const int* __restrict__ nr, int num, int* next)
{
    __shared__ Scal S[kMaxNR];
    __shared__ double sh[kMaxNV][kW];
    __shared__ int sys;
    __shared__ PArgs<TF> pa;
    static_assert(sizeof(PArgs<TF>) % 8 == 0, "argument block copied in 8-byte words");
    CtaCtx ctx{(int)(threadIdx.x >> 5), kW, (int)threadIdx.x, kT};
    for (;;) {
        if (threadIdx.x == 0) sys = atomicAdd(next, 1);
        __syncthreads();
        const int s = sys;
        if (s >= num) break;
        const unsigned long long* src = reinterpret_cast<const unsigned long long*>(sys_args + s);
        unsigned long long* dst = reinterpret_cast<unsigned long long*>(&pa);
        for (int i = threadIdx.x; i < (int)(sizeof(PArgs<TF>) / 8); i += kT) dst[i] = src[i];
        __syncthreads();
        const SysView sv{0, pa.n, pa.lvl_off, pa.lvl_off + 1, pa.out};
        if constexpr (MULTI) {
            const int r = __ldg(nr + s);
            if (r == 4) sqmr_body<TF, 4>(pa, ctx, sv, reinterpret_cast<Scal(&)[4]>(S), sh);
            else if (r == 2) sqmr_body<TF, 2>(pa, ctx, sv, reinterpret_cast<Scal(&)[2]>(S), sh);
            else sqmr_body<TF, 1>(pa, ctx, sv, reinterpret_cast<Scal(&)[1]>(S), sh);
        } else {
            sqmr_body<TF, 1>(pa, ctx, sv, reinterpret_cast<Scal(&)[1]>(S), sh);
        }
    }
}

// The kernels' addresses.  Each is defined in one translation unit of its own
// (sqmr_kernels_*.cu): every body takes the compiler some twenty seconds.
template <class TF, int CTAS, int NR>
const void* persistent_fn();
template <class TF>
const void* batched_fn();
template <class TF>
const void* rest_fn();
template <class TF, bool MULTI>
const void* many_fn();

#define CULIPX_SQMR_DECLARE(TF)                            \
    template <> const void* persistent_fn<TF, 1, 1>();     \
    template <> const void* persistent_fn<TF, 2, 1>();     \
    template <> const void* persistent_fn<TF, 1, 2>();     \
    template <> const void* persistent_fn<TF, 2, 2>();     \
    template <> const void* persistent_fn<TF, 1, 4>();     \
    template <> const void* persistent_fn<TF, 2, 4>();     \
    template <> const void* batched_fn<TF>();              \
    template <> const void* rest_fn<TF>();                 \
    template <> const void* many_fn<TF, false>();          \
    template <> const void* many_fn<TF, true>();
CULIPX_SQMR_DECLARE(double)
CULIPX_SQMR_DECLARE(float)

#define CULIPX_SQMR_PERSISTENT(TF, CTAS, NR)          \
    template <>                                       \
    const void* persistent_fn<TF, CTAS, NR>()         \
    {                                                 \
        return (const void*)k_sqmr_persistent<TF, CTAS, NR>; \
    }
#define CULIPX_SQMR_BATCHED(TF)                \
    template <>                                \
    const void* batched_fn<TF>()               \
    {                                          \
        return (const void*)k_sqmr_batched<TF>; \
    }
#define CULIPX_SQMR_REST(TF)                \
    template <>                             \
    const void* rest_fn<TF>()               \
    {                                       \
        return (const void*)k_sqmr_rest<TF>; \
    }
#define CULIPX_SQMR_MANY(TF, MULTI)                \
    template <>                                    \
    const void* many_fn<TF, MULTI>()               \
    {                                              \
        return (const void*)k_sqmr_many<TF, MULTI>; \
    }

}  // namespace persistent

}  // namespace culipx
