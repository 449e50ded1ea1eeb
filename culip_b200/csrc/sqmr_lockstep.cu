// Batched SQMR on the whole grid: all systems of a batch take their iterations
// together, in one cooperative launch.
//
// k_sqmr_batched gives a system to one CTA for its whole solve, so a batch of
// uneven systems lasts as long as its largest one on a single CTA (256
// systems, n log-uniform in [500, 20000], FP32 factor: 0.84 ms per iteration,
// of which the device was mostly idle).  Here each phase of an iteration runs
// over the rows of every system that is still iterating, spread evenly over
// the grid:
//   U     level-1 tiles: v+, U sweep                       | grid sync
//         level-0 rows: v+, U sweep, (K ev) kept unscaled  | grid sync
//         a CTA per system: ||v+||^2, the rotation         | grid sync
//   U'    level-1 tiles: SpMV, U' sweep, D^-1, p, x;
//         level-0 rows: D^-1, p, x                         | grid sync
//         a CTA per system: the dots, ||x||, tests         | grid sync
// (the level-0 fusion of sqmr_persistent.cuh, so for two-level factors only;
// others keep k_sqmr_batched).  A work unit is a warp's: one level-1 block row
// or up to 32 level-0 rows of one system.  A system's result does not depend
// on the others, on its place in the batch or on the grid: its sums are taken
// by one CTA over the rows' stored terms.
//
// The iterations end when no system of more than kLockRows rows is left: the
// small ones, whose count may be many times the large ones', go on in
// k_sqmr_rest with a CTA each (one easy system of 30 000 rows and 40 hard ones
// of 450: 17.0 ms all on the grid, 9.2 so, 22.5 with a CTA each from the start;
// of 9000 rows and 100 of 450: 23.7, 9.0 and 7.7).
//
// Bound: latency.  256 systems of 2.0 M rows, FP32 factor: half of the waiting at
// the barriers of the five phases, half for dependent loads; DRAM, L2 and L1 at
// 25, 24 and 33 % of their peaks, 0.46 ms an iteration.
#include "sqmr_persistent.cuh"
#include "sqmr_lockstep.h"

namespace culipx {

namespace persistent {

namespace {

struct LockArgs {
    int num, chunks, tiles;
    const int4* chunk;  // level-0 rows: first position in the level list, rows, system
    const int4* tile;   // level-1 block rows: block row, first row, rows, system
    const int* row_off; // per system its rows, and its block rows per level
    const int* qb;
    const int* qe;
    double* da;         // per row D^-1 Av and D^-1 v+
    double* dv;
    Scal* scal;
    LockCoef* coef;
    int* active;        // [0] systems of more than kLockRows rows still iterating, [1] iterations taken
    double* out;        // num x 8
};

__device__ __forceinline__ bool large(const LockArgs& k, int s)
{
    return __ldg(k.row_off + s + 1) - __ldg(k.row_off + s) > kLockRows;
}

template <class TF>
__device__ __forceinline__ ItemMeta meta_of_tile(const PArgs<TF>& a, const int4& t)
{
    ItemMeta m;
    m.I = t.x;
    m.fr = t.y;
    m.h = t.z;
    m.flags = __ldg(a.rowflags + t.x);
    m.pko = __ldg(a.pk_off + t.x);
    m.nd = __ldg(a.ndmask + t.x);
    return m;
}

// The sums of one system, by one CTA, over the rows' stored factors: thread by
// thread the terms of k_sqmr_batched's CTA and in its order (the iterates of an
// FP32 factor depend on it), so both kernels give the same bits.
//
// f(row) adds a row's terms to r.  Block rows of level L, warp by warp:
template <class TF, class F>
__device__ __forceinline__ void over_block_rows(const PArgs<TF>& a, const SysView& sv, int L, F f)
{
    const int lane = (int)lane_id(), w = threadIdx.x >> 5;
    const int q1 = __ldg(sv.qe + L);
#pragma unroll 4
    for (int q = __ldg(sv.qb + L) + w; q < q1; q += kW) {
        const int I = __ldg(a.lvl_rows + q);
        const int fr = __ldg(a.bs + I);
        if (fr + lane < __ldg(a.bs + I + 1)) f(fr + lane);
    }
}

// The pivot-tile items [c0, c1), warp by warp
template <class TF, class F>
__device__ __forceinline__ void over_items(const PArgs<TF>& a, const LvlBounds& b, F f)
{
    const int lane = (int)lane_id(), w = threadIdx.x >> 5;
#pragma unroll 4
    for (int t = b.c0 + w; t < b.c1; t += kW) {
        const int4 u = __ldg(reinterpret_cast<const int4*>(a.citem + t));
        if (lane < u.z) f(u.y + lane);
    }
}

// The simple rows at places i0, i0 + step, ... of [s0, s1) of the list.  The
// list ascends, so a run without gaps (a system of a batch in natural order)
// is known by its ends and needs no index loads.
template <class TF, class F>
__device__ __forceinline__ void over_simple(const PArgs<TF>& a, int s0, int s1, int first, int step, F f)
{
    if (s0 >= s1) return;
    const int g0 = __ldg(a.simple_rows + s0);
    if (__ldg(a.simple_rows + s1 - 1) - g0 == s1 - 1 - s0) {
#pragma unroll 8
        for (int i = first; i < s1 - s0; i += step) f(g0 + i);
    } else {
#pragma unroll 4
        for (int i = first; i < s1 - s0; i += step) f(__ldg(a.simple_rows + s0 + i));
    }
}

// U sweep of a level-0 row that starts from y (already in the caller's
// vector): D^-1 y less the level-1 values of `out`
template <class TF>
__device__ __forceinline__ double level0_u(const PArgs<TF>& a, int g, double d, const double* out)
{
    TF acc[1] = {(TF)d};
    const int2 kr = __ldg(a.u_rng + g);
    row_sub<TF, 1>(acc, kr.x, kr.y, a.u_colp, a.u_val, out);
    return (double)acc[0];
}

template <class TF>
__global__ void __launch_bounds__(kT, kCtasPerSm) k_sqmr_lockstep(PArgs<TF> a, LockArgs k)
{
    cg::grid_group grid = cg::this_grid();
    const int lane = (int)lane_id();
    const int wid = (int)(threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    const int nw = gridDim.x * kW;
    const int tid = threadIdx.x;
    const double one[1] = {1.0};
    __shared__ double sh[kMaxNV][kW];

    // ---- v0 = U'^-1 P' b; ||v0|| ----
    for (int c = wid; c < k.chunks; c += nw) {
        const int4 u = __ldg(k.chunk + c);
        if (lane < u.y) {
            const int g = __ldg(a.simple_rows + u.x + lane);
            a.v[0][g] = (double)(TF)a.b[g];
        }
    }
    grid.sync();
    for (int t = wid; t < k.tiles; t += nw) {
        const ItemMeta m = meta_of_tile(a, __ldg(k.tile + t));
        double v[1];
        ut_item<TF, 1, kRhsCaller>(a, m, a.b, one, a.v[0], v);
    }
    grid.sync();
    for (int s = blockIdx.x; s < k.num; s += gridDim.x) {
        double r[1] = {0.0};
        const int row1 = __ldg(k.row_off + s + 1);
#pragma unroll 4
        for (int g = __ldg(k.row_off + s) + tid; g < row1; g += kT) r[0] = fma_rn(a.v[0][g], a.v[0][g], r[0]);
        cta_reduce<1>(r, sh);
        if (tid == 0) {
            Scal& Q = k.scal[s];
            memset(&Q, 0, sizeof(Scal));
            Q.c[0] = -1.0;
            Q.norm_pb = sqrt(r[0]);
            Q.gamma = Q.norm_pb;
            Q.inv_pb = 1.0 / Q.norm_pb;
            k.coef[s].sc = Q.inv_pb;
        }
        __syncthreads();
    }
    grid.sync();
    // ---- v0 /= ||v0||, ev = P U^-1 D^-1 v0 (D^-1 v0 kept in da), level-0 (K ev) ----
    for (int t = wid; t < k.tiles; t += nw) {
        const int4 u = __ldg(k.tile + t);
        const ItemMeta m = meta_of_tile(a, u);
        double y[1] = {0.0}, d[1];
        if (lane < m.h) {
            y[0] = a.v[0][m.fr + lane] * k.coef[u.w].sc;
            a.v[0][m.fr + lane] = y[0];
        }
        u_item<TF, 1>(a, m, y, a.ev, d);
        if (lane < m.h) k.da[m.fr + lane] = d[0];
    }
    grid.sync();
    for (int c = wid; c < k.chunks; c += nw) {
        const int4 u = __ldg(k.chunk + c);
        if (lane < u.y) {
            const int g = __ldg(a.simple_rows + u.x + lane);
            const double y = a.v[0][g] * k.coef[u.z].sc;
            a.v[0][g] = y;
            const double d = y / (double)__ldg(a.dg + g);
            k.da[g] = d;
            a.ev[g] = level0_u(a, g, d, a.ev);
            double w[1];
            spmv_row<TF, 1>(a, g, a.ev, w);
            a.Av[g] = w[0];
        }
    }
    grid.sync();
    for (int s = blockIdx.x; s < k.num; s += gridDim.x) {
        const SysView sv{0, 0, k.qb + 2 * s, k.qe + 2 * s, nullptr};
        double r[1] = {0.0};
        auto add = [&](int g) { r[0] = fma_rn(k.da[g], k.da[g], r[0]); };
        over_block_rows(a, sv, 1, add);
        over_block_rows(a, sv, 0, add);
        cta_reduce<1>(r, sh);
        if (tid == 0) k.scal[s].eta = 1.0 / sqrt(r[0]);
        __syncthreads();
    }
    grid.sync();
    // ---- Av = U'^-1 P' K ev; alpha's dots for iteration 0 ----
    for (int t = wid; t < k.tiles; t += nw) {
        const ItemMeta m = meta_of_tile(a, __ldg(k.tile + t));
        double av[1];
        ut_item<TF, 1, kRhsSpmv, true>(a, m, a.ev, one, a.Av, av);
        DBlock<TF> D;
        D.load(a, m.fr, m.h, m.flags);
        const double vs = (lane < m.h) ? a.v[0][m.fr + lane] : 0.0;
        const double da = D.apply(av[0], m.h), dv = D.apply(vs, m.h);
        if (lane < m.h) {
            k.da[m.fr + lane] = da;
            k.dv[m.fr + lane] = dv;
        }
    }
    for (int c = wid; c < k.chunks; c += nw) {
        const int4 u = __ldg(k.chunk + c);
        if (lane < u.y) {
            const int g = __ldg(a.simple_rows + u.x + lane);
            const double dd = (double)__ldg(a.dg + g);
            k.da[g] = (double)(TF)a.Av[g] / dd;
            k.dv[g] = a.v[0][g] / dd;
        }
    }
    grid.sync();
    for (int s = blockIdx.x; s < k.num; s += gridDim.x) {
        const SysView sv{0, 0, k.qb + 2 * s, k.qe + 2 * s, nullptr};
        double r[2] = {0.0, 0.0};
        auto add = [&](int g) {
            const double vs = a.v[0][g];
            r[0] = fma_rn(vs, k.da[g], r[0]);
            r[1] = fma_rn(vs, k.dv[g], r[1]);
        };
        over_block_rows(a, sv, 0, add);
        over_block_rows(a, sv, 1, add);
        cta_reduce<2>(r, sh);
        if (tid == 0) {
            Scal& Q = k.scal[s];
            Q.alpha_next = r[0] / r[1];
            Q.vdv = r[1];
            if (!isfinite(Q.inv_pb) || !isfinite(Q.eta)) {
                Q.breakdown = 1;
                Q.done = 1;
            }
            LockCoef& C = k.coef[s];
            C.na = -Q.alpha_next;
            C.nb = -Q.beta[0];
            C.sc = 1.0;  // the scale of the Av that the initial phase leaves
            C.act = !Q.done;
            if (!Q.done && large(k, s)) atomicAdd(k.active, 1);
        }
        __syncthreads();
    }
    grid.sync();

    int it = 0;
    while (it < a.max_it && *(volatile int*)k.active > 0) {
        const int k0 = acc3(it), k1 = acc3(it + 1), km1 = acc3(it - 1);
        const double* const vk = a.v[it & 1];
        double* const vk1 = a.v[(it + 1) & 1];  // holds v_k-1 until written
        double* const pk = a.p[it & 1];         // holds p_k-2 until written
        const double* const pkm1 = a.p[(it + 1) & 1];
        // ---- U sweep on v+ = Av - alpha v - beta v-; ||v+||^2 ----
        for (int t = wid; t < k.tiles; t += nw) {
            const int4 u = __ldg(k.tile + t);
            const LockCoef& C = k.coef[u.w];
            if (!C.act) continue;
            const ItemMeta m = meta_of_tile(a, u);
            double y[1] = {0.0}, d[1];
            if (lane < m.h) {
                const int g = m.fr + lane;
                double v = fma_rn(C.na, vk[g], a.Av[g]);
                v = fma_rn(C.nb, vk1[g], v);
                vk1[g] = v;
                y[0] = v;
            }
            u_item<TF, 1>(a, m, y, a.ev, d);
        }
        grid.sync();
        for (int c = wid; c < k.chunks; c += nw) {
            const int4 u = __ldg(k.chunk + c);
            const LockCoef& C = k.coef[u.z];
            if (!C.act) continue;
            if (lane < u.y) {
                const int g = __ldg(a.simple_rows + u.x + lane);
                double v = (double)(TF)(a.Av[g] * C.sc);
                v = fma_rn(C.na, vk[g], v);
                v = fma_rn(C.nb, vk1[g], v);
                vk1[g] = v;
                a.ev[g] = level0_u(a, g, v / (double)__ldg(a.dg + g), a.ev);
                double w[1];
                spmv_row<TF, 1>(a, g, a.ev, w);
                a.Av[g] = w[0];
            }
        }
        grid.sync();
        for (int s = blockIdx.x; s < k.num; s += gridDim.x) {
            LockCoef& C = k.coef[s];
            if (!C.act) continue;
            const SysView sv{0, 0, k.qb + 2 * s, k.qe + 2 * s, nullptr};
            const LvlBounds b0 = level_bounds(a, sv, 0), b1 = level_bounds(a, sv, 1);
            double r[1] = {0.0};
            auto add = [&](int g) { r[0] = fma_rn(vk1[g], vk1[g], r[0]); };
            over_items(a, b1, add);
            over_simple(a, b1.s0, b1.s1, tid, kT, add);
            over_simple(a, b0.s0, b0.s1, tid, kT, add);
            cta_reduce<1>(r, sh);
            if (tid == 0) {
                Scal& Q = k.scal[s];
                scal_after_u(Q, r[0], k0, k1, km1);
                C.sc = Q.inv_delta;
                C.nbrr = -Q.beta_rr;
                C.ne = -Q.epsilon;
                C.ir = Q.inv_rho;
                C.tau = Q.tau;
            }
            __syncthreads();
        }
        grid.sync();
        // ---- U' sweep with the fused SpMV; D^-1 Av, D^-1 v+; p, x ----
        for (int t = wid; t < k.tiles; t += nw) {
            const int4 u = __ldg(k.tile + t);
            const LockCoef& C = k.coef[u.w];
            if (!C.act) continue;
            const ItemMeta m = meta_of_tile(a, u);
            const double sc[1] = {C.sc};
            double av[1];
            ut_item<TF, 1, kRhsSpmv, true>(a, m, a.ev, sc, a.Av, av);
            DBlock<TF> D;
            D.load(a, m.fr, m.h, m.flags);
            double vs = 0.0;
            const int g = m.fr + lane;
            if (lane < m.h) {
                vs = vk1[g] * sc[0];
                vk1[g] = vs;
                double p = fma_rn(C.nbrr, pkm1[g], vk[g]);
                p = fma_rn(C.ne, pk[g], p);
                p = p * C.ir;
                pk[g] = p;
                a.xt[g] = fma_rn(C.tau, p, a.xt[g]);
            }
            const double da = D.apply(av[0], m.h), dv = D.apply(vs, m.h);
            if (lane < m.h) {
                k.da[g] = da;
                k.dv[g] = dv;
            }
        }
        for (int c = wid; c < k.chunks; c += nw) {
            const int4 u = __ldg(k.chunk + c);
            const LockCoef& C = k.coef[u.z];
            if (!C.act) continue;
            if (lane < u.y) {
                const int g = __ldg(a.simple_rows + u.x + lane);
                const double dd = (double)__ldg(a.dg + g);
                const double vs = vk1[g] * C.sc;
                vk1[g] = vs;
                double p = fma_rn(C.nbrr, pkm1[g], vk[g]);
                p = fma_rn(C.ne, pk[g], p);
                p = p * C.ir;
                pk[g] = p;
                a.xt[g] = fma_rn(C.tau, p, a.xt[g]);
                k.da[g] = (double)(TF)(a.Av[g] * C.sc) / dd;
                k.dv[g] = vs / dd;
            }
        }
        grid.sync();
        for (int s = blockIdx.x; s < k.num; s += gridDim.x) {
            LockCoef& C = k.coef[s];
            if (!C.act) continue;
            const SysView sv{0, 0, k.qb + 2 * s, k.qe + 2 * s, nullptr};
            const LvlBounds b0 = level_bounds(a, sv, 0), b1 = level_bounds(a, sv, 1);
            double r[4] = {0.0, 0.0, 0.0, 0.0};
            auto add = [&](int g) {
                const double vkr = vk[g], vs = vk1[g], da = k.da[g], xv = a.xt[g];
                r[0] = fma_rn(vkr, da, r[0]);
                r[1] = fma_rn(vs, da, r[1]);
                r[2] = fma_rn(vs, k.dv[g], r[2]);
                r[3] = fma_rn(xv, xv, r[3]);
            };
            over_items(a, b1, add);
            over_simple(a, b1.s0, b1.s1, tid, kT, add);
            // level 0: the warps without an item, or all
            const int items = b1.c1 - b1.c0;
            if (items >= kW) over_simple(a, b0.s0, b0.s1, tid, kT, add);
            else if ((tid >> 5) >= items) over_simple(a, b0.s0, b0.s1, tid - 32 * items, kT - 32 * items, add);
            cta_reduce<4>(r, sh);
            if (tid == 0) {
                Scal& Q = k.scal[s];
                scal_after_ut(Q, r[0], r[1], r[2], r[3], it, k1, a.tol, a.max_it);
                C.na = -Q.alpha_next;
                C.nb = -Q.beta[k1];
                if (Q.done) {
                    C.act = 0;
                    if (large(k, s)) atomicSub(k.active, 1);
                }
            }
            __syncthreads();
        }
        grid.sync();
        ++it;
    }

    if (blockIdx.x == 0 && tid == 0) k.active[1] = it;
    // ---- x = P U^-1 D^-1 x~ (k_sqmr_rest writes that of an unfinished system again) ----
    for (int t = wid; t < k.tiles; t += nw) {
        const ItemMeta m = meta_of_tile(a, __ldg(k.tile + t));
        const double y[1] = {(lane < m.h) ? a.xt[m.fr + lane] : 0.0};
        double d[1];
        u_item<TF, 1>(a, m, y, a.x, d);
    }
    for (int s = wid; s < k.num; s += nw)
        if (lane == 0) {
            const Scal& Q = k.scal[s];
            double* o = k.out + 8 * (size_t)s;
            o[0] = Q.gamma / Q.norm_pb;
            o[1] = Q.done ? Q.iters : it;
            o[2] = Q.breakdown;
            o[3] = (Q.snap0 || Q.snap1) ? 1 : 0;
            o[4] = Q.norm_pb;
            o[5] = Q.done ? Q.stop_it : it;
            o[6] = 0.0;
        }
    grid.sync();
    for (int c = wid; c < k.chunks; c += nw) {
        const int4 u = __ldg(k.chunk + c);
        if (lane < u.y) {
            const int g = __ldg(a.simple_rows + u.x + lane);
            a.x[g] = level0_u(a, g, a.xt[g] / (double)__ldg(a.dg + g), a.x);
        }
    }
}

}  // namespace

size_t lockstep_bytes(int n, int num)
{
    return 2 * (size_t)n * sizeof(double) + (size_t)num * (sizeof(Scal) + sizeof(LockCoef)) + 64;
}

template <class TF>
int lockstep_launch(const PArgs<TF>& a, const LockPlan& p, const BatchArgs& bt, void* work, int grid, int rest_grid,
                    cudaStream_t s)
{
    LockArgs k;
    k.num = bt.num;
    k.chunks = p.chunks;
    k.tiles = p.tiles;
    k.chunk = p.units.as<int4>();
    k.tile = k.chunk + p.chunks;
    k.row_off = bt.row_off;
    k.qb = bt.qb;
    k.qe = bt.qe;
    k.coef = static_cast<LockCoef*>(work);
    k.scal = reinterpret_cast<Scal*>(k.coef + bt.num);
    k.da = reinterpret_cast<double*>(k.scal + bt.num);
    k.dv = k.da + a.n;
    k.active = reinterpret_cast<int*>(k.dv + a.n);
    k.out = bt.out;
    CULIPX_CUDA(cudaMemsetAsync(k.active, 0, sizeof(int), s));
    CULIPX_CUDA(cudaMemsetAsync(bt.next, 0, sizeof(int), s));
    void* args[] = {const_cast<PArgs<TF>*>(&a), &k};
    CULIPX_CUDA(cudaLaunchCooperativeKernel((const void*)k_sqmr_lockstep<TF>, dim3(grid), dim3(kT), args, 0, s));
    const Scal* scal = k.scal;
    const LockCoef* coef = k.coef;
    const int* at = k.active + 1;
    void* rest[] = {const_cast<PArgs<TF>*>(&a), const_cast<BatchArgs*>(&bt), &scal, &coef, &at};
    CULIPX_CUDA(cudaLaunchKernel(rest_fn<TF>(), dim3(rest_grid), dim3(kT), rest, 0, s));
    return CULIPX_OK;
}

template <class TF>
const void* lockstep_kernel()
{
    return (const void*)k_sqmr_lockstep<TF>;
}

template int lockstep_launch<double>(const PArgs<double>&, const LockPlan&, const BatchArgs&, void*, int, int,
                                     cudaStream_t);
template int lockstep_launch<float>(const PArgs<float>&, const LockPlan&, const BatchArgs&, void*, int, int,
                                    cudaStream_t);
template const void* lockstep_kernel<double>();
template const void* lockstep_kernel<float>();

}  // namespace persistent

}  // namespace culipx
