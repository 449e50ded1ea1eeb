// Preconditioner applies for a factor computed on fine rows
// (factor_two_level.cu): level 0's pivot blocks are identities without swaps,
// level 1 has no off-diagonal blocks, and the entries of a level-1 block row's
// rows of U' stand in one run of slots.
//
//   LEFT   x = U'^-1 P' b in one launch.  A level-0 row is a copy of b, so the
//          level-1 rows gather from b itself and wait for nothing.
//   RIGHT  x = P U^-1 b: the level-1 tiles, then the level-0 rows.
// Both load what belongs to the factor while the kernel before them drains
// (launch.cuh).
//
// The arithmetic and its order are k_sweep_level's (solve.cu).  Bound: dependent
// loads and the tile's serial substitution (scale system, FP64: L1TEX at 36 to
// 55 % of its peak, L2 and DRAM below 26 %).  With a lane per row every load of
// a warp touches up to 32 lines; a tile's run of U' is therefore read across the
// lanes (coalesced, gathers all in flight) into shared memory, where each lane
// then sums its own row.  A division in the chain is taken only
// where the tile's diagonal is not 1.  Measured, LEFT / RIGHT with k_sweep_level
// against this: scale FP64 21.3 / 18.1 -> 13.6 / 12.6 us, N = 1.5 M FP32
// 51 / 47 -> 38.5 / 39 us.
#include "factor.h"
#include "kernels_common.cuh"
#include "launch.cuh"

#include <algorithm>

namespace culipx {

namespace {

constexpr int kApplyWarps = 4;
constexpr int kRun = 448;   // entries of a tile's run that are staged (28 warps of FP64 per SM)
constexpr int kTriRegs = (32 * 33 / 2 + 31) / 32;

template <class T>
struct ApplyArgs {
    int n0, nr1;
    const int* l0_rows;
    const two::Tile* tiles;
    const int* rowflags;
    const int* perm;
    const unsigned* ndmask;
    const T* pk;
    const int2* rng;
    const int* col;
    const T* val;
    const T* b;
    T* x;
};

// the tile's packed triangle: loads in flight before its staging area is free
template <class T>
__device__ __forceinline__ void tri_load(const T* P, int count, T (&u)[kTriRegs])
{
    const int lane = lane_id();
#pragma unroll
    for (int j = 0; j < kTriRegs; ++j) u[j] = (lane + 32 * j < count) ? __ldg(P + lane + 32 * j) : T(0);
}

template <class T>
__device__ __forceinline__ void tri_store(T* tile, int count, const T (&u)[kTriRegs])
{
    const int lane = lane_id();
#pragma unroll
    for (int j = 0; j < kTriRegs; ++j)
        if (lane + 32 * j < count) tile[lane + 32 * j] = u[j];
}

// Substitution with the staged triangle, U' forward (row r of the triangle at
// r h - r (r - 1) / 2: columns r .. h - 1) or U backward (column c at
// c (c + 1) / 2: rows 0 .. c).  A diagonal entry of exactly 1 needs no
// division (t / 1 == t): only those that nd marks are divided, which leaves
// shuffle + fma on the chain, its factors loaded eight steps ahead.
template <class T, bool UPPER, bool DIV>
__device__ __forceinline__ T tri_solve_t(T acc, const T* tile, int h, unsigned nd)
{
    constexpr int B = 8;
    const int lane = lane_id();
    for (int k0 = 0; k0 < h; k0 += B) {
        T u[B];
#pragma unroll
        for (int j = 0; j < B; ++j) {
            const int k = UPPER ? h - 1 - k0 - j : k0 + j;
            const bool on = UPPER ? (k >= 0 && lane <= k) : (k < h && lane >= k && lane < h);
            const int at = UPPER ? k * (k + 1) / 2 + lane : k * h - k * (k - 1) / 2 - k + lane;
            u[j] = on ? tile[at] : T(0);
        }
#pragma unroll
        for (int j = 0; j < B; ++j) {
            const int k = UPPER ? h - 1 - k0 - j : k0 + j;
            if (UPPER ? k < 0 : k >= h) break;
            if (DIV && ((nd >> k) & 1u) && lane == k) acc = acc / u[j];
            const T xk = shfl(acc, k);
            if (UPPER ? lane < k : (lane > k && lane < h)) acc = fma_rn(-u[j], xk, acc);
        }
    }
    return acc;
}

template <class T, bool UPPER>
__device__ __forceinline__ T tri_solve(T acc, const T* tile, int h, unsigned nd)
{
    return nd ? tri_solve_t<T, UPPER, true>(acc, tile, h, nd) : tri_solve_t<T, UPPER, false>(acc, tile, h, 0u);
}

template <class T>
__global__ void __launch_bounds__(32 * kApplyWarps) k_two_left(ApplyArgs<T> a, int tile_ctas)
{
    __shared__ T run[kApplyWarps][2 * kRun];
    if ((int)blockIdx.x >= tile_ctas) {
        after_previous();
        // level 0: x = b (in place: nothing to do)
        const int stride = ((int)gridDim.x - tile_ctas) * 32 * kApplyWarps;
        for (int i = ((int)blockIdx.x - tile_ctas) * 32 * kApplyWarps + threadIdx.x; i < a.n0; i += stride) {
            const int g = __ldg(a.l0_rows + i) & two::kRowMask;
            a.x[g] = a.b[g];
        }
        return;
    }
    const int warp = threadIdx.x >> 5, lane = lane_id();
    const int t = blockIdx.x * kApplyWarps + warp;
    if (t >= a.nr1) {
        after_previous();
        return;
    }
    T* const sv = run[warp];
    T* const sx = sv + kRun;
    const int4* td = reinterpret_cast<const int4*>(a.tiles + t);
    const int4 d0 = __ldg(td), d1 = __ldg(td + 1);
    const int I = d0.x, fr = d0.y, h = d0.z, s0 = d1.x, s1 = d1.x + d0.w;
    const T* P = a.pk + (((long long)d1.w << 32) | (unsigned)d1.z);
    const int flags = __ldg(a.rowflags + I);
    const unsigned nd = __ldg(a.ndmask + I);
    const int tri = h * (h + 1) / 2;
    int2 kr = make_int2(0, 0);
    int from = 0;
    if (lane < h) {
        kr = __ldg(a.rng + fr + lane);
        from = __ldg(a.perm + fr + lane);
    }
    T u[kTriRegs];
    tri_load(P, tri, u);
    after_previous();  // b; what stands above is the factor's
    T acc = (lane < h) ? a.b[from] : T(0);
    if (s1 - s0 <= kRun) {
        constexpr int B = 7;
        for (int e0 = lane; e0 < s1 - s0; e0 += 32 * B) {
            int c[B];
            T v[B], xv[B];
#pragma unroll
            for (int j = 0; j < B; ++j) {
                const int e = e0 + 32 * j;
                c[j] = (e < s1 - s0) ? __ldg(a.col + s0 + e) : -1;
                v[j] = (e < s1 - s0) ? __ldg(a.val + s0 + e) : T(0);
            }
#pragma unroll
            for (int j = 0; j < B; ++j) xv[j] = (c[j] >= 0) ? a.b[c[j]] : T(0);
#pragma unroll
            for (int j = 0; j < B; ++j)
                if (c[j] >= 0) {
                    sv[e0 + 32 * j] = v[j];
                    sx[e0 + 32 * j] = xv[j];
                }
        }
        __syncwarp();
        for (int e = kr.x - s0; e < kr.y - s0; ++e) acc = fma_rn(-sv[e], sx[e], acc);
        __syncwarp();
    } else {
        constexpr int B = 8;
        for (int k = kr.x; k < kr.y; k += B) {
            int c[B];
            T v[B], xv[B];
#pragma unroll
            for (int j = 0; j < B; ++j) {
                c[j] = (k + j < kr.y) ? __ldg(a.col + k + j) : -1;
                v[j] = (k + j < kr.y) ? __ldg(a.val + k + j) : T(0);
            }
#pragma unroll
            for (int j = 0; j < B; ++j) xv[j] = (c[j] >= 0) ? a.b[c[j]] : T(0);
#pragma unroll
            for (int j = 0; j < B; ++j)
                if (c[j] >= 0) acc = fma_rn(-v[j], xv[j], acc);
        }
    }
    if (!(flags & kRowIdentity)) {
        T* const tile = run[warp];
        tri_store(tile, tri, u);
        __syncwarp();
        acc = tri_solve<T, false>(acc, tile, h, nd);
    }
    __syncwarp();  // in place: every lane has read its own place before any lane writes
    if (lane < h) a.x[fr + lane] = acc;
}

template <class T>
__global__ void __launch_bounds__(32 * kApplyWarps) k_two_right_tiles(ApplyArgs<T> a)
{
    __shared__ T tiles[kApplyWarps][32 * 33 / 2];
    const int warp = threadIdx.x >> 5, lane = lane_id();
    const int t = blockIdx.x * kApplyWarps + warp;
    if (t >= a.nr1) {
        after_previous();
        return;
    }
    T* const tile = tiles[warp];
    const int4* td = reinterpret_cast<const int4*>(a.tiles + t);
    const int4 d0 = __ldg(td), d1 = __ldg(td + 1);
    const int I = d0.x, fr = d0.y, h = d0.z;
    const T* P = a.pk + (((long long)d1.w << 32) | (unsigned)d1.z);
    const int flags = __ldg(a.rowflags + I);
    const unsigned nd = __ldg(a.ndmask + I);
    T u[kTriRegs];
    tri_load(P, h * (h + 1) / 2, u);
    const int to = (lane < h) ? __ldg(a.perm + fr + lane) : 0;
    after_previous();
    T acc = (lane < h) ? a.b[fr + lane] : T(0);
    if (!(flags & kRowIdentity)) {
        tri_store(tile, h * (h + 1) / 2, u);
        __syncwarp();
        acc = tri_solve<T, true>(acc, tile, h, nd);
    }
    __syncwarp();
    if (lane < h) a.x[to] = acc;
}

template <class T, int B>
__global__ void __launch_bounds__(256) k_two_right_rows(ApplyArgs<T> a)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = i < a.n0;
    int g = 0;
    int2 kr = make_int2(0, 0);
    int c[B];
    T v[B];
    if (in) {
        g = __ldg(a.l0_rows + i) & two::kRowMask;
        kr = __ldg(a.rng + g);
    }
#pragma unroll
    for (int j = 0; j < B; ++j) {
        c[j] = (kr.x + j < kr.y) ? __ldg(a.col + kr.x + j) : -1;
        v[j] = (kr.x + j < kr.y) ? __ldg(a.val + kr.x + j) : T(0);
    }
    after_previous();
    if (!in) return;
    T acc = a.b[g];
    for (int k = kr.x;;) {
        T xv[B];
#pragma unroll
        for (int j = 0; j < B; ++j) xv[j] = (c[j] >= 0) ? a.x[c[j]] : T(0);
#pragma unroll
        for (int j = 0; j < B; ++j)
            if (c[j] >= 0) acc = fma_rn(-v[j], xv[j], acc);
        k += B;
        if (k >= kr.y) break;
#pragma unroll
        for (int j = 0; j < B; ++j) {
            c[j] = (k + j < kr.y) ? __ldg(a.col + k + j) : -1;
            v[j] = (k + j < kr.y) ? __ldg(a.val + k + j) : T(0);
        }
    }
    a.x[g] = acc;
}

template <class T>
int apply(Factor* f, bool left, const void* d_b, void* d_x, cudaStream_t s)
{
    const Pattern& p = *f->pat;
    ApplyArgs<T> a;
    a.n0 = p.l0_count;
    a.nr1 = p.lvl_off[2] - p.lvl_off[1];
    a.l0_rows = p.two_l0_rows;
    a.tiles = p.two_tiles;
    a.rowflags = f->rowflags.as<int>();
    a.perm = f->perm.as<int>();
    a.ndmask = f->ndmask.as<unsigned>();
    a.pk = left ? f->pk_row.as<T>() : f->pk_col.as<T>();
    a.rng = left ? f->ut_rng.as<int2>() : f->u_rng.as<int2>();
    a.col = left ? f->ut_col.as<int>() : f->u_colp.as<int>();
    a.val = left ? f->ut_val.as<T>() : f->u_val.as<T>();
    a.b = static_cast<const T*>(d_b);
    a.x = static_cast<T*>(d_x);
    const int tile_ctas = (a.nr1 + kApplyWarps - 1) / kApplyWarps;
    if (left) {
        const int copies = (d_b == d_x) ? 0 : std::min((a.n0 + 511) / 512, 148 * 8);
        return launch_overlapped(k_two_left<T>, dim3(tile_ctas + copies), dim3(32 * kApplyWarps), s, true, a, tile_ctas);
    }
    CULIPX_TRY(launch_overlapped(k_two_right_tiles<T>, dim3(tile_ctas), dim3(32 * kApplyWarps), s, true, a));
    // a thread per row: fewer rows than fill the device are spread over it, as
    // a long row is its thread's serial chain (3000 rows of 200 entries, FP64:
    // 45 us for RIGHT with CTAs of 256, 27 with the general sweeps)
    const int threads = std::min(256, std::max(32, (a.n0 / (4 * 148) + 31) / 32 * 32));
    const dim3 grid((a.n0 + threads - 1) / threads), block(threads);
    if (p.two_entries > 12LL * a.n0) return launch_overlapped(k_two_right_rows<T, 16>, grid, block, s, true, a);
    return launch_overlapped(k_two_right_rows<T, 8>, grid, block, s, true, a);
}

}  // namespace

int two_level_apply(Factor* f, bool left, const void* d_b, void* d_x, cudaStream_t s)
{
    if (f->precision == CULIPX_F64) return apply<double>(f, left, d_b, d_x, s);
    return apply<float>(f, left, d_b, d_x, s);
}

}  // namespace culipx
