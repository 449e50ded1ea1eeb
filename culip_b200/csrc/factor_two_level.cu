// Numeric factorization on fine rows, for a two-level pattern whose level-0
// block rows have diagonal pivot blocks (Pattern::two_level: a KKT system in
// its natural order at fill level 0).
//
// There the factor has closed form up to the level-1 pivot tiles:
//   level 0   D_g = K_gg (perturbed as d_ldlt_1x1_step does), U = I on the
//             pivot blocks, U_gc = K_gc / D_g on the others;
//   level 1   each block row's tile K_JJ - sum_g U_gJ' D_g U_gJ, factored with
//             Bunch-Kaufman / Rook pivoting; no off-diagonal blocks.
// The general path (factor.cu, solve.cu) stores U by blocks, updates a tile
// block by block and then re-lays U out as fine rows.  Here K's rows are read
// as they are and the fine rows are written at once, in three launches:
//   k_two_rows    thread per level-0 row: D and the row of U
//   k_two_tiles   warp per level-1 block row: the Schur update, the tile's
//                 factorization, its packed triangles and its rows of U'
//   k_two_order   the rows of U into the order of the permuted columns; the
//                 level-1 block rows split into simple ones and work items
// Every value and every order of summation is the general path's: an update
// block's contributions to a tile entry are summed in row order and then
// subtracted, blocks in row order; entries of sparse blocks with |u| <= NZ_EPS
// are dropped.  Zeros that the general path multiplies with a NaN or an
// infinity are not in K's rows: spread_nonfinite puts their NaN in.
//
// Bound: the tiles' serial pivot steps (dependent loads and fixed latency, an
// issue slot in three used), not bandwidth; the order kernel's L1 requests
// (L1TEX at 76 %).  Measured on the scale system
// (n = 200 000, m = 100 000, 3125 tiles of 32, FP64): 120 us (rows 13, tiles
// 85, order 22) against 960 us for the general path's 31 launches, 590 of them
// in the tiles' block-by-block updates; N = 3000 with tiles of 4: 18 us against
// 130; 256 systems of 2.0 M rows in FP32: 0.46 ms against 3.4.
#include "factor.h"
#include "kernels_common.cuh"
#include "launch.cuh"
#include "pivot_tile.cuh"

#include <algorithm>

namespace culipx {

namespace {

constexpr int kTileWarps = 4;   // level-1 block rows per CTA
constexpr int kRowRegs = 8;     // entries of a row of U handled in registers

template <class T>
struct Pair {};
template <>
struct Pair<double> {
    using type = double2;
};
template <>
struct Pair<float> {
    using type = float2;
};

template <class T>
struct TwoArgs {
    int n0;               // level-0 fine rows
    int q1, nr1;          // first position of level 1 in lvl_rows, its block rows
    int method;
    double piv64;
    const T* kval;
    // the pattern's two-level form (pattern.h)
    const int* kp;
    const int* l0_rows;
    const int* ucol;
    const int2* low;
    const uint2* pairs;
    const int2* tail;
    const two::Tile* tiles;
    const int* tail_off;
    const int* slot;
    const int* l0_scan;
    const int* lvl_rows;
    const int* bs;
    typename Pair<T>::type* up;  // per entry of U: u and D u, both 0 if dropped
    T* u_sub;
    T* tri;
    T* dg;
    int* is_piv;
    int* perm;
    int* rowflags;
    int* u_col;
    int* u_colp;
    T* u_val;
    int2* u_rng;
    int* ut_col;
    T* ut_val;
    int2* ut_rng;
    int* iperm;           // per level-1 fine row its place after the tile's swaps
    const long long* pk_off;
    T* pk_col;
    T* pk_row;
    unsigned* ndmask;
    int* scan_s;
    int* scan_c;
    int* simple_rows;
    int* cplx;
    CItem* citem;
    unsigned char* kind;  // per level-1 block row: its rows if simple, else 0
    int* nonfinite;       // set by the rows, cleared by the last kernel
    int blocks;
};

// a level-0 pivot from K's diagonal entry (0 if K stores none), perturbed as
// d_ldlt_1x1_step (:556-560)
template <class T>
__device__ __forceinline__ T level0_pivot(const TwoArgs<T>& a, int tagged, int k0)
{
    T d = T(0);
    if (!(tagged & two::kNoDiag)) d = a.kval[k0];
    if (fabs(d) < 1e-8) d = T(1e-6);
    return d;
}

// Level-0 rows: D and the entries of U at their places of the pattern, each
// with D u for the tiles' updates.  The left solve is k_offdiag_fast's Givens
// form for a 1x1 pivot, its row constants taken once per row.
template <class T>
__global__ void __launch_bounds__(256) k_two_rows(TwoArgs<T> a)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    int tagged = 0, g = 0, k0 = 0, k1 = 0, o0 = 0;
    if (i < a.n0) {
        tagged = __ldg(a.l0_rows + i);
        g = tagged & two::kRowMask;
        k0 = __ldg(a.kp + g);
        k1 = __ldg(a.kp + g + 1);
        o0 = __ldg(a.slot + g);
    }
    after_previous();  // K's values; what stands above is the pattern's
    if (i >= a.n0) return;
    const T d11 = level0_pivot(a, tagged, k0);
    if (!isfinite(d11)) *a.nonfinite = 1;
    const T d22 = (tagged & two::kNextInBlock) ? level0_pivot(a, __ldg(a.l0_rows + i + 1), k1) : T(0);
    const T d12 = T(0);
    const T gr = sqrt(fma_rn(d11, d11, d12 * d12));
    const T gc = d11 / gr, gs = d12 / gr;
    const T td11 = fma_rn(gc, d11, gs * d12);
    const T td12 = fma_rn(gc, d12, gs * d22);
    const int kb = (tagged & two::kNoDiag) ? k0 : k0 + 1;
    for (int k = kb; k < k1; k += kRowRegs) {
        T v[kRowRegs];
#pragma unroll
        for (int j = 0; j < kRowRegs; ++j) v[j] = (k + j < k1) ? a.kval[k + j] : T(0);
#pragma unroll
        for (int j = 0; j < kRowRegs; ++j) {
            if (k + j >= k1) break;
            const int o = o0 + (k + j - kb);
            T u = fma_rn(gc, v[j], gs * T(0));
            u = fma_rn(-td12, T(0), u) / td11;
            // sparse blocks drop |u| <= NZ_EPS, dense ones keep every non-zero
            if (!(fabs(u) > T(kNzEps)) && !((tagged & two::kRowDense) && __ldg(a.ucol + o) < 0)) u = T(0);
            typename Pair<T>::type e;
            e.x = u;
            e.y = d11 * u;
            if (u == T(0)) e.y = T(0);
            a.up[o] = e;
        }
    }
    a.ut_rng[g] = make_int2(0, 0);
    a.dg[g] = d11;
    a.tri[3 * (size_t)g] = T(0);
    a.tri[3 * (size_t)g + 1] = d11;
    a.tri[3 * (size_t)g + 2] = T(0);
    a.perm[g] = g;
    a.is_piv[g] = 1;
    a.simple_rows[i] = g;
}

// What the general path's update of a tile by a whole block gives beyond the
// entries of K's rows where values are not finite (0 x inf and 0 x NaN are
// NaN): with lv = D u its factor for row a of the tile,
//   * a pivot of the block that is not finite makes lv NaN in every row a that
//     has an entry in the block, and a NaN or, next to other rows of the block,
//     an infinite entry does so in its own row: the tile's row is NaN;
//   * an infinite lv otherwise meets the zeros of U's row: the places of the
//     tile's row that are still finite are NaN.
// A lane looks through its row's entries; reached only with such values.
template <class T>
__device__ void spread_nonfinite(const TwoArgs<T>& a, T* tile, int h, int k0, int k1)
{
    const int b = lane_id();
    bool all = false, rest = false;
#pragma unroll 1
    for (int k = k0; k < k1; ++k) {
        const int2 w = __ldg(a.low + k);
        const auto q = a.up[w.y];
        if (q.x == T(0)) continue;  // dropped
        const int g = w.x & two::kColMask;
        int lo = 0, hi = a.blocks;  // the block row that holds g
        while (hi - lo > 1) {
            const int mid = (lo + hi) / 2;
            if (__ldg(a.bs + mid) <= g) lo = mid;
            else hi = mid;
        }
        const int g0 = __ldg(a.bs + lo), g1 = __ldg(a.bs + lo + 1);
        bool pivots = true;
#pragma unroll 1
        for (int r = g0; r < g1; ++r) pivots &= (bool)isfinite(a.dg[r]);
        all |= !pivots || q.x != q.x || q.y != q.y || (g1 - g0 > 1 && !isfinite(q.x));
        rest |= !isfinite(q.x) || !isfinite(q.y);
    }
    const unsigned alls = __ballot_sync(0xffffffffu, all), rests = __ballot_sync(0xffffffffu, rest);
    const T nan = T(0) / T(0);
    for (int r = 0; r < h; ++r) {
        T* const at = tile + r * kTileStride + b;
        if (b < h && (((alls >> r) & 1u) || (((rests >> r) & 1u) && isfinite(*at)))) *at = nan;
    }
}

// One level-1 block row per warp, the upper triangle T_ab at tile[a][b].  Lane b
// walks K's row fr + b for the diagonal's update and writes its row of U'; the
// entries off the diagonal take theirs from the pattern's pair list, a lane per
// entry, which keeps the lanes on the same path (walking a row's partners
// instead: 5000 of 13 200 instructions a tile).
template <class T>
__global__ void __launch_bounds__(32 * kTileWarps, 6) k_two_tiles(TwoArgs<T> a)
{
    __shared__ __align__(16) T tiles[kTileWarps][kTileElems];
    __shared__ T row_s[kTileWarps][kRowBuf];
    __shared__ int perm_s[kTileWarps][32];
    __shared__ int piv_s[kTileWarps][32];
    const int warp = threadIdx.x >> 5;
    const int t = blockIdx.x * kTileWarps + warp;
    if (t >= a.nr1) {
        after_previous();
        return;
    }
    const int b = lane_id();
    T* tile = tiles[warp];
    const int4* td = reinterpret_cast<const int4*>(a.tiles + t);
    const int4 d0 = __ldg(td), d1 = __ldg(td + 1);
    const int I = d0.x, fr = d0.y, h = d0.z;
    const int me = fr + b;
    int k0 = 0, k1 = 0;
    if (b < h) {
        k0 = __ldg(a.slot + me);
        k1 = (b + 1 < h) ? __ldg(a.slot + me + 1) : d1.x + d0.w;
    }
    after_previous();  // the rows of U; what stands above is the pattern's

    // The tile's entries of U' across the lanes: U' out, u and D u staged where
    // the tile will be, the marks of entries in the block of the one before as
    // bits; then each lane sums its row for the diagonal.
    constexpr int CAP = 448, B = 7;
    typename Pair<T>::type* const stage = reinterpret_cast<typename Pair<T>::type*>(tile);
    unsigned* const marks = reinterpret_cast<unsigned*>(perm_s[warp]);
    const int e0 = d1.x, e1 = d1.x + d0.w;
    int ut = k1;
    bool dropped = false;
    // K's values were complete before the rows' kernel let this one start
    const int q0 = __ldg(a.tail_off + t), q1 = __ldg(a.tail_off + t + 1);
    row_s[warp][b] = T(0);
    __syncwarp();
    for (int k = q0 + b; k < q1; k += 32) {  // K's diagonal, from which the update's sums are subtracted in turn
        const int2 e = __ldg(a.tail + k);
        if ((e.y >> 5) == (e.y & 31)) row_s[warp][e.y & 31] = __ldg(a.kval + e.x);
    }
    __syncwarp();
    T diag = row_s[warp][b], sum = T(0);
    for (int base = e0; base < e1; base += CAP) {
        const int n = min(CAP, e1 - base);
        for (int i0 = b; i0 < CAP && i0 - b < n; i0 += 32 * B) {
            int2 w[B];
            typename Pair<T>::type q[B];
#pragma unroll
            for (int j = 0; j < B; ++j) w[j] = (i0 + 32 * j < n) ? __ldg(a.low + base + i0 + 32 * j) : make_int2(0, -1);
#pragma unroll
            for (int j = 0; j < B; ++j)
                if (w[j].y >= 0) q[j] = a.up[w[j].y];
#pragma unroll
            for (int j = 0; j < B; ++j) {
                const unsigned m = __ballot_sync(0xffffffffu, w[j].x < 0);
                if (b == 0 && i0 + 32 * j < n) marks[(i0 + 32 * j) / 32] = m;
                if (w[j].y < 0) continue;
                stage[i0 + 32 * j] = q[j];
                a.ut_col[base + i0 + 32 * j] = w[j].x & two::kColMask;
                a.ut_val[base + i0 + 32 * j] = q[j].x;
                dropped |= q[j].x == T(0);
            }
        }
        __syncwarp();
        for (int e = max(k0, base); e < min(k1, base + n); ++e) {
            const auto q = stage[e - base];
            if (!((marks[(e - base) >> 5] >> ((e - base) & 31)) & 1u)) {  // another update block begins
                diag -= sum;
                sum = T(0);
            }
            if (q.x != T(0)) sum = fma_rn(q.x, q.y, sum);
        }
        __syncwarp();
    }
    if (__any_sync(0xffffffffu, dropped)) {  // the rows without the dropped entries
        ut = k0;
        for (int k = k0; k < k1; ++k) {
            const int2 w = __ldg(a.low + k);
            const T u = a.up[w.y].x;
            if (u == T(0)) continue;
            a.ut_col[ut] = w.x & two::kColMask;
            a.ut_val[ut] = u;
            ++ut;
        }
    }
    for (int e = b; e < kTileElems; e += 32) tile[e] = T(0);
    __syncwarp();
    for (int k = q0 + b; k < q1; k += 32) {
        const int2 e = __ldg(a.tail + k);
        tile[(e.y >> 5) * kTileStride + (e.y & 31)] = __ldg(a.kval + e.x);
    }
    __syncwarp();
    if (b < h) tile[b * kTileStride + b] = diag - sum;
    const bool spoilt = __any_sync(0xffffffffu, *a.nonfinite || (b < h && !isfinite(diag - sum)));
    const int p0 = d1.y, p1 = __ldg(&a.tiles[t + 1].pair);
    for (int i = p0 + b; i < p1; i += 32) {
        uint2 m = __ldg(a.pairs + i);
        if (m.x & two::kSameTarget) continue;  // its entry's first pair is another lane's
        T* const at = tile + (m.x >> two::kPlaceShift) * kTileStride + (m.y >> two::kPlaceShift);
        T v = *at;
        T s = T(0);
        auto add = [&]() {
            const T u = a.up[m.x & two::kSlotMask].x, du = a.up[m.y & two::kSlotMask].y;
            if (u != T(0) && du != T(0)) s = fma_rn(u, du, s);  // neither dropped
        };
        add();
        for (int j = i + 1; j < p1; ++j) {
            m = __ldg(a.pairs + j);
            if (!(m.x & two::kSameTarget)) break;
            if (!(m.y & two::kSameSum)) {
                v -= s;
                s = T(0);
            }
            add();
        }
        *at = v - s;
    }
    if (spoilt) {
        __syncwarp();
        spread_nonfinite(a, tile, h, k0, k1);
    }
    // the sweeps read a tile's run of slots whole
    for (int q = ut; q < k1; ++q) {
        a.ut_col[q] = 0;
        a.ut_val[q] = T(0);
    }
    __syncwarp();

    int* perm = perm_s[warp];
    int* piv = piv_s[warp];
    T* D = a.tri + 3 * (size_t)fr;
    perm[b] = b;
    piv[b] = 1;
    __syncwarp();
    bool diagonal = true;
    for (int r = 0; r < h; ++r) diagonal &= b <= r || b >= h || tile[r * kTileStride + b] == T(0);
    if (__all_sync(0xffffffffu, diagonal)) {
        // 1x1 pivots without swaps (k_pivot_blocks' short cut)
        if (b < h) {
            T d = tile[b * kTileStride + b];
            if (fabs(d) < 1e-8) d = T(1e-6);
            tile[b * kTileStride + b] = T(1);
            D[3 * b] = T(0);
            D[3 * b + 1] = d;
            D[3 * b + 2] = T(0);
        }
        __syncwarp();
    } else {
        factorize_tile_window(tile, row_s[warp], h, piv, D, perm, a.method, a.piv64);
    }
    __syncwarp();

    bool ident = true;
    if (b < h)
        for (int r = 0; r <= b; ++r) ident &= tile[r * kTileStride + b] == (r == b ? T(1) : T(0));
    ident = __all_sync(0xffffffffu, ident);
    const bool two = __any_sync(0xffffffffu, b < h && (D[3 * b + 2] != T(0) || D[3 * b] != T(0)));
    const bool pid = __all_sync(0xffffffffu, b >= h || perm[b] == b);
    const unsigned nd = __ballot_sync(0xffffffffu, b < h && tile[b * kTileStride + b] != T(1));
    if (b == 0) {
        a.rowflags[I] = (ident ? kRowIdentity : 0) | (two ? kRowHas2x2 : 0) | (pid ? kRowPermIdentity : 0);
        a.ndmask[I] = nd;
        a.kind[t] = (ident && pid && !two) ? (unsigned char)h : 0;
    }
    const int from = (b < h) ? perm[b] : b;  // the column now at place b
    const int s0 = shfl(k0, from), s1 = shfl(ut, from);
    if (b < h) {
        a.dg[me] = D[3 * b + 1];
        a.is_piv[me] = piv[b];
        a.perm[me] = fr + from;
        a.iperm[fr + from] = me;
        a.ut_rng[me] = make_int2(s0, s1);
        a.u_rng[me] = make_int2(0, 0);
    }
    // a 2x2 pivot's rounding residue left of its second row's diagonal, for the export
    if (two && b < h) a.u_sub[me] = b > 0 ? tile[b * kTileStride + b - 1] : T(0);
    if (!ident) {
        const long long pko = ((long long)d1.w << 32) | (unsigned)d1.z;
        T* pc = a.pk_col + pko;
        T* pr = a.pk_row + pko;
        // across the lanes: columns of the triangle into pc, rows into pr
        for (int k = 0; k < h; ++k) {
            if (b <= k) pc[k * (k + 1) / 2 + b] = tile[b * kTileStride + k];
            if (b >= k && b < h) pr[k * h - k * (k - 1) / 2 + b - k] = tile[k * kTileStride + b];
        }
    }
}

// The first split CTAs: the lists of solve.cu's k_split_count / k_split_fill, kOrderT
// level-1 block rows each, their prefix summed from one byte per earlier tile
// (the rows of a simple one, 0 for a work item; level 0 is all simple).  The
// others: a thread per level-0 row sorts its entries by their columns' places
// after the tiles' swaps (swaps stay inside a block, so rows keep their block
// order) and maps them back through the permutation.
constexpr int kOrderT = 256;

template <class T>
__device__ void split_rows(const TwoArgs<T>& a, int q0)
{
    __shared__ int sum_s[kOrderT / 32], sum_c[kOrderT / 32];
    const int tid = threadIdx.x, lane = lane_id(), w = tid >> 5;
    int s = 0, c = 0;  // simple rows and work items of this thread's share of the tiles before q0
    const uint4* kinds = reinterpret_cast<const uint4*>(a.kind);
    for (int i = tid; i < q0 / 16; i += kOrderT) {
        const uint4 v = kinds[i];
        const unsigned words[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            s += (int)__dp4a(words[j], 0x01010101u, 0u);
            c += __popc(__vcmpeq4(words[j], 0u)) / 8;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        c += __shfl_xor_sync(0xffffffffu, c, o);
    }
    if (lane == 0) {
        sum_s[w] = s;
        sum_c[w] = c;
    }
    __syncthreads();
    s = a.n0;
    c = 0;
    for (int k = 0; k < kOrderT / 32; ++k) {
        s += sum_s[k];
        c += sum_c[k];
    }
    __syncthreads();
    const int t = q0 + tid, q = a.q1 + t;
    const bool in = t < a.nr1;
    const int rows = in ? a.kind[t] : 0;
    const int item = in && rows == 0;
    int is = rows, ic = item;
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, is, o), y = __shfl_up_sync(0xffffffffu, ic, o);
        if (lane >= o) {
            is += x;
            ic += y;
        }
    }
    if (lane == 31) {
        sum_s[w] = is;
        sum_c[w] = ic;
    }
    __syncthreads();
    s += is - rows;
    c += ic - item;
    for (int k = 0; k < w; ++k) {
        s += sum_s[k];
        c += sum_c[k];
    }
    if (!in) return;
    a.scan_s[q] = s;
    a.scan_c[q] = c;
    const int I = __ldg(a.lvl_rows + q);
    const int fr = __ldg(a.bs + I);
    for (int r = 0; r < rows; ++r) a.simple_rows[s + r] = fr + r;
    if (item) {
        CItem it;
        it.I = I;
        it.fr = fr;
        it.h = __ldg(a.bs + I + 1) - fr;
        it.flags = a.rowflags[I];
        it.pk_off = __ldg(a.pk_off + I);
        it.nd = a.ndmask[I];
        it.pad = 0;
        a.cplx[c] = I;
        a.citem[c] = it;
    }
    if (t == a.nr1 - 1) {
        a.scan_s[q + 1] = s + rows;
        a.scan_c[q + 1] = c + item;
    }
}

template <class T>
__global__ void __launch_bounds__(kOrderT) k_two_order(TwoArgs<T> a, int splits)
{
    after_previous();
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.nonfinite = 0;  // the tiles have read it
    if ((int)blockIdx.x < splits) {
        split_rows(a, blockIdx.x * kOrderT);
        return;
    }
    const int i = ((int)blockIdx.x - splits) * kOrderT + threadIdx.x;
    if (i < a.q1) {  // the level-0 block rows' entries of the lists
        a.scan_s[i] = __ldg(a.l0_scan + i);
        a.scan_c[i] = 0;
        a.rowflags[__ldg(a.lvl_rows + i)] = kRowIdentity | kRowPermIdentity | kRowNoUpdates;
    }
    if (i >= a.n0) return;
    const int tagged = __ldg(a.l0_rows + i);
    const int g = tagged & two::kRowMask;
    const int o0 = __ldg(a.slot + g);
    const int len = __ldg(a.kp + g + 1) - __ldg(a.kp + g) - ((tagged & two::kNoDiag) ? 0 : 1);
    if (len <= kRowRegs) {
        int c[kRowRegs], nc[kRowRegs];
        T v[kRowRegs];
#pragma unroll
        for (int j = 0; j < kRowRegs; ++j) {
            c[j] = (j < len) ? __ldg(a.ucol + o0 + j) & two::kColMask : -1;
            v[j] = (j < len) ? a.up[o0 + j].x : T(0);
        }
        int kept = 0;
#pragma unroll
        for (int j = 0; j < kRowRegs; ++j) {
            const bool keep = v[j] != T(0);
            nc[j] = keep ? a.iperm[c[j]] : two::kColMask;
            kept += keep;
        }
#pragma unroll
        for (int j = 0; j < kRowRegs; ++j) {
            int rank = 0;
#pragma unroll
            for (int k = 0; k < kRowRegs; ++k)
                if (k != j) rank += nc[k] < nc[j];
            if (v[j] != T(0)) {
                a.u_colp[o0 + rank] = c[j];
                a.u_col[o0 + rank] = nc[j];
                a.u_val[o0 + rank] = v[j];
            }
        }
        a.u_rng[g] = make_int2(o0, o0 + kept);
        return;
    }
    int o = o0;
    for (int j = 0; j < len; ++j) {  // insertion: an entry moves within its block's few
        const T v = a.up[o0 + j].x;
        if (v == T(0)) continue;
        const int c = __ldg(a.ucol + o0 + j) & two::kColMask, nc = a.iperm[c];
        int k = o++;
        for (; k > o0 && a.u_col[k - 1] > nc; --k) {
            a.u_col[k] = a.u_col[k - 1];
            a.u_colp[k] = a.u_colp[k - 1];
            a.u_val[k] = a.u_val[k - 1];
        }
        a.u_col[k] = nc;
        a.u_colp[k] = c;
        a.u_val[k] = v;
    }
    a.u_rng[g] = make_int2(o0, o);
}

template <class T>
int run(Factor* f, const void* d_vals, cudaStream_t s, int* launches)
{
    const Pattern& p = *f->pat;
    TwoArgs<T> a;
    a.n0 = p.l0_count;
    a.q1 = p.lvl_off[1];
    a.nr1 = p.lvl_off[2] - p.lvl_off[1];
    a.method = f->pivot;
    a.piv64 = f->pivot_fp64;
    a.kval = static_cast<const T*>(d_vals);
    a.kp = p.two_kp;
    a.l0_rows = p.two_l0_rows;
    a.ucol = p.two_ucol;
    a.low = p.two_low;
    a.pairs = p.two_pairs;
    a.tail = p.two_tail;
    a.tiles = p.two_tiles;
    a.tail_off = p.two_tail_off;
    a.up = f->u_pair.as<typename Pair<T>::type>();
    a.slot = p.two_slot;
    a.l0_scan = p.two_l0_scan;
    a.lvl_rows = p.d_lvl_rows.as<int>();
    a.bs = p.d_bs.as<int>();
    a.u_sub = f->u_sub.as<T>();
    a.tri = f->tri.as<T>();
    a.dg = f->dg.as<T>();
    a.is_piv = f->is_piv.as<int>();
    a.perm = f->perm.as<int>();
    a.rowflags = f->rowflags.as<int>();
    a.u_col = f->u_col.as<int>();
    a.u_colp = f->u_colp.as<int>();
    a.u_val = f->u_val.as<T>();
    a.u_rng = f->u_rng.as<int2>();
    a.ut_col = f->ut_col.as<int>();
    a.ut_val = f->ut_val.as<T>();
    a.ut_rng = f->ut_rng.as<int2>();
    a.iperm = f->u_off.as<int>();
    a.pk_off = f->pk_off.as<long long>();
    a.pk_col = f->pk_col.as<T>();
    a.pk_row = f->pk_row.as<T>();
    a.ndmask = f->ndmask.as<unsigned>();
    a.scan_s = f->scan_s.as<int>();
    a.scan_c = f->scan_c.as<int>();
    a.simple_rows = f->simple_rows.as<int>();
    a.cplx = f->cplx.as<int>();
    a.citem = f->citem.as<CItem>();
    a.kind = f->kind.as<unsigned char>();
    a.nonfinite = f->nonfinite.as<int>();
    a.blocks = p.num_blocks;
    CULIPX_TRY(launch_overlapped(k_two_rows<T>, dim3((a.n0 + 255) / 256), dim3(256), s, !f->capturing, a));
    CULIPX_TRY(launch_overlapped(k_two_tiles<T>, dim3((a.nr1 + kTileWarps - 1) / kTileWarps), dim3(32 * kTileWarps),
                                 s, !f->capturing, a));
    const int splits = (a.nr1 + kOrderT - 1) / kOrderT;
    CULIPX_TRY(launch_overlapped(k_two_order<T>, dim3((a.n0 + kOrderT - 1) / kOrderT + splits), dim3(kOrderT), s,
                                 !f->capturing, a, splits));
    *launches += 3;
    return CULIPX_OK;
}

}  // namespace

int factor_two_level(Factor* f, const void* d_vals, cudaStream_t s, int* launches)
{
    if (f->precision == CULIPX_F64) return run<double>(f, d_vals, s, launches);
    return run<float>(f, d_vals, s, launches);
}

}  // namespace culipx
