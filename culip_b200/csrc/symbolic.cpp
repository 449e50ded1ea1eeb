// Symbolic analysis of a KKT sparsity pattern for the block-iLDL^T factor.
//
// Produces the same canonical output as the reference's host phase
// (libs/la/preconditioner/block_ildlt.impl.cuh):
//   coarse upper pattern           build_initial_coarse            :352-484
//   level-of-fill + diagonals      determine_coarse_level_fill..   :492-728
//   block CSC                      build_block_csc                 :732-762
//   row level sets, block order    find_level_sets                 :766-1011
//   formats, max_nnz, storage      build_blocks                    :1015-1280
//   U' sweep order                 solve_analysis_block            :2050-2150
// with different algorithms: per-row marker sets instead of global sorts, a
// longest-path pass over the block CSC for the levels (the level of block row
// c is 1 + the largest level of any row k < c with a block (k, c)), epoch-
// stamped visit arrays for the fill BFS, and counting sorts.  Rows inside a
// level are ascending (the reference's order there comes from OpenMP atomics).
#include "pattern.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <new>
#include <numeric>

#include <omp.h>

namespace culipx {

namespace {

int blk_size(const Pattern& p, int b) { return p.bs[b + 1] - p.bs[b]; }

// Coarse upper-triangular pattern with per-block counts of A's entries.
void coarse_pattern(Pattern& p, const int* rowptr, const int* colidx)
{
    const int cm = p.num_blocks;
    std::vector<std::vector<int>> rows_col(cm), rows_cnt(cm);
#pragma omp parallel
    {
        std::vector<int> cnt(cm, 0), touched;
        touched.reserve(256);
#pragma omp for schedule(dynamic, 64)
        for (int I = 0; I < cm; ++I) {
            touched.clear();
            for (int i = p.bs[I]; i < p.bs[I + 1]; ++i)
                for (int q = rowptr[i]; q < rowptr[i + 1]; ++q) {
                    const int c = colidx[q];
                    if (c < i) continue;
                    const int bc = p.row_block[c];
                    if (cnt[bc]++ == 0) touched.push_back(bc);
                }
            std::sort(touched.begin(), touched.end());
            rows_col[I].resize(touched.size());
            rows_cnt[I].resize(touched.size());
            for (size_t t = 0; t < touched.size(); ++t) {
                rows_col[I][t] = touched[t];
                rows_cnt[I][t] = cnt[touched[t]];
                cnt[touched[t]] = 0;
            }
        }
    }
    // level-of-fill and missing diagonals
    std::vector<std::vector<int>> fill(cm);
    const int max_level = p.fill_level;
#pragma omp parallel
    {
        std::vector<int> stamp(cm, -1), length(cm, 0), queue;
        queue.reserve(1024);
#pragma omp for schedule(dynamic, 16)
        for (int i = 0; i < cm; ++i) {
            if (max_level > 0) {
                queue.clear();
                queue.push_back(i);
                length[i] = 0;
                stamp[i] = i;
                for (size_t qh = 0; qh < queue.size(); ++qh) {
                    const int cur = queue[qh];
                    for (int j = p.bs[cur]; j < p.bs[cur + 1]; ++j)
                        for (int q = rowptr[j]; q < rowptr[j + 1]; ++q) {
                            const int kc = p.row_block[colidx[q]];
                            if (stamp[kc] == i) continue;
                            stamp[kc] = i;
                            if (kc < i && length[cur] < max_level) {
                                queue.push_back(kc);
                                length[kc] = length[cur] + 1;
                            }
                            if (kc > i && length[cur] > 0) fill[i].push_back(kc);
                        }
                }
            }
            // the reference inspects only the first block of the row
            const bool has_diag = !rows_col[i].empty() && rows_col[i][0] == i;
            if (!has_diag) fill[i].push_back(i);
            std::sort(fill[i].begin(), fill[i].end());
        }
    }
    p.cs_off.assign(cm + 1, 0);
    for (int I = 0; I < cm; ++I) p.cs_off[I + 1] = p.cs_off[I] + (int)(rows_col[I].size() + fill[I].size());
    p.coarse_nnz = p.cs_off[cm];
    p.fill_nnz = 0;
    for (int I = 0; I < cm; ++I) p.fill_nnz += (int)fill[I].size();
    p.cs_col.resize(p.coarse_nnz);
    p.blk_nnzA.resize(p.coarse_nnz);
#pragma omp parallel for schedule(static)
    for (int I = 0; I < cm; ++I) {
        // merge two sorted lists
        size_t a = 0, b = 0;
        int o = p.cs_off[I];
        const auto& rc = rows_col[I];
        const auto& fl = fill[I];
        while (a < rc.size() || b < fl.size()) {
            if (b >= fl.size() || (a < rc.size() && rc[a] < fl[b])) {
                p.cs_col[o] = rc[a];
                p.blk_nnzA[o] = rows_cnt[I][a];
                ++a;
            } else {
                p.cs_col[o] = fl[b];
                p.blk_nnzA[o] = 0;
                ++b;
            }
            ++o;
        }
    }
}

// Host arrays of the two-level form (Pattern::two_level).
struct TwoLevel {
    std::vector<int> l0_rows, l0_scan, slot, ucol, tail_off;
    std::vector<int2> low, tail;
    std::vector<uint2> pairs;
    std::vector<two::Tile> tiles;  // one more than there are, for the last one's end
};

// Fills the two-level form; false where the pattern has none: other than two
// levels, a level-0 pivot block with off-diagonal entries, an unsymmetric
// pattern (the general path reads the upper triangle only and takes any), or
// rows too long for a lane.  A lane walks a level-1 row and a thread a level-0
// row, while the general path gives a tile's update blocks to a warp one by
// one: about 1.4 us for each, measured, against at most 0.4 us here for each
// entry of a tile's longest row.
bool two_level_form(Pattern& p, const int* rowptr, const int* colidx, TwoLevel& w)
{
    if (p.num_levels != 2 || !p.l0_diagonal || p.n > two::kRowMask || p.nnz > two::kSlotMask) return false;
    const int q1 = p.lvl_off[1], q2 = p.lvl_off[2];
    w.slot.assign(p.n, 0);
    int entries = 0, lower = 0;
    for (int t = 0; t < q1; ++t) {
        const int I = p.lvl_rows[t];
        w.l0_scan.push_back((int)w.l0_rows.size());
        for (int i = p.bs[I]; i < p.bs[I + 1]; ++i) {
            const int k0 = rowptr[i], len = rowptr[i + 1] - k0;
            const bool diag = len > 0 && colidx[k0] == i;
            if ((len > 0 && colidx[k0] < i) || len > 256) return false;
            w.l0_rows.push_back(i | (i + 1 < p.bs[I + 1] ? two::kNextInBlock : 0) | (diag ? 0 : two::kNoDiag));
            w.slot[i] = entries;
            entries += len - diag;
        }
    }
    w.l0_scan.push_back((int)w.l0_rows.size());
    p.l0_count = (int)w.l0_rows.size();
    // level-1 rows: the entries before the row's own block mirror U's
    w.tail_off.push_back(0);
    for (int t = q1; t < q2; ++t) {
        const int I = p.lvl_rows[t], fr = p.bs[I];
        const int most = std::max(64, 3 * (p.csc_off[I + 1] - p.csc_off[I] - 1));
        for (int i = fr; i < p.bs[I + 1]; ++i) {
            int k1 = rowptr[i + 1];
            for (; k1 > rowptr[i] && colidx[k1 - 1] >= fr; --k1)
                if (colidx[k1 - 1] >= i) w.tail.push_back(make_int2(k1 - 1, (i - fr) * 32 + colidx[k1 - 1] - fr));
            if (k1 - rowptr[i] > most) return false;
            w.slot[i] = lower;
            lower += k1 - rowptr[i];
        }
        w.tail_off.push_back((int)w.tail.size());
        two::Tile tile = {I, fr, blk_size(p, I), lower - w.slot[fr], w.slot[fr], 0, p.pk_off[I]};
        w.tiles.push_back(tile);
    }
    w.tiles.push_back({0, 0, 0, 0, lower, 0, 0});
    if (entries != lower || entries == 0) return false;
    p.two_entries = entries;
    w.ucol.resize(entries);
    w.low.resize(entries);
#pragma omp parallel for schedule(static)
    for (int t = 0; t < q1; ++t) {
        const int I = p.lvl_rows[t], base = w.l0_scan[t];
        bool dense = false;
        for (int q = p.cs_off[I] + 1; q < p.cs_off[I + 1]; ++q) dense |= p.fmt[q] == kDense;
        for (int i = p.bs[I]; i < p.bs[I + 1]; ++i) {
            int k = rowptr[i];
            if (!(w.l0_rows[base + i - p.bs[I]] & two::kNoDiag)) ++k;
            int* out = w.ucol.data() + w.slot[i];
            for (int b = p.cs_off[I]; k < rowptr[i + 1]; ++k) {
                int c = colidx[k];
                if (dense) {
                    while (p.cs_col[b] != p.row_block[c]) ++b;
                    if (p.fmt[b] == kDense) {
                        c |= two::kDense;
                        w.l0_rows[base + i - p.bs[I]] |= two::kRowDense;
                    }
                }
                *out++ = c;
            }
        }
    }
    // the entries of U' and the pairs, tile by tile: first counted, then placed
    bool ok = true;
    std::vector<int> before(entries);
    std::vector<long long> pair_off(q2 - q1 + 1, 0);
#pragma omp parallel for schedule(static) reduction(&& : ok)
    for (int t = q1; t < q2; ++t) {
        const int I = p.lvl_rows[t], fr = p.bs[I];
        long long pairs = 0;
        for (int i = fr; i < p.bs[I + 1]; ++i) {
            int o = w.slot[i];
            for (int k = rowptr[i]; k < rowptr[i + 1] && colidx[k] < fr; ++k, ++o) {
                const int g = colidx[k];
                const int* r0 = colidx + rowptr[g];
                const int* r1 = colidx + rowptr[g + 1];
                const int* at = std::lower_bound(r0, r1, i);
                if (p.row_level[p.row_block[g]] != 0 || at == r1 || *at != i) {
                    ok = false;
                    break;
                }
                int n = 0;
                while (at - n > r0 && at[-n - 1] >= fr) ++n;
                before[o] = n;
                pairs += n;
                const bool same = k > rowptr[i] && p.row_block[g] == p.row_block[colidx[k - 1]];
                w.low[o] = make_int2(g | (same ? two::kSameBlock : 0), w.slot[g] + (int)(at - r0) - (r0[0] == g));
            }
        }
        pair_off[t - q1 + 1] = pairs;
    }
    if (!ok) return false;
    for (int t = 0; t < q2 - q1; ++t) pair_off[t + 1] += pair_off[t];
    // dense tiles (16 pairs an entry in full ones of 32) would take more memory
    // than their blocks do; the general path stores those dense
    if (pair_off[q2 - q1] > std::min(0x7fffffffLL, 8LL * entries + 4096)) return false;
    w.pairs.resize((size_t)pair_off[q2 - q1]);
    for (int t = 0; t <= q2 - q1; ++t) w.tiles[t].pair = (int)pair_off[t];
    int no_memory = 0;
#pragma omp parallel
    {
        struct Item {
            int place, block, b, a;
        };
        std::vector<Item> items;
#pragma omp for schedule(static)
        for (int t = q1; t < q2; ++t) {
            const int I = p.lvl_rows[t], fr = p.bs[I];
            items.clear();
            try {  // no exception may leave the parallel region
                items.reserve((size_t)(pair_off[t - q1 + 1] - pair_off[t - q1]));
            } catch (const std::bad_alloc&) {
#pragma omp atomic write
                no_memory = 1;
                continue;
            }
            for (int i = fr; i < p.bs[I + 1]; ++i)
                for (int k = rowptr[i], o = w.slot[i]; k < rowptr[i + 1] && colidx[k] < fr; ++k, ++o)
                    for (int n = 1; n <= before[o]; ++n) {
                        const int sb = w.low[o].y;
                        items.push_back({(w.ucol[sb - n] & two::kColMask) - fr + 32 * (i - fr),
                                         p.row_block[colidx[k]], sb, sb - n});
                    }
            // entry by entry; a stable sort keeps an entry's rows in order
            std::stable_sort(items.begin(), items.end(),
                             [](const Item& x, const Item& y) { return x.place < y.place; });
            uint2* out = w.pairs.data() + pair_off[t - q1];
            for (size_t k = 0; k < items.size(); ++k) {
                const Item& m = items[k];
                const bool target = k > 0 && items[k - 1].place == m.place;
                const bool sum = target && items[k - 1].block == m.block;
                *out++ = make_uint2((unsigned)m.b | (target ? two::kSameTarget : 0u) |
                                        ((unsigned)(m.place & 31) << two::kPlaceShift),
                                    (unsigned)m.a | (sum ? two::kSameSum : 0u) |
                                        ((unsigned)(m.place >> 5) << two::kPlaceShift));
            }
        }
    }
    if (no_memory) throw std::bad_alloc();
    return ok;
}

}  // namespace

int analyze_pattern(culipx_handle_t* h, int n, const int* rowptr, const int* colidx,
                    int num_blocks, const int* block_starts, int fill_level, double fill_factor,
                    int precision, Pattern** out, int num_systems, const int* system_row_offsets)
{
    if (!out || !rowptr || !colidx || !block_starts || n <= 0 || num_blocks <= 0 || num_blocks > n)
        return fail(CULIPX_INVALID_ARG, "culipx_pattern_analyze: bad arguments");
    if (fill_level < 0) return fail(CULIPX_INVALID_ARG, "culipx_pattern_analyze: fill_level < 0");
    if (!(fill_factor >= 1.0))
        return fail(CULIPX_INVALID_ARG, "culipx_pattern_analyze: fill_factor must be >= 1 (the driver clamps it, block_ildlt.cc:50)");
    if (precision != CULIPX_F64 && precision != CULIPX_F32)
        return fail(CULIPX_INVALID_ARG, "culipx_pattern_analyze: bad precision");
    if (rowptr[0] != 0) return fail(CULIPX_INVALID_ARG, "culipx_pattern_analyze: rowptr[0] != 0");

    auto pp = std::make_unique<culipx_pattern_t>();  // freed on every way out, exceptions too
    Pattern& p = *pp;
    p.handle = h;
    p.n = n;
    p.nnz = rowptr[n];
    p.precision = precision;
    p.fill_level = fill_level;
    p.fill_factor = fill_factor;
    p.num_blocks = num_blocks;
    const int cm = num_blocks;

    p.bs.assign(block_starts, block_starts + cm);
    p.bs.push_back(n);
    for (int b = 0; b < cm; ++b) {
        const int sz = p.bs[b + 1] - p.bs[b];
        if (sz < 1 || sz > 32)
            return fail(CULIPX_INVALID_ARG, "culipx_pattern_analyze: block %d has size %d (must be 1..32)", b, sz);
    }
    if (p.bs[0] != 0) return fail(CULIPX_INVALID_ARG, "culipx_pattern_analyze: block_starts[0] != 0");
    // systems of a block-diagonal union (default: one system): per block row
    // its system's first block row and block count, for the format rule
    std::vector<int> sys_first(cm, 0), sys_blocks(cm, cm);
    if (num_systems > 1 && system_row_offsets) {
        if (system_row_offsets[0] != 0 || system_row_offsets[num_systems] != n)
            return fail(CULIPX_INVALID_ARG, "culipx_pattern_analyze_systems: row offsets must run from 0 to n");
        int b0 = 0;
        for (int k = 0; k < num_systems; ++k) {
            int b1 = b0;
            while (b1 < cm && p.bs[b1] < system_row_offsets[k + 1]) ++b1;
            if (p.bs[b0] != system_row_offsets[k] || p.bs[b1] != system_row_offsets[k + 1] || b1 == b0)
                return fail(CULIPX_INVALID_ARG, "culipx_pattern_analyze_systems: system %d does not start and end on block boundaries", k);
            for (int I = b0; I < b1; ++I) {
                sys_first[I] = b0;
                sys_blocks[I] = b1 - b0;
            }
            b0 = b1;
        }
    }
    for (int i = 0; i < n; ++i) p.longest_row = std::max(p.longest_row, rowptr[i + 1] - rowptr[i]);
    for (int i = 0; i < n; ++i)
        for (int q = rowptr[i]; q < rowptr[i + 1]; ++q)
            if (colidx[q] < 0 || colidx[q] >= n || (q > rowptr[i] && colidx[q] <= colidx[q - 1]))
                return fail(CULIPX_INVALID_ARG, "culipx_pattern_analyze: row %d: columns must be sorted, unique, in range", i);
    p.row_block.resize(n);
    for (int b = 0; b < cm; ++b)
        for (int j = p.bs[b]; j < p.bs[b + 1]; ++j) p.row_block[j] = b;

    coarse_pattern(p, rowptr, colidx);
    const int cnz = p.coarse_nnz;
    p.blk_row.resize(cnz);
    p.blk_col.resize(cnz);
    for (int I = 0; I < cm; ++I)
        for (int q = p.cs_off[I]; q < p.cs_off[I + 1]; ++q) { p.blk_row[q] = I; p.blk_col[q] = p.cs_col[q]; }

    // block CSC by counting sort (rows ascend within a column)
    p.csc_off.assign(cm + 1, 0);
    for (int q = 0; q < cnz; ++q) p.csc_off[p.cs_col[q] + 1]++;
    for (int c = 0; c < cm; ++c) p.csc_off[c + 1] += p.csc_off[c];
    p.csc_blk.resize(cnz);
    {
        std::vector<int> pos(p.csc_off.begin(), p.csc_off.end() - 1);
        for (int q = 0; q < cnz; ++q) p.csc_blk[pos[p.cs_col[q]]++] = q;
    }

    // levels: longest path over the upper block pattern
    p.row_level.assign(cm, 0);
    for (int c = 0; c < cm; ++c) {
        int lv = 0;
        for (int q = p.csc_off[c]; q < p.csc_off[c + 1]; ++q) {
            const int k = p.blk_row[p.csc_blk[q]];
            if (k != c) lv = std::max(lv, p.row_level[k] + 1);
        }
        p.row_level[c] = lv;
    }
    p.num_levels = 0;
    for (int c = 0; c < cm; ++c) p.num_levels = std::max(p.num_levels, p.row_level[c] + 1);
    p.l0_diagonal = true;
    for (int c = 0; c < cm && p.l0_diagonal; ++c) {
        if (p.row_level[c] != 0) continue;
        for (int i = p.bs[c]; i < p.bs[c + 1]; ++i)
            for (int q = rowptr[i]; q < rowptr[i + 1]; ++q)
                if (colidx[q] != i && p.row_block[colidx[q]] == c) p.l0_diagonal = false;
    }
    const int nl = p.num_levels;
    p.lvl_off.assign(nl + 1, 0);
    for (int c = 0; c < cm; ++c) p.lvl_off[p.row_level[c] + 1]++;
    for (int L = 0; L < nl; ++L) p.lvl_off[L + 1] += p.lvl_off[L];
    p.lvl_rows.resize(cm);
    {
        std::vector<int> pos(p.lvl_off.begin(), p.lvl_off.end() - 1);
        for (int c = 0; c < cm; ++c) p.lvl_rows[pos[p.row_level[c]]++] = c;  // ascending
    }

    // factor order per level: pivots (row order) then off-diagonal blocks (block-id order)
    p.lb_off.assign(nl + 1, 0);
    p.lb.resize(cnz);
    p.max_level_blocks = 0;
    p.max_level_rows = 0;
    {
        int o = 0;
        for (int L = 0; L < nl; ++L) {
            p.lb_off[L] = o;
            for (int t = p.lvl_off[L]; t < p.lvl_off[L + 1]; ++t) p.lb[o++] = p.cs_off[p.lvl_rows[t]];  // diagonal is first
            for (int t = p.lvl_off[L]; t < p.lvl_off[L + 1]; ++t) {
                const int r = p.lvl_rows[t];
                for (int q = p.cs_off[r] + 1; q < p.cs_off[r + 1]; ++q) p.lb[o++] = q;
            }
            p.max_level_blocks = std::max(p.max_level_blocks, o - p.lb_off[L]);
            p.max_level_rows = std::max(p.max_level_rows, p.lvl_off[L + 1] - p.lvl_off[L]);
        }
        p.lb_off[nl] = o;
        p.row_offdiag_start.resize(cm);
        for (int L = 0; L < nl; ++L) {
            int s = 0;
            for (int t = p.lvl_off[L]; t < p.lvl_off[L + 1]; ++t) {
                p.row_offdiag_start[t] = s;
                s += p.cs_off[p.lvl_rows[t] + 1] - p.cs_off[p.lvl_rows[t]] - 1;
            }
        }
    }
    // U' sweep order: per column level, pivots then off-diagonal blocks (block-id order)
    p.sb_off.assign(nl + 1, 0);
    p.sb.resize(cnz);
    {
        int o = 0;
        for (int L = 0; L < nl; ++L) {
            p.sb_off[L] = o;
            for (int t = p.lvl_off[L]; t < p.lvl_off[L + 1]; ++t) p.sb[o++] = p.cs_off[p.lvl_rows[t]];
            const int o0 = o;
            for (int t = p.lvl_off[L]; t < p.lvl_off[L + 1]; ++t) {
                const int c = p.lvl_rows[t];
                for (int q = p.csc_off[c]; q < p.csc_off[c + 1] - 1; ++q) p.sb[o++] = p.csc_blk[q];
            }
            std::sort(p.sb.begin() + o0, p.sb.begin() + o);
        }
        p.sb_off[nl] = o;
    }

    // formats and max_nnz
    p.fmt.resize(cnz);
    p.max_nnz.resize(cnz);
    const bool dbl = (precision == CULIPX_F64);
    for (int I = 0; I < cm; ++I) {
        int sum_nnz = 0, sum_blocks = 0;
        for (int q = p.cs_off[I]; q < p.cs_off[I + 1]; ++q) {
            sum_nnz += p.blk_nnzA[q];
            sum_blocks += (p.blk_nnzA[q] != 0);
        }
        // a block row without any A entry has no defined average in the
        // reference (0/0); such rows get 0 here
        const int avg = (sum_blocks == 0) ? 0
                        : dbl ? (int)std::ceil((double)sum_nnz / (double)sum_blocks)
                              : (int)std::ceil((float)sum_nnz / (float)sum_blocks);
        const int r = blk_size(p, I);
        for (int q = p.cs_off[I]; q < p.cs_off[I + 1]; ++q) {
            const int J = p.cs_col[q];
            const int c = blk_size(p, J);
            const int src = p.blk_nnzA[q] ? p.blk_nnzA[q] : avg;
            const int cap = dbl ? (int)std::ceil(fill_factor * (double)src)
                                : (int)std::ceil((float)fill_factor * (float)src);
            const int mx = std::min(r * c, cap);
            p.max_nnz[q] = mx;
            const size_t vb = dbl ? 8 : 4;
            const double lhs = (double)((4 + vb) * (size_t)(long long)mx);
            const double rhs = dbl ? 0.5 * 8.0 * (double)r * (double)c : (double)(0.5f * 4.0f * (float)r * (float)c);
            // the last 10 % of a system's block rows keep dense blocks
            const bool sparse = (I != J) && ((double)(I - sys_first[I]) < 0.9 * (double)sys_blocks[I]) && (lhs < rhs);
            p.fmt[q] = sparse ? kSparse : kDense;
            if (sparse) ++p.num_sparse; else ++p.num_dense;
        }
    }

    // value-store layout in factor order
    p.desc.resize(cnz);
    {
        long long o = 0;
        for (int t = 0; t < cnz; ++t) {
            const int q = p.lb[t];
            const int r = blk_size(p, p.blk_row[q]), c = blk_size(p, p.blk_col[q]);
            BlockDesc& d = p.desc[q];
            d.row = p.blk_row[q];
            d.col = p.blk_col[q];
            d.cap = (p.fmt[q] == kDense) ? r * c : std::max(p.max_nnz[q], p.blk_nnzA[q]);
            d.val_off = (int)o;
            o += d.cap;
            if (p.fmt[q] == kSparse) p.sparse_slots += d.cap;
            if (o > 0x7fffffffLL) return fail(CULIPX_NOT_SUPPORTED, "culipx_pattern_analyze: factor storage exceeds 2^31 slots");
        }
        p.val_slots = o;
    }

    p.pk_off.assign(cm + 1, 0);
    for (int I = 0; I < cm; ++I) {
        const long long hI = blk_size(p, I);
        p.pk_off[I + 1] = p.pk_off[I] + (hI * (hI + 1) / 2 + 3) / 4 * 4;
    }
    TwoLevel form;
    p.two_level = two_level_form(p, rowptr, colidx, form);

    // device mirror (not for a host-only handle)
    if (h->device < 0) {
        *out = pp.release();
        return CULIPX_OK;
    }
    int st = CULIPX_OK;
    auto up = [&](DeviceBuffer& buf, const void* src, size_t bytes) {
        if (st == CULIPX_OK) st = buf.upload(h, src, bytes);
    };
    up(p.d_lvl_off, p.lvl_off.data(), sizeof(int) * (p.num_levels + 1));
    up(p.d_lvl_rows, p.lvl_rows.data(), sizeof(int) * cm);
    up(p.d_bs, p.bs.data(), sizeof(int) * (cm + 1));
    p.device_bytes = (long long)(p.d_lvl_off.bytes() + p.d_lvl_rows.bytes() + p.d_bs.bytes());
    p.k_rowptr.assign(rowptr, rowptr + n + 1);
    p.k_colidx.assign(colidx, colidx + p.nnz);
    if (!p.two_level && st == CULIPX_OK) st = block_mirror(p);
    if (p.two_level) {
        // one allocation and copy for all of them, each part on a 16-byte boundary
        const std::pair<const void*, size_t> parts[] = {
            {rowptr, sizeof(int) * (n + 1)},
            {form.l0_rows.data(), sizeof(int) * form.l0_rows.size()},
            {form.ucol.data(), sizeof(int) * form.ucol.size()},
            {form.low.data(), sizeof(int2) * form.low.size()},
            {form.tail.data(), sizeof(int2) * form.tail.size()},
            {form.tail_off.data(), sizeof(int) * form.tail_off.size()},
            {form.slot.data(), sizeof(int) * n},
            {form.l0_scan.data(), sizeof(int) * form.l0_scan.size()},
            {form.tiles.data(), sizeof(two::Tile) * form.tiles.size()},
            {form.pairs.data(), sizeof(uint2) * form.pairs.size()}};
        size_t total = 0;
        for (const auto& q : parts) total += (q.second + 15) / 16 * 16;
        std::vector<unsigned char> all(total);
        std::vector<size_t> at;
        total = 0;
        for (const auto& q : parts) {
            at.push_back(total);
            if (q.second) std::memcpy(all.data() + total, q.first, q.second);
            total += (q.second + 15) / 16 * 16;
        }
        up(p.d_two, all.data(), all.size());
        const unsigned char* d = p.d_two.as<unsigned char>();
        p.two_kp = reinterpret_cast<const int*>(d + at[0]);
        p.two_l0_rows = reinterpret_cast<const int*>(d + at[1]);
        p.two_ucol = reinterpret_cast<const int*>(d + at[2]);
        p.two_low = reinterpret_cast<const int2*>(d + at[3]);
        p.two_tail = reinterpret_cast<const int2*>(d + at[4]);
        p.two_tail_off = reinterpret_cast<const int*>(d + at[5]);
        p.two_slot = reinterpret_cast<const int*>(d + at[6]);
        p.two_l0_scan = reinterpret_cast<const int*>(d + at[7]);
        p.two_tiles = reinterpret_cast<const two::Tile*>(d + at[8]);
        p.two_pairs = reinterpret_cast<const uint2*>(d + at[9]);
    }
    if (st != CULIPX_OK) return st;
    p.device_bytes += (long long)p.d_two.bytes();
    *out = pp.release();
    return CULIPX_OK;
}

int block_mirror(Pattern& p)
{
    std::lock_guard<std::mutex> lock(p.mirror_lock);
    if (p.mirrored) return CULIPX_OK;
    culipx_handle_t* h = p.handle;
    const int cm = p.num_blocks, cnz = p.coarse_nnz;
    // gather destinations of A's upper entries
    std::vector<int> a_dst(p.nnz, -1), idx_init(p.val_slots, -1), nnz_init(cnz, 0);
#pragma omp parallel for schedule(dynamic, 64)
    for (int I = 0; I < cm; ++I) {  // a block row's slots are its own
        const int* cb = p.cs_col.data() + p.cs_off[I];
        const int clen = p.cs_off[I + 1] - p.cs_off[I];
        for (int i = p.bs[I]; i < p.bs[I + 1]; ++i)
            for (int q = p.k_rowptr[i]; q < p.k_rowptr[i + 1]; ++q) {
                const int c = p.k_colidx[q];
                if (c < i) continue;
                const int J = p.row_block[c];
                const int pos = (int)(std::lower_bound(cb, cb + clen, J) - cb);
                const int b = p.cs_off[I] + pos;
                const int w = blk_size(p, J);
                const int local = (i - p.bs[I]) * w + (c - p.bs[J]);
                const BlockDesc& d = p.desc[b];
                if (p.fmt[b] == kDense) {
                    a_dst[q] = d.val_off + local;
                } else {
                    const int slot = d.val_off + nnz_init[b]++;
                    a_dst[q] = slot;
                    idx_init[slot] = local;
                }
            }
    }

    // on a stream of its own: a copy on the legacy stream would end the
    // capture of a blocking stream
    const struct {
        DeviceBuffer& buf;
        const void* src;
        size_t size;
    } parts[] = {{p.d_cs_off, p.cs_off.data(), sizeof(int) * (cm + 1)},
                 {p.d_row_offdiag_start, p.row_offdiag_start.data(), sizeof(int) * cm},
                 {p.d_desc, p.desc.data(), sizeof(BlockDesc) * cnz},
                 {p.d_csc_off, p.csc_off.data(), sizeof(int) * (cm + 1)},
                 {p.d_csc_blk, p.csc_blk.data(), sizeof(int) * cnz},
                 {p.d_lb, p.lb.data(), sizeof(int) * cnz},
                 {p.d_a_dst, a_dst.data(), sizeof(int) * p.nnz},
                 {p.d_idx_init, idx_init.data(), sizeof(int) * p.val_slots},
                 {p.d_nnz_init, nnz_init.data(), sizeof(int) * cnz},
                 {p.d_fmt, p.fmt.data(), sizeof(int) * cnz},
                 {p.d_maxnnz, p.max_nnz.data(), sizeof(int) * cnz}};
    cudaStream_t s = nullptr;
    CULIPX_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    int st = CULIPX_OK;
    long long bytes = 0;
    auto up = [&]() -> int {
        for (const auto& q : parts) {
            CULIPX_TRY(q.buf.alloc(h, q.size));
            if (q.size) CULIPX_CUDA(cudaMemcpyAsync(q.buf.get(), q.src, q.size, cudaMemcpyHostToDevice, s));
            bytes += (long long)q.buf.bytes();
        }
        return CULIPX_OK;
    };
    st = up();
    const cudaError_t e = cudaStreamSynchronize(s);
    cudaStreamDestroy(s);
    if (st == CULIPX_OK && e != cudaSuccess)
        st = fail(CULIPX_CUDA_ERROR, "uploading the block form failed: %s", cudaGetErrorString(e));
    if (st != CULIPX_OK) {  // the next call starts over
        for (const auto& q : parts) q.buf.release();
        return st;
    }
    p.device_bytes += bytes;
    p.k_rowptr = std::vector<int>();
    p.k_colidx = std::vector<int>();
    p.mirrored = true;
    return CULIPX_OK;
}

}  // namespace culipx
