// Host-side symbolic analysis of one KKT sparsity pattern and the device
// mirror that the numeric kernels read.
#pragma once

#include "common.h"
#include "device.h"

#include <mutex>
#include <vector>

namespace culipx {

enum BlockFormat : int { kSparse = 0, kDense = 1 };  // BLOCK_FORMAT, block_ildlt.cuh:17-21

// Per-block descriptor as the kernels read it (16 bytes, one load).
struct BlockDesc {
    int row;      // block row
    int col;      // block column
    int val_off;  // first value slot in the value store (dense: r*c, sparse: capacity)
    int cap;      // sparse: capacity in entries (max_nnz); dense: r*c
};

// Packing of the two-level form's arrays (Pattern::d_l0_rows, d_ucol, d_low).
namespace two {
constexpr int kNextInBlock = 1 << 30;         // l0_rows: the next fine row is in the same block
constexpr int kRowDense = 1 << 29;            // l0_rows: the row has entries in dense blocks
constexpr int kNoDiag = (int)0x80000000u;     // l0_rows: K stores no diagonal entry for the row
constexpr int kRowMask = kRowDense - 1;
constexpr int kDense = (int)0x80000000u;      // ucol: the entry is in a dense block
constexpr int kColMask = 0x7fffffff;
constexpr int kSameBlock = (int)0x80000000u;  // low.x: same block row as the entry before it
// pairs: x = slot of U_gb | kSameTarget | a << 27, y = slot of U_ga | kSameSum | b << 27
constexpr int kSlotMask = (1 << 26) - 1;
constexpr unsigned kSameTarget = 1u << 26;    // same (a, b) as the pair before it
constexpr unsigned kSameSum = 1u << 26;       // and the same update block
constexpr int kPlaceShift = 27;

// a level-1 block row: its rows, its rows' run of entries of U', its first
// pair, the place of its packed pivot triangles (two 16-byte loads)
struct alignas(16) Tile {
    int I, fr, h, entries;
    int slot, pair;
    long long pk_off;
};
static_assert(sizeof(Tile) == 32, "Tile is two 16-byte words");
}  // namespace two

struct Pattern {
    culipx_handle_t* handle = nullptr;
    // the creator's reference plus one per factor / batch made from it through
    // the C ABI; the last release frees the pattern (and releases the handle)
    std::atomic<int> refs{1};
    int n = 0;
    long long nnz = 0;
    int precision = CULIPX_F64;
    int fill_level = 0;
    double fill_factor = 1.0;

    int num_blocks = 0;
    std::vector<int> bs;         // num_blocks + 1
    std::vector<int> row_block;  // n

    int coarse_nnz = 0, fill_nnz = 0;
    std::vector<int> cs_off, cs_col, blk_nnzA;
    std::vector<int> blk_row, blk_col, fmt, max_nnz;
    std::vector<int> csc_off, csc_blk;

    int num_levels = 0;
    std::vector<int> lvl_off, lvl_rows, row_level;
    // every level-0 block row's diagonal block of K is diagonal (no entry
    // between two rows of the same level-0 block row): a level-0 row's K row
    // then reads only itself and rows of later levels
    bool l0_diagonal = false;
    int longest_row = 0;         // entries of K's longest row
    // two levels whose level-0 block rows have diagonal pivot blocks, rows of
    // moderate length (a KKT system in its natural order at fill level 0): the
    // factor runs on K's fine rows (factor_two_level.cu).  The device arrays
    // below exist for such patterns only.
    bool two_level = false;
    int l0_count = 0;             // fine rows of level 0
    int two_entries = 0;          // entries of U
    // slots of the pivot tiles' packed triangles (h_I (h_I + 1) / 2 per block
    // row, rounded up to 4 slots: every tile on a 16-byte boundary)
    std::vector<long long> pk_off;
    std::vector<int> lb_off, lb;  // factor order per level: pivots, then off-diagonal (CSR order)
    // per row position t of lvl_rows: index of the row's first off-diagonal
    // block inside its level's off-diagonal list
    std::vector<int> row_offdiag_start;
    long long sparse_slots = 0;   // sum of the sparse blocks' capacities
    std::vector<int> sb_off, sb;  // U' sweep order per column level
    int max_level_blocks = 0, max_level_rows = 0;
    int num_sparse = 0, num_dense = 0;

    // value-store layout (level-list order)
    std::vector<BlockDesc> desc;
    long long val_slots = 0;

    DeviceBuffer d_lvl_off, d_lvl_rows, d_bs;
    // what the general factorization reads (block_mirror)
    DeviceBuffer d_row_offdiag_start, d_cs_off, d_desc, d_csc_off, d_csc_blk, d_lb, d_a_dst, d_idx_init,
        d_nnz_init, d_fmt, d_maxnnz;
    // two_level: K's structure, from which block_mirror builds those once a
    // factor of the pattern first takes the general path
    std::vector<int> k_rowptr, k_colidx;
    std::mutex mirror_lock;
    bool mirrored = false;
    // two_level, parts of d_two: the level-1 block rows; K's row offsets; the level-0 fine rows; the
    // columns of U's entries, row after row; the entries of U', level-1 row
    // after level-1 row (column, slot in U); the products U_ga D_g U_gb of the
    // tiles' updates left of the diagonal (a < b), tile by tile, those of an
    // entry (a, b) together and in row order; K's own entries of the level-1 pivot tiles with their
    // offsets per tile; per fine row its first entry in U (level 0) or U'
    // (level 1); per level-0 position of lvl_rows the fine rows before it
    DeviceBuffer d_two;
    const int *two_kp = nullptr, *two_l0_rows = nullptr, *two_ucol = nullptr, *two_tail_off = nullptr,
              *two_slot = nullptr, *two_l0_scan = nullptr;
    const two::Tile* two_tiles = nullptr;
    const int2 *two_low = nullptr, *two_tail = nullptr;
    const uint2* two_pairs = nullptr;
    long long device_bytes = 0;
};

// Builds the analysis on the host and uploads the device mirror.
int analyze_pattern(culipx_handle_t* h, int n, const int* rowptr, const int* colidx,
                    int num_blocks, const int* block_starts, int fill_level, double fill_factor,
                    int precision, Pattern** out, int num_systems = 1, const int* system_row_offsets = nullptr);

// The device arrays of the general factorization: uploaded with the analysis,
// for a two-level pattern on the first call that needs them.
int block_mirror(Pattern& p);

}  // namespace culipx

struct culipx_pattern_t : culipx::Pattern {};
