// rules.hpp -- host-side rules that choose a kernel's form, without CUDA: plain functions of
// sizes, so that they are tested by themselves.
#pragma once

#include <algorithm>

namespace hamlss {

// ------------------------------------------------------------- persistent CG (cg_persist.cuh)
constexpr int kPersistMaxRows = 3584;         // rows a block
constexpr int kPersistClusterBlocks = 16;
constexpr int kPersistMaxBlocks = 256;        // sets of partial sums (all_sums)

// Whether a launch of `blocks` blocks runs all at once, as both forms of the kernel need: a
// cluster of that size fits the device (active_clusters, from the occupancy query), or the
// grid's blocks are resident together (blocks_per_sm).  Partitioned devices and contexts that
// may use a part of one report less than the whole chip.
inline bool persist_can_run(bool cluster, int blocks, int active_clusters, int blocks_per_sm, int sm_count) {
    if (blocks < 1) return false;
    if (cluster) return blocks <= kPersistClusterBlocks && active_clusters >= 1;
    return blocks <= kPersistMaxBlocks && (long long)blocks_per_sm * sm_count >= blocks;
}

// Threads a block: one a row up to 256, unless the block reads many of its neighbours' rows each
// trip (`outside`: columns of its window that are not its own), which wait for L2 four a thread
// at a time.  The sums keep their order (the other warps' are zero).  28,000 rows of 5, 300
// trips, at 256 / 512 threads: 18,000 outside 5.1 / 3.6 ms, 24,000 6.0 / 4.1 ms (two launches a
// trip: 5.2); 33,000 rows, 6,000 outside 2.9 / 2.5 ms.
inline int persist_threads(int rows, int outside) { return rows <= 256 && outside <= 4096 ? 256 : 512; }

// --------------------------------------------------------------- FP64 products (spmv.cuh)
constexpr int kProdTile = 512;                // products a warp of k_spmv_prod holds

// Whether a matrix of long rows next to one another is left to a lane a row (k_spmv): all
// entries of the rows that one warp takes (`heaviest`: the most of any warp) go through its
// tile, and where a tile holds one row's part, one lane adds it while 31 wait.  Cycles of the
// slowest warp, measured: a tile ~1,500 for its loads and ~12 an addition; a lane a row ~225 an
// entry.  The rest of the matrix runs beside that warp and prefers k_spmv_prod by about a
// 200th of a cycle an entry.  A product of 100,000 rows of 10 with 40 neighbouring rows longer,
// k_spmv_prod / k_spmv: of 100 31 / 31 us, of 300 66 / 48, of 900 184 / 108; with 8 rows of 900
// 72 / 101.
inline bool prod_uneven(int longest, long long heaviest, long long nnz) {
    const long long tiles = (heaviest + kProdTile - 1) / kProdTile;
    const long long warp = tiles * (1500 + 12LL * std::min(longest, kProdTile));
    return warp - 225LL * longest > nnz / 200;
}

// Whether k_spmv_prod's entry indices stay in range: it steps by a tile past the last entry.
inline bool prod_indexable(long long nnz) { return nnz <= 2147483647LL - kProdTile; }

// Whether the gathers of neighbouring rows mostly fall on different lines: of the places that
// two neighbouring rows both have, fewer than half with columns at most kNearColumns apart.
// (Grids in natural or coloured order: nearly all.  Rows in random order, or random columns in
// a band of +-100: nearly none; spmv_stream.cuh's WIDE form then takes 94 us for 199, and 57
// for 59.)
constexpr int kNearColumns = 8;
constexpr int kNeighbourRows = 65536;         // rows looked at, about
inline bool gathers_scattered(int pairs, int near) { return pairs > 0 && 2LL * near < pairs; }

// ---------------------------------------------------------- triangular sweeps (ilu_sweep.cuh)
// Kernel of a triangle's sweep:
//   RING   one block, shared-memory rings, rows of at most 16 entries in 2, 4, 8 or 16 places
//   BLOCK  one block reading through the caches
//   GRID   the whole grid, a grid barrier (~2 us) a level
enum class TriMode { RING, BLOCK, GRID };
constexpr int kTriMaxRow = 16;

// Entry places of a RING triangle's rows, from its longest row.
inline int tri_places(int max_row) { return max_row <= 2 ? 2 : max_row <= 4 ? 4 : max_row <= 8 ? 8 : 16; }

// More than 4,096 rows a level on average: GRID (one block spends longer than a grid barrier
// on a level's rows).  Otherwise RING wherever its rows need 2 or 4 places (1.1 to 2 times
// BLOCK at every width, 200 to 4,000 rows a level of 1 to 4 entries).  With 8 and 16 places all
// rows pay for the longest one -- their empty places are copied too, and a step holds 416 or 224
// rows -- so RING and BLOCK are weighed.  Microseconds, measured: a RING step 0.3 and 0.003 a row
// (8 places), 0.35 and 0.0087 a row (16); a BLOCK level 0.95 and 0.00065 an entry, 0.0009 where
// rows have more than 8 on average.  An apply, RING / BLOCK: 8 of 8 places used, 500 rows a level
// 0.22 / 0.43 ms, 4,000 1.93 / 2.66; 2 of 8, 2,000 a level 0.95 / 0.56; 16 of 16, 500 a level 0.59 /
// 1.13; 4 of 16, 2,000 a level 2.48 / 0.76; one row of 14 in a 512^2 grid's rows of 2 3.4 / 2.3.
inline TriMode tri_mode(int n, int nlev, int nnz, int max_row) {
    if (nlev < 1) return TriMode::BLOCK;
    const double width = (double)n / nlev;
    if (width > 4096.0) return TriMode::GRID;
    if (max_row > kTriMaxRow) return TriMode::BLOCK;
    const int K = tri_places(max_row);
    if (K <= 4) return TriMode::RING;
    const double rows = K == 8 ? 416.0 : 224.0;                        // a step
    const double steps = nlev * std::max(1.0, width / rows + 0.5);     // (a level's last is partly filled)
    const double ring = K == 8 ? 0.3 * steps + 0.003 * n : 0.35 * steps + 0.0087 * n;
    const double block = 0.95 * nlev + (nnz > 8.0 * n ? 0.0009 : 0.00065) * nnz;
    return ring <= block ? TriMode::RING : TriMode::BLOCK;
}

// ------------------------------------------------------------- FGMRES multi-dots (fgmres.cu)
// A thread an entry (k_mdot_few) where there are few vectors and enough entries that the loads
// count: the figures stand at the kernel.
inline bool mdot_few(int n, int nv) { return nv <= 8 && n >= (1 << 19); }

// ----------------------------------------------------------- dense right operands (amg.cu)
// Entries of a right operand that an AMG setup holds dense, and of the slots beside it, on a
// context of its own and on a server's solve lane (8 and 12 bytes an entry).
constexpr long long kGatherDense = 16LL << 20;
constexpr long long kGatherDenseLane = 2LL << 20;
constexpr int kGatherSlots = 2 << 20;

// --------------------------------------------------------- the server's estimates (serve.cu)
// Device footprint of one request while it is admitted on a solve lane (bytes, an upper
// estimate): CSR (int32 row_ptr + int32 col_idx + FP64 values), its FP32 copy and the diagonal;
// Krylov workspace (eight FP64 and eight FP32 vectors, the FGMRES basis V and Z of 2m+1
// vectors); and the larger of
//   ILU(0)  the factor, L and U in sweep order, FP64 and FP32 -- a ring triangle's rows have the
//           places of its longest row (at most max_row entries), the others their own entries --,
//           diagonals with reciprocals, level sets and vectors
//   AMG     the hierarchy (operators of the coarse levels, P and R) bounded by twice the fine
//           operator, the dense right operand and its slots, and the coarse elimination's copy
// (max_row 5, m = 30: FGMRES + ILU(0) on 250^2 holds 50 MB.)
inline long long footprint_of(long long n, long long nnz, int m, int max_row) {
    const long long csr = 4 * (n + 1) + 12 * nnz;
    const long long f32 = 4 * nnz + 8 * n;
    const long long ws = 8 * 8 * n + 8 * 4 * n + (2LL * m + 1) * 8 * n + 64 * 1024;
    const long long ring = 2LL * tri_places(std::min(max_row, kTriMaxRow)) * (8 + 4 + 4 + 4) * n;
    const long long rows = 16 * nnz + 8 * n;
    const long long ilu = 8 * nnz + ring + (max_row > 4 ? rows : 0) + 100 * n;
    const long long small = std::min(n, 100000LL), square = small * small;      // (larger: the caps)
    const long long amg = 2 * (csr + f32) + 4 * 8 * n + std::min(20 * kGatherDenseLane, 5 * square) +
                          std::min(8LL << 20, 8 * square);
    return csr + f32 + 8 * n + ws + std::max(ilu, amg) + (1 << 20);
}

// Footprint of a request solved in the batch lane: the block's share of the batch's CSR (FP64 +
// FP32), the ILU(0) factor while it is made, its entries in level order, level sets, and the
// per-system vectors (2m + 5 in FP32, four in FP64).
inline long long footprint_small(long long n, long long nnz, int m) {
    return 36 * nnz + (8LL * m + 160) * n + 4096;
}

// ------------------------------------------------------------------ batched solves (batch.cu)
constexpr int kBatchSmall = 100;              // rows a warp solves by itself
constexpr int kBatchGroups = 6;
// Scheduling group of a system: the size classes (n <= 1,024, 4,096, 16,384, larger) are groups 2
// to 5; of the first class, systems of at most kBatchSmall rows are group 0 and the next ones, up
// to 200 rows (CG) or 640 (FGMRES), group 1, with narrower teams.  A width depends on the system
// alone, never on the batch, so that a system's result does not either.  Device time, ms, at 32 /
// 64 / 128 threads: CG, 121 rows, 40 systems 0.42 / 0.23 / 0.20, 2,000 0.48 / 0.47 / 0.77; 256 rows
// 0.88 / 0.49 / 0.32, 1.01 / 0.99 / 1.22; FGMRES + ILU(0), 256 rows 0.37 / 0.30 / 0.26, 0.47 / 0.59 /
// 0.95; 400 rows 0.52 / 0.39 / 0.34, 0.81 / 0.87 / 1.29; 1,024 rows 1.2 / 0.73 / 0.58, 1.9 / 2.0 / 2.4.
inline int batch_group(int n, bool cg) {
    if (n <= kBatchSmall) return 0;
    if (n <= (cg ? 200 : 640)) return 1;
    return n <= 1024 ? 2 : n <= 4096 ? 3 : n <= 16384 ? 4 : 5;
}
inline int batch_group_class(int group) { return std::max(0, group - 2); }
// (`width`: of the group's size class)
inline int batch_group_width(int group, int width) {
    return group == 0 ? 32 : group == 1 ? std::min(width, 64) : width;
}

}  // namespace hamlss
