// Device execution plan of the supernodal factorization and solves.
//
// The symbolic analysis yields the reference's supernodes, whose partition is
// part of the drop-in contract (SN_rp, SN_inner, the value layout).  Many of
// them are thin -- a separator node with a private neighbour in an ancestor
// separator always starts a new fundamental supernode -- and a chain of thin
// supernodes is a chain of large, nearly identical update matrices.  The GPU
// therefore computes on *fronts*: maximal runs of supernodes in which each is
// the last child of the next (so their rows are contiguous) merged while the
// structural zeros this adds stay within relaxation limits (the classical
// relaxed-supernode amalgamation).  A front's column set is that of its top
// supernode; zeros it carries stay exactly zero through every kernel.  The
// reference's per-supernode layout (row-major U0 squares, U1 rectangles at
// SN_tri_ptr / SN_rec_ptr) is produced from the fronts by an export kernel on
// request.
//
//  * the factor arena holds, per front, U0 (n0 x n0, row-major upper), U1
//    (n0 x n1, row-major), rows padded to kLdAlign entries (32-byte aligned
//    rows for vector and bulk copies), and an update-matrix region in which each front's
//    n1 x n1 contribution block V (Multifrontal.hpp:165) lives from its
//    front's level until its parent's level; V regions are reused across
//    levels by a best-fit allocator and zeroed by the level that owns them;
//  * fronts are grouped in levels by height in the front tree (leaves are
//    level 0); a level runs after all lower levels;
//  * within a level, children's update matrices are added into their parents
//    in child-rank passes (pass r adds every parent's r-th child), so no two
//    tasks of a launch write the same entry and the summation order is the
//    reference's (A, then children in order, Multifrontal.hpp:210-224);
//  * each front's pivots are eliminated in panels of kPanel rows: a potrf
//    launch factors the panel's diagonal block in place (one CTA per front),
//    a trsm launch solves the panel's row of the front against it (one CTA
//    per kRestChunk columns), an update launch applies the rank-kPanel
//    trailing update to the remaining rows of U0 and U1 as 64 x 64 GEMM
//    tiles, and in the update launch of a front's last panel its
//    V -= U1^T U1 tiles run with the full depth K = n0.
#pragma once

#include <cstdint>
#include <vector>

#include "symbolic.hpp"

namespace tb
{

constexpr int kPanel     = 64;    // pivot panel width
constexpr int kTile      = 64;    // GEMM output tile (kTile x kTile)
constexpr int kRestChunk = 64;    // rest columns per panel-solve CTA
constexpr int kSolveRest = 64;    // rows per solve-update task
constexpr int kLdAlign   = 4;     // row padding of every front block (entries)
constexpr std::uint64_t kDiagFlag = 1ull << 62;   // marks diagonal entries in the assembly map

// Relaxed amalgamation limits: a merge whose front has at most nrelax[0]
// rows is always taken; otherwise the fraction of structural zeros in the
// merged front must stay below zrelax[k] for the first k with
// rows <= nrelax[k] (zrelax[2] beyond).
struct Relaxation
{
    std::int32_t nrelax[3] = { 8, 32, 64 };
    double       zrelax[3] = { 0.8, 0.2, 0.1 };
};

// C[m0:m0+64, c0:c0+64] -= A[0:K, m0:m0+64]^T * B[0:K, c0:c0+64]; all
// operands row-major in the arena.  upper: only entries with (row <= col)
// in C's coordinates are written (diagonal tiles of symmetric blocks).
struct GemmTask
{
    std::int64_t a, b, c;          // arena offsets of A[0][0], B[0][0], C[0][0]
    std::int32_t lda, ldb, ldc;
    std::int32_t K, M, N;
    std::int32_t m0, c0;
    std::int32_t upper;
    std::int32_t pad;
};

// Panel [r0, r0+nb) of a front.  As a potrf task: factor the diagonal block
// in place.  As a trsm task: solve the panel's rows for the (up to kRestChunk)
// rest columns from c0 on, to the end of U0's or of U1's, against the factored block: rest column j is U0
// column r0+nb+j when j < n0-r0-nb, else U1 column j-(n0-r0-nb).  row0 is
// the front's first global row (failures report the failing global row);
// bit r of single_rows marks panel rows that form a 1 x 1 reference
// supernode, whose pivot is taken as sqrt(|a|) (Multifrontal.hpp:471).
struct PanelTask
{
    std::int64_t u0, u1;
    std::int32_t n0, n1;
    std::int32_t ld0, ld1;         // leading dimensions of U0 / U1
    std::int32_t r0, c0;
    std::int32_t row0;
    std::int32_t panel;            // index of the panel (its potrf task, SolveDiagTask and inverse block)
    std::int64_t single_rows;      // bit r set: panel row r is a 1 x 1 reference supernode
    std::int64_t img;              // FP32 path: the front's first operand-image block (see TcTask)
    std::int32_t img_t0, img_tf;   // its U0 column tiles, and U0 + U1 column tiles per k-chunk segment
    std::int32_t pend;             // potrf, FP64 level launches: rows r0 - pend .. r0 - 1 whose update of the diagonal
                                   // block the potrf applies itself (the other launches have a GEMM tile for it)
    std::int32_t pad;
};

// The FP32 path's Schur-complement tiles on the 5th-generation tensor cores
// read their operands from an *operand image*: every panel row of a front,
// once its trsm is done, split into TF32 hi and lo parts (x = hi + lo) and
// stored transposed in blocks of kImgRows U columns x kImgK U rows (row-major
// inside the block: the 32 k values of one U column are 128 contiguous bytes,
// one 128-byte-swizzled row of a K-major tensor-core operand).  Block
// (k-chunk kc, part hl, column tile ct) of front f is
//     img + (kc * 2 + hl) * tf + ct,
// where column tiles 0 .. t0-1 are U0 columns and t0 .. tf-1 are U1 columns
// (each 64-aligned), so every operand tile is a few whole blocks: one tensor
// map over the whole image serves every front.
constexpr int kImgRows = 64;
constexpr int kImgK    = 32;
constexpr int kTcM     = 128;     // tensor-core tile rows
constexpr int kTcNMax  = 256;     // widest tensor-core tile

// C[m0 : m0+kTcM, c0 : c0+nt] -= A^T B for K panel rows: A's columns are
// operand-image column tiles ta, ta+1 (the C rows), B's are tb .. tb+nt/64-1,
// over the k-chunks blk, blk + 2 tf, ... (hi; lo at + tf).  Rows >= M and
// columns >= N are not written; upper: only (row <= col) entries.
struct TcTask
{
    std::int64_t c;                // arena offset of C[0][0]
    std::int64_t blk;              // image block of (first k-chunk, hi, column tile 0)
    std::int32_t ldc, M, N;
    std::int32_t m0, c0;
    std::int32_t K;
    std::int32_t ta, tb, tf;
    std::int32_t nt;               // tile width: 64, 128, 192 or 256
    std::int32_t upper;
    std::int32_t pad;
};

// Add rows [row_begin, row_end) of child update W (m1 x m1, upper) into the
// parent front through lut (Multifrontal.hpp:324-436).
struct ExtendTask
{
    std::int64_t w, u0, u1, v;
    std::int64_t lut;              // offset into the lut array
    std::int32_t m1, mid;
    std::int32_t n0p, n1p;         // parent dimensions
    std::int32_t ldw;              // leading dimension of the child's W
    std::int32_t ld0p, ld1p, ldvp; // leading dimensions of the parent's U0 / U1 / V
    std::int32_t row_begin, row_end;
};

// Diagonal block of panel [r0, r0+nb) of a front whose first row is row0.
// Its inverse (kPanel x kPanel, row-major, identity-padded beyond nb) is
// block k of the inverse-diagonal buffer, k = the task's index.
struct SolveDiagTask
{
    std::int64_t u0;
    std::int32_t n0, r0, row0, ld0;
};

// One CTA of a solve step for panel [r0, r0+nb) of a front: rows [c0, c1)
// of the panel's rest (U0 rows below the panel, then the front's U1 columns,
// whose global rows come from SN_inner at offset inner), or c0 = -1, c1 = 0
// for a panel without rest rows.  The task with c0 <= 0 also applies the
// inverse diagonal block to the panel's own rows.  panel = index of the
// panel's SolveDiagTask.
struct SolveRestTask
{
    std::int64_t u0, u1, inner;
    std::int32_t n0, n1, r0, row0, c0, c1;
    std::int32_t ld0, ld1;
    std::int32_t panel, pad;
};

// Zero rows [row_begin, row_end) of the upper triangle of the n x n update
// matrix at arena offset `offset` (leading dimension ld): columns [r, n) of
// row r, `count` entries in all.  The strictly lower triangle is never read.
struct ZeroTask
{
    std::int64_t offset, count;
    std::int32_t n, ld, row_begin, row_end;
};

// Copy rows [r_begin, r_end) of reference supernode sn from its front into
// the reference layout: tri (n0s x n0s upper) and rec (n0s x n1s) blocks.
struct ExportTask
{
    std::int64_t fu0, fu1;         // front U0 / U1 arena offsets
    std::int64_t tri, rec;         // destination offsets (tri region / rec region)
    std::int64_t colmap;           // offset into colmap (== SN_outer[sn])
    std::int32_t fn0, fn1;         // front dimensions
    std::int32_t fld0, fld1;       // front leading dimensions
    std::int32_t roff;             // first row of sn within the front
    std::int32_t n0s, n1s;         // supernode dimensions
    std::int32_t r_begin, r_end;
    std::int32_t pad;
};

// One task of the factorization's task graph, executed by one CTA of the
// persistent factorization kernel: `index` into the task array of `kind`.
// Before it runs, counter wait[i] must have reached target[i] (unused
// waits: -1); when it is done it increments the counters signal[0..1]
// (-1: none).  The task list is in a topological order: every target is
// reached by tasks earlier in the list, which the plan check verifies.
constexpr int kDagWaits = 4;
constexpr int kDagMinSteps = 8;      // levels from the first with this many panel steps run as the task graph
constexpr int kSolveDagMinSteps = 4; // the same for the solves
constexpr int kDeferSteps = 3;       // panel steps over which a front's trailing update is deferred

struct DagTask
{
    std::int32_t kind, index;
    std::int32_t signal[2];
    std::int32_t wait[kDagWaits];
    std::int32_t target[kDagWaits];
};

enum class LaunchKind : std::int32_t { Zero = 0, Extend = 1, Trsm = 2, Gemm = 3, Invert = 4, Solve = 5, Potrf = 6,
                                       SuperInv = 8, SuperDiag = 9, SuperRest = 10, ExtendPull = 11, Front = 12 };

// Extend-add by parent rows (the level launches): one CTA adds, child by
// child in rank order, the rows of every child that map into one block of
// a parent's rows (pivot rows: U0 / U1; update rows: V).  The segments are
// ExtendTasks whose [row_begin, row_end) are those child rows.  Every parent
// entry receives the same additions in the same order as in the passes by
// child rank (the persistent schedule's extend tasks), in one launch per
// level instead of one per child rank.
struct ExtendPullTask
{
    std::int64_t seg_first;        // its segments in Plan::extend_segs
    std::int32_t seg_count;
    std::int32_t space;            // 0: pivot rows (U0 / U1), 1: update rows (V)
    std::int32_t b0, b1;           // its parent rows [b0, b1) in that space
};
constexpr std::int64_t kExtendPullEntries = 4096;    // target child entries per pull task

// A small front whole, in one CTA's shared memory: its assembled rows, the
// children's update matrices added in rank order, the panel factorization, the
// rest columns, and the update matrix written once (FrontTask, kernel
// front_kernel).  It replaces five launches (zero, extend-add, potrf, trsm,
// GEMM) and the passes over the front's entries between them.  Eligible: one
// panel of pivot rows, and everything in kFrontSmemMax; a level takes the
// kernel when at least half of its fronts are eligible (the others keep their
// launches, which cost about the same for a few fronts as for many).  Every
// front also has the separate tasks: those of the small ones come last in each
// launch's range (GEMM tiles: around the others'), so that the launches
// without them are ranges too.
struct FrontTask
{
    PanelTask    p;                // its only panel (r0 = 0)
    std::int64_t v;                // arena offset of its update matrix (leading dimension ld1); used when has_v
    std::int64_t seg_first;        // its children in rank order: ExtendTasks of all their rows in Plan::extend_segs
    std::int32_t seg_count;
    std::int32_t has_v;
};
constexpr std::int64_t kFrontSmemMax   = 220 * 1024;  // one CTA of 384 threads per SM
constexpr std::int64_t kFrontSmemMid   = 111 * 1024;  // two of 256 threads
constexpr std::int64_t kFrontSmemSmall = 74 * 1024;   // three of 128 threads
// Up to kFrontFew fronts (the chip's 148 SMs: every CTA is resident whatever its shared memory) a
// level's small fronts are one launch (fronts of 48 and 8 rows with 130 rest rows, 120 of them: 24 us
// against 36 in two launches).  From kFrontMany on, fronts that fit kFrontSmemSmall run with 128 threads,
// three CTAs an SM, where a whole level's throughput counts: 2,000 fronts of 24 rows and 60 rest rows
// 70 -> 59 us, 4,000 134 -> 115; 60 to 200 of them take 12 to 15 us with 256 threads and 14 to 15 with 128.
// (The two cross at about 300 fronts, 20.5 and 16.3 us; below 2,000 the level is a few us either way.)
constexpr std::int32_t kFrontFew = 148, kFrontMany = 2000;
// A front taken whole adds its children in one CTA, where the extend-add by
// parent rows spreads a wide parent's rows over the chip.  A front of more than
// kFrontWide rows in all whose children's update matrices have more than
// kFrontChildEntries entries together is wide-parented; a level keeps the
// launches for these fronts when it has fewer than kFrontSpread of them.
// Measured on groups of 3-row leaves under fronts of 8 rows and 200 rest rows,
// whole and apart: 3 such fronts with 65k entries of children 134 and 136 us,
// 130k 170 and 157, 347k 281 and 198, 1391k 790 and 404; 12 fronts with 347k
// each 309 and 256; 40 fronts with 347k each 470 and 563.  Fronts of up to 80
// rows are as fast whole with any number of children (25 rows, 2048 children:
// 1.3 and 2.7 ms; 64 rows, 64 children: 244 and 264 us).
constexpr std::int64_t kFrontChildEntries = 65536;
constexpr std::int32_t kFrontWide = 80, kFrontSpread = 32;

// Shared memory of front_kernel in doubles: the front's rows (diagonal block
// and rest columns, each rounded up to 8), the block's inverse, the update
// matrix by 8-row blocks from the diagonal on, the pivot floors and flags.
constexpr std::int64_t front_round8( std::int64_t x ) { return (x + 7) / 8 * 8; }
constexpr std::int64_t front_smem_bytes( std::int64_t n0, std::int64_t n1 )
{
    const std::int64_t a = front_round8( n0 ), b = front_round8( n1 );
    return 8 * (a * (a + b + 4) + a * (a + 4) + 4 * b * (b / 8 + 1) + kPanel + 2);
}

// Solve steps of fronts of at most kTinyRows rows and kTinyRest rest rows run a warp each, the
// others a CTA each.  A warp walks its rest rows eight at a
// time: with 32 or 64 of them it is slower than a CTA (C2 1.11 ms at 16, 1.12 at 32, 1.16 at 64;
// 56^3 with 64 right-hand sides 1.89, 1.94, 2.05), and so it is with up to 32 pivot rows (C2 1.55).
constexpr int kTinyRows = 8;
constexpr int kTinyRest = 16;

// The solve of a large front steps through its pivot rows 512 at a time
// (super-panels) instead of 64 at a time: the inverse of each 512 x 512
// diagonal block of U0 (T, FP64, upper triangular, row-major, built from
// the 64-row panel inverses after the factorization by doubling) turns eight
// sequential panel steps into one.  A level uses super-panels for every front of
// more than one panel when its largest front has at least kSuperMinRows pivot
// rows: it then runs two launches a super-panel step (its one-panel fronts in the
// first) where the panel steps of its fronts below that size alone took up to
// four (56^3 grid, 64 right-hand sides: 3.15 -> 2.93 ms; 40^3 grid: 354 -> 299
// us, with the one-panel fronts still in a launch of their own).  Lower lines
// cost more inverses than they save steps (the largest front at 193 rows:
// 131^2 mesh factor 394 -> 418 us, solve 90 -> 78 us).
constexpr int kSuperPanels  = 8;
constexpr int kSuperRows    = kSuperPanels * kPanel;   // 512
constexpr int kSuperMinRows = 256;

struct SuperPanel
{
    std::int64_t u0, u1, inner;    // the front's U0 / U1 arena offsets and its SN_inner offset
    std::int64_t t;                // offset of the inverse (ldt x ldt doubles, row-major)
    std::int32_t n0, n1, ld0, ld1;
    std::int32_t r0, rows;         // first pivot row of the block (a multiple of 512) and its row count
    std::int32_t row0;             // the front's first global row
    std::int32_t panel[kSuperPanels];   // inverse-block index of each 64-row panel (-1 beyond rows)
    std::int32_t ldt;              // the inverse's edge: rows rounded up to 64
    std::int32_t guard, pad;       // a front below kSuperMinRows: its solves use the inverse only where kGuardGrowth allows
};

// Guarded super-panels.  A product with the inverse of a whole block has a
// residual that grows with the block's condition number, panel by panel steps
// only with that of one panel.  Fronts below kSuperMinRows, which step by
// super-panels only because a larger front of their level does, keep the panel
// steps' residual: when a row's pivot is less than 1 / kGuardGrowth of its
// diagonal entry as the block's elimination starts (the sum over a column of
// U's squares against its diagonal entry's), the block's diag step goes panel
// by panel in one CTA.  Restated in FP64 over dense blocks of 80 to 255 rows,
// the inverse's residual is at most 2.5 times the panel steps' above the line;
// with rows within 1e-4 (squared) of each other it is 90 times, within 1e-8
// 10,000 times.  Scalar and 3-dof grid Laplacians have 0.2 and more in every
// front of 65 to 255 rows (median 0.75).
constexpr double kGuardGrowth = 8.0;
constexpr int    kGuardBlocks = 4;                     // 64-row blocks of a guarded super-panel

// Block (i, j) of a super-panel's inverse T, formed by doubling: with the
// inverses of two adjacent diagonal blocks of 2^s panels known, the block
// between them is -T_1 U_12 T_2, for s = 0, 1, 2 two launches of 64 x 64 block
// products each: W_ij = sum_{k=mid..j} U_ik T_kj (kept at block (j, i), which the
// solves never read), then T_ij = -sum_{k=i..mid-1} T_ik W_kj.  mid: the first
// panel of the second diagonal block; i == j: panel i's inverse is copied (in
// the first launch).  Against block back substitution by distance from the
// diagonal (a 64-row inverse on the left of every product), restated in FP64
// at 512 rows: a solve's residual is the same on a grid Laplacian's separator,
// 1.3 times on a dense matrix of condition 1e10, and 0.5 to 3 times with rows
// within 1e-8 (squared) of each other.
struct SuperInvTask
{
    std::int32_t sp, i, j, mid;
};

// A super-panel solve task.  Diag: the pair (blk, c0) of 64-row blocks, one
// term of the block's solution x_blk = sum_{i<=blk} T_{i,blk}^T y_i (forward,
// i = c0 <= blk) or sum_{j>=blk} T_{blk,j} (y_j + z_j) (back, j = c0 >= blk).
// Rest: block blk and rest rows [c0, c1) of the front after the super-panel
// (U0 rows, then its U1 columns): forward y_rest -= U_{blk,rest}^T x_blk; back
// z_blk -= U_{blk,rest} x_rest.
struct SuperSolveTask
{
    std::int32_t sp, blk, c0, c1;
};

// One launch: `count` tasks starting at `first` in the array of its kind.
// A panel step's GEMM tiles come as up to three launches: part 0 updates the
// next panel's rows (the next potrf / trsm wait for it; in the FP64 level
// launches without the diagonal block, which the potrf updates itself, so that
// only the trsm waits and the potrf runs beside it); part 1 the rows of the
// panels after it up to the next full update, whose steps' part 0 (and, FP64,
// potrf) wait for it;
// part 2 the rest of the trailing matrix and the update matrices, which only
// the next full update and the level's end wait for, so that it overlaps
// defer_steps panel steps.  (128-row tensor-core tiles may reach a part's rows
// early: a tile belongs to the part of its first row.)
struct Launch
{
    LaunchKind   kind;
    std::int32_t count;
    std::int64_t first;
    std::int32_t level;
    std::int32_t step;
    std::int32_t part = 0;
    // Gemm launches, FP32 path: the first small_count tiles belong to fronts
    // without an operand image (64 x 64 tiles); the updates of the other
    // tiles are the tensor-core tiles [tc_first, tc_first + tc_count)
    std::int64_t tc_first = 0;
    std::int32_t tc_count = 0;
    std::int32_t small_count = 0;
    // Solve launches: the last small_count tasks are tiny fronts (kTinyRows), a warp each
    // Front launches: small_count = the launch's shared memory in bytes, tc_count = its threads; part 1: other
    // fronts of the level keep their launches (the two may run side by side)
    // ExtendPull launches: the level's extend tasks in pass order are
    // [tc_first, tc_first + tc_count) of Plan::extend (what the persistent
    // schedule runs instead)
};

struct Plan
{
    Relaxation relax;
    std::int32_t defer_steps = kDeferSteps;   // panel steps over which a front's trailing update is deferred (1-4)
    std::int32_t tc_nmax = kTcNMax;           // widest tensor-core tile of the FP32 path (128 or 256)
    std::int32_t threads = 0;                 // host threads of the build and the check (<= 0: every hardware thread)

    // fronts: runs [sn_first, sn_last] of reference supernodes
    std::int32_t front_count = 0;
    std::vector<std::int32_t> front_sn_first, front_sn_last;
    std::vector<std::int32_t> front_row0, front_n0, front_n1;
    std::vector<std::int64_t> front_cols;      // offset of the column set in SN_inner
    std::vector<std::int32_t> front_parent;    // front_count = root
    std::vector<std::int32_t> front_of_sn;

    // arena layout (doubles): [U0 of all fronts][U1 of all fronts][update region];
    // rows are padded to a multiple of kLdAlign entries so every row of every
    // block starts on a 32-byte boundary
    std::int64_t u0_size = 0, u1_size = 0, v_size = 0;
    std::vector<std::int64_t> front_u0, front_u1, front_v;   // arena offsets
    std::vector<std::int32_t> front_ld0, front_ld1;          // U0 / U1 leading dimensions (V uses ld1)

    std::int32_t levels = 0;
    std::vector<std::int32_t> level_of;     // per front

    // extend-add lookup: lut[front_lut[t] + i] = position of column i of front
    // t in its parent (row of U0 when < mid, else position in the parent's
    // column set)
    std::vector<std::int32_t> lut;
    std::vector<std::int64_t> front_lut;

    // assembly map over the upper triangle of the permuted matrix
    std::vector<std::int64_t> asm_src;      // index into the caller's value array
    std::vector<std::int64_t> asm_dst;      // arena offset, | kDiagFlag on the diagonal

    // export to the reference layout: colmap[SN_outer[s] + l] = U0 column
    // (>= 0) or -(U1 column + 1) of column l of supernode s within its front
    std::vector<std::int32_t> colmap;
    std::vector<ExportTask>   exports;
    std::vector<std::int64_t> diag_offset;  // per row: arena offset of U(i,i)

    std::vector<GemmTask>      gemm;
    std::vector<TcTask>        tc;             // the GEMM updates as tensor-core tiles (FP32 path, level launches)
    std::vector<std::int64_t>  front_img;      // per front: first operand-image block
    std::int64_t img_blocks = 0;               // operand-image size in blocks of kImgRows x kImgK floats
    std::vector<PanelTask>     potrf;          // one per (front, panel)
    std::vector<PanelTask>     panel;          // trsm chunks
    std::vector<ExtendTask>    extend;
    std::vector<ZeroTask>      zero;
    std::vector<SolveDiagTask> sdiag;          // one per (front, panel); also the inverse-block list
    std::vector<SolveRestTask> srest;          // solve-step tasks, owner first per panel

    std::vector<Launch> factor_launches;    // in order, every front by the launches of its tasks' kinds
    std::vector<Launch> whole_launches;     // FP64 level schedule: the same with the small fronts taken whole (Front
                                            // launches) and left out of the others.  The factor is the same bit for bit;
                                            // the FP32 path keeps factor_launches, as its tensor-core updates are rounded
                                            // in their own order
    std::vector<DagTask> dag;               // the levels from dag_split_level up as one dependency-ordered task list
    std::int32_t dag_counters = 0;
    std::int32_t dag_min_steps = kDagMinSteps;   // set before build(): 0 puts every level in the task graph
    std::int32_t dag_split_level = 0;       // first level in the task graph
    std::int32_t dag_first_panel = 0;       // first panel (sdiag index) of that level
    std::vector<Launch> pre_dag_launches;   // the levels below, as launches, then their inversions
    double dag_makespan_us = 0.0;           // simulated duration of the scheduled list (schedule.cpp)
    std::vector<Launch> lower_launches;     // forward solve U^T y = b
    std::vector<Launch> upper_launches;     // back solve U x = y

    // Super-panel solve (see SuperPanel): the launch lists with the large
    // fronts' panel steps replaced by super-panel steps (per level: the other
    // fronts' step launches, then per super-panel step a diag and a rest
    // launch); the inverses are formed by the launches of sinv_launches after
    // the factorization.  Empty lists: no front is large enough.
    bool use_super = true;                  // set before build(): false keeps every front on panel steps
    std::vector<SuperPanel> spanels;
    std::vector<SuperInvTask> sinv;
    std::vector<Launch> sinv_launches;
    std::vector<SuperSolveTask> ssolve;
    std::vector<ExtendPullTask> extend_pull;
    std::vector<FrontTask> fronts;             // the small fronts taken whole, by level
    std::vector<char> front_small;             // per front: taken whole (FP64 level schedule)
    std::vector<ExtendTask> extend_segs;
    std::vector<Launch> lower_launches_sp, upper_launches_sp;
    std::int64_t super_inv_size = 0;        // doubles of all inverses

    // Solve task graph: the levels from solve_split_level up run as one
    // persistent launch per sweep, the levels below as the launches above.
    // A graph task is an srest task; its targets are the panels its rest
    // rows belong to (panel ids relative to solve_first_panel).  Forward:
    // a panel's tasks start once the solve_fwd_expected[p] graph tasks that
    // target it have applied their updates; each task signals its targets.
    // Back: a task starts once every target panel has all of its
    // solve_panel_tasks tasks done; each task signals its own panel.
    std::int32_t solve_split_level = 0;
    std::int32_t solve_default_split = 0;         // first level with kSolveDagMinSteps or more panel steps
    std::int32_t solve_first_panel = 0;
    std::int64_t solve_first_task = 0;
    std::vector<std::int32_t> solve_fwd_order;    // srest indices of the graph in forward order
    std::vector<std::int32_t> solve_bwd_order;    // the same in back-sweep order
    std::vector<std::int64_t> solve_target_ptr;   // per graph task (srest index - solve_first_task), + 1
    std::vector<std::int32_t> solve_targets;
    std::vector<std::int32_t> solve_fwd_expected; // per graph panel
    std::vector<std::int32_t> solve_panel_tasks;  // per graph panel

    double gemm_flops = 0.0;                // useful flops of all GEMM tiles (upper part of diagonal tiles)
    double gemm_tile_flops = 0.0;           // the flops the 64 x 64 tiles execute (full tiles, full depth)
    double factor_flops = 0.0;              // reference supernodes: Sum [n0^3/3 + n0^2 n1 + n0 n1^2]
    double front_flops  = 0.0;              // the same sum over fronts (work actually executed)
    double nnz_u = 0.0;                     // reference supernodes: Sum [n0(n0+1)/2 + n0 n1]
    double front_entries = 0.0;             // the same over fronts

    std::int64_t arena_size() const { return u0_size + u1_size + v_size; }

    void build( const Symbolic & sym );
    template<typename RangeOf, typename RangeCount>
    void build_super( const std::vector<std::vector<std::int32_t>> & front_panels, RangeOf range_of, RangeCount ranges,
                      const std::vector<std::vector<std::int32_t>> & by_level );
    // Fills the solve task graph for the levels from `split` up (levels: none).
    void build_solve_graph( const Symbolic & sym, std::int32_t split );
};

} // namespace tb
