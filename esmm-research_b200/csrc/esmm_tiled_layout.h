// Sizes and shared-memory layout of the tiled kernel (esmm_gemm_tiled.cuh) and of its block mode (esmm_gemm_blocks.cuh).
// Plain C++, so that the layout can be checked without a GPU.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define ESMM_HOST_DEVICE __host__ __device__
#else
#define ESMM_HOST_DEVICE
#endif

namespace esmm {

constexpr int TILE_M = 128;
constexpr int TILE_N = 128;
constexpr int SMEM_LIMIT = 232448; // 227 KB per CTA on sm_100

// ---- the pipeline ----
constexpr int ROW_BYTES = TILE_N * 4;            // 512: one k of an operand tile
constexpr int ROWS_PER_STAGE = 32;
constexpr int STAGE_HALF_BYTES = ROWS_PER_STAGE * ROW_BYTES;   // 16384: A rows, then B rows
constexpr int PSTAGE_BYTES = 2 * STAGE_HALF_BYTES;             // 32768
// Row-major A: the rows of A in a stage are 16 bytes further apart, so that the producers' 4-byte copies of eight k of four rows of
// A fall on all 32 banks.  (At 512 or 256 bytes they all fall on four, and every copied sector takes eight passes: 4096^3 dense 2621
// us, 2387 with the rows apart.)
ESMM_HOST_DEVICE constexpr int stage_a_row(int wmb, bool row_major) { return 256 * wmb + (row_major ? 16 : 0); }
constexpr int RM_STAGE_A_BYTES = ROWS_PER_STAGE * stage_a_row(2, true);   // 16896; B's rows after them start on 128 bytes, as the copy engine needs
static_assert(RM_STAGE_A_BYTES % 128 == 0, "B's rows in a stage");
constexpr int P_CONSUMER_WARPS = 8;
constexpr int P_MAX_STAGES = 6;

// ---- block mode ----
constexpr int BM_WARPS = 12;                                // warps of the CTA that take part
constexpr int BM_ROWS = 16;                                 // k per stage
constexpr int BM_STEP = 8;                                  // k multiplied as one run of straight-line code
constexpr int BM_PART = BM_ROWS * 128;                      // a stage's rows of one operand of one block
constexpr int BM_SLOT_BYTES = 4 * BM_PART;                  // X of block 0, X of block 1, Y of block 0, Y of block 1
constexpr int BM_SLOTS = 2;
constexpr int BM_LIST = 512;                                // entries of a block's list (a ring)
constexpr int BM_LIST_BYTES = BM_LIST * 2;
constexpr int BM_WARP_BYTES = BM_SLOTS * BM_SLOT_BYTES + 2 * BM_LIST_BYTES;
constexpr int BM_SMEM = BM_WARPS * BM_WARP_BYTES;           // the warps' rings and lists, from the start of shared memory

// Whether block mode pays, from samples of the patterns: work of the slots (32 x 32 block, k) that the pipeline would hold in shared
// memory are multiplied.  Samples without any live k say nothing about the rest of the operands: the pipeline then, whose worst
// case is the smaller one (4096^3: dense operands in block mode 2549 us instead of 2130; operands for block mode in the pipeline
// 308 instead of 167, of which a sample without a live k is no sign).
ESMM_HOST_DEVICE inline bool block_mode_pays(int work, int slots, int sixteenths)
{
    return slots > 0 && 16 * work <= sixteenths * slots;
}

// How many of a CTA's items (pairs of blocks) go as two single blocks each, at the end.  Up to 6 all of them: twelve warps then have a
// block or none, and a warp alone takes longer for a pair than three do for their blocks beside each other (1000 x 1508 x 2012 at 0.5 / 0.5, 5 or 6
// items, four pairs and the rest single 55.2 us, all single 49.9).  Up to 12 what is over when every scheduler (SM sub-partition) has as many
// pairs as every other (7 and 8 items as 2 and 4 pairs and 10 and 8 single blocks: 1500^3 at 0.5 / 0.5 50.1 -> 53.2, 512 x 4096 x 4096 pruned
// MLP 107.4 -> 108.6).  Then the end of a row of rounds: six, which are a round of single blocks, up to 24 items and where 5 or 6 are over
// after whole rounds; four elsewhere.  Whole calls, 4 / 6, 32-granular 0.5 / 0.5, 2048 x N x 1024, by items per CTA: 17.7 78.0 / 69.6 us, 29.8
// 113.9 / 106.6 (row-major A 173.8 / 163.6), 42 154.5 / 149.6, 53.6 191.4 / 187.1; 32 119.0 / 120.6, 45 158.9 / 160.7; 3000 x 3000 x 1000 at
// 0.7 / 0.7 (29.9) 207 / 190; 4096^3 64-granular (55.4) 652 / 662.  (Two are as good or better with 8 to 12 over, eight nowhere.)
ESMM_HOST_DEVICE inline int block_tail(int mine)
{
    if (mine <= 6) return mine;
    if (mine <= BM_WARPS) return (mine & 3) % 3;
    const int over = mine % BM_WARPS;
    return mine <= 2 * BM_WARPS || over == 5 || over == 6 ? 6 : 4;
}

// Row-major A: problems for which block_mode_pays has the pipeline as the faster one all the same, at shares above a quarter.  listed: k that
// are live for a sample's tile; span: k looked at; rows64: live (64-row half of a tile, column block, k); shape: RmShape of the problem.
//   * Row blocks that agree in pairs (work is twice rows64), so that the pipeline's warps, 64 rows each, waste nothing, and few k listed: an
//     item's start and end then outweigh its stages in block mode.  Whole call, pipeline / block mode, 64-granular 0.2 / 0.2 (0.13 listed)
//     4096^3 270 / 300 us, 2048^3 55 / 57, 1024^2 x 4096 32 / 39; but 0.1 / 0.1 (0.04) 2048^3 42 / 34, and 0.3 / 0.3 (0.26) 2048 x 11008 x 4096
//     589 / 537, while with at most six pairs of blocks per SM, single blocks all, 1024^2 x 4096 47 / 54 and 1100 x 700 x 12000 at 0.2 / 0.2
//     88 / 98.  Of more pairs not at ragged edges, which cost the pipeline more: 3000 x 3000 x 1000 at 0.2 / 0.2 98 / 66.
//   * Most k listed and more than 7/16 of them used, where the tiles come out even (a last round nearly full) or the blocks do not (seven
//     or eight pairs for twelve warps): 32-granular 0.7 / 0.7 4096^3 1798 / 1830, 3000 x 3000 x 1000 279 / 289, 512 x 4096 x 4096 285 / 314;
//     not so 2048^3 (0.86 of two rounds) 279 / 253.
// Neither where fewer than seven SMs of ten have a tile (64 x 4096 x 4096 at 1 / 0.4 149 / 85; 1000 x 1508 x 2012, 96 tiles, at 0.3 / 0.3 49 / 45).
enum RmShape { RM_FILLS = 1, RM_WHOLE = 2, RM_FEW = 4, RM_EVEN = 8 };

ESMM_HOST_DEVICE inline bool row_major_pipeline_pays(int work, int slots, int rows64, int listed, int span, int shape)
{
    if (!(shape & RM_FILLS) || 4 * work <= slots) return false;
    const bool short_lists = (shape & (RM_WHOLE | RM_FEW)) && 10 * work >= 19 * rows64 && 12 * listed >= span && ((shape & RM_FEW) ? 3 : 6) * listed <= span;
    return short_lists || (16 * work > 7 * slots && 4 * listed >= 3 * span && (shape & RM_EVEN));
}

inline int row_major_shape(int M, int N, long tiles, long pairs, int sms)
{
    const long rounds = (tiles + sms - 1) / sms;
    const bool even = 20 * tiles >= 19 * rounds * sms || (pairs > 6l * sms && pairs <= 8l * sms);
    return (10 * tiles >= 7l * sms ? RM_FILLS : 0) | (M % 64 == 0 && N % 64 == 0 ? RM_WHOLE : 0) | (pairs <= 6l * sms ? RM_FEW : 0) | (even ? RM_EVEN : 0);
}

struct PackedSmem {
    uint32_t stage_off, krow_off, krow_stride, rmask_off, rmask_stride, wlist_off, bar_off, misc_off, total;
};

// blocks: the kernel has block mode.
ESMM_HOST_DEVICE inline PackedSmem packed_smem_layout(int stages, int stage_bytes, int cap, bool blocks)
{
    PackedSmem L;
    uint32_t o = 0;
    L.stage_off = o;
    o += (uint32_t)stages * stage_bytes;
    L.krow_off = o;   // two buffers: k index of every listed row
    L.krow_stride = (uint32_t)cap * 2;
    o += 2 * L.krow_stride;
    L.rmask_off = o;  // two buffers: per row, bits 0-3 live row blocks, bits 4-7 live column blocks
    L.rmask_stride = (uint32_t)cap;
    o += 2 * L.rmask_stride;
    o = (o + 15u) & ~15u;
    L.wlist_off = o;  // per consumer warp: offsets of the live rows of its top and its bottom block
    o += P_CONSUMER_WARPS * 2 * 96;  // two lists of WLIST_BYTES per warp
    // Block mode lays its warps' rings over what is above, and over nothing below: the barriers' memory holds live mbarriers
    // (which have to be invalidated before their memory may serve another use), and its item counter is in misc.
    if (blocks && o < (uint32_t)BM_SMEM) o = BM_SMEM;
    L.bar_off = o;    // full[P_MAX_STAGES], empty[P_MAX_STAGES], list_full[2], list_empty[2]
    o += (2 * P_MAX_STAGES + 4) * 8;
    L.misc_off = o;   // nrows[2], abort, n_producers, runinfo[2], next item
    o += 32;
    L.total = o;
    return L;
}

}  // namespace esmm
