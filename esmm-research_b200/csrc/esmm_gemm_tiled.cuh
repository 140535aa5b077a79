// Joint-sparse FP32 SGEMM for sm_100a: the tiled kernel, on the packed (k-major) copy of A (esmm_gemm_packed.cu) or on row-major A
// (esmm_gemm_rowmajor.cu).
//
// Same arithmetic as esmm_ab_optimized_v3 of the reference
// (src/kernels/esmm_ab_optimized_v3.cu:18-235): for every output one FFMA chain in ascending
// k over the k whose joint bit (A pattern of its 32-row block AND B pattern of its 32-column
// block) is set; C is overwritten.  What differs is where the skipping happens.
//
// A comes from the packing preprocessor as [128-row tile][k][128 rows]; B is the caller's
// row-major matrix, i.e. [k][N].  So one k of a 128 x 128 tile of C needs one 512-byte row
// of each operand, and the pipeline moves exactly such rows:
//
//   * a mask warp walks the tile's K blocks one tile ahead and appends, for every K block,
//     the k rows that are live for the tile as a whole (the OR over its four 32-row blocks
//     AND the OR over its four 32-column blocks) to a row list, with one byte per row saying
//     for which row blocks and which column blocks the row is live.  On a tile whose K
//     blocks do not all share one live byte, K blocks with more than `brow_bits` live k are
//     appended whole (8 rows), so that they can be fetched as one box;
//   * three producer warps cut the row list into stages of 32 rows and fetch each stage's rows into
//     a ring slot ([32][512 B] of A, [32][512 B] of B), guarded by full / empty mbarriers.
//     Both operands are also described to the copy engine as 3-D tensors (column, k % 8,
//     k / 8), so a stage whose rows are "the same c consecutive k offsets of 32 / c
//     consecutive K blocks" (c = 1, 2, 4, 8: what uniform patterns such as 10000000,
//     11000000, 11110000 and 11111111 produce) is ONE box per operand, landing in ascending
//     k.  Other stages: the list is ascending, and rows with consecutive k are consecutive rows
//     of both operands, so every run of them goes as boxes of 8, 4, 2 and 1 rows, issued by the
//     lane at the box's first row, the boxes of a stage shared out among the producer warps (a
//     copy costs its warp about 50 cycles of issue, and warps issue in parallel).  A k that is
//     dead for the whole tile costs neither a copy nor shared memory nor a slot in any loop;
//   * a tile all of whose K blocks hold the same run of 1, 2, 4 or 8 consecutive live k, live for all
//     of its row and column blocks (what uniform patterns, and dense inputs, give), needs no row
//     list at all: its stages are computed arithmetically and are all-live;
//   * where 128 x 128 tiles would leave most of the GPU idle (small M x N), the same kernel runs
//     with 64 x 128 tiles: a 64-row tile reads the left or right half of a 128-row panel of A, a
//     consumer warp owns 32 x 32 outputs;
//   * 8 consumer warps own 64 rows x 32 columns of the tile each (two A pattern rows, one B
//     pattern row; a thread holds 8 x 8 outputs, 4 rows in each 32-row block).  Per stage a
//     warp forms its two 32-bit joint masks with two ballots.  If every row of the stage is
//     live for both row blocks - always the case for uniform patterns, at any density - it
//     runs straight-line code (4 sixteen-byte loads and 32 two-wide FMAs per k).  Otherwise it
//     walks the set bits of its masks, loading the next live row under the multiply-adds of
//     the current one.
//
// Lanes are laid out so that every group of 4 consecutive lanes touches 2 row chunks x 2
// column chunks: on this GPU a 16-byte shared load costs 2 wavefronts when each such group
// reads at most 32 distinct bytes and 4 otherwise.
//
// Every wait is bounded; a wait that expires raises the device status word and the CTA
// leaves after waiting (bounded again) for its copies in flight.
#pragma once

#include "esmm_gemm_blocks.cuh"

namespace esmm {

// Issuing a copy costs the issuing warp about 50 cycles per copy, whatever the mechanism (2-D tensor copy of one row
// or of an 8-row box, untiled bulk copy, or a warp-wide 16-byte cp.async per row: 3300 cycles for the 64 copies of a
// row-by-row stage from one warp, 1270 from three, 970 from four - measured), and different warps issue in parallel.
// So the rows of a stage are shared out among several producer warps.
//   3 producer warps: 8 consumer + 3 producer + 1 mask warp = 12 warps, 3 per SM sub-partition, every thread with
//     the 168 registers a 384-thread CTA allows (the consumers need about 150).
//   7 producer warps: 16 warps.  A 512-thread CTA starts with 128 registers per thread; the two warp groups of
//     consumers raise their allowance to 160 and the two warp groups of producers / mask warp lower theirs to 96
//     (setmaxnreg).  Each CTA's first tile decides whether all 7 copy (tiles of scattered single rows with little
//     work per consumer warp: a stage is then posted every 0.92 us instead of 1.19) or 3 do and 4 sleep.  Measured
//     against the 12-warp form: 512 x 1024 x 704, 32-granular patterns at 0.2 / 0.2 16.4 -> 14.4 us (larger operands of
//     this kind take block mode), but dense and uniform patterns 0.5 % slower.  A launch takes this form when the launch before it on the device
//     noted such tiles (see gemm_ab_packed_launch_form); esmm_tuning_set("PRODUCER_WARPS", 3 | 7 | 0) pins one.
constexpr int P_TMA_WARP = P_CONSUMER_WARPS;                   // first producer warp
// Block mode (esmm_gemm_blocks.cuh) where at most this many sixteenths of what the tiled pipeline would hold in shared memory are
// multiplied.  Measured at 4096^3, whole calls, pipeline / block mode: share 0.33 (32-granular, 0.5 / 0.5 of A's and B's
// k live) 921 / 718 us, 0.44 (64-granular, 0.5 / 0.5) 730 / 695, 0.53 (32-granular, 1 / 0.5) 1414 / 1344, 0.64 (32-granular,
// 0.8 / 0.8) 1900 / 1737, 0.67 (64-granular, 1 / 0.5) 1373 / 1346, 0.69 (64-granular, 0.8 / 0.8) 1675 / 1685, 0.83 (64-granular,
// 0.9 / 0.9) 2050 / 2087, 1 (dense) 2130 / 2549.
constexpr int BM_SIXTEENTHS = 11;
// The same for row-major A, where block mode has to transpose A for every pair of blocks: kernel alone, pipeline / block mode, share 0.11
// (32-granular, 0.2 / 0.2) 2048^3 79 / 64 us; pruned MLP (0.31) 2048 x 11008 x 4096 1267 / 827, 64 x 4096 x 4096 77 / 54; share 0.33
// (0.5 / 0.5) 2048^3 186 / 151, 1000 x 1508 x 2012 98 / 67; share 0.44 (64-granular, 0.5 / 0.5) 2048^3 142 / 140, 4096^3 882 / 811; share 0.50
// (32-granular, 0.7 / 0.7) 2048^3 281 / 252, 4096^3 1828 / 1833; share 0.53 (1 / 0.5) 257 / 265, 1683 / 1772.  Some problems above a
// quarter stay with the pipeline all the same: row_major_pipeline_pays.
constexpr int RM_SIXTEENTHS = 8;

// Optional timeline for tuning (build with -DESMM_TRACE): CTA 0 stamps %globaltimer at a few points
// into a device array that esmm_trace_read copies out.  Not part of the product build or of the ABI.
#ifdef ESMM_TRACE
static __device__ unsigned long long g_esmm_trace[1024];
#define ESMM_STAMP(idx)                                                                   \
    do {                                                                                  \
        if (blockIdx.x == 0 && lane == 0 && (idx) < 1024) g_esmm_trace[(idx)] = global_timer_ns(); \
    } while (0)
#else
#define ESMM_STAMP(idx) \
    do {                \
    } while (0)
#endif

struct PackedParams {
    int M, N, K;
    int nKB;         // ceil(K / 8)
    int kp;          // rows of the packed A matrix per 128-row tile (nKB * 8)
    int cap;         // capacity of a tile's row list (multiple of 32)
    int a_rows;      // rows of the A pattern array (ceil(M / 32))
    int b_rows;      // rows of the B pattern array (ceil(N / 32))
    int tiles_m, tiles_n, num_tiles;
    int group_m;     // tile rows per raster group
    int stages;
    int brow_bits;   // K blocks with more live k than this are fetched whole
    int row_density; // ... on tiles with at most this many live k per K block on average; denser tiles
                     // fetch every live K block whole
    int b_runs_ok;   // K % 8 == 0: the 3-D view of B stays inside the matrix
    int force_listed;  // tuning aid: take the index-list path even for all-live stages
    int no_run_tiles;  // tuning aid: build the row list even for tiles that need none
    int vec_patterns;  // K blocks per lane and load in the mask warp: 16, 4 (alignment permitting) or 0 = bytes
    int adaptive;      // 16-warp form: the CTA's first tile decides whether 3 or all 7 producer warps copy
    int *form_hint;    // host-mapped word, or null: CTA 0 notes whether its first tile wanted 7 producers ...
    int form_known;    // ... where that is not what the host read there
    int block_mode;    // 1, 0: always, never; -1: as the sampled tiles say
    int pat_words;     // pattern rows may be read as 32-bit words
    unsigned last_bits;  // of the last K block's byte: the bits whose k is < K, in all four bytes of the word
    int few_blocks;    // no more pairs of blocks than CTAs
    int rm_shape;      // row-major A: RmShape
    // row-major A: 32-row block mb uses A pattern rows (mb / a_div) * a_mul + [0, a_mul) of a_pat_rows
    int a_div, a_mul, a_pat_rows;
    int list_kb, lists;  // row-major A: K blocks per row list, row lists per tile
    const float *A;
    const uint8_t *a_pat;
    const uint8_t *b_pat;
    const float *a_packed;
    const float *B;
    float *C;
    int *status;
};

// Tensor maps of one launch.  *_box[i]: 2-D, 1 << i rows (1, 2, 4, 8) of 128 columns.  *_run[i]: 3-D
// (column, k % 8, k / 8) boxes of 128 x c x 32/c with c = 1 << i.
struct PackedMaps {
    CUtensorMap a_box[4], a_run[4];
    CUtensorMap b_box[4], b_run[4];
};

constexpr int RUN_TILE = 0x100;
constexpr int RUNS_LIKELY = 0x200;   // a listed tile whose stages may be whole runs of K blocks: the producers look for them

// A stage whose 32 rows are all live for both row blocks: 16 rows of straight-line code per
// loop trip (measured: 4 rows 1 % slower than 8, 16 rows 1.6 % faster, 32 no better than 16),
// so that the compiler can issue the loads of a row under the multiply-adds of the row before.
// RM: row-major A, whose rows in a stage are 16 bytes further apart (see esmm_tiled_layout.h).
template <int WMB, bool RM>
__device__ __forceinline__ void dense_rows(Acc &acc, const char *sA, const char *sB)
{
    constexpr int A_ROW = stage_a_row(WMB, RM);   // bytes of one k of the A tile
    // (Measured and dropped: a rolling prefetch across the loop's back edge; a non-blocking look at the next stage's
    // barrier under the last multiply-adds of this one, so that the wait at the stage change is skipped - no gain.)
#ifndef ESMM_DENSE_UNROLL
#define ESMM_DENSE_UNROLL 16
#endif
#pragma unroll 1
    for (int r0 = 0; r0 < ROWS_PER_STAGE; r0 += ESMM_DENSE_UNROLL) {
#pragma unroll
        for (int r = 0; r < ESMM_DENSE_UNROLL; ++r) {
            const KFrag f = load_kfrag<WMB>(sA + (r0 + r) * A_ROW, sB + (r0 + r) * ROW_BYTES);
            fma_top(acc, f);
            if (WMB == 2) fma_bottom(acc, f);
        }
    }
}

// ---- stages that are not all-live ------------------------------------------------------------------
// When the warp's two 32-row blocks have the same live rows (jt == jb) every live row goes into all
// 8 x 8 outputs (mode BOTH): the set bits of the mask, a warp-uniform value, are walked in ascending
// order with find-first-set, one row loaded ahead under the 32 two-wide FMAs of the row before.
// Otherwise the top and the bottom block are processed one after the other (modes TOP, BOTTOM): each
// accumulator still sees its own live k in ascending order, no multiply-add is predicated, and the
// only price is that B rows live for both blocks are read from shared memory twice.  A row then
// feeds only 16 two-wide FMAs, too few to hide a find-first-set chain and a load behind: the lanes
// first write the rows' offsets as a list (in parallel, while the stage may still be in flight) and
// the loop takes two rows per step from it.  (Measured on random 32-granular patterns: one pass over
// jt | jb with warp-uniform branches per block is 20 % slower than the two passes, bit walking in
// the half modes 3-5 % slower than lists, lists in mode BOTH 4 % slower than bit walking, a switch
// per nibble of the mask into straight-line code 38 % slower.  For masks made of bytes 0x00 / 0xFF
// (block-pruned operands) a walk in groups of 8 rows with one three-way choice per group gained nothing
// on a pruned-MLP shape - there the spread of live rows between the 8 warps of a stage is what costs -
// and made the other paths 1-5 % slower; preparing masks and lists one stage ahead (two list buffers)
// was 2-5 % slower on every workload.)
enum { MODE_BOTH = 0, MODE_TOP = 1, MODE_BOTTOM = 2 };

// What stands for a row in masks' walks and in lists: the byte offset in the stage's B rows, or (RM) a 32nd of it, of which the
// offsets in either operand's rows are multiples.
template <bool RM>
constexpr int ROW_SHIFT = RM ? 4 : 9;

template <int MODE, int WMB, bool RM>
__device__ __forceinline__ KFrag load_entry(const char *sA, const char *sB, unsigned off)
{
    KFrag f;
    const unsigned a_off = RM ? off * (stage_a_row(WMB, true) / 16) : WMB == 2 ? off : off >> 1;   // A rows are 512 or 256 bytes apart
    if (RM) off *= ROW_BYTES / 16;
    if (MODE != MODE_BOTTOM) f.at = *reinterpret_cast<const float4 *>(sA + a_off);
    if (MODE != MODE_TOP) f.ab = *reinterpret_cast<const float4 *>(sA + a_off + 128);
    f.b0 = *reinterpret_cast<const float4 *>(sB + off);
    f.b1 = *reinterpret_cast<const float4 *>(sB + off + 64);
    return f;
}

template <int MODE>
__device__ __forceinline__ void fma_entry(Acc &acc, const KFrag &f)
{
    if (MODE != MODE_BOTTOM) fma_top(acc, f);
    if (MODE != MODE_TOP) fma_bottom(acc, f);
}

// the lowest live row of m, which is removed from m
template <bool RM>
__device__ __forceinline__ unsigned pop_row(unsigned &m)
{
    const unsigned r = (unsigned)__ffs((int)m) - 1u;
    m &= m - 1u;
    return r << ROW_SHIFT<RM>;
}

// (128-row tiling only: in the 64-row tiling every stage that is not all-live takes the list.)
template <bool RM>
__device__ __forceinline__ void masked_rows_both(Acc &acc, const char *sA, const char *sB, unsigned m)
{
    if (m == 0u) return;
    KFrag f0 = load_entry<MODE_BOTH, 2, RM>(sA, sB, pop_row<RM>(m)), f1;
#pragma unroll 1
    while (true) {
        if (m == 0u) {
            fma_entry<MODE_BOTH>(acc, f0);
            break;
        }
        f1 = load_entry<MODE_BOTH, 2, RM>(sA, sB, pop_row<RM>(m));
        fma_entry<MODE_BOTH>(acc, f0);
        if (m == 0u) {
            fma_entry<MODE_BOTH>(acc, f1);
            break;
        }
        f0 = load_entry<MODE_BOTH, 2, RM>(sA, sB, pop_row<RM>(m));
        fma_entry<MODE_BOTH>(acc, f1);
    }
}

// A list holds, ascending, an entry (row << ROW_SHIFT, 16 bits) for every row of the stage that is
// live for one of the warp's blocks, padded with 8 zero entries so that look-ahead loads need no
// bounds checks.
constexpr int WLIST_ENTRIES = ROWS_PER_STAGE + 8;
constexpr int WLIST_BYTES = 96;   // WLIST_ENTRIES * 2, rounded up to a multiple of 16
static_assert(WLIST_ENTRIES * 2 <= WLIST_BYTES, "per-warp list does not fit");

__device__ __forceinline__ unsigned entry_of(const uint2 &w, int j)
{
    const unsigned word = (j & 2) ? w.y : w.x;
    return (j & 1) ? (word >> 16) : (word & 0xFFFFu);
}

// Two rows per step, the next pair loaded before the current pair is multiplied.
template <int MODE, int WMB, bool RM>
__device__ __forceinline__ void listed_rows(Acc &acc, const char *sA, const char *sB, const uint16_t *list, int cnt)
{
    const int n4 = cnt & ~3;
    uint2 ew = *reinterpret_cast<const uint2 *>(list);   // entries 0..3
    KFrag f0 = load_entry<MODE, WMB, RM>(sA, sB, entry_of(ew, 0));
    KFrag f1 = load_entry<MODE, WMB, RM>(sA, sB, entry_of(ew, 1));
#pragma unroll 1
    for (int i = 0; i < n4; i += 4) {
        const KFrag g0 = load_entry<MODE, WMB, RM>(sA, sB, entry_of(ew, 2));
        const KFrag g1 = load_entry<MODE, WMB, RM>(sA, sB, entry_of(ew, 3));
        fma_entry<MODE>(acc, f0);
        fma_entry<MODE>(acc, f1);
        ew = *reinterpret_cast<const uint2 *>(list + i + 4);   // padded: always readable
        f0 = load_entry<MODE, WMB, RM>(sA, sB, entry_of(ew, 0));
        f1 = load_entry<MODE, WMB, RM>(sA, sB, entry_of(ew, 1));
        fma_entry<MODE>(acc, g0);
        fma_entry<MODE>(acc, g1);
    }
    // up to three rows are left; f0, f1 already hold the first two of them (or padding)
    const int rem = cnt - n4;
    if (rem >= 1) fma_entry<MODE>(acc, f0);
    if (rem >= 2) fma_entry<MODE>(acc, f1);
    if (rem == 3) fma_entry<MODE>(acc, load_entry<MODE, WMB, RM>(sA, sB, entry_of(ew, 2)));
}

// Lanes write the list of the rows whose bit is set in `m`; returns the count.
template <bool RM>
__device__ __forceinline__ int build_list(uint16_t *list, unsigned m, int lane, int *status)
{
    const int cnt = __popc(m);
    const int mine = __popc(m & ((1u << lane) - 1u));
    if (((m >> lane) & 1u) && bounds_ok(mine < WLIST_ENTRIES, status, 25)) list[mine] = (uint16_t)(lane << ROW_SHIFT<RM>);
    if (lane < 8 && bounds_ok(cnt + lane < WLIST_ENTRIES, status, 25)) list[cnt + lane] = 0;
    return cnt;
}

// ---- mask warp helpers ---------------------------------------------------------------------------
// (Row-major A: patterns come from the caller, who may have marked k past K live, in a dense product by 0xFF throughout.  Such k
// are dropped here: there is no element of A to multiply, and the clamped address holds A[row][K - 1].)
// Pattern bytes of KPL (16 or 4) consecutive K blocks kb0 .. kb0 + KPL - 1, all inside the matrix, for the
// tile's RB 32-row blocks and four 32-column blocks: one 16-byte or 4-byte load per pattern row.  aw[j] /
// bw[j] get the four bytes of K block kb0 + j (byte i = block i).  Long K takes 16 per lane; shorter K
// takes 4, so that all lanes have work.
template <int RB, int KPL, bool RM>
__device__ __forceinline__ void load_patterns(const PackedParams &p, int tm, int tn, int kb0, bool valid,
                                              unsigned (&aw)[KPL], unsigned (&bw)[KPL])
{
    constexpr int W = KPL / 4;   // 32-bit words per pattern row
    unsigned ra[4][W], rb[4][W];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int mb = tm * RB + i, nb = tn * 4 + i;
#pragma unroll
        for (int w = 0; w < W; ++w) ra[i][w] = rb[i][w] = 0u;
        const PatternRows pr = a_pattern<RM>(p, mb);
        if (valid && i < RB && pr.first && bounds_ok(kb0 >= 0 && kb0 + KPL <= p.nKB, p.status, 21)) {
            for (int j = 0; j < pr.count; ++j) {
                const uint8_t *src = pr.first + (size_t)j * p.nKB + kb0;
                if (KPL == 16) {
                    const uint4 v = *reinterpret_cast<const uint4 *>(src);
                    ra[i][0] |= v.x, ra[i][W > 1 ? 1 : 0] |= v.y, ra[i][W > 2 ? 2 : 0] |= v.z, ra[i][W > 3 ? 3 : 0] |= v.w;
                } else {
                    ra[i][0] |= *reinterpret_cast<const unsigned *>(src);
                }
            }
        }
        if (valid && nb < p.b_rows && bounds_ok(kb0 >= 0 && kb0 + KPL <= p.nKB, p.status, 21)) {
            const uint8_t *src = p.b_pat + (size_t)nb * p.nKB + kb0;
            if (KPL == 16) {
                const uint4 v = *reinterpret_cast<const uint4 *>(src);
                rb[i][0] = v.x, rb[i][W > 1 ? 1 : 0] = v.y, rb[i][W > 2 ? 2 : 0] = v.z, rb[i][W > 3 ? 3 : 0] = v.w;
            } else {
                rb[i][0] = *reinterpret_cast<const unsigned *>(src);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < KPL; ++j) {
        const int sh = 8 * (j & 3);
        unsigned a = 0, b = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            a |= ((ra[i][j >> 2] >> sh) & 0xFFu) << (8 * i);
            b |= ((rb[i][j >> 2] >> sh) & 0xFFu) << (8 * i);
        }
        aw[j] = a;
        bw[j] = b;
    }
    // (nKB is a multiple of KPL here, so the last K block is some lane's last)
    if (RM && kb0 + KPL == p.nKB) aw[KPL - 1] &= p.last_bits;
}

// k offsets of one K block that are live for the tile as a whole: (OR of the A bytes) & (OR of the B bytes)
__device__ __forceinline__ unsigned tile_live(unsigned aw, unsigned bw)
{
    unsigned au = aw | (aw >> 16), bu = bw | (bw >> 16);
    au = (au | (au >> 8)) & 0xFFu;
    bu = (bu | (bu >> 8)) & 0xFFu;
    return au & bu;
}

// Appends the listed rows of one K block at position q; returns the new position.
__device__ __forceinline__ int append_rows(uint16_t *krow, uint8_t *rmask, int q, int kb, unsigned rows,
                                           unsigned aw, unsigned bw, int cap, int *status)
{
    while (rows) {
        const int kk = __ffs(rows) - 1;
        rows &= rows - 1;
        const unsigned as = aw >> kk, bs = bw >> kk;
        const unsigned abits = (as & 1u) | ((as >> 7) & 2u) | ((as >> 14) & 4u) | ((as >> 21) & 8u);
        const unsigned bbits = (bs & 1u) | ((bs >> 7) & 2u) | ((bs >> 14) & 4u) | ((bs >> 21) & 8u);
        if (bounds_ok(q < cap, status, 20)) {
            krow[q] = (uint16_t)(kb * BK + kk);
            rmask[q] = (uint8_t)(abits | (bbits << 4));
        }
        ++q;
    }
    return q;
}

__device__ __forceinline__ int warp_inclusive_scan(int v, int lane)
{
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(0xFFFFFFFFu, v, d);
        if (lane >= d) v += t;
    }
    return v;
}

// First pass of the mask warp over a tile's pattern bytes: the live byte of its first K block, whether all
// K blocks share it, the number of live k, and how many of those lie in K blocks with at most brow_bits live k.
// whether the live k of a K block are live for each of the tile's RB row blocks and 4 column blocks
template <int RB>
__device__ __forceinline__ bool blocks_cover(unsigned aw, unsigned bw, unsigned live)
{
    const unsigned l4 = live * 0x01010101u, am = RB == 4 ? 0xFFFFFFFFu : 0x0000FFFFu;
    return ((aw & l4 & am) == (l4 & am)) && ((bw & l4) == l4);
}

template <int RB, int KPL, bool RM>
__device__ __forceinline__ void tile_scan(const PackedParams &p, int tm, int tn, int kb_lo, int kb_hi, int lane, unsigned &live_first,
                                          bool &uniform, bool &full, int &live_total, int &live_small)
{
    for (int c0 = kb_lo; c0 < kb_hi; c0 += 32 * KPL) {
        const int kb0 = c0 + KPL * lane;
        unsigned aw[KPL], bw[KPL];
        load_patterns<RB, KPL, RM>(p, tm, tn, kb0, kb0 < kb_hi, aw, bw);
        if (c0 == kb_lo) live_first = __shfl_sync(0xFFFFFFFFu, tile_live(aw[0], bw[0]), 0);
        bool same = true, cover = true;
        int cnt = 0, small = 0;
#pragma unroll
        for (int j = 0; j < KPL; ++j) {
            const unsigned live = tile_live(aw[j], bw[j]);
            same = same && live == live_first;
            cover = cover && blocks_cover<RB>(aw[j], bw[j], live);
            cnt += __popc(live);
            small += __popc(live) <= p.brow_bits ? __popc(live) : 0;
        }
        uniform = uniform && __all_sync(0xFFFFFFFFu, kb0 >= kb_hi || same);
        full = full && __all_sync(0xFFFFFFFFu, kb0 >= kb_hi || cover);
        live_total += __reduce_add_sync(0xFFFFFFFFu, cnt);
        live_small += __reduce_add_sync(0xFFFFFFFFu, small);
    }
}

struct TileScan {
    unsigned live_first;
    bool uniform, full;
    int live_total, live_small;
};

// K block kb's byte of the pattern of 32-row block mb, 0 past the last block; with row-major A, without the bits of k past K
template <bool RM>
__device__ __forceinline__ unsigned a_byte(const PackedParams &p, int mb, int kb)
{
    unsigned v = 0u;
    if constexpr (RM) {
        const PatternRows pr = a_pattern<RM>(p, mb);
        if (pr.first)
            for (int j = 0; j < pr.count; ++j) v |= pr.first[(size_t)j * p.nKB + kb];
        if (kb == p.nKB - 1) v &= p.last_bits & 0xFFu;
    } else {
        if (mb < p.a_rows) v = p.a_pat[(size_t)mb * p.nKB + kb];
    }
    return v;
}

template <int RB, bool RM>
__device__ __forceinline__ TileScan tile_scan_any(const PackedParams &p, int tm, int tn, int kb_lo, int kb_hi, int lane)
{
    TileScan s = {0u, true, true, 0, 0};
    if (p.vec_patterns == 16) {
        tile_scan<RB, 16, RM>(p, tm, tn, kb_lo, kb_hi, lane, s.live_first, s.uniform, s.full, s.live_total, s.live_small);
    } else if (p.vec_patterns == 4) {
        tile_scan<RB, 4, RM>(p, tm, tn, kb_lo, kb_hi, lane, s.live_first, s.uniform, s.full, s.live_total, s.live_small);
    } else {
        for (int kb0 = kb_lo; kb0 < kb_hi; kb0 += 32) {
            const int kb = kb0 + lane;
            unsigned au = 0, bu = 0;
            if (kb < kb_hi) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int mb = tm * RB + i, nb = tn * 4 + i;
                    if (i < RB) au |= a_byte<RM>(p, mb, kb);
                    if (nb < p.b_rows) bu |= p.b_pat[(size_t)nb * p.nKB + kb];
                }
            }
            const unsigned live = au & bu;
            if (kb0 == kb_lo) s.live_first = __shfl_sync(0xFFFFFFFFu, live, 0);
            s.uniform = s.uniform && __all_sync(0xFFFFFFFFu, kb >= kb_hi || live == s.live_first);
            s.full = false;   // the byte-wise path keeps the general listing
            s.live_total += __reduce_add_sync(0xFFFFFFFFu, __popc(live));
            s.live_small += __reduce_add_sync(0xFFFFFFFFu, __popc(live) <= p.brow_bits ? __popc(live) : 0);
        }
    }
    return s;
}

// Second pass: the row list.  Lane l owns K blocks c0 + KPL l .. c0 + KPL l + KPL - 1 (consecutive lanes,
// consecutive K); K blocks with more than whole_above live k are listed whole.  Returns the row count.
// Rows are numbered from K block kb_lo's first on.
template <int RB, int KPL, bool RM>
__device__ __forceinline__ int tile_list(const PackedParams &p, int tm, int tn, int kb_lo, int kb_hi, int lane, int whole_above,
                                         uint16_t *krow, uint8_t *rmask)
{
    int pos = 0;
    for (int c0 = kb_lo; c0 < kb_hi; c0 += 32 * KPL) {
        const int kb0 = c0 + KPL * lane;
        unsigned aw[KPL], bw[KPL];
        load_patterns<RB, KPL, RM>(p, tm, tn, kb0, kb0 < kb_hi, aw, bw);
        unsigned rows[KPL];
        int c = 0;
#pragma unroll
        for (int j = 0; j < KPL; ++j) {
            const unsigned live = tile_live(aw[j], bw[j]);
            rows[j] = live == 0u ? 0u : (__popc(live) > whole_above ? 0xFFu : live);
            c += __popc(rows[j]);
        }
        const int incl = warp_inclusive_scan(c, lane);
        int q = pos + incl - c;
#pragma unroll
        for (int j = 0; j < KPL; ++j) q = append_rows(krow, rmask, q, kb0 - kb_lo + j, rows[j], aw[j], bw[j], p.cap, p.status);
        pos += __shfl_sync(0xFFFFFFFFu, incl, 31);
    }
    return pos;
}

#ifndef ESMM_CONS_REGS
#define ESMM_CONS_REGS 160
#define ESMM_PROD_REGS 96
#endif

// Sum over a tile's listed rows of the number of consumer warps (of 8) the row is live for.  (A call rather than
// inline code: it runs once per CTA, and the kernel's register allocation stays that of the code without it.)
template <int WMB>
__device__ __noinline__ int listed_warp_rows(const uint8_t *rmask, int n, int lane)
{
    int warp_rows = 0;
    for (int r = lane; r < n; r += 32) {
        const unsigned m = rmask[r], a = m & 15u, b = m >> 4;
        const int na = WMB == 2 ? ((a & 3u) != 0u) + ((a & 12u) != 0u) : __popc(a & 3u);
        warp_rows += na * __popc(b);
    }
    return __reduce_add_sync(0xFFFFFFFFu, warp_rows);
}

// Which way of working the launch takes: the same answer in every CTA.  All warps of the CTA call this; scratch: shared memory for the
// samples, free again on return.  (A call rather than inline code: it runs once per CTA, and what follows gets better registers: pruned
// MLP 2048 x 11008 x 4096 765 -> 748 us, 1000 x 1508 x 2012 at 0.5 / 0.5 59.4 -> 57.4, 4096^3 dense 2165 -> 2148.  Block mode as a call
// spills: 866, 67.6, 2170.)
// MODE_BLOCKS_WIDE_B: pairs of column blocks; MODE_BLOCKS_AGREE: which had the same patterns wherever samples were taken.
enum { MODE_PIPELINE = 0, MODE_BLOCKS = 1, MODE_BLOCKS_WIDE_B = 2, MODE_BLOCKS_AGREE = 4 };

template <bool RM>
__device__ __noinline__ int choose_mode(const PackedParams &p, char *scratch, int warp, int lane)
{
    // Operands whose samples are the same in all row blocks and in all column blocks of their tiles (uniform patterns, dense ones)
    // are for the pipeline, at the price of one barrier and no counting (1024 x 1024 x 768 at half density 28.6 -> 26.7 us, as
    // without the look; 1024^3 33.0 -> 32.8; pattern rows read byte by byte: 1126 x 776 x 840 at a quarter 24.6 -> 22.6).
    SampleWords words;
    words.differ = false;
    const int sample_m = warp * ((p.a_rows + 3) >> 2) / BM_SAMPLES, sample_n = ((5 * warp + 2) & 7) * p.tiles_n / BM_SAMPLES;
    if (warp < BM_SAMPLES) words = sample_words<RM>(p, sample_m, sample_n, warp, lane, false);
    if (!__syncthreads_or(words.differ) && p.block_mode <= 0) return MODE_PIPELINE;
    // two vectors per sample
    int4 *stats = reinterpret_cast<int4 *>(scratch);
    static_assert(2 * BM_SAMPLES * sizeof(int4) <= P_CONSUMER_WARPS * 2 * 96 && BM_SAMPLES <= P_CONSUMER_WARPS, "samples");
    if (warp < BM_SAMPLES) {
        if (!p.pat_words) words = sample_words<RM>(p, sample_m, sample_n, warp, lane, true);
        const TileStats s = tile_stats(words);
        int4 x, y;
        x.x = __reduce_add_sync(0xFFFFFFFFu, s.slots);
        x.y = __reduce_add_sync(0xFFFFFFFFu, s.work);
        x.z = __reduce_add_sync(0xFFFFFFFFu, s.a_differ);
        x.w = __reduce_add_sync(0xFFFFFFFFu, s.b_differ);
        y.x = __reduce_add_sync(0xFFFFFFFFu, s.listed);
        y.y = __reduce_add_sync(0xFFFFFFFFu, s.rows64);
        y.z = __reduce_add_sync(0xFFFFFFFFu, s.single);
        y.w = 0;
        if (lane == 0) {
            stats[warp] = x;
            stats[BM_SAMPLES + warp] = y;
        }
    }
    __syncthreads();
    int slots = 0, work = 0, a_differ = 0, b_differ = 0;
#pragma unroll
    for (int i = 0; i < BM_SAMPLES; ++i) {
        const int4 x = stats[i];
        slots += x.x;
        work += x.y;
        a_differ += x.z;
        b_differ += x.w;
    }
    bool blocks = p.block_mode > 0 || block_mode_pays(work, slots, RM ? RM_SIXTEENTHS : BM_SIXTEENTHS);
    if (RM && blocks && p.block_mode <= 0 && (p.rm_shape & RM_FILLS)) {
        int listed = 0, rows64 = 0;
        for (int i = 0; i < BM_SAMPLES; ++i) {
            const int4 y = stats[BM_SAMPLES + i];
            listed += y.x;
            rows64 += y.y;
        }
        blocks = !row_major_pipeline_pays(work, slots, rows64, listed, BM_SAMPLES * min(32 * 4 * BK, p.K), p.rm_shape);
    }
    if (blocks && blockIdx.x == 0 && threadIdx.x == 0 && p.form_hint != nullptr) {
        // the note for the next launch (see gemm_ab_packed_launch_form)
        int listed = 0, rows64 = 0, single = 0;
        for (int i = 0; i < BM_SAMPLES; ++i) {
            const int4 y = stats[BM_SAMPLES + i];
            listed += y.x;
            rows64 += y.y;
            single += y.z;
        }
        const int note = p.few_blocks && 2 * single >= listed && rows64 <= 3 * listed ? 1 : 0;
        if (note != p.form_known) *p.form_hint = note;
    }
    __syncthreads();   // the samples have been read by all
    if (!blocks) return MODE_PIPELINE;
    // Pairs on the side whose blocks differ less.  Where neither does more, on B's: an item then has one block of A, which row-major A is
    // transposed for (16 and not 32 copies a stage), and with packed A the faster code; not at N's edge (1500^3, 64-granular 0.5 / 0.5
    // 49.3 us, 48.5 with A's).
    const bool wide_b = RM || !(p.N & 63) ? b_differ <= a_differ : b_differ < a_differ;
    return MODE_BLOCKS | (wide_b ? MODE_BLOCKS_WIDE_B : 0) | (wide_b && b_differ == 0 ? MODE_BLOCKS_AGREE : 0);
}

// The CTA's next row list: the tile's next one, or the first of its next tile.
template <bool RM>
__device__ __forceinline__ void next_list(const PackedParams &p, int &tile, int &list)
{
    if (RM && ++list < p.lists) return;
    list = 0;
    tile += gridDim.x;
}

// RM: A is the caller's row-major matrix.  The producers then transpose the tile's rows of A with 4-byte copies, the rest is the same.
// (Before, a kernel of its own fetched boxes of 128 rows x 8 k, multiplied with scalar FMAs and could not leave out dead k of A.
// Kernel alone, before -> now: 2048^3 64-granular 0.5 / 0.5 232 -> 149 us, 32-granular 0.2 / 0.2 106 -> 72; 4096^3 dense 2806 -> 2387, half
// 1844 -> 1210; 2048 x 2048 x 1000 dense 210 -> 199.)
// BLOCKS: with block mode; without it for launches too short to look whether it would pay (the code is then that of the pipeline
// alone: up to 1.3 us of a 15 us call).
template <int WMB, int NPW, bool RM, bool BLOCKS>
__device__ __forceinline__ void tiled_sgemm(const PackedMaps &maps, const PackedParams &p)
{
    static_assert(NPW == 3 || NPW == 7, "consumers, producers and the mask warp fill whole warp groups");
    constexpr int P_TMA_WARPS = NPW;
    constexpr int P_MASK_WARP = P_CONSUMER_WARPS + NPW;
    constexpr bool P_REBALANCE_REGS = NPW == 7;
    constexpr int TM_ROWS = 64 * WMB;                  // rows of a tile of C: 128 or 64
    constexpr int RB = 2 * WMB;                        // 32-row blocks per tile
    constexpr int A_ROW = stage_a_row(WMB, RM);        // bytes of one k of the A tile in shared memory
    constexpr uint32_t STAGE_ROW_BYTES = TM_ROWS * 4 + ROW_BYTES;
    constexpr int STAGE_A_BYTES = RM ? RM_STAGE_A_BYTES : STAGE_HALF_BYTES, STAGE_BYTES = STAGE_A_BYTES + STAGE_HALF_BYTES;
    extern __shared__ __align__(1024) char smem[];
    const PackedSmem L = packed_smem_layout(p.stages, STAGE_BYTES, p.cap, BLOCKS);
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + L.bar_off);
    const uint32_t full0 = smem_u32(bars);
    const uint32_t empty0 = smem_u32(bars + P_MAX_STAGES);
    const uint32_t lfull0 = smem_u32(bars + 2 * P_MAX_STAGES);
    const uint32_t lempty0 = smem_u32(bars + 2 * P_MAX_STAGES + 2);
    volatile int *nrows = reinterpret_cast<volatile int *>(smem + L.misc_off);
    volatile int *abort_flag = nrows + 2;
    volatile int *n_producers = nrows + 3;   // 16-warp form: producer warps that copy (set with the first tile's list)
    // per list buffer: 0, or RUN_TILE | log2(c) | kk0 << 4 for a tile whose every K block has the same c = 1, 2,
    // 4 or 8 consecutive live k (kk0 .. kk0 + c - 1), live for all of the tile's row and column blocks.  Such
    // a tile needs no row list: stage s is the 3-D box of K blocks 32 s / c .. and every stage is all-live.
    volatile int *runinfo = nrows + 4;
    int *next_item = const_cast<int *>(nrows) + 6;   // block mode's item counter

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(full0 + 8 * s, RM ? 1 + 32 * P_TMA_WARPS : 1);
            mbar_init(empty0 + 8 * s, P_CONSUMER_WARPS);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(lfull0 + 8 * b, 1);
            mbar_init(lempty0 + 8 * b, P_CONSUMER_WARPS + P_TMA_WARPS);
        }
        *abort_flag = 0;
        *next_item = BM_WARPS;
        fence_barrier_init();
        fence_proxy_async();
    }
    __syncthreads();
    grid_dependency_wait();   // (patterns and the packed copy of A come from the kernel before this one)

    // The mode: every CTA looks at the same BM_SAMPLES samples, spread over the rows, the columns and K, so that all of them
    // come to the same answer.  The mask warp scans the CTA's first tile meanwhile, which the pipeline starts with.
    TileScan scan = {0u, true, true, 0, 0};
    if (warp == P_MASK_WARP && (int)blockIdx.x < p.num_tiles) {
        int tm, tn;
        tile_coords(blockIdx.x, p.tiles_m, p.tiles_n, tm, tn, p.group_m);
        scan = tile_scan_any<RB, RM>(p, tm, tn, 0, RM ? p.list_kb : p.nKB, lane);
    }
    if (BLOCKS && p.block_mode != 0) {
        const int mode = choose_mode<RM>(p, smem + L.wlist_off, warp, lane);
        if (mode != MODE_PIPELINE) {
            if (warp < BM_WARPS) {
                // The code of a whole launch, so that no two kinds of it compete for the instruction cache (items at N's edge alone
                // with predicates of their own: 2330 x 932 x 5020 128 -> 136 us).  Blocks all whole: copies without predicates; column
                // blocks that agree in pairs, where samples were taken: one list for both until they differ; and which operand's blocks come in
                // pairs is a constant.  Without / with the first two: pruned MLP 2048 x 11008 x 4096 744 -> 724, 4096^3 64-granular 0.5 / 0.5
                // 692 -> 674 us, 32-granular 0.2 / 0.2 164 either way (165 with one list until they differ, which is at once).  The constant:
                // 720 -> 701, 672 -> 651 (with column blocks in pairs, too: 680 with A's), 162 -> 160, 2330 x 932 x 5020 125 -> 123;
                // row-major 2048 x 11008 x 4096 856 -> 827.  Row blocks that agree have no code for it: A 64-granular, B 32-granular 677 us
                // with it, 655 without.
                const bool wide_b = (mode & MODE_BLOCKS_WIDE_B) != 0;
                if ((p.N & 63) || (RM && (p.M & 63))) {
                    if (wide_b) block_mode<RM, true, false>(p, smem, warp, lane, true, next_item);
                    else block_mode<RM, true, false>(p, smem, warp, lane, false, next_item);
                } else if (!wide_b) block_mode<RM, false, false>(p, smem, warp, lane, false, next_item);
                else if (mode & MODE_BLOCKS_AGREE) block_mode<RM, false, true>(p, smem, warp, lane, true, next_item);
                else block_mode<RM, false, false>(p, smem, warp, lane, true, next_item);
            }
            return;
        }
    }

    bool ok = true;
    if (warp == 0) ESMM_STAMP(0);

    // (16-warp form: registers move from the producer / mask warp groups to the consumer warp groups; 8 x 32 x 160 +
    // 8 x 32 x 96 = 65536, all the CTA starts with.  Each instruction heads its own side's code.)
    if (warp == P_MASK_WARP) {
        if (P_REBALANCE_REGS) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(ESMM_PROD_REGS));
        // ---------------- mask warp: the tile's list of live k rows ----------------
        int it = 0, list = 0;
        for (int tile = blockIdx.x; tile < p.num_tiles && ok; next_list<RM>(p, tile, list), ++it) {
            const int buf = it & 1;
            const int kb_lo = RM ? list * p.list_kb : 0, kb_hi = RM ? min(kb_lo + p.list_kb, p.nKB) : p.nKB;
            int tm, tn;
            tile_coords(tile, p.tiles_m, p.tiles_n, tm, tn, p.group_m);
            // A first pass over the list's pattern bytes (the first one's is done) decides the listing policy.
            if (it > 0) scan = tile_scan_any<RB, RM>(p, tm, tn, kb_lo, kb_hi, lane);
            const unsigned live_first = scan.live_first;
            const bool uniform = scan.uniform, full = scan.full;
            const int live_total = scan.live_total, live_small = scan.live_small;
            ok = mbar_wait(lempty0 + 8 * buf, ((it >> 1) & 1) ^ 1, abort_flag);
            if (!ok) break;
            uint16_t *krow = reinterpret_cast<uint16_t *>(smem + L.krow_off + buf * L.krow_stride);
            uint8_t *rmask = reinterpret_cast<uint8_t *>(smem + L.rmask_off + buf * L.rmask_stride);
            // uniform tile: list live k only.  Otherwise the policy is two numbers: K blocks with more than brow_bits
            // live k are listed whole, on tiles with at most row_density live k per K block on average; denser
            // tiles list every live K block whole.  With the producers fetching runs of consecutive rows as boxes,
            // listing exactly the live k is best at every density measured (brow_bits 7, row_density 8: a K
            // block is then listed whole only when it is whole; 6 / 6 was 2-4 % slower on independent
            // 32-granular patterns at 0.5 / 0.5 and 0.3 / 0.7).
            const int whole_above = uniform ? BK : (live_total <= p.row_density * (kb_hi - kb_lo) ? p.brow_bits : 0);
            // a run tile?  c = 1, 2, 4 or 8 consecutive live k, whole stages only, 3-D view of B valid
            int run_code = 0;
            {
                const int c = __popc(live_first);
                const int kk0 = __ffs((int)live_first) - 1;
                if (uniform && full && live_first != 0u && (c & (c - 1)) == 0 &&
                    (live_first >> kk0) == (1u << c) - 1u && ((kb_hi - kb_lo) * c) % ROWS_PER_STAGE == 0 && p.b_runs_ok &&
                    !p.force_listed && !p.no_run_tiles)
                    run_code = RUN_TILE | (31 - __clz(c)) | (kk0 << 4);
            }
            int pos = 0;
            if (run_code) {
                pos = (kb_hi - kb_lo) * __popc(live_first);
            } else if (p.vec_patterns == 16) {
                pos = tile_list<RB, 16, RM>(p, tm, tn, kb_lo, kb_hi, lane, whole_above, krow, rmask);
            } else if (p.vec_patterns == 4) {
                pos = tile_list<RB, 4, RM>(p, tm, tn, kb_lo, kb_hi, lane, whole_above, krow, rmask);
            } else {
                for (int kb0 = kb_lo; kb0 < kb_hi; kb0 += 32) {
                    const int kb = kb0 + lane;
                    unsigned aw = 0, bw = 0;  // byte i: pattern of the tile's i-th 32-row / 32-column block
                    if (kb < kb_hi) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const int mb = tm * RB + i, nb = tn * 4 + i;
                            if (i < RB) aw |= a_byte<RM>(p, mb, kb) << (8 * i);
                            if (nb < p.b_rows) bw |= (unsigned)p.b_pat[(size_t)nb * p.nKB + kb] << (8 * i);
                        }
                    }
                    const unsigned live = tile_live(aw, bw);            // k live for the tile as a whole
                    const unsigned rows = live == 0u ? 0u : (__popc(live) > whole_above ? 0xFFu : live);
                    const int c = __popc(rows);
                    const int incl = warp_inclusive_scan(c, lane);
                    append_rows(krow, rmask, pos + incl - c, kb - kb_lo, rows, aw, bw, p.cap, p.status);
                    pos += __shfl_sync(0xFFFFFFFFu, incl, 31);
                }
            }
            // rows past the end of the last stage read as dead
            if (!run_code) {
                const int q = pos + lane;
                if (q < ((pos + 31) & ~31) && bounds_ok(q < p.cap, p.status, 22)) {
                    krow[q] = 0;
                    rmask[q] = 0;
                }
            }
            // a tile of mostly single rows: no stage of it is a run of whole K blocks, bar a rare coincidence
            const bool sparse_rows = !run_code && !uniform && whole_above == p.brow_bits && 2 * live_small >= pos;
            if (it == 0 && (NPW == 7 || (blockIdx.x == 0 && p.form_hint != nullptr))) {
                // 16-warp form: how many producer warps copy.  A row-by-row stage costs its producers the same 64
                // copies whatever the patterns, and its consumers one pass per row that is live for their own
                // 64 (32) rows x 32 columns.  Where the CTA's first tile is mostly such rows and a consumer warp
                // works on 12 of a stage's 32 rows or fewer, three producers cannot keep up and all seven copy;
                // otherwise three do and four stay idle.
                bool wants7 = false;
                if (sparse_rows) {
                    __syncwarp();
                    wants7 = listed_warp_rows<WMB>(rmask, min(pos, p.cap), lane) <= 3 * pos;
                }
                if (lane == 0) {
                    *n_producers = !p.adaptive || wants7 ? 7 : 3;
                    // (either form computes the same C; the note only steers the shape of the next launch)
                    if (blockIdx.x == 0 && p.form_hint != nullptr && (wants7 ? 1 : 0) != p.form_known) *p.form_hint = wants7 ? 1 : 0;
                }
            }
            if (lane == 0) {
                nrows[buf] = pos;
                runinfo[buf] = run_code | (sparse_rows ? 0 : RUNS_LIKELY);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(lfull0 + 8 * buf);
            if (it == 0) ESMM_STAMP(1);
        }
    } else if (warp >= P_TMA_WARP) {
        if (P_REBALANCE_REGS) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(ESMM_PROD_REGS));
        // ---------------- producer warps: one lane per row of the stage ----------------
        // All of them walk the row list and take the same decisions; producer q issues the copies of
        // rows 32 q / P .. of each stage, producer 0 also the stage's byte count and whole-stage boxes.
        // (A copy may complete before producer 0 has posted the byte count: the barrier's transaction
        // count then goes negative for a moment, which it is allowed to, and the phase cannot complete
        // before producer 0's arrival.)
        const int q = warp - P_TMA_WARP;
        if (q == 0 && lane < 16 && (!RM || lane >= 8)) tma_prefetch_descriptor(&maps.a_box[0] + lane);
        int slot = 0;
        uint32_t phase = 0;
        uint32_t issued_bits = 0, parity_bits = 0;  // per slot: ever issued / parity of last issue
        int it = 0, list = 0;
        int copying = P_TMA_WARPS;   // producer warps that share the copies out
        for (int tile = blockIdx.x; tile < p.num_tiles && ok; next_list<RM>(p, tile, list), ++it) {
            const int buf = it & 1;
            ok = NPW == 7 && q >= copying ? mbar_wait_idle(lfull0 + 8 * buf, (it >> 1) & 1, abort_flag)
                                          : mbar_wait(lfull0 + 8 * buf, (it >> 1) & 1, abort_flag);
            if (!ok) break;
            if (NPW == 7 && it == 0) copying = *n_producers;
            if (NPW == 7 && q >= copying) {
                // an idle producer: it only hands the list buffer back, once per tile
                __syncwarp();
                if (lane == 0) mbar_arrive(lempty0 + 8 * buf);
                continue;
            }
            int tm, tn;
            tile_coords(tile, p.tiles_m, p.tiles_n, tm, tn, p.group_m);
            const uint16_t *krow = reinterpret_cast<const uint16_t *>(smem + L.krow_off + buf * L.krow_stride);
            const int n = nrows[buf];
            const int run_code = runinfo[buf] & (RUN_TILE | 0xFF);
            const bool look_for_runs = (runinfo[buf] & RUNS_LIKELY) != 0 && p.b_runs_ok;
            // packed A is stored in panels of 128 rows: a 64-row tile is the left or right half of one
            const int panel = WMB == 2 ? tm : tm >> 1;
            const int a_x = WMB == 2 ? 0 : (tm & 1) * TM_ROWS;
            const int a_row0 = panel * p.kp, b_col0 = tn * TILE_N;
            if constexpr (RM) {
                const int lc = run_code & 15, kk0 = (run_code >> 4) & 7;
                const int k_lo = list * p.list_kb * BK;            // what the list's k are counted from
                for (int r0 = 0; r0 < n; r0 += ROWS_PER_STAGE) {
                    const int cnt = min(ROWS_PER_STAGE, n - r0);
                    int k = -1;                                    // of the stage's row `lane`
                    if (run_code) k = (((r0 + lane) >> lc) << 3) + kk0 + (lane & ((1 << lc) - 1));
                    else if (lane < cnt && bounds_ok(r0 + lane < p.cap, p.status, 27)) k = krow[r0 + lane];
                    // B in boxes, as below
                    const int k_prev = __shfl_up_sync(0xFFFFFFFFu, k, 1);
                    const unsigned starts = __ballot_sync(0xFFFFFFFFu, lane < cnt && (lane == 0 || k != k_prev + 1));
                    int box_log = -1;
                    if (lane < cnt && !run_code) {
                        const int first = 31 - __clz((int)(starts & (0xFFFFFFFFu >> (31 - lane))));
                        const unsigned later = lane == 31 ? 0u : (starts >> (first + 1)) << (first + 1);
                        const int len = (later ? __ffs((int)later) - 1 : cnt) - first, o = lane - first, full8 = len & ~7;
                        if (o < full8) box_log = (o & 7) == 0 ? 3 : -1;
                        else if ((len & 4) && o == full8) box_log = 2;
                        else if ((len & 2) && o == full8 + (len & 4)) box_log = 1;
                        else if ((len & 1) && o == len - 1) box_log = 0;
                        if (((lane * P_TMA_WARPS) >> 5) != q) box_log = -1;
                    }
                    ok = mbar_wait(empty0 + 8 * slot, phase ^ 1, abort_flag);
                    ok = __all_sync(0xFFFFFFFFu, ok);
                    if (!ok) break;
                    const uint32_t full = full0 + 8 * slot;
                    const uint32_t s0 = smem_u32(smem + L.stage_off) + (uint32_t)slot * STAGE_BYTES;
                    if (q == 0 && lane == 0) {
                        mbar_arrive_expect_tx(full, (uint32_t)cnt * ROW_BYTES);
                        if (run_code) tma_load_3d(s0 + STAGE_A_BYTES, &maps.b_run[lc], b_col0, kk0, list * p.list_kb + (r0 >> lc), full);
                    }
                    if (box_log >= 0) tma_load_2d(s0 + STAGE_A_BYTES + lane * ROW_BYTES, &maps.b_box[box_log], b_col0, k_lo + k, full);
                    // A: 4-byte copies, eight lanes on the k and four on the rows, so that neighbouring k of a row come as one
                    // sector; row groups shared out among the producers.  Rows past the end of A, k past its width (in K
                    // blocks listed whole; no mask has their bit) and past the end of the list: any element, never multiplied
                    // or never stored.
                    // What bounds the form: these copies go through the banks the consumers load from, one pass per sector since a
                    // stage's rows of A are 16 bytes further apart.  Kernel alone, before that -> now (packed A: 2144): 4096^3 dense
                    // 2621 -> 2387 us, 64-granular 0.5 / 0.5 977 -> 874; 2048 x 2048 x 1000 dense 233 -> 199.  (Rows in place and their
                    // 16-byte chunks exchanged instead: 4096^3 dense 2445, then with 16 lanes on the k 2501, with 32 2642.)
                    constexpr int KL = RM_KL, RL = 32 / KL;
                    const int kk = lane & (KL - 1), rr = lane / KL;
                    int kg[32 / KL];
#pragma unroll
                    for (int g = 0; g < 32 / KL; ++g) kg[g] = min(k_lo + max(__shfl_sync(0xFFFFFFFFu, k, KL * g + kk), 0), p.K - 1);
#pragma unroll 1
                    for (int rg = q; rg < TM_ROWS / RL; rg += P_TMA_WARPS) {
                        const float *row = p.A + (size_t)min(tm * TM_ROWS + rg * RL + rr, p.M - 1) * p.K;
                        const uint32_t d = s0 + kk * A_ROW + (rg * RL + rr) * 4;
#pragma unroll
                        for (int g = 0; g < 32 / KL; ++g) cp_async_4(d + g * KL * A_ROW, row + kg[g]);
                    }
                    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(full) : "memory");
                    issued_bits |= 1u << slot;
                    parity_bits = (parity_bits & ~(1u << slot)) | (phase << slot);
                    if (++slot == p.stages) {
                        slot = 0;
                        phase ^= 1;
                    }
                }
            } else if (run_code) {
                // a run tile: whole stages, each one box per operand, no row list
                const int lc = run_code & 15, kk0 = (run_code >> 4) & 7;
                for (int r0 = 0; r0 < n; r0 += ROWS_PER_STAGE) {
                    // (every producer waits for every stage's slot, also where it has nothing to copy: a
                    // parity wait only tells "this phase" from "the one before", so no producer may get
                    // more than one lap of the ring ahead of the consumers)
                    ok = mbar_wait(empty0 + 8 * slot, phase ^ 1, abort_flag);
                    if (!ok) break;
                    const uint32_t full = full0 + 8 * slot;
                    if (q == 0 && lane == 0) {
                        mbar_arrive_expect_tx(full, (uint32_t)ROWS_PER_STAGE * STAGE_ROW_BYTES);
                        const uint32_t s0 = smem_u32(smem + L.stage_off) + (uint32_t)slot * STAGE_BYTES;
                        const int kb0 = r0 >> lc;
                        tma_load_3d(s0, &maps.a_run[lc], a_x, kk0, panel * p.nKB + kb0, full);
                        tma_load_3d(s0 + STAGE_A_BYTES, &maps.b_run[lc], b_col0, kk0, kb0, full);
                    }
                    if (q == 0) {
                        issued_bits |= 1u << slot;
                        parity_bits = (parity_bits & ~(1u << slot)) | (phase << slot);
                    }
                    if (it == 0 && q == 0) ESMM_STAMP(400 + r0 / ROWS_PER_STAGE);
                    if (++slot == p.stages) {
                        slot = 0;
                        phase ^= 1;
                    }
                }
            }
            // (the k of a stage's rows are read one stage ahead, under the copies of the stage before)
            int k_next = !RM && !run_code && lane < n && bounds_ok(lane < p.cap, p.status, 27) ? (int)krow[lane] : -1;
            for (int r0 = 0; r0 < n && !RM && !run_code; r0 += ROWS_PER_STAGE) {
                const int cnt = min(ROWS_PER_STAGE, n - r0);
                const bool valid = lane < cnt;
                if (it == 0 && q == 0 && r0 < 80 * ROWS_PER_STAGE) ESMM_STAMP(700 + 4 * (r0 / ROWS_PER_STAGE));
                const int k = k_next;
                {
                    const int rn = r0 + ROWS_PER_STAGE + lane;
                    k_next = rn < n && bounds_ok(rn < p.cap, p.status, 27) ? (int)krow[rn] : -1;
                }
                // a uniform run?  rows = k offsets kk0 .. kk0 + c - 1 of 32 / c consecutive K blocks
                const int k_first = __shfl_sync(0xFFFFFFFFu, k, 0);
                const int kb0 = k_first >> 3, kk0 = k_first & 7;
                int run = -1;  // log2(c)
                if (cnt == ROWS_PER_STAGE && look_for_runs) {
#pragma unroll
                    for (int lc = 3; lc >= 0; --lc) {
                        const int c = 1 << lc;
                        const int expect = ((kb0 + (lane >> lc)) << 3) + kk0 + (lane & (c - 1));
                        if (run < 0 && kk0 + c <= BK && __all_sync(0xFFFFFFFFu, k == expect)) run = lc;
                    }
                }
                // otherwise: the list is ascending, and rows with consecutive k are consecutive rows of packed A and of
                // B alike, so a run of L such rows is fetched in boxes of 8, 4, 2 and 1 rows (L = 8 a + 4 b + 2 c +
                // d, largest first): fewer copies for the same bytes.  The lane at a box's first row issues it.
                const int k_prev = __shfl_up_sync(0xFFFFFFFFu, k, 1);
                const unsigned starts = __ballot_sync(0xFFFFFFFFu, valid && (lane == 0 || k != k_prev + 1));
                int box_log = -1;   // log2 of the height of the box this lane issues
                if (valid && run < 0) {
                    const int first = 31 - __clz((int)(starts & (0xFFFFFFFFu >> (31 - lane))));   // my run's first lane
                    const unsigned later = lane == 31 ? 0u : (starts >> (first + 1)) << (first + 1);
                    const int len = (later ? __ffs((int)later) - 1 : cnt) - first;
                    const int o = lane - first;
                    const int full8 = len & ~7;
                    if (o < full8) box_log = (o & 7) == 0 ? 3 : -1;
                    else if ((len & 4) && o == full8) box_log = 2;
                    else if ((len & 2) && o == full8 + (len & 4)) box_log = 1;
                    else if ((len & 1) && o == len - 1) box_log = 0;
                }
                // my share of the stage: the boxes that start in my lane group
                if (((lane * copying) >> 5) != q) box_log = -1;
                if (it == 0 && q == 0 && r0 < 80 * ROWS_PER_STAGE) ESMM_STAMP(701 + 4 * (r0 / ROWS_PER_STAGE));
                ok = mbar_wait(empty0 + 8 * slot, phase ^ 1, abort_flag);
                ok = __all_sync(0xFFFFFFFFu, ok);
                if (!ok) break;
                if (it == 0 && q == 0 && r0 < 80 * ROWS_PER_STAGE) ESMM_STAMP(702 + 4 * (r0 / ROWS_PER_STAGE));
                {
                    const uint32_t full = full0 + 8 * slot;
                    const uint32_t s0 = smem_u32(smem + L.stage_off) + (uint32_t)slot * STAGE_BYTES;
                    const uint32_t sa = s0 + lane * A_ROW;
                    const uint32_t sb = s0 + STAGE_A_BYTES + lane * ROW_BYTES;
                    if (run >= 0) {
                        if (q == 0 && lane == 0) {
                            tma_load_3d(sa, &maps.a_run[run], a_x, kk0, panel * p.nKB + kb0, full);
                            tma_load_3d(sb, &maps.b_run[run], b_col0, kk0, kb0, full);
                        }
                    } else if (box_log >= 0) {
                        tma_load_2d(sa, &maps.a_box[box_log], a_x, a_row0 + k, full);
                        tma_load_2d(sb, &maps.b_box[box_log], b_col0, k, full);
                    }
                    if (q == 0 && lane == 0) mbar_arrive_expect_tx(full, (uint32_t)cnt * STAGE_ROW_BYTES);
                    issued_bits |= 1u << slot;
                    parity_bits = (parity_bits & ~(1u << slot)) | (phase << slot);
                }
                if (it == 0 && q == 0) ESMM_STAMP(400 + r0 / ROWS_PER_STAGE);
                if (it == 0 && q == 0 && r0 < 80 * ROWS_PER_STAGE) ESMM_STAMP(703 + 4 * (r0 / ROWS_PER_STAGE));
                if (++slot == p.stages) {
                    slot = 0;
                    phase ^= 1;
                }
            }
            if (!ok) break;
            __syncwarp();
            if (lane == 0) mbar_arrive(lempty0 + 8 * buf);
        }
        if (RM) cp_async_wait_all();   // (after a wait that ran out, copies may still be in flight)
        if (!ok && lane == 0) {
            // leave only after the copies already issued have landed (bounded)
            for (int s = 0; s < p.stages; ++s) {
                if (!(issued_bits & (1u << s))) continue;
                const uint32_t par = (parity_bits >> s) & 1u;
                for (int tries = 0; tries < (1 << 16); ++tries)
                    if (mbar_try_wait(full0 + 8 * s, par)) break;
            }
        }
    } else {
        if (P_REBALANCE_REGS) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(ESMM_CONS_REGS));
        // ---------------- consumer warps: 32 WMB rows x 32 columns of the tile each ----------------
        const int wm = warp >> 2, wn = warp & 3;              // 2 x 4 warps
        const int lm = (lane >> 1) & 7;                       // group of 4 rows within a 32-row block
        const int ln = (lane & 1) | ((lane >> 4) << 1);       // 16-byte column chunk
        const uint32_t a_thr = (uint32_t)(wm * 32 * WMB + lm * 4) * 4;                // within a row of A
        const uint32_t b_thr = STAGE_A_BYTES + (uint32_t)(wn * 32 + ln * 4) * 4;  // within a row of B
        const int t_shift = WMB * wm, b_shift = 4 + wn;
        uint16_t *wlist_t = reinterpret_cast<uint16_t *>(smem + L.wlist_off + warp * 2 * WLIST_BYTES);
        uint16_t *wlist_b = wlist_t + WLIST_BYTES / 2;
        int slot = 0;
        uint32_t phase = 0;
        int it = 0, list = 0;
        Acc acc;
        for (int tile = blockIdx.x; tile < p.num_tiles && ok; next_list<RM>(p, tile, list), ++it) {
            const int buf = it & 1;
            ok = mbar_wait(lfull0 + 8 * buf, (it >> 1) & 1, abort_flag);
            if (!ok) break;
            int tm, tn;
            tile_coords(tile, p.tiles_m, p.tiles_n, tm, tn, p.group_m);
            const uint8_t *rmask = reinterpret_cast<const uint8_t *>(smem + L.rmask_off + buf * L.rmask_stride);
            const int n = nrows[buf];
            const bool run_tile = (runinfo[buf] & RUN_TILE) != 0;
            if (warp == 0) ESMM_STAMP(600 + 4 * it);

            if (!RM || list == 0) acc_clear(acc);

            // joint masks of a stage: bit r = row r is live for (top | bottom) block x my columns.  The
            // masks of the next stage are formed under the multiply-adds of the current one (the list's
            // buffer is padded by one stage, so reading one stage past the end is harmless).
            unsigned rm = run_tile ? 0xFFu : rmask[lane];   // (cap >= 64: the first stage is always inside the list)
            for (int r0 = 0; r0 < n; r0 += ROWS_PER_STAGE) {
                unsigned jt = 0xFFFFFFFFu, jb = 0xFFFFFFFFu;   // a run tile: every row live for every block
                if (!run_tile) {
                    const unsigned colb = (rm >> b_shift) & 1u;
                    jt = __ballot_sync(0xFFFFFFFFu, ((rm >> t_shift) & colb) != 0u);
                    jb = WMB == 2 ? __ballot_sync(0xFFFFFFFFu, ((rm >> (t_shift + 1)) & colb) != 0u) : jt;
                    rm = bounds_ok(r0 + ROWS_PER_STAGE + lane < p.cap, p.status, 23) ? rmask[r0 + ROWS_PER_STAGE + lane] : 0u;
                }
                const bool dense = (jt & jb) == 0xFFFFFFFFu && !p.force_listed;
                // in the 64-row tiling a row feeds 16 two-wide FMAs, as in the half modes: lists there too
                int cnt_t = 0, cnt_b = 0;
                if (WMB == 1 ? !dense : jt != jb) {
                    cnt_t = build_list<RM>(wlist_t, jt, lane, p.status);
                    if (WMB == 2) cnt_b = build_list<RM>(wlist_b, jb, lane, p.status);
                    __syncwarp();
                }
                ok = mbar_wait(full0 + 8 * slot, phase, abort_flag);
                if (!ok) break;
                if (!bounds_ok(slot >= 0 && slot < p.stages && L.stage_off + (uint32_t)(slot + 1) * STAGE_BYTES <= L.krow_off,
                               p.status, 24)) {
                    ok = false;   // a stage outside the ring: leave through the time-out path rather than read it
                    break;
                }
                const char *sA = smem + L.stage_off + (size_t)slot * STAGE_BYTES + a_thr;
                const char *sB = smem + L.stage_off + (size_t)slot * STAGE_BYTES + b_thr;
                if (warp == 0 && it == 0) ESMM_STAMP(10 + r0 / ROWS_PER_STAGE);
                if (dense) {
                    dense_rows<WMB, RM>(acc, sA, sB);
                } else if (WMB == 1) {
                    listed_rows<MODE_TOP, 1, RM>(acc, sA, sB, wlist_t, cnt_t);
                } else if (jt == jb) {
                    masked_rows_both<RM>(acc, sA, sB, jt);
                } else {
                    listed_rows<MODE_TOP, 2, RM>(acc, sA, sB, wlist_t, cnt_t);
                    listed_rows<MODE_BOTTOM, 2, RM>(acc, sA, sB, wlist_b, cnt_b);
                }
                if (warp == 0 && it == 0) ESMM_STAMP(200 + r0 / ROWS_PER_STAGE);
                __syncwarp();
                if (lane == 0) mbar_arrive(empty0 + 8 * slot);
                if (++slot == p.stages) {
                    slot = 0;
                    phase ^= 1;
                }
            }
            if (!ok) break;
            __syncwarp();
            if (lane == 0) mbar_arrive(lempty0 + 8 * buf);
            if (warp == 0) ESMM_STAMP(601 + 4 * it);
            if (RM && list + 1 < p.lists) continue;   // (the tile's sums go on through its next list)

            // epilogue: C is overwritten (beta = 0)
            const int row0 = tm * TM_ROWS + wm * 32 * WMB + lm * 4;
            const int col0 = tn * TILE_N + wn * 32 + ln * 4;
#pragma unroll
            for (int pr = 0; pr < 2 * WMB; ++pr) {
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int i = 2 * pr + e;                        // row of the thread tile
                    const int row = row0 + (i & 3) + 32 * (i >> 2);
                    float v[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) v[j] = acc_get(acc, pr, e, j);
                    if (row < p.M) {
                        float *c = p.C + (size_t)row * p.N + col0;
                        const size_t c_floats = (size_t)p.M * p.N, off = (size_t)row * p.N + col0;
                        if (col0 < p.N && bounds_ok(off + 4 <= c_floats, p.status, 26))
                            *reinterpret_cast<float4 *>(c) = make_float4(v[0], v[1], v[2], v[3]);
                        if (col0 + 16 < p.N && bounds_ok(off + 20 <= c_floats, p.status, 26))
                            *reinterpret_cast<float4 *>(c + 16) = make_float4(v[4], v[5], v[6], v[7]);
                    }
                }
            }
            if (warp == 0) ESMM_STAMP(602 + 4 * it);
        }
    }

    if (warp == 0) ESMM_STAMP(5);
    if (!ok && lane == 0) atomicExch(p.status, (int)ESMM_ERR_TIMEOUT);
}

// esmm_gemm_rowmajor.cu.  (A file of its own, so that a program's first call loads the kernels it uses and not the others: first call of a
// process with row-major A 14 ms with all twelve in one module, 6.5 with its four; packed A 16 and 8.)
cudaError_t rowmajor_allow_smem(int bytes);
cudaError_t rowmajor_launch(int tile_rows, bool blocks, int grid, size_t smem, cudaStream_t stream, const PackedMaps &maps,
                            const PackedParams &p);

}  // namespace esmm
