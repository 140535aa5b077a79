// Block mode of the packed joint-sparse SGEMM: every warp of the CTA works on its own blocks of C, with its own list of live k
// and its own copies.
//
// The tiled pipeline (esmm_gemm_tiled.cuh) fetches every k that is live for any part of a 128 x 128 tile and moves in steps
// of 32 such rows, eight warps together.  On operands whose 32-row and 32-column blocks are zero in different places most of
// a fetched row is of no use to most of the warps, and a step lasts as long as its busiest warp.  Here nothing is shared:
//
//   * an item is a pair of adjacent 32 x 32 blocks of C: 32 rows x 64 columns where B's patterns agree in pairs of column blocks as
//     often as A's in pairs of row blocks, or more often (and N is a multiple of 64), else 64 rows x 32 columns.  The operand that spans 64 is called X, the one that
//     spans 32 Y;
//   * a warp joins the pattern bytes of each block to a list of its live k (ascending, 16 bits each, a ring of 512
//     that is refilled as it is used up).  Lanes
//     0-15 own the first block and walk its list, lanes 16-31 the second: a step is one live k of EACH block, 4 sixteen-byte
//     loads and 32 two-wide FMAs per thread for its 8 x 8 outputs, whether the two k are the same or not.  (One block after the
//     other on the whole warp, 4 x 8 outputs per thread, takes 6 loads for the same work.)
//   * the rows of 16 steps are one stage of the warp's own ring of two, fetched with 16-byte cp.async copies: 128 bytes of X and
//     128 of Y per block and k, Y only once where the blocks have the same list.  No copy is spent on a k that is dead for the
//     block, and no multiply-add unless one list is longer than the other;
//   * the warps of a CTA draw items from a counter in shared memory; the last ones come as single blocks spread over the whole
//     warp, so that the warps finish together (a problem with few blocks consists of nothing else).
//
// What bounds it: the FMA pipe together with everything else that is issued.  A stage (16 steps) is 512 two-wide FMAs and 64 loads; with
// everything, items' starts and ends included, it is 739 instructions at 4096^3 64-granular 0.5 / 0.5, where it was 785 (ncu), and the
// kernel takes 670 us instead of 716, the FMA pipe active 75 % of the time instead of 71.  So the others are kept few: one load per list
// for a lane's entries, one instruction per address, no predicates where all of B's blocks are whole, one list for blocks that agree.
// The rest is lost to the end of a launch (3-4 % between SMs, whose items differ, 2 % inside them).  Measured, whole calls, the tiled pipeline before ->
// block mode: 2048 x 11008 x 4096 pruned MLP 1016 -> 701 us, 4096^3 with independent 32-granular patterns at 0.2 / 0.2 308 -> 163 and at
// 0.5 / 0.5 921 -> 710, 1000 x 1508 x 2012 at 0.5 / 0.5 80.7 -> 49.  Also measured: one block after the other on the whole warp (4096^3 at 0.5 /
// 0.5 824), 8 k per stage (971), lists made for all of K before the first copy (762), rows past a list's end skipped in a second code
// path instead of multiplied by zeros (752: the accumulators are then moved between registers at every stage); eight warps that multiply
// and four that list and copy for them (pruned MLP 1129: a warp alone on its scheduler's spare slots takes 2000 cycles for a stage's 250
// instructions), the copies among the multiply-adds and an item's first stage under the last of the one before (823-875: 470 M
// instructions instead of 411 M).
//
// There is no barrier between warps and nothing to wait for but a warp's own copies.  Every output sees one FMA per live k, in
// ascending k, as in the tiled pipeline: the results are the same bits.
#pragma once

#include <climits>

#include "esmm_gemm_shared.cuh"

namespace esmm {

constexpr int RM_KL = 8;                                    // row-major A: lanes of a 4-byte copy instruction on the k (4: 9 % slower, 16: 12 %)
constexpr int BM_SAMPLES = 8;                               // tiles looked at to choose the mode

// bits of the k of K blocks kb .. kb + 3 that are < K
__device__ __forceinline__ unsigned inside_k(int kb, int K)
{
    const int left = K - kb * BK;
    return left >= 32 ? 0xFFFFFFFFu : left <= 0 ? 0u : (1u << left) - 1u;
}

// Pattern bytes of K blocks kb .. kb + 3 of one pattern row (null: no such row), zero past the end.  words: the row may be
// read as 32-bit words.
__device__ __forceinline__ unsigned pattern_word(const uint8_t *row, int kb, int nKB, bool words, int *status)
{
    if (row == nullptr || kb >= nKB) return 0u;
    if (!bounds_ok(kb >= 0 && (!words || (kb + 4 <= nKB && ((uintptr_t)(row + kb) & 3) == 0)), status, 36)) return 0u;   // checked build: site 36
    if (words) return *reinterpret_cast<const unsigned *>(row + kb);
    unsigned v = 0u;
#pragma unroll
    for (int j = 0; j < 4; ++j) v |= (unsigned)row[min(kb + j, nKB - 1)] << (8 * j);   // (four loads in flight)
    return v & inside_k(kb, nKB * BK);
}

// The pattern rows of one 32-row (32-column) block: count rows from `first` on, whose OR is the block's pattern; none: no such block.
struct PatternRows {
    const uint8_t *first;
    int count;
};

__device__ __forceinline__ unsigned pattern_word(const PatternRows &r, int kb, int nKB, bool words, int *status)
{
    unsigned v = pattern_word(r.first, kb, nKB, words, status);
    for (int t = 1; t < r.count; ++t) v |= pattern_word(r.first + (size_t)t * nKB, kb, nKB, words, status);
    return v;
}

template <typename Params>
__device__ __forceinline__ PatternRows b_pattern(const Params &p, int block)
{
    return {block < p.b_rows ? p.b_pat + (size_t)block * p.nKB : nullptr, 1};
}

// A's patterns have one row per 32 rows of A, or (ROW_MAJOR) one for every a_div blocks, or a_mul for each.
template <bool ROW_MAJOR, typename Params>
__device__ __forceinline__ PatternRows a_pattern(const Params &p, int block)
{
    if (block >= p.a_rows) return {nullptr, 1};
    if constexpr (ROW_MAJOR) {
        const int row = block / p.a_div * p.a_mul;
        return {p.a_pat + (size_t)row * p.nKB, min(p.a_mul, p.a_pat_rows - row)};
    } else {
        return {p.a_pat + (size_t)block * p.nKB, 1};
    }
}

// A sample: one 32-bit word, four K blocks, of each pattern row of a 128 x 128 tile per lane; zero where there is no such block.
// Pattern rows that may not be read as words: the first of the four K blocks only, where `whole` is not asked for.
struct SampleWords {
    unsigned a[4], b[4];
    int na, nb;      // row blocks, column blocks of the tile
    bool differ;     // two row blocks, or two column blocks, are not the same
};

// Sample `part` of BM_SAMPLES: up to 128 K blocks of the tile, a single round trip to memory.
template <bool ROW_MAJOR, typename Params>
__device__ __forceinline__ SampleWords sample_words(const Params &p, int tm, int tn, int part, int lane, bool whole)
{
    SampleWords s;
    s.na = min(4, p.a_rows - tm * 4);
    s.nb = min(4, p.b_rows - tn * 4);
    const int span = (p.nKB + 3) >> 2, first = max(0, (span - 32) * part / (BM_SAMPLES - 1));
    const int kb = 4 * (first + lane);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const PatternRows ra = a_pattern<ROW_MAJOR>(p, tm * 4 + i), rb = b_pattern(p, tn * 4 + i);
        if (p.pat_words || whole) {
            s.a[i] = pattern_word(ra, kb, p.nKB, p.pat_words, p.status);
            s.b[i] = pattern_word(rb, kb, p.nKB, p.pat_words, p.status);
        } else {
            s.a[i] = s.b[i] = 0u;
            if (kb < p.nKB) {
                for (int t = 0; ra.first && t < ra.count; ++t) s.a[i] |= ra.first[(size_t)t * p.nKB + kb];
                if (rb.first) s.b[i] = rb.first[kb];
            }
        }
    }
    s.differ = false;
#pragma unroll
    for (int i = 1; i < 4; ++i)
        s.differ = s.differ || (i < s.na && s.a[i] != s.a[0]) || (i < s.nb && s.b[i] != s.b[0]);
    return s;
}

// What one lane counts in its words.  (block, k) counts.
struct TileStats {
    int listed;      // k live for the tile as a whole
    int slots;       // listed k times the tile's 32 x 32 blocks: what the tiled pipeline holds in shared memory
    int work;        // (32 x 32 block, k) pairs that are live: what is multiplied
    int rows64;      // (64 x 32 blocks, k) pairs with a live k: what the tiled pipeline's warps step through
    int single;      // listed k in K blocks that are not live as a whole
    int a_differ, b_differ;   // bits in which adjacent row blocks (column blocks) of a pair differ
};

__device__ __forceinline__ TileStats tile_stats(const SampleWords &w)
{
    const unsigned(&a)[4] = w.a;
    const unsigned(&b)[4] = w.b;
    TileStats s = {0, 0, 0, 0, 0, 0, 0};
    const unsigned live = (a[0] | a[1] | a[2] | a[3]) & (b[0] | b[1] | b[2] | b[3]);
    s.listed = __popc(live);
    s.slots = s.listed * w.na * w.nb;
    s.single = s.listed - __popc(__vcmpeq4(live, 0xFFFFFFFFu));
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int i = 0; i < 4; ++i) s.work += __popc(a[i] & b[j]);
        s.rows64 += __popc((a[0] | a[1]) & b[j]) + __popc((a[2] | a[3]) & b[j]);
    }
    if (w.na > 1) s.a_differ += __popc(a[0] ^ a[1]);
    if (w.na > 3) s.a_differ += __popc(a[2] ^ a[3]);
    if (w.nb > 1) s.b_differ += __popc(b[0] ^ b[1]);
    if (w.nb > 3) s.b_differ += __popc(b[2] ^ b[3]);
    return s;
}

__device__ __forceinline__ int exclusive_scan(int v, int lane)
{
    int x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(0xFFFFFFFFu, x, d);
        if (lane >= d) x += t;
    }
    return x - v;
}

// Appends k0 + b for every set bit b of m to a list ring, from this lane's position q on; the entries before `taken` are done with.
__device__ __forceinline__ void append_live(uint16_t *list, int q, int taken, unsigned m, int k0, int *status)
{
    while (m) {
        const int bit = __ffs((int)m) - 1;
        m &= m - 1u;
        if (bounds_ok(q >= taken && q - taken < BM_LIST, status, 28)) list[q & (BM_LIST - 1)] = (uint16_t)(k0 + bit);   // checked build: site 28
        ++q;
    }
}

// A block's list of live k while its item is worked on: `list` is a ring; entries taken .. made - 1 are listed and not yet copied.
struct LiveList {
    uint16_t *list;
    int made, taken;
    __device__ __forceinline__ int pending() const { return made - taken; }
};

// BM_STEP steps of a stage: 8 x 8 outputs per thread, each half-warp on its own rows of X and Y.
__device__ __forceinline__ void pair_steps(Acc &acc, const char *sx, const char *sy)
{
#pragma unroll
    for (int r = 0; r < BM_STEP; ++r) {
        const int lo = r * 128, hi = r * 128 + 64;
        KFrag f;
        f.at = *reinterpret_cast<const float4 *>(sx + lo);
        f.ab = *reinterpret_cast<const float4 *>(sx + hi);
        f.b0 = *reinterpret_cast<const float4 *>(sy + lo);
        f.b1 = *reinterpret_cast<const float4 *>(sy + hi);
        fma_top(acc, f);
        fma_bottom(acc, f);
    }
}

// BM_STEP k of a single block: 4 x 8 outputs per thread.  Odd rows hold their upper half first; sx_odd: the lane's chunk of X in them.
__device__ __forceinline__ void single_steps(Acc &acc, const char *sx, const char *sx_odd, const char *sy)
{
#pragma unroll
    for (int r = 0; r < BM_STEP; ++r) {
        KFrag f;
        f.at = *reinterpret_cast<const float4 *>(((r & 1) ? sx_odd : sx) + r * 128);
        f.b0 = *reinterpret_cast<const float4 *>(sy + r * 128 + (r & 1) * 64);
        f.b1 = *reinterpret_cast<const float4 *>(sy + r * 128 + 64 - (r & 1) * 64);
        fma_top(acc, f);
    }
}

// Row-major A: the eight 16-byte chunks of row r of a stage lie at their number XOR rm_swizzle(r), so that 4-byte copies of eight k of
// four rows of A fall on all 32 banks; 16-byte copies and the loads below meet as few bank conflicts as without.  (Odd rows' halves
// swapped and nothing more, block mode of 2048^3 alone: 64-granular 0.5 / 0.5 175 us, 143 so; 32-granular 0.5 / 0.5 207 and 171.)
__host__ __device__ constexpr int rm_swizzle(int r) { return ((r >> 1) & 3) | ((r & 1) << 2); }

// pair_steps and single_steps on such rows.  The lane's chunks: xg and xg + 4, yg and yg + 4; of a single block lm, ln and ln + 4.
__device__ __forceinline__ void rm_pair_steps(Acc &acc, const char *sx, const char *sy, int xg, int yg)
{
#pragma unroll
    for (int r = 0; r < BM_STEP; ++r) {
        const int sw = rm_swizzle(r), lo = r * 128 + (sw & 4) * 16, hi = r * 128 + 64 - (sw & 4) * 16;
        const char *x = sx + ((xg ^ (sw & 3)) << 4), *y = sy + ((yg ^ (sw & 3)) << 4);
        KFrag f;
        f.at = *reinterpret_cast<const float4 *>(x + lo);
        f.ab = *reinterpret_cast<const float4 *>(x + hi);
        f.b0 = *reinterpret_cast<const float4 *>(y + lo);
        f.b1 = *reinterpret_cast<const float4 *>(y + hi);
        fma_top(acc, f);
        fma_bottom(acc, f);
    }
}

__device__ __forceinline__ void rm_single_steps(Acc &acc, const char *sx, const char *sy, int lm, int ln)
{
#pragma unroll
    for (int r = 0; r < BM_STEP; ++r) {
        const int sw = rm_swizzle(r);
        const char *y = sy + ((ln ^ (sw & 3)) << 4);
        KFrag f;
        f.at = *reinterpret_cast<const float4 *>(sx + ((lm ^ sw) << 4) + r * 128);
        f.b0 = *reinterpret_cast<const float4 *>(y + r * 128 + (sw & 4) * 16);
        f.b1 = *reinterpret_cast<const float4 *>(y + r * 128 + 64 - (sw & 4) * 16);
        fma_top(acc, f);
    }
}

// Whether a listed k is inside the operands; row-major A and B end at K, packed A at the K blocks' end (checked build: site 37).
template <typename Params>
__device__ __forceinline__ bool k_ok(const Params &p, size_t k) { return bounds_ok(k < (size_t)p.K, p.status, 37); }

__device__ __forceinline__ void cp_async_4(uint32_t dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}

// dst <- 16 bytes at row + OFFSET
template <int OFFSET>
__device__ __forceinline__ void copy_16(uint32_t dst, const char *row)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1+%2], 16;" ::"r"(dst), "l"(row), "n"(OFFSET) : "memory");
}

// base + k * stride in one instruction (of the multiply-adds' pipe, where the compiler takes two)
__device__ __forceinline__ const char *row_of(const char *base, unsigned k, unsigned stride)
{
    const char *r;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(k), "r"(stride), "l"(base));
    return r;
}

__device__ __forceinline__ void fill_4(uint32_t dst, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(dst), "f"(v) : "memory"); }

__device__ __forceinline__ void fill_16(uint32_t dst, float v)
{
    asm volatile("st.shared.v4.f32 [%0], {%1, %1, %1, %1};" ::"r"(dst), "f"(v) : "memory");
}

// One item: blocks x0 and x0 + 1 of X (TWO) or x0 alone, times block y of Y.
// ROW_MAJOR: A is the caller's matrix instead of the k-major packed copy; 4-byte copies transpose it on the way.
// EDGE: blocks of B may be cut off by its last column, blocks of row-major A by its last row.  AGREE: X's blocks had the same patterns in
// pairs wherever samples were taken.
template <bool TWO, bool ROW_MAJOR, bool EDGE, bool AGREE, typename Params>
__device__ __forceinline__ void block_item(const Params &p, char *ring, int lane, bool wide_b, int x0, int y)
{
    LiveList l0, l1;
    l0.list = reinterpret_cast<uint16_t *>(ring + BM_SLOTS * BM_SLOT_BYTES);
    l1.list = l0.list + BM_LIST;
    // every 4 consecutive lanes touch 2 chunks of X and 2 of Y (see the tiled pipeline)
    const int half = lane >> 4, xg = (lane >> 1) & 3, yg = (lane & 1) | ((lane >> 2) & 2);   // pair: 4 x 4 lanes per block
    const int lm = (lane >> 1) & 7, ln = (lane & 1) | ((lane >> 4) << 1);                    // single block: 8 x 4 lanes
    // Copies of a pair from packed A: eight lanes per row, a lane's rows are 4 r4 .. 4 r4 + 3, so that its list entries are one load and the
    // rows of one copy instruction are whole.
    const int r4 = lane >> 3, c8 = lane & 7;
    const uint32_t dst = smem_u32(ring) + (uint32_t)(r4 * 512 + ((ROW_MAJOR ? c8 ^ rm_swizzle(r4 * 4) : c8) << 4));
    // Single blocks: four lanes per row of the stage, eight rows at a time; a lane moves the 16-byte chunks c4
    // and c4 + 4 of its row.  Rows are 128 bytes apart; odd rows have their two halves swapped, so that the eight rows of one copy
    // instruction fall on all banks.  (Fewer addresses: 100 x 6000 x 3000, single blocks only, 54.7 us so, 56.6 in the order above.)
    const int r8 = lane >> 2, c4 = lane & 3;
    const uint32_t dst0 = smem_u32(ring) + (uint32_t)(r8 * 128 + c4 * 16 + (r8 & 1) * 64), dst1 = dst0 + 64 - (r8 & 1) * 128;
    const unsigned n4 = (unsigned)p.N * 4u;                       // bytes of a row of B
    const unsigned x_stride = wide_b ? n4 : TILE_M * 4u, y_stride = wide_b ? TILE_M * 4u : n4;

    const PatternRows px = wide_b ? b_pattern(p, x0) : a_pattern<ROW_MAJOR>(p, x0);
    const PatternRows px1 = !TWO ? PatternRows{nullptr, 1} : wide_b ? b_pattern(p, x0 + 1) : a_pattern<ROW_MAJOR>(p, x0 + 1);
    const PatternRows py = wide_b ? a_pattern<ROW_MAJOR>(p, y) : b_pattern(p, y);
    // 32 floats of packed A are contiguous within a panel of 128 rows; a row of B has N floats.  Chunks of B past its
    // last column are not copied: whatever is multiplied there ends in columns of C that do not exist.
    const int a_blk = wide_b ? y : x0, b_blk = wide_b ? x0 : y;
    const char *a_src = nullptr;
    if constexpr (!ROW_MAJOR) a_src = reinterpret_cast<const char *>(p.a_packed + (size_t)(a_blk >> 2) * p.kp * TILE_M + (a_blk & 3) * 32);
    const char *b_src = reinterpret_cast<const char *>(p.B + b_blk * 32);
    const char *xs = (wide_b ? b_src : a_src) + c8 * 16, *ys = (wide_b ? a_src : b_src) + c8 * 16;
    const int b_chunks = (p.N - b_blk * 32) >> 2;
    const int x_chunks = wide_b ? b_chunks : 16, y_chunks = wide_b ? 8 : b_chunks;
    // Row-major A: the lane's k of a copy, its row within a chunk of four and where it lands.  Rows of A past its last one: one of the rows
    // before them; columns of B past its last one: others of the same row (what is multiplied there ends in rows and columns of C that do
    // not exist).
    const int a_kk = lane & (RM_KL - 1), a_rr = lane / RM_KL;
    const char *a_rows = reinterpret_cast<const char *>(p.A) + ((size_t)a_blk * 32 + a_rr) * p.K * 4;
    const char *b_rows = b_src + (!EDGE || c8 < b_chunks ? c8 * 16 : 0);
    const int b_next = c8 + 8 < b_chunks ? 128 : 0;               // from the lane's chunk of one block of B to the next block's
    const uint32_t dst_a = smem_u32(ring) + (uint32_t)(a_kk * 128 + (rm_swizzle(a_kk) << 4) + a_rr * 4);
    const unsigned k16 = (unsigned)p.K * 16u;                     // four rows
    const bool plain = p.K <= 65536 && (!EDGE || p.M >= 4);       // list entries are whole k; (EDGE) no chunk of four rows is before A
    const bool x_ok0 = c8 < x_chunks, x_ok1 = c8 + 8 < x_chunks, y_ok = c8 < y_chunks;

    Acc acc;
    acc_clear(acc);

    // The lane's pattern bits of the 128 K blocks kb0 .. (m0, m1: joint bits of either block; wy, w0, w1: the words of the
    // 128 K blocks after them, on their way) and how many quarters of them are listed already.
    int kb0 = -128, part = 0, live = 0;
    // A list that holds less than a stage gives nothing as long as more of it is to come (the other list may be full and keep it from being
    // refilled), so that a full stage's entries start at a multiple of BM_ROWS.
    int taken_mask = BM_ROWS;
    static_assert((BM_ROWS & (BM_ROWS - 1)) == 0, "mask");
    unsigned m0 = 0u, m1 = 0u, wy = 0u, w0 = 0u, w1 = 0u;
    auto load_words = [&](int kb) {
        wy = pattern_word(py, kb, p.nKB, p.pat_words, p.status) & inside_k(kb, p.K);
        w0 = pattern_word(px, kb, p.nKB, p.pat_words, p.status);
        w1 = pattern_word(px1, kb, p.nKB, p.pat_words, p.status);
    };
    auto next_words = [&]() {
        kb0 += 128;
        if (kb0 >= p.nKB) taken_mask = 2 * BM_ROWS - 1;
        part = 0;
        m0 = w0 & wy;
        m1 = w1 & wy;
        live = __reduce_add_sync(0xFFFFFFFFu, __popc(m0) | (__popc(m1) << 16));   // (both counts in one word)
        if (kb0 + 128 < p.nKB) load_words(kb0 + 128 + 4 * lane);
    };
    load_words(4 * lane);
    next_words();
    l0.made = l0.taken = l1.made = l1.taken = 0;
    bool one_list = TWO && AGREE;   // so far both blocks have the same live k: list 0 stands for both
    int wrap0 = INT_MAX, wrap1 = INT_MAX;   // (ROW_MAJOR) list positions from which on an entry is k - 65536

    // Lists further K blocks until each list holds a stage or there is no room: all 128 at once where they fit, or a
    // quarter of them (then a lane takes one byte).
    auto refill = [&]() {
        bool wrote = false;
        while (kb0 < p.nKB && (l0.pending() < BM_ROWS || (TWO && l1.pending() < BM_ROWS))) {
            const int room = BM_LIST - max(l0.pending(), l1.pending());
            unsigned a0 = m0, a1 = m1;
            int k0 = (kb0 + 4 * lane) * BK;
            if (part == 0 && max(live & 0xFFFF, live >> 16) <= room) {
                part = 4;
            } else {
                if (room < 32 * BK) break;
                const int from = part * 8 + (lane >> 2), sh = (lane & 3) * 8;
                a0 = (__shfl_sync(0xFFFFFFFFu, m0, from) >> sh) & 0xFFu;
                a1 = (__shfl_sync(0xFFFFFFFFu, m1, from) >> sh) & 0xFFu;
                k0 = (kb0 + part * 32 + lane) * BK;
                ++part;
            }
            const int c = __popc(a0) | (__popc(a1) << 16);
            const int before = exclusive_scan(c, lane);
            const int total = __shfl_sync(0xFFFFFFFFu, before + c, 31);
            if (one_list && !__all_sync(0xFFFFFFFFu, a0 == a1)) {   // from here on a list each
                one_list = false;
                __syncwarp();
                for (int i = l0.taken + lane; i < l0.made; i += 32) l1.list[i & (BM_LIST - 1)] = l0.list[i & (BM_LIST - 1)];
            }
            append_live(l0.list, l0.made + (before & 0xFFFF), l0.taken, a0, k0, p.status);
            if (TWO && !one_list) append_live(l1.list, l1.made + (before >> 16), l1.taken, a1, k0, p.status);
            if (ROW_MAJOR && k0 >= 65536 && wrap0 == INT_MAX) wrap0 = l0.made, wrap1 = l1.made;
            l0.made += total & 0xFFFF;
            l1.made += total >> 16;
            wrote = true;
            if (part == 4) next_words();
        }
        if (wrote) __syncwarp();
    };

    uint32_t slot = 0;
    int count = 0;                 // steps of the stage that is multiplied
    bool same = false;             // both blocks have the same 16 k there: Y is held once
    do {
        cp_async_wait_group<0>();
        __syncwarp();              // the stage is complete for all lanes, and the one before it read by all
        refill();
        // ---- copies of the next stage ----
        const int d0 = min(BM_ROWS, l0.pending()) & taken_mask, d1 = TWO ? min(BM_ROWS, l1.pending()) & taken_mask : 0;
        const uint32_t to = BM_SLOT_BYTES - slot;
        bool same_next = false;
        if constexpr (ROW_MAJOR) {
            auto entry = [&](int blk, int row) {
                const int pos = (blk ? l1.taken : l0.taken) + row;
                const uint16_t *list = blk && !one_list ? l1.list : l0.list;
                return (unsigned)list[pos & (BM_LIST - 1)] + (pos >= (blk && !one_list ? wrap1 : wrap0) ? 65536u : 0u);
            };
            same_next = TWO && d0 == BM_ROWS && d1 == BM_ROWS &&
                        (one_list || __all_sync(0xFFFFFFFFu, entry(0, lane & 15) == entry(1, lane & 15)));
            // A: X of either block, or Y.  RM_KL lanes on the k, four on the rows of a 16-byte chunk.
            const bool a_twice = TWO && !(wide_b && same_next), b_twice = TWO && !(!wide_b && same_next);
            const uint32_t to_a = dst_a + to + (wide_b ? 2 * BM_PART : 0), to_b = dst + to + (wide_b ? 0 : 2 * BM_PART);
            if (plain && d0 == BM_ROWS && (!TWO || d1 == BM_ROWS)) {
                auto copy_a = [&](int blk, const uint16_t *list) {
                    const int down = blk && !wide_b ? 32 : 0;
                    const char *base = a_rows + (size_t)down * p.K * 4;
                    const unsigned k0 = list[0], k1 = list[RM_KL];
                    const char *g0 = base + k0 * 4u, *g1 = base + k1 * 4u;
                    if (!k_ok(p, k0) || !k_ok(p, k1)) return;
                    const int last_q = (p.M - 1 - a_blk * 32 - down - a_rr) >> 2;   // (EDGE)
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const uint32_t e = (to_a ^ (q << 4)) + blk * BM_PART;
                        if (EDGE) {
                            const long rows = (long)min(q, last_q) * (int)k16;
                            cp_async_4(e, g0 + rows);
                            cp_async_4(e + RM_KL * 128, g1 + rows);
                        } else {
                            cp_async_4(e, row_of(g0, q, k16));
                            cp_async_4(e + RM_KL * 128, row_of(g1, q, k16));
                        }
                    }
                };
                auto copy_b = [&](int blk, const uint16_t *list, bool both) {
                    const uint2 v = *reinterpret_cast<const uint2 *>(list);
                    const char *base = b_rows + (wide_b && blk ? (EDGE ? b_next : 128) : 0);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const unsigned w = j & 2 ? v.y : v.x, k = j & 1 ? w >> 16 : w & 0xFFFFu;
                        if (!k_ok(p, k)) continue;
                        const char *g = row_of(base, k, n4);
                        const uint32_t e = (to_b ^ (rm_swizzle(j) << 4)) + j * 128 + blk * BM_PART;
                        copy_16<0>(e, g);
                        if (both) {
                            if (EDGE) copy_16<0>(e + BM_PART, g + b_next);
                            else copy_16<128>(e + BM_PART, g);
                        }
                    }
                };
                // (One body for both lists: its instructions, not their number, are what the loop has too many of.  Unrolled, 32-granular
                // 0.5 / 0.5, 2048^3: 171 us instead of 154.  Edges in this code for every launch: 4096^3 64-granular 850 instead of 811.)
                const uint16_t *list0 = l0.list + (l0.taken & (BM_LIST - 1)), *list1 = one_list ? list0 : l1.list + (l1.taken & (BM_LIST - 1));

                if (TWO && wide_b && same_next) {
                    copy_a(0, list0 + a_kk);
                    copy_b(0, list0 + r4 * 4, true);
                } else {
#pragma unroll 1
                    for (int blk = 0; blk < (TWO ? 2 : 1); ++blk) {
                        const uint16_t *list = blk ? list1 : list0;
                        copy_a(blk, list + a_kk);
                        if (!blk || b_twice) copy_b(blk, list + r4 * 4, false);
                    }
                }
            } else if (max(d0, d1) > 0) {
                // Past the end of a list X = -0 and Y = +0 (below).  Rows past the end of A: any row, what is multiplied there ends in
                // rows of C that do not exist.
#pragma unroll 1
                for (int i = 0; i < (a_twice ? 4 : 2); ++i) {
                    const int blk = i >> 1, row = (i & 1) * RM_KL + a_kk, row0 = (a_blk + (wide_b ? 0 : blk)) * 32 + a_rr;
                    const bool listed = row < (blk ? d1 : d0);
                    const unsigned k = listed ? entry(blk, row) : 0u;
                    if (listed && !k_ok(p, k)) continue;
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const uint32_t e = (to_a ^ (q << 4)) + (i & 1) * (RM_KL * 128) + blk * BM_PART;
                        if (listed) cp_async_4(e, p.A + (size_t)min(row0 + 4 * q, p.M - 1) * p.K + k);
                        else fill_4(e, wide_b ? 0.0f : -0.0f);
                    }
                }
#pragma unroll 1
                for (int i = 0; i < (b_twice ? 8 : 4); ++i) {
                    const int blk = i >> 2, j = i & 3, row = r4 * 4 + j;
                    const uint32_t e = (to_b ^ (rm_swizzle(j) << 4)) + j * 128 + blk * BM_PART;
                    if (row < (blk ? d1 : d0)) {
                        const size_t k = entry(blk, row);
                        if (k_ok(p, k) && c8 + (wide_b ? blk * 8 : 0) < b_chunks) copy_16<0>(e, b_rows + (wide_b ? blk * 128 : 0) + k * n4);
                    } else {
                        fill_16(e, wide_b ? -0.0f : 0.0f);
                    }
                }
            }
        } else {
            if (!TWO && d0 == BM_ROWS) {
                const uint16_t *entry = l0.list + (l0.taken & (BM_LIST - 1)) + r8;
                const unsigned k[2] = {entry[0], entry[8]};
                const char *xs4 = xs - c8 * 16 + c4 * 16, *ys4 = ys - c8 * 16 + c4 * 16;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (!k_ok(p, k[h])) continue;
                    const char *gx = row_of(xs4, k[h], x_stride), *gy = row_of(ys4, k[h], y_stride);
                    const uint32_t e0 = dst0 + to + h * 1024, e1 = dst1 + to + h * 1024;
                    if (!EDGE || c4 < x_chunks) copy_16<0>(e0, gx);
                    if (!EDGE || c4 + 4 < x_chunks) copy_16<64>(e1, gx);
                    if (!EDGE || c4 < y_chunks) copy_16<0>(e0 + 2 * BM_PART, gy);
                    if (!EDGE || c4 + 4 < y_chunks) copy_16<64>(e1 + 2 * BM_PART, gy);
                }
            } else if (TWO && d0 == BM_ROWS && d1 == BM_ROWS) {
                const uint2 v0 = *reinterpret_cast<const uint2 *>(l0.list + (l0.taken & (BM_LIST - 1)) + r4 * 4);
                uint2 v1 = v0;
                same_next = true;
                if (!one_list) {
                    v1 = *reinterpret_cast<const uint2 *>(l1.list + (l1.taken & (BM_LIST - 1)) + r4 * 4);
                    same_next = __all_sync(0xFFFFFFFFu, v0.x == v1.x && v0.y == v1.y);
                }
                if (same_next) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const unsigned w0 = j & 2 ? v0.y : v0.x, k0 = j & 1 ? w0 >> 16 : w0 & 0xFFFFu;
                        const uint32_t e = dst + to + j * 128;
                        if (!k_ok(p, k0)) continue;
                        const char *gx = row_of(xs, k0, x_stride), *gy = row_of(ys, k0, y_stride);
                        if (!EDGE || x_ok0) copy_16<0>(e, gx);
                        if (!EDGE || y_ok) copy_16<0>(e + 2 * BM_PART, gy);
                        if (!EDGE || x_ok1) copy_16<128>(e + BM_PART, gx);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const unsigned w0 = j & 2 ? v0.y : v0.x, w1 = j & 2 ? v1.y : v1.x;
                        const unsigned k0 = j & 1 ? w0 >> 16 : w0 & 0xFFFFu, k1 = j & 1 ? w1 >> 16 : w1 & 0xFFFFu;
                        const uint32_t e = dst + to + j * 128;
                        if (!k_ok(p, k0) || !k_ok(p, k1)) continue;
                        if (!EDGE || x_ok0) copy_16<0>(e, row_of(xs, k0, x_stride));
                        if (!EDGE || y_ok) copy_16<0>(e + 2 * BM_PART, row_of(ys, k0, y_stride));
                        if (!EDGE || x_ok1) copy_16<128>(e + BM_PART, row_of(xs, k1, x_stride));
                        if (!EDGE || y_ok) copy_16<0>(e + 3 * BM_PART, row_of(ys, k1, y_stride));
                    }
                }
            } else if (max(d0, d1) > 0) {
                // Past the end of a list X = -0 and Y = +0: a multiply-add with them changes no accumulator, not even a zero's sign.
#pragma unroll 1
                for (int i = 0; i < (TWO ? 8 : 4); ++i) {      // (row of four, block)
                    const int j = i & 3, row = r4 * 4 + j, blk = TWO ? i >> 2 : 0;
                    const uint32_t e = (TWO || !(row & 1) ? dst : dst ^ 64u) + to + j * 128 + blk * BM_PART;
                    if (row < (blk ? d1 : d0)) {
                        const size_t k = blk && !one_list ? l1.list[(l1.taken + row) & (BM_LIST - 1)] : l0.list[(l0.taken + row) & (BM_LIST - 1)];
                        if (!k_ok(p, k)) continue;
                        if (blk ? x_ok1 : x_ok0) copy_16<0>(e, xs + k * x_stride + blk * 128);
                        if (y_ok) copy_16<0>(e + 2 * BM_PART, ys + k * y_stride);
                    } else {
                        fill_16(e, -0.0f);
                        fill_16(e + 2 * BM_PART, 0.0f);
                    }
                }
            }
        }
        l0.taken += d0;
        l1.taken += d1;
        cp_async_commit();
        // ---- the stage itself ----
        const char *st = ring + slot;
        if (ROW_MAJOR) {
            const char *sx = st + (TWO ? half * BM_PART : 0), *sy = st + (TWO && !same ? 2 + half : 2) * BM_PART;
#pragma unroll 1
            for (int r = 0; r < count; r += BM_STEP) {
                if (TWO) rm_pair_steps(acc, sx + r * 128, sy + r * 128, xg, yg);
                else rm_single_steps(acc, sx + r * 128, sy + r * 128, lm, ln);
            }
        } else if (TWO) {
            const char *sx = st + half * BM_PART + xg * 16, *sy = st + (same ? 2 : 2 + half) * BM_PART + yg * 16;
#pragma unroll 1
            for (int r = 0; r < count; r += BM_STEP) pair_steps(acc, sx + r * 128, sy + r * 128);
        } else {
            const char *sx = st + lm * 16, *sx_odd = st + (lm ^ 4) * 16, *sy = st + 2 * BM_PART + ln * 16;
#pragma unroll 1
            for (int r = 0; r < count; r += BM_STEP) single_steps(acc, sx + r * 128, sx_odd + r * 128, sy + r * 128);
        }
        count = max(d0, d1);
        same = same_next;
        slot = to;
    } while (count > 0);

    // ---- C is overwritten (beta = 0) ----
    // x values 4 * xv .. + 3 and, in a pair, + 16; y values 4 * yv .. + 3 and + 16, of block xb
    const size_t c_floats = (size_t)p.M * p.N;
    const int xb = x0 + (TWO ? half : 0), xv = TWO ? xg : lm, yv = TWO ? yg : ln;
#pragma unroll
    for (int q = 0; q < 2; ++q) {                       // the two groups of 4 x values
        if (q == 1 && !TWO) break;
        if (!wide_b) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int row = xb * 32 + q * 16 + xv * 4 + i, col = y * 32 + yv * 4;
                float v8[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) v8[j] = acc_get(acc, 2 * q + (i >> 1), i & 1, j);
                const size_t off = (size_t)row * p.N + col;
                if (row < p.M && col < p.N && bounds_ok(off + 4 <= c_floats, p.status, 29))
                    *reinterpret_cast<float4 *>(p.C + off) = make_float4(v8[0], v8[1], v8[2], v8[3]);
                if (row < p.M && col + 16 < p.N && bounds_ok(off + 20 <= c_floats, p.status, 29))
                    *reinterpret_cast<float4 *>(p.C + off + 16) = make_float4(v8[4], v8[5], v8[6], v8[7]);
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int row = y * 32 + yv * 4 + (j & 3) + 16 * (j >> 2), col = xb * 32 + q * 16 + xv * 4;
                const size_t off = (size_t)row * p.N + col;
                if (row < p.M && col < p.N && bounds_ok(off + 4 <= c_floats, p.status, 29))
                    *reinterpret_cast<float4 *>(p.C + off) =
                        make_float4(acc_get(acc, 2 * q, 0, j), acc_get(acc, 2 * q, 1, j), acc_get(acc, 2 * q + 1, 0, j), acc_get(acc, 2 * q + 1, 1, j));
            }
        }
    }
}

// All of a warp's share of block mode.  smem: the CTA's dynamic shared memory; next: the CTA's item counter (initially
// BM_WARPS: a warp's first item is its own number).
template <bool ROW_MAJOR, bool EDGE, bool AGREE, typename Params>
__device__ __forceinline__ void block_mode(const Params &p, char *smem, int warp, int lane, bool wide_b, int *next)
{
    char *ring = smem + warp * BM_WARP_BYTES;
    // X spans pairs of blocks, Y single ones
    const int x_blocks = wide_b ? p.b_rows : p.a_rows, y_blocks = wide_b ? p.a_rows : p.b_rows;
    const int pairs_x = (x_blocks + 1) >> 1;
    const int tiles_m = wide_b ? y_blocks : pairs_x, tiles_n = wide_b ? pairs_x : y_blocks;
    const long items = (long)tiles_m * tiles_n;
    const int mine = blockIdx.x < items ? (int)((items - 1 - blockIdx.x) / gridDim.x) + 1 : 0;
    const int tail = block_tail(mine), whole = mine - tail;   // the last `tail` items go as two single blocks each

    for (int v = warp; v < whole + 2 * tail;) {
        const int item = blockIdx.x + (v < whole ? v : whole + ((v - whole) >> 1)) * gridDim.x;
        int tm, tn;
        tile_coords(item, tiles_m, tiles_n, tm, tn, wide_b ? 32 : 16);
        const int y = wide_b ? tm : tn, x0 = 2 * (wide_b ? tn : tm) + (v < whole ? 0 : (v - whole) & 1);
        if (v < whole && x0 + 1 < x_blocks) block_item<true, ROW_MAJOR, EDGE, AGREE>(p, ring, lane, wide_b, x0, y);
        else if (x0 < x_blocks) block_item<false, ROW_MAJOR, EDGE, AGREE>(p, ring, lane, wide_b, x0, y);
        int nx = 0;
        if (lane == 0) nx = atomicAdd(next, 1);
        v = __shfl_sync(0xFFFFFFFFu, nx, 0);
    }
    cp_async_wait_group<0>();
}

}  // namespace esmm
