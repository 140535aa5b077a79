// Joint-sparse FP32 SGEMM for sm_100a, few rows: the strip kernel, for M <= 32 (one 32-row pattern block of A) and for problems of a
// few row blocks that have too few tiles for the GPU.
//
// Same arithmetic as the packed kernel (esmm_gemm_tiled.cuh) and as esmm_ab_optimized_v3 of the reference
// (src/kernels/esmm_ab_optimized_v3.cu:157, 183-203): for every output one FMA chain in ascending k over the k whose joint bit is set.
// With a single row block of A the large kernel has M / 128 x N / 128 = N / 128 tiles, runs half of its consumer warps on rows that do
// not exist and leaves a third of the SMs idle (N = 11008: 86 tiles).  Here the work is cut the other way:
//
//   * one CTA per row block and 32-column strip of C (N / 32 of them per row block, several resident per SM).  That is exactly one
//     pattern block of A and one of B, so its live k are a_pat[rb][kb] & b_pat[strip][kb]: every listed row is live for the whole CTA,
//     there are no per-warp masks and no index lists in the inner loop;
//   * all threads first build the strip's list of live k (pattern bytes read as 32-bit words); then stages of 64 k travel through a
//     ring of four (three or two, where K is long and an SM has room for more strips so) as 16-byte asynchronous copies: per k 128
//     bytes of B and 32, 64 or 128 bytes of packed A (8, 16 or 32 of the block's rows: as many as M needs);
//   * two warps copy, a stage each in turn, two or four multiply.  A stage's barrier takes an arrival of every copying lane when its
//     copies have landed (cp.async.mbarrier.arrive.noinc); the multiplying warps hand the slot back.  No warp does both: copies in the
//     multiplying warps' own instruction stream, with a barrier of the whole CTA per 32 k, were what the kernel before spent most of
//     its time on (the first call below: FMA pipe 22 % active);
//   * a multiplying thread holds 4 x 4, 4 x 2 or 2 x 2 outputs as row pairs times one broadcast column.  The operands of four k are
//     loaded (volatile, so that they stay put) one batch ahead of the multiply-adds that use them, two register sets in ping-pong,
//     over the stages' borders too;
//   * the multiplying warps of an SM's strips lie on different SM sub-partitions.  The hardware starts a CTA's first warp on any of
//     the four, so a CTA with two multiplying warps takes its turn from a counter per SM and places them by its own %warpid (without:
//     K = 4096 dense, 32 rows, three and four strips per SM 13-20 % slower on average and up to twice as long where all fall
//     together).
//
// What bounds it: a multiplying warp is alone or nearly so on its SM sub-partition, so its loads' issue and its multiply-adds add up:
// 13 cycles a k for 4 x 2 outputs (8 of multiply-adds) with no copies and no barriers at all, 15 with them; on SMs with three or more
// strips shared memory (10 of its wavefronts per strip of 32 rows and k, 7.5 of 16).  Measured, whole calls, the kernel before -> this
// one: M = 16, N = 11008, K = 4096 pruned MLP (819 live k per strip, 344 strips) 28.5 -> 19.0 us; M = 8 28.4 -> 14.5; M = 1 19.4 ->
// 9.7; M = 32 34.1 -> 27.3; dense, N = 4096, K = 4096, M = 16 61.5 -> 33.5; dense, N = 11008, M = 1 100.5 -> 47.4; N = 512, K =
// 16384, M = 6 148 -> 70.  Also measured: stages of 32 k 10-20 % slower, of 128 in a ring of two as fast, k of a batch 2 or 8 and
// three batches ahead as fast, counters in shared memory with release / acquire instead of barriers 3-5 % slower; lanes past B's last
// column that all copy the matrix's first bytes instead of others of their row: N = 300, 32 row blocks 118 us instead of 61. Every
// wait is bounded: a wait that runs out raises the abort flag, nothing is stored and the status word tells.
#include <algorithm>
#include <cstring>
#include <mutex>

#include "esmm_gemm_shared.cuh"

namespace esmm {

constexpr int SK_COLS = 32;                     // columns of a strip = one B pattern block
constexpr int SK_ROWS = 32;                     // rows of a row block = one A pattern block
constexpr int SK_STAGE_ROWS = 64;               // k per stage
constexpr int SK_ROW_BYTES = 128;               // one k of B in shared memory
constexpr int SK_MAX_STAGES = 4;                // of the ring; two at least
constexpr int SK_MAX_KP = 16384;                // longest K the row list is sized for
constexpr int SK_COPY_WARPS = 2;                // warps that copy
constexpr int SK_BATCH = 4;                     // k per register set of operands
constexpr int SK_SETS = 2;                      // register sets

// Whose turn it is, per SM: the CTAs of two multiplying warps that an SM gets one after the other have them on different SM
// sub-partitions.  (A hint: whatever the counters hold, every CTA has its two.)
constexpr int SK_TURNS = 256;
__device__ unsigned g_sk_turn[SK_TURNS];

struct SkinnyParams {
    int M, N, K, nKB, kp, cap;
    int row_blocks, stages;
    const uint8_t *a_pat;
    const uint8_t *b_pat;
    const float *a_packed;  // [panel][k][128]: a quarter of a panel's rows are read
    const float *B;
    float *C;
    int *status;
};

// bits of the k of K blocks kb .. kb + 3 that are < K (a pattern may mark more of a ragged last K block live: there is no B for them)
__device__ __forceinline__ unsigned sk_inside(int kb, int K)
{
    const int left = K - kb * BK;
    return left >= 32 ? 0xFFFFFFFFu : left <= 0 ? 0u : (1u << left) - 1u;
}

__device__ __forceinline__ int sk_scan(int v, int lane)
{
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(0xFFFFFFFFu, v, d);
        if (lane >= d) v += t;
    }
    return v;
}

__device__ __forceinline__ void sk_copy_16(uint32_t dst, const char *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// (one group of copies per stage and lane)
__device__ __forceinline__ void sk_copies_arrive(uint32_t bar)
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void mbar_arrive_if(uint32_t bar, bool on)
{
    asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %1, 0;\n@p mbarrier.arrive.shared::cta.b64 _, [%0];\n}" ::"r"(bar), "r"((int)on) : "memory");
}

// Shared memory: ring | list (u16 x cap) | warp sums | full and empty barriers, abort flag
__host__ __device__ constexpr int sk_stage_bytes(int rows) { return SK_STAGE_ROWS * (rows * 4 + SK_ROW_BYTES); }
__host__ __device__ constexpr size_t sk_sum_off(int rows, int stages, int cap)
{
    return (size_t)stages * sk_stage_bytes(rows) + (((size_t)cap * 2 + 15) & ~(size_t)15);
}
__host__ __device__ constexpr size_t sk_smem(int rows, int stages, int cap)
{
    return sk_sum_off(rows, stages, cap) + 32 + 2 * SK_MAX_STAGES * 8 + 16;
}

// ROWS: rows of C that are fetched and multiplied, 8, 16 or 32.  CW: warps that multiply.  RT: rows per thread.
template <int ROWS, int CW, int RT>
__global__ void __launch_bounds__((CW + SK_COPY_WARPS) * 32)
esmm_joint_sgemm_skinny_kernel(const SkinnyParams p)
{
    constexpr int A_ROW_BYTES = ROWS * 4;                           // one k of A in shared memory
    constexpr int A_HALF = SK_STAGE_ROWS * A_ROW_BYTES;             // A rows, then B rows
    constexpr int STAGE_BYTES = sk_stage_bytes(ROWS);
    constexpr int SK_WARPS = CW + SK_COPY_WARPS, SK_THREADS = SK_WARPS * 32;
    static_assert(SK_WARPS < 8 && (CW == 2 ? SK_WARPS == 4 : CW == 4), "warp sums; roles");
    extern __shared__ __align__(1024) char smem[];
    uint16_t *krow = reinterpret_cast<uint16_t *>(smem + (size_t)p.stages * STAGE_BYTES);
    char *rest = smem + sk_sum_off(ROWS, p.stages, p.cap);
    volatile int *wsum = reinterpret_cast<volatile int *>(rest);
    const uint32_t full0 = smem_u32(rest + 32), empty0 = full0 + SK_MAX_STAGES * 8;
    volatile int *abort_flag = reinterpret_cast<volatile int *>(rest + 32 + 2 * SK_MAX_STAGES * 8);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int strip = blockIdx.x / p.row_blocks, rb = blockIdx.x - strip * p.row_blocks;
    const uint8_t *a_pat = p.a_pat + (size_t)rb * p.nKB;
    if (threadIdx.x == 0) {
        for (int s = 0; s < SK_MAX_STAGES; ++s) {
            mbar_init(full0 + 8 * s, 32);         // a copying warp's lanes, when their copies have landed
            mbar_init(empty0 + 8 * s, CW);
        }
        *abort_flag = 0;
        if (CW == 2) {
            unsigned sm, slot;
            asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
            asm volatile("mov.u32 %0, %%warpid;" : "=r"(slot));
            wsum[SK_WARPS] = (int)(slot + 2u * atomicAdd(&g_sk_turn[sm % SK_TURNS], 1u)) & 3;
        }
    }
    grid_dependency_wait();   // (the A patterns and the packed copy come from the kernel before this one)

    int n = 0;
    // ---------------- the strip's list of live k ----------------
    // Thread t owns the K blocks t * per .. t * per + per - 1 (consecutive threads, ascending k; per a multiple
    // of 4 so that a thread's pattern bytes are whole 32-bit words where the arrays allow): count, prefix over
    // the CTA, write.
    {
        constexpr int MAX_WORDS = ((SK_MAX_KP / BK + SK_THREADS - 1) / SK_THREADS + 3) / 4;   // 4 words of 4 K blocks per thread at most
        const uint8_t *bp = p.b_pat + (size_t)strip * p.nKB;
        const int per = ((p.nKB + SK_THREADS - 1) / SK_THREADS + 3) & ~3;
        const int kb_lo = min((int)threadIdx.x * per, p.nKB), kb_hi = min(kb_lo + per, p.nKB);
        const bool words = (p.nKB & 3) == 0 && ((reinterpret_cast<uintptr_t>(a_pat) | reinterpret_cast<uintptr_t>(bp)) & 3) == 0;
        unsigned live[MAX_WORDS];
        int c = 0;
#pragma unroll
        for (int w = 0; w < MAX_WORDS; ++w) {
            const int kb = kb_lo + 4 * w;
            unsigned v = 0u;
            if (kb < kb_hi) {
                if (words) {
                    v = *reinterpret_cast<const unsigned *>(a_pat + kb) & *reinterpret_cast<const unsigned *>(bp + kb);
                } else {
                    for (int j = 0; j < 4 && kb + j < kb_hi; ++j) v |= (unsigned)(a_pat[kb + j] & bp[kb + j]) << (8 * j);
                }
            }
            v &= sk_inside(kb, p.K);
            live[w] = v;
            c += __popc(v);
        }
        const int incl = sk_scan(c, lane);
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        int q = incl - c;
#pragma unroll
        for (int w = 0; w < SK_WARPS; ++w) {
            if (w < warp) q += wsum[w];
            n += wsum[w];
        }
#pragma unroll
        for (int w = 0; w < MAX_WORDS; ++w) {
            unsigned v = live[w];
            int e = q + __popc(v);
            const int k0 = (kb_lo + 4 * w) * BK, qn = e;
            while (v) {                                              // from both ends of the word
                const int lo = __ffs((int)v) - 1, hi = 31 - __clz((int)v);   // bit 8 j + kk: K block kb_lo + 4 w + j, offset kk
                --e;
                if (bounds_ok(q < p.cap, p.status, 30)) krow[q] = (uint16_t)(k0 + lo);   // checked build: site 30
                if (bounds_ok(e < p.cap, p.status, 30)) krow[e] = (uint16_t)(k0 + hi);
                ++q;
                v &= ~((1u << lo) | (1u << hi));
            }
            q = qn;
        }
        __syncthreads();
    }
    const int num_stages = (n + SK_STAGE_ROWS - 1) / SK_STAGE_ROWS;
    const int col0 = strip * SK_COLS;
    // the warps' roles: strips that share an SM have their multiplying warps on different SM sub-partitions
    const int role = CW == 2 ? (warp + wsum[SK_WARPS]) & 3 : warp;
    bool ok = true;

    if (role < CW) {
        // ---------------- multiplying warps: WROWS rows x WCOLS columns each, 4 rows x CT columns per thread ----------------
        constexpr int WROWS = ROWS < 16 ? ROWS : 16, ROW_SPLIT = ROWS / WROWS, WCOLS = SK_COLS * ROW_SPLIT / CW;
        constexpr int RG = WROWS / RT, CG = 32 / RG, CT = WCOLS / CG;     // groups of lanes on the rows, on the columns
        static_assert(CT == 2 || CT == 4, "columns per thread");
        static_assert(RT == 2 || RT == 4, "rows per thread");
        // every 4 consecutive lanes touch 2 row groups x 2 column groups (few distinct bytes per load)
        const int rg = RG == 4 ? ((lane >> 1) & 1) | ((lane >> 4) << 1) : ((lane >> 1) & 1) | ((lane >> 3) << 1);
        const int cg = RG == 4 ? (lane & 1) | (((lane >> 2) & 3) << 1) : (lane & 1) | (((lane >> 2) & 1) << 1);
        static_assert(RG == 4 || RG == 8, "lanes");
        const int row0 = (role % ROW_SPLIT) * WROWS + rg * RT, colw = (role / ROW_SPLIT) * WCOLS + cg * CT;
        const uint32_t tA = smem_u32(smem) + row0 * 4, tB = smem_u32(smem) + A_HALF + colw * 4;
        // c[pr][j] = rows 2 pr, 2 pr + 1 of column j
        float2 c[RT / 2][CT];
#pragma unroll
        for (int i = 0; i < RT / 2; ++i)
#pragma unroll
            for (int j = 0; j < CT; ++j) c[i][j] = make_float2(0.0f, 0.0f);

        // Operands of SK_BATCH consecutive k of a stage.  The next batch is loaded before the current one is multiplied (two
        // register sets, ping-pong), across the stages' borders too, so that a load has a whole batch of multiply-adds to land
        // under; the loads are volatile so that they stay where they are written.
        struct Ops {
            float2 a[SK_BATCH][RT / 2];
            float b[SK_BATCH][CT];
        };
        auto load_rows = [&](Ops &o, uint32_t s_off, int r) {
#pragma unroll
            for (int i = 0; i < SK_BATCH; ++i) {
                const uint32_t pa = tA + s_off + (uint32_t)((r + i) * A_ROW_BYTES), pb = tB + s_off + (uint32_t)((r + i) * SK_ROW_BYTES);
                if constexpr (RT == 4)
                    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                                 : "=f"(o.a[i][0].x), "=f"(o.a[i][0].y), "=f"(o.a[i][RT / 2 - 1].x), "=f"(o.a[i][RT / 2 - 1].y) : "r"(pa));
                else
                    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(o.a[i][0].x), "=f"(o.a[i][0].y) : "r"(pa));
                if constexpr (CT == 4)
                    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                                 : "=f"(o.b[i][0]), "=f"(o.b[i][1]), "=f"(o.b[i][2]), "=f"(o.b[i][3]) : "r"(pb));
                else
                    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(o.b[i][0]), "=f"(o.b[i][1]) : "r"(pb));
            }
        };
        auto fma_rows = [&](const Ops &o, int count) {
#pragma unroll
            for (int i = 0; i < SK_BATCH; ++i)
                if (i < count) {
#pragma unroll
                    for (int pr = 0; pr < RT / 2; ++pr)
#pragma unroll
                        for (int j = 0; j < CT; ++j) c[pr][j] = __ffma2_rn(o.a[i][pr], make_float2(o.b[i][j], o.b[i][j]), c[pr][j]);
                }
        };

        constexpr int BATCHES = SK_STAGE_ROWS / SK_BATCH, AHEAD = SK_SETS - 1;
        static_assert(BATCHES % SK_SETS == 0, "a stage's first batch is in set 0");
        Ops o[SK_SETS];
        if (num_stages > 0) {
            ok = mbar_wait(full0, 0, abort_flag);
            if (ok) {
#pragma unroll
                for (int b = 0; b < AHEAD; ++b) load_rows(o[b], 0, b * SK_BATCH);
            }
        }
        // (after a wait that ran out the sums are worthless and not stored; the loop goes on, as the waits no longer do)
        int slot = 0;
        uint32_t phase = 0u;
        for (int s = 0; s < num_stages; ++s) {
            const int cnt = n - s * SK_STAGE_ROWS;
            const uint32_t s_off = (uint32_t)slot * STAGE_BYTES;
            if (cnt > SK_STAGE_ROWS) {
                const bool wrap = slot + 1 == p.stages;
                const int next = wrap ? 0 : slot + 1;
                const uint32_t next_bar = full0 + 8 * next, next_phase = phase ^ (wrap ? 1u : 0u);
                bool ready = false;
#pragma unroll
                for (int b = 0; b < BATCHES; ++b) {
                    if (b + AHEAD < BATCHES) {
                        load_rows(o[(b + AHEAD) % SK_SETS], s_off, (b + AHEAD) * SK_BATCH);
                    } else {
                        if (b + AHEAD == BATCHES && !ready) ok = ok && mbar_wait(next_bar, next_phase, abort_flag);
                        load_rows(o[(b + AHEAD) % SK_SETS], (uint32_t)next * STAGE_BYTES, (b + AHEAD - BATCHES) * SK_BATCH);
                    }
                    if (b == BATCHES - 4) ready = mbar_test_wait(next_bar, next_phase);   // (its answer comes under the multiply-adds)
                    fma_rows(o[b % SK_SETS], SK_BATCH);
                }
                __syncwarp();
                mbar_arrive_if(empty0 + 8 * slot, lane == 0);
                slot = next;
                phase = next_phase;
            } else {
                // the last stage (batches loaded past its last row are in bounds and never multiplied)
#pragma unroll
                for (int b = 0; b < BATCHES; ++b) {
                    if (b * SK_BATCH >= cnt) break;
                    if (b + AHEAD < BATCHES) load_rows(o[(b + AHEAD) % SK_SETS], s_off, (b + AHEAD) * SK_BATCH);
                    fma_rows(o[b % SK_SETS], cnt - b * SK_BATCH);
                }
            }
        }
        // C is overwritten (beta = 0)
        const int col = col0 + colw;
#pragma unroll
        for (int e = 0; e < RT; ++e) {
            const int r = rb * SK_ROWS + row0 + e;
            float v[CT];
#pragma unroll
            for (int j = 0; j < CT; ++j) v[j] = (e & 1) ? c[e >> 1][j].y : c[e >> 1][j].x;
            if (ok && r < p.M && col < p.N && bounds_ok((size_t)r * p.N + col + CT <= (size_t)p.M * p.N, p.status, 33)) {
                float *dst = p.C + (size_t)r * p.N + col;
                if constexpr (CT == 4) *reinterpret_cast<float4 *>(dst) = make_float4(v[0], v[1], v[2], v[3]);
                else *reinterpret_cast<float2 *>(dst) = make_float2(v[0], v[1]);
            }
        }
    } else {
        // ---------------- copies: a warp takes every other stage ----------------
        // 32 rows at a time.  B: 8 lanes per row, 4 rows an instruction, rows 8 apart, so that a lane's 8 list entries are one load;
        // A likewise.  (Rows of 128 bytes are too short for the tensor copy engine: about 57 cycles of issue per copy and warp.)
        constexpr int A_LANES = ROWS / 4, A_N = A_LANES;            // lanes per row of A; instructions per 32 rows
        const int b_row = (lane >> 3) * 8, b_chunk = lane & 7;
        const int a_row = lane / A_LANES * A_N, a_chunk = lane % A_LANES;
        // (columns past B's last one: another chunk of the same row; what is multiplied there is not stored)
        const char *b_src = reinterpret_cast<const char *>(p.B + col0 + (col0 + b_chunk * 4 < p.N ? b_chunk * 4 : 0));
        const char *a_src = reinterpret_cast<const char *>(p.a_packed + (size_t)(rb >> 2) * p.kp * TILE_M + (rb & 3) * 32 + a_chunk * 4);
        const unsigned n4 = (unsigned)p.N * 4u;
        const uint32_t dst_a = smem_u32(smem) + (uint32_t)(a_row * A_ROW_BYTES + a_chunk * 16);
        const uint32_t dst_b = smem_u32(smem) + (uint32_t)(A_HALF + b_row * SK_ROW_BYTES + b_chunk * 16);
        int slot = role - CW;
        uint32_t phase = 1u;                                        // of the slot's empty barrier that the warp waits for
        static_assert(SK_COPY_WARPS <= 2, "a warp's first slot and its steps along the ring");
        int s = role - CW;
        for (; (s + 1) * SK_STAGE_ROWS <= n; s += SK_COPY_WARPS, slot += SK_COPY_WARPS) {
            if (slot >= p.stages) {
                slot -= p.stages;
                phase ^= 1u;
            }
            if (!bounds_ok((s + 1) * SK_STAGE_ROWS <= p.cap, p.status, 31)) break;
            ok = mbar_wait(empty0 + 8 * slot, phase, abort_flag);
            if (!ok) break;
#pragma unroll
            for (int h = 0; h < SK_STAGE_ROWS / 32; ++h) {
                const uint32_t s_off = (uint32_t)slot * STAGE_BYTES;
                const uint16_t *list = krow + s * SK_STAGE_ROWS + h * 32;
                const uint4 bk = *reinterpret_cast<const uint4 *>(list + b_row);
                unsigned ka[8];
                const unsigned kb[8] = {bk.x & 0xFFFFu, bk.x >> 16, bk.y & 0xFFFFu, bk.y >> 16, bk.z & 0xFFFFu, bk.z >> 16, bk.w & 0xFFFFu, bk.w >> 16};
                if (A_N == 8) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) ka[j] = kb[j];
                } else if (A_N == 4) {
                    const uint2 v = *reinterpret_cast<const uint2 *>(list + a_row);
                    ka[0] = v.x & 0xFFFFu, ka[1] = v.x >> 16, ka[2] = v.y & 0xFFFFu, ka[3] = v.y >> 16;
                } else {
                    const unsigned v = *reinterpret_cast<const unsigned *>(list + a_row);
                    ka[0] = v & 0xFFFFu, ka[1] = v >> 16;
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    if (!bounds_ok(kb[j] < (unsigned)p.K, p.status, 32)) continue;   // site 32: a k outside B / the packed panel
                    sk_copy_16(dst_b + s_off + (h * 32 + j) * SK_ROW_BYTES, b_src + (size_t)kb[j] * n4);
                }
#pragma unroll
                for (int j = 0; j < A_N; ++j) {
                    if (!bounds_ok(ka[j] < (unsigned)p.kp, p.status, 32)) continue;
                    sk_copy_16(dst_a + s_off + (h * 32 + j) * A_ROW_BYTES, a_src + (size_t)ka[j] * (TILE_M * 4));
                }
            }
            sk_copies_arrive(full0 + 8 * slot);
        }
        // The list's end: its rows and no others.  Rows to fill the stage, which nothing multiplies, were the same one of A for all strips
        // of a row block, which queued for it in L2 (whole stages / the listed rows only, us, product alone: 16 x 11008 x 128 with a quarter
        // of A's and of B's k live 6.6 / 2.9, 1 x 16000 x 256 likewise 7.6 / 2.9, 33 x 8192 x 8 dense 8.4 / 3.2).
        // For 8 and 16 rows as a whole stage is copied (in the other form, a loop, lists of one stage take 0.7 us longer), for 32 a loop.  What
        // the compiler makes of the loops over whole stages, here and above, depends on this part and on its place: so, and after the
        // multiplying warps' code, nothing is slower than without it (128 x 4096 x 4096 dense 101.3 us, 102.7 without it, 101 to 121 in nine
        // other forms and places; one strip of 48 k 3.1 and 3.1).
        const int left = n - s * SK_STAGE_ROWS;
        if (ok && left > 0) {
            if (slot >= p.stages) {
                slot -= p.stages;
                phase ^= 1u;
            }
            ok = mbar_wait(empty0 + 8 * slot, phase, abort_flag);
            const uint32_t s_off = (uint32_t)slot * STAGE_BYTES;
            if constexpr (ROWS < 32) {
#pragma unroll 2
                for (int h = 0; h < SK_STAGE_ROWS / 32; ++h) {
                    if (!ok || h * 32 >= left) break;
                    const uint16_t *list = krow + s * SK_STAGE_ROWS + h * 32;
                    const uint4 bk = *reinterpret_cast<const uint4 *>(list + b_row);
                    const unsigned kb[8] = {bk.x & 0xFFFFu, bk.x >> 16, bk.y & 0xFFFFu, bk.y >> 16, bk.z & 0xFFFFu, bk.z >> 16, bk.w & 0xFFFFu, bk.w >> 16};
                    const int b_left = left - h * 32 - b_row, a_left = left - h * 32 - a_row;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        if (j >= b_left || !bounds_ok(kb[j] < (unsigned)p.K, p.status, 32)) continue;
                        sk_copy_16(dst_b + s_off + (h * 32 + j) * SK_ROW_BYTES, b_src + (size_t)kb[j] * n4);
                    }
#pragma unroll
                    for (int j = 0; j < A_N; ++j) {
                        const unsigned k = list[a_row + j];
                        if (j >= a_left || !bounds_ok(k < (unsigned)p.kp, p.status, 32)) continue;
                        sk_copy_16(dst_a + s_off + (h * 32 + j) * A_ROW_BYTES, a_src + (size_t)k * (TILE_M * 4));
                    }
                }
            } else {
                const uint32_t to = smem_u32(smem) + s_off + b_chunk * 16;   // (a row of A is as long as one of B)
#pragma unroll (CW == 4 ? 1 : 2)
                for (int r = (lane >> 3) * 4; ok && r < left; r += 16) {
                    const uint2 v = *reinterpret_cast<const uint2 *>(krow + s * SK_STAGE_ROWS + r);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const unsigned w = j & 2 ? v.y : v.x, k = j & 1 ? w >> 16 : w & 0xFFFFu;
                        if (r + j >= left || !bounds_ok(k < (unsigned)p.K, p.status, 32)) continue;
                        sk_copy_16(to + A_HALF + (r + j) * SK_ROW_BYTES, b_src + (size_t)k * n4);
                        sk_copy_16(to + (r + j) * A_ROW_BYTES, a_src + (size_t)k * (TILE_M * 4));
                    }
                }
            }
            if (ok) sk_copies_arrive(full0 + 8 * slot);
        }
        cp_async_wait_all();      // nothing of this thread is in flight when it leaves
    }
    if (!ok && lane == 0) atomicExch(p.status, (int)ESMM_ERR_TIMEOUT);
}

// Once per device: the SM count, and the shared-memory allowance of every variant raised to the device's maximum.  The allowance belongs
// to the kernel in its context and not to a launch: set to each launch's own size, a call of another thread with a shorter list lowered
// it between this call's setting and its launch, which was then refused.
static int skinny_prepare(int dev, int *sms)
{
    static std::mutex mu;
    static int sm_count[64];
    if (dev < 0 || dev >= 64) return ESMM_ERR_CUDA;
    std::lock_guard<std::mutex> lock(mu);
    if (!sm_count[dev]) {
        int n = 0, smem = 0;
        auto allow = [&](auto kernel) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); };
        ESMM_CUDA_TRY(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
        ESMM_CUDA_TRY(cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
        ESMM_CUDA_TRY(allow(esmm_joint_sgemm_skinny_kernel<8, 2, 2>));
        ESMM_CUDA_TRY(allow(esmm_joint_sgemm_skinny_kernel<16, 4, 2>));
        ESMM_CUDA_TRY(allow(esmm_joint_sgemm_skinny_kernel<16, 2, 4>));
        ESMM_CUDA_TRY(allow(esmm_joint_sgemm_skinny_kernel<32, 4, 4>));
        ESMM_CUDA_TRY(allow(esmm_joint_sgemm_skinny_kernel<32, 2, 4>));
        sm_count[dev] = n;
    }
    *sms = sm_count[dev];
    return ESMM_OK;
}

// Whether this kernel takes a problem (otherwise the tiled kernel does).  Of M <= 32 all; of fewer than two whole panels of 128 rows
// those for which it takes less time whatever the operands: a strip and row block of 32 rows is counted as 1 per SM, a 64-row tile of
// eight of them as 5 (a strip takes 13.7 cycles a k with several on an SM, a tile 87, and the tiled kernel is as fast as 1.2 times
// that on blocks that differ), a 128-row tile as 9.1.  Tiled / strips, us, K = 4096: 64 x 1024 dense 184 / 42, 64 x 4096 185 / 64, 64
// x 4096 a quarter live 51.8 / 19.8, 96 x 4096 pruned MLP 44.8 / 27.2, 64 x 11008 x 2048 pruned MLP (4.7 per SM) 33.9 / 24.1, 100 x
// 6000 x 3000 0.5 / 0.5 (5.1) 53.9 / 36.2; on the other side 256 x 4096 dense (6.9) 188 / 205 and pruned MLP 60.4 / 51.7, 1000 x 1508
// x 2012 0.5 / 0.5 (10.4) 48.5 / 51.2.  At K up to 256 what a strip costs beside its k counts for more, and the lines are 4 and 8: dense,
// 64 x 11008 x 128 (4.65 per SM) 12.2 / 15.8, 160 x 4096 x 128 (4.3) 12.1 / 15.4, 160 x 8192 x 64 (8.6) 12.3 / 18.6, 224 x 6000 x 256 (8.9)
// 26.6 / 29.7; on the other side 64 x 8192 x 128 (3.5) 12.1 / 10.7, 96 x 11008 x 256 (7.0) 25.6 / 24.8.  (Half-density operands of the
// first group are up to 1.5 us faster in strips.)  Taller problems stay with the tiled kernel and its launch shapes, which callers can ask
// for (esmm_last_tiled_kernel_warps).
bool gemm_ab_skinny_applies(int M, int N, int K)
{
    const int kp = ceil_div(K, BK) * BK;
    if (kp > SK_MAX_KP || M >= STRIP_ROW_LIMIT || tuning_get("NO_SKINNY", 0)) return false;
    if (M <= SK_ROWS) return N >= 4 * SK_COLS;
    if (tiled_kernel_tuned()) return false;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) return false;
    const long units = (long)ceil_div(M, SK_ROWS) * ceil_div(N, SK_COLS), across = ceil_div(N, TILE_N);
    const long rounds64 = (ceil_div(M, 64) * across + sms - 1) / sms, rounds128 = (ceil_div(M, TILE_M) * across + sms - 1) / sms;
    return K <= 256 ? units <= sms * std::min(4 * rounds64, 8 * rounds128) : (double)units <= sms * std::min(5.0 * rounds64, 9.1 * rounds128);
}

int gemm_ab_skinny_launch(int M, int N, int K, const float *d_a_packed, const float *d_B, float *d_C,
                          const uint8_t *d_a_pat, const uint8_t *d_b_pat, cudaStream_t stream)
{
    SkinnyParams p;
    memset(&p, 0, sizeof p);
    p.M = M;
    p.N = N;
    p.K = K;
    p.nKB = ceil_div(K, BK);
    p.kp = p.nKB * BK;
    p.cap = p.kp + SK_STAGE_ROWS;
    p.row_blocks = ceil_div(M, SK_ROWS);
    p.a_pat = d_a_pat;
    p.b_pat = d_b_pat;
    p.a_packed = d_a_packed;
    p.B = d_B;
    p.C = d_C;
    p.status = device_status_ptr();
    if (!p.status) return ESMM_ERR_CUDA;
    int dev = 0, sms = 0;
    ESMM_CUDA_TRY(cudaGetDevice(&dev));
    const int pst = skinny_prepare(dev, &sms);
    if (pst != ESMM_OK) return pst;
    const int strips = ceil_div(N, SK_COLS), forced = tuning_get("SKINNY_ROWS", 0);
    const int rows = M > 16 || forced == 32 ? 32 : M > 8 || forced == 16 ? 16 : 8;
    const long units = (long)strips * p.row_blocks;
    auto launch = [&](auto kernel, int r, int warps) -> int {
        // the ring as deep as it can be with as many CTAs on an SM as there are for it, up to four
        const size_t room = (size_t)(SMEM_LIMIT + 1024) / std::min(4l, (units + sms - 1) / sms) - 1024;
        p.stages = SK_MAX_STAGES;
        while (p.stages > 2 && sk_smem(r, p.stages, p.cap) > room) --p.stages;
        const size_t smem = sk_smem(r, p.stages, p.cap);
        ESMM_CUDA_TRY(launch_dependent(kernel, dim3((unsigned)units), dim3(warps * 32), smem, stream, p));
        ESMM_CUDA_TRY(cudaGetLastError());
        return ESMM_OK;
    };
    // Four multiplying warps where an SM has one or two strips; with three, shared memory bounds the kernel and two warps, which
    // load less of A, are faster.  The multiplying part alone, us, two / four warps, K = 4096: M = 16 dense, one strip per SM 31.1 / 28.6;
    // M = 16 pruned MLP, SMs with two strips 9.2 / 8.6, with three 9.9 / 11.6; M = 32 one strip 10.3 / 7.6, two 14.2 / 11.7, three 14.9 / 16.2.
    const bool spread = units <= 2 * sms;
    if (rows == 8) return launch(esmm_joint_sgemm_skinny_kernel<8, 2, 2>, 8, 4);
    if (rows == 16)
        return spread ? launch(esmm_joint_sgemm_skinny_kernel<16, 4, 2>, 16, 6) : launch(esmm_joint_sgemm_skinny_kernel<16, 2, 4>, 16, 4);
    return spread ? launch(esmm_joint_sgemm_skinny_kernel<32, 4, 4>, 32, 6) : launch(esmm_joint_sgemm_skinny_kernel<32, 2, 4>, 32, 4);
}

}  // namespace esmm
