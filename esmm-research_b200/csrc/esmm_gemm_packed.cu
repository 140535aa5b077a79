// The tiled kernel on packed A: its instantiations, and the host side of both forms (esmm_gemm_ab_packed, esmm_gemm_ab).
#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>

#include "esmm_gemm_tiled.cuh"

namespace esmm {

template <int WMB, int NPW, bool BLOCKS>
__global__ void __launch_bounds__((P_CONSUMER_WARPS + NPW + 1) * 32, 1)
esmm_joint_sgemm_packed_kernel(const __grid_constant__ PackedMaps maps, const __grid_constant__ PackedParams p)
{
    tiled_sgemm<WMB, NPW, false, BLOCKS>(maps, p);
}

#ifdef ESMM_TRACE
extern "C" int esmm_trace_read(unsigned long long *host, int n)
{
    return (int)cudaMemcpyFromSymbol(host, g_esmm_trace, sizeof(unsigned long long) * (n < 1024 ? n : 1024));
}
#endif

// esmm_gemm_skinny.cu: the kernel for few rows
bool gemm_ab_skinny_applies(int M, int N, int K);
int gemm_ab_skinny_launch(int M, int N, int K, const float *d_a_packed, const float *d_B, float *d_C,
                          const uint8_t *d_a_pat, const uint8_t *d_b_pat, cudaStream_t stream);

// The launch shape follows the operands: the 16-warp form pays on tiles of scattered single rows and costs about
// half a percent elsewhere, and which kind the operands are is known on the device only.  So CTA 0 of every
// launch notes what its first tile would have wanted in a word of host-mapped memory (one per device, set up at
// the first launch) where the word said otherwise when the host launched it (a launch's end waits for the store across
// PCIe: 512 x 1024 x 704, 32-granular 0.2 / 0.2, 16.4 us with a note every time, 14.4 now), and the next launch on that
// device reads the word, without waiting for anything: repeated products of like operands - what a benchmark loop or a
// layer with fixed weights issues - get the right shape from the second call on, and a stale or missing note costs one
// launch in the other.  The results are bit-identical in both shapes.  esmm_tuning_set("PRODUCER_WARPS", 3 | 7 | 0) pins the
// shape instead.  (Scattered rows reach the pipeline in launches too short to look at the samples.  Larger operands of that
// kind go to block mode, where twelve warps work in either shape and the 16-warp form, whose registers do not hold block mode's
// accumulators without spilling, is as a rule the slower one: whole calls, 12 / 16 warps, 4096^3 32-granular 0.2 / 0.2 158 / 182 us,
// 64-granular 0.5 / 0.5 652 / 731, 1000 x 1508 x 2012 at 0.5 / 0.5 47.9 / 50.7; 2048^3 32-granular 0.5 / 0.5 118 / 115.  There the note
// is set only with no more pairs of blocks than CTAs: 512 x 512 x 4096 at 0.3 / 0.3 24.1 / 24.7.)
static std::atomic<int> g_last_tiled_warps[64];   // per device: warps per CTA of the last launch of the tiled kernel

struct FormHint {
    volatile int *host = nullptr;   // what the host reads
    int *device = nullptr;          // the same word as the kernels address it
};

static FormHint form_hint_word(int dev)
{
    static std::mutex mu;
    static FormHint words[64];
    if (dev < 0 || dev >= 64) return FormHint();
    std::lock_guard<std::mutex> lock(mu);
    if (!words[dev].host) {
        void *h = nullptr, *d = nullptr;
        if (cudaHostAlloc(&h, 64, cudaHostAllocMapped | cudaHostAllocPortable) != cudaSuccess ||
            cudaHostGetDevicePointer(&d, h, 0) != cudaSuccess) {
            (void)cudaGetLastError();   // no note then: the 12-warp form is launched
            if (h) (void)cudaFreeHost(h);
            return FormHint();
        }
        memset(h, 0, 64);
        words[dev].host = static_cast<volatile int *>(h);
        words[dev].device = static_cast<int *>(d);
    }
    return words[dev];
}

// Once per device: the SM count, and the shared-memory allowance of all forms of the kernel, for packed or for row-major A, raised to
// the device's maximum.  (Raising it also loads the forms' code, so that the first launch in another shape does not pay for that.)
static int prepare_device(int dev, bool row_major, int *sms)
{
    static std::mutex mu;
    static int sm_count[64][2] = {{0}};
    if (dev < 0 || dev >= 64) return ESMM_ERR_CUDA;
    std::lock_guard<std::mutex> lock(mu);
    int &known = sm_count[dev][row_major];
    if (!known) {
        int n = 0, smem = 0;
        auto allow_smem = [](auto kernel, int bytes) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); };
        ESMM_CUDA_TRY(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
        ESMM_CUDA_TRY(cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
        if (row_major) {
            ESMM_CUDA_TRY(rowmajor_allow_smem(smem));
        } else {
            ESMM_CUDA_TRY(allow_smem(esmm_joint_sgemm_packed_kernel<1, 3, false>, smem));
            ESMM_CUDA_TRY(allow_smem(esmm_joint_sgemm_packed_kernel<1, 3, true>, smem));
            ESMM_CUDA_TRY(allow_smem(esmm_joint_sgemm_packed_kernel<1, 7, false>, smem));
            ESMM_CUDA_TRY(allow_smem(esmm_joint_sgemm_packed_kernel<1, 7, true>, smem));
            ESMM_CUDA_TRY(allow_smem(esmm_joint_sgemm_packed_kernel<2, 3, false>, smem));
            ESMM_CUDA_TRY(allow_smem(esmm_joint_sgemm_packed_kernel<2, 3, true>, smem));
            ESMM_CUDA_TRY(allow_smem(esmm_joint_sgemm_packed_kernel<2, 7, false>, smem));
            ESMM_CUDA_TRY(allow_smem(esmm_joint_sgemm_packed_kernel<2, 7, true>, smem));
        }
        known = n;
    }
    *sms = known;
    return ESMM_OK;
}

int gemm_ab_packed_launch_form(int M, int N, int K, const float *d_a_packed, const float *d_B, float *d_C,
                               const uint8_t *d_a_pat, const uint8_t *d_b_pat, cudaStream_t stream, bool follow_hint);

// The once-per-device set-up of the tiled kernel on the current device, for callers that want it outside a timed region.
int gemm_ab_packed_prepare()
{
    int dev = 0, sms = 0;
    ESMM_CUDA_TRY(cudaGetDevice(&dev));
    const int st = prepare_device(dev, false, &sms);
    if (st == ESMM_OK && tuning_get("PRODUCER_WARPS", -1) < 0) (void)form_hint_word(dev);
    return st;
}

int gemm_ab_packed_launch(int M, int N, int K, const float *d_a_packed, const float *d_B, float *d_C,
                          const uint8_t *d_a_pat, const uint8_t *d_b_pat, cudaStream_t stream)
{
    return gemm_ab_packed_launch_form(M, N, K, d_a_packed, d_B, d_C, d_a_pat, d_b_pat, stream, true);
}

// follow_hint = false: the 12-warp form unless PRODUCER_WARPS says otherwise, and no host-mapped word (for the
// entry point that may not allocate).
static int tiled_launch(int M, int N, int K, const float *d_a_packed, const float *d_A, int a_tile_m, const float *d_B, float *d_C,
                        const uint8_t *d_a_pat, const uint8_t *d_b_pat, cudaStream_t stream, bool follow_hint);

int gemm_ab_packed_launch_form(int M, int N, int K, const float *d_a_packed, const float *d_B, float *d_C,
                               const uint8_t *d_a_pat, const uint8_t *d_b_pat, cudaStream_t stream, bool follow_hint)
{
    if (!d_a_packed || !d_B || !d_C || !d_a_pat || !d_b_pat) return ESMM_ERR_NULL;
    if (M <= 0 || N <= 0 || K <= 0 || (K & 3) || (N & 3)) return ESMM_ERR_SHAPE;
    if (((uintptr_t)d_a_packed | (uintptr_t)d_B | (uintptr_t)d_C) & 15) return ESMM_ERR_ALIGN;
    if (gemm_ab_skinny_applies(M, N, K))
        return gemm_ab_skinny_launch(M, N, K, d_a_packed, d_B, d_C, d_a_pat, d_b_pat, stream);
    return tiled_launch(M, N, K, d_a_packed, nullptr, 32, d_B, d_C, d_a_pat, d_b_pat, stream, follow_hint);
}

constexpr int RM_MAX_KB = 8332;   // longest K taken with row-major A, in K blocks
// Row-major A of more K blocks than RM_WHOLE_LIST_KB: a tile's rows are listed RM_LIST_KB K blocks at a time, its sums go on from
// one list to the next.  Whole lists leave a ring of fewer than five stages from there on and no ring at all past K = 27488, where
// block mode, whatever the operands, was the alternative.  Whole lists or block mode / lists in parts, kernel alone, 2048 x 2048 x K:
// K = 12288 dense 2568 / 2577 us, 24576 dense 5148 / 5160 and 64-granular 0.5 / 0.5 2144 / 1945, 32768 dense 8497 / 5991.
constexpr int RM_LIST_KB = 1024, RM_WHOLE_LIST_KB = 1336;

// Row-major A, A patterns with one row per a_tile_m rows.
int gemm_ab_launch(int M, int N, int K, const float *d_A, const float *d_B, float *d_C,
                   const uint8_t *d_a_pat, const uint8_t *d_b_pat, int a_tile_m, cudaStream_t stream)
{
    if (!d_A || !d_B || !d_C || !d_a_pat || !d_b_pat) return ESMM_ERR_NULL;
    if (M <= 0 || N <= 0 || K <= 0 || (K & 3) || (N & 3)) return ESMM_ERR_SHAPE;
    if (a_tile_m <= 0 || (a_tile_m < 32 ? (32 % a_tile_m) : (a_tile_m % 32))) return ESMM_ERR_UNSUPPORTED;
    if (((uintptr_t)d_A | (uintptr_t)d_B | (uintptr_t)d_C) & 15) return ESMM_ERR_ALIGN;
    if (ceil_div(K, BK) > RM_MAX_KB) return ESMM_ERR_TOO_LARGE;
    return tiled_launch(M, N, K, nullptr, d_A, a_tile_m, d_B, d_C, d_a_pat, d_b_pat, stream, false);
}

// A packed (d_a_packed) or row-major (d_A, with a_tile_m).
static int tiled_launch(int M, int N, int K, const float *d_a_packed, const float *d_A, int a_tile_m, const float *d_B, float *d_C,
                        const uint8_t *d_a_pat, const uint8_t *d_b_pat, cudaStream_t stream, bool follow_hint)
{
    const bool row_major = d_a_packed == nullptr;
    PackedParams p;
    memset(&p, 0, sizeof p);
    p.M = M;
    p.N = N;
    p.K = K;
    p.nKB = ceil_div(K, BK);
    p.kp = p.nKB * BK;
    if (p.kp > 65535 && !row_major) return ESMM_ERR_TOO_LARGE;  // row list entries are 16-bit k indices
    p.cap = ((p.kp + 31) & ~31) + 32;
    p.list_kb = p.nKB;
    p.lists = 1;
    if (row_major && p.nKB > RM_WHOLE_LIST_KB) {
        p.list_kb = RM_LIST_KB;
        p.lists = ceil_div(p.nKB, RM_LIST_KB);
        p.cap = RM_LIST_KB * BK + 32;
    }
    p.A = d_A;
    p.a_div = a_tile_m >= 32 ? a_tile_m / 32 : 1;
    p.a_mul = a_tile_m >= 32 ? 1 : 32 / a_tile_m;
    p.a_pat_rows = ceil_div(M, a_tile_m);
    p.a_rows = ceil_div(M, 32);
    p.b_rows = ceil_div(N, PAT_N);
    int dev = 0, sms = 0;
    ESMM_CUDA_TRY(cudaGetDevice(&dev));
    {
        const int pst = prepare_device(dev, row_major, &sms);
        if (pst != ESMM_OK) return pst;
    }
    // Tile height: 128 rows, or 64 where that fills the GPU better.  Rounds of tiles per SM, a 64-row
    // tile counted as 0.55 of a 128-row one (it does half the multiply-adds at a worse ratio of
    // shared-memory loads).  ESMM_TILE_M = 64 | 128 overrides.
    p.tiles_n = ceil_div(N, TILE_N);
    const int panels = ceil_div(M, TILE_M);
    const long t128 = (long)panels * p.tiles_n, t64 = (long)ceil_div(M, 64) * p.tiles_n;
    const double cost128 = (double)((t128 + sms - 1) / sms), cost64 = 0.55 * (double)((t64 + sms - 1) / sms);
    int tile_rows = cost64 < cost128 ? 64 : TILE_M;
    const int forced_rows = tuning_get("TILE_M", 0);
    if (forced_rows == 64 || forced_rows == TILE_M) tile_rows = forced_rows;
    p.tiles_m = ceil_div(M, tile_rows);
    p.num_tiles = p.tiles_m * p.tiles_n;
    p.group_m = tuning_get("GROUP_M", GROUP_M);
    if (p.group_m < 1) p.group_m = 1;
    p.brow_bits = tuning_get("BROW_BITS", 7);
    if (p.brow_bits < 0) p.brow_bits = 0;
    if (p.brow_bits > 8) p.brow_bits = 8;
    p.row_density = tuning_get("ROW_DENSITY", 8);
    p.force_listed = tuning_get("FORCE_LISTED", 0);
    p.no_run_tiles = tuning_get("NO_RUN_TILES", 0);
    const uintptr_t pat_bits = (uintptr_t)d_a_pat | (uintptr_t)d_b_pat;
    p.vec_patterns = 0;
    if (p.nKB % 4 == 0 && (pat_bits & 3) == 0) p.vec_patterns = 4;
    if (p.nKB % 16 == 0 && (pat_bits & 15) == 0 && p.nKB >= 512) p.vec_patterns = 16;
    const int forced_vec = tuning_get("VEC_PATTERNS", -1);   // 0, 4, 16: tuning and tests
    if (forced_vec == 0 || (forced_vec == 4 && p.vec_patterns >= 4) ||
        (forced_vec == 16 && p.nKB % 16 == 0 && (pat_bits & 15) == 0))
        p.vec_patterns = forced_vec;
    p.pat_words = p.nKB % 4 == 0 && (pat_bits & 3) == 0;
    p.last_bits = (K & 7) ? ((1u << (K & 7)) - 1u) * 0x01010101u : 0xFFFFFFFFu;
    p.a_pat = d_a_pat;
    p.b_pat = d_b_pat;
    p.a_packed = d_a_packed;
    p.B = d_B;
    p.C = d_C;

    // 3 = 12 warps; 7 = 16 warps, 7 producers copying; 0 = 16 warps, 3 or 7 copying as each CTA's first tile says;
    // not set = 3 or 0 as the last launch on this device noted
    int producer_warps = tuning_get("PRODUCER_WARPS", -1);
    if (row_major) {
        producer_warps = 3;
    } else if (producer_warps != 3 && producer_warps != 7 && producer_warps != 0) {
        producer_warps = 3;
        if (follow_hint) {
            const FormHint hint = form_hint_word(dev);
            if (hint.host) {
                p.form_hint = hint.device;
                p.form_known = *hint.host != 0 ? 1 : 0;
                if (p.form_known) producer_warps = 0;
            }
        }
    }
    const bool wide = producer_warps != 3;
    p.adaptive = producer_warps == 0;
    if (!row_major && dev >= 0 && dev < 64) g_last_tiled_warps[dev].store(wide ? 16 : 12, std::memory_order_relaxed);
    const int threads = (P_CONSUMER_WARPS + (wide ? 7 : 3) + 1) * 32;

    int grid = tuning_get("GRID", sms);
    const long pairs = std::max((long)ceil_div(p.a_rows, 2) * p.b_rows, (long)p.a_rows * ceil_div(p.b_rows, 2));
    p.few_blocks = pairs <= grid;
    p.rm_shape = row_major_shape(M, N, p.num_tiles, pairs, sms);
    // Where blocks differ the samples cost a launch a microsecond or two, which short ones do not win back: the pipeline, without looking, where an SM
    // has fewer than 768 k of tiles to go through (58 x 7368 x 648: 15.2 us, 17.4 with the look; 2502 x 1112 x 456, 912 k of tiles
    // per SM: 37.1 in the pipeline, 31.5 in block mode).
    const long tile_rounds = (p.num_tiles + sms - 1) / sms;
    p.block_mode = tuning_get("BLOCK_MODE", tile_rounds * p.kp < 768 ? 0 : -1);
    const bool blocks = p.block_mode != 0;

    int stages = tuning_get("STAGES", P_MAX_STAGES);
    if (stages > P_MAX_STAGES) stages = P_MAX_STAGES;
    if (stages < 2) stages = 2;
    const int stage_bytes = row_major ? RM_STAGE_A_BYTES + STAGE_HALF_BYTES : PSTAGE_BYTES;
    while (stages > 2 && packed_smem_layout(stages, stage_bytes, p.cap, blocks).total > SMEM_LIMIT) --stages;
    const PackedSmem L = packed_smem_layout(stages, stage_bytes, p.cap, blocks);
    if (L.total > SMEM_LIMIT) return ESMM_ERR_TOO_LARGE;
    p.stages = stages;

    p.status = device_status_ptr();
    if (!p.status) return ESMM_ERR_CUDA;

    // Packed A is a matrix of 128 columns and panels * kp rows, of which a tile reads all 128 columns
    // or the 64 of its half; B is K rows of N columns.  Rows
    // (or columns of B) outside the matrices are zero-filled by the copy engine and still counted
    // in the stage's byte total.  The 3-D views split the row index into (k % 8, k / 8); for B
    // that is only valid when K is a multiple of 8 (otherwise the view would reach past row K).
    p.b_runs_ok = (K % BK) == 0;
    PackedMaps maps;
    const uint64_t a_rows_total = (uint64_t)panels * p.kp;
    int st = 0;
    memset(&maps, 0, sizeof maps);
    for (int i = 0; i < 4 && !st; ++i) {
        if (!row_major)
            st = make_map_2d(&maps.a_box[i], d_a_packed, TILE_M, a_rows_total, tile_rows, 1u << i, CU_TENSOR_MAP_SWIZZLE_NONE,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
        if (!st) st = make_map_2d(&maps.b_box[i], d_B, (uint64_t)N, (uint64_t)K, TILE_N, 1u << i, CU_TENSOR_MAP_SWIZZLE_NONE,
                                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
    }
    for (int i = 0; i < 4 && !st; ++i) {
        const uint32_t c = 1u << i;
        if (!row_major)
            st = make_map_3d(&maps.a_run[i], d_a_packed, TILE_M, BK, (uint64_t)panels * p.nKB, (uint64_t)TILE_M * 4,
                         (uint64_t)TILE_M * 4 * BK, tile_rows, c, ROWS_PER_STAGE / c);
        if (!st) {
            if (p.b_runs_ok)
                st = make_map_3d(&maps.b_run[i], d_B, (uint64_t)N, BK, (uint64_t)p.nKB, (uint64_t)N * 4,
                                 (uint64_t)N * 4 * BK, TILE_N, c, ROWS_PER_STAGE / c);
            else
                maps.b_run[i] = maps.b_box[0];  // never used
        }
    }
    if (st) return st;

    // (in block mode a CTA has work as soon as there are pairs of blocks for it)
    const long most = p.block_mode ? std::max((long)p.num_tiles, pairs) : (long)p.num_tiles;
    if (grid > most) grid = (int)most;
    if (grid < 1) grid = 1;
    auto launch = [&](auto kernel, int threads) -> int {
        ESMM_CUDA_TRY(launch_dependent(kernel, dim3(grid), dim3(threads), L.total, stream, maps, p));
        return ESMM_OK;
    };
    int lst;
    auto pick = [&](auto with, auto without) { return blocks ? launch(with, threads) : launch(without, threads); };
    if (row_major) {
        ESMM_CUDA_TRY(rowmajor_launch(tile_rows, blocks, grid, L.total, stream, maps, p));
        lst = ESMM_OK;
    } else if (tile_rows == 64) {
        lst = wide ? pick(esmm_joint_sgemm_packed_kernel<1, 7, true>, esmm_joint_sgemm_packed_kernel<1, 7, false>)
                   : pick(esmm_joint_sgemm_packed_kernel<1, 3, true>, esmm_joint_sgemm_packed_kernel<1, 3, false>);
    } else {
        lst = wide ? pick(esmm_joint_sgemm_packed_kernel<2, 7, true>, esmm_joint_sgemm_packed_kernel<2, 7, false>)
                   : pick(esmm_joint_sgemm_packed_kernel<2, 3, true>, esmm_joint_sgemm_packed_kernel<2, 3, false>);
    }
    if (lst != ESMM_OK) return lst;
    ESMM_CUDA_TRY(cudaGetLastError());
    return ESMM_OK;
}

int last_tiled_warps()
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    return g_last_tiled_warps[dev].load(std::memory_order_relaxed);
}

}  // namespace esmm

extern "C" int esmm_last_tiled_kernel_warps(void) { return esmm::last_tiled_warps(); }

extern "C" int esmm_gemm_ab_packed(int M, int N, int K, const float *d_a_packed, const float *d_B, float *d_C,
                                   const uint8_t *d_a_pat, const uint8_t *d_b_pat, void *stream)
{
    return esmm::gemm_ab_packed_launch(M, N, K, d_a_packed, d_B, d_C, d_a_pat, d_b_pat, (cudaStream_t)stream);
}

extern "C" int esmm_gemm_ab(int M, int N, int K, const float *d_A, const float *d_B, float *d_C,
                            const uint8_t *d_a_pat, const uint8_t *d_b_pat, int a_tile_m, void *stream)
{
    return esmm::gemm_ab_launch(M, N, K, d_A, d_B, d_C, d_a_pat, d_b_pat, a_tile_m, (cudaStream_t)stream);
}
