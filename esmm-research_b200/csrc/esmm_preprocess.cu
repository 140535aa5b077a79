// A/B pattern preprocessor for sm_100a: one coalesced pass over the matrix, 16-byte loads,
// row reduction in registers, packed stores.  Pattern bytes are bit-exact with
// preprocess_a_patterns_kernel / preprocess_b_patterns_kernel of the reference
// (src/preprocessors/ab_preprocessor.cu:31-84, :91-144).
//
// Kernel names keep "preprocess" in them: the reference's sweep scripts split timings by
// that substring (scripts/benchmark.py:456-458).
#include <cstdio>
#include <cstring>

#include "esmm_common.cuh"

namespace esmm {

constexpr int PRE_THREADS = 128;

// `v != 0.0f` as an integer test: -0.0f is zero, NaN and denormals are nonzero.
__device__ __forceinline__ unsigned nz(float v) { return (__float_as_uint(v) << 1) != 0u; }

__device__ __forceinline__ unsigned nz4(const float4 &v)
{
    return nz(v.x) | (nz(v.y) << 1) | (nz(v.z) << 2) | (nz(v.w) << 3);
}

// SPLIT = 1: one warp owns tile_m rows x 128 columns (16 K blocks).  Lane l reads columns 4l..4l+3 of
// every row (one 512-byte request per row per warp), ORs the nonzero bits of its 4 columns
// over the rows in registers, then pairs of lanes join their nibbles into a pattern byte.
// SPLIT = PRE_WARPS: the CTA's four warps share the rows, eight in turn, and join their nibbles in shared memory.  A warp waits for
// memory once per eight rows, and on a small A there is little else to do meanwhile: 2048^2 at tile_m 128
// 12.4 -> 6.2 us, at 64 8.3 -> 4.6, 1024^2 at 32 6.2 -> 4.6.
// Needs K % 4 == 0 and a 16-byte aligned A.
constexpr int PRE_WARPS = PRE_THREADS / 32;

template <int SPLIT>
__global__ void __launch_bounds__(PRE_THREADS)
esmm_preprocess_a_patterns_kernel(const float *A, int M, int K, int tile_m, int nMB,
                                  int nKB, int k_chunks, uint8_t *__restrict__ out, int *status)
{
    grid_launch_dependents();   // (both as in the packing kernel below)
    grid_dependency_wait();
    // checked build, sites 10 (loads of A) and 11 (pattern stores)
    const size_t a_floats = (size_t)M * K, out_bytes = (size_t)nMB * nKB;
    __shared__ uint8_t nibs[PRE_WARPS][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, part = SPLIT > 1 ? warp : 0;
    const long step = SPLIT > 1 ? gridDim.x : (long)gridDim.x * PRE_WARPS;
    const long tasks = (long)nMB * k_chunks;
    for (long task = SPLIT > 1 ? blockIdx.x : (long)blockIdx.x * PRE_WARPS + warp; task < tasks; task += step) {
        const int mb = (int)(task / k_chunks);
        const int kc = (int)(task - (long)mb * k_chunks);
        const int col = kc * 128 + lane * 4;
        unsigned nib = 0;
        if (col < K) {
            const int row0 = mb * tile_m;
            const int rows = min(tile_m, M - row0);
            const float *src = A + (size_t)row0 * K + col;
            int r = 8 * part;
            for (; r + 8 <= rows; r += 8 * SPLIT) {
                float4 v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (bounds_ok((size_t)(row0 + r + u) * K + col + 4 <= a_floats, status, 10))
                        v[u] = __ldcg(reinterpret_cast<const float4 *>(src + (size_t)(r + u) * K));
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) nib |= nz4(v[u]);
            }
            for (const int end = min(rows, r + 8); r < end; ++r)   // (a group of fewer than eight rows; of the warps one at most has it)
                if (bounds_ok((size_t)(row0 + r) * K + col + 4 <= a_floats, status, 10))
                    nib |= nz4(__ldcg(reinterpret_cast<const float4 *>(src + (size_t)r * K)));
        }
        if (SPLIT > 1) {
            nibs[warp][lane] = (uint8_t)nib;
            __syncthreads();
            if (warp == 0)
#pragma unroll
                for (int w = 1; w < PRE_WARPS; ++w) nib |= nibs[w][lane];
            __syncthreads();
        }
        const unsigned other = __shfl_xor_sync(0xFFFFFFFFu, nib, 1);
        const int kb = kc * 16 + (lane >> 1);
        if (part == 0 && !(lane & 1) && kb < nKB && bounds_ok((size_t)mb * nKB + kb < out_bytes, status, 11))
            out[(size_t)mb * nKB + kb] = (uint8_t)(nib | (other << 4));
    }
}

// Pattern scan fused with the re-layout the packed GEMM variant reads: besides the pattern
// bytes the warp writes its 32 rows x 32 columns transposed into
//   packed[((tile * nKB + kb) * 8 + k) * 128 + row_in_tile],   tile = row / 128,
// i.e. k-major rows of 128 floats per 128-row tile, so that one K block of a tile is 4 KB of
// contiguous memory.  A k whose pattern bit is clear for the warp's 32-row block is not written: the
// GEMM never multiplies it, so whatever the buffer holds there is harmless.
//
// Lane = (row r4 of four, column group cq of eight): lane loads rows 4 i + r4, columns 4 cq .. 4 cq + 3.  All rows of a column are OR-ed as
// bit patterns before the one test for zero (without the sign bit), and one reduction over the warp gives the 32 live bits, which
// are the block's four pattern bytes as they stand.  The transpose goes through shared memory 16 bytes at a time, chunk cq of row r at
// position cq ^ (r & 7), so that neither the stores (eight lanes a row) nor the loads (a lane a row) meet a bank twice; four stores
// of 128 bytes per chunk follow, of live columns only.
// What bounds it: HBM.  In a train of calls 4096^2 takes 11.4 us with a fifth of the columns live, 16.2 with half and 21.8 with all (12.3, 15.4
// and 20.5 us of bytes at the measured copy bandwidth); 32 x 64 columns per warp with every element's own test, store and load through shared
// memory, 1277 instructions for 64 live columns where these tasks have 796 (ncu), took 15.2, 18.5 and 22.3 and had 16 warps per SM for these 32.
constexpr int PACK_WARPS = 4;
constexpr int PACK_COLS = 32;

__global__ void __launch_bounds__(PACK_WARPS * 32)
esmm_preprocess_a_pack32_kernel(const float *A, int M, int K, int nMB, int nKB, int k_chunks,
                                uint8_t *__restrict__ out, float *__restrict__ packed, int *status, int early)
{
    // The product kernel, launched as a dependent of this one, may be placed where SMs become free once every CTA of this
    // grid has got here; it waits for this grid's end itself.
    if (early) grid_launch_dependents();
    // This kernel is a dependent launch too, of whatever was before it: it is launched as that ends rather than after, which takes 2 us off
    // every call of a train of them (1000 x 1508 x 2012 57.4 -> 55.2 us, 1024^3 at half density 32.9 -> 30.9).  The product kernels don't
    // call it early: strips placed beside those of the call before are 15-100 % slower.  Nothing of A is read before the wait, and what is
    // read goes past L1, which may have been filled while A was written.
    grid_dependency_wait();
    // checked build, sites 10 (loads of A), 11 (pattern stores), 12 (stores into the packed copy)
    const size_t a_floats = (size_t)M * K, out_bytes = (size_t)nMB * nKB;
    const size_t packed_floats = (size_t)((M + 127) / 128) * nKB * BK * 128;
    __shared__ __align__(16) float4 pack_smem[PACK_WARPS][32 * PACK_COLS / 4];
    float4 *tile = pack_smem[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31, r4 = lane >> 3, cq = lane & 7;
    const long warps_total = (long)gridDim.x * PACK_WARPS;
    const long tasks = (long)nMB * k_chunks;
    for (long task = (long)blockIdx.x * PACK_WARPS + (threadIdx.x >> 5); task < tasks; task += warps_total) {
        const int mb = (int)(task / k_chunks);
        const int kc = (int)(task - (long)mb * k_chunks);
        const int col = kc * PACK_COLS + cq * 4;
        const int row0 = mb * 32;
        const float *src = A + (size_t)(row0 + r4) * K + col;
        float4 v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int row = row0 + 4 * i + r4;
            v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (col < K && row < M && bounds_ok((size_t)row * K + col + 4 <= a_floats, status, 10))
                v[i] = __ldcg(reinterpret_cast<const float4 *>(src + (size_t)(4 * i) * K));
        }
        unsigned any[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            any[0] |= __float_as_uint(v[i].x);
            any[1] |= __float_as_uint(v[i].y);
            any[2] |= __float_as_uint(v[i].z);
            any[3] |= __float_as_uint(v[i].w);
            tile[(4 * i + r4) * 8 + (cq ^ ((4 * i + r4) & 7))] = v[i];
        }
        unsigned nib = 0u;
#pragma unroll
        for (int q = 0; q < 4; ++q) nib |= (any[q] << 1) != 0u ? 1u << q : 0u;
        const unsigned live = __reduce_or_sync(0xFFFFFFFFu, nib << (4 * cq));   // bit c: column c of the 32
        if (lane == 0) {
            uint8_t *bytes = out + (size_t)mb * nKB + kc * 4;
            if (kc * 4 + 4 <= nKB && (reinterpret_cast<uintptr_t>(bytes) & 3) == 0) {
                if (bounds_ok((size_t)mb * nKB + kc * 4 + 4 <= out_bytes, status, 11)) *reinterpret_cast<unsigned *>(bytes) = live;
            } else {
                for (int j = 0; j < 4; ++j)
                    if (kc * 4 + j < nKB && bounds_ok((size_t)mb * nKB + kc * 4 + j < out_bytes, status, 11)) bytes[j] = (uint8_t)(live >> (8 * j));
            }
        }
        __syncwarp();
        // (a live column is inside A)
        const size_t dst0 = ((size_t)(mb >> 2) * nKB * BK + kc * PACK_COLS) * 128 + (mb & 3) * 32 + lane;
        float *dst = packed + dst0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (!((live >> (4 * j)) & 0xFu)) continue;
            const float4 x = tile[lane * 8 + (j ^ (lane & 7))];
            if (!bounds_ok(dst0 + (size_t)(4 * j + 3) * 128 < packed_floats, status, 12)) continue;
            if ((live >> (4 * j)) & 1u) dst[(4 * j + 0) * 128] = x.x;
            if ((live >> (4 * j)) & 2u) dst[(4 * j + 1) * 128] = x.y;
            if ((live >> (4 * j)) & 4u) dst[(4 * j + 2) * 128] = x.z;
            if ((live >> (4 * j)) & 8u) dst[(4 * j + 3) * 128] = x.w;
        }
        __syncwarp();
    }
}

// Any K, any alignment: one thread per pattern byte.  Only used when the fast kernel's
// alignment conditions do not hold.
__global__ void esmm_preprocess_a_patterns_generic_kernel(const float *__restrict__ A, int M, int K,
                                                          int tile_m, int nMB, int nKB,
                                                          uint8_t *__restrict__ out, int *status)
{
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long)nMB * nKB) return;
    const int mb = (int)(idx / nKB), kb = (int)(idx % nKB);
    unsigned pat = 0;
    for (int r = mb * tile_m; r < min(M, (mb + 1) * tile_m); ++r)
        for (int k = 0; k < BK; ++k) {
            const int c = kb * BK + k;
            if (c < K && bounds_ok((size_t)r * K + c < (size_t)M * K, status, 10)) pat |= nz(A[(size_t)r * K + c]) << k;
        }
    out[idx] = (uint8_t)pat;
}

// One warp owns 128 columns (4 pattern column blocks) x 32 k rows (4 K blocks).  Per k row
// every lane tests its 4 columns; a ballot gives 8 bits per column block, nonzero means the
// row is live for that block.  Lanes 0..3 each collect one column block and store the 4
// bytes of the 4 K blocks.  Needs N % 4 == 0 and a 16-byte aligned B.
__global__ void __launch_bounds__(PRE_THREADS)
esmm_preprocess_b_patterns_kernel(const float *__restrict__ B, int K, int N, int nNB, int nKB,
                                  int n_strips, int k_groups, uint8_t *__restrict__ out, int *status)
{
    // checked build, sites 14 (loads of B) and 15 (pattern stores)
    const size_t b_floats = (size_t)K * N, out_bytes = (size_t)nNB * nKB;
    const int lane = threadIdx.x & 31;
    const long warps_total = (long)gridDim.x * (PRE_THREADS / 32);
    const long tasks = (long)n_strips * k_groups;
    for (long task = (long)blockIdx.x * (PRE_THREADS / 32) + (threadIdx.x >> 5); task < tasks;
         task += warps_total) {
        const int kg = (int)(task / n_strips);
        const int strip = (int)(task - (long)kg * n_strips);
        const int col = strip * 128 + lane * 4;
        const bool col_ok = col < N;
        const float *src = B + col;
        unsigned word = 0;  // lane j < 4: byte g = pattern of (column block strip*4+j, K block kg*4+g)
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            const int k0 = (kg * 4 + g) * BK;
            float4 v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (col_ok && k0 + u < K && bounds_ok((size_t)(k0 + u) * N + col + 4 <= b_floats, status, 14))
                    v[u] = __ldg(reinterpret_cast<const float4 *>(src + (size_t)(k0 + u) * N));
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const unsigned bal = __ballot_sync(0xFFFFFFFFu, nz4(v[u]) != 0u);
                const unsigned mine = (bal >> (8 * (lane & 3))) & 0xFFu;
                word |= (mine ? 1u : 0u) << (8 * g + u);
            }
        }
        if (lane < 4) {
            const int nb = strip * 4 + lane;
            if (nb < nNB) {
                uint8_t *dst = out + (size_t)nb * nKB + kg * 4;
                if (kg * 4 + 4 <= nKB && (nKB & 3) == 0) {
                    if (bounds_ok((size_t)nb * nKB + kg * 4 + 4 <= out_bytes, status, 15)) *reinterpret_cast<uint32_t *>(dst) = word;
                } else {
                    for (int g = 0; g < 4; ++g)
                        if (kg * 4 + g < nKB && bounds_ok((size_t)nb * nKB + kg * 4 + g < out_bytes, status, 15))
                            dst[g] = (uint8_t)(word >> (8 * g));
                }
            }
        }
    }
}

__global__ void esmm_preprocess_b_patterns_generic_kernel(const float *__restrict__ B, int K, int N,
                                                          int nNB, int nKB, uint8_t *__restrict__ out, int *status)
{
    const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long)nNB * nKB) return;
    const int nb = (int)(idx / nKB), kb = (int)(idx % nKB);
    unsigned pat = 0;
    for (int k = 0; k < BK; ++k) {
        const int r = kb * BK + k;
        if (r >= K) break;
        for (int c = nb * PAT_N; c < min(N, (nb + 1) * PAT_N); ++c)
            if (bounds_ok((size_t)r * N + c < (size_t)K * N, status, 14)) pat |= nz(B[(size_t)r * N + c]) << k;
    }
    out[idx] = (uint8_t)pat;
}

static int sm_count()
{
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    return sms;
}

int preprocess_a_launch(const float *d_A, int M, int K, int tile_m, uint8_t *d_out, cudaStream_t stream)
{
    if (!d_A || !d_out) return ESMM_ERR_NULL;
    if (M <= 0 || K <= 0 || tile_m <= 0) return ESMM_ERR_SHAPE;
    const int nMB = ceil_div(M, tile_m), nKB = ceil_div(K, BK);
    int *status = kCheckedBuild ? device_status_ptr() : nullptr;   // only the checked build's kernels write it
    if ((K & 3) == 0 && ((uintptr_t)d_A & 15) == 0) {
        const int k_chunks = ceil_div(K, 128);
        const long tasks = (long)nMB * k_chunks;
        const int sms = sm_count();
        if (sms <= 0) return record_cuda_error_text("no CUDA device");
        // Four warps to a task where a warp each would leave the GPU's 64 warps per SM unfilled: 6000^2 (8836 tasks) 27.0 -> 24.6 us,
        // 4096^2 8.3 either way.
        const bool split = tile_m >= 8 * PRE_WARPS && tasks < (long)sms * 64;
        long blocks = split ? tasks : (tasks + PRE_WARPS - 1) / PRE_WARPS;
        const long cap = (long)sms * 16 * 4;
        if (blocks > cap) blocks = cap;
        const auto kernel = split ? esmm_preprocess_a_patterns_kernel<PRE_WARPS> : esmm_preprocess_a_patterns_kernel<1>;
        ESMM_CUDA_TRY(launch_dependent(kernel, dim3((unsigned)blocks), dim3(PRE_THREADS), 0, stream, d_A, M, K, tile_m, nMB, nKB, k_chunks, d_out, status));
    } else {
        const long total = (long)nMB * nKB;
        esmm_preprocess_a_patterns_generic_kernel<<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(
            d_A, M, K, tile_m, nMB, nKB, d_out, status);
    }
    ESMM_CUDA_TRY(cudaGetLastError());
    return ESMM_OK;
}

// strips: the strip kernel comes next, or may.
int preprocess_a_pack_launch(const float *d_A, int M, int K, uint8_t *d_out, float *d_packed,
                             cudaStream_t stream, bool strips)
{
    if (!d_A || !d_out || !d_packed) return ESMM_ERR_NULL;
    if (M <= 0 || K <= 0 || (K & 3)) return ESMM_ERR_SHAPE;
    if (((uintptr_t)d_A | (uintptr_t)d_packed) & 15) return ESMM_ERR_ALIGN;
    const int nMB = ceil_div(M, 32), nKB = ceil_div(K, BK);
    const int sms = sm_count();
    if (sms <= 0) return record_cuda_error_text("no CUDA device");
    int *status = kCheckedBuild ? device_status_ptr() : nullptr;
    const int k_chunks = ceil_div(K, PACK_COLS);
    const long tasks = (long)nMB * k_chunks;
    long blocks = (tasks + PACK_WARPS - 1) / PACK_WARPS;
    const long cap = (long)sms * 8 * 8;
    if (blocks > cap) blocks = cap;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(PACK_WARPS * 32);
    cfg.stream = stream;
    // The strip kernel's CTAs are placed while this kernel ends, and an SM whose shared memory is carved out for less than they need takes
    // none of them until it has (M = 16, K = 4096: 344 strips on 132 of 148 SMs; packing and product by calls of their own, dense, 100 x 1000
    // x 4096 95.5 us without the carve-out, 42.6 with it, 33 x 4096 x 2048 50.1 and 35.0; before tiles it makes no difference).
    cudaLaunchAttribute attr[2];
    int attrs = 0;
    if (!tuning_get("NO_DEPENDENT_LAUNCH", 0)) {
        attr[attrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[attrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (strips) {
        attr[attrs].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
        attr[attrs++].val.sharedMemCarveout = cudaSharedmemCarveoutMaxShared;
    }
    cfg.attrs = attr;
    cfg.numAttrs = attrs;
    // Strips of one row block are placed late where this grid fills the GPU.  Of several row blocks they take the same either way (33 x 4096 x
    // 2048 dense 35.0 and 35.1 us), and tiles, which may come instead, lose by it (255 x 11008 x 8192 dense 1082 us early, 1090 late).
    const int early = !strips || M > 32 || blocks <= sms;
    ESMM_CUDA_TRY(cudaLaunchKernelEx(&cfg, esmm_preprocess_a_pack32_kernel, d_A, M, K, nMB, nKB, k_chunks, d_out, d_packed, status, early));
    ESMM_CUDA_TRY(cudaGetLastError());
    return ESMM_OK;
}

int preprocess_b_launch(const float *d_B, int K, int N, uint8_t *d_out, cudaStream_t stream)
{
    if (!d_B || !d_out) return ESMM_ERR_NULL;
    if (K <= 0 || N <= 0) return ESMM_ERR_SHAPE;
    const int nNB = ceil_div(N, PAT_N), nKB = ceil_div(K, BK);
    int *status = kCheckedBuild ? device_status_ptr() : nullptr;
    if ((N & 3) == 0 && ((uintptr_t)d_B & 15) == 0 && ((uintptr_t)d_out & 3) == 0) {
        const int n_strips = ceil_div(N, 128), k_groups = ceil_div(nKB, 4);
        const long tasks = (long)n_strips * k_groups;
        const int sms = sm_count();
        if (sms <= 0) return record_cuda_error_text("no CUDA device");
        long blocks = (tasks + PRE_THREADS / 32 - 1) / (PRE_THREADS / 32);
        const long cap = (long)sms * 16 * 4;
        if (blocks > cap) blocks = cap;
        esmm_preprocess_b_patterns_kernel<<<(unsigned)blocks, PRE_THREADS, 0, stream>>>(
            d_B, K, N, nNB, nKB, n_strips, k_groups, d_out, status);
    } else {
        const long total = (long)nNB * nKB;
        esmm_preprocess_b_patterns_generic_kernel<<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(
            d_B, K, N, nNB, nKB, d_out, status);
    }
    ESMM_CUDA_TRY(cudaGetLastError());
    return ESMM_OK;
}

}  // namespace esmm

extern "C" {

int esmm_num_k_blocks(int K) { return K > 0 ? esmm::ceil_div(K, esmm::BK) : 0; }

size_t esmm_a_pattern_bytes(int M, int K, int tile_m)
{
    if (M <= 0 || K <= 0 || tile_m <= 0) return 0;
    return (size_t)esmm::ceil_div(M, tile_m) * esmm::ceil_div(K, esmm::BK);
}

size_t esmm_b_pattern_bytes(int K, int N)
{
    if (N <= 0 || K <= 0) return 0;
    return (size_t)esmm::ceil_div(N, esmm::PAT_N) * esmm::ceil_div(K, esmm::BK);
}

int esmm_preprocess_a(const float *d_A, int M, int K, int tile_m, uint8_t *d_out, void *stream)
{
    return esmm::preprocess_a_launch(d_A, M, K, tile_m, d_out, (cudaStream_t)stream);
}

size_t esmm_a_packed_bytes(int M, int K)
{
    if (M <= 0 || K <= 0) return 0;
    return (size_t)esmm::ceil_div(M, 128) * 128 * (size_t)esmm::ceil_div(K, esmm::BK) * esmm::BK * sizeof(float);
}

int esmm_preprocess_a_packed(const float *d_A, int M, int K, uint8_t *d_out, float *d_packed, void *stream)
{
    return esmm::preprocess_a_pack_launch(d_A, M, K, d_out, d_packed, (cudaStream_t)stream, M < esmm::STRIP_ROW_LIMIT);
}

int esmm_preprocess_b(const float *d_B, int K, int N, uint8_t *d_out, void *stream)
{
    return esmm::preprocess_b_launch(d_B, K, N, d_out, (cudaStream_t)stream);
}

int esmm_preprocess_ab(const float *d_A, const float *d_B, int M, int N, int K, int tile_m,
                       const uint8_t *d_b_cached, esmm_ab_pattern_metadata *meta)
{
    if (!meta) return ESMM_ERR_NULL;
    memset(meta, 0, sizeof *meta);
    if (!d_A || (!d_B && !d_b_cached)) return ESMM_ERR_NULL;
    if (M <= 0 || N <= 0 || K <= 0 || tile_m <= 0) return ESMM_ERR_SHAPE;
    meta->numMBlocks = esmm::ceil_div(M, tile_m);
    meta->numNBlocks = esmm::ceil_div(N, esmm::PAT_N);
    meta->numKBlocks = esmm::ceil_div(K, esmm::BK);
    ESMM_CUDA_TRY(cudaMalloc(&meta->d_a_patterns, (size_t)meta->numMBlocks * meta->numKBlocks));
    if (d_b_cached) {
        meta->d_b_patterns = const_cast<uint8_t *>(d_b_cached);
        meta->owns_b_patterns = 0;
    } else {
        cudaError_t e = cudaMalloc(&meta->d_b_patterns, (size_t)meta->numNBlocks * meta->numKBlocks);
        if (e != cudaSuccess) {
            cudaFree(meta->d_a_patterns);
            meta->d_a_patterns = nullptr;
            return esmm::record_cuda_error(e, "cudaMalloc(b patterns)");
        }
        meta->owns_b_patterns = 1;
    }
    int st = esmm::preprocess_a_launch(d_A, M, K, tile_m, meta->d_a_patterns, 0);
    if (st == ESMM_OK && meta->owns_b_patterns) st = esmm::preprocess_b_launch(d_B, K, N, meta->d_b_patterns, 0);
    if (st != ESMM_OK) esmm_free_ab_pattern_metadata(meta);
    return st;
}

int esmm_free_ab_pattern_metadata(esmm_ab_pattern_metadata *meta)
{
    if (!meta) return ESMM_ERR_NULL;
    if (meta->d_a_patterns) cudaFree(meta->d_a_patterns);
    if (meta->owns_b_patterns && meta->d_b_patterns) cudaFree(meta->d_b_patterns);
    meta->d_a_patterns = nullptr;
    meta->d_b_patterns = nullptr;
    return ESMM_OK;
}

}  // extern "C"
