// Pieces shared by the joint-sparse GEMM kernels: tiled (packed and row-major A), its block mode, and the strip kernel.
#pragma once

#include <cstdio>
#include <cstdlib>

#include "esmm_common.cuh"
#include "esmm_tiled_layout.h"

namespace esmm {

constexpr int GROUP_M = 8;         // tile rows per raster group

#ifdef __CUDACC__
// Tiles are walked in groups of `group_m` tile rows (GROUP_M unless the launch says otherwise), column by column
// inside a group, so that the CTAs running at the same time share a compact set of A row panels and B column panels
// in L2.  A pass over a group touches the group's A panels and all of B, and B comes from DRAM again for every group.
__device__ __forceinline__ void tile_coords(int tile, int tiles_m, int tiles_n, int &tm, int &tn, int group_m = GROUP_M)
{
    const int per_group = group_m * tiles_n;
    const int group = tile / per_group;
    const int first_m = group * group_m;
    const int gsize = min(tiles_m - first_m, group_m);
    const int r = tile - group * per_group;
    tm = first_m + r % gsize;
    tn = r / gsize;
}

// One k of the tile for one thread: its 4 rows of the top block, 4 rows of the bottom block
// and 2 x 4 columns are one 16-byte load each.
struct KFrag {
    float4 at, ab, b0, b1;
};

// WMB = 32-row blocks per consumer warp: 2 in the 128 x 128 tiling, 1 in the 64 x 128 tiling (where a
// thread holds 4 x 8 outputs and the "bottom" half of everything below is compiled out).
template <int WMB>
__device__ __forceinline__ KFrag load_kfrag(const char *pa, const char *pb)
{
    KFrag f;
    f.at = *reinterpret_cast<const float4 *>(pa);
    if (WMB == 2) f.ab = *reinterpret_cast<const float4 *>(pa + 128);
    f.b0 = *reinterpret_cast<const float4 *>(pb);
    f.b1 = *reinterpret_cast<const float4 *>(pb + 64);
    return f;
}

// The thread's 8 x 8 outputs are held as row pairs for the packed FP32 multiply-add of sm_100 (fma.rn.f32x2: two
// independent IEEE FMAs per instruction, half the issue slots of scalar FFMA):
//   c[p][j] = (c of row 2p, column j; c of row 2p + 1, column j)
// so an FMA takes the row pair (a[2p], a[2p+1]) as it comes from shared memory and one column of B in both halves.  Row
// pairs 0, 1 are the top 32-row block, 2, 3 the bottom one.  Every output still sees one FMA per live k, in ascending k.
// The row pair is the outer loop, so that eight instructions in a row use the same pair: this loop alone, operands in
// shared memory, reaches 67.6 TFLOP/s, which is what fma.rn.f32x2 does with no loads at all; 63.3 with the column as
// the outer loop, and 62.4 with the columns kept as pairs too (diagonal and anti-diagonal of 2 x 2 blocks).
struct Acc {
    float2 c[4][8];
};

__device__ __forceinline__ void acc_clear(Acc &acc)
{
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc.c[i][j] = make_float2(0.0f, 0.0f);
}

// row 2p (e = 0) or 2p + 1 (e = 1), column j
__device__ __forceinline__ float acc_get(const Acc &acc, int p, int e, int j) { return e ? acc.c[p][j].y : acc.c[p][j].x; }

__device__ __forceinline__ void fma_pair_row(Acc &c, int p, float2 ar, const KFrag &f)
{
    const float b[8] = {f.b0.x, f.b0.y, f.b0.z, f.b0.w, f.b1.x, f.b1.y, f.b1.z, f.b1.w};
#pragma unroll
    for (int j = 0; j < 8; ++j) c.c[p][j] = __ffma2_rn(ar, make_float2(b[j], b[j]), c.c[p][j]);
}

__device__ __forceinline__ void fma_top(Acc &c, const KFrag &f)
{
    fma_pair_row(c, 0, make_float2(f.at.x, f.at.y), f);
    fma_pair_row(c, 1, make_float2(f.at.z, f.at.w), f);
}

__device__ __forceinline__ void fma_bottom(Acc &c, const KFrag &f)
{
    fma_pair_row(c, 2, make_float2(f.ab.x, f.ab.y), f);
    fma_pair_row(c, 3, make_float2(f.ab.z, f.ab.w), f);
}

__device__ __forceinline__ void cp_async_commit()
{
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// returns when at most N of this thread's copy groups are still in flight
template <int N>
__device__ __forceinline__ void cp_async_wait_group()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// returns when all of this thread's copies have landed, those too that belong to no committed group (the ones that signal a barrier)
__device__ __forceinline__ void cp_async_wait_all()
{
    asm volatile("cp.async.wait_all;" ::: "memory");
}
#endif  // __CUDACC__

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                  const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_tiled_fn()
{
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
    return fn;
}

// Row-major FP32 matrix of `outer` rows x `inner` columns, box = box_outer x box_inner.
inline int make_map_2d(CUtensorMap *map, const void *base, uint64_t inner, uint64_t outer,
                       uint32_t box_inner, uint32_t box_outer, CUtensorMapSwizzle swz,
                       CUtensorMapL2promotion l2)
{
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return record_cuda_error_text("cuTensorMapEncodeTiled entry point not available");
    cuuint64_t dims[2] = {inner, outer};
    cuuint64_t strides[1] = {inner * 4};
    cuuint32_t box[2] = {box_inner, box_outer};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void *>(base), dims, strides,
                     box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz, l2, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        char buf[96];
        snprintf(buf, sizeof buf, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
        return record_cuda_error_text(buf);
    }
    return ESMM_OK;
}

// 3-D FP32 tensor (d0 fastest, contiguous; strides of d1 and d2 in bytes), box b0 x b1 x b2.
inline int make_map_3d(CUtensorMap *map, const void *base, uint64_t d0, uint64_t d1, uint64_t d2,
                       uint64_t stride1, uint64_t stride2, uint32_t b0, uint32_t b1, uint32_t b2)
{
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return record_cuda_error_text("cuTensorMapEncodeTiled entry point not available");
    cuuint64_t dims[3] = {d0, d1, d2};
    cuuint64_t strides[2] = {stride1, stride2};
    cuuint32_t box[3] = {b0, b1, b2};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void *>(base), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        char buf[96];
        snprintf(buf, sizeof buf, "cuTensorMapEncodeTiled (3-D) failed with CUresult %d", (int)r);
        return record_cuda_error_text(buf);
    }
    return ESMM_OK;
}

}  // namespace esmm
