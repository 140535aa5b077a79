// The tiled kernel on row-major A (esmm_gemm_ab): its four instantiations and their launch.
#include "esmm_gemm_tiled.cuh"

namespace esmm {

template <int WMB, bool BLOCKS>
__global__ void __launch_bounds__((P_CONSUMER_WARPS + 4) * 32, 1)
esmm_joint_sgemm_kernel(const __grid_constant__ PackedMaps maps, const __grid_constant__ PackedParams p)
{
    tiled_sgemm<WMB, 3, true, BLOCKS>(maps, p);
}

cudaError_t rowmajor_allow_smem(int bytes)
{
    cudaError_t e = cudaSuccess;
    auto allow = [&](auto kernel) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    };
    allow(esmm_joint_sgemm_kernel<1, false>);
    allow(esmm_joint_sgemm_kernel<1, true>);
    allow(esmm_joint_sgemm_kernel<2, false>);
    allow(esmm_joint_sgemm_kernel<2, true>);
    return e;
}

cudaError_t rowmajor_launch(int tile_rows, bool blocks, int grid, size_t smem, cudaStream_t stream, const PackedMaps &maps,
                            const PackedParams &p)
{
    auto launch = [&](auto kernel) {
        return launch_dependent(kernel, dim3(grid), dim3((P_CONSUMER_WARPS + 4) * 32), smem, stream, maps, p);
    };
    if (tile_rows == 64) return blocks ? launch(esmm_joint_sgemm_kernel<1, true>) : launch(esmm_joint_sgemm_kernel<1, false>);
    return blocks ? launch(esmm_joint_sgemm_kernel<2, true>) : launch(esmm_joint_sgemm_kernel<2, false>);
}

}  // namespace esmm
