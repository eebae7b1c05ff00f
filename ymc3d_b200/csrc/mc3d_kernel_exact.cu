/*
 * mc3d_kernel_exact.cu -- the photon kernel with reproducible IEEE math.
 * Built with -fmad=false -prec-div=true -prec-sqrt=true: every operation is
 * correctly rounded and nothing is contracted, so a trajectory matches the CPU
 * transcription bit for bit.
 */
#include "mc3d_engine.cuh"
#include "mc3d_launch.h"

namespace mc3d {

/* Divisions by a voxel size or mu_t by their reciprocals and two corrections, the same
 * correctly rounded quotients as IEEE division (1e5 layered photons: 81.9 ms with
 * divisions, 66.4 ms without); the _wide kernels divide (MC3D_VARIANT_DIVIDE).  96
 * registers, 20 warps an SM, as the fast kernels (4e5 photons: 84.9 ms with 80, 81.0). */
__global__ void __maxnreg__(96) photon_kernel_exact(const __grid_constant__ KernelParams P)
{
    photon_kernel_body<MathExact, false>(P);
}

/* with the per-voxel absorption map */
__global__ void __maxnreg__(96)
    photon_kernel_exact_amap(const __grid_constant__ KernelParams P)
{
    photon_kernel_body<MathExact, true>(P);
}

__global__ void __maxnreg__(96)
    photon_kernel_exact_wide(const __grid_constant__ KernelParams P)
{
    photon_kernel_body<MathExactWide, false>(P);
}

__global__ void __maxnreg__(96)
    photon_kernel_exact_wide_amap(const __grid_constant__ KernelParams P)
{
    photon_kernel_body<MathExactWide, true>(P);
}

typedef void (*photon_kernel_t)(KernelParams);

static photon_kernel_t pick(bool amap, int variant)
{
    if (variant & MC3D_VARIANT_DIVIDE)
        return amap ? photon_kernel_exact_wide_amap : photon_kernel_exact_wide;
    return amap ? photon_kernel_exact_amap : photon_kernel_exact;
}

cudaError_t launch_photon_exact(const KernelParams &P, int grid, int block, size_t smem,
                                cudaStream_t stream, int variant)
{
    pick(P.amap != nullptr, variant)<<<grid, block, smem, stream>>>(P);
    return cudaGetLastError();
}

cudaError_t occupancy_photon_exact(int block, size_t smem, int *blocks_per_sm, int variant)
{
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, pick(false, variant),
                                                         block, smem);
}

cudaError_t smem_limit_photon_exact(size_t smem)
{
    const photon_kernel_t all[] = {photon_kernel_exact, photon_kernel_exact_amap,
                                   photon_kernel_exact_wide, photon_kernel_exact_wide_amap};
    for (photon_kernel_t k : all) {
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t attributes_photon_exact(cudaFuncAttributes *attr)
{
    return cudaFuncGetAttributes(attr, photon_kernel_exact);
}

} /* namespace mc3d */
