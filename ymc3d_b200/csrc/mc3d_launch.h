/*
 * mc3d_launch.h -- launchers of the device code, one per translation unit.
 * The fast and exact photon kernels live in separate files because their math
 * depends on compile flags (-use_fast_math vs -fmad=false).
 */
#ifndef MC3D_LAUNCH_H
#define MC3D_LAUNCH_H

#include <float.h>
#include <math.h>
#include <cuda_runtime.h>
#include "mc3d_device_types.h"

namespace mc3d {

/* kernel variant bits: one step per voxel face instead of merged steps */
#define MC3D_VARIANT_VOXEL_STEPS 2
/* one geometry in the launch: its descriptor is read from the kernel parameters */
#define MC3D_VARIANT_ONE_GEOM 4
/* exact math with IEEE divisions by voxel sizes and mu_t (outside [2^-60, 2^60]) */
#define MC3D_VARIANT_DIVIDE 8
/* fast math for grids with more than MC3D_NARROW_DIM voxels along an axis: the other
 * kernels' voxel indices are exact up to 2^22 */
#define MC3D_VARIANT_WIDE 16
#define MC3D_NARROW_DIM (1 << 21)

static inline int photon_variant_wide(int nx, int ny, int nz)
{
    return nx > MC3D_NARROW_DIM || ny > MC3D_NARROW_DIM || nz > MC3D_NARROW_DIM
               ? MC3D_VARIANT_WIDE : 0;
}

/* mu_t as fast math's kernels, which flush denormals, have it in every expression */
static inline float flushed_mu_t(float mut) { return fabsf(mut) < FLT_MIN ? 0.0f : mut; }

/* dynamic shared memory of a photon kernel: the threads' rows, optical tables, geometry
 * descriptors */
static inline size_t photon_smem(int props_entries, int ngeoms, int block)
{
    return sizeof(unsigned long long) * MC3D_THREAD_WORDS * (size_t)block +
           sizeof(float4) * (size_t)props_entries + sizeof(GeomDev) * (size_t)ngeoms;
}

cudaError_t launch_photon_fast(const KernelParams &P, int grid, int block, size_t smem,
                               cudaStream_t stream, int variant);
cudaError_t launch_photon_exact(const KernelParams &P, int grid, int block, size_t smem,
                                cudaStream_t stream, int variant);
cudaError_t launch_photon_f64(const KernelParams &P, int grid, int block, size_t smem,
                              cudaStream_t stream, int variant);
cudaError_t occupancy_photon_fast(int block, size_t smem, int *blocks_per_sm, int variant);
cudaError_t occupancy_photon_f64(int block, size_t smem, int *blocks_per_sm, int variant);
cudaError_t smem_limit_photon_f64(size_t smem);
cudaError_t attributes_photon_f64(cudaFuncAttributes *attr);
cudaError_t occupancy_photon_exact(int block, size_t smem, int *blocks_per_sm, int variant);
cudaError_t smem_limit_photon_fast(size_t smem);
cudaError_t smem_limit_photon_exact(size_t smem);
cudaError_t attributes_photon_fast(cudaFuncAttributes *attr);
cudaError_t attributes_photon_exact(cudaFuncAttributes *attr);

/* first rejected seeding attempt per job, assuming none before it (UINT64_MAX if none);
 * seeds, if not NULL, gets the state of every launched stream under the same assumption */
cudaError_t launch_seed_scan(const JobDev *jobs, int njobs, const uint32_t *mult,
                             int64_t nmult, const mc3d_seed_consts &sc, int64_t total_streams,
                             unsigned long long *first_reject, uint64_t *seeds,
                             cudaStream_t stream);
/* states of streams [first, first+count) of job 0 of `jobs` */
cudaError_t launch_seed_dump(const KernelParams &P, int64_t first, int64_t count,
                             uint64_t *x_out, uint32_t *a_out, cudaStream_t stream);
/* bytes of scratch that the two launches below need for a grid: two maps of whole
 * words a row, three with the distances of the refractive-index classes; none for a grid
 * at most two voxels wide */
size_t safe_distance_scratch(int nx, int ny, int nz, bool index_map);
/* safe-distance map of a tissue grid: nx * ny * (nz + MC3D_SAFE_CAP) bytes */
cudaError_t launch_safe_distance(const uint8_t *tissue, int nx, int ny, int nz, uint8_t *radius,
                                 uint8_t *scratch, cudaStream_t stream);
/* Packed cells (tissue | box radius << 8) of a grid, nz + MC3D_SAFE_CAP slices.
 * one_tissue: the tissue of a grid that holds no other, else -1 (no scratch then).
 * classes (256 entries, host memory): the refractive-index class of each tissue where
 * some tissues share one, else NULL; one_index: every tissue of the grid is of one
 * class, so that only the faces bound its index (no map of the classes then). */
cudaError_t launch_cells(const uint8_t *tissue, int nx, int ny, int nz, int one_tissue,
                         const uint8_t *classes, bool one_index, uint16_t *cells, uint8_t *scratch,
                         cudaStream_t stream);
cudaError_t launch_mwc_draws(const uint64_t *x, const uint32_t *a, int64_t ngen, int64_t n,
                             float *out, cudaStream_t stream);

} /* namespace mc3d */

#endif
