/*
 * mc3d_safedist.cu -- the safe-distance map of a voxel grid, for merged steps.
 *
 * r(v) is the largest r <= MC3D_SAFE_CAP such that every voxel of the cube of
 * half-width r (Chebyshev radius, in voxels) around v lies inside the grid and
 * has v's tissue.  A photon in voxel v can then cross that whole cube in one
 * step: the voxel-face crossings inside it change nothing in the reference's
 * step (src/mc3d_gpu.cu:181-339 with ni == nt: no Fresnel event, and no
 * absorption or scattering on a hit).
 *
 * The medium does not end at the grid's bottom face: the reference clamps the
 * voxel index (the texture's clamp addressing, src/mc3d_gpu.cu:416-418), so below
 * the grid every column continues with its last voxel.  The map therefore covers
 * nz + MC3D_SAFE_CAP slices, the extra ones standing for that continuation, and
 * only the top and lateral faces (air above, mirrors at the sides) bound it; a
 * photon deeper than the map reads its last slice, which is exact because every
 * slice below the grid is the same.
 *
 * Computation: r is the L-infinity distance transform of the boundary set B
 * (voxels on the top or lateral faces, or with one of their 26 neighbours in
 * another tissue): the nearest other-tissue voxel u of v, at Chebyshev distance
 * d, has a neighbour w of v's tissue at distance d - 1, and w is in B; so r(v) =
 * min over b in B of |v - b|_inf.  That transform is separable:
 *   D1 = distance along x to B, D2 = min_k max(|k|, D1 shifted k along y),
 *   D3 = the same along z over D2.
 * B is kept as one bit per voxel, so D1 is two bit scans.  D2 and D3 work on tiles
 * of 64 voxels by 64 lines in shared memory, two voxels to a register, scanning
 * outward from the voxel until the offset reaches the best value found.  D3 also
 * writes the packed cells.  The scan's 16-bit minima and maxima bound it (issue):
 * 256x256x128 layered, both maps: 3.41 ms with a byte and a 64-bit index per voxel in
 * every pass, 0.57 ms now; 1024x1024x256 in four tissues of one index: 89 ms with both
 * maps, 4.1 ms with the classes' distances from the faces.  The traffic alone, 33 MB and
 * 0.94 GB, would take 5 us and 0.14 ms.
 */
#include <stdint.h>
#include "mc3d_launch.h"

namespace mc3d {

namespace {

/* bytes of a row in the scratch maps: whole 32-bit words */
__host__ __device__ inline int64_t map_pitch(int nx) { return ((int64_t)nx + 3) & ~3ll; }
/* 32-bit words of a row of the boundary bits; never more than map_pitch / 4 */
__host__ __device__ inline int bit_words(int nx) { return (nx + 31) / 32; }

struct ClassTable {
    uint8_t c[256];
};

/* B, one bit per voxel of the map.  A warp takes 32 voxels along x and kSlab slices.
 * The 3x3x3 neighbourhood of a voxel is uniform when its three slices are (3x3 each,
 * nine loads) and their middle voxels agree, so going up z each slice is looked at
 * once.  With CLASSES two tissues are alike when their classes are. */
const int kSlab = 8;

template <bool CLASSES>
__global__ void __launch_bounds__(256) boundary_kernel(const uint8_t *__restrict__ t, int nx, int ny,
                                                       int nz, int nz_map,
                                                       const __grid_constant__ ClassTable lut,
                                                       uint32_t *__restrict__ bits)
{
    __shared__ uint8_t cls[256];
    if (CLASSES) {
        cls[threadIdx.x] = lut.c[threadIdx.x];
        __syncthreads();
    }
    const int words = bit_words(nx);
    const int64_t plane = (int64_t)nx * ny;
    const int lane = threadIdx.x & 31;
    const int64_t slabs = (nz_map + kSlab - 1) / kSlab;
    const int64_t tasks = slabs * ny * words;
    for (int64_t task = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); task < tasks;
         task += (int64_t)gridDim.x * 8) {
        const int w = (int)(task % words);
        const int64_t rest = task / words;
        const int j = (int)(rest % ny);
        const int k0 = (int)(rest / ny) * kSlab;
        const int i = w * 32 + lane;
        const bool inside = i > 0 && i < nx - 1 && j > 0 && j < ny - 1; /* off the lateral faces */
        const uint8_t *col = t + (int64_t)j * nx + i;
        auto other = [&](uint8_t a, uint8_t b) { return a != b && (!CLASSES || cls[a] != cls[b]); };
        /* slice k: its middle voxel, and whether its 3x3 voxels agree with it */
        auto slice = [&](int k, uint8_t *mid) {
            const uint8_t *p = col + (int64_t)min(k, nz - 1) * plane;
            const uint8_t c = p[0];
            bool same = true;
#pragma unroll
            for (int dj = -1; dj <= 1; dj++)
#pragma unroll
                for (int di = -1; di <= 1; di++)
                    if (di || dj) same = same && !other(p[dj * (int64_t)nx + di], c);
            *mid = c;
            return same;
        };
        uint8_t c0 = 0, c1 = 0, c2 = 0;
        bool s0 = false, s1 = false, s2 = false;
        if (inside) {
            s0 = slice(max(k0 - 1, 0), &c0);
            s1 = slice(k0, &c1);
        }
        const int k_end = min(k0 + kSlab, nz_map);
        for (int k = k0; k < k_end; k++) {
            bool b = true;
            if (inside) {
                s2 = slice(k + 1, &c2);
                b = k == 0 || !(s0 && s1 && s2) || other(c0, c1) || other(c2, c1);
                s0 = s1; c0 = c1;
                s1 = s2; c1 = c2;
            }
            const unsigned word = __ballot_sync(0xffffffffu, b && i < nx);
            if (lane == 0) bits[((int64_t)k * ny + j) * words + w] = word;
        }
    }
}

/* D1: offset along x to the nearest set bit of the row, capped; four voxels a thread */
__global__ void __launch_bounds__(256) pass_x_kernel(const uint32_t *__restrict__ bits, int nx,
                                                     int64_t rows, uint8_t *__restrict__ out)
{
    const int words = bit_words(nx);
    const int64_t quads = map_pitch(nx) / 4;
    const int64_t n = rows * quads;
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n;
         v += (int64_t)gridDim.x * blockDim.x) {
        const int64_t row = v / quads;
        const int x0 = (int)(v % quads) * 4;
        const int w = x0 >> 5;
        const uint32_t *r = bits + row * words;
        const uint32_t a = w >= 2 ? r[w - 2] : 0, b = w >= 1 ? r[w - 1] : 0, c = r[w];
        const uint32_t d = w + 1 < words ? r[w + 1] : 0, e = w + 2 < words ? r[w + 2] : 0;
        uint32_t packed = 0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int s = (x0 & 31) + q; /* the voxel's bit in its word */
            /* the 64 bits that end at the voxel, and the 64 that start there */
            const uint64_t left = ((uint64_t)__funnelshift_rc(b, c, s + 1) << 32) |
                                  __funnelshift_rc(a, b, s + 1);
            const uint64_t right = ((uint64_t)__funnelshift_r(d, e, s) << 32) |
                                   __funnelshift_r(c, d, s);
            const int dl = __clzll((long long)left); /* 64 when there is none */
            const int dr = right ? __ffsll((long long)right) - 1 : 64;
            packed |= (uint32_t)min(min(dl, dr), MC3D_SAFE_CAP) << (8 * q);
        }
        reinterpret_cast<uint32_t *>(out)[v] = packed;
    }
}

/* what the z pass writes */
enum { OUT_MAP = 0, OUT_RADIUS, OUT_CELLS };
/* the safe distance of the refractive-index classes that the cells need */
enum { INDEX_AS_TISSUE = 0, INDEX_MAP, INDEX_FACES };

/* The merged kernel's cell: tissue | box radius << 8.  r is the safe distance of the
 * tissue grid (the box holds one tissue); rn is the safe distance of the grid of
 * refractive-index classes (tissues whose index is equal in every optical set used
 * with the geometry share a class).  The box radius min(r, rn - 1) keeps a shell of
 * one voxel between the box and any index change, top face or lateral face, so
 * every reflection happens in a one-voxel step, while a box may still end at a
 * boundary between tissues of equal index, where the reference's step only moves
 * the photon on. */
__device__ inline uint16_t cell_of(int tissue, int r, int rn)
{
    return (uint16_t)(tissue | (min(r, max(rn - 1, 0)) << 8));
}

/* safe distance where only the top and lateral faces bound the medium */
__device__ inline int faces_distance(int i, int j, int k, int nx, int ny)
{
    return min(min(min(i, nx - 1 - i), min(j, ny - 1 - j)), min(k, MC3D_SAFE_CAP));
}

struct PassArgs {
    const uint8_t *in;     /* map rows of map_pitch(nx) bytes, ny rows a slice */
    uint8_t *out;          /* OUT_MAP: the same layout; OUT_RADIUS: nx bytes a row */
    uint16_t *cells;       /* OUT_CELLS */
    const uint8_t *tissue; /* OUT_CELLS: the grid */
    const uint8_t *rn;     /* INDEX_MAP: the classes' distances, map rows */
    int nx, ny, nz, nz_map;
};

const int kLines = 64;                              /* lines of a tile */
const int kTileRows = kLines + 2 * MC3D_SAFE_CAP;   /* with its halo */

/* min over offsets d along an axis (Z: z, else y) of max(|d|, in shifted by d), capped.
 * Outside the lateral and top faces there is nothing nearer than the cap; below the
 * map the last slice goes on. */
template <bool Z, int OUT, int INDEX>
__global__ void __launch_bounds__(256) pass_minmax_kernel(const __grid_constant__ PassArgs A)
{
    __shared__ uint32_t tile[kTileRows][32]; /* 64 voxels a row, two to a word */
    const int64_t pitch = map_pitch(A.nx);
    const int n = Z ? A.nz_map : A.ny;      /* along the axis */
    const int m = Z ? A.ny : A.nz_map;      /* across it */
    const int64_t step = Z ? pitch * A.ny : pitch; /* bytes from line to line */
    const int64_t across = Z ? pitch : pitch * A.ny;
    const int xt = (A.nx + 63) / 64;
    const int lt = (n + kLines - 1) / kLines;
    const int64_t tiles = (int64_t)xt * lt * m;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int64_t tl = blockIdx.x; tl < tiles; tl += gridDim.x) {
        const int x0 = (int)(tl % xt) * 64;
        const int64_t rest = tl / xt;
        const int l0 = (int)(rest % lt) * kLines;
        const int other = (int)(rest / lt);
        const uint8_t *base = A.in + other * across + x0;
        __syncthreads(); /* the last tile has been read */
        for (int w = threadIdx.x; w < kTileRows * 16; w += 256) {
            const int row = w >> 4, q = w & 15;
            int line = l0 - MC3D_SAFE_CAP + row;
            if (Z) line = min(line, n - 1);
            uint32_t v = 0x3f3f3f3fu; /* MC3D_SAFE_CAP */
            if (line >= 0 && line < n && x0 + q * 4 < pitch)
                v = *reinterpret_cast<const uint32_t *>(base + line * step + q * 4);
            tile[row][2 * q] = __byte_perm(v, 0, 0x4140);
            tile[row][2 * q + 1] = __byte_perm(v, 0, 0x4342);
        }
        __syncthreads();
        const int i = x0 + 2 * lane;
        const int last = min(kLines, n - l0);
        if (i < A.nx) {
            for (int q = warp; q < last; q += 8) {
                const uint32_t *at = &tile[q + MC3D_SAFE_CAP][lane];
                uint32_t best = at[0];
                uint32_t d2 = 0x00010001u;
                /* two offsets a turn; one past the best value changes nothing, and with
                 * the cap odd the last is within the halo */
                static_assert(MC3D_SAFE_CAP % 2 == 1, "the scan would leave its tile");
                for (int d = 32; __vmaxu2(best, d2) != d2; d += 64, d2 += 0x00020002u) {
                    best = __vminu2(best, __vmaxu2(d2, __vminu2(at[-d], at[d])));
                    best = __vminu2(best, __vmaxu2(d2 + 0x00010001u,
                                                   __vminu2(at[-d - 32], at[d + 32])));
                }
                const int l = l0 + q;
                const int j = Z ? other : l, k = Z ? l : other;
                const int64_t row = (int64_t)k * A.ny + j;
                const int r0 = (int)(best & 0xffffu), r1 = (int)(best >> 16);
                if (OUT == OUT_MAP) {
                    *reinterpret_cast<uint16_t *>(A.out + row * pitch + i) =
                        (uint16_t)(r0 | (r1 << 8));
                } else {
                    const uint8_t *t = A.tissue + ((int64_t)min(k, A.nz - 1) * A.ny + j) * A.nx;
                    for (int h = 0; h < 2 && i + h < A.nx; h++) {
                        const int r = h ? r1 : r0;
                        if (OUT == OUT_RADIUS) {
                            A.out[row * A.nx + i + h] = (uint8_t)r;
                        } else {
                            const int rn = INDEX == INDEX_AS_TISSUE ? r
                                           : INDEX == INDEX_MAP
                                               ? A.rn[row * pitch + i + h]
                                               : faces_distance(i + h, j, k, A.nx, A.ny);
                            A.cells[row * A.nx + i + h] = cell_of(t[i + h], r, rn);
                        }
                    }
                }
            }
        }
    }
}

/* the cells of a grid of one tissue, which only its faces bound */
__global__ void __launch_bounds__(256) one_tissue_kernel(int tissue, int nx, int ny, int nz_map,
                                                         uint16_t *__restrict__ cells)
{
    const int64_t n = (int64_t)nx * ny * nz_map;
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n;
         v += (int64_t)gridDim.x * blockDim.x) {
        const int64_t row = v / nx;
        const int r = faces_distance((int)(v % nx), (int)(row % ny), (int)(row / ny), nx, ny);
        cells[v] = cell_of(tissue, r, r);
    }
}

/* Whether every voxel lies on a lateral face: all safe distances are 0 then, and rows
 * padded to whole words would take up to four times the grid's own size. */
bool all_on_faces(int nx, int ny) { return nx <= 2 || ny <= 2; }

/* the cells of such a grid */
__global__ void __launch_bounds__(256) on_faces_kernel(const uint8_t *__restrict__ t, int64_t plane,
                                                       int nz, int nz_map,
                                                       uint16_t *__restrict__ cells)
{
    const int64_t n = plane * nz_map;
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n;
         v += (int64_t)gridDim.x * blockDim.x)
        cells[v] = cell_of(t[min(v, plane * (nz - 1) + v % plane)], 0, 0);
}

/* blocks for `want` pieces of work: enough to fill the GPU several times */
int grid_for(int64_t want) { return (int)(want < 148 * 32 ? (want > 0 ? want : 1) : 148 * 32); }

/* B and D1, D2 of the grid (of its classes, if given) into map rows at d2 */
cudaError_t launch_d2(const uint8_t *tissue, int nx, int ny, int nz, const uint8_t *classes,
                      uint8_t *d1, uint8_t *d2, cudaStream_t stream)
{
    const int nz_map = nz + MC3D_SAFE_CAP;
    const int64_t rows = (int64_t)ny * nz_map;
    uint32_t *bits = reinterpret_cast<uint32_t *>(d2); /* read before D2 is written */
    ClassTable lut = {};
    if (classes)
        for (int t = 0; t < 256; t++) lut.c[t] = classes[t];
    const int64_t tasks = (int64_t)((nz_map + kSlab - 1) / kSlab) * ny * bit_words(nx);
    const int blocks = grid_for((tasks + 7) / 8);
    if (classes)
        boundary_kernel<true><<<blocks, 256, 0, stream>>>(tissue, nx, ny, nz, nz_map, lut, bits);
    else boundary_kernel<false><<<blocks, 256, 0, stream>>>(tissue, nx, ny, nz, nz_map, lut, bits);
    pass_x_kernel<<<grid_for((rows * (map_pitch(nx) / 4) + 255) / 256), 256, 0, stream>>>(
        bits, nx, rows, d1);
    PassArgs a = {};
    a.in = d1; a.out = d2;
    a.nx = nx; a.ny = ny; a.nz = nz; a.nz_map = nz_map;
    const int64_t tiles = (int64_t)((nx + 63) / 64) * ((ny + kLines - 1) / kLines) * nz_map;
    pass_minmax_kernel<false, OUT_MAP, INDEX_AS_TISSUE><<<grid_for(tiles), 256, 0, stream>>>(a);
    return cudaGetLastError();
}

int64_t z_tiles(int nx, int ny, int nz)
{
    return (int64_t)((nx + 63) / 64) * ((nz + MC3D_SAFE_CAP + kLines - 1) / kLines) * ny;
}

} /* namespace */

size_t safe_distance_scratch(int nx, int ny, int nz, bool index_map)
{
    if (all_on_faces(nx, ny)) return 0;
    const size_t map = (size_t)map_pitch(nx) * ny * ((size_t)nz + MC3D_SAFE_CAP);
    return map * (index_map ? 3 : 2);
}

cudaError_t launch_safe_distance(const uint8_t *tissue, int nx, int ny, int nz, uint8_t *radius,
                                 uint8_t *scratch, cudaStream_t stream)
{
    if (all_on_faces(nx, ny))
        return cudaMemsetAsync(radius, 0, (size_t)nx * ny * ((size_t)nz + MC3D_SAFE_CAP), stream);
    const size_t map = safe_distance_scratch(nx, ny, nz, false) / 2;
    cudaError_t e = launch_d2(tissue, nx, ny, nz, nullptr, scratch, scratch + map, stream);
    if (e != cudaSuccess) return e;
    PassArgs a = {};
    a.in = scratch + map; a.out = radius; a.tissue = tissue;
    a.nx = nx; a.ny = ny; a.nz = nz; a.nz_map = nz + MC3D_SAFE_CAP;
    pass_minmax_kernel<true, OUT_RADIUS, INDEX_AS_TISSUE>
        <<<grid_for(z_tiles(nx, ny, nz)), 256, 0, stream>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_cells(const uint8_t *tissue, int nx, int ny, int nz, int one_tissue,
                         const uint8_t *classes, bool one_index, uint16_t *cells, uint8_t *scratch,
                         cudaStream_t stream)
{
    const int nz_map = nz + MC3D_SAFE_CAP;
    if (one_tissue >= 0) {
        const int64_t n = (int64_t)nx * ny * nz_map;
        one_tissue_kernel<<<grid_for((n + 255) / 256), 256, 0, stream>>>(one_tissue, nx, ny, nz_map,
                                                                         cells);
        return cudaGetLastError();
    }
    if (all_on_faces(nx, ny)) {
        const int64_t plane = (int64_t)nx * ny;
        on_faces_kernel<<<grid_for((plane * nz_map + 255) / 256), 256, 0, stream>>>(
            tissue, plane, nz, nz_map, cells);
        return cudaGetLastError();
    }
    const size_t map = safe_distance_scratch(nx, ny, nz, false) / 2;
    uint8_t *d1 = scratch, *d2 = scratch + map, *rn = scratch + 2 * map;
    const int blocks = grid_for(z_tiles(nx, ny, nz));
    PassArgs a = {};
    a.in = d2; a.tissue = tissue; a.cells = cells;
    a.nx = nx; a.ny = ny; a.nz = nz; a.nz_map = nz_map;
    cudaError_t e = cudaSuccess;
    if (classes && !one_index) { /* the classes' distances first */
        e = launch_d2(tissue, nx, ny, nz, classes, d1, d2, stream);
        if (e != cudaSuccess) return e;
        PassArgs c = a;
        c.out = rn;
        pass_minmax_kernel<true, OUT_MAP, INDEX_AS_TISSUE><<<blocks, 256, 0, stream>>>(c);
        a.rn = rn;
    }
    e = launch_d2(tissue, nx, ny, nz, nullptr, d1, d2, stream);
    if (e != cudaSuccess) return e;
    if (!classes)
        pass_minmax_kernel<true, OUT_CELLS, INDEX_AS_TISSUE><<<blocks, 256, 0, stream>>>(a);
    else if (one_index)
        pass_minmax_kernel<true, OUT_CELLS, INDEX_FACES><<<blocks, 256, 0, stream>>>(a);
    else pass_minmax_kernel<true, OUT_CELLS, INDEX_MAP><<<blocks, 256, 0, stream>>>(a);
    return cudaGetLastError();
}

} /* namespace mc3d */
