/*
 * mc3d_engine.cuh -- the photon-tracking hot path on sm_100a.
 *
 * One persistent kernel runs every photon of every job in a launch.  The unit of
 * work is an RNG *stream*: stream i of a job owns multiplier a_(i mod M) of the
 * safe-prime table and runs the job's photons i, i+S, i+2S, ... one after
 * another, continuing the same multiply-with-carry sequence, exactly as one
 * photon slot of the reference does (src/mc3d_gpu.cu:74-111, 128-376) minus the
 * masked steps a frozen slot burns until the next host round trip.  Threads take
 * streams from a global counter, so the trajectories depend on (table, seed,
 * photons, streams) and the math and step mode only -- never on the grid shape or on
 * scheduling -- and the tallies, being 64-bit integer sums, are bit-reproducible.
 * Fast merged steps know two things more of their launch: the optical sets that share
 * a geometry, which decide where a box may end (cell_of), and whether it maps the
 * absorption of a single geometry (scatter).
 *
 * Per-step physics follows src/mc3d_gpu.cu:175-340 operation for operation,
 * including its quirks (Fresnel denominator, 0/0 -> transmit at normal incidence,
 * mirror short-circuit after a Fresnel reflection, freeze one step after entering
 * air, i/j/k re-derived from the position every 45 steps, the NaN/db==0 quickfix
 * at the end of each 45-step chunk).  The math policy fixes the transport type
 * and how the elementary operations are evaluated: MathExact uses correctly
 * rounded IEEE operations and the reproducible series of mc3d_exactmath.h
 * (bit-identical to the CPU transcription), MathFast uses the GPU's approximate
 * instructions like the reference's -use_fast_math build, MathF64 steps in FP64.
 * With fast math the face crossings inside cubes of uniform tissue can be merged
 * into one step (photon_step's JUMP).
 */
#ifndef MC3D_ENGINE_CUH
#define MC3D_ENGINE_CUH

#include <limits.h>
#include <stdint.h>
#include <cuda_runtime.h>
#include "mc3d_rng.h"
#include "mc3d_exactmath.h"
#include "mc3d_device_types.h"

namespace mc3d {

#define MC3D_TAB_STRIDE 3   /* float4 per tissue in the optical table */
#define MC3D_TAB64_STRIDE 9 /* doubles per tissue in the FP64 one */

/* ---------------------------------------------------------------- math policies
 * A policy fixes the transport arithmetic type (real) and how the elementary
 * operations are evaluated, and reads the per-tissue coefficients of the optical
 * table (three float4 per tissue, see photon_step).  mul(a, b) is a product rounded
 * on its own; mad(a, b, c) is a b + c, one rounding with fast math and two with the
 * others.  The step uses these two wherever a product feeds a sum, so which
 * products fuse is written down and not the compiler's choice: the tallies do not
 * change with the code around an expression or with the register budget.  One kernel
 * writes it down differently from the others (SPLIT_SIN2, see scatter). */

/* Two values of one step side by side (its x and y axes): the fast policy computes on
 * both with one instruction, the others one after the other. */
template <class R>
struct Pair {
    R a, b;
};

template <class M, class R>
struct PairwiseOps {
    using P2 = Pair<R>;
    static __device__ __forceinline__ P2 mul(P2 x, P2 y)
    {
        return {M::mul(x.a, y.a), M::mul(x.b, y.b)};
    }
    static __device__ __forceinline__ P2 add(P2 x, P2 y) { return {x.a + y.a, x.b + y.b}; }
    static __device__ __forceinline__ P2 sub(P2 x, P2 y) { return {x.a - y.a, x.b - y.b}; }
    static __device__ __forceinline__ P2 mad(P2 x, P2 y, P2 z)
    {
        return {M::mad(x.a, y.a, z.a), M::mad(x.b, y.b, z.b)};
    }
    static __device__ __forceinline__ P2 div(P2 x, P2 y)
    {
        return {M::div(x.a, y.a), M::div(x.b, y.b)};
    }
    static __device__ __forceinline__ P2 div_r(P2 x, P2 y, P2 r)
    {
        return {M::div_r(x.a, y.a, r.a), M::div_r(x.b, y.b, r.b)};
    }
    static __device__ __forceinline__ P2 floor(P2 x) { return {M::floor(x.a), M::floor(x.b)}; }
};

/* FP32 pairs in the packed instructions of sm_100, each rounding as its scalar form */
struct PackedOps {
    using P2 = Pair<float>;
    static __device__ __forceinline__ uint64_t pack(P2 x)
    {
        uint64_t r;
        asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x.a), "f"(x.b));
        return r;
    }
    static __device__ __forceinline__ P2 unpack(uint64_t v)
    {
        P2 r;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(r.a), "=f"(r.b) : "l"(v));
        return r;
    }
    static __device__ __forceinline__ P2 mul(P2 x, P2 y)
    {
        uint64_t r;
        asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack(x)), "l"(pack(y)));
        return unpack(r);
    }
    static __device__ __forceinline__ P2 add(P2 x, P2 y)
    {
        uint64_t r;
        asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack(x)), "l"(pack(y)));
        return unpack(r);
    }
    static __device__ __forceinline__ P2 sub(P2 x, P2 y)
    {
        uint64_t r;
        asm("sub.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack(x)), "l"(pack(y)));
        return unpack(r);
    }
    static __device__ __forceinline__ P2 mad(P2 x, P2 y, P2 z)
    {
        uint64_t r;
        asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;"
            : "=l"(r)
            : "l"(pack(x)), "l"(pack(y)), "l"(pack(z)));
        return unpack(r);
    }
    static __device__ __forceinline__ float rcp(float x)
    {
        float r;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
        return r;
    }
    /* as __fdividef: the product with the approximate reciprocal */
    static __device__ __forceinline__ P2 div(P2 x, P2 y) { return mul(x, P2{rcp(y.a), rcp(y.b)}); }
    static __device__ __forceinline__ P2 div_r(P2 x, P2, P2 r) { return mul(x, r); }
    /* Of |x| <= 2^22 (or NaN, +-inf): 1.5 2^23 + x lies where floats are whole numbers, so
     * rounded down it holds the floor.  Two packed sums in place of two instructions of the
     * quarter-rate unit, which the step keeps busy half the time. */
    static __device__ __forceinline__ P2 floor(P2 x)
    {
        const P2 whole = {12582912.0f, 12582912.0f};
        uint64_t r;
        asm("add.rm.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack(x)), "l"(pack(whole)));
        return sub(unpack(r), whole);
    }
};

/* The same for grids of any size */
struct PackedWideOps : PackedOps {
    static __device__ __forceinline__ P2 floor(P2 x) { return {floorf(x.a), floorf(x.b)}; }
};

/* The FP32 policies read every coefficient as the float the reference computes
 * per step, precomputed on the host. */
struct FloatTable {
    using real = float;
    using Geom = GeomDev;
    using Row = const float4 *; /* of the table in shared memory, MC3D_TAB_STRIDE a tissue */
    static constexpr bool kShared = true; /* table and geometries are read from shared memory */
    static __device__ __forceinline__ Row row(Row tab, int t) { return tab + MC3D_TAB_STRIDE * t; }
    static __device__ __forceinline__ Row table(const KernelParams &, Row shared, int offset)
    {
        return shared + offset;
    }
    static __device__ __forceinline__ const Geom *geom(const KernelParams &, const GeomDev *shared,
                                                       int i)
    {
        return shared + i;
    }
    /* A voxel index clamped into the grid; the first voxel for the NaN position of a
     * photon that the quickfix is about to remove. */
    static __device__ __forceinline__ int cell(float f, int last)
    {
        return min(max((int)f, 0), last);
    }
    static __device__ __forceinline__ float n(const float4 *tt) { return tt[0].w; }
    static __device__ __forceinline__ float mu_t(const float4 *tt) { return tt[1].x; }
    /* mua / mu_t, 0 where mu_t is not positive */
    static __device__ __forceinline__ float albedo_c(const float4 *tt) { return tt[1].z; }
    static __device__ __forceinline__ float rmu_t(const float4 *tt) { return tt[1].y; }
    /* Henyey-Greenstein cos(theta) for the draw xi in (0, 1] (src/mc3d_gpu.cu:282-286) */
    template <class M>
    static __device__ __forceinline__ float hg_cos(const float4 *tt, float xi)
    {
        const float4 t2 = tt[2];
        const float c = M::div(t2.x, M::mad(t2.z, xi, t2.y));
        return M::mul(tt[1].w, M::mad(-c, c, t2.w));
    }
    /* thresholds of src/mc3d_types.h:11-18, see the constants below */
    static __device__ __forceinline__ bool w_below_threshold(float w) { return w <= 0x1.a36e2ep-14f; }
    static __device__ __forceinline__ bool w_above_threshold(float w) { return w > 0x1.a36e2ep-14f; }
    static __device__ __forceinline__ bool uz_within(float u) { return u <= 0x1.fffeb0p-1f; }
    static __device__ __forceinline__ float roulette_survivor(float w)
    {
        return (float)((double)w / 0.1);
    }
    static __device__ __forceinline__ float zero_threshold() { return (float)(1 - 0.99999); }
    /* Whether a step needs the work that few do (photon_step).  One chain of compares,
     * each taking the result so far: written in C the terms are combined by predicate
     * instructions of their own (8.6 of the step's 192, 5.2 of 188 this way). */
    static __device__ __forceinline__ bool rare(uint32_t changed, float W, float mu_t, float uz,
                                                float least_u, float x, float Lx, float y, float Ly)
    {
        uint32_t any;
        asm("{\n\t.reg .pred p;\n\t"
            "setp.ne.u32 p, %1, 0;\n\t"
            "setp.leu.or.f32 p, %2, %3, p;\n\t"
            "setp.eq.or.f32 p, %4, 0f00000000, p;\n\t"
            "setp.gtu.or.f32 p, %5, %6, p;\n\t"
            "setp.lt.or.f32 p, %7, %8, p;\n\t"
            "setp.leu.or.f32 p, %9, 0f00000000, p;\n\t"
            "setp.geu.or.f32 p, %9, %10, p;\n\t"
            "setp.leu.or.f32 p, %11, 0f00000000, p;\n\t"
            "setp.geu.or.f32 p, %11, %12, p;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(any)
            : "r"(changed), "f"(W), "f"(0x1.a36e2ep-14f), "f"(mu_t), "f"(fabsf(uz)),
              "f"(0x1.fffeb0p-1f), "f"(least_u), "f"(zero_threshold()), "f"(x), "f"(Lx), "f"(y),
              "f"(Ly));
        return any != 0;
    }
    /* fixed-point weight, 2^-32 resolution */
    static __device__ __forceinline__ uint64_t qw(float w) { return __float2ull_rn(w * 4294967296.0f); }
};

struct MathExact : FloatTable {
    static constexpr bool kFast = false;
    using Pairs = PairwiseOps<MathExact, float>;
    static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
    static __device__ __forceinline__ float mad(float a, float b, float c) { return a * b + c; }
    static __device__ __forceinline__ float div(float a, float b) { return a / b; }
    /* a / b, correctly rounded, by r = 1 / b correctly rounded, as MathF64::div_r */
    static __device__ __forceinline__ float div_r(float a, float b, float r)
    {
        float q = a * r;
        q = __fmaf_rn(__fmaf_rn(-q, b, a), r, q);
        return __fmaf_rn(__fmaf_rn(-q, b, a), r, q);
    }
    /* x + u t for a hit, x + us / mu_t for a scattering; us is u or u s */
    static __device__ __forceinline__ float advance(float x, float us, bool hit, float t, float mu_t,
                                                    float rmu_t)
    {
        return x + (hit ? us * t : div_r(us, mu_t, rmu_t));
    }
    static __device__ __forceinline__ float sqrt(float x) { return sqrtf(x); }
    static __device__ __forceinline__ float rsqrt(float x) { return 1.0f / sqrtf(x); }
    static __device__ __forceinline__ float log(float x) { return mc3d_xm_logf(x); }
    static __device__ __forceinline__ float acos(float x) { return mc3d_xm_acosf(x); }
    static __device__ __forceinline__ float sin(float x) { return mc3d_xm_sinf(x); }
    /* sin and cos of the azimuth 2 pi e 2^-32 */
    static __device__ __forceinline__ void sincos_draw(uint32_t e, float *s, float *c)
    {
        mc3d_xm_sincospif(2 * (mc3d_u32_to_float_rz(e) * 0x1p-32f), s, c);
    }
    static __device__ __forceinline__ float floor(float x) { return floorf(x); }
    static __device__ __forceinline__ float fmin(float a, float b) { return fminf(a, b); }
    static __device__ __forceinline__ float fabs(float x) { return fabsf(x); }
    static __device__ __forceinline__ float copysign(float a, float b) { return copysignf(a, b); }
};

/* The same with IEEE divisions, for voxel sizes and coefficients whose reciprocals, or
 * the residuals of the quotients, leave FP32's normal range. */
struct MathExactWide : MathExact {
    using Pairs = PairwiseOps<MathExactWide, float>; /* x and y divide too */
    static __device__ __forceinline__ float div_r(float a, float b, float) { return a / b; }
    static __device__ __forceinline__ float advance(float x, float us, bool hit, float t, float mu_t,
                                                    float)
    {
        return x + (hit ? us * t : us / mu_t);
    }
};

/* Compiled only in a translation unit built with -use_fast_math, where the
 * operators and functions below map to the approximate hardware paths. */
struct MathFast : FloatTable {
    static constexpr bool kFast = true;
    using Pairs = PackedOps;
    /* The index f - 1 as a multiple of the least denormal float has f - 1 itself as its
     * bits (up to 2^24, and larger bits for larger f), a sign bit below 1, and NaN's bits
     * plus one wrap below 0: a fused multiply and an add with the clamps in place of a
     * conversion, which runs at a quarter of their rate.  With PackedOps::floor: the
     * quarter-rate unit has 13 instead of 18 instructions a step; layered 1e7 163.4 ->
     * 161.2 ms, per-face 1e6 100.7 -> 96.7 ms, skin model 3.36 -> 3.15 ms. */
    static __device__ __forceinline__ int cell(float f, int last)
    {
        float v;
        asm("fma.rn.f32 %0, %1, 0f00000001, 0f80000001;" : "=f"(v) : "f"(f));
        return __viaddmin_s32_relu(__float_as_int(v), 1, last);
    }
    static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
    static __device__ __forceinline__ float mad(float a, float b, float c) { return __fmaf_rn(a, b, c); }
    /* every denominator divided here is a direction cosine, a sum of products of
     * cosines and sines, a refractive-index sum or 1 - g + 2 g xi, all far below the
     * 2^126 where __fdividef stops being defined; x / 0 still gives +-inf or NaN */
    static __device__ __forceinline__ float div(float a, float b) { return __fdividef(a, b); }
    static __device__ __forceinline__ float div_r(float a, float, float r) { return __fmul_rn(a, r); }
    static __device__ __forceinline__ float advance(float x, float us, bool hit, float t, float,
                                                    float rmu_t)
    {
        return __fmaf_rn(us, hit ? t : rmu_t, x);
    }
    static __device__ __forceinline__ float sqrt(float x) { return sqrtf(x); }
    static __device__ __forceinline__ float rsqrt(float x) { return rsqrtf(x); }
    static __device__ __forceinline__ float log(float x) { return logf(x); }
    static __device__ __forceinline__ float acos(float x) { return acosf(x); }
    static __device__ __forceinline__ float sin(float x) { return sinf(x); }
    /* the SFU's sin/cos on the azimuth less pi, in [-pi, pi) */
    static __device__ __forceinline__ void sincos_draw(uint32_t e, float *s, float *c)
    {
        float sn, cs;
        const float x = __fmaf_rn(mc3d_u32_to_float_rz(e), 0x1p-31f, -1.0f);
        __sincosf(__fmul_rn(3.14159265358979f, x), &sn, &cs);
        *s = -sn;
        *c = -cs;
    }
    static __device__ __forceinline__ float floor(float x) { return floorf(x); }
    static __device__ __forceinline__ float fmin(float a, float b) { return fminf(a, b); }
    static __device__ __forceinline__ float fabs(float x) { return fabsf(x); }
    static __device__ __forceinline__ float copysign(float a, float b) { return copysignf(a, b); }
};

/* The same for grids with more than MC3D_NARROW_DIM voxels along an axis */
struct MathFastWide : MathFast {
    using Pairs = PackedWideOps;
    static __device__ __forceinline__ int cell(float f, int last)
    {
        return FloatTable::cell(f, last);
    }
};

/* FP64 stepping: the same loop with every transport quantity in double, the
 * coefficients derived in double from the sets' float (mua, mus, g, n), and
 * the reference's double literals compared in double.  Random numbers stay the
 * reference's 32-bit draws.  Built with IEEE division and square root; the
 * precision reference for the FP32 policies. */
struct MathF64 {
    using real = double;
    static constexpr bool kFast = false;
    using Pairs = PairwiseOps<MathF64, double>;
    static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
    static __device__ __forceinline__ double mad(double a, double b, double c) { return a * b + c; }
    static __device__ __forceinline__ double div(double a, double b) { return a / b; }
    /* a / b, correctly rounded, by r = 1 / b correctly rounded: the product with r and two
     * corrections by the residual, which a fused multiply-add gives exactly (Markstein,
     * IBM J. Res. Dev. 34, 1990: a quotient within one ulp becomes the nearest; the first
     * correction brings it there).  5 instructions and no branch instead of about 16. */
    static __device__ __forceinline__ double div_r(double a, double b, double r)
    {
        double q = a * r;
        q = __fma_rn(__fma_rn(-q, b, a), r, q);
        return __fma_rn(__fma_rn(-q, b, a), r, q);
    }
    static __device__ __forceinline__ double advance(double x, double us, bool hit, double t,
                                                     double mu_t, double rmu_t)
    {
        return x + (hit ? us * t : div_r(us, mu_t, rmu_t));
    }
    static __device__ __forceinline__ double sqrt(double x) { return ::sqrt(x); }
    static __device__ __forceinline__ double rsqrt(double x) { return 1.0 / ::sqrt(x); }
    static __device__ __forceinline__ double log(double x) { return ::log(x); }
    static __device__ __forceinline__ double acos(double x) { return ::acos(x); }
    static __device__ __forceinline__ double sin(double x) { return ::sin(x); }
    static __device__ __forceinline__ void sincos_draw(uint32_t e, double *s, double *c)
    {
        ::sincospi(2 * (double)(mc3d_u32_to_float_rz(e) * 0x1p-32f), s, c);
    }
    static __device__ __forceinline__ double floor(double x) { return ::floor(x); }
    static __device__ __forceinline__ double fmin(double a, double b) { return ::fmin(a, b); }
    static __device__ __forceinline__ double fabs(double x) { return ::fabs(x); }
    static __device__ __forceinline__ double copysign(double a, double b) { return ::copysign(a, b); }
    using Geom = GeomDev64;
    using Row = const double *; /* of the table in global memory, MC3D_TAB64_STRIDE a tissue */
    static constexpr bool kShared = false;
    static __device__ __forceinline__ Row row(Row tab, int t) { return tab + MC3D_TAB64_STRIDE * t; }
    static __device__ __forceinline__ Row table(const KernelParams &P, const float4 *, int offset)
    {
        return P.props64 + (offset / MC3D_TAB_STRIDE) * MC3D_TAB64_STRIDE;
    }
    static __device__ __forceinline__ const Geom *geom(const KernelParams &P, const GeomDev *, int i)
    {
        return P.geoms64 + i;
    }
    /* A voxel index clamped into the grid.  NaN, less the face rule's one, wraps to the
     * last voxel. */
    static __device__ __forceinline__ int cell(double f, int last)
    {
        return min(max(f == f ? (int)f : INT_MAX, 0), last);
    }
    static __device__ __forceinline__ double mu_t(Row tt) { return tt[0]; }
    static __device__ __forceinline__ double rmu_t(Row tt) { return tt[1]; }
    static __device__ __forceinline__ double albedo_c(Row tt) { return tt[2]; }
    static __device__ __forceinline__ double n(Row tt) { return tt[3]; }
    template <class M>
    static __device__ __forceinline__ double hg_cos(Row tt, double xi)
    {
        const double c = tt[4] / (tt[5] + tt[6] * xi);
        return div_r(tt[7] - c * c, tt[6], tt[8]);
    }
    static __device__ __forceinline__ bool w_below_threshold(double w) { return w < 0.0001; }
    static __device__ __forceinline__ bool w_above_threshold(double w) { return w >= 0.0001; }
    static __device__ __forceinline__ bool uz_within(double u) { return u <= 0.99999; }
    static __device__ __forceinline__ double roulette_survivor(double w) { return w / 0.1; }
    static __device__ __forceinline__ double zero_threshold() { return 1 - 0.99999; }
    static __device__ __forceinline__ bool rare(uint32_t changed, double W, double mu_t, double uz,
                                                double least_u, double x, double Lx, double y,
                                                double Ly)
    {
        return changed | !w_above_threshold(W) | (mu_t == 0) | !uz_within(fabs(uz)) |
               (least_u < zero_threshold()) | !(x > 0) | !(x < Lx) | !(y > 0) | !(y < Ly);
    }
    static __device__ __forceinline__ uint64_t qw(double w)
    {
        return __double2ull_rn(w * 4294967296.0);
    }
};

/* ------------------------------------------------------------ reference constants
 * src/mc3d_types.h:11-18.  SURVIVAL_CHANCE, W_THRESHOLD and UZ_THRESH are double
 * literals there, so a float compared with them is widened to double.  No float
 * lies between each literal and the float bound below, so these float comparisons
 * decide exactly as the double ones do (the unit tests enumerate the neighbours):
 *   (double)e <  0.1      <=>  e <  0x1.99999ap-4f   ((float)0.1 is above 0.1)
 *   (double)w <  0.0001   <=>  w <= 0x1.a36e2ep-14f  ((float)0.0001 is below it)
 *   (double)u <= 0.99999  <=>  u <= 0x1.fffeb0p-1f   ((float)0.99999 is below it)
 * The roulette division W / 0.1 stays in double, as in the reference. */
#define MC3D_SURVIVAL_CHANCE 0.1
#define MC3D_SURVIVAL_LT_F 0x1.99999ap-4f
#define MC3D_W_THRESHOLD_LE_F 0x1.a36e2ep-14f
#define MC3D_UZ_THRESH 0.99999
#define MC3D_UZ_THRESH_LE_F 0x1.fffeb0p-1f
/* fast math: |1 - sin^2(theta_t)| below this takes the FP64 Fresnel branch */
#define MC3D_NEAR_CRITICAL_F 0x1p-5f
#define MC3D_NUM_PHOTON_STEPS 45
#define MC3D_TISSUE_AIR 0


/* 1 for a direction that moves up the axis (u >= 0), 0 for one that moves down */
template <class R>
static __device__ __forceinline__ R upward(R u)
{
    return u >= 0 ? (R)1 : (R)0;
}

/* Voxel index of x along one axis (src/mc3d_gpu.cu:53-63), as a real: exact below
 * 2^24, NaN for a NaN position; up = upward(u).  The reference takes i = floor(x / d),
 * steps up when x lies on the upper face, and keeps a voxel only when x is above its
 * lower face or on it moving up.  So floor's value stands unless x lies on the face
 * that the photon moves through (one voxel on) or, floor's argument having been
 * rounded up, below the lower face (one voxel back).  Written as arithmetic on 0 and
 * 1: as predicates the three axes need more of them than a thread has. */
template <class M, class R = typename M::real>
static __device__ __forceinline__ R grid_index(R x, R up, R d, R rd)
{
    const R fi = M::floor(M::div_r(x, d, rd));
    const R on_face = x == M::mul(fi + up, d) ? (R)1 : (R)0;
    const R below = x >= M::mul(fi, d) ? (R)0 : (R)1;
    return M::mad(on_face, M::mad((R)2, up, (R)-1), fi) - below;
}

/* grid_index of the x and y axes */
template <class M, class G, class R = typename M::real>
static __device__ __forceinline__ Pair<R> grid_index2(Pair<R> x, Pair<R> up, const G &g)
{
    using Two = typename M::Pairs;
    using P2 = Pair<R>;
    const P2 d = {(R)g.dx, (R)g.dy};
    const P2 q = Two::div_r(x, d, P2{(R)g.rdx, (R)g.rdy});
    const P2 f = Two::floor(q);
    const P2 face = Two::mul(Two::add(f, up), d), lo = Two::mul(f, d);
    const P2 on_face = {x.a == face.a ? (R)1 : (R)0, x.b == face.b ? (R)1 : (R)0};
    const P2 below = {x.a >= lo.a ? (R)0 : (R)1, x.b >= lo.b ? (R)0 : (R)1};
    const P2 way = Two::mad(P2{(R)2, (R)2}, up, P2{(R)-1, (R)-1});
    return Two::sub(Two::mad(on_face, way, f), below);
}

/* src/mc3d_gpu.cu:24-27 with the clamp addressing of the texture (:416-418).
 * With JUMP the lookup reads the packed map (tissue | box radius << 8, one
 * 16-bit load), so the box radius rides in bits 8-15 of the result (0 above
 * the surface, where the tissue is air). */
template <class M, bool JUMP = false, class G, class R>
static __device__ __forceinline__ int tissue_at(const G &g, R fi, R fj, R fk, R z, R uz)
{
    const int ci = M::cell(fi, g.last_x);
    const int cj = M::cell(fj, g.last_y);
    const int ck = M::cell(fk, g.last_z);
    int t;
    if (JUMP) {
        /* 32-bit index: plans take merged steps only for maps below 2^32 cells */
        t = __ldg(g.cells + (((uint32_t)ck * (uint32_t)g.ny + (uint32_t)cj) * (uint32_t)g.nx +
                             (uint32_t)ci));
    } else {
        t = __ldg(g.tissue + ((int64_t)ck * g.ny + cj) * g.nx + ci);
    }
    return ((z <= 0) & (uz < 0)) ? MC3D_TISSUE_AIR : t;
}

/* Distance to one face of the step's box along an axis (src/mc3d_gpu.cu:29-49): the
 * box reaches r voxels beyond the photon's voxel fi on either side.  The border is
 * a rounded product, as the reference's separate multiply gives it: fused into the
 * subtraction that follows, a photon lying exactly on a face would see its distance
 * to that face as the product's rounding error instead of 0. */
template <class M, class R = typename M::real>
static __device__ __forceinline__ R face_distance(R x, R u, R up, R fi, R r, R d, R *border)
{
    /* fi + r + 1 upward, fi - r downward (whole numbers: exact) */
    *border = M::mul(fi + M::mad(up, M::mad((R)2, r, (R)1), -r), d);
    return M::div(*border - x, u);
}

/* face_distance of the x and y axes */
template <class M, class G, class R = typename M::real>
static __device__ __forceinline__ Pair<R> face_distance2(Pair<R> x, Pair<R> u, Pair<R> up,
                                                         Pair<R> fi, R r, const G &g,
                                                         Pair<R> *border)
{
    using Two = typename M::Pairs;
    const R span = M::mad((R)2, r, (R)1);
    const Pair<R> off = {M::mad(up.a, span, -r), M::mad(up.b, span, -r)};
    *border = Two::mul(Two::add(fi, off), Pair<R>{(R)g.dx, (R)g.dy});
    return Two::div(Two::sub(*border, x), u);
}

/* src/mc3d_gpu.cu:113-126 */
template <class M, class R = typename M::real>
static __device__ __forceinline__ bool mirror(R *x, R *ux, R length)
{
    bool refl = (*x >= length) || (*x <= 0);
    *x = (*x >= length) ? 2 * length - *x : *x;
    *x = (*x <= 0) ? M::fabs(*x) : *x;
    *ux = refl ? -1 * (*ux) : *ux;
    return refl;
}

template <class R>
struct PhotonT {
    R x, y, z, ux, uy, uz, W, s;
    R i, j, k; /* voxel index, as a real: the step's borders need no conversion */
    int tissue;
};

/* Per-thread tallies live in shared memory, one row per thread, so that the
 * step loop keeps only the photon in registers.  They are touched when a photon
 * ends or at a roulette event, and flushed to the job's totals when the thread
 * moves to another stream.  Slot order is mc3d_totals (include/mc3d.h). */
enum {
    T_PHOTONS = 0, T_STEPS, T_W_LAUNCHED, T_R_IN, T_R_OUT, T_T_IN, T_T_OUT, T_ABSORBED,
    T_RR_KILLED, T_RR_CREATED, T_LOST, T_CAPPED, T_QUICKFIX, T_FRESNEL
};

struct Acc {
    unsigned long long *row; /* the thread's MC3D_THREAD_WORDS words of shared memory */
    __device__ __forceinline__ unsigned long long &operator[](int t) const { return row[t]; }
    /* of the thread's stream: photons left and job-local index */
    __device__ __forceinline__ int64_t &left() const { return (int64_t &)row[MC3D_NUM_TOTALS]; }
    __device__ __forceinline__ int64_t &local() const { return (int64_t &)row[MC3D_NUM_TOTALS + 1]; }
};

/* Henyey-Greenstein scattering of the direction of p, src/mc3d_gpu.cu:282-294, by the
 * draws e_hg (cosine) and e_phi (azimuth): the direction by the general formula, and
 * the angles for the one along the z axis. */
template <class R>
struct Spin {
    R ux, uy, uz, costheta, sintheta, cosphi, sinphi;
};

template <class M, bool SPLIT_SIN2, class R = typename M::real>
static __device__ __forceinline__ Spin<R> scatter(typename M::Row tt, const PhotonT<R> &p,
                                                  uint32_t e_hg, uint32_t e_phi)
{
    Spin<R> o;
    const R xi = (R)(1.0f - mc3d_u32_to_float_rz(e_hg) * 0x1p-32f);
    o.costheta = M::template hg_cos<M>(tt, xi);
    /* 1 - cos^2 with one rounding, but with two in the fast merged-step kernel that maps
     * one geometry's absorption: that kernel has always rounded the square by itself, and
     * a seeded run repeats its tallies */
    o.sintheta = M::sqrt(SPLIT_SIN2 ? (R)1 - M::mul(o.costheta, o.costheta)
                                    : M::mad(-o.costheta, o.costheta, (R)1));
    M::sincos_draw(e_phi, &o.sinphi, &o.cosphi);
    const R sin2 = M::mad(-p.uz, p.uz, (R)1);
    const R invsqrt = M::rsqrt(sin2);
    const R Ax = M::mad(-p.uy, o.sinphi, M::mul(M::mul(p.ux, p.uz), o.cosphi));
    const R Ay = M::mad(p.ux, o.sinphi, M::mul(M::mul(p.uy, p.uz), o.cosphi));
    o.ux = M::mad(p.ux, o.costheta, M::mul(M::mul(o.sintheta, Ax), invsqrt));
    o.uy = M::mad(p.uy, o.costheta, M::mul(M::mul(o.sintheta, Ay), invsqrt));
    o.uz = M::mad(p.uz, o.costheta, M::mul(M::mul(-M::sqrt(sin2), o.sintheta), o.cosphi));
    return o;
}

/* One step of src/mc3d_gpu.cu:175-340 for a live photon.  Returns true when the
 * photon froze during this step; *db receives the step's boundary distance.
 *
 * JUMP (merged steps): p.tissue carries a box radius r in bits 8-15, and the
 * step's box is the cube of voxels within Chebyshev distance r of the photon's
 * voxel.  The box holds only the photon's tissue, and a shell of one voxel around
 * it has the photon's refractive index and stays clear of the top and lateral
 * faces (cell_of): a step that reaches a box face crosses into a voxel of the
 * same index, with no Fresnel event, no mirror and no air rule, exactly as the
 * reference's step at that face would (snapped, next voxel by the face rule; that
 * voxel may hold another tissue of the same index, whose coefficients the next
 * step uses).
 * The face crossings inside the box, which in the reference only move the
 * photon (no absorption or scattering; their four random numbers are drawn and
 * discarded), are merged into this one step.  Every reflection therefore
 * happens in a one-voxel step (r = 0), where the reference's rule applies
 * unchanged: a reflected photon keeps the voxel index it started the step with
 * (src/mc3d_gpu.cu:334-339).  That rule can leave the index one voxel off when a
 * coordinate that was not snapped rounded onto a face; the photon then takes
 * zero-length steps until the quickfix at its chunk's end removes it, which is
 * part of the weight the reference loses.
 *
 * Bound by instruction issue, so the straight line holds what most lanes do and all else
 * stands behind one test: 188 thread-instructions a merged step (283 when every rule had
 * its own branch), layered 1e7 photons 221.7 -> 163.4 ms. */
template <class M, bool AMAP, bool JUMP, bool ONE_GEOM, class R = typename M::real>
static __device__ __forceinline__ bool photon_step(const typename M::Geom &g, typename M::Row tab,
                                                   PhotonT<R> &p, uint64_t &rx, uint32_t ra,
                                                   const Acc &acc, R *db_out,
                                                   unsigned long long *amap, bool *lat_mirror)
{
    constexpr bool SPLIT_SIN2 = M::kFast && AMAP && JUMP && ONE_GEOM; /* see scatter */
    /* per tissue: (mua, mus, g, n), (mu_t, 1/mu_t, mua/mu_t, 1/(2g)),
     * (1-g^2, 1-g, 2g, 1+g^2) -- each the float the reference computes per step */
    const typename M::Row tt = M::row(tab, JUMP ? (p.tissue & 0xff) : p.tissue);
    const R mu_t = M::mu_t(tt);

    /* the box's nearest face, src/mc3d_gpu.cu:29-49 */
    const R r = JUMP ? (R)(p.tissue >> 8) : (R)0;
    using P2 = Pair<R>;
    const P2 up = {upward(p.ux), upward(p.uy)};
    const R up_z = upward(p.uz);
    P2 bxy;
    R bz;
    const P2 t_xy = face_distance2<M>({p.x, p.y}, {p.ux, p.uy}, up, {p.i, p.j}, r, g, &bxy);
    const R t_z = face_distance<M>(p.z, p.uz, up_z, p.k, r, g.dz, &bz);
    const R db = M::fmin(t_xy.a, M::fmin(t_xy.b, t_z));
    *db_out = db;

    /* move to that face or to the interaction, whichever is nearer: one expression
     * for both, u 1 db or u s / mu_t from the position, snapped to the face hit */
    const R ds = M::mul(db, mu_t);
    const bool hit = ds <= p.s;
    const R m = hit ? (R)1 : p.s;
    const R rmu_t = M::rmu_t(tt);
    R newx = M::advance(p.x, M::mul(p.ux, m), hit, db, mu_t, rmu_t);
    R newy = M::advance(p.y, M::mul(p.uy, m), hit, db, mu_t, rmu_t);
    R newz = M::advance(p.z, M::mul(p.uz, m), hit, db, mu_t, rmu_t);
    const R face = hit ? db : (R)__int_as_float(0x7fc00000); /* NaN: no face */
    newx = (face == t_xy.a) ? bxy.a : newx;
    newy = (face == t_xy.b) ? bxy.b : newy;
    newz = (face == t_z) ? bz : newz;
    const R s = p.s - ds; /* what a hit leaves of the free path */

    const P2 nextij = grid_index2<M>(P2{newx, newy}, up, g);
    R nexti = nextij.a, nextj = nextij.b;
    R nextk = grid_index<M>(newz, up_z, g.dz, g.rdz);
    int next_tissue = tissue_at<M, JUMP>(g, nexti, nextj, nextk, newz, p.uz);

    /* the step's draws: roulette, scattering cosine and azimuth, next free path */
    rx = mc3d_mwc_next(rx, ra);
    uint32_t e_rr = (uint32_t)rx;
    rx = mc3d_mwc_next(rx, ra);
    uint32_t e_hg = (uint32_t)rx;
    rx = mc3d_mwc_next(rx, ra);
    uint32_t e_phi = (uint32_t)rx;
    rx = mc3d_mwc_next(rx, ra);
    uint32_t e_s = (uint32_t)rx;

    /* Absorption, src/mc3d_gpu.cu:262-263.  Fast math selects; the others multiply by 0 or
     * 1 as the reference does, which makes an infinite weight (a medium with gain) NaN at
     * the next face. */
    R W;
    if (M::kFast) {
        W = p.W - (hit ? (R)0 : M::mul(M::albedo_c(tt), p.W));
    } else {
        const R dW = mu_t > 0 ? M::mul(M::albedo_c(tt), p.W) : (R)0;
        W = p.W - M::mul(dW, hit ? (R)0 : (R)1);
    }
    if (AMAP && !hit && mu_t > 0) {
        /* absorption map, the reference's disabled tally (src/mc3d_gpu.cu:265-272):
         * the current voxel clamped into the grid, fixed-point weight removed.  A
         * merged step can end its flight several voxels from where it started, so
         * there the voxel of the interaction point is used.  A photon without a
         * position (NaN, of a tissue with g = 0) tallies where its cell is looked up. */
        const int ai = M::cell(JUMP ? nexti : p.i, g.last_x);
        const int aj = M::cell(JUMP ? nextj : p.j, g.last_y);
        const int ak = M::cell(JUMP ? nextk : p.k, g.nz - 1);
        const uint64_t dq = M::qw(p.W) - M::qw(W);
        if (dq) atomicAdd(amap + ((int64_t)ak * g.ny + aj) * g.nx + ai, (unsigned long long)dq);
    }

    /* the scattered direction, or for a hit the old one */
    R nux = p.ux, nuy = p.uy, nuz = p.uz;
    const Spin<R> spin = scatter<M, SPLIT_SIN2>(tt, p, e_hg, e_phi);
    nux = (!hit) ? spin.ux : nux;
    nuy = (!hit) ? spin.uy : nuy;
    nuz = (!hit) ? spin.uz : nuz;

    /* The normalised direction and the next free path.  Fast math computes them here,
     * while the load is under way, and again for the few steps that change them (a lone
     * photon's step takes 3 % less); where they are long, once, at the step's end. */
    R ux, uy, uz, newS;
    auto finish = [&]() {
        const R norm = M::rsqrt(M::mad(nuz, nuz, M::mad(nuy, nuy, M::mul(nux, nux))));
        ux = M::mul(nux, norm);
        uy = M::mul(nuy, norm);
        uz = M::mul(nuz, norm);
        newS = -M::log((R)(1.0f - mc3d_u32_to_float_rz(e_s) * 0x1p-32f));
    };
    if (M::kFast) finish();

    /* What few steps need, behind one test: another tissue, a weight below the
     * roulette's threshold, air, components that snap to zero, the scattering of a
     * photon along the z axis, and the lateral faces.  The cell is looked up above
     * and first looked at here, so the scattering hides the load. */
    const R zero_thresh = M::zero_threshold();
    const bool steep = !M::uz_within(M::fabs(p.uz));
    const uint32_t changed = (uint32_t)(next_tissue ^ p.tissue) & 0xffu;
    const R least_u = M::fmin(M::fabs(nux), M::fmin(M::fabs(nuy), M::fabs(nuz)));
    if (M::rare(changed, W, mu_t, p.uz, least_u, newx, g.Lx, newy, g.Ly)) {
        bool refl = false;
        bool again = steep && !hit;   /* the scattering anew */
        bool redo = steep | (least_u < zero_thresh); /* the normalisation anew */
        const bool lateral = !(newx > 0) | !(newx < g.Lx) | !(newy > 0) | !(newy < g.Ly);
        const bool low = !M::w_above_threshold(W) | (mu_t == 0);
        /* Two of three lanes that come here only touch a lateral face: with one geometry
         * they pass the three parts below at once (layered 1e6 22.4 -> 21.8 ms, pencil beam
         * 1e6 18.6 -> 18.1).  Launches over several geometries, whose inclusions change the
         * index in half of a warp's steps, lose by the extra test (22.5 -> 23.2 ms). */
        if (!ONE_GEOM || (changed != 0) | low | redo) {
            if (((next_tissue ^ p.tissue) & 0xff) != 0 &&
                M::n(tt) != M::n(M::row(tab, next_tissue & 0xff))) {
                /* Fresnel, src/mc3d_gpu.cu:226-257 */
                const R ni = M::n(tt), nt = M::n(M::row(tab, next_tissue & 0xff));
                const bool mx = p.i != nexti, my = p.j != nextj, mz = p.k != nextk;
                R cos_ai = mx ? p.ux : (my ? p.uy : p.uz);
                cos_ai = M::fabs(cos_ai);
                cos_ai = (cos_ai > 1) ? 1 : cos_ai;
                const R ni_nt = M::div(ni, nt);
                /* sin(acos(c)); fast math evaluates it as sqrt((1 - c)(1 + c)), the same
                 * value without the polynomial of acosf (and more accurate near c = 1) */
                const R sin_ai = M::kFast ? M::sqrt(M::mul((R)1 - cos_ai, (R)1 + cos_ai))
                                          : M::sin(M::acos(cos_ai));
                const R sin_at = M::mul(ni_nt, sin_ai);
                R cos_at = M::sqrt(M::mad(-sin_at, sin_at, (R)1));
                const R cs = M::mul(cos_ai, sin_at), cc = M::mul(cos_ai, cos_at);
                const R R1 = M::div(M::mad(sin_ai, cos_at, -cs), M::mad(sin_ai, cos_at, cs));
                const R R2 = M::div(M::mad(-sin_ai, sin_at, cc), M::mad(sin_at, sin_at, cc));
                /* 0.5 is a double literal there too */
                R Rf = 0.5 * R1 * R1 * M::mad(R2, R2, (R)1);
                Rf = (sin_at > 1) ? 1 : Rf;
                R lat = ni_nt; /* scale of the transmitted lateral cosines */
                if (M::kFast && M::fabs(M::mad(-sin_at, sin_at, (R)1)) < MC3D_NEAR_CRITICAL_F) {
                    /* Near the critical angle 1 - sin_at^2 cancels in float and R is steep:
                     * the same formulas in FP64, sin_ai from cos_ai directly, and the
                     * transmitted direction renormalised in FP64. */
                    const double c = cos_ai;
                    const double rn = (double)ni / (double)nt;
                    const double si = sqrt((1.0 - c) * (1.0 + c));
                    const double st = rn * si;
                    const double ca = sqrt(fmax((1.0 - st) * (1.0 + st), 0.0));
                    const double R1 = (si * ca - c * st) / (si * ca + c * st);
                    const double R2 = (c * ca - si * st) / (c * ca + st * st);
                    Rf = (st >= 1.0) ? (R)1 : (R)(0.5 * R1 * R1 * (1.0 + R2 * R2));
                    const bool xa = mx;
                    const bool ya = !xa && my;
                    const bool za = !xa && !ya && mz;
                    const double ax = xa ? 0.0 : (double)p.ux;
                    const double ay = ya ? 0.0 : (double)p.uy;
                    const double az = za ? 0.0 : (double)p.uz;
                    const double lat2 = rn * rn * (ax * ax + ay * ay + az * az);
                    const double sc = 1.0 / sqrt(ca * ca + lat2);
                    cos_at = (R)(ca * sc);
                    lat = (R)(rn * sc);
                }
                /* The reflection is the step's first draw, so the other four are each one
                 * draw later than taken above. */
                refl = mc3d_u32_to_float_rz(e_rr) * 0x1p-32f < Rf;
                e_rr = e_hg;
                e_hg = e_phi;
                e_phi = e_s;
                rx = mc3d_mwc_next(rx, ra);
                e_s = (uint32_t)rx;
                if (hit) {
                    const R tx = mx ? M::copysign(cos_at, M::mul(p.ux, cos_at)) : M::mul(p.ux, lat);
                    const R ty = (my && !mx) ? M::copysign(cos_at, M::mul(p.uy, cos_at))
                                             : M::mul(p.uy, lat);
                    const R tz = (mz && !my && !mx) ? M::copysign(cos_at, M::mul(p.uz, cos_at))
                                                    : M::mul(p.uz, lat);
                    nux = refl ? (mx ? -p.ux : p.ux) : tx;
                    nuy = refl ? (my ? -p.uy : p.uy) : ty;
                    nuz = refl ? (mz ? -p.uz : p.uz) : tz;
                }
                again = !hit; /* an interaction that rounded onto the face */
                redo = true;
                acc[T_FRESNEL] += 1;
            }
            if (low) {
                /* Russian roulette, src/mc3d_gpu.cu:275-277 */
                if (M::w_below_threshold(W) && !hit && mu_t != 0) {
                    const float eps = mc3d_u32_to_float_rz(e_rr) * 0x1p-32f;
                    const R newW = (eps < MC3D_SURVIVAL_LT_F) ? M::roulette_survivor(W) : (R)0;
                    /* absorbed weight is booked at the photon's end as Q(W0) - Q(W_end) - lost;
                     * a roulette event moves its share from there to the roulette tallies */
                    if (newW == 0) {
                        uint64_t k = M::qw(W);
                        acc[T_RR_KILLED] += k;
                        acc[T_ABSORBED] -= k;
                    } else {
                        uint64_t c = M::qw(newW) - M::qw(W);
                        acc[T_RR_CREATED] += c;
                        acc[T_ABSORBED] += c;
                    }
                    W = newW;
                }
                if (W <= 0 || mu_t == 0) { /* freeze (:303-311): the photon stays where it is */
                    p.W = W;
                    p.s = hit ? s : p.s - p.s;
                    *lat_mirror = false;
                    if (!refl && !(p.x > 0 && p.x < g.Lx && p.y > 0 && p.y < g.Ly))
                        *lat_mirror = mirror<M>(&p.x, &p.ux, (R)g.Lx) || mirror<M>(&p.y, &p.uy, (R)g.Ly);
                    return true;
                }
                if (!(W > 0)) { /* NaN weight: no free path, -log(1) */
                    e_s = 0;
                    redo = true;
                }
            }
            if (redo) {
                if (again) {
                    const Spin<R> sp = scatter<M, SPLIT_SIN2>(tt, p, e_hg, e_phi);
                    nux = steep ? M::mul(sp.sintheta, sp.cosphi) : sp.ux;
                    nuy = steep ? M::mul(sp.sintheta, sp.sinphi) : sp.uy;
                    nuz = steep ? M::copysign(sp.costheta, M::mul(sp.costheta, p.uz)) : sp.uz;
                }
                nux = (M::fabs(nux) < zero_thresh) ? 0 : nux;
                nuy = (M::fabs(nuy) < zero_thresh) ? 0 : nuy;
                nuz = (M::fabs(nuz) < zero_thresh) ? 0 : nuz;
                if (M::kFast) finish();
            }
        }
        /* The mirrors, short-circuited as in src/mc3d_gpu.cu:330, both axes at once.  A
         * mirror turns its component before or after the normalisation, which keeps the
         * sign. */
        if (lateral && !refl) {
            R &mx = M::kFast ? ux : nux, &my = M::kFast ? uy : nuy;
            const bool in_x = (newx >= g.Lx) | (newx <= 0);
            const bool in_y = !in_x & ((newy >= g.Ly) | (newy <= 0));
            const R length = in_x ? (R)g.Lx : (R)g.Ly;
            R c = in_x ? newx : newy;
            c = c >= length ? 2 * length - c : c;
            c = M::fabs(c);
            newx = in_x ? c : newx;
            newy = in_y ? c : newy;
            mx = in_x ? -mx : mx;
            my = in_y ? -my : my;
            refl = in_x | in_y;
        }
        if (hit && refl) { /* a reflected photon keeps its voxel (:334-339) */
            nexti = p.i;
            nextj = p.j;
            nextk = p.k;
            next_tissue = p.tissue;
        }
    }
    if (!M::kFast) finish();
    p.ux = ux;
    p.uy = uy;
    p.uz = uz;
    p.s = hit ? s : newS;
    p.W = W;
    p.x = newx;
    p.y = newy;
    p.z = newz;
    p.i = nexti;
    p.j = nextj;
    p.k = nextk;
    p.tissue = next_tissue;
    return false;
}

/* i, j, k and tissue from the position, as at the start of every launch of
 * photontrack_step (src/mc3d_gpu.cu:168-171). */
template <class M, bool JUMP = false, class R = typename M::real>
static __device__ __forceinline__ void derive_cell(const typename M::Geom &g, PhotonT<R> &p)
{
    p.i = grid_index<M>(p.x, upward(p.ux), g.dx, g.rdx);
    p.j = grid_index<M>(p.y, upward(p.uy), g.dy, g.rdy);
    p.k = grid_index<M>(p.z, upward(p.uz), g.dz, g.rdz);
    p.tissue = tissue_at<M, JUMP>(g, p.i, p.j, p.k, p.z, p.uz);
}

/* Whether photontrack_get_grid_coord's face rule puts (x, u) in the stored cell on
 * every axis: strictly inside, or on the lower face moving up, or on the upper face
 * moving down.  Then re-deriving the cell and tissue at a launch boundary changes
 * nothing (above the surface the air rule would apply, which needs z > 0 here). */
template <class R, class G>
static __device__ __forceinline__ bool cell_consistent(const G &g, const PhotonT<R> &p)
{
    const R xl = p.i * (R)g.dx, xh = (p.i + (R)1) * (R)g.dx;
    const R yl = p.j * (R)g.dy, yh = (p.j + (R)1) * (R)g.dy;
    const R zl = p.k * (R)g.dz, zh = (p.k + (R)1) * (R)g.dz;
    const bool ox = (p.x > xl && p.x < xh) || (p.x == xl && p.ux >= 0) || (p.x == xh && p.ux < 0);
    const bool oy = (p.y > yl && p.y < yh) || (p.y == yl && p.uy >= 0) || (p.y == yh && p.uy < 0);
    const bool oz = (p.z > zl && p.z < zh) || (p.z == zl && p.uz >= 0) || (p.z == zh && p.uz < 0);
    return ox && oy && oz && p.z > 0;
}

template <class R>
static __device__ __forceinline__ bool finite_state(const PhotonT<R> &p)
{
    return isfinite(p.x) && isfinite(p.y) && isfinite(p.z) && isfinite(p.s) &&
           isfinite(p.ux) && isfinite(p.uy) && isfinite(p.uz);
}

/* The boundary distance the reference's one-voxel DDA (src/mc3d_gpu.cu:29-49,
 * :194) gives a step that starts in state p.  It is 0 when the photon sits on a
 * face of its voxel and moves out through it, which happens when a scattering
 * move rounds onto a voxel face and the new direction points back across it. */
template <class M, class R = typename M::real>
static __device__ __forceinline__ R voxel_db(const typename M::Geom &g, const PhotonT<R> &p)
{
    R b;
    const R t_x = face_distance<M>(p.x, p.ux, upward(p.ux), p.i, (R)0, g.dx, &b);
    const R t_y = face_distance<M>(p.y, p.uy, upward(p.uy), p.j, (R)0, g.dy, &b);
    const R t_z = face_distance<M>(p.z, p.uz, upward(p.uz), p.k, (R)0, g.dz, &b);
    return M::fmin(t_x, M::fmin(t_y, t_z));
}

/* The NaN/Inf/db==0 quickfix run after each 45-step launch (src/mc3d_gpu.cu:343-353);
 * zero_db tells whether the launch's last step had db == 0.  Returns true (and
 * zeroes the photon) when it fires. */
template <class R>
static __device__ __forceinline__ bool quickfix(PhotonT<R> &p, bool zero_db)
{
    if (!finite_state(p) || zero_db) {
        p.x = 0; p.y = 0; p.z = 0;
        p.ux = 0; p.uy = 0; p.uz = 1;
        p.W = 0; p.s = 0;
        return true;
    }
    return false;
}

/* The steps a frozen slot keeps executing until the end of its 45-step launch.
 * They change nothing but the mirror (which flips u while the photon sits on a
 * lateral face) and the boundary distance the quickfix looks at. */
template <class M, class R = typename M::real>
static __device__ __forceinline__ R masked_steps(const typename M::Geom &g, PhotonT<R> &p, int masked, R db)
{
    for (int t = 0; t < masked; t++) {
        db = voxel_db<M>(g, p);
        if (!mirror<M>(&p.x, &p.ux, (R)g.Lx)) mirror<M>(&p.y, &p.uy, (R)g.Ly);
    }
    return db;
}

/* --------------------------------------------------------------- kernel body */
static __device__ __forceinline__ void acc_clear(const Acc &a)
{
#pragma unroll
    for (int t = 0; t < MC3D_NUM_TOTALS; t++) a[t] = 0;
}

static __device__ __forceinline__ void acc_flush(const Acc &a, unsigned long long *tot)
{
#pragma unroll
    for (int t = 0; t < MC3D_NUM_TOTALS; t++) {
        unsigned long long v = a[t];
        if (v) atomicAdd(tot + t, v);
        a[t] = 0;
    }
}

static __device__ __forceinline__ unsigned long long *job_totals(const KernelParams &P, int job)
{
    return P.totals + (int64_t)P.jobs[job].index * MC3D_NUM_TOTALS;
}

/* Multiplier of job-local stream `local`: table line 1 + local mod (L - 1).  The
 * remainder by Barrett reduction with magic = floor((2^64 - 1) / (L - 1)): the
 * quotient estimate is at most one short, so one correction gives the remainder
 * (local < 2^63). */
static __device__ __forceinline__ uint32_t stream_multiplier(const KernelParams &P, int64_t local)
{
    const uint64_t d = (uint64_t)(P.num_multipliers - 1);
    const uint64_t q = __umul64hi((uint64_t)local, P.mult_magic);
    uint64_t r = (uint64_t)local - q * d;
    r = (r >= d) ? r - d : r;
    return P.multipliers[1 + r];
}

/* job owning global stream index gs (binary search over the stream prefix) */
static __device__ __forceinline__ int find_job(const JobDev *jobs, int njobs, int64_t gs)
{
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (jobs[mid].stream_base <= gs) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

/* initial packed state of stream `local` of job `jb` (gpumcml_rng/gpumcml_rng.cu:95-114),
 * honouring the seeding attempts that earlier streams of the job rejected */
static __device__ __forceinline__ uint64_t stream_seed(const KernelParams &P, const JobDev &jb,
                                                       int64_t local, uint32_t fora)
{
    int64_t offset = 0;
    int lo = 0, hi = jb.rej_count - 1;
    while (lo <= hi) { /* last listed stream <= local */
        int mid = (lo + hi) >> 1;
        if (P.rejections[jb.rej_offset + mid].stream <= local) {
            offset = P.rejections[jb.rej_offset + mid].cum;
            lo = mid + 1;
        } else {
            hi = mid - 1;
        }
    }
    uint64_t xs = mc3d_seed_jump(&P.seed, jb.seed, (uint64_t)(local + offset));
    return mc3d_seed_attempt(xs, P.seed.begin, fora);
}

/* A photon on its way from one thread of the block to another, in the tally words of
 * the receiving thread's row (the stream's words go to their own place). */
template <class R>
struct ParkedT {
    uint64_t rx;
    R x, y, z, ux, uy, uz, W, s, i, j, k;
    int32_t tissue;
    uint32_t ra;
    int32_t psteps, job;
};
static_assert(sizeof(ParkedT<double>) <= 8 * MC3D_NUM_TOTALS, "a photon outgrows the tally words");

#define MC3D_MAX_WARPS 8 /* per block: 256 threads */

/* The persistent photon loop.  JUMP selects merged steps (photon_step) and needs
 * every geometry's safe-distance map. */
template <class M, bool AMAP, bool JUMP = false, bool ONE_GEOM = false>
__device__ __forceinline__ void photon_kernel_body(const KernelParams &P)
{
    using R = typename M::real;
    /* dynamic shared memory (photon_smem): the threads' rows, then the optical tables,
     * then (several geometries) the geometry descriptors, read from there instead of
     * being held per thread.  Sized by the block, so the rest stays with the L1 cache,
     * which holds cells. */
    extern __shared__ float4 sh_base[];
    unsigned long long *sh_rows = reinterpret_cast<unsigned long long *>(sh_base);
    float4 *sh_tab = reinterpret_cast<float4 *>(sh_rows + MC3D_THREAD_WORDS * blockDim.x);
    for (int t = threadIdx.x; M::kShared && t < P.props_entries; t += blockDim.x)
        sh_tab[t] = P.props_table[t];
    GeomDev *sh_geom = reinterpret_cast<GeomDev *>(sh_tab + P.props_entries);
    if (M::kShared && !ONE_GEOM)
        for (int t = threadIdx.x; t < P.ngeoms; t += blockDim.x) sh_geom[t] = P.geoms[t];
    const Acc acc{sh_rows + MC3D_THREAD_WORDS * threadIdx.x};
    acc_clear(acc);
    __shared__ volatile int sh_drain;          /* a thread found no stream left */
    __shared__ int sh_live[2][MC3D_MAX_WARPS]; /* photons per warp, two chunks' worth */
    if (threadIdx.x == 0) sh_drain = 0;
    __syncthreads();

    int job = -1;
    unsigned long long *amap = nullptr;
    /* valid before the first stream too: a lane that gets none still passes run_chunk,
     * which names its geometry and table */
    const typename M::Geom *gp = M::geom(P, sh_geom, 0);
    typename M::Row tab = M::table(P, sh_tab, 0);
    /* the photon's geometry: the launch's only one from the kernel parameters */
    auto geometry = [&]() -> const typename M::Geom & {
        if constexpr (ONE_GEOM) return P.geom0;
        else return *gp;
    };
    auto set_job = [&](int j) {
        job = j;
        gp = M::geom(P, sh_geom, P.jobs[job].geom);
        tab = M::table(P, sh_tab, P.jobs[job].props_offset);
        if (AMAP) amap = P.amap + P.jobs[job].amap_offset;
    };
    int64_t &left = acc.left(), &local = acc.local();
    left = 0;
    uint64_t rx = 0;
    uint32_t ra = 1;
    PhotonT<R> p;
    bool alive = false;
    bool drained = false; /* no stream left to take */
    int psteps = 0; /* steps of the photon before its present chunk */
    /* a lane without photons left in its stream takes the next stream */
    auto take_stream = [&]() {
        if (!alive && !drained) {
            while (left == 0) {
                drained = P.cancel && *((volatile const int *)P.cancel);
                if (drained) break;
                int64_t gs = (int64_t)atomicAdd((unsigned long long *)P.work_counter, 1ull);
                drained = gs >= P.total_streams;
                if (drained) break;
                const int next_job = find_job(P.jobs, P.njobs, gs);
                /* the per-thread tallies are the job's: flushed when the job changes */
                if (job >= 0 && next_job != job)
                    acc_flush(acc, job_totals(P, job));
                set_job(next_job);
                const JobDev &jb = P.jobs[job];
                local = gs - jb.stream_base + jb.stream_first;
                left = jb.per_stream + (local < jb.remainder ? 1 : 0);
                ra = stream_multiplier(P, local);
                rx = P.seeds ? P.seeds[gs] : stream_seed(P, jb, local, ra);
            }
        }
    };
    /* a lane without a photon starts the next of its stream */
    auto start_photon = [&]() {
        if (!alive && left != 0) {
            const auto &g = geometry();
            /* photontrack_reinitialize, src/mc3d_gpu.cu:74-111 */
            if (P.jobs[job].beam == 0) {
                p.x = (R)g.Lx * (R)mc3d_rand_co(&rx, ra);
                p.y = (R)g.Ly * (R)mc3d_rand_co(&rx, ra);
            } else {
                p.x = (R)g.Lx / 2;
                p.y = (R)g.Ly / 2;
            }
            p.z = 0;
            p.ux = 0; p.uy = 0; p.uz = 1;
            /* specular reflection from air into tissue type 1 (src/mc3d_gpu.cu:67-70, 500) */
            const R n0 = M::n(M::row(tab, MC3D_TISSUE_AIR)), n1 = M::n(M::row(tab, 1));
            const R rsp = M::div(n0 - n1, n0 + n1);
            p.W = M::mad(-rsp, rsp, (R)1);
            p.s = -M::log((R)mc3d_rand_oc(&rx, ra));
            derive_cell<M, JUMP>(g, p);
            psteps = 0;
            alive = true;
            left--;
        }
    };
    /* One chunk of 45 steps, the reference's launch, and its end.  A photon starts only at
     * a chunk's start, as a reference slot starts only at a launch boundary: a lane whose
     * photon ended waits out the rest of the chunk (the reference's masked steps).  The
     * barrier after the steps makes that wait real: without it a lane that leaves the step
     * loop early runs on alone, and from then on the warp steps in pieces (4.7 lanes a
     * chunk's end instead of 32, layered 1e6 photons). */
    auto run_chunk = [&]() {
        const auto &g = geometry();
        /* The chunk's steps, fewer where the step cap comes first.  Merged steps: the
         * quickfix must see the boundary distance of the reference's one-voxel DDA
         * for the chunk's last step, not the merged box's (which is never 0 inside a
         * uniform cube), or merged steps would lose less weight to it than the
         * reference does.  It is taken from that step's start state, so the loop
         * stops before that step and goes round once more for it. */
        const int cap = alive ? min(MC3D_NUM_PHOTON_STEPS, (int)P.max_steps - psteps) : 0;
        int stop = JUMP ? min(cap, MC3D_NUM_PHOTON_STEPS - 1) : cap;
        int chunk = 0;
        R db;
        bool lat_mirror;
        bool froze = false;
        bool vzero = false;
        for (;;) {
            while (!froze && chunk < stop) {
                froze = photon_step<M, AMAP, JUMP, ONE_GEOM>(g, tab, p, rx, ra, acc, &db, amap,
                                                             &lat_mirror);
                chunk++;
            }
            if (!JUMP || froze || stop == cap) break;
            vzero = voxel_db<M>(g, p) == 0;
            stop = cap;
        }
        __syncwarp();
        if (!alive) return;
        psteps += chunk;

        bool done = false;
        uint64_t lost = 0;
        if (froze) {
            /* If the freeze step's mirror did not fire and the photon is off the
             * lateral faces, the masked steps change nothing and see the freeze
             * step's boundary distance again: no need to replay them.  The
             * replayed masked steps are one-voxel steps; without them a merged
             * kernel takes the one-voxel distance of the frozen state, which is
             * the freeze step's start state. */
            bool zero;
            if (lat_mirror || !(p.x > 0 && p.x < g.Lx && p.y > 0 && p.y < g.Ly)) {
                if (chunk < MC3D_NUM_PHOTON_STEPS)
                    zero = masked_steps<M>(g, p, MC3D_NUM_PHOTON_STEPS - chunk, db) == 0;
                else
                    zero = JUMP ? vzero : db == 0;
            } else {
                zero = JUMP ? voxel_db<M>(g, p) == 0 : db == 0;
            }
            R w_before = p.W;
            if (quickfix(p, zero)) { acc[T_QUICKFIX]++; lost = M::qw(w_before); }
            done = true;
        } else if (chunk == MC3D_NUM_PHOTON_STEPS) {
            R w_before = p.W;
            if (quickfix(p, JUMP ? vzero : db == 0)) {
                acc[T_QUICKFIX]++;
                lost = M::qw(w_before);
                done = true;
            } else {
                /* fast math: re-derive only where the stored cell breaks the face rule
                 * (exact math always re-derives, as the reference's relaunch does) */
                if (!M::kFast || !cell_consistent(g, p)) derive_cell<M, JUMP>(g, p);
            }
        }
        if (!done && psteps >= P.max_steps) {
            lost = M::qw(p.W);
            p.W = 0;
            acc[T_CAPPED]++;
            done = true;
        }
        if (done) {
            /* photon_detector, src/mc3d_photons.cu:151-171 */
            const JobDev &jb = P.jobs[job];
            const int ix = (int)grid_index<M>(p.x, upward(p.ux), g.dx, g.rdx);
            const int iy = (int)grid_index<M>(p.y, upward(p.uy), g.dy, g.rdy);
            bool inside = (ix >= 0) && (iy >= 0) && (ix < g.nx) && (iy < g.ny);
            uint64_t q = M::qw(p.W);
            int64_t bin = jb.bin_offset + (int64_t)iy * g.nx + ix;
            int slot;
            if (p.z <= 0) {
                slot = inside ? T_R_IN : T_R_OUT;
                if (inside && q) {
                    atomicAdd(P.drs + bin, (unsigned long long)q);
                    atomicAdd(P.drs_sq + bin, (unsigned long long)M::qw(M::mul(p.W, p.W)));
                }
            } else {
                slot = inside ? T_T_IN : T_T_OUT;
                if (inside && q) atomicAdd(P.trans + bin, (unsigned long long)q);
            }
            acc[slot] += q;
            /* the launch weight 1 - Rsp again, as at the photon's start */
            const R n0 = M::n(M::row(tab, MC3D_TISSUE_AIR)), n1 = M::n(M::row(tab, 1));
            const R rsp = M::div(n0 - n1, n0 + n1);
            const uint64_t qw0 = M::qw(M::mad(-rsp, rsp, (R)1));
            acc[T_W_LAUNCHED] += qw0;
            acc[T_ABSORBED] += qw0 - q - lost;
            acc[T_LOST] += lost;
            acc[T_PHOTONS] += 1;
            acc[T_STEPS] += psteps;
            if (P.photon_log) {
                int64_t nstream = jb.per_stream + (local < jb.remainder ? 1 : 0);
                int64_t kphot = nstream - left - 1;
                int64_t pid = jb.photon_base + local + kphot * jb.streams;
                PhotonRecord r;
                r.x = (float)p.x; r.y = (float)p.y; r.z = (float)p.z;
                r.ux = (float)p.ux; r.uy = (float)p.uy; r.uz = (float)p.uz;
                r.W = (float)p.W; r.s = (float)p.s;
                r.steps = (uint32_t)psteps;
                r.tissue = (uint32_t)(p.tissue & 0xff);
                r.rng = rx;
                P.photon_log[pid] = r;
            }
            alive = false;
        }
    };

    /* The drain.  Once the streams run out, lanes fall idle one by one and the last
     * photons of a launch, up to 15 times the mean length, would leave warps stepping
     * for one or two lanes each and, by sharing an SM, slowing one another.  So from
     * then on the block's warps meet at each chunk's start and, whenever its photons
     * fit into fewer warps, close ranks: at most seven times, a photon's state passing
     * through shared memory.  Where a photon is stepped changes nothing in its
     * trajectory. */
    int turn = 0;
    auto close_ranks = [&]() { /* false when the block has no photon left */
        const unsigned live = __ballot_sync(0xffffffffu, alive);
        int *count = sh_live[turn];
        turn ^= 1; /* the other half is written only after all have read this one */
        if ((threadIdx.x & 31) == 0) count[threadIdx.x >> 5] = __popc(live);
        __syncthreads();
        int total = 0, before = 0, warps = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
            if (w == (int)(threadIdx.x >> 5)) before = total;
            total += count[w];
            warps += count[w] != 0;
        }
        if (total == 0) return false;
        if ((total + 31) / 32 < warps) {
            /* the rows become free of tallies, then carry the photons */
            if (job >= 0) acc_flush(acc, job_totals(P, job));
            const int64_t my_left = left, my_local = local;
            __syncthreads();
            if (alive) {
                const int to = before + __popc(live & ((1u << (threadIdx.x & 31)) - 1u));
                const Acc other{sh_rows + MC3D_THREAD_WORDS * to};
                *reinterpret_cast<ParkedT<R> *>(other.row) = ParkedT<R>{
                    rx, p.x, p.y, p.z, p.ux, p.uy, p.uz, p.W, p.s, p.i, p.j, p.k,
                    p.tissue, ra, psteps, job};
                other.left() = my_left;
                other.local() = my_local;
            }
            __syncthreads();
            alive = (int)threadIdx.x < total;
            if (alive) {
                const ParkedT<R> q = *reinterpret_cast<const ParkedT<R> *>(acc.row);
                rx = q.rx;
                p.x = q.x; p.y = q.y; p.z = q.z;
                p.ux = q.ux; p.uy = q.uy; p.uz = q.uz;
                p.W = q.W; p.s = q.s;
                p.i = q.i; p.j = q.j; p.k = q.k;
                p.tissue = q.tissue;
                ra = q.ra;
                psteps = q.psteps;
                set_job(q.job);
            } else {
                left = 0;
            }
            asm volatile("" ::: "memory"); /* the row is read before it is cleared */
            acc_clear(acc);
        }
        return true;
    };

    if (M::kFast) {
        /* two loops: with the drain's code in it the compiler reloads the launch's
         * constants in every step (6.6 of 196 instructions) */
        for (;;) {
            take_stream();
            start_photon();
            if (drained) sh_drain = 1;
            if (__any_sync(0xffffffffu, sh_drain != 0)) break;
            run_chunk();
        }
        for (;;) {
            start_photon();
            if (!close_ranks()) break;
            run_chunk();
        }
    } else {
        /* one loop: a second copy of the steps, several times as long, gains next to
         * nothing (2e6 FP64 photons: 148.2 ms, with two loops 147.3; 1e6 exact ones: 135.5
         * and 136.2) */
        for (bool drain = false;;) {
            if (!drain) take_stream();
            start_photon();
            if (drained) sh_drain = 1;
            drain = drain || __any_sync(0xffffffffu, sh_drain != 0);
            if (drain && !close_ranks()) break;
            run_chunk();
        }
    }
    if (job >= 0) acc_flush(acc, job_totals(P, job));
}

} /* namespace mc3d */

#endif /* MC3D_ENGINE_CUH */
