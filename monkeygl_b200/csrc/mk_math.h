// mk_math.h -- scalar expressions of MonkeyGL's kernels shared by the CUDA
// kernels and host code.
//
// MonkeyGL evaluates a few expressions in double precision on the device (a
// double literal promotes the whole expression).  They are evaluated here in
// double too, operation for operation, with explicit roundings on the device
// so that no multiply-add is contracted differently from MonkeyGL's build:
// FP64 runs at half the FP32 rate on sm_100, and the values then equal
// MonkeyGL's by construction.
#pragma once

#include <math.h>
#include <string.h>
#include <stdint.h>

#if defined(__CUDACC__)
#define MK_HD __host__ __device__ __forceinline__
#else
#define MK_HD inline
#endif

namespace mk {

// (float)(((double)a - 0.866) * (double)scale): the ray parameter of
// core/kernel.cu:197 (and :313, :415), whose 0.866 literal makes the
// expression double: the difference and the product are rounded to double,
// then the product to float.  Host builds are compiled with
// -ffp-contract=off, and a difference times a factor has no multiply-add to
// contract anyway.
MK_HD float ray_fy(float a, float scale) {
#if defined(__CUDA_ARCH__)
    return __double2float_rn(__dmul_rn(__dsub_rn((double)a, 0.866), (double)scale));
#else
    return (float)(((double)a - 0.866) * (double)scale);
#endif
}

// float -> int16 with truncation and saturation (PTX cvt.rzi.s16.f32
// semantics, which MonkeyGL's "short v = 32768 * tex3D(...)" compiles to).
MK_HD short f2s_sat(float v) {
    if (!(v == v)) return 0;
    if (v >= 32767.0f) return 32767;
    if (v <= -32768.0f) return -32768;
    return (short)v;
}

// a after n additions of `step`, each rounded to float, as MonkeyGL's loop
// makes them.  Between two powers of two all floats have one spacing, so every
// addition moves a by the same amount (after the first sum in that range: a
// step that falls halfway between two floats is rounded to the even one, and
// from an even one always the same way); that amount is an exact difference
// and n times it an exact product.  Where the sum leaves the range, one
// addition at a time.
MK_HD float add_steps(float a, float step, int n) {
    if (n > 4) {
        const float a1 = a + step, a2 = a1 + step, d = (a2 + step) - a2;
#ifdef __CUDA_ARCH__
        const float end = __fmaf_rn((float)(n - 2), d, a2);
        const bool same = ((__float_as_uint(a1) ^ __float_as_uint(end)) >> 23) == 0u;
#else
        const float end = fmaf((float)(n - 2), d, a2);
        uint32_t u, v;
        memcpy(&u, &a1, 4);
        memcpy(&v, &end, 4);
        const bool same = ((u ^ v) >> 23) == 0u;
#endif
        if (same) return end;
    }
    for (; n > 0; --n) a += step;
    return a;
}

// Pixel of thread t in a 32x8 tile of a 256-thread block: eight 8x4 warp tiles,
// and inside one the lanes along a Z curve, so that the four lanes the texture
// unit serves together are 2x2 pixels and touch fewer texels than four in a
// row.
MK_HD int tile_x(int t) { return ((t >> 5) & 3) * 8 + ((t & 1) | ((t >> 1) & 2) | ((t >> 2) & 4)); }
MK_HD int tile_y(int t) { return (t >> 7) * 4 + (((t >> 1) & 1) | ((t >> 2) & 2)); }

// a / d, correctly rounded, given y = 1 / d correctly rounded: two corrections
// of a * y by the remainder, which one fused multiply-add gives (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor",
// IBM J. Res. Dev. 34(1), 1990: with y correctly rounded, the correction of a
// quotient within one ulp is correctly rounded; the first correction brings a * y
// there).  For d, 1 / d and a / d well inside the range of normal numbers
// (div_by_ok); an infinite a gives NaN.
MK_HD float div_by(float a, float d, float y) {
    float q = a * y;
    q = fmaf(fmaf(-q, d, a), y, q);
    return fmaf(fmaf(-q, d, a), y, q);
}

MK_HD double div_by(double a, double d, double y) {
    double q = a * y;
    q = fma(fma(-q, d, a), y, q);
    return fma(fma(-q, d, a), y, q);
}

MK_HD bool div_by_ok(float d) {
    const float m = fabsf(d);
    return m >= 1e-18f && m <= 1e18f;
}

}  // namespace mk
