// mk_reslice_impl.cuh -- device code of the planar reslice: one output pixel
// of MonkeyGL's d_renderPlane_{MIP,MinIP,Average} (core/kernel.cu:570-793),
// shared by the one-plane kernel (mk_reslice.cu) and the serving kernel
// (mk_server.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "mk_internal.h"
#include "mk_math.h"

namespace mk {

struct PlaneParams {
    int W, H;
    float ext[3], inv_ext[3];  // spacing * dim and its reciprocal
    int fast;                  // 1: the extents suit div_by
    float h[3], v[3], n[3], lt[3];
    float ps;
    int invertZ;
    float halfNum;
    int mode;
    const uint8_t *voi_lut;   // u8 epilogue: display value of int16 v at [v + 32768]
};

// FAST: the three divisions by the volume's extents go through div_by.  The
// extremum is taken of the texture values, before the scaling and conversion to
// short, which are non-decreasing.  Bound by the texture unit's data path: 21
// samples, 512^2 oblique, 23.6 us with a row of 32 pixels a warp and compiled
// divisions, 21.6 with div_by, 16.0 with 2x2 pixels in each quad of lanes
// (tile_x).  (Two samples in flight: 22 us, four: 16.5.)
template <int MODE, bool FAST>
__device__ __forceinline__ short reslice_samples(const PlaneParams &P, cudaTextureObject_t tex, int x, int y) {
    float best = (MODE == MK_MPR_MIP) ? -INFINITY : INFINITY;
    double sum = 0.0;          // MonkeyGL's double accumulator (core/kernel.cu:773)
    // The contraction of MonkeyGL's sums pt + x*ps*h + y*ps*v into fused
    // multiply-adds is spelled out, left to right: of the fused and unfused
    // orders, this one reproduces MonkeyGL's kernel pixel for pixel, and
    // writing it out keeps every kernel that inlines this function on it.
    const float xs = __fmul_rn((float)x, P.ps), ys = __fmul_rn((float)y, P.ps);
    for (float t = -P.halfNum; t <= P.halfNum; t += 1) {
        const float fLength = __fmul_rn(t, P.ps);
        float f[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float pt = __fmaf_rn(fLength, P.n[k], P.lt[k]);
            const float a = __fmaf_rn(ys, P.v[k], __fmaf_rn(xs, P.h[k], pt));
            f[k] = FAST ? div_by(a, P.ext[k], P.inv_ext[k]) : __fdiv_rn(a, P.ext[k]);
        }
        // "fz = 1.0 - fz" in double, then rounded to float: identical to the
        // float subtraction for every float fz (the exact difference rounds once)
        if (!P.invertZ) f[2] = 1.0f - f[2];
        const bool inside = f[0] >= 0 && f[0] <= 1 && f[1] >= 0 && f[1] <= 1 && f[2] >= 0 && f[2] <= 1;
        const float v = inside ? tex3D<float>(tex, f[0], f[1], f[2]) : -1.0f;
        if (MODE == MK_MPR_AVERAGE) sum = __dadd_rn(sum, (double)(32768 * v));
        else if (MODE == MK_MPR_MIP) best = fmaxf(best, v);
        else best = fminf(best, v);
    }
    if (MODE == MK_MPR_AVERAGE) {
        // fSum / (2 * halfNum + 1) in double, converted to short (truncated,
        // saturated as the conversion instruction does)
        const double q = __ddiv_rn(sum, (double)(2 * P.halfNum + 1));
        return (short)min(max(__double2int_rz(q), -32768), 32767);
    }
    return f2s_sat(32768 * best);
}

template <int MODE>
__device__ __forceinline__ short reslice_pixel(const PlaneParams &P, cudaTextureObject_t tex, int x, int y) {
    return P.fast ? reslice_samples<MODE, true>(P, tex, x, y) : reslice_samples<MODE, false>(P, tex, x, y);
}

// One 32x8 tile (bx, by) of a plane by a 256-thread block.
template <int MODE, bool U8>
__device__ __forceinline__ void plane_tile(const PlaneParams &P, cudaTextureObject_t tex, void *out, int bx, int by) {
    const int x = bx * 32 + tile_x(threadIdx.x);
    const int y = by * 8 + tile_y(threadIdx.x);
    if (x >= P.W || y >= P.H) return;
    const short r = reslice_pixel<MODE>(P, tex, x, y);
    if (U8) {
        // display window: one table read per pixel (the table is built on
        // the host; 64 KB, resident in L1/L2)
        static_cast<uint8_t *>(out)[(size_t)y * P.W + x] = __ldg(P.voi_lut + ((int)r + 32768));
    } else {
        static_cast<short *>(out)[(size_t)y * P.W + x] = r;
    }
}

// Host: kernel parameters of one plane (validates the request).
int fill_plane_params(const VolumeState &v, const mk_plane_params *p, PlaneParams &P);

}  // namespace mk
