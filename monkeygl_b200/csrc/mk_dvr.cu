// mk_dvr.cu -- differentiable direct volume rendering: forward and a
// hand-written backward of the front-to-back compositing, with respect to the
// transfer-function LUT entries and the voxel values.
//
// This has no counterpart in MonkeyGL.  It uses MonkeyGL's orthographic VR
// camera (the pixel -> ray mapping of core/kernel.cu:161-206) with the method
// made differentiable: a fixed step along the ray (no adaptive refinement), a
// float32 volume in [0, 1] sampled with exact trilinear weights (texel
// centres at (i+0.5)/dim, clamp to edge), the value used directly as the LUT
// coordinate (entry i centred at (i+0.5)/n, linear interpolation, clamp), and
// compositing
//     C = sum_i T_i a_i c_i,   T_0 = 1,   T_{i+1} = T_i (1 - a_i),
// stopped after the sample that takes T below t_min.  The image is C (RGB).
// The texture unit is not used for the volume: its float32 trilinear filter
// combines the x and y weights in fixed point below 8 fractional bits, so a
// backward pass could not reproduce the weights of the forward one.
//
// Backward.  With g = dL/dC and U_i the colour composited behind sample i
// seen from unit transmittance just after it (U_last = 0,
// U_{i-1} = a_i c_i + (1 - a_i) U_i),
//     dL/dc_i = T_i a_i g,     dL/da_i = T_i g . (c_i - U_i).
// The backward reverse-marches each ray from its last sample, reconstructing
// T_i = T_{i+1} / (1 - a_i) from the transmittance the forward saved after
// the last sample; the forward also saves T every K samples (checkpoints),
// which reset the reconstruction at each checkpoint and give T_i where
// a_i = 1 leaves nothing to divide by (a re-march from the checkpoint).  A
// ray accumulates its dL/dLUT in registers while its samples stay in one LUT
// cell and its dL/dvolume while they stay in one voxel cell; a change of
// cell flushes the sums -- the LUT sums of the lanes flushing one cell are
// combined by warp shuffles before the shared-memory bins, which go to global
// memory once per block; the voxel sums take eight global reductions.
#include <cuda_runtime.h>
#include <float.h>
#include <limits.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include "mk_internal.h"

namespace mk {

constexpr int kDvrMaxLut = 1024;
constexpr int kDvrSeg = 16;              // samples per recomputed segment
constexpr int kDvrMaxCkpt = 512;         // checkpoints per ray
constexpr int kDvrViewsPerLaunch = 32;

struct DvrView {
    float M[9];
    float mls[3];
    float scale, xT, yT;
    float step;
    float t_min;
    int ckpt_shift;                      // samples between checkpoints = 1 << ckpt_shift (>= kDvrSeg)
    int max_ckpt;
    unsigned long long work_off;         // floats from the workspace start
};

struct DvrBatch {
    int W, H;
    int lut_len;
    int dim[3];
    int sxy;                             // dim[0] * dim[1]
    float fdim[3];
    DvrView v[kDvrViewsPerLaunch];
};

struct Ray {
    float px, py, pz;                    // normalized position at a = 0
    float dx, dy, dz;                    // change of normalized position per unit a
    float a0;                            // first sample on the grid a0 + i * step
    int n;                               // samples inside the volume
};

__device__ __forceinline__ Ray make_ray(const DvrBatch &B, const DvrView &V, int x, int y) {
    Ray r;
    const float u = (x - B.W / 2.0f - V.xT) / B.H;
    const float v = (y - B.H / 2.0f - V.yT) / B.H;
    float base[3], dir[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        // pos(a) = M (u, (a - 0.866) s, v) * mls + 0.5
        base[k] = (V.M[3 * k] * u + V.M[3 * k + 1] * (-0.866f * V.scale) + V.M[3 * k + 2] * v) * V.mls[k] + 0.5f;
        dir[k] = V.M[3 * k + 1] * V.scale * V.mls[k];
    }
    float lo = 0.0f, hi = 1.732f;
    bool hit = true;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if (fabsf(dir[k]) < 1e-12f) {
            if (base[k] < 0.0f || base[k] > 1.0f) hit = false;
            continue;
        }
        float t0 = (0.0f - base[k]) / dir[k], t1 = (1.0f - base[k]) / dir[k];
        if (t0 > t1) {
            const float t = t0;
            t0 = t1;
            t1 = t;
        }
        lo = fmaxf(lo, t0);
        hi = fminf(hi, t1);
    }
    r.px = base[0];
    r.py = base[1];
    r.pz = base[2];
    r.dx = dir[0];
    r.dy = dir[1];
    r.dz = dir[2];
    r.a0 = ceilf(lo / V.step) * V.step;
    r.n = (hit && lo < hi) ? max(0, (int)floorf((hi - r.a0) / V.step) + 1) : 0;
    return r;
}

// Cell and weights of sample i: texel coordinate pos*dim - 0.5, its integer
// part and fraction.  One expression (explicit fused multiply-adds) serves the
// forward and backward kernels, so both see the same cells and weights.
struct Cell {
    int ix, iy, iz;
    float wx, wy, wz;
};

__device__ __forceinline__ Cell sample_cell(const DvrBatch &B, const Ray &r, float step, int i) {
    const float a = __fmaf_rn((float)i, step, r.a0);
    const float cx = __fmaf_rn(__fmaf_rn(a, r.dx, r.px), B.fdim[0], -0.5f);
    const float cy = __fmaf_rn(__fmaf_rn(a, r.dy, r.py), B.fdim[1], -0.5f);
    const float cz = __fmaf_rn(__fmaf_rn(a, r.dz, r.pz), B.fdim[2], -0.5f);
    const float fx = floorf(cx), fy = floorf(cy), fz = floorf(cz);
    Cell c;
    c.ix = (int)fx;
    c.iy = (int)fy;
    c.iz = (int)fz;
    c.wx = cx - fx;
    c.wy = cy - fy;
    c.wz = cz - fz;
    return c;
}

__device__ __forceinline__ float lerp(float a, float b, float w) { return __fmaf_rn(w, b - a, a); }

// Trilinear value of a cell; cells inside the volume read their eight voxels
// without clamping (the common case), the boundary half-voxel clamps to edge.
__device__ __forceinline__ float trilinear(const DvrBatch &B, const float *__restrict__ vol, const Cell &c) {
    const int X = B.dim[0];
    float v0, v1, v2, v3, v4, v5, v6, v7;
    if ((unsigned)c.ix < (unsigned)(X - 1) && (unsigned)c.iy < (unsigned)(B.dim[1] - 1) &&
        (unsigned)c.iz < (unsigned)(B.dim[2] - 1)) {
        const float *p = vol + (c.iz * B.sxy + c.iy * X + c.ix);
        v0 = __ldg(p);
        v1 = __ldg(p + 1);
        v2 = __ldg(p + X);
        v3 = __ldg(p + X + 1);
        p += B.sxy;
        v4 = __ldg(p);
        v5 = __ldg(p + 1);
        v6 = __ldg(p + X);
        v7 = __ldg(p + X + 1);
    } else {
        const int x0 = min(max(c.ix, 0), X - 1), x1 = min(max(c.ix + 1, 0), X - 1);
        const int y0 = min(max(c.iy, 0), B.dim[1] - 1) * X, y1 = min(max(c.iy + 1, 0), B.dim[1] - 1) * X;
        const int z0 = min(max(c.iz, 0), B.dim[2] - 1) * B.sxy, z1 = min(max(c.iz + 1, 0), B.dim[2] - 1) * B.sxy;
        v0 = __ldg(vol + z0 + y0 + x0);
        v1 = __ldg(vol + z0 + y0 + x1);
        v2 = __ldg(vol + z0 + y1 + x0);
        v3 = __ldg(vol + z0 + y1 + x1);
        v4 = __ldg(vol + z1 + y0 + x0);
        v5 = __ldg(vol + z1 + y0 + x1);
        v6 = __ldg(vol + z1 + y1 + x0);
        v7 = __ldg(vol + z1 + y1 + x1);
    }
    const float a0 = lerp(v0, v1, c.wx), a1 = lerp(v2, v3, c.wx), a2 = lerp(v4, v5, c.wx), a3 = lerp(v6, v7, c.wx);
    return lerp(lerp(a0, a1, c.wy), lerp(a2, a3, c.wy), c.wz);
}

// LUT lookup: x = s*n - 0.5 clamped to [0, n-1]; cell k = floor, weight w of
// entry k+1.  L[k] holds the entries, D[k] = L[k+1] - L[k] (D[n-1] = 0).
struct LutCell {
    int k;
    float w;
    bool inside;                         // 0 <= x < n-1: the value's slope is n
};

__device__ __forceinline__ LutCell lut_cell(float s, int n) {
    LutCell c;
    const float x = __fmaf_rn(s, (float)n, -0.5f);
    c.inside = (x >= 0.0f) && (x < (float)(n - 1));
    const float xc = fminf(fmaxf(x, 0.0f), (float)(n - 1));
    c.k = (int)xc;
    c.w = xc - (float)c.k;
    return c;
}

__device__ __forceinline__ float4 lut_value(const float4 *L, const float4 *D, const LutCell &c) {
    const float4 a = L[c.k], d = D[c.k];
    return make_float4(__fmaf_rn(c.w, d.x, a.x), __fmaf_rn(c.w, d.y, a.y), __fmaf_rn(c.w, d.z, a.z),
                       __fmaf_rn(c.w, d.w, a.w));
}

__device__ __forceinline__ void load_lut(const float4 *__restrict__ lut_g, float4 *L, float4 *D, int n) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const float4 a = lut_g[i];
        L[i] = a;
        if (i + 1 < n) {
            const float4 b = lut_g[i + 1];
            D[i] = make_float4(b.x - a.x, b.y - a.y, b.z - a.z, b.w - a.w);
        } else {
            D[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
}

__device__ __forceinline__ int pixel_x(int bx, int tile_w) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    return bx * tile_w + (warp % (tile_w / 8)) * 8 + (lane & 7);
}

__device__ __forceinline__ int pixel_y(int by, int tile_w) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    return by * 8 + (warp / (tile_w / 8)) * 4 + (lane >> 3);
}

// ---------------------------------------------------------------------------
// forward: 256 threads = 32x8 pixels as 8x4 warp tiles; blockIdx.z = view

__global__ void __launch_bounds__(256) k_dvr_forward(const __grid_constant__ DvrBatch B,
                                                     const float *__restrict__ vol,
                                                     const float4 *__restrict__ lut_g, float *__restrict__ images,
                                                     float *__restrict__ trans, float *__restrict__ work) {
    extern __shared__ float4 sm[];
    float4 *L = sm, *D = sm + B.lut_len;
    load_lut(lut_g, L, D, B.lut_len);
    __syncthreads();
    const DvrView &V = B.v[blockIdx.z];
    const int x = pixel_x(blockIdx.x, 32), y = pixel_y(blockIdx.y, 32);
    if (x >= B.W || y >= B.H) return;
    const size_t npix = (size_t)B.W * B.H, pix = (size_t)y * B.W + x;
    float *wk = work ? work + V.work_off : nullptr;
    const int cmask = (1 << V.ckpt_shift) - 1;
    float T = 1.0f, cr = 0.0f, cg = 0.0f, cb = 0.0f;
    const Ray r = make_ray(B, V, x, y);
    int i = 0;
    for (; i < r.n; ++i) {
        if (wk && (i & cmask) == 0) wk[(size_t)(i >> V.ckpt_shift) * npix + pix] = T;
        const float s = trilinear(B, vol, sample_cell(B, r, V.step, i));
        const float4 c = lut_value(L, D, lut_cell(s, B.lut_len));
        const float wgt = T * c.w;
        cr = __fmaf_rn(wgt, c.x, cr);
        cg = __fmaf_rn(wgt, c.y, cg);
        cb = __fmaf_rn(wgt, c.z, cb);
        T *= (1.0f - c.w);
        if (T < V.t_min) {
            ++i;
            break;
        }
    }
    const size_t o = (size_t)blockIdx.z * npix + pix;
    images[3 * o + 0] = cr;
    images[3 * o + 1] = cg;
    images[3 * o + 2] = cb;
    trans[o] = T;
    if (wk) {
        reinterpret_cast<int *>(wk + (size_t)V.max_ckpt * npix)[pix] = i;   // samples taken
        wk[(size_t)(V.max_ckpt + 1) * npix + pix] = T;                      // transmittance after them
    }
}

// ---------------------------------------------------------------------------
// backward: 128 threads = 16x8 pixels as 8x4 warp tiles; blockIdx.z = view

// Adds the LUT-gradient runs that lanes end at this step (cell k: a0 to
// entry k, a1 to entry k + 1) to the block's shared bins.  Every lane of the
// warp calls it.  Lanes ending a run on the same cell are summed by warp
// shuffles first (a butterfly per cell), so a cell takes one set of
// shared-memory atomics per warp and step; a lane alone on its cell adds
// directly.
__device__ __forceinline__ void flush_lut_warp(float *bins, int n, bool flush, int k, const float4 &a0,
                                               const float4 &a1) {
    const unsigned FULL = 0xffffffffu;
    if (__ballot_sync(FULL, flush) == 0u) return;
    const int lane = threadIdx.x & 31;
    const unsigned peers = __match_any_sync(FULL, flush ? k : -1);
    const bool alone = flush && __popc(peers) == 1;
    if (alone) {
        atomicAdd(&bins[4 * k + 0], a0.x);
        atomicAdd(&bins[4 * k + 1], a0.y);
        atomicAdd(&bins[4 * k + 2], a0.z);
        atomicAdd(&bins[4 * k + 3], a0.w);
        if (k + 1 < n) {
            atomicAdd(&bins[4 * k + 4], a1.x);
            atomicAdd(&bins[4 * k + 5], a1.y);
            atomicAdd(&bins[4 * k + 6], a1.z);
            atomicAdd(&bins[4 * k + 7], a1.w);
        }
    }
    unsigned shared = __ballot_sync(FULL, flush && !alone);
    while (shared) {
        const int leader = __ffs(shared) - 1;
        const unsigned grp = __shfl_sync(FULL, peers, leader);
        const bool in = (grp >> lane) & 1u;
        float v[8] = {in ? a0.x : 0.f, in ? a0.y : 0.f, in ? a0.z : 0.f, in ? a0.w : 0.f,
                      in ? a1.x : 0.f, in ? a1.y : 0.f, in ? a1.z : 0.f, in ? a1.w : 0.f};
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
            for (int c = 0; c < 8; ++c) v[c] += __shfl_xor_sync(FULL, v[c], o);
        }
        if (lane == leader) {
#pragma unroll
            for (int c = 0; c < 4; ++c) atomicAdd(&bins[4 * k + c], v[c]);
            if (k + 1 < n) {
#pragma unroll
                for (int c = 0; c < 4; ++c) atomicAdd(&bins[4 * k + 4 + c], v[4 + c]);
            }
        }
        shared &= ~grp;
    }
}

__device__ __forceinline__ void flush_vol(float *__restrict__ gv, const DvrBatch &B, int ix, int iy, int iz,
                                          const float (&acc)[8]) {
    if (ix == INT_MIN) return;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        if (acc[c] == 0.0f) continue;
        const int x = min(max(ix + (c & 1), 0), B.dim[0] - 1);
        const int y = min(max(iy + ((c >> 1) & 1), 0), B.dim[1] - 1);
        const int z = min(max(iz + (c >> 2), 0), B.dim[2] - 1);
        atomicAdd(&gv[z * B.sxy + y * B.dim[0] + x], acc[c]);
    }
}

__device__ __forceinline__ bool gradient_finite(float r, float g, float b) {
    return fabsf(r) + fabsf(g) + fabsf(b) <= FLT_MAX;
}

// Reverse march.  A ray walks its samples from the last to the first,
// reconstructing T_i = T_{i+1} / (1 - a_i) from the transmittance saved after
// its last sample; at every checkpoint (each 2^ckpt_shift samples) T is taken
// from the forward pass instead, so a reconstruction never runs for more
// than one checkpoint interval.  A sample with a_i = 1 (nothing to divide
// by) takes T_i by re-marching forward from its interval's checkpoint.  Each
// sample is fetched once otherwise.  The walk is warp-uniform (lanes past
// their first sample idle), so the LUT-gradient runs that end in one step
// can be combined across the warp.  ODD: only the rays whose
// pixel gradient is not finite (after k_dvr_backward_bricks, which leaves them
// out).
template <bool VOLGRAD, bool ODD>
__global__ void __launch_bounds__(128) k_dvr_backward(const __grid_constant__ DvrBatch B,
                                                      const float *__restrict__ vol,
                                                      const float4 *__restrict__ lut_g,
                                                      const float *__restrict__ work,
                                                      const float *__restrict__ grad_images,
                                                      float *__restrict__ grad_lut, float *__restrict__ grad_vol) {
    extern __shared__ float4 sm[];
    const int n = B.lut_len;
    float4 *L = sm, *D = sm + n;
    float *bins = reinterpret_cast<float *>(sm + 2 * n);
    const DvrView &V = B.v[blockIdx.z];
    const int x = pixel_x(blockIdx.x, 16), y = pixel_y(blockIdx.y, 16);
    const bool in_image = x < B.W && y < B.H;
    const size_t npix = (size_t)B.W * B.H, pix = in_image ? (size_t)y * B.W + x : 0;
    const size_t o = (size_t)blockIdx.z * npix + pix;
    float gr = 0.f, gg = 0.f, gb = 0.f, T = 0.f;
    if (in_image) {
        gr = grad_images[3 * o];
        gg = grad_images[3 * o + 1];
        gb = grad_images[3 * o + 2];
    }
    if (ODD && !__syncthreads_or(!gradient_finite(gr, gg, gb))) return;
    load_lut(lut_g, L, D, n);
    for (int i = threadIdx.x; i < 4 * n; i += blockDim.x) bins[i] = 0.0f;
    __syncthreads();

    const float *wk = work + V.work_off;
    int ns = 0;
    if (in_image) {
        ns = reinterpret_cast<const int *>(wk + (size_t)V.max_ckpt * npix)[pix];
        T = wk[(size_t)(V.max_ckpt + 1) * npix + pix];
        if (gr == 0.0f && gg == 0.0f && gb == 0.0f) ns = 0;
        if (ODD && gradient_finite(gr, gg, gb)) ns = 0;
    }
    const Ray r = make_ray(B, V, x, y);
    const int cmask = (1 << V.ckpt_shift) - 1;
    int steps = ns;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) steps = max(steps, __shfl_xor_sync(0xffffffffu, steps, off));
    float Ur = 0.f, Ug = 0.f, Ub = 0.f;
    int lk = -1;
    float4 la0 = make_float4(0.f, 0.f, 0.f, 0.f), la1 = la0;
    int vx = INT_MIN, vy = 0, vz = 0;
    float va[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) va[c] = 0.0f;

    for (int t = 0; t < steps; ++t) {
        const int i = ns - 1 - t;
        const bool live = i >= 0;
        LutCell h;
        h.k = -1;
        h.w = 0.0f;
        h.inside = false;
        float d_cr = 0.f, d_cg = 0.f, d_cb = 0.f, d_a = 0.f;
        Cell c = {};
        if (live) {
            c = sample_cell(B, r, V.step, i);
            h = lut_cell(trilinear(B, vol, c), n);
            const float4 q = lut_value(L, D, h);
            const float d = 1.0f - q.w;
            float Ti;
            if ((i & cmask) == 0) {
                Ti = wk[(size_t)(i >> V.ckpt_shift) * npix + pix];
            } else if (d != 0.0f) {
                Ti = T / d;
            } else {
                Ti = wk[(size_t)(i >> V.ckpt_shift) * npix + pix];
                for (int j = i & ~cmask; j < i; ++j)
                    Ti *= 1.0f - lut_value(L, D, lut_cell(trilinear(B, vol, sample_cell(B, r, V.step, j)), n)).w;
            }
            T = Ti;
            d_cr = Ti * q.w * gr;
            d_cg = Ti * q.w * gg;
            d_cb = Ti * q.w * gb;
            d_a = Ti * (gr * (q.x - Ur) + gg * (q.y - Ug) + gb * (q.z - Ub));
            Ur = q.w * q.x + (1.0f - q.w) * Ur;
            Ug = q.w * q.y + (1.0f - q.w) * Ug;
            Ub = q.w * q.z + (1.0f - q.w) * Ub;
        }
        const bool change = live && h.k != lk;
        flush_lut_warp(bins, n, change && lk >= 0, lk, la0, la1);
        if (change) {
            lk = h.k;
            la0 = make_float4(0.f, 0.f, 0.f, 0.f);
            la1 = la0;
        }
        if (live) {
            const float w1 = h.w, w0 = 1.0f - h.w;
            la0.x += w0 * d_cr;
            la0.y += w0 * d_cg;
            la0.z += w0 * d_cb;
            la0.w += w0 * d_a;
            la1.x += w1 * d_cr;
            la1.y += w1 * d_cg;
            la1.z += w1 * d_cb;
            la1.w += w1 * d_a;
            if (VOLGRAD && h.inside) {
                const float4 dd = D[h.k];
                const float ds = (float)n * (d_cr * dd.x + d_cg * dd.y + d_cb * dd.z + d_a * dd.w);
                if (ds != 0.0f) {
                    if (c.ix != vx || c.iy != vy || c.iz != vz) {
                        flush_vol(grad_vol, B, vx, vy, vz, va);
                        vx = c.ix;
                        vy = c.iy;
                        vz = c.iz;
#pragma unroll
                        for (int k = 0; k < 8; ++k) va[k] = 0.0f;
                    }
                    const float y0z0 = (1.0f - c.wy) * (1.0f - c.wz) * ds, y1z0 = c.wy * (1.0f - c.wz) * ds;
                    const float y0z1 = (1.0f - c.wy) * c.wz * ds, y1z1 = c.wy * c.wz * ds;
                    va[0] += (1.0f - c.wx) * y0z0;
                    va[1] += c.wx * y0z0;
                    va[2] += (1.0f - c.wx) * y1z0;
                    va[3] += c.wx * y1z0;
                    va[4] += (1.0f - c.wx) * y0z1;
                    va[5] += c.wx * y0z1;
                    va[6] += (1.0f - c.wx) * y1z1;
                    va[7] += c.wx * y1z1;
                }
            }
        }
    }
    flush_lut_warp(bins, n, lk >= 0, lk, la0, la1);
    if (VOLGRAD) flush_vol(grad_vol, B, vx, vy, vz, va);
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * n; i += blockDim.x) {
        const float v = bins[i];
        if (v != 0.0f) atomicAdd(&grad_lut[i], v);
    }
}

// ---------------------------------------------------------------------------
// Bricked path (scratch given): the volume is rearranged, per call, into
// bricks of 8^3 cells before the rays are marched.
//
// A ray sample reads the eight voxels of its cell.  In the x-fastest volume
// the 32 lanes of a warp, whose pixels spread over a plane across the rays,
// touch up to 24 different 128-byte lines with each of the eight loads, and
// the kernels above run at the rate at which the load/store unit takes lines
// (about 190 cycles per warp and sample, 99% of L1TEX).  On 256^3 with eight
// views of 256^2 the rearrangement takes 66-77 us, the forward 640 us (plain:
// 5.2 ms) and the backward 1430 us (plain: 6.2 ms); the load/store unit (93%)
// and instruction issue (78%) now share the forward's bound.  Here a cell's plane
// of four voxels is one float4 ("quad"), so a sample is two 16-byte loads;
// a 128-byte line holds 4x2 cells of one plane, and a quarter warp (the lanes
// a 16-byte load serves together) covers 4x2 pixels.
//
// A brick holds the 8x8x9 quads of its cells (its last plane is the next
// brick's first, kept twice so that a cell never needs two bricks), and is
// built only if a sample in it can matter, which the LUT decides from the
// brick's smallest and largest voxel:
//  * forward: where every LUT entry the brick can reach has alpha 0, a sample
//    leaves colour and transmittance as they are ("clear" brick);
//  * backward: there the only gradient is dL/dalpha of those entries.  Where
//    in addition all voxels of the brick are equal (padding, clipped air),
//    every sample in it adds the same term, which is added once, times the
//    number of samples ("flat" brick).
// Byte maps of the Chebyshev distance to the next brick that is not clear
// (forward) or not flat (backward) let a ray leave such regions in one step.
//
// Cell (ix, iy, iz), ix = -1 .. X-1, has cell coordinates (ix+1, ...); cells
// at the border repeat the edge voxel, which is the clamping above.

constexpr int kDvrBrickQuads = 576;      // 8 x 8 x 9
constexpr float kDvrExitMargin = 0.05f;  // cells; covers the rounding of the linear exit model
constexpr float kDvrSlow = 1e-4f;        // cells a sample (samples_inside)

struct DvrBricks {
    int nb[3];
    const float4 *quads;
    float4 *gquads;                      // voxel gradients in the same layout (backward)
    const uint8_t *dist;                 // per brick; 0: its samples are evaluated
    const float *flat;                   // per flat brick: the value of its voxels (backward)
};

// Offset of a cell's first quad inside its brick (the second is 64 further).
__device__ __forceinline__ int quad_offset(int lx, int ly, int lz) {
    return lz * 64 + (ly >> 1) * 16 + (lx >> 2) * 8 + (ly & 1) * 4 + (lx & 3);
}

// One block per row of four bricks: their 33 x 9 x 9 voxels (a warp reads a
// row of them, lane = x), each brick's range, the LUT entries it can reach,
// and, for a needed brick, its quads (and zeroed gradient quads).  The lanes
// keep the range of their column over the rows, so the ranges cost two
// instructions a row and one reduction a block.
template <bool BACKWARD>
__global__ void __launch_bounds__(256) k_dvr_build(int X, int Y, int Z, int nbx, const float *__restrict__ vol,
                                                   const float4 *__restrict__ lut, int n, float4 *__restrict__ quads,
                                                   float4 *__restrict__ gquads, uint8_t *__restrict__ needed,
                                                   float *__restrict__ flat, double *__restrict__ lut_sums) {
    __shared__ float v[81][33];
    __shared__ float s_lo[8][33], s_hi[8][33];
    __shared__ int s_need[4];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (BACKWARD && blockIdx.x + blockIdx.y + blockIdx.z == 0)
        for (int i = tid; i < 4 * n; i += 256) lut_sums[i] = 0.0;
    const int x0 = blockIdx.x * 32 - 1, y0 = blockIdx.y * 8 - 1, z0 = blockIdx.z * 8 - 1;
    const int gx = min(max(x0 + lane, 0), X - 1), gx32 = min(x0 + 32, X - 1);
    float lo = INFINITY, hi = -INFINITY, lo32 = INFINITY, hi32 = -INFINITY;
    bool odd = false;                    // a value the range test cannot place
#pragma unroll
    for (int t = 0; t < 11; ++t) {
        const int row = t * 8 + warp, lz = row / 9, ly = row - lz * 9;
        if (row >= 81) break;
        const int gy = min(max(y0 + ly, 0), Y - 1), gz = min(max(z0 + lz, 0), Z - 1);
        const float *p = vol + ((size_t)gz * Y + gy) * X;
        const float a = __ldg(p + gx);
        v[row][lane] = a;
        odd |= !(fabsf(a) <= 2.0f);      // (beyond, the rounding could pass an entry)
        lo = fminf(lo, a);
        hi = fmaxf(hi, a);
        if (lane == 0) {
            const float e = __ldg(p + gx32);
            v[row][32] = e;
            odd |= !(fabsf(e) <= 2.0f);
            lo32 = fminf(lo32, e);
            hi32 = fmaxf(hi32, e);
        }
    }
    s_lo[warp][lane] = lo;
    s_hi[warp][lane] = hi;
    if (lane == 0) {
        s_lo[warp][32] = lo32;
        s_hi[warp][32] = hi32;
    }
    odd = __syncthreads_or(odd);
    if (warp < 4) {
        // warp j: brick j, columns 8 j .. 8 j + 8
        lo = INFINITY;
        hi = -INFINITY;
        for (int i = lane; i < 72; i += 32) {
            lo = fminf(lo, s_lo[i / 9][warp * 8 + i % 9]);
            hi = fmaxf(hi, s_hi[i / 9][warp * 8 + i % 9]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        // entries a sample between lo and hi can reach, one more on each
        // side for the rounding of the interpolation
        bool seen = odd;
        if (!odd) {
            const float a = fminf(fmaxf(__fmaf_rn(lo, (float)n, -0.5f), 0.0f), (float)(n - 1));
            const float b = fminf(fmaxf(__fmaf_rn(hi, (float)n, -0.5f), 0.0f), (float)(n - 1));
            const int i0 = max((int)a - 1, 0), i1 = min((int)b + 2, n - 1);
            for (int i = i0 + lane; i <= i1; i += 32) {
                const float4 c = __ldg(lut + i);
                // a colour that is not finite would show even at alpha 0
                seen |= c.w != 0.0f || !(fabsf(c.x) <= FLT_MAX && fabsf(c.y) <= FLT_MAX && fabsf(c.z) <= FLT_MAX);
            }
        }
        seen = __any_sync(0xffffffffu, seen);
        if (lane == 0) {
            const int bx = blockIdx.x * 4 + warp;
            const int need = bx >= nbx ? 0 : seen ? 2 : BACKWARD && lo != hi ? 1 : 0;
            s_need[warp] = need;
            if (bx < nbx) {
                const size_t b = ((size_t)blockIdx.z * gridDim.y + blockIdx.y) * nbx + bx;
                needed[b] = (uint8_t)need;
                if (BACKWARD) flat[b] = lo;
            }
        }
    }
    __syncthreads();
    const size_t b0 = ((size_t)blockIdx.z * gridDim.y + blockIdx.y) * nbx + blockIdx.x * 4;
    // 64 threads a brick, one per cell of a plane
    const int j = tid >> 6, r = tid & 63, need = s_need[j];
    if (need == 0) return;
    const int lx = j * 8 + ((r & 3) | ((r >> 1) & 4)), ly = ((r >> 2) & 1) | ((r >> 3) & 6);
    float4 *q = quads + (b0 + j) * kDvrBrickQuads + r;
    float4 *g = BACKWARD && gquads && need == 2 ? gquads + (b0 + j) * kDvrBrickQuads + r : nullptr;
#pragma unroll
    for (int lz = 0; lz < 9; ++lz) {
        const float *p = &v[lz * 9 + ly][lx];
        q[lz * 64] = make_float4(p[0], p[1], p[33], p[34]);
        // where nothing is seen no voxel has a gradient
        if (g) g[lz * 64] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

__device__ __forceinline__ void add_lut_sums(int n, const double *__restrict__ sums, float *__restrict__ grad_lut) {
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        if (sums[i] != 0.0) atomicAdd(&grad_lut[i], (float)sums[i]);
}

__global__ void __launch_bounds__(256) k_dvr_lut_add(int n, const double *__restrict__ sums, float *__restrict__ grad_lut) {
    add_lut_sums(n, sums, grad_lut);
}

// The gradient quads of one brick, summed per voxel and added to the gradient
// volume (voxels on a brick's faces get a sum from each brick); the first
// block also adds the LUT sums to the LUT gradient.
__global__ void __launch_bounds__(256) k_dvr_fold(int X, int Y, int Z, const float4 *__restrict__ gquads,
                                                  const uint8_t *__restrict__ needed, float *__restrict__ grad_vol,
                                                  int n, const double *__restrict__ sums, float *__restrict__ grad_lut) {
    __shared__ float4 q[kDvrBrickQuads];
    const size_t b = ((size_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
    if (b == 0) add_lut_sums(n, sums, grad_lut);
    if (needed[b] != 2) return;
    for (int i = threadIdx.x; i < kDvrBrickQuads; i += 256) q[i] = gquads[b * kDvrBrickQuads + i];
    __syncthreads();
    const int x0 = blockIdx.x * 8 - 1, y0 = blockIdx.y * 8 - 1, z0 = blockIdx.z * 8 - 1;
    for (int i = threadIdx.x; i < 729; i += 256) {
        const int lx = i % 9, ly = (i / 9) % 9, lz = i / 81;
        float s = 0.0f;
        if (lx < 8 && ly < 8) s += q[quad_offset(lx, ly, lz)].x;
        if (lx > 0 && ly < 8) s += q[quad_offset(lx - 1, ly, lz)].y;
        if (lx < 8 && ly > 0) s += q[quad_offset(lx, ly - 1, lz)].z;
        if (lx > 0 && ly > 0) s += q[quad_offset(lx - 1, ly - 1, lz)].w;
        if (s == 0.0f) continue;
        const int gx = min(max(x0 + lx, 0), X - 1), gy = min(max(y0 + ly, 0), Y - 1), gz = min(max(z0 + lz, 0), Z - 1);
        atomicAdd(grad_vol + ((size_t)gz * Y + gy) * X + gx, s);
    }
}

// Cell coordinates and weights of sample i: sample_cell with the cell counted
// from -1.  The floor is an addition of 1.5 * 2^23 rounded down (exact for
// the |c| < 2^22 there are; floorf and the conversion to int would go through
// the quarter-rate unit), and the sample number is kept as a float.  The
// samples of a ray lie in the cells -1 .. X-1 (to a few hundredths, see
// use_bricks); inside a known brick only the low three bits are used.
struct BrickCell {
    int x, y, z;
    float wx, wy, wz;
};

__device__ __forceinline__ void floor_cell(float c, int &i, float &w) {
    const float magic = 12582912.0f;     // 0x4b400000
    const float t = __fadd_rd(c, magic);
    i = __float_as_int(t) - (0x4b400000 - 1);
    w = c - (t - magic);
}

__device__ __forceinline__ BrickCell brick_cell(const DvrBatch &B, const Ray &r, float step, float i) {
    const float a = __fmaf_rn(i, step, r.a0);
    BrickCell q;
    floor_cell(__fmaf_rn(__fmaf_rn(a, r.dx, r.px), B.fdim[0], -0.5f), q.x, q.wx);
    floor_cell(__fmaf_rn(__fmaf_rn(a, r.dy, r.py), B.fdim[1], -0.5f), q.y, q.wy);
    floor_cell(__fmaf_rn(__fmaf_rn(a, r.dz, r.pz), B.fdim[2], -0.5f), q.z, q.wz);
    return q;
}

// The brick of a cell (clamped to those there are).
__device__ __forceinline__ uint32_t brick_of(const DvrBatch &B, const DvrBricks &K, BrickCell &c) {
    c.x = min(max(c.x, 0), B.dim[0]);
    c.y = min(max(c.y, 0), B.dim[1]);
    c.z = min(max(c.z, 0), B.dim[2]);
    return ((uint32_t)(c.z >> 3) * K.nb[1] + (c.y >> 3)) * K.nb[0] + (c.x >> 3);
}

// Samples per cell along each axis; 0: slower than 1e-4 cells a sample, with
// DRIFT, or not moving at all.
template <bool DRIFT>
__device__ __forceinline__ float3 inverse_rate(const DvrBatch &B, const Ray &r, float step) {
    const float x = r.dx * step * B.fdim[0], y = r.dy * step * B.fdim[1], z = r.dz * step * B.fdim[2];
    const float slow = DRIFT ? kDvrSlow : 0.0f;
    return make_float3(fabsf(x) > slow ? 1.0f / x : 0.0f, fabsf(y) > slow ? 1.0f / y : 0.0f,
                       fabsf(z) > slow ? 1.0f / z : 0.0f);
}

// Further samples (after sample i in cell c, or BACK, before it) certain to stay
// in the bricks within `reach` of the one that holds c.  DRIFT: an axis is slower
// than kDvrSlow and yet moves (a camera turned in steps leaves 1e-8 in its
// matrix), and a ray on a brick's face crosses it by one rounding.  So the last
// of those samples is looked at: every operation of a coordinate is rounded
// monotonically, so the samples between lie between.
template <bool BACK, bool DRIFT>
__device__ __forceinline__ int samples_inside(const DvrBatch &B, const Ray &r, float step, const float3 &inv, int i,
                                              const BrickCell &c, int reach) {
    float t = 4096.0f;
    const int b[3] = {c.x >> 3, c.y >> 3, c.z >> 3};
    const float p[3] = {c.x + c.wx, c.y + c.wy, c.z + c.wz};
    const float iv[3] = {BACK ? -inv.x : inv.x, BACK ? -inv.y : inv.y, BACK ? -inv.z : inv.z};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float lo = (float)((b[k] - reach) * 8), hi = (float)((b[k] + reach + 1) * 8);
        const float room = iv[k] > 0.0f ? hi - kDvrExitMargin - p[k] : lo + kDvrExitMargin - p[k];
        if (iv[k] != 0.0f) t = fminf(t, room * iv[k]);
    }
    const int n = t > 0.0f ? (int)t : 0;
    if (DRIFT) {
        const int j = BACK ? max(i - n, 0) : min(i + n, r.n - 1);
        const BrickCell e = brick_cell(B, r, step, (float)j);
        if (abs((e.x >> 3) - b[0]) > reach || abs((e.y >> 3) - b[1]) > reach || abs((e.z >> 3) - b[2]) > reach) return 0;
    }
    return n;
}

__device__ __forceinline__ float quad_trilinear(const float4 &a, const float4 &b, float wx, float wy, float wz) {
    const float a0 = lerp(a.x, a.y, wx), a1 = lerp(a.z, a.w, wx), a2 = lerp(b.x, b.y, wx), a3 = lerp(b.z, b.w, wx);
    return lerp(lerp(a0, a1, wy), lerp(a2, a3, wy), wz);
}

__device__ __forceinline__ float brick_trilinear(const float4 *__restrict__ q, const BrickCell &c) {
    return quad_trilinear(__ldg(q), __ldg(q + 64), c.wx, c.wy, c.wz);
}

// The pixel and view of this thread.  A block covers 16 pixels by 2 per warp,
// as 8x4 warp tiles whose quarter warps are 4x2 pixels.  Blocks are taken
// from the middle of the image outwards, all views of a tile in turn, so that
// the long rays start first.
struct DvrPixel {
    int x, y, view;
};

__device__ __forceinline__ int middle_out(int i, int n) {
    const int m = (n - 1) >> 1;          // m, m + 1, m - 1, m + 2, ...
    return m + ((i & 1) ? (i + 1) >> 1 : -(i >> 1));
}

__device__ __forceinline__ DvrPixel dvr_pixel(const DvrBatch &B, int views) {
    const int h = blockDim.x >> 4, tx = (B.W + 15) >> 4, ty = (B.H + h - 1) / h;
    const int t = blockIdx.x / views, row = t / tx, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    DvrPixel p;
    p.view = blockIdx.x - t * views;
    p.x = middle_out(t - row * tx, tx) * 16 + (warp & 1) * 8 + (lane & 3) + ((lane >> 2) & 4);
    p.y = middle_out(row, ty) * h + (warp >> 1) * 4 + ((lane >> 2) & 3);
    return p;
}

// Forward over bricks: the samples, their order and every operation on them
// are k_dvr_forward's, without those that change nothing.
constexpr int kForwardThreads = 128;

template <int kAhead, bool DRIFT>
__global__ void __launch_bounds__(kForwardThreads) k_dvr_forward_bricks(const __grid_constant__ DvrBatch B,
                                                            const __grid_constant__ DvrBricks K, int views,
                                                            const float4 *__restrict__ lut_g,
                                                            float *__restrict__ images, float *__restrict__ trans,
                                                            float *__restrict__ work) {
    extern __shared__ float4 sm[];
    float4 *L = sm, *D = sm + B.lut_len;
    load_lut(lut_g, L, D, B.lut_len);
    __syncthreads();
    const DvrPixel px = dvr_pixel(B, views);
    const DvrView &V = B.v[px.view];
    const int x = px.x, y = px.y;
    if (x >= B.W || y >= B.H) return;
    const size_t npix = (size_t)B.W * B.H, pix = (size_t)y * B.W + x;
    float *wk = work ? work + V.work_off : nullptr;
    const int cmask = (1 << V.ckpt_shift) - 1;
    float T = 1.0f, cr = 0.0f, cg = 0.0f, cb = 0.0f;
    const Ray r = make_ray(B, V, x, y);
    const float3 inv = inverse_rate<DRIFT>(B, r, V.step);
    // a threshold above 1 ends every ray at its first sample
    const bool may_skip = !(T < V.t_min);
    int i = 0, look = 0;                 // look: first sample whose brick is not known
    const float4 *brick = K.quads;
    bool more = r.n > 0;
    while (more) {
        bool sample = true;
        if (i >= look) {
            BrickCell c = brick_cell(B, r, V.step, (float)i);
            const uint32_t b = brick_of(B, K, c);
            const int d = K.dist[b];
            look = min(i + 1 + samples_inside<false, DRIFT>(B, r, V.step, inv, i, c, max(d - 1, 0)), r.n);
            brick = K.quads + (size_t)b * kDvrBrickQuads;
            if (d > 0) {
                sample = false;
                if (may_skip) {
                    // (a transmittance that is not finite turns 0 * T, and with
                    // it the colour, to NaN)
                    if (!(fabsf(T) <= FLT_MAX)) cr = cg = cb = T * 0.0f;
                    if (wk)
                        for (int j = (i + cmask) & ~cmask; j < look; j += cmask + 1)
                            wk[(size_t)(j >> V.ckpt_shift) * npix + pix] = T;
                    i = look;
                    more = i < r.n;
                } else {
                    if (wk) wk[pix] = T;
                    i = 1;
                    more = false;
                }
            }
        }
        if (sample) {
            // the loads of up to kAhead samples of the brick, then their
            // compositing in order
            const int m = min(look - i, kAhead);
            BrickCell c[kAhead];
            float4 qa[kAhead], qb[kAhead];
#pragma unroll
            for (int k = 0; k < kAhead; ++k) {
                c[k] = brick_cell(B, r, V.step, (float)(i + k));
                const float4 *q = brick + quad_offset(c[k].x & 7, c[k].y & 7, c[k].z & 7);
                if (k < m) {
                    qa[k] = __ldg(q);
                    qb[k] = __ldg(q + 64);
                }
            }
#pragma unroll
            for (int k = 0; k < kAhead; ++k) {
                if (k < m && more) {
                    if (wk && (i & cmask) == 0) wk[(size_t)(i >> V.ckpt_shift) * npix + pix] = T;
                    const float4 q = lut_value(L, D, lut_cell(quad_trilinear(qa[k], qb[k], c[k].wx, c[k].wy, c[k].wz), B.lut_len));
                    const float wgt = T * q.w;
                    cr = __fmaf_rn(wgt, q.x, cr);
                    cg = __fmaf_rn(wgt, q.y, cg);
                    cb = __fmaf_rn(wgt, q.z, cb);
                    T *= (1.0f - q.w);
                    ++i;
                    more = i < r.n && !(T < V.t_min);
                }
            }
        }
    }
    const size_t o = (size_t)px.view * npix + pix;
    images[3 * o + 0] = cr;
    images[3 * o + 1] = cg;
    images[3 * o + 2] = cb;
    trans[o] = T;
    if (wk) {
        reinterpret_cast<int *>(wk + (size_t)V.max_ckpt * npix)[pix] = i;   // samples taken
        wk[(size_t)(V.max_ckpt + 1) * npix + pix] = T;                      // transmittance after them
    }
}

// The LUT gradient of one ray.  Its colour part is T_i a_i times the pixel's
// gradient, so a LUT cell needs four sums: (w0, w1) x (T a, dL/da).  They are
// kept per lane in shared memory for a window of WIN cells about the values
// the ray meets (noise about a tissue value stays inside it), so a sample
// costs one 16-byte read and write without a conflict, and the block's bins
// are touched only when a ray leaves its window.  The same noise spans more
// cells of a longer table: ten from 257 entries on (microseconds a backward with
// six / ten cells: 256 entries, eight views of 256^2 on 256^3, all visible 3740 /
// 3897; 500 entries 5503 / 4633, one view of 321x243 1142 / 841, where the plain
// kernel takes 1091), and six again where the table fills the shared memory (three
// blocks per SM: 900 entries, 64^3, 1681 / 2050; 256^3 7830 / 8633).
constexpr int kWinShort = 6, kWinLong = 10;
constexpr int kWinShortLut = 256, kWinLongLut = 750;
constexpr int kBackThreads = 128;

static int window_cells(int lut_len) {
    return lut_len > kWinShortLut && lut_len <= kWinLongLut ? kWinLong : kWinShort;
}

__device__ __forceinline__ void bin_add(float *bins, int n, int k, float gr, float gg, float gb, const float4 &a) {
    if (a.x != 0.0f) {
        atomicAdd(&bins[4 * k + 0], gr * a.x);
        atomicAdd(&bins[4 * k + 1], gg * a.x);
        atomicAdd(&bins[4 * k + 2], gb * a.x);
    }
    if (a.z != 0.0f) atomicAdd(&bins[4 * k + 3], a.z);
    if (k + 1 < n) {
        if (a.y != 0.0f) {
            atomicAdd(&bins[4 * k + 4], gr * a.y);
            atomicAdd(&bins[4 * k + 5], gg * a.y);
            atomicAdd(&bins[4 * k + 6], gb * a.y);
        }
        if (a.w != 0.0f) atomicAdd(&bins[4 * k + 7], a.w);
    }
}

// The voxel sums of a cell: one 16-byte reduction per plane.
__device__ __forceinline__ void flush_quads(float4 *g, uint32_t cell, const float (&v)[8]) {
    if (cell == 0xffffffffu) return;
    float4 *p = g + cell;
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};"
                 :: "l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]) : "memory");
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};"
                 :: "l"(p + 64), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
}

// Backward over bricks: k_dvr_backward's reverse march; the lanes of a warp do
// not wait for one another.  Of the colour behind a sample only its product
// with the pixel's gradient, U . g, is needed: one recurrence instead of three.
// The blocks' LUT sums are added up in double: thousands of blocks add to the
// same few entries, and in fp32 that order-dependent sum was the largest
// error of the LUT gradient (6e-7 relative, 1.6e-6 at worst).
// 72-80 registers and 24 KB of shared memory at 256 LUT entries: six blocks per
// SM (seven spill and leave too little L1: 1.45 -> 1.85 ms on 256^3, eight
// views of 256^2; five: 1.52).  The next sample's loads are issued before a
// sample is summed.  Tried and left: four lanes per ray (2.26 ms; forward 1.14
// against 0.64: the brick look-ups are then made by every lane).
template <bool VOLGRAD, bool DRIFT, int WIN>
__global__ void __launch_bounds__(kBackThreads, 6)
k_dvr_backward_bricks(const __grid_constant__ DvrBatch B, const __grid_constant__ DvrBricks K, int views,
                      const float4 *__restrict__ lut_g, const float *__restrict__ work,
                      const float *__restrict__ grad_images, double *__restrict__ lut_sums,
                      float *__restrict__ grad_vol) {
    extern __shared__ float4 sm[];
    const int n = B.lut_len, tid = threadIdx.x;
    float4 *L = sm, *D = sm + n;
    float4 *win = sm + 2 * n + tid;      // [WIN][kBackThreads]
    float *bins = reinterpret_cast<float *>(sm + 2 * n + WIN * kBackThreads);
    load_lut(lut_g, L, D, n);
    for (int i = tid; i < 4 * n; i += kBackThreads) bins[i] = 0.0f;
#pragma unroll
    for (int k = 0; k < WIN; ++k) win[k * kBackThreads] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();

    const DvrPixel px = dvr_pixel(B, views);
    const DvrView &V = B.v[px.view];
    const bool in_image = px.x < B.W && px.y < B.H;
    const size_t npix = (size_t)B.W * B.H, pix = in_image ? (size_t)px.y * B.W + px.x : 0;
    const float *wk = work + V.work_off;
    const size_t o = (size_t)px.view * npix + pix;
    float gr = 0.f, gg = 0.f, gb = 0.f, T = 0.f;
    int ns = 0;
    if (in_image) {
        gr = grad_images[3 * o];
        gg = grad_images[3 * o + 1];
        gb = grad_images[3 * o + 2];
        ns = reinterpret_cast<const int *>(wk + (size_t)V.max_ckpt * npix)[pix];
        T = wk[(size_t)(V.max_ckpt + 1) * npix + pix];
        // (a gradient that is not finite spreads to every cell and voxel the
        // ray meets, zero terms too: k_dvr_backward takes those rays)
        if ((gr == 0.0f && gg == 0.0f && gb == 0.0f) || !gradient_finite(gr, gg, gb)) ns = 0;
    }
    const Ray r = make_ray(B, V, px.x, px.y);
    const float3 inv = inverse_rate<DRIFT>(B, r, V.step);
    const int cmask = (1 << V.ckpt_shift) - 1;
    float U = 0.0f;                      // U . g
    int wbase = 0;                       // first LUT cell of the window
    unsigned used = 0u;                  // its cells that hold a sum
    uint32_t cell = 0xffffffffu;         // quad of the voxel sums (none yet)
    float va[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) va[c] = 0.0f;
    uint32_t brick = 0;
    bool flat = false;
    float flat_value = 0.0f;
    int look = ns;                       // samples below `look` lie in bricks not known yet
    int i = ns - 1;
    uint32_t at = 0;                     // quad of sample i, its weights and values
    float wx = 0.f, wy = 0.f, wz = 0.f;
    float4 qa = make_float4(0.f, 0.f, 0.f, 0.f), qb = qa;
    while (i >= 0) {
        int count = 1;                   // samples this step stands for
        if (i < look) {
            BrickCell c = brick_cell(B, r, V.step, (float)i);
            const uint32_t b = brick_of(B, K, c);
            const int d = K.dist[b];
            flat = d > 0;
            look = max(i - samples_inside<true, DRIFT>(B, r, V.step, inv, i, c, max(d - 1, 0)), 0);
            brick = b * kDvrBrickQuads;
            wx = c.wx;
            wy = c.wy;
            wz = c.wz;
            if (flat) {
                flat_value = K.flat[b];
                count = i - look + 1;
            } else {
                at = brick + quad_offset(c.x & 7, c.y & 7, c.z & 7);
                qa = __ldg(K.quads + at);
                qb = __ldg(K.quads + at + 64);
            }
        }
        const float cwx = wx, cwy = wy, cwz = wz;
        const uint32_t cat = at;
        const LutCell h = lut_cell(flat ? flat_value : quad_trilinear(qa, qb, wx, wy, wz), n);
        if (!flat && i > look) {
            // the next sample's voxels are on their way while this one is summed
            const BrickCell c = brick_cell(B, r, V.step, (float)(i - 1));
            at = brick + quad_offset(c.x & 7, c.y & 7, c.z & 7);
            wx = c.wx;
            wy = c.wy;
            wz = c.wz;
            qa = __ldg(K.quads + at);
            qb = __ldg(K.quads + at + 64);
        }
        const float4 q = lut_value(L, D, h);
        const float d = 1.0f - q.w;
        const int ck = i & ~cmask;       // the last checkpoint at or before sample i
        if (ck > i - count) {
            T = wk[(size_t)(ck >> V.ckpt_shift) * npix + pix];
        } else if (d == 0.0f) {
            T = wk[(size_t)(ck >> V.ckpt_shift) * npix + pix];
            for (int j = ck; j < i; ++j) {
                BrickCell e = brick_cell(B, r, V.step, (float)j);
                const uint32_t b = brick_of(B, K, e);
                if (K.dist[b] != 0) continue;          // alpha 0
                const uint32_t qe = b * kDvrBrickQuads + quad_offset(e.x & 7, e.y & 7, e.z & 7);
                T *= 1.0f - lut_value(L, D, lut_cell(brick_trilinear(K.quads + qe, e), n)).w;
            }
        } else if (d != 1.0f) {
            T = T / d;
        }
        const float ta = T * q.w, p = gr * q.x + gg * q.y + gb * q.z;
        const float d_a = T * (p - U);
        U = q.w * p + d * U;
        // LUT sums
        int slot = h.k - wbase;
        if ((unsigned)slot >= (unsigned)WIN) {
            while (used) {
                const int u = __ffs(used) - 1;
                used &= used - 1u;
                bin_add(bins, n, wbase + u, gr, gg, gb, win[u * kBackThreads]);
                win[u * kBackThreads] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            wbase = max(h.k - WIN / 2, 0);
            slot = h.k - wbase;
        }
        used |= 1u << slot;
        {
            const float w1 = h.w, w0 = 1.0f - h.w, da = (float)count * d_a;
            float4 a = win[slot * kBackThreads];
            a.x += w0 * ta;
            a.y += w1 * ta;
            a.z += w0 * da;
            a.w += w1 * da;
            win[slot * kBackThreads] = a;
        }
        // voxel sums
        if (VOLGRAD && h.inside) {
            const float4 dd = D[h.k];
            const float ds = (float)n * (ta * (gr * dd.x + gg * dd.y + gb * dd.z) + d_a * dd.w);
            if (ds != 0.0f) {
                const float y0z0 = (1.0f - cwy) * (1.0f - cwz) * ds, y1z0 = cwy * (1.0f - cwz) * ds;
                const float y0z1 = (1.0f - cwy) * cwz * ds, y1z1 = cwy * cwz * ds;
                const float x0 = 1.0f - cwx, x1 = cwx;
                if (flat || !(fabsf(ds) <= FLT_MAX)) {
                    // not finite: to the voxels themselves, whatever the brick holds
                    const float v[8] = {x0 * y0z0, x1 * y0z0, x0 * y1z0, x1 * y1z0, x0 * y0z1, x1 * y0z1, x0 * y1z1, x1 * y1z1};
                    for (int j = i; j > i - count; --j) {
                        const BrickCell c = brick_cell(B, r, V.step, (float)j);
                        flush_vol(grad_vol, B, c.x - 1, c.y - 1, c.z - 1, v);
                    }
                } else {
                    if (cat != cell) {
                        flush_quads(K.gquads, cell, va);
                        cell = cat;
#pragma unroll
                        for (int k = 0; k < 8; ++k) va[k] = 0.0f;
                    }
                    va[0] += x0 * y0z0;
                    va[1] += x1 * y0z0;
                    va[2] += x0 * y1z0;
                    va[3] += x1 * y1z0;
                    va[4] += x0 * y0z1;
                    va[5] += x1 * y0z1;
                    va[6] += x0 * y1z1;
                    va[7] += x1 * y1z1;
                }
            }
        }
        i -= count;
    }
    if (VOLGRAD) flush_quads(K.gquads, cell, va);
    __syncwarp();
#pragma unroll 1
    for (int u = 0; u < WIN; ++u) {
        const bool has = (used >> u) & 1u;
        const float4 a = win[u * kBackThreads];
        const float4 a0 = make_float4(gr * a.x, gg * a.x, gb * a.x, a.z), a1 = make_float4(gr * a.y, gg * a.y, gb * a.y, a.w);
        flush_lut_warp(bins, n, has, wbase + u, a0, a1);
    }
    __syncthreads();
    for (int k = tid; k < 4 * n; k += kBackThreads) {
        const float v = bins[k];
        if (v != 0.0f) atomicAdd(&lut_sums[k], (double)v);
    }
}

// ---------------------------------------------------------------------------
// host side

// Checkpoint spacing of a view: 16 samples, doubled until at most 512
// checkpoints cover the longest ray (1.732 in the ray parameter).
static void view_layout(const mk_dvr_params &p, int &ckpt_shift, int &max_ckpt) {
    const int steps = (int)(1.74f / p.step) + 2;
    int sh = 4;
    while (((steps + (1 << sh) - 1) >> sh) > kDvrMaxCkpt) ++sh;
    ckpt_shift = sh;
    max_ckpt = (steps + (1 << sh) - 1) >> sh;
}

// Workspace floats of one view: max_ckpt checkpoint planes, a plane of sample
// counts and a plane of final transmittances.
static size_t view_floats(const mk_dvr_params &p) {
    int sh, mc;
    view_layout(p, sh, mc);
    return (size_t)(mc + 2) * p.width * p.height;
}

static int check_views(const mk_dvr_params *views, int nviews) {
    if (!views || nviews <= 0) {
        set_last_error("mk_dvr: no views");
        return MK_ERR_INVALID_ARGUMENT;
    }
    const mk_dvr_params &a = views[0];
    for (int i = 0; i < nviews; ++i) {
        const mk_dvr_params &p = views[i];
        if (p.width <= 0 || p.height <= 0 || p.width > 16384 || p.height > 16384 || p.dims[0] <= 0 ||
            p.dims[1] <= 0 || p.dims[2] <= 0 || p.lut_len < 2 || p.lut_len > kDvrMaxLut || !(p.step >= 1e-5f) ||
            !(p.scale > 0.0f) || !(p.t_min >= 0.0f)) {
            set_last_error("mk_dvr: bad view parameters (image size 1..16384, dims > 0, 2 <= lut_len <= 1024, "
                           "step >= 1e-5, scale > 0, t_min >= 0)");
            return MK_ERR_INVALID_ARGUMENT;
        }
        if ((double)p.dims[0] * p.dims[1] * p.dims[2] >= 2147483648.0) {
            set_last_error("mk_dvr: the volume must have fewer than 2^31 voxels");
            return MK_ERR_INVALID_ARGUMENT;
        }
        if (p.width != a.width || p.height != a.height || p.lut_len != a.lut_len || p.dims[0] != a.dims[0] ||
            p.dims[1] != a.dims[1] || p.dims[2] != a.dims[2]) {
            set_last_error("mk_dvr: the views of one call must share width, height, dims and lut_len");
            return MK_ERR_INVALID_ARGUMENT;
        }
    }
    return MK_OK;
}

static void fill_batch(const mk_dvr_params *views, int first, int count, size_t work_off0, DvrBatch &B) {
    memset(&B, 0, sizeof(B));
    const mk_dvr_params &a = views[first];
    B.W = a.width;
    B.H = a.height;
    B.lut_len = a.lut_len;
    for (int k = 0; k < 3; ++k) {
        B.dim[k] = a.dims[k];
        B.fdim[k] = (float)a.dims[k];
    }
    B.sxy = a.dims[0] * a.dims[1];
    size_t off = work_off0;
    for (int i = 0; i < count; ++i) {
        const mk_dvr_params &p = views[first + i];
        DvrView &V = B.v[i];
        for (int m = 0; m < 9; ++m) V.M[m] = p.transform[m];
        for (int k = 0; k < 3; ++k) V.mls[k] = p.max_len_spacing[k];
        V.scale = p.scale;
        V.xT = p.x_translate;
        V.yT = p.y_translate;
        V.step = p.step;
        V.t_min = p.t_min;
        view_layout(p, V.ckpt_shift, V.max_ckpt);
        V.work_off = off;
        off += view_floats(p);
    }
}

// Scratch of the bricked path: the bricks' quads (twice with voxel
// gradients), then flat values, LUT gradient sums, need bytes and the distance
// map and its intermediate.
struct BrickLayout {
    int nb[3];
    size_t n;                            // bricks
    size_t gquads, flat, lut, needed, tmp, dist, bytes;
};

static BrickLayout brick_layout(const int dims[3], bool gradients) {
    BrickLayout l;
    for (int k = 0; k < 3; ++k) l.nb[k] = dims[k] / 8 + 1;       // dims + 1 cells
    l.n = (size_t)l.nb[0] * l.nb[1] * l.nb[2];
    const size_t quads = l.n * kDvrBrickQuads * sizeof(float4), pad = (l.n + 255) & ~(size_t)255;
    l.gquads = quads;
    l.flat = quads * (gradients ? 2 : 1);
    l.lut = l.flat + 4 * pad;
    l.needed = l.lut + 4 * kDvrMaxLut * sizeof(double);
    l.tmp = l.needed + pad;
    l.dist = l.tmp + pad;
    l.bytes = l.dist + pad;
    return l;
}

// Whether these views gain from bricks, and may use them.  Measured at a
// quarter of a sample per voxel (one view of 128^2, 256^3, plain / bricks):
// forward 426 / 122 us where most is transparent, 426 / 377 us where all is
// visible; backward 1256 / 734 and 1369 / 1312 us.  At a sixteenth the visible
// case turns (backward 1245 / 1401 us).  Below about five million samples the
// rays must also be long for the shorter chain of a ray to outweigh three to
// six more launches (240 samples; a forward alone of 183x96x116 with rays of
// 220: 93 / 102 us, a training step of 40^3, 57: 236 / 296 us, of 128^3, 260:
// 640 / 460 us; eight 128^2 views of 64^3, six million samples: 644 / 473 us),
// and for the backward the LUT must have 64 entries: with a few, long runs in
// one LUT cell make the plain one cheap (16 entries, 249x73x51, rays of 250:
// 215 / 316 us a step).  With a long table few blocks fit an SM: above 750
// entries the backward needs four samples per voxel (800 entries, one view of
// 321x243 on 211x190x157, two per voxel: 1298 / 1443 us; 128^3, six: 1612 / 1304),
// and without voxel gradients, whose reductions make the plain kernel dear, above
// 512 long rays (600 entries, 64^3, rays of 107: 1323 / 1479 us).  The exit model
// of a ray (linear in the sample number) holds to a few hundredths of a cell
// while a unit of the ray parameter is at most 3e4 cells along an axis; quads
// are addressed with 32 bits.
constexpr double kDvrSamplesPerVoxel = 0.25;
constexpr double kDvrManySamples = 5.0e6;
constexpr double kDvrLongRay = 240.0;
constexpr int kDvrLongLut = 64;
constexpr int kDvrLutOnlyLut = 512;
constexpr double kDvrLongLutSamplesPerVoxel = 4.0;
constexpr double kDvrMaxCellsPerUnit = 3.0e4;

static bool use_bricks(const mk_dvr_params *views, int nviews, bool backward, bool gradients) {
    const mk_dvr_params &a = views[0];
    double samples = 0.0, depth = 0.0;
    for (int i = 0; i < nviews; ++i) {
        const mk_dvr_params &p = views[i];
        double across = 1.732;           // the longest way through the volume, in the ray parameter
        for (int k = 0; k < 3; ++k) {
            const double unit = fabs((double)p.transform[3 * k + 1] * p.scale * p.max_len_spacing[k]);
            if (!(unit * a.dims[k] <= kDvrMaxCellsPerUnit)) return false;
            if (unit > 0.0) across = fmin(across, 1.0 / unit);
        }
        // half of that for every pixel, and at most the box's volume in (u, v,
        // ray parameter) over that of a sample
        const float *m = p.transform;
        const double det = fabs((double)m[0] * ((double)m[4] * m[8] - (double)m[5] * m[7]) -
                                (double)m[1] * ((double)m[3] * m[8] - (double)m[5] * m[6]) +
                                (double)m[2] * ((double)m[3] * m[7] - (double)m[4] * m[6]));
        const double mls = fabs((double)p.max_len_spacing[0] * p.max_len_spacing[1] * p.max_len_spacing[2]);
        const double box = (double)p.height * p.height / (p.scale * det * mls);
        samples += fmin((double)p.width * p.height * 0.5 * across, box) / p.step;
        depth = fmax(depth, across / p.step);
    }
    for (int k = 0; k < 3; ++k)
        if (a.dims[k] > 4096) return false;
    const BrickLayout l = brick_layout(a.dims, false);
    if (l.nb[1] > 65535 || l.nb[2] > 65535 || l.n * kDvrBrickQuads >= 0xffffffffull) return false;
    if (samples < kDvrManySamples && (depth < kDvrLongRay || (backward && a.lut_len < kDvrLongLut))) return false;
    if (backward && !gradients && a.lut_len > kDvrLutOnlyLut && depth < kDvrLongRay) return false;
    const double per_voxel = backward && a.lut_len > kWinLongLut ? kDvrLongLutSamplesPerVoxel : kDvrSamplesPerVoxel;
    return samples >= per_voxel * a.dims[0] * a.dims[1] * (double)a.dims[2];
}

// Build the bricks of `volume` under `lut` in `scratch`, and their distances.
template <bool BACKWARD>
static int build_bricks(const mk_dvr_params &p, const float *volume, const float *lut, void *scratch, bool gradients,
                        DvrBricks &K, cudaStream_t s) {
    const BrickLayout l = brick_layout(p.dims, gradients);
    char *base = static_cast<char *>(scratch);
    float4 *quads = reinterpret_cast<float4 *>(base);
    float4 *gquads = gradients ? reinterpret_cast<float4 *>(base + l.gquads) : nullptr;
    float *flat = reinterpret_cast<float *>(base + l.flat);
    uint8_t *needed = reinterpret_cast<uint8_t *>(base + l.needed);
    uint8_t *dist = reinterpret_cast<uint8_t *>(base + l.dist);
    k_dvr_build<BACKWARD><<<dim3((l.nb[0] + 3) / 4, l.nb[1], l.nb[2]), 256, 0, s>>>(
        p.dims[0], p.dims[1], p.dims[2], l.nb[0], volume, reinterpret_cast<const float4 *>(lut), p.lut_len, quads, gquads, needed,
        flat, reinterpret_cast<double *>(base + l.lut));
    MK_CUDA_TRY(cudaGetLastError());
    for (int k = 0; k < 3; ++k) K.nb[k] = l.nb[k];
    K.quads = quads;
    K.gquads = gquads;
    K.dist = dist;
    K.flat = flat;
    return launch_brick_distance(needed, l.nb[0], l.nb[1], l.nb[2], false, reinterpret_cast<uint8_t *>(base + l.tmp), dist, s);
}

// Blocks of `threads` threads over the views of a batch (dvr_pixel).
static unsigned dvr_blocks(const DvrBatch &B, int views, int threads) {
    const unsigned h = threads / 16;
    return ((B.W + 15) / 16) * ((B.H + h - 1) / h) * (unsigned)views;
}

// Samples whose loads a ray has in flight: four where the launch is too small to
// fill the SMs and the longest rays set its time, two where there are rays enough
// (four cost registers, and so resident warps).  One to 32 views of 128^2 to 700^2
// on three volumes, mostly transparent and all visible: up to 130,000 rays four
// take 1-18% less (one view of 321x243: 107 us, against 118 with two and 150 with
// one), from 150,000 on the two are level within 5%, either way by volume and
// table, with two ahead by more in the largest launches (eight views of 256^2 on
// 256^3: 638 us, against 670 and 686 with one).  The line is in that level stretch.
constexpr long long kDvrManyRays = 300000;

static void launch_forward_bricks(const DvrBatch &B, const DvrBricks &K, int views, bool drift, const float4 *lut,
                                  float *images, float *trans, float *work, size_t smem, cudaStream_t s) {
    const bool many = (long long)B.W * B.H * views >= kDvrManyRays;
    auto kern = many ? (drift ? k_dvr_forward_bricks<2, true> : k_dvr_forward_bricks<2, false>)
                     : (drift ? k_dvr_forward_bricks<4, true> : k_dvr_forward_bricks<4, false>);
    kern<<<dvr_blocks(B, views, kForwardThreads), kForwardThreads, smem, s>>>(B, K, views, lut, images, trans, work);
}

static decltype(&k_dvr_backward_bricks<true, true, kWinLong>) backward_bricks(bool volgrad, bool drift, bool wide) {
    if (volgrad) {
        if (drift) return wide ? k_dvr_backward_bricks<true, true, kWinLong> : k_dvr_backward_bricks<true, true, kWinShort>;
        return wide ? k_dvr_backward_bricks<true, false, kWinLong> : k_dvr_backward_bricks<true, false, kWinShort>;
    }
    if (drift) return wide ? k_dvr_backward_bricks<false, true, kWinLong> : k_dvr_backward_bricks<false, true, kWinShort>;
    return wide ? k_dvr_backward_bricks<false, false, kWinLong> : k_dvr_backward_bricks<false, false, kWinShort>;
}

// Whether rays of these views drift along an axis (samples_inside): a launch of
// its own, so that other views do not pay for the look at each run's end
// (one view of 321x243: 148 -> 150 us).
static bool views_drift(const mk_dvr_params *views, int nviews) {
    for (int i = 0; i < nviews; ++i) {
        const mk_dvr_params &p = views[i];
        for (int k = 0; k < 3; ++k) {
            const float d = p.transform[3 * k + 1] * p.scale * p.max_len_spacing[k];
            if (d != 0.0f && !(fabsf(d * p.step * (float)p.dims[k]) >= 2.0f * kDvrSlow)) return true;
        }
    }
    return false;
}

// Scratch the caller gave, if it is enough and aligned for these views.
static bool bricks_fit(const mk_dvr_params *views, int nviews, bool backward, bool gradients, const void *scratch,
                       size_t bytes) {
    return scratch && (reinterpret_cast<uintptr_t>(scratch) & 255) == 0 && use_bricks(views, nviews, backward, gradients) &&
           bytes >= brick_layout(views[0].dims, gradients).bytes;
}

}  // namespace mk

using namespace mk;

extern "C" int mk_dvr_workspace_floats(const mk_dvr_params *views, int nviews, size_t *floats) {
    if (!floats) {
        set_last_error("mk_dvr_workspace_floats: null argument");
        return MK_ERR_INVALID_ARGUMENT;
    }
    int rc = check_views(views, nviews);
    if (rc != MK_OK) return rc;
    size_t total = 0;
    for (int i = 0; i < nviews; ++i) total += view_floats(views[i]);
    *floats = total;
    return MK_OK;
}

extern "C" int mk_dvr_scratch_bytes(const mk_dvr_params *views, int nviews, int gradients, size_t *bytes) {
    if (!bytes) {
        set_last_error("mk_dvr_scratch_bytes: null argument");
        return MK_ERR_INVALID_ARGUMENT;
    }
    int rc = check_views(views, nviews);
    if (rc != MK_OK) return rc;
    const bool backward = gradients != 0, volgrad = backward && gradients != 2;
    *bytes = use_bricks(views, nviews, backward, volgrad) ? brick_layout(views[0].dims, volgrad).bytes : 0;
    return MK_OK;
}

extern "C" int mk_dvr_forward_scratch(const mk_dvr_params *views, int nviews, const float *volume, const float *lut,
                                      float *images, float *transmittance, float *workspace, void *scratch,
                                      size_t scratch_bytes, void *stream) {
    if (!volume || !lut || !images || !transmittance) {
        set_last_error("mk_dvr_forward: null argument");
        return MK_ERR_INVALID_ARGUMENT;
    }
    int rc = check_views(views, nviews);
    if (rc != MK_OK) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t npix = (size_t)views[0].width * views[0].height;
    const size_t smem = 2 * (size_t)views[0].lut_len * sizeof(float4);
    const bool bricks = bricks_fit(views, nviews, false, false, scratch, scratch_bytes);
    const bool drift = bricks && views_drift(views, nviews);
    DvrBricks K = {};
    if (bricks) {
        rc = build_bricks<false>(views[0], volume, lut, scratch, false, K, s);
        if (rc != MK_OK) return rc;
    } else {
        MK_CUDA_TRY(cudaFuncSetAttribute(k_dvr_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    }
    size_t off = 0;
    DvrBatch B;
    for (int first = 0; first < nviews; first += kDvrViewsPerLaunch) {
        const int count = min(kDvrViewsPerLaunch, nviews - first);
        fill_batch(views, first, count, off, B);
        for (int i = 0; i < count; ++i) off += view_floats(views[first + i]);
        dim3 grid((B.W + 31) / 32, (B.H + 7) / 8, count);
        const float4 *l4 = reinterpret_cast<const float4 *>(lut);
        float *im = images + (size_t)first * npix * 3, *tr = transmittance + (size_t)first * npix;
        if (bricks) launch_forward_bricks(B, K, count, drift, l4, im, tr, workspace, smem, s);
        else k_dvr_forward<<<grid, 256, smem, s>>>(B, volume, l4, im, tr, workspace);
        MK_CUDA_TRY(cudaGetLastError());
    }
    return MK_OK;
}

extern "C" int mk_dvr_forward(const mk_dvr_params *views, int nviews, const float *volume, const float *lut,
                              float *images, float *transmittance, float *workspace, void *stream) {
    return mk_dvr_forward_scratch(views, nviews, volume, lut, images, transmittance, workspace, nullptr, 0, stream);
}

extern "C" int mk_dvr_backward_scratch(const mk_dvr_params *views, int nviews, const float *volume, const float *lut,
                                       const float *workspace, const float *grad_images, float *grad_lut,
                                       float *grad_volume, void *scratch, size_t scratch_bytes, void *stream) {
    if (!volume || !lut || !workspace || !grad_images || !grad_lut) {
        set_last_error("mk_dvr_backward: null argument");
        return MK_ERR_INVALID_ARGUMENT;
    }
    int rc = check_views(views, nviews);
    if (rc != MK_OK) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t npix = (size_t)views[0].width * views[0].height;
    const bool bricks = bricks_fit(views, nviews, true, grad_volume != nullptr, scratch, scratch_bytes);
    const int win = window_cells(views[0].lut_len);
    const size_t smem = 3 * (size_t)views[0].lut_len * sizeof(float4), smem_b = smem + win * kBackThreads * sizeof(float4);
    DvrBricks K = {};
    double *lut_sums = nullptr;
    auto kern = grad_volume ? k_dvr_backward<true, false> : k_dvr_backward<false, false>;
    auto kern_odd = grad_volume ? k_dvr_backward<true, true> : k_dvr_backward<false, true>;
    const bool drift = bricks && views_drift(views, nviews);
    auto kern_b = backward_bricks(grad_volume != nullptr, drift, win == kWinLong);
    if (bricks) {
        MK_CUDA_TRY(cudaFuncSetAttribute(kern_b, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_b));
        MK_CUDA_TRY(cudaFuncSetAttribute(kern_odd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        lut_sums = reinterpret_cast<double *>(static_cast<char *>(scratch) + brick_layout(views[0].dims, grad_volume != nullptr).lut);
        rc = build_bricks<true>(views[0], volume, lut, scratch, grad_volume != nullptr, K, s);
        if (rc != MK_OK) return rc;
    } else {
        MK_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    }
    size_t off = 0;
    DvrBatch B;
    for (int first = 0; first < nviews; first += kDvrViewsPerLaunch) {
        const int count = min(kDvrViewsPerLaunch, nviews - first);
        fill_batch(views, first, count, off, B);
        for (int i = 0; i < count; ++i) off += view_floats(views[first + i]);
        dim3 grid((B.W + 15) / 16, (B.H + 7) / 8, count);
        const float4 *l4 = reinterpret_cast<const float4 *>(lut);
        const float *gi = grad_images + (size_t)first * npix * 3;
        if (bricks) {
            kern_b<<<dvr_blocks(B, count, kBackThreads), kBackThreads, smem_b, s>>>(B, K, count, l4, workspace, gi, lut_sums,
                                                                                  grad_volume);
            MK_CUDA_TRY(cudaGetLastError());
            kern_odd<<<grid, 128, smem, s>>>(B, volume, l4, workspace, gi, grad_lut, grad_volume);
        } else {
            kern<<<grid, 128, smem, s>>>(B, volume, l4, workspace, gi, grad_lut, grad_volume);
        }
        MK_CUDA_TRY(cudaGetLastError());
    }
    if (bricks && !grad_volume) {
        k_dvr_lut_add<<<1, 256, 0, s>>>(4 * views[0].lut_len, lut_sums, grad_lut);
        MK_CUDA_TRY(cudaGetLastError());
    }
    if (bricks && grad_volume) {
        const mk_dvr_params &p = views[0];
        const BrickLayout l = brick_layout(p.dims, true);
        k_dvr_fold<<<dim3(l.nb[0], l.nb[1], l.nb[2]), 256, 0, s>>>(
            p.dims[0], p.dims[1], p.dims[2], K.gquads, reinterpret_cast<const uint8_t *>(scratch) + l.needed, grad_volume,
            4 * p.lut_len, lut_sums, grad_lut);
        MK_CUDA_TRY(cudaGetLastError());
    }
    return MK_OK;
}

extern "C" int mk_dvr_backward(const mk_dvr_params *views, int nviews, const float *volume, const float *lut,
                               const float *workspace, const float *grad_images, float *grad_lut,
                               float *grad_volume, void *stream) {
    return mk_dvr_backward_scratch(views, nviews, volume, lut, workspace, grad_images, grad_lut, grad_volume, nullptr, 0,
                                   stream);
}
