// mk_brickdist.cu -- distance maps over bricks: how far a ray may go before it
// can meet a brick that matters.
//
// From one byte per brick (0: empty) the map holds, per brick, the Chebyshev
// distance in bricks to the nearest brick that is not empty, capped at
// kMaxBrickDist: 0 for a brick that is not empty itself, d > 0 where all
// bricks within d - 1 along every axis are empty.  A ray in such a brick may
// leave the whole cube of 2 d - 1 bricks in one step; with a bit per brick it
// stopped at every brick face.  Bricks outside the grid count as empty.
#include <cuda_runtime.h>
#include <stdint.h>

#include "mk_internal.h"

namespace mk {

namespace {

// Smallest distance along a line of n bytes (stride apart) at position i to a
// value v: min over k of max(|k|, v at i + k).
__device__ __forceinline__ int line_distance(const uint8_t *v, int stride, int i, int n) {
    int best = v[0];
#pragma unroll
    for (int k = 1; k < kMaxBrickDist; ++k) {
        int m = kMaxBrickDist;
        if (i - k >= 0) m = v[-k * stride];
        if (i + k < n) m = min(m, (int)v[k * stride]);
        best = min(best, max(m, k));
    }
    return best;
}

// x and y of one z slice per block, in shared memory (the maximum distance is
// separable); latency-bound, a few microseconds.  A block has read its slice
// before it writes it, so out may be occupied.
__global__ void __launch_bounds__(1024) k_brick_distance_xy(const uint8_t *occupied, int nbx, int nby, uint8_t *out) {
    extern __shared__ uint8_t smem[];
    const int n = nbx * nby;
    uint8_t *a = smem, *b = smem + n;
    const size_t off = (size_t)blockIdx.x * n;
    for (int i = threadIdx.x; i < n; i += blockDim.x) a[i] = occupied[off + i] ? 0 : kMaxBrickDist;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) b[i] = (uint8_t)line_distance(a + i, 1, i % nbx, nbx);
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) out[off + i] = (uint8_t)line_distance(b + i, nbx, i / nbx, nby);
}

__global__ void __launch_bounds__(256) k_brick_distance_z(const uint8_t *__restrict__ in, int nxy, int nbz,
                                                          uint8_t *__restrict__ dist) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)nxy * nbz) return;
    dist[i] = (uint8_t)line_distance(in + i, nxy, (int)(i / nxy), nbz);
}

// Small grids, all three axes in one block (one launch less: 2.5 us).
constexpr int kOneBlockBricks = 8192;
__global__ void __launch_bounds__(1024) k_brick_distance_small(const uint8_t *occupied, int nbx, int nby, int nbz,
                                                               uint8_t *dist) {
    __shared__ uint8_t a[kOneBlockBricks], b[kOneBlockBricks];
    const int nxy = nbx * nby, n = nxy * nbz;
    for (int i = threadIdx.x; i < n; i += blockDim.x) a[i] = occupied[i] ? 0 : kMaxBrickDist;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) b[i] = (uint8_t)line_distance(a + i, 1, i % nbx, nbx);
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) a[i] = (uint8_t)line_distance(b + i, nbx, i / nbx % nby, nby);
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x) dist[i] = (uint8_t)line_distance(a + i, nxy, i / nxy, nbz);
}

// Every empty brick is its own step (also for slices too large for shared
// memory).
__global__ void __launch_bounds__(256) k_brick_distance_one(const uint8_t *occupied, size_t n, uint8_t *dist) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dist[i] = occupied[i] ? 0 : 1;
}

constexpr size_t kMaxSliceSmem = 200 * 1024;

}  // namespace

int launch_brick_distance(const uint8_t *occupied, int nbx, int nby, int nbz, bool one, uint8_t *tmp, uint8_t *dist,
                          cudaStream_t s) {
    const size_t nxy = (size_t)nbx * nby, n = nxy * nbz;
    const unsigned blocks = (unsigned)((n + 255) / 256);
    if (one || 2 * nxy > kMaxSliceSmem) {
        k_brick_distance_one<<<blocks, 256, 0, s>>>(occupied, n, dist);
    } else if (n <= kOneBlockBricks) {
        k_brick_distance_small<<<1, 1024, 0, s>>>(occupied, nbx, nby, nbz, dist);
    } else {
        if (2 * nxy > 48 * 1024)
            MK_CUDA_TRY(cudaFuncSetAttribute(k_brick_distance_xy, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)kMaxSliceSmem));
        k_brick_distance_xy<<<nbz, 1024, 2 * nxy, s>>>(occupied, nbx, nby, tmp);
        MK_CUDA_TRY(cudaGetLastError());
        k_brick_distance_z<<<blocks, 256, 0, s>>>(tmp, (int)nxy, nbz, dist);
    }
    MK_CUDA_TRY(cudaGetLastError());
    return MK_OK;
}

}  // namespace mk
