// tri_inverse.cuh — inverses of small FP64 triangles in shared memory, from 16 x 16
// blocks: 64 x 64 by a CTA of 256 threads (the diagonal blocks of the blocked DTRSV
// and DTRSM), 32 x 32 by 128 (those of the triangular inverse).
#pragma once

#include <cuda_runtime.h>

namespace gbx_tri {

constexpr int NB = 64, LD = NB + 1;

// Element (i, k) of all blocks at [k * LD + i]; o: the block's first row and column.
// X = inverse of the 16 x 16 block of D at o, by one warp: substitution, lane =
// column j, rows r = 2 u + part.
template <int LD>
__device__ __forceinline__ void invert16(const double *D, double *X, int o)
{
    const int lane = threadIdx.x & 31, j = lane & 15, part = lane >> 4;
    const double rd = 1.0 / D[(o + j) * LD + o + j];
    const double *d = D + o * LD + o + part;
    double s[8];
#pragma unroll
    for (int u = 0; u < 8; u++) s[u] = (2 * u + part == j) ? 1.0 : 0.0;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const double ri = __shfl_sync(0xffffffffu, rd, i);
        const double w = __shfl_sync(0xffffffffu, s[i >> 1] * ri, j + 16 * (i & 1));
        if (part == (i & 1)) X[(o + j) * LD + o + i] = w;
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (2 * u + 1 > i && 2 * u + part > i) s[u] = fma(-d[i * LD + 2 * u], w, s[u]);
    }
}

// The 32 x 32 block at o from its two inverted 16 x 16 ones, by four warps (t =
// 0 .. 127, two elements each): W = D21 X11, then, after a barrier, X21 = -X22 W
// and X12 = 0.  W: 16 x 17 of scratch.
template <int LD>
__device__ __forceinline__ void join32_w(const double *D, const double *X, double *W, int o, int t)
{
    const int v = t & 15, g = t >> 4;
#pragma unroll
    for (int u = 0; u < 2; u++) {   // row v, column j
        const int j = g + 8 * u;
        double w = 0.0;
#pragma unroll 4
        for (int k = j; k < 16; k++) w = fma(D[(o + k) * LD + o + 16 + v], X[(o + j) * LD + o + k], w);
        W[j * 17 + v] = w;
    }
}
template <int LD>
__device__ __forceinline__ void join32_x(double *X, const double *W, int o, int t)
{
    const int v = t & 15, g = t >> 4;
#pragma unroll
    for (int u = 0; u < 2; u++) {   // row i, column v
        const int i = g + 8 * u;
        double w = 0.0;
#pragma unroll 4
        for (int k = 0; k <= i; k++) w = fma(-X[(o + 16 + k) * LD + o + 16 + i], W[v * 17 + k], w);
        X[(o + v) * LD + o + 16 + i] = w;
        X[(o + 16 + v) * LD + o + i] = 0.0;
    }
}

// X = inverse of the lower triangular 64 x 64 block D (W: 32 x 33 scratch), by
// the whole CTA: the four 16 x 16 diagonal blocks, a warp each, then
// X21 = -X22 (D21 X11) for the two 32 x 32 blocks and for the whole.
// What bounds it: the FP64 pipe, which an instruction of a warp holds 16 to 19
// cycles whatever its predicate, so the loops skip the zero parts by warp: the
// two products of the whole take 20k cycles.  Substitution on 32 x 32
// blocks by four warps each, with a barrier per row, took 5 us more.
__device__ __forceinline__ void invert64(const double *D, double *X, double *W)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < 4) invert16<LD>(D, X, 16 * warp);
    __syncthreads();
    const int half = warp >> 2;
    join32_w<LD>(D, X, W + 16 * 17 * half, 32 * half, threadIdx.x & 127);
    __syncthreads();
    join32_x<LD>(X, W + 16 * 17 * half, 32 * half, threadIdx.x & 127);
    __syncthreads();
    // W = D21 X11, lane = row, this warp's columns j = warp + 8 u
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const int j = warp + 8 * u;
        double v = 0.0;
#pragma unroll 4
        for (int k = j; k < 32; k++) v = fma(D[k * LD + 32 + lane], X[j * LD + k], v);
        W[j * 33 + lane] = v;
    }
    __syncthreads();
    // X21 = -X22 W, lane = column, this warp's rows i = warp + 8 u; X12 = 0
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const int i = warp + 8 * u;
        double v = 0.0;
#pragma unroll 4
        for (int k = 0; k <= i; k++) v = fma(-X[(32 + k) * LD + 32 + i], W[lane * 33 + k], v);
        X[lane * LD + 32 + i] = v;
        X[(32 + lane) * LD + i] = 0.0;
    }
    __syncthreads();
}

}  // namespace gbx_tri
