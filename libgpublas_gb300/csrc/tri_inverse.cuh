// tri_inverse.cuh — inverse of a 64 x 64 FP64 triangle in shared memory by one
// CTA of 256 threads: the diagonal blocks of the blocked DTRSV and DTRSM.
#pragma once

#include <cuda_runtime.h>

namespace gbx_tri {

constexpr int NB = 64, LD = NB + 1;   // element (row i, column k) at [k * LD + i]

// X = inverse of the lower triangular 64 x 64 block D (D[k * 65 + i] is row i,
// column k; the same layout for X; W: 32 x 33 scratch), by the whole CTA: the
// four 16 x 16 diagonal blocks by substitution, a warp each, then
// X21 = -X22 (D21 X11) for the two 32 x 32 blocks and for the whole.
// What bounds it: the FP64 pipe, which an instruction of a warp holds 16 to 19
// cycles whatever its predicate, so the loops skip the zero parts by warp: the
// two products of the whole take 20k cycles.  Substitution on 32 x 32
// blocks by four warps each, with a barrier per row, took 5 us more.
__device__ __forceinline__ void invert64(const double *D, double *X, double *W)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < 4) {   // lane = column j, rows r = 2 u + part
        const int o = 16 * warp, j = lane & 15, part = lane >> 4;
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
    __syncthreads();
    {   // 32 x 32 blocks, four warps each; this thread: two columns of one row, or two rows of one column
        const int o = 32 * (warp >> 2), v = lane & 15, g = 2 * (warp & 3) + (lane >> 4);
        double *Wb = W + 16 * 17 * (warp >> 2);
#pragma unroll
        for (int u = 0; u < 2; u++) {   // W = D21 X11: row v, column j
            const int j = g + 8 * u;
            double w = 0.0;
#pragma unroll 4
            for (int k = j; k < 16; k++) w = fma(D[(o + k) * LD + o + 16 + v], X[(o + j) * LD + o + k], w);
            Wb[j * 17 + v] = w;
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 2; u++) {   // X21 = -X22 W: row i, column v; X12 = 0
            const int i = g + 8 * u;
            double w = 0.0;
#pragma unroll 4
            for (int k = 0; k <= i; k++) w = fma(-X[(o + 16 + k) * LD + o + 16 + i], Wb[v * 17 + k], w);
            X[(o + v) * LD + o + 16 + i] = w;
            X[(o + 16 + v) * LD + o + i] = 0.0;
        }
    }
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
