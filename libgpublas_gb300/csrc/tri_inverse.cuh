// tri_inverse.cuh — inverse of a 64 x 64 FP64 triangle in shared memory by one
// CTA of 256 threads: the diagonal blocks of the blocked DTRSV and DTRSM.
#pragma once

#include <cuda_runtime.h>

namespace gbx_tri {

constexpr int NB = 64, LD = NB + 1;   // element (row i, column k) at [k * LD + i]

// X = inverse of the lower triangular 64 x 64 block D (D[k * 65 + i] is row i,
// column k; the same layout for X; W: 32 x 33 scratch), by the whole CTA:
// the two 32 x 32 diagonal blocks by substitution, lane j owning column j
// and four warps sharing a block's rows, then X21 = -X22 (D21 X11).  An FP64
// warp instruction holds the SM's pipe 16 to 19 cycles whatever its predicate,
// so the loops skip the zero parts by warp.
__device__ __forceinline__ void invert64(const double *D, double *X, double *W)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int b = warp >> 2, part = warp & 3, o = 32 * b;   // diagonal block, rows r = 4 u + part
    const double rd = 1.0 / D[(o + lane) * LD + o + lane];   // lane i: 1 / D_ii of this warp's block
    double s[8];
#pragma unroll
    for (int u = 0; u < 8; u++) s[u] = (4 * u + part == lane) ? 1.0 : 0.0;
#pragma unroll
    for (int i = 0; i < 32; i++) {
        const double ri = __shfl_sync(0xffffffffu, rd, i);
        if ((i & 3) == part) X[(o + lane) * LD + o + i] = s[i >> 2] * ri;
        asm volatile("bar.sync %0, 128;" :: "r"(1 + b) : "memory");
        const double w = X[(o + lane) * LD + o + i];
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (4 * u + 3 > i && 4 * u + part > i) s[u] = fma(-D[(o + i) * LD + o + 4 * u + part], w, s[u]);
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
