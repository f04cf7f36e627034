// grouped_dev.cuh — device code shared by the grouped kernel (batched.cu)
// and the serving loop's persistent kernel (serve_loop.cu): the operation
// descriptor and the small triangular solve.
#pragma once

#include "tri_inverse.cuh"

#include <cuda_runtime.h>

namespace gbx_grouped {

struct DevOp {
    int kind;                     // GBX_OP_GEMM / GBX_OP_TRSM
    int ta, tb;                   // GEMM transpositions; TRSM: ta = op(A) transposed
    int lower, unit, left;        // TRSM: effective triangle of the solved matrix, diag, side
    int m, n, k;
    double alpha, beta;
    const double *A;
    long long lda;
    const double *B;
    long long ldb;
    double *C;
    long long ldc;
};

// ---------------------------------------------------------------- TRSM item
// Solves T y = alpha*b for up to NSYS systems of order n (<= 256), where
// for side 'L' T = op(A) and the systems are columns of B (m x nrhs), and for
// side 'R' T = op(A)^T and the systems are rows of B.  Blocks of 16 rows in solve
// order (the effective triangle of T): the block's solution is its inverted
// diagonal block times its right-hand sides, then every later row subtracts its
// 16 products; warp 0 inverts the next diagonal block meanwhile (T only).
// What bounds it: the FP64 pipe, n^2 / 2 FMAs per system, and the chain of
// n / 16 inversions.  Row by row, with a division and two barriers each, small
// plans waited for their longest solve: 324 DGEMMs and 80 DTRSMs took 1.42 ms,
// now 0.92.
constexpr int TRSM_BLK = 16, TRSM_LD = TRSM_BLK + 1;
// doubles of shared memory for systems of order n at most
constexpr int trsm_smem(int n, int nsys) { return n * nsys + 3 * TRSM_BLK * TRSM_LD; }

template <int NSYS, int NTHREADS>
__device__ void trsm_item(const DevOp &o, int sys0, double *smem)
{
    static_assert(NSYS == 16 && NTHREADS == 256, "one thread per element of a block's solution");
    const int n = o.left ? o.m : o.n;                 // order of T
    const int nsys_total = o.left ? o.n : o.m;
    const int nsys = min(NSYS, nsys_total - sys0);
    double *D = smem;                                  // a diagonal block, [k * 17 + i]
    double *inv = D + TRSM_BLK * TRSM_LD;              // two inverses
    double *X = inv + 2 * TRSM_BLK * TRSM_LD;          // X[p * NSYS + s], p in solve order
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, s = threadIdx.x % NSYS;
    // row of position p in solve order
    auto g = [&](int p) { return o.lower ? p : n - 1 - p; };
    // element (i, s) of system vector s
    auto bidx = [&](int i, int s) -> long long {
        return o.left ? (long long)(sys0 + s) * o.ldc + i : (long long)i * o.ldc + (sys0 + s);
    };
    // T at positions p, q: side L: op(A)(i,j); side R: op(A)(j,i)
    auto T = [&](int p, int q) -> double {
        int r = g(p), c = g(q);
        if (!o.left) { const int t = r; r = c; c = t; }
        return o.ta ? o.A[(long long)r * o.lda + c] : o.A[(long long)c * o.lda + r];
    };
    auto invert = [&](int b) {
        const int p0 = b * TRSM_BLK;
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {   // identity beyond n
            const int i = (lane + 32 * u) % TRSM_BLK, k = (lane + 32 * u) / TRSM_BLK;
            v[u] = i == k ? 1.0 : 0.0;
            if (p0 + i < n && k <= i && !(o.unit && i == k)) v[u] = T(p0 + i, p0 + k);
        }
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int i = (lane + 32 * u) % TRSM_BLK, k = (lane + 32 * u) / TRSM_BLK;
            D[k * TRSM_LD + i] = v[u];
        }
        __syncwarp();
        gbx_tri::invert16<TRSM_LD>(D, inv + (b & 1) * TRSM_BLK * TRSM_LD, 0);
        __syncwarp();
    };
    for (int t = threadIdx.x; t < n * NSYS; t += NTHREADS) {
        const int p = t / NSYS;
        X[t] = s < nsys ? o.alpha * o.C[bidx(g(p), s)] : 0.0;
    }
    if (warp == 0) invert(0);
    __syncthreads();
    const int nb = (n + TRSM_BLK - 1) / TRSM_BLK;
    for (int b = 0; b < nb; b++) {
        const int p0 = b * TRSM_BLK, i = threadIdx.x / NSYS;
        const double *c = inv + (b & 1) * TRSM_BLK * TRSM_LD + i;
        double x = 0.0;
        if (p0 + i < n) {
#pragma unroll
            for (int k = 0; k < TRSM_BLK; k++)
                if (k <= i) x = fma(c[k * TRSM_LD], X[(p0 + k) * NSYS + s], x);
        }
        __syncthreads();
        if (p0 + i < n) X[(p0 + i) * NSYS + s] = x;
        __syncthreads();
        if (b + 1 == nb) break;
        if (warp == 0) {
            invert(b + 1);
        } else {
            const double *xb = X + p0 * NSYS + s;
            for (int p = p0 + TRSM_BLK + (threadIdx.x - 32) / NSYS; p < n; p += (NTHREADS - 32) / NSYS) {
                double acc = X[p * NSYS + s];
#pragma unroll 1
                for (int k0 = 0; k0 < TRSM_BLK; k0 += 8) {
                    double tk[8];
#pragma unroll
                    for (int k = 0; k < 8; k++) tk[k] = T(p, p0 + k0 + k);
#pragma unroll
                    for (int k = 0; k < 8; k++) acc = fma(-tk[k], xb[(k0 + k) * NSYS], acc);
                }
                X[p * NSYS + s] = acc;
            }
        }
        __syncthreads();
    }
    for (int t = threadIdx.x; t < n * NSYS; t += NTHREADS)
        if (s < nsys) o.C[bidx(g(t / NSYS), s)] = X[t];
}

}  // namespace gbx_grouped
