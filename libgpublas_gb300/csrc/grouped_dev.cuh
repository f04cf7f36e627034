// grouped_dev.cuh — device code shared by the grouped kernel (batched.cu)
// and the serving loop's persistent kernel (serve_loop.cu): the operation
// descriptor and the small triangular solve.
#pragma once

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
// side 'R' T = op(A)^T and the systems are rows of B.  Substitution in solve order
// (the effective triangle of T), every element's products subtracted one by one in
// increasing order: the solution of a row-by-row substitution, backward stable
// however ill-conditioned T is.  (With inverted 16 x 16 diagonal blocks the
// componentwise backward error at a block condition of 4e8 was 1.7e-11.)
// Blocks of 16 rows: two warps solve a block, eight systems each, while the others
// subtract the block before from the rows after the next one, and one of them
// fetches what the next block needs; then all subtract the block from the next.
// What bounds it: the FP64 pipe, n^2 / 2 FMAs per system, and the chain over the
// rows, five FP64 instructions each (65 cycles).
constexpr int TRSM_BLK = 16, TRSM_LD = TRSM_BLK + 1;
// doubles of shared memory for systems of order n at most
constexpr int trsm_smem(int n, int nsys) { return n * nsys + 3 * TRSM_BLK * TRSM_LD; }

static __device__ __noinline__ double trsm_ratio(double a, double d) { return a / d; }

// v / d with r = 1 / d (0: d is zero, not finite or far from 1): the quotient
// v r and one correction by its residual, which an FMA gives exactly (Markstein,
// IBM J. Res. Dev. 34(1), 1990): the rounded quotient, three dependent operations
// instead of a division's dozen.  A v outside the range where neither quotient
// nor residual can leave the normal numbers is divided.  live: the lane's
// result matters; by whole warps.
__device__ __forceinline__ double trsm_quotient(double v, double d, double r, bool live)
{
    const unsigned e = (unsigned)__double2hiint(v) >> 20 & 0x7ffu;
    const bool zero = (__double_as_longlong(v) << 1) == 0;
    const double q = v * r;
    double x = fma(fma(-d, q, v), r, q);
    if (zero) x = q;   // with its sign
    const bool rare = r == 0.0 || (!zero && e - 523u > 1000u);
    if (__any_sync(0xffffffffu, live && rare)) {
        if (live && rare) x = trsm_ratio(v, d);
    }
    return x;
}

template <int NSYS, int NTHREADS>
__device__ void trsm_item(const DevOp &o, int sys0, double *smem)
{
    static_assert(NSYS == 16 && NTHREADS == 256, "one thread per element of a block");
    constexpr int BLK = TRSM_BLK, LD = TRSM_LD;
    const int n = o.left ? o.m : o.n;                 // order of T
    const int nsys_total = o.left ? o.n : o.m;
    const int nsys = min(NSYS, nsys_total - sys0);
    double *D = smem;                  // two diagonal blocks, element (i, k) at [k * 17 + i], 1 / d_k at [k * 17 + 16]
    double *E = D + 2 * BLK * LD;      // the rows of the next block, columns of this one
    double *X = E + BLK * LD;          // X[p * NSYS + s], p in solve order
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
    // diagonal block b (identity beyond n) and, if it is not the first, its rows'
    // columns of the block before; by one warp
    auto fetch = [&](int b) {
        const int p0 = b * BLK, i = lane % BLK, k0 = lane / BLK;
        double *d = D + (b & 1) * BLK * LD;
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int k = k0 + 2 * u;
            v[u] = i == k ? 1.0 : 0.0;
            if (p0 + i < n && k <= i && !(o.unit && i == k)) v[u] = T(p0 + i, p0 + k);
        }
#pragma unroll
        for (int u = 0; u < 8; u++) d[(k0 + 2 * u) * LD + i] = v[u];
        if (b > 0) {
#pragma unroll
            for (int u = 0; u < 8; u++) v[u] = p0 + i < n ? T(p0 + i, p0 - BLK + k0 + 2 * u) : 0.0;
#pragma unroll
            for (int u = 0; u < 8; u++) E[(k0 + 2 * u) * LD + i] = v[u];
        }
        __syncwarp();
        if (!o.unit) {
            const double p = d[i * LD + i];
            const unsigned e = (unsigned)__double2hiint(p) >> 20 & 0x7ffu;
            const double r = e - 623u <= 800u ? 1.0 / p : 0.0;
            if (lane < BLK) d[i * LD + BLK] = r;
        }
    };
    for (int t = threadIdx.x; t < n * NSYS; t += NTHREADS) {
        const int p = t / NSYS;
        X[t] = s < nsys ? o.alpha * o.C[bidx(g(p), s)] : 0.0;
    }
    if (warp == 7) fetch(0);
    __syncthreads();
    const int nb = (n + BLK - 1) / BLK;
    for (int b = 0; b < nb; b++) {
        const int p0 = b * BLK;
        if (warp < 2) {
            // lanes: system 8 warp + lane % 8, rows lane / 8 + 4 u
            const double *d = D + (b & 1) * BLK * LD;
            const int part = lane >> 3;
            double *x = X + (size_t)(p0 + part) * NSYS + 8 * warp + (lane & 7);
            double v[4];
#pragma unroll
            for (int u = 0; u < 4; u++) v[u] = p0 + part + 4 * u < n ? x[4 * u * NSYS] : 0.0;
#pragma unroll
            for (int k = 0; k < BLK; k++) {
                if (!o.unit) {
                    const double q = trsm_quotient(v[k >> 2], d[k * LD + k], d[k * LD + BLK], part == (k & 3));
                    if (part == (k & 3)) v[k >> 2] = q;
                }
                const double xk = __shfl_sync(0xffffffffu, v[k >> 2], (lane & 7) + 8 * (k & 3));
#pragma unroll
                for (int u = k >> 2; u < 4; u++)
                    if (u > (k >> 2) || part > (k & 3)) v[u] = fma(-d[k * LD + part + 4 * u], xk, v[u]);
            }
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (p0 + part + 4 * u < n) x[4 * u * NSYS] = v[u];
        } else {
            if (warp == 7 && b + 1 < nb) fetch(b + 1);
            if (b > 0) {
                const double *xb = X + (p0 - BLK) * NSYS + s;
                for (int p = p0 + BLK + (threadIdx.x - 64) / NSYS; p < n; p += (NTHREADS - 64) / NSYS) {
                    double acc = X[p * NSYS + s];
#pragma unroll 1
                    for (int k0 = 0; k0 < BLK; k0 += 8) {
                        double tk[8];
#pragma unroll
                        for (int k = 0; k < 8; k++) tk[k] = T(p, p0 - BLK + k0 + k);
#pragma unroll
                        for (int k = 0; k < 8; k++) acc = fma(-tk[k], xb[(k0 + k) * NSYS], acc);
                    }
                    X[p * NSYS + s] = acc;
                }
            }
        }
        __syncthreads();
        if (b + 1 == nb) break;
        const int i = threadIdx.x / NSYS;
        if (p0 + BLK + i < n) {
            double acc = X[(p0 + BLK + i) * NSYS + s];
#pragma unroll
            for (int k = 0; k < BLK; k++) acc = fma(-E[k * LD + i], X[(p0 + k) * NSYS + s], acc);
            X[(p0 + BLK + i) * NSYS + s] = acc;
        }
        __syncthreads();
    }
    for (int t = threadIdx.x; t < n * NSYS; t += NTHREADS)
        if (s < nsys) o.C[bidx(g(t / NSYS), s)] = X[t];
}

}  // namespace gbx_grouped
