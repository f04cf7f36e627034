// tri_inverse.cuh — inverses of small FP64 triangles in shared memory: 64 x 64 by a
// CTA of 256 threads (the diagonal blocks of the blocked DTRSV and DTRSM), 32 x 32
// by 128 (those of the triangular inverse).
//
// They are joined from inverted 16 x 16 blocks, X21 = -X22 (D21 X11), two products
// where substitution has a chain of rows.  But X22 multiplies what D21 X11 has
// lost to cancellation: for ill-conditioned triangles the error is that of
// substitution times the condition number of D22 (Du Croz and Higham, IMA J. Numer.
// Anal. 12(1), 1992).  The Cholesky factor of a Gaussian kernel with a nugget of 1e-8,
// condition 1e5, left a solve 230 times the backward error that substitution does,
// with 1e-10, 1e6, 3500 times.  So the joined inverse is kept only if the largest
// row sum of |X| |D|, which bounds the condition of every block it is joined from,
// is at most COND (600 random triangles: within 2 of substitution below 100), and is
// computed again by substitution otherwise.
#pragma once

#include <cuda_runtime.h>

namespace gbx_tri {

constexpr int NB = 64, LD = NB + 1;
constexpr float COND = 16.0f;

// |x| as a float, to 21 bits; at least 2^-126 unless zero, infinite beyond the FP32
// range and for NaN.  On the integer pipe: a conversion is an FP64 instruction.
__device__ __forceinline__ float abs_float(double x)
{
    const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
    if (h < 0x38100000u) return h ? 0x1p-126f : 0.0f;
    return __uint_as_float(h < 0x47f00000u ? (h - 0x38000000u) << 3 : 0x7f800000u);
}

// The row sums of |D|, D lower triangular N x N, by 2 N threads t: half a row each,
// left in the spare word that ends a column of X, or of D.
template <int N, int LD>
__device__ __forceinline__ void row_sums(double *D, double *X, int t)
{
    const int i = t % N, h = t / N;
    float v = 0.0f;
#pragma unroll 8
    for (int k = h * (N / 2); k < (h + 1) * (N / 2); k++)
        if (k <= i) v += abs_float(D[k * LD + i]);
    *(float *)((h ? D : X) + i * LD + N) = v;
}

// Whether the largest row sum of |X| |D| is at most COND, X lower triangular, after
// row_sums and a barrier; by the whole CTA of 4 N threads, four to a row.
template <int N, int LD>
__device__ __forceinline__ bool well_conditioned(const double *D, const double *X)
{
    const int lane = threadIdx.x & 31, i = (threadIdx.x >> 5) * 8 + (lane & 7), q = lane >> 3;
    float v = 0.0f;
#pragma unroll 8
    for (int s = 0; s < N / 4; s++) {   // (columns eight apart for the lanes of a half warp: no bank conflicts)
        const int k = (q >> 1) * (N / 2) + (s >> 3) * 16 + (q & 1) * 8 + (s & 7);
        const float r = *(const float *)(X + k * LD + N) + *(const float *)(D + k * LD + N);
        if (k <= i) v = fmaf(abs_float(X[k * LD + i]), r, v);
    }
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    v += __shfl_xor_sync(0xffffffffu, v, 16);
    return __syncthreads_and(v <= COND);   // (NaN: no)
}

// X = inverse of the lower triangular N x N block D by substitution, by the whole CTA
// of 4 N threads; R: N doubles.  Panels of 16 rows, a warp to eight columns: the
// panel's rows one after another, then all later rows subtract its 16.
template <int N, int LD>
__device__ __forceinline__ void invert_by_substitution(const double *D, double *X, double *R)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < N) R[tid] = 1.0 / D[tid * LD + tid];
    for (int t = tid; t < N * N; t += 4 * N) X[(t / N) * LD + t % N] = t / N == t % N ? 1.0 : 0.0;
    __syncthreads();
#pragma unroll 1
    for (int p = 0; p < N; p += 16) {
        if (8 * warp < p + 16) {
            const int part = lane >> 3;
            const double *d = D + p * LD + p + part;
            double *x = X + (8 * warp + (lane & 7)) * LD + p + part;
            double v[4];
#pragma unroll
            for (int u = 0; u < 4; u++) v[u] = x[4 * u];
#pragma unroll
            for (int k = 0; k < 16; k++) {
                const double xk = __shfl_sync(0xffffffffu, v[k >> 2] * R[p + k], (lane & 7) + 8 * (k & 3));
                if (part == (k & 3)) v[k >> 2] = xk;
#pragma unroll
                for (int u = k >> 2; u < 4; u++)
                    if (u > (k >> 2) || part > (k & 3)) v[u] = fma(-d[k * LD + 4 * u], xk, v[u]);
            }
#pragma unroll
            for (int u = 0; u < 4; u++) x[4 * u] = v[u];
        }
        __syncthreads();
        const int rows = N - 16 - p;
        for (int t = tid; t < rows * (p + 16); t += 4 * N) {
            const int r = p + 16 + t % rows, c = t / rows;
            double acc = X[c * LD + r];
#pragma unroll
            for (int k = 0; k < 16; k++) acc = fma(-D[(p + k) * LD + r], X[c * LD + p + k], acc);
            X[c * LD + r] = acc;
        }
        __syncthreads();
    }
}

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

// The same out of line, for a kernel that has other things in its registers.
static __device__ __noinline__ void invert64_by_substitution(const double *D, double *X, double *R)
{
    invert_by_substitution<NB, LD>(D, X, R);
}

// X = inverse of the lower triangular 64 x 64 block D (W: 32 x 33 scratch), by
// the whole CTA: the four 16 x 16 diagonal blocks, a warp each, then
// X21 = -X22 (D21 X11) for the two 32 x 32 blocks and for the whole; or, if the
// answer is false, by substitution.
// What bounds it: the FP64 pipe, which an instruction of a warp holds 16 to 19
// cycles whatever its predicate, so the loops skip the zero parts by warp: the
// two products of the whole take 20k cycles.  Substitution on 32 x 32
// blocks by four warps each, with a barrier per row, took 5 us more.
template <bool OUT_OF_LINE>
__device__ __forceinline__ bool invert64(double *D, double *X, double *W)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < 4) invert16<LD>(D, X, 16 * warp);
    else row_sums<NB, LD>(D, X, threadIdx.x - 128);
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
    const bool joined = well_conditioned<NB, LD>(D, X);
    if (!joined) {
        if (OUT_OF_LINE) invert64_by_substitution(D, X, W);
        else invert_by_substitution<NB, LD>(D, X, W);
    }
    return joined;
}

}  // namespace gbx_tri
