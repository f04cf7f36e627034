// l2_ext.cu — DGER, DSYMV and DTRSV: the Level-2 routines on either side of
// a Cholesky or TRSM step (rank-1 update, symmetric matrix-vector product,
// triangular solve with one right-hand side).  The reference lists them in
// blas_level2/ger.cc, symv.cc and trsv.cc (CBLAS bodies that its build
// leaves out, meson.build:53-75; prototypes blas.h:94-100, 134-142,
// 193-200).
//
//   * DGER: A += alpha x y^T streams A once (read + write, 16 B per FMA:
//     HBM-bound); 512-row x 32-column tiles, netlib's skip of zero y_j.
//   * DSYMV: y = alpha A x + beta y reads only the stored triangle.  Each
//     64x64 tile of the triangle is staged in shared memory and used twice
//     (A_IJ x_J for rows I and A_IJ^T x_I for rows J), so the kernel does 2
//     FMAs per 8 bytes: on GB300's FP64 pipe (2 lanes per clock per SM) that
//     is the bound, not HBM.  Per-tile partial vectors are summed in a fixed
//     order by a second kernel (deterministic).
//   * DTRSV: one cooperative launch in which every CTA owns a 64-row block
//     and passes its part of the solution to the later blocks through global
//     memory as soon as it is known (see trsv_solve).
#include "gbx_internal.h"
#include "gemm_host.h"
#include "tri_inverse.cuh"

#include <cuda_runtime.h>
#include <stdint.h>
#include <algorithm>

namespace {

inline cudaStream_t S(gbx_ctx *ctx) { return (cudaStream_t)gbx_ctx_get_stream(ctx); }
inline long long base_off(int n, int inc) { return inc >= 0 ? 0 : (long long)(n - 1) * (-inc); }

// ------------------------------------------------------------------- DGER
constexpr int GER_ROWS = 512, GER_COLS = 32;

// 512 rows x 32 columns per CTA, two rows per thread, eight columns' loads in
// flight.  The bound is HBM (16 bytes per element and one DFMA: the FP64
// pipe alone would take two thirds of that time), so nothing else per
// element may use the FP64 pipe: alpha y_j is formed once per CTA and the
// test for a zero y_j (netlib leaves that column alone) is a bit in an
// integer mask.  With the product and the test per element the FP64 pipe was
// the bound: 8192 x 8192 took 387 us, now 162 us (1.07 GB, 6.6 TB/s).
// vec: A is 16-byte aligned and lda even, so that a thread's two adjacent
// rows are one 128-bit access in every column.
__global__ void __launch_bounds__(256)
ger_kernel(int m, int n, double alpha, const double *__restrict__ x, int incx, const double *__restrict__ y,
           int incy, double *__restrict__ A, long long lda, int vec)
{
    __shared__ double coef[GER_COLS];
    __shared__ unsigned s_keep;
    const int c0 = blockIdx.y * GER_COLS, cols = min(GER_COLS, n - c0);
    const int tid = threadIdx.x;
    if (tid < 32) {
        const double yj = tid < cols ? __ldg(y + (long long)(c0 + tid) * incy) : 0.0;
        coef[tid] = alpha * yj;
        // y_j != 0 on the bit pattern (NaN counts as nonzero)
        const unsigned keep = __ballot_sync(0xffffffffu, (__double_as_longlong(yj) << 1) != 0);
        if (tid == 0) s_keep = keep;
    }
    __syncthreads();
    const unsigned keep = s_keep;
    // vec: rows r, r + 1 with r even; otherwise rows r and r + 256
    const int r = blockIdx.x * GER_ROWS + (vec ? 2 * tid : tid);
    const int r2 = vec ? r + 1 : r + 256;
    if (r >= m) return;
    double *ap = A + (long long)c0 * lda + r;
    const double x0 = __ldg(x + (long long)r * incx);
    const double x1 = r2 < m ? __ldg(x + (long long)r2 * incx) : 0.0;
    if (keep == 0xffffffffu >> (GER_COLS - cols) && r2 < m) {   // no column is skipped
        if (vec) {
#pragma unroll 1
            for (int j = 0; j < cols; j += 8) {
                double2 v[8];
#pragma unroll
                for (int u = 0; u < 8; u++)
                    if (j + u < cols) v[u] = *(const double2 *)(ap + (j + u) * lda);
#pragma unroll
                for (int u = 0; u < 8; u++)
                    if (j + u < cols) {
                        const double c = coef[j + u];
                        v[u].x = fma(x0, c, v[u].x);
                        v[u].y = fma(x1, c, v[u].y);
                        *(double2 *)(ap + (j + u) * lda) = v[u];
                    }
            }
        } else {
#pragma unroll 1
            for (int j = 0; j < cols; j += 8) {
                double v[8], w[8];
#pragma unroll
                for (int u = 0; u < 8; u++)
                    if (j + u < cols) {
                        v[u] = ap[(j + u) * lda];
                        w[u] = ap[(j + u) * lda + 256];
                    }
#pragma unroll
                for (int u = 0; u < 8; u++)
                    if (j + u < cols) {
                        const double c = coef[j + u];
                        ap[(j + u) * lda] = fma(x0, c, v[u]);
                        ap[(j + u) * lda + 256] = fma(x1, c, w[u]);
                    }
            }
        }
        return;
    }
    for (int j = 0; j < cols; j++) {
        if (!((keep >> j) & 1)) continue;
        double *q = ap + j * lda;
        const double c = coef[j];
        *q = fma(x0, c, *q);
        if (r2 < m) q[r2 - r] = fma(x1, c, q[r2 - r]);
    }
}

// ------------------------------------------------------------------ DSYMV
constexpr int SY_T = 64;

// One tile (I, J) of the stored triangle per CTA (I >= J for lower, I <= J
// for upper in block indices).  Writes the row partial (A_IJ x_J, 64 values)
// to part[I][J] and, off the diagonal, the column partial (A_IJ^T x_I) to
// part[J][I]; part[b][q] is the q-th partial of output block b.
__global__ void __launch_bounds__(256)
symv_tiles(int n, int nb, int lower, const double *__restrict__ A, long long lda, const double *__restrict__ x,
           int incx, double *__restrict__ part)
{
    __shared__ double s[SY_T][SY_T + 1];
    __shared__ double sxI[SY_T], sxJ[SY_T];
    __shared__ double red[4][SY_T];
    // tile index -> (I, J) with I >= J (lower) in row-major triangle order
    // (FP32 square root and integer correction: an FP64 one by every thread
    // cost the FP64 pipe nearly half as much as the tile's products:
    // n = 8192 took 198 us, now 136 us)
    const int t = blockIdx.x;
    int I = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
    while ((long long)(I + 1) * (I + 2) / 2 <= t) I++;
    while ((long long)I * (I + 1) / 2 > t) I--;
    int J = (int)(t - (long long)I * (I + 1) / 2);
    if (!lower) { const int tmp = I; I = J; J = tmp; }   // upper: I <= J
    const int r0 = I * SY_T, c0 = J * SY_T;
    const int tid = threadIdx.x;
    for (int q = tid; q < SY_T * SY_T; q += blockDim.x) {
        const int i = q % SY_T, j = q / SY_T;
        const int gi = r0 + i, gj = c0 + j;
        double v = 0.0;
        if (gi < n && gj < n) {
            if (I != J) v = A[(long long)gj * lda + gi];
            else {
                const bool stored = lower ? gi >= gj : gi <= gj;
                v = stored ? A[(long long)gj * lda + gi] : A[(long long)gi * lda + gj];   // mirror
            }
        }
        s[i][j] = v;
    }
    if (tid < SY_T) {
        sxJ[tid] = (c0 + tid < n) ? x[(long long)(c0 + tid) * incx] : 0.0;
        sxI[tid] = (r0 + tid < n) ? x[(long long)(r0 + tid) * incx] : 0.0;
    }
    __syncthreads();
    const int l = tid & (SY_T - 1), part4 = tid >> 6;
    // row sums: row l over columns part4*16 .. +15
    double r = 0.0;
#pragma unroll
    for (int j = 0; j < 16; j++) r = fma(s[l][part4 * 16 + j], sxJ[part4 * 16 + j], r);
    red[part4][l] = r;
    __syncthreads();
    double *rowp = part + ((size_t)I * nb + J) * SY_T;
    if (tid < SY_T) rowp[tid] = (red[0][tid] + red[1][tid]) + (red[2][tid] + red[3][tid]);
    if (I == J) return;
    __syncthreads();
    // column sums: column l over rows part4*16 .. +15
    double c = 0.0;
#pragma unroll
    for (int i = 0; i < 16; i++) c = fma(s[part4 * 16 + i][l], sxI[part4 * 16 + i], c);
    red[part4][l] = c;
    __syncthreads();
    double *colp = part + ((size_t)J * nb + I) * SY_T;
    if (tid < SY_T) colp[tid] = (red[0][tid] + red[1][tid]) + (red[2][tid] + red[3][tid]);
}

// y_i = alpha * sum_q part[b][q][i] + beta y_i  (beta == 0 sets y).  One CTA
// per output block, four threads per row, each summing a quarter of the
// partials in order with eight loads in flight (one thread per row walking
// all 128 partials of n = 8192 took 19.6 us, now 6.8 us).
__global__ void __launch_bounds__(4 * SY_T)
symv_finish(int n, int nb, const double *__restrict__ part, double alpha, double beta, double *__restrict__ y,
            int incy)
{
    __shared__ double red[4][SY_T];
    const int b = blockIdx.x, l = threadIdx.x & (SY_T - 1), g = threadIdx.x / SY_T;
    const int q0 = (int)((long long)nb * g / 4), q1 = (int)((long long)nb * (g + 1) / 4);
    const double *p = part + (size_t)b * nb * SY_T + l;
    double s = 0.0;
#pragma unroll 8
    for (int q = q0; q < q1; q++) s += p[(size_t)q * SY_T];
    red[g][l] = s;
    __syncthreads();
    const int i = b * SY_T + l;
    if (g || i >= n) return;
    s = (red[0][l] + red[1][l]) + (red[2][l] + red[3][l]);
    double *yp = y + (long long)i * incy;
    *yp = (beta == 0.0) ? alpha * s : fma(alpha, s, beta * *yp);
}

// ------------------------------------------------------------------ DTRSV
constexpr int TV_NB = gbx_tri::NB, TV_LD = gbx_tri::LD, TV_THREADS = 256, TV_STAGES = 3;
constexpr int TV_TILE = TV_NB * TV_LD;
constexpr size_t TV_SMEM = sizeof(double) * ((TV_STAGES + 1) * TV_TILE + 4 * TV_NB + TV_NB + 8 * 16);
constexpr int TV_FOLD = 24;
constexpr unsigned long long TV_TIMEOUT_NS = 2000000000ull;
constexpr int TV_TIMEOUT_CODE = 9;

struct TrsvArgs {
    int n, nblk, fwd, tr, unit, incx;
    const double *A;
    long long lda;
    double *x;          // element 0 of the vector
    double *xw;         // solution in solve order, nblk * 64 values, all bits set until known
    int *status, *status_host;
};

__device__ __forceinline__ unsigned long long tv_now()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// 8-byte asynchronous copy; ok == 0 writes zero and reads nothing.
__device__ __forceinline__ void tv_copy8(double *dst, const double *src, int ok)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;"
                 :: "r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(ok ? 8 : 0) : "memory");
}

// op(A) in solve order: T(p, c) = op(A)(g(p), g(c)) with g(p) = p for a lower
// op(A) and n - 1 - p for an upper one, so that T is always lower triangular
// and solved forwards.  Address of T(p, c); p, c < n.
__device__ __forceinline__ const double *tv_at(const TrsvArgs &a, int p, int c)
{
    const long long r = a.fwd ? p : a.n - 1 - p, q = a.fwd ? c : a.n - 1 - c;
    return a.tr ? a.A + r * a.lda + q : a.A + q * a.lda + r;
}

// Starts the copy of the 64 x 64 block (s, K), K < s, to dst[k * 65 + i]:
// neighbouring threads take neighbouring addresses in memory.
__device__ __forceinline__ void tv_fetch(const TrsvArgs &a, double *dst, int s, int K)
{
    const int t = threadIdx.x & 63, g = threadIdx.x >> 6;
    const int i0 = a.tr ? g : t, k0 = a.tr ? t : g;
    const int p0 = s * TV_NB + i0, c0 = K * TV_NB + k0;
    const long long sgn = a.fwd ? 1 : -1;
    const double *src = tv_at(a, min(p0, a.n - 1), c0);
    const long long step = 4 * sgn * a.lda;
    double *d = dst + k0 * TV_LD + i0;
#pragma unroll
    for (int u = 0; u < 16; u++) {
        const int ok = p0 + (a.tr ? 4 * u : 0) < a.n;
        tv_copy8(d, ok ? src + u * step : a.A, ok);
        d += a.tr ? 4 : 4 * TV_LD;
    }
}

// This warp's 16 values of solution block K (columns 16 q .. of it): lanes
// 0-15 hold them in v once known.  The values themselves are the flags: a
// block's owner stores them over the "all bits set" pattern.  A wait that
// lasts 2 s gives up: the status word is set and the values become NaN, so
// that every later block still finishes.
__device__ __forceinline__ double tv_load(const double *p, int lane)
{
    return lane < 16 ? *(const volatile double *)(p + lane) : 0.0;
}
__device__ __forceinline__ double tv_wait(const TrsvArgs &a, const double *p, double v, int lane)
{
    if (__all_sync(0xffffffffu, __double_as_longlong(v) != -1ll)) return v;
    const unsigned long long t0 = tv_now();
    while (true) {
        if (__double_as_longlong(v) == -1ll) v = tv_load(p, lane);
        if (__all_sync(0xffffffffu, __double_as_longlong(v) != -1ll)) return v;
        if (__any_sync(0xffffffffu, tv_now() - t0 > TV_TIMEOUT_NS)) {
            if (lane == 0) {
                atomicCAS(a.status, 0, TV_TIMEOUT_CODE);
                *(volatile int *)a.status_host = TV_TIMEOUT_CODE;
                __threadfence_system();
            }
            return __longlong_as_double(0x7ff8000000000000ll);
        }
    }
}

// x := T^-1 x, blocks of 64 rows in solve order; CTA b owns blocks b,
// b + gridDim.x, ...  All CTAs are resident (cooperative launch), and a block
// waits only for earlier ones.  For its block s a CTA
//   * inverts the diagonal block (while it waits anyway, except the first);
//   * subtracts T(s, K) x_K for every earlier block K as x_K appears, the
//     64 x 64 blocks of T prefetched three deep into shared memory (they do
//     not depend on x), 16 of the products per thread and block;
//   * x_s = inv (b - sum) goes to the later blocks through xw and to x.
// What bounds it: the chain over the blocks, each link one hand-over through
// L2 (about 1 us) and the products between x_(s-1) and x_s, 1 us per 64 x 64
// on the SM's two FP64 lanes.  From the 24th block on there is time to form
// M = inv T(s, s-1) beforehand, so that x_s = inv (b - sum over K < s-1) -
// M x_(s-1) needs one product after x_(s-1) instead of two (M costs 47 us,
// by which the chain has come to that block).  64 rows per block: half of it
// would double the hand-overs, double of it the products per link.
// n = 8192: 300 us for N or T; one launch per 64 rows, each forming
// x_s in every CTA, took 4.1 ms.
__global__ void __launch_bounds__(TV_THREADS)
trsv_solve(TrsvArgs a)
{
    extern __shared__ __align__(16) double tv_sm[];
    double *stage = tv_sm;                          // TV_STAGES blocks
    double *X = stage + TV_STAGES * TV_TILE;        // inverse of the diagonal block
    double *red = X + TV_TILE;                      // [4][64]
    double *st = red + 4 * TV_NB;                   // [64]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int i = tid & 63, q = tid >> 6;           // row, quarter of the columns
    double *xs = st + TV_NB + 16 * warp;            // this warp's 16 solution values

    for (int s = blockIdx.x; s < a.nblk; s += gridDim.x) {
        const int p = s * TV_NB + i;
        // diagonal block into stage 0 (identity beyond n)
        for (int t = tid; t < TV_NB * TV_NB; t += TV_THREADS) {
            const int u = t & 63, v = t >> 6;
            const int r = a.tr ? v : u, k = a.tr ? u : v;
            const int pr = s * TV_NB + r, pk = s * TV_NB + k;
            double d = r == k ? 1.0 : 0.0;
            if (k <= r && pr < a.n && !(a.unit && r == k)) d = *tv_at(a, pr, pk);
            stage[k * TV_LD + r] = d;
        }
        const bool fold = s >= TV_FOLD;
        if (fold) tv_fetch(a, stage + TV_TILE, s, s - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const double b = p < a.n ? a.x[(long long)(a.fwd ? p : a.n - 1 - p) * a.incx] : 0.0;
        __syncthreads();
        gbx_tri::invert64(stage, X, stage + 2 * TV_TILE);
        double M[16];
        if (fold) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            // M(i, 16 q ..): row i of the inverse reaches column i at most
            const double *T1 = stage + TV_TILE + 16 * q * TV_LD;
#pragma unroll
            for (int k = 0; k < 16; k++) M[k] = 0.0;
            const int jend = (warp & 1) ? 64 : 32;
            for (int j = 0; j < jend; j++) {
                const double v = X[j * TV_LD + i];
#pragma unroll
                for (int k = 0; k < 16; k++) M[k] = fma(v, T1[k * TV_LD + j], M[k]);
            }
            __syncthreads();
        }
        const int nk = fold ? s - 1 : s;   // blocks subtracted one by one
#pragma unroll
        for (int f = 0; f < TV_STAGES - 1; f++) {
            if (f < nk) tv_fetch(a, stage + f * TV_TILE, s, f);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        double acc = 0.0, xv = 0.0;
        if (s > 0) xv = tv_load(a.xw + 16 * q, lane);
        for (int K = 0; K < nk; K++) {
            asm volatile("cp.async.wait_group %0;" :: "n"(TV_STAGES - 2) : "memory");
            __syncthreads();   // block K is in, block K - 1 consumed
            if (K + TV_STAGES - 1 < nk)
                tv_fetch(a, stage + ((K + TV_STAGES - 1) % TV_STAGES) * TV_TILE, s, K + TV_STAGES - 1);
            asm volatile("cp.async.commit_group;" ::: "memory");
            xv = tv_wait(a, a.xw + (long long)K * TV_NB + 16 * q, xv, lane);
            __syncwarp();
            if (lane < 16) xs[lane] = xv;
            __syncwarp();
            if (K + 1 < s) xv = tv_load(a.xw + (long long)(K + 1) * TV_NB + 16 * q, lane);
            const double *T = stage + (K % TV_STAGES) * TV_TILE + 16 * q * TV_LD + i;
#pragma unroll
            for (int k = 0; k < 16; k++) acc = fma(T[k * TV_LD], xs[k], acc);
        }
        red[q * TV_NB + i] = acc;
        __syncthreads();
        if (tid < TV_NB) st[i] = b - ((red[i] + red[TV_NB + i]) + (red[2 * TV_NB + i] + red[3 * TV_NB + i]));
        __syncthreads();
        double v = 0.0;
        if ((warp & 1) || q < 2) {   // rows < 32 end at column 31
#pragma unroll
            for (int k = 0; k < 16; k++) v = fma(X[(16 * q + k) * TV_LD + i], st[16 * q + k], v);
        }
        if (fold) {
            xv = tv_wait(a, a.xw + (long long)(s - 1) * TV_NB + 16 * q, xv, lane);
            __syncwarp();
            if (lane < 16) xs[lane] = xv;
            __syncwarp();
#pragma unroll
            for (int k = 0; k < 16; k++) v = fma(-M[k], xs[k], v);
        }
        red[q * TV_NB + i] = v;
        __syncthreads();
        if (tid < TV_NB) {
            const double r = (red[i] + red[TV_NB + i]) + (red[2 * TV_NB + i] + red[3 * TV_NB + i]);
            // the "not yet known" pattern is a NaN: publish another NaN in its place
            const double o = __double_as_longlong(r) == -1ll ? __longlong_as_double(0x7ff8000000000000ll) : r;
            *(volatile double *)(a.xw + p) = o;
            if (p < a.n) a.x[(long long)(a.fwd ? p : a.n - 1 - p) * a.incx] = r;
        }
        __syncthreads();   // shared memory is reused by the next block
    }
}

}  // namespace

// ------------------------------------------------------------------ checks
extern "C" int gbx_check_ger_args(int m, int n, int incx, int incy, int lda)
{
    if (m < 0) return 1;
    if (n < 0) return 2;
    if (incx == 0) return 5;
    if (incy == 0) return 7;
    if (lda < std::max(1, m)) return 9;
    return 0;
}

extern "C" int gbx_check_symv_args(char uplo, int n, int lda, int incx, int incy)
{
    if (!gbx_lsame(uplo, 'U') && !gbx_lsame(uplo, 'L')) return 1;
    if (n < 0) return 2;
    if (lda < std::max(1, n)) return 5;
    if (incx == 0) return 7;
    if (incy == 0) return 10;
    return 0;
}

extern "C" int gbx_check_trsv_args(char uplo, char trans, char diag, int n, int lda, int incx)
{
    if (!gbx_lsame(uplo, 'U') && !gbx_lsame(uplo, 'L')) return 1;
    if (!gbx_lsame(trans, 'N') && !gbx_lsame(trans, 'T') && !gbx_lsame(trans, 'C')) return 2;
    if (!gbx_lsame(diag, 'U') && !gbx_lsame(diag, 'N')) return 3;
    if (n < 0) return 4;
    if (lda < std::max(1, n)) return 6;
    if (incx == 0) return 8;
    return 0;
}

// ------------------------------------------------------------ entry points
extern "C" gbx_status gbx_dger(gbx_ctx *ctx, int m, int n, double alpha, const double *x, int incx,
                               const double *y, int incy, double *A, int lda)
{
    if (!ctx) return GBX_ERR_ARG;
    const int info = gbx_check_ger_args(m, n, incx, incy, lda);
    if (info) return gbx_fail(ctx, GBX_ERR_ARG, "DGER parameter %d", info);
    if (m == 0 || n == 0 || alpha == 0.0) return GBX_OK;
    dim3 g((m + GER_ROWS - 1) / GER_ROWS, (n + GER_COLS - 1) / GER_COLS);
    if (g.y > 65535) return gbx_fail(ctx, GBX_ERR_UNSUPPORTED, "DGER: n too large");
    gbx_timer_begin(ctx, GBX_TIMER_GEMV);
    const int vec = (((uintptr_t)A) & 15) == 0 && lda % 2 == 0;
    ger_kernel<<<g, 256, 0, S(ctx)>>>(m, n, alpha, x + base_off(m, incx), incx, y + base_off(n, incy), incy, A,
                                      lda, vec);
    gbx_timer_end(ctx);
    gbx_count_launch(ctx, 1);
    return gbx_check_launch(ctx, "dger");
}

extern "C" gbx_status gbx_dsymv(gbx_ctx *ctx, char uplo, int n, double alpha, const double *A, int lda,
                                const double *x, int incx, double beta, double *y, int incy)
{
    if (!ctx) return GBX_ERR_ARG;
    const int info = gbx_check_symv_args(uplo, n, lda, incx, incy);
    if (info) return gbx_fail(ctx, GBX_ERR_ARG, "DSYMV parameter %d", info);
    if (n == 0 || (alpha == 0.0 && beta == 1.0)) return GBX_OK;
    const double *xb = x + base_off(n, incx);
    double *yb = y + base_off(n, incy);
    const int nb = (n + SY_T - 1) / SY_T;
    double *part;
    gbx_status st = gbx_ws(ctx, GBX_WS_GEMV, sizeof(double) * (size_t)nb * nb * SY_T, (void **)&part);
    if (st != GBX_OK) return st;
    const long long tiles = (long long)nb * (nb + 1) / 2;
    if (tiles > 0x7fffffffLL) return gbx_fail(ctx, GBX_ERR_UNSUPPORTED, "DSYMV: n too large");
    if (alpha != 0.0) {
        gbx_timer_begin(ctx, GBX_TIMER_GEMV);
        symv_tiles<<<(unsigned)tiles, 256, 0, S(ctx)>>>(n, nb, gbx_lsame(uplo, 'L'), A, lda, xb, incx, part);
        gbx_timer_end(ctx);
        gbx_count_launch(ctx, 1);
    } else {
        cudaMemsetAsync(part, 0, sizeof(double) * (size_t)nb * nb * SY_T, S(ctx));
    }
    symv_finish<<<nb, 4 * SY_T, 0, S(ctx)>>>(n, nb, part, alpha, beta, yb, incy);
    gbx_count_launch(ctx, 1);
    return gbx_check_launch(ctx, "dsymv");
}

extern "C" gbx_status gbx_dtrsv(gbx_ctx *ctx, char uplo, char trans, char diag, int n, const double *A, int lda,
                                double *x, int incx)
{
    if (!ctx) return GBX_ERR_ARG;
    const int info = gbx_check_trsv_args(uplo, trans, diag, n, lda, incx);
    if (info) return gbx_fail(ctx, GBX_ERR_ARG, "DTRSV parameter %d", info);
    if (n == 0) return GBX_OK;
    const int tri = gbx_op_tri(uplo, trans, diag);
    const int nblk = (n + TV_NB - 1) / TV_NB;
    double *xw;
    TrsvArgs p{};
    gbx_status st;
    if ((st = gbx_ws(ctx, GBX_WS_TMP2, sizeof(double) * (size_t)nblk * TV_NB, (void **)&xw)) != GBX_OK) return st;
    if ((st = gbx_ctx_status(ctx, &p.status, &p.status_host)) != GBX_OK) return st;
    p.n = n;
    p.nblk = nblk;
    p.fwd = (tri & gbx_gemm::TRI_LOWER) != 0;
    p.tr = !gbx_lsame(trans, 'N');
    p.unit = (tri & gbx_gemm::TRI_UNIT) != 0;
    p.A = A;
    p.lda = lda;
    p.x = x + base_off(n, incx);
    p.incx = incx;
    p.xw = xw;
    // every value "not yet known" (all bits set)
    cudaError_t e = cudaMemsetAsync(xw, 0xFF, sizeof(double) * (size_t)nblk * TV_NB, S(ctx));
    // a per-device function attribute; setting it is a cheap host call
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(trsv_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TV_SMEM);
    if (e != cudaSuccess) return gbx_fail(ctx, GBX_ERR_CUDA, "dtrsv: %s", cudaGetErrorString(e));
    const int grid = std::min(nblk, gbx_ctx_sms(ctx));   // one CTA per SM is always resident
    void *args[] = {&p};
    gbx_timer_begin(ctx, GBX_TIMER_GEMV);
    e = cudaLaunchCooperativeKernel((const void *)trsv_solve, dim3(grid), dim3(TV_THREADS), args, TV_SMEM, S(ctx));
    gbx_timer_end(ctx);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return gbx_fail(ctx, GBX_ERR_CUDA, "dtrsv: %s", cudaGetErrorString(e));
    }
    gbx_count_launch(ctx, 1);
    return gbx_check_launch(ctx, "dtrsv");
}
