// potrf.cu — Cholesky factorisation of one diagonal block, lower triangle.
// Not a BLAS routine: it is the diagonal step of the blocked right-looking
// Cholesky that drives the serving trace (the other steps are the
// intercepted dtrsm_/dsyrk_/dgemm_ calls).
//
// Blocked in 32-column steps.  On GB300 one SM does about 4 GFLOP/s of FP64,
// so a factorisation of a 256 x 256 block confined to one CTA costs over a
// millisecond; here only the 32 x 32 diagonal factorisations are serial:
//   * potrf_step(j0): every CTA (four warps) factors the
//     32 x 32 diagonal block at j0 (redundantly) together with 8 rows of the
//     panel below it, which take the same column operations; the last CTA to
//     finish writes the diagonal block back;
//   * potrf_syrk(j0): the trailing update A22 -= A21 A21^T, one 16 x 16
//     lower tile per CTA (8k FMAs each).  The GEMM core would put this
//     product on one or two 128 x 128 tiles, i.e. one or two SMs: 63 µs for
//     a 64 x 64 x 64 update.
// A non-positive pivot sets *info to its 1-based column (LAPACK convention,
// first failure wins); the rest of the block is then unspecified.
#include "gbx_internal.h"
#include "launch.cuh"

#include <cuda_runtime.h>

namespace {

using namespace gbx_launch;

constexpr int PB = 32;          // panel width: one lane per row of the diagonal block
constexpr int PR = 8;           // panel rows per CTA
constexpr int PT_THREADS = 128;

// 1 / d to within an ulp or two for a positive d: an approximate reciprocal y
// and one step of Halley's third-order iteration, y (1 + e + e^2) with
// e = 1 - d y (e < 2^-18 leaves e^3 < 2^-54), three dependent FP64 operations
// where a division takes a dozen (64 cycles each on this part).  NaN for a d
// whose reciprocal is near the ends of the range: its column is divided by d.
__device__ __forceinline__ double potrf_recip(double d)
{
    const unsigned ex = ((unsigned)(__double_as_longlong(d) >> 52)) & 0x7ffu;
    if (ex - 23u > 2000u) return __longlong_as_double(0x7ff8000000000000ll);
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = fma(-d, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// The division of the rare columns, out of line (the steps are unrolled).
__device__ __noinline__ double potrf_ratio(double a, double d) { return a / d; }

// One step j0.  Warp w holds columns 4q + w of the diagonal block (lane = row,
// a[q]) and of this CTA's 8 panel rows (lane = row + 8 (q mod 4), p[q / 4]).
// The factorisation is A = L' D L'^T with L' = L diag(L)^-1: at step k every warp
// scales the published column k by -1/d_k and subtracts its multiples from its
// own later columns; the warp of column k + 1 updates that one first, publishes
// it with its reciprocal and arrives on a named barrier that only the others
// wait on, so the chain from pivot to pivot is one multiplication, two FMAs (the
// panel's column too) and a reciprocal.  The square roots come at the end, one
// per column in parallel.  A warp has one FP64 instruction in flight at a time,
// 65 cycles each whether they depend on one another or not, and four warps fill
// the SM's pipe (a one-warp version took 64 us); the chain's seven operations
// and hand-over set 500 to 900 cycles per column.
// Measured: 18 us per step; with a barrier of 256 threads and a reciprocal
// square root per column it was 30 us.
__global__ void __launch_bounds__(PT_THREADS)
potrf_step(int n, int j0, double *__restrict__ A, long long lda, int *__restrict__ info, unsigned *done)
{
    pdl_enter();
    __shared__ double colA[PB][PB];   // column k, unscaled, once final
    __shared__ double colP[PB][PR];
    __shared__ double rec[PB];        // reciprocal (then reciprocal square root) of pivot k
    __shared__ int s_last;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int b = min(PB, n - j0);
    const int r0 = j0 + b + blockIdx.x * PR;   // first panel row (b = PB whenever there is a panel)
    const int pr = lane & (PR - 1), pg = lane >> 3;
    double *D = A + (long long)j0 * lda + j0;
    double a[8], p[2];
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const int j = 4 * q + warp;
        a[q] = (lane < b && j <= lane) ? D[(long long)j * lda + lane] : (j == lane ? 1.0 : 0.0);
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int j = 4 * (pg + 4 * h) + warp;
        p[h] = (r0 + pr < n && j < b) ? A[(long long)(j0 + j) * lda + r0 + pr] : 0.0;
    }
    // publishes column k (this warp's): values, reciprocal of the pivot, panel
    auto publish = [&](int k, double ak, double pk) {
        colA[k][lane] = ak;
        if (pg == ((k >> 2) & 3)) colP[k][pr] = pk;
        const double r = potrf_recip(__shfl_sync(0xffffffffu, ak, k));
        if (lane == 0) rec[k] = r;
        bar_arrive(1 + (k & 7), PT_THREADS);
    };
    if (warp == 0) publish(0, a[0], p[0]);
#pragma unroll
    for (int k = 0; k < PB - 1; k++) {
        if (warp != (k & 3)) bar_wait(1 + (k & 7), PT_THREADS);
        const double r = rec[k];
        double m = -(colA[k][lane] * r);
        if ((__double_as_longlong(r) & 0x7ff0000000000000ll) == 0x7ff0000000000000ll)   // uniform
            m = -potrf_ratio(colA[k][lane], colA[k][k]);
        const double pk = colP[k][pr];
        constexpr unsigned ALL = 0xffffffffu;
        if (warp == ((k + 1) & 3)) {
            a[(k + 1) >> 2] = fma(m, colA[k][k + 1], a[(k + 1) >> 2]);
            const double mk = __shfl_sync(ALL, m, k + 1);
            publish(k + 1, a[(k + 1) >> 2], fma(pk, mk, p[(k + 1) >> 4]));
        }
#pragma unroll
        for (int q = 0; q < 8; q++)
            if (4 * q + 3 > k && 4 * q + warp > k + (warp == ((k + 1) & 3) ? 1 : 0)) {
                a[q] = fma(m, colA[k][4 * q + warp], a[q]);
            }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (16 * h + 15 <= k) continue;
            // a lane's columns up to k + 1 are published already: its value no longer matters
            const double mj = __shfl_sync(ALL, m, (4 * (pg + 4 * h) + warp) & 31);
            p[h] = fma(pk, mj, p[h]);
        }
    }
    if (warp != ((PB - 1) & 3)) bar_wait(1 + ((PB - 1) & 7), PT_THREADS);
    __syncthreads();
    // 1-based column of the first non-positive pivot (zero, negative or NaN, by
    // the bit pattern), or 0; every warp gets the same answer
    const double d = colA[lane][lane];
    const unsigned neg =
        __ballot_sync(0xffffffffu, (unsigned long long)__double_as_longlong(d) - 1ull >= 0x7ff0000000000000ull);
    const int bad = __ffs((int)neg);
    const double y = rsqrt(d);   // L_ik = a_ik / sqrt(d_k)
    if (warp == 0) rec[lane] = y;
    __syncthreads();
    if (!bad) {
        for (int t = tid; t < PR * PB; t += PT_THREADS) {
            const int q = t % PR, k = t / PR;
            if (r0 + q < n && k < b) A[(long long)(j0 + k) * lda + r0 + q] = colP[k][q] * rec[k];
        }
    }
    // The factored diagonal block goes back to A only when every CTA has read
    // the original (the last CTA to finish writes it; all CTAs hold the same
    // factor), so no CTA can read a half-written block.
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        s_last = atomicAdd(done, 1u) == gridDim.x - 1;
        if (s_last) {
            *done = 0u;
            if (bad) atomicCAS(info, 0, j0 + bad);
        }
    }
    __syncthreads();
    if (!s_last || bad) return;
    for (int k = warp; k < b; k += 4)
        if (lane < b && k <= lane) D[(long long)k * lda + lane] = colA[k][lane] * rec[k];
}

// A22 (m x m, lower) -= A21 A21^T with A21 m x PB: one 16 x 16 tile of the
// lower triangle per CTA, blockIdx.x enumerating the tiles (ti >= tj) row by
// row; the two 16 x PB row blocks of A21 are staged in shared memory.
__global__ void __launch_bounds__(256)
potrf_syrk(int m, const double *__restrict__ A21, double *__restrict__ A22, long long lda)
{
    pdl_enter();
    __shared__ double Li[16][PB + 1], Lj[16][PB + 1];
    const int b = blockIdx.x;
    int ti = (int)((sqrtf(8.0f * (float)b + 1.0f) - 1.0f) * 0.5f);
    while ((ti + 1) * (ti + 2) / 2 <= b) ti++;
    while (ti * (ti + 1) / 2 > b) ti--;
    const int tj = b - ti * (ti + 1) / 2;
    const int i0 = ti * 16, j0 = tj * 16;
    for (int t = threadIdx.x; t < 16 * PB; t += blockDim.x) {
        const int r = t & 15, k = t >> 4;
        Li[r][k] = i0 + r < m ? A21[(long long)k * lda + i0 + r] : 0.0;
        Lj[r][k] = j0 + r < m ? A21[(long long)k * lda + j0 + r] : 0.0;
    }
    __syncthreads();
    const int r = threadIdx.x & 15, c = threadIdx.x >> 4;
    const int gi = i0 + r, gj = j0 + c;
    if (gi >= m || gj > gi) return;
    double acc = 0.0;
#pragma unroll 8
    for (int k = 0; k < PB; k++) acc = fma(Li[r][k], Lj[c][k], acc);
    A22[(long long)gj * lda + gi] -= acc;
}

}  // namespace

extern "C" gbx_status gbx_dpotrf_small(gbx_ctx *ctx, char uplo, int n, double *A, int lda, int *info)
{
    if (!ctx || !info) return GBX_ERR_ARG;
    if (!gbx_lsame(uplo, 'L')) return gbx_fail(ctx, GBX_ERR_UNSUPPORTED, "dpotrf_small: lower only");
    if (n < 0 || n > 256 || lda < (n > 1 ? n : 1))
        return gbx_fail(ctx, GBX_ERR_ARG, "dpotrf_small: n = %d (<= 256), lda = %d", n, lda);
    cudaStream_t s = (cudaStream_t)gbx_ctx_get_stream(ctx);
    int *words, *mirror;
    gbx_status st = gbx_ctx_status(ctx, &words, &mirror);   // word 12: the step's finish counter
    if (st != GBX_OK) return st;
    unsigned *done = (unsigned *)(words + 12);
    cudaMemsetAsync(info, 0, sizeof(int), s);
    for (int j0 = 0; j0 < n; j0 += PB) {
        const int b = n - j0 < PB ? n - j0 : PB;
        const int rows = n - j0 - b;
        const int grid = rows > 0 ? (rows + PR - 1) / PR : 1;
        launch_pdl(potrf_step, grid, PT_THREADS, 0, s, n, j0, A, lda, info, done);
        gbx_count_launch(ctx, 1);
        if ((st = gbx_check_launch(ctx, "dpotrf_small")) != GBX_OK) return st;
        if (rows > 0) {
            const double *A21 = A + (long long)j0 * lda + j0 + b;
            double *A22 = A + (long long)(j0 + b) * lda + j0 + b;
            const int nt = (rows + 15) / 16;
            launch_pdl(potrf_syrk, nt * (nt + 1) / 2, 256, 0, s, rows, A21, A22, lda);
            gbx_count_launch(ctx, 1);
            if ((st = gbx_check_launch(ctx, "dpotrf_small update")) != GBX_OK) return st;
        }
    }
    return GBX_OK;
}
