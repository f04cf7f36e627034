// potrf.cu — Cholesky factorisation of one diagonal block, lower triangle.
// Not a BLAS routine: it is the diagonal step of the blocked right-looking
// Cholesky that drives the serving trace (the other steps are the
// intercepted dtrsm_/dsyrk_/dgemm_ calls).
//
// Blocked in 32-column steps.  On GB300 one SM does about 4 GFLOP/s of FP64,
// so a factorisation of a 256 x 256 block confined to one CTA costs over a
// millisecond; here only the 32 x 32 diagonal factorisations are serial:
//   * potrf_step(j0): every CTA factors the
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
#include "tc_ptx.cuh"

#include <cuda_runtime.h>

namespace {

using namespace gbx_launch;

constexpr int PB = 32;          // panel width: one lane per row of the diagonal block
constexpr int PR = 8;           // panel rows per CTA
constexpr int PT_THREADS = 320;

// 1 / d to within an ulp or two for a positive d: an approximate reciprocal y
// and one step of Chebyshev's third-order iteration, y (1 + e + e^2) with
// e = 1 - d y (e < 2^-18 leaves e^3 < 2^-54), three dependent FP64 operations
// where a division takes a dozen (65 cycles each on this part).  Not for a d
// whose reciprocal is near the ends of the range: its column is divided by d.
__device__ __forceinline__ bool potrf_rare(double d)
{
    return (unsigned)(__double_as_longlong(d) >> 52) - 23u > 2000u;   // negative ones too
}
__device__ __forceinline__ double potrf_recip(double d)
{
    double y;
    asm volatile("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = fma(-d, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// The division of the rare columns, out of line (the steps are unrolled).
__device__ __noinline__ double potrf_ratio(double a, double d) { return a / d; }

// One step j0.  Warps 0-7 have the diagonal block, lane = row: columns w and w + 8
// in a[0], a[1], and of the columns from 16 on, whose rows begin at 16, two in
// one register: 16 + w in lanes 0-15 and 24 + w in lanes 16-31.  Warps 8 and 9 have
// four each of this CTA's panel rows: lane = row + 4 (column mod 8), p[column / 8].
// The factorisation is A = L' D L'^T with L' = L diag(L)^-1: at step k the warp of
// column k + 1 waits for column k, scales it by -1/d_k, subtracts its multiple
// from column k + 1 and hands that on, on a named barrier of the two warps; the
// scaled column m_k goes to the other warps, which subtract its multiples from
// their columns, and to the panel, on an mbarrier of its own, so that no warp
// waits for a slower one.  A warp whose turn is next leaves the step before to
// its turn, when the reciprocal is under way.  The square roots come at the end,
// one per column in parallel.
// What bounds it: the chain, five FP64 operations per column (66 cycles each, of
// which a warp has one in flight), an approximate reciprocal and a hand-over
// (90 cycles), 600 cycles in all; for the first columns the SM's FP64 pipe (16.7
// cycles an instruction), 850.
// Measured: 256 columns (8 steps with their updates) 132 us.  They were 178 with
// four warps that passed column and reciprocal on barriers where everybody waits
// for everybody (19 us a step, now 12; with a barrier of 256 threads and a
// reciprocal square root per column it was 30).
// A wait that did not end at once, out of line and bounded.  The arrival is that of
// a warp of the same CTA, which comes whatever an earlier call has left in the
// status word: only the deadline ends the wait, and sets *failed.
__device__ __noinline__ void potrf_wait_long(uint64_t *bar, int *status, int *failed)
{
    if (!gbx_tc::mbar_wait_timed(bar, 0u, status, gbx_tc::TC_TIMEOUT_FULL)) *(volatile int *)failed = 1;
}

__global__ void __launch_bounds__(PT_THREADS)
potrf_step(int n, int j0, double *__restrict__ A, long long lda, int *__restrict__ info, unsigned *done, int *status,
           int *status_host)
{
    __shared__ double colA[PB][PB];   // column k, unscaled, once final
    __shared__ double colM[PB][PB];   // -(column k) / d_k
    __shared__ double colP[PB][PR];
    __shared__ double rec[PB];        // reciprocal (then reciprocal square root) of pivot k
    __shared__ __align__(8) uint64_t barM[PB];
    __shared__ int s_last, s_failed;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_failed = 0;
    if (tid < PB) gbx_tc::mbar_init(barM + tid, 1);
    __syncthreads();
    pdl_enter();
    const int b = min(PB, n - j0);
    const int r0 = j0 + b + blockIdx.x * PR;   // first panel row (b = PB whenever there is a panel)
    double *D = A + (long long)j0 * lda + j0;
    constexpr unsigned ALL = 0xffffffffu;
    auto wait = [&](uint64_t *bar) {
        if (!gbx_tc::mbar_try_wait(bar, 0u)) potrf_wait_long(bar, status, &s_failed);
    };
    if (warp < 8) {
        const int row = 16 + (lane & 15), jb = 16 + warp + 8 * (lane >> 4);   // of ab
        double a[2], ab;
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int j = 8 * q + warp;
            a[q] = (lane < b && j <= lane) ? D[(long long)j * lda + lane] : (j == lane ? 1.0 : 0.0);
        }
        ab = (row < b && jb <= row) ? D[(long long)jb * lda + row] : (jb == row ? 1.0 : 0.0);
        if (warp == 0) {
            colA[0][lane] = a[0];
            bar_arrive(1, 64);
        }
        // column 8 q + warp of the first 16, and the last ones, at step k; a
        // published column's value no longer matters
        auto update_a = [&](int k, int q) {
            if (8 * q + 7 > k && 8 * q + warp > k) a[q] = fma(colM[k][lane], colA[k][8 * q + warp], a[q]);
        };
        auto update_b = [&](int k) {
            if (24 + warp > k) ab = fma(colM[k][row], colA[k][jb], ab);
        };
#pragma unroll
        for (int k = 0; k < PB - 1; k++) {
            const int k1 = k + 1, k2 = k + 2;
            if (warp == (k1 & 7)) {
                bar_wait(1 + (k & 7), 64);
                const double d = colA[k][k];
                const int i = k1 < 16 ? lane : row;
                const double c = colA[k][i], c1 = colA[k][k1 < 16 ? k1 : jb];
                const double r = potrf_recip(d);
                if (k > 0) {   // step k - 1, for column k + 1
                    wait(barM + k - 1);
                    if (k1 < 16) update_a(k - 1, (k1 >> 3) & 1);
                    else update_b(k - 1);
                }
                const double x = k1 < 16 ? a[(k1 >> 3) & 1] : ab;
                double m = -(c * r), v = fma(m, c1, x);
                if (potrf_rare(d)) {   // uniform
                    m = -potrf_ratio(c, d);
                    v = fma(m, c1, x);
                }
                colM[k][i] = m;
                if (lane == 0) rec[k] = r;
                __syncwarp();
                if (lane == 0) gbx_tc::mbar_arrive(barM + k);
                if (k1 < 16) {
                    a[(k1 >> 3) & 1] = v;
                    colA[k1][lane] = v;
                } else {
                    ab = v;
                    if ((lane >> 4) == ((k1 >> 3) & 1)) colA[k1][row] = v;
                }
                if (k1 < PB - 1) bar_arrive(1 + (k1 & 7), 64);
                // the rest of the step before and of this one
                if (k1 < 16) {
                    if (k > 0) {
                        update_a(k - 1, 1 - ((k1 >> 3) & 1));
                        update_b(k - 1);
                    }
                    update_a(k, 1 - ((k1 >> 3) & 1));
                    update_b(k);
                }
            } else if (k1 == PB - 1 || warp != (k2 & 7)) {   // the next warp waits in its turn
                wait(barM + k);
                update_a(k, 0);
                update_a(k, 1);
                update_b(k);
            }
        }
    } else {
        const int pr = 4 * (warp - 8) + (lane & 3), pg = lane >> 2;
        double p[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int j = pg + 8 * q;
            p[q] = (r0 + pr < n && j < b) ? A[(long long)(j0 + j) * lda + r0 + pr] : 0.0;
        }
#pragma unroll
        for (int k = 0; k < PB - 1; k++) {
            const double pk = __shfl_sync(ALL, p[k >> 3], (lane & 3) + 4 * (k & 7));
            wait(barM + k);
            // every warp has had its second turn: its loads of the diagonal
            // block are done, and the last CTA to get here may overwrite it
            if (k == 24 && tid == 8 * 32) {
                __threadfence();
                s_last = atomicAdd(done, 1u) == gridDim.x - 1;
                if (s_last) *done = 0u;
            }
            const double d = colA[k][k];
            const double t = potrf_rare(d) ? -potrf_ratio(pk, d) : -(pk * rec[k]);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (8 * q + 7 <= k) continue;
                const double v = fma(t, colA[k][pg + 8 * q], p[q]);
                if (8 * q > k || pg + 8 * q > k) p[q] = v;
            }
        }
#pragma unroll
        for (int q = 0; q < 4; q++) colP[pg + 8 * q][pr] = p[q];
    }
    __syncthreads();
    if (s_failed) {   // uniform: nothing is stored, and the host is told
        if (tid == 0) {
            *(volatile int *)status_host = *(volatile int *)status;
            __threadfence_system();
        }
        return;
    }
    // 1-based column of the first non-positive pivot (zero, negative or NaN, by
    // the bit pattern), or 0; every warp gets the same answer
    const double d = colA[lane][lane];
    const unsigned neg =
        __ballot_sync(0xffffffffu, (unsigned long long)__double_as_longlong(d) - 1ull >= 0x7ff0000000000000ull);
    const int bad = __ffs((int)neg);
    if (tid == 0 && s_last && bad) atomicCAS(info, 0, j0 + bad);
    if (bad) return;
    if (warp == 0) rec[lane] = rsqrt(d);   // L_ik = a_ik / sqrt(d_k)
    __syncthreads();
    for (int t = tid; t < PR * PB; t += PT_THREADS) {
        const int q = t % PR, k = t / PR;
        if (r0 + q < n && k < b) A[(long long)(j0 + k) * lda + r0 + q] = colP[k][q] * rec[k];
    }
    // all CTAs hold the same factor; the last to have read the block writes it
    if (!s_last) return;
    for (int k = warp; k < b; k += PT_THREADS / 32)
        if (lane < b && k <= lane) D[(long long)k * lda + lane] = colA[k][lane] * rec[k];
}

// A22 (m x m, lower) -= A21 A21^T with A21 m x PB: one 16 x 16 tile of the
// lower triangle per CTA, blockIdx.x enumerating the tiles (ti >= tj) row by
// row; the two 16 x PB row blocks of A21 are staged in shared memory.
__global__ void __launch_bounds__(256)
potrf_syrk(int m, const double *A21, double *A22, long long lda)
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
        launch_pdl(potrf_step, grid, PT_THREADS, 0, s, n, j0, A, lda, info, done, words, mirror);
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
