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
//   * DTRSV: one cooperative launch in which every CTA owns 16 rows of a block
//     and passes its part of the solution to the later blocks through global
//     memory as soon as it is known (see trsv_solve).
#include "gbx_internal.h"
#include "gemm_host.h"
#include "launch.cuh"
#include "tri_inverse.cuh"

#include <cuda_runtime.h>
#include <stdint.h>
#include <algorithm>

namespace {

using gbx_launch::launch_pdl_short;

inline cudaStream_t S(gbx_ctx *ctx) { return (cudaStream_t)gbx_ctx_get_stream(ctx); }
inline long long base_off(int n, int inc) { return inc >= 0 ? 0 : (long long)(n - 1) * (-inc); }

// ------------------------------------------------------------------- DGER
constexpr int GER_ROWS = 512, GER_COLS = 32;

// 512 rows x `width` (at most 32) columns per CTA, two rows per thread, eight
// columns' loads in flight.  The bound is HBM (16 bytes per element and one DFMA:
// the FP64 pipe alone would take two thirds of that time), so nothing else per
// element may use the FP64 pipe: alpha y_j is formed once per CTA and the
// test for a zero y_j (netlib leaves that column alone) is a bit in an
// integer mask.  With the product and the test per element the FP64 pipe was
// the bound: 8192 x 8192 took 387 us, now 156 us (1.07 GB, 6.9 TB/s).
// A row count that leaves threads without their second row, or zeros in y, takes
// the same batches of eight: one column at a time, 300 x 4000 took 25 us, now 11.
// vec: A is 16-byte aligned and lda even, so that a thread's two adjacent
// rows are one 128-bit access in every column.
__global__ void __launch_bounds__(256)
ger_kernel(int m, int n, int width, double alpha, const double *x, int incx, const double *y, int incy, double *A,
           long long lda, int vec)
{
    gbx_launch::pdl_enter();
    __shared__ double coef[GER_COLS];
    __shared__ unsigned s_keep;
    const int c0 = blockIdx.y * width, cols = min(width, n - c0);
    const int tid = threadIdx.x;
    if (tid < 32) {
        const double yj = tid < cols ? y[(long long)(c0 + tid) * incy] : 0.0;
        coef[tid] = alpha * yj;
        // y_j != 0 on the bit pattern (NaN counts as nonzero)
        const unsigned keep = __ballot_sync(0xffffffffu, (__double_as_longlong(yj) << 1) != 0);
        if (tid == 0) s_keep = keep;
    }
    __syncthreads();
    const unsigned keep = s_keep;   // no bit beyond cols
    // vec: rows r, r + 1 with r even; otherwise rows r and r + 256
    const int r = blockIdx.x * GER_ROWS + (vec ? 2 * tid : tid);
    const int r2 = vec ? r + 1 : r + 256;
    if (r >= m) return;
    double *ap = A + (long long)c0 * lda + r;
    const bool two = r2 < m;
    const double x0 = x[(long long)r * incx];
    const double x1 = two ? x[(long long)r2 * incx] : 0.0;
    if (vec && two) {
#pragma unroll 1
        for (int j = 0; j < cols; j += 8) {
            double2 v[8];
#pragma unroll
            for (int u = 0; u < 8; u++)
                if (keep >> (j + u) & 1) v[u] = *(const double2 *)(ap + (j + u) * lda);
#pragma unroll
            for (int u = 0; u < 8; u++)
                if (keep >> (j + u) & 1) {
                    const double c = coef[j + u];
                    v[u].x = fma(x0, c, v[u].x);
                    v[u].y = fma(x1, c, v[u].y);
                    *(double2 *)(ap + (j + u) * lda) = v[u];
                }
        }
        return;
    }
#pragma unroll 1
    for (int j = 0; j < cols; j += 8) {
        double v[8], w[8];
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (keep >> (j + u) & 1) {
                v[u] = ap[(j + u) * lda];
                if (two) w[u] = ap[(j + u) * lda + 256];
            }
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (keep >> (j + u) & 1) {
                const double c = coef[j + u];
                ap[(j + u) * lda] = fma(x0, c, v[u]);
                if (two) ap[(j + u) * lda + 256] = fma(x1, c, w[u]);
            }
    }
}

// ------------------------------------------------------------------ DSYMV
constexpr int SY_T = 64;

// One tile (I, J) of the stored triangle per CTA (I >= J for lower, I <= J
// for upper in block indices).  Writes the row partial (A_IJ x_J, 64 values)
// to part[I][J] and, off the diagonal, the column partial (A_IJ^T x_I) to
// part[J][I]; part[b][q] is the q-th partial of output block b.
__global__ void __launch_bounds__(256)
symv_tiles(int n, int nb, int lower, const double *A, long long lda, const double *x,
           int incx, double *part)
{
    gbx_launch::pdl_enter();
    __shared__ double s[SY_T][SY_T + 1];
    __shared__ double sxI[SY_T], sxJ[SY_T];
    __shared__ double red[4][SY_T];
    // tile index -> (I, J) with I >= J (lower) in row-major triangle order
    // (FP32 square root and integer correction: an FP64 one by every thread
    // cost the FP64 pipe nearly half as much as the tile's products:
    // n = 8192 took 198 us, then 136)
    const int t = blockIdx.x;
    int I = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
    while ((long long)(I + 1) * (I + 2) / 2 <= t) I++;
    while ((long long)I * (I + 1) / 2 > t) I--;
    int J = (int)(t - (long long)I * (I + 1) / 2);
    if (!lower) { const int tmp = I; I = J; J = tmp; }   // upper: I <= J
    const int r0 = I * SY_T, c0 = J * SY_T;
    const int tid = threadIdx.x;
    double v[SY_T * SY_T / 256];   // all loads in flight before the first store to shared memory:
    // n = 300 7.3 us instead of 13.9, n = 8192 125 instead of 136
#pragma unroll
    for (int f = 0; f < SY_T * SY_T / 256; f++) {
        const int q = tid + f * 256, i = q % SY_T, j = q / SY_T;
        const int gi = r0 + i, gj = c0 + j;
        v[f] = 0.0;
        if (gi < n && gj < n) {
            const bool stored = I != J || (lower ? gi >= gj : gi <= gj);   // else its mirror image
            v[f] = stored ? A[(long long)gj * lda + gi] : A[(long long)gi * lda + gj];
        }
    }
#pragma unroll
    for (int f = 0; f < SY_T * SY_T / 256; f++) s[(tid + f * 256) % SY_T][(tid + f * 256) / SY_T] = v[f];
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
symv_finish(int n, int nb, const double *part, double alpha, double beta, double *y,
            int incy)
{
    gbx_launch::pdl_enter();
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
constexpr int TV_NB = gbx_tri::NB, TV_LD = gbx_tri::LD, TV_THREADS = 256;
constexpr int TV_TILE = TV_NB * TV_LD;
constexpr int TV_R = 16, TV_SL = TV_NB / TV_R, TV_RLD = TV_R + 1;   // rows and number of a block's slices
constexpr int TV_STAGES = 8, TV_WT = 8 * TV_RLD;   // a warp's ring: 16 rows x 8 columns per stage
constexpr int TV_RED = TV_R * 18;
constexpr int TV_W1 = 3 * TV_NB * TV_RLD + 8 * TV_STAGES * TV_WT + 2 * TV_RED;   // for a slice
constexpr int TV_W2 = 2 * TV_TILE + 32 * 33;                                    // to invert a block
constexpr size_t TV_SMEM = sizeof(double) * (TV_TILE + (TV_W1 > TV_W2 ? TV_W1 : TV_W2));
constexpr int TV_FOLD = 8;
constexpr unsigned long long TV_TIMEOUT_NS = 2000000000ull;
constexpr int TV_TIMEOUT_CODE = 9;

struct TrsvArgs {
    int n, nblk, fwd, tr, unit, incx;
    const double *A;
    long long lda;
    double *x;          // element 0 of the vector
    double *xw;         // solution in solve order, nblk * 64 values, all bits set until known
    double *zw;         // b - (the blocks subtracted one by one), likewise
    double *inv;        // inverted diagonal blocks, element (i, k) at [64 k + i]
    int *ready;         // per block: all bits set until its inverse is there, then 1 if M may be used, else 0
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

// Row of its block that is row r of slice sl: eight from the block's upper half
// and eight from the lower, so that the triangular work of the slices is equal.
__device__ __forceinline__ int tv_row(int sl, int r) { return r < 8 ? 8 * sl + r : 48 - 8 * sl + r; }

// A lane's share of the copy of a slice's 16 x 8 parts, columns c0 + 64 K .. of
// block row s, to dst[k * 17 + i]: four elements whose addresses differ by
// off[], 64 columns further per block.
struct TvPart {
    const double *src, *any;
    long long off[3], kstep;
    int dst, dstep, ok;

    __device__ __forceinline__ TvPart(const TrsvArgs &a, int s, int sl, int c0, int lane)
    {
        const int k0 = a.tr ? lane & 7 : lane >> 4, i0 = a.tr ? lane >> 3 : lane & 15;
        const long long col = a.fwd ? a.lda : -a.lda;   // one column (N) or row (T) on
        any = a.A;
        ok = 0;
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (s * TV_NB + tv_row(sl, i0 + (a.tr ? 4 * u : 0)) < a.n) ok |= 1 << u;
        // (a lane whose first row is beyond n reads nothing)
        src = tv_at(a, min(s * TV_NB + tv_row(sl, i0), a.n - 1), c0 + k0);
#pragma unroll
        for (int u = 1; u < 4; u++)
            off[u - 1] = col * (a.tr ? tv_row(sl, i0 + 4 * u) - tv_row(sl, i0) : 2 * u);
        kstep = TV_NB * (a.tr ? (a.fwd ? 1 : -1) : col);
        dst = k0 * TV_RLD + i0;
        dstep = a.tr ? 4 : 2 * TV_RLD;
    }
    // the next block's part
    __device__ __forceinline__ void fetch(double *ring)
    {
        double *d = ring + dst;
        tv_copy8(d, ok & 1 ? src : any, ok & 1);
#pragma unroll
        for (int u = 1; u < 4; u++) tv_copy8(d + u * dstep, ok >> u & 1 ? src + off[u - 1] : any, ok >> u & 1);
        src += kstep;
    }
};

// Values that other CTAs publish are their own flags: a value is stored over
// the "all bits set" pattern.  Waits until the lanes of `mask` hold theirs
// (v: loaded before, p: this lane's address).  A wait that lasts 2 s gives
// up: the status word is set and the values become NaN, so that every later
// block still finishes.
__device__ __forceinline__ double tv_load(const double *p) { return *(const volatile double *)p; }
__device__ __forceinline__ void tv_timeout(const TrsvArgs &a)
{
    atomicCAS(a.status, 0, TV_TIMEOUT_CODE);
    *(volatile int *)a.status_host = TV_TIMEOUT_CODE;
    __threadfence_system();
}
__device__ __forceinline__ double tv_wait(const TrsvArgs &a, const double *p, double v, unsigned mask, int lane)
{
    const bool mine = mask >> lane & 1;
    if (!__any_sync(0xffffffffu, mine && __double_as_longlong(v) == -1ll)) return v;
    const unsigned long long t0 = tv_now();
    while (true) {
        if (mine && __double_as_longlong(v) == -1ll) v = tv_load(p);
        if (!__any_sync(0xffffffffu, mine && __double_as_longlong(v) == -1ll)) return v;
        if (__any_sync(0xffffffffu, tv_now() - t0 > TV_TIMEOUT_NS)) {
            if (lane == 0) tv_timeout(a);
            return __longlong_as_double(0x7ff8000000000000ll);
        }
    }
}
__device__ __forceinline__ void tv_publish(double *p, double r)
{
    // the "not yet known" pattern is a NaN: another NaN in its place
    *(volatile double *)p = __double_as_longlong(r) == -1ll ? __longlong_as_double(0x7ff8000000000000ll) : r;
}

// Waits for the inverse of block s and starts the copy of the slice's rows of
// it to dst[k * 17 + i], *fold: M may be used for it; by the whole CTA.
__device__ __forceinline__ void tv_fetch_inv(const TrsvArgs &a, double *dst, int s, int sl, int *fold)
{
    const int tid = threadIdx.x;
    if (tid == 0) {
        const unsigned long long t0 = tv_now();
        int r;
        while ((r = *(volatile int *)(a.ready + s)) < 0)
            if (tv_now() - t0 > TV_TIMEOUT_NS) {
                tv_timeout(a);
                break;
            }
        *fold = r > 0;
        __threadfence();
    }
    __syncthreads();
    const double *src = a.inv + (size_t)s * TV_NB * TV_NB + tv_row(sl, tid & 15);
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const int k = (tid >> 4) + 16 * u;
        tv_copy8(dst + k * TV_RLD + (tid & 15), src + k * TV_NB, 1);
    }
}

// Sum over the CTA of the 16 values that its threads (row lane & 15, columns
// 4 (2 warp + lane / 16) ..) have for each row: in warps 0-3, lanes 4 r' + ..:
// row 4 warp + (lane & 3).
__device__ __forceinline__ double tv_sum(double *red, double v, int lane, int warp)
{
    red[(2 * warp + (lane >> 4)) * 18 + (lane & 15)] = v;
    __syncthreads();
    double r = 0.0;
    if (warp < 4) {
        const double *q = red + 2 * (lane >> 2) * 18 + 4 * warp + (lane & 3);
        r = q[0] + q[18];
        r += __shfl_xor_sync(0xffffffffu, r, 4);
        r += __shfl_xor_sync(0xffffffffu, r, 8);
        r += __shfl_xor_sync(0xffffffffu, r, 16);
    }
    return r;
}

// x := T^-1 x, blocks of 64 rows in solve order, each in four slices of 16
// rows (tv_row); CTA b owns slices b, b + gridDim.x, ...  All CTAs are resident
// (cooperative launch).  A slice waits for earlier blocks and for sums of its
// own block's slices, which wait for earlier blocks only.
//   * The CTAs invert the diagonal blocks first, CTA b block b (again before
//     every fourth slice, for as many blocks as the next four rounds reach).
//   * A slice subtracts T(s, K) x_K for every earlier block K as x_K appears:
//     warp w columns 8 w .. 8 w + 7 of each, prefetched seven blocks deep into
//     its own ring (they do not depend on x), without barriers.
//   * The four slices exchange z = b - sum through zw; x_s = inv z goes to the
//     later blocks through xw and to x.
//   * From block TV_FOLD on, for well-conditioned diagonal blocks (whose inverse was
//     joined), M = inv T(s, s-1) is formed beforehand, so that x_s = inv (b - sum over
//     K < s-1) - M x_(s-1): the exchange and the inverse lie before x_(s-1), which
//     needs one product.  It multiplies b - sum and T x by the inverse before they
//     cancel, so its backward error grows with the condition number (against the form
//     without M, 400 triangles: up to 16 both stay below 2 u; at 16 to 64 20 times as
//     much, at 1e7 400 times).
// What bounds it: the chain over the blocks, each link one hand-over through
// L2 and the product with x_(s-1), 1.2 us; for the last blocks the FP64 pipe,
// which takes 0.33 us for each 16 x 64 part and 11 us for M.  (With a block per
// CTA, 1.3 us of the pipe for each 64 x 64 part, a link took 2.3 us; two CTAs
// per SM fill the pipe but share it with the link: n = 8192 6 % slower, 16000
// 10 % faster.)  n = 8192: N or T 300 us with a block per CTA, now 208
// to 218 (by where the exchanged words lie); without M, for ill-conditioned blocks, 334.  M for
// every block from the 8th on: from the 12th n = 2000 is 3 us slower, from the
// 6th all sizes the same.
__global__ void __launch_bounds__(TV_THREADS)
trsv_solve(TrsvArgs a)
{
    extern __shared__ __align__(16) double tv_sm[];
    __shared__ int s_fold[2];
    double *T1 = tv_sm;                              // T(s, s-1)
    double *work = T1 + TV_TILE;                     // to invert a block
    double *Ia = work;                               // the slice's rows of the inverse, [k * 17 + i]: two
    double *Ms = Ia + 2 * TV_NB * TV_RLD;            // of M, likewise
    double *ring = Ms + TV_NB * TV_RLD;
    double *red = ring + 8 * TV_STAGES * TV_WT;      // two sums
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int i = lane & 15, h4 = 4 * (lane >> 4);   // row; columns 8 warp + h4 .. + 3
    ring += warp * TV_STAGES * TV_WT;
    const int r16 = (4 * warp + (lane & 3)) & 15;    // row of the sums, warps 0-3
    const bool out = warp < 4 && lane < 4;

    int round = 0;
    for (int t = blockIdx.x; t < TV_SL * a.nblk; t += gridDim.x, round++) {
        const int ib = blockIdx.x + round / TV_SL * gridDim.x;
        if (round % TV_SL == 0 && ib < a.nblk) {
            double *D = work, *X = D + TV_TILE;
#pragma unroll
            for (int f = 0; f < TV_NB * TV_NB / TV_THREADS; f++) {   // identity beyond n
                const int e = tid + f * TV_THREADS, u = e & 63, v = e >> 6;
                const int r = a.tr ? v : u, k = a.tr ? u : v;
                const int pr = ib * TV_NB + r, pk = ib * TV_NB + k;
                const int in = k <= r && pr < a.n && !(a.unit && r == k);
                if (in) tv_copy8(D + k * TV_LD + r, tv_at(a, pr, pk), 1);
                else D[k * TV_LD + r] = r == k ? 1.0 : 0.0;
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            const int may = gbx_tri::invert64<true>(D, X, X + TV_TILE);
            double *o = a.inv + (size_t)ib * TV_NB * TV_NB;
            for (int e = tid; e < TV_NB * TV_NB; e += TV_THREADS) o[e] = X[(e >> 6) * TV_LD + (e & 63)];
            __threadfence();
            __syncthreads();
            if (tid == 0) *(volatile int *)(a.ready + ib) = may;
        }
        const int s = t / TV_SL, sl = t % TV_SL;
        const int row = s * TV_NB + tv_row(sl, r16);
        double *I = Ia + (round & 1) * TV_NB * TV_RLD;
        if (s >= TV_FOLD && round == 0) tv_fetch(a, T1, s, s - 1);
        if (round % TV_SL == 0) tv_fetch_inv(a, I, s, sl, s_fold + (round & 1));
        asm volatile("cp.async.commit_group;" ::: "memory");
        const bool fold = s >= TV_FOLD && s_fold[round & 1];   // the same in all slices of the block
        const int nk = fold ? s - 1 : s;                 // blocks subtracted one by one
        TvPart part(a, s, sl, 8 * warp, lane);
#pragma unroll 1
        for (int f = 0; f < TV_STAGES - 1; f++) {
            if (f < nk) part.fetch(ring + f * TV_WT);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        double b = 0.0;
        const long long xi = (long long)(a.fwd ? row : a.n - 1 - row) * a.incx;
        if (out && row < a.n) b = a.x[xi];
        asm volatile("cp.async.wait_group %0;" ::"n"(TV_STAGES - 1) : "memory");   // T1, I
        __syncthreads();
        double M[4];
        if (fold) {
            // warps 0-3 have the slice's upper eight rows, 4-7 the lower: the
            // inverse is lower triangular.  Thread: one row, four columns.
            const int m8 = (lane & 7) + 8 * (warp >> 2), c4 = 16 * (warp & 3) + 4 * (lane >> 3);
            const int jend = 8 * (warp < 4 ? sl + 1 : 8 - sl);
            const double *c = T1 + c4 * TV_LD;
#pragma unroll
            for (int k = 0; k < 4; k++) M[k] = 0.0;
            for (int j = 0; j < jend; j++) {
                const double v = I[j * TV_RLD + m8];
#pragma unroll
                for (int k = 0; k < 4; k++) M[k] = fma(v, c[k * TV_LD + j], M[k]);
            }
#pragma unroll
            for (int k = 0; k < 4; k++) Ms[(c4 + k) * TV_RLD + m8] = M[k];
        }
        __syncthreads();
        if (fold) {
#pragma unroll
            for (int k = 0; k < 4; k++) M[k] = -Ms[(8 * warp + h4 + k) * TV_RLD + i];
        }
        const int sn = (t + gridDim.x) / TV_SL;          // the next slice's
        if (sn < a.nblk && sn >= TV_FOLD) tv_fetch(a, T1, sn, sn - 1);
        if (sn < a.nblk && (round + 1) % TV_SL != 0)
            tv_fetch_inv(a, Ia + ((round + 1) & 1) * TV_NB * TV_RLD, sn, sl, s_fold + ((round + 1) & 1));
        asm volatile("cp.async.commit_group;" ::: "memory");
        // x of four blocks at a time: lane 8 u + c has column 8 warp + c of block 4 g + u
        const double *xp = a.xw + (lane >> 3) * TV_NB + 8 * warp + (lane & 7);
        double acc0 = 0.0, acc1 = 0.0, xv = 0.0, xn = 0.0;
        if ((lane >> 3) < s) xn = tv_load(xp);
        auto x_of = [&](int K) {   // this warp's eight values of x_K are in lanes 8 (K & 3) ..
            if ((K & 3) == 0) {
                xv = xn;
                if (K + 4 + (lane >> 3) < s) xn = tv_load(xp + (long long)(K + 4) * TV_NB);
            }
            xv = tv_wait(a, xp + (long long)(K & ~3) * TV_NB, xv, 0xffu << 8 * (K & 3), lane);
        };
        for (int K = 0; K < nk; K++) {
            if (K + TV_STAGES - 1 < nk) part.fetch(ring + (K + TV_STAGES - 1) % TV_STAGES * TV_WT);
            asm volatile("cp.async.commit_group;" ::: "memory");
            x_of(K);
            asm volatile("cp.async.wait_group %0;" ::"n"(TV_STAGES - 1) : "memory");
            __syncwarp();
            const double *T = ring + K % TV_STAGES * TV_WT + h4 * TV_RLD + i;
            const int l = 8 * (K & 3) + h4;
            acc0 = fma(T[0], __shfl_sync(0xffffffffu, xv, l), acc0);
            acc1 = fma(T[TV_RLD], __shfl_sync(0xffffffffu, xv, l + 1), acc1);
            acc0 = fma(T[2 * TV_RLD], __shfl_sync(0xffffffffu, xv, l + 2), acc0);
            acc1 = fma(T[3 * TV_RLD], __shfl_sync(0xffffffffu, xv, l + 3), acc1);
            __syncwarp();   // the stage may be overwritten
        }
        const double sum = tv_sum(red, acc0 + acc1, lane, warp);
        if (out) tv_publish(a.zw + row, b - sum);
        double v0 = 0.0, v1 = 0.0;
        if (warp < 8 - sl) {   // the rows end at column 63 - 8 sl
            const double *zp = a.zw + (long long)s * TV_NB + 8 * warp + (lane & 7);
            const double z = tv_wait(a, zp, tv_load(zp), 0xffffffffu, lane);
            const double *c = I + (8 * warp + h4) * TV_RLD + i;
            v0 = fma(c[0], __shfl_sync(0xffffffffu, z, h4), v0);
            v1 = fma(c[TV_RLD], __shfl_sync(0xffffffffu, z, h4 + 1), v1);
            v0 = fma(c[2 * TV_RLD], __shfl_sync(0xffffffffu, z, h4 + 2), v0);
            v1 = fma(c[3 * TV_RLD], __shfl_sync(0xffffffffu, z, h4 + 3), v1);
            v0 += v1;
            v1 = 0.0;
        }
        if (fold) {
            x_of(s - 1);
            const int l = 8 * ((s - 1) & 3) + h4;
            v0 = fma(M[0], __shfl_sync(0xffffffffu, xv, l), v0);
            v1 = M[1] * __shfl_sync(0xffffffffu, xv, l + 1);
            v0 = fma(M[2], __shfl_sync(0xffffffffu, xv, l + 2), v0);
            v1 = fma(M[3], __shfl_sync(0xffffffffu, xv, l + 3), v1);
            v0 += v1;
        }
        const double r = tv_sum(red + TV_RED, v0, lane, warp);
        if (out) {
            tv_publish(a.xw + row, r);
            if (row < a.n) a.x[xi] = r;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();   // shared memory is reused by the next slice
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
    // 32 columns per CTA, 16 or 8 as long as there is at most one CTA per SM
    // (1000 x 800: 9.6 us with 32, 6.7 with 16)
    dim3 g((m + GER_ROWS - 1) / GER_ROWS, (n + GER_COLS - 1) / GER_COLS);
    int width = GER_COLS;
    while (width > 8 && (long long)g.x * ((n + width / 2 - 1) / (width / 2)) <= gbx_ctx_sms(ctx)) width /= 2;
    g.y = (n + width - 1) / width;
    if (g.y > 65535) return gbx_fail(ctx, GBX_ERR_UNSUPPORTED, "DGER: n too large");
    gbx_timer_begin(ctx, GBX_TIMER_GEMV);
    const int vec = (((uintptr_t)A) & 15) == 0 && lda % 2 == 0;
    launch_pdl_short(gbx_ctx_sms(ctx), ger_kernel, g, 256, S(ctx), m, n, width, alpha, x + base_off(m, incx), incx,
                     y + base_off(n, incy), incy, A, lda, vec);
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
        launch_pdl_short(gbx_ctx_sms(ctx), symv_tiles, dim3((unsigned)tiles), 256, S(ctx), n, nb, gbx_lsame(uplo, 'L'), A,
                         lda, xb, incx, part);
        gbx_timer_end(ctx);
        gbx_count_launch(ctx, 1);
    } else {
        cudaMemsetAsync(part, 0, sizeof(double) * (size_t)nb * nb * SY_T, S(ctx));
    }
    launch_pdl_short(gbx_ctx_sms(ctx), symv_finish, dim3(nb), 4 * SY_T, S(ctx), n, nb, part, alpha, beta, yb, incy);
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
    // the inverses; x and z in solve order and the blocks' ready words (eight bytes
    // each).  A capture cannot allocate: without the second slot they lie behind the
    // inverses, in the slack of a slot that DTRSM of this order has used.  (Not
    // always there: n = 1000 51 -> 53 us, 7000 183 -> 188, 8000 215 -> 211.)
    const size_t ibytes = sizeof(double) * (size_t)nblk * TV_NB * TV_NB;
    const size_t wbytes = sizeof(double) * (size_t)nblk * (2 * TV_NB + 1);
    const bool behind = !gbx_ws_ready(ctx, GBX_WS_TMP2, wbytes) && gbx_ws_ready(ctx, GBX_WS_TMP1, ibytes + wbytes) &&
                        gbx_capturing(ctx);
    if ((st = gbx_ws(ctx, GBX_WS_TMP1, ibytes, (void **)&p.inv)) != GBX_OK) return st;
    if (behind) xw = p.inv + ibytes / sizeof(double);
    else if ((st = gbx_ws(ctx, GBX_WS_TMP2, wbytes, (void **)&xw)) != GBX_OK) return st;
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
    p.zw = xw + (size_t)nblk * TV_NB;
    p.ready = (int *)(p.zw + (size_t)nblk * TV_NB);
    // every value "not yet known" (all bits set)
    cudaError_t e = cudaMemsetAsync(xw, 0xFF, wbytes, S(ctx));
    // a per-device function attribute; setting it is a cheap host call
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(trsv_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TV_SMEM);
    if (e != cudaSuccess) return gbx_fail(ctx, GBX_ERR_CUDA, "dtrsv: %s", cudaGetErrorString(e));
    // one CTA per SM is always resident; whole blocks, so that a block's slices run side by side
    const int grid = TV_SL * std::min(nblk, std::max(1, gbx_ctx_sms(ctx) / TV_SL));
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
