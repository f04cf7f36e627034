// gemm_small.cu — FP64 GEMM launches of at most one CTA per SM: the core's tiles
// launched so that they overlap the end of the kernel before them, and a
// half-height tile for products (SGEMM's too) that would leave most SMs idle.  (Not larger
// ones: CTAs placed while the kernel before still runs spread unevenly over the
// SMs, and the FP64 pipe of the fullest SM sets the time: DGEMM 756 x 330 x 1710,
// 1008 tiles, took 873 us overlapped and 769 not.)
#include "gbx_internal.h"
#include "gemm_host.h"
#include "launch.cuh"

#include <cuda_runtime.h>

using namespace gbx_gemm;
using gbx_launch::launch_pdl;
using gbx_launch::pdl_enter;

namespace {

// 8 x 16 tile of a full C = alpha op(A) op(B) + beta C by 128 threads, one
// element each.  A warp has one FP64 instruction in flight, 65 cycles each, and
// the SM's pipe takes 16 to 19 cycles per warp: the eight warps of the core's
// 16 x 16 tile take 128 to 150 cycles per k and the four of this one 65 to 77,
// the latency of the FMA chain itself; what is
// left is the latency of the loads, so a panel is 64 k deep (one round of loads
// up to K = 64) and C is fetched under the products.  Each element is one FMA
// chain over k in increasing order and the core's epilogue: the bits of any
// other tile.  DGEMM 64^3 in a stream of calls: 9.2 us with the 16 x 16 tile, 5.6
// with this one (the rate at which Python issues the calls).
constexpr int SM_BM = 8, SM_BN = 16, SM_BK = 64, SM_THREADS = SM_BM * SM_BN;

template <typename T>
__global__ void __launch_bounds__(SM_THREADS)
gemm_small_kernel(GemmArgs<T> p)
{
    pdl_enter();
    __shared__ T As[2][SM_BK][SM_BM], Bs[2][SM_BK][SM_BN];
    const int m0 = (int)(blockIdx.x % p.tiles_m) * SM_BM, n0 = (int)(blockIdx.x / p.tiles_m) * SM_BN;
    const int tid = threadIdx.x, tx = tid % SM_BN, ty = tid / SM_BN;
    const int row = m0 + ty, col = n0 + tx;
    T *cp = p.C + (long long)col * p.ldc + row;
    const bool beta0 = Ops<T>::is_zero(p.beta);
    const bool live = row < p.m && col < p.n;
    const T cold = live && !beta0 ? *cp : T(0);
    constexpr int NA = SM_BM * SM_BK / SM_THREADS, NB = SM_BN * SM_BK / SM_THREADS;
    T ra[NA], rb[NB];
    // neighbouring threads along the contiguous index: rows of A or k for A^T,
    // k for B or columns for B^T
    auto load = [&](int k0) {
#pragma unroll
        for (int q = 0; q < NA; q++) {
            const int t = tid + q * SM_THREADS;
            const int r = m0 + (p.ta ? t / SM_BK : t % SM_BM), k = k0 + (p.ta ? t % SM_BK : t / SM_BM);
            ra[q] = r < p.m && k < p.k ? p.A[p.ta ? (long long)r * p.lda + k : (long long)k * p.lda + r] : T(0);
        }
#pragma unroll
        for (int q = 0; q < NB; q++) {
            const int t = tid + q * SM_THREADS;
            const int c = n0 + (p.tb ? t % SM_BN : t / SM_BK), k = k0 + (p.tb ? t / SM_BN : t % SM_BK);
            rb[q] = c < p.n && k < p.k ? p.B[p.tb ? (long long)k * p.ldb + c : (long long)c * p.ldb + k] : T(0);
        }
    };
    auto store = [&](int s) {
#pragma unroll
        for (int q = 0; q < NA; q++) {
            const int t = tid + q * SM_THREADS;
            As[s][p.ta ? t % SM_BK : t / SM_BM][p.ta ? t / SM_BK : t % SM_BM] = ra[q];
        }
#pragma unroll
        for (int q = 0; q < NB; q++) {
            const int t = tid + q * SM_THREADS;
            Bs[s][p.tb ? t / SM_BN : t % SM_BK][p.tb ? t % SM_BN : t / SM_BK] = rb[q];
        }
    };
    T acc = T(0);
    load(0);
    store(0);
    __syncthreads();
    for (int k0 = 0, s = 0; k0 < p.k; k0 += SM_BK, s ^= 1) {
        const bool more = k0 + SM_BK < p.k;
        if (more) load(k0 + SM_BK);
#pragma unroll 1
        for (int kk = 0; kk < SM_BK && k0 + kk < p.k; kk += 8) {   // (zero padding past k)
#pragma unroll
            for (int u = 0; u < 8; u++) acc = fma(As[s][kk + u][ty], Bs[s][kk + u][tx], acc);
        }
        if (more) {
            store(s ^ 1);
            __syncthreads();
        }
    }
    if (live) *cp = beta0 ? Ops<T>::mul(p.alpha, acc) : Ops<T>::axpby(p.alpha, acc, p.beta, cold);
}

template <int TM, int BK>
__global__ void __launch_bounds__(GEMM_THREADS)
gemm_overlap_kernel(GemmArgs<double> p)
{
    pdl_enter();
    gemm_simt_tile<double, TM, TM, BK>(p, blockIdx.x);
}

}  // namespace

namespace gbx_gemm {

// The FP64 launches this file takes; bm: the core's tile (64, 32, 16).  Half-
// height tiles when 16 x 16 tiles would leave half the SMs idle and the operands
// are plain; otherwise the core's tile, overlapping, up to one CTA per SM.
bool launch_gemm_short(gbx_ctx *ctx, GemmArgs<double> p, int bm)
{
    const int sms = gbx_ctx_sms(ctx);
    cudaStream_t s = (cudaStream_t)gbx_ctx_get_stream(ctx);
    const bool plain = p.c_part == C_FULL && !p.tri_a && !p.tri_b && !p.sym_a && !p.sym_b;
    const long long t16 = ((p.m + 15LL) / 16) * ((p.n + 15) / 16);
    if (bm == 16 && plain && 2 * t16 <= sms) {
        p.tiles_m = (p.m + SM_BM - 1) / SM_BM;
        p.tiles_n = (p.n + SM_BN - 1) / SM_BN;
        launch_pdl(gemm_small_kernel<double>, (unsigned)(p.tiles_m * p.tiles_n), SM_THREADS, 0, s, p);
        return true;
    }
    p.tiles_m = (p.m + bm - 1) / bm;
    p.tiles_n = (p.n + bm - 1) / bm;
    const long long blocks = p.c_part == C_FULL ? (long long)p.tiles_m * p.tiles_n
                                                : (long long)p.tiles_m * (p.tiles_m + 1) / 2;
    if (blocks > sms || (p.c_part != C_FULL && p.m != p.n)) return false;
    launch_pdl(bm == 64 ? gemm_overlap_kernel<4, 8> : (bm == 32 ? gemm_overlap_kernel<2, 8> : gemm_overlap_kernel<1, 16>),
               (unsigned)blocks, GEMM_THREADS, 0, s, p);
    return true;
}

// SGEMM where the core's 16 x 16 tiles would leave half the SMs idle (the same
// bits again; the core loads 8 k per panel).  Through sgemm_, which waits for the
// result: 134 x 76 x 125 25 -> 22 us, 60 x 50 x 1000 56 -> 39.
bool launch_gemm_short(gbx_ctx *ctx, GemmArgs<float> p)
{
    const long long t16 = ((p.m + 15LL) / 16) * ((p.n + 15) / 16);
    if (p.c_part != C_FULL || p.tri_a || p.tri_b || p.sym_a || p.sym_b || 2 * t16 > gbx_ctx_sms(ctx)) return false;
    p.tiles_m = (p.m + SM_BM - 1) / SM_BM;
    p.tiles_n = (p.n + SM_BN - 1) / SM_BN;
    launch_pdl(gemm_small_kernel<float>, (unsigned)(p.tiles_m * p.tiles_n), SM_THREADS, 0,
               (cudaStream_t)gbx_ctx_get_stream(ctx), p);
    return true;
}

}  // namespace gbx_gemm
