// l1.cu — Level-1 streaming kernels: daxpy, ddot, dnrm2, idamax, idamin, dscal.
//
// Replaces the reference's (dead, never-built) cuBLAS Level-1 wrappers
// blas_level1/axpy.cc:10-50, dot.cc:9-48, nrm2.cc:9-41, amax.cc:32-43,
// amin.cc:32-43.  All of them are HBM-bound: the kernels read each element
// once with 128-bit loads when the pointers allow it, run a grid sized to a
// multiple of the SM count, and reduce deterministically (a fixed partition
// into per-block partials, which the block that finishes last combines in a
// fixed order), so repeated calls give bit-identical results.  One launch per
// call, placed before the previous call's kernel has drained (launch.cuh): the
// vector work of a CG iteration (DDOT, two DAXPYs, DNRM2, IDAMAX) on vectors of
// 10,001 elements takes 17 us, in eight serial launches 39 us.
#include "gbx_internal.h"
#include "l1_kernels.cuh"

#include <cuda_runtime.h>
#include <algorithm>

using namespace gbx_l1;
using gbx_launch::launch_pdl;

namespace {

inline int grid_for(gbx_ctx *ctx, long long n, int per_thread)
{
    long long want = (n + (long long)L1_THREADS * per_thread - 1) / ((long long)L1_THREADS * per_thread);
    long long cap = (long long)gbx_ctx_sms(ctx) * L1_BLOCKS_PER_SM;
    if (want < 1) want = 1;
    return (int)(want < cap ? want : cap);
}

inline cudaStream_t S(gbx_ctx *ctx) { return (cudaStream_t)gbx_ctx_get_stream(ctx); }

// Blocks of a reduction: two elements per thread, so that the loads and FP64
// operations of a short vector spread over as many SMs as there are (eight per
// thread kept a vector of 10,000 on five of them), up to one block per SM; beyond
// that eight per thread, because every block takes its turn at the count of
// finished blocks (300,000 elements: 586 blocks 8.5 us, 152 5.5).
inline int reduction_grid(gbx_ctx *ctx, long long n)
{
    return std::max(grid_for(ctx, n, 8), std::min(grid_for(ctx, n, 2), gbx_ctx_sms(ctx)));
}

// Partials (at most three values per block) and counter of a reduction.  One block
// needs neither; its call allocates them all the same, so that any reduction can be
// captured on a context that has run one.
template <typename P>
gbx_status reduction_ws(gbx_ctx *ctx, int g, P **part, gbx_red *red)
{
    const size_t bytes = 3 * sizeof(double) * (size_t)gbx_ctx_sms(ctx) * L1_BLOCKS_PER_SM;
    *part = nullptr;
    *red = gbx_red{};
    if (g > 1) return gbx_reduction(ctx, bytes, (void **)part, red);
    return gbx_reduction_reserve(ctx, bytes);
}

// element offset of the first element a kernel should touch: netlib walks a
// negative-increment vector from its far end.
inline long long base_off(int n, int inc) { return inc >= 0 ? 0 : (long long)(n - 1) * (-inc); }

}  // namespace

extern "C" gbx_status gbx_daxpy(gbx_ctx *ctx, int n, double alpha, const double *x, int incx,
                                double *y, int incy)
{
    if (!ctx) return GBX_ERR_ARG;
    if (n <= 0 || alpha == 0.0) return GBX_OK;
    int g = grid_for(ctx, n, 2);
    gbx_timer_begin(ctx, GBX_TIMER_LEVEL1);
    if (incx == 1 && incy == 1) {
        launch_pdl(axpy_unit, g, L1_THREADS, 0, S(ctx), n, alpha, x, y);
    } else {
        launch_pdl(axpy_strided, g, L1_THREADS, 0, S(ctx), n, alpha, x + base_off(n, incx), incx,
                                                    y + base_off(n, incy), incy);
    }
    gbx_timer_end(ctx);
    gbx_count_launch(ctx, 1);
    return gbx_check_launch(ctx, "daxpy");
}

extern "C" gbx_status gbx_dscal(gbx_ctx *ctx, int n, double alpha, double *x, int incx)
{
    if (!ctx) return GBX_ERR_ARG;
    if (n <= 0 || incx <= 0 || alpha == 1.0) return GBX_OK;
    int g = grid_for(ctx, n, 4);
    launch_pdl(scal_kernel, g, L1_THREADS, 0, S(ctx), n, alpha, x, incx);
    gbx_count_launch(ctx, 1);
    return gbx_check_launch(ctx, "dscal");
}

extern "C" gbx_status gbx_ddot(gbx_ctx *ctx, int n, const double *x, int incx,
                               const double *y, int incy, double *res)
{
    if (!ctx || !res) return GBX_ERR_ARG;
    if (n <= 0) {
        zero_result<<<1, 1, 0, S(ctx)>>>(res);
        gbx_count_launch(ctx, 1);
        return gbx_check_launch(ctx, "ddot");
    }
    const int g = reduction_grid(ctx, n);
    double *part;
    gbx_red red;
    gbx_status st = reduction_ws(ctx, g, &part, &red);
    if (st != GBX_OK) return st;
    gbx_timer_begin(ctx, GBX_TIMER_LEVEL1);
    launch_pdl(dot_kernel, g, L1_THREADS, 0, S(ctx), n, x + base_off(n, incx), incx, y + base_off(n, incy), incy, part, red, res);
    gbx_timer_end(ctx);
    gbx_count_launch(ctx, 1);
    return gbx_check_launch(ctx, "ddot");
}

extern "C" gbx_status gbx_dnrm2(gbx_ctx *ctx, int n, const double *x, int incx, double *res)
{
    if (!ctx || !res) return GBX_ERR_ARG;
    if (n < 1 || incx < 1) {
        zero_result<<<1, 1, 0, S(ctx)>>>(res);
        gbx_count_launch(ctx, 1);
        return gbx_check_launch(ctx, "dnrm2");
    }
    const int g = reduction_grid(ctx, n);
    double *part;
    gbx_red red;
    gbx_status st = reduction_ws(ctx, g, &part, &red);
    if (st != GBX_OK) return st;
    gbx_timer_begin(ctx, GBX_TIMER_LEVEL1);
    launch_pdl(nrm2_kernel, g, L1_THREADS, 0, S(ctx), n, x, incx, part, red, res);
    gbx_timer_end(ctx);
    gbx_count_launch(ctx, 1);
    return gbx_check_launch(ctx, "dnrm2");
}

static gbx_status iamax_common(gbx_ctx *ctx, int n, const double *x, int incx, int *res, bool is_min)
{
    if (!ctx || !res) return GBX_ERR_ARG;
    if (n < 1 || incx <= 0) {
        zero_index<<<1, 1, 0, S(ctx)>>>(res);
        gbx_count_launch(ctx, 1);
        return gbx_check_launch(ctx, is_min ? "idamin" : "idamax");
    }
    const int g = reduction_grid(ctx, n);
    unsigned long long *keys;
    gbx_red red;
    gbx_status st = reduction_ws(ctx, g, &keys, &red);
    if (st != GBX_OK) return st;
    long long *idx = g > 1 ? (long long *)(keys + g) : nullptr;
    gbx_timer_begin(ctx, GBX_TIMER_LEVEL1);
    if (is_min) launch_pdl(iamax_kernel<true>, g, L1_THREADS, 0, S(ctx), n, x, incx, keys, idx, red, res);
    else launch_pdl(iamax_kernel<false>, g, L1_THREADS, 0, S(ctx), n, x, incx, keys, idx, red, res);
    gbx_timer_end(ctx);
    gbx_count_launch(ctx, 1);
    return gbx_check_launch(ctx, is_min ? "idamin" : "idamax");
}

extern "C" gbx_status gbx_idamax(gbx_ctx *ctx, int n, const double *x, int incx, int *res)
{
    return iamax_common(ctx, n, x, incx, res, false);
}

extern "C" gbx_status gbx_idamin(gbx_ctx *ctx, int n, const double *x, int incx, int *res)
{
    return iamax_common(ctx, n, x, incx, res, true);
}
