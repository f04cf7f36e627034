// gemm_host.h — host-side entry points of the GEMM core shared by the
// Level-3 translation units.
#pragma once

#include "gbx_internal.h"
#include "gemm_simt.cuh"

namespace gbx_gemm {
template <typename T>
gbx_status launch_gemm(gbx_ctx *ctx, GemmArgs<T> p, const char *what);
// FP64 launches of few waves and small SGEMMs (gemm_small.cu); false: not one of them.
bool launch_gemm_short(gbx_ctx *ctx, GemmArgs<double> p, int bm);
bool launch_gemm_short(gbx_ctx *ctx, GemmArgs<float> p);
// What SGEMM's splitting kernel (sgemm_tc.cu) marks with the call's tag.
enum {
    SPLIT_UNCOVERED,      // an element outside [2^-90, 2^60]
    SPLIT_A_SMALL,        // one of A below 2^-34
    SPLIT_A_TINY,         // below 2^-60
    SPLIT_B_SMALL,
    SPLIT_B_TINY
};
// The operands are the SIMT core's.
__device__ __forceinline__ bool split_uncovered(const unsigned *marks, unsigned tag)
{
    return marks[SPLIT_UNCOVERED] == tag || (marks[SPLIT_A_TINY] == tag && marks[SPLIT_B_SMALL] == tag) ||
           (marks[SPLIT_A_SMALL] == tag && marks[SPLIT_B_TINY] == tag);
}
// The SIMT SGEMM of a full C, which does nothing unless they are when it runs.
gbx_status launch_gemm_if(gbx_ctx *ctx, GemmArgs<float> p, const char *what, const unsigned *marks, unsigned tag);
// SGEMM on the tensor cores (sgemm_tc.cu); *done: the call was taken.
gbx_status sgemm_tensor(gbx_ctx *ctx, const GemmArgs<float> &p, const char *what, bool *done);
// C = beta * C on the whole matrix or one triangle (beta == 0 sets zero);
// herm: the diagonal's imaginary part is set to zero (Hermitian C).
template <typename T>
gbx_status scale_matrix(gbx_ctx *ctx, int m, int n, T beta, T *C, long long ldc, int part, int herm = 0);
}  // namespace gbx_gemm
