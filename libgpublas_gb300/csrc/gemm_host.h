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
// The SIMT SGEMM of a full C, which does nothing unless *flag == tag when it runs.
gbx_status launch_gemm_if(gbx_ctx *ctx, GemmArgs<float> p, const char *what, const unsigned *flag,
                          unsigned tag);
// SGEMM on the tensor cores (sgemm_tc.cu); *done: the call was taken.
gbx_status sgemm_tensor(gbx_ctx *ctx, const GemmArgs<float> &p, const char *what, bool *done);
// C = beta * C on the whole matrix or one triangle (beta == 0 sets zero);
// herm: the diagonal's imaginary part is set to zero (Hermitian C).
template <typename T>
gbx_status scale_matrix(gbx_ctx *ctx, int m, int n, T beta, T *C, long long ldc, int part, int herm = 0);
}  // namespace gbx_gemm
