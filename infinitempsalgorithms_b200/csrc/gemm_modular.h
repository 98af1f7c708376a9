// FP64 complex GEMM by residue arithmetic on the int8 tensor cores (see gemm_modular.cu).
#pragma once
#include "imps_internal.h"

namespace imps {

// C = alpha op(A) op(B) + beta C (column-major complex, one product) when the sizes make the
// residue path faster than the FP64 tensor cores (t_fp64: their modelled time in us) and its
// scratch is to be had; returns false, with nothing done, otherwise.
bool zgemm_modular(Context* ctx, Op opA, Op opB, int M, int N, int K, cplx alpha, const dcplx* A, int64_t lda,
                   const dcplx* B, int64_t ldb, cplx beta, dcplx* C, int64_t ldc, double t_fp64);

}  // namespace imps
