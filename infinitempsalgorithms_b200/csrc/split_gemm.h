// int8 split-precision complex GEMM on tcgen05 (see gemm_i8.cu).
#pragma once
#include <cuda.h>

#include "imps_internal.h"

namespace imps {

// One operand cut into `s` int8 planes (K-major, padded), plus per-line scales.
struct SplitOperand {
  DevBuf data;    // s planes of Rp x Kp bytes
  DevBuf scale;   // per complex row (A side) / column (B side): power of two > max |re|,|im|
  DevBuf mx;      // per line: bits of the largest |re|, |im|
  int rows = 0;   // complex rows (A: M, B: N)
  int K = 0;      // complex inner dimension
  int s = 0;      // slices stored
  int64_t Rp = 0, Kp = 0;
};

// op(A) (M x K), op in {N, C}: expanded real rows (2M) x (2K) int8 planes; have_max: S.mx
// already holds the rows' maxima (op N)
void split_operand_a(Context* ctx, SplitOperand& S, Op op, int M, int K, const dcplx* A, int64_t lda, int s,
                     bool have_max = false);
// S.mx for this many lines, cleared, for a kernel that collects them while it writes the operand
unsigned long long* split_line_max(Context* ctx, SplitOperand& S, int lines);
// op(B) (K x N), op in {N, C}: N rows x (2K) int8 planes
void split_operand_b(Context* ctx, SplitOperand& S, Op op, int K, int N, const dcplx* B, int64_t ldb, int s);
// C (complex, ldc) = alpha * op(A) op(B) (+ C when accumulate) using `s` slice diagonals
void split_gemm(Context* ctx, const SplitOperand& A, const SplitOperand& B, int s, double alpha, bool accumulate,
                dcplx* C, int64_t ldc);

// 3D tensor map over int8 planes (Kp bytes, rows, planes), box (box_k, box_rows, 1), swizzled
// over box_k = 64 or 128 bytes; plane_bytes: stride of the planes, 0 for rows x Kp
CUtensorMap plane_map(const int8_t* base, int64_t Kp, int64_t rows, int planes, int box_k, int box_rows,
                      int64_t plane_bytes = 0);

// Slices needed for a requested relative accuracy `tol` (clamped to 2..8).
int slices_for_tol(double tol);

}  // namespace imps
