// One round of Cholesky QR on split-tf32 products: A <- A R^-1 with R^T R = G, all blocks 128 wide (see chol_qr.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace hb {

constexpr int kQrBlock = 128;  // columns of a block; a leaf of skinny.h
constexpr int kQrRows = 64;    // rows of the long side that a block of threads solves

// X = B T^-1 for 128 columns and upper-triangular T whose inverse is given; B: `rows` x 128, row stride ld, or its transpose (from_rows:
// element (row, k) at src[k * ld + row]).  X goes to whichever of these are wanted:
//   out   : fp32, row stride ld_out
//   same  : split-tf32 rows, high parts at same + r * ld_same, low parts lo_same behind them
//   trans : split-tf32 columns, high parts of column c from row 0 on at trans + c * ld_trans, low parts lo_trans behind them
// All strides are multiples of 4 elements, all pointers 16-byte aligned, rows a multiple of kQrRows.
struct QrLeafSolve {
  const float* src;
  int64_t ld, stride;
  int from_rows;
  const float* inv;  // [128, 128], zeros below the diagonal
  int64_t stride_inv;
  float* out;
  int64_t ld_out, stride_out;
  float* same;
  int64_t ld_same, lo_same, stride_same;
  float* trans;
  int64_t ld_trans, lo_trans, stride_trans;
};
cudaError_t launch_qr_leaf_solve(const QrLeafSolve& S, int rows, int batch, cudaStream_t stream);

// A[b][i][j] = X[b][i][j] / norm[b][j]; A_trans: [batch, k, 2 n], the split-tf32 operand of A^T.  X, A (may be X): contiguous [batch, n, k], n a
// multiple of 64, k of 128.
cudaError_t launch_qr_unit_columns(const float* X, const float* norm, float* A, float* A_trans, int batch, int n, int k, cudaStream_t stream);

// G: [batch, k, k] symmetric positive definite, overwritten; A: [batch, n, k]; contiguous, n % 64 == 0, k % 128 == 0.
//   A       : <- X = A R^-1
//   X_trans : [batch, k, 2 n] <- the split-tf32 operand of X^T (null: not wanted)
// Workspaces: L [batch, k, 2 k] (the split rows of R^T below its diagonal blocks), inv [batch, k / 128, 128, 128], X_same [batch, n, 2 k].
// info[b] is incremented per leaf with a bad pivot.  *launches += kernels issued.
struct QrRound {
  float *G, *A, *X_trans, *L, *inv, *X_same;
  int n, k, batch;
  int* info;
  int* status;
};
cudaError_t launch_chol_qr_round(const QrRound& Q, int* launches, cudaStream_t stream);

}  // namespace hb
