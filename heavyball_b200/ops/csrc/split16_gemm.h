// fp32 GEMM at near-fp32 accuracy from products of fp16 pairs, with the epilogues of tf32_gemm.h (see split16_gemm.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "tf32_gemm.h"

namespace hb {

// Operand: [rows, 2 * kp] fp16 with kp = K rounded up to 64; a row holds [hi | lo], hi = fp16(x 2^e), lo = fp16((x 2^e - hi) 2^11),
// where the exponent e of the row takes its largest value to [2^14, 2^15), 126 at most (rows below 2^-112 stay under that; rows with an
// infinity have e = 0); columns [K, kp) of both halves are zero.  `unit` holds 2^-e per row and, in the mantissa, the number of the
// row's values below 2^-14 2^-e other than zero, which a pair holds in fewer than 22 bits (2^19 and more: any number);
// [batch, split16_units(rows)] (padded to whole tiles; the padding is read but never reaches a result).
inline int64_t split16_kp(int64_t K) { return (K + 63) / 64 * 64; }
inline int64_t split16_units(int64_t rows) { return (rows + 255) / 256 * 256; }

// The matrix that an operand was made from: element (r, c) of batch entry b is p[b * batch + r * row + c * k].  A product reads it where a
// result hangs on values that the pairs do not hold, so it has to be what it was when it was split.
struct Split16Source {
  const float* p;
  int64_t batch, row, k;
};

struct Split16Operand {
  void* data;    // fp16
  float* unit;
  Split16Source src;
};

// src: [batch, R, C] fp32 (row stride ld, batch stride `stride`).  Writes either or both operands (data null = not wanted):
//   same : rows = src rows, K = C;   trans: rows = src columns, K = R
struct Split16Pass {
  const float* src;
  int64_t ld, stride;
  int R, C;
  Split16Operand same, trans;
};
// One or two passes over matrices of one batch in a launch.
cudaError_t launch_split16(const Split16Pass* passes, int n, int batch, cudaStream_t stream);

// out[b] = epilogue(A[b] * B[b]^T); epilogue and flags as for launch_tf32_gemm, without split outputs (E.S null).
cudaError_t launch_split16_gemm(Split16Operand A, Split16Operand B, int M, int N, int K, int batch, const Tf32Epilogue& E, int* status,
                                cudaStream_t stream);

// Tile choice: 0 = by problem size, 128 or 256 = forced (tests and measurements).
void set_split16_gemm_tile_override(int tile);

}  // namespace hb
