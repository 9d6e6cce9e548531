// Passes over batches of fp32 matrices that only memory bounds, each in the place of several of the library's (see matrix_passes.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace hb {

// dst[b][c][r] = src[b][r][c]; src: [batch, R, C], dst: [batch, C, R], both contiguous, not overlapping; batch <= 65535.
cudaError_t launch_transpose(const float* src, float* dst, int batch, int R, int C, cudaStream_t stream);

// a <- a + b, b <- triu(a - b) for contiguous [batch, n, n] matrices.
cudaError_t launch_sum_triu_diff(float* a, float* b, int batch, int n, cudaStream_t stream);

// out[i] = g[i] + (damp + eps |g[i]|) v[i].
cudaError_t launch_dampen(const float* g, const float* v, float* out, int64_t count, float damp, float eps, cudaStream_t stream);

// line[b] -= triu(step[b]) / ell[b] * lr; step: [batch, n, n], line: row-major upper triangles [batch, n (n + 1) / 2]; batch <= 65535.
cudaError_t launch_triu_step(const float* step, const float* ell, float* line, int batch, int n, float lr, cudaStream_t stream);

// x[b][i] *= by[b] for i < count; batch <= 65535.
cudaError_t launch_scale_matrices(float* x, const float* by, int batch, int64_t count, cudaStream_t stream);

}  // namespace hb
