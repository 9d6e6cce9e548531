// Largest eigenvalue of batched symmetric positive semi-definite matrices (see power_iteration.cu).
#pragma once
#include <cuda_runtime.h>

namespace hb {

constexpr int kMaxPowerSize = 2048;

// out[b] <- sqrt(x^T A A x) with x after `iterations` steps x <- A A x / |A A x| from the row of A of largest norm; A: contiguous [batch, n, n]
// symmetric fp32, n <= kMaxPowerSize.
cudaError_t launch_power_iteration(const float* A, int batch, int n, int iterations, float* out, cudaStream_t stream);

}  // namespace hb
