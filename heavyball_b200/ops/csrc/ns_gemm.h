// Host-visible declarations for the Newton–Schulz GEMM family (ns_gemm.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <memory>

namespace hb {

enum GemmMode : int { kModeGram = 0, kModePoly = 1, kModeApply = 2 };

// D[M, N] = A[M, K] * B[N, K]^T (b_mn: B is [K, N], N contiguous) per batch entry; all leading dimensions and strides
// in elements.
struct GemmParams {
  int M, N, K, batch;
  int mode;
  int symmetric;            // compute tiles with tile_n >= tile_m only and mirror them through CT
  int b_mn;                 // B is stored [K, N]: its tiles are read through MN-major descriptors
  int same_operand;         // A and B are the same matrix (set by the launcher): diagonal tiles load it once
  __nv_bfloat16* C;         // bf16 output [M, N] (may be null)
  int64_t ldc, strideC;
  __nv_bfloat16* CT;        // bf16 transposed output [N, M] (may be null; equals C for symmetric results)
  int64_t ldct, strideCT;
  float* F;                 // fp32 output scaled by f_scale, [M, N] or [N, M] when f_transposed (may be null)
  int64_t ldf, strideF;
  int f_transposed;
  float f_scale;
  const __nv_bfloat16* S;   // poly mode: epilogue operand, same shape as the output
  int64_t lds, strideS;
  float ca, cb, cc;         // poly mode: D <- cc * acc + cb * S + ca * I
  int* status;              // set to 1 if a bounded wait expired
};

// Tile choice of launch_ns_products: 0 = by problem size (ns_tiles.h, default), 128 / 256 = force that output tile (tests, tuning).
int ns_gemm_tile_override();
void set_ns_gemm_tile_override(int tile);

struct NsProduct {
  const void* A;
  int64_t lda, strideA;
  const void* B;
  int64_t ldb, strideB;
  GemmParams P;
};
// Independent products, in as few launches as their tile sizes allow, ready to be issued any number of times while their buffers live on the
// current device: an iteration alternates between two buffers, so its five steps are made of as many different launches as two.
struct NsLaunches;
struct NsPlan {
  std::shared_ptr<NsLaunches> launches;
};
cudaError_t prepare_ns_products(const NsProduct* products, int n, NsPlan* plan);
void set_ns_coefficients(const NsPlan& plan, float ca, float cb, float cc);
// `launches` (may be null) is advanced by their number.
cudaError_t launch_ns_plan(const NsPlan& plan, int* launches, cudaStream_t stream);
// Both at once.
cudaError_t launch_ns_products(const NsProduct* products, int n, int* launches, cudaStream_t stream);

// One matrix to be normalised and rounded into the bf16 iterate (as it is, or transposed).
struct NsSource {
  const void* src;
  const float* sumsq;  // squared Frobenius norm
  void* dst;
  uint64_t seed;
  int64_t ld;
  int rows, cols, trans;
  int index;           // position within its bucket (part of the rounding noise's address)
};
// `first`: n_mats + 1 prefix sums of the matrices' 64 x 64 tile counts; both tables in device memory.
cudaError_t launch_ns_prepare(const NsSource* mats, const int* first, int n_mats, int total_tiles, int src_dt, float eps,
                              cudaStream_t stream);

}  // namespace hb
