// fp32-in / fp32-out batched GEMM at near-fp32 accuracy on the tf32 tensor-core path of sm_100a ("3xTF32"), with the
// element-wise stages of SOAP and PSGD fused into its epilogue.
//
// The preconditioner algebra of SOAP and PSGD (eigenbasis projections, Gram statistics, Kronecker factor
// products; heavyball/utils.py:1205-1259, 1391-1411, 3084-3122, 3557-3576 of the reference run them as fp32 cuBLAS
// einsums) needs more than tf32's 10 mantissa bits, and fp32 SIMT GEMMs run at a twentieth of the tensor-core rate.
// Each operand is therefore split once into hi = tf32(x) and lo = tf32(x - hi), stored side by side as rows of
// [hi | lo], and the product is taken as
//     A B^T ~= hi_a hi_b^T + hi_a lo_b^T + lo_a hi_b^T
// by walking A as (hi, hi, lo) and B as (hi, lo, hi) along K: ONE K-major tf32 GEMM over 3K with a single fp32
// accumulator in tensor memory.  The dropped lo*lo term and the rounding of lo to tf32 are both below 2^-21.
// Measured error: about 2^-18 of |A||B|^T for K = 2048 (fp32 SIMT: 2^-21, one tf32 pass: 2^-11); it is set by the
// rounding of the tensor core's accumulator.  One split buffer serves as either operand, so a symmetric product
// X X^T needs one split of X, and matrices that change rarely (eigenbases, preconditioner factors) stay split.
//
// Kernels and epilogues: gemm_epilogue.cuh; which tile when: gemm_rules.h.  SOAP's statistics and refresh run on this product (lerp into the
// statistics matrix; added to a view for Schur complements and solves) and so does the rotation of its moments, projections and PSGD on that of
// split16_gemm.cu.  Adam / LaProp on moment
// buffers, a result written as a split operand - as it is or transposed - and products of upper-triangular matrices are here for callers of
// ops.tf32_gemm and ops.matmul3.
// Waits are bounded as in the bf16 kernels: on expiry the CTA flags `status`, drains, frees TMEM and returns.
#include "tf32_gemm.h"

#include "gemm_epilogue.cuh"
#include "gemm_rules.h"
#include "per_device.h"

namespace hb {
namespace {

constexpr int TBK = 32;
// tf32 x tf32 -> fp32, both operands K-major
constexpr uint32_t tf32_desc(int m, int n) { return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24); }

struct Tf32Kind {
  static constexpr int kBlock = TBK;
  static constexpr bool kScaled = false, kCrossFirst = false;
  static constexpr int kTermLoA = 2, kTermLoB = 1;  // A: hi, hi, lo   B: hi, lo, hi
  static constexpr uint32_t kDesc = tf32_desc(TBM, TBN), kPairDesc = tf32_desc(kPairTile, kPairTile);
  __device__ static __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t desc, uint32_t accumulate) {
    tc_mma_tf32(d, a, b, desc, accumulate);
  }
  __device__ static __forceinline__ void mma_pair(uint32_t d, uint64_t a, uint64_t b, uint32_t desc, uint32_t accumulate) {
    tc_mma_tf32_pair(d, a, b, desc, accumulate);
  }
};

// One block moves a 64 x 64 tile of the source through shared memory and writes the [hi | lo] rows it covers of either
// or both operand orientations (see tf32_gemm.h).  The zero padding [K, kp) of every row is written too.  256 threads
// = 16 float4 lanes x 16 rows, four passes each way; global accesses are 16 bytes wide (the source falls back to
// scalars when its rows are not 16-byte aligned).  Grid: (ceil(kp(C) / 64), ceil(kp(R) / 64), batch).
__global__ void __launch_bounds__(256) tf32_split_kernel(const float* __restrict__ src, int64_t ld_src, int64_t stride_src,
                                                        int R, int C, float* __restrict__ dst_same,
                                                        float* __restrict__ dst_trans, int kpC, int kpR) {
  __shared__ float tile[64][65];  // [source row][source column]
  griddep_wait();
  griddep_launch();
  const float* s = src + (int64_t)blockIdx.z * stride_src;
  const int c0 = blockIdx.x * 64, r0 = blockIdx.y * 64;
  const int lane4 = (threadIdx.x & 15) * 4, line = threadIdx.x >> 4;
  const bool vec_ok = (ld_src & 3) == 0 && (stride_src & 3) == 0 && (((uintptr_t)src) & 15) == 0;
#pragma unroll
  for (int pass = 0; pass < 4; ++pass) {
    const int lr = line + 16 * pass, sr = r0 + lr, sc = c0 + lane4;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (sr < R) {
      const float* row = s + (int64_t)sr * ld_src;
      if (vec_ok && sc + 3 < C) {
        const float4 t = *reinterpret_cast<const float4*>(row + sc);
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (sc + e < C) v[e] = row[sc + e];
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) tile[lr][lane4 + e] = v[e];
  }
  __syncthreads();
  if (dst_same != nullptr) {  // rows = source rows, k = source columns
    float* d = dst_same + (int64_t)blockIdx.z * R * 2 * kpC;
#pragma unroll
    for (int pass = 0; pass < 4; ++pass) {
      const int lr = line + 16 * pass, r = r0 + lr, k = c0 + lane4;
      if (r >= R || k >= kpC) continue;  // kp is a multiple of 32, so a float4 never straddles it
      float hi[4], lo[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float x = tile[lr][lane4 + e];
        // lo is rounded to tf32 here (the tensor core would truncate it): halves the error of the two cross terms
        hi[e] = tf32_hi(x);
        lo[e] = tf32_hi(x - hi[e]);
      }
      float* row = d + (int64_t)r * 2 * kpC + k;
      *reinterpret_cast<float4*>(row) = make_float4(hi[0], hi[1], hi[2], hi[3]);
      *reinterpret_cast<float4*>(row + kpC) = make_float4(lo[0], lo[1], lo[2], lo[3]);
    }
  }
  if (dst_trans != nullptr) {  // rows = source columns, k = source rows
    float* d = dst_trans + (int64_t)blockIdx.z * C * 2 * kpR;
#pragma unroll
    for (int pass = 0; pass < 4; ++pass) {
      const int lc = line + 16 * pass, c = c0 + lc, k = r0 + lane4;
      if (c >= C || k >= kpR) continue;
      float hi[4], lo[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float x = tile[lane4 + e][lc];
        hi[e] = tf32_hi(x);
        lo[e] = tf32_hi(x - hi[e]);
      }
      float* row = d + (int64_t)c * 2 * kpR + k;
      *reinterpret_cast<float4*>(row) = make_float4(hi[0], hi[1], hi[2], hi[3]);
      *reinterpret_cast<float4*>(row + kpR) = make_float4(lo[0], lo[1], lo[2], lo[3]);
    }
  }
}

// fp32 tensor [batch, rows, cols], row stride ld elements; box = 32 columns x 128 rows, 128-byte swizzle.
bool make_f32_map(CUtensorMap* map, const void* base, int rows, int64_t cols, int64_t ld, int64_t batch_stride, int batch) {
  EncodeTiledFn fn = tensor_map_encoder();
  if (fn == nullptr) return false;
  cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)batch};
  cuuint64_t strides[2] = {(cuuint64_t)ld * 4, (cuuint64_t)batch_stride * 4};
  cuuint32_t box[3] = {TBK, TBM, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

cudaError_t launch_tf32_split(const float* src, int64_t ld_src, int64_t stride_src, int R, int C, int batch, float* dst_same,
                              float* dst_trans, cudaStream_t stream) {
  if (R == 0 || C == 0 || batch == 0 || (dst_same == nullptr && dst_trans == nullptr)) return cudaSuccess;
  const int kpC = (int)tf32_split_kp(C), kpR = (int)tf32_split_kp(R);
  dim3 grid((kpC + 63) / 64, (kpR + 63) / 64, batch);
  return launch_chained(tf32_split_kernel, grid, 256, 0, stream, src, ld_src, stride_src, R, C, dst_same, dst_trans, kpC, kpR);
}

static int g_tf32_tile_override = 0;  // 0 = by size, 128 / 256 = forced (tests and measurements)
int tf32_gemm_tile_override() { return g_tf32_tile_override; }
void set_tf32_gemm_tile_override(int tile) { g_tf32_tile_override = (tile == 128 || tile == 256) ? tile : 0; }

// Pairs of CTAs that can be resident at once on the current device; also sets the kernels' shared memory up there.
static cudaError_t resident_pairs(int* out) {
  static PerDevice<int> pairs;
  int device = 0;
  const cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  return pairs.get(device, cudaSuccess, out, [](int& found) {
    cudaError_t s = cudaFuncSetAttribute(gemm128_kernel<Tf32Kind>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTSmemBytes);
    if (s == cudaSuccess) s = cudaFuncSetAttribute(gemm_pair_kernel<Tf32Kind>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGPairSmemBytes);
    return s != cudaSuccess ? s : max_resident_pairs(gemm_pair_kernel<Tf32Kind>, kGPairThreads, kGPairSmemBytes, &found);
  });
}

cudaError_t tf32_gemm_tiles(int M, int N, int K, int batch, int symmetric, int* choice) {
  int max_pairs = 0;
  const cudaError_t e = resident_pairs(&max_pairs);
  if (e == cudaSuccess) *choice = tf32_tiles(M, N, K, batch, symmetric != 0, max_pairs);
  return e;
}

cudaError_t launch_tf32_gemm(const float* A2, const float* B2, int M, int N, int K, int batch, const Tf32Epilogue& E,
                             int* status, cudaStream_t stream) {
  const int64_t kp = tf32_split_kp(K);
  return launch_tf32_gemm(Tf32Operand{A2, 2 * kp, M * 2 * kp, kp}, Tf32Operand{B2, 2 * kp, N * 2 * kp, kp}, M, N, K, batch, E, status, stream);
}

cudaError_t launch_tf32_gemm(Tf32Operand A, Tf32Operand B, int M, int N, int K, int batch, const Tf32Epilogue& E, int* status, cudaStream_t stream) {
  int max_pairs = 0;
  const cudaError_t e = resident_pairs(&max_pairs);
  if (e != cudaSuccess) return e;
  if (M == 0 || N == 0 || batch == 0) return cudaSuccess;
  if ((E.mode == kEpiAdam || E.mode == kEpiLaProp) && (E.m == nullptr || E.v == nullptr)) return cudaErrorInvalidValue;
  if ((E.mode == kEpiLerp || E.mode == kEpiAdd) && E.C == nullptr) return cudaErrorInvalidValue;
  if (E.tri && (M != N || M != K || E.symmetric)) return cudaErrorInvalidValue;
  if (E.symmetric && (A.p != B.p || M != N || E.C == nullptr || E.S != nullptr || (E.mode != kEpiStore && E.mode != kEpiLerp && E.mode != kEpiAdd)))
    return cudaErrorInvalidValue;
  const int64_t kp = tf32_split_kp(K);
  if (A.lo < kp || B.lo < kp || A.lo % 4 != 0 || B.lo % 4 != 0) return cudaErrorInvalidValue;
  CUtensorMap ma, mb, mc;
  if (!make_f32_map(&ma, A.p, M, A.lo + kp, A.ld, A.stride, batch) || !make_f32_map(&mb, B.p, N, B.lo + kp, B.ld, B.stride, batch))
    return cudaErrorInvalidValue;

  TileChoice tiles = tf32_tiles(M, N, K, batch, E.symmetric != 0, max_pairs);
  if (g_tf32_tile_override == 128) tiles = kSmallTiles;
  if (g_tf32_tile_override == 256 && tiles == kSmallTiles) tiles = kPairTiles;
  if (tiles != kSmallTiles) {
    const int big_m = (M + kPairTile - 1) / kPairTile, big_n = (N + kPairTile - 1) / kPairTile;
    const int per_batch = (int)output_tiles(M, N, kPairTile, E.symmetric != 0);
    const int64_t total = (int64_t)per_batch * batch;
    Tf32Epilogue E2 = E;
    if (tiles == kPairTilesSmallDiagonal) E2.symmetric = 2;
    return launch_chained(gemm_pair_kernel<Tf32Kind>, dim3(2 * (int)(total < max_pairs ? total : max_pairs)), kGPairThreads, kGPairSmemBytes, stream,
                          ma, mb, M, N, (int)kp, (int)A.lo, (int)B.lo, big_m, big_n, per_batch, (int)total, E2, PairOperands{}, status);
  }

  // plain products leave through the bulk-store path (bulk stores end on 16-byte boundaries: with N a multiple of 4 they write nothing
  // past it); everything else is written by the epilogue threads themselves
  const int bulk = (!E.symmetric && !E.tri && E.mode == kEpiStore && E.S == nullptr && E.C != nullptr && (N & 3) == 0 && (E.ldc & 3) == 0 &&
                    (E.strideC & 3) == 0 && (((uintptr_t)E.C) & 15) == 0) ? 1 : 0;
  mc = ma;  // placeholder when the bulk-store path is not taken (never dereferenced then)
  if (bulk && !make_f32_map(&mc, E.C, M, N, E.ldc, E.strideC, batch)) return cudaErrorInvalidValue;
  const int tiles_m = (M + TBM - 1) / TBM, tiles_n = (N + TBN - 1) / TBN;
  dim3 grid(E.symmetric ? tiles_n * (tiles_n + 1) / 2 : tiles_m * tiles_n, batch);
  return launch_chained(gemm128_kernel<Tf32Kind>, grid, kTThreads, kTSmemBytes, stream, ma, mb, mc, M, N, (int)kp, (int)A.lo, (int)B.lo, E, PairOperands{}, bulk,
                        status);
}

}  // namespace hb
