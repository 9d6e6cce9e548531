// fp32 product over a long dimension for block Gram-Schmidt with a narrow panel (the eigenbasis-refresh QR):
//
//   tall_t_mul : C[b] = X[b]^T W[b]     X: [n, m] (leading dimension ldx), W: [n, p], p <= 32, contraction over the
//                                       long dimension n.  The library's GEMM for this shape is a 32x32x16 SIMT
//                                       kernel that walks n serially (18 us whatever m is); here n is split over
//                                       CTAs and the partial products are kept apart (deterministic), to be summed
//                                       by the caller.
//
// Tiles staged in shared memory, 8 x 4 register tiles, plain FMAs: the products are tiny (at most 2 * 1024 * 1024 * 32 flops per
// matrix) and latency, not throughput, is what the panel loop pays for.  The matching rank-m update W -= X C has
// plenty of row parallelism and stays a library GEMM (a version written here the same way was slower).
#include "skinny.h"

#include "per_device.h"
#include "tc_common.cuh"

#include <stdint.h>

namespace hb {
namespace {

constexpr int kTileM = 128;   // columns of X (rows of the result) per CTA
constexpr int kTileR = 64;    // rows of the long dimension staged at a time
constexpr int kMaxSplits = 16;

// grid: (ceil(m / 128), splits, batch); block: 128 threads = 16 (groups of 8 result rows) x 8 (groups of 4 columns).
// Each thread keeps an 8 x 4 register tile: per staged row it reads 8 + 4 values from shared memory (three 16-byte
// loads) for 32 FMAs.  A first version with one value per load and four FMAs was issue-bound at 20 us per call.
template <bool kVec>
__global__ void __launch_bounds__(128) tall_t_mul_kernel(const float* __restrict__ X, long long ldx, long long strideX,
                                                        const float* __restrict__ W, long long ldw, long long strideW,
                                                        int n, int m, int p, float* __restrict__ C, int splits) {
  __shared__ __align__(16) float xs[kTileR][kTileM];
  __shared__ __align__(16) float ws[kTileR][32];
  const int b = blockIdx.z, split = blockIdx.y, m0 = blockIdx.x * kTileM;
  const float* x = X + (long long)b * strideX;
  const float* w = W + (long long)b * strideW;
  const int t = threadIdx.x, tm = t >> 3, tp = t & 7;
  float acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  const int rows_per_split = (n + splits - 1) / splits;
  const int r_begin = split * rows_per_split, r_end = min(n, r_begin + rows_per_split);
  for (int r0 = r_begin; r0 < r_end; r0 += kTileR) {
    // stage X[r0 .. r0+63][m0 .. m0+127] and W[r0 .. r0+63][0 .. 31]; loads are issued before any is consumed
    if (kVec) {
      float4 xv[16], wv[4];
#pragma unroll
      for (int it = 0; it < 16; ++it) {  // 64 rows x 32 float4 per row, 128 threads
        const int idx = t + 128 * it, rr = idx >> 5, c4 = (idx & 31) * 4;
        const int r = r0 + rr, c = m0 + c4;
        xv[it] = (r < r_end && c < m) ? *reinterpret_cast<const float4*>(x + (long long)r * ldx + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (c + 3 >= m && c < m) {  // tail of the m range: mask the lanes past it
          if (c + 1 >= m) xv[it].y = 0.f;
          if (c + 2 >= m) xv[it].z = 0.f;
          xv[it].w = 0.f;
        }
      }
#pragma unroll
      for (int it = 0; it < 4; ++it) {  // 64 rows x 8 float4 per row
        const int idx = t + 128 * it, rr = idx >> 3, c4 = (idx & 7) * 4;
        const int r = r0 + rr;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < r_end && c4 < p) {
          const float* src = w + (long long)r * ldw + c4;
          v.x = src[0];
          if (c4 + 1 < p) v.y = src[1];
          if (c4 + 2 < p) v.z = src[2];
          if (c4 + 3 < p) v.w = src[3];
        }
        wv[it] = v;
      }
#pragma unroll
      for (int it = 0; it < 16; ++it) {
        const int idx = t + 128 * it;
        *reinterpret_cast<float4*>(&xs[idx >> 5][(idx & 31) * 4]) = xv[it];
      }
#pragma unroll
      for (int it = 0; it < 4; ++it) {
        const int idx = t + 128 * it;
        *reinterpret_cast<float4*>(&ws[idx >> 3][(idx & 7) * 4]) = wv[it];
      }
    } else {
      for (int idx = t; idx < kTileR * kTileM; idx += 128) {
        const int rr = idx >> 7, c = idx & 127, r = r0 + rr;
        xs[rr][c] = (r < r_end && m0 + c < m) ? x[(long long)r * ldx + m0 + c] : 0.f;
      }
      for (int idx = t; idx < kTileR * 32; idx += 128) {
        const int rr = idx >> 5, c = idx & 31, r = r0 + rr;
        ws[rr][c] = (r < r_end && c < p) ? w[(long long)r * ldw + c] : 0.f;
      }
    }
    __syncthreads();
#pragma unroll 4
    for (int rr = 0; rr < kTileR; ++rr) {
      const float4 a0 = *reinterpret_cast<const float4*>(&xs[rr][tm * 8]);
      const float4 a1 = *reinterpret_cast<const float4*>(&xs[rr][tm * 8 + 4]);
      const float4 bv = *reinterpret_cast<const float4*>(&ws[rr][tp * 4]);
      const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      const float bw[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bw[j], acc[i][j]);
    }
    __syncthreads();
  }
  float* c = C + ((long long)split * gridDim.z + b) * m * p;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int row = m0 + tm * 8 + i;
    if (row >= m) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int col = tp * 4 + j;
      if (col < p) c[(long long)row * p + col] = acc[i][j];
    }
  }
}

}  // namespace

int tall_splits(int n) {  // two staged tiles of rows per CTA, up to 16 splits; very long inputs (the flattened parameter
                          // vector of a low-rank preconditioner: millions of rows) are cut so that every SM gets several CTAs
  const int s = (n + 2 * kTileR - 1) / (2 * kTileR);
  const int cap = n > 65536 ? 2048 : kMaxSplits;
  return s < 1 ? 1 : (s > cap ? cap : s);
}

cudaError_t launch_tall_t_mul(const float* X, long long ldx, long long strideX, const float* W, long long ldw,
                              long long strideW, int batch, int n, int m, int p, float* C, cudaStream_t stream) {
  if (batch == 0 || m == 0 || p == 0) return cudaSuccess;
  const int splits = tall_splits(n);
  dim3 grid((m + kTileM - 1) / kTileM, splits, batch);
  const bool vec = (ldx % 4 == 0) && (strideX % 4 == 0) && ((reinterpret_cast<uintptr_t>(X) & 15) == 0);
  if (vec)
    tall_t_mul_kernel<true><<<grid, 128, 0, stream>>>(X, ldx, strideX, W, ldw, strideW, n, m, p, C, splits);
  else
    tall_t_mul_kernel<false><<<grid, 128, 0, stream>>>(X, ldx, strideX, W, ldw, strideW, n, m, p, C, splits);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------ 128 x 128 triangular leaves
// Both leaf kernels work on one (up to) 128 x 128 block per CTA of 1024 threads, the block and its inverse in shared memory
// as 4 x 4 sub-blocks of 32.  A refresh of an eigenbasis factors 16 leaves per 2048-wide factor and round, one after the
// other, so the latency of one CTA is all that counts; it is set by the length of the dependent chain, not by the 0.7 MFLOP.
//   factor R^T R = G, panel of 32 rows by panel: the 32 x 32 diagonal block in one warp (lane = column, the column in
//     registers, pivots and multipliers by shuffle), the rows of the panel to its right by substitution (thread = column,
//     column in registers), the trailing blocks by a rank-32 update (4 x up to 3 elements per thread).  Every element
//     receives the same products in the same order as in an element-wise right-looking factorisation; that form needed two
//     barriers per pivot, 256 of them, and a leaf took 108 us (two SOAP steps on 8 x 1024^2, 32 leaves: 9.82 -> 8.19 ms).
//   invert R: the four diagonal blocks (one warp each, lane = column in registers), then the blocks above the diagonal by
//     distance d = 1, 2, 3:  X_IJ = -X_II (sum_{K = I+1 .. J} R_IK X_KJ), J = I + d, four rows per warp.
// A non-positive or non-finite pivot is replaced by 1 and counted in info[b] (the result for that matrix is then
// meaningless, the others are unaffected).
namespace {

constexpr int kLeafThreads = 1024;
constexpr int kLeafLd = kTriBlock + 4;  // rows start on 16-byte boundaries: four values of a row per (broadcast) load
constexpr int kLeafBytes = 2 * kTriBlock * kLeafLd * (int)sizeof(float);
constexpr int kSub = 32, kSubs = kTriBlock / kSub;

// Loads the upper part of a block of `size` rows; a short block is completed by an identity.  x <- 0.
__device__ __forceinline__ void load_upper(const float* __restrict__ g, long long ld, int size, float* t, float* x) {
  float v[kTriBlock * kTriBlock / kLeafThreads];
#pragma unroll
  for (int e = 0; e < kTriBlock * kTriBlock / kLeafThreads; ++e) {
    const int idx = threadIdx.x + e * kLeafThreads, i = idx >> 7, j = idx & (kTriBlock - 1);
    v[e] = (i == j) ? 1.f : 0.f;
    if (i < size && j < size && j >= i) v[e] = g[(long long)i * ld + j];
  }
#pragma unroll
  for (int e = 0; e < kTriBlock * kTriBlock / kLeafThreads; ++e) {
    const int idx = threadIdx.x + e * kLeafThreads, i = idx >> 7, j = idx & (kTriBlock - 1);
    t[i * kLeafLd + j] = v[e];
    x[i * kLeafLd + j] = 0.f;
  }
}

// x <- t^-1 for the upper-triangular block t; the part of x below the diagonal blocks is scratch.
__device__ __forceinline__ void invert_upper(const float* t, float* x) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < kSubs) {  // right-looking back substitution: row i of this lane's column is final when step i starts
    const float* d = t + warp * kSub * (kLeafLd + 1);
    float* xd = x + warp * kSub * (kLeafLd + 1);
    float acc[kSub];
#pragma unroll
    for (int i = 0; i < kSub; ++i) acc[i] = 0.f;
#pragma unroll
    for (int i = kSub - 1; i >= 0; --i) {
      const float piv = d[i * kLeafLd + i];
      const float xi = i == lane ? 1.0f / piv : (i < lane ? -acc[i] / piv : 0.f);
      xd[i * kLeafLd + lane] = xi;
#pragma unroll
      for (int k = 0; k < i; ++k) acc[k] = fmaf(d[k * kLeafLd + i], xi, acc[k]);
    }
  }
  __syncthreads();
  const int I = warp >> 3, r0 = (warp & 7) * 4;  // four rows of the I-th block at the current distance
#pragma unroll 1
  for (int dist = 1; dist < kSubs; ++dist) {
    const int J = I + dist;
    const bool on = J < kSubs;
    if (on) {  // S = sum_K R_IK X_KJ, parked in the mirror position below the diagonal
      float s[4] = {0.f, 0.f, 0.f, 0.f};
      for (int k = kSub * (I + 1); k < kSub * (J + 1); k += 4) {
        float xv[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) xv[e] = x[(k + e) * kLeafLd + kSub * J + lane];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const float4 a = *(const float4*)(t + (kSub * I + r0 + r) * kLeafLd + k);
          s[r] = fmaf(a.x, xv[0], s[r]); s[r] = fmaf(a.y, xv[1], s[r]); s[r] = fmaf(a.z, xv[2], s[r]); s[r] = fmaf(a.w, xv[3], s[r]);
        }
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) x[(kSub * J + r0 + r) * kLeafLd + kSub * I + lane] = s[r];
    }
    __syncthreads();
    if (on) {
      float s[4] = {0.f, 0.f, 0.f, 0.f};
      for (int k = r0; k < kSub; k += 4) {  // X_II is upper triangular: columns left of the row are zero
        float sv[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) sv[e] = x[(kSub * J + k + e) * kLeafLd + kSub * I + lane];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const float4 a = *(const float4*)(x + (kSub * I + r0 + r) * kLeafLd + kSub * I + k);
          s[r] = fmaf(a.x, sv[0], s[r]); s[r] = fmaf(a.y, sv[1], s[r]); s[r] = fmaf(a.z, sv[2], s[r]); s[r] = fmaf(a.w, sv[3], s[r]);
        }
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) x[(kSub * I + r0 + r) * kLeafLd + kSub * J + lane] = -s[r];
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kLeafThreads) tri_inv_blocks_kernel(const float* __restrict__ Q, long long ld, long long strideQ,
                                                                     int n, float* __restrict__ X) {
  extern __shared__ __align__(16) float leaf_smem[];
  float *t = leaf_smem, *x = leaf_smem + kTriBlock * kLeafLd;
  const int blk = blockIdx.x, b = blockIdx.y, r0 = blk * kTriBlock;
  load_upper(Q + (long long)b * strideQ + (long long)r0 * ld + r0, ld, min(kTriBlock, n - r0), t, x);
  __syncthreads();
  invert_upper(t, x);
  float* out = X + ((long long)b * gridDim.x + blk) * kTriBlock * kTriBlock;
  for (int idx = threadIdx.x; idx < kTriBlock * kTriBlock; idx += kLeafThreads) {
    const int i = idx >> 7, j = idx & (kTriBlock - 1);
    out[idx] = j >= i ? x[i * kLeafLd + j] : 0.f;
  }
}

__global__ void __launch_bounds__(kLeafThreads) chol_inv_leaf_kernel(const float* __restrict__ G, long long ldg, long long strideG,
                                                                     float* __restrict__ R, long long ldr, long long strideR,
                                                                     float* __restrict__ X, long long strideX, int size,
                                                                     int* __restrict__ info) {
  extern __shared__ __align__(16) float leaf_smem[];
  float *t = leaf_smem, *x = leaf_smem + kTriBlock * kLeafLd;
  __shared__ float inv_piv[kSub];
  __shared__ int failed;
  const int b = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) failed = 0;
  griddep_wait();
  griddep_launch();
  load_upper(G + (long long)b * strideG, ldg, size, t, x);
  __syncthreads();

  for (int base = 0; base < size; base += kSub) {
    float* d = t + base * (kLeafLd + 1);
    if (warp == 0) {
      float a[kSub];
      bool bad = false;
#pragma unroll
      for (int i = 0; i < kSub; ++i) a[i] = d[i * kLeafLd + lane];
#pragma unroll
      for (int k = 0; k < kSub; ++k) {
        const float piv = __shfl_sync(0xffffffffu, a[k], k);
        const bool ok = piv > 0.f && piv < 3.0e38f;
        const float inv = ok ? rsqrtf(piv) : 1.f;
        bad = bad || !ok;
        if (lane == k) {
          a[k] = ok ? piv * inv : 1.f;  // sqrt of the pivot
          inv_piv[k] = inv;
        } else {
          a[k] *= inv;
        }
#pragma unroll
        for (int i = k + 1; i < kSub; ++i) a[i] = fmaf(-__shfl_sync(0xffffffffu, a[k], i), a[k], a[i]);
      }
#pragma unroll
      for (int i = 0; i < kSub; ++i)
        if (i <= lane) d[i * kLeafLd + lane] = a[i];
      if (lane == 0 && bad) failed = 1;
    }
    __syncthreads();
    const int rest = kTriBlock - base - kSub;  // columns right of the panel
    if (tid < rest) {
      float* col = d + kSub + tid;
      float a[kSub];
#pragma unroll
      for (int i = 0; i < kSub; ++i) a[i] = col[i * kLeafLd];
#pragma unroll
      for (int k = 0; k < kSub; ++k) {
        a[k] *= inv_piv[k];
#pragma unroll
        for (int i = k + 1; i < kSub; ++i) a[i] = fmaf(-d[k * kLeafLd + i], a[k], a[i]);
        col[k * kLeafLd] = a[k];
      }
    }
    __syncthreads();
    if (warp * 4 < rest) {  // rows i0 .. i0+3 of the trailing block, columns from the 32-block of i0 on
      const int i0 = warp * 4, first = i0 & ~(kSub - 1);
      const float* panel = d + kSub;  // panel[k * ld + i] = r_ki of trailing row / column i
      float* trail = t + (base + kSub) * (kLeafLd + 1);
      for (int j = first + lane; j < rest; j += kSub) {
        float acc[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[r] = trail[(i0 + r) * kLeafLd + j];
#pragma unroll 8
        for (int k = 0; k < kSub; ++k) {
          const float4 m = *(const float4*)(panel + k * kLeafLd + i0);
          const float rkj = panel[k * kLeafLd + j];
          acc[0] = fmaf(-m.x, rkj, acc[0]); acc[1] = fmaf(-m.y, rkj, acc[1]);
          acc[2] = fmaf(-m.z, rkj, acc[2]); acc[3] = fmaf(-m.w, rkj, acc[3]);
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
          if (j >= i0 + r) trail[(i0 + r) * kLeafLd + j] = acc[r];
      }
    }
    __syncthreads();
  }

  invert_upper(t, x);

  float* r = R + (long long)b * strideR;
  float* out = X + (long long)b * strideX;
  for (int idx = tid; idx < kTriBlock * kTriBlock; idx += kLeafThreads) {
    const int i = idx >> 7, j = idx & (kTriBlock - 1);
    if (R != nullptr && i < size && j < size) r[(long long)i * ldr + j] = j >= i ? t[i * kLeafLd + j] : 0.f;
    out[idx] = j >= i ? x[i * kLeafLd + j] : 0.f;
  }
  if (tid == 0 && failed && info != nullptr) atomicAdd(info + b, 1);
}

cudaError_t configure_leaf_kernels() {
  static PerDevice<bool> configured;
  int device = 0;
  const cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  bool done = false;
  return configured.get(device, cudaSuccess, &done, [](bool&) {
    const cudaError_t s = cudaFuncSetAttribute(tri_inv_blocks_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kLeafBytes);
    return s != cudaSuccess ? s : cudaFuncSetAttribute(chol_inv_leaf_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kLeafBytes);
  });
}

}  // namespace

cudaError_t launch_tri_inv_blocks(const float* Q, long long ld, long long strideQ, int batch, int n, float* X,
                                  cudaStream_t stream) {
  if (batch == 0 || n == 0) return cudaSuccess;
  cudaError_t e = configure_leaf_kernels();
  if (e != cudaSuccess) return e;
  dim3 grid((n + kTriBlock - 1) / kTriBlock, batch);
  tri_inv_blocks_kernel<<<grid, kLeafThreads, kLeafBytes, stream>>>(Q, ld, strideQ, n, X);
  return cudaGetLastError();
}

cudaError_t launch_chol_inv_leaf(const float* G, long long ldg, long long strideG, float* R, long long ldr, long long strideR,
                                 float* X, long long strideX, int batch, int size, int* info, cudaStream_t stream) {
  if (batch == 0 || size == 0) return cudaSuccess;
  if (size > kTriBlock) return cudaErrorInvalidValue;
  cudaError_t e = configure_leaf_kernels();
  if (e != cudaSuccess) return e;
  return launch_chained(chol_inv_leaf_kernel, dim3(batch), kLeafThreads, kLeafBytes, stream, G, ldg, strideG, R, ldr, strideR, X, strideX, size, info);
}

// ------------------------------------------------------------------------------------------ packed upper triangles
// PSGD stores a triangular factor as the row-major upper triangle ("line").  Row i of the triangle is the contiguous
// piece dense[i, i:n] and sits at line offset i*n - i*(i-1)/2, so packing and unpacking are row copies: one block per
// (row, matrix), no index tensors (index_put / index_select read an 8-byte index per element and first materialise
// 16 n^2 bytes of indices).
namespace {

template <typename T>
__global__ void __launch_bounds__(256) triu_pack_kernel(const T* __restrict__ dense, T* __restrict__ line, int n) {
  const long long i = blockIdx.x, b = blockIdx.y;
  const long long len = (long long)n * (n + 1) / 2;
  const T* src = dense + (b * n + i) * n + i;
  T* dst = line + b * len + i * n - i * (i - 1) / 2;
  for (int j = threadIdx.x; j < n - (int)i; j += blockDim.x) dst[j] = src[j];
}

template <typename T>
__global__ void __launch_bounds__(256) triu_unpack_kernel(const T* __restrict__ line, T* __restrict__ dense, int n) {
  const long long i = blockIdx.x, b = blockIdx.y;
  const long long len = (long long)n * (n + 1) / 2;
  const T* src = line + b * len + i * n - i * (i - 1) / 2 - i;  // indexed by the dense column
  T* dst = dense + (b * n + i) * n;
  for (int j = threadIdx.x; j < n; j += blockDim.x) dst[j] = j >= (int)i ? src[j] : T(0);
}

}  // namespace

cudaError_t launch_triu_pack(const void* dense, void* line, int elem_bytes, int batch, int n, cudaStream_t stream) {
  if (batch == 0 || n == 0) return cudaSuccess;
  dim3 grid(n, batch);
  if (elem_bytes == 4) triu_pack_kernel<uint32_t><<<grid, 256, 0, stream>>>((const uint32_t*)dense, (uint32_t*)line, n);
  else if (elem_bytes == 2) triu_pack_kernel<uint16_t><<<grid, 256, 0, stream>>>((const uint16_t*)dense, (uint16_t*)line, n);
  else return cudaErrorInvalidValue;
  return cudaGetLastError();
}

cudaError_t launch_triu_unpack(const void* line, void* dense, int elem_bytes, int batch, int n, cudaStream_t stream) {
  if (batch == 0 || n == 0) return cudaSuccess;
  dim3 grid(n, batch);
  if (elem_bytes == 4) triu_unpack_kernel<uint32_t><<<grid, 256, 0, stream>>>((const uint32_t*)line, (uint32_t*)dense, n);
  else if (elem_bytes == 2) triu_unpack_kernel<uint16_t><<<grid, 256, 0, stream>>>((const uint16_t*)line, (uint16_t*)dense, n);
  else return cudaErrorInvalidValue;
  return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------ around the eigenbasis refresh
// Passes over n x k matrices that only memory bounds: a block turns a few rows in shared memory, so that both sides are read and written
// in whole lines (16 of 1024^2: 33 us, back 34; the library's gather and scatter, element by element through 64-bit indices, 54 and 78).
__global__ void __launch_bounds__(256) permute_columns_kernel(const float* __restrict__ x, const long long* __restrict__ order, float* __restrict__ out,
                                                             int n, int k, int rows, int inverse) {
  extern __shared__ float turned[];  // rows x k
  const int r0 = blockIdx.x * rows, count = min(rows, n - r0);
  const long long base = ((long long)blockIdx.y * n + r0) * k;
  const long long* o = order + (long long)blockIdx.y * k;
  for (int j = threadIdx.x; j < k; j += blockDim.x) {
    const long long to = inverse ? o[j] : j;
    if (to < 0 || to >= k) continue;
#pragma unroll 8
    for (int r = 0; r < count; ++r) turned[r * k + to] = x[base + (long long)r * k + j];
  }
  __syncthreads();
  for (int j = threadIdx.x; j < k; j += blockDim.x) {
    const long long from = inverse ? j : o[j];
    if (from < 0 || from >= k) continue;
#pragma unroll 8
    for (int r = 0; r < count; ++r) out[base + (long long)r * k + j] = turned[r * k + from];
  }
}

cudaError_t launch_permute_columns(const float* x, const long long* order, float* out, int batch, int n, int k, int inverse, cudaStream_t stream) {
  if (batch == 0 || n == 0 || k == 0) return cudaSuccess;
  if (k > kMaxPermuted || batch > 65535) return cudaErrorInvalidValue;
  const int rows = kMaxPermuted / k < 8 ? kMaxPermuted / k : 8;  // 48 KB of shared memory at most
  permute_columns_kernel<<<dim3((n + rows - 1) / rows, batch), 256, (size_t)rows * k * sizeof(float), stream>>>(x, order, out, n, k, rows, inverse);
  return cudaGetLastError();
}

__global__ void __launch_bounds__(256) identity_defect_kernel(const float* __restrict__ G, long long ld, long long strideG, int k, float limit,
                                                             int* __restrict__ bad) {
  const int r = blockIdx.x * 8 + (threadIdx.x >> 5);
  bool off = false;
  if (r < k) {
    const float* row = G + blockIdx.y * strideG + r * ld;
#pragma unroll 8
    for (int c = threadIdx.x & 31; c < k; c += 32) off |= !(fabsf(row[c] - (c == r ? 1.0f : 0.0f)) <= limit);
  }
  if (__syncthreads_or(off) && threadIdx.x == 0) atomicOr(bad + blockIdx.y, 1);
}

cudaError_t launch_identity_defect(const float* G, long long ld, long long strideG, int batch, int k, float limit, int* bad, cudaStream_t stream) {
  if (batch == 0 || k == 0) return cudaSuccess;
  if (batch > 65535) return cudaErrorInvalidValue;
  identity_defect_kernel<<<dim3((k + 7) / 8, batch), 256, 0, stream>>>(G, ld, strideG, k, limit, bad);
  return cudaGetLastError();
}

}  // namespace hb
