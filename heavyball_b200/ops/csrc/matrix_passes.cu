// Element-wise passes around the matrix products of a PSGD fit and of an eigenbasis refresh.  Chains of the library's kernels move every
// intermediate through memory, and those that read across rows or broadcast a row run at a quarter of the bandwidth.  Each expression here
// is one pass with 16-byte accesses and the roundings of the chain it replaces: one per operation, divisions in full, subnormal values kept
// (the instructions are spelled out because the fast-math flags of this library would contract and approximate them).
// 8 of 1024^2 (33.5 MB each), chain / here: transposed copy 39 / 12 us, t1 + t2 and triu(t1 - t2) 59 / 18, damped gradient 57 / 13, packed step 42 / 16.
#include "matrix_passes.h"

namespace hb {
namespace {

__device__ __forceinline__ float add(float a, float b) {
  float r;
  asm("add.rn.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float sub(float a, float b) {
  float r;
  asm("sub.rn.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float mul(float a, float b) {
  float r;
  asm("mul.rn.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float div(float a, float b) {
  float r;
  asm("div.rn.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// 64 x 64 values per block through shared memory, 16 bytes per access either way where rows start on 16-byte boundaries.
__global__ void __launch_bounds__(256) transpose_kernel(const float* __restrict__ src, float* __restrict__ dst, int R, int C, int vec) {
  __shared__ float tile[64][65];
  const float* s = src + (int64_t)blockIdx.z * R * C;
  float* d = dst + (int64_t)blockIdx.z * R * C;
  const int c0 = blockIdx.x * 64, r0 = blockIdx.y * 64, q = (threadIdx.x & 15) * 4, line = threadIdx.x >> 4;
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const int r = line + 16 * p;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (r0 + r < R) {
      const float* row = s + (int64_t)(r0 + r) * C + c0 + q;
      if (vec) {
        if (c0 + q < C) {
          const float4 t = *(const float4*)row;
          v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
        }
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (c0 + q + e < C) v[e] = row[e];
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) tile[r][q + e] = v[e];
  }
  __syncthreads();
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const int c = line + 16 * p;
    if (c0 + c >= C) continue;
    float* row = d + (int64_t)(c0 + c) * R + r0 + q;
    if (vec) {
      if (r0 + q < R) *(float4*)row = make_float4(tile[q][c], tile[q + 1][c], tile[q + 2][c], tile[q + 3][c]);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (r0 + q + e < R) row[e] = tile[q + e][c];
    }
  }
}

template <typename V>  // float4, or float where n is not a multiple of 4
__global__ void __launch_bounds__(256) sum_triu_diff_kernel(V* __restrict__ a, V* __restrict__ b, int64_t count, int n) {
  constexpr int kWide = sizeof(V) / sizeof(float);
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += step) {
    V x = a[i], y = b[i];
    const int64_t at = i * kWide;
    const int col = (int)(at % n), row = (int)(at / n % n);
    float *px = (float*)&x, *py = (float*)&y;
#pragma unroll
    for (int e = 0; e < kWide; ++e) {
      const float u = px[e], w = py[e];
      px[e] = add(u, w);
      py[e] = col + e >= row ? sub(u, w) : 0.0f;
    }
    a[i] = x;
    b[i] = y;
  }
}

template <typename V>
__global__ void __launch_bounds__(256) dampen_kernel(const V* __restrict__ g, const V* __restrict__ v, V* __restrict__ out, int64_t count, float damp,
                                                    float eps) {
  constexpr int kWide = sizeof(V) / sizeof(float);
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += step) {
    V x = g[i];
    const V y = v[i];
    float* px = (float*)&x;
    const float* py = (const float*)&y;
#pragma unroll
    for (int e = 0; e < kWide; ++e) px[e] = add(px[e], mul(add(mul(fabsf(px[e]), eps), damp), py[e]));
    out[i] = x;
  }
}

// One row of one triangle per block: as packing it (skinny.cu), with the arithmetic on the way.
__global__ void __launch_bounds__(256) triu_step_kernel(const float* __restrict__ step, const float* __restrict__ ell, float* __restrict__ line, int n,
                                                       float lr) {
  const int64_t i = blockIdx.x, b = blockIdx.y, len = (int64_t)n * (n + 1) / 2;
  const float* s = step + (b * n + i) * n + i;
  float* t = line + b * len + i * n - i * (i - 1) / 2;
  const float by = ell[b];
#pragma unroll 4
  for (int j = threadIdx.x; j < n - (int)i; j += blockDim.x) t[j] = sub(t[j], mul(div(s[j], by), lr));
}

template <typename V>
__global__ void __launch_bounds__(256) scale_matrices_kernel(V* __restrict__ x, const float* __restrict__ by, int64_t count) {
  constexpr int kWide = sizeof(V) / sizeof(float);
  const int64_t base = blockIdx.y * count, step = (int64_t)gridDim.x * blockDim.x;
  const float s = by[blockIdx.y];
#pragma unroll 2
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += step) {
    V v = x[base + i];
    float* p = (float*)&v;
#pragma unroll
    for (int e = 0; e < kWide; ++e) p[e] = mul(p[e], s);
    x[base + i] = v;
  }
}

unsigned blocks_for(int64_t items) {
  const int64_t blocks = (items + 511) / 512;  // two steps a thread until the device is full several times over
  return (unsigned)(blocks < 1 ? 1 : blocks > 4736 ? 4736 : blocks);
}

}  // namespace

cudaError_t launch_transpose(const float* src, float* dst, int batch, int R, int C, cudaStream_t stream) {
  if (batch == 0 || R == 0 || C == 0) return cudaSuccess;
  if (batch > 65535 || (R + 63) / 64 > 65535) return cudaErrorInvalidValue;
  const int vec = (R & 3) == 0 && (C & 3) == 0 && (((uintptr_t)src | (uintptr_t)dst) & 15) == 0;
  transpose_kernel<<<dim3((C + 63) / 64, (R + 63) / 64, batch), 256, 0, stream>>>(src, dst, R, C, vec);
  return cudaGetLastError();
}

cudaError_t launch_sum_triu_diff(float* a, float* b, int batch, int n, cudaStream_t stream) {
  const int64_t count = (int64_t)batch * n * n;
  if (count == 0) return cudaSuccess;
  if ((n & 3) == 0 && (((uintptr_t)a | (uintptr_t)b) & 15) == 0)
    sum_triu_diff_kernel<<<blocks_for(count / 4), 256, 0, stream>>>((float4*)a, (float4*)b, count / 4, n);
  else
    sum_triu_diff_kernel<<<blocks_for(count), 256, 0, stream>>>(a, b, count, n);
  return cudaGetLastError();
}

cudaError_t launch_dampen(const float* g, const float* v, float* out, int64_t count, float damp, float eps, cudaStream_t stream) {
  if (count == 0) return cudaSuccess;
  if ((count & 3) == 0 && (((uintptr_t)g | (uintptr_t)v | (uintptr_t)out) & 15) == 0)
    dampen_kernel<<<blocks_for(count / 4), 256, 0, stream>>>((const float4*)g, (const float4*)v, (float4*)out, count / 4, damp, eps);
  else
    dampen_kernel<<<blocks_for(count), 256, 0, stream>>>(g, v, out, count, damp, eps);
  return cudaGetLastError();
}

cudaError_t launch_triu_step(const float* step, const float* ell, float* line, int batch, int n, float lr, cudaStream_t stream) {
  if (batch == 0 || n == 0) return cudaSuccess;
  if (batch > 65535) return cudaErrorInvalidValue;
  triu_step_kernel<<<dim3(n, batch), 256, 0, stream>>>(step, ell, line, n, lr);
  return cudaGetLastError();
}

cudaError_t launch_scale_matrices(float* x, const float* by, int batch, int64_t count, cudaStream_t stream) {
  if (batch == 0 || count == 0) return cudaSuccess;
  if (batch > 65535) return cudaErrorInvalidValue;
  if ((count & 3) == 0 && ((uintptr_t)x & 15) == 0)
    scale_matrices_kernel<<<dim3(blocks_for(count / 4), batch), 256, 0, stream>>>((float4*)x, by, count / 4);
  else
    scale_matrices_kernel<<<dim3(blocks_for(count), batch), 256, 0, stream>>>(x, by, count);
  return cudaGetLastError();
}

}  // namespace hb
