// Power iteration on A^2 for the step length of a PSGD fit: heavyball/utils.py's estimate of the largest eigenvalue, started from A's largest row.
//
// As single operations that is thirty dependent launches per factor: row norms, their maximum, a gather, A over the largest norm, and for every
// product a matrix-vector kernel, a norm, a clamp and a division.  Here a cluster of CTAs takes a matrix from beginning to end.  A CTA owns a
// share of the rows, which it reads once for the norms and twice a step (from the L2: 4 MB at 1024), a warp four rows at a time; every CTA keeps
// the whole vectors in shared memory, and each product's entries are stored into all of them.  What is left of each step is the reading and one
// cluster barrier per product.  A is scaled by a power of two near its largest row norm on the way, entry by entry: what may not leave fp32 are the
// squares of its entries and their sums along a row.
// Two factors of 8 of 1024^2, two iterations each, in the graph of a fit: 245 us of the library's kernels, 2 x 51 here.
#include "power_iteration.h"

#include "per_device.h"
#include "tc_common.cuh"

namespace hb {
namespace {

constexpr int kPowerThreads = 512, kPowerWarps = kPowerThreads / 32;
constexpr int kPowerRows = 4;  // of a warp at a time

// Subnormal values are kept (squares of a small A's entries), against the flags of this library.
__device__ __forceinline__ float fma_full(float a, float b, float c) {
  float r;
  asm("fma.rn.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float mul_full(float a, float b) {
  float r;
  asm("mul.rn.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float add_full(float a, float b) {
  float r;
  asm("add.rn.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float sqrt_full(float a) {
  float r;
  asm("sqrt.rn.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ float div_full(float a, float b) {
  float r;
  asm("div.rn.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// A and the vectors are scaled by powers of two, which rounds nothing; what is left of the vector's length is divided out at the end.  Of a value
// that is not finite: NaN.
__device__ __forceinline__ float power_of_two(float v) { return v < 1.7e38f ? __uint_as_float(__float_as_uint(v) & 0x7F800000u) : v - v; }
__device__ __forceinline__ float inverse_power(float p) { return p > 0.0f ? __uint_as_float((254u << 23) - __float_as_uint(p)) : p; }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = add_full(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
  return v;
}
__device__ __forceinline__ float block_sum(float v, float* scratch) {
  v = warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
  __syncthreads();
  return warp_sum((threadIdx.x & 31) < kPowerWarps ? scratch[threadIdx.x & 31] : 0.0f);
}
// One value per row, from the lanes that hold it to the same place of every CTA.
__device__ __forceinline__ void store_everywhere(float* to, float v, int lane, int ctas) {
  if (lane < ctas) cluster_store(cluster_addr(to, (uint32_t)lane), __float_as_int(v));
}

// The row to start from: a NaN before any number, then the largest norm, of equal ones the first row.  Which of them it is decides what a
// block-diagonal matrix converges to.
__device__ __forceinline__ bool ranks_before(float norm, int row, float than, int than_row) {
  if (isnan(norm) || isnan(than)) return isnan(norm) && (!isnan(than) || row < than_row);
  return norm > than || (norm == than && row < than_row);
}

// For each row r of [first, last): done(r, s, lane) with s from zero through s <- term(s, a_rk, k).
template <bool kWide, class Term, class Done>
__device__ __forceinline__ void over_rows(const float* __restrict__ A, int n, int first, int last, const Term& term, const Done& done) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int r0 = first + warp * kPowerRows; r0 < last; r0 += kPowerWarps * kPowerRows) {
    float s[kPowerRows] = {};
    const float* row[kPowerRows];
#pragma unroll
    for (int i = 0; i < kPowerRows; ++i) row[i] = A + (int64_t)min(r0 + i, last - 1) * n;
    if (kWide) {
#pragma unroll 2
      for (int k = lane * 4; k < n; k += 128) {
        float4 a[kPowerRows];
#pragma unroll
        for (int i = 0; i < kPowerRows; ++i) a[i] = *(const float4*)(row[i] + k);
#pragma unroll
        for (int i = 0; i < kPowerRows; ++i) {
          s[i] = term(s[i], a[i].x, k);
          s[i] = term(s[i], a[i].y, k + 1);
          s[i] = term(s[i], a[i].z, k + 2);
          s[i] = term(s[i], a[i].w, k + 3);
        }
      }
    } else {
      for (int k = lane; k < n; k += 32) {
#pragma unroll
        for (int i = 0; i < kPowerRows; ++i) s[i] = term(s[i], row[i][k], k);
      }
    }
#pragma unroll
    for (int i = 0; i < kPowerRows; ++i) {
      const float total = warp_sum(s[i]);
      if (r0 + i < last) done(r0 + i, total, lane);
    }
  }
}

template <bool kWide>
__global__ void __launch_bounds__(kPowerThreads) power_iteration_kernel(const float* __restrict__ matrices, int n, int iterations, int ctas,
                                                                       float* __restrict__ out) {
  extern __shared__ __align__(16) float vectors[];  // three of n, padded to 16 bytes
  __shared__ float scratch[kPowerWarps], best_norm[kPowerWarps];
  __shared__ int best_row[kPowerWarps];
  const int pad = (n + 3) & ~3;
  float *const x = vectors, *const ax = vectors + pad, *const aax = vectors + 2 * pad;
  const int rank = (int)cluster_rank(), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float* A = matrices + (int64_t)(blockIdx.x / ctas) * n * n;
  const int per = (n + ctas - 1) / ctas, first = min(n, rank * per), last = min(n, first + per);
  cluster_sync();  // every CTA's shared memory is there to be written

  over_rows<kWide>(A, n, first, last, [](float s, float a, int) { return fma_full(a, a, s); },
                   [&](int r, float s, int l) { store_everywhere(aax + r, sqrt_full(s), l, ctas); });
  cluster_sync();
  float norm = -1.0f;
  int at = 0;
  for (int i = threadIdx.x; i < n; i += kPowerThreads)
    if (ranks_before(aax[i], i, norm, at)) {
      norm = aax[i];
      at = i;
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float other = __shfl_xor_sync(0xFFFFFFFFu, norm, o);
    const int other_at = __shfl_xor_sync(0xFFFFFFFFu, at, o);
    if (ranks_before(other, other_at, norm, at)) {
      norm = other;
      at = other_at;
    }
  }
  if (lane == 0) {
    best_norm[warp] = norm;
    best_row[warp] = at;
  }
  __syncthreads();
  norm = best_norm[0];
  at = best_row[0];
  for (int w = 1; w < kPowerWarps; ++w)
    if (ranks_before(best_norm[w], best_row[w], norm, at)) {
      norm = best_norm[w];
      at = best_row[w];
    }
  const float top = norm < 1.17549435e-38f ? 1.17549435e-38f : norm;
  const float unit = power_of_two(top), by = inverse_power(unit);
  for (int k = threadIdx.x; k < n; k += kPowerThreads) x[k] = mul_full(A[(int64_t)at * n + k], by);
  cluster_sync();  // x is complete, and nobody reads the norms any more

  const auto times = [&](const float* v, float* to) {
    over_rows<kWide>(A, n, first, last, [&](float s, float a, int k) { return fma_full(mul_full(a, by), v[k], s); }, [&](int r, float s, int l) { store_everywhere(to + r, s, l, ctas); });
    cluster_sync();
  };
  const auto times_itself = [&](const float* v) {
    float s = 0.0f;
    for (int k = threadIdx.x; k < n; k += kPowerThreads) s = fma_full(x[k], v[k], s);
    return block_sum(s, scratch);
  };
  bool vanished = false;  // a vector shorter than 1e-12 counts as one of that length
  for (int it = 0; it < iterations; ++it) {
    times(x, ax);
    times(ax, aax);
    float s = 0.0f;
    for (int k = threadIdx.x; k < n; k += kPowerThreads) s = fma_full(aax[k], aax[k], s);
    const float length = sqrt_full(block_sum(s, scratch));
    vanished = length < 1e-12f;
    const float inv = vanished ? 1e12f : inverse_power(power_of_two(length));
    for (int k = threadIdx.x; k < n; k += kPowerThreads) x[k] = mul_full(aax[k], inv);
    __syncthreads();
  }
  times(x, ax);
  times(ax, aax);
  const float product = times_itself(aax), square = times_itself(x);
  if (rank == 0 && threadIdx.x == 0) out[blockIdx.x / ctas] = mul_full(sqrt_full(vanished || square == 0.0f ? product : div_full(product, square)), unit);
}

}  // namespace

cudaError_t launch_power_iteration(const float* A, int batch, int n, int iterations, float* out, cudaStream_t stream) {
  const bool wide = (n & 3) == 0 && ((uintptr_t)A & 15) == 0;
  const auto kernel = wide ? power_iteration_kernel<true> : power_iteration_kernel<false>;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.blockDim = dim3(kPowerThreads);
  cfg.dynamicSmemBytes = 3 * ((n + 3) & ~3) * sizeof(float);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const auto shape = [&](int ctas) {
    attr[0].val.clusterDim.x = ctas;
    cfg.gridDim = dim3(batch * ctas);
  };
  struct Device {
    int clusters, sms;  // of sixteen that it holds at once
  } on{};
  static PerDevice<Device> devices;
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e == cudaSuccess)
    e = devices.get(device, cudaSuccess, &on, [device](Device& found) {
      for (const auto k : {power_iteration_kernel<true>, power_iteration_kernel<false>})
        if (const cudaError_t s = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1); s != cudaSuccess) return s;
      cudaLaunchConfig_t c{};
      cudaLaunchAttribute a[1];
      a[0].id = cudaLaunchAttributeClusterDimension;
      a[0].val.clusterDim.x = 16;
      a[0].val.clusterDim.y = a[0].val.clusterDim.z = 1;
      c.gridDim = dim3(16);
      c.blockDim = dim3(kPowerThreads);
      c.dynamicSmemBytes = 3 * kMaxPowerSize * sizeof(float);
      c.attrs = a;
      c.numAttrs = 1;
      if (const cudaError_t s = cudaOccupancyMaxActiveClusters(&found.clusters, power_iteration_kernel<true>, &c); s != cudaSuccess) return s;
      return cudaDeviceGetAttribute(&found.sms, cudaDevAttrMultiProcessorCount, device);
    });
  if (e != cudaSuccess) return e;
  if (n > kMaxPowerSize || iterations < 0) return cudaErrorInvalidValue;
  if (batch == 0 || n == 0) return cudaSuccess;
  // Sixteen where every matrix still gets its cluster at once and has rows for them, else eight (two iterations, 8 / 16 CTAs: four of 512^2
  // 21 / 23 us, of 1024^2 48 / 37, of 2048^2 146 / 138, three of them 146 / 88).  Many small matrices fill the device by themselves, and waves of short
  // CTAs with barriers between them are all that larger clusters add: while there are more than two CTAs per SM, half as many, as long as each has
  // no more than 128 rows (8 / 4 / 2 / 1 CTAs: 64 of 64^2 26 / 13 / 12 / 14 us, 1024 of them 382 / 167 / 81 / 57, 256 of 128^2 106 / 51 / 31 / 24, 64 of 256^2
  // 40 / 22 / 24 / 35, 300 of 512^2 305 / 230 / 366 / 400).
  int ctas = batch <= on.clusters && n >= 512 ? 16 : 8;
  while (ctas > 1 && ctas <= 8 && (int64_t)batch * ctas > 2 * on.sms && ctas / 2 * 128 >= n) ctas /= 2;
  shape(ctas);
  return cudaLaunchKernelEx(&cfg, kernel, A, n, iterations, ctas, out);
}

}  // namespace hb
