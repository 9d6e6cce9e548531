// fp32-in / fp32-out batched GEMM at fp32-level accuracy on the fp16 tensor-core path of sm_100a.
//
// The 3-term split product of tf32_gemm.cu with fp16 in the place of tf32: both carry 11 significant bits, so hi + lo keep 22 bits
// of a value either way, but fp16 operands are half as wide and their products run at twice the rate.  What fp16 lacks is range,
// hence one power of two per operand row that takes the row's largest value to the top of it and comes off again in the epilogue
// (exact both ways).  Values down to 2^-29 of their row's largest keep all 22 bits; below that the error is 2^-51 of the largest:
// far under the rounding of any sum in which both take part, but everything to a result that the largest has no part in (because it meets a
// zero, in triangular or block-diagonal factors).  The operand pass counts such values per row, the epilogue finds the results that may hang
// on them and computes those from the matrices (settle_slowly in gemm_epilogue.cuh).  Subnormal values are scaled like others.
//
// Three walks over K share one fp32 accumulator: hi lo^T and lo hi^T first, with lo stored times 2^11 (so that small values keep it,
// too), then hi hi^T on top, whose first instruction takes 2^-11 off the accumulator (the scale-input-d operand of tcgen05.mma).  The
// large sum is rounded once per 16 of K that way; with the high parts first, as tf32 walks them, the two small sums would be rounded
// at its magnitude as well.  Error against 64 bits, relative 2-norm, K = 1024 / 2048 / 8192: 1.2e-6 / 2.5e-6 / 9.7e-6 (tf32: 1.1e-5 /
// 2.1e-5 / 8.4e-5), the same with rows over thirty decades and with entries over eight decades along K.  Entry by entry, whatever the range:
// 2^-20 + (K / 16 + 4) 2^-23 of |A| |B|^T, tested over thirty decades along K opposite zeros.
//
// Measured on one B200, of measured peak (1.64 PFLOP/s / 3): 2 of 5504 x 2048 x 2048 205 us = 451 TFLOP/s, 0.82 (split tf32 340 us);
// 4 of 2048^3 159 us = 431, 0.79 (265); 8 of 1024^3 50 us = 346, 0.63, one wave (76).
#include "split16_gemm.h"

#include <cuda_fp16.h>

#include "gemm_epilogue.cuh"
#include "per_device.h"

namespace hb {
namespace {

constexpr int HBK = 64;  // fp16 elements of K in a 128-byte row
// fp16 x fp16 -> fp32, both operands K-major
constexpr uint32_t half_desc(int m, int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24); }

struct HalfKind {
  static constexpr int kBlock = HBK;
  static constexpr bool kScaled = true, kCrossFirst = true;
  static constexpr int kTermLoA = 1, kTermLoB = 0;  // A: hi, lo, hi   B: lo, hi, hi
  static constexpr uint32_t kDesc = half_desc(TBM, TBN), kPairDesc = half_desc(kPairTile, kPairTile);
  __device__ static __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t desc, uint32_t accumulate) {
    tc_mma_bf16(d, a, b, desc, accumulate);  // kind::f16; the operand type is in the descriptor
  }
  __device__ static __forceinline__ void mma_pair(uint32_t d, uint64_t a, uint64_t b, uint32_t desc, uint32_t accumulate) {
    tc_mma_bf16_pair(d, a, b, desc, accumulate);
  }
};

// ------------------------------------------------------------------------------------------ operand split
// One launch, two kinds of block; a row's exponent has to be known before its first value can be stored, so both kinds first look for
// the largest value and then convert:
//   blocks [0, row_blocks) : eight source rows, one per warp -> `same`
//   the others             : clusters of up to eight share a strip of 32 source columns, 256 rows at a time each, and exchange their
//                            column maxima -> `trans`, turned through shared memory
// What both saw first stays in registers (1024 columns of a row, 256 rows of a strip); only longer ones are read again, from L1 or L2.
// Bound by memory: 4 of 2048^2 rows 24 us (5.6 TB/s; split tf32, twice the bytes out, 37), columns 38 us, both 50 (59); one block per
// strip of 16 columns instead of a cluster 70 us for the columns.  Watching the smallest value costs the columns 4 % (43 -> 45 us from a cold
// L2), the rows nothing; counting every value as it is converted cost 9 %.
constexpr int kSplitThreads = 256;
constexpr int kRowChunk = 1024;
constexpr int kStrip = 32, kStripRows = 256, kMaxSplitCluster = 8;

// Largest absolute value (not counting NaN) and smallest one other than zero, the latter as its bits without the sign, shifted left, less
// one: zeros come out above everything.
struct RowRange {
  float top = 0.0f;
  uint32_t low = 0xFFFFFFFFu;
  __device__ __forceinline__ void add(float x) {
    top = fmaxf(top, fabsf(x));
    low = min(low, (__float_as_uint(x) << 1) - 1u);
  }
};
struct RowScale {
  float mul, unit;       // 2^e, 2^-e
  uint32_t short_below;  // 2^(-14 - e) in the form of RowRange::low: values under it are too small for 22 bits in a pair
};
__device__ __forceinline__ RowScale row_scale(uint32_t top_bits) {
  const int field = (int)(top_bits >> 23);
  // rows with an infinity stay as they are: all of their results are NaN (lo = inf - inf)
  if (field == 255) return {1.0f, 1.0f, 0u};
  const int e = min(126, 141 - field), f = 113 - e;  // f: exponent field of 2^(-14 - e); 0 and below: subnormal
  return {pow2(e), pow2(-e), ((f > 0 ? (uint32_t)f << 23 : 1u << (22 + f)) << 1) - 1u};
}
__device__ __forceinline__ uint32_t is_short(float x, uint32_t short_below) { return (__float_as_uint(x) << 1) - 1u < short_below ? 1u : 0u; }
// without flushing subnormals
__device__ __forceinline__ float scaled(float x, float mul) {
  float y;
  asm("mul.rn.f32 %0, %1, %2;" : "=f"(y) : "f"(x), "f"(mul));
  return y;
}
__device__ __forceinline__ void split_pair(float x, uint16_t& hi, uint16_t& lo) {
  const __half h = __float2half_rn(x);
  hi = __half_as_ushort(h);
  lo = __half_as_ushort(__float2half_rn((x - __half2float(h)) * 2048.0f));
}
__device__ __forceinline__ void split_store4(uint16_t* row, int64_t kp, const float (&x)[4]) {
  uint16_t h[4], l[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) split_pair(x[e], h[e], l[e]);
  *(uint2*)row = make_uint2((uint32_t)h[0] | ((uint32_t)h[1] << 16), (uint32_t)h[2] | ((uint32_t)h[3] << 16));
  *(uint2*)(row + kp) = make_uint2((uint32_t)l[0] | ((uint32_t)l[1] << 16), (uint32_t)l[2] | ((uint32_t)l[3] << 16));
}
__device__ __forceinline__ float4 load4(const float* p, int left, bool vec) {
  if (vec && left >= 4) return *(const float4*)p;
  return make_float4(left > 0 ? p[0] : 0.f, left > 1 ? p[1] : 0.f, left > 2 ? p[2] : 0.f, left > 3 ? p[3] : 0.f);
}

// position of row r of column c in the turned tile: four columns of a thread and four rows of a warp fall into distinct banks
__device__ __forceinline__ int turned(int c, int r) { return c * kStripRows + (r ^ (c & ~3)); }

// One or two source matrices per batch entry: the two operands of a product come from one launch, side by side (the blocks of the first
// come first), with the cluster of the one that needs the larger.  Such passes are short - 8 of 1024 x 128 rows 7.5 us, 8 of 128 x 128 columns 8.6 - and a pass of its own for the second operand was
// one more step of a chain of dependent launches: a PSGD fit of 8 of 1024^2 takes 1645 us with a launch each, 1621 with one.
struct SplitJob {
  const float* src;
  int64_t ld, stride;
  uint16_t *same, *trans;
  float *same_unit, *trans_unit;
  int R, C, row_blocks, blocks;  // of `blocks`, the first `row_blocks` write rows (both multiples of the cluster)
};
struct SplitJobs {
  SplitJob job[2];
};

__device__ __forceinline__ void split16_block(const float* __restrict__ src, int64_t ld_src, int64_t stride_src, int R, int C, int block, int row_blocks,
                                              int cluster, uint16_t* __restrict__ same, float* __restrict__ same_unit,
                                              uint16_t* __restrict__ trans, float* __restrict__ trans_unit) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t batch = blockIdx.y;
  const float* s = src + batch * stride_src;
  const bool vec = (ld_src & 3) == 0 && (stride_src & 3) == 0 && (((uintptr_t)src) & 15) == 0;

  if (block < row_blocks) {  // whole clusters take this branch (row_blocks is a multiple of `cluster`)
    const int r = block * (kSplitThreads / 32) + warp;
    if (r >= R) return;
    const int kp = (C + 63) / 64 * 64;
    const float* row = s + (int64_t)r * ld_src;
    float4 v[kRowChunk / 128];
    RowRange range;
    uint32_t n_short = 0;
    const auto fetch = [&](int base) {
#pragma unroll
      for (int i = 0; i < kRowChunk / 128; ++i) {
        const int c = base + i * 128 + lane * 4;
        v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c < C) v[i] = load4(row + c, C - c, vec);
      }
    };
    for (int base = 0; base < C; base += kRowChunk) {
      fetch(base);
#pragma unroll
      for (int i = 0; i < kRowChunk / 128; ++i) {
        range.add(v[i].x);
        range.add(v[i].y);
        range.add(v[i].z);
        range.add(v[i].w);
      }
    }
    const RowScale f = row_scale(__reduce_max_sync(0xFFFFFFFFu, __float_as_uint(range.top)));
    uint16_t* dst = same + (batch * R + r) * 2 * kp;
    for (int base = 0; base < C; base += kRowChunk) {
      if (C > kRowChunk) fetch(base);
      if (range.low < f.short_below) {
#pragma unroll
        for (int i = 0; i < kRowChunk / 128; ++i)
          n_short += is_short(v[i].x, f.short_below) + is_short(v[i].y, f.short_below) + is_short(v[i].z, f.short_below) + is_short(v[i].w, f.short_below);
      }
#pragma unroll
      for (int i = 0; i < kRowChunk / 128; ++i) {
        const int c = base + i * 128 + lane * 4;
        if (c < kp) {
          const float x[4] = {scaled(v[i].x, f.mul), scaled(v[i].y, f.mul), scaled(v[i].z, f.mul), scaled(v[i].w, f.mul)};
          split_store4(dst + c, kp, x);
        }
      }
    }
    n_short = min(__reduce_add_sync(0xFFFFFFFFu, n_short), kManyShort);
    if (lane == 0) same_unit[batch * ((R + 255) / 256 * 256) + r] = __uint_as_float(__float_as_uint(f.unit) | n_short);
    return;
  }

  __shared__ __align__(16) float tile[kStrip * kStripRows];
  __shared__ uint32_t warp_tops[kSplitThreads / 32][kStrip];
  __shared__ uint32_t tops[kStrip];  // of this block's rows; the blocks of the cluster read each other's
  __shared__ uint32_t short_below[kStrip], shorts[kStrip];
  __shared__ float muls[kStrip];
  const int at = block - row_blocks, rank = at % cluster, c0 = at / cluster * kStrip;
  const int q = threadIdx.x & 7, line = threadIdx.x >> 3, c = c0 + q * 4, kp = (R + 63) / 64 * 64;
  const int first = rank * kStripRows, step = cluster * kStripRows;
  float4 v[kStripRows / 32];
  const auto fetch = [&](int r0) {  // rows r0 + line + 32 i, four columns each
#pragma unroll
    for (int i = 0; i < kStripRows / 32; ++i) {
      const int r = r0 + line + 32 * i;
      v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < R && c < C) v[i] = load4(s + (int64_t)r * ld_src + c, C - c, vec);
    }
  };
  RowRange range[4];
  for (int r0 = first; r0 < R; r0 += step) {
    fetch(r0);
#pragma unroll
    for (int i = 0; i < kStripRows / 32; ++i) {
      range[0].add(v[i].x);
      range[1].add(v[i].y);
      range[2].add(v[i].z);
      range[3].add(v[i].w);
    }
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    float top = fmaxf(range[e].top, __shfl_xor_sync(0xFFFFFFFFu, range[e].top, 8));
    top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, 16));
    if (lane < 8) warp_tops[warp][lane * 4 + e] = __float_as_uint(top);
  }
  __syncthreads();
  if (threadIdx.x < kStrip) {
    uint32_t t = 0;
#pragma unroll
    for (int w = 0; w < kSplitThreads / 32; ++w) t = max(t, warp_tops[w][threadIdx.x]);
    tops[threadIdx.x] = t;
    shorts[threadIdx.x] = 0;
  }
  if (cluster > 1) cluster_sync(); else __syncthreads();
  if (threadIdx.x < kStrip) {
    uint32_t t = tops[threadIdx.x];
    for (int k = 1; k < cluster; ++k)
      t = max(t, (uint32_t)cluster_load(cluster_addr(&tops[threadIdx.x], (rank + k) % cluster)));
    const RowScale f = row_scale(t);
    muls[threadIdx.x] = f.mul;
    short_below[threadIdx.x] = f.short_below;
    if (rank == 0 && c0 + (int)threadIdx.x < C) trans_unit[batch * ((C + 255) / 256 * 256) + c0 + threadIdx.x] = f.unit;
  }
  if (cluster > 1) cluster_sync(); else __syncthreads();  // no block leaves while its maxima may still be read
  const int oc = threadIdx.x >> 4, k4 = (threadIdx.x & 15) * 4;  // output: rows c0 + oc (+ 16) of the operand, four of K at a time
  for (int r0 = first; r0 < R; r0 += step) {
    if (R > step) fetch(r0);
#pragma unroll
    for (int i = 0; i < kStripRows / 32; ++i) {
      const int r = line + 32 * i;
      tile[turned(q * 4 + 0, r)] = scaled(v[i].x, muls[q * 4 + 0]);
      tile[turned(q * 4 + 1, r)] = scaled(v[i].y, muls[q * 4 + 1]);
      tile[turned(q * 4 + 2, r)] = scaled(v[i].z, muls[q * 4 + 2]);
      tile[turned(q * 4 + 3, r)] = scaled(v[i].w, muls[q * 4 + 3]);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const uint32_t below = short_below[q * 4 + e];
      if (range[e].low < below) {  // this thread has some in column e
        uint32_t n = 0;
#pragma unroll
        for (int i = 0; i < kStripRows / 32; ++i) n += is_short(e == 0 ? v[i].x : e == 1 ? v[i].y : e == 2 ? v[i].z : v[i].w, below);
        atomicAdd(&shorts[q * 4 + e], n);
      }
    }
    __syncthreads();
#pragma unroll
    for (int g = 0; g < kStrip; g += 16) {
      if (c0 + oc + g >= C) continue;
      uint16_t* dst = trans + (batch * C + c0 + oc + g) * 2 * kp + r0;
#pragma unroll
      for (int k = k4; k < kStripRows; k += 64) {
        if (r0 + k < kp) {
          const float4 t = *(const float4*)&tile[turned(oc + g, k)];
          const float x[4] = {t.x, t.y, t.z, t.w};
          split_store4(dst + k, kp, x);
        }
      }
    }
    __syncthreads();
  }
  // (rank 0's unit is there: the cluster has met since)
  if (threadIdx.x < kStrip && c0 + (int)threadIdx.x < C && shorts[threadIdx.x] != 0)
    atomicAdd((uint32_t*)&trans_unit[batch * ((C + 255) / 256 * 256) + c0 + threadIdx.x], min(shorts[threadIdx.x], kManyShort));
}

// A kernel of its own for a single matrix: with the arguments behind a choice the column passes are 3 % slower (2 of 4096^2 71.7 -> 73.9 us).
__global__ void __launch_bounds__(kSplitThreads, 4) split16_kernel(const float* __restrict__ src, int64_t ld_src, int64_t stride_src, int R, int C,
                                                                 int row_blocks, int cluster, uint16_t* __restrict__ same,
                                                                 float* __restrict__ same_unit, uint16_t* __restrict__ trans,
                                                                 float* __restrict__ trans_unit) {
  griddep_wait();
  griddep_launch();
  split16_block(src, ld_src, stride_src, R, C, blockIdx.x, row_blocks, cluster, same, same_unit, trans, trans_unit);
}
__global__ void __launch_bounds__(kSplitThreads, 4) split16_two_kernel(const __grid_constant__ SplitJobs jobs, int cluster) {
  griddep_wait();
  griddep_launch();
  const bool second = (int)blockIdx.x >= jobs.job[0].blocks;  // the same for the blocks of a cluster
  const SplitJob& J = jobs.job[second];
  split16_block(J.src, J.ld, J.stride, J.R, J.C, (int)blockIdx.x - (second ? jobs.job[0].blocks : 0), J.row_blocks, cluster, J.same, J.same_unit,
                J.trans, J.trans_unit);
}

// fp16 operand [batch, rows, cols]; box = 64 columns x 128 rows, 128-byte swizzle
bool make_half_map(CUtensorMap* map, const void* base, int rows, int64_t cols, int batch) {
  EncodeTiledFn fn = tensor_map_encoder();
  if (fn == nullptr) return false;
  cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)batch};
  cuuint64_t strides[2] = {(cuuint64_t)cols * 2, (cuuint64_t)cols * rows * 2};
  cuuint32_t box[3] = {HBK, TBM, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// fp32 output for the 128 x 128 kernel's bulk stores; box = 32 columns x 128 rows
bool make_store_map(CUtensorMap* map, float* base, int rows, int cols, int64_t ld, int64_t stride, int batch) {
  EncodeTiledFn fn = tensor_map_encoder();
  if (fn == nullptr) return false;
  cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)batch};
  cuuint64_t strides[2] = {(cuuint64_t)ld * 4, (cuuint64_t)stride * 4};
  cuuint32_t box[3] = {32, TBM, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Whether a product takes pairs, from the waves that 128 x 128 tiles (four in the place of a pair) and pairs need.  150 sizes measured,
// 128 / pairs:
//   - More than one wave of small tiles, in about as many waves of pairs: pairs from K = 512 on (8 of 3000 x 4096 x 768 531 / 356 us, 6 of
//     5504 x 1536 x 512 219 / 159, 16 of 512 x 1024 x 640 45.3 / 41.8).  With a shorter K the three walks do not cover a pair's epilogue (16 of
//     1024 x 768 x 128 28.7 / 36.0, 3000 x 2048 x 384 25.3 / 30.7), except where the mirrored stores of a symmetric product make either
//     epilogue long (3 of 4096 x 4096 x 256 119 / 107).  A half more waves cost more than the tile gains (16 of 1000 x 1000 x 4096
//     symmetric, two waves or three, 253 / 277).
//   - One wave of either: pairs where most of them have work and K is long (4 of 768 x 1024 x 5504 120 / 103, 3 of 384 x 2048 x 3000 60.5 / 62.4);
//     else the small tiles, which are more (640 x 512 x 2048 30.2 / 41.3).
// The worst of the 150 loses 11 %, the mean 0.2 %.
bool split16_take_pairs(int M, int N, int K, bool symmetric, int64_t small_waves, int64_t big_waves, int64_t big, int64_t pairs) {
  if (M <= 128 || N <= 128) return false;
  if (small_waves >= 2) return 3 * big_waves <= 4 * small_waves && (K >= 512 || (symmetric && small_waves >= 4));
  return K >= 3000 && 7 * big >= 4 * pairs && big_waves == 1;
}

int g_split16_tile = 0;

}  // namespace

void set_split16_gemm_tile_override(int tile) { g_split16_tile = (tile == 128 || tile == 256) ? tile : 0; }

cudaError_t launch_split16(const Split16Pass* passes, int n, int batch, cudaStream_t stream) {
  SplitJobs jobs{};
  if (n < 1 || n > 2 || batch == 0) return n < 1 || n > 2 ? cudaErrorInvalidValue : cudaSuccess;
  int cluster = 1;  // strips longer than one block's rows are shared
  for (int i = 0; i < n; ++i)
    while (passes[i].trans.data != nullptr && cluster < kMaxSplitCluster && cluster * kStripRows < passes[i].R) cluster *= 2;
  int used = 0, blocks = 0;
  for (int i = 0; i < n; ++i) {
    const Split16Pass& p = passes[i];
    if (p.R == 0 || p.C == 0 || (p.same.data == nullptr && p.trans.data == nullptr)) continue;
    const int strips = p.trans.data != nullptr ? (p.C + kStrip - 1) / kStrip : 0;
    int row_blocks = p.same.data != nullptr ? (p.R + kSplitThreads / 32 - 1) / (kSplitThreads / 32) : 0;
    row_blocks = (row_blocks + cluster - 1) / cluster * cluster;
    jobs.job[used] = {p.src, p.ld, p.stride, (uint16_t*)p.same.data, (uint16_t*)p.trans.data, p.same.unit, p.trans.unit,
                      p.R, p.C, row_blocks, row_blocks + strips * cluster};
    blocks += jobs.job[used++].blocks;
  }
  if (used == 0) return cudaSuccess;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(blocks, batch);
  cfg.blockDim = dim3(kSplitThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  if (used == 2) return cudaLaunchKernelEx(&cfg, split16_two_kernel, jobs, cluster);
  const SplitJob& J = jobs.job[0];
  return cudaLaunchKernelEx(&cfg, split16_kernel, J.src, J.ld, J.stride, J.R, J.C, J.row_blocks, cluster, J.same, J.same_unit, J.trans, J.trans_unit);
}

cudaError_t launch_split16_gemm(Split16Operand A, Split16Operand B, int M, int N, int K, int batch, const Tf32Epilogue& E, int* status,
                                cudaStream_t stream) {
  static PerDevice<int> pairs;
  int device = 0, max_pairs = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e == cudaSuccess)
    e = pairs.get(device, cudaSuccess, &max_pairs, [](int& found) {
      cudaError_t s = cudaFuncSetAttribute(gemm128_kernel<HalfKind>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTSmemBytes);
      if (s == cudaSuccess) s = cudaFuncSetAttribute(gemm_pair_kernel<HalfKind>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGPairSmemBytes);
      return s != cudaSuccess ? s : max_resident_pairs(gemm_pair_kernel<HalfKind>, kGPairThreads, kGPairSmemBytes, &found);
    });
  if (e != cudaSuccess) return e;
  if (M == 0 || N == 0 || batch == 0) return cudaSuccess;
  const bool moments = E.mode == kEpiAdam || E.mode == kEpiLaProp;
  if (K == 0 || A.src.p == nullptr || B.src.p == nullptr || E.S != nullptr || (moments && (E.m == nullptr || E.v == nullptr))) return cudaErrorInvalidValue;
  if (!moments && E.C == nullptr) return cudaErrorInvalidValue;
  if (E.tri && (M != N || M != K || E.symmetric)) return cudaErrorInvalidValue;
  if (E.symmetric && (A.data != B.data || M != N || E.C == nullptr || moments)) return cudaErrorInvalidValue;
  const int64_t kp = split16_kp(K);
  const auto pair_operand = [](const Split16Operand& o, int64_t rows) {
    return PairOperand{o.unit, split16_units(rows), o.src.p, o.src.batch, o.src.row, o.src.k};
  };
  const PairOperands P{pair_operand(A, M), pair_operand(B, N), K};
  CUtensorMap ma, mb;
  if (!make_half_map(&ma, A.data, M, 2 * kp, batch) || !make_half_map(&mb, B.data, N, 2 * kp, batch)) return cudaErrorInvalidValue;
  const auto tiles = [&](int tile) {
    const int m = (M + tile - 1) / tile, n = (N + tile - 1) / tile;
    return E.symmetric ? n * (n + 1) / 2 : m * n;
  };
  const int64_t small = (int64_t)tiles(TBM) * batch, big = (int64_t)tiles(kPairTile) * batch;
  const int64_t small_waves = (small + 4 * max_pairs - 1) / (4 * max_pairs), big_waves = (big + max_pairs - 1) / max_pairs;
  bool pair = split16_take_pairs(M, N, K, E.symmetric != 0, small_waves, big_waves, big, max_pairs);
  if (g_split16_tile != 0) pair = g_split16_tile == 256;
  if (pair) {
    const int tm = (M + kPairTile - 1) / kPairTile, tn = (N + kPairTile - 1) / kPairTile;
    const int grid = 2 * (int)(big < max_pairs ? big : max_pairs);
    return launch_chained(gemm_pair_kernel<HalfKind>, dim3(grid), kGPairThreads, kGPairSmemBytes, stream, ma, mb, M, N, (int)kp, (int)kp, (int)kp, tm, tn,
                          tiles(kPairTile), (int)big, E, P, status);
  }
  // bulk stores end on 16-byte boundaries: with N a multiple of 4 they write nothing past it
  const int bulk = (!E.symmetric && !E.tri && E.mode == kEpiStore && (N & 3) == 0 && (E.ldc & 3) == 0 && (E.strideC & 3) == 0 &&
                    (((uintptr_t)E.C) & 15) == 0) ? 1 : 0;
  CUtensorMap mc = ma;  // placeholder when the bulk-store path is not taken (never dereferenced then)
  if (bulk && !make_store_map(&mc, E.C, M, N, E.ldc, E.strideC, batch)) return cudaErrorInvalidValue;
  return launch_chained(gemm128_kernel<HalfKind>, dim3(tiles(TBM), batch), kTThreads, kTSmemBytes, stream, ma, mb, mc, M, N, (int)kp, (int)kp, (int)kp, E, P, bulk,
                        status);
}

}  // namespace hb
