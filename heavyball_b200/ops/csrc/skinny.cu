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
// Both leaf kernels work on one (up to) 128 x 128 block per CTA of 512 threads, the block and its inverse in shared memory
// as 4 x 4 sub-blocks of 32.  A refresh of an eigenbasis factors 16 leaves per 2048-wide factor and round, one after the
// other, so the latency of one CTA is all that counts; it is set by the length of the dependent chain, not by the 0.7 MFLOP.
//   factor R^T R = G, panel of 32 rows by panel: the 32 x 32 diagonal block in one warp (lane = column, the column in registers), four pivots at
//     a time, whose 4 x 4 block every lane factors for itself; rows and reciprocal pivots go through shared memory, where three more warps
//     pick them up four at a time and carry the columns to the right along (a barrier per step).  Then the trailing blocks by a rank-32
//     update, 4 x 4 values per lane.  Every element receives the same products in the same order as in an element-wise right-looking
//     factorisation.
//   invert R, column of blocks by column while the next panel is factored:  X_JJ by one warp (lane = column in registers), then upwards
//     X_IJ = -X_II (sum_{K = I+1 .. J} R_IK X_KJ) by eight warps, 2 x 2 values per lane.
// 54 -> 25 us for 16 leaves (SM clocks of the former / this form: diagonal blocks 4 x 15.7k / 4.1k to 8k, with the inverse's columns under them;
// rows to the right 3 x 2.7k / hidden; trailing 9.3k / 6k; inverse 20.7k / 9.9k behind the last panel; load 4k / 2k; store 5.4k / 2.1k).  The former
// shuffled every multiplier: in a branch on the warp's number, which the compiler takes for divergent, shuffles go one at a time, 490 clocks
// a pivot.  Hence the warp's number by a shuffle, too (uniform), and loads in groups before the arithmetic that uses them.
// A non-positive or non-finite pivot is replaced by 1 and counted in info[b] (the result for that matrix is then
// meaningless, the others are unaffected).
namespace {

constexpr int kLeafThreads = 512;
constexpr int kLeafLd = kTriBlock + 4;  // rows start on 16-byte boundaries: four values of a row per (broadcast) load
constexpr int kLeafBytes = 2 * kTriBlock * kLeafLd * (int)sizeof(float);
constexpr int kSub = 32, kSubs = kTriBlock / kSub;
constexpr int kLoads = kTriBlock * kTriBlock / 4 / kLeafThreads;

// Named barriers of part of a block.
enum LeafBarrier : int { kLowWarps = 1, kHighWarps = 2, kPanelStep = 4 };  // kPanelStep .. + 7: the eight steps of a panel
template <int kThreads>
__device__ __forceinline__ void part_sync(int id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(kThreads) : "memory"); }
template <int kThreads>
__device__ __forceinline__ void part_arrive(int id) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(kThreads) : "memory"); }


// Loads the upper part of a block of `size` rows (what lies left of the diagonal is anything); a short block is completed by an identity.
__device__ __forceinline__ void load_upper(const float* __restrict__ g, long long ld, int size, float* t) {
  if (size == kTriBlock && (ld & 3) == 0 && ((uintptr_t)g & 15) == 0) {
    float4 v[kLoads];
#pragma unroll
    for (int e = 0; e < kLoads; ++e) {
      const int idx = threadIdx.x + e * kLeafThreads, i = idx >> 5, j = (idx & 31) * 4;
      v[e] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (j + 3 >= i) v[e] = *(const float4*)(g + (long long)i * ld + j);
    }
#pragma unroll
    for (int e = 0; e < kLoads; ++e) {
      const int idx = threadIdx.x + e * kLeafThreads, i = idx >> 5, j = (idx & 31) * 4;
      *(float4*)(t + i * kLeafLd + j) = v[e];
    }
  } else {
    for (int idx = threadIdx.x; idx < kTriBlock * kTriBlock; idx += kLeafThreads) {
      const int i = idx >> 7, j = idx & (kTriBlock - 1);
      float v = i == j ? 1.f : 0.f;
      if (i < size && j < size && j >= i) v = g[(long long)i * ld + j];
      t[i * kLeafLd + j] = v;
    }
  }
}

struct Pivot {
  float inv, root;
  bool ok;
};
__device__ __forceinline__ Pivot pivot_of(float piv) {
  Pivot p;
  p.ok = piv > 0.f && piv < 3.0e38f;
  const float r = rsqrtf(piv);
  p.inv = p.ok ? r : 1.f;
  p.root = p.ok ? piv * p.inv : 1.f;
  return p;
}

// A panel on its way from the warp that factors to those that follow: reciprocal pivots and rows, four at a time.
struct Panel {
  float4 inv[kSub / 4];
  float4 row[kSub / 4][kSub];
};

// 32 x 32 diagonal block by one warp
__device__ __forceinline__ bool factor_diagonal(float* d, Panel& P) {
  const int lane = threadIdx.x & 31;
  float a[kSub], p[4][4];
  bool bad = false;
#pragma unroll
  for (int i = 0; i < kSub; ++i) a[i] = d[i * kLeafLd + lane];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = r; c < 4; ++c) p[r][c] = d[r * kLeafLd + c];
#pragma unroll
  for (int k = 0; k < kSub; k += 4) {
    float m[4][4], inv[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const Pivot v = pivot_of(p[r][r]);
      bad |= !v.ok;
      inv[r] = v.inv;
#pragma unroll
      for (int c = r + 1; c < 4; ++c) m[r][c] = p[r][c] * v.inv;
#pragma unroll
      for (int i = r + 1; i < 4; ++i)
#pragma unroll
        for (int c = i; c < 4; ++c) p[i][c] = fmaf(-m[r][i], m[r][c], p[i][c]);
      a[k + r] = lane == k + r ? v.root : a[k + r] * v.inv;
#pragma unroll
      for (int i = r + 1; i < 4; ++i) a[k + i] = fmaf(-m[r][i], a[k + r], a[k + i]);
    }
    float4* row = P.row[k >> 2];
    row[lane] = make_float4(a[k], a[k + 1], a[k + 2], a[k + 3]);
    if (lane == 0) P.inv[k >> 2] = make_float4(inv[0], inv[1], inv[2], inv[3]);
    __syncwarp();
    part_arrive<128>(kPanelStep + (k >> 2));
#pragma unroll
    for (int i0 = k + 4; i0 < kSub; i0 += 4) {
      float4 r[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) r[e] = row[i0 + e];
#pragma unroll
      for (int e = 0; e < 4; ++e) a[i0 + e] = fmaf(-r[e].x, a[k], a[i0 + e]);
#pragma unroll
      for (int e = 0; e < 4; ++e) a[i0 + e] = fmaf(-r[e].y, a[k + 1], a[i0 + e]);
#pragma unroll
      for (int e = 0; e < 4; ++e) a[i0 + e] = fmaf(-r[e].z, a[k + 2], a[i0 + e]);
#pragma unroll
      for (int e = 0; e < 4; ++e) a[i0 + e] = fmaf(-r[e].w, a[k + 3], a[i0 + e]);
      if (i0 == k + 4) {
#pragma unroll
        for (int r2 = 0; r2 < 4; ++r2)
#pragma unroll
          for (int c = r2; c < 4; ++c) p[r2][c] = __shfl_sync(0xffffffffu, a[i0 + r2], i0 + c);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kSub; ++i)
    if (i <= lane) d[i * kLeafLd + lane] = a[i];
  return bad;
}

// the rows of the panel right of its diagonal block, a column per lane, step by step behind the warp that factors
__device__ __forceinline__ void follow_panel(float* col, const Panel& P, bool on) {
  if (!on) {
    for (int step = 0; step < kSub / 4; ++step) part_sync<128>(kPanelStep + step);
    return;
  }
  float a[kSub];
#pragma unroll
  for (int i = 0; i < kSub; ++i) a[i] = col[i * kLeafLd];
#pragma unroll
  for (int k = 0; k < kSub; k += 4) {
    part_sync<128>(kPanelStep + (k >> 2));
    const float4* row = P.row[k >> 2];
    const float4 inv4 = P.inv[k >> 2];
    const float inv[4] = {inv4.x, inv4.y, inv4.z, inv4.w};
    float4 m[4];
#pragma unroll
    for (int e = 1; e < 4; ++e) m[e] = row[k + e];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      a[k + r] *= inv[r];
#pragma unroll
      for (int i = r + 1; i < 4; ++i) a[k + i] = fmaf(-(r == 0 ? m[i].x : r == 1 ? m[i].y : m[i].z), a[k + r], a[k + i]);
    }
#pragma unroll
    for (int i0 = k + 4; i0 < kSub; i0 += 4) {
      float4 r[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) r[e] = row[i0 + e];
#pragma unroll
      for (int e = 0; e < 4; ++e) a[i0 + e] = fmaf(-r[e].x, a[k], a[i0 + e]);
#pragma unroll
      for (int e = 0; e < 4; ++e) a[i0 + e] = fmaf(-r[e].y, a[k + 1], a[i0 + e]);
#pragma unroll
      for (int e = 0; e < 4; ++e) a[i0 + e] = fmaf(-r[e].z, a[k + 2], a[i0 + e]);
#pragma unroll
      for (int e = 0; e < 4; ++e) a[i0 + e] = fmaf(-r[e].w, a[k + 3], a[i0 + e]);
    }
  }
#pragma unroll
  for (int i = 0; i < kSub; ++i)
    col[i * kLeafLd] = a[i];
}

// xd <- d^-1 for an upper-triangular 32 x 32 block by one warp: right-looking back substitution, four rows at a time; zeros below the diagonal.
__device__ __forceinline__ void invert_diagonal(const float* d, float* xd) {
  const int lane = threadIdx.x & 31;
  float x[kSub];
#pragma unroll
  for (int i = 0; i < kSub; ++i) x[i] = 0.f;
#pragma unroll
  for (int q = kSub - 4; q >= 0; q -= 4) {
    float4 r4[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) r4[e] = *(const float4*)(d + (q + e) * kLeafLd + q);
#pragma unroll
    for (int i = q + 3; i >= q; --i) {
      const float v[4] = {r4[i - q].x, r4[i - q].y, r4[i - q].z, r4[i - q].w};
#pragma unroll
      for (int c = 3; c > 0; --c)
        if (q + c > i) x[i] = fmaf(v[c], x[q + c], x[i]);
      const float piv = v[i - q], own = 1.0f / piv, other = -x[i] / piv;
      x[i] = i == lane ? own : (i < lane ? other : 0.f);
    }
#pragma unroll
    for (int i0 = q - 4; i0 >= 0; i0 -= 4) {
#pragma unroll
      for (int e = 0; e < 4; ++e) r4[e] = *(const float4*)(d + (i0 + e) * kLeafLd + q);
#pragma unroll
      for (int e = 0; e < 4; ++e) x[i0 + e] = fmaf(r4[e].w, x[q + 3], x[i0 + e]);
#pragma unroll
      for (int e = 0; e < 4; ++e) x[i0 + e] = fmaf(r4[e].z, x[q + 2], x[i0 + e]);
#pragma unroll
      for (int e = 0; e < 4; ++e) x[i0 + e] = fmaf(r4[e].y, x[q + 1], x[i0 + e]);
#pragma unroll
      for (int e = 0; e < 4; ++e) x[i0 + e] = fmaf(r4[e].x, x[q], x[i0 + e]);
    }
  }
#pragma unroll
  for (int i = 0; i < kSub; ++i) xd[i * kLeafLd + lane] = x[i];
}

// s += a b for a lane's 2 x 2 values of a product of 32 x 32 blocks: `a` at its first row, `b` at its first column.
__device__ __forceinline__ void tile_times(float (&s)[2][2], const float* a, const float* b) {
#pragma unroll
  for (int k = 0; k < kSub; k += 8) {
    float4 m[2][2];
    float2 v[8];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      m[0][e] = *(const float4*)(a + k + 4 * e);
      m[1][e] = *(const float4*)(a + kLeafLd + k + 4 * e);
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = *(const float2*)(b + (k + e) * kLeafLd);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float4 p4 = m[0][e >> 2], q4 = m[1][e >> 2];
      const float p = (e & 3) == 0 ? p4.x : (e & 3) == 1 ? p4.y : (e & 3) == 2 ? p4.z : p4.w;
      const float q = (e & 3) == 0 ? q4.x : (e & 3) == 1 ? q4.y : (e & 3) == 2 ? q4.z : q4.w;
      s[0][0] = fmaf(p, v[e].x, s[0][0]); s[0][1] = fmaf(p, v[e].y, s[0][1]);
      s[1][0] = fmaf(q, v[e].x, s[1][0]); s[1][1] = fmaf(q, v[e].y, s[1][1]);
    }
  }
}
// Column J of the inverse above its diagonal block, by eight warps that meet at barrier `kBar`.
template <int kBar>
__device__ __forceinline__ void invert_column(const float* t, float* x, int J, int warp) {
  const int lane = threadIdx.x & 31, r0 = (warp >> 1) * 8 + (lane >> 3) * 2, c0 = (warp & 1) * 16 + (lane & 7) * 2;
#pragma unroll 1
  for (int I = J - 1; I >= 0; --I) {
    float s[2][2] = {};
#pragma unroll 1
    for (int K = I + 1; K <= J; ++K) tile_times(s, t + (kSub * I + r0) * kLeafLd + kSub * K, x + kSub * K * kLeafLd + kSub * J + c0);
    float* park = x + kSub * J * kLeafLd + kSub * I;
    *(float2*)(park + r0 * kLeafLd + c0) = make_float2(s[0][0], s[0][1]);
    *(float2*)(park + (r0 + 1) * kLeafLd + c0) = make_float2(s[1][0], s[1][1]);
    s[0][0] = s[0][1] = s[1][0] = s[1][1] = 0.f;
    part_sync<256>(kBar);
    tile_times(s, x + (kSub * I + r0) * kLeafLd + kSub * I, park + c0);
    float* to = x + (kSub * I + r0) * kLeafLd + kSub * J + c0;
    *(float2*)to = make_float2(-s[0][0], -s[0][1]);
    *(float2*)(to + kLeafLd) = make_float2(-s[1][0], -s[1][1]);
    part_sync<256>(kBar);
  }
}


// x <- t^-1 for the upper-triangular block t; the part of x below the diagonal blocks is scratch.
__device__ __forceinline__ void invert_upper(const float* t, float* x, int warp) {
  if (warp < kSubs) invert_diagonal(t + warp * kSub * (kLeafLd + 1), x + warp * kSub * (kLeafLd + 1));
  __syncthreads();
  if (warp < 8) {
    invert_column<kLowWarps>(t, x, 3, warp);
  } else {
    invert_column<kHighWarps>(t, x, 1, warp - 8);
    invert_column<kHighWarps>(t, x, 2, warp - 8);
  }
  __syncthreads();
}

__device__ __forceinline__ void store_upper(const float* x, float* out) {
#pragma unroll
  for (int e = 0; e < kLoads; ++e) {
    const int idx = threadIdx.x + e * kLeafThreads, i = idx >> 5, j = (idx & 31) * 4;
    const float4 v = *(const float4*)(x + i * kLeafLd + j);
    *(float4*)(out + i * kTriBlock + j) = make_float4(j >= i ? v.x : 0.f, j + 1 >= i ? v.y : 0.f, j + 2 >= i ? v.z : 0.f, j + 3 >= i ? v.w : 0.f);
  }
}

__global__ void __launch_bounds__(kLeafThreads) tri_inv_blocks_kernel(const float* __restrict__ Q, long long ld, long long strideQ,
                                                                     int n, float* __restrict__ X) {
  extern __shared__ __align__(16) float leaf_smem[];
  float *t = leaf_smem, *x = leaf_smem + kTriBlock * kLeafLd;
  const int blk = blockIdx.x, b = blockIdx.y, r0 = blk * kTriBlock;
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);
  load_upper(Q + (long long)b * strideQ + (long long)r0 * ld + r0, ld, min(kTriBlock, n - r0), t);
  __syncthreads();
  invert_upper(t, x, warp);
  store_upper(x, X + ((long long)b * gridDim.x + blk) * kTriBlock * kTriBlock);
}

__global__ void __launch_bounds__(kLeafThreads) chol_inv_leaf_kernel(const float* __restrict__ G, long long ldg, long long strideG,
                                                                     float* __restrict__ R, long long ldr, long long strideR,
                                                                     float* __restrict__ X, long long strideX, int size,
                                                                     int* __restrict__ info) {
  extern __shared__ __align__(16) float leaf_smem[];
  float *t = leaf_smem, *x = leaf_smem + kTriBlock * kLeafLd;
  __shared__ __align__(16) Panel P;
  __shared__ int failed;
  const int b = blockIdx.x, tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = tid & 31;
  if (tid == 0) failed = 0;
  griddep_wait();
  griddep_launch();
  load_upper(G + (long long)b * strideG, ldg, size, t);
  __syncthreads();
  const int panels = (size + kSub - 1) / kSub;
#pragma unroll 1
  for (int J = 0; J < kSubs; ++J) {
    float* d = t + J * kSub * (kLeafLd + 1);
    float* xd = x + J * kSub * (kLeafLd + 1);
    const int nb = kSubs - 1 - J;  // blocks right of the diagonal
    // warp 0: the diagonal block; 1 .. 3: the columns right of it; 8 .. 15: column J - 1 of the inverse
    if (warp == 0) {
      if (J < panels) {
        const bool bad = factor_diagonal(d, P);
        if (lane == 0 && bad) failed = 1;
      }
    } else if (warp < 4) {
      if (J < panels) follow_panel(d + (warp <= nb ? warp * kSub : 0) + lane, P, warp <= nb);
    } else if (warp >= 8 && J > 0) {
      if (warp == 8) invert_diagonal(d - kSub * (kLeafLd + 1), xd - kSub * (kLeafLd + 1));
      part_sync<256>(kLowWarps);
      invert_column<kLowWarps>(t, x, J - 1, warp - 8);
    }
    __syncthreads();
    // trailing blocks (I, K), I <= K, sixteen rows of a block per warp; a lane has 4 x 4 values
    if (J < panels && warp < nb * (nb + 1)) {
      const int I = warp < 2 * nb ? 0 : warp < 4 * nb - 2 ? 1 : 2, K = (warp >> 1) - (I == 0 ? 0 : I == 1 ? nb - 1 : 2 * nb - 3);
      const int i0 = kSub * I + (warp & 1) * 16 + (lane >> 3) * 4, j0 = kSub * K + (lane & 7) * 4;
      const float* panel = d + kSub;
      float* trail = d + kSub * (kLeafLd + 1);
      float v[4][4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float4 q = *(const float4*)(trail + (i0 + r) * kLeafLd + j0);
        v[r][0] = q.x; v[r][1] = q.y; v[r][2] = q.z; v[r][3] = q.w;
      }
#pragma unroll 4
      for (int k = 0; k < kSub; k += 4) {
        float4 m[4], c[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          m[e] = *(const float4*)(panel + (k + e) * kLeafLd + i0);
          c[e] = *(const float4*)(panel + (k + e) * kLeafLd + j0);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float mv[4] = {m[e].x, m[e].y, m[e].z, m[e].w}, cv[4] = {c[e].x, c[e].y, c[e].z, c[e].w};
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) v[i][j] = fmaf(-mv[i], cv[j], v[i][j]);
        }
      }
      // (left of the diagonal: nobody reads it)
#pragma unroll
      for (int r = 0; r < 4; ++r) *(float4*)(trail + (i0 + r) * kLeafLd + j0) = make_float4(v[r][0], v[r][1], v[r][2], v[r][3]);
    }
    __syncthreads();
  }
  if (warp == 0) invert_diagonal(t + (kSubs - 1) * kSub * (kLeafLd + 1), x + (kSubs - 1) * kSub * (kLeafLd + 1));
  __syncthreads();
  if (warp < 8) invert_column<kLowWarps>(t, x, kSubs - 1, warp);
  __syncthreads();
  store_upper(x, X + (long long)b * strideX);
  if (R != nullptr) {
    float* r = R + (long long)b * strideR;
    for (int idx = tid; idx < kTriBlock * kTriBlock; idx += kLeafThreads) {
      const int i = idx >> 7, j = idx & (kTriBlock - 1);
      if (i < size && j < size) r[(long long)i * ldr + j] = j >= i ? t[i * kLeafLd + j] : 0.f;
    }
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

// Four rows and a column of 16-byte stores per step (8 of 1024^2: 9 us, with one row per block and 4-byte stores 14).
__global__ void __launch_bounds__(256) triu_unpack_wide_kernel(const uint32_t* __restrict__ line, uint32_t* __restrict__ dense, int n) {
  const long long b = blockIdx.y, len = (long long)n * (n + 1) / 2;
  const int i0 = blockIdx.x * 4;  // n is a multiple of 4
  for (int j = threadIdx.x * 4; j < n; j += blockDim.x * 4) {
    uint32_t v[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const long long i = i0 + r;
      const uint32_t* src = line + b * len + i * n - i * (i - 1) / 2 - i + j;
#pragma unroll
      for (int e = 0; e < 4; ++e) v[r][e] = j + e >= i ? src[e] : 0u;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) *(uint4*)(dense + (b * n + i0 + r) * n + j) = make_uint4(v[r][0], v[r][1], v[r][2], v[r][3]);
  }
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
  if (elem_bytes == 4 && (n & 3) == 0 && ((uintptr_t)dense & 15) == 0)
    triu_unpack_wide_kernel<<<dim3(n / 4, batch), 256, 0, stream>>>((const uint32_t*)line, (uint32_t*)dense, n);
  else if (elem_bytes == 4) triu_unpack_kernel<uint32_t><<<grid, 256, 0, stream>>>((const uint32_t*)line, (uint32_t*)dense, n);
  else if (elem_bytes == 2) triu_unpack_kernel<uint16_t><<<grid, 256, 0, stream>>>((const uint16_t*)line, (uint16_t*)dense, n);
  else return cudaErrorInvalidValue;
  return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------ around the eigenbasis refresh
// Passes over n x k matrices that only memory bounds: a block turns a few rows in shared memory, so that both sides are read and written
// in whole lines (16 of 1024^2, the library's gather and scatter, element by element through 64-bit indices, 54 and 78 us).  16 bytes per access
// where rows start on such boundaries and are long enough to give the threads of a block a vector each, us there and back with 16 / 4 bytes:
// 3000 of 16^2 14, 11 / 8, 9; 64 of 256^2 7.6, 7.8 / 6.5, 7.3; 64 of 512^2 30, 27 / 28, 31; 16 of 768^2 12, 13 / 13, 15; 16 of 1024^2 28, 26 / 32, 39;
// 11 of 2048^2 94, 85 / 206, 202.  A thread's eight loads are of eight rows (through a flat index 16 of 1024^2 33 in the place of 28).
template <typename V>  // float4 or float
__global__ void __launch_bounds__(256) permute_columns_kernel(const float* __restrict__ x, const long long* __restrict__ order, float* __restrict__ out,
                                                             int n, int k, int rows, int inverse) {
  constexpr int kWide = sizeof(V) / sizeof(float);
  extern __shared__ __align__(16) float turned[];  // rows x k
  const int r0 = blockIdx.x * rows, count = min(rows, n - r0), vectors = k / kWide;
  const long long base = ((long long)blockIdx.y * n + r0) * k;
  const long long* o = order + (long long)blockIdx.y * k;
  const V* from = (const V*)(x + base);
  V* to = (V*)(out + base);
  if (!inverse) {
    for (int j = threadIdx.x; j < vectors; j += blockDim.x) {
#pragma unroll 8
      for (int r = 0; r < count; ++r) ((V*)turned)[r * vectors + j] = from[r * vectors + j];
    }
    __syncthreads();
  }
  for (int j = threadIdx.x; j < vectors; j += blockDim.x) {
    int at[kWide];
#pragma unroll
    for (int e = 0; e < kWide; ++e) {
      const long long v = o[j * kWide + e];
      at[e] = v < 0 || v >= k ? -1 : (int)v;
    }
    if (inverse) {
#pragma unroll 8
      for (int r = 0; r < count; ++r) {
        const V v = from[r * vectors + j];
#pragma unroll
        for (int e = 0; e < kWide; ++e)
          if (at[e] >= 0) turned[r * k + at[e]] = ((const float*)&v)[e];
      }
    } else {
#pragma unroll 8
      for (int r = 0; r < count; ++r) {
        V v;
#pragma unroll
        for (int e = 0; e < kWide; ++e) ((float*)&v)[e] = at[e] >= 0 ? turned[r * k + at[e]] : 0.0f;
        to[r * vectors + j] = v;
      }
    }
  }
  if (inverse) {
    __syncthreads();
#pragma unroll 4
    for (int i = threadIdx.x; i < count * vectors; i += blockDim.x) to[i] = ((const V*)turned)[i];
  }
}

cudaError_t launch_permute_columns(const float* x, const long long* order, float* out, int batch, int n, int k, int inverse, cudaStream_t stream) {
  if (batch == 0 || n == 0 || k == 0) return cudaSuccess;
  if (k > kMaxPermuted || batch > 65535) return cudaErrorInvalidValue;
  const int rows = kMaxPermuted / k < 8 ? kMaxPermuted / k : 8;  // 48 KB of shared memory at most
  const bool vec = k >= 768 && (k & 3) == 0 && (((uintptr_t)x | (uintptr_t)out) & 15) == 0;
  const auto kernel = vec ? permute_columns_kernel<float4> : permute_columns_kernel<float>;
  kernel<<<dim3((n + rows - 1) / rows, batch), 256, (size_t)rows * k * sizeof(float), stream>>>(x, order, out, n, k, rows, inverse);
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
