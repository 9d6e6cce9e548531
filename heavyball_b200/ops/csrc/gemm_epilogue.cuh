// Epilogue and kernels (128 x 128 tiles, and 256 x 256 on CTA pairs) shared by the split-operand GEMMs (tf32_gemm.cu, split16_gemm.cu).
//
// 128 x 128 tiles, one per CTA, 192 threads, two CTAs per SM (a ring of six stages and one CTA per SM is no faster, not even for launches
// of a few tiles: a tile by itself takes 0.43 us per 128 bytes of K because its products and its loads share the shared memory):
//   warp 0     : TMA producer, cp.async.bulk.tensor 3-D loads (128-byte swizzle, 128 bytes of K per row) into a 3-stage ring
//   warp 1     : tcgen05.mma.cta_group::1, 128 x 128 x 32 bytes of K per instruction, accumulator in 128 TMEM columns
//   warps 2..5 : tcgen05.ld, then the epilogue.  Plain stores go through the (now idle) ring and four bulk tensor stores, the
//                others through epilogue_direct.
#pragma once
#include "pair_drain.h"
#include "tc_common.cuh"
#include "tf32_gemm.h"

namespace hb {
namespace {

constexpr int TBM = 128, TBN = 128;
constexpr int kTStages = 3;
constexpr int kTTileBytes = TBM * 128;               // 16 KiB per operand tile
constexpr int kTStageBytes = 2 * kTTileBytes;
constexpr int kTSmemBytes = kTStages * kTStageBytes + 1024;
constexpr int kTThreads = 192;
constexpr uint32_t kTTmemCols = 128;

__device__ __forceinline__ float tf32_hi(float x) {
  uint32_t bits;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(bits) : "f"(x));
  return __uint_as_float(bits);
}

__device__ __forceinline__ float lerp_w(float s, float x, float w) { return s * (1.0f - w) + x * w; }

constexpr int kStageLd = 36;                         // floats per staged row: rows stay 16-byte aligned and float4
                                                     // accesses of a quarter-warp fall into distinct banks
constexpr int kStageWarpBytes = 32 * kStageLd * 4;   // one warp's 32 rows x 32 columns

// What the epilogue knows of an operand of scaled fp16 pairs (split16_gemm.h): what one unit of each of its rows stands for with the number of
// values that the row's pairs hold in fewer bits than split tf32 would, and the matrix that it was made from: element (row, k) of batch
// entry b is src[b * src_batch + row * src_row + k * src_k].
struct PairOperand {
  const float* unit;
  int64_t unit_batch;
  const float* src;
  int64_t src_batch, src_row, src_k;
};
struct PairOperands {
  PairOperand a, b;
  int K;
};

// kRows (32 or 16) rows of an operand's matrix, 16 of K at a time (zeros outside it), fetched in the order in which they lie in memory - four
// neighbours at once where they are aligned - and put down as rows of the stage.
template <int kRows>
struct SourceWalk {
  static constexpr int kPieces = kRows / 8;        // a lane's, of four values
  static constexpr int kAcross = kRows / 4;        // not along_k: lanes side by side along the rows
  static constexpr int kStep = 32 / kAcross;       // ... whose pieces are that many of K apart
  const float* p;              // of this lane's first value
  int64_t one, piece, advance;  // to the next value of a piece, to the next piece, to the next 16 of K
  int rows, left;              // rows and values of K from the first value on
  int at;                      // where it goes
  bool along_k, wide;
  __device__ __forceinline__ SourceWalk(const PairOperand& op, int lane, int batch, int row0, int n_rows, int K) {
    along_k = op.src_k == 1;
    const int r = along_k ? lane >> 2 : lane % kAcross * 4, k = along_k ? (lane & 3) * 4 : lane / kAcross;
    p = op.src + batch * op.src_batch + (row0 + r) * op.src_row + k * op.src_k;
    one = along_k ? 1 : op.src_row;
    piece = along_k ? 8 * op.src_row : kStep * op.src_k;
    advance = 16 * op.src_k;
    rows = n_rows - row0 - r;
    left = K - k;
    at = r * kStageLd + k;
    const int64_t between = along_k ? op.src_row : op.src_k;
    wide = one == 1 && (between & 3) == 0 && (op.src_batch & 3) == 0 && ((uintptr_t)op.src & 15) == 0;
  }
  __device__ __forceinline__ void fetch(float4 (&v)[kPieces]) {
    const bool inside = along_k ? rows > 8 * (kPieces - 1) && left >= 4 : rows >= 4 && left > kStep * (kPieces - 1);
    if (__all_sync(0xFFFFFFFFu, wide && inside)) {
#pragma unroll
      for (int i = 0; i < kPieces; ++i) v[i] = *(const float4*)(p + i * piece);
    } else {
#pragma unroll
      for (int i = 0; i < kPieces; ++i) {
        const int n = along_k ? (rows > 8 * i ? left : 0) : (left > kStep * i ? rows : 0);  // values of the piece that are inside
        const float* q = p + i * piece;
        v[i] = make_float4(n > 0 ? q[0] : 0.0f, n > 1 ? q[one] : 0.0f, n > 2 ? q[2 * one] : 0.0f, n > 3 ? q[3 * one] : 0.0f);
      }
    }
    p += advance;
    left -= 16;
  }
  __device__ __forceinline__ void put(float* stage, const float4 (&v)[kPieces]) const {
    float* s = stage + at;
    if (along_k) {
#pragma unroll
      for (int i = 0; i < kPieces; ++i) *(float4*)(s + 8 * i * kStageLd) = v[i];
    } else {
#pragma unroll
      for (int i = 0; i < kPieces; ++i, s += kStep) {
        s[0] = v[i].x;
        s[kStageLd] = v[i].y;
        s[2 * kStageLd] = v[i].z;
        s[3 * kStageLd] = v[i].w;
      }
    }
  }
};

__device__ __forceinline__ float pow2(int e) { return __uint_as_float((uint32_t)(127 + e) << 23); }

// A row's unit carries the number of its values below 2^-14 units in the mantissa.
__device__ __forceinline__ float unit_of(float u) { return __uint_as_float(__float_as_uint(u) & 0x7F800000u); }
__device__ __forceinline__ uint32_t short_values(float u, bool inside) { return inside ? __float_as_uint(u) & 0x7FFFFFu : 0u; }

constexpr uint32_t kManyShort = 1u << 19;  // counts of short values from here on stand for "any number"

// Accumulators of a block (32 x 32, in tensor memory) with values short of bits or with units whose product may leave the range of fp32 <-
// entries of the product.
// A value below 2^-14 in units of its row is held with an error of up to 2^-36 of a unit instead of 22 bits of itself.  With the other
// operand's values (2^15 at most) and the product of low parts that is left out, n of them bring an error of at most n 2^-20: where the
// accumulator is 4 n or more, less than 2^-22 of the result.  Smaller accumulators of such rows and columns may consist of nothing else:
// the block is computed from the matrices themselves, in fp32 arithmetic (subnormals kept), sums of 16 at a time, the next 16 of K on their
// way meanwhile.  (One such value among ordinary ones, as in one of a hundred thousand rows of 1024 normally distributed values, does not
// lead there: sums over ordinary values are around 2^25 and more.)
// Measured, a warp by itself: 1.3 us per 16 of K, most of it the latency of the loads (a second step of prefetch, in registers or by cp.async, was
// slower: spills, and more instructions than it hides).  A product half of which comes this way takes sixteen times its tf32 time (4 of 2048^3
// 4.3 ms, 8 of 128^3 43 us instead of 14); steps on 4 of 2048 x 1024 with half of the gradient's rows 1e-14 of the others, against split tf32:
// PSGD with a fit 6.6 / 3.7 ms, SOAP without refresh 5.1 / 1.2 (ordinary gradients 2.8 / 3.6 and 0.9 / 1.1).
// `tri`: entries below the diagonal are zeros whatever the values.
__device__ __noinline__ void settle_slowly(uint32_t tmem, int lane, float* stage, const PairOperands& P, int batch, int row0, int col0, int M, int N,
                                           int tri) {
  const float row = P.a.unit[batch * P.a.unit_batch + row0 + lane], col = P.b.unit[batch * P.b.unit_batch + col0 + lane];
  uint32_t acc[32];
  tmem_ld32(tmem, acc);
  tmem_ld_wait();
  const uint32_t n_row = short_values(row, row0 + lane < M), n_col = short_values(col, col0 + lane < N);
  const float by_row = 4.0f * (n_row >= kManyShort ? (float)P.K : (float)n_row), by_col = 4.0f * (n_col >= kManyShort ? (float)P.K : (float)n_col);
  bool small = false;
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    const float least = by_row + __shfl_sync(0xFFFFFFFFu, by_col, j);
    small |= row0 + lane < M && col0 + j < N && !(tri && row0 + lane > col0 + j) && fabsf(__uint_as_float(acc[j])) < least;
  }
  if (!__any_sync(0xFFFFFFFFu, small)) {  // units in two steps of half the exponent each: neither leaves the range unless the result does
    const int e_row = (int)(__float_as_uint(unit_of(row)) >> 23) - 127, e_mine = (int)(__float_as_uint(unit_of(col)) >> 23) - 127;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const int e = max(-252, min(252, e_row + __shfl_sync(0xFFFFFFFFu, e_mine, j))), half = e >> 1;  // (padding holds anything)
      acc[j] = __float_as_uint(__uint_as_float(acc[j]) * pow2(half) * pow2(e - half));
    }
    tmem_st32(tmem, acc);
    return;
  }
  // Half of the columns at a time: with all 32 the registers do not suffice, and what is spilled comes back from the L2 (shared memory leaves
  // the L1 next to nothing).  A lane has rows y + 8 i and columns x + 4 j, even and odd k in the halves of one register pair: eight loads from the
  // stage for 64 products in 32 instructions, no two of a quarter warp in one bank.
  const int x = lane & 3, y = lane >> 2;
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {
    float out[4][4];
    float4 next_a[4], next_b[2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) out[i][j] = 0.0f;
    SourceWalk<32> walk_a(P.a, lane, batch, row0, M, P.K);
    SourceWalk<16> walk_b(P.b, lane, batch, col0 + 16 * half, N, P.K);
    walk_a.fetch(next_a);
    walk_b.fetch(next_b);
#pragma unroll 1
    for (int left = P.K; left > 0; left -= 16) {
      __syncwarp();
      walk_a.put(stage, next_a);       // columns 0 .. 15 of the stage
      walk_b.put(stage + 16, next_b);  // columns 16 .. 31 of its first 16 rows
      __syncwarp();
      if (left > 16) {
        walk_a.fetch(next_a);
        walk_b.fetch(next_b);
      }
      unsigned long long sum[4][4];  // two floats each
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) sum[i][j] = 0ull;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        ulonglong2 a[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = *(const ulonglong2*)(stage + (y + 8 * i) * kStageLd + q * 4);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const ulonglong2 b = *(const ulonglong2*)(stage + (x + 4 * j) * kStageLd + 16 + q * 4);
#pragma unroll
          for (int i = 0; i < 4; ++i) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(sum[i][j]) : "l"(a[i].x), "l"(b.x));
#pragma unroll
          for (int i = 0; i < 4; ++i) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(sum[i][j]) : "l"(a[i].y), "l"(b.y));
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float both = __uint_as_float((uint32_t)sum[i][j]);
          asm("add.rn.f32 %0, %0, %1;" : "+f"(both) : "f"(__uint_as_float((uint32_t)(sum[i][j] >> 32))));
          asm("add.rn.f32 %0, %0, %1;" : "+f"(out[i][j]) : "f"(both));
        }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) stage[(y + 8 * i) * kStageLd + x + 4 * j] = out[i][j];
    __syncwarp();
    uint32_t settled[16];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float4 t = *(const float4*)(stage + lane * kStageLd + q * 4);
      settled[q * 4] = __float_as_uint(t.x); settled[q * 4 + 1] = __float_as_uint(t.y);
      settled[q * 4 + 2] = __float_as_uint(t.z); settled[q * 4 + 3] = __float_as_uint(t.w);
    }
    tmem_st16(tmem + 16u * (uint32_t)half, settled);
  }
  __syncwarp();
}

// Units of a warp's 32 rows (lane = row) and four blocks of 32 columns (lane = column), fetched while the products are under way; `slow`: the blocks
// that are not ordinary - some value short of bits, or a unit far from one - and are settled in tensor memory before the epilogue proper, which
// thereby keeps its registers.
struct BlockUnits {
  float row, col[4];
  uint32_t slow;
};
__device__ __forceinline__ bool ordinary_unit(float u, bool inside) { return !inside || (short_values(u, true) == 0 && u > 0x1p-63f && u < 0x1p63f); }
__device__ __forceinline__ BlockUnits fetch_units(const PairOperands& P, int lane, int batch, int row0, int col0, int M, int N) {
  BlockUnits u;
  u.row = P.a.unit[batch * P.a.unit_batch + row0 + lane];
#pragma unroll
  for (int cb = 0; cb < 4; ++cb) u.col[cb] = P.b.unit[batch * P.b.unit_batch + col0 + cb * 32 + lane];
  u.slow = 0;
#pragma unroll
  for (int cb = 0; cb < 4; ++cb)
    if (!__all_sync(0xFFFFFFFFu, ordinary_unit(u.row, row0 + lane < M) && ordinary_unit(u.col[cb], col0 + cb * 32 + lane < N))) u.slow |= 1u << cb;
  return u;
}
__device__ __forceinline__ void settle_blocks(const BlockUnits& u, uint32_t tmem, int lane, float* stage, const PairOperands& P, int batch, int row0,
                                              int col0, int M, int N, int tri) {
#pragma unroll 1
  for (uint32_t left = u.slow; left != 0; left &= left - 1) {
    const int cb = __ffs((int)left) - 1;
    settle_slowly(tmem + (uint32_t)(cb * 32), lane, stage, P, batch, row0, col0 + cb * 32, M, N, tri);
  }
}
__device__ __forceinline__ float row_unit_of(const BlockUnits& u, int cb) { return u.slow >> cb & 1 ? 1.0f : u.row; }
__device__ __forceinline__ float col_unit_of(const BlockUnits& u, int cb) {
  return u.slow >> cb & 1 ? 1.0f : cb < 2 ? (cb == 0 ? u.col[0] : u.col[1]) : (cb == 2 ? u.col[2] : u.col[3]);
}

// Accumulators of an ordinary 32 x 32 block (lane = row) -> entries of the product.
__device__ __forceinline__ void unscale32(uint32_t (&acc)[32], float row_unit, float col_unit) {
#pragma unroll
  for (int j = 0; j < 32; ++j) acc[j] = __float_as_uint(__uint_as_float(acc[j]) * (row_unit * __shfl_sync(0xFFFFFFFFu, col_unit, j)));
}

// The usual case of the epilogue below: a 32 x 32 block inside the output, C aligned, no split output.  With the mode known at compile
// time, no bounds to check and all reads in flight before the first use a tile's epilogue is a third as long (8 of 128^3, whole
// launch: added to C 15.8 -> 9.3 us, symmetric 13.1 -> 7.8, Adam 21.1 -> 12.6, stored in bulk 7.2).
// `c`, `cm`, `m`, `v`: the block's first element in the output, in its mirror image (null: not stored) and in the moments.
template <bool kScaled, int kMode>
__device__ __forceinline__ void epilogue_block(uint32_t tmem, int lane, float* stage, const Tf32Epilogue& E, float* c, float* cm, float* m,
                                               float* v, int64_t ld_state, float row_unit, float col_unit) {
  constexpr bool kOld = kMode == kEpiLerp || kMode == kEpiAdd, kMoments = kMode == kEpiAdam || kMode == kEpiLaProp;
  const int sub = lane >> 3, cg = (lane & 7) * 4;
  float* const mine = stage + lane * kStageLd;
  float* const turned = stage + sub * kStageLd + cg;
  float* const crow = c + (int64_t)sub * E.ldc + cg;
  const int64_t cstep = 4 * E.ldc, sstep = 4 * ld_state;
  float4 pa[8], pb[8];
  if constexpr (kOld) {  // what is read from memory is on its way before the first value is needed
#pragma unroll
    for (int i = 0; i < 8; ++i) pa[i] = *(const float4*)(crow + i * cstep);
  }
  if constexpr (kMoments) {
    m += sub * ld_state + cg;
    v += sub * ld_state + cg;
#pragma unroll
    for (int i = 0; i < 8; ++i) {  // (with four at a time, which spills nothing: 16 of 1024^3 with Adam 169 instead of 140 us)
      pa[i] = *(const float4*)(m + i * sstep);
      pb[i] = *(const float4*)(v + i * sstep);
    }
  }
  {
    uint32_t acc[32];
    tmem_ld32(tmem, acc);
    tmem_ld_wait();
    if constexpr (kScaled) unscale32(acc, row_unit, col_unit);
#pragma unroll
    for (int q = 0; q < 8; ++q)
      *(float4*)(mine + q * 4) =
          make_float4(__uint_as_float(acc[q * 4]) * E.alpha, __uint_as_float(acc[q * 4 + 1]) * E.alpha,
                      __uint_as_float(acc[q * 4 + 2]) * E.alpha, __uint_as_float(acc[q * 4 + 3]) * E.alpha);
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float4 x4 = *(const float4*)(turned + i * 4 * kStageLd);
    float x[4] = {x4.x, x4.y, x4.z, x4.w};
    if constexpr (kOld) {
      const float o[4] = {pa[i].x, pa[i].y, pa[i].z, pa[i].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) x[e] = kMode == kEpiLerp ? o[e] + (x[e] - o[e]) * E.w : o[e] + x[e];
      if (cm != nullptr) *(float4*)(turned + i * 4 * kStageLd) = make_float4(x[0], x[1], x[2], x[3]);
    }
    if constexpr (kMoments) {
      float m4[4] = {pa[i].x, pa[i].y, pa[i].z, pa[i].w}, s4[4] = {pb[i].x, pb[i].y, pb[i].z, pb[i].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        s4[e] = lerp_w(s4[e], x[e] * x[e], 1.0f - E.b2);
        const float d = fmaxf(sqrtf(s4[e]), E.eps);
        m4[e] = lerp_w(m4[e], kMode == kEpiAdam ? x[e] : x[e] / d, 1.0f - E.b1);
        x[e] = kMode == kEpiAdam ? m4[e] / d : m4[e];
      }
      *(float4*)(m + i * sstep) = make_float4(m4[0], m4[1], m4[2], m4[3]);
      *(float4*)(v + i * sstep) = make_float4(s4[0], s4[1], s4[2], s4[3]);
    }
    *(float4*)(crow + i * cstep) = make_float4(x[0], x[1], x[2], x[3]);
  }
  if constexpr (!kMoments) {
    if (cm != nullptr) {  // consecutive lanes hold consecutive rows: a column of the block is one line of the mirror image
      __syncwarp();
      float* out = cm + lane;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float4 t = *(const float4*)(mine + q * 4);
        out[0] = t.x;
        out[E.ldc] = t.y;
        out[2 * E.ldc] = t.z;
        out[3 * E.ldc] = t.w;
        out += 4 * E.ldc;
      }
    }
  }
  __syncwarp();  // the stage is rewritten by the next block
}

// Fused epilogue of one warp: its 32 accumulator rows of the 128x128 tile, 32 columns at a time.  A thread reads
// its own row from tensor memory; global memory wants the other orientation (consecutive lanes on consecutive
// columns), so the block is turned through the warp's `stage` in shared memory (the idle operand ring):
//   pass 1 (lane = row):                   accumulators * alpha -> stage
//   pass 2 (8 lanes per row, 4 rows/step): moments, lerp, C store, split-operand store - every global access is a full
//                                          128-byte line per row; the final values go back to the stage when needed
//   pass 3 (lane = row):                   outputs that run along the rows: transposed split operand, mirror tile
// Values outside [M, N] are never stored; the zero padding of a split output (columns [K, kp) of the operand being
// produced) is.
// `tmem_warp`: tensor-memory address of the warp's first row and the tile's first column; `row0` / `col_base`: their
// global indices; `n_cb`: 32-column blocks in the tile; `off_diagonal`: the tile is not on the diagonal (mirror stores).
// `zero_acc`: the tile had no product (its accumulator was never written): the values are zeros.
// `kScaled`: the operands are fp16 pairs, described by `P` and by the units `U` of the warp's blocks; their products have no split outputs.
template <bool kScaled>
__device__ __forceinline__ void epilogue_direct(uint32_t tmem_warp, int lane, float* stage, int row0, int col_base, int n_cb,
                                                bool off_diagonal, bool zero_acc, int batch, int M, int N,
                                                const Tf32Epilogue& E, const PairOperands& P, const BlockUnits& U) {
  const int64_t b64 = batch;
  const bool state_vec = (N & 3) == 0;
  const bool c_vec = (E.ldc & 3) == 0 && ((E.strideC & 3) == 0) && ((((uintptr_t)E.C) & 15) == 0);
  const bool moments = E.mode == kEpiAdam || E.mode == kEpiLaProp;
  const bool mirror = E.symmetric && off_diagonal && E.C != nullptr;
  const bool s_cols = !kScaled && E.S != nullptr && E.s_transposed, s_rows = !kScaled && E.S != nullptr && !E.s_transposed;
  const bool along_rows = mirror || s_cols;
  const int sub = lane >> 3, cg = (lane & 7) * 4;
  const float w1 = 1.0f - E.b1, w2 = 1.0f - E.b2;
  float* mine = stage + lane * kStageLd;
#pragma unroll 1
  for (int cb = 0; cb < n_cb; ++cb) {
    const int col0 = col_base + cb * 32;
    float row_unit = 1.0f, col_unit = 1.0f;
    if constexpr (kScaled) {
      row_unit = row_unit_of(U, cb);
      col_unit = col_unit_of(U, cb);
    }
    if (!zero_acc && !s_rows && !s_cols && c_vec && E.C != nullptr && row0 + 32 <= M && col0 + 32 <= N && (!moments || state_vec)) {
      const uint32_t t = tmem_warp + (uint32_t)(cb * 32);
      float* c = E.C + b64 * E.strideC + (int64_t)row0 * E.ldc + col0;
      float* cm = mirror ? E.C + b64 * E.strideC + (int64_t)col0 * E.ldc + row0 : nullptr;
      const int64_t st = (b64 * M + row0) * (int64_t)N + col0;
      switch (E.mode) {
        case kEpiStore: epilogue_block<kScaled, kEpiStore>(t, lane, stage, E, c, cm, nullptr, nullptr, 0, row_unit, col_unit); break;
        case kEpiLerp: epilogue_block<kScaled, kEpiLerp>(t, lane, stage, E, c, cm, nullptr, nullptr, 0, row_unit, col_unit); break;
        case kEpiAdd: epilogue_block<kScaled, kEpiAdd>(t, lane, stage, E, c, cm, nullptr, nullptr, 0, row_unit, col_unit); break;
        case kEpiAdam: epilogue_block<kScaled, kEpiAdam>(t, lane, stage, E, c, nullptr, E.m + st, E.v + st, N, row_unit, col_unit); break;
        default: epilogue_block<kScaled, kEpiLaProp>(t, lane, stage, E, c, nullptr, E.m + st, E.v + st, N, row_unit, col_unit); break;
      }
      continue;
    }
    {
      uint32_t acc[32];
      if (!zero_acc) {
        tmem_ld32(tmem_warp + (uint32_t)(cb * 32), acc);
        tmem_ld_wait();
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) acc[j] = 0u;
      }
      if constexpr (kScaled)
        if (!zero_acc) unscale32(acc, row_unit, col_unit);
#pragma unroll
      for (int q = 0; q < 8; ++q)
        *(float4*)(mine + q * 4) =
            make_float4(__uint_as_float(acc[q * 4]) * E.alpha, __uint_as_float(acc[q * 4 + 1]) * E.alpha,
                        __uint_as_float(acc[q * 4 + 2]) * E.alpha, __uint_as_float(acc[q * 4 + 3]) * E.alpha);
    }
    __syncwarp();

    const int col = col0 + cg;
    // What the epilogue reads from global memory (moments, or the old value of C) is fetched four steps at a time
    // before the first of them is used: a step-by-step load -> compute -> store chain pays one memory round trip per step
    // (stores may alias the next step's loads, so the compiler cannot hoist them), which for the small products of a
    // blocked solve was longer than the product itself.
    const bool fast_state = moments && state_vec && col + 3 < N;
    const bool fast_old = (E.mode == kEpiLerp || E.mode == kEpiAdd) && E.C != nullptr && c_vec && col + 3 < N;
    float4 pa[4], pb[4];
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
    if (fast_state || fast_old) {
#pragma unroll
      for (int i4 = 0; i4 < 4; ++i4) {
        const int row = row0 + (half * 4 + i4) * 4 + sub;
        pa[i4] = make_float4(0.f, 0.f, 0.f, 0.f);
        pb[i4] = pa[i4];
        if (row < M) {
          if (fast_state) {
            pa[i4] = *(const float4*)(E.m + (b64 * M + row) * (int64_t)N + col);
            pb[i4] = *(const float4*)(E.v + (b64 * M + row) * (int64_t)N + col);
          } else {
            pa[i4] = *(const float4*)(E.C + b64 * E.strideC + (int64_t)row * E.ldc + col);
          }
        }
      }
    }
#pragma unroll
    for (int i4 = 0; i4 < 4; ++i4) {
      const int it = half * 4 + i4;
      const int lr = it * 4 + sub, row = row0 + lr;
      float* sp = stage + lr * kStageLd + cg;
      const float4 x4 = *(const float4*)sp;
      float x[4] = {x4.x, x4.y, x4.z, x4.w};
      if (row < M && col < N) {
        if (moments) {
          float* mp = E.m + (b64 * M + row) * (int64_t)N + col;
          float* vp = E.v + (b64 * M + row) * (int64_t)N + col;
          const bool fast = fast_state;
          float m4[4], s4[4];
          if (fast) {
            const float4 a = pa[i4], c = pb[i4];
            m4[0] = a.x; m4[1] = a.y; m4[2] = a.z; m4[3] = a.w;
            s4[0] = c.x; s4[1] = c.y; s4[2] = c.z; s4[3] = c.w;
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              m4[e] = col + e < N ? mp[e] : 0.f;
              s4[e] = col + e < N ? vp[e] : 0.f;
            }
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            s4[e] = lerp_w(s4[e], x[e] * x[e], w2);
            const float d = fmaxf(sqrtf(s4[e]), E.eps);
            if (E.mode == kEpiAdam) {
              m4[e] = lerp_w(m4[e], x[e], w1);
              x[e] = m4[e] / d;
            } else {
              m4[e] = lerp_w(m4[e], x[e] / d, w1);
              x[e] = m4[e];
            }
          }
          if (fast) {
            *(float4*)mp = make_float4(m4[0], m4[1], m4[2], m4[3]);
            *(float4*)vp = make_float4(s4[0], s4[1], s4[2], s4[3]);
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (col + e < N) { mp[e] = m4[e]; vp[e] = s4[e]; }
          }
        }
        if (E.C != nullptr) {
          float* cp = E.C + b64 * E.strideC + (int64_t)row * E.ldc + col;
          const bool fast = c_vec && col + 3 < N;
          if (E.mode == kEpiLerp || E.mode == kEpiAdd) {
            // lerp: o + (x - o) w;  add: o + x  (the same expression with the old value left out of the difference)
            const float keep = E.mode == kEpiLerp ? 1.f : 0.f, w = E.mode == kEpiLerp ? E.w : 1.f;
            if (fast) {
              const float4 o = pa[i4];
              x[0] = o.x + (x[0] - keep * o.x) * w; x[1] = o.y + (x[1] - keep * o.y) * w;
              x[2] = o.z + (x[2] - keep * o.z) * w; x[3] = o.w + (x[3] - keep * o.w) * w;
            } else {
#pragma unroll
              for (int e = 0; e < 4; ++e)
                if (col + e < N) { const float o = cp[e]; x[e] = o + (x[e] - keep * o) * w; }
            }
          }
          if (fast) {
            *(float4*)cp = make_float4(x[0], x[1], x[2], x[3]);
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (col + e < N) cp[e] = x[e];
          }
        }
      }
      if (s_rows && row < M && col < E.kpS) {  // operand rows = output rows, K over the output columns (zero from N to kp)
        float* srow = E.S + b64 * E.strideS + (int64_t)row * (2 * E.kpS) + col;
        float hi[4], lo[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float y = col + e < N ? x[e] : 0.f;
          hi[e] = tf32_hi(y);
          lo[e] = tf32_hi(y - hi[e]);
        }
        *(float4*)srow = make_float4(hi[0], hi[1], hi[2], hi[3]);
        *(float4*)(srow + E.kpS) = make_float4(lo[0], lo[1], lo[2], lo[3]);
      }
      if (along_rows) *(float4*)sp = make_float4(x[0], x[1], x[2], x[3]);
    }
    }

    if (along_rows) {
      __syncwarp();
      const int row = row0 + lane;
      float v[32];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float4 t = *(const float4*)(mine + q * 4);
        v[q * 4] = t.x; v[q * 4 + 1] = t.y; v[q * 4 + 2] = t.z; v[q * 4 + 3] = t.w;
      }
      if (mirror && row < M) {  // consecutive lanes hold consecutive rows: one accumulator column is one contiguous line
        float* ccol = E.C + b64 * E.strideC + row;
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (col0 + j < N) ccol[(int64_t)(col0 + j) * E.ldc] = v[j];
      }
      if (s_cols && row < E.kpS) {
        // operand rows = output columns, K over the output rows (zero from M up to kp)
        float* sb = E.S + b64 * E.strideS + row;
        const int64_t ld = 2 * E.kpS;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          if (col0 + j < N) {
            const float y = row < M ? v[j] : 0.f;
            const float hi = tf32_hi(y);
            float* dst = sb + (int64_t)(col0 + j) * ld;
            dst[0] = hi;
            dst[E.kpS] = tf32_hi(y - hi);
          }
        }
      }
    }
    __syncwarp();  // the stage is rewritten by the next block of columns
  }
}

// `Kind`: operand type.  kBlock elements of K fill a 128-byte row; kDesc is the instruction descriptor for a 128 x 128 tile; the product
// is three walks over K, of which walk kTermLoA takes the low parts of A and walk kTermLoB those of B; kCrossFirst: these two come
// first, and the sum they leave is scaled by 2^-11 when the walk over the high parts begins.  kPairDesc, mma_pair: the same for the pair
// kernel.  `lo_a`, `lo_b`: how far the low parts of an operand's rows lie behind the high parts.
template <class Kind>
__global__ void __launch_bounds__(kTThreads, 2)
gemm128_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
               const __grid_constant__ CUtensorMap map_c, int M, int N, int kp, int lo_a, int lo_b, const Tf32Epilogue E,
               const __grid_constant__ PairOperands P, int bulk_store, int* status) {
  constexpr int TBK = Kind::kBlock;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[kTStages];
  __shared__ __align__(8) uint64_t empty_bar[kTStages];
  __shared__ __align__(8) uint64_t accum_bar, drain_bar;  // drain_bar: teardown only
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool leader = elect_one();  // issues the loads (warp 0) and the products (warp 1), and waits for them in the teardown
  uint8_t* tiles = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int tiles_n = (N + TBN - 1) / TBN;
  int tm = blockIdx.x / tiles_n, tn = blockIdx.x % tiles_n;
  if (E.symmetric) {  // blockIdx.x counts the tiles on or above the diagonal, row by row
    int left = blockIdx.x;
    tm = 0;
    while (left >= tiles_n - tm) { left -= tiles_n - tm; ++tm; }
    tn = tm + left;
  }
  const int batch = blockIdx.y;
  int kb_lo = 0, kb_hi = kp / TBK;  // K blocks of one term of the split product that this tile walks
  if (E.tri) {
    kb_lo = min(kb_hi, tm * (TBM / TBK));
    kb_hi = tn < tm ? kb_lo : min(kb_hi, (tn + 1) * (TBN / TBK));
  }
  const int seg_kb = kb_hi - kb_lo;
  const int num_kb = 3 * seg_kb;    // three terms of the split product
  const float alpha = E.alpha;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kTStages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(&accum_bar, 1);
    mbar_init(&drain_bar, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) { tmem_alloc(&tmem_base_slot, kTTmemCols); tmem_relinquish(); }
  griddep_wait();
  // a kernel of this stream already gave up on a wait: do not pile more work on a broken pipeline
  const bool skip = __syncthreads_or(threadIdx.x == 0 && status != nullptr && *(volatile const int*)status != 0);
  griddep_launch();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;

  int issued = 0;
  if (skip) {
  } else if (warp == 0) {
    if (leader) {
      for (int kb = 0; kb < num_kb; ++kb) {
        const int s = kb % kTStages, round = kb / kTStages;
        if (!mbar_wait(&empty_bar[s], (round & 1) ^ 1, &abort_flag)) break;
        uint8_t* dst = tiles + s * kTStageBytes;
        const int seg = kb / seg_kb, k0 = (kb_lo + kb - seg * seg_kb) * TBK;
        mbar_expect_tx(&full_bar[s], kTStageBytes);
        tma_load_3d(dst, &map_a, &full_bar[s], k0 + (seg == Kind::kTermLoA ? lo_a : 0), tm * TBM, batch);
        tma_load_3d(dst + kTTileBytes, &map_b, &full_bar[s], k0 + (seg == Kind::kTermLoB ? lo_b : 0), tn * TBN, batch);
        issued = kb + 1;
      }
    }
  } else if (warp == 1) {
    if (leader) {
      bool ok = true;
      for (int kb = 0; kb < num_kb && ok; ++kb) {
        const int s = kb % kTStages, round = kb / kTStages;
        ok = mbar_wait(&full_bar[s], round & 1, &abort_flag);
        if (!ok) break;
        tc_fence_after();
        const uint32_t a_addr = smem_u32(tiles + s * kTStageBytes);
        const uint64_t a_desc = make_smem_desc(a_addr), b_desc = make_smem_desc(a_addr + kTTileBytes);
#pragma unroll
        for (int k = 0; k < 4; ++k)  // 32 B along K inside the swizzle atom = +2 address units
          if (Kind::kCrossFirst && k == 0 && kb == 2 * seg_kb)
            tc_mma_f16_d11(tmem_base, a_desc, b_desc, Kind::kDesc);
          else
            Kind::mma(tmem_base, a_desc + 2 * k, b_desc + 2 * k, Kind::kDesc, (kb | k) ? 1u : 0u);
        tc_commit(&empty_bar[s]);
      }
      if (ok) tc_commit(&accum_bar);
    }
  } else {
    const int quarter = warp & 3, r = quarter * 32 + lane;
    BlockUnits U{};
    if constexpr (Kind::kScaled) U = fetch_units(P, lane, batch, tm * TBM + quarter * 32, tn * TBN, M, N);
    const bool have = (num_kb == 0) || mbar_wait(&accum_bar, 0, &abort_flag);
    tc_fence_after();
    if constexpr (Kind::kScaled)  // (its stage: behind what the epilogues use)
      if (have && num_kb != 0 && U.slow != 0)
        settle_blocks(U, tmem_base + ((uint32_t)(quarter * 32) << 16), lane, (float*)(tiles + (TBN / 32) * kTTileBytes + quarter * kStageWarpBytes), P,
                      batch, tm * TBM + quarter * 32, tn * TBN, M, N, E.tri);
    if (have && bulk_store) {
      // every load has landed and every MMA has retired: the ring is free and stages the output tile as four
      // [128 rows x 32 fp32] boxes in the swizzled layout the bulk store expects
#pragma unroll 1
      for (int cb = 0; cb < TBN / 32; ++cb) {
        uint32_t acc[32];
        tmem_ld32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(cb * 32), acc);
        tmem_ld_wait();
        if constexpr (Kind::kScaled) unscale32(acc, row_unit_of(U, cb), col_unit_of(U, cb));
        uint8_t* box = tiles + cb * kTTileBytes;
#pragma unroll
        for (int q = 0; q < 8; ++q)
          *(float4*)(box + swz(r, q)) =
              make_float4(__uint_as_float(acc[q * 4]) * alpha, __uint_as_float(acc[q * 4 + 1]) * alpha,
                          __uint_as_float(acc[q * 4 + 2]) * alpha, __uint_as_float(acc[q * 4 + 3]) * alpha);
      }
    } else if (have) {
      epilogue_direct<Kind::kScaled>(tmem_base + ((uint32_t)(quarter * 32) << 16), lane, (float*)(tiles + quarter * kStageWarpBytes),
                      tm * TBM + quarter * 32, tn * TBN, TBN / 32, tm != tn, num_kb == 0, batch, M, N, E, P, U);
    }
    tc_fence_before();
    if (bulk_store) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (have && warp == 2 && lane == 0) {
#pragma unroll
        for (int cb = 0; cb < TBN / 32; ++cb)
          if (tn * TBN + cb * 32 < N) tma_store_3d(&map_c, tiles + cb * kTTileBytes, tn * TBN + cb * 32, tm * TBM, batch);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      }
    }
  }

  __syncthreads();
  if (abort_flag) {  // after an expired wait: loads and products in flight end before shared and tensor memory go away
    if (warp == 0 && leader) ring_drain(full_bar, issued, kTStages);
    if (warp == 1 && leader) products_drain(&drain_bar);
    __syncthreads();
    if (threadIdx.x == 0 && status != nullptr) atomicExch(status, 1);
  }
  if (warp == 1) { __syncwarp(); tc_fence_after(); tmem_dealloc(tmem_base, kTTmemCols); }
}

// ------------------------------------------------------------------------------------------ pair kernel
// 256 x 256 tiles on CTA pairs (cta_group::2), one persistent pair per two SMs; structure as in ns_gemm.cu: each CTA stages 128 rows of
// A and half of B (32 KiB per 128 bytes of K, 5 stages), two accumulators, eight epilogue warps of 32 rows x 128 columns under the next
// tile's main loop.
// In the place of the one-CTA 256 x 256 tile that split tf32 used (64 KiB stages, one accumulator over all of tensor memory, its epilogue
// exposed), same bits: 16 of 1024^3 166 -> 147 us, symmetric 169 -> 114, 2 of 5504 x 2048 x 2048 405 -> 342, 11 of 2048^3 718 -> 690.
constexpr int kGPairStages = 5;
constexpr int kGPairStageBytes = 2 * kTTileBytes;
constexpr int kGPairEpiWarps = 8;
constexpr int kGPairThreads = 64 + 32 * kGPairEpiWarps;
constexpr int kGPairSmemBytes = kGPairStages * kGPairStageBytes + kGPairEpiWarps * kStageWarpBytes + 1024;

// Epilogues of scaled operands may compute blocks from the matrices (65 ms for a tile all of whose blocks are, at K = 2^17), and everything in the
// pair waits for them; 2^18 polls last around 10 ms.
constexpr uint32_t kLongSpinLimit = kSpinLimit << 5;

struct WalkTile {
  int kb_lo, seg;  // K blocks of one term that the tile walks: [kb_lo, kb_lo + seg)
};
__device__ __forceinline__ WalkTile walk_tile(const PairTile& t, int kp, int tri, int block) {
  int lo = 0, hi = kp / block;
  if (tri) {
    lo = min(hi, t.tm * (kPairTile / block));
    hi = t.tn < t.tm ? lo : min(hi, (t.tn + 1) * (kPairTile / block));
  }
  return {lo, hi - lo};
}

template <class Kind>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGPairThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, int M, int N, int kp, int lo_a, int lo_b,
                    int tiles_m, int tiles_n, int per_batch, int total, const Tf32Epilogue E, const __grid_constant__ PairOperands P, int* status) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[kGPairStages];   // used in the even CTA: both CTAs' loads of a stage have landed
  __shared__ __align__(8) uint64_t empty_bar[kGPairStages];  // in each CTA: the products that read the stage have finished
  __shared__ __align__(8) uint64_t acc_full[2];              // in each CTA: accumulator finished
  __shared__ __align__(8) uint64_t acc_empty[2];             // in the even CTA: all sixteen epilogue warps have read it
  __shared__ __align__(8) uint64_t drain_bar;                // in each CTA, teardown only: all products have finished
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag, skip_flag;
  __shared__ int fills;                                      // ring fills this CTA issued

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool leader = elect_one();  // issues the loads (warp 0) and the products (warp 1), and waits for them in the teardown
  const uint32_t rank = cluster_rank();
  uint8_t* ring = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kGPairStages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], 2 * kGPairEpiWarps); }
    mbar_init(&drain_bar, 1);
    abort_flag = 0;
    fills = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) { tmem_alloc_pair(&tmem_base_slot, 512); tmem_relinquish_pair(); }
  griddep_wait();
  // a kernel of this stream already gave up on a wait: do not pile more work on a broken pipeline (the even CTA decides)
  if (threadIdx.x == 0) skip_flag = status != nullptr && *(volatile const int*)status != 0;
  tc_fence_before();
  __syncthreads();
  cluster_sync();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  const bool skip = cluster_load(cluster_addr(&skip_flag, 0)) != 0;

  if (skip) {
  } else if (warp == 0) {
    if (leader) {
      int n = 0;  // ring fills so far
      bool ok = true;
      for (int idx = pair; idx < total && ok; idx += pairs) {
        const PairTile t = pair_tile(idx, tiles_m, tiles_n, per_batch, E.symmetric);
        const WalkTile h = walk_tile(t, kp, E.tri, Kind::kBlock);
        const int a_row = t.tm * kPairTile + (int)rank * 128, b_row = t.tn * kPairTile + (int)rank * 128;
        for (int term = 0; term < 3 && ok; ++term) {
          const int ka = (term == Kind::kTermLoA ? lo_a : 0), kb_off = (term == Kind::kTermLoB ? lo_b : 0);
          for (int kb = 0; kb < h.seg; ++kb, ++n) {
            const int s = n % kGPairStages, round = n / kGPairStages, k0 = (h.kb_lo + kb) * Kind::kBlock;
            ok = mbar_wait<Kind::kScaled ? kLongSpinLimit : kSpinLimit>(&empty_bar[s], (round & 1) ^ 1, &abort_flag);
            if (!ok) break;
            uint8_t* dst = ring + s * kGPairStageBytes;
            const uint32_t bar = cluster_addr(&full_bar[s], 0);
            if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * kGPairStageBytes);
            tma_load_3d_pair(dst, &map_a, bar, ka + k0, a_row, t.batch);  // rows past the operand's end arrive as zeros and count
            tma_load_3d_pair(dst + kTTileBytes, &map_b, bar, kb_off + k0, b_row, t.batch);
          }
        }
      }
      fills = n;
      griddep_launch();  // this CTA's last loads are on their way: the next kernel may take over SMs that drain
    }
  } else if (warp == 1) {
    if (leader && rank == 0) {
      int n = 0, it = 0;
      bool ok = true;
      for (int idx = pair; idx < total && ok; idx += pairs, ++it) {
        const PairTile t = pair_tile(idx, tiles_m, tiles_n, per_batch, E.symmetric);
        const int seg = walk_tile(t, kp, E.tri, Kind::kBlock).seg, num_kb = 3 * seg, acc = it & 1;
        ok = mbar_wait<Kind::kScaled ? kLongSpinLimit : kSpinLimit>(&acc_empty[acc], ((it >> 1) & 1) ^ 1, &abort_flag);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d = tmem_base + (uint32_t)acc * 256u;
        for (int kb = 0; kb < num_kb; ++kb, ++n) {
          const int s = n % kGPairStages, round = n / kGPairStages;
          ok = mbar_wait<Kind::kScaled ? kLongSpinLimit : kSpinLimit>(&full_bar[s], round & 1, &abort_flag);
          if (!ok) break;
          tc_fence_after();
          const uint32_t base = smem_u32(ring + s * kGPairStageBytes);
          const uint64_t a_desc = make_smem_desc(base), b_desc = make_smem_desc(base + kTTileBytes);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (Kind::kCrossFirst && k == 0 && kb == 2 * seg)
              tc_mma_f16_d11_pair(d, a_desc, b_desc, Kind::kPairDesc);
            else
              Kind::mma_pair(d, a_desc + 2 * k, b_desc + 2 * k, Kind::kPairDesc, (kb | k) ? 1u : 0u);
          tc_commit_pair(&empty_bar[s]);
        }
        if (ok) tc_commit_pair(&acc_full[acc]);
      }
    }
  } else {
    const int quarter = warp & 3, half = (warp - 2) >> 2;  // tensor-memory lanes this warp may read; its half of the columns
    float* const stage = (float*)(ring + kGPairStages * kGPairStageBytes + (warp - 2) * kStageWarpBytes);
    const uint32_t tmem_warp = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * 128);
    int it = 0;
    for (int idx = pair; idx < total; idx += pairs, ++it) {
      const PairTile t = pair_tile(idx, tiles_m, tiles_n, per_batch, E.symmetric);
      const int acc = it & 1, row0 = t.tm * kPairTile + (int)rank * 128 + quarter * 32, col0 = t.tn * kPairTile + half * 128;
      const int blocks = min(4, (N - col0 + 31) / 32);
      BlockUnits U{};
      if constexpr (Kind::kScaled)
        if (row0 < M && blocks > 0) U = fetch_units(P, lane, t.batch, row0, col0, M, N);
      const bool ok = mbar_wait<Kind::kScaled ? kLongSpinLimit : kSpinLimit>(&acc_full[acc], (it >> 1) & 1, &abort_flag);
      if (!__all_sync(0xFFFFFFFFu, ok)) break;
      tc_fence_after();
      // a tile on the diagonal: computed whole, or (symmetric == 2) as three of 128 x 128 whose middle one is mirrored
      const bool thirds = E.symmetric == 2 && t.tm == t.tn;
      const bool mirrored = thirds ? rank == 0 && half == 1 : t.tm != t.tn;
      if constexpr (Kind::kScaled)
        if (U.slow != 0 && walk_tile(t, kp, E.tri, Kind::kBlock).seg != 0)
          settle_blocks(U, tmem_warp + (uint32_t)(acc * 256), lane, stage, P, t.batch, row0, col0, M, N, E.tri);
      if (row0 < M && blocks > 0 && !(thirds && rank == 1 && half == 0))
        epilogue_direct<Kind::kScaled>(tmem_warp + (uint32_t)(acc * 256), lane, stage, row0, col0, blocks, mirrored,
                              walk_tile(t, kp, E.tri, Kind::kBlock).seg == 0, t.batch, M, N, E, P, U);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) cluster_arrive(cluster_addr(&acc_empty[acc], 0));
    }
    tc_fence_before();
  }

  // After an expired wait in either CTA, both wait (with a limit) for every product and every load that the pair issued before its
  // shared and tensor memory go away.
  __syncthreads();
  if (threadIdx.x == 0 && abort_flag) cluster_store(cluster_addr(&abort_flag, rank ^ 1), 1);
  cluster_sync();
  if (abort_flag) {
    if (rank == 0 && warp == 1 && leader) tc_commit_pair(&drain_bar);  // the thread that issued the products
    if (threadIdx.x == 0) mbar_drain(&drain_bar, 0);
    if (rank == 0 && threadIdx.x == 0) {
      const int even = fills, odd = cluster_load(cluster_addr(&fills, 1)), top = max(even, odd);
      for (int n = pair_drain_first(even, odd, kGPairStages); n < top; ++n) {
        const int s = n % kGPairStages, kind = pair_fill_kind(n, even, odd);
        if (kind == kFillOddOnly) mbar_expect_tx(&full_bar[s], (uint32_t)kGPairStageBytes);
        if (kind == kFillEvenOnly) mbar_complete_tx(&full_bar[s], (uint32_t)kGPairStageBytes);
        mbar_drain(&full_bar[s], (n / kGPairStages) & 1);
      }
    }
    cluster_sync();
  }
  if (threadIdx.x == 0 && abort_flag && status != nullptr) atomicExch(status, 1);
  if (warp == 1) { __syncwarp(); tc_fence_after(); tmem_dealloc_pair(tmem_base, 512); }
}

}  // namespace
}  // namespace hb
