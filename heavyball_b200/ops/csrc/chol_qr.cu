// A round of Cholesky QR, A <- A R^-1 with R^T R = G = A^T A, as the eigenbasis refresh runs it: recursive, 128-wide leaves
// (chol_inv_leaf of skinny.cu), everything between them products on split tf32.
//
//   factor [lo, hi):  factor [lo, mid);  Y = G[lo:mid, mid:hi]^T R[lo:mid, lo:mid]^-1;  G[mid:hi, mid:hi] -= Y Y^T;  factor [mid, hi)
//   solve X R = B:    X_1 = B_1 R_11^-1;  B_2 -= X_1 R_12;  X_2 = B_2 R_22^-1
//
// A refresh is a chain of a few hundred dependent launches, so what counts is how many there are and how long each takes by itself.  Y is the
// transpose of R[lo:mid, mid:hi], and every product that reads either - the Schur complement, the updates inside later solves, those of the
// rows of A - wants its rows split into [hi | lo].  So the factor exists in that form alone (L, rows of R^T), written by the kernel that solves
// against a leaf, and its blocks are operands by address; rows of A are split by the same kernel, in both orientations.  That leaves no
// operand passes, no copies and no transposes between the products: 49 launches in the place of 95 for a 1024-wide round.  Two rounds and the
// check, replayed, in that form / this: 16 of 1024^2 2.96 / 2.00 ms, 11 of 2048^2 8.33 / 6.09, 8 of 256^2 0.376 / 0.237 (half of it from the
// leaf kernel, which bounds it now: 16 leaves of 25 us, 10 products over whole columns of 91 and 18, the others 8 to 25 us each).
// The products, their tiles and their sums are those of the launch-by-launch form (utils/orthogonal.py), and so are the bits of the result.
#include "chol_qr.h"

#include "per_device.h"
#include "skinny.h"
#include "tc_common.cuh"
#include "tf32_gemm.h"

namespace hb {
namespace {

constexpr int kLeafSolveThreads = 512, kLeafSolveWarps = kLeafSolveThreads / 32;
constexpr int kRowLd = kQrBlock + 4;  // floats per staged row: four values of K per lane and load, lanes on distinct banks
constexpr int leaf_solve_bytes(int lane_rows) { return (kQrBlock * kQrBlock + 32 * lane_rows * kRowLd) * (int)sizeof(float); }

__device__ __forceinline__ float qr_tf32(float x) {
  uint32_t bits;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(bits) : "f"(x));
  return __uint_as_float(bits);
}
__device__ __forceinline__ unsigned long long twice(float x) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "r"(__float_as_uint(x)));
  return r;
}

// 32 kLaneRows rows x 128 columns of X per block, sums over K in its order in fp32.  A warp has 8 columns of all rows, a lane kLaneRows of the rows:
// per k two (broadcast) loads of the inverse, half a load of B and four paired multiply-adds per row.  Only k up to the warp's last column: the
// inverse is upper triangular.  Column groups are dealt to warps so that the four schedulers get the same number of steps.
template <int kLaneRows>
__global__ void __launch_bounds__(kLeafSolveThreads, 2) qr_leaf_solve_kernel(const QrLeafSolve S) {
  constexpr int kRows = 32 * kLaneRows;
  extern __shared__ __align__(16) float qr_smem[];
  float *const t = qr_smem, *const b = qr_smem + kQrBlock * kQrBlock;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r0 = blockIdx.x * kRows;
  const int64_t batch = blockIdx.y;
  griddep_wait();
  griddep_launch();
  const float* inv = S.inv + batch * S.stride_inv;
#pragma unroll
  for (int i = 0; i < kQrBlock / kLeafSolveWarps; ++i) {  // (what lies left of the diagonal is needed as far as its group of eight columns)
    const int r = warp + kLeafSolveWarps * i;
    if (lane * 4 + 7 >= r) *(float4*)(t + r * kQrBlock + lane * 4) = *(const float4*)(inv + r * kQrBlock + lane * 4);
  }
  const float* src = S.src + batch * S.stride;
  if (!S.from_rows) {
#pragma unroll
    for (int i = 0; i < kRows / kLeafSolveWarps; ++i) {
      const int r = warp + kLeafSolveWarps * i;
      *(float4*)(b + r * kRowLd + lane * 4) = *(const float4*)(src + (int64_t)(r0 + r) * S.ld + lane * 4);
    }
  } else if (threadIdx.x < 32 * kRows / 4) {  // 4 x 4 values per thread, turned in registers
    const int r = threadIdx.x % (kRows / 4) * 4, k = threadIdx.x / (kRows / 4) * 4;
    float4 v[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = *(const float4*)(src + (int64_t)(k + e) * S.ld + r0 + r);
    *(float4*)(b + (r + 0) * kRowLd + k) = make_float4(v[0].x, v[1].x, v[2].x, v[3].x);
    *(float4*)(b + (r + 1) * kRowLd + k) = make_float4(v[0].y, v[1].y, v[2].y, v[3].y);
    *(float4*)(b + (r + 2) * kRowLd + k) = make_float4(v[0].z, v[1].z, v[2].z, v[3].z);
    *(float4*)(b + (r + 3) * kRowLd + k) = make_float4(v[0].w, v[1].w, v[2].w, v[3].w);
  }
  __syncthreads();

  // groups g, 7 - g, 8 + g and 15 - g on one scheduler
  const int c0 = ((warp & 4) != 0 ? (warp ^ 3) : warp) * 8;
  unsigned long long acc[kLaneRows][4];  // two neighbouring columns each
#pragma unroll
  for (int r = 0; r < kLaneRows; ++r)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[r][j] = 0ull;
#pragma unroll 2
  for (int k = 0; k < c0 + 8; k += 4) {
    float4 x[kLaneRows];
#pragma unroll
    for (int r = 0; r < kLaneRows; ++r) x[r] = *(const float4*)(b + (lane + 32 * r) * kRowLd + k);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const ulonglong2 m0 = *(const ulonglong2*)(t + (k + e) * kQrBlock + c0), m1 = *(const ulonglong2*)(t + (k + e) * kQrBlock + c0 + 4);
#pragma unroll
      for (int r = 0; r < kLaneRows; ++r) {
        const unsigned long long p = twice(e == 0 ? x[r].x : e == 1 ? x[r].y : e == 2 ? x[r].z : x[r].w);
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[r][0]) : "l"(p), "l"(m0.x));
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[r][1]) : "l"(p), "l"(m0.y));
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[r][2]) : "l"(p), "l"(m1.x));
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[r][3]) : "l"(p), "l"(m1.y));
      }
    }
  }
  __syncthreads();  // B has been read: its place takes X
#pragma unroll
  for (int r = 0; r < kLaneRows; ++r) {
    *(ulonglong2*)(b + (lane + 32 * r) * kRowLd + c0) = make_ulonglong2(acc[r][0], acc[r][1]);
    *(ulonglong2*)(b + (lane + 32 * r) * kRowLd + c0 + 4) = make_ulonglong2(acc[r][2], acc[r][3]);
  }
  __syncthreads();

  if (S.out != nullptr || S.same != nullptr) {
#pragma unroll
    for (int i = 0; i < kRows / kLeafSolveWarps; ++i) {
      const int r = warp + kLeafSolveWarps * i;
      const float4 x = *(const float4*)(b + r * kRowLd + lane * 4);
      if (S.out != nullptr) *(float4*)(S.out + batch * S.stride_out + (int64_t)(r0 + r) * S.ld_out + lane * 4) = x;
      if (S.same != nullptr) {
        const float4 hi = make_float4(qr_tf32(x.x), qr_tf32(x.y), qr_tf32(x.z), qr_tf32(x.w));
        float* to = S.same + batch * S.stride_same + (int64_t)(r0 + r) * S.ld_same + lane * 4;
        *(float4*)to = hi;
        *(float4*)(to + S.lo_same) = make_float4(qr_tf32(x.x - hi.x), qr_tf32(x.y - hi.y), qr_tf32(x.z - hi.z), qr_tf32(x.w - hi.w));
      }
    }
  }
  if (S.trans != nullptr) {  // consecutive lanes on consecutive rows: 32 of a column are a line
#pragma unroll 4
    for (int i = warp; i < kLaneRows * kQrBlock; i += kLeafSolveWarps) {
      const int c = i / kLaneRows, r = i % kLaneRows * 32 + lane;
      const float x = b[r * kRowLd + c], hi = qr_tf32(x);
      float* to = S.trans + batch * S.stride_trans + (int64_t)c * S.ld_trans + r0 + r;
      to[0] = hi;
      to[S.lo_trans] = qr_tf32(x - hi);
    }
  }
}

// 64 x 64 values per block: divided by their column's norm (in full, subnormal values kept), stored, and turned through shared memory into rows of
// the operand.  One pass in the place of a division (138 us for 11 of 2048^2, the library's broadcast along rows) and an operand pass (86).
__global__ void __launch_bounds__(256) qr_unit_columns_kernel(const float* X, const float* __restrict__ norm, float* A, float* __restrict__ trans, int n,
                                                             int k) {
  __shared__ float tile[64][65];
  const int64_t b = blockIdx.z;
  const int c0 = blockIdx.x * 64, r0 = blockIdx.y * 64, q = (threadIdx.x & 15) * 4, line = threadIdx.x >> 4;
  const float4 by = *(const float4*)(norm + b * k + c0 + q);
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const int64_t at = (b * n + r0 + line + 16 * p) * k + c0 + q;
    float4 v = *(const float4*)(X + at);
    asm("div.rn.f32 %0, %0, %1;" : "+f"(v.x) : "f"(by.x));
    asm("div.rn.f32 %0, %0, %1;" : "+f"(v.y) : "f"(by.y));
    asm("div.rn.f32 %0, %0, %1;" : "+f"(v.z) : "f"(by.z));
    asm("div.rn.f32 %0, %0, %1;" : "+f"(v.w) : "f"(by.w));
    *(float4*)(A + at) = v;
    tile[line + 16 * p][q] = v.x;
    tile[line + 16 * p][q + 1] = v.y;
    tile[line + 16 * p][q + 2] = v.z;
    tile[line + 16 * p][q + 3] = v.w;
  }
  __syncthreads();
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const int c = line + 16 * p;
    float hi[4], lo[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float x = tile[q + e][c];
      hi[e] = qr_tf32(x);
      lo[e] = qr_tf32(x - hi[e]);
    }
    float* row = trans + (b * k + c0 + c) * 2 * n + r0 + q;
    *(float4*)row = make_float4(hi[0], hi[1], hi[2], hi[3]);
    *(float4*)(row + n) = make_float4(lo[0], lo[1], lo[2], lo[3]);
  }
}

// g[j][i] <- g[i][j] for rows [lo, mid) and columns [mid, hi) of symmetric matrices, 32 x 32 at a time.
__global__ void __launch_bounds__(256) qr_mirror_kernel(float* g, int k, int lo, int mid) {
  __shared__ float tile[32][33];
  griddep_wait();
  griddep_launch();
  float* m = g + (int64_t)blockIdx.z * k * k;
  const int i0 = lo + blockIdx.y * 32, j0 = mid + blockIdx.x * 32, x = threadIdx.x & 31, y = threadIdx.x >> 5;
#pragma unroll
  for (int r = y; r < 32; r += 8) tile[r][x] = m[(int64_t)(i0 + r) * k + j0 + x];
  __syncthreads();
#pragma unroll
  for (int r = y; r < 32; r += 8) m[(int64_t)(j0 + r) * k + i0 + x] = tile[x][r];
}

// Where a block of `width` columns is cut: the recursion of utils/orthogonal.py and utils/core.py.
int first_part(int width) { return width / 2 / kQrBlock * kQrBlock > kQrBlock ? width / 2 / kQrBlock * kQrBlock : kQrBlock; }

struct Round {
  const QrRound& Q;
  cudaStream_t stream;
  int* launches;
  cudaError_t error = cudaSuccess;

  void note(cudaError_t e, int kernels = 1) {
    if (error == cudaSuccess) error = e;
    *launches += kernels;
  }
  float* g(int row, int col) const { return Q.G + (int64_t)row * Q.k + col; }
  Tf32Operand l(int row, int col) const { return {Q.L + (int64_t)row * 2 * Q.k + col, 2 * Q.k, (int64_t)Q.k * 2 * Q.k, Q.k}; }

  // C[rows, cols] -= A B^T over K columns of both
  void subtract(Tf32Operand A, Tf32Operand B, float* C, int64_t stride, int rows, int cols, int K, bool symmetric) {
    Tf32Epilogue E{};
    E.mode = kEpiAdd;
    E.alpha = -1.0f;
    E.C = C;
    E.ldc = Q.k;
    E.strideC = stride;
    E.symmetric = symmetric ? 1 : 0;
    note(launch_tf32_gemm(A, B, rows, cols, K, Q.batch, E, Q.status, stream));
  }
  void leaf_solve(QrLeafSolve S, int block, int rows) {
    const int64_t size = kQrBlock * kQrBlock;
    S.inv = Q.inv + block * size;
    S.stride_inv = Q.k / kQrBlock * size;
    note(launch_qr_leaf_solve(S, rows, Q.batch, stream));
  }

  // Columns [lo, hi) of X with X R = B.  Rows [row0, row0 + rows) of L (of_l: B lies below the diagonal of G), or all rows of A.
  void solve(int lo, int hi, bool of_l, int row0, int rows) {
    if (hi - lo == kQrBlock) {
      QrLeafSolve S{};
      S.ld = Q.k;
      if (of_l) {
        S.src = g(row0, lo);
        S.stride = (int64_t)Q.k * Q.k;
        put_l(S, row0, lo);
      } else {
        S.src = Q.A + lo;
        S.stride = (int64_t)Q.n * Q.k;
        S.out = Q.A + lo;  // in the place of B, whose rows a block of threads has read when it writes them
        S.ld_out = Q.k;
        S.stride_out = (int64_t)Q.n * Q.k;
        if (hi < Q.k) {  // (nothing to the right of the last block: never an operand)
          S.same = Q.X_same + lo;
          S.ld_same = 2 * Q.k;
          S.lo_same = Q.k;
          S.stride_same = (int64_t)Q.n * 2 * Q.k;
        }
        if (Q.X_trans != nullptr) {
          S.trans = Q.X_trans + (int64_t)lo * 2 * Q.n;
          S.ld_trans = 2 * Q.n;
          S.lo_trans = Q.n;
          S.stride_trans = (int64_t)Q.k * 2 * Q.n;
        }
      }
      leaf_solve(S, lo / kQrBlock, rows);
      return;
    }
    const int mid = lo + first_part(hi - lo);
    solve(lo, mid, of_l, row0, rows);
    const Tf32Operand x = of_l ? l(row0, lo) : Tf32Operand{Q.X_same + lo, 2 * Q.k, (int64_t)Q.n * 2 * Q.k, Q.k};
    float* const b = of_l ? g(row0, mid) : Q.A + mid;
    subtract(x, l(mid, lo), b, of_l ? (int64_t)Q.k * Q.k : (int64_t)Q.n * Q.k, rows, hi - mid, mid - lo, false);
    solve(mid, hi, of_l, row0, rows);
  }
  void put_l(QrLeafSolve& S, int row, int col) const {
    const Tf32Operand to = l(row, col);
    S.same = const_cast<float*>(to.p);
    S.ld_same = to.ld;
    S.lo_same = to.lo;
    S.stride_same = to.stride;
  }

  // `even`: all products that updated this block began at multiples of 256.
  void factor(int lo, int hi, bool even) {
    if (hi - lo == kQrBlock) {
      const int64_t size = kQrBlock * kQrBlock;
      note(launch_chol_inv_leaf(g(lo, lo), Q.k, (int64_t)Q.k * Q.k, nullptr, 0, 0, Q.inv + lo / kQrBlock * size, Q.k / kQrBlock * size, Q.batch,
                                kQrBlock, Q.info, stream));
      return;
    }
    const int mid = lo + first_part(hi - lo);
    const bool mirrored = even && mid % 256 == 0;
    factor(lo, mid, even);
    if (mid - lo == kQrBlock) {  // one leaf wide: read from above the diagonal
      QrLeafSolve S{};
      S.src = g(lo, mid);
      S.ld = Q.k;
      S.stride = (int64_t)Q.k * Q.k;
      S.from_rows = 1;
      put_l(S, mid, lo);
      leaf_solve(S, lo / kQrBlock, hi - mid);
    } else {
      // wider: worked on in place below the diagonal, where products have stored the same block mirrored - except within a 256 x 256 tile on
      // the diagonal, both halves of which are computed; the upper one counts
      if (!mirrored) note(launch_chained(qr_mirror_kernel, dim3((hi - mid) / 32, (mid - lo) / 32, Q.batch), 256, 0, stream, Q.G, Q.k, lo, mid));
      solve(lo, mid, true, mid, hi - mid);
    }
    subtract(l(mid, lo), l(mid, lo), g(mid, mid), (int64_t)Q.k * Q.k, hi - mid, hi - mid, mid - lo, true);
    factor(mid, hi, mirrored);
  }
};

}  // namespace

cudaError_t launch_qr_leaf_solve(const QrLeafSolve& S, int rows, int batch, cudaStream_t stream) {
  static PerDevice<int> resident;  // blocks of 32 rows
  int device = 0, slots = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e == cudaSuccess)
    e = resident.get(device, cudaSuccess, &slots, [device](int& found) {
      int sms = 0;
      cudaError_t s = cudaFuncSetAttribute(qr_leaf_solve_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, leaf_solve_bytes(1));
      if (s == cudaSuccess) s = cudaFuncSetAttribute(qr_leaf_solve_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, leaf_solve_bytes(2));
      if (s == cudaSuccess) s = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
      found = 2 * sms;
      return s;
    });
  if (e != cudaSuccess) return e;
  if (rows % kQrRows != 0 || batch > 65535) return cudaErrorInvalidValue;
  if (rows == 0 || batch == 0) return cudaSuccess;
  // few rows: the chain waits for one block, and one of 32 rows is done sooner (rows of 16 matrices, 64 / 32 per block: 128 rows 11.8 / 8.2 us, 512
  // rows 12.0 / 11.7); more than fit at once: 64, the inverse is read half as often
  if ((int64_t)(rows / 32) * batch <= slots)
    return launch_chained(qr_leaf_solve_kernel<1>, dim3(rows / 32, batch), kLeafSolveThreads, leaf_solve_bytes(1), stream, S);
  return launch_chained(qr_leaf_solve_kernel<2>, dim3(rows / 64, batch), kLeafSolveThreads, leaf_solve_bytes(2), stream, S);
}

cudaError_t launch_qr_unit_columns(const float* X, const float* norm, float* A, float* A_trans, int batch, int n, int k, cudaStream_t stream) {
  if (n % 64 != 0 || k % kQrBlock != 0 || batch > 65535 || n / 64 > 65535) return cudaErrorInvalidValue;
  if (batch == 0 || n == 0 || k == 0) return cudaSuccess;
  qr_unit_columns_kernel<<<dim3(k / 64, n / 64, batch), 256, 0, stream>>>(X, norm, A, A_trans, n, k);
  return cudaGetLastError();
}

cudaError_t launch_chol_qr_round(const QrRound& Q, int* launches, cudaStream_t stream) {
  if (Q.n % kQrRows != 0 || Q.k % kQrBlock != 0 || Q.k == 0 || Q.batch > 65535) return cudaErrorInvalidValue;
  if (Q.n == 0 || Q.batch == 0) return cudaSuccess;
  Round R{Q, stream, launches};
  R.factor(0, Q.k, true);
  R.solve(0, Q.k, false, 0, Q.n);
  return R.error;
}

}  // namespace hb
