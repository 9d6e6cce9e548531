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
// GEMM kernel (one 128x128 output tile per CTA, 192 threads, two CTAs per SM):
//   warp 0     : TMA producer, cp.async.bulk.tensor 3-D loads (128-byte swizzle, 32 fp32 per row) into a 3-stage ring
//   warp 1     : tcgen05.mma.cta_group::1.kind::tf32, 128x128x8 per instruction, accumulator in 128 TMEM columns
//   warps 2..5 : tcgen05.ld, then the epilogue.  Plain stores go through the (now idle) ring and four bulk tensor
//                stores.  Fused epilogues work in registers and store directly: scale; lerp into the statistics
//                matrix (GG <- lerp(GG, G G^T)); Adam / LaProp in the eigenbasis (moments read and written in
//                place, the preconditioned value goes on); and, for any of them, the result written in the split
//                [hi | lo] layout - as it is or transposed - so the next product of the chain needs no split pass.
// Waits are bounded as in the bf16 kernels: on expiry the CTA flags `status`, drains, frees TMEM and returns.
#include "tf32_gemm.h"

#include "gemm_epilogue.cuh"
#include "per_device.h"

namespace hb {
namespace {

constexpr int TBK = 32;
// tf32 x tf32 -> fp32, both operands K-major, M = 128, N = 128
constexpr uint32_t kTf32InstrDesc =
    (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(TBN >> 3) << 17) | ((uint32_t)(TBM >> 4) << 24);

struct Tf32Kind {
  static constexpr int kBlock = TBK;
  static constexpr bool kScaled = false, kCrossFirst = false;
  static constexpr int kTermLoA = 2, kTermLoB = 1;  // A: hi, hi, lo   B: hi, lo, hi
  static constexpr uint32_t kDesc = kTf32InstrDesc;
  __device__ static __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t desc, uint32_t accumulate) {
    tc_mma_tf32(d, a, b, desc, accumulate);
  }
};

// ------------------------------------------------------------------------------------------ 256 x 256 tiles
// A 128 x 128 tile asks the L2 for 32 KiB of operands per 256 tensor-core cycles (tf32 runs at half the bf16 rate on
// operands twice as wide), which is more than the L2 delivers to 148 SMs at once; a 256 x 256 tile needs half of that
// per FLOP.  One CTA per SM: four 128 x 128 fp32 accumulators = all 512 columns of tensor memory, 64 KiB ring stages
// (two 128-row boxes per operand), two 128 x 256 x 8 instructions per 8 of K sharing the B rows.  Eight epilogue
// warps: two per 32-lane quarter of tensor memory, one for each 128-row half of the tile.
constexpr int TBM2 = 256, TBN2 = 256;
constexpr int kTStageBytes2 = 4 * kTTileBytes;                  // 64 KiB
constexpr int kTSmemBytes2 = kTStages * kTStageBytes2 + 1024;
constexpr int kTThreads2 = 320;                                 // producer, MMA, 8 epilogue warps
constexpr uint32_t kTTmemCols2 = 512;
constexpr uint32_t kTf32InstrDesc256 =
    (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(TBN2 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);

__global__ void __launch_bounds__(kTThreads2, 1)
tf32_gemm256_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, int M, int N, int kp,
                    const Tf32Epilogue E, int* status) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[kTStages];
  __shared__ __align__(8) uint64_t empty_bar[kTStages];
  __shared__ __align__(8) uint64_t accum_bar, drain_bar;  // drain_bar: teardown only
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool leader = elect_one();  // issues the loads (warp 0) and the products (warp 1), and waits for them in the teardown
  uint8_t* tiles = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int tiles_n = (N + TBN2 - 1) / TBN2;
  int tm = blockIdx.x / tiles_n, tn = blockIdx.x % tiles_n;
  if (E.symmetric) {
    int left = blockIdx.x;
    tm = 0;
    while (left >= tiles_n - tm) { left -= tiles_n - tm; ++tm; }
    tn = tm + left;
  }
  const int batch = blockIdx.y;
  int kb_lo = 0, kb_hi = kp / TBK;
  if (E.tri) {
    kb_lo = min(kb_hi, tm * (TBM2 / TBK));
    kb_hi = tn < tm ? kb_lo : min(kb_hi, (tn + 1) * (TBN2 / TBK));
  }
  const int seg_kb = kb_hi - kb_lo;
  const int num_kb = 3 * seg_kb;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kTStages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(&accum_bar, 1);
    mbar_init(&drain_bar, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) { tmem_alloc(&tmem_base_slot, kTTmemCols2); tmem_relinquish(); }
  griddep_wait();
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
        uint8_t* dst = tiles + s * kTStageBytes2;
        const int seg = kb / seg_kb, k0 = (kb_lo + kb - seg * seg_kb) * TBK;
        const int ka = k0 + (seg == 2 ? kp : 0), kb_col = k0 + (seg == 1 ? kp : 0);   // A: hi, hi, lo   B: hi, lo, hi
        mbar_expect_tx(&full_bar[s], kTStageBytes2);   // rows past the operand's end arrive as zeros and count as bytes
        tma_load_3d(dst, &map_a, &full_bar[s], ka, tm * TBM2, batch);
        tma_load_3d(dst + kTTileBytes, &map_a, &full_bar[s], ka, tm * TBM2 + 128, batch);
        tma_load_3d(dst + 2 * kTTileBytes, &map_b, &full_bar[s], kb_col, tn * TBN2, batch);
        tma_load_3d(dst + 3 * kTTileBytes, &map_b, &full_bar[s], kb_col, tn * TBN2 + 128, batch);
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
        const uint32_t base = smem_u32(tiles + s * kTStageBytes2);
        const uint64_t a_top = make_smem_desc(base), a_bot = make_smem_desc(base + kTTileBytes);
        // 256 B rows = 32 eight-row groups, 1 KiB apart: the two 128-row boxes are contiguous
        const uint64_t b_desc = make_smem_desc(base + 2 * kTTileBytes);
#pragma unroll
        for (int k = 0; k < TBK / 8; ++k) {
          const uint32_t acc = (kb | k) ? 1u : 0u;
          tc_mma_tf32(tmem_base, a_top + 2 * k, b_desc + 2 * k, kTf32InstrDesc256, acc);
          tc_mma_tf32(tmem_base + 256u, a_bot + 2 * k, b_desc + 2 * k, kTf32InstrDesc256, acc);
        }
        tc_commit(&empty_bar[s]);
      }
      if (ok) tc_commit(&accum_bar);
    }
  } else {
    const int quarter = warp & 3, half = (warp - 2) >> 2;   // warps 2..5: rows 0..127 of the tile, warps 6..9: rows 128..255
    const bool have = (num_kb == 0) || mbar_wait(&accum_bar, 0, &abort_flag);
    tc_fence_after();
    const int row0 = tm * TBM2 + half * 128 + quarter * 32;
    if (have && row0 < M)
      epilogue_direct<false>(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * 256), lane,
                      (float*)(tiles + (warp - 2) * kStageWarpBytes), row0, tn * TBN2, TBN2 / 32, tm != tn, num_kb == 0,
                      batch, M, N, E);
    tc_fence_before();
  }

  __syncthreads();
  if (abort_flag) {
    if (warp == 0 && leader) ring_drain(full_bar, issued, kTStages);
    if (warp == 1 && leader) products_drain(&drain_bar);
    __syncthreads();
    if (threadIdx.x == 0 && status != nullptr) atomicExch(status, 1);
  }
  if (warp == 1) { __syncwarp(); tc_fence_after(); tmem_dealloc(tmem_base, kTTmemCols2); }
}

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

cudaError_t launch_tf32_gemm(const float* A2, const float* B2, int M, int N, int K, int batch, const Tf32Epilogue& E,
                             int* status, cudaStream_t stream) {
  static PerDevice<bool> configured;
  int device = 0;
  bool done = false;
  cudaError_t e = cudaGetDevice(&device);
  if (e == cudaSuccess)
    e = configured.get(device, cudaSuccess, &done, [](bool&) {
      const cudaError_t s = cudaFuncSetAttribute(gemm128_kernel<Tf32Kind>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTSmemBytes);
      return s != cudaSuccess ? s : cudaFuncSetAttribute(tf32_gemm256_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTSmemBytes2);
    });
  if (e != cudaSuccess) return e;
  if (M == 0 || N == 0 || batch == 0) return cudaSuccess;
  if ((E.mode == kEpiAdam || E.mode == kEpiLaProp) && (E.m == nullptr || E.v == nullptr)) return cudaErrorInvalidValue;
  if ((E.mode == kEpiLerp || E.mode == kEpiAdd) && E.C == nullptr) return cudaErrorInvalidValue;
  if (E.tri && (M != N || M != K || E.symmetric)) return cudaErrorInvalidValue;
  if (E.symmetric && (A2 != B2 || M != N || E.C == nullptr || E.S != nullptr || (E.mode != kEpiStore && E.mode != kEpiLerp && E.mode != kEpiAdd)))
    return cudaErrorInvalidValue;
  const int64_t kp = tf32_split_kp(K), ld = 2 * kp;
  CUtensorMap ma, mb, mc;
  if (!make_f32_map(&ma, A2, M, ld, ld, (int64_t)M * ld, batch) || !make_f32_map(&mb, B2, N, ld, ld, (int64_t)N * ld, batch))
    return cudaErrorInvalidValue;

  // big tiles once there are enough of them to fill the machine (one CTA per SM) and K is long enough to pay for a
  // serial epilogue; small problems keep 128 x 128 tiles, two CTAs per SM
  const int big_m = (M + TBM2 - 1) / TBM2, big_n = (N + TBN2 - 1) / TBN2;
  const int64_t big_tiles = (int64_t)(E.symmetric ? big_n * (big_n + 1) / 2 : big_m * big_n) * batch;
  bool big = M >= TBM2 && N >= TBN2 && K >= 512 && big_tiles >= 96;
  if (g_tf32_tile_override == 128) big = false;
  if (g_tf32_tile_override == 256) big = true;
  if (big) {
    dim3 grid(E.symmetric ? big_n * (big_n + 1) / 2 : big_m * big_n, batch);
    return launch_chained(tf32_gemm256_kernel, grid, kTThreads2, kTSmemBytes2, stream, ma, mb, M, N, (int)kp, E, status);
  }

  // plain products leave through the bulk-store path (bulk stores end on 16-byte boundaries: with N a multiple of 4 they write nothing
  // past it); everything else is written by the epilogue threads themselves
  const int bulk = (!E.symmetric && !E.tri && E.mode == kEpiStore && E.S == nullptr && E.C != nullptr && (N & 3) == 0 && (E.ldc & 3) == 0 &&
                    (E.strideC & 3) == 0 && (((uintptr_t)E.C) & 15) == 0) ? 1 : 0;
  mc = ma;  // placeholder when the bulk-store path is not taken (never dereferenced then)
  if (bulk && !make_f32_map(&mc, E.C, M, N, E.ldc, E.strideC, batch)) return cudaErrorInvalidValue;
  const int tiles_m = (M + TBM - 1) / TBM, tiles_n = (N + TBN - 1) / TBN;
  dim3 grid(E.symmetric ? tiles_n * (tiles_n + 1) / 2 : tiles_m * tiles_n, batch);
  return launch_chained(gemm128_kernel<Tf32Kind>, grid, kTThreads, kTSmemBytes, stream, ma, mb, mc, M, N, (int)kp, E, nullptr, 0, nullptr, 0, bulk, status);
}

}  // namespace hb
