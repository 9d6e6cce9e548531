// Newton–Schulz / Polar-Express building blocks for sm_100a.
//
// One polynomial step X <- (a I + b S + c S^2) X with S = X X^T (heavyball/utils.py:550-577, 605-631)
// is executed as three batched bf16 GEMMs with fp32 accumulation in tensor memory:
//     gram : S  = X  X^T                       (symmetric: upper-triangular tiles only, mirrored)
//     poly : Y  = c S S + b S + a I            (symmetric; S is both operands and an epilogue input)
//     apply: X' = Y X
// Gram and polynomial are "TN" products D[M,N] = A[M,K] * B[N,K]^T with both operands K-major; the apply product takes
// X as it lies in memory ([K, N], N contiguous) through an MN-major B descriptor, so the iterate exists once and no
// transposed copy of it is ever written (half of the bytes of every apply epilogue and of the prologue; GPT-2-small's
// 48 matrices: 2634 -> 2513 us, a Llama-3-8B layer: 19.97 -> 18.71 ms).  The three differ only in the B box, its descriptor
// and the epilogue.  Two kernels share them: 128 x 128 tiles, and 256 x 256 tiles on CTA pairs for large launches (ns_tiles.h).
//
// Kernel structure (one 128x128 output tile per CTA, 192 threads, two CTAs resident per SM so one
// CTA's epilogue overlaps the other's main loop):
//   warp 0      : TMA producer  - cp.async.bulk.tensor (3-D maps, 128B swizzle) into a 3-stage ring
//   warp 1      : MMA issuer    - tcgen05.mma.cta_group::1.kind::f16, 128x128x16 per instruction,
//                                 accumulator = 128 TMEM columns; tcgen05.commit releases ring slots
//   warps 2..5  : epilogue      - tcgen05.ld 32x32b from their TMEM lane quarter, fused scalar math (the
//                                 S tile of the polynomial arrives by TMA in a freed ring slot), bf16
//                                 tile and its transpose staged in swizzled shared memory and written
//                                 with cp.async.bulk.tensor stores; fp32 final output stored directly
// Every mbarrier wait is bounded; on expiry the CTA raises a flag in global memory, drains what it
// issued, frees its TMEM columns and returns, so a protocol bug cannot wedge the device.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "ns_gemm.h"
#include "ns_tiles.h"

#include <algorithm>
#include <mutex>
#include <unordered_map>
#include <vector>
#include "pair_drain.h"
#include "per_device.h"
#include "tc_common.cuh"

namespace hb {

constexpr int BM = 128, BN = 128, BK = 64;
constexpr int kStages = 3;
constexpr int kTileBytes = BM * BK * 2;            // 16 KiB per operand tile
constexpr int kStageBytes = 2 * kTileBytes;        // A + B
constexpr int kSmemBytes = kStages * kStageBytes + 1024;  // + slack for 1 KiB alignment
constexpr int kGemmThreads = 192;
constexpr uint32_t kTmemCols = 128;

// bf16 x bf16 -> fp32, both operands K-major, M = 128, N = 128.
constexpr uint32_t kInstrDesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);

// B given as [K, N] with N contiguous (MN-major): boxes of 64 columns x 64 rows of K, one 128-byte swizzle atom wide.
// Consecutive groups of 64 columns are one box apart, groups of 8 rows of K 1 KiB; 16 rows of K are 2 KiB.
constexpr int kMnBoxBytes = 64 * BK * 2;
constexpr uint32_t kMnStep = (16 * 128) >> 4;
constexpr uint32_t kInstrBMn = 1u << 16;

// ------------------------------------------------------------------------------------------ grouped launches
// One launch covers the same stage of every shape bucket of a step (up to kMaxGroups products of different sizes): the tiles
// of all of them share the machine, and a step is 15 launches instead of 15 per bucket (five small odd matrices in four shapes:
// 654 -> 276 us; GPT-2-small's 48 matrices in four shapes: 2513 -> 1920 us together with the pair kernel below).
constexpr int kMaxGroups = 8;
struct GemmGroup {
  CUtensorMap a, b, c, ct, s;  // s: the polynomial's epilogue operand (pair kernel); absent operands repeat `a`
  GemmParams P;
  int tiles_m, tiles_n, per_batch;
  int f_bulk;                  // F leaves through bulk stores, described by `c` (pair kernel)
};
// kRoom groups at most.  A launch's arguments are copied by the host, and 7 KB take longer than 3.5: up to kFewGroups groups go in a
// smaller struct (five small odd matrices in four shapes, a step's 15 launches: 80 -> 65 us of host time).
constexpr int kFewGroups = 4;
template <int kRoom>
struct GemmGroups {
  int n, total;
  int first[kRoom];            // index of each group's first tile within the launch
  int* status;
  GemmGroup g[kRoom];
};

struct TileAt : PairTile {
  int group;
};
template <int kRoom>
__device__ __forceinline__ TileAt tile_at(const GemmGroups<kRoom>& L, int idx) {
  TileAt t;
  t.group = 0;
#pragma unroll
  for (int i = 1; i < kRoom; ++i)
    if (i < L.n && idx >= L.first[i]) t.group = i;
  const GemmGroup& G = L.g[t.group];
  static_cast<PairTile&>(t) = pair_tile(idx - L.first[t.group], G.tiles_m, G.tiles_n, G.per_batch, G.P.symmetric);
  return t;
}

// ------------------------------------------------------------------------------------------ kernel
template <int kRoom>
__global__ void __launch_bounds__(kGemmThreads, 2) ns_gemm_kernel(const __grid_constant__ GemmGroups<kRoom> L) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[kStages];
  __shared__ __align__(8) uint64_t empty_bar[kStages];
  __shared__ __align__(8) uint64_t accum_bar, drain_bar;  // drain_bar: teardown only
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool leader = elect_one();  // issues the loads (warp 0) and the products (warp 1), and waits for them in the teardown
  uint8_t* tiles = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);

  const TileAt tile = tile_at(L, blockIdx.x);
  const GemmGroup& G = L.g[tile.group];
  const GemmParams P = G.P;  // by value: through the reference every use would be a load (nothing survives the asm fences)
  const int tm = tile.tm, tn = tile.tn, batch = tile.batch;
  const int num_kb = (P.K + BK - 1) / BK;
  const bool poly = P.mode == kModePoly;
  const bool same_ab = P.same_operand && tm == tn;  // A and B tiles coincide
  // after the main loop the ring is reused: slot sx receives the S tile (poly), the next two stage
  // the output tile and its transpose for the bulk stores
  const int sx = num_kb % kStages;
  uint8_t* s_tile = tiles + sx * kStageBytes;
  uint8_t* c_stage = tiles + ((sx + 1) % kStages) * kStageBytes;
  uint8_t* ct_stage = tiles + ((sx + 2) % kStages) * kStageBytes;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(&accum_bar, 1);
    mbar_init(&drain_bar, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) { tmem_alloc(&tmem_base_slot, kTmemCols); tmem_relinquish(); }
  griddep_wait();
  // a kernel of this stream already gave up on a wait: do not pile more work on a broken pipeline
  const bool skip = __syncthreads_or(threadIdx.x == 0 && L.status != nullptr && *(volatile const int*)L.status != 0);
  griddep_launch();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;

  int issued = 0;  // producer: ring fills whose loads were issued
  if (skip) {
  } else if (warp == 0) {
    if (leader) {
      const int total = num_kb + (poly ? 1 : 0);
      for (int kb = 0; kb < total; ++kb) {
        const int s = kb % kStages, round = kb / kStages;
        if (!mbar_wait(&empty_bar[s], (round & 1) ^ 1, &abort_flag)) break;
        uint8_t* a_dst = tiles + s * kStageBytes;
        if (kb < num_kb) {
          // diagonal tiles of a symmetric product multiply a row block with itself: one load feeds both operands
          mbar_expect_tx(&full_bar[s], same_ab ? kTileBytes : kStageBytes);
          tma_load_3d(a_dst, &G.a, &full_bar[s], kb * BK, tm * BM, batch);
          if (P.b_mn) {  // [K, N] operand: two boxes of 64 columns x 64 rows of K
            tma_load_3d(a_dst + kTileBytes, &G.b, &full_bar[s], tn * BN, kb * BK, batch);
            tma_load_3d(a_dst + kTileBytes + kMnBoxBytes, &G.b, &full_bar[s], tn * BN + 64, kb * BK, batch);
          } else if (!same_ab) {
            tma_load_3d(a_dst + kTileBytes, &G.b, &full_bar[s], kb * BK, tn * BN, batch);
          }
        } else {
          mbar_expect_tx(&full_bar[s], kStageBytes);  // S[tm-block, tn-block] for the polynomial epilogue, as two 64-column halves
          tma_load_3d(a_dst, &G.a, &full_bar[s], tn * BN, tm * BM, batch);
          tma_load_3d(a_dst + kTileBytes, &G.a, &full_bar[s], tn * BN + BK, tm * BM, batch);
        }
        issued = kb + 1;
      }
    }
  } else if (warp == 1) {
    if (leader) {
      bool ok = true;
      for (int kb = 0; kb < num_kb && ok; ++kb) {
        const int s = kb % kStages, round = kb / kStages;
        ok = mbar_wait(&full_bar[s], round & 1, &abort_flag);
        if (!ok) break;
        tc_fence_after();
        const uint32_t a_addr = smem_u32(tiles + s * kStageBytes);
        const uint64_t a_desc = make_smem_desc(a_addr);
        const uint64_t b_desc = same_ab ? a_desc : (P.b_mn ? make_smem_desc_mn(a_addr + kTileBytes, kMnBoxBytes) : make_smem_desc(a_addr + kTileBytes));
        const uint32_t b_step = P.b_mn ? kMnStep : 2u, idesc = kInstrDesc | (P.b_mn ? kInstrBMn : 0u);
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) {
          // advancing 16 bf16 (32 B) along K inside the swizzle atom = +2 in 16-byte address units
          tc_mma_bf16(tmem_base, a_desc + 2 * k, b_desc + b_step * k, idesc, (kb | k) ? 1u : 0u);
        }
        tc_commit(&empty_bar[s]);
      }
      if (ok) tc_commit(&accum_bar);
    }
  } else {
    // ---------------------------------------------------------------- epilogue warps (128 threads)
    const int quarter = warp & 3;            // TMEM lane quarter this warp may read
    const int r = quarter * 32 + lane;       // row inside the tile
    const int row = tm * BM + r;             // global output row
    bool have = (num_kb == 0) || mbar_wait(&accum_bar, 0, &abort_flag);
    if (have && poly) have = mbar_wait(&full_bar[sx], (num_kb / kStages) & 1, &abort_flag);
    tc_fence_after();
    const bool mirror = P.symmetric ? (tn != tm) : true;
    const bool want_c = P.C != nullptr, want_ct = P.CT != nullptr && mirror;
    if (have) {
      const int64_t b64 = batch;
#pragma unroll 1
      for (int cb = 0; cb < BN / 32; ++cb) {
        uint32_t acc[32];
        if (num_kb > 0) {
          tmem_ld32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(cb * 32), acc);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) acc[j] = 0u;
        }
        const int half = cb >> 1, q0 = (cb & 1) * 4;  // 64-column half of the tile, first 16-byte chunk in it
        const int col0 = tn * BN + cb * 32;
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(acc[j]);

        if (poly) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint4 sv = *(const uint4*)(s_tile + half * kTileBytes + swz(r, q0 + q));
            const uint32_t w[4] = {sv.x, sv.y, sv.z, sv.w};
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const int j = q * 8 + e;
              const float sval = bf16_bits_to_float((uint16_t)((w[e >> 1] >> ((e & 1) * 16)) & 0xFFFF));
              v[j] = P.cc * v[j] + P.cb * sval + ((col0 + j == row) ? P.ca : 0.f);
            }
          }
        }
        // rounded once, so that the tile and its mirrored / transposed copy agree bit for bit
        uint16_t h[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) h[j] = rne_bf16_bits(v[j]);

        if (want_c) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint4 o;
            o.x = (uint32_t)h[q * 8 + 0] | ((uint32_t)h[q * 8 + 1] << 16);
            o.y = (uint32_t)h[q * 8 + 2] | ((uint32_t)h[q * 8 + 3] << 16);
            o.z = (uint32_t)h[q * 8 + 4] | ((uint32_t)h[q * 8 + 5] << 16);
            o.w = (uint32_t)h[q * 8 + 6] | ((uint32_t)h[q * 8 + 7] << 16);
            *(uint4*)(c_stage + half * kTileBytes + swz(r, q0 + q)) = o;
          }
        }
        if (want_ct) {  // transposed tile: row = column of the accumulator, column = r
          uint8_t* dst = ct_stage + (r >> 6) * kTileBytes + (r & 7) * 2;
          const int qr = (r & 63) >> 3;
#pragma unroll
          for (int j = 0; j < 32; ++j) *(uint16_t*)(dst + swz(cb * 32 + j, qr)) = h[j];
        }
        if (P.F != nullptr && row < P.M) {
          float* f = P.F + b64 * P.strideF;
          if (P.f_transposed) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (col0 + j < P.N) f[(int64_t)(col0 + j) * P.ldf + row] = bf16_bits_to_float(h[j]) * P.f_scale;
          } else {
            float* frow = f + (int64_t)row * P.ldf + col0;
            if (col0 + 32 <= P.N && (P.ldf & 3) == 0 && (((uintptr_t)f) & 15) == 0) {
#pragma unroll
              for (int q = 0; q < 8; ++q)
                *(float4*)(frow + q * 4) =
                    make_float4(bf16_bits_to_float(h[q * 4]) * P.f_scale, bf16_bits_to_float(h[q * 4 + 1]) * P.f_scale,
                                bf16_bits_to_float(h[q * 4 + 2]) * P.f_scale, bf16_bits_to_float(h[q * 4 + 3]) * P.f_scale);
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (col0 + j < P.N) frow[j] = bf16_bits_to_float(h[j]) * P.f_scale;
            }
          }
        }
      }
    }
    tc_fence_before();
    if (want_c || want_ct) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic-proxy writes -> visible to the bulk copy
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (have && warp == 2 && lane == 0) {
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          if (want_c && tn * BN + hh * BK < P.N)
            tma_store_3d(&G.c, c_stage + hh * kTileBytes, tn * BN + hh * BK, tm * BM, batch);
          if (want_ct && tm * BM + hh * BK < P.M)
            tma_store_3d(&G.ct, ct_stage + hh * kTileBytes, tm * BM + hh * BK, tn * BN, batch);
        }
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      }
    }
  }

  // ---- teardown: after an expired wait, nothing may still land in shared memory or be multiplied when they are given back
  __syncthreads();
  if (abort_flag) {
    if (warp == 0 && leader) ring_drain(full_bar, issued, kStages);
    if (warp == 1 && leader) products_drain(&drain_bar);
    __syncthreads();
    if (threadIdx.x == 0 && L.status != nullptr) atomicExch(L.status, 1);
  }
  if (warp == 1) { __syncwarp(); tc_fence_after(); tmem_dealloc(tmem_base, kTmemCols); }
}

// ------------------------------------------------------------------------------------------ pair kernel
// Same products with a 256x256 output tile per PAIR of CTAs (cta_group::2, a cluster of two on neighbouring SMs), one
// persistent pair per two SMs.  Each CTA stages 128 rows of A and half of B (32 KiB per 64 of K, 5 stages) and holds 128 rows
// of the accumulator, 256 of the 512 columns of tensor memory, so two accumulators fit and the epilogue of one tile runs
// under the main loop of the next.
//   warp 0      : TMA producer of its CTA; completion of both CTAs' loads is counted on the even CTA's barrier
//   warp 1      : of the even CTA: issues 256x256x16 instructions for the pair; commits release a ring slot in both CTAs
//   warps 2..9  : epilogue of 32 rows x 128 columns each, 64 columns at a time and independent of the other warps: tensor
//                 memory -> registers -> swizzled staging (for the polynomial the S block lands there first, by TMA, and
//                 every thread overwrites what it read) -> bulk tensor store; the transposed copy is made by ldmatrix.trans /
//                 stmatrix from that staging.  A 768-long K leaves 6100 cycles per tile to hide this in.
constexpr int kPairStages = 5;
constexpr int kPairStageBytes = 2 * kTileBytes;                       // this CTA's 128 rows of A | its half of B
constexpr int kWarpStage = 32 * 64 * 2;                               // 32 rows x 64 columns of bf16
constexpr int kPairEpiWarps = 8;
constexpr int kPairThreads = 64 + 32 * kPairEpiWarps;
constexpr int kPairSmemBytes = kPairStages * kPairStageBytes + kPairEpiWarps * 2 * kWarpStage + 1024;  // C and C^T of a warp
constexpr uint32_t kInstrDescPair = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kPairTile >> 3) << 17) | ((uint32_t)(kPairTile >> 4) << 24);
template <int kRoom>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1) ns_gemm_pair_kernel(const __grid_constant__ GemmGroups<kRoom> L) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[kPairStages];   // used in the even CTA: both CTAs' loads of a stage have landed
  __shared__ __align__(8) uint64_t empty_bar[kPairStages];  // in each CTA: the products that read the stage have finished
  __shared__ __align__(8) uint64_t acc_full[2];             // in each CTA: accumulator finished
  __shared__ __align__(8) uint64_t acc_empty[2];            // in the even CTA: all sixteen epilogue warps have read it
  __shared__ __align__(8) uint64_t s_bar[kPairEpiWarps];
  __shared__ __align__(8) uint64_t drain_bar;               // in each CTA, teardown only: all products have finished
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag, skip_flag;
  __shared__ int fills, fill_bytes[kPairStages];            // ring fills this CTA issued, bytes of the last one of each stage

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool leader = elect_one();  // issues the loads (warp 0) and the products (warp 1), and waits for them in the teardown
  const uint32_t rank = cluster_rank();
  uint8_t* ring = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int total = L.total, pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kPairStages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], 2 * kPairEpiWarps); }
    for (int w = 0; w < kPairEpiWarps; ++w) mbar_init(&s_bar[w], 1);
    mbar_init(&drain_bar, 1);
    abort_flag = 0;
    fills = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) { tmem_alloc_pair(&tmem_base_slot, 512); tmem_relinquish_pair(); }
  griddep_wait();
  // a kernel of this stream already gave up on a wait: do not pile more work on a broken pipeline (the even CTA decides)
  if (threadIdx.x == 0) skip_flag = L.status != nullptr && *(volatile const int*)L.status != 0;
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
        const TileAt t = tile_at(L, idx);
        const GemmGroup& G = L.g[t.group];
        const GemmParams P = G.P;  // by value: through the reference every use would be a load (nothing survives the asm fences)
        const bool same_ab = P.same_operand && t.tm == t.tn;
        const int num_kb = (P.K + BK - 1) / BK;
        const int a_row = t.tm * kPairTile + (int)rank * 128, b_row = t.tn * kPairTile + (int)rank * 128;
        for (int kb = 0; kb < num_kb; ++kb, ++n) {
          const int s = n % kPairStages, round = n / kPairStages;
          ok = mbar_wait(&empty_bar[s], (round & 1) ^ 1, &abort_flag);
          if (!ok) break;
          uint8_t* dst = ring + s * kPairStageBytes;
          const uint32_t bar = cluster_addr(&full_bar[s], 0);
          fill_bytes[s] = same_ab ? kTileBytes : kPairStageBytes;
          if (rank == 0) mbar_expect_tx(&full_bar[s], same_ab ? 2 * kTileBytes : 2 * kPairStageBytes);
          tma_load_3d_pair(dst, &G.a, bar, kb * BK, a_row, t.batch);
          if (P.b_mn) {
            tma_load_3d_pair(dst + kTileBytes, &G.b, bar, b_row, kb * BK, t.batch);
            tma_load_3d_pair(dst + kTileBytes + kMnBoxBytes, &G.b, bar, b_row + 64, kb * BK, t.batch);
          } else if (!same_ab) {
            tma_load_3d_pair(dst + kTileBytes, &G.b, bar, kb * BK, b_row, t.batch);
          }
        }
      }
      fills = n;
      griddep_launch();  // this CTA's last loads are on their way: the next kernel of the chain may take over SMs that drain
    }
  } else if (warp == 1) {
    if (leader && rank == 0) {
      int n = 0, it = 0;
      bool ok = true;
      for (int idx = pair; idx < total && ok; idx += pairs, ++it) {
        const TileAt t = tile_at(L, idx);
        const GemmGroup& G = L.g[t.group];
        const GemmParams P = G.P;  // by value: through the reference every use would be a load (nothing survives the asm fences)
        const bool same_ab = P.same_operand && t.tm == t.tn;
        const int num_kb = (P.K + BK - 1) / BK;
        const int acc = it & 1;
        ok = mbar_wait(&acc_empty[acc], ((it >> 1) & 1) ^ 1, &abort_flag);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d = tmem_base + (uint32_t)acc * 256u;
        const uint32_t b_step = P.b_mn ? kMnStep : 2u, idesc = kInstrDescPair | (P.b_mn ? kInstrBMn : 0u);
        for (int kb = 0; kb < num_kb; ++kb, ++n) {
          const int s = n % kPairStages, round = n / kPairStages;
          ok = mbar_wait(&full_bar[s], round & 1, &abort_flag);
          if (!ok) break;
          tc_fence_after();
          const uint32_t base = smem_u32(ring + s * kPairStageBytes);
          const uint64_t a_desc = make_smem_desc(base);
          const uint64_t b_desc = same_ab ? a_desc : (P.b_mn ? make_smem_desc_mn(base + kTileBytes, kMnBoxBytes) : make_smem_desc(base + kTileBytes));
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) tc_mma_bf16_pair(d, a_desc + 2 * k, b_desc + b_step * k, idesc, (kb | k) ? 1u : 0u);
          tc_commit_pair(&empty_bar[s]);
        }
        if (ok) tc_commit_pair(&acc_full[acc]);
      }
    }
  } else {
    const int quarter = warp & 3, half = (warp - 2) >> 2;  // tensor-memory lanes this warp may read; its half of the columns
    uint8_t* const stage = ring + kPairStages * kPairStageBytes + (warp - 2) * 2 * kWarpStage;
    uint64_t* const sb = &s_bar[warp - 2];
    const uint32_t tmem_warp = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * 128);
    int it = 0, s_block = -1;  // s_block: parity of the S load in flight, -1 without one
    bool ok = true;
    for (int idx = pair; idx < total && ok; idx += pairs, ++it) {
      const TileAt t = tile_at(L, idx);
      const GemmGroup& G = L.g[t.group];
      const GemmParams P = G.P;  // by value: through the reference every use would be a load (nothing survives the asm fences)
      const bool poly = P.mode == kModePoly, f_bulk = G.f_bulk != 0;
      const int acc = it & 1, row0 = t.tm * kPairTile + (int)rank * 128 + quarter * 32, row = row0 + lane;
      const int first = t.tn * kPairTile + half * 128;
      const bool mirror = P.symmetric ? (t.tn != t.tm) : true;
      const bool want_c = P.C != nullptr, want_ct = P.CT != nullptr && mirror;
      const bool two = P.CT == nullptr && !poly;  // without a transposed copy its buffer is a second one for C
      if (poly && lane == 0) {  // the first S block arrives while the tile is still being multiplied
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        mbar_expect_tx(sb, kWarpStage);
        tma_load_3d(stage, &G.s, sb, first, row0, t.batch);
        s_block = 0;
      }
      __syncwarp();
      ok = mbar_wait(&acc_full[acc], (it >> 1) & 1, &abort_flag);
      if (!__all_sync(0xFFFFFFFFu, ok)) { ok = false; break; }
      tc_fence_after();
#pragma unroll 1
      for (int q = 0; q < 2; ++q) {
        const int col0 = first + q * 64;
        uint8_t* c_st = stage + (two ? q * kWarpStage : 0);
        uint8_t* ct_st = stage + kWarpStage;
        uint32_t acc_r[2][32];
        tmem_ld32(tmem_warp + (uint32_t)(acc * 256 + q * 64), acc_r[0]);
        tmem_ld32(tmem_warp + (uint32_t)(acc * 256 + q * 64 + 32), acc_r[1]);
        tmem_ld_wait();
        if (q == 1) {  // last read of this accumulator
          tc_fence_before();
          __syncwarp();
          if (lane == 0) cluster_arrive(cluster_addr(&acc_empty[acc], 0));
        }
        if (poly) {
          ok = mbar_wait(sb, q, &abort_flag);  // two blocks per tile: the phase is the block
          if (!__all_sync(0xFFFFFFFFu, ok)) { ok = false; break; }
          s_block = -1;
        } else if (!f_bulk) {  // the store that read this buffer last
          if (lane == 0) {
            if (two) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
            else asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          }
          __syncwarp();
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t packed[16];  // rounded once, so that the tile, its mirrored copy and F agree bit for bit
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(acc_r[h][c * 8 + e]);
            uint4* slot = (uint4*)(c_st + swz(lane, h * 4 + c));
            if (poly) {
              const uint4 sv = *slot;
              const uint32_t w[4] = {sv.x, sv.y, sv.z, sv.w};
#pragma unroll
              for (int e = 0; e < 8; ++e) {
                const float sval = bf16_bits_to_float((uint16_t)((w[e >> 1] >> ((e & 1) * 16)) & 0xFFFF));
                v[e] = P.cc * v[e] + P.cb * sval + ((col0 + h * 32 + c * 8 + e == row) ? P.ca : 0.f);
              }
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const __nv_bfloat162 two_values = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
              packed[c * 4 + e] = *reinterpret_cast<const uint32_t*>(&two_values);
            }
            if (want_c || want_ct) *slot = make_uint4(packed[c * 4], packed[c * 4 + 1], packed[c * 4 + 2], packed[c * 4 + 3]);
          }
          if (P.F != nullptr) {
            const int fc = col0 + h * 32;
            if (f_bulk) {  // 32 x 32 fp32 block, one staging buffer per half
              if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
              __syncwarp();
              uint8_t* f_st = stage + h * kWarpStage;
#pragma unroll
              for (int c = 0; c < 8; ++c)
                *(float4*)(f_st + swz(lane, c)) =
                    make_float4(bf16_bits_to_float((uint16_t)(packed[c * 2] & 0xFFFF)) * P.f_scale, bf16_bits_to_float((uint16_t)(packed[c * 2] >> 16)) * P.f_scale,
                                bf16_bits_to_float((uint16_t)(packed[c * 2 + 1] & 0xFFFF)) * P.f_scale, bf16_bits_to_float((uint16_t)(packed[c * 2 + 1] >> 16)) * P.f_scale);
              asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
              __syncwarp();
              if (lane == 0) {
                if (fc < P.N && row0 < P.M) tma_store_3d(&G.c, f_st, fc, row0, t.batch);
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
              }
            } else if (row < P.M) {
              float* f = P.F + (int64_t)t.batch * P.strideF;
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                const float y = bf16_bits_to_float((uint16_t)((packed[j >> 1] >> ((j & 1) * 16)) & 0xFFFF)) * P.f_scale;
                if (fc + j < P.N) f[P.f_transposed ? (int64_t)(fc + j) * P.ldf + row : (int64_t)row * P.ldf + fc + j] = y;
              }
            }
          }
        }
        if (want_c || want_ct) {
          __syncwarp();
          if (want_ct) {  // 8 columns at a time: four 8x8 blocks of the staged tile, transposed on the way to the registers
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              uint32_t blk[4];
              ldmatrix_x4_trans(smem_u32(c_st + swz(lane, c)), blk);
              const int ct_row = c * 8 + (lane & 7), chunk = lane >> 3;
              stmatrix_x4(smem_u32(ct_st + ct_row * 64 + ((chunk ^ ((ct_row >> 1) & 3)) << 4)), blk);
            }
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) {
            if (col0 < P.N && row0 < P.M) {
              if (want_c) tma_store_3d(&G.c, c_st, col0, row0, t.batch);
              if (want_ct) tma_store_3d(&G.ct, ct_st, row0, col0, t.batch);
            }
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        }
        if (poly && q == 0 && lane == 0) {
          asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          mbar_expect_tx(sb, kWarpStage);
          tma_load_3d(c_st, &G.s, sb, col0 + 64, row0, t.batch);
          s_block = 1;
        }
      }
    }
    if (lane == 0) {
      if (s_block >= 0) mbar_drain(sb, s_block);
      asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    }
    tc_fence_before();
  }

  // After an expired wait in either CTA, both wait (with a limit) for every product and every load that the pair issued before its
  // shared and tensor memory go away; the blocks of S and the stores were waited for above.
  __syncthreads();
  if (threadIdx.x == 0 && abort_flag) cluster_store(cluster_addr(&abort_flag, rank ^ 1), 1);
  cluster_sync();
  if (abort_flag) {
    if (rank == 0 && warp == 1 && leader) tc_commit_pair(&drain_bar);  // the thread that issued the products
    if (threadIdx.x == 0) mbar_drain(&drain_bar, 0);
    if (rank == 0 && threadIdx.x == 0) {
      const int even = fills, odd = cluster_load(cluster_addr(&fills, 1)), top = max(even, odd);
      for (int n = pair_drain_first(even, odd, kPairStages); n < top; ++n) {
        const int s = n % kPairStages, kind = pair_fill_kind(n, even, odd);
        if (kind == kFillOddOnly) mbar_expect_tx(&full_bar[s], (uint32_t)cluster_load(cluster_addr(&fill_bytes[s], 1)));
        if (kind == kFillEvenOnly) mbar_complete_tx(&full_bar[s], (uint32_t)fill_bytes[s]);
        mbar_drain(&full_bar[s], (n / kPairStages) & 1);
      }
    }
    cluster_sync();
  }
  if (threadIdx.x == 0 && abort_flag && L.status != nullptr) atomicExch(L.status, 1);
  if (warp == 1) { __syncwarp(); tc_fence_after(); tmem_dealloc_pair(tmem_base, 512); }
}

// ------------------------------------------------------------------------------------------ prologue
// X = SR_bf16(G / max(||G||_F, eps)), written in the source orientation (`trans` == 0) or transposed, whichever makes the
// Gram matrix the small one.  `sumsq[b]` holds ||G_b||_F^2.
// One block handles a 64 x 64 tile: 256 threads as 16 column-groups (4 columns each) x 16 rows, four row
// passes.  Loads are 16 B (fp32) / 8 B (bf16), stores 8 bytes; the transpose goes through shared memory.
// All matrices of a step share the launch: block b belongs to the matrix whose tile range holds it.
__global__ void __launch_bounds__(256) ns_prepare_kernel(const NsSource* __restrict__ mats, const int* __restrict__ first, int n_mats,
                                                        int src_dt, float eps) {
  __shared__ uint16_t tile[64][66];
  const int at = find_range(first, n_mats, blockIdx.x);
  const NsSource S = mats[at];
  const int R = S.rows, C = S.cols, b = S.index, trans = S.trans, tiles_c = (C + 63) >> 6;
  const int local = blockIdx.x - first[at], by = local / tiles_c, bx = local - by * tiles_c;
  const void* src = S.src;
  const int64_t ld = S.ld;
  const float inv = 1.0f / fmaxf(sqrtf(*S.sumsq), eps);
  const Philox rng(S.seed);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int c0 = bx * 64 + tx * 4;
  const bool vec = (C & 3) == 0 && (((uintptr_t)src) & 15) == 0;
  uint16_t* dst_b = (uint16_t*)S.dst;
  float x[4][4];
#pragma unroll
  for (int pass = 0; pass < 4; ++pass) {  // every load of the tile is in flight before the first value is used
    const int r = by * 64 + ty + 16 * pass;
#pragma unroll
    for (int k = 0; k < 4; ++k) x[pass][k] = 0.f;
    if (r < R && c0 < C) {
      const int64_t idx = (int64_t)r * C + c0;
      if (vec) {
        if (src_dt == kF32) {
          const float4 t = *(const float4*)((const float*)src + idx);
          x[pass][0] = t.x; x[pass][1] = t.y; x[pass][2] = t.z; x[pass][3] = t.w;
        } else {
          const uint2 t = *(const uint2*)((const uint16_t*)src + idx);
          x[pass][0] = bf16_bits_to_float(t.x & 0xFFFF); x[pass][1] = bf16_bits_to_float(t.x >> 16);
          x[pass][2] = bf16_bits_to_float(t.y & 0xFFFF); x[pass][3] = bf16_bits_to_float(t.y >> 16);
        }
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (c0 + k < C)
            x[pass][k] = src_dt == kF32 ? ((const float*)src)[idx + k] : bf16_bits_to_float(((const uint16_t*)src)[idx + k]);
      }
    }
  }
  uint4 rnd = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
  for (int pass = 0; pass < 4; ++pass) {
    const int rl = ty + 16 * pass, r = by * 64 + rl;
    uint16_t h[4] = {0, 0, 0, 0};
    if (r < R && c0 < C) {
      const int64_t idx = (int64_t)r * C + c0;
      // rounding to bf16 takes 16 random bits: a draw serves two row passes (low halves, then high halves)
      if ((pass & 1) == 0) rnd = rng((uint32_t)idx, (uint32_t)(idx >> 32), (uint32_t)b, 7u);
      const uint32_t rr[4] = {rnd.x >> (pass & 1) * 16, rnd.y >> (pass & 1) * 16, rnd.z >> (pass & 1) * 16, rnd.w >> (pass & 1) * 16};
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (c0 + k < C) h[k] = sr_bf16_bits(x[pass][k] * inv, rr[k]);
      if (!trans) {
        uint2 o;
        o.x = (uint32_t)h[0] | ((uint32_t)h[1] << 16);
        o.y = (uint32_t)h[2] | ((uint32_t)h[3] << 16);
        *(uint2*)(dst_b + (int64_t)r * ld + c0) = o;  // columns past C land in the row padding (ld is a multiple of 8)
      }
    }
    if (trans) {
#pragma unroll
      for (int k = 0; k < 4; ++k) tile[rl][tx * 4 + k] = h[k];
    }
  }
  if (!trans) return;
  __syncthreads();
  // transposed output: this thread owns source rows r0..r0+3 (consecutive in the output row) of four source columns
  const int r0 = by * 64 + tx * 4;
#pragma unroll
  for (int pass = 0; pass < 4; ++pass) {
    const int cl = ty + 16 * pass, c = bx * 64 + cl;
    if (c < C && r0 < R) {
      uint2 o;
      o.x = (uint32_t)tile[tx * 4 + 0][cl] | ((uint32_t)tile[tx * 4 + 1][cl] << 16);
      o.y = (uint32_t)tile[tx * 4 + 2][cl] | ((uint32_t)tile[tx * 4 + 3][cl] << 16);
      *(uint2*)(dst_b + (int64_t)c * ld + r0) = o;
    }
  }
}

// ------------------------------------------------------------------------------------------ host side
// Tensor [batch, rows, cols] with leading dimension `ld` elements (bf16, or fp32 when `f32`); box = box_cols x box_rows,
// swizzled over the width of a box row (128 or 64 bytes).
static bool encode_map(CUtensorMap* map, const void* base, int rows, int cols, int64_t ld, int64_t batch_stride, int batch,
                       int box_cols, int box_rows, bool f32) {
  EncodeTiledFn fn = tensor_map_encoder();
  if (fn == nullptr) return false;
  const int elem = f32 ? 4 : 2;
  cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)batch};
  cuuint64_t strides[2] = {(cuuint64_t)ld * elem, (cuuint64_t)batch_stride * elem};
  cuuint32_t box[3] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return fn(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims,
            strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            box_cols * elem == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A step launches the same ~60 products over the same workspace addresses (the caching allocator hands the buffers
// back), and every launch needs up to five descriptors: they are kept by their defining values instead of being
// encoded again (about 0.6 us each on the host, which is what limits a step once the matrices are split over ranks).
static bool make_map(CUtensorMap* map, const void* base, int rows, int cols, int64_t ld, int64_t batch_stride, int batch,
                     int box_cols = BK, int box_rows = BM, bool f32 = false) {
  struct Key {
    const void* base; int64_t ld, stride; int rows, cols, batch, box;
    bool operator==(const Key& o) const {
      return base == o.base && ld == o.ld && stride == o.stride && rows == o.rows && cols == o.cols && batch == o.batch && box == o.box;
    }
  };
  struct Hash {
    size_t operator()(const Key& k) const {
      size_t h = std::hash<const void*>()(k.base);
      for (int64_t v : {k.ld, k.stride, (int64_t)k.rows, (int64_t)k.cols, (int64_t)k.batch, (int64_t)k.box})
        h ^= std::hash<int64_t>()(v) + 0x9e3779b97f4a7c15ull + (h << 6) + (h >> 2);
      return h;
    }
  };
  static std::unordered_map<Key, CUtensorMap, Hash> cache;
  static std::mutex guard;
  const Key key{base, ld, batch_stride, rows, cols, batch, (box_cols << 16) | (box_rows << 1) | (f32 ? 1 : 0)};
  std::lock_guard<std::mutex> lock(guard);
  auto it = cache.find(key);
  if (it != cache.end()) {
    *map = it->second;
    return true;
  }
  if (!encode_map(map, base, rows, cols, ld, batch_stride, batch, box_cols, box_rows, f32)) return false;
  if (cache.size() >= 4096) cache.clear();
  cache.emplace(key, *map);
  return true;
}

static int g_tile_override = 0;
int ns_gemm_tile_override() { return g_tile_override; }
void set_ns_gemm_tile_override(int tile) { g_tile_override = tile; }

// Pairs of CTAs that the current device holds at once, after allowing both kernels their shared memory there.
static cudaError_t resident_pairs(int* out) {
  static PerDevice<int> pairs;
  int device = 0;
  const cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  return pairs.get(device, cudaSuccess, out, [](int& found) {
    cudaError_t s = cudaSuccess;
    for (const void* kernel : {(const void*)ns_gemm_kernel<kFewGroups>, (const void*)ns_gemm_kernel<kMaxGroups>})
      if (s == cudaSuccess) s = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    for (const void* kernel : {(const void*)ns_gemm_pair_kernel<kFewGroups>, (const void*)ns_gemm_pair_kernel<kMaxGroups>})
      if (s == cudaSuccess) s = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmemBytes);
    return s != cudaSuccess ? s : max_resident_pairs(ns_gemm_pair_kernel<kMaxGroups>, kPairThreads, kPairSmemBytes, &found);
  });
}

// One launch of the pair kernel (`pair`) or of the 128 x 128 kernel over up to kMaxGroups products.
struct NsLaunch {
  GemmGroups<kMaxGroups> L;
  bool pair;
  int blocks;
};
struct NsLaunches {
  std::vector<NsLaunch> all;
};

static cudaError_t prepare_group(const NsProduct* const* products, int n, bool pair, int max_pairs, NsLaunch& out) {
  GemmGroups<kMaxGroups>& L = out.L;
  out.pair = pair;
  L.n = n;
  L.total = 0;
  L.status = products[0]->P.status;
  for (int i = 0; i < n; ++i) {
    const NsProduct& X = *products[i];
    GemmGroup& G = L.g[i];
    GemmParams& P = G.P;
    P = X.P;
    P.same_operand = (!P.b_mn && X.A == X.B && X.lda == X.ldb && X.strideA == X.strideB && P.M == P.N) ? 1 : 0;
    const int tile = pair ? kPairTile : BM;
    G.tiles_m = (P.M + tile - 1) / tile;
    G.tiles_n = (P.N + tile - 1) / tile;
    G.per_batch = P.symmetric ? G.tiles_m * (G.tiles_m + 1) / 2 : G.tiles_m * G.tiles_n;
    L.first[i] = L.total;
    L.total += G.per_batch * P.batch;
    // fp32 results leave through bulk stores when rows start on 16-byte boundaries and no bf16 copy needs the staging
    G.f_bulk = pair && P.F != nullptr && !P.f_transposed && P.C == nullptr && P.CT == nullptr && (P.ldf & 3) == 0 &&
               (P.strideF & 3) == 0 && (((uintptr_t)P.F) & 15) == 0;
    bool ok = make_map(&G.a, X.A, P.M, P.K, X.lda, X.strideA, P.batch);
    ok = ok && (P.b_mn ? make_map(&G.b, X.B, P.K, P.N, X.ldb, X.strideB, P.batch, BK, BK)
                       : make_map(&G.b, X.B, P.N, P.K, X.ldb, X.strideB, P.batch));
    G.c = G.ct = G.s = G.a;  // placeholders where an operand is absent (never dereferenced by the kernels then)
    if (P.C != nullptr) ok = ok && make_map(&G.c, P.C, P.M, P.N, P.ldc, P.strideC, P.batch, 64, pair ? 32 : BM);
    if (G.f_bulk) ok = ok && make_map(&G.c, P.F, P.M, P.N, P.ldf, P.strideF, P.batch, 32, 32, true);
    if (P.CT != nullptr) ok = ok && make_map(&G.ct, P.CT, P.N, P.M, P.ldct, P.strideCT, P.batch, pair ? 32 : 64, pair ? 64 : BM);
    if (pair && P.mode == kModePoly) ok = ok && make_map(&G.s, P.S, P.M, P.N, P.lds, P.strideS, P.batch, 64, 32);
    if (!ok) return cudaErrorInvalidValue;
  }
  out.blocks = pair ? 2 * std::min(L.total, max_pairs) : L.total;
  return cudaSuccess;
}

cudaError_t prepare_ns_products(const NsProduct* products, int n, NsPlan* plan) {
  int max_pairs = 0;
  const cudaError_t found = resident_pairs(&max_pairs);
  if (found != cudaSuccess) return found;
  std::vector<NsExtent> extents;
  extents.reserve(n);
  for (int i = 0; i < n; ++i)
    extents.push_back({products[i].P.M, products[i].P.N, products[i].P.K, products[i].P.batch, products[i].P.symmetric != 0});
  const int force = ns_gemm_tile_override();
  const bool pairs = force == 0 && ns_take_pairs(extents.data(), n, max_pairs);
  std::vector<const NsProduct*> side[2];
  for (int i = 0; i < n; ++i) side[force == 256 || (pairs && ns_pair_sized(extents[i])) ? 1 : 0].push_back(&products[i]);
  plan->launches = std::make_shared<NsLaunches>();
  plan->launches->all.reserve(side[0].size() / kMaxGroups + side[1].size() / kMaxGroups + 2);
  for (int pair = 1; pair >= 0; --pair) {
    auto& list = side[pair];
    // tiles are dealt out in order: the ones with the longest main loop first
    std::stable_sort(list.begin(), list.end(), [](const NsProduct* a, const NsProduct* b) { return a->P.K > b->P.K; });
    for (size_t i = 0; i < list.size(); i += kMaxGroups) {
      plan->launches->all.emplace_back();
      const cudaError_t e =
          prepare_group(list.data() + i, (int)std::min<size_t>(kMaxGroups, list.size() - i), pair != 0, max_pairs, plan->launches->all.back());
      if (e != cudaSuccess) return e;
    }
  }
  return cudaSuccess;
}

void set_ns_coefficients(const NsPlan& plan, float ca, float cb, float cc) {
  for (NsLaunch& launch : plan.launches->all)
    for (int i = 0; i < launch.L.n; ++i) {
      launch.L.g[i].P.ca = ca;
      launch.L.g[i].P.cb = cb;
      launch.L.g[i].P.cc = cc;
    }
}

template <int kRoom>
static cudaError_t launch_groups(const NsLaunch& launch, const GemmGroups<kRoom>& L, cudaStream_t stream) {
  void* args[] = {const_cast<GemmGroups<kRoom>*>(&L)};
  return launch.pair ? launch_chained_with((const void*)ns_gemm_pair_kernel<kRoom>, dim3(launch.blocks), kPairThreads, kPairSmemBytes, stream, args)
                     : launch_chained_with((const void*)ns_gemm_kernel<kRoom>, dim3(launch.blocks), kGemmThreads, kSmemBytes, stream, args);
}

cudaError_t launch_ns_plan(const NsPlan& plan, int* launches, cudaStream_t stream) {
  for (const NsLaunch& launch : plan.launches->all) {
    if (launch.L.total > 0) {
      cudaError_t e;
      if (launch.L.n <= kFewGroups) {
        GemmGroups<kFewGroups> few;
        few.n = launch.L.n;
        few.total = launch.L.total;
        few.status = launch.L.status;
        std::copy_n(launch.L.first, launch.L.n, few.first);
        std::copy_n(launch.L.g, launch.L.n, few.g);
        e = launch_groups(launch, few, stream);
      } else {
        e = launch_groups(launch, launch.L, stream);
      }
      if (e != cudaSuccess) return e;
    }
    if (launches != nullptr) ++*launches;
  }
  return cudaSuccess;
}

cudaError_t launch_ns_products(const NsProduct* products, int n, int* launches, cudaStream_t stream) {
  NsPlan plan;
  const cudaError_t e = prepare_ns_products(products, n, &plan);
  return e != cudaSuccess ? e : launch_ns_plan(plan, launches, stream);
}

cudaError_t launch_ns_prepare(const NsSource* mats, const int* first, int n_mats, int total_tiles, int src_dt, float eps,
                              cudaStream_t stream) {
  if (total_tiles == 0) return cudaSuccess;
  ns_prepare_kernel<<<total_tiles, 256, 0, stream>>>(mats, first, n_mats, src_dt, eps);
  return cudaGetLastError();
}

}  // namespace hb
