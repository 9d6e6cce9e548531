// Multi-tensor fused optimizer chain: one launch executes, for every element of every tensor of a
// param group,  [ECC/bf16/fp32 decode] -> [MARS] -> [momentum / second-moment rule] -> [caution] ->
// [weight decay] -> [parameter write | update write] -> [stochastic-rounding / ECC encode].
//
// Replaces the per-tensor compiled regions of the reference (heavyball/utils.py:1842-2334 Adam family,
// 736-776 momentum, 3616-3627 MARS, 2373-2406 parameter update, 3652-3658 caution).  Arithmetic is
// restated from heavyball_b200/utils/first_order.py, which is also the test oracle.
//
// Work decomposition: tensors are cut into chunks (chain_chunks.h); block b owns chunk b, and its warps find the tensor in a
// table of prefix sums, 32 entries at a time (find_range).  All tensor addresses come from a table (in device memory, or in the
// launch's arguments where tensors and elements are few), so the launch count is independent of the number of tensors.
//
// Two kernels: the general one below takes every storage kind, rule and destination from run-time parameters; the specialised
// instances after it (Kinds) cover the launches that most steps consist of.
#include "chain_chunks.h"
#include "common.cuh"
#include "fused_chain.h"

#include <algorithm>
#include <type_traits>

namespace hb {

constexpr int kThreads = 256;

// Random bits are only generated for storage kinds that consume them (bf16 rounding, ECC residuals).
__device__ inline uint4 draw(int dt, const Philox& rng, uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3) {
  if (dt == kF32 || dt == kF16 || dt == kNone) return make_uint4(0u, 0u, 0u, 0u);
  return rng(c0, c1, c2, c3);
}

__device__ inline float lerp_to(float s, float x, float beta) {  // s*beta' + x*(1-beta') in the oracle's order
  float w = 1.0f - beta;
  return s * (1.0f - w) + x * w;
}

__device__ __forceinline__ float trust_region(float u) {
  const float x = u * (1.0f / 1.5f);
  const float t = tanhf(x);
  const float y = copysignf(log1pf(fabsf(x)), t) * 0.1f + t * 0.9f;
  return fminf(fmaxf(y * 1.5f, -2.0f), 2.0f);
}

// Block sums of a launch -> one atomic per block and tensor.
template <bool kCountCaution>
__device__ __forceinline__ void finish_block(const ChainParams& P, const TensorMeta& M, float sumsq_local, float nonzero_local,
                                             int masked_local) {
  if (P.accum_sumsq && M.scale != nullptr) {  // per-tensor squared norm of the update just written (feeds Newton–Schulz)
    __shared__ float warp_sq[kThreads / 32];
    float v = sumsq_local;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, o);
    if ((threadIdx.x & 31) == 0) warp_sq[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
      float tot = 0.f;
      for (int w = 0; w < kThreads / 32; ++w) tot += warp_sq[w];
      atomicAdd(M.scale, tot);
    }
    if (P.accum_sumsq == 2) {  // block counts are exact integers (<= 8192); their sum stays exact up to 2^24 elements
      __syncthreads();
      float c = nonzero_local;
      for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xFFFFFFFFu, c, o);
      if ((threadIdx.x & 31) == 0) warp_sq[threadIdx.x >> 5] = c;
      __syncthreads();
      if (threadIdx.x == 0) {
        float tot = 0.f;
        for (int w = 0; w < kThreads / 32; ++w) tot += warp_sq[w];
        atomicAdd(M.scale + 1, tot);
      }
    }
  }
  if (kCountCaution) {
    __shared__ int warp_sums[kThreads / 32];
    int v = masked_local;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, o);
    if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
      int tot = 0;
      for (int w = 0; w < kThreads / 32; ++w) tot += warp_sums[w];
      if (tot) atomicAdd(M.masked, tot);
    }
  }
}

template <bool kCountCaution>
__global__ void __launch_bounds__(kThreads, 4) fused_chain_kernel(const TensorMeta* __restrict__ metas,
                                                              const int* __restrict__ chunk_prefix, ChainParams P) {
  // ---- locate (tensor, chunk)
  const int b = blockIdx.x, t = find_range(chunk_prefix, P.n_tensors, b);
  const TensorMeta M = metas[t];
  const int64_t base = (int64_t)(b - chunk_prefix[t]) * kChunk;
  const bool vec_ok = M.vec_ok != 0;
  const Philox rng(P.seed);

  float cscale = 1.0f;
  if (P.use_tensor_scale && M.scale != nullptr) cscale = *M.scale;
  if (P.caution_apply && M.masked != nullptr) {
    float n = (float)M.numel;
    cscale *= n / fmaxf(n - (float)(*M.masked), 1.0f);
  }
  float gclip = 1.0f, ortho_c = 0.f;
  const bool ortho = P.g_clip_mode == kClipOrtho && M.gsq != nullptr;
  if (ortho) {
    const float px = M.gsq[0], pp = M.gsq[1], xx = M.gsq[2];
    ortho_c = px / (pp + P.g_clip_at);
    if (P.g_clip_numel != 0.f) {
      const float proj_sq = fmaxf(xx - 2.f * ortho_c * px + ortho_c * ortho_c * pp, 0.f);
      gclip = sqrtf(fmaxf(xx, 0.f)) / fmaxf(sqrtf(proj_sq), 1e-6f);
    }
  } else if (P.g_clip_mode != kClipNone && M.gsq != nullptr) {
    float sq = *M.gsq;
    if (P.g_clip_mode == kClipRms) sq /= (P.g_clip_numel > 0.f ? P.g_clip_numel : (float)M.numel);
    gclip = P.g_clip_at / fmaxf(sqrtf(sq), fmaxf(P.g_clip_at, 1e-8f));
  }
  float ugraft = 1.0f;
  if (P.u_op == kUopSignGraft && M.scale != nullptr) ugraft = sqrtf(fmaxf(M.scale[0], 0.f)) / fmaxf(sqrtf(M.scale[1]), 1e-6f);
  int masked_local = 0;
  float sumsq_local = 0.f, nonzero_local = 0.f;

#pragma unroll 2
  for (int it = 0; it < kChunk / (kThreads * 4); ++it) {
    const int64_t i = base + ((int64_t)it * kThreads + threadIdx.x) * 4;
    if (i >= M.numel) break;
    const int nv = (int)min((int64_t)4, M.numel - i);
    const uint32_t ctr = (uint32_t)(i >> 2), ctr_hi = (uint32_t)(i >> 34);

    // local state first, then the gradient: with peers the gradient loads are NVLink round trips (about 2 us each),
    // and everything issued before the first use of one of them overlaps with it
    F4 s0 = load4(M.s0, M.s0e, P.dt_s, i, nv, vec_ok);
    F4 s1 = load4(M.s1, M.s1e, P.dt_s, i, nv, vec_ok);
    F4 s2 = load4(M.s2, M.s2e, P.dt_s, i, nv, vec_ok);
    F4 g;
    if (P.n_src > 0 && P.g_mc_delta != 0 && vec_ok && nv == 4 && (P.dt_g == kF32 || P.dt_g == kBF16 || P.dt_g == kF16)) {
      // one load, summed over all ranks inside the NVSwitch
      g = mc_ld_reduce4((const char*)M.g + P.g_mc_delta, P.dt_g, i);
#pragma unroll
      for (int k = 0; k < 4; ++k) g.v[k] *= P.g_scale;
    } else if (P.n_src > 0) {  // reduce the same element over every rank's gradient slab (peer loads over NVLink)
#pragma unroll
      for (int k = 0; k < 4; ++k) g.v[k] = 0.f;
      for (int r0 = 0; r0 < P.n_src; r0 += 4) {  // four sources in flight at a time, summed in rank order
        F4 part[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (r0 + j < P.n_src) part[j] = load4((const char*)M.g + P.g_delta[r0 + j], nullptr, P.dt_g, i, nv, vec_ok);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (r0 + j < P.n_src) {
#pragma unroll
            for (int k = 0; k < 4; ++k) g.v[k] += part[j].v[k];
          }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) g.v[k] *= P.g_scale;
    } else {
      g = load4(M.g, nullptr, P.dt_g, i, nv, vec_ok);
    }
    F4 u = P.u_is_input ? load4(M.u, nullptr, P.dt_u, i, nv, vec_ok) : g;
    if (P.u_is_input && P.u_op == kUopTrustRegion) {
#pragma unroll
      for (int k = 0; k < 4; ++k) u.v[k] = trust_region(u.v[k]);
    }
    if (P.u_is_input && (P.u_op == kUopSignGraft || P.u_op == kUopSign)) {
#pragma unroll
      for (int k = 0; k < 4; ++k) u.v[k] = u.v[k] > 0.f ? ugraft : (u.v[k] < 0.f ? -ugraft : 0.f);
    }
    F4 p = (P.out_mode == kOutParam || ortho || P.post_state == kPostDecayIn) ? load4(M.p, M.pe, P.dt_p, i, nv, vec_ok) : F4{};
    F4 out;

    if (ortho) {  // remove the component along the parameter (and keep the norm): caution still sees the raw gradient
#pragma unroll
      for (int k = 0; k < 4; ++k) u.v[k] = (u.v[k] - ortho_c * p.v[k]) * gclip;
    } else if (P.g_clip_mode != kClipNone && !P.u_is_input) {  // the clip acts on the update, caution still sees the raw gradient
#pragma unroll
      for (int k = 0; k < 4; ++k) u.v[k] *= gclip;
    }
    if (P.mars) {  // g <- lerp(g, g_prev, a); g_prev <- raw g
      F4 old = load4(M.mars, M.marse, P.dt_s, i, nv, vec_ok);
      F4 raw = u;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        u.v[k] = u.v[k] * (1.0f - P.mars_a) + old.v[k] * P.mars_a;
        g.v[k] = u.v[k];
      }
      store4(M.mars, M.marse, P.dt_s, i, nv, vec_ok, raw, draw(P.dt_s, rng, ctr, ctr_hi ^ 0x40000000u, (uint32_t)t, 4u));
    }

#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float x = u.v[k], r;
      switch (P.algo) {
        case kAdam: {
          s0.v[k] = lerp_to(s0.v[k], x, P.b1);
          s1.v[k] = lerp_to(s1.v[k], x * x, P.b2);
          r = s0.v[k] / fmaxf(sqrtf(s1.v[k]), P.eps);
        } break;
        case kLaProp: {
          s1.v[k] = lerp_to(s1.v[k], x * x, P.b2);
          s0.v[k] = lerp_to(s0.v[k], x / fmaxf(sqrtf(s1.v[k]), P.eps), P.b1);
          r = s0.v[k];
        } break;
        case kAdopt: {
          s0.v[k] = lerp_to(s0.v[k], x / fmaxf(sqrtf(s1.v[k]), P.eps), P.b1);
          r = s0.v[k];
          s1.v[k] = s1.v[k] * (1.0f - P.b3) + x * x * P.b3;  // b3 = 1 - debiased beta2 of the next step
        } break;
        case kAdemamix: {
          s0.v[k] = lerp_to(s0.v[k], x, P.b1);
          s2.v[k] = lerp_to(s2.v[k], x, P.b3);
          s1.v[k] = lerp_to(s1.v[k], x * x, P.b2);
          r = (s0.v[k] + s2.v[k] * P.alpha) / fmaxf(sqrtf(s1.v[k]), P.eps);
        } break;
        case kRmsprop: {
          s1.v[k] = lerp_to(s1.v[k], x * x, P.b2);
          r = x / fmaxf(sqrtf(s1.v[k]), P.eps);
        } break;
        case kUnscaledAdam: {
          s1.v[k] = lerp_to(s1.v[k], x * x, P.b2);
          float d = fmaxf(sqrtf(s1.v[k]), P.eps);
          s0.v[k] = lerp_to(s0.v[k], x / d, P.b1);
          r = s0.v[k] * d;
        } break;
        case kExpAvg: {
          s0.v[k] = lerp_to(s0.v[k], x, P.b1);
          r = s0.v[k];
        } break;
        case kNesterovEma: {
          s0.v[k] = lerp_to(s0.v[k], x, P.b1);
          r = x + s0.v[k];
        } break;
        case kHeavyball: {
          s0.v[k] = s0.v[k] * P.b1 + x;
          r = s0.v[k];
        } break;
        case kNesterovMom: {
          s0.v[k] = s0.v[k] * P.b1 + x;
          r = x + s0.v[k] * P.b1;
        } break;
        case kNadam: {  // b3 = (1 - mu) / (1 - mu_product), alpha = mu_next / (1 - mu_product mu_next), set on the host
          s0.v[k] = lerp_to(s0.v[k], x, P.b1);
          s1.v[k] = lerp_to(s1.v[k], x * x, P.b2);
          float d = fmaxf(sqrtf(s1.v[k]), P.eps);
          r = x / d * P.b3 + s0.v[k] / d * P.alpha;
        } break;
        default:
          r = x;
      }
      out.v[k] = r;
    }

    if (P.post_state == kPostMsam) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float m = lerp_to(s0.v[k], out.v[k], P.b3);
        float d = P.wd;
        if (P.cautious_wd && ((__float_as_uint(s2.v[k]) ^ __float_as_uint(m)) >> 31)) d = 0.f;
        s0.v[k] = m;
        s2.v[k] = s2.v[k] * (1.0f - d * P.lr) + m * -P.lr;
        out.v[k] = m;
      }
    } else if (P.post_state == kPostDecayIn) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float d = P.wd;
        if (P.cautious_wd && ((__float_as_uint(p.v[k]) ^ __float_as_uint(out.v[k])) >> 31)) d = 0.f;
        out.v[k] += p.v[k] * d;
      }
    }

    // plain bf16 rounding consumes 16 random bits per element: the first two state tensors share one draw
    // (low / high halves); ECC residuals need 32 bits and keep a draw each
    const uint4 r0 = (P.n_state >= 1) ? draw(P.dt_s, rng, ctr, ctr_hi, (uint32_t)t, 0u) : make_uint4(0u, 0u, 0u, 0u);
    if (P.n_state >= 1) store4(M.s0, M.s0e, P.dt_s, i, nv, vec_ok, s0, r0);
    if (P.n_state >= 2)
      store4(M.s1, M.s1e, P.dt_s, i, nv, vec_ok, s1,
             P.dt_s == kBF16 ? make_uint4(r0.x >> 16, r0.y >> 16, r0.z >> 16, r0.w >> 16)
                             : draw(P.dt_s, rng, ctr, ctr_hi, (uint32_t)t, 1u));
    if (P.n_state >= 3) store4(M.s2, M.s2e, P.dt_s, i, nv, vec_ok, s2, draw(P.dt_s, rng, ctr, ctr_hi, (uint32_t)t, 2u));
    if (P.out_mode == kOutScheduleFree) {  // z lives in slot s2 (loaded above), p and z are both written
      F4 pp = load4(M.p, M.pe, P.dt_p, i, nv, vec_ok);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float uu = out.v[k];
        if (P.wd != 0.f) {
          float d = P.wd;
          if (P.cautious_wd && ((__float_as_uint(pp.v[k]) ^ __float_as_uint(uu)) >> 31)) d = 0.f;
          uu += pp.v[k] * d;
        }
        pp.v[k] = pp.v[k] + (s2.v[k] - pp.v[k]) * P.b3 + uu * (P.lr * (P.alpha * (1.0f - P.b3)) - P.lr);
        s2.v[k] = s2.v[k] + uu * -P.lr;
      }
      store4(M.s2, M.s2e, P.dt_s, i, nv, vec_ok, s2, draw(P.dt_s, rng, ctr, ctr_hi, (uint32_t)t, 2u));
      store4(M.p, M.pe, P.dt_p, i, nv, vec_ok, pp, draw(P.dt_p, rng, ctr, ctr_hi, (uint32_t)t, 3u));
      continue;
    }

    if (kCountCaution) {  // phase one of caution: mask, count, park the masked update
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        bool disagree = (__float_as_uint(g.v[k]) ^ __float_as_uint(out.v[k])) >> 31;
        if (k < nv && disagree) { out.v[k] = 0.f; ++masked_local; }
      }
      store4(M.u, nullptr, P.dt_u, i, nv, vec_ok, out, draw(P.dt_u, rng, ctr, ctr_hi, (uint32_t)t, 5u));
      continue;
    }
    if (P.out_mode == kOutUpdate) {
      store4(M.u, nullptr, P.dt_u, i, nv, vec_ok, out, draw(P.dt_u, rng, ctr, ctr_hi, (uint32_t)t, 5u));
      if (P.accum_sumsq) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (k < nv) {
            sumsq_local += out.v[k] * out.v[k];
            nonzero_local += out.v[k] != 0.f ? 1.f : 0.f;
          }
      }
      continue;
    }
    // parameter epilogue: p <- p (1 - d lr) - lr u
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float uu = out.v[k] * cscale;
      float d = P.wd;
      if (P.cautious_wd && ((__float_as_uint(p.v[k]) ^ __float_as_uint(uu)) >> 31)) d = 0.f;
      p.v[k] = p.v[k] * (1.0f - d * P.lr) + uu * -P.lr;
    }
    const uint4 prnd = draw(P.dt_p, rng, ctr, ctr_hi, (uint32_t)t, 3u);
    if (P.n_dst > 0 && P.p_mc_delta != 0 && vec_ok && nv == 4) {  // one store, replicated to every rank by the NVSwitch
      mc_store4((char*)M.p + P.p_mc_delta, M.pe, P.dt_p, i, p, prnd);
    } else if (P.n_dst > 0) {  // single writer per element: every replica receives bit-identical parameters
      for (int r = 0; r < P.n_dst; ++r)  // the residual of an error-corrected parameter stays with this rank (its only reader)
        store4((char*)M.p + P.p_delta[r], P.p_delta[r] == 0 ? M.pe : nullptr, P.dt_p, i, nv, vec_ok, p, prnd);
    } else {
      store4(M.p, M.pe, P.dt_p, i, nv, vec_ok, p, prnd);
    }
  }

  finish_block<kCountCaution>(P, M, sumsq_local, nonzero_local, masked_local);
}

// ---------------------------------------------------------------------------------------------
// Specialised instances for the launches without peers, gradient clips, sign updates, post-state, schedule-free output and
// third state, which are the bulk of every step: storage kinds, destination and source of the update are compile-time
// constants, and a kind's batch of vectors per thread is loaded before anything is computed or stored (stores may alias later loads,
// so the compiler cannot move those up by itself: a vector at a time is a memory round trip each).  Against the general kernel:
// AdamW on the 39.5 M fp32 parameters of GPT-2-small's embeddings 242 -> 170 us (6.5 TB/s), cautious AdamW with error-corrected
// state on 8 x 2048^2 965 -> 562 us, 353 us with the loads separated from the codec, and 290 us with
// the rule compiled in (ChainKind).
// Storage kinds outside the list below (fp16, 16-bit residuals, plain bf16 state, bf16 gradients into an update with fp32 state or
// without state), peers, clips and the other launches named here run the general kernel at its speed.
// ---------------------------------------------------------------------------------------------
// One rule with at most two states on one element: advances the states and returns the new direction.
template <int A>
__device__ __forceinline__ float rule_one(const ChainParams& P, float x, float& s0, float& s1) {
  const float d0 = fmaxf(sqrtf(s1), P.eps);  // ADOPT normalises by the second moment before this gradient entered it
  if (A == kAdam || A == kLaProp || A == kRmsprop || A == kUnscaledAdam || A == kNadam) s1 = lerp_to(s1, x * x, P.b2);
  const float d = fmaxf(sqrtf(s1), P.eps);
  switch (A) {
    case kAdam: s0 = lerp_to(s0, x, P.b1); return s0 / d;
    case kLaProp: s0 = lerp_to(s0, x / d, P.b1); return s0;
    case kAdopt:
      s0 = lerp_to(s0, x / d0, P.b1);
      s1 = s1 * (1.0f - P.b3) + x * x * P.b3;
      return s0;
    case kRmsprop: return x / d;
    case kUnscaledAdam: s0 = lerp_to(s0, x / d, P.b1); return s0 * d;
    case kExpAvg: s0 = lerp_to(s0, x, P.b1); return s0;
    case kNesterovEma: s0 = lerp_to(s0, x, P.b1); return x + s0;
    case kHeavyball: s0 = s0 * P.b1 + x; return s0;
    case kNesterovMom: s0 = s0 * P.b1 + x; return x + s0 * P.b1;
    case kNadam: s0 = lerp_to(s0, x, P.b1); return x / d * P.b3 + s0 / d * P.alpha;
    default: return x;
  }
}

__device__ __forceinline__ F4 apply_rule(const ChainParams& P, const F4& u, F4& s0, F4& s1) {
  F4 out = u;
#define HB_CASE(A)                                                                                  \
  case A:                                                                                           \
    _Pragma("unroll") for (int k = 0; k < 4; ++k) out.v[k] = rule_one<A>(P, u.v[k], s0.v[k], s1.v[k]); \
    break;
  switch (P.algo) {
    HB_CASE(kAdam) HB_CASE(kLaProp) HB_CASE(kAdopt) HB_CASE(kRmsprop) HB_CASE(kUnscaledAdam) HB_CASE(kExpAvg)
    HB_CASE(kNesterovEma) HB_CASE(kHeavyball) HB_CASE(kNesterovMom) HB_CASE(kNadam)
    default: break;
  }
#undef HB_CASE
  return out;
}

// RULE: one moment rule, with or without MARS, known at compile time (kAnyRule: whatever the launch asks for; kAnyOfTwo: any rule with two states).
constexpr int kAnyRule = -1, kAnyOfTwo = -2;
constexpr int rule_states(int rule) { return rule == kAdam || rule == kAnyOfTwo ? 2 : 1; }

template <int DTP, int DTG, int DTU, int DTS, int OUT, int UIN, bool COUNT, int RULE = kAnyRule, bool MARS = false>
struct ChainKind {
  static constexpr int dt_p = DTP, dt_g = DTG, dt_u = DTU, dt_s = DTS, out_mode = OUT;
  static constexpr bool u_in = UIN != 0, count = COUNT, state = DTS != kNone;
  static constexpr bool reads_g = !u_in || count, reads_p = OUT == kOutParam;
  // Vectors per thread loaded together, and blocks per SM.  Two vectors through a rule need about 80 registers: three blocks.
  // The codec and its random bits are up to 190 instructions per element and want warps rather than vectors in flight: with
  // error-corrected state one vector is as many as fit.  What such a launch then waits for is that vector's loads (a third of its stalls) and the
  // ten dependent rounds of a random draw.  So the random bits are drawn side by side between the loads and their first use (cautious Adam with MARS
  // on 8 x 2048^2: 287 -> 265 us), and where the rule is a constant - which also takes the spills of the ten-way switch away (255) - the next
  // vector is fetched ahead of this one's arithmetic (231; three blocks, at two 248).  Without MARS 228 -> 162 us; Adam into fp32
  // parameters 195 -> 169, into error-corrected ones 245 -> 222; exponential average of 25 M elements (one state: four blocks) 122 -> 75;
  // momentum with MARS of a Llama-3-8B layer, at the clock that the products around it leave, 1.71 -> 1.42 ms.
  // Compiled in are the rules whose steps have been measured as workloads: Adam with codec state into fp32 and error-corrected parameters and under
  // caution, PSGD's exponential average, Muon's Nesterov average from fp32 gradients and, with MARS, from bf16 ones; of fp32 state only that
  // average, which spills without (85 M elements: 228 -> 202 us; Adam 165.6 -> 165.4, not worth a kernel).  An instance is two kernels of the same
  // length again, so others come in by measurement.  What the rest pays, 33.5 M elements, before these changes / with the rule left open: heavy-ball
  // momentum of fp32 gradients 156 / 154 us, of bf16 ones 129 / 128, with MARS 229 / 207; into fp32 parameters 136 / 135; LaProp 197 / 183, under
  // caution 233 / 214.
  // Launches without codec state draw the bits of 16-bit parameters early too (64 M elements, Adam into bf16: 254 -> 235 us; a parked update
  // into bf16, four vectors: 111 -> 91; into error-corrected parameters, where four vectors no longer fit: 159 -> 166, with two vectors 167 -> 145).
  static constexpr bool ecc = DTS == kBF16E8;
  // With the rule left open and an error-corrected parameter beside the states, bits that wait for their use cost more than the waits they fill (one
  // state, 33.5 M elements: drawn at use 181 us, early 190; two 243 to 247, early 239 to 249).
  static constexpr bool s_draws = ecc && (RULE != kAnyRule || DTP != kBF16E8);
  static constexpr bool p_draws = (DTP == kBF16E8 || DTP == kBF16) && !ecc && OUT == kOutParam;
  // Otherwise a thread should have about 128 bytes on their way: two vectors of Adam's four arrays, four where a launch reads
  // two arrays (momentum of GPT-2-small's fp32 matrices, 85M elements, two arrays read and two written, 1.36 GB:
  // 202 us, the rate of a copy).
  static constexpr int batch = ecc ? 1 : (DTP == kBF16E8 && !state) ? 2 : (state && (reads_p || count) ? 2 : 4);
  static constexpr int rule_n = rule_states(RULE);
  static constexpr bool one_state = RULE != kAnyRule && rule_n == 1;
  static constexpr bool ahead = ecc && RULE != kAnyRule;  // the next vector is fetched ahead
  static constexpr int min_blocks = ahead ? (one_state ? 4 : 3) : state && !(ecc && !count) ? 3 : 4;
  // Adam's four fp32 arrays at two vectors are in flight either way (166 us with the test per load on 39.5 M elements, 169 with one for all; into an
  // update, two states, 33.5 M elements: 126.5 / 129.7), one state's are not (87 us with one test for all, 93 per load)
  static constexpr bool either = state && (reads_p || RULE == kAnyOfTwo) && DTS == kF32 && DTG == kF32;
  static bool takes(const ChainParams& P, bool counting) {
    return counting == COUNT && P.out_mode == OUT && P.u_is_input == UIN && (!reads_p || P.dt_p == DTP) &&
           (!reads_g || P.dt_g == DTG) && ((OUT == kOutParam && !u_in) || P.dt_u == DTU) && P.dt_s == DTS &&
           (RULE == kAnyRule || ((P.algo == RULE || RULE == kAnyOfTwo) && P.n_state == rule_states(RULE) && (P.mars != 0) == MARS));
  }
  static __device__ __forceinline__ bool mars(const ChainParams& P) { return RULE == kAnyRule ? P.mars != 0 : MARS; }
  static __device__ __forceinline__ int n_state(const ChainParams& P) { return RULE == kAnyRule ? P.n_state : rule_n; }
  static __device__ __forceinline__ F4 apply(const ChainParams& P, const F4& u, F4& s0, F4& s1) {
    if constexpr (RULE == kAnyRule || RULE == kAnyOfTwo) {
      return apply_rule(P, u, s0, s1);
    } else {
      F4 out;
#pragma unroll
      for (int k = 0; k < 4; ++k) out.v[k] = rule_one<RULE>(P, u.v[k], s0.v[k], s1.v[k]);
      return out;
    }
  }
};

// Random bits of the states of four elements, drawn while their loads are on their way.
struct StateDraws {
  uint4 s0, s1, mars;
};
__device__ __forceinline__ void pin(uint4& r) { asm volatile("" : "+r"(r.x), "+r"(r.y), "+r"(r.z), "+r"(r.w)); }
__device__ __forceinline__ StateDraws draw_states(bool mars, int n_state, const Philox& rng, int64_t i, uint32_t t) {
  const uint32_t ctr = (uint32_t)(i >> 2), ctr_hi = (uint32_t)(i >> 34);
  const uint4 c0 = make_uint4(ctr, ctr_hi, t, 0u), c1 = make_uint4(ctr, ctr_hi, t, 1u), cm = make_uint4(ctr, ctr_hi ^ 0x40000000u, t, 4u);
  StateDraws r{};
  if (mars && n_state >= 2) {
    uint4 c[3] = {c0, c1, cm};
    rng.rounds(c);
    r = {c[0], c[1], c[2]};
  } else if (mars) {
    uint4 c[2] = {c0, cm};
    rng.rounds(c);
    r.s0 = c[0];
    r.mars = c[1];
  } else if (n_state >= 2) {
    uint4 c[2] = {c0, c1};
    rng.rounds(c);
    r.s0 = c[0];
    r.s1 = c[1];
  } else {
    uint4 c[1] = {c0};
    rng.rounds(c);
    r.s0 = c[0];
  }
  pin(r.s0);
  pin(r.s1);
  pin(r.mars);
  return r;
}

template <int kCase>
using LoadAs = std::integral_constant<int, kCase>;

template <class K, class Table>
__global__ void __launch_bounds__(kThreads, K::min_blocks) plain_chain_kernel(const __grid_constant__ Table T, ChainParams P) {
  // a launch that applies a parked update walks backwards: what the launch before it wrote last is still in the L2
  const int b = (K::u_in && K::reads_p) ? (int)(gridDim.x - 1 - blockIdx.x) : (int)blockIdx.x;
  int t = 0;
  if constexpr (std::is_same<Table, DeviceTable>::value) {
    t = find_range(T.prefix, P.n_tensors, b);
  } else {
    for (int i = 1; i < P.n_tensors; ++i)
      if (T.prefix[i] <= b) t = i;
  }
  const TensorMeta& M = T.metas[t];
  const int64_t numel = M.numel, base = (int64_t)(b - T.prefix[t]) * P.chunk, end = min(numel, base + P.chunk);
  const bool vec_ok = M.vec_ok != 0;
  const Philox rng(P.seed);
  void *const mp = M.p, *const mpe = M.pe, *const mg = M.g, *const mu = M.u;
  void *const m0 = M.s0, *const m0e = M.s0e, *const m1 = M.s1, *const m1e = M.s1e, *const mm = M.mars, *const mme = M.marse;

  float cscale = 1.0f;
  if (K::reads_p) {
    if (P.use_tensor_scale && M.scale != nullptr) cscale = *M.scale;
    if (P.caution_apply && M.masked != nullptr) {
      const float n = (float)numel;
      cscale *= n / fmaxf(n - (float)(*M.masked), 1.0f);
    }
  }
  constexpr int kBatch = K::batch;
  int masked_local = 0;
  float sumsq_local = 0.f, nonzero_local = 0.f;

  const int64_t first = base + threadIdx.x * 4;
  const auto fetch_as = [&](auto load_case, int64_t i, Raw4& s0, Raw4& s1, Raw4& old, Raw4& g, Raw4& u, Raw4& p) {
    constexpr int kCase = decltype(load_case)::value;
    const int nv = (int)max((int64_t)0, min((int64_t)4, end - i));
    if (K::state) {
      s0 = load_raw<K::dt_s, kCase>(m0, m0e, i, nv, vec_ok);
      if (!K::one_state) s1 = load_raw<K::dt_s, kCase>(m1, m1e, i, nv, vec_ok);
      if (K::mars(P)) old = load_raw<K::dt_s, kCase>(mm, mme, i, nv, vec_ok);
    }
    if (K::reads_g) g = load_raw<K::dt_g, kCase>(mg, nullptr, i, nv, vec_ok);
    if (K::u_in) u = load_raw<K::dt_u, kCase>(mu, nullptr, i, nv, vec_ok);
    if (K::reads_p) p = load_raw<K::dt_p, kCase>(mp, mpe, i, nv, vec_ok);
  };
  Raw4 s0_next{}, s1_next{}, old_next{}, g_next{}, u_next{}, p_next{};
  const auto fetch_next = [&](int64_t i) {
    if (vec_ok && i + 4 <= end) fetch_as(LoadAs<kWhole>{}, i, s0_next, s1_next, old_next, g_next, u_next, p_next);
    else fetch_as(LoadAs<kElements>{}, i, s0_next, s1_next, old_next, g_next, u_next, p_next);
  };
  if constexpr (K::ahead) fetch_next(first);

#pragma unroll 1
  for (int64_t i0 = first; i0 < end; i0 += kBatch * kThreads * 4) {
    Raw4 s0[kBatch], s1[kBatch], old[kBatch], g[kBatch], u[kBatch], p[kBatch];
    StateDraws rnd[kBatch];
    if constexpr (K::ahead) {  // (past the end: nothing is read)
      s0[0] = s0_next; s1[0] = s1_next; old[0] = old_next; g[0] = g_next; u[0] = u_next; p[0] = p_next;
      fetch_next(i0 + kThreads * 4);
    } else if constexpr (K::either) {
#pragma unroll
      for (int v = 0; v < kBatch; ++v) fetch_as(LoadAs<kEither>{}, i0 + v * (kThreads * 4), s0[v], s1[v], old[v], g[v], u[v], p[v]);
    } else if (vec_ok && i0 + (kBatch - 1) * (kThreads * 4) + 4 <= end) {  // only a part's last batch is not whole
#pragma unroll
      for (int v = 0; v < kBatch; ++v) fetch_as(LoadAs<kWhole>{}, i0 + v * (kThreads * 4), s0[v], s1[v], old[v], g[v], u[v], p[v]);
    } else {
#pragma unroll
      for (int v = 0; v < kBatch; ++v) fetch_as(LoadAs<kElements>{}, i0 + v * (kThreads * 4), s0[v], s1[v], old[v], g[v], u[v], p[v]);
    }
    uint4 p_rnd[kBatch];
    if constexpr (K::p_draws) {
#pragma unroll
      for (int v = 0; v < kBatch; ++v) {
        const int64_t i = i0 + v * (kThreads * 4);
        p_rnd[v] = make_uint4((uint32_t)(i >> 2), (uint32_t)(i >> 34), (uint32_t)t, 3u);
      }
      rng.rounds(p_rnd);
#pragma unroll
      for (int v = 0; v < kBatch; ++v) pin(p_rnd[v]);
    }
    if constexpr (K::s_draws) {
#pragma unroll
      for (int v = 0; v < kBatch; ++v) rnd[v] = draw_states(K::mars(P), K::n_state(P), rng, i0 + v * (kThreads * 4), (uint32_t)t);
    }
#pragma unroll
    for (int v = 0; v < kBatch; ++v) {
      const int64_t i = i0 + v * (kThreads * 4);
      const int nv = (int)max((int64_t)0, min((int64_t)4, end - i));
      if (nv == 0) break;
      const uint32_t ctr = (uint32_t)(i >> 2), ctr_hi = (uint32_t)(i >> 34);
      F4 grad{}, x;
      if (K::reads_g) grad = decode_raw<K::dt_g>(g[v]);
      x = K::u_in ? decode_raw<K::u_in ? K::dt_u : (int)kNone>(u[v]) : grad;
      if (K::u_in && P.u_op == kUopTrustRegion) {
#pragma unroll
        for (int k = 0; k < 4; ++k) x.v[k] = trust_region(x.v[k]);
      }
      if (K::state && K::mars(P)) {  // g <- lerp(g, g_prev, a); g_prev <- raw g
        const F4 raw = x, before = decode_raw<K::dt_s>(old[v]);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          x.v[k] = x.v[k] * (1.0f - P.mars_a) + before.v[k] * P.mars_a;
          grad.v[k] = x.v[k];
        }
        store_values<K::dt_s>(mm, mme, i, nv, vec_ok, raw, K::s_draws ? rnd[v].mars : draw(K::dt_s, rng, ctr, ctr_hi ^ 0x40000000u, (uint32_t)t, 4u));
      }
      F4 out = x;
      if (K::state) {
        F4 a{}, b{};
        if (m0 != nullptr) a = decode_raw<K::dt_s>(s0[v]);
        if (!K::one_state && m1 != nullptr) b = decode_raw<K::dt_s>(s1[v]);
        out = K::apply(P, x, a, b);
        if (K::n_state(P) >= 1) store_values<K::dt_s>(m0, m0e, i, nv, vec_ok, a, K::s_draws ? rnd[v].s0 : draw(K::dt_s, rng, ctr, ctr_hi, (uint32_t)t, 0u));
        if (K::n_state(P) >= 2) store_values<K::dt_s>(m1, m1e, i, nv, vec_ok, b, K::s_draws ? rnd[v].s1 : draw(K::dt_s, rng, ctr, ctr_hi, (uint32_t)t, 1u));
      }
      if (K::count) {  // phase one of caution: mask, count, park the masked update
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const bool disagree = (__float_as_uint(grad.v[k]) ^ __float_as_uint(out.v[k])) >> 31;
          if (k < nv && disagree) { out.v[k] = 0.f; ++masked_local; }
        }
      }
      if (!K::reads_p) {
        store_values<K::dt_u>(mu, nullptr, i, nv, vec_ok, out, draw(K::dt_u, rng, ctr, ctr_hi, (uint32_t)t, 5u));
        if (!K::count && P.accum_sumsq) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (k < nv) {
              sumsq_local += out.v[k] * out.v[k];
              nonzero_local += out.v[k] != 0.f ? 1.f : 0.f;
            }
        }
        continue;
      }
      // parameter epilogue: p <- p (1 - d lr) - lr u
      F4 np = decode_raw<K::reads_p ? K::dt_p : (int)kNone>(p[v]);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float uu = out.v[k] * cscale;
        float d = P.wd;
        if (P.cautious_wd && ((__float_as_uint(np.v[k]) ^ __float_as_uint(uu)) >> 31)) d = 0.f;
        np.v[k] = np.v[k] * (1.0f - d * P.lr) + uu * -P.lr;
      }
      store_values<K::dt_p>(mp, mpe, i, nv, vec_ok, np, K::p_draws ? p_rnd[v] : draw(K::dt_p, rng, ctr, ctr_hi, (uint32_t)t, 3u));
    }
  }
  finish_block<K::count>(P, M, sumsq_local, nonzero_local, masked_local);
}

// ---------------------------------------------------------------------------------------------
// Segmented sum of squares: out[t] += sum(x_t^2).  One block per chunk, one atomic per block.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) sumsq_kernel(const TensorMeta* __restrict__ metas,
                                                        const int* __restrict__ chunk_prefix, int n_tensors, int dt,
                                                        float* __restrict__ out) {
  const int b = blockIdx.x, lo = find_range(chunk_prefix, n_tensors, b);
  const TensorMeta M = metas[lo];
  const int64_t base = (int64_t)(b - chunk_prefix[lo]) * kChunk;
  float acc = 0.f;
#pragma unroll 2
  for (int it = 0; it < kChunk / (kThreads * 4); ++it) {
    const int64_t i = base + ((int64_t)it * kThreads + threadIdx.x) * 4;
    if (i >= M.numel) break;
    const int nv = (int)min((int64_t)4, M.numel - i);
    F4 x = load4(M.u, nullptr, dt, i, nv, M.vec_ok != 0);
#pragma unroll
    for (int k = 0; k < 4; ++k) acc += x.v[k] * x.v[k];
  }
  __shared__ float warp_sums[kThreads / 32];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xFFFFFFFFu, acc, o);
  if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float tot = 0.f;
    for (int w = 0; w < kThreads / 32; ++w) tot += warp_sums[w];
    atomicAdd(out + lo, tot);
  }
}

// ---------------------------------------------------------------------------------------------
// Segmented dot product and absolute maximum over the same chunk table: out[t] = sum(x_t * y_t) or max |x_t|.
// x comes from TensorMeta::u, y from TensorMeta::g; `out` starts at zero.  One block per chunk; the block results
// meet in out[t] through one atomic each (float add; for the maximum an unsigned integer max on the bit pattern,
// which orders non-negative floats like their values and puts NaN above everything, so a NaN input gives NaN).
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ float nan_max(float acc, float a) { return (a > acc || a != a) ? a : acc; }

template <int OP>
__global__ void __launch_bounds__(kThreads) segmented_reduce_kernel(const TensorMeta* __restrict__ metas,
                                                                   const int* __restrict__ chunk_prefix, int n_tensors,
                                                                   int dt, float* __restrict__ out) {
  const int b = blockIdx.x, lo = find_range(chunk_prefix, n_tensors, b);
  const TensorMeta M = metas[lo];
  const int64_t base = (int64_t)(b - chunk_prefix[lo]) * kChunk;
  float acc = 0.f;
#pragma unroll 2
  for (int it = 0; it < kChunk / (kThreads * 4); ++it) {
    const int64_t i = base + ((int64_t)it * kThreads + threadIdx.x) * 4;
    if (i >= M.numel) break;
    const int nv = (int)min((int64_t)4, M.numel - i);
    const F4 x = load4(M.u, nullptr, dt, i, nv, M.vec_ok != 0);
    if (OP == kReduceDot) {
      const F4 y = load4(M.g, nullptr, dt, i, nv, M.vec_ok != 0);
#pragma unroll
      for (int k = 0; k < 4; ++k) acc += x.v[k] * y.v[k];
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) acc = nan_max(acc, fabsf(x.v[k]));  // lanes past the end read as zero
    }
  }
  __shared__ float warp_res[kThreads / 32];
  for (int o = 16; o > 0; o >>= 1) {
    const float other = __shfl_down_sync(0xFFFFFFFFu, acc, o);
    acc = OP == kReduceDot ? acc + other : nan_max(acc, other);
  }
  if ((threadIdx.x & 31) == 0) warp_res[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float tot = warp_res[0];
    for (int w = 1; w < kThreads / 32; ++w) tot = OP == kReduceDot ? tot + warp_res[w] : nan_max(tot, warp_res[w]);
    if (OP == kReduceDot)
      atomicAdd(out + lo, tot);
    else
      atomicMax(reinterpret_cast<unsigned int*>(out + lo), __float_as_uint(tot));
  }
}

namespace {

template <class... Ks>
struct KindList {};
using Kinds = KindList<
    //        parameter gradient update state
    // rules known at compile time
    ChainKind<kF32, kF32, kNone, kBF16E8, kOutParam, 0, false, kAdam>,
    ChainKind<kBF16E8, kBF16, kNone, kBF16E8, kOutParam, 0, false, kAdam>,
    ChainKind<kNone, kF32, kF32, kBF16E8, kOutUpdate, 0, false, kExpAvg>,
    ChainKind<kNone, kF32, kF32, kBF16E8, kOutUpdate, 0, false, kNesterovEma>,
    ChainKind<kNone, kBF16, kF32, kBF16E8, kOutUpdate, 0, false, kNesterovEma, true>,
    ChainKind<kNone, kF32, kF32, kF32, kOutUpdate, 0, false, kNesterovEma>,
    ChainKind<kNone, kF32, kF32, kBF16E8, kOutUpdate, 0, true, kAdam, false>,
    ChainKind<kNone, kF32, kF32, kBF16E8, kOutUpdate, 0, true, kAdam, true>,
    // any rule with two states
    ChainKind<kNone, kF32, kF32, kF32, kOutUpdate, 0, false, kAnyOfTwo>,
    // any rule
    ChainKind<kF32, kF32, kNone, kF32, kOutParam, 0, false>,       // first-order rules on fp32 parameters
    ChainKind<kBF16, kBF16, kNone, kF32, kOutParam, 0, false>,     // ... on bf16 parameters
    ChainKind<kF32, kF32, kNone, kBF16E8, kOutParam, 0, false>,    // ... with error-corrected state
    ChainKind<kBF16E8, kBF16, kNone, kBF16E8, kOutParam, 0, false>,
    ChainKind<kNone, kF32, kF32, kNone, kOutUpdate, 0, false>,     // gradient into an fp32 update
    ChainKind<kNone, kF32, kF32, kF32, kOutUpdate, 0, false>,      // momentum into an fp32 update
    ChainKind<kNone, kF32, kF32, kBF16E8, kOutUpdate, 0, false>,
    ChainKind<kNone, kBF16, kF32, kBF16E8, kOutUpdate, 0, false>,
    ChainKind<kNone, kF32, kF32, kF32, kOutUpdate, 0, true>,       // caution, first launch
    ChainKind<kNone, kF32, kF32, kBF16E8, kOutUpdate, 0, true>,
    ChainKind<kNone, kF32, kF32, kNone, kOutUpdate, 1, true>,      // caution on a finished update
    ChainKind<kNone, kBF16, kF32, kNone, kOutUpdate, 1, true>,
    ChainKind<kF32, kNone, kF32, kNone, kOutParam, 1, false>,      // finished update -> parameter
    ChainKind<kBF16, kNone, kF32, kNone, kOutParam, 1, false>,
    ChainKind<kBF16E8, kNone, kF32, kNone, kOutParam, 1, false>>;

using PlainLaunch = void (*)(DeviceTable, ChainParams);
using InlineLaunch = void (*)(InlineTable, ChainParams);

struct PlainKind {
  PlainLaunch kernel = nullptr;
  InlineLaunch kernel_inline = nullptr;
  int vectors = 0;  // in flight per thread
};

// The first specialised instance that covers the launch; without a kernel when the general one has to run it.
template <class... Ks>
PlainKind find_kind(KindList<Ks...>, const ChainParams& P, bool count) {
  const bool plain = P.n_state <= 2 && P.algo != kAdemamix && P.n_src == 0 && P.n_dst == 0 && P.g_clip_mode == kClipNone &&
                     (P.u_op == kUopNone || (P.u_op == kUopTrustRegion && P.u_is_input)) && P.post_state == kPostNone && P.out_mode != kOutScheduleFree &&
                     (!P.u_is_input || (P.algo == kIdentity && P.n_state == 0 && !P.mars)) && !(count && P.accum_sumsq);
  PlainKind hit;
  if (plain) ((hit.kernel == nullptr && Ks::takes(P, count) ? (void)(hit = {plain_chain_kernel<Ks, DeviceTable>, plain_chain_kernel<Ks, InlineTable>, Ks::batch}) : (void)0), ...);
  return hit;
}

}  // namespace

int chain_chunk_elems() { return kChunk; }

int chain_chunk_elems_for(const ChainParams& P, bool count_caution, int64_t total_elems) {
  const PlainKind kind = find_kind(Kinds{}, P, count_caution);
  return kind.kernel != nullptr ? chain_chunk(kind.vectors, total_elems) : kChunk;
}

cudaError_t launch_fused_chain(const TensorMeta* metas, const int* chunk_prefix, int total_chunks, const ChainParams& P0,
                               bool count_caution, cudaStream_t stream) {
  if (total_chunks <= 0) return cudaSuccess;
  ChainParams P = P0;
  if (P.chunk == 0) P.chunk = kChunk;
  if (const PlainLaunch kernel = find_kind(Kinds{}, P, count_caution).kernel)
    kernel<<<total_chunks, kThreads, 0, stream>>>(DeviceTable{metas, chunk_prefix}, P);
  else if (P.chunk != kChunk)
    return cudaErrorInvalidValue;  // the general kernel is compiled for one chunk size
  else if (count_caution)
    fused_chain_kernel<true><<<total_chunks, kThreads, 0, stream>>>(metas, chunk_prefix, P);
  else
    fused_chain_kernel<false><<<total_chunks, kThreads, 0, stream>>>(metas, chunk_prefix, P);
  return cudaGetLastError();
}

bool chain_takes_inline(const ChainParams& P, bool count_caution, int n_tensors, int64_t total_elems) {
  return n_tensors <= kInlineTensors && total_elems <= (1 << 23) && find_kind(Kinds{}, P, count_caution).kernel != nullptr;
}

cudaError_t launch_fused_chain_inline(const TensorMeta* host_metas, const int* host_prefix, int total_chunks, const ChainParams& P,
                                      bool count_caution, cudaStream_t stream) {
  if (total_chunks <= 0) return cudaSuccess;
  const InlineLaunch kernel = find_kind(Kinds{}, P, count_caution).kernel_inline;
  if (kernel == nullptr || P.n_tensors > kInlineTensors || P.chunk == 0) return cudaErrorInvalidValue;
  InlineTable T;
  std::copy(host_prefix, host_prefix + P.n_tensors + 1, T.prefix);
  std::copy(host_metas, host_metas + P.n_tensors, T.metas);
  kernel<<<total_chunks, kThreads, 0, stream>>>(T, P);
  return cudaGetLastError();
}

cudaError_t launch_sumsq(const TensorMeta* metas, const int* chunk_prefix, int total_chunks, int n_tensors, int dt,
                         float* out, cudaStream_t stream) {
  if (total_chunks <= 0) return cudaSuccess;
  sumsq_kernel<<<total_chunks, kThreads, 0, stream>>>(metas, chunk_prefix, n_tensors, dt, out);
  return cudaGetLastError();
}

cudaError_t launch_segmented_reduce(const TensorMeta* metas, const int* chunk_prefix, int total_chunks, int n_tensors,
                                    int dt, int op, float* out, cudaStream_t stream) {
  if (total_chunks <= 0) return cudaSuccess;
  if (op == kReduceDot)
    segmented_reduce_kernel<kReduceDot><<<total_chunks, kThreads, 0, stream>>>(metas, chunk_prefix, n_tensors, dt, out);
  else if (op == kReduceAbsMax)
    segmented_reduce_kernel<kReduceAbsMax><<<total_chunks, kThreads, 0, stream>>>(metas, chunk_prefix, n_tensors, dt, out);
  else
    return cudaErrorInvalidValue;
  return cudaGetLastError();
}

}  // namespace hb
