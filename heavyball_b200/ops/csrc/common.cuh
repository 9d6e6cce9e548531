// Device helpers shared by the optimizer kernels: counter-based RNG, dtype-generic vector load/store,
// stochastic rounding to bf16 and the ULP error-correction codec (16-bit float + integer residual).
//
// Numerics follow the PyTorch definitions in heavyball_b200/utils/core.py (parity targets
// heavyball/utils.py:1288-1324 codec, 2341-2370 stochastic rounding).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace hb {

// Storage kinds understood by the element-wise kernels.
enum DType : int { kF32 = 0, kBF16 = 1, kF16 = 2, kBF16E8 = 3, kBF16E16 = 4, kF16E8 = 5, kF16E16 = 6, kNone = 7 };

__host__ __device__ inline bool is_ecc(int d) { return d >= kBF16E8 && d <= kF16E16; }
__host__ __device__ inline bool is_bf16_like(int d) { return d == kBF16 || d == kBF16E8 || d == kBF16E16; }
__host__ __device__ inline bool ecc_wide(int d) { return d == kBF16E16 || d == kF16E16; }

// Index of the range that holds position `b`: the last entry of the ascending table `first` (n entries, first[0] == 0) that is
// <= b.  A warp tests 32 entries at a time (one load for up to 32 ranges, two up to 1024) where a binary search is a chain of
// five to ten dependent loads, paid by every block before its first data load.  Executed by whole warps.
__device__ inline int find_range(const int* __restrict__ first, int n, int b) {
  int lo = 0, len = n;
  while (len > 1) {
    const int step = (len + 31) >> 5, at = lo + (int)(threadIdx.x & 31) * step;
    const unsigned below = __ballot_sync(0xFFFFFFFFu, at < lo + len && first[at] <= b);  // lane 0 always counts
    const int k = 31 - __clz(below);
    len = min(step, len - k * step);
    lo += k * step;
  }
  return lo;
}

// ---------------------------------------------------------------------------------------------
// Philox-4x32-10.  Streams are addressed by (seed, tensor index, element index / 4, draw id), never
// by launch geometry, so results do not depend on grid shape or on which rank runs the update.
// ---------------------------------------------------------------------------------------------
struct Philox {
  uint32_t k0, k1;
  __device__ Philox(uint64_t seed) : k0((uint32_t)seed), k1((uint32_t)(seed >> 32)) {}
  __device__ inline uint4 operator()(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3) const {
    uint32_t a = k0, b = k1;
#pragma unroll
    for (int i = 0; i < 10; ++i) {
      uint32_t hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
      uint32_t hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
      c0 = hi1 ^ c1 ^ a;
      c1 = lo1;
      c2 = hi0 ^ c3 ^ b;
      c3 = lo0;
      a += 0x9E3779B9u;
      b += 0xBB67AE85u;
    }
    return make_uint4(c0, c1, c2, c3);
  }
  // Counters -> random bits.  A round waits for the one before; several draws of a thread side by side fill those waits.  The products are
  // 64 bits wide here; a single draw, among other arithmetic, is better off with halves (Adam with bf16 state on 33.5 M elements, the general
  // kernel: 338 us, with wide products 364; with 16-bit residuals 550 / 594).
  template <int N>
  __device__ __forceinline__ void rounds(uint4 (&c)[N]) const {
    uint32_t a = k0, b = k1;
#pragma unroll
    for (int i = 0; i < 10; ++i) {
#pragma unroll
      for (int n = 0; n < N; ++n) {
        const uint64_t p0 = (uint64_t)0xD2511F53u * c[n].x, p1 = (uint64_t)0xCD9E8D57u * c[n].z;
        c[n] = make_uint4((uint32_t)(p1 >> 32) ^ c[n].y ^ a, (uint32_t)p1, (uint32_t)(p0 >> 32) ^ c[n].w ^ b, (uint32_t)p0);
      }
      a += 0x9E3779B9u;
      b += 0xBB67AE85u;
    }
  }
};

__device__ inline float u32_to_unit(uint32_t x) { return (float)(x >> 8) * (1.0f / 16777216.0f); }  // [0, 1)

// ---------------------------------------------------------------------------------------------
// bf16 stochastic rounding: add 16 uniform low bits, truncate.
// ---------------------------------------------------------------------------------------------
__device__ inline uint16_t sr_bf16_bits(float x, uint32_t rnd16) {
  uint32_t b = __float_as_uint(x);
  b += (rnd16 & 0xFFFFu);
  return (uint16_t)(b >> 16);
}
__device__ inline float bf16_bits_to_float(uint16_t h) { return __uint_as_float(((uint32_t)h) << 16); }
__device__ inline uint16_t rne_bf16_bits(float x) { return __bfloat16_as_ushort(__float2bfloat16_rn(x)); }
__device__ inline float f16_bits_to_float(uint16_t h) { return __half2float(__ushort_as_half(h)); }
__device__ inline uint16_t rne_f16_bits(float x) { return __half_as_ushort(__float2half_rn(x)); }

// log2(ulp) - 1 of a 16-bit float given its bits.
__device__ inline int half_ulp_log2(uint16_t bits, bool bf16) {
  int m = bf16 ? 7 : 10, bias = bf16 ? 127 : 15;
  int e = (bits & 0x7FFF) >> m;
  return (e == 0 ? 1 - bias - m : e - (bias + m)) - 1;
}

// The codec's scale is a power of two taken from the primary's exponent.  For bf16 values of at least 2^-95 (biased exponent
// 32) that power and its reciprocal are floats whose exponent fields follow from the primary's by one subtraction, and every
// product with them is exact: the same results as ldexpf for a fraction of its instructions.  An error-corrected Adam step
// does six of these per element and is bound by instruction issue (Muon step of a Llama-3-8B layer: 19.7 -> 18.9 ms).
constexpr uint32_t kEccFastExp = 32u << 23;

__device__ inline float ecc_decode(uint16_t prim, int corr, bool bf16, float inv_smax) {
  const float base = bf16 ? bf16_bits_to_float(prim) : f16_bits_to_float(prim);
  const uint32_t ebits = __float_as_uint(base) & 0x7F800000u;
  if (bf16 && ebits >= kEccFastExp)  // 2^(e - 135): half a unit in the last place
    return fmaf((float)corr * inv_smax, __uint_as_float(ebits - (8u << 23)), base);
  return base + ldexpf((float)corr * inv_smax, half_ulp_log2(prim, bf16));
}

// Returns the residual (integer units) for fp32 value x once prim = RNE(x) is chosen.
__device__ inline int ecc_residual(float x, uint16_t prim, bool bf16, float smax, float unit_rand) {
  const float base = bf16 ? bf16_bits_to_float(prim) : f16_bits_to_float(prim);
  const uint32_t ebits = __float_as_uint(base) & 0x7F800000u;
  float e;
  if (bf16 && ebits >= kEccFastExp)
    e = (x - base) * __uint_as_float((262u << 23) - ebits);
  else
    e = ldexpf(x - base, -half_ulp_log2(prim, bf16));
  e = fminf(fmaxf(e, -1.0f), 1.0f) * smax;
  return __float2int_rd(e + unit_rand);
}

// The same for four bf16 values with 8-bit residuals, the usual kind.  One test of the exponents serves the four (false: the
// caller takes the element-wise path), and conversions between integers and floats go through the low mantissa bits of 2^23
// instead of the conversion unit, which delivers 4 lanes a cycle: byte -> float as 2^23 + byte, floor -> byte by adding
// 1.5 * 2^23 rounded down.  Same bits as the element-wise codec.
__device__ inline bool ecc8_decode4(uint32_t lo, uint32_t hi, uint32_t res, float (&v)[4]) {
  const uint32_t b[4] = {lo << 16, lo & 0xFFFF0000u, hi << 16, hi & 0xFFFF0000u};
  const uint32_t e[4] = {b[0] & 0x7F800000u, b[1] & 0x7F800000u, b[2] & 0x7F800000u, b[3] & 0x7F800000u};
  if (min(min(e[0], e[1]), min(e[2], e[3])) < kEccFastExp) return false;
  const uint32_t biased = res ^ 0x80808080u;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float c = __uint_as_float(__byte_perm(biased, 0x4B000000u, 0x7650u + k)) - 8388736.0f;  // 2^23 + 128
    v[k] = fmaf(c * (1.0f / 127.0f), __uint_as_float(e[k] - (8u << 23)), __uint_as_float(b[k]));
  }
  return true;
}

__device__ inline bool ecc8_encode4(const float (&x)[4], const uint32_t (&rnd)[4], uint32_t& lo, uint32_t& hi, uint32_t& res) {
  const __nv_bfloat162 p0 = __floats2bfloat162_rn(x[0], x[1]), p1 = __floats2bfloat162_rn(x[2], x[3]);
  lo = *reinterpret_cast<const uint32_t*>(&p0);
  hi = *reinterpret_cast<const uint32_t*>(&p1);
  const uint32_t b[4] = {lo << 16, lo & 0xFFFF0000u, hi << 16, hi & 0xFFFF0000u};
  const uint32_t e[4] = {b[0] & 0x7F800000u, b[1] & 0x7F800000u, b[2] & 0x7F800000u, b[3] & 0x7F800000u};
  if (min(min(e[0], e[1]), min(e[2], e[3])) < kEccFastExp) return false;
  uint32_t r[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float d = (x[k] - __uint_as_float(b[k])) * __uint_as_float((262u << 23) - e[k]);
    const float y = fminf(fmaxf(d, -1.0f), 1.0f) * 127.0f + u32_to_unit(rnd[k]);
    r[k] = __float_as_uint(__fadd_rd(y, 12582912.0f));  // 1.5 * 2^23 + floor(y): the low byte is the residual
  }
  res = __byte_perm(__byte_perm(r[0], r[1], 0x0040), __byte_perm(r[2], r[3], 0x0040), 0x5410);
  return true;
}

// ---------------------------------------------------------------------------------------------
// 4-wide generic load / store.  `p` is the primary buffer, `c` the ECC residual buffer (or null).
// ---------------------------------------------------------------------------------------------
struct F4 {
  float v[4];
};

// All loops below have compile-time trip counts and constant indices so that the 4-element
// temporaries live in registers (dynamic indexing would push them to local memory).
__device__ inline void unpack_h4(const void* src, int n_valid, bool fast, uint16_t (&h)[4]) {
  const uint16_t* hp = (const uint16_t*)src;
  if (fast) {
    uint2 t = *(const uint2*)hp;
    h[0] = t.x & 0xFFFF; h[1] = t.x >> 16; h[2] = t.y & 0xFFFF; h[3] = t.y >> 16;
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) h[k] = (k < n_valid) ? hp[k] : (uint16_t)0;
  }
}

__device__ inline F4 load4(const void* p, const void* c, int dt, int64_t i, int n_valid, bool vec_ok) {
  F4 r;
#pragma unroll
  for (int k = 0; k < 4; ++k) r.v[k] = 0.f;
  if (dt == kNone || p == nullptr) return r;
  const bool fast = vec_ok && n_valid == 4;
  if (dt == kF32) {
    const float* f = (const float*)p + i;
    if (fast) {
      float4 t = *(const float4*)f;
      r.v[0] = t.x; r.v[1] = t.y; r.v[2] = t.z; r.v[3] = t.w;
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (k < n_valid) r.v[k] = f[k];
    }
    return r;
  }
  uint16_t h[4];
  unpack_h4((const uint16_t*)p + i, n_valid, fast, h);
  const bool bf = is_bf16_like(dt);
  if (!is_ecc(dt)) {
#pragma unroll
    for (int k = 0; k < 4; ++k) r.v[k] = bf ? bf16_bits_to_float(h[k]) : f16_bits_to_float(h[k]);
    return r;
  }
  int corr[4];
  if (ecc_wide(dt)) {
    uint16_t w[4];
    unpack_h4((const uint16_t*)c + i, n_valid, fast, w);
#pragma unroll
    for (int k = 0; k < 4; ++k) corr[k] = (int)(int16_t)w[k];
  } else {
    const int8_t* cp = (const int8_t*)c + i;
    if (fast) {
      uint32_t t = *(const uint32_t*)cp;
#pragma unroll
      for (int k = 0; k < 4; ++k) corr[k] = (int)(int8_t)((t >> (8 * k)) & 0xFF);
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) corr[k] = (k < n_valid) ? (int)cp[k] : 0;
    }
  }
  const float inv = ecc_wide(dt) ? (1.0f / 32767.0f) : (1.0f / 127.0f);
#pragma unroll
  for (int k = 0; k < 4; ++k) r.v[k] = ecc_decode(h[k], corr[k], bf, inv);
  return r;
}

__device__ inline void pack_h4(void* dst, int n_valid, bool fast, const uint16_t (&h)[4]) {
  uint16_t* hp = (uint16_t*)dst;
  if (fast) {
    uint2 t;
    t.x = (uint32_t)h[0] | ((uint32_t)h[1] << 16);
    t.y = (uint32_t)h[2] | ((uint32_t)h[3] << 16);
    *(uint2*)hp = t;
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < n_valid) hp[k] = h[k];
  }
}

// rnd supplies 4 x 32 random bits: low 16 bits feed bf16 stochastic rounding, the 24 high bits the
// stochastic floor of the ECC residual.
__device__ inline void store4(void* p, void* c, int dt, int64_t i, int n_valid, bool vec_ok, const F4& x, uint4 rnd) {
  if (dt == kNone || p == nullptr) return;
  const bool fast = vec_ok && n_valid == 4;
  const uint32_t rr[4] = {rnd.x, rnd.y, rnd.z, rnd.w};
  if (dt == kF32) {
    float* f = (float*)p + i;
    if (fast) {
      *(float4*)f = make_float4(x.v[0], x.v[1], x.v[2], x.v[3]);
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (k < n_valid) f[k] = x.v[k];
    }
    return;
  }
  const bool bf = is_bf16_like(dt);
  uint16_t h[4];
  if (!is_ecc(dt)) {
#pragma unroll
    for (int k = 0; k < 4; ++k) h[k] = bf ? sr_bf16_bits(x.v[k], rr[k]) : rne_f16_bits(x.v[k]);
    pack_h4((uint16_t*)p + i, n_valid, fast, h);
    return;
  }
  int corr[4];
  const float smax = ecc_wide(dt) ? 32767.0f : 127.0f;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    h[k] = bf ? rne_bf16_bits(x.v[k]) : rne_f16_bits(x.v[k]);
    corr[k] = ecc_residual(x.v[k], h[k], bf, smax, u32_to_unit(rr[k]));
  }
  pack_h4((uint16_t*)p + i, n_valid, fast, h);
  if (c == nullptr) return;  // primary-only copy (a peer's replica of a parameter whose residual lives with its owner)
  if (ecc_wide(dt)) {
    uint16_t w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) w[k] = (uint16_t)(int16_t)corr[k];
    pack_h4((uint16_t*)c + i, n_valid, fast, w);
  } else {
    int8_t* cp = (int8_t*)c + i;
    if (fast) {
      uint32_t t = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) t |= ((uint32_t)(uint8_t)(int8_t)corr[k]) << (8 * k);
      *(uint32_t*)cp = t;
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (k < n_valid) cp[k] = (int8_t)corr[k];
    }
  }
}

// ---------------------------------------------------------------------------------------------
// The load in two halves, for storage kinds known at compile time: the words of four elements, and their values.  Decoding an
// error-corrected value branches on its exponent, and loads behind a branch that waits for a load wait with it: a kernel that
// decoded each array as it arrived paid one memory round trip per array instead of one for all.
// ---------------------------------------------------------------------------------------------
struct Raw4 {
  uint32_t w[4];
};

// kWhole: all four elements are there and every buffer starts on a 16-byte boundary.  The caller decides that once for all of its loads: with the
// element-wise loads of the other case beside it, the compiler predicates those, and the instructions that put 16-bit values together wait for the
// wide load they would have replaced - one memory round trip per array again (update masked against a bf16 gradient, 64 M elements: 171 us with
// the two cases per load, 104 with one).
enum LoadCase : int { kElements, kWhole, kEither };
template <int DT, int kCase>
__device__ __forceinline__ Raw4 load_raw(const void* p, const void* c, int64_t i, int n_valid, bool vec_ok) {
  Raw4 r{{0u, 0u, 0u, 0u}};
  if (DT == kNone || p == nullptr) return r;
  const bool fast = kCase == kWhole || (kCase == kEither && vec_ok && n_valid == 4);
  if (DT == kF32) {
    const uint32_t* f = (const uint32_t*)p + i;
    if (fast) {
      const uint4 t = *(const uint4*)f;
      r.w[0] = t.x; r.w[1] = t.y; r.w[2] = t.z; r.w[3] = t.w;
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (k < n_valid) r.w[k] = f[k];
    }
    return r;
  }
  const uint16_t* h = (const uint16_t*)p + i;
  const uint8_t* e = (const uint8_t*)c + i;
  if (fast) {
    const uint2 t = *(const uint2*)h;
    r.w[0] = t.x; r.w[1] = t.y;
    if (DT == kBF16E8) r.w[2] = *(const uint32_t*)e;
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < n_valid) {
        r.w[k >> 1] |= (uint32_t)h[k] << (16 * (k & 1));
        if (DT == kBF16E8) r.w[2] |= (uint32_t)e[k] << (8 * k);
      }
  }
  return r;
}

template <int DT>
__device__ inline F4 decode_raw(const Raw4& r) {
  static_assert(DT == kF32 || DT == kBF16 || DT == kBF16E8 || DT == kNone, "storage kinds of the specialised kernels");
  F4 out;
  if (DT == kBF16E8) {
    if (ecc8_decode4(r.w[0], r.w[1], r.w[2], out.v)) return out;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      out.v[k] = ecc_decode((uint16_t)(r.w[k >> 1] >> (16 * (k & 1))), (int)(int8_t)(r.w[2] >> (8 * k)), true, 1.0f / 127.0f);
    return out;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k)
    out.v[k] = DT == kF32 ? __uint_as_float(r.w[k]) : __uint_as_float((k & 1) ? (r.w[k >> 1] & 0xFFFF0000u) : (r.w[k >> 1] << 16));
  return out;
}

// store4 for a storage kind known at compile time.
template <int DT>
__device__ inline void store_values(void* p, void* c, int64_t i, int n_valid, bool vec_ok, const F4& x, uint4 rnd) {
  if (DT == kBF16E8 && p != nullptr && c != nullptr && vec_ok && n_valid == 4) {
    const uint32_t rr[4] = {rnd.x, rnd.y, rnd.z, rnd.w};
    uint2 prim;
    uint32_t res;
    if (ecc8_encode4(x.v, rr, prim.x, prim.y, res)) {
      *(uint2*)((uint16_t*)p + i) = prim;
      *(uint32_t*)((int8_t*)c + i) = res;
      return;
    }
  }
  store4(p, c, DT, i, n_valid, vec_ok, x, rnd);
}

// ---------------------------------------------------------------------------------------------
// NVSwitch multicast accesses (multimem): one instruction acts on the same address of every GPU bound to the
// multicast object.  Addresses must be 16-byte (v4.f32) / 8-byte (v2) aligned.
// ---------------------------------------------------------------------------------------------
__device__ inline F4 mc_ld_reduce4(const void* mc, int dt, int64_t i) {
  F4 r;
  if (dt == kF32) {
    asm volatile("multimem.ld_reduce.relaxed.sys.global.add.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(r.v[0]), "=f"(r.v[1]), "=f"(r.v[2]), "=f"(r.v[3])
                 : "l"((const float*)mc + i)
                 : "memory");
  } else {  // four 16-bit values, accumulated in fp32 inside the switch
    uint32_t a, b;
    if (dt == kBF16)
      asm volatile("multimem.ld_reduce.relaxed.sys.global.add.acc::f32.v2.bf16x2 {%0, %1}, [%2];"
                   : "=r"(a), "=r"(b) : "l"((const uint16_t*)mc + i) : "memory");
    else
      asm volatile("multimem.ld_reduce.relaxed.sys.global.add.acc::f32.v2.f16x2 {%0, %1}, [%2];"
                   : "=r"(a), "=r"(b) : "l"((const uint16_t*)mc + i) : "memory");
    const uint16_t h[4] = {(uint16_t)(a & 0xFFFF), (uint16_t)(a >> 16), (uint16_t)(b & 0xFFFF), (uint16_t)(b >> 16)};
#pragma unroll
    for (int k = 0; k < 4; ++k) r.v[k] = dt == kBF16 ? bf16_bits_to_float(h[k]) : f16_bits_to_float(h[k]);
  }
  return r;
}

// Stores the primary of four elements to every GPU through the multicast address `mc`; the residual of an
// error-corrected value (if any) goes to the local buffer `c`.  Same rounding as store4.
__device__ inline void mc_store4(void* mc, void* c, int dt, int64_t i, const F4& x, uint4 rnd) {
  if (dt == kF32) {
    asm volatile("multimem.st.relaxed.sys.global.v4.f32 [%0], {%1, %2, %3, %4};"
                 ::"l"((float*)mc + i), "f"(x.v[0]), "f"(x.v[1]), "f"(x.v[2]), "f"(x.v[3])
                 : "memory");
    return;
  }
  const uint32_t rr[4] = {rnd.x, rnd.y, rnd.z, rnd.w};
  const bool bf = is_bf16_like(dt);
  uint16_t h[4];
  int corr[4] = {0, 0, 0, 0};
  const float smax = ecc_wide(dt) ? 32767.0f : 127.0f;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (is_ecc(dt)) {
      h[k] = bf ? rne_bf16_bits(x.v[k]) : rne_f16_bits(x.v[k]);
      corr[k] = ecc_residual(x.v[k], h[k], bf, smax, u32_to_unit(rr[k]));
    } else {
      h[k] = bf ? sr_bf16_bits(x.v[k], rr[k]) : rne_f16_bits(x.v[k]);
    }
  }
  const float lo = __uint_as_float((uint32_t)h[0] | ((uint32_t)h[1] << 16));
  const float hi = __uint_as_float((uint32_t)h[2] | ((uint32_t)h[3] << 16));
  asm volatile("multimem.st.relaxed.sys.global.v2.f32 [%0], {%1, %2};" ::"l"((uint16_t*)mc + i), "f"(lo), "f"(hi) : "memory");
  if (is_ecc(dt) && c != nullptr) {
    if (ecc_wide(dt)) {
      uint16_t w[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) w[k] = (uint16_t)(int16_t)corr[k];
      pack_h4((uint16_t*)c + i, 4, true, w);
    } else {
      uint32_t t = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) t |= ((uint32_t)(uint8_t)(int8_t)corr[k]) << (8 * k);
      *(uint32_t*)((int8_t*)c + i) = t;
    }
  }
}

}  // namespace hb
