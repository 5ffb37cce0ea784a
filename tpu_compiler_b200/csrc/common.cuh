// Shared device/host helpers for the B200 interpreter backend.
//
// The requantisation and rounding primitives restate, for the device, the
// reference's QuantizationArithmetic.cpp free functions
// (lib/Dialect/TPU/Quantization/QuantizationArithmetic.cpp):
//   qdm_requant      <- applyMultiplierAndRShiftAndSaturateInt8(.., qdm=true)  :518-539
//                       (SaturatingRoundingDoublingHighMul :501-509,
//                        RoundingDivideByPOT :487-499, saturateInt8 :301-334)
//   mul_rshift_sat8  <- the same function with qdm=false                      :526
//   rshift_sat8      <- applyRShiftAndSaturateInt8                            :481-483
//   f32_to_bf16_bits <- F32ToBF16                                             :873-910
//   f32_to_int8_rne  <- F32ToInt8(v, 0) / F32ToInt (round half to even on |v|) :918-947
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#define TPUCB_HD __host__ __device__ __forceinline__

namespace tpucb {

TPUCB_HD int clamp_i8(int q) { return q > 127 ? 127 : (q < -128 ? -128 : q); }

// gemmlowp-style rounding doubling high multiply followed by a rounding right
// shift and int8 saturation. v: int32 accumulator (bias already added),
// M: multiplier as int32, r: right shift in [0,31].
TPUCB_HD int qdm_requant(int32_t v, int32_t M, int r) {
  long long ab = (long long)v * (long long)M;
  long long x = ab + (ab >= 0 ? (1ll << 30) : (1ll - (1ll << 30)));
  // C++ division by 2^31 truncates toward zero.
  long long fl = x >> 31;
  if (x < 0 && (x & 0x7fffffffll) != 0) fl += 1;
  int32_t hi = (int32_t)fl;
  int32_t q;
  if (hi == 0 || r == 0) {
    q = hi;
  } else {
    int32_t mask = (int32_t)((1ll << r) - 1);
    int32_t rem = hi & mask;
    int32_t thr = (mask >> 1) + (hi < 0 ? 1 : 0);
    q = (hi >> r) + (rem > thr ? 1 : 0);
  }
  return clamp_i8(q);
}

// saturateInt8(floor(v * M / 2^r + 0.5)) for small integer v (|v*M| < 2^24 in the
// reference's float; here integer, exact for |v*M| < 2^31): (v*M + 2^(r-1)) >> r.
TPUCB_HD int mul_rshift_sat8(int32_t v, int32_t M, int r) {
  int32_t t = v * M;
  int32_t q = r == 0 ? t : ((t + (1 << (r - 1))) >> r);
  return clamp_i8(q);
}

TPUCB_HD int rshift_sat8(int32_t v, int r) {
  int32_t q = r == 0 ? v : ((v + (1 << (r - 1))) >> r);
  return clamp_i8(q);
}

TPUCB_HD uint32_t f32_bits(float f) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(f);
#else
  union { float f; uint32_t u; } c;
  c.f = f;
  return c.u;
#endif
}
TPUCB_HD float bits_f32(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  union { float f; uint32_t u; } c;
  c.u = u;
  return c.f;
#endif
}

// Round-to-nearest-even BF16 with the hardware quirk that any exponent-all-ones
// result (inf/NaN, either sign) becomes +max-finite 0x7f7f.
TPUCB_HD uint16_t f32_to_bf16_bits(float f, bool rounding = true) {
  uint32_t u = f32_bits(f);
  if (!rounding) return (uint16_t)(u >> 16);
  u += 0x7fffu + ((u >> 16) & 1u);
  uint16_t h = (uint16_t)(u >> 16);
  if ((h & 0x7f80) == 0x7f80) h = 0x7f7f;
  return h;
}
TPUCB_HD float bf16_bits_to_f32(uint16_t h) { return bits_f32((uint32_t)h << 16); }
TPUCB_HD float bf16_round(float f, bool rounding = true) {
  return bf16_bits_to_f32(f32_to_bf16_bits(f, rounding));
}

#ifdef __CUDACC__
// the part of x that a kind::tf32 product does not read: x - (upper 19 bits of x), exact
__device__ __forceinline__ float4 tf32_remainder(const float4 &x) {
  float4 l;
  l.x = __fsub_rn(x.x, __uint_as_float(__float_as_uint(x.x) & 0xffffe000u));
  l.y = __fsub_rn(x.y, __uint_as_float(__float_as_uint(x.y) & 0xffffe000u));
  l.z = __fsub_rn(x.z, __uint_as_float(__float_as_uint(x.z) & 0xffffe000u));
  l.w = __fsub_rn(x.w, __uint_as_float(__float_as_uint(x.w) & 0xffffe000u));
  return l;
}

// n / d and n % d of an element index: 32-bit arithmetic while it fits, which is always but for tensors of tens of
// gigabytes (a 64-bit division is a call of some forty instructions).
__device__ __forceinline__ unsigned div_rem(size_t &n, unsigned d) {
  if ((n >> 32) == 0) {
    const unsigned a = (unsigned)n, q = a / d;
    n = q;
    return a - q * d;
  }
  const size_t q = n / d;
  const unsigned r = (unsigned)(n - q * d);
  n = q;
  return r;
}

// Programmatic dependent launch (kernels launched through launch_k with the stream-serialisation attribute): a kernel
// lets its successor in the stream be scheduled early (pdl_trigger) and waits for its predecessor's memory operations
// before its own first global access (pdl_wait). Both are no-ops in a kernel launched the ordinary way.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// First statement of every kernel that has no set-up worth overlapping. It waits before it lets its successor in: with
// nothing to overlap, blocks of the successor that stand about early only take room from this kernel's own (MobileNet-v2
// batch 7: 231 us, the other way round 261).
__device__ __forceinline__ void pdl_prologue() {
  pdl_wait();
  pdl_trigger();
}

// Two F32ToBF16 roundings in one conversion instruction: {bf16(hi), bf16(lo)} packed in a word.
// The hardware conversion equals the reference's add-and-shift rule whenever its result is
// finite; a result with an all-ones exponent (inf/NaN in, or rounding past max-finite) takes
// the exact bit rule instead, which also covers the NaN payloads that wrap in the reference.
__device__ __forceinline__ uint32_t bf16x2_round_bits(float lo, float hi) {
  uint32_t p;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p) : "f"(hi), "f"(lo));
  if (((p & 0x7f807f80u) + 0x00800080u) & 0x80008000u)
    p = (uint32_t)f32_to_bf16_bits(lo) | ((uint32_t)f32_to_bf16_bits(hi) << 16);
  return p;
}
// round(v) half-to-even as int32 (saturating at the int32 range, NaN -> 0): the integer that
// F32ToInt8(v, 0) saturates to int8 afterwards.
__device__ __forceinline__ int f32_to_i32_rne(float v) {
  int r;
  asm("cvt.rni.s32.f32 %0, %1;" : "=r"(r) : "f"(v));
  return r;
}

// Per-channel constants of the short form of qdm_requant(acc + bias, M, r):
//   x  = acc * M + c64,  c64 = bias * M + 2^30 (one wide multiply-add)
//   hi = x >> 31 (floor; one funnel shift): adding 2^30 and flooring equals the reference's
//        sign-dependent nudge followed by a division that truncates toward zero, for either sign
//   q  = (hi + rnd - [hi < 0 and r > 0]) >> r,  rnd = 2^(r-1) (0 when r = 0): round half away
//        from zero, as RoundingDivideByPOT does
// With ReLU, negative results become 0 anyway: rnd moves into c64 and the sign term is dropped.
// The value returned is not yet saturated; pack4_sat does that.
struct QdmConst {
  int32_t M, r, rnd, s1; // s1 = 31 when r > 0, else 32: (uint)hi >> s1 is the sign term
  long long c64;
};
__device__ __forceinline__ QdmConst make_qdm_const(int32_t bias, int32_t M, int32_t r, bool relu) {
  QdmConst c;
  c.M = M;
  c.r = r;
  const long long rnd = r > 0 ? (1ll << (r - 1)) : 0ll;
  c.c64 = (long long)bias * (long long)M + (1ll << 30);
  if (relu) c.c64 += rnd << 31;
  c.rnd = (int32_t)rnd;
  c.s1 = r > 0 ? 31 : 32;
  return c;
}
template <bool RELU> __device__ __forceinline__ int qdm_fast(int32_t acc, const QdmConst &q) {
  long long x;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(x) : "r"(acc), "r"(q.M), "l"(q.c64));
  const int32_t hi = (int32_t)__funnelshift_r((uint32_t)x, (uint32_t)(x >> 32), 31);
  if (RELU) return max(hi, 0) >> q.r;
  uint32_t adj;
  asm("shr.u32 %0, %1, %2;" : "=r"(adj) : "r"((uint32_t)hi), "r"((uint32_t)q.s1)); // shifts >= 32 give 0
  return (hi + q.rnd - (int)adj) >> q.r;
}
#endif

// F32ToInt8(v, 0): round half to even on the magnitude, then saturate.
__device__ __forceinline__ int f32_to_int8_rne(float v) {
  // rintf is round-half-even and symmetric in sign, identical to the reference's
  // modf-based rule for every finite v; clamp before the int conversion.
  float r = rintf(v);
  r = fminf(fmaxf(r, -128.0f), 127.0f);
  return (int)r;
}
// F32ToInt8(v, 1): C cast (truncate) then saturate.
__device__ __forceinline__ int f32_to_int8_rz(float v) {
  float r = truncf(v);
  r = fminf(fmaxf(r, -128.0f), 127.0f);
  return (int)r;
}

// d = {c[15:0], sat8(a), sat8(b)}: two int32 saturated to int8 and merged below the low half of c.
__device__ __forceinline__ uint32_t pack_sat_s8(int a, int b, uint32_t c) {
  uint32_t d;
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
// bytes (q0, q1, q2, q3) from low to high, each saturated to [-128, 127]
__device__ __forceinline__ uint32_t pack4_sat(int q0, int q1, int q2, int q3) {
  return pack_sat_s8(q1, q0, pack_sat_s8(q3, q2, 0u));
}
// the same with unsigned saturation to [0, 255]
__device__ __forceinline__ uint32_t pack_sat_u8(int a, int b, uint32_t c) {
  uint32_t d;
  asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
// max(byte, 0) of four packed int8 values: the sign of every byte spread over it by one permute, then one logic operation
__device__ __forceinline__ uint32_t relu_bytes(uint32_t w) {
  uint32_t s;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(s) : "r"(w), "r"(0u), "r"(0xBA98u));
  return w & ~s;
}

// ---- The requantisation on the floating-point pipes --------------------------------------------------------------------
// Exact, with three (ReLU) or four full-rate instructions per value. The integer forms (requant_fast in conv_gemm_i8.cuh)
// need a multiply-high at a quarter of that rate and shifts and multiply-adds at half of it, and their instruction pipes
// bound every convolution with a short K. With s = acc + bias, the reference's
//   hi = floor((s M + 2^30) / 2^31),  q = round half away from zero(hi / 2^r)
// is computed as follows (m = M / 2^31; every quantity scaled by 2^-100, see below).
//   f = the float with the bits of acc + sb: A + s, exact, because one unit of the bit pattern is 1 around A
//   u = fma.rm(f, m, d), d = C + 1/2 - A m: rounds C + s m + 1/2 down to an integer, once: C + hi
// ReLU (A = 2^23; negative s give some f below A and a result <= 0, which the caller clamps): C = 2^23 + 2^(r-1), and
//   v = fma.rm(u, c, e), c = 2^-r, e = -2^23 c: floor((hi + 2^(r-1)) / 2^r)
// else (A = 1.5 2^23, C = kFqC): h = u - C exactly, and
//   v = fma.rn(h, c, 128), c = 2^-r (1 + 2^-23): the factor moves exact ties away from zero and nothing else across one
// The products are scaled so that v's unit is 2^-149, the smallest subnormal: the bits of v ARE the integer (the sign bit
// makes negative ones very negative integers, which saturate), and the packing instruction takes them as they are.
// float_requant (host) checks per channel, from the sum of |weights|, that s and hi stay in range, or that results are saturated
// where they do not, and that d is a float; a layer that fails keeps the integer forms.
struct FloatRequant {
  uint32_t sb; // bias + bits of A
  float m, d, c;
};
constexpr float kFqScale = 7.888609052210118e-31f; // 2^-100
constexpr double kFqC = 8388608.0 + 2097152.0 - 8.0;

#ifdef __CUDACC__
// one value, and four of them packed, each with its channel's constants
template <bool RELU> __device__ __forceinline__ int float_requant1(uint32_t a, const FloatRequant &q) {
  float u, v;
  asm("fma.rm.f32 %0, %1, %2, %3;" : "=f"(u) : "f"(__uint_as_float(a + q.sb)), "f"(q.m), "f"(q.d));
  if (RELU) asm("fma.rm.f32 %0, %1, %2, %3;" : "=f"(v) : "f"(u), "f"(q.c), "f"(q.c * -6.617444900424222e-24f)); // -2^-77: the unit 2^-149 against c's 2^-49
  else asm("fma.rn.f32 %0, %1, %2, %3;" : "=f"(v) : "f"(__fsub_rn(u, (float)kFqC * kFqScale)), "f"(q.c), "f"(__uint_as_float(128u)));
  return __float_as_int(v);
}
template <bool RELU> __device__ __forceinline__ uint32_t float_requant_pack(int v0, int v1, int v2, int v3) {
  if (RELU) return relu_bytes(pack_sat_s8(v1, v0, pack_sat_s8(v3, v2, 0u)));
  return pack_sat_u8(v1, v0, pack_sat_u8(v3, v2, 0u)) ^ 0x80808080u;
}
// two 32-bit values as a register pair
__device__ __forceinline__ unsigned long long pack_b32x2(uint32_t lo, uint32_t hi) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
  return d;
}
// Two values of one channel: the packed multiply-adds round each half as the single ones do and take one issue slot for two.
// The constants are held as pairs whose making the compiler may not repeat (it did, before some uses).
__device__ __forceinline__ unsigned long long hold_pair(float v) {
  unsigned long long d;
  asm volatile("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(v));
  return d;
}
struct FloatRequantShared { // what the channels share without ReLU
  unsigned long long k, h;
  __device__ __forceinline__ void set() {
    k = hold_pair(-(float)kFqC * kFqScale);
    h = hold_pair(__uint_as_float(128u));
  }
};
template <bool RELU> struct FloatRequantPairs {
  uint32_t sb;
  unsigned long long m, d, c, e; // e: ReLU the last addend, else unused
  __device__ __forceinline__ void set(const FloatRequant &q) {
    sb = q.sb;
    m = hold_pair(q.m);
    d = hold_pair(q.d);
    c = hold_pair(q.c);
    if (RELU) e = hold_pair(q.c * -6.617444900424222e-24f); // as above
  }
};
template <bool RELU>
__device__ __forceinline__ void float_requant2(uint32_t a0, uint32_t a1, const FloatRequantPairs<RELU> &q, const FloatRequantShared &s, int &v0,
                                               int &v1) {
  unsigned long long f = pack_b32x2(a0 + q.sb, a1 + q.sb);
  asm("fma.rm.f32x2 %0, %0, %1, %2;" : "+l"(f) : "l"(q.m), "l"(q.d));
  if (RELU) {
    asm("fma.rm.f32x2 %0, %0, %1, %2;" : "+l"(f) : "l"(q.c), "l"(q.e));
  } else {
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(f) : "l"(s.k));
    asm("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(f) : "l"(q.c), "l"(s.h));
  }
  asm("mov.b64 {%0, %1}, %2;" : "=r"(v0), "=r"(v1) : "l"(f));
}
// four values of one channel, packed
template <bool RELU>
__device__ __forceinline__ uint32_t float_requant4(uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, const FloatRequantPairs<RELU> &q,
                                                   const FloatRequantShared &s) {
  int v0, v1, v2, v3;
  float_requant2<RELU>(a0, a1, q, s, v0, v1);
  float_requant2<RELU>(a2, a3, q, s, v2, v3);
  return float_requant_pack<RELU>(v0, v1, v2, v3);
}
#endif

// sign-extended byte J of a word in one byte-permute: in prmt's default mode bit 3 of a selector
// nibble replicates the sign of the selected byte (the __byte_perm intrinsic masks that bit off,
// hence the inline PTX).
template <int J> __device__ __forceinline__ int sext_byte(uint32_t w) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(w), "r"(0u), "r"((uint32_t)(J | ((8 | J) << 4) | ((8 | J) << 8) | ((8 | J) << 12))));
  return (int)d;
}

} // namespace tpucb
