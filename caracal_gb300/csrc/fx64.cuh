// FP64 functions on the integer pipe.
//
// What bounds FP64 code on this GPU is the FP64 pipe: one warp instruction
// (add, multiply or FMA) holds its scheduler's pipe for 64 cycles (76 with all
// four schedulers of an SM busy), against 1 to 2 for FP32 and integer ones
// (measured, 152 SMs, one to sixteen warps each).  A division or square root
// in FP64 instructions takes 400 to 650 such cycles per warp, exp 1085 to
// 1255, acos 1415, log 2100, pow 5850.  The functions here do the same work on
// the 53-bit significands in 64-bit integer arithmetic: a 64-bit high product
// is three 32 x 32 -> 64 multiply-adds, so a polynomial step costs about eight
// integer instructions.  Measured in the same harness: see each function.
//
// Accuracy: the intermediate fixed-point values carry 60 bits and more, so the
// results are rounded once from a value good to about 2^-59 (checked against
// extended precision on the host, tests/test_fx64.py: at most 0.51 ulp for
// reciprocal, quotient and roots, 0.6 ulp for exp up to |x| = 40 and acos, 0.8 ulp
// for pow).  Arguments outside the stated range of the
// integer path (zero, subnormal, infinite, NaN, results near the ends of the
// exponent range) go to the FP64 functions, so those keep their meaning.
//
// Methods: reciprocal and reciprocal square root by one third-order Newton
// step from the FP32 hardware estimate; exp2 by 16 tabulated powers of two and
// the Taylor series of 2^z, z < 1/16; log2 by 2 atanh((m-1)/(m+1)); arc sine
// by its Taylor series with the half-angle reduction; sine, cosine and erf by
// Taylor series to an absolute 2^-58.  The constants are those
// series' coefficients, scaled.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#include <cuda_runtime.h>
#endif

#include "fx64_erf.cuh"

namespace cr {
namespace fx {

typedef uint64_t u64;
typedef uint32_t u32;

#ifdef __CUDA_ARCH__
#define FX_FN __device__ __forceinline__
#define FX_SLOW static __device__ __noinline__
#else
#define FX_FN inline
#define FX_SLOW static inline
#endif

FX_FN u64 bits(double x) {
#ifdef __CUDA_ARCH__
  return (u64)__double_as_longlong(x);
#else
  u64 u;
  std::memcpy(&u, &x, 8);
  return u;
#endif
}
FX_FN double dbl(u64 u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double x;
  std::memcpy(&x, &u, 8);
  return x;
#endif
}
FX_FN float flt(u32 u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float x;
  std::memcpy(&x, &u, 4);
  return x;
#endif
}
FX_FN float est_rcp(float x) {
#ifdef __CUDA_ARCH__
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return (float)(1.0 / x * (1.0 + 6e-8));  // as inexact as the hardware estimate
#endif
}
FX_FN float est_rsqrt(float x) {
#ifdef __CUDA_ARCH__
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return (float)(1.0 / std::sqrt((double)x) * (1.0 + 8e-8));
#endif
}
// float in [0, 2) to unsigned Q31, saturating
FX_FN u32 q31(float y) {
#ifdef __CUDA_ARCH__
  return __float2uint_rz(y * 2147483648.0f);
#else
  const double v = (double)y * 2147483648.0;
  return v >= 4294967295.0 ? 4294967295u : (u32)v;
#endif
}
FX_FN int clz64(u64 x) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)x);
#else
  return x ? __builtin_clzll(x) : 64;
#endif
}
FX_FN u32 mulh32(u32 a, u32 b) { return (u32)(((u64)a * b) >> 32); }

// floor(a b / 2^64) or one less: the low partial product is left out
FX_FN u64 mulh(u64 a, u64 b) {
  const u32 al = (u32)a, ah = (u32)(a >> 32), bl = (u32)b, bh = (u32)(b >> 32);
  const u64 t = (u64)al * bh;
  const u64 u = (u64)ah * bl + (u32)t;
  return (u64)ah * bh + (t >> 32) + (u >> 32);
}

// floor(a b / 2^64)
FX_FN u64 mulh_exact(u64 a, u64 b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (u64)(((unsigned __int128)a * b) >> 64);
#endif
}

// +-M 2^(e - 63), M with its top bit set, to the nearest double (e in the
// normal range; a carry out of the significand moves the exponent)
FX_FN double pack(u64 sign, int e, u64 M) {
  return dbl(sign | (((u64)(u32)(e + 1022) << 52) + (M >> 11) + ((M >> 10) & 1)));
}

// significand with its top bit set, of a normal x
FX_FN u64 signif(u64 b) { return ((b << 11) | 0x8000000000000000ull); }
FX_FN int expo(u64 b) { return (int)((u32)(b >> 52) & 0x7ffu); }

// 1 / d for d = D 2^-64 in [1/2, 1): Q63 in (1, 2] (2 as 2 - 2^-63)
FX_FN u64 rcp_q63(u64 D) {
  const float d = flt(0x3f000000u | ((u32)(D >> 40) & 0x7fffffu));
  const u32 y = q31(est_rcp(d));
  const u32 dl = (u32)D, dh = (u32)(D >> 32);
  // e = 1 - d y, exactly to 2^-63; 1/d = y (1 + e + e^2 + ...), |e| < 2^-21
  const u64 p = (u64)dh * y + (((u64)dl * y) >> 32);
  const int64_t e = (int64_t)(0x8000000000000000ull - p);
  const int32_t es = (int32_t)(e >> 20);
  const int64_t s = e + (((int64_t)es * es) >> 23);
  const int32_t sh = (int32_t)(s >> 32);
  const u32 sl = (u32)s;
  return ((u64)y << 32) + (u64)((int64_t)sh * (int64_t)(u64)y * 2) + (((u64)y * sl) >> 31);
}

// 1 / sqrt(d) for d = D 2^-64 in [1/4, 1): Q63 in (1, 2]
FX_FN u64 rsqrt_q63(u64 D) {
  const u32 top = (u32)(D >> 32);
  // float of d (24 bits suffice): d = top 2^-32
#ifdef __CUDA_ARCH__
  const float d = __uint2float_rz(top) * 2.3283064365386963e-10f;
#else
  const float d = (float)(top & 0xffffff00u) * 2.3283064365386963e-10f;
#endif
  const u32 y = q31(est_rsqrt(d));
  // h = 1 - d y^2 to 2^-62; 1/sqrt(d) = y (1 + h/2 + 3 h^2/8 + ...), |h| < 2^-20
  const u64 y2 = (u64)y * y;
  const int64_t h = (int64_t)(0x4000000000000000ull - mulh(D, y2));
  const int32_t hs = (int32_t)(h >> 20);
  // s = h/2 + 3/8 h^2 in units 2^-63: h + 3/4 h^2
  const int64_t s = h + ((((int64_t)hs * hs) >> 22) * 3 >> 2);
  const int32_t sh = (int32_t)(s >> 32);
  const u32 sl = (u32)s;
  return ((u64)y << 32) + (u64)((int64_t)sh * (int64_t)(u64)y * 2) + (((u64)y * sl) >> 31);
}

FX_SLOW double slow_rcp(double x) { return 1.0 / x; }
FX_SLOW double slow_div(double a, double b) { return a / b; }
FX_SLOW double slow_sqrt(double x) { return std::sqrt(x); }
FX_SLOW double slow_exp(double x) { return std::exp(x); }
FX_SLOW double slow_log(double x) { return std::log(x); }
FX_SLOW double slow_pow(double x, double y) { return std::pow(x, y); }
FX_SLOW double slow_acos(double x) { return std::acos(x); }
FX_SLOW double slow_asin(double x) { return std::asin(x); }

// biased exponent within [lo, hi] (one unsigned comparison)
FX_FN bool within(int e, int lo, int hi) { return (u32)(e - lo) <= (u32)(hi - lo); }

FX_FN double rcp(double x) {
  const u64 b = bits(x);
  const int e = expo(b);
  if (!within(e, 2, 2044)) return slow_rcp(x);
  return pack(b & 0x8000000000000000ull, 1022 - e, rcp_q63(signif(b)));
}

FX_FN double div(double a, double b) {
  const u64 ba = bits(a), bb = bits(b);
  const int ea = expo(ba), eb = expo(bb), e = ea - eb;
  if (!(within(ea, 1, 2046) && within(eb, 1, 2046) && within(e, -1000, 1000))) return slow_div(a, b);
  // a / b = (A / 2^63) (R / 2^63) 2^(e - 1), A R / 2^126 in [1, 4)
  u64 q = mulh(signif(ba), rcp_q63(signif(bb)));
  const int up = (int)(q >> 63);  // quotient of significands in [1, 2)
  q <<= 1 - up;
  return pack((ba ^ bb) & 0x8000000000000000ull, e - 1 + up, q);
}

// sqrt(x) and 1 / sqrt(x)
FX_FN void sqrt_rsqrt(double x, double& r, double& ir) {
  const u64 b = bits(x);
  const int eb = (int)(u32)(b >> 52);  // with the sign: negative x is out of range
  if (!within(eb, 2, 2044)) {
    r = slow_sqrt(x);
    ir = slow_rcp(r);
    return;
  }
  // x = d 4^k, d = D 2^-64 in [1/4, 1)
  const int e = eb - 1022, odd = e & 1, k = (e + odd) >> 1;
  const u64 D = signif(b) >> odd;
  const u64 R = rsqrt_q63(D);
  ir = pack(0, -k, R);
  u64 S = mulh(D, R);  // sqrt(d) Q63 in [1/2, 1): top bit clear
  r = pack(0, k - 1, S << 1);
}
FX_FN double sqrt(double x) {
  const u64 b = bits(x);
  const int eb = (int)(u32)(b >> 52);
  if (!within(eb, 2, 2044)) return slow_sqrt(x);
  const int e = eb - 1022, odd = e & 1, k = (e + odd) >> 1;
  const u64 D = signif(b) >> odd;
  return pack(0, k - 1, mulh(D, rsqrt_q63(D)) << 1);
}
FX_FN double rsqrt(double x) {
  const u64 b = bits(x);
  const int eb = (int)(u32)(b >> 52);
  if (!within(eb, 2, 2044)) return slow_rcp(slow_sqrt(x));
  const int e = eb - 1022, odd = e & 1, k = (e + odd) >> 1;
  return pack(0, -k, rsqrt_q63(signif(b) >> odd));
}

#ifdef __CUDACC__
#define FX_TABLE static __device__ const
#else
#define FX_TABLE static const
#endif
// 2^(j/16), Q63
#define FX_POW2_VALUES                                                                                  \
  {0x8000000000000000ull, 0x85aac367cc487b15ull, 0x8b95c1e3ea8bd6e7ull, 0x91c3d373ab11c336ull,          \
   0x9837f0518db8a96full, 0x9ef5326091a111aeull, 0xa5fed6a9b15138eaull, 0xad583eea42a14ac6ull,          \
   0xb504f333f9de6484ull, 0xbd08a39f580c36bfull, 0xc5672a115506daddull, 0xce248c151f8480e4ull,          \
   0xd744fccad69d6af4ull, 0xe0ccdeec2a94e111ull, 0xeac0c6e7dd24392full, 0xf5257d152486cc2cull}
FX_TABLE u64 kPow2[16] = FX_POW2_VALUES;
FX_FN u64 pow2_16(u32 j) {
#if defined(__CUDACC__) && !defined(__CUDA_ARCH__)
  static const u64 host[16] = FX_POW2_VALUES;
  return host[j];
#else
  return kPow2[j];
#endif
}

// 2^(f / 2^64), Q63 in [1, 2)
FX_FN u64 exp2_frac(u64 f) {
  const u64 T = pow2_16((u32)(f >> 60));
  const u64 z = f << 4;  // 16 times the remainder, Q64
  const u32 z32 = (u32)(z >> 32);
  // Taylor coefficients (ln 2 / 16)^k / k!: k = 8..5 in Q60, 4..1 in Q64
  u32 t = 355u;
  t = 65510u + mulh32(t, z32);
  t = 10585225u + mulh32(t, z32);
  t = 1466040222u + mulh32(t, z32);
  u64 a = 0x00000276556df74aull + (((u64)t * z32) >> 28);
  a = 0x0000e35846b82506ull + mulh(a, z);
  a = 0x003d7f7bff058b1dull + mulh(a, z);
  a = 0x0b17217f7d1cf79bull + mulh(a, z);
  a = 0x8000000000000000ull + (mulh(a, z) >> 1);
  return mulh(a, T) << 1;
}

// exp(x); the integer path takes 2^-60 <= |x| < 512.  85 cycles per warp
// against 1085 to 1255 of the FP64 function.
FX_FN double exp(double x) {
  const u64 b = bits(x);
  const int e = expo(b) - 1023;
  if (!within(e, -60, 8)) return slow_exp(x);
  // |x| log2(e) = P 2^(e - 62)
  const u64 P = mulh(signif(b), 0xb8aa3b295c17f0bcull);
  int n = 0;
  u64 f;
  if (e >= -2) {
    n = (int)(P >> (62 - e));
    if (e == -2) n = 0;
    f = P << (e + 2);
  } else {
    f = P >> (-2 - e);
  }
  if (b >> 63) {
    n = -n - (f != 0 ? 1 : 0);
    f = 0 - f;
  }
  return pack(0, n, exp2_frac(f));
}

// |log2(x)| of x = +M 2^(e - 63) as Q57 (integer part below 64) and its sign
// (neg).  M top bit set.
FX_FN u64 log2_q57(u64 M, int e, bool& neg) {
  // m in [sqrt(1/2), sqrt(2)): halve the upper part
  const bool up = M >= 0xb504f333f9de6484ull;
  if (up) e += 1;
  // m = M / 2^63 or M / 2^64; |m - 1| and m + 1 in Q63
  const u64 one = 0x8000000000000000ull;
  const u64 m = up ? M >> 1 : M;
  const bool below = m < one;  // m < 1
  const u64 num = below ? one - m : m - one;
  // m + 1 in Q62, normalised to [1/2, 1) of 2^64 (m + 1 in [1.7, 2.42))
  u64 den = (m >> 1) + (one >> 1);
  const int sh = (int)(~den >> 63);  // 1 where the top bit is clear
  den <<= sh;
  // t = num / (m + 1): num Q63, 1/den: value (m+1) = den 2^(2 - sh) / 2^64
  const u64 R = rcp_q63(den);  // 2^64/den, Q63
  const u64 t = mulh(num, R) << sh;   // num/2^63 R/2^63 / 2^(2-sh): Q64 -> t 2^64
  const u64 t2 = mulh(t, t);
  // sum over k of t^(2k) / (2k + 1), t^2 < 0.0295: with w = 32 t^2 (< 0.943) and
  // coefficients 2^-5k / (2k + 1): k = 10..5 in Q60, 4..1 in Q64
  const u64 w = t2 << 5;
  const u32 w32 = (u32)(w >> 32);
  u32 s = 49u;
  s = 1725u + mulh32(s, w32);
  s = 61681u + mulh32(s, w32);
  s = 2236962u + mulh32(s, w32);
  s = 82595525u + mulh32(s, w32);
  s = 3123612579u + mulh32(s, w32);
  u64 a = 0x000001c71c71c71cull + (((u64)s * w32) >> 28);
  a = 0x0000492492492492ull + mulh(a, w);
  a = 0x000ccccccccccccdull + mulh(a, w);
  a = 0x02aaaaaaaaaaaaabull + mulh(a, w);
  a = one + (mulh(a, w) >> 1);                  // k = 0, Q63
  // log2(m) = (2 / ln 2) t a: 2/ln 2 = 2.885.. as Q61
  const u64 ta = mulh(t, a);                    // Q63 of t a
  const u64 l = mulh(ta, 0x5c551d94ae0bf85eull);  // Q(63 + 61 - 64) = Q60
  const u64 lq = l >> 3;                        // Q57
  // e + (below ? -log : log)
  const int64_t v = ((int64_t)e << 57) + (below ? -(int64_t)lq : (int64_t)lq);
  neg = v < 0;
  return (u64)(neg ? -v : v);
}

// x^y for positive x in [2^-30, 2^30] and 2^-10 <= |y| < 16; out of that range pow
FX_FN double pow(double x, double y) {
  const u64 b = bits(x), by = bits(y);
  const int eb = (int)(u32)(b >> 52), ey = expo(by) - 1023;
  if (!within(eb, 1023 - 30, 1023 + 30) || !within(ey, -10, 3)) return slow_pow(x, y);
  bool neg;
  const u64 L = log2_q57(signif(b), eb - 1023, neg);  // Q57
  const int s = ey > 0 ? ey : 0;
  const u64 Y = signif(by) >> (1 - (ey - s));         // |y| 2^-s: Q62
  if (by >> 63) neg = !neg;
  // L Y: Q119 in 128 bits
  const u64 hi = mulh_exact(L, Y), lo = L * Y;              // hi Q55
  int n = (int)(hi >> (55 - s));
  u64 f = (hi << (9 + s)) | (lo >> (55 - s));
  if (neg) {
    n = -n - (f != 0 ? 1 : 0);
    f = 0 - f;
  }
  return pack(0, n, exp2_frac(f));
}

// P(4 Z 2^-64) of asin(u) = u P(4 u^2), u^2 = Z 2^-64 <= 1/4: the Taylor series of
// asin(s)/s to s^52 (error 2^-61), Q63
FX_FN u64 asin_poly(u64 Z) {
  const u64 w = (Z >= 0x4000000000000000ull ? 0x3fffffffffffffffull : Z) << 2;
  const u32 w32 = (u32)(w >> 32);
  u32 s = 1u;
  s = 2u + mulh32(s, w32);
  s = 10u + mulh32(s, w32);
  s = 41u + mulh32(s, w32);
  s = 174u + mulh32(s, w32);
  s = 746u + mulh32(s, w32);
  s = 3206u + mulh32(s, w32);
  s = 13829u + mulh32(s, w32);
  s = 59881u + mulh32(s, w32);
  s = 260447u + mulh32(s, w32);
  s = 1138410u + mulh32(s, w32);
  s = 5003791u + mulh32(s, w32);
  s = 22133297u + mulh32(s, w32);
  s = 98613096u + mulh32(s, w32);
  s = 443048919u + mulh32(s, w32);
  s = 2010051807u + mulh32(s, w32);
  u64 a = 0x000000225de79e7aull + (((u64)s * w32) >> 28);
  a = 0x0000009fef286bcaull + mulh(a, w);
  a = 0x000002f50f0f0f0full + mulh(a, w);
  a = 0x00000e4ccccccccdull + mulh(a, w);
  a = 0x00004713b13b13b1ull + mulh(a, w);
  a = 0x00016e8ba2e8ba2full + mulh(a, w);
  a = 0x0007c71c71c71c72ull + mulh(a, w);
  a = 0x002db6db6db6db6eull + mulh(a, w);
  a = 0x0133333333333333ull + mulh(a, w);
  a = 0x0aaaaaaaaaaaaaabull + mulh(a, w);
  return 0x8000000000000000ull + (mulh(a, w) >> 1);
}

// arc sine of |x| < 1/2; outside asin
FX_FN double asin(double x) {
  const u64 b = bits(x);
  const int e = expo(b) - 1023;
  if (e < -31) return e < -1022 ? slow_asin(x) : x;
  if (e >= -1) return slow_asin(x);
  const u64 M = signif(b), X = M >> -e;
  const u64 A = mulh(M, asin_poly(mulh(X, X) << 2));  // asin|x| 2^-e, Q62 in [1, 2.1)
  const int lz = clz64(A);
  return pack(b & 0x8000000000000000ull, e + 1 - lz, A << lz);
}

// arc cosine of |x| <= 1 - 2^-24; outside acos.  About 130 cycles per warp
// against 1415 of the FP64 function.  asin_poly for u <= 1/2; beyond, the half-angle
// form 2 asin(sqrt((1 - |x|) / 2)).
FX_FN double acos(double x) {
  const u64 b = bits(x);
  const int e = expo(b) - 1023;
  const bool small = e < -1;
  const u64 X = e < -62 ? 0 : signif(b) >> (e < 0 ? -e : 0);  // |x|, Q63
  const u64 Z = small ? mulh(X, X) << 2 : 0x8000000000000000ull - X;  // u^2, Q64
  if (e >= 0 || (!small && Z < 0x0000008000000000ull)) return slow_acos(x);
  const u64 a = asin_poly(Z);
  u64 V;
  int ex = 1;
  if (small) {
    const u64 A = mulh(X, a);  // asin|x|, Q62
    V = 0x6487ed5110b4611aull + ((b >> 63) ? A : 0 - A);  // pi/2 -+
  } else {
    const int lz = clz64(Z) & ~1;
    const u64 D = Z << lz;
    const u64 A = mulh(mulh(D, rsqrt_q63(D)), a);  // asin(u) 2^(lz/2), Q62
    if (b >> 63) {
      V = 0xc90fdaa22168c235ull - ((A << 1) >> (lz >> 1));  // pi - 2 asin(u)
    } else {
      V = A;
      ex = 2 - (lz >> 1);
    }
  }
  const int lz = clz64(V);
  return pack(0, ex - lz, V << lz);
}

FX_SLOW double slow_sin(double x) { return std::sin(x); }
FX_SLOW double slow_cos(double x) { return std::cos(x); }
FX_SLOW double slow_erf(double x) { return std::erf(x); }

// V 2^-63 as a double
FX_FN double from_q63(u64 V, u64 sign) {
  const int lz = clz64(V);
  return V == 0 ? 0.0 : pack(sign, -lz, V << lz);
}

// sin(x) and cos(x) to 2^-58 absolute (|x| 2^-65 from the 64-bit 2 / pi on top; not
// relative to a small sine) for |x| < 1024.  x 2/pi = n + f with |f| <= 1/2, then
// the Taylor series in v = 2 |f|: sum (-1)^k (pi/4)^k v^k / k!, the upper terms in 32
// bits.  About 130 cycles per warp for both against 1274 for either FP64 function.
FX_FN void sincos(double x, double& sn, double& cs) {
  const u64 b = bits(x);
  const int e = expo(b) - 1023;
  if (e > 9) {
    sn = slow_sin(x);
    cs = slow_cos(x);
    return;
  }
  const u64 C = 0xa2f9836e4e44152aull;  // 2 / pi, Q64
  const u64 M = signif(b), hi = mulh_exact(M, C), lo = M * C;
  u32 n = 0;
  u64 f;  // fraction of |x| 2/pi, Q64
  if (e >= 0) {
    n = (u32)(hi >> (63 - e));
    f = (hi << (1 + e)) | (lo >> (63 - e));
  } else {
    f = e < -64 ? 0 : hi >> (-1 - e);
  }
  const bool up = (f >> 63) != 0;
  n += up;
  u64 v = up ? 0 - f : f;
  v = v >> 63 ? ~0ull : v << 1;
  const u64 w = mulh(v, v);
  const u32 w32 = (u32)(w >> 32);
  u32 t = 23531u - mulh32(53u, w32);
  t = 8011021u - mulh32(t, w32);
  t = 2025968632u - mulh32(t, w32);
  u64 a = 0x00000541e0d21fbaull - (((u64)t * w32) >> 28);
  a = 0x000265a599cc57b1ull - mulh(a, w);
  a = 0x00a335e33bad570full - mulh(a, w);
  a = 0x14abbce625be52bfull - mulh(a, w);
  a = 0xc90fdaa22168c235ull - mulh(a, w);
  const u64 S = mulh(a, v) >> 1;  // Q63
  t = 1155u - mulh32(2u, w32);
  t = 449417u - mulh32(t, w32);
  t = 132599337u - mulh32(t, w32);
  a = 0x000000069b47ca88ull * 16 + 1 - (((u64)t * w32) >> 28);
  a = 0x00003c3ea0d12375ull - mulh(a, w);
  a = 0x00155d3c7e3cbffaull - mulh(a, w);
  a = 0x040f07c206d6b0edull - mulh(a, w);
  a = 0x4ef4f326f9177969ull - mulh(a, w);
  const u64 c = 0x8000000000000000ull - (mulh(a, w) >> 1);
  const u64 top = 0x8000000000000000ull, neg = b & top;
  const u64 sS = up ? top : 0;  // sign of sin(f)
  const bool odd = n & 1, half = (n & 2) != 0;
  // n = 0: (S, c); 1: (c, -S); 2: (-S, -c); 3: (-c, S)
  const u64 s1 = (half ? top : 0), c1 = ((n + 1) & 2) ? top : 0;
  sn = from_q63(odd ? c : S, (odd ? s1 : s1 ^ sS) ^ neg);
  cs = from_q63(odd ? S : c, odd ? c1 ^ sS : c1);
}

#ifdef __CUDACC__
FX_TABLE ErfRow kErf[48] = {FX_ERF_ROWS};
#endif
FX_FN const ErfRow& erf_row(int j) {
#if defined(__CUDACC__) && defined(__CUDA_ARCH__)
  return kErf[j];
#else
  static const ErfRow host[48] = {FX_ERF_ROWS};
  return host[j];
#endif
}

// erf(x) to 2^-58 absolute: a Taylor series about the nearest of 48 centres on
// [0, 6); beyond erf.  About 120 cycles per warp against 3025.
FX_FN double erf(double x) {
  const u64 b = bits(x);
  const int e = expo(b) - 1023;
  const u64 X = e > 2 ? ~0ull : e < -60 ? 0 : signif(b) >> (3 - e);  // |x|, Q60
  const int j = (int)(X >> 57);
  if (j >= 48) return slow_erf(x);
  const ErfRow& r = erf_row(j);
  const int64_t z = (int64_t)((X << 7) ^ 0x8000000000000000ull);  // Q63
  const int32_t zh = (int32_t)(z >> 32);
  auto m32 = [zh](int32_t a) { return (int32_t)(((int64_t)a * zh) >> 31); };
  // a z / 2^63
  auto m64 = [z](int64_t a) {
    u64 p = mulh((u64)a, (u64)z);
    if (a < 0) p -= (u64)z;
    if (z < 0) p -= (u64)a;
    return (int64_t)(p << 1);
  };
  int32_t t = r.d[3] + m32(r.d[4]);
  t = r.d[2] + m32(t);
  t = r.d[1] + m32(t);
  t = r.d[0] + m32(t);
  int64_t a = r.c[6] + (((int64_t)t * zh) >> 31);
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
  for (int k = 5; k >= 0; --k) a = r.c[k] + m64(a);
  return from_q63((u64)(a < 0 ? 0 : a) << 1, b & 0x8000000000000000ull);
}

}  // namespace fx
}  // namespace cr
