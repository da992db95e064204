// FP64 vectors times fixed FP64 matrices on the integer pipe.
//
// One FP64 FMA holds its scheduler 64 to 76 cycles on this GPU, a 32 x 32 ->
// 64 integer multiply-add about 2.  A matrix-vector product whose matrix is
// known beforehand runs in block fixed point instead: a vector's elements
// become 56-bit integers under the exponent of its largest element (exact for
// elements within 2^3 of it), the matrix likewise under its own, both cut into
// two 28-bit limbs; a product is then three multiply-adds into two 64-bit sums
// (the low x low part, below 2^-56, is left out), and each sum becomes one
// FP64 number at the end.  The error per output is at most n 2^-55 of
// max|K| max|x| (n terms), against about n 2^-53 of the same for the FP64 sum.
// A vector with a NaN or infinity gives NaN.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

#include "fx64.cuh"

namespace cr {

constexpr int kLimbBits = 28;
constexpr int kLimbMask = (1 << kLimbBits) - 1;
constexpr int kFixedNan = 0x7ff;  // exponent field of a vector with a NaN or infinity

struct Limbs {
  int hi, lo;  // hi 2^28 + lo, 0 <= lo < 2^28
};

#ifdef __CUDACC__
__device__ __forceinline__ int exponent_field(double x) { return (int)(((unsigned)__double2hiint(x) >> 20) & 0x7ffu); }

// x / 2^(emax - 1078 + guard) as an integer below 2^(56 - guard) (emax: the
// largest exponent field of the vector; subnormals count as 0)
__device__ __forceinline__ int64_t to_fixed(double x, int emax, int guard) {
  const unsigned h = (unsigned)__double2hiint(x);
  const int e = (int)((h >> 20) & 0x7ffu), sh = emax - e;
  uint64_t m = ((uint64_t)((h & 0xfffffu) | 0x100000u) << 32) | (unsigned)__double2loint(x);
  m = (e == 0 || sh > 55) ? 0 : (m << 3) >> (sh + guard);
  return (h >> 31) ? -(int64_t)m : (int64_t)m;
}
__device__ __forceinline__ Limbs to_limbs(int64_t v) {
  return Limbs{(int)(v >> kLimbBits), (int)v & kLimbMask};
}

// a running sum of products
struct FixedSum {
  int64_t hh, cr;
  __device__ __forceinline__ void add(Limbs x, Limbs k) {
    hh += (int64_t)x.hi * k.hi;
    cr += (int64_t)x.hi * k.lo;
    cr += (int64_t)x.lo * k.hi;
  }
  __device__ __forceinline__ void sub(Limbs x, Limbs k) {
    hh -= (int64_t)x.hi * k.hi;
    cr -= (int64_t)x.hi * k.lo;
    cr -= (int64_t)x.lo * k.hi;
  }
  __device__ __forceinline__ int64_t value() const { return hh + ((cr + (1 << (kLimbBits - 1))) >> kLimbBits); }
};

// S 2^ex as FP64
__device__ __forceinline__ double from_fixed(int64_t S, int ex) {
  const uint64_t a = (uint64_t)(S < 0 ? -S : S);
  const int lz = __clzll((long long)a), e = ex - lz + 63;
  const double r = fx::pack((uint64_t)S & 0x8000000000000000ull, e, a << lz);
  if (a == 0 || e < -1021) return 0.0;
  return e > 1022 ? __longlong_as_double(0x7ff0000000000000ll) : r;
}
#endif

// Guard bits of a product of n terms: two folded elements sum below
// 2^(57 - guard), so both 64-bit sums stay in range for any matrix.
inline int fixed_guard(int n) { return n <= 20 ? 0 : n <= 40 ? 1 : n <= 80 ? 2 : 3; }

// Host side: a matrix block as limbs under the exponent of its largest entry;
// sum_l K[l] x[l] = value 2^(ek + emax - 1078 + guard) with x under emax.
inline int fixed_exponent(const std::vector<double>& K) {
  double m = 0.0;
  for (double v : K) m = std::max(m, std::fabs(v));
  return m > 0.0 ? std::ilogb(m) + 1 : -1000;
}
inline void fixed_limbs(const std::vector<double>& K, int ek, std::vector<Limbs>& out) {
  for (double v : K) {
    const long long n = std::llrint(std::ldexp(v, 56 - ek));
    const long long lo = n & kLimbMask;
    out.push_back(Limbs{(int)((n - lo) >> kLimbBits), (int)lo});
  }
}

}  // namespace cr
