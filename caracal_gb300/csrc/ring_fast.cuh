// Free ring polymer of P = 2 M beads (M = 4, 8, 16, 32) by fast cosine
// transforms in fixed point, on the integer pipe.
//
// Caracal's map on the distinct beads x_0 .. x_M is y = T_M(z) 2/P with
// z_k = (w_k / 2) D_k T_M(s)_k, s_0 = x_0, s_M = x_M, s_l = 2 x_l, w_0 = w_M = 1,
// else 2, and the type-I cosine transform
//   T_M(s)_k = s_0 + (-1)^k s_M + sum_{l=1}^{M-1} s_l cos(pi k l / M);
// T_M splits by the parity of k into T_{M/2} and a type-III transform of size
// M/2, which follows Lee's recursion (B. G. Lee, IEEE Trans. ASSP 32 (1984)
// 1243).  For M = 32 that is 49 multiplications and 165 additions instead of
// 545 multiplications for each of the four parity-split matrix products.  What
// bounds it here is the integer pipe: an addition is two instructions, a
// product by a 64-bit constant about eight, against 64 to 76 cycles for either
// in FP64.
//
// A lane transforms one coordinate of one array (even lanes q, odd lanes p, the
// two of a coordinate next to each other) as 64-bit integers under one
// exponent; q enters relative to its bead-0 value (the constant vector is mode
// 0, which K1 keeps and K2 drops) and normalised to its spread, so the products
// round on bead spreads.  The elements take 58 - log2(M) bits: with |x| < 2^b
// the modes' magnitudes sum to at most 2 M^1.5 2^b, both terms of z together to
// as much again after their halving, and Lee's intermediates stay within twice
// such a sum, below 2^63.
#pragma once
#include "fixed_map.cuh"

namespace cr {

// Mode tables of one engine: A_k = (w_k / 2) cos(w_k dt), B_k = (w_k / 2)
// sin(w_k dt) / w_k and C_k = -(w_k / 2) w_k sin(w_k dt) as Q62 under the
// exponents 0, eb, ec.
struct FastRing {
  const int64_t* tab;  // [3][M + 1]
  int eb, ec;
};

#ifdef __CUDACC__
namespace ring {

struct LeeFactor {
  int whole;
  uint64_t part;  // Q64
};
// 1 / (2 cos(pi (2k+1) / (2N))) for N = 2, 4, 8, 16 at [N/2 - 1 + k]
__device__ constexpr LeeFactor lee(int i) {
  constexpr LeeFactor t[15] = {{0, 0xb504f333f9de6484ull}, {0, 0x8a8bd3ded9c4a5ffull}, {1, 0x4e7ae9144f0fbc8cull}, {0, 0x8281f68be5d29734ull}, {0, 0x99f1bd0f00b9ef95ull}, {0, 0xe664d77d8c6ac20dull}, {2, 0x901b3a0e7684f241ull}, {0, 0x809e8ce30ecb89f8ull}, {0, 0x85c2781f5f0af1e0ull}, {0, 0x91233e8832d3a10aull}, {0, 0xa5961cc5df1e33cdull}, {0, 0xc9c4805bea10819aull}, {1, 0x0f8892a4eced8d66ull}, {1, 0xb8f24b0406140cb6ull}, {5, 0x19e4e0394e376bd3ull}};
  return t[i];
}

// x c / 2^64 for c in [0, 2^64)
__device__ __forceinline__ int64_t mul_q64(int64_t x, uint64_t c) {
  const uint64_t r = fx::mulh((uint64_t)x, c);
  return (int64_t)(x < 0 ? r - c : r);
}
// x c / 2^64, both signed
__device__ __forceinline__ int64_t mul_s64(int64_t x, int64_t c) {
  uint64_t r = fx::mulh((uint64_t)x, (uint64_t)c);
  if (x < 0) r -= (uint64_t)c;
  if (c < 0) r -= (uint64_t)x;
  return (int64_t)r;
}
template <int I>
__device__ __forceinline__ int64_t mul_lee(int64_t x) {
  constexpr LeeFactor f = lee(I);
  return mul_q64(x, f.part) + x * f.whole;
}

template <int N>
struct Dct3 {
  template <int K>
  static __device__ __forceinline__ void outs(const int64_t (&G)[N / 2], const int64_t (&H)[N / 2], int64_t (&X)[N]) {
    if constexpr (K < N / 2) {
      const int64_t h = mul_lee<N / 2 - 1 + K>(H[K]);
      X[K] = G[K] + h;
      X[N - 1 - K] = G[K] - h;
      outs<K + 1>(G, H, X);
    }
  }
  static __device__ __forceinline__ void run(const int64_t (&x)[N], int64_t (&X)[N]) {
    constexpr int H = N / 2;
    int64_t xe[H], z[H], G[H], Hh[H];
#pragma unroll
    for (int m = 0; m < H; ++m) {
      xe[m] = x[2 * m];
      z[m] = m > 0 ? x[2 * m + 1] + x[2 * m - 1] : x[1];
    }
    Dct3<H>::run(xe, G);
    Dct3<H>::run(z, Hh);
    outs<0>(G, Hh, X);
  }
};
template <>
struct Dct3<1> {
  static __device__ __forceinline__ void run(const int64_t (&x)[1], int64_t (&X)[1]) { X[0] = x[0]; }
};

template <int M>
struct Dct1 {
  static __device__ __forceinline__ void run(const int64_t (&s)[M + 1], int64_t (&y)[M + 1]) {
    constexpr int N = M / 2;
    int64_t u[N + 1], v[N], ye[N + 1], yo[N];
    u[0] = s[0] + s[M];
    v[0] = s[0] - s[M];
#pragma unroll
    for (int l = 1; l < N; ++l) {
      u[l] = s[l] + s[M - l];
      v[l] = s[l] - s[M - l];
    }
    u[N] = s[N];
    Dct1<N>::run(u, ye);
    Dct3<N>::run(v, yo);
#pragma unroll
    for (int k = 0; k <= N; ++k) y[2 * k] = ye[k];
#pragma unroll
    for (int k = 0; k < N; ++k) y[2 * k + 1] = yo[k];
  }
};
template <>
struct Dct1<2> {
  static __device__ __forceinline__ void run(const int64_t (&s)[3], int64_t (&y)[3]) {
    const int64_t a = s[0] + s[2];
    y[0] = a + s[1];
    y[1] = s[0] - s[2];
    y[2] = a - s[1];
  }
};

__device__ constexpr int log2i(int x) { return x <= 1 ? 0 : 1 + log2i(x / 2); }
__device__ __forceinline__ int64_t shr(int64_t x, int n) { return x >> (n < 63 ? n : 63); }

// One coordinate row x[0 .. M] of q (isp 0) or p (isp 1) in shared memory, in place;
// msc is 1/m for q, m for p.  Every lane of the warp takes part; lanes that are not
// active point at an active lane's row and write nothing.  Returns whether the new
// row is finite; put(l, y) receives it.
//
// A warp passes through this once or twice only, so what it fetches as code
// bounds it: unrolled as a whole (9000 instructions for M = 32) it waited for
// instructions half of the time.  So only the transforms, which need their
// arrays in registers, are straight code, once for both passes, and everything
// element by element loops over the row in shared memory.
template <int M, class Put>
__device__ __forceinline__ bool row(double* buf, Put put, bool isp, bool active, double msc, const FastRing& T) {
  constexpr int kGuard = log2i(M) - 2, kBits = 56 - kGuard, kNone = -100000;
  long long* fix = reinterpret_cast<long long*>(buf);
  const double first = isp ? 0.0 : buf[0];
  int e = 0;
#pragma unroll 4
  for (int l = 0; l <= M; ++l) e = max(e, exponent_field(buf[l]));
  const bool bad = e == kFixedNan;
  uint64_t mag = 0;
  const int64_t x0 = isp ? 0 : to_fixed(buf[0], e, kGuard);
#pragma unroll 4
  for (int l = 0; l <= M; ++l) {
    const int64_t x = to_fixed(buf[l], e, kGuard) - x0;
    mag |= (uint64_t)(x < 0 ? -x : x);
    if (active) fix[l] = x;
  }
  const int up = fx::clz64(mag) - (64 - kBits);  // -1 .. : left shift to kBits bits
  const int ex = mag == 0 ? kNone : e - 1078 + kGuard - up;
  const int left = up < 0 ? 0 : up < 63 ? up : 0, right = up < 0 ? 1 : 0;
  // z = A X + msc B O with the partner's modes O
  const bool obad = __shfl_xor_sync(0xffffffffu, (int)bad, 1) != 0;
  const int eo = __shfl_xor_sync(0xffffffffu, ex, 1);
  const uint64_t mb = fx::bits(msc);
  const uint64_t mq = fx::signif(mb);
  const int ev = ex + 1, eu = eo == kNone ? kNone : eo + (isp ? T.ec : T.eb) + (fx::expo(mb) - 1023) + 2;
  const int E = max(ev, eu);
  const long long* A = (const long long*)T.tab;
  const long long* B = A + (isp ? 2 : 1) * (M + 1);
  // x_l normalised, twice it between the ends
#pragma unroll 4
  for (int l = 0; l <= M; ++l) {
    const long long x = (fix[l] << left) >> right << (l > 0 && l < M ? 1 : 0);
    if (active) fix[l] = x;
  }
#pragma unroll 1
  for (int pass = 0;; ++pass) {
    int64_t x[M + 1], X[M + 1];
#pragma unroll
    for (int l = 0; l <= M; ++l) x[l] = fix[l];
    Dct1<M>::run(x, X);
    if (active) {
#pragma unroll
      for (int l = 0; l <= M; ++l) fix[l] = X[l];
    }
    if (pass == 1) break;
#pragma unroll 4
    for (int k = 0; k <= M; ++k) {
      const int64_t own = fix[k], o = __shfl_xor_sync(0xffffffffu, own, 1);
      const int64_t v = mul_s64(own << 1, __ldg(A + k));
      const int64_t u = mul_q64(mul_s64(o << 1, __ldg(B + k)), mq);
      if (active) fix[k] = shr(v, E - ev) + shr(u, E - eu);
    }
    }
  bool fine = true;
  if (active) {
    fine = !(bad || obad);
#pragma unroll 4
    for (int l = 0; l <= M; ++l) {
      double y = from_fixed(fix[l], E - log2i(M)) + first;
      if (bad || obad) y = __longlong_as_double(0x7ff8000000000000ll);
      fine = fine && exponent_field(y) != 0x7ff;
      put(l, y);
    }
  }
  return fine;
}

}  // namespace ring
#endif

}  // namespace cr
