// Arithmetic whose roundings the source decides.
//
// The compiler contracts a product and a sum as it sees fit, so one expression in
// two instantiations of a template (a surface by one thread and by four lanes) may
// differ in the last bit.  A product of Nums stays open until something is added to
// it or it is subtracted (one fused operation; of two products the second is rounded)
// or it is stored or multiplied on (rounded); sums are operations that the compiler
// does not contract.  The bits of a result are then those of the source, whatever
// surrounds it, at the cost of the contracted code.
#pragma once
#include <cuda_runtime.h>

#include <type_traits>

namespace cr {

__device__ __forceinline__ float sum_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double sum_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float fused(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fused(double a, double b, double c) { return __fma_rn(a, b, c); }

template <class F>
struct Prod {
  F a, b;
  __device__ __forceinline__ F value() const { return a * b; }
};

template <class F>
struct Num {
  F v;
  Num() = default;
  template <class T, class = typename std::enable_if<std::is_arithmetic<T>::value>::type>
  __device__ __forceinline__ constexpr Num(T x) : v((F)x) {}  // NOLINT: constants promote implicitly
  __device__ __forceinline__ Num(Prod<F> p) : v(p.value()) {}  // NOLINT
  template <class G>
  __device__ __forceinline__ explicit Num(Num<G> x) : v((F)x.v) {}
  __device__ __forceinline__ explicit operator double() const { return (double)v; }
};

template <class F>
__device__ __forceinline__ Num<F> operator-(Num<F> x) { return Num<F>(-x.v); }
template <class F>
__device__ __forceinline__ Prod<F> operator-(Prod<F> p) { return Prod<F>{-p.a, p.b}; }

template <class F>
__device__ __forceinline__ Prod<F> operator*(Num<F> x, Num<F> y) { return Prod<F>{x.v, y.v}; }
template <class F>
__device__ __forceinline__ Prod<F> operator*(Prod<F> p, Num<F> y) { return Prod<F>{p.value(), y.v}; }
template <class F>
__device__ __forceinline__ Prod<F> operator*(Num<F> x, Prod<F> q) { return Prod<F>{x.v, q.value()}; }
template <class F>
__device__ __forceinline__ Prod<F> operator*(Prod<F> p, Prod<F> q) { return Prod<F>{p.value(), q.value()}; }

template <class F>
__device__ __forceinline__ Num<F> operator+(Num<F> x, Num<F> y) { return Num<F>(sum_rn(x.v, y.v)); }
template <class F>
__device__ __forceinline__ Num<F> operator+(Prod<F> p, Num<F> y) { return Num<F>(fused(p.a, p.b, y.v)); }
template <class F>
__device__ __forceinline__ Num<F> operator+(Num<F> x, Prod<F> q) { return Num<F>(fused(q.a, q.b, x.v)); }
template <class F>
__device__ __forceinline__ Num<F> operator+(Prod<F> p, Prod<F> q) { return Num<F>(fused(p.a, p.b, q.value())); }

template <class F>
__device__ __forceinline__ Num<F> operator-(Num<F> x, Num<F> y) { return x + (-y); }
template <class F>
__device__ __forceinline__ Num<F> operator-(Prod<F> p, Num<F> y) { return p + (-y); }
template <class F>
__device__ __forceinline__ Num<F> operator-(Num<F> x, Prod<F> q) { return x + (-q); }
template <class F>
__device__ __forceinline__ Num<F> operator-(Prod<F> p, Prod<F> q) { return p + (-q); }

template <class F, class T>
__device__ __forceinline__ Num<F>& operator+=(Num<F>& x, T y) { return x = x + y; }
template <class F>
__device__ __forceinline__ Num<F>& operator*=(Num<F>& x, Num<F> y) { return x = x * y; }

template <class F>
__device__ __forceinline__ bool operator<(Num<F> x, Num<F> y) { return x.v < y.v; }
template <class F>
__device__ __forceinline__ bool operator<=(Num<F> x, Num<F> y) { return x.v <= y.v; }
template <class F>
__device__ __forceinline__ bool operator>=(Num<F> x, Num<F> y) { return x.v >= y.v; }

}  // namespace cr
