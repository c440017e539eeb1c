// Complex element types (interleaved re, im) and their arithmetic: products
// from fused multiply-adds of the real parts, quotients by Smith's algorithm
// (R. L. Smith, "Algorithm 116: Complex division", CACM 5(8), 1962).
#pragma once

#include "nla_common.cuh"

namespace nla {
namespace cx {

template <typename R>
struct alignas(2 * sizeof(R)) cpx {
  R re, im;
};

template <typename R> __device__ __forceinline__ cpx<R> mk(R a, R b) { return cpx<R>{a, b}; }
template <typename R> __device__ __forceinline__ cpx<R> zero() { return cpx<R>{R(0), R(0)}; }
template <typename R> __device__ __forceinline__ cpx<R> conj_if(cpx<R> a, bool c) { return c ? mk(a.re, -a.im) : a; }
// c + a b
template <typename R> __device__ __forceinline__ cpx<R> fma_c(cpx<R> a, cpx<R> b, cpx<R> c) {
  return mk(fma(a.re, b.re, fma(-a.im, b.im, c.re)), fma(a.re, b.im, fma(a.im, b.re, c.im)));
}
// c - a b
template <typename R> __device__ __forceinline__ cpx<R> fms_c(cpx<R> a, cpx<R> b, cpx<R> c) {
  return mk(fma(-a.re, b.re, fma(a.im, b.im, c.re)), fma(-a.re, b.im, fma(-a.im, b.re, c.im)));
}
// a / b, Smith's algorithm.
template <typename R> __device__ __forceinline__ cpx<R> div(cpx<R> a, cpx<R> b) {
  if (fabs(b.re) >= fabs(b.im)) {
    const R t = b.im / b.re, den = b.re + b.im * t;
    return mk((a.re + a.im * t) / den, (a.im - a.re * t) / den);
  }
  const R t = b.re / b.im, den = b.im + b.re * t;
  return mk((a.re * t + a.im) / den, (a.im * t - a.re) / den);
}
template <typename R> __device__ __forceinline__ cpx<R> operator+(cpx<R> a, cpx<R> b) { return mk(a.re + b.re, a.im + b.im); }
template <typename R> __device__ __forceinline__ cpx<R> operator-(cpx<R> a, cpx<R> b) { return mk(a.re - b.re, a.im - b.im); }

}  // namespace cx

template <typename R> struct Elem<cx::cpx<R>> {
  using compute = cx::cpx<R>;
  __device__ static compute load(const compute* p) { return *p; }
  __device__ static void store(compute* p, compute v) { *p = v; }
};

}  // namespace nla
