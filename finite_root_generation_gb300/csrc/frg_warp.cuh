// What the warp-per-path kernels share: shuffles of complex values, comparisons of FP64
// magnitudes in the integer pipes, products kept out of fused multiply-adds.
#pragma once

#include <cuda_runtime.h>

#include "frg_complex.cuh"

namespace frg {

constexpr unsigned FULL = 0xffffffffu;

template <typename T>
__device__ __forceinline__ cx<T> warp_shfl(cx<T> v, int src) {
  return cx<T>(__shfl_sync(FULL, v.re, src), __shfl_sync(FULL, v.im, src));
}
// Largest |re| or |im| of values, NaN taking no part (as fmax drops it): FP32 directly,
// FP64 on the bit patterns, whose order as integers is the order of the magnitudes.
template <typename T> struct MaxAbs;
template <> struct MaxAbs<float> {
  float m = 0.f;
  __device__ __forceinline__ void take(cx<float> v) { m = fmaxf(m, fmaxf(fabsf(v.re), fabsf(v.im))); }
  __device__ __forceinline__ void across(int off) { m = fmaxf(m, __shfl_xor_sync(FULL, m, off)); }
  __device__ __forceinline__ float value() const { return m; }
};
template <> struct MaxAbs<double> {
  long long m = 0;
  __device__ __forceinline__ void one(double x) {
    const long long b = __double_as_longlong(x) & 0x7fffffffffffffffll;
    if (b > m && b <= 0x7ff0000000000000ll) m = b;
  }
  __device__ __forceinline__ void take(cx<double> v) { one(v.re); one(v.im); }
  __device__ __forceinline__ void across(int off) {
    const long long o = __shfl_xor_sync(FULL, m, off);
    if (o > m) m = o;
  }
  __device__ __forceinline__ double value() const { return __longlong_as_double(m); }
};

// running maximum and minimum of magnitudes >= 0, NaN taking no part
__device__ __forceinline__ float max_mag(float m, float x) { return fmaxf(m, x); }
__device__ __forceinline__ float min_mag(float m, float x) { return fminf(m, x); }
__device__ __forceinline__ double max_mag(double m, double x) {
  const long long b = __double_as_longlong(x);
  return b > __double_as_longlong(m) && b <= 0x7ff0000000000000ll ? x : m;
}
__device__ __forceinline__ double min_mag(double m, double x) {
  return (unsigned long long)__double_as_longlong(x) < (unsigned long long)__double_as_longlong(m) ? x : m;
}

// x > m for magnitudes, false for a NaN x
__device__ __forceinline__ bool mag_above(float x, float m) { return x > m; }
__device__ __forceinline__ bool mag_above(double x, double m) {
  const long long b = __double_as_longlong(x);
  return b > __double_as_longlong(m) && b <= 0x7ff0000000000000ll;
}

// 1 / b when |b|^2 is at hand (FP64: conj(b) / |b|^2; FP32 keeps Smith's form)
__device__ __forceinline__ cx<double> cinv_norm(cx<double> b, double n2) {
  const double r = 1.0 / n2;
  return cx<double>(b.re * r, -b.im * r);
}
__device__ __forceinline__ cx<float> cinv_norm(cx<float> b, float) { return cinv(b); }

// products that no later addition may absorb into a fused multiply-add
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
template <typename T>
__device__ __forceinline__ cx<T> mul_rn(T s, cx<T> a) { return cx<T>(mul_rn(s, a.re), mul_rn(s, a.im)); }
// s * a + b, fused
template <typename T>
__device__ __forceinline__ cx<T> axpy(T s, cx<T> a, cx<T> b) { return cx<T>(fma(s, a.re, b.re), fma(s, a.im, b.im)); }


// -x when `neg`, on the sign bit: a negation that no arithmetic absorbs (a selected or
// stored one) would be an FP64 instruction of its own
__device__ __forceinline__ double neg_if(double x, bool neg) {
  return __hiloint2double(__double2hiint(x) ^ (neg ? 0x80000000 : 0), __double2loint(x));
}
__device__ __forceinline__ float neg_if(float x, bool neg) { return neg ? -x : x; }
template <typename T>
__device__ __forceinline__ cx<T> neg(cx<T> a) { return cx<T>(neg_if(a.re, true), neg_if(a.im, true)); }

// An FP64 complex value held by a pair of lanes (2 k, 2 k + 1): each lane computes one
// component of every result (the even lane the real part) and the pair exchanges, so a
// product takes 2 FP64 instructions and a sum 1 where a lane alone takes 4 and 2. The
// operations are cx<double>'s. `re` and `ims` (the imaginary part on the odd lane, its
// negative on the even one) serve a left factor, `own` and `oth` the rest.
struct PairCx {
  double re, ims, own, oth;
  __device__ __forceinline__ static bool odd() { return threadIdx.x & 1; }
  __device__ __forceinline__ PairCx() {}
  __device__ __forceinline__ explicit PairCx(cx<double> v)
      : re(v.re), ims(neg_if(v.im, !odd())), own(odd() ? v.im : v.re), oth(odd() ? v.re : v.im) {}
  __device__ __forceinline__ explicit PairCx(double v) : PairCx(cx<double>(v)) {}
  __device__ __forceinline__ static PairCx of(double own) {
    PairCx r;
    r.own = own;
    r.oth = __shfl_xor_sync(FULL, own, 1);
    r.re = odd() ? r.oth : own;
    r.ims = neg_if(odd() ? own : r.oth, !odd());
    return r;
  }
};
__device__ __forceinline__ PairCx operator*(PairCx a, PairCx b) {
  return PairCx::of(fma(a.re, b.own, __dmul_rn(a.ims, b.oth)));
}
__device__ __forceinline__ PairCx operator+(PairCx a, PairCx b) { return PairCx::of(a.own + b.own); }
__device__ __forceinline__ PairCx operator-(PairCx a, PairCx b) { return PairCx::of(a.own - b.own); }
__device__ __forceinline__ PairCx operator-(PairCx a) {
  PairCx r;
  r.re = -a.re; r.ims = -a.ims; r.own = -a.own; r.oth = -a.oth;
  return r;
}
// a real multiple, absorbed by the sum it enters as cx<double>'s is (one fused multiply-add)
struct PairScaled {
  double s, own;
};
__device__ __forceinline__ PairScaled operator*(double s, PairCx a) { return {s, a.own}; }
__device__ __forceinline__ PairScaled operator-(PairScaled a) { return {-a.s, a.own}; }
__device__ __forceinline__ PairCx operator+(PairScaled a, PairCx b) { return PairCx::of(fma(a.s, a.own, b.own)); }
__device__ __forceinline__ PairCx operator-(PairScaled a, PairCx b) { return PairCx::of(fma(a.s, a.own, -b.own)); }
__device__ __forceinline__ PairCx operator+(PairCx b, PairScaled a) { return PairCx::of(fma(a.s, a.own, b.own)); }

__device__ __forceinline__ void cx_put(cx<double>* p, PairCx v) { reinterpret_cast<double*>(p)[PairCx::odd()] = v.own; }

}  // namespace frg
