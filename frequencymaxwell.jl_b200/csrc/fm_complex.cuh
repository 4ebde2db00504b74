// Complex arithmetic on float2 / double2 for the fmcuda kernels.
#pragma once
#include <cuda_runtime.h>
#include <type_traits>

namespace fm {

template <typename R> struct CT;
template <> struct CT<float>  { using T = float2; };
template <> struct CT<double> { using T = double2; };
template <typename R> using cplx = typename CT<R>::T;

template <typename T> struct RealOf;
template <> struct RealOf<float2>  { using R = float; };
template <> struct RealOf<double2> { using R = double; };

__host__ __device__ __forceinline__ float2 mk(float a, float b) { return make_float2(a, b); }
__host__ __device__ __forceinline__ double2 mk(double a, double b) { return make_double2(a, b); }

template <typename T> __host__ __device__ __forceinline__ T cadd(T a, T b) { return mk(a.x + b.x, a.y + b.y); }
template <typename T> __host__ __device__ __forceinline__ T csub(T a, T b) { return mk(a.x - b.x, a.y - b.y); }
template <typename T> __host__ __device__ __forceinline__ T cmul(T a, T b) {
  return mk(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// cmul with its fused multiply-adds written out: the same bits wherever it is used
template <typename T> __device__ __forceinline__ T cmul_fixed(T a, T b) {
  return mk(fma(a.x, b.x, -(a.y * b.y)), fma(a.y, b.x, a.x * b.y));
}
// a * conj(b)
template <typename T> __host__ __device__ __forceinline__ T cmulc(T a, T b) {
  return mk(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
template <typename T> __host__ __device__ __forceinline__ T cconj(T a) { return mk(a.x, -a.y); }
template <typename T, typename R> __host__ __device__ __forceinline__ T cscale(T a, R s) { return mk(a.x * s, a.y * s); }
// multiply by i*sgn  (sgn = +1 -> i, -1 -> -i)
template <int SGN, typename T> __host__ __device__ __forceinline__ T cmul_i(T a) {
  return SGN > 0 ? mk(-a.y, a.x) : mk(a.y, -a.x);
}
template <typename T> __host__ __device__ __forceinline__ T cinv(T a) {
  auto d = a.x * a.x + a.y * a.y;
  return mk(a.x / d, -a.y / d);
}
template <typename T> __host__ __device__ __forceinline__ T czero() { return mk(decltype(T{}.x)(0), decltype(T{}.x)(0)); }

__device__ __forceinline__ double2 to_d(float2 a) { return make_double2(a.x, a.y); }
__device__ __forceinline__ double2 to_d(double2 a) { return a; }
template <typename T> __device__ __forceinline__ T from_d(double2 a);
template <> __device__ __forceinline__ float2 from_d<float2>(double2 a) { return make_float2((float)a.x, (float)a.y); }
template <> __device__ __forceinline__ double2 from_d<double2>(double2 a) { return a; }

// starts bringing the 128-byte line at p to L2
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// ---- FP32 -> FP64 without the conversion unit ----
// The conversion instruction issues about one lane per clock and scheduler on sm_100a, which caps a kernel that
// widens every value it reads near 5 TB/s of FP32 data.  Moving the fields of the float into those of a double with
// three integer instructions gives the value times WIDEN_SCALE = 2^-896 exactly, for zeros and subnormal numbers too
// (the exponent field is kept unbiased and a double's smallest exponents take it).  The factor is taken out again by
// exact powers of two.  Infinities and NaNs would come out finite, so the users add nonfinite_mark() of the values.
constexpr double WIDEN_HALF = 0x1p448;  // WIDEN_HALF^2 * WIDEN_SCALE = 1
__device__ __forceinline__ double widen(float x) {
  const int i = __float_as_int(x);
  return __hiloint2double((i >> 3) & 0x8fffffff, i << 29);
}
__device__ __forceinline__ double2 widen(float2 a) { return make_double2(widen(a.x), widen(a.y)); }
// accumulates zero for finite values and NaN otherwise
__device__ __forceinline__ void nonfinite_mark(float& t, float2 a) { t = fmaf(a.x, 0.0f, fmaf(a.y, 0.0f, t)); }
// the mark as a double: 0 or NaN (the hardware's NaN result is 0x7fffffff, whose bits are a double's NaN too)
__device__ __forceinline__ double mark_d(float t) { return __hiloint2double(__float_as_int(t), 0); }

}  // namespace fm
