// The fill's arithmetic, written once for both of its number types: double
// (the plain path) and df (double-float: FP64-class values on the FP32 pipes).
#pragma once

#include "df64.cuh"

namespace {

__device__ __forceinline__ df operator+(df a, df b) { return df_add(a, b); }
__device__ __forceinline__ df operator-(df a, df b) { return df_sub(a, b); }
__device__ __forceinline__ df operator-(df a) { return df_neg(a); }
__device__ __forceinline__ df operator*(df a, df b) { return df_mul(a, b); }

// Num<T>: what the two types do differently.  Tail is the type that carries
// terms below 2^-24 of a sum.  LESS: sincos_ and exp_ also give sin x - x and
// e^x - 1, accurate relative to themselves where x needs no reduction (double:
// the functions' values again).
template <typename T>
struct Num;

template <>
struct Num<double> {
  typedef double Tail;
  static constexpr bool LESS = false;
  __device__ __forceinline__ static double of(double x) { return x; }
  __device__ __forceinline__ static double to_double(double x) { return x; }
  __device__ __forceinline__ static double head(double x) { return x; }
  __device__ __forceinline__ static double tail(double x) { return x; }
  __device__ __forceinline__ static double diff(double a, double b) { return a - b; }
  __device__ __forceinline__ static double sumsq(double x, double y, double z) { return x * x + y * y + z * z; }
  __device__ __forceinline__ static void mac(double &a, double x, double y) { a = fma(x, y, a); }
  __device__ __forceinline__ static double fin(double a) { return a; }
  __device__ __forceinline__ static double dot2(double a, double b, double c, double d) { return fma(a, b, c * d); }
  __device__ __forceinline__ static double muladd(double a, double b, double c) { return fma(a, b, c); }
  __device__ __forceinline__ static double sqrt_(double a) { return sqrt(a); }
  __device__ __forceinline__ static double rcp(double a) { return 1.0 / a; }
  __device__ __forceinline__ static void sqrt_rcp(double a, double &R, double &Ri) {
    Ri = rsqrt(a);
    R = a * Ri;
  }
  __device__ __forceinline__ static void sincos_(double x, double &s, double &c, double &sm) {
    sincos(x, &s, &c);
    sm = s;
  }
  __device__ __forceinline__ static double exp_(double x, double &m1) { return m1 = exp(x); }
  __device__ __forceinline__ static double log_(double x) { return log(x); }
  __device__ __forceinline__ static double atan2_(double y, double x) { return atan2(y, x); }
  __device__ __forceinline__ static double abs_(double x) { return fabs(x); }
  __device__ __forceinline__ static double pow2(double x, double p) { return x * p; }  // p: a power of two
  __device__ __forceinline__ static double shfl(double x, int o) { return __shfl_xor_sync(0xffffffffu, x, o); }
};

template <>
struct Num<df> {
  typedef float Tail;
  static constexpr bool LESS = true;
  __device__ __forceinline__ static df of(double x) { return df_make(x); }
  __device__ __forceinline__ static double to_double(df x) { return df_to_double(x); }
  __device__ __forceinline__ static float head(df x) { return x.hi; }
  __device__ __forceinline__ static df tail(float x) { return {x, 0.f}; }
  __device__ __forceinline__ static df diff(df a, df b) { return df_diff(a, b); }
  __device__ __forceinline__ static df sumsq(df x, df y, df z) { return df_sumsq(x, y, z); }
  __device__ __forceinline__ static void mac(df &a, df x, df y) { df_mac(a, x, y); }
  __device__ __forceinline__ static df fin(df a) { return df_fin(a); }
  __device__ __forceinline__ static df dot2(df a, df b, df c, df d) { return df_dot2(a, b, c, d); }
  __device__ __forceinline__ static df muladd(df a, df b, df c) { return df_muladd(a, b, c); }
  __device__ __forceinline__ static df sqrt_(df a) { return df_sqrt(a); }
  __device__ __forceinline__ static df rcp(df a) { return df_rcp(a); }
  __device__ __forceinline__ static void sqrt_rcp(df a, df &R, df &Ri) { df_sqrt_rcp(a, R, Ri); }
  // sm = sin x - x
  __device__ __forceinline__ static void sincos_(df x, df &s, df &c, df &sm) {
    if (fabsf(x.hi) < 200.f) {
      df_sincos_df(x, s, c, sm);
    } else {
      df_sincos(df_to_double(x), s, c);  // FP64 reduction for phases of 200 rad and more
      sm = df_sub(s, x);
    }
  }
  __device__ __forceinline__ static df exp_(df x, df &m1) { return df_exp_df(x, m1); }  // m1 = e^x - 1
  __device__ __forceinline__ static df log_(df x) { return df_log(x); }
  __device__ __forceinline__ static df atan2_(df y, df x) { return df_atan2(y, x); }
  __device__ __forceinline__ static df abs_(df x) { return df_abs(x); }
  __device__ __forceinline__ static df pow2(df x, float p) { return df_scale2(x, p); }
  __device__ __forceinline__ static df shfl(df x, int o) {
    return {__shfl_xor_sync(0xffffffffu, x.hi, o), __shfl_xor_sync(0xffffffffu, x.lo, o)};
  }
};

template <typename T>
struct V3 {
  T x, y, z;
};
template <typename T>
__device__ __forceinline__ V3<T> operator+(V3<T> a, V3<T> b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
template <typename T>
__device__ __forceinline__ V3<T> operator-(V3<T> a, V3<T> b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
template <typename T>
__device__ __forceinline__ V3<T> operator*(T s, V3<T> a) { return {s * a.x, s * a.y, s * a.z}; }
template <typename T>
__device__ __forceinline__ T vdot(V3<T> a, V3<T> b) { return Num<T>::muladd(a.z, b.z, Num<T>::dot2(a.x, b.x, a.y, b.y)); }
template <typename T>
__device__ __forceinline__ V3<T> vcross(V3<T> a, V3<T> b) {
  return {Num<T>::dot2(a.y, b.z, -a.z, b.y), Num<T>::dot2(a.z, b.x, -a.x, b.z), Num<T>::dot2(a.x, b.y, -a.y, b.x)};
}
template <typename T>
__device__ __forceinline__ V3<T> vscale2(V3<T> a, float p) {
  return {Num<T>::pow2(a.x, p), Num<T>::pow2(a.y, p), Num<T>::pow2(a.z, p)};
}
template <typename T>
__device__ __forceinline__ V3<T> vzero() {
  const T z = Num<T>::of(0.0);
  return {z, z, z};
}

template <typename T>
struct C1 {
  T r, i;
};
template <typename T>
__device__ __forceinline__ C1<T> operator+(C1<T> a, C1<T> b) { return {a.r + b.r, a.i + b.i}; }
template <typename T>
__device__ __forceinline__ C1<T> operator-(C1<T> a, C1<T> b) { return {a.r - b.r, a.i - b.i}; }
template <typename T>
__device__ __forceinline__ C1<T> operator*(T s, C1<T> a) { return {s * a.r, s * a.i}; }
template <typename T>
__device__ __forceinline__ C1<T> cmul(C1<T> a, C1<T> b) {
  return {Num<T>::dot2(a.r, b.r, -a.i, b.i), Num<T>::dot2(a.r, b.i, a.i, b.r)};
}

// Sums of eight values over the warp: three exchange steps leave each group of
// four lanes one value, two more finish it.  Lane l returns the sum of value
// reduce8_index(l): 9 additions a chunk, against 40 for eight butterflies.
__device__ __forceinline__ int reduce8_index(int lane) { return ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1); }
template <typename T>
__device__ __forceinline__ T reduce8(const T (&v)[8], int lane) {
  T a[4], b[2];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const bool up = lane & 16;
    const T keep = up ? v[k + 4] : v[k], give = up ? v[k] : v[k + 4];
    a[k] = keep + Num<T>::shfl(give, 16);
  }
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const bool up = lane & 8;
    const T keep = up ? a[k + 2] : a[k], give = up ? a[k] : a[k + 2];
    b[k] = keep + Num<T>::shfl(give, 8);
  }
  const bool up = lane & 4;
  const T keep = up ? b[1] : b[0], give = up ? b[0] : b[1];
  T c = keep + Num<T>::shfl(give, 4);
  c = c + Num<T>::shfl(c, 2);
  return c + Num<T>::shfl(c, 1);
}

}  // namespace
