// Complex arithmetic of the z-marching operator kernels (stencil2.cuh, hh.cu):
// paired FP32 instructions for complex64, scalar FP64 for complex128, and
// neighbour exchange within a warp.
#pragma once

#include <type_traits>

#include "operator_common.cuh"

namespace fdfd {

template <typename C>
__device__ __forceinline__ C zif(bool z, C v) {
  return z ? czero<C>() : v;
}

template <typename C>
__device__ __forceinline__ C shfl_up1(C v) {
  return mk(__shfl_up_sync(0xffffffffu, v.x, 1), __shfl_up_sync(0xffffffffu, v.y, 1));
}
template <typename C>
__device__ __forceinline__ C shfl_down1(C v) {
  return mk(__shfl_down_sync(0xffffffffu, v.x, 1), __shfl_down_sync(0xffffffffu, v.y, 1));
}

// Complex64 arithmetic of the curls and the diagonal term on the paired FP32
// instructions of sm_100 and later (__fadd2_rn, __fmul2_rn, __ffma2_rn:
// both lanes rounded to nearest, as the scalar forms are), half the
// instructions of the scalar forms; complex128 keeps the scalar forms.
__device__ __forceinline__ float2 f2(float s) { return make_float2(s, s); }
__device__ __forceinline__ float2 psub(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
__device__ __forceinline__ double2 psub(double2 a, double2 b) { return csub(a, b); }
// a·s + b for real s
__device__ __forceinline__ float2 pfma(float2 a, float s, float2 b) { return __ffma2_rn(a, f2(s), b); }
__device__ __forceinline__ double2 pfma(double2 a, double s, double2 b) { return cadd(cscale(a, s), b); }
// a·u − b·v for coefficients a, b that are real when RC
template <bool RC>
__device__ __forceinline__ float2 pdiff(float2 a, float2 u, float2 b, float2 v) {
  if constexpr (RC) {
    return __ffma2_rn(f2(a.x), u, __fmul2_rn(f2(-b.x), v));
  } else {
    float2 t = __fmul2_rn(make_float2(b.y, -b.y), make_float2(v.y, v.x));  // −b·v
    t = __ffma2_rn(f2(-b.x), v, t);
    t = __ffma2_rn(make_float2(-a.y, a.y), make_float2(u.y, u.x), t);     // + a·u
    return __ffma2_rn(f2(a.x), u, t);
  }
}
template <bool RC>
__device__ __forceinline__ double2 pdiff(double2 a, double2 u, double2 b, double2 v) {
  return csub(mulc<RC>(a, u), mulc<RC>(b, v));
}
// conj(a0)·b0 + conj(a1)·b1 + conj(a2)·b2
__device__ __forceinline__ float2 pdot3(float2 a0, float2 b0, float2 a1, float2 b1, float2 a2, float2 b2) {
  float2 t = __fmul2_rn(f2(a0.x), b0);
  t = __ffma2_rn(make_float2(a0.y, -a0.y), make_float2(b0.y, b0.x), t);
  t = __ffma2_rn(f2(a1.x), b1, t);
  t = __ffma2_rn(make_float2(a1.y, -a1.y), make_float2(b1.y, b1.x), t);
  t = __ffma2_rn(f2(a2.x), b2, t);
  return __ffma2_rn(make_float2(a2.y, -a2.y), make_float2(b2.y, b2.x), t);
}
// (re, im) += conj(a)·b
template <typename R, typename C>
__device__ __forceinline__ void dot_into(R &re, R &im, C a, C b) {
  re = fma(a.y, b.y, fma(a.x, b.x, re));
  im = fma(-a.y, b.x, fma(a.x, b.y, im));
}
// a·u + b·v for coefficients a, b that are real when RC (corner averaging)
template <bool RC>
__device__ __forceinline__ float2 wsum(float2 a, float2 u, float2 b, float2 v) {
  return cadd(mulc<RC>(a, u), mulc<RC>(b, v));
}
template <bool RC>
__device__ __forceinline__ double2 wsum(double2 a, double2 u, double2 b, double2 v) {
  return cadd(mulc<RC>(a, u), mulc<RC>(b, v));
}
// A complex64 curl coefficient as csum takes it: its real part twice (the
// operand of a paired multiply; 16 bytes, one shared-memory load).
template <typename R> struct Coef;
template <> struct __align__(16) Coef<float> {
  float2 xx;
  float y, pad;
};
__device__ __forceinline__ Coef<float> coef_of(float2 c) { return {make_float2(c.x, c.x), c.y, 0.f}; }

// a·u + b·v for coefficients a (real when AR) and b (real when BR): the real
// parts in paired instructions, the imaginary ones in scalar instructions
// (paired ones would first swap the halves of u and v).
template <bool AR, bool BR>
__device__ __forceinline__ float2 csum(const Coef<float> &a, float2 u, const Coef<float> &b, float2 v) {
  if constexpr (AR && BR) {
    return __ffma2_rn(a.xx, u, __fmul2_rn(b.xx, v));
  } else {
    float2 t = make_float2(-b.y * v.y, b.y * v.x);
    t = __ffma2_rn(b.xx, v, t);
    t = make_float2(fmaf(-a.y, u.y, t.x), fmaf(a.y, u.x, t.y));
    return __ffma2_rn(a.xx, u, t);
  }
}

// complex128 runs at the FP64 pipe's rate — a warp's FP64 instruction holds
// it for 64 cycles, predicated off or not — so its products take only the
// parts they need, axis by axis: a·u − b·v with a real when AR, b when BR.
template <bool AR, bool BR>
__device__ __forceinline__ double2 pdiff_by(double2 a, double2 u, double2 b, double2 v) {
  double2 t = make_double2(a.x * u.x, a.x * u.y);
  if (!AR) t = make_double2(fma(-a.y, u.y, t.x), fma(a.y, u.x, t.y));
  t = make_double2(fma(-b.x, v.x, t.x), fma(-b.x, v.y, t.y));
  if (!BR) t = make_double2(fma(b.y, v.y, t.x), fma(-b.y, v.x, t.y));
  return t;
}

// f(XR, YR, ZR) for three warp-uniform flags as compile-time constants: one
// branch to a body that holds only the FP64 instructions it needs (FINE =
// false: only the all-real and the all-complex body, less code).
template <bool FINE = true, typename F>
__device__ __forceinline__ void by_axis(bool xr, bool yr, bool zr, F f) {
  using T = std::true_type;
  using N = std::false_type;
  if constexpr (!FINE) {
    if (xr && yr && zr) f(T{}, T{}, T{});
    else f(N{}, N{}, N{});
  } else if (xr) {
    if (yr) {
      if (zr) f(T{}, T{}, T{});
      else f(T{}, T{}, N{});
    } else {
      if (zr) f(T{}, N{}, T{});
      else f(T{}, N{}, N{});
    }
  } else {
    if (yr) {
      if (zr) f(N{}, T{}, T{});
      else f(N{}, T{}, N{});
    } else {
      if (zr) f(N{}, N{}, T{});
      else f(N{}, N{}, N{});
    }
  }
}

}  // namespace fdfd
