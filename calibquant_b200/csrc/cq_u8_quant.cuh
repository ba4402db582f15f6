// uint8 format: the arithmetic of the quantizers.
#pragma once

#include "cq_common.cuh"

namespace cq {
namespace calib {

template <typename T> struct Pk2;
template <> struct Pk2<__half> { static __device__ __forceinline__ __half2 magic() { return __float2half2_rn(1024.f); } };
template <> struct Pk2<__nv_bfloat16> { static __device__ __forceinline__ __nv_bfloat162 magic() { return __float2bfloat162_rn(128.f); } };

// order-preserving 16-bit keys of fp16 / bfloat16 patterns
__device__ __forceinline__ unsigned short key16(unsigned short b) {
  return (b & 0x8000u) ? (unsigned short)~b : (unsigned short)(b | 0x8000u);
}
__device__ __forceinline__ unsigned short unkey16(unsigned short k) {
  return (k & 0x8000u) ? (unsigned short)(k & 0x7fffu) : (unsigned short)~k;
}
template <typename T>
__device__ __forceinline__ float ref_code(float x, float s, float z, int levels) {
  const float y = rnd<T>(rnd<T>(__fdiv_rn(x, s)) + z);
  return rintf(fminf(fmaxf(y, 0.f), (float)levels));
}
template <typename T> struct Finite16;
template <> struct Finite16<__half> { static constexpr unsigned short MAXPOS = 0x7bffu; };
template <> struct Finite16<__nv_bfloat16> { static constexpr unsigned short MAXPOS = 0x7f7fu; };

// scale and zero point of a channel from its extremes, every operation rounded to the data type
template <typename T>
__device__ __forceinline__ void scale_zero(float mn, float mx, float clip, int levels, float& s, float& z) {
  const float x_min = rnd<T>(mn * clip), x_max = rnd<T>(mx * clip);
  s = rnd<T>(__fdiv_rn(rnd<T>(x_max - x_min), (float)levels));
  z = rnd<T>(__fdiv_rn(-x_min, s));
}
// With scale > 0 the code  rint(clamp(rnd(rnd(x / s) + z)))  is a non-decreasing step function of x: the largest number of the
// data type whose code is <= k, by bisection over the ordered 16-bit patterns with the reference arithmetic itself.  The
// search starts around s (k + 1/2 - z), which the roundings move by a few patterns (many only where x is close to zero), and widens
// as needed: 6 evaluations instead of 18 in the usual case.
template <typename T>
__device__ __forceinline__ T threshold(float s, float z, int k, int levels) {
  const int k_min = key16((unsigned short)(Finite16<T>::MAXPOS | 0x8000u)), k_max = key16(Finite16<T>::MAXPOS);
  auto above = [&](int key) {
    const unsigned short b = unkey16((unsigned short)key);
    return ref_code<T>(Elem<T>::to_f(*reinterpret_cast<const T*>(&b)), s, z, levels) > (float)k;
  };
  const T guess = Elem<T>::from_f(s * ((float)k + 0.5f - z));
  const int g = min(max((int)key16(*reinterpret_cast<const unsigned short*>(&guess)), k_min), k_max);
  int lo = max(g - 4, k_min), hi = min(g + 4, k_max), w = 16;
  bool a_lo = above(lo), a_hi = above(hi);
  while (a_lo && lo > k_min) { hi = lo; a_hi = true; lo = max(lo - w, k_min); w *= 8; a_lo = above(lo); }
  while (!a_hi && hi < k_max) { lo = hi; a_lo = false; hi = min(hi + w, k_max); w *= 8; a_hi = above(hi); }
  unsigned short theta;
  if (a_lo) theta = Finite16<T>::MAXPOS == 0x7f7fu ? 0xff80u : 0xfc00u;      // every finite number exceeds level k: -inf
  else if (!a_hi) theta = Finite16<T>::MAXPOS;                              // only +inf exceeds the largest finite number
  else {
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (above(mid)) hi = mid; else lo = mid;
    }
    theta = unkey16((unsigned short)lo);
  }
  return *reinterpret_cast<const T*>(&theta);
}

}  // namespace calib
}  // namespace cq
