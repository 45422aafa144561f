// pair_spec.cuh — storage of template pairs' spectra for the paired correlation (corr_pair.cu).
#pragma once

#include "fft_pair.cuh"

namespace gisspa {

// A template pair's spectra at one point, as the column pass reads them.  FP32: U = T1 - i T2
// and V = T1 + i T2 (so that I conj U = A1 + i A2 and I conj V = A1 - i A2) as
// (U.re, V.re, U.im, V.im).  FP16 / BF16: T1 and T2 themselves, rounded as the one-template
// form rounds them.
struct PairFp32 {
  using T = float4;
  __device__ __forceinline__ static float2 plus(float2 i, T t) { return cmulc(i, make_float2(t.x, t.z)); }
  __device__ __forceinline__ static Cx2 both(float2 i, T t) {
    const float2 a = cmulc(i, make_float2(t.x, t.z)), b = cmulc(i, make_float2(t.y, t.w));
    return Cx2{make_float2(a.x, b.x), make_float2(a.y, b.y)};
  }
  // T1 + T2 (U + V = 2 T1, V - U = 2 i T2)
  __device__ __forceinline__ static double2 sum(T t) {
    return make_double2(0.5 * (((double)t.x + t.y) + ((double)t.w - t.z)),
                        0.5 * (((double)t.z + t.w) + ((double)t.x - t.y)));
  }
  __device__ __forceinline__ static T pack(float2 t1, float2 t2) {
    return make_float4(t1.x + t2.y, t1.x - t2.y, t1.y - t2.x, t1.y + t2.x);
  }
};
template <typename SPEC>
struct PairHalf {
  struct __align__(8) T {
    typename SPEC::T t1, t2;
  };
  __device__ __forceinline__ static Cx2 both(float2 i, T t) {
    const float2 a1 = cmulc(i, SPEC::load(&t.t1)), a2 = cmulc(i, SPEC::load(&t.t2));
    return Cx2{make_float2(a1.x - a2.y, a1.x + a2.y), make_float2(a1.y + a2.x, a1.y - a2.x)};
  }
  __device__ __forceinline__ static float2 plus(float2 i, T t) {
    const Cx2 c = both(i, t);
    return make_float2(c.re.x, c.im.x);
  }
  __device__ __forceinline__ static double2 sum(T t) {
    const float2 a = SPEC::load(&t.t1), b = SPEC::load(&t.t2);
    return make_double2((double)a.x + b.x, (double)a.y + b.y);
  }
  __device__ __forceinline__ static T pack(float2 t1, float2 t2) { return T{SPEC::pack(t1), SPEC::pack(t2)}; }
};

}  // namespace gisspa
