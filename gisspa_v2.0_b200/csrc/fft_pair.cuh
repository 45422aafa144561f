// fft_pair.cuh — register Stockham FFTs of the paired-template correlation (corr_pair.cu): one
// complex number per value (float2) or two side by side (Cx2), the same butterflies for both.
//
// Exchanges go through shared memory at padded positions whose offsets are affine in the
// element number, so every access of a stage is one base address plus a constant: the XOR
// swizzle of fft.cuh cost three to four integer instructions per access, a quarter of all
// instructions the column and row passes issued.
#pragma once

#include "fft.cuh"

namespace gisspa {

// Two complex numbers a, b as (a.re, b.re), (a.im, b.im): every add, subtract and constant
// multiply of a butterfly is one paired FP32 instruction for both, and a multiplication by i
// is a renaming, where (re, im) pairs need moves.
struct Cx2 {
  float2 re, im;
};

__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return cadd(a, b); }
__device__ __forceinline__ float2 vsub(float2 a, float2 b) { return csub(a, b); }
__device__ __forceinline__ Cx2 vadd(Cx2 a, Cx2 b) { return Cx2{cadd(a.re, b.re), cadd(a.im, b.im)}; }
__device__ __forceinline__ Cx2 vsub(Cx2 a, Cx2 b) { return Cx2{csub(a.re, b.re), csub(a.im, b.im)}; }

// x times the complex number w (scalar products: a twiddle that is used once or twice is not
// worth duplicating into both halves of a pair)
__device__ __forceinline__ float2 vmulw(float2 x, float2 w) { return cmul(x, w); }
__device__ __forceinline__ Cx2 vmulw(Cx2 x, float2 w) {
  return Cx2{make_float2(x.re.x * w.x - x.im.x * w.y, x.re.y * w.x - x.im.y * w.y),
             make_float2(x.re.x * w.y + x.im.x * w.x, x.re.y * w.y + x.im.y * w.x)};
}

// a = e + SIGN i o, b = e - SIGN i o
template <int SIGN>
__device__ __forceinline__ void bf_i(float2 e, float2 o, float2& a, float2& b) {
  const float2 p = make_float2(e.x - o.y, e.y + o.x), m = make_float2(e.x + o.y, e.y - o.x);
  a = SIGN > 0 ? p : m;
  b = SIGN > 0 ? m : p;
}
template <int SIGN>
__device__ __forceinline__ void bf_i(Cx2 e, Cx2 o, Cx2& a, Cx2& b) {
  const Cx2 p{csub(e.re, o.im), cadd(e.im, o.re)}, m{cadd(e.re, o.im), csub(e.im, o.re)};
  a = SIGN > 0 ? p : m;
  b = SIGN > 0 ? m : p;
}

// a = e + w o, b = e - w o for the constant w = exp(SIGN 2 pi i K / R): with w = c (1 + i t),
// t = tan, u = (1 + i t) o takes one multiply-add per part and a, b = e +- c u one more each
// (six instead of eight); where |sin| > |cos| the cotangent form, so that |t| <= 1.
template <int R, int K, int SIGN>
__device__ __forceinline__ void bf_w(float2 e, float2 o, float2& a, float2& b) {
  constexpr double c = root_cos<R>(K), s = SIGN * root_sin<R>(K);
  if constexpr (c * c >= s * s) {
    constexpr float t = (float)(s / c), f = (float)c;
    const float2 u = make_float2(fmaf(-t, o.y, o.x), fmaf(t, o.x, o.y));
    a = pfma(u, make_float2(f, f), e);
    b = pfma(u, make_float2(-f, -f), e);
  } else {
    constexpr float t = (float)(c / s), f = (float)s;
    // w o = s (t o.x - o.y, t o.y + o.x)
    const float2 u = make_float2(fmaf(t, o.x, -o.y), fmaf(t, o.y, o.x));
    a = pfma(u, make_float2(f, f), e);
    b = pfma(u, make_float2(-f, -f), e);
  }
}
template <int R, int K, int SIGN>
__device__ __forceinline__ void bf_w(Cx2 e, Cx2 o, Cx2& a, Cx2& b) {
  constexpr double c = root_cos<R>(K), s = SIGN * root_sin<R>(K);
  if constexpr (8 * K == R || 8 * K == 3 * R) {  // t = +-1
    constexpr float f = (float)c;
    constexpr bool plus = s * c > 0;
    const float2 ur = plus ? csub(o.re, o.im) : cadd(o.re, o.im);
    const float2 ui = plus ? cadd(o.im, o.re) : csub(o.im, o.re);
    const float2 fp = make_float2(f, f), fm = make_float2(-f, -f);
    a = Cx2{pfma(ur, fp, e.re), pfma(ui, fp, e.im)};
    b = Cx2{pfma(ur, fm, e.re), pfma(ui, fm, e.im)};
  } else if constexpr (c * c >= s * s) {
    constexpr float t = (float)(s / c), f = (float)c;
    const float2 ur = pfma(o.im, make_float2(-t, -t), o.re), ui = pfma(o.re, make_float2(t, t), o.im);
    const float2 fp = make_float2(f, f), fm = make_float2(-f, -f);
    a = Cx2{pfma(ur, fp, e.re), pfma(ui, fp, e.im)};
    b = Cx2{pfma(ur, fm, e.re), pfma(ui, fm, e.im)};
  } else {
    // w o = s (-vr, ui) with vr = o.im - t o.re, ui = o.re + t o.im
    constexpr float t = (float)(c / s), f = (float)s;
    const float2 vr = pfma(o.re, make_float2(-t, -t), o.im), ui = pfma(o.im, make_float2(t, t), o.re);
    const float2 fp = make_float2(f, f), fm = make_float2(-f, -f);
    a = Cx2{pfma(vr, fm, e.re), pfma(ui, fp, e.im)};
    b = Cx2{pfma(vr, fp, e.re), pfma(ui, fm, e.im)};
  }
}

// x times the constant exp(SIGN 2 pi i K / R)
template <int R, int K, int SIGN>
__device__ __forceinline__ float2 vmulc(float2 v) { return mul_wr<R, K, SIGN>(v); }
template <int R, int K, int SIGN>
__device__ __forceinline__ Cx2 vmulc(Cx2 v) {
  constexpr int KK = K % R;
  if constexpr (KK == 0) {
    return v;
  } else {
    constexpr float c = (float)root_cos<R>(KK), s = (float)(SIGN * root_sin<R>(KK));
    const float2 cc = make_float2(c, c), sp = make_float2(s, s), sm = make_float2(-s, -s);
    return Cx2{pfma(v.im, sm, pmul(v.re, cc)), pfma(v.re, sp, pmul(v.im, cc))};
  }
}

// In-register DFT of length R, natural order in and out; V is float2 or Cx2.
template <typename V, int R, int SIGN>
struct RegDft {
  template <int K>
  __device__ __forceinline__ static void combine(V* a, const V* e, const V* o) {
    if constexpr (K < R / 2) {
      if constexpr (K == 0) {
        a[0] = vadd(e[0], o[0]);
        a[R / 2] = vsub(e[0], o[0]);
      } else if constexpr (4 * K == R) {
        bf_i<SIGN>(e[K], o[K], a[K], a[K + R / 2]);
      } else {
        bf_w<R, K, SIGN>(e[K], o[K], a[K], a[K + R / 2]);
      }
      combine<K + 1>(a, e, o);
    }
  }
  __device__ __forceinline__ static void run(V* a) {
    if constexpr (R == 2) {
      const V t = a[1];
      a[1] = vsub(a[0], t);
      a[0] = vadd(a[0], t);
    } else if constexpr (R > 2) {
      V e[R / 2], o[R / 2];
#pragma unroll
      for (int m = 0; m < R / 2; ++m) {
        e[m] = a[2 * m];
        o[m] = a[2 * m + 1];
      }
      RegDft<V, R / 2, SIGN>::run(e);
      RegDft<V, R / 2, SIGN>::run(o);
      combine<0>(a, e, o);
    }
  }
};

__device__ __forceinline__ float2 vscale_add(float2 x, float c1, float2 t1, float c2, float2 t2) {
  return pfma(t2, make_float2(c2, c2), pfma(t1, make_float2(c1, c1), x));
}
__device__ __forceinline__ Cx2 vscale_add(Cx2 x, float c1, Cx2 t1, float c2, Cx2 t2) {
  return Cx2{vscale_add(x.re, c1, t1.re, c2, t2.re), vscale_add(x.im, c1, t1.im, c2, t2.im)};
}
__device__ __forceinline__ float2 vlin(float c1, float2 t1, float c2, float2 t2) {
  return pfma(t2, make_float2(c2, c2), pmul(t1, make_float2(c1, c1)));
}
__device__ __forceinline__ Cx2 vlin(float c1, Cx2 t1, float c2, Cx2 t2) {
  return Cx2{vlin(c1, t1.re, c2, t2.re), vlin(c1, t1.im, c2, t2.im)};
}

// 5-point DFT from the symmetric pairs, as Dft<5> (fft.cuh)
template <typename V, int SIGN>
struct RegDft<V, 5, SIGN> {
  __device__ __forceinline__ static void run(V* a) {
    constexpr float c1 = (float)cos20(4), c2 = (float)cos20(8), s1 = (float)sin20(4), s2 = (float)sin20(8);
    const V t1 = vadd(a[1], a[4]), t2 = vadd(a[2], a[3]), t3 = vsub(a[1], a[4]), t4 = vsub(a[2], a[3]);
    const V x0 = a[0];
    const V p1 = vscale_add(x0, c1, t1, c2, t2), p2 = vscale_add(x0, c2, t1, c1, t2);
    const V q = vlin(s1, t3, s2, t4), r = vlin(s2, t3, -s1, t4);
    a[0] = vadd(x0, vadd(t1, t2));
    bf_i<SIGN>(p1, q, a[1], a[4]);
    bf_i<SIGN>(p2, r, a[2], a[3]);
  }
};

// 20 = 4 x 5, as DftAB<4, 5>
template <typename V, int SIGN>
struct RegDft<V, 20, SIGN> {
  template <int N2, int K1>
  __device__ __forceinline__ static void twiddle(V (&y)[5][4]) {
    if constexpr (N2 < 5) {
      if constexpr (K1 < 4) {
        y[N2][K1] = vmulc<20, N2 * K1, SIGN>(y[N2][K1]);
        twiddle<N2, K1 + 1>(y);
      } else {
        twiddle<N2 + 1, 0>(y);
      }
    }
  }
  __device__ __forceinline__ static void run(V* a) {
    V y[5][4];
#pragma unroll
    for (int n2 = 0; n2 < 5; ++n2) {
#pragma unroll
      for (int n1 = 0; n1 < 4; ++n1) y[n2][n1] = a[5 * n1 + n2];
      RegDft<V, 4, SIGN>::run(y[n2]);
    }
    twiddle<0, 0>(y);
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) {
      V z[5];
#pragma unroll
      for (int n2 = 0; n2 < 5; ++n2) z[n2] = y[n2][k1];
      RegDft<V, 5, SIGN>::run(z);
#pragma unroll
      for (int k2 = 0; k2 < 5; ++k2) a[k1 + 4 * k2] = z[k2];
    }
  }
};

// Column plans: two stages of radix R1 and R2, R1 R2 = L, one exchange; L / R1 threads hold a
// column's R1 points each in the first stage.
template <int L>
struct ColPlan;
template <> struct ColPlan<256> { static constexpr int R1 = 16, R2 = 16; };
template <> struct ColPlan<320> { static constexpr int R1 = 20, R2 = 16; };
template <> struct ColPlan<512> { static constexpr int R1 = 32, R2 = 16; };
template <> struct ColPlan<1024> { static constexpr int R1 = 32, R2 = 32; };

// Row plans: T lanes per row with R1 = L / T points each, stages R1, R2 and (L = 320) R3.
template <int L>
struct RowPlan2;
template <> struct RowPlan2<256> { static constexpr int T = 16, R1 = 16, R2 = 16, R3 = 1; };
template <> struct RowPlan2<320> { static constexpr int T = 16, R1 = 20, R2 = 4, R3 = 4; };
template <> struct RowPlan2<512> { static constexpr int T = 16, R1 = 32, R2 = 16, R3 = 1; };
template <> struct RowPlan2<1024> { static constexpr int T = 32, R1 = 32, R2 = 32, R3 = 1; };

// Place of element i in a row's first exchange: thread t stores the block R1 t .. R1 t + R1 - 1;
// one pad per block makes the blocks' stride odd, so that the lanes of a shared-memory phase
// fall in distinct banks.  (A second exchange needs no pad.)
template <int L>
__host__ __device__ constexpr int row_pos1(int i) {
  return i + i / RowPlan2<L>::R1;
}
// Values of one row's buffer.  The two rows of a pair sit side by side and a phase of 16 lanes
// takes 8 lanes of each: a stride of 8 mod 16 puts the second row's banks beside the first's.
template <int L>
__host__ __device__ constexpr int row_buf() {
  return (row_pos1<L>(L - 1) + 1 + 7) / 16 * 16 + 8;
}
static_assert(row_buf<512>() >= row_pos1<512>(511) + 1 && row_buf<320>() >= row_pos1<320>(319) + 1, "row buffers");

// Multiplies the inputs of a radix-R butterfly by their twiddles w1^m, m = 1 .. R - 1.
template <typename V, int R>
__device__ __forceinline__ void twiddle_inputs(V* a, float2 w1) {
  float2 w[R];
  tw_powers<R>(w1, w);
#pragma unroll
  for (int m = 1; m < R; ++m) a[m] = vmulw(a[m], w[m]);
}

}  // namespace gisspa
