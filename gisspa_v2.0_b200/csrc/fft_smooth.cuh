// fft_smooth.cuh — device routine of the mixed-radix Stockham transform in shared memory (register
// transforms of 2 to 16 points per stage), shared by the generic FFT engine and the correlation of
// window sizes without hand-tuned kernels.
#pragma once

#include "fft.cuh"
#include "fft_generic.cuh"

namespace gisspa {

// One butterfly of a Stockham stage of radix R for rows of length n, after stages whose
// radices multiply to Ns: butterfly j < m = n/R reads x_q = in[j + q m], applies the twiddles
// w^(q k), k = j mod Ns, w = e^(-+2 pi i/(Ns R)) (tw[p] = e^(-2 pi i p/n), one read and its powers),
// takes the R-point DFT and writes out[(j / Ns) Ns R + k + p Ns]: after the last stage the row is in
// natural order.
template <int R, int SIGN>
__device__ __forceinline__ void smooth_butterfly(const float2* __restrict__ in, float2* __restrict__ out, int m,
                                                 int Ns, int tstep, unsigned div_ns, int j,
                                                 const float2* __restrict__ tw) {
  float2 x[R];
#pragma unroll
  for (int q = 0; q < R; ++q) x[q] = in[j + q * m];
  int base = j * R;
  if (Ns > 1) {
    const int g = fast_div(j, div_ns), k = j - g * Ns;
    base = g * Ns * R + k;
    float2 w[R];
    tw_powers<R>(table_tw<SIGN>(TwGlobal{tw}, k * tstep), w);
#pragma unroll
    for (int q = 1; q < R; ++q) x[q] = cmul(x[q], w[q]);
  }
  Dft<R, SIGN>::run(x);
#pragma unroll
  for (int p = 0; p < R; ++p) out[base + p * Ns] = x[p];
}

template <int R, int SIGN>
__device__ __forceinline__ void smooth_stage(const float2* __restrict__ a, float2* __restrict__ b, int rows, int n,
                                             int ld, int Ns, unsigned div_m, unsigned div_ns,
                                             const float2* __restrict__ tw) {
  const int m = n / R, nb = rows * m, tstep = m / Ns;
  for (int t = threadIdx.x; t < nb; t += blockDim.x) {
    const int r = fast_div(t, div_m), j = t - r * m;
    smooth_butterfly<R, SIGN>(a + r * ld, b + r * ld, m, Ns, tstep, div_ns, j, tw);
  }
}

// Runs every stage of `plan` on `rows` rows of length n (row stride ld) held in a, ping-
// ponging with b (same shape).  The caller has synchronised the block after filling a; returns
// the buffer holding the result, in natural order, after a final __syncthreads.
template <int SIGN>
__device__ __forceinline__ float2* smooth_stages(float2* a, float2* b, int rows, int n, int ld, const SmoothPlan& plan,
                                                 const float2* __restrict__ tw) {
  int Ns = 1;
#pragma unroll 1
  for (int s = 0; s < plan.ns; ++s) {
    const int R = plan.r[s];
    const unsigned dm = plan.div_m[s], dn = plan.div_ns[s];
    switch (R) {
      case 2: smooth_stage<2, SIGN>(a, b, rows, n, ld, Ns, dm, dn, tw); break;
      case 3: smooth_stage<3, SIGN>(a, b, rows, n, ld, Ns, dm, dn, tw); break;
      case 4: smooth_stage<4, SIGN>(a, b, rows, n, ld, Ns, dm, dn, tw); break;
      case 5: smooth_stage<5, SIGN>(a, b, rows, n, ld, Ns, dm, dn, tw); break;
      case 6: smooth_stage<6, SIGN>(a, b, rows, n, ld, Ns, dm, dn, tw); break;
      case 7: smooth_stage<7, SIGN>(a, b, rows, n, ld, Ns, dm, dn, tw); break;
      case 8: smooth_stage<8, SIGN>(a, b, rows, n, ld, Ns, dm, dn, tw); break;
      case 10: smooth_stage<10, SIGN>(a, b, rows, n, ld, Ns, dm, dn, tw); break;
      case 12: smooth_stage<12, SIGN>(a, b, rows, n, ld, Ns, dm, dn, tw); break;
      case 14: smooth_stage<14, SIGN>(a, b, rows, n, ld, Ns, dm, dn, tw); break;
      case 15: smooth_stage<15, SIGN>(a, b, rows, n, ld, Ns, dm, dn, tw); break;
      default: smooth_stage<16, SIGN>(a, b, rows, n, ld, Ns, dm, dn, tw); break;
    }
    __syncthreads();
    float2* tmp = a;
    a = b;
    b = tmp;
    Ns *= R;
  }
  return a;
}

}  // namespace gisspa
