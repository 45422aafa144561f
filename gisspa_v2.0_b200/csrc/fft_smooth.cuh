// fft_smooth.cuh — device routine of the mixed-radix Stockham transform in shared memory (register
// transforms of 2 to 16 points per stage), shared by the generic FFT engine and the correlation of
// window sizes without hand-tuned kernels.
#pragma once

#include "fft.cuh"
#include "fft_generic.cuh"

namespace gisspa {

// x[q] *= W_n^(q p), 1 <= q < R (conjugated for the inverse transform): one table read.
template <int R, int SIGN>
__device__ __forceinline__ void twiddle_powers(float2 (&x)[R], const float2* __restrict__ tw, int p) {
  float2 w[R];
  tw_powers<R>(table_tw<SIGN>(TwGlobal{tw}, p), w);
#pragma unroll
  for (int q = 1; q < R; ++q) x[q] = cmul(x[q], w[q]);
}

// The whole CTA, or a group of whole warps of it (named barrier 1 + index).
struct CtaTeam {
  __device__ __forceinline__ int id() const { return threadIdx.x; }
  __device__ __forceinline__ int size() const { return blockDim.x; }
  __device__ __forceinline__ void sync() const { __syncthreads(); }
};
struct WarpsTeam {
  int index, threads;
  __device__ __forceinline__ int id() const { return threadIdx.x - index * threads; }
  __device__ __forceinline__ int size() const { return threads; }
  __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(1 + index), "r"(threads) : "memory"); }
};

// One Stockham stage of radix R on `rows` rows of length n, after stages whose radices multiply to
// Ns: butterfly j < m = n/R of a row takes x_q = in(row, j + q m), applies the twiddles w^(q k),
// k = j mod Ns, w = e^(-+2 pi i/(Ns R)) (tw[p] = e^(-2 pi i p/n), one read and its powers), takes the
// R-point DFT and hands its outputs p to out(row, base, x) for the places base + p Ns, base =
// (j / Ns) Ns R + k: after the last stage the row is in natural order.
// team: the threads that share the work.
template <int R, int SIGN, typename Team, typename In, typename Out>
__device__ __forceinline__ void smooth_stage(const Team& team, int rows, int n, int Ns, unsigned div_m,
                                             unsigned div_ns, const float2* __restrict__ tw, In&& in, Out&& out) {
  const int m = n / R, nb = rows * m, tstep = m / Ns;
  for (int t = team.id(); t < nb; t += team.size()) {
    const int r = fast_div(t, div_m), j = t - r * m;
    float2 x[R];
    in(r, j, m, x);
    int base = j * R;
    if (Ns > 1) {
      const int g = fast_div(j, div_ns), k = j - g * Ns;
      base = g * Ns * R + k;
      twiddle_powers<R, SIGN>(x, tw, k * tstep);
    }
    Dft<R, SIGN>::run(x);
    out(r, base, x);
  }
}

template <int SIGN, typename Team, typename In, typename Out>
__device__ __forceinline__ void smooth_any(const Team& team, const SmoothPlan& plan, int s, int rows, int n, int Ns,
                                           const float2* __restrict__ tw, In&& in, Out&& out) {
  const unsigned dm = plan.div_m[s], dn = plan.div_ns[s];
  switch (plan.r[s]) {
    case 2: smooth_stage<2, SIGN>(team, rows, n, Ns, dm, dn, tw, in, out); break;
    case 3: smooth_stage<3, SIGN>(team, rows, n, Ns, dm, dn, tw, in, out); break;
    case 4: smooth_stage<4, SIGN>(team, rows, n, Ns, dm, dn, tw, in, out); break;
    case 5: smooth_stage<5, SIGN>(team, rows, n, Ns, dm, dn, tw, in, out); break;
    case 6: smooth_stage<6, SIGN>(team, rows, n, Ns, dm, dn, tw, in, out); break;
    case 7: smooth_stage<7, SIGN>(team, rows, n, Ns, dm, dn, tw, in, out); break;
    case 8: smooth_stage<8, SIGN>(team, rows, n, Ns, dm, dn, tw, in, out); break;
    case 10: smooth_stage<10, SIGN>(team, rows, n, Ns, dm, dn, tw, in, out); break;
    case 12: smooth_stage<12, SIGN>(team, rows, n, Ns, dm, dn, tw, in, out); break;
    case 14: smooth_stage<14, SIGN>(team, rows, n, Ns, dm, dn, tw, in, out); break;
    case 15: smooth_stage<15, SIGN>(team, rows, n, Ns, dm, dn, tw, in, out); break;
    default: smooth_stage<16, SIGN>(team, rows, n, Ns, dm, dn, tw, in, out); break;
  }
}

// Loads from and stores to rows in shared memory (row stride ld).
struct SmoothLoad {
  const float2* a;
  int ld;
  template <int R>
  __device__ __forceinline__ void operator()(int r, int j, int m, float2 (&x)[R]) const {
    const float2* in = a + r * ld + j;
#pragma unroll
    for (int q = 0; q < R; ++q) x[q] = in[q * m];
  }
};
struct SmoothStore {
  float2* b;
  int ld, Ns;
  template <int R>
  __device__ __forceinline__ void operator()(int r, int base, const float2 (&x)[R]) const {
    float2* out = b + r * ld + base;
#pragma unroll
    for (int p = 0; p < R; ++p) out[p * Ns] = x[p];
  }
};

// Runs stages [s0, s1) of `plan` (Ns: the product of the radices before s0) on `rows` rows of length
// n (row stride ld) held in a, ping-ponging with b (same shape).  The caller has synchronised the
// team after filling a; returns the buffer holding the result after a final synchronisation.
template <int SIGN, typename Team>
__device__ __forceinline__ float2* smooth_stages(const Team& team, float2* a, float2* b, int rows, int n, int ld,
                                                 const SmoothPlan& plan, int s0, int s1, int Ns,
                                                 const float2* __restrict__ tw) {
#pragma unroll 1
  for (int s = s0; s < s1; ++s) {
    smooth_any<SIGN>(team, plan, s, rows, n, Ns, tw, SmoothLoad{a, ld}, SmoothStore{b, ld, Ns});
    team.sync();
    float2* tmp = a;
    a = b;
    b = tmp;
    Ns *= plan.r[s];
  }
  return a;
}

}  // namespace gisspa
