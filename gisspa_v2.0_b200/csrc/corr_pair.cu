// corr_pair.cu — the correlation of sweep 1 with two templates per transform.
//
// A pair of real templates t1, t2 is carried through one complex transform: with T1, T2 their
// spectra and I a window's, W(k) = I(k) (conj T1(k) + i conj T2(k)) is the spectrum of
// c1 + i c2, the two correlation maps.  W is not Hermitian, but both halves come from the half
// spectra that are stored: with A_j = I conj T_j on the half plane,
//   W(k) = A1(k) + i A2(k),     W(-k) = conj(A1(k) - i A2(k)).
// Column pass: one thread team per column kx of the half plane transforms columns kx and -kx
// along ky side by side (the inverse transform of column -kx is the conjugate of the one of
// A1 - i A2), so both share the loads of I, the twiddles and the addresses.  Row pass: an
// ordinary complex transform of length L per row gives row y of both maps as its real and
// imaginary parts, with no Hermitian unpacking.
//
// Measured on B200 (window 512, FP32, 24 templates x 6 windows per launch, 1.9 GHz): 0.60 us per
// (window, template) correlation, column pass 0.34, row pass 0.26, against 0.83 for the
// one-template passes (correlate.cu); a 4096^2 search with 40 templates 393 instead of 518 ms,
// 1855 x 1919 at window 320 37 instead of 54 ms (0.58 us with the order in which Q is read, see the
// row pass; 1.7 us at window 1024 instead of 2.5).  The column pass is bound by L2 traffic (1.5 MB
// of spectra read and 1 MB of Q written per correlation; without its stores it takes 0.20, with
// a Q of 32 MB that stays in L2 0.26), the row pass by latency at 12 warps per SM (61 % of
// issue slots; 552 instructions per row and template pair against 1090).
#include <algorithm>
#include <cfloat>

#include "../../include/gisspa.h"
#include "correlate.cuh"
#include "fft_pair.cuh"
#include "pair_spec.cuh"

namespace gisspa {
namespace {

// Barrier of a team: a warp or half warp, or whole warps through named barrier 1 + team.
template <int T>
__device__ __forceinline__ void team_sync(int team) {
  if constexpr (T <= 32)
    __syncwarp();
  else
    asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "n"(T) : "memory");
}

// Writes v into the low or high half of w.
__device__ __forceinline__ void put_half(unsigned& w, int high, int v) {
  w = high ? (w & 0xFFFFu) | (unsigned)v << 16 : (w & 0xFFFF0000u) | (unsigned)v;
}

// Column pass: NC columns kx (and their mirror images -kx) per CTA, one (window, template pair)
// per blockIdx.y.  Stage 1: L / R1 threads per column, R1 points each, the loads coalesced
// along ky.  One exchange, then stage 2's butterflies are dealt over the CTA with the column as
// the fastest index, so its outputs leave in row segments straight from registers: no
// transposing tile.  A stage 2 butterfly holds rows y and y + L/2 of its column, which Q keeps
// side by side: Q[p][y][.] (y < L/2) is a row of (re, im, re', im'), with column kx < L/2 at kx,
// L/2 at L/2 and column L - kx (0 < kx < L/2) at L/2 + kx, so that a CTA's columns and their
// mirror images are two aligned segments of 16 NC bytes per row pair.
template <int L, int NC>
constexpr int col_buf() {
  // the phases of stage 2's loads take 8 columns (NC = 8: an odd stride) or 4 columns and 2
  // consecutive elements (NC = 4: a stride of 2 mod 8)
  constexpr int n = L + L / ColPlan<L>::R1;
  return NC >= 8 ? n | 1 : (n + 7) / 8 * 8 + 2;
}
template <int L, int NC>
constexpr int col_threads() {
  return NC * (L / ColPlan<L>::R1 > L / ColPlan<L>::R2 || L == 320 ? L / ColPlan<L>::R2 : L / ColPlan<L>::R1);
}
template <int L, typename SPEC, int NC, int MINB>
__global__ void __launch_bounds__(col_threads<L, NC>(), MINB)
    pair_cols_kernel(const float2* __restrict__ I, const typename SPEC::T* __restrict__ T, float4* __restrict__ Q,
                     int b0, int g0, int DP, const float2* __restrict__ twL, int chained) {
  constexpr int R1 = ColPlan<L>::R1, R2 = ColPlan<L>::R2, T1 = L / R1, T2 = L / R2, NZ = L / 2, HS = NZ + 1;
  constexpr int NT = col_threads<L, NC>(), BUF = col_buf<L, NC>();
  static_assert(R1 * R2 == L && NC * T1 <= NT && NC * T2 % NT == 0, "plan");
  extern __shared__ __align__(16) float4 xbuf[];  // [NC][BUF]
  griddep_launch_dependents();
  if (!chained) griddep_wait();  // the spectra may come from the kernel just before
  const int c0 = blockIdx.x * NC, tid = threadIdx.x;
  // all windows of a template pair, then the next pair: the row pass starts with the last ones
  const int E = gridDim.y / DP, d = blockIdx.y / E, e = blockIdx.y - d * E, p = e * DP + d;
  if (NC * T1 == NT || tid < NC * T1) {
    const int team = tid / T1, t = tid - team * T1, c = c0 + team;
    const float2* Ic = I + ((size_t)(b0 + e) * HS + c) * L + t;
    const typename SPEC::T* Tc = T + ((size_t)(g0 + d) * HS + c) * L + t;
    Cx2 v[R1];
    if (c == 0) {
      // columns 0 and L/2 are their own mirror images: they ride together
#pragma unroll
      for (int m = 0; m < R1; ++m) {
        const float2 a = SPEC::plus(__ldg(Ic + m * T1), Tc[m * T1]);
        const float2 b = SPEC::plus(__ldg(Ic + (size_t)NZ * L + m * T1), Tc[(size_t)NZ * L + m * T1]);
        v[m] = Cx2{make_float2(a.x, b.x), make_float2(a.y, b.y)};
      }
    } else {
#pragma unroll
      for (int m = 0; m < R1; ++m) v[m] = SPEC::both(__ldg(Ic + m * T1), Tc[m * T1]);
    }
    RegDft<Cx2, R1, +1>::run(v);
    float4* st = xbuf + team * BUF + (R1 + 1) * t;
#pragma unroll
    for (int r = 0; r < R1; ++r) st[r] = make_float4(v[r].re.x, v[r].re.y, v[r].im.x, v[r].im.y);
  }
  __syncthreads();
  if (chained) griddep_wait();  // Q is still being read by the previous row pass
  const int col = tid % NC, j0 = tid / NC;
  const unsigned long long keep = l2_keep_policy();
  const unsigned flip = c0 + col ? 0x80000000u : 0u;  // column -kx: the conjugate
  float4* Qp = Q + (size_t)p * NZ * L + c0 + col;
#pragma unroll
  for (int q = 0; q < NC * T2 / NT; ++q) {
    const int j = j0 + (NT / NC) * q;
    const float4* ld = xbuf + col * BUF + j;
    Cx2 x[R2];
#pragma unroll
    for (int m = 0; m < R2; ++m) {
      const float4 y = ld[m * (R1 + 1)];
      x[m] = Cx2{make_float2(y.x, y.y), make_float2(y.z, y.w)};
    }
    twiddle_inputs<Cx2, R2>(x, table_tw<+1>(TwGlobal{twL}, j));
    RegDft<Cx2, R2, +1>::run(x);
#pragma unroll
    for (int r = 0; r < R2 / 2; ++r) {
      const Cx2 u = x[r], w = x[r + R2 / 2];
      float4* o = Qp + (size_t)(j + r * R1) * L;
      store_hint(o, make_float4(u.re.x, u.im.x, w.re.x, w.im.x), keep);
      store_hint(o + NZ,
                 make_float4(u.re.y, __uint_as_float(__float_as_uint(u.im.y) ^ flip), w.re.y,
                             __uint_as_float(__float_as_uint(w.im.y) ^ flip)),
                 keep);
    }
  }
}

// Row pass: one team of 2 T threads per (row pair y, y + L/2; share of the launch's template
// pairs), even threads on row y and odd ones on row y + L/2: RB row pairs of one window per CTA,
// each one's template pairs dealt over DS teams, which keep the per-pixel sums of squares (and
// maxima) in registers and add them up in shared memory at the end.  Every team runs its own
// double-buffered stream of bulk copies (a row pair of Q is one contiguous block) on its own
// mbarriers, with no barrier of the CTA between pairs.  Every wait is bounded: on timeout the
// team raises *a.err and fetches no further rows.
// Q, 160 MB per launch, passes through an L2 that kept 33 MB of it.  The pairs are taken in descending
// order, the last written (whose stores ask to be kept) first: 57 MB; and each row pair's lines,
// dead once read, are discarded from L2, from where the next column pass would otherwise write them
// back to DRAM.  A 4096^2 search at window 512: 321 -> 311 ms by the discarding, -> 304 ms by the
// order and the stores' hint (the order alone: half of that).
template <int L, int RB, int DS, int EPI, int MINB>
__global__ void __launch_bounds__(2 * RowPlan2<L>::T* RB* DS, MINB)
    pair_rows_kernel(CorrArgs a, const float2* __restrict__ twL) {
  using P = RowPlan2<L>;
  constexpr int T = P::T, TT = 2 * T, E = L / T, R1 = P::R1, R2 = P::R2, R3 = P::R3;
  constexpr int RL = R3 > 1 ? R3 : R2, BL = E / RL;  // the last stage: radix, butterflies per thread
  constexpr int NT = RB * DS, BUF = row_buf<L>(), PAIR = 2 * BUF;  // float2 per row, per row pair
  constexpr bool TOPK = EPI == EPI_TOPK, MAXP = EPI == EPI_SUMMAX, BEST = TOPK || MAXP;
  static_assert(R1 * R2 * R3 == L && E == R1 && E % R2 == 0 && E % RL == 0, "plan");
  static_assert(TT == 32 || NT <= 15, "named barriers");
  extern __shared__ __align__(128) float2 stage[];  // [NT][2][PAIR]
  __shared__ __align__(8) uint64_t bars[NT][2];
  __shared__ unsigned pmax[MAXP ? kMaxListedTemplates : 1];
  const int team = threadIdx.x / TT, u = threadIdx.x - team * TT, t = u >> 1, h = u & 1;
  const int row = team % RB, s = team / RB;
  const int e = blockIdx.y, y = blockIdx.x * RB + row, win = a.b0 + e;
  const int angle = a.angle_state ? a.angle_state->index : a.angle;
  const int DP = (a.D + 1) / 2, np = (DP - s + DS - 1) / DS;  // this team's pairs s, s + DS, ..., from the last
  float2* buf = stage + (size_t)team * 2 * PAIR;
  if (u == 0) {
    mbar_init(&bars[team][0], 1);
    mbar_init(&bars[team][1], 1);
    fence_mbar_init();
  }
  if constexpr (MAXP)
    for (int d = threadIdx.x; d < a.D; d += NT * TT) pmax[d] = 0u;
  // the last stage's twiddles are loop invariant
  float2 wl[BL];
#pragma unroll
  for (int q = 0; q < BL; ++q) wl[q] = table_tw<+1>(TwGlobal{twL}, t + T * q);
  float s2[E], best[BEST ? E : 1];
  unsigned barg[TOPK ? E / 2 : 1];  // index within the launch + 1, two pixels to a word; 0: none
#pragma unroll
  for (int i = 0; i < E; ++i) {
    s2[i] = 0.f;
    if constexpr (BEST) best[i] = TOPK ? -FLT_MAX : -INFINITY;
    if constexpr (TOPK) barg[i / 2] = 0u;
  }
  const float inv = 1.0f / (float)(L * L);
  __syncthreads();
  griddep_launch_dependents();
  griddep_wait();  // Q comes from the column pass just before
  constexpr unsigned kBytes = L * (unsigned)sizeof(float4);
  static_assert(kBytes % 128 == 0, "whole lines");
  auto row_pair = [&](int k) {
    return reinterpret_cast<const float4*>(a.Q) + ((size_t)(e * DP + s + DS * (np - 1 - k)) * (L / 2) + y) * L;
  };
  auto issue = [&](int k) {
    fence_proxy_async_smem();
    mbar_expect_tx(&bars[team][k & 1], kBytes);
    bulk_g2s(buf + (k & 1) * PAIR, row_pair(k), kBytes, &bars[team][k & 1]);
  };
  if (u == 0) {
    if (np > 0) issue(0);
    if (np > 1) issue(1);
  }
  // where the upper half of the row's columns lies in Q: L - k at L/2 + k, L/2 at L/2
  const int up = 3 * (L / 2) - t, mid = t == 0 ? L / 2 : up - L / 2;
  bool ok = true;
  int failed = 0;
  for (int k = 0; k < np; ++k) {
    if (ok) {
      ok = mbar_wait(&bars[team][k & 1], (k >> 1) & 1, 4000000000LL);
      failed = k;
    }
    const int d = 2 * (s + DS * (np - 1 - k));
    const bool two = d + 1 < a.D;  // an odd template count leaves the last pair half empty
    float m1 = -INFINITY, m2 = -INFINITY;
    float2* in = buf + (k & 1) * PAIR + h;  // element i of this thread's row at 2 i
    float2* x = buf + (k & 1) * PAIR + h * BUF;
    float2 v[E];
#pragma unroll
    for (int m = 0; m < E; ++m) v[m] = in[2 * (m < E / 2 ? t + T * m : m == E / 2 ? mid : up - T * m)];
    if (ok) discard_lines(row_pair(k), kBytes, u, TT);  // (the row pair has been copied)
    team_sync<TT>(team);
    RegDft<float2, R1, +1>::run(v);
#pragma unroll
    for (int r = 0; r < R1; ++r) x[(R1 + 1) * t + r] = v[r];
    team_sync<TT>(team);
    if constexpr (R3 > 1) {
#pragma unroll
      for (int q = 0; q < E / R2; ++q)
#pragma unroll
        for (int m = 0; m < R2; ++m) v[q * R2 + m] = x[row_pos1<L>(t + T * q) + m * row_pos1<L>(L / R2)];
      team_sync<TT>(team);
#pragma unroll
      for (int q = 0; q < E / R2; ++q) {
        const int j = t + T * q;
        twiddle_inputs<float2, R2>(v + q * R2, table_tw<+1>(TwGlobal{twL}, (j % R1) * R3));
        RegDft<float2, R2, +1>::run(v + q * R2);
#pragma unroll
        for (int r = 0; r < R2; ++r) x[(j / R1) * R1 * R2 + j % R1 + r * R1] = v[q * R2 + r];
      }
      team_sync<TT>(team);
    }
#pragma unroll
    for (int q = 0; q < BL; ++q) {
      float2 z[RL];
#pragma unroll
      for (int m = 0; m < RL; ++m)
        z[m] = R3 > 1 ? x[t + T * q + m * (L / RL)] : x[t + T * q + m * (R1 + 1)];
      if (q == BL - 1) {  // the row has been read: its buffer takes the pair after the next
        team_sync<TT>(team);
        if (u == 0 && ok && k + 2 < np) issue(k + 2);
      }
      twiddle_inputs<float2, RL>(z, wl[q]);
      RegDft<float2, RL, +1>::run(z);
      // z[r] = (c1, c2) at transform column t + T q + r L / RL (raw values: the 1/L^2 is applied
      // when folding)
#pragma unroll
      for (int r = 0; r < RL; ++r) {
        const int i = q * RL + r;
        const float c1 = z[r].x, c2 = two ? z[r].y : 0.f;
        s2[i] = fmaf(c2, c2, fmaf(c1, c1, s2[i]));
        if constexpr (MAXP) {
          const float cm = two ? z[r].y : c1;
          best[i] = fmaxf(best[i], fmaxf(c1, cm));
          m1 = fmaxf(m1, c1);
          m2 = fmaxf(m2, cm);
        }
        if constexpr (TOPK) {  // (templates in descending order: equal values keep the lowest)
          if (two && c2 >= best[i]) {
            best[i] = c2;
            put_half(barg[i / 2], i & 1, d + 2);
          }
          if (c1 >= best[i]) {
            best[i] = c1;
            put_half(barg[i / 2], i & 1, d + 1);
          }
        }
      }
    }
    if constexpr (MAXP) {
      if (a.pair_max) {
        const unsigned k1 = __reduce_max_sync(0xffffffffu, float_key(m1 * inv));
        const unsigned k2 = __reduce_max_sync(0xffffffffu, float_key(m2 * inv));
        const int lane = threadIdx.x & 31;
        if (lane == 0) atomicMax(&pmax[d], k1);
        if (lane == 1 && two) atomicMax(&pmax[d + 1], k2);
      }
    }
  }
  if (!ok && u == 0) {
    atomicOr(a.err, 1u);
    // copies still in flight land before the CTA's shared memory is reused or goes away
    for (int k = failed; k < min(failed + 2, np); ++k) mbar_wait(&bars[team][k & 1], (k >> 1) & 1, 400000000LL);
  }
  if constexpr (DS > 1) {
    // the teams of a row pair meet in shared memory (every copy has landed and been read)
    __syncthreads();
    constexpr int NV = BEST ? 2 : 1, PER = (NV * E + (TOPK ? E / 2 : 0)) * TT;  // floats per team
    float* part = reinterpret_cast<float*>(stage);  // [DS - 1][RB][PER]
    static_assert((size_t)(DS - 1) * PER * sizeof(float) <= (size_t)DS * 2 * PAIR * sizeof(float2), "scratch");
    if (s > 0) {
      float* o = part + (size_t)((s - 1) * RB + row) * PER + u;
#pragma unroll
      for (int i = 0; i < E; ++i) {
        o[i * TT] = s2[i];
        if constexpr (BEST) o[(E + i) * TT] = best[i];
        if constexpr (TOPK)
          if (!(i & 1)) o[(2 * E + i / 2) * TT] = __uint_as_float(barg[i / 2]);
      }
    }
    __syncthreads();
    if (s > 0) return;
    for (int w = 0; w < DS - 1; ++w) {
      const float* o = part + (size_t)(w * RB + row) * PER + u;
#pragma unroll
      for (int i = 0; i < E; ++i) {
        s2[i] += o[i * TT];
        if constexpr (MAXP) best[i] = fmaxf(best[i], o[(E + i) * TT]);
        if constexpr (TOPK) {
          const float b = o[(E + i) * TT];
          const unsigned g2 = __float_as_uint(o[(2 * E + i / 2) * TT]);
          const unsigned g = i & 1 ? g2 >> 16 : g2 & 0xFFFFu, own = i & 1 ? barg[i / 2] >> 16 : barg[i / 2] & 0xFFFFu;
          if (g && (b > best[i] || (b == best[i] && (g < own || !own)))) {
            best[i] = b;
            put_half(barg[i / 2], i & 1, (int)g);
          }
        }
      }
    }
  } else if constexpr (MAXP) {
    __syncthreads();
  }
  if constexpr (MAXP) {
    if (a.pair_max)
      for (int d = threadIdx.x; d < a.D; d += RB * TT) {
        const int v = a.n0 + d, da = v / a.nt_real;  // image v: template v % nt at the da-th angle
        atomicMax(a.pair_max + pair_index(win, v - da * a.nt_real, angle + da, a.n_windows, a.n_angles), pmax[d]);
      }
  }
  // Fold into the per-pixel state with reductions that return nothing (no warp waits on the
  // state's memory latency); each pixel receives one per launch and launches are
  // stream-ordered, so the additions happen in a fixed order.  The zero lag moves to
  // (L/2, L/2): row y of the transform is window row y + L/2, row y + L/2 is row y.
  const int id0 = angle * a.nt_total + a.n0 - 1;
  const size_t base = ((size_t)win * L + y + (h ? 0 : L / 2)) * L;
#pragma unroll
  for (int i = 0; i < E; ++i) {
    const int xc = t + T * (i / RL) + (i % RL) * (L / RL);
    const size_t pix = base + (xc + L / 2) % L;
    atomicAdd(a.S2 + pix, (double)(s2[i] * (inv * inv)));
    if constexpr (BEST) {
      const unsigned key = float_key(best[i] * inv);
      if constexpr (TOPK) {
        const unsigned g = i & 1 ? barg[i / 2] >> 16 : barg[i / 2] & 0xFFFFu;
        if (g)
          atomicMax(a.peak + pix,
                    (unsigned long long)key << 32 | (unsigned)(0xFFFFFFFFu - (unsigned)(id0 + (int)g)));
      } else {
        atomicMax(a.peak32 + pix, key);
      }
    }
  }
}

// Half spectra X[n][kx][ky] of single templates -> pairs, scaled and with DC zeroed as
// finalize_spectra (prep.cu) does; an odd last template is paired with zeros.
template <typename SPEC>
__global__ void __launch_bounds__(256) pair_pack_kernel(const float2* __restrict__ X, int n, int l,
                                                        const double* __restrict__ sums,
                                                        typename SPEC::T* __restrict__ out, double base) {
  const int g = blockIdx.y;
  const bool two = 2 * g + 1 < n;
  const long long per = (long long)(l / 2 + 1) * l;
  const double L2 = (double)l * l;
  float fs[2] = {0.f, 0.f};
  for (int j = 0; j < (two ? 2 : 1); ++j) {
    const int i = 2 * g + j;
    const double mean = sums[2 * i] / L2, var = sums[2 * i + 1] / L2 - mean * mean;
    fs[j] = (float)(var != 0 ? base / sqrt(var) : base);
  }
  const float2* X1 = X + (size_t)2 * g * per;
  for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < per; k += (long long)gridDim.x * blockDim.x) {
    float2 t1 = make_float2(0.f, 0.f), t2 = t1;
    if (k) {  // mean subtracted: DC is exactly zero
      t1 = cscale(X1[k], fs[0]);
      if (two) t2 = cscale(X1[per + k], fs[1]);
    }
    out[(size_t)g * per + k] = SPEC::pack(t1, t2);
  }
}

// Adds the spectra of all templates (as stored) to the running sum, in FP64, one slot of tsum per
// blockIdx.y: the sum of the correlations over all templates and angles is the correlation with
// the sum of the templates (pair_sum_finish).
constexpr int kSumSlots = 8;
template <typename SPEC>
__global__ void __launch_bounds__(256) pair_sum_kernel(const typename SPEC::T* __restrict__ T, int np, long long per,
                                                       double2* __restrict__ tsum) {
  const int per_y = (np + gridDim.y - 1) / gridDim.y, g0 = blockIdx.y * per_y, g1 = min(np, g0 + per_y);
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= per) return;
  double2 acc = make_double2(0.0, 0.0);
#pragma unroll 8
  for (int g = g0; g < g1; ++g) {
    const double2 v = SPEC::sum(T[(size_t)g * per + k]);
    acc.x += v.x;
    acc.y += v.y;
  }
  double2* o = tsum + (size_t)blockIdx.y * per + k;
  o->x += acc.x;
  o->y += acc.y;
}

__global__ void pair_sum_finish_kernel(const double2* __restrict__ tsum, long long per, float2* __restrict__ out) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= per) return;
  double2 a = make_double2(0.0, 0.0);
  for (int y = 0; y < kSumSlots; ++y) {
    a.x += tsum[y * per + k].x;
    a.y += tsum[y * per + k].y;
  }
  out[k] = make_float2((float)a.x, (float)a.y);
}

template <typename... P, typename... A>
void launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  GISSPA_CUDA(cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...));
  ++launch_counter();
}

// Columns per CTA and CTAs per SM of the column pass; row pairs per CTA of the row pass and its
// resident warps per SM (the register cap).
template <int L>
struct PairShape;
template <> struct PairShape<256> { static constexpr int NC = 8, MA = 4, RB = 2, WARPS = 16; };
template <> struct PairShape<320> { static constexpr int NC = 8, MA = 3, RB = 2, WARPS = 16; };
template <> struct PairShape<1024> { static constexpr int NC = 4, MA = 3, RB = 1, WARPS = 12; };
template <> struct PairShape<512> { static constexpr int NC = 8, MA = 3, RB = 1, WARPS = 12; };

template <int L, typename SPEC>
void cols(const CorrLaunch& cl, const float2* I, const void* T, float2* Q, const CorrArgs& a, const float2* twL,
          cudaStream_t s) {
  using S = PairShape<L>;
  auto* kernel = pair_cols_kernel<L, SPEC, S::NC, S::MA>;
  constexpr size_t smem = (size_t)S::NC * col_buf<L, S::NC>() * sizeof(float4);
  static PerDeviceOnce once;
  once([&] { GISSPA_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); });
  const int DP = (cl.D + 1) / 2;
  launch_pdl(kernel, dim3(L / 2 / S::NC, cl.E * DP), dim3(col_threads<L, S::NC>()), smem, s, I,
             static_cast<const typename SPEC::T*>(T), reinterpret_cast<float4*>(Q), a.b0, a.n0 / 2, DP, twL,
             cl.chained ? 1 : 0);
}

template <int L, int EPI, int DS>
void rows_ds(const CorrLaunch& cl, const CorrArgs& a, const float2* twL, cudaStream_t s) {
  using S = PairShape<L>;
  constexpr int threads = 2 * RowPlan2<L>::T * S::RB * DS;
  auto* kernel = pair_rows_kernel<L, S::RB, DS, EPI, S::WARPS * 32 / threads>;
  constexpr size_t smem = (size_t)S::RB * DS * 4 * row_buf<L>() * sizeof(float2);
  static PerDeviceOnce once;
  once([&] { GISSPA_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); });
  launch_pdl(kernel, dim3(L / 2 / S::RB, cl.E), dim3(threads), smem, s, a, twL);
}

// Shares per row pair: a launch has L / 2 x E row pairs, each a team's serial chain over the
// template pairs; where that leaves half or more of the chip's warp slots empty the chains are
// cut in two or three.
template <int L, int EPI>
void rows(const CorrLaunch& cl, const CorrArgs& a, const float2* twL, cudaStream_t s) {
  const int slots = 148 * PairShape<L>::WARPS / (RowPlan2<L>::T / 16), chains = L / 2 * cl.E, pairs = (cl.D + 1) / 2;
  const int ds = std::min(slots / chains, pairs);
  if (ds >= 3 && PairShape<L>::RB == 1)
    rows_ds<L, EPI, PairShape<L>::RB == 1 ? 3 : 2>(cl, a, twL, s);
  else if (ds >= 2)
    rows_ds<L, EPI, 2>(cl, a, twL, s);
  else
    rows_ds<L, EPI, 1>(cl, a, twL, s);
}

template <int L>
void launch(const CorrLaunch& cl, const float2* I, const void* T, float2* Q, const CorrArgs& a, const float2* twL,
            cudaStream_t s, cudaEvent_t* ev) {
  if (ev) GISSPA_CUDA(cudaEventRecord(ev[0], s));
  switch (cl.spec) {
    case GISSPA_SPEC_FP32: cols<L, PairFp32>(cl, I, T, Q, a, twL, s); break;
    case GISSPA_SPEC_FP16: cols<L, PairHalf<SpecFp16>>(cl, I, T, Q, a, twL, s); break;
    default: cols<L, PairHalf<SpecBf16>>(cl, I, T, Q, a, twL, s); break;
  }
  if (ev) GISSPA_CUDA(cudaEventRecord(ev[1], s));
  switch (cl.epi) {
    case EPI_SUM: rows<L, EPI_SUM>(cl, a, twL, s); break;
    case EPI_SUMMAX: rows<L, EPI_SUMMAX>(cl, a, twL, s); break;
    default: rows<L, EPI_TOPK>(cl, a, twL, s); break;
  }
  if (ev) GISSPA_CUDA(cudaEventRecord(ev[2], s));
}

}  // namespace

bool pair_supported(int L, int epi) {
  return (L == 256 || L == 320 || L == 512 || L == 1024) && (epi == EPI_SUM || epi == EPI_SUMMAX || epi == EPI_TOPK);
}

// Windows and templates per launch.  E fills the row pass's team slots with one chain per row
// pair; D then makes the state's reductions (12 bytes per pixel and launch) small beside the D/2
// row pairs of Q they stand for, with at most 160 MB of Q.  At window 1024 one window's chains fill
// 0.58 of the slots and three's 1.73 (two rounds, 0.86): three windows and 240 MB of Q, evened out
// over the windows (a 3838 x 3710 search: 85.8 ms; 1 window x 20 templates 105, 3 x 10 88.9, 5 x 16
// 91.7; one-template passes 116).
void pair_batch(int L, int W, int nt, int& D, int& E) {
  if (L == 1024)
    E = ceil_div(W, ceil_div(W, 3));
  else
    E = std::max(1, std::min(W, 148 * (L == 512 ? 12 : 16) / (L / 2)));
  const long long cap = ((L == 1024 ? 240LL : 160LL) << 20) / ((long long)L * L * 4) / E;
  D = (int)std::min<long long>(std::max<long long>(cap, 2), kMaxListedTemplates) & ~1;
  const int n = (nt + D - 1) / D;  // launches per window batch, evened out
  D = ((nt + n - 1) / n + 1) & ~1;
}

size_t pair_spectrum_bytes(int L, int spec) {
  return (size_t)(L / 2 + 1) * L * (spec == GISSPA_SPEC_FP32 ? sizeof(float4) : 2 * sizeof(__half2));
}

size_t pair_sum_bytes(int L) { return sizeof(double2) * kSumSlots * (size_t)(L / 2 + 1) * L; }

void pair_pack(const float2* X, int n, int L, const double* sums, int spec, void* out, double base, cudaStream_t s) {
  const dim3 grid((unsigned)std::min(ceil_div((long long)(L / 2 + 1) * L, 1024), 512), (unsigned)((n + 1) / 2));
  if (spec == GISSPA_SPEC_FP16)
    pair_pack_kernel<PairHalf<SpecFp16>>
        <<<grid, 256, 0, s>>>(X, n, L, sums, static_cast<PairHalf<SpecFp16>::T*>(out), base);
  else if (spec == GISSPA_SPEC_BF16)
    pair_pack_kernel<PairHalf<SpecBf16>>
        <<<grid, 256, 0, s>>>(X, n, L, sums, static_cast<PairHalf<SpecBf16>::T*>(out), base);
  else
    throw CudaError{cudaErrorInvalidValue, "FP32 pairs come from tmpl_spectra"};
  GISSPA_LAUNCH_CHECK();
}

void pair_sum(const void* T, int nt, int L, int spec, void* tsum, cudaStream_t s) {
  const long long per = (long long)(L / 2 + 1) * L;
  const int np = (nt + 1) / 2;
  const dim3 grid((unsigned)ceil_div(per, 256), (unsigned)std::min(kSumSlots, np));
  double2* ts = static_cast<double2*>(tsum);
  switch (spec) {
    case GISSPA_SPEC_FP32:
      pair_sum_kernel<PairFp32><<<grid, 256, 0, s>>>(static_cast<const PairFp32::T*>(T), np, per, ts);
      break;
    case GISSPA_SPEC_FP16:
      pair_sum_kernel<PairHalf<SpecFp16>>
          <<<grid, 256, 0, s>>>(static_cast<const PairHalf<SpecFp16>::T*>(T), np, per, ts);
      break;
    default:
      pair_sum_kernel<PairHalf<SpecBf16>>
          <<<grid, 256, 0, s>>>(static_cast<const PairHalf<SpecBf16>::T*>(T), np, per, ts);
      break;
  }
  GISSPA_LAUNCH_CHECK();
}

void pair_sum_finish(const void* tsum, int L, float2* out, cudaStream_t s) {
  const long long per = (long long)(L / 2 + 1) * L;
  pair_sum_finish_kernel<<<ceil_div(per, 256), 256, 0, s>>>(static_cast<const double2*>(tsum), per, out);
  GISSPA_LAUNCH_CHECK();
}

void pair_launch(const CorrLaunch& cl, const float2* I, const void* T, float2* Q, const CorrArgs& args,
                 const float2* twL, cudaStream_t s, cudaEvent_t* ev) {
  switch (cl.L) {
    case 256: launch<256>(cl, I, T, Q, args, twL, s, ev); break;
    case 320: launch<320>(cl, I, T, Q, args, twL, s, ev); break;
    case 512: launch<512>(cl, I, T, Q, args, twL, s, ev); break;
    case 1024: launch<1024>(cl, I, T, Q, args, twL, s, ev); break;
    default: throw CudaError{cudaErrorInvalidValue, "window size without paired correlation kernels"};
  }
}

}  // namespace gisspa
