// tmpl_spectra.cu — per-angle FP32 template spectra at the window sizes with register transforms
// (256, 320, 512, 1024): RotateTemplate (norm.cu:479-521) in two kernels.  (FP16 and BF16 spectra
// stay with the one-template kernels of prep.cu and fft_generic.cu: this transform differs from
// those in its last bits, and a value within 1e-7 of a rounding boundary of a 16-bit type would land
// on its other side: 2e-5 of a BF16 search's sums.)
//
// Two real templates make one complex image t1 + i t2, so one transform serves both.
//   rows:    samples both rotated, masked templates along a row (no rotated image is stored),
//            transforms the row and writes it; adds up each template's sum and sum of squares
//   columns: splits column pairs kx, -kx into the two templates' columns
//            (T1 = (F(kx) + conj F(-kx)) / 2, T2 = (F(kx) - conj F(-kx)) / 2i), transforms both
//            side by side along y, scales by 1 / (L^2 sigma), zeroes DC and writes the layout that
//            the correlation reads
// Per template and angle 12 L^2 bytes move, against 56 L^2 for rotating, transforming rows,
// transposing, transforming columns and scaling in kernels of their own; both are bound by L2 / HBM
// traffic and by the latency of the bilinear gathers.
#include <cmath>

#include "correlate.cuh"
#include "fft_pair.cuh"
#include "pair_spec.cuh"
#include "tmpl_spectra.cuh"

namespace gisspa {
namespace {

constexpr int kRows = 8;  // rows (or columns) per CTA

template <int L>
constexpr int spectra_threads() {
  // stage 1 takes L / R1 threads a row, stage 2 L / R2 butterflies a row: the larger at L = 320
  return kRows * (L == 320 ? L / ColPlan<L>::R2 : L / ColPlan<L>::R1);
}
// Row buffer: one pad per block of R1; odd, so that 8 rows or columns fall in distinct banks.
template <int L>
constexpr int spectra_buf() {
  return (L + L / ColPlan<L>::R1) | 1;
}

__device__ __forceinline__ double warp_add(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Bilinear sampling position of a rotated image (rotate_subIMG, kernels.cu:545-579, with its float
// expressions).
struct Sample {
  int k0, dx, dy;
  float fx, fy;
  bool inside;
};
template <int L>
__device__ __forceinline__ Sample sample_at(float x, float y, float cose, float sine) {
  const float x2 = (cose * x + sine * y) + L / 2;
  const float y2 = (-sine * x + cose * y) + L / 2;
  Sample s;
  s.inside = !(x2 < 0 || x2 > L - 1.0f || y2 < 0 || y2 > L - 1.0f);
  const int ii = s.inside ? (int)floorf(x2) : 0, jj = s.inside ? (int)floorf(y2) : 0;
  s.dx = ii == L - 1 ? 0 : 1;
  s.dy = jj == L - 1 ? 0 : L;
  s.k0 = ii + jj * L;
  s.fx = x2 - ii;
  s.fy = y2 - jj;
  return s;
}
__device__ __forceinline__ float sample(const float* __restrict__ src, const Sample& s) {
  const float gx = 1.0f - s.fx, gy = 1.0f - s.fy;
  const float v = src[s.k0] * gx * gy + src[s.k0 + s.dx] * s.fx * gy + src[s.k0 + s.dx + s.dy] * s.fx * s.fy +
                  src[s.k0 + s.dy] * gx * s.fy;
  return s.inside ? v : 0.f;
}

// blockIdx.x: 8 rows, blockIdx.y: pair of the launch, pair list[blockIdx.y] where a list is given.
// Pair G holds images 2 G and 2 G + 1 of n = nt x angles (image v: template v % nt at angle
// st[v / nt], or at (cose, sine) without st).  A template always shares its transform with the
// same partner at one angle, so its values do not depend on what else is transformed.
template <int L>
__global__ void __launch_bounds__(spectra_threads<L>())
    rotated_rows_kernel(const float* __restrict__ src, const int* __restrict__ list, int n, int nt, float cose,
                        float sine, const float* __restrict__ pre, const float* __restrict__ mask, const float2* __restrict__ twL, float2* __restrict__ F,
                        double* __restrict__ sums, const AngleState* __restrict__ st) {
  constexpr int R1 = ColPlan<L>::R1, R2 = ColPlan<L>::R2, T1 = L / R1, T2 = L / R2, NT = spectra_threads<L>(),
                BUF = spectra_buf<L>();
  extern __shared__ __align__(16) float2 xrow[];  // [kRows][BUF]
  __shared__ double part[NT / 32][4];
  const int g = blockIdx.y, G = list ? list[g] : g, y0 = blockIdx.x * kRows, tid = threadIdx.x;
  const bool two = 2 * G + 1 < n;
  const int v1 = 2 * G, v2 = two ? v1 + 1 : v1, n1 = v1 % nt, n2 = v2 % nt;
  const float* s1 = src + (size_t)n1 * L * L;
  const float* s2 = src + (size_t)n2 * L * L;
  const float p1 = pre ? pre[n1] : 1.f, p2 = !two ? 0.f : pre ? pre[n2] : 1.f;
  float cose2 = cose, sine2 = sine;
  if (st) {
    cose = st[v1 / nt].cose;
    sine = st[v1 / nt].sine;
    cose2 = st[v2 / nt].cose;
    sine2 = st[v2 / nt].sine;
  }
  const bool same = v1 / nt == v2 / nt;
  double a1 = 0, q1 = 0, a2 = 0, q2 = 0;
  if (kRows * T1 == NT || tid < kRows * T1) {
    const int r = tid / T1, t = tid - r * T1, j = y0 + r;
    const float* mk = mask + (size_t)j * L;
    const float y = (float)(j - L / 2);
    float2 v[R1];
#pragma unroll
    for (int m = 0; m < R1; ++m) {
      const int i = t + T1 * m;
      const float mv = mk[i];
      float2 o = make_float2(0.f, 0.f);
      if (mv != 0.f) {
        const float x = (float)(i - L / 2);
        Sample w = sample_at<L>(x, y, cose, sine);
        o.x = sample(s1, w) * (mv * p1);
        if (!same) w = sample_at<L>(x, y, cose2, sine2);
        o.y = two ? sample(s2, w) * (mv * p2) : 0.f;
      }
      a1 += (double)o.x;
      q1 += (double)o.x * o.x;
      a2 += (double)o.y;
      q2 += (double)o.y * o.y;
      v[m] = o;
    }
    RegDft<float2, R1, -1>::run(v);
    float2* o = xrow + r * BUF + (R1 + 1) * t;
#pragma unroll
    for (int k = 0; k < R1; ++k) o[k] = v[k];
  }
  a1 = warp_add(a1);
  q1 = warp_add(q1);
  a2 = warp_add(a2);
  q2 = warp_add(q2);
  if ((tid & 31) == 0) {
    part[tid >> 5][0] = a1;
    part[tid >> 5][1] = q1;
    part[tid >> 5][2] = a2;
    part[tid >> 5][3] = q2;
  }
  __syncthreads();
  if (tid < 4 && (two || tid < 2)) {
    double a = 0;
    for (int w = 0; w < NT / 32; ++w) a += part[w][tid];
    atomicAdd(sums + 4 * g + tid, a);
  }
  float2* Fg = F + ((size_t)g * L + y0) * L;
  for (int q = tid; q < kRows * T2; q += NT) {
    const int r = q / T2, j = q - r * T2;
    const float2* ld = xrow + r * BUF + j;
    float2 x[R2];
#pragma unroll
    for (int m = 0; m < R2; ++m) x[m] = ld[m * (R1 + 1)];
    twiddle_inputs<float2, R2>(x, table_tw<-1>(TwGlobal{twL}, j));
    RegDft<float2, R2, -1>::run(x);
#pragma unroll
    for (int k = 0; k < R2; ++k) Fg[(size_t)r * L + j + k * R1] = x[k];
  }
}

// Where the column kernel puts pair G's values at point k.
struct PairOut {  // the paired correlation's interleaved pairs
  PairFp32::T* out;
  __device__ __forceinline__ void put(int G, int, size_t per, size_t k, float2 t1, float2 t2) const {
    out[(size_t)G * per + k] = PairFp32::pack(t1, t2);
  }
};
struct SingleOut {  // one half spectrum per image
  float2* out;
  __device__ __forceinline__ void put(int G, int n, size_t per, size_t k, float2 t1, float2 t2) const {
    out[(size_t)2 * G * per + k] = t1;
    if (2 * G + 1 < n) out[((size_t)2 * G + 1) * per + k] = t2;
  }
};

// blockIdx.x: 8 columns of the half plane, blockIdx.y: template pair.
template <int L, typename OUT>
__global__ void __launch_bounds__(spectra_threads<L>())
    spectra_cols_kernel(const float2* __restrict__ F, const int* __restrict__ list, int n,
                        const double* __restrict__ sums, double base, const float2* __restrict__ twL, OUT out) {
  constexpr int R1 = ColPlan<L>::R1, R2 = ColPlan<L>::R2, T1 = L / R1, T2 = L / R2, NT = spectra_threads<L>(),
                BUF = spectra_buf<L>(), HS = L / 2 + 1;
  extern __shared__ __align__(16) float4 xcol[];  // [kRows][BUF]
  __shared__ float fs[2];
  const int g = blockIdx.y, G = list ? list[g] : g, c0 = blockIdx.x * kRows, tid = threadIdx.x;
  if (tid < 2) {
    // half of the factor undoes the split's doubling
    const double L2 = (double)L * L, mean = sums[4 * g + 2 * tid] / L2,
                 var = sums[4 * g + 2 * tid + 1] / L2 - mean * mean;
    fs[tid] = 0.5f * (float)(var != 0 ? base / sqrt(var) : base);
  }
  if (kRows * T1 == NT || tid < kRows * T1) {
    const int col = tid % kRows, t = tid / kRows, c = min(c0 + col, L / 2), cm = c ? L - c : 0;
    const float2* Fg = F + (size_t)g * L * L;
    Cx2 v[R1];
#pragma unroll
    for (int m = 0; m < R1; ++m) {
      const float2 f = Fg[(size_t)(t + T1 * m) * L + c], h = Fg[(size_t)(t + T1 * m) * L + cm];
      v[m] = Cx2{make_float2(f.x + h.x, f.y + h.y), make_float2(f.y - h.y, h.x - f.x)};
    }
    RegDft<Cx2, R1, -1>::run(v);
    float4* o = xcol + col * BUF + (R1 + 1) * t;
#pragma unroll
    for (int k = 0; k < R1; ++k) o[k] = make_float4(v[k].re.x, v[k].re.y, v[k].im.x, v[k].im.y);
  }
  __syncthreads();
  const float f1 = fs[0], f2 = fs[1];
  for (int q = tid; q < kRows * T2; q += NT) {
    const int col = q / T2, j = q - col * T2, c = c0 + col;
    if (c >= HS) continue;
    const float4* ld = xcol + col * BUF + j;
    Cx2 x[R2];
#pragma unroll
    for (int m = 0; m < R2; ++m) {
      const float4 y = ld[m * (R1 + 1)];
      x[m] = Cx2{make_float2(y.x, y.y), make_float2(y.z, y.w)};
    }
    twiddle_inputs<Cx2, R2>(x, table_tw<-1>(TwGlobal{twL}, j));
    RegDft<Cx2, R2, -1>::run(x);
#pragma unroll
    for (int k = 0; k < R2; ++k) {
      float2 t1 = make_float2(x[k].re.x * f1, x[k].im.x * f1), t2 = make_float2(x[k].re.y * f2, x[k].im.y * f2);
      if (c == 0 && j + k * R1 == 0) t1 = t2 = make_float2(0.f, 0.f);  // mean subtracted: DC is exactly zero
      out.put(G, n, (size_t)HS * L, (size_t)c * L + j + k * R1, t1, t2);
    }
  }
}

// A power of two per template that brings its masked, unrotated deviation to about 1: the two
// templates of a pair are of one size in the shared transform whatever the mask leaves of each,
// and as a power of two it changes no bit of either (the scaling by 1 / sigma takes it out again).
__global__ void prescale_kernel(const double* __restrict__ sums, int n, double L2, float* __restrict__ pre) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const double mean = sums[2 * t] / L2, var = sums[2 * t + 1] / L2 - mean * mean;
  pre[t] = (var > 0 && isfinite(var)) ? ldexpf(1.f, -max(-60, min(60, ilogb(var) / 2))) : 1.f;
}

template <int L>
void run(const TmplSpectra& p, cudaStream_t s) {
  const int np = p.list ? p.n_list : (p.nt * p.na + 1) / 2;
  if (np <= 0) return;
  constexpr int NT = spectra_threads<L>();
  constexpr size_t smr = sizeof(float2) * kRows * spectra_buf<L>(), smc = sizeof(float4) * kRows * spectra_buf<L>();
  GISSPA_CUDA(cudaMemsetAsync(p.sums, 0, sizeof(double) * 4 * np, s));
  static PerDeviceOnce once_rows;
  if (smr > 48 * 1024)
    once_rows([&] {
      GISSPA_CUDA(cudaFuncSetAttribute(rotated_rows_kernel<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smr));
    });
  rotated_rows_kernel<L><<<dim3(L / kRows, np), NT, smr, s>>>(p.src, p.list, p.nt * p.na, p.nt, p.cose, p.sine, p.pre,
                                                               p.mask, p.twL, p.F, p.sums, p.st);
  GISSPA_LAUNCH_CHECK();
  if (!p.out) return;
  auto cols = [&](auto out) {
    auto* kernel = spectra_cols_kernel<L, decltype(out)>;
    static PerDeviceOnce once;
    once([&] { GISSPA_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smc)); });
    kernel<<<dim3((L / 2 + kRows) / kRows, np), NT, smc, s>>>(p.F, p.list, p.nt * p.na, p.sums, 1.0 / ((double)L * L), p.twL,
                                                             out);
    GISSPA_LAUNCH_CHECK();
  };
  if (p.paired)
    cols(PairOut{static_cast<PairFp32::T*>(p.out)});
  else
    cols(SingleOut{static_cast<float2*>(p.out)});
}

}  // namespace

void tmpl_prescale(int l, TmplSpectra p, float* pre, cudaStream_t s) {
  p.cose = 1.f;
  p.sine = 0.f;
  p.st = nullptr;
  p.list = nullptr;
  p.na = 1;
  p.pre = nullptr;
  p.out = nullptr;  // the rows' sums only
  tmpl_spectra(l, p, s);
  prescale_kernel<<<ceil_div(p.nt, 128), 128, 0, s>>>(p.sums, p.nt, (double)l * l, pre);
  GISSPA_LAUNCH_CHECK();
}

bool tmpl_spectra_supported(int l) { return l == 256 || l == 320 || l == 512 || l == 1024; }

void tmpl_spectra(int l, const TmplSpectra& p, cudaStream_t s) {
  switch (l) {
    case 256: run<256>(p, s); break;
    case 320: run<320>(p, s); break;
    case 512: run<512>(p, s); break;
    case 1024: run<1024>(p, s); break;
    default: throw CudaError{cudaErrorInvalidValue, "window size without fused template spectra"};
  }
}

}  // namespace gisspa
