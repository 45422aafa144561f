// corr_generic.cu — the correlation and its epilogues for window sizes without hand-tuned
// kernels.  Same results as pass A + pass B (correlate.cu) within FP32 rounding: the
// transforms run in shared memory (mixed radix, fft_smooth.cuh) in a fused two-pass form, or on the
// generic FFT engine (Bluestein for other lengths) in an unfused form; the epilogues reproduce
// pass B's per-pixel sums and maxima, chunk picks with the reference's tie order, norm_type=0
// peaks and sums, and maps.  The reference's chunks are 256 consecutive pixels of the window's
// linear index (norm.cu:583-597), so for L that is not a multiple of 256 they straddle rows:
// the chunk scans work on linear indices.
#include "../../include/gisspa.h"
#include "corr_generic.cuh"
#include "fft_smooth.cuh"

namespace gisspa {
namespace {

constexpr int kT = 256;

// Z[p][kx][ky] = I[b0 + e][kx][ky] conj(T[n0 + d][kx][ky]), p = e D + d (half spectra, kx-major)
template <typename SPEC>
__global__ void gen_product_kernel(const float2* __restrict__ I, const typename SPEC::T* __restrict__ T, int b0,
                                   int n0, int D, long long H, float2* __restrict__ Z) {
  const int p = blockIdx.y, e = p / D, d = p - e * D;
  const float2* Ib = I + (size_t)(b0 + e) * H;
  const typename SPEC::T* Tn = T + (size_t)(n0 + d) * H;
  for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < H; k += (long long)gridDim.x * blockDim.x)
    Z[(size_t)p * H + k] = cmulc(Ib[k], SPEC::load(Tn + k));
}

// After the column transforms Z[p][kx][y] holds row y's half spectrum over kx <= L/2; each
// row of a real map is Hermitian: X[p][y][k] = Z[p][k][y] (k <= L/2), conj(Z[p][L - k][y]).
__global__ void gen_hermitian_rows_kernel(const float2* __restrict__ Z, int L, float2* __restrict__ X) {
  const int p = blockIdx.y;
  const long long L2 = (long long)L * L, H = (long long)(L / 2 + 1) * L;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < L2; q += (long long)gridDim.x * blockDim.x) {
    const int y = (int)(q / L), k = (int)(q - (long long)y * L);
    float2 v;
    if (k <= L / 2) {
      v = Z[(size_t)p * H + (size_t)k * L + y];
    } else {
      const float2 w = Z[(size_t)p * H + (size_t)(L - k) * L + y];
      v = make_float2(w.x, -w.y);
    }
    X[(size_t)p * L2 + q] = v;
  }
}

// raw correlation at the shifted window pixel (oy, ox): the zero lag sits at (L/2, L/2)
__device__ __forceinline__ float gen_raw(const float2* X, int p, int L, int oy, int ox) {
  const int y = oy + L / 2 - (oy + L / 2 >= L ? L : 0), x = ox + L / 2 - (ox + L / 2 >= L ? L : 0);
  return X[(size_t)p * L * L + (size_t)y * L + x].x;
}

// EPI_SUM / EPI_TOPK: per window pixel over the launch's D templates, folded into the state
__global__ void gen_sum_kernel(const float2* __restrict__ X, CorrArgs a, int L, int topk) {
  const int e = blockIdx.y;
  const long long L2 = (long long)L * L;
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= L2) return;
  const int oy = (int)(q / L), ox = (int)(q - (long long)oy * L);
  const float inv = 1.0f / (float)L2;
  const int angle = a.angle_state ? a.angle_state->index : a.angle;
  float s1 = 0.f, s2 = 0.f, best = -INFINITY;
  int barg = -1;
  for (int d = 0; d < a.D; ++d) {
    const float c = gen_raw(X, e * a.D + d, L, oy, ox) * inv;
    s1 += c;
    s2 = fmaf(c, c, s2);
    if (c > best) {
      best = c;
      barg = angle * a.nt_total + a.n0 + d;
    }
  }
  const size_t pix = (size_t)(a.b0 + e) * L2 + q;
  atomicAdd(a.S1 + pix, (double)s1);
  atomicAdd(a.S2 + pix, (double)s2);
  if (topk && barg >= 0)
    atomicMax(a.peak + pix, ((unsigned long long)float_key(best) << 32) | (unsigned)(0xFFFFFFFFu - (unsigned)barg));
}

// block-wide max of a u64 key (blockDim.x == kT)
__device__ __forceinline__ unsigned long long block_max_u64(unsigned long long k, unsigned long long* sh) {
  for (int off = 16; off > 0; off >>= 1) {
    const unsigned long long o = __shfl_xor_sync(0xffffffffu, k, off);
    k = o > k ? o : k;
  }
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = k;
  __syncthreads();
  if (threadIdx.x < 32) {
    k = threadIdx.x < kT / 32 ? sh[threadIdx.x] : 0ull;
    for (int off = 16; off > 0; off >>= 1) {
      const unsigned long long o = __shfl_xor_sync(0xffffffffu, k, off);
      k = o > k ? o : k;
    }
  }
  return k;  // valid in thread 0
}

// EPI_CHUNK: one block per (chunk, pair): z-score, chunk max with the reference's tie order
// (the lowest bit-reversed position wins), threshold and centre test -> candidate
__global__ void gen_chunk_kernel(const float2* __restrict__ X, CorrArgs a, int L) {
  __shared__ unsigned long long sh[kT / 32];
  const int p = blockIdx.y, e = p / a.D, d = p - e * a.D, win = a.b0 + e;
  const int chunk = blockIdx.x, t = threadIdx.x;
  const long long L2 = (long long)L * L, q = (long long)chunk * 256 + t;
  const int oy = (int)(q / L), ox = (int)(q - (long long)oy * L);
  const float c = gen_raw(X, p, L, oy, ox) / (float)L2;
  const float2 m = a.musig[(size_t)win * L2 + q];
  const float z = (c - m.x) * m.y;
  const unsigned long long key = ((unsigned long long)float_key(z) << 32) | (unsigned)(255 - brev8(t));
  const unsigned long long best = block_max_u64(key, sh);
  if (threadIdx.x != 0) return;
  const float zb = key_float((uint32_t)(best >> 32));
  if (!(zb >= a.thresh)) return;
  const int tb = brev8(255 - (unsigned)(best & 0xffu));
  const int id = chunk * 256 + tb;
  const int px = id % L, py = id / L;
  const int cx = a.offx[win % a.bx] + px, cy = a.offy[win / a.bx] + py;
  if (!(cx >= a.dmin && cx < a.nx - a.dmin && cy >= a.dmin && cy < a.ny - a.dmin)) return;
  const unsigned slot = atomicAdd(a.cand_count, 1u);
  if (slot >= a.cand_cap) return;
  Cand cd;
  cd.score = zb;
  cd.x = px;
  cd.y = py;
  cd.window = win;
  cd.templ = a.n0 + d;
  cd.angle = a.angle_state ? a.angle_state->index : a.angle;
  cd.chunk = chunk;
  cd.pad = 0;
  a.cand[slot] = cd;
}

// EPI_NONORM: one block per (chunk, pair): peak with the border zeroed (the largest value,
// then the lowest chunk, then the reference's in-chunk order) and the sums of the raw map
__global__ void gen_nonorm_kernel(const float2* __restrict__ X, CorrArgs a, int L) {
  __shared__ unsigned long long sh[kT / 32];
  __shared__ double s1s[kT / 32], s2s[kT / 32];
  const int p = blockIdx.y, e = p / a.D, d = p - e * a.D, win = a.b0 + e;
  const int chunk = blockIdx.x, t = threadIdx.x;
  const long long q = (long long)chunk * 256 + t;
  const int oy = (int)(q / L), ox = (int)(q - (long long)oy * L);
  const float v = gen_raw(X, p, L, oy, ox);
  double s1 = v, s2 = (double)v * v;
  for (int off = 16; off > 0; off >>= 1) {
    s1 += __shfl_xor_sync(0xffffffffu, s1, off);
    s2 += __shfl_xor_sync(0xffffffffu, s2, off);
  }
  if ((t & 31) == 0) {
    s1s[t >> 5] = s1;
    s2s[t >> 5] = s2;
  }
  float val = v;
  if (ox < a.border || ox > L - a.border || oy < a.border || oy > L - a.border) val = 0.f;
  const unsigned long long key = ((unsigned long long)float_key(val) << 32) | (unsigned)(255 - brev8(t));
  const unsigned long long best = block_max_u64(key, sh);  // includes a __syncthreads
  if (t != 0) return;
  double b1 = 0, b2 = 0;
  for (int w = 0; w < kT / 32; ++w) {
    b1 += s1s[w];
    b2 += s2s[w];
  }
  const size_t qq = (size_t)win * a.nt_total + a.n0 + d;
  atomicAdd(a.nn_sum + 2 * qq, b1);
  atomicAdd(a.nn_sum + 2 * qq + 1, b2);
  const float vb = key_float((uint32_t)(best >> 32));
  if (vb > 0.f) {
    const unsigned long long g =
        ((unsigned long long)float_key(vb) << 32) | ((unsigned long long)(0xFFFFFu - chunk) << 8) | (best & 0xffu);
    atomicMax(a.nn_key + qq, g);
  }
}

// EPI_MAP: c maps [pair][L][L], zero lag at (L/2, L/2)
__global__ void gen_map_kernel(const float2* __restrict__ X, CorrArgs a, int L) {
  const int p = blockIdx.y;
  const long long L2 = (long long)L * L;
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= L2) return;
  const int oy = (int)(q / L), ox = (int)(q - (long long)oy * L);
  a.map_out[(size_t)p * L2 + q] = gen_raw(X, p, L, oy, ox) / (float)L2;
}

// ---- fused two-pass form for window sizes whose prime factors are 2, 3, 5 and 7
// Both passes are bound by instruction issue and shared memory.  Stages of 2 to 16 points in
// registers (336 = 7 6 8) instead of 2, 3, 4, 5 and 7 with table reads per point, multiplications
// instead of divisions by run-time sizes, rows per CTA that fill its passes, and an intermediate
// that both passes move in whole sectors took a top-K search of 1500 x 1401 pixels at window 336
// (20 templates, 30 angles) from 59.1 to 35.0 ms; the first and last stages' own loads and stores,
// accumulators in registers, groups of warps with their own barriers and fewer, even launches from
// there to 23.8.

// Rows per CTA of gen_rows_kernel: even, a divisor of L, about 1280 pixels per CTA, and for
// the chunk scans (EPI_CHUNK, EPI_NONORM) RB L a multiple of 256; 0 when no such RB exists.
__host__ __device__ constexpr int gen_rows_rb(int L, int epi) {
  int rb0 = 1;
  if (epi == EPI_CHUNK || epi == EPI_NONORM) {
    int g = 256;
    while (L % g) g >>= 1;
    rb0 = 256 / g;
  }
  const int step = rb0 % 2 ? 2 * rb0 : rb0;
  int rb = step;
  while (rb * L < 1280 && rb + step <= L) rb += step;
  while (rb <= L && L % rb) rb += step;
  return rb <= L ? rb : 0;
}


// Where the column pass leaves Z[p][kx][y]: four rows of a column together (L is a multiple of 16),
// the columns side by side, so that both passes move whole 32-byte sectors: from [kx][y] the row
// pass read 16 bytes of a sector per column, twice.
__device__ __forceinline__ size_t gen_z_index(int p, int kx, int y, int L, int hz) {
  return (((size_t)p * (L >> 2) + (y >> 2)) * hz + kx) * 4 + (y & 3);
}

// Column pass: rows gr = p (L/2+1) + kx of the launch's half-spectrum products
// I[b0 + e][kx][.] conj(T[n0 + d][kx][.]) (p = e D + d), each inverse-transformed along ky in
// shared memory: Z (gen_z_index).  The first stage reads its points from memory, the last writes
// them there (four neighbouring butterflies fill a sector).  rpc <= kGenMaxCols
constexpr int kGenMaxCols = 128;
template <typename SPEC>
__global__ void __launch_bounds__(256, 3) gen_cols_kernel(const float2* __restrict__ I,
                                                          const typename SPEC::T* __restrict__ T, int b0, int n0,
                                                          int D, int L, int nrows, int rpc, SmoothPlan plan,
                                                          const float2* __restrict__ tw, float2* __restrict__ Z) {
  extern __shared__ float2 sm[];
  __shared__ long long iof[kGenMaxCols], tof[kGenMaxCols], zof[kGenMaxCols];
  const int hz = L / 2 + 1;
  const long long H = (long long)hz * L;
  const int row0 = blockIdx.x * rpc;
  const int rows_here = min(rpc, nrows - row0);
  float2* a = sm;
  float2* b = sm + (size_t)rpc * L;
  for (int r = threadIdx.x; r < rows_here; r += 256) {
    const int gr = row0 + r, p = gr / hz, kx = gr - p * hz, e = p / D, d = p - e * D;
    iof[r] = (b0 + e) * H + (long long)kx * L;
    tof[r] = (n0 + d) * H + (long long)kx * L;
    zof[r] = (long long)gen_z_index(p, kx, 0, L, hz);
  }
  __syncthreads();
  smooth_any<1>(CtaTeam{}, plan, 0, rows_here, L, 1, tw,
                [&](int r, int j, int m, auto& x) {
                  constexpr int R = sizeof(x) / sizeof(float2);
                  const float2* i = I + iof[r] + j;
                  const typename SPEC::T* t = T + tof[r] + j;
#pragma unroll
                  for (int q = 0; q < R; ++q) x[q] = cmulc(__ldg(i + q * m), SPEC::load(t + q * m));
                },
                SmoothStore{a, L, 1});
  __syncthreads();
  const int last = plan.ns - 1, Ns = L / plan.r[last];
  const float2* f = smooth_stages<1>(CtaTeam{}, a, b, rows_here, L, L, plan, 1, last, plan.r[0], tw);
  smooth_any<1>(CtaTeam{}, plan, last, rows_here, L, Ns, tw, SmoothLoad{f, L}, [&](int r, int base, const auto& x) {
    constexpr int R = sizeof(x) / sizeof(float2);
    float2* o = Z + zof[r];
#pragma unroll
    for (int p = 0; p < R; ++p) {
      const int y = base + p * Ns;
      o[(y >> 2) * (4 * hz) + (y & 3)] = x[p];
    }
  });
}

// Where the row passes' threads load a template's Hermitian half rows: of a team of `threads`, thread
// t < (threads / hr) hr takes complex row r2 = t mod hr of the CTA's and columns k0 = t / hr, k0 +
// step, ...  (hr <= threads)
struct GenRowLoad {
  int r2, k0, step, ya, yb;
  __device__ __forceinline__ GenRowLoad(int t, int threads, int L, int Y0, int hr) {
    step = threads / hr;
    k0 = t / hr;
    r2 = t - k0 * hr;
    if (k0 >= step) k0 = L;  // no columns
    ya = Y0 + r2 + L / 2;
    yb = ya + hr;
    ya -= ya >= L ? L : 0;
    yb -= yb >= L ? L : 0;
  }
  // X_r + i X_{r + hr} of pair p over all columns into row (row r2 of the template's rows)
  __device__ __forceinline__ void run(const float2* __restrict__ Z, int p, int L, int hz, float2* row) const {
    const float2* A = Z + gen_z_index(p, 0, ya, L, hz);
    const float2* B = Z + gen_z_index(p, 0, yb, L, hz);
#pragma unroll 4
    for (int k = k0; k < hz; k += step) {
      const float2 u = A[4 * k], v = B[4 * k];
      row[k] = make_float2(u.x - v.y, u.y + v.x);
      if (k > 0 && 2 * k < L) row[L - k] = make_float2(u.x + v.y, v.x - u.y);
    }
  }
};

// Row pass of EPI_SUM and EPI_TOPK: one CTA per (block of RB window rows, window of the launch), RB
// / 2 complex rows (as gen_rows_kernel).  The CTA's groups of warps take every `groups`-th template
// of the launch, each with its own buffers and barrier.  The plan ends in a stage of 8 points, whose
// butterflies stay with their threads for all templates: a thread keeps the sums (and maxima) of its
// 16 pixels in registers, and the groups meet in shared memory at the end.
constexpr int kFold = 8, kFoldThreads = 512;
// Warps of a group: a thread for each of the last stage's butterflies
__host__ __device__ constexpr int gen_fold_warps(int L, int RB) { return (RB / 2 * L / kFold + 31) / 32; }
template <int EPI>
__global__ void __launch_bounds__(kFoldThreads)
    gen_fold_kernel(const float2* __restrict__ Z, CorrArgs a, int L, int RB, int ld, int groups, SmoothPlan plan,
                    const float2* __restrict__ tw) {
  extern __shared__ float2 sm[];
  constexpr bool TOPK = EPI == EPI_TOPK;
  constexpr int NV = TOPK ? 4 : 2;  // values per pixel
  const int hz = L / 2 + 1, hr = RB / 2, m = L / kFold, per = hr * m, threads = 32 * gen_fold_warps(L, RB);
  const int e = blockIdx.y, Y0 = blockIdx.x * RB, g = threadIdx.x / threads;
  const long long L2 = (long long)L * L;
  const float inv = 1.0f / (float)L2;
  const WarpsTeam team{g, threads};
  const int t = team.id(), r = t / m, j = t - r * m;  // this thread's butterfly
  const bool own = t < per;
  float2* buf0 = sm + (size_t)g * 2 * hr * ld;  // hr complex rows, row stride ld
  float2* buf1 = buf0 + (size_t)hr * ld;
  const GenRowLoad rows(t, threads, L, Y0, hr);
  float s1[2][kFold], s2[2][kFold], best[TOPK ? 2 : 1][kFold];
  unsigned arg[TOPK ? kFold : 1];  // template of the launch + 1 of the two pixels' maxima, 16 bits each
#pragma unroll
  for (int i = 0; i < kFold; ++i) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      s1[h][i] = s2[h][i] = 0.f;
      if constexpr (TOPK) best[h][i] = -INFINITY;
    }
    if constexpr (TOPK) arg[i] = 0u;
  }
  for (int d = g; d < a.D; d += groups) {
    rows.run(Z, e * a.D + d, L, hz, buf0 + rows.r2 * ld);
    team.sync();
    const float2* f = smooth_stages<1>(team, buf0, buf1, hr, L, ld, plan, 0, plan.ns - 1, 1, tw);
    if (own) {
      float2 x[kFold];
      SmoothLoad{f, ld}(r, j, m, x);
      twiddle_powers<kFold, 1>(x, tw, j);
      Dft<kFold, 1>::run(x);
#pragma unroll
      for (int i = 0; i < kFold; ++i) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float c = (h ? x[i].y : x[i].x) * inv;
          s1[h][i] += c;
          s2[h][i] = fmaf(c, c, s2[h][i]);
          if constexpr (TOPK) {
            if (c > best[h][i]) {
              best[h][i] = c;
              arg[i] = h ? (arg[i] & 0xFFFFu) | (unsigned)(d + 1) << 16 : (arg[i] & 0xFFFF0000u) | (unsigned)(d + 1);
            }
          }
        }
      }
    }
    team.sync();  // the buffers are rewritten next
  }
  // every pixel's shares, in the groups' order; group g takes every groups-th of the 8 columns
  float* sh = reinterpret_cast<float*>(sm);  // [kFold][NV][groups][per]
  const int angle = a.angle_state ? a.angle_state->index : a.angle, all = groups * per;
  const size_t wpix = (size_t)(a.b0 + e) * L2;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    __syncthreads();
    if (own) {
      float* o = sh + g * per + t;
#pragma unroll
      for (int i = 0; i < kFold; ++i) {
        o[(NV * i) * all] = s1[h][i];
        o[(NV * i + 1) * all] = s2[h][i];
        if constexpr (TOPK) {
          o[(NV * i + 2) * all] = best[h][i];
          o[(NV * i + 3) * all] = __uint_as_float(h ? arg[i] >> 16 : arg[i] & 0xFFFFu);
        }
      }
    }
    __syncthreads();
    if (!own) continue;
    for (int i = g; i < kFold; i += groups) {
      const float* o = sh + (size_t)NV * i * all + t;
      float v1 = 0.f, v2 = 0.f, b = -INFINITY;
      unsigned w = 0;
      for (int q = 0; q < groups; ++q, o += per) {
        v1 += o[0];
        v2 += o[all];
        if constexpr (TOPK) {
          const float c = o[2 * all];
          const unsigned n = __float_as_uint(o[3 * all]);
          if (n && (!w || c > b || (c == b && n < w))) {
            b = c;
            w = n;
          }
        }
      }
      const int xc = j + i * m, ox = xc + L / 2 - (xc + L / 2 >= L ? L : 0);
      const size_t pix = wpix + (size_t)(Y0 + r + h * hr) * L + ox;
      atomicAdd(a.S1 + pix, (double)v1);
      atomicAdd(a.S2 + pix, (double)v2);
      if constexpr (TOPK) {
        if (w) {
          const unsigned id = (unsigned)(angle * a.nt_total + a.n0) + w - 1;
          atomicMax(a.peak + pix, ((unsigned long long)float_key(b) << 32) | (unsigned)(0xFFFFFFFFu - id));
        }
      }
    }
  }
}

// Row pass of the other epilogues: one CTA per (block of RB window rows, window of the launch), over the launch's D
// templates.  Window (state) row Y0 + r is transform row (Y0 + r + L/2) mod L, and state
// column ox is transform column (ox + L/2) mod L (zero lag at (L/2, L/2)).  Rows r and
// r + RB/2 are real, so their Hermitian spectra X_r[k] (= Z[p][k][y] for k <= L/2,
// conj Z[p][L-k][y] above) go through one complex transform as X_r + i X_{r+RB/2}: the real
// and imaginary parts of the result are the two rows.  Thread t holds the CTA's pixels
// q = 256 i + t (state linear index Y0 L + q, q < RB L); for the chunk scans (EPI_CHUNK,
// EPI_NONORM) RB L is a multiple of 256, so these are whole chunks of the reference's
// 256-pixel scan and q = 256 i + t is pixel t of the CTA's chunk i.  The rows of up to TB
// templates go through one transform pass (fewer block barriers, more butterflies per thread);
// the epilogue then takes those templates in order.
template <int EPI>
__global__ void __launch_bounds__(256, 3) gen_rows_kernel(const float2* __restrict__ Z, CorrArgs a, int L, unsigned div_l,
                                                       int RB, int ld, int TB, SmoothPlan plan,
                                                       const float2* __restrict__ tw) {
  extern __shared__ float2 sm[];
  const int hz = L / 2 + 1;
  const int hr = RB / 2, npix = RB * L, nch = npix / 256, t = threadIdx.x, lane = t & 31, wid = t >> 5;
  float2* buf0 = sm;  // TB templates x hr complex rows, row stride ld
  float2* buf1 = sm + (size_t)TB * hr * ld;
  unsigned long long* red = reinterpret_cast<unsigned long long*>(sm + (size_t)2 * TB * hr * ld);  // [nch][8]
  double* dred = reinterpret_cast<double*>(red + (size_t)nch * 8);                            // [2][8]
  char* st = reinterpret_cast<char*>(dred + 16);
  __shared__ unsigned hits;  // EPI_CHUNK: the group's templates with a pixel at the threshold
  const int e = blockIdx.y, win = a.b0 + e, Y0 = blockIdx.x * RB;
  const long long L2 = (long long)L * L;
  const size_t wpix = (size_t)win * L2 + (size_t)Y0 * L;
  const float inv = 1.0f / (float)L2;
  const int angle = a.angle_state ? a.angle_state->index : a.angle;
  const GenRowLoad rows(t, 256, L, Y0, hr);
  float2* ms = reinterpret_cast<float2*>(st);  // CHUNK: (mu, 1/sigma) of the CTA's pixels
  if constexpr (EPI == EPI_CHUNK)
    for (int q = t; q < npix; q += 256) ms[q] = a.musig[wpix + q];
  // pixel q's place in a template's transformed rows (complex row, column) and which part
  auto place = [&](int q, bool& upper) {
    const int r = fast_div(q, div_l), ox = q - r * L, x = ox + L / 2 - (ox + L / 2 >= L ? L : 0);
    upper = r >= hr;
    return (upper ? r - hr : r) * ld + x;
  };

  for (int d0 = 0; d0 < a.D; d0 += TB) {
    const int nd = min(TB, a.D - d0);
    if (EPI == EPI_CHUNK && t == 0) hits = 0u;
    for (int q = 0; q < nd; ++q) rows.run(Z, e * a.D + d0 + q, L, hz, buf0 + (q * hr + rows.r2) * ld);
    __syncthreads();
    const float2* fg = smooth_stages<1>(CtaTeam{}, buf0, buf1, nd * hr, L, ld, plan, 0, plan.ns, 1, tw);

    if constexpr (EPI == EPI_CHUNK) {
      unsigned hit = 0;
      for (int q = t; q < npix; q += 256) {
        bool up;
        const float2* f = fg + place(q, up);
        const float2 m = ms[q];
        for (int g = 0; g < nd; ++g) {
          const float2 w = f[g * hr * ld];
          if (((up ? w.y : w.x) * inv - m.x) * m.y >= a.thresh) hit |= 1u << g;
        }
      }
      hit = __reduce_or_sync(0xffffffffu, hit);
      if (lane == 0 && hit) atomicOr(&hits, hit);
      __syncthreads();
    }

    for (int g = 0; g < nd; ++g) {
      const int d = d0 + g, p = e * a.D + d;
      const float2* f = fg + g * hr * ld;

      if constexpr (EPI == EPI_CHUNK) {
        if (hits >> g & 1) {  // CTA-uniform
          for (int i = 0; i < nch; ++i) {
            const int q = 256 * i + t;
            bool up;
            const float2 w = f[place(q, up)];
            const float z = ((up ? w.y : w.x) * inv - ms[q].x) * ms[q].y;
            unsigned long long key = ((unsigned long long)float_key(z) << 32) | (unsigned)(255 - brev8(t));
            for (int off = 16; off > 0; off >>= 1) {
              const unsigned long long o = __shfl_xor_sync(0xffffffffu, key, off);
              key = o > key ? o : key;
            }
            if (lane == 0) red[i * 8 + wid] = key;
          }
          __syncthreads();
          for (int i = t; i < nch; i += 256) {
            unsigned long long best = 0;
            for (int w = 0; w < 8; ++w) best = red[i * 8 + w] > best ? red[i * 8 + w] : best;
            const float zb = key_float((uint32_t)(best >> 32));
            if (!(zb >= a.thresh)) continue;
            const int id = Y0 * L + i * 256 + brev8(255 - (unsigned)(best & 0xffu));
            const int px = id % L, py = id / L;
            const int cx = a.offx[win % a.bx] + px, cy = a.offy[win / a.bx] + py;
            if (!(cx >= a.dmin && cx < a.nx - a.dmin && cy >= a.dmin && cy < a.ny - a.dmin)) continue;
            const unsigned slot = atomicAdd(a.cand_count, 1u);
            if (slot >= a.cand_cap) continue;
            Cand cd;
            cd.score = zb;
            cd.x = px;
            cd.y = py;
            cd.window = win;
            cd.templ = a.n0 + d;
            cd.angle = angle;
            cd.chunk = id >> 8;
            cd.pad = 0;
            a.cand[slot] = cd;
          }
          __syncthreads();  // reduction slots reused next
        }
      } else if constexpr (EPI == EPI_NONORM) {
        double t1 = 0.0, t2 = 0.0;
        for (int i = 0; i < nch; ++i) {
          const int q = 256 * i + t;
          const int r = fast_div(q, div_l), ox = q - r * L, oy = Y0 + r;
          bool up;
          const float2 w = f[place(q, up)];
          const float v = up ? w.y : w.x;
          t1 += v;
          t2 += (double)v * v;
          float val = v;
          if (ox < a.border || ox > L - a.border || oy < a.border || oy > L - a.border) val = 0.f;
          unsigned long long key = ((unsigned long long)float_key(val) << 32) | (unsigned)(255 - brev8(t));
          for (int off = 16; off > 0; off >>= 1) {
            const unsigned long long o = __shfl_xor_sync(0xffffffffu, key, off);
            key = o > key ? o : key;
          }
          if (lane == 0) red[i * 8 + wid] = key;
        }
        for (int off = 16; off > 0; off >>= 1) {
          t1 += __shfl_xor_sync(0xffffffffu, t1, off);
          t2 += __shfl_xor_sync(0xffffffffu, t2, off);
        }
        if (lane == 0) {
          dred[wid] = t1;
          dred[8 + wid] = t2;
        }
        __syncthreads();
        const size_t qq = (size_t)win * a.nt_total + a.n0 + d;
        if (t == 0) {
          double b1 = 0, b2 = 0;
          for (int w = 0; w < 8; ++w) {
            b1 += dred[w];
            b2 += dred[8 + w];
          }
          atomicAdd(a.nn_sum + 2 * qq, b1);
          atomicAdd(a.nn_sum + 2 * qq + 1, b2);
        }
        for (int i = t; i < nch; i += 256) {
          unsigned long long best = 0;
          for (int w = 0; w < 8; ++w) best = red[i * 8 + w] > best ? red[i * 8 + w] : best;
          const float vb = key_float((uint32_t)(best >> 32));
          if (vb > 0.f) {
            const int chunk = Y0 * L / 256 + i;
            atomicMax(a.nn_key + qq, ((unsigned long long)float_key(vb) << 32) |
                                         ((unsigned long long)(0xFFFFFu - chunk) << 8) | (best & 0xffu));
          }
        }
        __syncthreads();  // reduction slots reused next
      } else if constexpr (EPI == EPI_MAP) {
        float* out = a.map_out + (size_t)p * L2 + (size_t)Y0 * L;
        for (int q = t; q < npix; q += 256) {
          bool up;
          const float2 w = f[place(q, up)];
          out[q] = (up ? w.y : w.x) * inv;
        }
      }
    }
    __syncthreads();  // the transform buffers are rewritten next
  }
}

// Row stride in shared memory: the loads write hr rows of a column at a time, 16 / hr columns per
// half warp, to distinct banks.
int gen_rows_ld(int L, int RB) { return L + std::max(1, 16 / (RB / 2)); }

size_t gen_rows_smem(int L, int RB, int epi, int tb) {
  const size_t ld = gen_rows_ld(L, RB), npix = (size_t)RB * L, nch = npix / 256;
  size_t b = sizeof(float2) * tb * RB * ld + sizeof(unsigned long long) * nch * 8 + sizeof(double) * 16;
  if (epi == EPI_SUM || epi == EPI_TOPK)  // the groups' buffers, then their pixels' values
    b = std::max<size_t>(sizeof(float2) * tb * RB * ld, sizeof(float) * (epi == EPI_TOPK ? 4 : 2) * tb * RB / 2 * L);
  if (epi == EPI_CHUNK) b += sizeof(float2) * npix;
  return b;
}

constexpr size_t kGenSmemMax = 200 * 1024;
constexpr int kGenColPoints = 4352;  // per CTA of the column pass (68 KB: three CTAs per SM)

// Templates per transform pass of gen_rows_kernel: as fill its CTA's passes best (smooth_rows), three
// CTAs per SM where one template's rows leave room for that.
constexpr int kGenTB = 16;
int gen_rows_tb(int L, int RB, int epi, const SmoothPlan& plan) {
  const size_t one = gen_rows_smem(L, RB, epi, 1), two = gen_rows_smem(L, RB, epi, 2);
  const size_t room = kGenSmemMax / 3 > one ? kGenSmemMax / 3 - one : 0;
  const int tb = std::min<long long>(kGenTB, 1 + room / (two - one));
  if (epi == EPI_SUM || epi == EPI_TOPK) return std::max(1, std::min(std::min(tb, 15), kFoldThreads / 32 / gen_fold_warps(L, RB)));  // (15 barriers)
  return smooth_rows(plan, L, 256, tb * (RB / 2) * L, RB / 2) / (RB / 2);
}

// A row kernel with its dynamic shared-memory limit raised to kGenSmemMax, once per device, at the
// first launch that needs more than the default 48 KB (the first angle of a sweep runs before any
// graph capture).
template <auto K>
auto gen_kernel(size_t smem) {
  if (smem > 48 * 1024) {
    static PerDeviceOnce once;
    once([] { GISSPA_CUDA(cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGenSmemMax)); });
  }
  return K;
}

}  // namespace

bool generic_fused(int L, int epi) {
  if (L > kSmoothMax || smooth_plan(L).ns == 0) return false;
  const int rb = gen_rows_rb(L, epi);
  if ((epi == EPI_SUM || epi == EPI_TOPK) && gen_fold_warps(L, rb) * 32 > kFoldThreads) return false;
  return rb > 0 && gen_rows_smem(L, rb, epi, 1) <= kGenSmemMax && (size_t)2 * sizeof(float2) * L <= kGenSmemMax;
}

bool correlate_fast(int L) { return L == 256 || L == 320 || L == 512 || L == 1024; }

size_t generic_z_elems(int L, int P) { return (size_t)P * (L / 2 + 1) * L; }
size_t generic_x_elems(int L, int P, int epi) { return generic_fused(L, epi) ? 0 : (size_t)P * L * L; }

void correlate_generic(const CorrLaunch& cl, const float2* I, const void* T, const CorrArgs& a, FftEngine& fft,
                       float2* z, float2* x, cudaStream_t s, cudaEvent_t* ev) {
  const int L = cl.L, P = cl.E * cl.D;
  const long long H = (long long)(L / 2 + 1) * L, L2 = (long long)L * L;
  if (ev) GISSPA_CUDA(cudaEventRecord(ev[0], s));
  if (generic_fused(L, cl.epi)) {
    const SmoothPlan plan = smooth_plan(L);
    const float2* tw = fft.twiddles(L);
    const unsigned div_l = fast_div_mul(L);
    const int nrows = P * (L / 2 + 1);
    const int rpc = std::min(kGenMaxCols, smooth_rows(plan, L, 256, kGenColPoints));
    const size_t smc = 2 * sizeof(float2) * (size_t)rpc * L;
    const unsigned gc = (unsigned)ceil_div(nrows, rpc);
    auto cols = [&](auto kernel, const auto* t) {
      kernel<<<gc, 256, smc, s>>>(I, t, a.b0, a.n0, cl.D, L, nrows, rpc, plan, tw, z);
    };
    switch (cl.spec) {
      case GISSPA_SPEC_FP32: cols(gen_kernel<gen_cols_kernel<SpecFp32>>(smc), static_cast<const float2*>(T)); break;
      case GISSPA_SPEC_FP16: cols(gen_kernel<gen_cols_kernel<SpecFp16>>(smc), static_cast<const __half2*>(T)); break;
      case GISSPA_SPEC_BF16:
        cols(gen_kernel<gen_cols_kernel<SpecBf16>>(smc), static_cast<const __nv_bfloat162*>(T));
        break;
      default: throw CudaError{cudaErrorInvalidValue, "unknown spectrum precision"};
    }
    GISSPA_LAUNCH_CHECK();
    if (ev) GISSPA_CUDA(cudaEventRecord(ev[1], s));
    const int rb = gen_rows_rb(L, cl.epi), ld = gen_rows_ld(L, rb);
    const int most = gen_rows_tb(L, rb, cl.epi, plan), tb = ceil_div(cl.D, ceil_div(cl.D, most));
    const size_t smr = gen_rows_smem(L, rb, cl.epi, tb);
    const dim3 gr((unsigned)(L / rb), (unsigned)cl.E);
    auto rows = [&](auto kernel) { kernel<<<gr, 256, smr, s>>>(z, a, L, div_l, rb, ld, tb, plan, tw); };
    auto fold = [&](auto kernel) {
      kernel<<<gr, 32 * tb * gen_fold_warps(L, rb), smr, s>>>(z, a, L, rb, ld, tb, smooth_plan(L, kFold), tw);
    };
    switch (cl.epi) {
      case EPI_SUM: fold(gen_kernel<gen_fold_kernel<EPI_SUM>>(smr)); break;
      case EPI_TOPK: fold(gen_kernel<gen_fold_kernel<EPI_TOPK>>(smr)); break;
      case EPI_CHUNK: rows(gen_kernel<gen_rows_kernel<EPI_CHUNK>>(smr)); break;
      case EPI_NONORM: rows(gen_kernel<gen_rows_kernel<EPI_NONORM>>(smr)); break;
      case EPI_MAP: rows(gen_kernel<gen_rows_kernel<EPI_MAP>>(smr)); break;
      default: throw CudaError{cudaErrorInvalidValue, "unknown epilogue"};
    }
    GISSPA_LAUNCH_CHECK();
    if (ev) GISSPA_CUDA(cudaEventRecord(ev[2], s));
    return;
  }
  const dim3 gp((unsigned)std::min(ceil_div(H, kT), 4096), (unsigned)P);
  switch (cl.spec) {
    case GISSPA_SPEC_FP32:
      gen_product_kernel<SpecFp32><<<gp, kT, 0, s>>>(I, static_cast<const float2*>(T), a.b0, a.n0, cl.D, H, z);
      break;
    case GISSPA_SPEC_FP16:
      gen_product_kernel<SpecFp16><<<gp, kT, 0, s>>>(I, static_cast<const __half2*>(T), a.b0, a.n0, cl.D, H, z);
      break;
    case GISSPA_SPEC_BF16:
      gen_product_kernel<SpecBf16><<<gp, kT, 0, s>>>(I, static_cast<const __nv_bfloat162*>(T), a.b0, a.n0, cl.D, H,
                                                     z);
      break;
    default: throw CudaError{cudaErrorInvalidValue, "unknown spectrum precision"};
  }
  GISSPA_LAUNCH_CHECK();
  fft.rows(z, (long long)P * (L / 2 + 1), L, +1, 1.f, s);  // columns over ky
  gen_hermitian_rows_kernel<<<dim3((unsigned)std::min(ceil_div(L2, kT), 4096), (unsigned)P), kT, 0, s>>>(z, L, x);
  GISSPA_LAUNCH_CHECK();
  if (ev) GISSPA_CUDA(cudaEventRecord(ev[1], s));
  fft.rows(x, (long long)P * L, L, +1, 1.f, s);  // rows over kx: real maps
  const unsigned chunks = (unsigned)(L2 / 256);  // L % 16 == 0 makes L^2 a multiple of 256
  switch (cl.epi) {
    case EPI_SUM:
    case EPI_TOPK:
      gen_sum_kernel<<<dim3((unsigned)ceil_div(L2, kT), (unsigned)cl.E), kT, 0, s>>>(x, a, L, cl.epi == EPI_TOPK);
      break;
    case EPI_CHUNK: gen_chunk_kernel<<<dim3(chunks, (unsigned)P), kT, 0, s>>>(x, a, L); break;
    case EPI_NONORM: gen_nonorm_kernel<<<dim3(chunks, (unsigned)P), kT, 0, s>>>(x, a, L); break;
    case EPI_MAP: gen_map_kernel<<<dim3((unsigned)ceil_div(L2, kT), (unsigned)P), kT, 0, s>>>(x, a, L); break;
    default: throw CudaError{cudaErrorInvalidValue, "unknown epilogue"};
  }
  GISSPA_LAUNCH_CHECK();
  if (ev) GISSPA_CUDA(cudaEventRecord(ev[2], s));
}

}  // namespace gisspa
