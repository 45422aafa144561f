// serial_sum.cu — the reference's LoadImage statistics (norm.cu:157-167): two running FP32 sums
// over the micrograph in row order, every addition rounded, evaluated in parallel and bit for bit.
//
// While a running sum s stays inside one binade, s = k u with a fixed unit u = 2^(e - 23) and an
// integer 2^23 <= |k| < 2^24, adding t rounds k + t / u to the nearest integer, ties to even.
// Except for exact ties the rounded increment does not depend on k, and a tie only on k's
// parity; so a run of terms is a map parity -> (increment, parity), and such maps compose:
// (D0, d) = increment from even k, and how much more from odd k (after the first tie both cases
// leave k even, so |d| <= 1), with bounds (mn, mx) on the increments of all prefixes.  A run whose
// prefixes keep k inside the binade (by one unit at either end) has the result k + D0 (+ d); the
// additions that leave it are done one by one.
//
//   1. block_sum_kernel: FP64 sums of 4096-term blocks (only to choose binades)
//   2. binade_kernel: the largest running sum's exponent
//   3. chunk_map_kernel, block_map_kernel: the maps of every 256-term chunk and every block in the
//      kBinades binades below it
//   4. walk_kernel: one CTA per sum composes 256 blocks at a time and takes those that fit; the
//      first that does not goes chunk by chunk, and the chunks that leave the binade term by term
// One thread adding the 16.8 M terms of a 4096^2 micrograph took 65 ms (a dependent FP32 addition
// per term).  This takes 0.6 ms where the mean is well away from zero and 10.6 ms for a zero-mean
// micrograph, whose running sum changes its binade often: the chunks in which it does (a serial
// chain of 256 additions each) bound it.  2048^2: 0.23 and 3.0 ms instead of 16.
// (Blocks of one size only, 1024 terms: 13.5 and 3.8 ms.  Maps of 16 terms for the failing part: 36 ms,
// one warp's checks cost more than the additions that they save.)
#include <cmath>

#include "prep.cuh"

namespace gisspa {
namespace {

constexpr int kChunk = 256, kPerLane = 32;         // terms per chunk, per lane of step 3
constexpr int kLanes = kChunk / kPerLane;           // lanes per chunk
constexpr int kBlock = 4096, kCB = kBlock / kChunk;  // terms per block, chunks per block
constexpr int kBinades = 16;
constexpr int kOut = 1 << 29;  // a bound no prefix may reach
constexpr int kWarps = 8;      // warps per CTA of step 3

// The terms of the two sums (norm.cu:160-163) with the reference's roundings.
__device__ __forceinline__ float term1(float v, float fnx, float fny) { return __fdiv_rn(__fdiv_rn(v, fnx), fny); }
__device__ __forceinline__ float term2(float v, float fnx, float fny) {
  return __fdiv_rn(__fdiv_rn(__fmul_rn(v, v), fnx), fny);
}

struct RunMap {
  int D0, d, mn, mx;
};
__device__ __forceinline__ RunMap identity_map() { return RunMap{0, 0, kOut, -kOut}; }
// a, then b.  (Sums may wrap only after a prefix has left +-2^24, which mn or mx then keeps.)
__device__ __forceinline__ RunMap compose(const RunMap& a, const RunMap& b) {
  RunMap r;
  const int a1 = a.D0 + a.d;
  r.D0 = a.D0 + b.D0 + ((a.D0 & 1) ? b.d : 0);
  const int r1 = a1 + b.D0 + ((a1 & 1) ? 0 : b.d);  // from odd k: odd + a1
  r.d = r1 - r.D0;
  r.mn = min(a.mn, min(a.D0, a1) + b.mn);
  r.mx = max(a.mx, max(a.D0, a1) + b.mx);
  return r;
}
// Appends the term t: inv = 1 / u, a power of two.
__device__ __forceinline__ void append(RunMap& m, float t, float inv) {
  const float y = t * inv;
  if (!(fabsf(y) < 4194304.f)) {  // half the binade's width in one step, or no number: not taken
    m.mx = kOut;
    return;
  }
  // nearest integer, ties to even, by two additions (and no conversion instruction)
  constexpr float kMagic = 12582912.f;  // 1.5 2^23
  const float z = __fadd_rn(y, kMagic), f = y - __fsub_rn(z, kMagic);
  int q = __float_as_int(z) - 0x4B400000;
  const bool tie = fabsf(f) == 0.5f;
  if (tie) {
    // q is the even neighbour, right for even k; odd k takes the other one
    const int other = q + (f > 0.f ? 1 : -1);
    const bool odd0 = m.D0 & 1, odd1 = !((m.D0 + m.d) & 1);
    const int i0 = odd0 ? other : q, i1 = odd1 ? other : q;
    m.d += i1 - i0;
    q = i0;
  }
  m.D0 += q;
  m.mn = min(m.mn, m.D0 + min(m.d, 0));
  m.mx = max(m.mx, m.D0 + max(m.d, 0));
}
__device__ __forceinline__ RunMap shfl_up_map(const RunMap& m, int o) {
  return RunMap{__shfl_up_sync(0xffffffffu, m.D0, o), __shfl_up_sync(0xffffffffu, m.d, o),
                __shfl_up_sync(0xffffffffu, m.mn, o), __shfl_up_sync(0xffffffffu, m.mx, o)};
}
// Inclusive composition over each group of W lanes, in lane order.
template <int W = 32>
__device__ __forceinline__ RunMap scan_map(RunMap m, int lane) {
#pragma unroll
  for (int o = 1; o < W; o <<= 1) {
    const RunMap p = shfl_up_map(m, o);
    if ((lane & (W - 1)) >= o) m = compose(p, m);
  }
  return m;
}

__global__ void __launch_bounds__(256) block_sum_kernel(const float* __restrict__ img, long long n, float fnx,
                                                        float fny, double* __restrict__ sums, int nblocks) {
  const int c = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (c >= nblocks) return;
  double a = 0, b = 0;
  const long long base = (long long)c * kBlock;
#pragma unroll 8
  for (int i = lane; i < kBlock; i += 32)
    if (base + i < n) {
      const float v = img[base + i];
      a += v;
      b += (double)v * v;
    }
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  if (lane == 0) {
    const double s = 1.0 / ((double)fnx * fny);
    sums[c] = a * s;
    sums[nblocks + c] = b * s;
  }
}

// etop[j]: the exponent of the largest running sum j, plus one for the drift of the rounded sum.
__global__ void __launch_bounds__(1024) binade_kernel(const double* __restrict__ sums, int nblocks,
                                                      int* __restrict__ etop) {
  __shared__ double sh[1024];
  __shared__ double big[32];
  for (int j = 0; j < 2; ++j) {
    // each thread a contiguous run: its total, then the prefixes inside it
    const int per = (nblocks + 1023) / 1024, c0 = threadIdx.x * per, c1 = min(nblocks, c0 + per);
    double t = 0;
    for (int c = c0; c < c1; ++c) t += sums[(size_t)j * nblocks + c];
    sh[threadIdx.x] = t;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
      const double x = threadIdx.x >= o ? sh[threadIdx.x - o] : 0.0;
      __syncthreads();
      sh[threadIdx.x] += x;
      __syncthreads();
    }
    double p = sh[threadIdx.x] - t, m = 0;
    for (int c = c0; c < c1; ++c) {
      p += sums[(size_t)j * nblocks + c];
      m = fmax(m, fabs(p));
    }
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) big[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < 32; ++w) m = fmax(m, big[w]);
      etop[j] = (m > 0 && isfinite(m)) ? max(-80, min(100, ilogb(m) + 1)) : 0;
    }
    __syncthreads();
  }
}

// 1 / u of the binade with exponent e (-100 <= e <= 100: a normal float).
__device__ __forceinline__ float unit_inv(int e) { return __uint_as_float((unsigned)(127 + 23 - e) << 23); }

__global__ void __launch_bounds__(kWarps * 32) chunk_map_kernel(const float* __restrict__ img, long long n, float fnx,
                                                                float fny, const int* __restrict__ etop,
                                                                int4* __restrict__ tab, int nchunks) {
  constexpr int kTerms = 32 * kPerLane;       // a warp's
  __shared__ float t[kWarps][kTerms + 32];  // one pad per lane's run: the runs' stride is odd
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, j = blockIdx.y;
  const long long base = ((long long)blockIdx.x * kWarps + w) * kTerms;
  if (base / kChunk >= nchunks) return;
#pragma unroll 4
  for (int i = lane; i < kTerms; i += 32) {
    float v = 0.f;
    if (base + i < n) v = j ? term2(img[base + i], fnx, fny) : term1(img[base + i], fnx, fny);
    t[w][i + i / kPerLane] = v;  // past the end: zeros, which change nothing
  }
  __syncwarp();
  const int e0 = etop[j], c = (int)(base / kChunk) + lane / kLanes;
  const float* mine = &t[w][lane * (kPerLane + 1)];
#pragma unroll 1
  for (int b0 = 0; b0 < kBinades; b0 += 4) {
    RunMap m[4];
    float inv[4];
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      m[b] = identity_map();
      inv[b] = unit_inv(e0 - b0 - b);
    }
    for (int i = 0; i < kPerLane; ++i) {
      const float v = mine[i];
#pragma unroll
      for (int b = 0; b < 4; ++b) append(m[b], v, inv[b]);
    }
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const RunMap s = scan_map<kLanes>(m[b], lane);
      if ((lane & (kLanes - 1)) == kLanes - 1 && c < nchunks)
        tab[((size_t)j * kBinades + b0 + b) * nchunks + c] = make_int4(s.D0, s.d, s.mn, s.mx);
    }
  }
}

__device__ __forceinline__ RunMap to_map(int4 v) { return RunMap{v.x, v.y, v.z, v.w}; }

// The maps of whole blocks (nchunks: whole blocks of chunks).
__global__ void block_map_kernel(const int4* __restrict__ chunks, int nblocks, int4* __restrict__ blocks) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 2 * kBinades * nblocks) return;
  RunMap m = identity_map();
#pragma unroll
  for (int q = 0; q < kCB; ++q) m = compose(m, to_map(chunks[(size_t)i * kCB + q]));
  blocks[i] = make_int4(m.D0, m.d, m.mn, m.mx);
}

// k, e of a normal s (false for zero, subnormals, infinities and NaN, and outside |e| <= 100).
__device__ __forceinline__ bool split(float s, int& k, int& e) {
  const unsigned u = __float_as_uint(s);
  e = (int)((u >> 23) & 255u) - 127;
  k = (int)((u & 0x7FFFFFu) | 0x800000u);
  if (u >> 31) k = -k;
  return e >= -100 && e <= 100;
}
__device__ __forceinline__ float join(int k, int e) {
  return (float)k * __uint_as_float((unsigned)(127 + e - 23) << 23);
}
// Whether the runs' prefixes keep k inside its binade, a unit away from its ends.
__device__ __forceinline__ bool fits(int k, const RunMap& m) {
  constexpr int lo = (1 << 23) + 1, hi = (1 << 24) - 1;
  return k > 0 ? (k + m.mn >= lo && k + m.mx <= hi) : (k + m.mx <= -lo && k + m.mn >= -hi);
}

constexpr int kWalk = 256;  // threads of step 4
struct WalkShared {
  float t[kBlock];
  int4 map[kCB][3];  // a block's chunks, in the sum's binade and the two beside it
  RunMap tot[kWalk / 32];
  int bad[kWalk / 32];
  float s;
};
// Of the CTA's maps in thread order: how many the sum s = k 2^(e - 23) takes whole; s after them.
__device__ __forceinline__ int take(WalkShared& sh, float& s, int k, int e, const RunMap& own) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  RunMap m = scan_map(own, lane);
  if (lane == 31) sh.tot[w] = m;
  __syncthreads();
  if (w) {
    RunMap p = sh.tot[0];
    for (int i = 1; i < w; ++i) p = compose(p, sh.tot[i]);
    m = compose(p, m);
  }
  // an inclusive prefix is within bounds exactly when every run up to it fits
  const unsigned bad = __ballot_sync(0xffffffffu, !fits(k, m));
  if (lane == 0) sh.bad[w] = bad ? w * 32 + __ffs(bad) - 1 : kWalk;
  __syncthreads();
  int good = kWalk;
#pragma unroll
  for (int i = 0; i < kWalk / 32; ++i) good = min(good, sh.bad[i]);
  if ((int)threadIdx.x == good - 1) sh.s = join(k + m.D0 + ((k & 1) ? m.d : 0), e);
  __syncthreads();
  if (good) s = sh.s;
  return good;
}

__global__ void __launch_bounds__(kWalk) walk_kernel(const float* __restrict__ img, long long n, float fnx, float fny,
                                                     const int* __restrict__ etop, const int4* __restrict__ chunks,
                                                     const int4* __restrict__ blocks, int nblocks,
                                                     float* __restrict__ out) {
  __shared__ __align__(16) WalkShared sh;
  const int tid = threadIdx.x, j = blockIdx.x, e0 = etop[j];
  const int4* tc = chunks + (size_t)j * kBinades * nblocks * kCB;
  const int4* tb = blocks + (size_t)j * kBinades * nblocks;
  float s = 0.f;  // (the same in every thread)
  int c = 0;
  while (c < nblocks) {
    int k, e;
    const bool normal = split(s, k, e);
    const int b = e0 - e;
    if (normal && b >= 0 && b < kBinades) {
      RunMap m = identity_map();
      if (c + tid < nblocks)
        m = to_map(tb[(size_t)b * nblocks + c + tid]);
      else
        m.mx = kOut;  // past the last block
      const int done = take(sh, s, k, e, m);
      c += done;
      if (done == kWalk || c >= nblocks) continue;
    }
    // block c leaves the binade: its terms and its chunks' maps
    const bool ours = split(s, k, e);
    const long long base = (long long)c * kBlock;
    {
      constexpr int kEach = kBlock / kWalk;
      float v[kEach];
#pragma unroll
      for (int q = 0; q < kEach; ++q) {
        const long long at = base + tid + q * kWalk;
        v[q] = at < n ? img[at] : 0.f;
      }
      if (tid < 3 * kCB) {
        const int q = tid / 3, b3 = e0 - (e - 1 + tid % 3);
        int4 m = make_int4(0, 0, 0, kOut);  // no map of this binade: not taken
        if (ours && b3 >= 0 && b3 < kBinades) m = tc[((size_t)b3 * nblocks + c) * kCB + q];
        sh.map[q][tid % 3] = m;
      }
#pragma unroll
      for (int q = 0; q < kEach; ++q) sh.t[tid + q * kWalk] = j ? term2(v[q], fnx, fny) : term1(v[q], fnx, fny);
    }
    __syncthreads();
    if (tid < 32) {  // one warp, every lane the same
      const int eb = e;
      bool ok = ours;  // k, e hold the sum
#pragma unroll 1
      for (int q = 0; q < kCB; ++q) {
        if (ok) {
          const RunMap m = to_map(sh.map[q][e - eb + 1]);
          if (fits(k, m)) {
            k += m.D0 + ((k & 1) ? m.d : 0);
            continue;
          }
          s = join(k, e);
        }
        const float4* t = reinterpret_cast<const float4*>(sh.t + q * kChunk);
        float4 x[4], y[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = t[i];
#pragma unroll 4
        for (int r = 4; r <= kChunk / 4; r += 4) {  // the next 16 terms load while these are added
#pragma unroll
          for (int i = 0; i < 4; ++i) y[i] = t[min(r + i, kChunk / 4 - 1)];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, x[i].x), x[i].y), x[i].z), x[i].w);
            x[i] = y[i];
          }
        }
        ok = split(s, k, e) && ours && e >= eb - 1 && e <= eb + 1;
      }
      if (ok) s = join(k, e);
      if (tid == 0) sh.s = s;
    }
    __syncthreads();
    s = sh.s;
    ++c;
  }
  if (tid == 0) out[j] = s;
}

__global__ void stats_finish_kernel(const float* __restrict__ sums, float* __restrict__ stats) {
  const float avg = sums[0], sum_s2 = sums[1];
  const float var = __fsqrt_rn(__fsub_rn(sum_s2, __fmul_rn(avg, avg)));
  const float up = __fadd_rn(avg, __fmul_rn(6.f, var));
  const float lo = __fsub_rn(avg, __fmul_rn(6.f, var));
  stats[0] = avg;
  stats[1] = (float)(int)up;  // int truncation (norm.cu:166-167)
  stats[2] = (float)(int)lo;
  stats[3] = (sum_s2 > __fmul_rn(avg, avg)) ? 1.f : 0.f;
  if (!(up == up) || !(lo == lo)) stats[3] = 0.f;
}

int blocks_of(long long n) { return (int)((n + kBlock - 1) / kBlock); }

}  // namespace

size_t serial_stats_bytes(long long n) {
  // maps of chunks and blocks, FP64 block sums, exponents and the two sums
  return (size_t)blocks_of(n) * (2 * kBinades * (kCB + 1) * sizeof(int4) + 2 * sizeof(double)) + 16;
}

void serial_stats(const float* img, int nx, int ny, float* stats, void* scratch, cudaStream_t s) {
  const long long n = (long long)nx * ny;
  const int nb = blocks_of(n), nc = nb * kCB;
  int4* chunks = static_cast<int4*>(scratch);
  int4* blocks = chunks + (size_t)2 * kBinades * nc;
  double* sums = reinterpret_cast<double*>(blocks + (size_t)2 * kBinades * nb);
  int* etop = reinterpret_cast<int*>(sums + 2 * (size_t)nb);
  float* out = reinterpret_cast<float*>(etop + 2);
  const float fnx = (float)nx, fny = (float)ny;
  block_sum_kernel<<<ceil_div(nb, 8), 256, 0, s>>>(img, n, fnx, fny, sums, nb);
  GISSPA_LAUNCH_CHECK();
  binade_kernel<<<1, 1024, 0, s>>>(sums, nb, etop);
  GISSPA_LAUNCH_CHECK();
  // (whole blocks: the last one's chunks past the image are zeros)
  chunk_map_kernel<<<dim3(ceil_div((long long)nb * kBlock, kWarps * 32 * kPerLane), 2), kWarps * 32, 0, s>>>(
      img, n, fnx, fny, etop, chunks, nc);
  GISSPA_LAUNCH_CHECK();
  block_map_kernel<<<ceil_div(2 * kBinades * nb, 128), 128, 0, s>>>(chunks, nb, blocks);
  GISSPA_LAUNCH_CHECK();
  walk_kernel<<<2, kWalk, 0, s>>>(img, n, fnx, fny, etop, chunks, blocks, nb, out);
  GISSPA_LAUNCH_CHECK();
  stats_finish_kernel<<<1, 1, 0, s>>>(out, stats);
  GISSPA_LAUNCH_CHECK();
}

}  // namespace gisspa
