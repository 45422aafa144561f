// fft_generic.cuh — batched 1D/2D complex FFTs for every size outside the hot loop
// (template and image preparation, window spectra, per-angle template spectra).
//
// Power-of-two lengths up to 16384 run one shared-memory radix-2 transform per row; lengths
// up to 8192 whose prime factors are 2, 3, 5 and 7 run one shared-memory mixed-radix
// Stockham transform per row; other lengths use Bluestein's chirp-z algorithm on top of the
// power-of-two transform.  2D transforms are
// rows -> transpose -> rows (-> transpose).  All transforms are unnormalised.
#pragma once

#include <utility>

#include <atomic>
#include <map>
#include <memory>
#include <vector>

#include "common.cuh"

namespace gisspa {

// Incremented on every device buffer (re)allocation and release in the process: a captured
// CUDA graph holds raw buffer addresses and is rebuilt when this has moved since its capture.
inline std::atomic<unsigned long long>& alloc_generation() {
  static std::atomic<unsigned long long> g{0};
  return g;
}

// Grow-only device buffer.
class DevBuf {
 public:
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  DevBuf(DevBuf&& o) noexcept : p_(o.p_), n_(o.n_) { o.p_ = nullptr; o.n_ = 0; }
  ~DevBuf() { release(); }
  void* ensure(size_t bytes) {
    if (bytes > n_) {
      release();
      ++alloc_generation();
      GISSPA_CUDA(cudaMalloc(&p_, bytes));
      n_ = bytes;
    }
    return p_;
  }
  void release() {
    if (p_) {
      ++alloc_generation();
      cudaFree(p_);
    }
    p_ = nullptr;
    n_ = 0;
  }
  template <typename T>
  T* as() const { return static_cast<T*>(p_); }
  size_t size() const { return n_; }
  void swap(DevBuf& o) noexcept {
    std::swap(p_, o.p_);
    std::swap(n_, o.n_);
  }

 private:
  void* p_ = nullptr;
  size_t n_ = 0;
};

// Stockham stages of a row of length n: radices from kSmoothRadices (register transforms of that
// length) whose product is n, as few as possible, the largest as small as possible; ns = 0 when n
// has a prime factor above 7 (such lengths use Bluestein's algorithm).  Odd radices come first: the
// first stage writes its outputs R apart, in distinct banks for odd R.
constexpr int kSmoothRadices[] = {2, 3, 4, 5, 6, 7, 8, 10, 12, 14, 15, 16};
struct SmoothPlan {
  static constexpr int kMax = 14;  // radices of 2^13 and one more
  int ns = 0;
  int r[kMax] = {};
  unsigned div_m[kMax] = {}, div_ns[kMax] = {};  // fast_div of n / r and of the radices before
};
// i / d for i d < 2^32 (mul: fast_div_mul(d))
__host__ __device__ constexpr unsigned fast_div_mul(unsigned d) {
  return d > 1 ? (unsigned)(((1ull << 32) + d - 1) / d) : 0;
}
__device__ __forceinline__ int fast_div(int i, unsigned mul) { return mul ? (int)__umulhi((unsigned)i, mul) : i; }
// last: a divisor of n to end with (0: any).
SmoothPlan smooth_plan(int n, int last = 0);
// Rows of length n per CTA of `threads`, a multiple of `step`, of at most max_points points (or
// `step`): the count whose butterflies fill the CTA's passes best.
int smooth_rows(const SmoothPlan& plan, int n, int threads, int max_points, int step = 1);
// Longest row the mixed-radix kernel takes (two shared-memory copies of 8192 complex = 128 KB).
constexpr int kSmoothMax = 8192;

class FftEngine {
 public:
  // Table of exp(-2 pi i p / n), p < n (device pointer, cached per n).
  const float2* twiddles(int n);
  // In-place transform of `rows` contiguous rows of length n (any n >= 1).
  void rows(float2* data, long long rows, int n, int sign, float scale, cudaStream_t s);
  // out[b][c][r] = in[b][r][c] for rows x cols matrices; optional row subset
  // [0, out_rows) of the transposed result (i.e. input columns [0, out_rows)).
  void transpose(const float2* in, float2* out, int batch, int rows, int cols, cudaStream_t s, int out_rows = -1);
  // In-place 2D transform of batch x ny x nx, using tmp (same size) as scratch.
  void fft2(float2* data, float2* tmp, int batch, int ny, int nx, int sign, float scale, cudaStream_t s);

 private:
  struct Blue {
    int n = 0, m = 0;
    DevBuf chirp, bfwd, binv;
  };
  Blue& bluestein(int n);
  std::map<int, DevBuf> tw_;
  std::map<int, std::unique_ptr<Blue>> blue_;
  DevBuf scratch_;
};

bool is_pow2(long long n);

}  // namespace gisspa
