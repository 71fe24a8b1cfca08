// AC-RANSAC hypothesis scoring (include/gbsfm.h, gbsfm_acransac_score): the
// per-model body of ACRANSAC's main loop
// (libs/feature/include/mvg/feature/estimator_acransac.h:170-200) for a batch
// of candidate resection models, one CTA per model:
//   1. the squared reprojection error of every correspondence
//      (ResectionSquaredResidualError, libs/sfm/include/mvg/sfm/sfm_robust.h:
//      197-204) as a 64-bit key (the bits of a non-negative double order like
//      the double) with the correspondence index as payload;
//   2. a bitonic sort of the (key, index) pairs: the pairs are distinct, so
//      the result is std::sort's order of (error, index) pairs.  Up to 8192
//      correspondences in registers (k_score_block), above that in a per-CTA
//      global slice (k_acransac_score);
//   3. bestNFA (estimator_acransac.h:75-97) as a block-wide argmin over k,
//      the smallest k winning ties as the reference's strict '<' scan does.
// The logcombi tables (:40-65, float-rounded as the reference stores them)
// are built on the device from a table of log10(i), summed in the
// reference's order.
#include <math_constants.h>

#include <cfloat>
#include <cmath>
#include <cstring>
#include <limits>

#include "../../include/gbsfm.h"
#include "gbba_internal.h"

namespace gbba {
namespace {

constexpr int kScoreThreads = 512;
constexpr int64_t kBlockPairs = 8192;  // sorted in registers: a 13-bit index, 128 KB of shared memory

__global__ void __launch_bounds__(256) k_log10_table(int64_t n, double* __restrict__ lg) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i <= n; i += (int64_t)gridDim.x * blockDim.x)
    lg[i] = i > 0 ? log10((double)i) : 0.0;
}

// logcombi(k, n): 0 for k >= n or k <= 0, else the sum over i = 1..min(k, n-k)
// of log10(n - i + 1) - log10(i), in that order.
__device__ double logcombi(int64_t k, int64_t n, const double* __restrict__ lg) {
  if (k >= n || k <= 0) return 0.0;
  if (n - k < k) k = n - k;
  double r = 0.0;
  for (int64_t i = 1; i <= k; ++i) r += lg[n - i + 1] - lg[i];
  return r;
}

// logc_n[k] = logcombi(k, n), logc_k[m] = logcombi(sample_size, m), k, m in 0..n.
// logc_n is one running sum (its k-th value the sum of the first min(k, n - k)
// terms): block 0 walks it once, the terms staged by all its threads, the
// other blocks form logc_k.  A chain of n / 2 FP64 additions bounds it: 2,000
// correspondences 56 us beside the scoring, against 149 with a sum of its own for every k.  The
// scoring kernel is launched beside it and waits for it before it reads the
// tables.
constexpr int kLogcThreads = 256;
constexpr int kLogcChunk = 1024;
__global__ void __launch_bounds__(kLogcThreads) k_logcombi(int64_t n, int sample_size, const double* __restrict__ lg,
                                                           float* __restrict__ logc_n, float* __restrict__ logc_k) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (blockIdx.x > 0) {
    for (int64_t i = (blockIdx.x - 1) * (int64_t)kLogcThreads + threadIdx.x; i <= n;
         i += (gridDim.x - 1) * (int64_t)kLogcThreads)
      logc_k[i] = (float)logcombi(sample_size, i, lg);
    return;
  }
  __shared__ double term[kLogcChunk];
  double r = 0.0;
  const int64_t half = n / 2;
  if (threadIdx.x == 0) logc_n[0] = logc_n[n] = 0.0f;
  for (int64_t i0 = 1; i0 <= half; i0 += kLogcChunk) {
    const int m = (int)min((int64_t)kLogcChunk, half - i0 + 1);
    for (int i = threadIdx.x; i < m; i += kLogcThreads) term[i] = lg[n - (i0 + i) + 1] - lg[i0 + i];
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll 8
      for (int i = 0; i < m; ++i) {
        r += term[i];
        term[i] = r;
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < m; i += kLogcThreads) {
      const float v = (float)term[i];
      const int64_t k = i0 + i;
      if (k < n) {  // k = n only when n = 1, where the value is 0
        logc_n[k] = v;
        logc_n[n - k] = v;
      }
    }
    __syncthreads();
  }
}

// |Project(P, X) - x|^2 with Project = (P [X; 1]).head(2) / z, the products
// and sums kept apart (no contraction) in the order of the matrix rows.
__device__ __forceinline__ double resection_error(const double* __restrict__ m, double X0, double X1, double X2,
                                                  double x, double y) {
  double h[3];
#pragma unroll
  for (int r = 0; r < 3; ++r)
    h[r] = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(m[4 * r], X0), __dmul_rn(m[4 * r + 1], X1)),
                               __dmul_rn(m[4 * r + 2], X2)),
                     m[4 * r + 3]);
  const double dx = h[0] / h[2] - x, dy = h[1] / h[2] - y;
  return __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
}

__device__ __forceinline__ bool pair_less(unsigned long long ka, uint32_t va, unsigned long long kb, uint32_t vb) {
  return ka < kb || (ka == kb && va < vb);
}

// Ascending bitonic sort of p (a power of two) pairs.
__device__ void bitonic_sort(unsigned long long* keys, uint32_t* vals, int64_t p) {
  for (int64_t size = 2; size <= p; size <<= 1) {
    for (int64_t stride = size >> 1; stride > 0; stride >>= 1) {
      for (int64_t t = threadIdx.x; t < p / 2; t += blockDim.x) {
        const int64_t i = 2 * t - (t & (stride - 1));  // lower element of the t-th compared pair
        const int64_t j = i + stride;
        const bool up = (i & size) == 0;
        const unsigned long long ki = keys[i], kj = keys[j];
        const uint32_t vi = vals[i], vj = vals[j];
        if (pair_less(kj, vj, ki, vi) == up) {
          keys[i] = kj;
          keys[j] = ki;
          vals[i] = vj;
          vals[j] = vi;
        }
      }
      __syncthreads();
    }
  }
}

struct ScoreArgs {
  int64_t n, h, p;
  const double *x2d, *x3d, *models;
  const float *logc_n, *logc_k;
  int sample_size;
  double loge0, logalpha0, mult_error, max_threshold;
  float margin;  // of bestNFA's FP32 pass
  double* nfa;
  int32_t* inliers;
  double* error_max;
  uint32_t* order;
  unsigned long long* scratch_keys;  // global slices when p > kSmemPairs
  uint32_t* scratch_vals;
};

// Up to 8192 correspondences: one CTA of 256 threads per model, E pairs per
// thread in registers (E = p / 256, thread t holds ranks tE .. tE + E - 1).
// A pair is one 64-bit word, the error's bits 62..12 above a 13-bit index: the
// compared strides below E stay in a thread, those below 32 E are shuffles,
// and only the few larger ones go through shared memory (2,048 pairs: 6 of 66
// steps, where every step was a barrier).  Neighbours that agree in the 51
// bits are put in order of the whole (error, index) afterwards.
// bestNFA first runs in FP32 and the FP64 formula is evaluated only where that
// comes within `margin` (an upper bound of its error, from the caller) of the
// smallest value: the FP64 log10 of every error took as long as the residuals.
// Bound by the residuals' FP64 arithmetic (41 operations a correspondence):
// 1,024 models x 2,000 correspondences 196 us, against 391.
constexpr int kSortThreads = 256;
template <int E>
__device__ __forceinline__ void sort_words(unsigned long long (&w)[E], unsigned long long* xbuf) {
  constexpr int P = E * kSortThreads;
  const int t = threadIdx.x;
  auto exchange = [](unsigned long long& lo, unsigned long long& hi, bool up) {
    const bool swap = (lo > hi) == up;
    const unsigned long long a = lo, b = hi;
    lo = swap ? b : a;
    hi = swap ? a : b;
  };
#pragma unroll 1
  for (int size = 2; size <= P; size <<= 1) {
    // strides across warps, then across lanes
#pragma unroll 1
    for (int d = size / (2 * E); d >= 1; d >>= 1) {
      const bool up = ((t * E) & size) == 0;
      const bool keep_min = ((t & d) == 0) == up;
      if (d >= 32) {
        __syncthreads();
#pragma unroll
        for (int e = 0; e < E; ++e) xbuf[e * kSortThreads + t] = w[e];
        __syncthreads();
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const unsigned long long o = xbuf[e * kSortThreads + (t ^ d)];
          w[e] = (o < w[e]) == keep_min ? o : w[e];
        }
      } else {
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const unsigned long long o = __shfl_xor_sync(0xffffffffu, w[e], d);
          w[e] = (o < w[e]) == keep_min ? o : w[e];
        }
      }
    }
    // strides inside a thread
#pragma unroll
    for (int s = E / 2; s >= 1; s >>= 1) {
      if (s >= size) continue;
#pragma unroll
      for (int e = 0; e < E; ++e)
        if ((e & s) == 0) exchange(w[e], w[e + s], ((t * E + e) & size) == 0);
    }
  }
}

// log10 of (the double whose bits 62..12 are given) + FLT_MIN, within the
// FP32 rounding of its value: through a float of the truncated mantissa, or in
// FP64 outside the floats' normal range.
__device__ __forceinline__ float log10_low(unsigned long long bits51) {
  const int ex = (int)(bits51 >> 40) - 1023 + 127;
  if (ex <= 0 || ex >= 254) return (float)log10(__longlong_as_double((long long)(bits51 << 12)) + (double)FLT_MIN);
  return log10f(__uint_as_float(((unsigned)ex << 23) | ((unsigned)(bits51 >> 17) & 0x7fffffu)) + FLT_MIN);
}

template <int E>
__global__ void __launch_bounds__(kSortThreads) k_score_block(ScoreArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int P = E * kSortThreads;
  constexpr unsigned kIndex = 0x1fffu;
  unsigned long long* xbuf = reinterpret_cast<unsigned long long*>(smem);  // [P] exchange, then the sorted words
  unsigned long long* errs = xbuf + P;                                     // [n] the errors' bits
  __shared__ double sh_model[12];
  __shared__ float sh_min[kSortThreads / 32];
  __shared__ double sh_best[kSortThreads / 32];
  __shared__ int sh_best_k[kSortThreads / 32];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, n = (int)a.n;
  const unsigned long long thr = a.max_threshold >= 0.0 ? (unsigned long long)__double_as_longlong(a.max_threshold + 0.0) : 0ull;
  const bool any = a.max_threshold >= 0.0;
  bool waited = false;
  for (int64_t m = blockIdx.x; m < a.h; m += gridDim.x) {
    if (t < 12) sh_model[t] = a.models[12 * m + t];
    __syncthreads();
    for (int i = t; i < n; i += kSortThreads) {
      const double e = resection_error(sh_model, a.x3d[3 * i], a.x3d[3 * i + 1], a.x3d[3 * i + 2], a.x2d[2 * i],
                                       a.x2d[2 * i + 1]);
      errs[i] = (unsigned long long)__double_as_longlong(e + 0.0);  // +0.0 for -0.0: the bit order is the double order
    }
    __syncthreads();
    unsigned long long w[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      // (the order of the words before the sort is free: coalesced)
      const int i = e * kSortThreads + t;
      w[e] = ~0ull;
      if (i < n) {
        const unsigned long long b = errs[i];
        w[e] = (b >> 63 ? ~0ull << 13 : (b >> 12) << 13) | (unsigned)i;  // a NaN's sign bit: past every error
      }
    }
    sort_words<E>(w, xbuf);
    __syncthreads();
#pragma unroll
    for (int e = 0; e < E; ++e) xbuf[t * E + e] = w[e];
    __syncthreads();
    // words that agree in the error's 51 bits: by the whole (error, index)
    auto tie = [&](int i) { return i + 1 < n && (xbuf[i] >> 13) == (xbuf[i + 1] >> 13); };
    bool ties = false;
    for (int i = t; i < n; i += kSortThreads) ties |= tie(i);
    if (__syncthreads_or(ties)) {
      for (bool moved = true; moved;) {
        bool any_swap = false;
#pragma unroll 1
        for (int odd = 0; odd < 2; ++odd) {
          for (int i = 2 * t + odd; i < n; i += 2 * kSortThreads) {
            if (!tie(i)) continue;
            const unsigned long long x = xbuf[i], y = xbuf[i + 1];
            const unsigned ix = (unsigned)x & kIndex, iy = (unsigned)y & kIndex;
            if (errs[iy] < errs[ix] || (errs[iy] == errs[ix] && iy < ix)) {
              xbuf[i] = y;
              xbuf[i + 1] = x;
              any_swap = true;
            }
          }
          __syncthreads();
        }
        moved = __syncthreads_or(any_swap) != 0;
      }
    }
    if (!waited) {  // the logcombi tables are ready when the kernel before has finished
      asm volatile("griddepcontrol.wait;" ::: "memory");
      waited = true;
    }
    // bestNFA: k = sample_size + 1 .. n while e[k-1] <= max_threshold
    auto passes = [&](int k) { return any && errs[(unsigned)xbuf[k - 1] & kIndex] <= thr; };
    auto nfa32 = [&](int k) {
      const float logalpha = (float)a.logalpha0 + (float)a.mult_error * log10_low(xbuf[k - 1] >> 13);
      return (float)a.loge0 + logalpha * (float)(k - a.sample_size) + __ldcg(a.logc_n + k) + __ldcg(a.logc_k + k);
    };
    float low = CUDART_INF_F;
    for (int k = a.sample_size + 1 + t; k <= n; k += kSortThreads)
      if (passes(k)) low = fminf(low, nfa32(k));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) low = fminf(low, __shfl_xor_sync(0xffffffffu, low, o));
    if (lane == 0) sh_min[warp] = low;
    __syncthreads();
#pragma unroll
    for (int v = 0; v < kSortThreads / 32; ++v) low = fminf(low, sh_min[v]);
    const float limit = low + a.margin;
    double best = CUDART_INF;
    int best_k = a.sample_size;
    for (int k = a.sample_size + 1 + t; k <= n; k += kSortThreads) {
      if (!passes(k) || nfa32(k) > limit) continue;
      const double e = __longlong_as_double((long long)errs[(unsigned)xbuf[k - 1] & kIndex]);
      const double logalpha = a.logalpha0 + a.mult_error * log10(e + (double)FLT_MIN);
      const double v = a.loge0 + logalpha * (double)(k - a.sample_size) + (double)__ldcg(a.logc_n + k) +
                       (double)__ldcg(a.logc_k + k);
      if (v < best) {  // k ascends per thread: the first of equal values stays
        best = v;
        best_k = k;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int ok = __shfl_xor_sync(0xffffffffu, best_k, o);
      if (ob < best || (ob == best && ok < best_k)) {
        best = ob;
        best_k = ok;
      }
    }
    if (lane == 0) {
      sh_best[warp] = best;
      sh_best_k[warp] = best_k;
    }
    __syncthreads();
    if (t == 0) {
      for (int v = 1; v < kSortThreads / 32; ++v)
        if (sh_best[v] < best || (sh_best[v] == best && sh_best_k[v] < best_k)) {
          best = sh_best[v];
          best_k = sh_best_k[v];
        }
      const bool found = best < CUDART_INF;
      a.nfa[m] = best;
      a.inliers[m] = found ? best_k : a.sample_size;
      a.error_max[m] = found ? __longlong_as_double((long long)errs[(unsigned)xbuf[best_k - 1] & kIndex]) : CUDART_INF;
    }
    if (a.order)
      for (int i = t; i < n; i += kSortThreads) a.order[m * a.n + i] = (unsigned)xbuf[i] & kIndex;
    __syncthreads();
  }
}

// Above 8192 correspondences: the pairs in a per-CTA global slice.
__global__ void __launch_bounds__(kScoreThreads) k_acransac_score(ScoreArgs a) {
  __shared__ double sh_model[12];
  __shared__ double sh_best[kScoreThreads / 32];
  __shared__ int64_t sh_best_k[kScoreThreads / 32];
  unsigned long long* keys = a.scratch_keys + blockIdx.x * a.p;
  uint32_t* vals = a.scratch_vals + blockIdx.x * a.p;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int64_t m = blockIdx.x; m < a.h; m += gridDim.x) {
    if (threadIdx.x < 12) sh_model[threadIdx.x] = a.models[12 * m + threadIdx.x];
    __syncthreads();
    for (int64_t i = threadIdx.x; i < a.p; i += blockDim.x) {
      if (i < a.n) {
        const double e = resection_error(sh_model, a.x3d[3 * i], a.x3d[3 * i + 1], a.x3d[3 * i + 2], a.x2d[2 * i],
                                         a.x2d[2 * i + 1]);
        // +0.0 for -0.0 so that the bit order is the double order
        keys[i] = (unsigned long long)__double_as_longlong(e + 0.0);
        vals[i] = (uint32_t)i;
      } else {
        keys[i] = ~0ull;
        vals[i] = 0xffffffffu;
      }
    }
    __syncthreads();
    bitonic_sort(keys, vals, a.p);
    // bestNFA: k = sample_size + 1 .. n while e[k-1] <= max_threshold
    double best = CUDART_INF;
    int64_t best_k = a.sample_size;
    for (int64_t k = a.sample_size + 1 + threadIdx.x; k <= a.n; k += blockDim.x) {
      const double e = __longlong_as_double((long long)keys[k - 1]);
      if (!(e <= a.max_threshold)) break;  // sorted: every later k fails too
      const double logalpha = a.logalpha0 + a.mult_error * log10(e + (double)FLT_MIN);
      const double v = a.loge0 + logalpha * (double)(k - a.sample_size) + (double)a.logc_n[k] + (double)a.logc_k[k];
      if (v < best) {  // k ascends per thread: the first of equal values stays
        best = v;
        best_k = k;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int64_t ok = __shfl_xor_sync(0xffffffffu, best_k, o);
      if (ob < best || (ob == best && ok < best_k)) {
        best = ob;
        best_k = ok;
      }
    }
    if (lane == 0) {
      sh_best[warp] = best;
      sh_best_k[warp] = best_k;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < kScoreThreads / 32; ++w)
        if (sh_best[w] < best || (sh_best[w] == best && sh_best_k[w] < best_k)) {
          best = sh_best[w];
          best_k = sh_best_k[w];
        }
      const bool found = best < CUDART_INF;
      a.nfa[m] = best;
      a.inliers[m] = (int32_t)(found ? best_k : a.sample_size);
      a.error_max[m] = found ? __longlong_as_double((long long)keys[best_k - 1]) : CUDART_INF;
    }
    if (a.order)
      for (int64_t i = threadIdx.x; i < a.n; i += blockDim.x) a.order[m * a.n + i] = vals[i];
    __syncthreads();
  }
}

int64_t next_pow2(int64_t n) {
  int64_t p = 2;
  while (p < n) p <<= 1;
  return p;
}

PerDeviceOnce g_score_smem[3];

}  // namespace
}  // namespace gbba

using namespace gbba;

extern "C" gbba_status gbsfm_acransac_score(gbba_handle* h, const gbsfm_acransac_params* prm, int64_t num_points,
                                            const double* x2d, const double* x3d, int64_t num_models,
                                            const double* models, double* nfa, int32_t* num_inliers,
                                            double* error_max, uint32_t* order, int32_t memory) {
  if (!prm || prm->sample_size < 1 || prm->max_models < 1 || num_models < 0 || num_points <= prm->sample_size)
    return GBBA_ERROR_INVALID_ARGUMENT;
  if (num_models > 0 && (!x2d || !x3d || !models || !nfa || !num_inliers || !error_max))
    return GBBA_ERROR_INVALID_ARGUMENT;
  if (num_points > 0x7fffffffLL) return GBBA_ERROR_TOO_LARGE;
  return sfm_guard(h, [&]() {
    if (num_models == 0) return GBBA_SUCCESS;
    const int64_t n = num_points;
    const bool in_block = n <= kBlockPairs;
    const int64_t p = in_block ? std::max<int64_t>(kSortThreads, next_pow2(n)) : next_pow2(n);
    const size_t smem = in_block ? sizeof(unsigned long long) * (size_t)(p + n) : 0;
    // CTAs per SM: the shared memory and 64 registers a thread allow
    const int64_t per_sm = in_block ? std::max<int64_t>(1, std::min<int64_t>(4, (220 << 10) / (int64_t)smem)) : 2;
    const unsigned grid = (unsigned)std::min<int64_t>(num_models, (int64_t)h->sm_count * per_sm);
    const size_t scratch = in_block ? 0 : (size_t)grid * p * (sizeof(unsigned long long) + sizeof(uint32_t));
    h->arena.reset();
    h->arena.reserve(sizeof(double) * (5 * n + 12 * num_models + 3 * num_models + n + 1) + 2 * sizeof(float) * (n + 1) +
                     sizeof(int32_t) * num_models + (order ? sizeof(uint32_t) * num_models * n : 0) + scratch +
                     256 * 16);
    ScoreArgs a;
    a.n = n;
    a.h = num_models;
    a.p = p;
    a.x2d = in_view(h, x2d, 2 * n, memory);
    a.x3d = in_view(h, x3d, 3 * n, memory);
    a.models = in_view(h, models, 12 * num_models, memory);
    a.nfa = out_view(h, nfa, num_models, memory);
    a.inliers = out_view(h, num_inliers, num_models, memory);
    a.error_max = out_view(h, error_max, num_models, memory);
    a.order = out_view(h, order, num_models * n, memory);
    double* lg = h->arena.take<double>(n + 1);
    float* logc_n = h->arena.take<float>(n + 1);
    float* logc_k = h->arena.take<float>(n + 1);
    a.logc_n = logc_n;
    a.logc_k = logc_k;
    a.scratch_keys = in_block ? nullptr : h->arena.take<unsigned long long>(grid * p);
    a.scratch_vals = in_block ? nullptr : h->arena.take<uint32_t>(grid * p);
    a.sample_size = prm->sample_size;
    // loge0 = log10(MAX_MODELS * (nData - sample_size)) (estimator_acransac.h:147)
    a.loge0 = log10((double)prm->max_models * (double)(n - prm->sample_size));
    a.logalpha0 = prm->logalpha0;
    a.mult_error = prm->mult_error;
    a.max_threshold = prm->max_threshold;
    // The FP32 pass is off by at most: in log10 of the error (at most 309 in
    // size), 2^-22 from the truncated mantissa and a few units in the last
    // place; then one rounding (2^-24) of each of five terms, none above
    // `most` in size (the tables: log10 of at most 2^n).
    const double most = std::fabs(a.loge0) + (std::fabs(a.logalpha0) + 309.0 * std::fabs(a.mult_error)) * (double)n +
                        2.0 * (double)n;
    const double margin = 2.0 * ((double)n * std::fabs(a.mult_error) * 4e-5 + 5e-7 * most);
    a.margin = std::isfinite(margin) && margin < 1e30 ? (float)margin : std::numeric_limits<float>::infinity();
    KernelTimer timer(h);
    k_log10_table<<<grid_for(h, n + 1, 256), 256, 0, h->active>>>(n, lg);
    check_launch(h);
    k_logcombi<<<1 + grid_for(h, n + 1, kLogcThreads), kLogcThreads, 0, h->active>>>(n, prm->sample_size, lg, logc_n,
                                                                                     logc_k);
    check_launch(h);
    if (in_block) {
      auto launch = [&](auto kern) {
        if (smem > 48 * 1024)
          g_score_smem[kern == k_score_block<8> ? 0 : kern == k_score_block<16> ? 1 : 2].run([&]() {
            GBBA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)(2 * sizeof(unsigned long long) * kBlockPairs)));
          });
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(grid);
        cfg.blockDim = dim3(kSortThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = h->active;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        GBBA_CUDA(cudaLaunchKernelEx(&cfg, kern, a));
        check_launch(h);
      };
      switch (p / kSortThreads) {
        case 1: launch(k_score_block<1>); break;
        case 2: launch(k_score_block<2>); break;
        case 4: launch(k_score_block<4>); break;
        case 8: launch(k_score_block<8>); break;
        case 16: launch(k_score_block<16>); break;
        default: launch(k_score_block<32>); break;
      }
    } else {
      k_acransac_score<<<grid, kScoreThreads, 0, h->active>>>(a);
      check_launch(h);
    }
    timer.stop();
    out_back(h, nfa, a.nfa, num_models, memory);
    out_back(h, num_inliers, a.inliers, num_models, memory);
    out_back(h, error_max, a.error_max, num_models, memory);
    out_back(h, order, a.order, num_models * n, memory);
    GBBA_CUDA(cudaStreamSynchronize(h->active));
    return GBBA_SUCCESS;
  });
}
