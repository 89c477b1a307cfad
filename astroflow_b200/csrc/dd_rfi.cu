// RFI stages and input layout for the B200 dedispersion path.
//
//  * time binning with sqrt compression (src/core/dedispered.cu:337-376);
//  * IQRM channel masks (src/core/iqrm.cu:21-185, 203-345), computed entirely on
//    the device: per-channel sums are exact 64-bit integers (the reference's
//    double sums of integer samples are exact, so the statistics agree), and
//    differences, quartiles, threshold and votes run in one block per (window,
//    lag) instead of the reference's two host round trips per lag;
//  * window-mask application (src/rfi/rfimarker.cu:309-390), zero-DM over a
//    channel range with an exact integer mean, and the static channel mask
//    (rfimarker.cu:469-488), fused into the pass that writes the channel-major
//    layout the dedispersion kernels read.
// Host-side arithmetic of the reference (its percentile and threshold code runs
// on the CPU) is reproduced with explicitly rounded intrinsics so that no
// multiply-add contraction changes it.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <cstdio>

#include "dd_internal.h"

namespace dd {
namespace {

template <typename T> struct Lim;
template <> struct Lim<uint8_t> { static constexpr uint64_t vmax = 255u; };
template <> struct Lim<uint16_t> { static constexpr uint64_t vmax = 65535u; };
template <> struct Lim<uint32_t> { static constexpr uint64_t vmax = 4294967295u; };

// ---------------------------------------------------------------- binning
// One thread per channel and output sample (grid: channel blocks x output rows,
// rows strided by gridDim.y); smax_full = sqrt(vmax * ds) of the full bins,
// evaluated on the host with the same IEEE square root.
template <typename T>
__global__ void k_time_binning(const T* __restrict__ in, T* __restrict__ out, int64_t nchans,
                               int64_t ndata, int ds, int64_t nout, double smax_full) {
  const int64_t c = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (c >= nchans) return;
  const uint64_t vmax = Lim<T>::vmax;
  for (int64_t k = blockIdx.y; k < nout; k += gridDim.y) {
    const int64_t t0 = k * ds;
    const int64_t t1 = t0 + ds < ndata ? t0 + ds : ndata;
    uint64_t sum = 0;
    for (int64_t t = t0; t < t1; ++t) sum += static_cast<uint64_t>(in[c + t * nchans]);
    const uint64_t cnt = static_cast<uint64_t>(t1 - t0);
    const double s = sqrt(static_cast<double>(sum));
    const double smax = cnt == static_cast<uint64_t>(ds)
                            ? smax_full
                            : sqrt(static_cast<double>(vmax * (cnt ? cnt : 1)));
    const double v = __dmul_rn(__ddiv_rn(s, smax > 0.0 ? smax : 1.0), static_cast<double>(vmax));
    out[c + k * nchans] = static_cast<T>(v < static_cast<double>(vmax) ? v : static_cast<double>(vmax));
  }
}

// The value of a full bin depends only on the integer sum of its ds samples, so
// for 8- and 16-bit samples every value is tabulated once per plan (lut[sum],
// sum in [0, ds * vmax]) by the same expression as k_time_binning, and the
// binning becomes a gather: V channels per thread (V * sizeof(T) = 4 bytes, one
// word per load and store).  A last, partial bin uses the expression directly.
template <typename T>
__global__ void k_binning_lut(T* __restrict__ lut, int64_t n, double smax_full) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint64_t vmax = Lim<T>::vmax;
  const double s = sqrt(static_cast<double>(i));
  const double v = __dmul_rn(__ddiv_rn(s, smax_full > 0.0 ? smax_full : 1.0), static_cast<double>(vmax));
  lut[i] = static_cast<T>(v < static_cast<double>(vmax) ? v : static_cast<double>(vmax));
}

template <typename T>
__device__ __forceinline__ T binned_value(uint64_t sum, uint64_t cnt) {
  const uint64_t vmax = Lim<T>::vmax;
  const double s = sqrt(static_cast<double>(sum));
  const double smax = sqrt(static_cast<double>(vmax * (cnt ? cnt : 1)));
  const double v = __dmul_rn(__ddiv_rn(s, smax > 0.0 ? smax : 1.0), static_cast<double>(vmax));
  return static_cast<T>(v < static_cast<double>(vmax) ? v : static_cast<double>(vmax));
}

// DS: the bin width (2, 4, 8), or 0 for any.  W: the word of channels that a thread loads,
// 32 bits, or less where rows do not start on one.  A block covers 256 words of channels
// and `rows` bins; with a fixed width the samples of several bins are loaded before the
// first is summed (sixteen loads in flight per thread; 2,048 channels x 300,001 samples in
// bins of four 242 us with one bin at a time; 2,870 channels, whose rows are whole pairs,
// 1380 us with the expression evaluated per bin, now 253).
template <typename T, typename W, int DS>
__global__ void __launch_bounds__(256) k_time_binning_lut(const T* __restrict__ in, T* __restrict__ out,
                                                          int64_t nchans, int64_t ndata, int ds, int64_t nout,
                                                          int rows, const T* __restrict__ lut) {
  constexpr int V = sizeof(W) / sizeof(T);
  constexpr int R = DS ? 16 / DS : 1;  // bins at a time
  const int64_t c = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) * V;
  if (c >= nchans) return;
  auto add = [](uint32_t w, uint32_t (&sum)[V]) {
#pragma unroll
    for (int v = 0; v < V; ++v) sum[v] += (w >> (8 * sizeof(T) * v)) & static_cast<uint32_t>(Lim<T>::vmax);
  };
  auto store = [&](int64_t k, const uint32_t (&sum)[V], int cnt) {
    uint32_t o = 0;
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const T b = cnt == ds ? __ldg(lut + sum[v]) : binned_value<T>(sum[v], static_cast<uint64_t>(cnt));
      o |= static_cast<uint32_t>(b) << (8 * sizeof(T) * v);
    }
    *reinterpret_cast<W*>(out + k * nchans + c) = static_cast<W>(o);
  };
  const int64_t k1 = min(nout, (static_cast<int64_t>(blockIdx.y) + 1) * rows);
  int64_t k = static_cast<int64_t>(blockIdx.y) * rows;
  if constexpr (DS > 0) {
    const int64_t full = min(k1, ndata / DS);
    for (; k + R <= full; k += R) {
      const T* p = in + k * DS * nchans + c;
      uint32_t w[R * DS];
#pragma unroll
      for (int i = 0; i < R * DS; ++i) w[i] = __ldg(reinterpret_cast<const W*>(p + i * nchans));
#pragma unroll
      for (int r = 0; r < R; ++r) {
        uint32_t sum[V];
#pragma unroll
        for (int v = 0; v < V; ++v) sum[v] = 0;
#pragma unroll
        for (int i = 0; i < DS; ++i) add(w[r * DS + i], sum);
        store(k + r, sum, DS);
      }
    }
  }
  for (; k < k1; ++k) {
    const int64_t t0 = k * ds, t1 = min(t0 + ds, ndata);
    uint32_t sum[V];
#pragma unroll
    for (int v = 0; v < V; ++v) sum[v] = 0;
    for (int64_t t = t0; t < t1; ++t) add(__ldg(reinterpret_cast<const W*>(in + t * nchans + c)), sum);
    store(k, sum, static_cast<int>(t1 - t0));
  }
}
template <typename T, typename W>
void launch_time_binning_lut(const void* in, void* out, int64_t ndata, int64_t nchans, int ds,
                             int64_t nout, const void* lut, cudaStream_t st) {
  const int64_t words = nchans / static_cast<int64_t>(sizeof(W) / sizeof(T));
  const int64_t gx = (words + 255) / 256;
  // bins per block: at least those loaded together; fewer than sixteen where the threads
  // would not fill the GPU (1024 channels, 5,000 samples in bins of sixteen 30 -> 12 us), more
  // where the grid would pass its limit
  const int least = ds == 2 || ds == 4 || ds == 8 ? 16 / ds : 1;
  int rows = 16;
  while (rows > least && (nout + rows - 1) / rows * words < 148 * 2048) rows /= 2;
  while ((nout + rows - 1) / rows > 65535) rows *= 2;
  const dim3 g(static_cast<unsigned>(gx), static_cast<unsigned>((nout + rows - 1) / rows));
  const T* i = static_cast<const T*>(in);
  T* o = static_cast<T*>(out);
  const T* l = static_cast<const T*>(lut);
  switch (ds) {
    case 2: k_time_binning_lut<T, W, 2><<<g, 256, 0, st>>>(i, o, nchans, ndata, ds, nout, rows, l); break;
    case 4: k_time_binning_lut<T, W, 4><<<g, 256, 0, st>>>(i, o, nchans, ndata, ds, nout, rows, l); break;
    case 8: k_time_binning_lut<T, W, 8><<<g, 256, 0, st>>>(i, o, nchans, ndata, ds, nout, rows, l); break;
    default: k_time_binning_lut<T, W, 0><<<g, 256, 0, st>>>(i, o, nchans, ndata, ds, nout, rows, l); break;
  }
  DD_LAUNCHED();
}

// ---------------------------------------------------------------- IQRM sums
// Calls f(a, b, w) for the runs [a, b) of samples of [lo, hi) that the same windows
// cover, so that overlapping windows (5 s every 2.5 s) share one read of the chunk; w
// is the first window that ends after a (starts and ends both grow along the list).
template <typename F>
__device__ __forceinline__ void for_window_runs(const uint32_t* __restrict__ win, int nwin,
                                                int64_t lo, int64_t hi, F&& f) {
  int first = 0, last = nwin;
  while (first < last) {
    const int mid = (first + last) >> 1;
    if (static_cast<int64_t>(win[2 * mid + 1]) > lo) last = mid; else first = mid + 1;
  }
  for (int64_t a = lo; a < hi;) {
    while (first < nwin && static_cast<int64_t>(win[2 * first + 1]) <= a) ++first;
    int64_t b = hi;
    bool covered = false;
    for (int w = first; w < nwin; ++w) {
      const int64_t t0 = win[2 * w], t1 = win[2 * w + 1];
      if (t1 < b) b = t1;
      if (t0 > a) {
        if (t0 < b) b = t0;
        break;
      }
      covered = true;
    }
    if (covered) f(a, b, first);
    a = b;
  }
}
// Adds one channel's sums of the run that starts at sample a to the windows covering
// it, from window w on.
__device__ __forceinline__ void add_window_sums(const uint32_t* __restrict__ win, int nwin, int w, int64_t a,
                                                int64_t csub, int64_t i, unsigned long long s,
                                                unsigned long long q,
                                                unsigned long long* __restrict__ sums) {
  for (; w < nwin && static_cast<int64_t>(win[2 * w]) <= a; ++w) {
    atomicAdd(&sums[(static_cast<int64_t>(w) * 2) * csub + i], s);
    atomicAdd(&sums[(static_cast<int64_t>(w) * 2 + 1) * csub + i], q);
  }
}

// Many short windows: a grid z each (their runs would hold a few samples, and a run costs
// its windows' bounds and sums).
__device__ __forceinline__ void take_window(const uint32_t*& win, int& nwin, int64_t csub,
                                            unsigned long long*& sums) {
  if (gridDim.z == 1) return;
  win += 2 * static_cast<int64_t>(blockIdx.z);
  sums += 2 * csub * blockIdx.z;
  nwin = 1;
}

// One channel per thread; grid.y: chunks of samples.
template <typename T>
__global__ void k_iqrm_stats(const T* __restrict__ x, int64_t nsamp, int64_t nchans, int64_t cs,
                             int64_t csub, const uint32_t* win, int nwin,
                             int64_t chunk, unsigned long long* sums) {
  int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= csub) return;
  const int64_t c = cs + i;
  take_window(win, nwin, csub, sums);
  const int64_t lo = static_cast<int64_t>(blockIdx.y) * chunk;
  const int64_t hi = lo + chunk < nsamp ? lo + chunk : nsamp;
  for_window_runs(win, nwin, lo, hi, [&](int64_t a, int64_t b, int w) {
    unsigned long long s = 0, s2 = 0;
    for (int64_t t = a; t < b; ++t) {
      unsigned long long v = x[t * nchans + c];
      s += v;
      s2 += v * v;
    }
    add_window_sums(win, nwin, w, a, csub, i, s, s2, sums);
  });
}

// 8-bit samples, four channels per thread: thread k covers channels (cs & ~3) + 4k
// .. + 3, one 32-bit word per row.  The words of four rows are transposed by byte
// permutes into one word per channel, whose sum and sum of squares are one dot
// product each: one operation per sample where taking the bytes apart took three.
// A chunk holds at most 1024 rows, so that the 32-bit partial sums cannot overflow
// (1024 x 255^2 < 2^32).  Needs nchans % 4 == 0 and an aligned input.  Bound by the
// reads (2,048 channels x 75,001 samples in two overlapping windows: 59 us, 298 us
// with one read per window, byte-wise sums and 1024-row chunks only).
__global__ void __launch_bounds__(128) k_iqrm_stats_u8w(
    const uint8_t* __restrict__ x, int64_t nsamp, int64_t nchans, int64_t cs, int64_t csub,
    const uint32_t* win, int nwin, int64_t chunk, unsigned long long* sums) {
  const int64_t c4 = (cs & ~int64_t(3)) + 4 * (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x);
  if (c4 >= cs + csub) return;
  take_window(win, nwin, csub, sums);
  const int64_t lo = static_cast<int64_t>(blockIdx.y) * chunk;
  const int64_t hi = lo + chunk < nsamp ? lo + chunk : nsamp;
  for_window_runs(win, nwin, lo, hi, [&](int64_t a, int64_t b, int w) {
    uint32_t s[4] = {0u, 0u, 0u, 0u}, q[4] = {0u, 0u, 0u, 0u};
    auto add4 = [&](uint32_t v0, uint32_t v1, uint32_t v2, uint32_t v3) {
      const uint32_t lo01 = __byte_perm(v0, v1, 0x5140), hi01 = __byte_perm(v0, v1, 0x7362);
      const uint32_t lo23 = __byte_perm(v2, v3, 0x5140), hi23 = __byte_perm(v2, v3, 0x7362);
      const uint32_t o[4] = {__byte_perm(lo01, lo23, 0x5410), __byte_perm(lo01, lo23, 0x7632),
                             __byte_perm(hi01, hi23, 0x5410), __byte_perm(hi01, hi23, 0x7632)};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        s[k] = __dp4a(o[k], 0x01010101u, s[k]);
        q[k] = __dp4a(o[k], o[k], q[k]);
      }
    };
    const uint8_t* p = x + a * nchans + c4;
    auto row = [&](int64_t r) { return __ldg(reinterpret_cast<const uint32_t*>(p + r * nchans)); };
    const int64_t n = b - a;
    int64_t r = 0;
    for (; r + 16 <= n; r += 16) {  // sixteen rows' loads in flight
      uint32_t v[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) v[k] = row(r + k);
#pragma unroll
      for (int k = 0; k < 16; k += 4) add4(v[k], v[k + 1], v[k + 2], v[k + 3]);
    }
    for (; r < n; ++r) add4(row(r), 0u, 0u, 0u);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int64_t ch = c4 + k;
      if (ch >= cs && ch < cs + csub) add_window_sums(win, nwin, w, a, csub, ch - cs, s[k], q[k], sums);
    }
  });
}

// 16-bit samples, two channels per thread (one 32-bit word per row): 32-bit sums and
// 64-bit sums of squares per chunk.  Needs nchans % 2 == 0 and an aligned input.
__global__ void __launch_bounds__(128) k_iqrm_stats_u16w(
    const uint16_t* __restrict__ x, int64_t nsamp, int64_t nchans, int64_t cs, int64_t csub,
    const uint32_t* win, int nwin, int64_t chunk, unsigned long long* sums) {
  const int64_t c2 = (cs & ~int64_t(1)) + 2 * (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x);
  if (c2 >= cs + csub) return;
  take_window(win, nwin, csub, sums);
  const int64_t lo = static_cast<int64_t>(blockIdx.y) * chunk;
  const int64_t hi = lo + chunk < nsamp ? lo + chunk : nsamp;
  for_window_runs(win, nwin, lo, hi, [&](int64_t a, int64_t b, int w) {
    uint32_t s[2] = {0u, 0u};
    unsigned long long q[2] = {0u, 0u};
    const uint16_t* p = x + a * nchans + c2;
    auto add = [&](uint32_t v) {
      const uint32_t l = v & 0xffffu, h = v >> 16;
      s[0] += l;
      s[1] += h;
      q[0] += static_cast<unsigned long long>(l) * l;
      q[1] += static_cast<unsigned long long>(h) * h;
    };
    auto row = [&](int64_t r) { return __ldg(reinterpret_cast<const uint32_t*>(p + r * nchans)); };
    const int64_t n = b - a;
    int64_t r = 0;
    for (; r + 16 <= n; r += 16) {
      uint32_t v[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) v[k] = row(r + k);
#pragma unroll
      for (int k = 0; k < 16; ++k) add(v[k]);
    }
    for (; r < n; ++r) add(row(r));
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int64_t ch = c2 + k;
      if (ch >= cs && ch < cs + csub) add_window_sums(win, nwin, w, a, csub, ch - cs, s[k], q[k], sums);
    }
  });
}

__device__ __forceinline__ int iqrm_target(int lag, int i, int csub) {
  if (lag < 0) return i < csub + lag ? i - lag : csub - 1;
  return i < lag ? 0 : i - lag;
}

// Percentile of iqrm.cu:299-306 (host code there): pos = q*(n-1) in double,
// linear interpolation with the float difference promoted to double, between the
// order statistics at floor(pos) and ceil(pos).
__device__ __forceinline__ double pct_pos(int n, float q) {
  return __dmul_rn(static_cast<double>(q), static_cast<double>(n - 1));
}
__device__ __forceinline__ float pct_value(double pos, float lo, float hi) {
  const double w = __dsub_rn(pos, floor(pos));
  const float dlt = __fsub_rn(hi, lo);
  return static_cast<float>(__dadd_rn(static_cast<double>(lo), __dmul_rn(static_cast<double>(dlt), w)));
}
// Floats as unsigned words of the same order, and back.
__device__ __forceinline__ uint32_t order_key(float v) {
  const uint32_t u = __float_as_uint(v);
  return (u & 0x80000000u) ? ~u : u | 0x80000000u;
}
__device__ __forceinline__ float key_value(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? k ^ 0x80000000u : ~k);
}

// Statistic per channel of every window, make_stat_from_sums (iqrm.cu:72-91); clears
// the vote counters and the masks.  grid: windows x channels.
__global__ void k_iqrm_stat(const unsigned long long* __restrict__ sums,
                            const uint32_t* __restrict__ win, int64_t nchans, int64_t csub,
                            int mode, int variant, float* __restrict__ xs, int* __restrict__ recv,
                            int* __restrict__ cast_, uint8_t* __restrict__ masks) {
  const int64_t w = blockIdx.x;
  const int64_t i = static_cast<int64_t>(blockIdx.y) * blockDim.x + threadIdx.x;
  if (i < nchans) masks[w * nchans + i] = 0;
  const unsigned W = win[2 * w + 1] - win[2 * w];
  if (i >= csub || W == 0) return;
  const unsigned long long* s1 = sums + w * 2 * csub;
  const unsigned long long* s2 = s1 + csub;
  float x;
  const double mean = __ddiv_rn(static_cast<double>(s1[i]), static_cast<double>(W));
  if (mode == 0) {
    x = static_cast<float>(mean);
  } else {
    const double e2 = __ddiv_rn(static_cast<double>(s2[i]), static_cast<double>(W));
    double var = (variant & 8) ? __fma_rn(-mean, mean, e2) : __dsub_rn(e2, __dmul_rn(mean, mean));
    if (var < 0.0) var = 0.0;
    x = static_cast<float>(sqrt(var));
  }
  xs[w * csub + i] = x;
  recv[w * csub + i] = 0;
  cast_[w * csub + i] = 0;
}

// One block per (window, lag): the lagged differences, their quartiles and the votes
// of this lag.  The six order statistics the percentiles need come from a bisection
// over the 32 bits of the differences' order keys: per bit, the block counts the keys
// below each of the three candidates (warp sums by one reduction instruction, one
// barrier).  Bound by the latency of those 32 rounds (30 us for 4,096 channels, the
// whole decision 42 us); one block per window that sorted every lag's differences in
// turn took 364 us for 8 lags of 4,096 channels and 597 us for 26 lags of 2,048.  Few
// channels take few warps, so that a round's barrier is short.
// Dynamic shared memory: the csub keys.
template <int THREADS>
__global__ void __launch_bounds__(THREADS) k_iqrm_lag(
    const uint32_t* __restrict__ win, int csub, float nsigma, const int32_t* __restrict__ lags,
    int nlags, int variant, const float* __restrict__ xs, int* __restrict__ recv,
    int* __restrict__ cast_, uint8_t* __restrict__ flags) {
  extern __shared__ uint32_t keys[];
  constexpr int kWarpsL = THREADS / 32;
  __shared__ uint32_t part[2][3][kWarpsL];
  const int l = blockIdx.y, w = blockIdx.x;
  if (win[2 * w + 1] == win[2 * w]) return;
  const int lag = lags[l];
  const float* x = xs + static_cast<int64_t>(w) * csub;
  uint8_t* fl = flags + (static_cast<int64_t>(w) * nlags + l) * csub;
  int* rc = recv + static_cast<int64_t>(w) * csub;
  int* cc = cast_ + static_cast<int64_t>(w) * csub;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // Lagged difference with edge clipping, make_diff_with_clipping (iqrm.cu:94-117).
  for (int k = threadIdx.x; k < csub; k += THREADS) {
    float v;
    if (lag < 0) {
      const int cut = csub + lag;
      v = k < cut ? __fsub_rn(x[k], x[k - lag]) : __fsub_rn(x[cut], x[csub - 1]);
    } else {
      v = k < lag ? __fsub_rn(x[lag], x[0]) : __fsub_rn(x[k], x[k - lag]);
    }
    keys[k] = order_key(v);
  }
  __syncthreads();
  // block sums of three counts; two buffers, so that one barrier per call suffices
  int buf = 0;
  auto block_sums = [&](uint32_t (&c)[3]) {
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const uint32_t t = __reduce_add_sync(0xffffffffu, c[j]);
      if (lane == 0) part[buf][j][warp] = t;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 3; ++j)
      c[j] = __reduce_add_sync(0xffffffffu, lane < kWarpsL ? part[buf][j][lane] : 0u);
    buf ^= 1;
  };
  const double pos[3] = {pct_pos(csub, 0.25f), pct_pos(csub, 0.50f), pct_pos(csub, 0.75f)};
  uint32_t rank[3], key[3] = {0u, 0u, 0u};
#pragma unroll
  for (int j = 0; j < 3; ++j) rank[j] = static_cast<uint32_t>(floor(pos[j]));
  for (int bit = 31; bit >= 0; --bit) {
    // the largest t with at most rank keys below it is the key of that rank
    uint32_t c[3] = {0u, 0u, 0u};
    const uint32_t t0 = key[0] | (1u << bit), t1 = key[1] | (1u << bit), t2 = key[2] | (1u << bit);
    for (int k = threadIdx.x; k < csub; k += THREADS) {
      const uint32_t v = keys[k];
      c[0] += v < t0;
      c[1] += v < t1;
      c[2] += v < t2;
    }
    block_sums(c);
    if (c[0] <= rank[0]) key[0] = t0;
    if (c[1] <= rank[1]) key[1] = t1;
    if (c[2] <= rank[2]) key[2] = t2;
  }
  // the next order statistic: the same key again, or the least one above it
  uint32_t c[3] = {0u, 0u, 0u}, up[3] = {~0u, ~0u, ~0u};
  for (int k = threadIdx.x; k < csub; k += THREADS) {
    const uint32_t v = keys[k];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      if (v <= key[j]) ++c[j];
      else up[j] = min(up[j], v);
    }
  }
  block_sums(c);
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const uint32_t t = __reduce_min_sync(0xffffffffu, up[j]);
    if (lane == 0) part[buf][j][warp] = t;
  }
  __syncthreads();
  float pct[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const uint32_t above = __reduce_min_sync(0xffffffffu, lane < kWarpsL ? part[buf][j][lane] : ~0u);
    const bool next = ceil(pos[j]) > floor(pos[j]) && c[j] < rank[j] + 2u;
    pct[j] = pct_value(pos[j], key_value(key[j]), key_value(next ? above : key[j]));
  }
  float s;
  if (variant & 4) s = fabsf(__fmul_rn(__fsub_rn(pct[2], pct[0]), __frcp_rn(1.349f)));
  else s = fabsf(__fdiv_rn(__fsub_rn(pct[2], pct[0]), 1.349f));
  const bool skip = !(s > 0.f) || !isfinite(s);
  // flag_and_count_kernel (iqrm.cu:120-151).
  const float med = pct[1], thr = __fmul_rn(nsigma, s);
  for (int i = threadIdx.x; i < csub; i += THREADS) {
    const bool hit = !skip && __fsub_rn(key_value(keys[i]), med) > thr;
    fl[i] = hit ? 1 : 0;
    if (hit) {
      atomicAdd(&rc[i], 1);
      atomicAdd(&cc[iqrm_target(lag, i, csub)], 1);
    }
  }
}

// merge_lags_to_mask_kernel (iqrm.cu:154-185).  grid: windows x channels.
__global__ void k_iqrm_merge(const uint32_t* __restrict__ win, int64_t nchans, int64_t cs, int csub,
                             const int32_t* __restrict__ lags, int nlags,
                             const int* __restrict__ recv, const int* __restrict__ cast_,
                             const uint8_t* __restrict__ flags, uint8_t* __restrict__ masks) {
  const int w = blockIdx.x;
  const int i = blockIdx.y * blockDim.x + threadIdx.x;
  if (i >= csub || win[2 * w + 1] == win[2 * w]) return;
  const int ri = recv[static_cast<int64_t>(w) * csub + i];
  if (ri <= 0) return;
  const int* cc = cast_ + static_cast<int64_t>(w) * csub;
  for (int l = 0; l < nlags; ++l) {
    if (!flags[(static_cast<int64_t>(w) * nlags + l) * csub + i]) continue;
    if (cc[iqrm_target(lags[l], i, csub)] < ri) {
      masks[static_cast<int64_t>(w) * nchans + cs + i] = 1;
      return;
    }
  }
}

// OR of the masks of all windows covering each segment of samples.
__global__ void k_segment_masks(const uint8_t* __restrict__ masks, int nwin,
                                const uint32_t* __restrict__ win, const uint32_t* __restrict__ seg_t0,
                                int nseg, int64_t nchans, uint8_t* __restrict__ segmask) {
  const int s = blockIdx.y;
  const int64_t c = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (c >= nchans || s >= nseg) return;
  const uint32_t a = seg_t0[s];
  uint8_t m = 0;
  for (int w = 0; w < nwin; ++w)
    if (win[2 * w] <= a && a < win[2 * w + 1]) m |= masks[static_cast<int64_t>(w) * nchans + c];
  segmask[static_cast<int64_t>(s) * nchans + c] = m;
}

__device__ __forceinline__ int find_seg(const uint32_t* seg_t0, int nseg, int64_t t) {
  int lo = 0, hi = nseg - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (static_cast<int64_t>(seg_t0[mid]) <= t) lo = mid; else hi = mid - 1;
  }
  return lo;
}

template <typename T>
__global__ void k_apply_masks(T* __restrict__ x, int64_t nsamp, int64_t nchans,
                              const uint8_t* __restrict__ segmask, const uint32_t* __restrict__ seg_t0,
                              int nseg) {
  const int64_t c = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (c >= nchans) return;
  for (int64_t t = blockIdx.y; t < nsamp; t += gridDim.y) {
    const int s = find_seg(seg_t0, nseg, t);
    if (segmask[static_cast<int64_t>(s) * nchans + c]) x[t * nchans + c] = 0;
  }
}

// Zero-DM offset per sample: one warp per sample row, warp-shuffle reduction of
// the sum and count of the non-zero (post-IQRM) values of [cs, ce).
template <typename T>
__global__ void k_zdm_offsets(const T* __restrict__ x, int64_t nsamp, int64_t nchans, int64_t cs,
                              int64_t ce, const uint8_t* __restrict__ segmask,
                              const uint32_t* __restrict__ seg_t0, int nseg,
                              uint32_t* __restrict__ off) {
  const int lane = threadIdx.x & 31;
  const int64_t t = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (t >= nsamp) return;
  const uint8_t* sm = nullptr;
  if (segmask) sm = segmask + static_cast<int64_t>(find_seg(seg_t0, nseg, t)) * nchans;
  unsigned long long s = 0;
  unsigned int n = 0;
  const T* row = x + t * nchans;
  for (int64_t c = cs + lane; c < ce; c += 32) {
    uint64_t v = row[c];
    if (sm && sm[c]) v = 0;
    if (v) { s += v; n += 1; }
  }
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    n += __shfl_xor_sync(0xffffffffu, n, o);
  }
  if (lane == 0) off[t] = n ? static_cast<uint32_t>((s + n - 1) / n) : 0u;
}

// The same for 8- and 16-bit samples, a 32-bit word of channels per lane and load.
// Needs whole, aligned words
// (nchans a multiple of the samples per word); words are read from cs rounded down and
// channels outside [cs, ce) are cleared.  Bound: issue (eleven instructions a word), then
// the latency of a row's loads and of its segment's search, which overlap.  2,048 channels
// x 75,001 samples: 95 us with a byte per lane and load, 60 us with the segment searched
// first, emulated byte compares and minima and 64-bit adds, now 46 us.
template <typename T>
__global__ void __launch_bounds__(256) k_zdm_offsets_w(
    const T* __restrict__ x, int64_t nsamp, int64_t nchans, int64_t cs, int64_t ce,
    const uint8_t* __restrict__ segmask, const uint32_t* __restrict__ seg_t0, int nseg,
    uint32_t* __restrict__ off) {
  constexpr int V = 4 / sizeof(T);
  constexpr int kLoads = 8;  // loads in flight
  const int lane = threadIdx.x & 31;
  const int64_t t = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (t >= nsamp) return;
  const int64_t c0 = cs / V * V;
  const int words = static_cast<int>((ce - c0 + V - 1) / V);
  const uint32_t* row = reinterpret_cast<const uint32_t*>(x + t * nchans + c0);
  const uint8_t* sm = nullptr;
  const int head = static_cast<int>(cs - c0), tail = static_cast<int>(c0 + static_cast<int64_t>(words) * V - ce);
  uint32_t s = 0, n = 0;  // (a lane's 8-bit samples of one row: below 2^32 / 255)
  unsigned long long sum = 0;
  auto take = [&](int i, uint32_t v) {
    if (sm) {
      if constexpr (V == 4) {
        v &= ~(*reinterpret_cast<const uint32_t*>(sm + 4 * i) * 255u);  // mask bytes are 0 or 1
      } else {
        const uint32_t m = *reinterpret_cast<const uint16_t*>(sm + 2 * i);
        v &= ~(__byte_perm(m, 0u, 0x4140) * 65535u);
      }
    }
    if (head | tail) {
      if (i == 0) v &= ~0u << (8 * sizeof(T) * head);
      if (i == words - 1) v &= ~0u >> (8 * sizeof(T) * tail);
    }
    // the top bit of a sample's lane: it is not zero
    if constexpr (V == 4) {
      s = __dp4a(v, 0x01010101u, s);
      n += __popc((((v & 0x7f7f7f7fu) + 0x7f7f7f7fu) | v) & 0x80808080u);
    } else {
      sum += (v & 0xffffu) + (v >> 16);
      n += __popc((((v & 0x7fff7fffu) + 0x7fff7fffu) | v) & 0x80008000u);
    }
  };
  const auto find = [&] { sm = segmask + static_cast<int64_t>(find_seg(seg_t0, nseg, t)) * nchans + c0; };
  int i = 0;
  for (; i + 32 * kLoads <= words; i += 32 * kLoads) {
    uint32_t v[kLoads];
#pragma unroll
    for (int k = 0; k < kLoads; ++k) v[k] = __ldg(row + i + lane + 32 * k);
    if (i == 0 && segmask) find();  // while the first loads are on their way
#pragma unroll
    for (int k = 0; k < kLoads; ++k) take(i + lane + 32 * k, v[k]);
  }
  if (i == 0 && segmask) find();
  for (i += lane; i < words; i += 32) take(i, __ldg(row + i));
  sum += s;
  for (int o = 16; o > 0; o >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
    n += __shfl_xor_sync(0xffffffffu, n, o);
  }
  if (lane == 0) off[t] = n ? static_cast<uint32_t>((sum + n - 1) / n) : 0u;
}

// Range zero-DM subtraction with a float mean (zdm_sat_sub of
// rfimarker.cu:218-225 with alpha 1 and clipping): float(v) - mean, clipped to
// [0, max of T], truncated.
template <typename T>
__device__ __forceinline__ T zdm_float_sub(T v, float mean) {
  float r = __fsub_rn(static_cast<float>(v), mean);
  if (r < 0.0f) r = 0.0f;
  const float vmax = static_cast<float>(Lim<T>::vmax);
  if (r > vmax) r = vmax;
  return static_cast<T>(r);
}

// The value of sample t of channel c after the RFI stages.
template <typename T>
__device__ __forceinline__ T prepared_value(const PrepArgs& a, const T* x, int64_t t, int64_t c) {
  T v = x[t * a.nchans + c];
  if (a.segmask) {
    const int s = find_seg(a.seg_t0, a.nseg, t);
    if (a.segmask[static_cast<int64_t>(s) * a.nchans + c]) v = 0;
  }
  if (a.zdm_off && c >= a.zdm_cs && c < a.zdm_ce) {
    const uint32_t m = a.zdm_off[t];
    v = static_cast<T>(static_cast<uint32_t>(v) > m ? static_cast<uint32_t>(v) - m : 0u);
  }
  if (a.zdm_mean && c >= a.zdm_cs && c < a.zdm_ce) v = zdm_float_sub<T>(v, a.zdm_mean[t]);
  if (a.keep && !a.keep[c]) v = 0;
  return v;
}

// Tile of a layout kernel's block: the grid is one-dimensional with the channel groups
// fastest, so that the blocks running at a time read whole rows of the chunk.
__device__ __forceinline__ int64_t prep_tile(const PrepArgs& a, int64_t c0, int64_t* group) {
  const unsigned groups = (static_cast<unsigned>(a.c1 - c0) + 63u) / 64u;  // 32-bit division
  const unsigned t = blockIdx.x / groups;
  *group = blockIdx.x - t * groups;
  return t;
}

// Fused RFI application and transpose to the channel-major layout.
// Tile: 64 samples x 64 channels, 256 threads.
template <typename T>
__global__ void k_prep(PrepArgs a) {
  __shared__ T tile[64][65];
  const T* x = static_cast<const T*>(a.x);
  int64_t group;
  const int64_t tb = prep_tile(a, a.c0, &group) * 64;
  const int64_t cb = a.c0 + group * 64;
  const int tx = threadIdx.x & 63;   // channel within tile (read phase)
  const int ty = threadIdx.x >> 6;   // 0..3
  const int64_t c = cb + tx;
  for (int r = ty; r < 64; r += 4) {
    const int64_t t = tb + r;
    T v = 0;
    if (t < a.nsamp && c < a.c1) {
      v = prepared_value<T>(a, x, t, c);
    }
    tile[r][tx] = v;
  }
  __syncthreads();
  if (a.out) {
    T* out = static_cast<T*>(a.out);
    // write phase: thread -> (channel row, sample)
    for (int r = ty; r < 64; r += 4) {
      const int64_t cc = cb + r;
      const int64_t t = tb + tx;
      if (cc < a.c1 && t < a.nsamp) {
        const int64_t row = (cc - a.c0) * a.ds + (t % a.ds);
        out[row * a.pitch + t / a.ds] = tile[tx][r];
      }
    }
  }
}

// Folded layout with a float mean per sample to subtract: word s of channel c holds the
// samples s + f * seg, f = 0 .. F-1 (F = 4 of 8 bits, 2 of 16).  Tile: 64 words x 64
// channels, 256 threads.
template <typename T>
__global__ void __launch_bounds__(256) k_prep_fold(PrepArgs a) {
  constexpr int F = 4 / sizeof(T);
  __shared__ uint32_t tile[64][65];  // [channel][word]
  const T* x = static_cast<const T*>(a.x);
  int64_t group;
  const int64_t sb = prep_tile(a, a.c0, &group) * 64;
  const int64_t cb = a.c0 + group * 64;
  const int tx = threadIdx.x & 63, ty = threadIdx.x >> 6;
  const int64_t c = cb + tx;
  for (int r = ty; r < 64; r += 4) {
    uint32_t w = 0;
    if (c < a.c1)
#pragma unroll
      for (int f = 0; f < F; ++f) {
        const int64_t t = sb + r + f * a.seg;
        if (t < a.nsamp) w |= static_cast<uint32_t>(prepared_value<T>(a, x, t, c)) << (8 * sizeof(T) * f);
      }
    tile[tx][r] = w;
  }
  __syncthreads();
  uint32_t* out = static_cast<uint32_t*>(a.out);
  for (int r = ty; r < 64; r += 4)
    if (cb + r < a.c1 && sb + tx < a.nwords) out[(cb + r - a.c0) * a.pitch + sb + tx] = tile[r][tx];
}

// Both layouts without downsampling, with word loads: output word i of channel c holds
// the samples t = WS * i + fs * f, f = 0 .. F-1, of the channel (F = 4 of 8 bits, 2 of
// 16, 1 of 32): WS 1 and fs seg fold the chunk, WS F and fs 1 keep its order.  A thread
// loads four channels (4, 8 or 16 bytes) of the F samples of four words, applies the masks and the
// zero-DM offset to whole words, puts the samples of each channel together by byte
// permutes, and the block stores 64 words of 64 channels through shared memory, which
// each output word passes once.  Channel words are read from c0 & ~3; RAGGED: rows do not
// start on a word of four channels (nchans % 4 or the input's address), channels are
// loaded one by one (2,870 channels x 75,001 samples folded 263 us, 1152 us with the
// segment search and offset per sample of k_prep_fold).  Bound by its loads beside the
// memory (warps wait on them 4.4 cycles per issue, issue is 65 % busy, DRAM moves 4.9
// TB/s): row pointers and counts are set up once per thread, the tile comes from one 32-bit
// division, and nothing is 64-bit per load.  4096 channels x 151,000 samples in time
// order 216 us (5.7 TB/s; 480 us with four loads in flight per thread and 64-bit rows);
// 131,072 samples folded, delays to DM 3000, 480 us (2.4 GB; 690 us with all channels
// written up to the plan's largest delay, 905 with every load and store predicated and
// two-way bank conflicts).  The phase rows of downsampled brute force are laid out by one
// launch, grid y = phase (WS 0: strides times ds, ws taken from the arguments).
struct PrepWords {
  int64_t fs, nwords, pitch;  // nwords: words to store per channel; pitch in words
  int ws;
  int64_t phase_pitch;  // WS 0: output words between phases
};
// Byte masks of four channels as masks of their samples, word v of the four channels.
template <typename T>
__device__ __forceinline__ uint32_t expand_mask(uint32_t m4, int v) {
  if constexpr (sizeof(T) == 1) return m4;
  if constexpr (sizeof(T) == 2) return __byte_perm(m4, 0u, v ? 0x3322 : 0x1100);
  return __byte_perm(m4, 0u, 0x1111 * v);
}
template <typename T, int WS, bool RAGGED>
__global__ void __launch_bounds__(256, RAGGED ? 4 : sizeof(T) == 1 && WS == 1 ? 5 : 6) k_prep_w(PrepArgs a, PrepWords q) {
  constexpr int F = 4 / sizeof(T);   // samples per word
  const int ph = WS == 0 ? static_cast<int>(blockIdx.y) : 0;  // phase: its first sample
  const int ws = WS ? WS : q.ws;
  constexpr int V = sizeof(T);       // 32-bit words per four channels
  // [16 * b + w][word] for channel 4w + b: with 66 words a row, the 16 channel groups and
  // two words that a warp stores at a time fall into 32 banks
  __shared__ uint32_t tile[64][66];
  int64_t group;
  const int64_t sb = prep_tile(a, a.c0 & ~int64_t(3), &group) * 64;
  if (a.limit && ph + ws * sb >= a.limit[group]) return;
  const int64_t cb = (a.c0 & ~int64_t(3)) + group * 64;
  const int w = threadIdx.x & 15, r0 = threadIdx.x >> 4;
  const int64_t c = cb + 4 * w;
  const bool cvalid = c < a.nchans;
  uint32_t keep[V], inrange[V];  // per lane: not a bad channel / zero-DM applies
#pragma unroll
  for (int v = 0; v < V; ++v) {
    keep[v] = ~0u;
    inrange[v] = 0;
  }
  if (cvalid && (a.keep || a.zdm_off)) {
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int64_t ch = c + b;
      if (RAGGED && ch >= a.nchans) break;
      const int v = b * V / 4;  // the word and lane of channel b
      const uint32_t lane = V == 1 ? 0xffu << (8 * b) : V == 2 ? 0xffffu << (16 * (b & 1)) : ~0u;
      if (a.keep && !a.keep[ch]) keep[v] &= ~lane;
      if (a.zdm_off && ch >= a.zdm_cs && ch < a.zdm_ce) inrange[v] |= lane;
    }
  }
  // this thread's words of the tile are r0 + 16k: of each sample slot f, how many of the
  // tile's words have a sample, and the samples.  All of them are on their way before the
  // first mask or offset is looked for (the same input: 124 -> 116 us, and no spills).
  const int64_t step = static_cast<int64_t>(16 * ws) * a.nchans;
  int have[F];
  uint32_t in[4][F][V];
#pragma unroll
  for (int f = 0; f < F; ++f) {
    const int64_t t0 = ph + ws * sb + q.fs * f;
    const T* src = static_cast<const T*>(a.x) + (t0 + ws * r0) * a.nchans + c;
    const int64_t left = a.nsamp - t0;  // words i with ws * i < left
    have[f] = !cvalid || left <= 0 ? 0 : left >= ws * 64 ? 64 : (static_cast<int>(left) + ws - 1) / ws;
    auto load = [&](int k) {
      if constexpr (RAGGED) {
        T e[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) e[b] = c + b < a.nchans ? __ldg(src + k * step + b) : T(0);
#pragma unroll
        for (int v = 0; v < V; ++v) {
          in[k][f][v] = 0;
#pragma unroll
          for (int b = 0; b < F; ++b) in[k][f][v] |= static_cast<uint32_t>(e[F * v + b]) << (8 * sizeof(T) * b);
        }
      } else if constexpr (V == 1) {
        in[k][f][0] = __ldg(reinterpret_cast<const uint32_t*>(src + k * step));
      } else if constexpr (V == 4) {
        const uint4 u = __ldg(reinterpret_cast<const uint4*>(src + k * step));
        in[k][f][0] = u.x;
        in[k][f][1] = u.y;
        in[k][f][2] = u.z;
        in[k][f][3] = u.w;
      } else {
        const uint2 u = __ldg(reinterpret_cast<const uint2*>(src + k * step));
        in[k][f][0] = u.x;
        in[k][f][V - 1] = u.y;
      }
    };
    if (have[f] == 64) {  // (all tiles but a slot's last)
#pragma unroll
      for (int k = 0; k < 4; ++k) load(k);
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
#pragma unroll
        for (int v = 0; v < V; ++v) in[k][f][v] = 0;
        if (r0 + 16 * k < have[f]) load(k);
      }
    }
  }
  if (a.segmask || a.keep) {
#pragma unroll
    for (int f = 0; f < F; ++f) {
      if (!have[f]) continue;
      // the mask of the IQRM segment that holds the tile's rows of this slot
      const int64_t t0 = ph + ws * sb + q.fs * f;
      const auto seg_mask = [&](int sg) {
        const uint8_t* p = a.segmask + static_cast<int64_t>(sg) * a.nchans + c;
        if constexpr (RAGGED) {
          uint32_t m = 0;
#pragma unroll
          for (int b = 0; b < 4; ++b)
            if (c + b < a.nchans && p[b]) m |= 0xffu << (8 * b);
          return ~m;
        }
        return ~__vcmpne4(*reinterpret_cast<const uint32_t*>(p), 0u);
      };
      const int sg = a.segmask ? find_seg(a.seg_t0, a.nseg, t0) : 0;
      if (a.segmask && sg + 1 < a.nseg && static_cast<int64_t>(a.seg_t0[sg + 1]) <= t0 + ws * 63) {
        // rows of several segments: one by one
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (r0 + 16 * k >= have[f]) continue;
          const uint32_t m4 = seg_mask(find_seg(a.seg_t0, a.nseg, t0 + ws * (r0 + 16 * k)));
#pragma unroll
          for (int v = 0; v < V; ++v) in[k][f][v] &= expand_mask<T>(m4, v) & keep[v];
        }
      } else {
        const uint32_t m4 = a.segmask ? seg_mask(sg) : ~0u;
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const uint32_t m = expand_mask<T>(m4, v) & keep[v];
#pragma unroll
          for (int k = 0; k < 4; ++k) in[k][f][v] &= m;
        }
      }
    }
  }
  if (a.zdm_off) {
#pragma unroll
    for (int f = 0; f < F; ++f) {
      const uint32_t* offs = a.zdm_off + (ph + ws * (sb + r0) + q.fs * f);
      uint32_t off[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) off[k] = r0 + 16 * k < have[f] ? __ldg(offs + 16 * k * ws) : 0u;
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const uint32_t u = in[k][f][v];
          in[k][f][v] = V == 1   ? __vsubus4(u, (min(off[k], 255u) * 0x01010101u) & inrange[v])
                        : V == 2 ? __vsubus2(u, (min(off[k], 65535u) * 0x00010001u) & inrange[v])
                                 : u - min(u, off[k] & inrange[v]);
        }
    }
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    uint32_t o[4];
    if constexpr (V == 1) {
      const uint32_t v0 = in[k][0][0], v1 = in[k][1][0], v2 = in[k][F - 2][0], v3 = in[k][F - 1][0];
      const uint32_t lo01 = __byte_perm(v0, v1, 0x5140), hi01 = __byte_perm(v0, v1, 0x7362);
      const uint32_t lo23 = __byte_perm(v2, v3, 0x5140), hi23 = __byte_perm(v2, v3, 0x7362);
      o[0] = __byte_perm(lo01, lo23, 0x5410);
      o[1] = __byte_perm(lo01, lo23, 0x7632);
      o[2] = __byte_perm(hi01, hi23, 0x5410);
      o[3] = __byte_perm(hi01, hi23, 0x7632);
    } else if constexpr (V == 4) {
#pragma unroll
      for (int b = 0; b < 4; ++b) o[b] = in[k][0][b];
    } else {
      o[0] = __byte_perm(in[k][0][0], in[k][1][0], 0x5410);
      o[1] = __byte_perm(in[k][0][0], in[k][1][0], 0x7632);
      o[2] = __byte_perm(in[k][0][V - 1], in[k][1][V - 1], 0x5410);
      o[3] = __byte_perm(in[k][0][V - 1], in[k][1][V - 1], 0x7632);
    }
#pragma unroll
    for (int b = 0; b < 4; ++b) tile[16 * b + w][r0 + 16 * k] = o[b];
  }
  __syncthreads();
  // a warp stores channels row, row + 8, ... of the tile, 64 words each
  const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
  const int words = static_cast<int>(min(q.nwords - sb, static_cast<int64_t>(64)));
  const int ch0 = static_cast<int>(max(a.c0 - cb, static_cast<int64_t>(0)));
  const int ch1 = static_cast<int>(min(a.c1 - cb, static_cast<int64_t>(64)));
  uint32_t* dst = static_cast<uint32_t*>(a.out) + (cb + row - a.c0) * q.pitch + sb + lane;
  if constexpr (WS == 0) dst += ph * q.phase_pitch;
  const uint32_t* from = &tile[16 * (row & 3) + (row >> 2)][lane];
  if (words == 64 && ch0 == 0 && ch1 == 64) {
#pragma unroll
    for (int r = 0; r < 8; ++r, dst += 8 * q.pitch) {
      dst[0] = from[2 * r * 66];
      dst[32] = from[2 * r * 66 + 32];
    }
    return;
  }
  for (int r = 0; r < 8; ++r, dst += 8 * q.pitch) {
    if (row + 8 * r < ch0 || row + 8 * r >= ch1) continue;
    if (lane < words) dst[0] = from[2 * r * 66];
    if (lane + 32 < words) dst[32] = from[2 * r * 66 + 32];
  }
}

// Full-layout copy of the prepared input (parity checks only): all channels.
template <typename T>
__global__ void k_prep_full(PrepArgs a) {
  const T* x = static_cast<const T*>(a.x);
  T* out = static_cast<T*>(a.full_out);
  const int64_t c = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (c >= a.nchans) return;
  for (int64_t t = blockIdx.y; t < a.nsamp; t += gridDim.y) {
    out[t * a.nchans + c] = prepared_value<T>(a, x, t, c);
  }
}

}  // namespace

int64_t binning_lut_entries(int nbits, int ds) {
  if (nbits != 8 && nbits != 16) return 0;
  const int64_t n = static_cast<int64_t>(ds) * (nbits == 8 ? 255 : 65535) + 1;
  return n <= (int64_t(1) << 24) ? n : 0;
}

void launch_binning_lut(void* lut, int nbits, int ds, cudaStream_t st) {
  const int64_t n = binning_lut_entries(nbits, ds);
  if (!n) throw Error{DD_ERR_RUNTIME, "no binning table for these samples"};
  const uint64_t vmax = nbits == 8 ? 255u : 65535u;
  const double smax_full = std::sqrt(static_cast<double>(vmax * static_cast<uint64_t>(ds)));
  const unsigned grid = static_cast<unsigned>((n + 255) / 256);
  if (nbits == 8) k_binning_lut<uint8_t><<<grid, 256, 0, st>>>(static_cast<uint8_t*>(lut), n, smax_full);
  else k_binning_lut<uint16_t><<<grid, 256, 0, st>>>(static_cast<uint16_t*>(lut), n, smax_full);
  DD_LAUNCHED();
}

void launch_time_binning(const void* in, void* out, int nbits, int64_t ndata, int64_t nchans,
                         int ds, const void* lut, cudaStream_t st) {
  const int64_t nout = (ndata + ds - 1) / ds;
  if (lut && (nbits == 8 || nbits == 16)) {
    // the widest word that every row starts on
    const auto starts = [&](int64_t bytes) {
      return nchans * (nbits / 8) % bytes == 0 && reinterpret_cast<uintptr_t>(in) % bytes == 0 &&
             reinterpret_cast<uintptr_t>(out) % bytes == 0;
    };
    if (nbits == 16 && starts(4)) launch_time_binning_lut<uint16_t, uint32_t>(in, out, ndata, nchans, ds, nout, lut, st);
    else if (nbits == 16) launch_time_binning_lut<uint16_t, uint16_t>(in, out, ndata, nchans, ds, nout, lut, st);
    else if (starts(4)) launch_time_binning_lut<uint8_t, uint32_t>(in, out, ndata, nchans, ds, nout, lut, st);
    else if (starts(2)) launch_time_binning_lut<uint8_t, uint16_t>(in, out, ndata, nchans, ds, nout, lut, st);
    else launch_time_binning_lut<uint8_t, uint8_t>(in, out, ndata, nchans, ds, nout, lut, st);
    return;
  }
  const dim3 grid(static_cast<unsigned>((nchans + 255) / 256),
                  static_cast<unsigned>(std::min<int64_t>(nout, 65535)));
  const uint64_t vmax = nbits == 8 ? 255u : nbits == 16 ? 65535u : 4294967295u;
  const double smax_full = std::sqrt(static_cast<double>(vmax * static_cast<uint64_t>(ds)));
  switch (nbits) {
    case 8: k_time_binning<uint8_t><<<grid, 256, 0, st>>>(static_cast<const uint8_t*>(in), static_cast<uint8_t*>(out), nchans, ndata, ds, nout, smax_full); break;
    case 16: k_time_binning<uint16_t><<<grid, 256, 0, st>>>(static_cast<const uint16_t*>(in), static_cast<uint16_t*>(out), nchans, ndata, ds, nout, smax_full); break;
    default: k_time_binning<uint32_t><<<grid, 256, 0, st>>>(static_cast<const uint32_t*>(in), static_cast<uint32_t*>(out), nchans, ndata, ds, nout, smax_full); break;
  }
  DD_LAUNCHED();
}

void launch_iqrm_stats(const void* x, int nbits, int64_t nsamp, int64_t nchans, int64_t cs,
                       int64_t csub, const uint32_t* d_win, int nwin, unsigned long long* d_sums,
                       cudaStream_t st) {
  DD_CUDA_TRY(cudaMemsetAsync(d_sums, 0, sizeof(unsigned long long) * 2 * csub * nwin, st));
  // chunks of at most 1024 samples (32-bit partial sums), fewer where the grid would
  // hold less than eight blocks per SM: a thread reads its channels row by row, so the
  // bytes in flight grow with the blocks
  const int threads = nbits == 32 ? 256 : 128;
  const bool u8w = nbits == 8 && nchans % 4 == 0 && reinterpret_cast<uintptr_t>(x) % 4 == 0;
  const bool u16w = nbits == 16 && nchans % 2 == 0 && reinterpret_cast<uintptr_t>(x) % 4 == 0;
  const int64_t per = u8w ? 4 : u16w ? 2 : 1;
  const int64_t cols = (csub + (cs % per) + per - 1) / per;
  const int64_t gx = (cols + threads - 1) / threads;
  int64_t chunk = 1024;
  while (chunk > 64 && gx * ((nsamp + chunk - 1) / chunk) < 148 * 8) chunk /= 2;
  // windows that start less than 64 samples apart are read one by one (240 channels, 100
  // samples, windows of 32 every 2: 184 us with runs of two samples, 82 by one block per
  // window before that, now 38; windows of 400 every 200 are better read together, 114 us
  // against 172 apart)
  const bool apart = nsamp < 64 * static_cast<int64_t>(nwin) && nwin <= 65535;
  const dim3 grid(static_cast<unsigned>(gx), static_cast<unsigned>((nsamp + chunk - 1) / chunk), apart ? nwin : 1);
  if (u8w)
    k_iqrm_stats_u8w<<<grid, threads, 0, st>>>(static_cast<const uint8_t*>(x), nsamp, nchans, cs, csub, d_win, nwin, chunk, d_sums);
  else if (u16w)
    k_iqrm_stats_u16w<<<grid, threads, 0, st>>>(static_cast<const uint16_t*>(x), nsamp, nchans, cs, csub, d_win, nwin, chunk, d_sums);
  else if (nbits == 8)
    k_iqrm_stats<uint8_t><<<grid, threads, 0, st>>>(static_cast<const uint8_t*>(x), nsamp, nchans, cs, csub, d_win, nwin, chunk, d_sums);
  else if (nbits == 16)
    k_iqrm_stats<uint16_t><<<grid, threads, 0, st>>>(static_cast<const uint16_t*>(x), nsamp, nchans, cs, csub, d_win, nwin, chunk, d_sums);
  else
    k_iqrm_stats<uint32_t><<<grid, threads, 0, st>>>(static_cast<const uint32_t*>(x), nsamp, nchans, cs, csub, d_win, nwin, chunk, d_sums);
  DD_LAUNCHED();
}

size_t iqrm_scratch_bytes(int nwin, int64_t csub, int nlags) {
  return static_cast<size_t>(nwin) * csub * (4 + 4 + 4 + nlags) + 256;
}

// k_iqrm_lag holds one window's csub differences in shared memory.  Bands are limited to
// the largest power of two of words that a block's opt-in shared memory holds (32,768
// channels on sm_100), with room for the kernel's own.
void check_iqrm_channels(int64_t csub) {
  int dev = 0, optin = 0;
  DD_CUDA_TRY(cudaGetDevice(&dev));
  DD_CUDA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  int64_t most = 1;
  while (2 * most * static_cast<int64_t>(sizeof(uint32_t)) <= optin) most *= 2;
  if (csub > most) {
    char msg[200];
    std::snprintf(msg, sizeof(msg),
                  "IQRM over %lld channels: a window's differences are held in a block's shared memory "
                  "(%d bytes), at most %lld channels",
                  static_cast<long long>(csub), optin, static_cast<long long>(most));
    throw Error{DD_ERR_INVALID, msg};
  }
}

void launch_iqrm_decide(const unsigned long long* d_sums, int nwin, const uint32_t* d_win,
                        int64_t nchans, int64_t cs, int64_t csub, int mode, float nsigma,
                        const int32_t* d_lags, int nlags, int variant, void* scratch,
                        uint8_t* d_masks, cudaStream_t st) {
  // scratch (iqrm_scratch_bytes): statistics, vote counters, flags
  char* p = static_cast<char*>(scratch);
  float* xs = reinterpret_cast<float*>(p); p += sizeof(float) * nwin * csub;
  int* recv = reinterpret_cast<int*>(p); p += sizeof(int) * nwin * csub;
  int* cast_ = reinterpret_cast<int*>(p); p += sizeof(int) * nwin * csub;
  uint8_t* flags = reinterpret_cast<uint8_t*>(p);
  check_iqrm_channels(csub);
  const int n = static_cast<int>(csub);
  const dim3 all(static_cast<unsigned>(nwin), static_cast<unsigned>((nchans + 255) / 256));
  k_iqrm_stat<<<all, 256, 0, st>>>(d_sums, d_win, nchans, csub, mode, variant, xs, recv, cast_, d_masks);
  DD_LAUNCHED();
  const auto lag = [&](auto kernel, int threads) {
    const size_t smem = sizeof(uint32_t) * csub;
    allow_dynamic_smem(kernel, smem);
    kernel<<<dim3(static_cast<unsigned>(nwin), static_cast<unsigned>(nlags)), threads, smem, st>>>(
        d_win, n, nsigma, d_lags, nlags, variant, xs, recv, cast_, flags);
    DD_LAUNCHED();
  };
  if (csub <= 32) lag(k_iqrm_lag<32>, 32);
  else if (csub <= 128) lag(k_iqrm_lag<128>, 128);
  else lag(k_iqrm_lag<512>, 512);
  const dim3 band(static_cast<unsigned>(nwin), static_cast<unsigned>((csub + 255) / 256));
  k_iqrm_merge<<<band, 256, 0, st>>>(d_win, nchans, cs, n, d_lags, nlags, recv, cast_, flags, d_masks);
  DD_LAUNCHED();
}

void launch_segment_masks(const uint8_t* d_masks, int nwin, const uint32_t* d_win,
                          const uint32_t* d_seg_t0, int nseg, int64_t nchans, uint8_t* d_segmask,
                          cudaStream_t st) {
  dim3 grid(static_cast<unsigned>((nchans + 255) / 256), static_cast<unsigned>(nseg));
  k_segment_masks<<<grid, 256, 0, st>>>(d_masks, nwin, d_win, d_seg_t0, nseg, nchans, d_segmask);
  DD_LAUNCHED();
}

void launch_apply_masks_inplace(void* x, int nbits, int64_t nsamp, int64_t nchans,
                                const uint8_t* d_segmask, const uint32_t* d_seg_t0, int nseg,
                                cudaStream_t st) {
  dim3 grid(static_cast<unsigned>((nchans + 255) / 256), static_cast<unsigned>(nsamp < 8192 ? nsamp : 8192));
  switch (nbits) {
    case 8: k_apply_masks<uint8_t><<<grid, 256, 0, st>>>(static_cast<uint8_t*>(x), nsamp, nchans, d_segmask, d_seg_t0, nseg); break;
    case 16: k_apply_masks<uint16_t><<<grid, 256, 0, st>>>(static_cast<uint16_t*>(x), nsamp, nchans, d_segmask, d_seg_t0, nseg); break;
    default: k_apply_masks<uint32_t><<<grid, 256, 0, st>>>(static_cast<uint32_t*>(x), nsamp, nchans, d_segmask, d_seg_t0, nseg); break;
  }
  DD_LAUNCHED();
}

void launch_zdm_offsets(const void* x, int nbits, int64_t nsamp, int64_t nchans, int64_t cs,
                        int64_t ce_excl, const uint8_t* d_segmask, const uint32_t* d_seg_t0,
                        int nseg, uint32_t* d_off, cudaStream_t st) {
  const unsigned blocks = static_cast<unsigned>((nsamp + 7) / 8);
  if (nbits <= 16 && ce_excl > cs && nchans % (32 / nbits) == 0 && reinterpret_cast<uintptr_t>(x) % 4 == 0 &&
      (!d_segmask || reinterpret_cast<uintptr_t>(d_segmask) % 4 == 0)) {
    if (nbits == 8)
      k_zdm_offsets_w<uint8_t><<<blocks, 256, 0, st>>>(static_cast<const uint8_t*>(x), nsamp, nchans, cs, ce_excl, d_segmask, d_seg_t0, nseg, d_off);
    else
      k_zdm_offsets_w<uint16_t><<<blocks, 256, 0, st>>>(static_cast<const uint16_t*>(x), nsamp, nchans, cs, ce_excl, d_segmask, d_seg_t0, nseg, d_off);
    DD_LAUNCHED();
    return;
  }
  switch (nbits) {
    case 8: k_zdm_offsets<uint8_t><<<blocks, 256, 0, st>>>(static_cast<const uint8_t*>(x), nsamp, nchans, cs, ce_excl, d_segmask, d_seg_t0, nseg, d_off); break;
    case 16: k_zdm_offsets<uint16_t><<<blocks, 256, 0, st>>>(static_cast<const uint16_t*>(x), nsamp, nchans, cs, ce_excl, d_segmask, d_seg_t0, nseg, d_off); break;
    default: k_zdm_offsets<uint32_t><<<blocks, 256, 0, st>>>(static_cast<const uint32_t*>(x), nsamp, nchans, cs, ce_excl, d_segmask, d_seg_t0, nseg, d_off); break;
  }
  DD_LAUNCHED();
}

void launch_prep(const PrepArgs& a, cudaStream_t st) {
  const auto blocks = [&](int64_t tiles, int64_t c0) {
    const int64_t n = tiles * ((a.c1 - c0 + 63) / 64);
    if (n >= (int64_t(1) << 31)) throw Error{DD_ERR_INVALID, "chunk too large for the layout kernel"};
    return static_cast<unsigned>(n);
  };
  // the word-wise kernel applies integer zero-DM offsets only
  const int F = 32 / a.nbits;
  const auto run = [&](auto kernel, auto kernel_ragged, dim3 grid, const PrepWords& q, bool r) {
    if (r) kernel_ragged<<<grid, 256, 0, st>>>(a, q);
    else kernel<<<grid, 256, 0, st>>>(a, q);
    DD_LAUNCHED();
  };
  const bool wide = a.out && !a.zdm_mean;
  const bool ragged = a.nchans % 4 != 0 || reinterpret_cast<uintptr_t>(a.x) % (a.nbits / 2) != 0;
  if (wide && a.nbits <= 16 && a.ds > 1 && a.ds <= 16 && a.pitch % F == 0 && reinterpret_cast<uintptr_t>(a.out) % 4 == 0) {
    // (of phase 0; where a later one has a word less, its last one is zero)
    const int64_t words = ((a.nsamp + a.ds - 1) / a.ds + F - 1) / F;
    const PrepWords q{a.ds, words, a.ds * (a.pitch / F), F * a.ds, a.pitch / F};
    const dim3 grid(blocks((words + 63) / 64, a.c0 & ~int64_t(3)), static_cast<unsigned>(a.ds));
    if (a.nbits == 8) run(k_prep_w<uint8_t, 0, false>, k_prep_w<uint8_t, 0, true>, grid, q, ragged);
    else run(k_prep_w<uint16_t, 0, false>, k_prep_w<uint16_t, 0, true>, grid, q, ragged);
  } else if (wide && (a.fold > 1 || (a.ds == 1 && a.pitch % F == 0 && reinterpret_cast<uintptr_t>(a.out) % 4 == 0))) {
    const PrepWords q = a.fold > 1 ? PrepWords{a.seg, a.nwords, a.pitch, 1, 0}
                                   : PrepWords{1, (a.nsamp + F - 1) / F, a.pitch / F, F, 0};
    const dim3 grid(blocks((q.nwords + 63) / 64, a.c0 & ~int64_t(3)));
    if (a.nbits == 32) run(k_prep_w<uint32_t, 1, false>, k_prep_w<uint32_t, 1, true>, grid, q, ragged);
    else if (a.nbits == 8 && a.fold > 1) run(k_prep_w<uint8_t, 1, false>, k_prep_w<uint8_t, 1, true>, grid, q, ragged);
    else if (a.nbits == 8) run(k_prep_w<uint8_t, 4, false>, k_prep_w<uint8_t, 4, true>, grid, q, ragged);
    else if (a.fold > 1) run(k_prep_w<uint16_t, 1, false>, k_prep_w<uint16_t, 1, true>, grid, q, ragged);
    else run(k_prep_w<uint16_t, 2, false>, k_prep_w<uint16_t, 2, true>, grid, q, ragged);
  } else if (a.out && a.fold > 1) {
    const unsigned grid = blocks((a.nwords + 63) / 64, a.c0);
    if (a.nbits == 8) k_prep_fold<uint8_t><<<grid, 256, 0, st>>>(a);
    else k_prep_fold<uint16_t><<<grid, 256, 0, st>>>(a);
    DD_LAUNCHED();
  } else if (a.out) {
    const unsigned grid = blocks((a.nsamp + 63) / 64, a.c0);
    switch (a.nbits) {
      case 8: k_prep<uint8_t><<<grid, 256, 0, st>>>(a); break;
      case 16: k_prep<uint16_t><<<grid, 256, 0, st>>>(a); break;
      default: k_prep<uint32_t><<<grid, 256, 0, st>>>(a); break;
    }
    DD_LAUNCHED();
  }
  if (a.full_out) {
    dim3 grid(static_cast<unsigned>((a.nchans + 255) / 256), static_cast<unsigned>(a.nsamp < 8192 ? a.nsamp : 8192));
    switch (a.nbits) {
      case 8: k_prep_full<uint8_t><<<grid, 256, 0, st>>>(a); break;
      case 16: k_prep_full<uint16_t><<<grid, 256, 0, st>>>(a); break;
      default: k_prep_full<uint32_t><<<grid, 256, 0, st>>>(a); break;
    }
    DD_LAUNCHED();
  }
}

}  // namespace dd
