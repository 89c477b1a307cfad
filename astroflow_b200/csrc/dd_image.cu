// DM-time images on the GPU: the image step the reference runs on the host with
// OpenCV after every GPU call (include/data.h:620-727, preprocess_typed_
// dedisperseddata_with_slicing) and after the CPU path (data.h:299-369):
//
//   slice of columns -> float -> resize to target x target
//   (INTER_AREA when both dimensions exceed the target, else INTER_LANCZOS4)
//   -> min-max normalise to uint8 -> gray to RGB -> COLORMAP_VIRIDIS
//
// Resampling (both separable: a horizontal pass over every source row the
// output row needs, then a vertical combination), with the rounding of OpenCV's
// float path reproduced operation by operation (each product and each sum
// rounded to float, no fused multiply-add):
//   * area, general scale: each output pixel is the overlap-weighted mean of the
//     source pixels its cell covers (weight = overlap / cell width, overlaps
//     below 1e-3 of a pixel dropped, the last cell clipped to the source);
//     horizontal sums in increasing source column, vertical sums in increasing
//     source row;
//   * area, integer scales (both dimensions multiples of the target): the plain
//     block mean, row sums added row by row, times 1/area;
//   * Lanczos-4: taps at floor(f) - 3 .. floor(f) + 4 of f = (d + 0.5) * scale -
//     0.5 (indices clamped to the source), weights sin(pi x) sin(pi x / 4) /
//     (pi^2 x^2 / 4) at the tap distances, evaluated in double through the
//     angle-addition form, rounded to float and normalised by the float
//     reciprocal of their float sum; horizontal taps summed first to last,
//     vertical taps last to first.
// The weight tables are built on the host in double; the GPU only applies them.
// Normalisation: scale = 255 / (max - min) in double (0 when the image is flat),
// shift = -min * scale, u8 = round-half-even(fmaf(x, (float)scale,
// (float)shift)) clamped to [0, 255]; the color map is a 256-entry BGR table
// supplied by the caller.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>

#include "dd_internal.h"

namespace dd {
namespace {

constexpr int kImgThreads = 256;
constexpr int kStageFloats = 12288;  // source row staged in shared memory up to this width
constexpr double kPi = 3.14159265358979323846;

enum AxisMethod { kAreaGeneral = 0, kAreaInteger = 1, kLanczos = 2 };

// One axis (source size -> target size) as CSR lists of (source index, weight)
// per output index.  Lanczos lists have 8 taps; integer area lists hold the
// block's first index only (the block length is the scale).
struct AxisTab {
  std::vector<int32_t> off, idx;
  std::vector<float> w;
};

AxisTab area_table(int64_t ssize, int dsize) {
  AxisTab t;
  const double scale = static_cast<double>(ssize) / dsize;
  t.off.push_back(0);
  for (int d = 0; d < dsize; ++d) {
    const double f1 = d * scale, f2 = f1 + scale;
    const double cell = std::min(scale, static_cast<double>(ssize) - f1);
    int64_t s1 = static_cast<int64_t>(std::ceil(f1)), s2 = static_cast<int64_t>(std::floor(f2));
    s2 = std::min<int64_t>(s2, ssize - 1);
    s1 = std::min<int64_t>(s1, ssize - 1);
    if (static_cast<double>(s1) - f1 > 1e-3) {
      t.idx.push_back(static_cast<int32_t>(s1 - 1));
      t.w.push_back(static_cast<float>((static_cast<double>(s1) - f1) / cell));
    }
    for (int64_t s = s1; s < s2; ++s) {
      t.idx.push_back(static_cast<int32_t>(s));
      t.w.push_back(static_cast<float>(1.0 / cell));
    }
    if (f2 - static_cast<double>(s2) > 1e-3) {
      t.idx.push_back(static_cast<int32_t>(s2));
      t.w.push_back(static_cast<float>(std::min(std::min(f2 - static_cast<double>(s2), 1.0), cell) / cell));
    }
    t.off.push_back(static_cast<int32_t>(t.idx.size()));
  }
  return t;
}

AxisTab integer_area_table(int64_t ssize, int dsize) {
  AxisTab t;
  const int64_t k = ssize / dsize;
  for (int d = 0; d <= dsize; ++d) t.off.push_back(d);
  for (int d = 0; d < dsize; ++d) {
    t.idx.push_back(static_cast<int32_t>(d * k));
    t.w.push_back(0.0f);
  }
  return t;
}

// Lanczos-4 weights of the 8 taps for fractional position x in (0, 1).
void lanczos4_weights(float x, float* out) {
  if (x < FLT_EPSILON) {
    for (int i = 0; i < 8; ++i) out[i] = 0.0f;
    out[3] = 1.0f;
    return;
  }
  // sin(pi x_i / 4) for x_i = x + 3 - i rotates by 45 degrees from tap to tap;
  // sin(pi x_i) alternates in sign and cancels in the normalisation.
  const double r = std::sqrt(0.5);
  const double rot[8][2] = {{1, 0}, {-r, -r}, {0, 1}, {r, -r}, {-1, 0}, {r, r}, {0, -1}, {-r, r}};
  const double a0 = -(static_cast<double>(x) + 3) * kPi * 0.25;
  const double s0 = std::sin(a0), c0 = std::cos(a0);
  volatile float sum = 0.0f;
  for (int i = 0; i < 8; ++i) {
    const double a = -(static_cast<double>(x) + 3 - i) * kPi * 0.25;
    out[i] = static_cast<float>((rot[i][0] * s0 + rot[i][1] * c0) / (a * a));
    sum = sum + out[i];
  }
  volatile float inv = 1.0f / sum;
  for (int i = 0; i < 8; ++i) {
    volatile float v = out[i] * inv;
    out[i] = v;
  }
}

AxisTab lanczos_table(int64_t ssize, int dsize) {
  AxisTab t;
  const double scale = static_cast<double>(ssize) / dsize;
  for (int d = 0; d < dsize; ++d) {
    const float f = static_cast<float>((d + 0.5) * scale - 0.5);
    const int64_t s = static_cast<int64_t>(std::floor(f));
    volatile float frac = f - static_cast<float>(s);
    float w[8];
    lanczos4_weights(frac, w);
    t.off.push_back(8 * d);
    for (int i = 0; i < 8; ++i) {
      t.idx.push_back(static_cast<int32_t>(std::min(std::max<int64_t>(s - 3 + i, 0), ssize - 1)));
      t.w.push_back(w[i]);
    }
  }
  t.off.push_back(8 * dsize);
  return t;
}

struct ImgLaunch {
  const void* src;      // [rows][pitch] uint32 or uint64
  int64_t pitch;        // elements between rows
  int elem;             // 4 or 8
  int64_t rows, cols;   // slice size
  const int64_t* col0;  // per slice of the group: first column
  int method;
  int target;
  const int32_t* hoff; const int32_t* hidx; const float* hw;
  // general area, horizontal: per output column its first source column, source
  // count and weights (first, interior, last); the interior ones are all equal
  const int32_t* ha_i0; const int32_t* ha_n; const float4* ha_w;
  const int32_t* voff; const int32_t* vidx; const float* vw;
  int ky, kx;           // integer area: block size
  float inv_area;
  float* out;           // [slice][target][target]
  const int* out_slot;  // per slice of the group: its index among the call's slices
  int by_slot;          // `out` is indexed by that (else by position in the launch)
};

__device__ __forceinline__ float to_float(const void* src, int elem, int64_t i) {
  if (elem == 8) return __ull2float_rn(static_cast<const unsigned long long*>(src)[i]);
  return __uint2float_rn(static_cast<const uint32_t*>(src)[i]);
}

// ---------------------------------------------------------------- two-pass resize
// Horizontal pass: every source row of a slice once into `target` floats, then a
// vertical pass over those.  A warp owns 32 output columns (one per lane) and walks down
// the rows, whose pieces (the source columns these outputs need, 2.6 KB at 20 columns
// per output) come through a ring of four asynchronous copies of its own, so that nothing
// is synchronised beyond the warp.  Bound by the shared loads of the sequential sums (lanes
// start 20 words apart: four-way bank conflicts) close to the reads of the sums.
// 3,001 rows x 2^18 columns in 26 slices, whole image step: 0.77 ms, the horizontal
// passes at 5.2 TB/s of sums; 1.28 ms with a block per output row that staged each of
// its source rows between two barriers and read the rows at cell edges twice.
struct HLaunch {
  const char* src;       // element 0 of the DM-time rows
  const char* end;       // past their last element
  int64_t pitch;         // elements between rows
  int64_t rows;          // rows of the pass
  const int32_t* row;    // Lanczos: their source rows (nullptr: all of them, in order)
  int target, rows_per_block, win_bytes;
  const int64_t* col0;   // per slice: first column
  const int32_t* seg0;   // per 32 output columns: first source column and their number
  const int32_t* segn;
  const int32_t* hidx; const float* hw;                          // Lanczos, integer area
  const int32_t* ha_i0; const int32_t* ha_n; const float4* ha_w; // general area
  int kx;
  float* out;            // [slice][rows][target]
};
constexpr int kRing = 4;
constexpr int kRingMaxBytes = 6144;

__device__ __forceinline__ float elem_float(uint32_t v) { return __uint2float_rn(v); }
__device__ __forceinline__ float elem_float(unsigned long long v) { return __ull2float_rn(v); }

template <int METHOD, typename E>
__global__ void __launch_bounds__(kImgThreads) k_hresize(HLaunch L) {
  extern __shared__ __align__(16) char ring[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int seg = blockIdx.y, slice = blockIdx.z;
  char* slots = ring + static_cast<size_t>(warp) * kRing * L.win_bytes;
  const int first = L.seg0[seg], count = L.segn[seg];
  const int dx = min(seg * 32 + lane, L.target - 1);
  const int64_t r0 = static_cast<int64_t>(blockIdx.x) * L.rows_per_block + warp;
  const int64_t r1 = min(L.rows, static_cast<int64_t>(blockIdx.x + 1) * L.rows_per_block);
  const char* base = L.src + (L.col0[slice] + first) * static_cast<int64_t>(sizeof(E));
  const int64_t row_bytes = L.pitch * static_cast<int64_t>(sizeof(E));
  auto piece = [&](int64_t r) {
    if (METHOD == kLanczos && L.row) r = __ldg(L.row + r);
    return base + r * row_bytes;
  };
  // copies row r's piece into slot s: whole 16-byte units inside the rows' memory, its
  // first and last elements by plain loads where a unit would leave it
  auto fetch = [&](int64_t r, int s) {
    if (r < r1) {
      const char* p = piece(r);
      const char* e = p + count * static_cast<int64_t>(sizeof(E));
      const char* lo = reinterpret_cast<const char*>(reinterpret_cast<uintptr_t>(p) & ~uintptr_t(15));
      const char* a = lo < L.src ? lo + 16 : lo;
      const char* b = reinterpret_cast<const char*>((reinterpret_cast<uintptr_t>(e) + 15) & ~uintptr_t(15));
      if (b > L.end) b -= 16;
      char* dst = slots + s * L.win_bytes;
      for (const char* q = a + 16 * lane; q < b; q += 16 * 32) {
        const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst + (q - lo)));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(q) : "memory");
      }
      const char* h = p + lane * sizeof(E);  // head: elements below a
      if (h < e && h < a) *reinterpret_cast<E*>(dst + (h - lo)) = *reinterpret_cast<const E*>(h);
      const char* t = (b > p ? b : p) + lane * sizeof(E);  // tail: elements from b on
      if (lane < 4 && t < e) *reinterpret_cast<E*>(dst + (t - lo)) = *reinterpret_cast<const E*>(t);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  // this lane's output column
  int x0 = 0, n = 0;
  float4 w4 = make_float4(0, 0, 0, 0);
  int xi[8];
  float wi[8];
  if constexpr (METHOD == kAreaGeneral) {
    x0 = L.ha_i0[dx] - first;
    n = L.ha_n[dx];
    w4 = L.ha_w[dx];
  } else if constexpr (METHOD == kAreaInteger) {
    x0 = L.hidx[dx] - first;
    n = L.kx;
  } else {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      xi[k] = L.hidx[8 * dx + k] - first;
      wi[k] = L.hw[8 * dx + k];
    }
  }
#pragma unroll
  for (int k = 0; k < kRing - 1; ++k) fetch(r0 + 8 * k, k);
  int s = 0;
  for (int64_t r = r0; r < r1; r += 8) {
    fetch(r + 8 * (kRing - 1), (s + kRing - 1) & (kRing - 1));
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kRing - 1) : "memory");
    __syncwarp();
    const E* row = reinterpret_cast<const E*>(slots + s * L.win_bytes + (reinterpret_cast<uintptr_t>(piece(r)) & 15));
    float h;
    if constexpr (METHOD == kAreaGeneral) {
      // first, interior and last sources, each product and sum rounded to float
      const E* x = row + x0;
      h = __fmul_rn(elem_float(x[0]), w4.x);
#pragma unroll 4
      for (int i = 1; i < n - 1; ++i) h = __fadd_rn(h, __fmul_rn(elem_float(x[i]), w4.y));
      if (n > 1) h = __fadd_rn(h, __fmul_rn(elem_float(x[n - 1]), w4.z));
    } else if constexpr (METHOD == kAreaInteger) {
      const E* x = row + x0;
      h = elem_float(x[0]);
      for (int i = 1; i < n; ++i) h = __fadd_rn(h, elem_float(x[i]));
    } else {
      h = __fmul_rn(elem_float(row[xi[0]]), wi[0]);
#pragma unroll
      for (int k = 1; k < 8; ++k) h = __fadd_rn(h, __fmul_rn(elem_float(row[xi[k]]), wi[k]));
    }
    if (seg * 32 + lane < L.target) L.out[(slice * L.rows + r) * L.target + dx] = h;
    __syncwarp();  // the slot is refilled by the next iteration's copy
    s = (s + 1) & (kRing - 1);
  }
}

// Order keys of floats (as unsigned words) for the extrema.
__device__ __forceinline__ uint32_t float_key(float v) {
  const uint32_t u = __float_as_uint(v);
  return (u & 0x80000000u) ? ~u : u | 0x80000000u;
}
__device__ __forceinline__ float key_float(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? k ^ 0x80000000u : ~k);
}
// Extrema of a block's values into the image's pair of keys (least inverted, largest),
// both of which start at zero.
__device__ __forceinline__ void block_extrema(float mn, float mx, uint2* ext) {
  __shared__ uint32_t s_ext[2];
  if (threadIdx.x < 2) s_ext[threadIdx.x] = 0u;
  __syncthreads();
  const uint32_t a = __reduce_max_sync(0xffffffffu, ~float_key(mn));
  const uint32_t b = __reduce_max_sync(0xffffffffu, float_key(mx));
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&s_ext[0], a);
    atomicMax(&s_ext[1], b);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicMax(&ext->x, s_ext[0]);
    atomicMax(&ext->y, s_ext[1]);
  }
}

// Vertical pass: one block per output row and slice, summing the horizontal results of
// its source rows in the order of k_resize; the extrema of each image on the way.
__global__ void __launch_bounds__(kImgThreads) k_vresize(const float* h, int64_t rows, int target,
                                                         int method, const int32_t* voff,
                                                         const int32_t* vidx, const float* vw, int ky,
                                                         float inv_area, const int* out_slot,
                                                         int by_slot, float* img, uint2* ext) {
  const int dy = blockIdx.x, slice = blockIdx.y;
  const int v0 = voff[dy], v1 = voff[dy + 1];
  const int nv = method == kAreaInteger ? ky : v1 - v0;
  const float* src = h + slice * rows * target;
  float* out = img + (static_cast<int64_t>(by_slot ? out_slot[slice] : slice) * target + dy) * target;
  float mn = FLT_MAX, mx = -FLT_MAX;
  for (int dx = threadIdx.x; dx < target; dx += kImgThreads) {
    float acc = 0.0f;
    for (int j = 0; j < nv; ++j) {
      const int k = method == kLanczos ? v1 - 1 - j : v0 + j;  // Lanczos: last tap first
      const int64_t sy = method == kAreaInteger ? static_cast<int64_t>(vidx[dy]) + j : vidx[k];
      const float v = src[sy * target + dx];
      if (method == kAreaInteger) {
        acc = j == 0 ? v : __fadd_rn(acc, v);
      } else if (method == kLanczos) {
        const float t = __fmul_rn(v, vw[k]);
        acc = j == 0 ? t : __fadd_rn(acc, t);
      } else {
        acc = __fadd_rn(j == 0 ? 0.0f : acc, __fmul_rn(v, vw[k]));
      }
    }
    const float o = method == kAreaInteger ? __fmul_rn(acc, inv_area) : acc;
    out[dx] = o;
    mn = fminf(mn, o);
    mx = fmaxf(mx, o);
  }
  if (ext) block_extrema(mn, mx, ext + out_slot[slice]);
}

// ---------------------------------------------------------------- one-pass resize
// For slices whose pieces do not fit the ring or whose horizontal results would take
// too much memory.  One block per (output row, slice).  Each source row the output row needs is
// brought into shared memory as float (when it fits), then every thread
// resamples its output columns from it.
#ifndef DD_IMG_MINB
#define DD_IMG_MINB 3
#endif
__global__ void __launch_bounds__(kImgThreads, DD_IMG_MINB) k_resize(ImgLaunch L) {
  __shared__ __align__(16) float row[kStageFloats];
  const int dy = blockIdx.x;
  const int s = blockIdx.y;
  const int64_t c0 = L.col0[s];
  const bool staged = L.cols <= kStageFloats;
  constexpr int kMaxPer = 4;  // output columns per thread (target <= 1024)
  float acc[kMaxPer];
  float* out = L.out + (static_cast<int64_t>(L.by_slot ? L.out_slot[s] : s) * L.target + dy) * L.target;
  const int per = (L.target + kImgThreads - 1) / kImgThreads;
  const int v0 = L.voff[dy], v1 = L.voff[dy + 1];
  const int nv = L.method == kAreaInteger ? L.ky : v1 - v0;
  int a_i0[kMaxPer], a_n[kMaxPer];
  float4 a_w[kMaxPer];
  if (L.method == kAreaGeneral) {
    for (int q = 0; q < per && q < kMaxPer; ++q) {
      const int dx = threadIdx.x + q * kImgThreads;
      if (dx >= L.target) break;
      a_i0[q] = L.ha_i0[dx];
      a_n[q] = L.ha_n[dx];
      a_w[q] = L.ha_w[dx];
    }
  }
  for (int j = 0; j < nv; ++j) {
    // taps in summation order: Lanczos vertical taps last to first
    const int k = L.method == kLanczos ? v1 - 1 - j : v0 + j;
    const int64_t sy = L.method == kAreaInteger ? static_cast<int64_t>(L.vidx[dy]) + j : L.vidx[k];
    const int64_t base = sy * L.pitch + c0;
    if (staged) {
      __syncthreads();
      if (L.elem == 4 && (base & 3) == 0) {  // 16-byte loads of four 32-bit sums
        const uint4* src4 = reinterpret_cast<const uint4*>(static_cast<const uint32_t*>(L.src) + base);
        const int64_t n4 = L.cols >> 2;
        for (int64_t i = threadIdx.x; i < n4; i += kImgThreads) {
          const uint4 v = __ldg(src4 + i);
          reinterpret_cast<float4*>(row)[i] = make_float4(__uint2float_rn(v.x), __uint2float_rn(v.y),
                                                          __uint2float_rn(v.z), __uint2float_rn(v.w));
        }
        for (int64_t i = 4 * n4 + threadIdx.x; i < L.cols; i += kImgThreads)
          row[i] = to_float(L.src, L.elem, base + i);
      } else {
        for (int64_t i = threadIdx.x; i < L.cols; i += kImgThreads) row[i] = to_float(L.src, L.elem, base + i);
      }
      __syncthreads();
    }
    for (int q = 0; q < per && q < kMaxPer; ++q) {
      const int dx = threadIdx.x + q * kImgThreads;
      if (dx >= L.target) break;
      float h;
      if (L.method == kAreaInteger) {
        const int64_t sx = L.hidx[dx];
        h = staged ? row[sx] : to_float(L.src, L.elem, base + sx);
        for (int i = 1; i < L.kx; ++i)
          h = __fadd_rn(h, staged ? row[sx + i] : to_float(L.src, L.elem, base + sx + i));
      } else {
        if (L.method == kLanczos) {
          const int h0 = L.hoff[dx], h1 = L.hoff[dx + 1];
          const int sx = L.hidx[h0];
          h = __fmul_rn(staged ? row[sx] : to_float(L.src, L.elem, base + sx), L.hw[h0]);
          for (int e = h0 + 1; e < h1; ++e) {
            const int x = L.hidx[e];
            h = __fadd_rn(h, __fmul_rn(staged ? row[x] : to_float(L.src, L.elem, base + x), L.hw[e]));
          }
        } else {
          // first, interior and last sources, each product and sum rounded to float
          const int x0 = a_i0[q], n = a_n[q];
          const float4 w = a_w[q];
          h = __fmul_rn(staged ? row[x0] : to_float(L.src, L.elem, base + x0), w.x);
          for (int i = 1; i < n - 1; ++i)
            h = __fadd_rn(h, __fmul_rn(staged ? row[x0 + i] : to_float(L.src, L.elem, base + x0 + i), w.y));
          if (n > 1)
            h = __fadd_rn(h, __fmul_rn(staged ? row[x0 + n - 1] : to_float(L.src, L.elem, base + x0 + n - 1), w.z));
        }
      }
      if (L.method == kAreaInteger) {
        acc[q] = j == 0 ? h : __fadd_rn(acc[q], h);
      } else if (L.method == kLanczos) {
        const float t = __fmul_rn(h, L.vw[k]);
        acc[q] = j == 0 ? t : __fadd_rn(acc[q], t);
      } else {
        acc[q] = __fadd_rn(j == 0 ? 0.0f : acc[q], __fmul_rn(h, L.vw[k]));
      }
    }
  }
  for (int q = 0; q < per && q < kMaxPer; ++q) {
    const int dx = threadIdx.x + q * kImgThreads;
    if (dx >= L.target) break;
    out[dx] = L.method == kAreaInteger ? __fmul_rn(acc[q], L.inv_area) : acc[q];
  }
}

// Per image: min and max of the resized floats (one-pass resize).
__global__ void __launch_bounds__(1024) k_minmax(const float* img, int64_t npix, int by_slot, const int* slot, uint2* ext) {
  const float* p = img + static_cast<int64_t>(by_slot ? slot[blockIdx.y] : blockIdx.y) * npix;
  float mn = FLT_MAX, mx = -FLT_MAX;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < npix;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const float v = p[i];
    mn = fminf(mn, v);
    mx = fmaxf(mx, v);
  }
  block_extrema(mn, mx, ext + slot[blockIdx.y]);
}

struct Lut {
  uint8_t bgr[768];
};

// Normalise (the scale and shift of the image's extrema), then color: four pixels per
// thread, twelve bytes (B, G, R each) out as three words; pixel by pixel where the
// pixels of an image are not a multiple of four.
__global__ void __launch_bounds__(256) k_colorize(const float* img, int64_t npix, int by_slot,
                                                  const int* slot, const uint2* ext, Lut lut,
                                                  uint8_t* out) {
  __shared__ uint32_t s_lut[256];
  __shared__ float2 s_ab;
  for (int i = threadIdx.x; i < 256; i += blockDim.x)
    s_lut[i] = lut.bgr[3 * i] | (lut.bgr[3 * i + 1] << 8) | (lut.bgr[3 * i + 2] << 16);
  const int64_t img_i = slot[blockIdx.y];
  if (threadIdx.x == 0) {
    const float mn = key_float(~ext[img_i].x), mx = key_float(ext[img_i].y);
    const double d = static_cast<double>(mx) - static_cast<double>(mn);
    const double scale = d > DBL_EPSILON ? __ddiv_rn(255.0, d) : 0.0;
    const double shift = 0.0 - static_cast<double>(mn) * scale;
    s_ab = make_float2(__double2float_rn(scale), __double2float_rn(shift));
  }
  __syncthreads();
  const float2 k = s_ab;
  auto color = [&](float x) {
    return s_lut[min(max(__float2int_rn(__fmaf_rn(x, k.x, k.y)), 0), 255)];
  };
  const int64_t p = 4 * (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x);
  const float* src = img + (by_slot ? img_i : blockIdx.y) * npix + p;
  uint8_t* o = out + (img_i * npix + p) * 3;
  if (npix % 4 == 0 && reinterpret_cast<uintptr_t>(img) % 16 == 0 && reinterpret_cast<uintptr_t>(out) % 4 == 0) {
    if (p >= npix) return;
    const float4 v = *reinterpret_cast<const float4*>(src);
    const uint32_t c0 = color(v.x), c1 = color(v.y), c2 = color(v.z), c3 = color(v.w);
    uint32_t* w = reinterpret_cast<uint32_t*>(o);
    w[0] = c0 | (c1 << 24);
    w[1] = (c1 >> 8) | (c2 << 16);
    w[2] = (c2 >> 16) | (c3 << 8);
    return;
  }
  for (int q = 0; q < 4 && p + q < npix; ++q) {
    const uint32_t c = color(src[q]);
    o[3 * q] = static_cast<uint8_t>(c);
    o[3 * q + 1] = static_cast<uint8_t>(c >> 8);
    o[3 * q + 2] = static_cast<uint8_t>(c >> 16);
  }
}

// Tables of a call in one device block: filled on the host, copied once.
struct Tables {
  std::vector<char> host;
  char* dev = nullptr;
  template <typename T>
  size_t add(const std::vector<T>& v) {
    const size_t at = (host.size() + 15) & ~size_t(15);
    host.resize(at + std::max<size_t>(v.size() * sizeof(T), 16));
    if (!v.empty()) std::memcpy(host.data() + at, v.data(), v.size() * sizeof(T));
    return at;
  }
  template <typename T>
  const T* at(size_t off) const { return reinterpret_cast<const T*>(dev + off); }
};

// Scratch of the image step comes stream-ordered from a pool of its own per device that
// keeps up to kPoolBytes across calls: the default pool returns its memory at every
// synchronisation, and mapping 27 MB again cost a call more than its kernels.  The pool
// serves all streams and threads; what a call takes is bounded (kHorizontalBytes and the
// float images of those slices).
constexpr uint64_t kPoolBytes = uint64_t(64) << 20;
constexpr int kMaxDevices = 64;
std::mutex g_pool_mutex;
cudaMemPool_t g_pool[kMaxDevices] = {};
cudaMemPool_t image_pool(cudaStream_t st) {
  int dev = 0;
  DD_CUDA_TRY(cudaStreamGetDevice(st, &dev));
  if (dev < 0 || dev >= kMaxDevices) return nullptr;
  std::lock_guard<std::mutex> lock(g_pool_mutex);
  if (!g_pool[dev]) {
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    DD_CUDA_TRY(cudaMemPoolCreate(&pool, &props));
    uint64_t keep = kPoolBytes;
    DD_CUDA_TRY(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    g_pool[dev] = pool;
  }
  return g_pool[dev];
}
void* scratch_alloc(size_t bytes, cudaStream_t st, std::vector<void*>& scratch) {
  void* p = nullptr;
  const cudaMemPool_t pool = image_pool(st);
  bytes = std::max<size_t>(bytes, 16);
  if (pool) DD_CUDA_TRY(cudaMallocFromPoolAsync(&p, bytes, pool, st));
  else DD_CUDA_TRY(cudaMallocAsync(&p, bytes, st));
  scratch.push_back(p);
  return p;
}

// Bytes of horizontal results in flight at most (they stay in L2 between the passes).
constexpr int64_t kHorizontalBytes = int64_t(32) << 20;

template <int METHOD>
void launch_hresize(const HLaunch& L, int elem, dim3 grid, cudaStream_t st) {
  const size_t smem = static_cast<size_t>(8 * kRing) * L.win_bytes;
  if (elem == 4) {
    allow_dynamic_smem(k_hresize<METHOD, uint32_t>, smem);
    k_hresize<METHOD, uint32_t><<<grid, kImgThreads, smem, st>>>(L);
  } else {
    allow_dynamic_smem(k_hresize<METHOD, unsigned long long>, smem);
    k_hresize<METHOD, unsigned long long><<<grid, kImgThreads, smem, st>>>(L);
  }
  DD_LAUNCHED();
}

}  // namespace
}  // namespace dd

using namespace dd;

extern "C" int dd_images(const void* dm_time, int32_t elem_bytes, int64_t nrows, int64_t row_pitch,
                         int32_t nslices, const int64_t* col_start, const int64_t* col_count,
                         int32_t target, const uint8_t* lut_bgr, uint8_t* images, float* resized,
                         void* stream) {
  if (!dm_time || !col_start || !col_count || (!images && !resized) || (images && !lut_bgr)) {
    set_error("NULL argument");
    return DD_ERR_INVALID;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  std::vector<void*> scratch;
  int rc = DD_OK;
  try {
    set_error("");
    if (elem_bytes != 4 && elem_bytes != 8) throw Error{DD_ERR_INVALID, "elem_bytes must be 4 or 8"};
    if (nrows < 1 || nslices < 0 || target < 1 || target > 4 * kImgThreads)
      throw Error{DD_ERR_INVALID, "bad image geometry"};
    if (nslices == 0) return DD_OK;
    scratch.reserve(16);  // (a block is noted as soon as it is allocated)
    for (int32_t i = 0; i < nslices; ++i)
      if (col_count[i] < 1 || col_start[i] < 0 || col_start[i] + col_count[i] > row_pitch)
        throw Error{DD_ERR_INVALID, "slice outside the rows"};
    const int64_t npix = static_cast<int64_t>(target) * target;
    uint2* ext = nullptr;
    if (images) {
      ext = static_cast<uint2*>(scratch_alloc(sizeof(uint2) * nslices, st, scratch));
      DD_CUDA_TRY(cudaMemsetAsync(ext, 0, sizeof(uint2) * nslices, st));
    }
    // slices of equal width share one launch and one pair of tables
    std::map<int64_t, std::vector<int32_t>> by_width;
    for (int32_t i = 0; i < nslices; ++i) by_width[col_count[i]].push_back(i);
    struct Group {
      int64_t cols = 0, n = 0;
      int method = 0, win = 0;
      bool taps = false;  // the horizontal pass makes the vertical taps' rows only, in their order
      size_t c0, slot, hoff, hidx, hw, voff, vidx, vw, i0, nn, w, seg0, segn, vtap = 0;
    };
    std::vector<Group> groups;
    Tables tabs;
    const int nseg = (target + 31) / 32;
    for (const auto& kv : by_width) {
      Group g;
      g.cols = kv.first;
      g.n = static_cast<int64_t>(kv.second.size());
      const bool area = nrows > target && g.cols > target;
      const bool integer = area && nrows % target == 0 && g.cols % target == 0;
      g.method = integer ? kAreaInteger : area ? kAreaGeneral : kLanczos;
      AxisTab h = integer ? integer_area_table(g.cols, target)
                  : area  ? area_table(g.cols, target)
                          : lanczos_table(g.cols, target);
      AxisTab v = integer ? integer_area_table(nrows, target)
                  : area  ? area_table(nrows, target)
                          : lanczos_table(nrows, target);
      std::vector<int64_t> c0;
      std::vector<int> slot;
      for (int32_t i : kv.second) {
        c0.push_back(col_start[i]);
        slot.push_back(i);
      }
      std::vector<int32_t> i0, n;
      std::vector<float4> w;
      if (g.method == kAreaGeneral) {
        i0.resize(target);
        n.resize(target);
        w.resize(target);
        for (int d = 0; d < target; ++d) {
          const int a = h.off[d], b = h.off[d + 1];
          if (b <= a) throw Error{DD_ERR_RUNTIME, "empty area cell"};
          i0[d] = h.idx[a];
          n[d] = b - a;
          const float mid = b - a > 2 ? h.w[a + 1] : h.w[a];
          for (int e = a; e < b; ++e) {
            if (h.idx[e] != h.idx[a] + (e - a) || (e > a && e < b - 1 && h.w[e] != mid))
              throw Error{DD_ERR_RUNTIME, "area table is not a contiguous run"};
          }
          w[d] = make_float4(h.w[a], mid, h.w[b - 1], 0.0f);
        }
      }
      // source columns of every 32 output columns
      const int kx = static_cast<int>(g.cols / target);
      std::vector<int32_t> seg0(nseg), segn(nseg);
      int most = 0;
      for (int sgm = 0; sgm < nseg; ++sgm) {
        int lo = INT32_MAX, hi = 0;
        for (int d = 32 * sgm; d < std::min(target, 32 * sgm + 32); ++d)
          for (int e = h.off[d]; e < h.off[d + 1]; ++e) {
            lo = std::min(lo, h.idx[e]);
            hi = std::max(hi, h.idx[e] + (integer ? kx : 1));
          }
        seg0[sgm] = lo;
        segn[sgm] = hi - lo;
        most = std::max(most, hi - lo);
      }
      g.win = static_cast<int>(std::min<int64_t>((static_cast<int64_t>(most) * elem_bytes + 31) / 16 * 16, 1 << 20));
      g.c0 = tabs.add(c0);
      g.slot = tabs.add(slot);
      g.hoff = tabs.add(h.off);
      g.hidx = tabs.add(h.idx);
      g.hw = tabs.add(h.w);
      g.voff = tabs.add(v.off);
      g.vidx = tabs.add(v.idx);
      g.vw = tabs.add(v.w);
      g.i0 = tabs.add(i0);
      g.nn = tabs.add(n);
      g.w = tabs.add(w);
      // Lanczos reads eight source rows per output row: of many more only those pass (60,000
      // rows to 64 in 20 slices: 667 us with all of them, 93 a row at a time in one pass, now
      // 28; 16,000 rows to 512 in 8 slices 608, 494, 203)
      g.taps = g.method == kLanczos && nrows > 12 * static_cast<int64_t>(target);
      if (g.taps) {
        std::vector<int32_t> order(v.idx.size());
        for (size_t i = 0; i < order.size(); ++i) order[i] = static_cast<int32_t>(i);
        g.vtap = tabs.add(order);
      }
      g.seg0 = tabs.add(seg0);
      g.segn = tabs.add(segn);
      groups.push_back(g);
    }
    tabs.dev = static_cast<char*>(scratch_alloc(tabs.host.size(), st, scratch));
    DD_CUDA_TRY(cudaMemcpyAsync(tabs.dev, tabs.host.data(), tabs.host.size(), cudaMemcpyHostToDevice, st));
    Lut lut;
    if (images) std::memcpy(lut.bgr, lut_bgr, sizeof(lut.bgr));
    float* fimg = nullptr;  // float images of one chunk of slices, unless the caller takes them
    int64_t fslices = 0;
    auto float_images = [&](int64_t n) {
      if (resized) return resized;
      if (n > fslices) {
        fimg = static_cast<float*>(scratch_alloc(static_cast<size_t>(sizeof(float) * npix * n), st, scratch));
        fslices = n;
      }
      return fimg;
    };
    auto colorize = [&](const float* img, const int* slots, int64_t n) {
      if (!images) return;
      k_colorize<<<dim3(static_cast<unsigned>((npix + 1023) / 1024), static_cast<unsigned>(n)), 256, 0, st>>>(
          img, npix, resized ? 1 : 0, slots, ext, lut, images);
      DD_LAUNCHED();
    };
    float* hres = nullptr;
    int64_t hslices = 0;
    for (const Group& g : groups) {
      const float inv_area = g.method == kAreaInteger
                                 ? static_cast<float>(1.0 / (static_cast<double>(g.cols / target) * (nrows / target)))
                                 : 1.0f;
      const int ky = static_cast<int>(nrows / target), kx = static_cast<int>(g.cols / target);
      const int64_t hrows = g.taps ? 8 * target : nrows;
      const int64_t hbytes = hrows * target * static_cast<int64_t>(sizeof(float));  // per slice
      if (g.win <= kRingMaxBytes && hbytes <= kHorizontalBytes && nseg <= 65535) {
        const int64_t per = std::min<int64_t>(std::min<int64_t>(g.n, kHorizontalBytes / hbytes), 65535);
        if (per > hslices) {
          hres = static_cast<float*>(scratch_alloc(static_cast<size_t>(per * hbytes), st, scratch));
          hslices = per;
        }
        // eight rows per warp and turn; fewer rows per block where the grid is small
        int rpb = 128;
        while (rpb > 32 && (hrows + rpb - 1) / rpb * nseg * per < 148 * 4) rpb /= 2;
        for (int64_t s0 = 0; s0 < g.n; s0 += per) {
          const int64_t ns = std::min(per, g.n - s0);
          float* img = float_images(per);
          HLaunch L{};
          L.src = static_cast<const char*>(dm_time);
          L.end = L.src + nrows * row_pitch * elem_bytes;
          L.pitch = row_pitch;
          L.rows = hrows;
          L.row = g.taps ? tabs.at<int32_t>(g.vidx) : nullptr;
          L.target = target;
          L.rows_per_block = rpb;
          L.win_bytes = g.win;
          L.col0 = tabs.at<int64_t>(g.c0) + s0;
          L.seg0 = tabs.at<int32_t>(g.seg0);
          L.segn = tabs.at<int32_t>(g.segn);
          L.hidx = tabs.at<int32_t>(g.hidx);
          L.hw = tabs.at<float>(g.hw);
          L.ha_i0 = tabs.at<int32_t>(g.i0);
          L.ha_n = tabs.at<int32_t>(g.nn);
          L.ha_w = tabs.at<float4>(g.w);
          L.kx = kx;
          L.out = hres;
          const dim3 hg(static_cast<unsigned>((hrows + rpb - 1) / rpb), static_cast<unsigned>(nseg), static_cast<unsigned>(ns));
          if (g.method == kAreaGeneral) launch_hresize<kAreaGeneral>(L, elem_bytes, hg, st);
          else if (g.method == kAreaInteger) launch_hresize<kAreaInteger>(L, elem_bytes, hg, st);
          else launch_hresize<kLanczos>(L, elem_bytes, hg, st);
          k_vresize<<<dim3(static_cast<unsigned>(target), static_cast<unsigned>(ns)), kImgThreads, 0, st>>>(
              hres, hrows, target, g.method, tabs.at<int32_t>(g.voff), tabs.at<int32_t>(g.taps ? g.vtap : g.vidx),
              tabs.at<float>(g.vw), ky, inv_area, tabs.at<int>(g.slot) + s0, resized ? 1 : 0, img, ext);
          DD_LAUNCHED();
          colorize(img, tabs.at<int>(g.slot) + s0, ns);
        }
        continue;
      }
      // (a launch takes the slices as its grid's y: 65535 at most)
      const int64_t step = std::min<int64_t>(std::min<int64_t>(g.n, 65535), std::max<int64_t>(1, kHorizontalBytes / (npix * 4)));
      for (int64_t g0 = 0; g0 < g.n; g0 += step) {
        ImgLaunch L{};
        float* img = float_images(step);
        L.src = dm_time;
        L.pitch = row_pitch;
        L.elem = elem_bytes;
        L.rows = nrows;
        L.cols = g.cols;
        L.col0 = tabs.at<int64_t>(g.c0) + g0;
        L.out_slot = tabs.at<int>(g.slot) + g0;
        L.method = g.method;
        L.target = target;
        L.hoff = tabs.at<int32_t>(g.hoff);
        L.hidx = tabs.at<int32_t>(g.hidx);
        L.hw = tabs.at<float>(g.hw);
        L.voff = tabs.at<int32_t>(g.voff);
        L.vidx = tabs.at<int32_t>(g.vidx);
        L.vw = tabs.at<float>(g.vw);
        L.ha_i0 = tabs.at<int32_t>(g.i0);
        L.ha_n = tabs.at<int32_t>(g.nn);
        L.ha_w = tabs.at<float4>(g.w);
        L.ky = ky;
        L.kx = kx;
        L.inv_area = inv_area;
        L.out = img;
        L.by_slot = resized ? 1 : 0;
        const unsigned ns = static_cast<unsigned>(std::min(g.n - g0, step));
        k_resize<<<dim3(static_cast<unsigned>(target), ns), kImgThreads, 0, st>>>(L);
        DD_LAUNCHED();
        if (images) {
          k_minmax<<<dim3(8, ns), 1024, 0, st>>>(img, npix, L.by_slot, L.out_slot, ext);
          DD_LAUNCHED();
        }
        colorize(img, L.out_slot, ns);
      }
    }
  } catch (const Error& e) {
    set_error(e.msg);
    rc = e.code;
  } catch (const std::exception& e) {
    set_error(e.what());
    rc = DD_ERR_RUNTIME;
  }
  for (void* p : scratch) cudaFreeAsync(p, st);
  return rc;
}
