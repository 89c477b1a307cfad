// Shared-memory staged shift-and-add kernels: the dedispersion sums of
// src/core/dedispered.cu:416-476 (subband stages 1 and 2) and
// include/cpucal.hpp:154-190 (brute force), all of the form
//
//   out[r][t] = sum_i src_i[base + off(r, i) + t],   t in [0, T) of the block's tile.
//
// A block owns kSumRows output rows (eight where coarse trial steps spread them too far,
// sum_kind_rows8), dealt to its warp groups (RB rows each), and T
// consecutive words of them.  Sources are processed in groups of two or four.  The time
// window of each source that the block's rows need,
// [base + min_r off, base + max_r off + T), is brought into shared memory by one
// bulk asynchronous copy (cp.async.bulk, completion counted in bytes on an
// mbarrier); up to `stages` groups are in flight in a ring of buffers.
// The warps take turns as the producer (run_pipeline), each refilling a buffer once
// every warp has released it (an "empty" mbarrier with one arrival per warp).  The
// window bounds and each row's offset inside its window come from descriptors
// precomputed on the host (SumDesc), which the producing warp has loaded ahead (one
// lane per source and row).
//
// Layouts.  Folded chunks (the default where the delays are short against the chunk)
// hold in one 32-bit word samples that lie a segment apart, so every delay is a whole
// number of words and each source word is one aligned shared load; their lanes own
// interleaved words (l, l + 32, ...).  Chunks in time order (short against their
// delays: a beam's pushes) pay one funnel shift of two words per unaligned word; their
// lanes own an odd number of consecutive words (8- and 16-bit samples) or read the
// subband sums' one-sample-shifted twin (sum_u16_twin).  Downsampled brute force reads
// one phase row per delay, 32-bit samples are whole words.  All of these keep a warp's
// shared loads free of bank conflicts.
// 8-bit samples are added two at a time by two-way dot products with the weights
// (1, 2^15) (see dot_lo), 16-bit samples in packed lanes or whole beside their high
// halves.  Outputs leave through shared memory as 16-byte chunks where a lane's words
// are scattered (16-bit stage-1 sums in time order and their twin).  Sums of more
// sources than a 15-bit field holds are added to the output in several flushes.
// A missing source (source count not a multiple of the group) reads a zeroed window.
//
// Every wait on an mbarrier is bounded (about two seconds of SM clock); a wait
// that gives up records an error code in L.err and the block stops summing, and
// the other blocks of the launch stop at their next wait.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

#include "dd_internal.h"

namespace dd {
namespace {

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
constexpr long long kWaitCycles = 4000000000LL;

// ------------------------------------------------------------------ mbarrier helpers
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(count)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Waits for the phase with the given parity to complete; false after ~2 s, or
// as soon as this block (*failed) or any block of the launch (*gerr) has failed.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* failed,
                                          volatile int* gerr) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  for (uint32_t i = 1;; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 255u) == 0) {  // the failure checks read memory: keep them off the wake-up path
      if (*failed || *gerr) return false;
      if (clock64() - t0 > kWaitCycles) return false;
    }
  }
}
// One bulk copy global -> shared, completing `bytes` on `bar`.
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes,
                                          uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}

// 8-bit samples are summed by two-way dot products: dot_lo adds bytes 0 and 1 of a
// word to an accumulator with the weights 1 and 2^15 (dot_hi: bytes 2 and 3), so one
// instruction takes two samples out of the word, puts each into its own field (bits
// 0..14 and 15..31) and adds them.  A field holds kDotSources samples (128 x 255 =
// 32640 < 2^15).  The dot products issue at half rate on the multiply-add pipe (63
// lanes per cycle and SM measured, beside byte permutes at 62 on the integer pipe),
// so a word costs two of them where splitting it by two byte permutes and adding the
// 16-bit lanes took four operations on two pipes.
constexpr int kDotSources = 128;
constexpr uint32_t kDotWeights = 0x80000001u;
__device__ __forceinline__ uint32_t dot_lo(uint32_t w, uint32_t acc) {
  return __dp2a_lo(kDotWeights, w, acc);
}
__device__ __forceinline__ uint32_t dot_hi(uint32_t w, uint32_t acc) {
  return __dp2a_hi(kDotWeights, w, acc);
}
// The two fields as packed 16-bit sums (first sample low): a + (its high field << 15).
__device__ __forceinline__ uint32_t dot_pack(uint32_t a) { return a + (a & 0xffff8000u); }
// acc plus the high half of w, one dot product (a multiply-high issues at half its
// rate: 31 lanes per cycle and SM).
__device__ __forceinline__ uint32_t high_add(uint32_t w, uint32_t acc) {
  return __dp2a_lo(w, 0x0100u, acc);
}

// Per-block view of the sum.  Row r of the block covers launch columns
// [col - skew(r), col - skew(r) + T): stage 1 shifts each row by its delay at the
// subband's top channel (SumLaunch::skew), so that the windows of the block's rows
// nearly coincide; the other sums have no skew.
struct Geo {
  const char* src;     // source 0 (byte address)
  int64_t src_pitch;   // bytes between consecutive sources
  const SumDesc* desc; // descriptor of source 0 for this block's row group
  int64_t base;        // element index added to every offset
  int nsrc, nrows;     // nrows <= 0: nothing to do
  int64_t valid;       // source elements: from here on they are zero (past the chunk)
  char* out;           // row 0, launch column 0 (byte address)
  int64_t out_pitch;   // bytes between output rows
  const int32_t* skew; // per row, or nullptr
  int64_t col;         // first column of the block before skews
  int64_t ncols;       // columns of the launch
};
__device__ __forceinline__ int64_t row_col(const Geo& g, int r) {
  return g.col - (g.skew ? __ldg(g.skew + r) : 0);
}

template <bool PHASES = false, int ROWS = kSumRows>
__device__ __forceinline__ Geo make_geo(const SumLaunch& L, int T, uint3 blk) {
  Geo g;
  const int64_t tile = blk.x;
  g.col = tile * T;
  g.ncols = L.ncols;
  g.skew = nullptr;
  g.valid = L.valid;
  const SumDesc* drow = L.desc + static_cast<int64_t>(blk.y) * L.desc_pitch;
  switch (L.mode) {
    case SumLaunch::kStage1: {
      // rows: nominal DMs j0.. of subband sb; sources: the subband's channels
      const int64_t j0 = static_cast<int64_t>(blk.y) * ROWS;
      const int64_t sb = blk.z;
      const int64_t c0 = sb * L.group;
      g.src = L.src + c0 * L.src_pitch;
      g.desc = drow + c0;
      g.nsrc = static_cast<int>(min(static_cast<int64_t>(L.group), L.nsrc_total - c0));
      g.nrows = static_cast<int>(min(static_cast<int64_t>(ROWS), L.nrows_total - j0));
      g.out = L.out + (j0 * L.nsb_out + sb) * L.out_pitch + L.out_col0 * L.out_elem;
      g.out_pitch = L.nsb_out * L.out_pitch;
      g.skew = L.skew + (static_cast<int64_t>(blk.y) * L.nsb_out + sb) * kSumRows;
      break;
    }
    case SumLaunch::kStage2: {
      // rows: fine DMs of nominal DM j; sources: the subband sums of j
      const int per_nom = (L.group + ROWS - 1) / ROWS;
      const int64_t j = blk.y / per_nom;
      const int64_t m0 = j * L.group + static_cast<int64_t>(blk.y % per_nom) * ROWS;
      const int64_t mend = min((j + 1) * L.group, L.nrows_total);
      g.src = L.src + blk.z * L.plane_bytes + j * L.nsrc_total * L.src_pitch;
      g.desc = drow;
      g.nsrc = static_cast<int>(L.nsrc_total);
      g.nrows = static_cast<int>(max(static_cast<int64_t>(0), min(static_cast<int64_t>(ROWS), mend - m0)));
      g.out = L.out + m0 * L.out_pitch + L.out_col0 * L.out_elem;
      g.out_pitch = L.out_pitch;
      break;
    }
    default: {  // brute force: rows = DMs, sources = channels
      const int64_t m0 = static_cast<int64_t>(blk.y) * ROWS;
      g.src = L.src;
      g.desc = drow;
      g.nsrc = static_cast<int>(L.nsrc_total);
      g.nrows = static_cast<int>(min(static_cast<int64_t>(ROWS), L.nrows_total - m0));
      g.out = L.out + m0 * L.out_pitch + L.out_col0 * L.out_elem;
      g.out_pitch = L.out_pitch;
      if constexpr (PHASES) {
        // slice blk.z: column t is sample start + t * ds of every channel's delayed row
        const int64_t start = static_cast<int64_t>(blk.z) * L.sps;
        g.desc += (start % L.ds) * L.desc_pattern;
        g.base = start / L.ds + g.col;
        g.src_pitch = L.src_pitch;
        g.ncols = min(L.ncols, (L.nin - start + L.ds - 1) / L.ds);
        g.out += static_cast<int64_t>(blk.z) * L.ncols * L.out_elem;
        return g;
      }
      break;
    }
  }
  g.src_pitch = L.src_pitch;
  g.base = L.base + g.col;
  return g;
}

// Shared state of the pipeline.  A stage holds QS sources: two, or four with their
// twins.
struct __align__(16) Pipe {
  uint64_t full[kSumMaxStages];   // completes when a stage's windows have landed
  uint64_t empty[kSumMaxStages];  // completes when all warps released a stage
  // per row: word index and shift (bits) of sample 0 in the window of source i of
  // the stage at [2i], [2i+1]; twin windows (four sources): word indices only
  int row[kSumMaxStages][kSumRows][4];
  uint32_t first[kWarps];      // first source with samples of the chunk, by warp
  int failed;
};
__device__ __forceinline__ int4 row_info(const Pipe& P, int s, int r) {
  return *reinterpret_cast<const int4*>(&P.row[s][r][0]);
}

// The descriptors of one group of QS sources, held by the warp that will stage it:
// lane 16i + r has row r's offset into the windows of sources i and i + 2.
template <int QS>
struct GroupDesc {
  int lo[QS / 2], span[QS / 2], rel[QS / 2];
  __device__ __forceinline__ void load(const Geo& g, int q, int lane) {
    static_assert(kSumRows == 16, "lane = 16 * source + row");
#pragma unroll
    for (int h = 0; h < QS / 2; ++h) {
      const int src = QS * q + (lane >> 4) + 2 * h;
      lo[h] = span[h] = rel[h] = 0;
      if (src < g.nsrc) {
        const SumDesc* d = g.desc + src;
        const int2 v = __ldg(reinterpret_cast<const int2*>(d));
        lo[h] = v.x;
        span[h] = v.y;
        // rows past nrows take offset lo (rel 0): their reads stay in the window
        if ((lane & 15) < g.nrows) rel[h] = __ldg(&d->rel[lane & 15]);
      }
    }
  }
  // the phase rows (downsampled brute force) of the lane's sources
  __device__ __forceinline__ int phase(const Geo& g, int q, int lane) const {
    const int src = QS * q + (lane >> 4);
    if (src >= g.nsrc) return 0;
    return (__ldg(&g.desc[src].phase[(lane >> 3) & 1]) >> (4 * (lane & 7))) & 15;
  }
};

// Stages source pair q in stage s, by all lanes of one warp: lane 16i + r writes row
// r's offsets into the window of source 2q + i, and lane 16i issues that window's
// copy.  The caller has made sure stage s is free.
template <int SB>
__device__ __forceinline__ void produce(const Geo& g, Pipe& P, uint32_t* sw, int ww, int zero_q,
                                        int tile_bytes, const GroupDesc<2>& d, int q, int s, int lane) {
  const int i = lane >> 4, r = lane & 15;
  const int src = 2 * q + i;
  uint32_t nbytes = 0;
  const char* gsrc = nullptr;
  int2 rw = make_int2(zero_q, 0);
  if (src < g.nsrc && g.base + d.lo[0] < g.valid) {
    const int64_t firstb = (g.base + d.lo[0]) * SB;
    const int64_t a0 = firstb & ~int64_t(15);
    const int ob = static_cast<int>(firstb - a0) + d.rel[0] * SB;
    rw = make_int2((2 * s + i) * ww + (ob >> 2), (ob & 3) * 8);
    if (r == 0) {
      const int64_t last = firstb + static_cast<int64_t>(d.span[0]) * SB + tile_bytes + 8;  // + funnel word
      nbytes = static_cast<uint32_t>((last - a0 + 15) & ~int64_t(15));
      gsrc = g.src + static_cast<int64_t>(src) * g.src_pitch + a0;
    }
  }
  *reinterpret_cast<int2*>(&P.row[s][r][2 * i]) = rw;
  const uint32_t total = nbytes + __shfl_xor_sync(0xffffffffu, nbytes, 16);
  __syncwarp();
  if (lane == 0) mbar_arrive_expect_tx(&P.full[s], total);
  __syncwarp();
  if (nbytes) bulk_copy(sw + (2 * s + i) * ww, gsrc, nbytes, &P.full[s]);
}

// The same for downsampled brute force: a source is its channel's ds phase rows (L.ds),
// each staged from the same element on into its own part of the window, and row r reads
// the phase that its delay falls on.
template <int SB>
__device__ __forceinline__ void produce_phases(const SumLaunch& L, const Geo& g, Pipe& P, uint32_t* sw,
                                               int ww, int zero_q, int tile_bytes, const GroupDesc<2>& d,
                                               int phase, int q, int s, int lane) {
  const int i = lane >> 4, r = lane & 15;
  const int src = 2 * q + i;
  uint32_t nbytes = 0;
  const char* gsrc = nullptr;
  int2 rw = make_int2(zero_q, 0);
  if (src < g.nsrc && g.base + d.lo[0] < g.valid) {
    const int64_t firstb = (g.base + d.lo[0]) * SB;
    const int64_t a0 = firstb & ~int64_t(15);
    const int ob = static_cast<int>(firstb - a0) + d.rel[0] * SB;
    rw = make_int2((2 * s + i) * ww + phase * (L.sub_bytes >> 2) + (ob >> 2), (ob & 3) * 8);
    if (r == 0) {
      const int64_t last = firstb + static_cast<int64_t>(d.span[0]) * SB + tile_bytes + 8;
      nbytes = static_cast<uint32_t>((last - a0 + 15) & ~int64_t(15));
      gsrc = g.src + static_cast<int64_t>(src) * g.src_pitch + a0;
    }
  }
  *reinterpret_cast<int2*>(&P.row[s][r][2 * i]) = rw;
  const uint32_t total = (nbytes + __shfl_xor_sync(0xffffffffu, nbytes, 16)) * static_cast<uint32_t>(L.ds);
  __syncwarp();
  if (lane == 0) mbar_arrive_expect_tx(&P.full[s], total);
  __syncwarp();
  if (nbytes)
    for (int ph = 0; ph < L.ds; ++ph)
      bulk_copy(sw + (2 * s + i) * ww + ph * (L.sub_bytes >> 2), gsrc + ph * L.phase_pitch, nbytes, &P.full[s]);
}

// The same for the twin-window sums (16-bit sources with a one-sample-shifted twin,
// twin[i] = sums[i - 1], four sources per stage): each source is staged twice, the
// sums and the twin, each from the 16-byte boundary at or below the first element
// the block's rows read there, and row r of source 4q + i is pointed into the copy
// in which its first element starts a 32-bit word: an even element index e at byte
// 2e of the sums, an odd one at byte 2(e + 1) of the twin.  Lane 16i + r takes
// sources i and i + 2; lanes 0 and 16 issue the copies.
__device__ __forceinline__ void produce_twin(const Geo& g, Pipe& P, uint32_t* sw, int ww, int zero_q,
                                             int tile_bytes, int64_t twin_off, const GroupDesc<4>& d,
                                             int q, int s, int lane) {
  const int i = lane >> 4, r = lane & 15;
  uint32_t n0[2] = {0, 0}, n1[2] = {0, 0};
  const char *c0[2] = {nullptr, nullptr}, *c1[2] = {nullptr, nullptr};
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int k = i + 2 * h;  // source of the stage
    const int src = 4 * q + k;
    const int win0 = 2 * (4 * s + k) * ww;  // the sums; the twin follows at win0 + ww
    int idx = zero_q;
    if (src < g.nsrc) {
      const int64_t e0 = g.base + d.lo[h];  // first element any row of the block reads
      // element e sits at byte 2e of the sums and at byte 2(e + 1) of the twin
      const int64_t a0 = (2 * e0) & ~int64_t(15);
      const int64_t a1 = (2 * (e0 + 1)) & ~int64_t(15);
      const int64_t o = e0 + d.rel[h];
      idx = (o & 1) ? win0 + ww + static_cast<int>((2 * (o + 1) - a1) >> 2)
                    : win0 + static_cast<int>((2 * o - a0) >> 2);
      if (r == 0) {
        const int64_t last = 2 * (e0 + d.span[h]) + tile_bytes;  // past the last byte any row reads
        n0[h] = static_cast<uint32_t>((last - a0 + 15) & ~int64_t(15));
        n1[h] = static_cast<uint32_t>((last + 2 - a1 + 15) & ~int64_t(15));
        c0[h] = g.src + static_cast<int64_t>(src) * g.src_pitch + a0;
        c1[h] = g.src + static_cast<int64_t>(src) * g.src_pitch + twin_off + a1;
      }
    }
    P.row[s][r][k] = idx;
  }
  uint32_t total = n0[0] + n1[0] + n0[1] + n1[1];
  total += __shfl_xor_sync(0xffffffffu, total, 16);
  __syncwarp();
  if (lane == 0) mbar_arrive_expect_tx(&P.full[s], total);
  __syncwarp();
#pragma unroll
  for (int h = 0; h < 2; ++h)
    if (n0[h]) {
      const int win0 = 2 * (4 * s + i + 2 * h) * ww;
      bulk_copy(sw + win0, c0[h], n0[h], &P.full[s]);
      bulk_copy(sw + win0 + ww, c1[h], n1[h], &P.full[s]);
    }
}

// The same for sources of 32-bit words (folded samples and their sums), QS per
// stage: every offset is a whole word, so a row's offset needs no shift.  EW words per
// element: 1, or 2 for 64-bit sums (offsets and tile in elements).
template <int EW, int QS>
__device__ __forceinline__ void produce_words(const Geo& g, Pipe& P, uint32_t* sw, int ww, int zero_q,
                                              int tile, const GroupDesc<QS>& d, int q, int s, int lane) {
  const int i = lane >> 4, r = lane & 15;
  uint32_t nbytes[QS / 2] = {};
  const char* gsrc[QS / 2] = {};
#pragma unroll
  for (int h = 0; h < QS / 2; ++h) {
    const int k = i + 2 * h;  // source of the stage
    const int src = QS * q + k;
    int idx = zero_q;
    const int64_t e0 = g.base + d.lo[h];
    if (src < g.nsrc && e0 < g.valid) {
      constexpr int kAlign = 4 / EW - 1;  // elements of a 16-byte unit, less one
      const int64_t a0 = e0 & ~int64_t(kAlign);
      idx = (QS * s + k) * ww + EW * (static_cast<int>(e0 - a0) + d.rel[h]);
      if (r == 0) {
        nbytes[h] = static_cast<uint32_t>((e0 + d.span[h] + tile - a0 + kAlign) & ~int64_t(kAlign)) * 4u * EW;
        gsrc[h] = g.src + static_cast<int64_t>(src) * g.src_pitch + 4 * EW * a0;
      }
    }
    P.row[s][r][k] = idx;
  }
  uint32_t total = nbytes[0] + (QS == 4 ? nbytes[QS / 2 - 1] : 0u);
  total += __shfl_xor_sync(0xffffffffu, total, 16);
  __syncwarp();
  if (lane == 0) mbar_arrive_expect_tx(&P.full[s], total);
  __syncwarp();
#pragma unroll
  for (int h = 0; h < QS / 2; ++h)
    if (nbytes[h]) bulk_copy(sw + (QS * s + i + 2 * h) * ww, gsrc[h], nbytes[h], &P.full[s]);
}

// Delays past the chunk's end leave a block's first sources (the lowest frequencies)
// without samples: takes them off the block's sources, in whole groups of QS, so that
// they are neither staged nor summed.  Only blocks that reach past the end look.
template <int QS>
__device__ __forceinline__ void skip_empty_sources(const SumLaunch& L, Geo& g, Pipe& P) {
  if (g.base + L.max_off < g.valid) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t first = static_cast<uint32_t>(g.nsrc);
  for (int i = threadIdx.x; i < g.nsrc && i < static_cast<int>(first); i += kThreads)
    if (g.base + __ldg(&g.desc[i].lo) < g.valid) first = i;
  first = __reduce_min_sync(0xffffffffu, first);
  if (lane == 0) P.first[warp] = first;
  __syncthreads();
  first = __reduce_min_sync(0xffffffffu, P.first[lane & (kWarps - 1)]);
  const int skip = static_cast<int>(first) / QS * QS;
  g.src += skip * g.src_pitch;
  g.desc += skip;
  g.nsrc -= skip;
}

// Pipeline driver shared by the kernels: calls body(stage, cur) for every group of
// QS sources once their windows are in shared memory, and setup() once the first
// windows are on their way (SKIP: sources may lie past the chunk's end); false when the block has nothing to store (kModeTwin: each source is staged
// with its shifted twin, see produce_twin; kModeWords: see produce_words; QS is 4 for
// both; kModeDwords: the same for 64-bit elements; `tile` is in bytes, for words and
// dwords in elements).  The warps take turns at
// staging: warp q % kWarps stages group q, D groups before they are summed, and has
// loaded the group's descriptors kWarps groups earlier, so that no warp carries the
// staging beside its sums and none waits for a descriptor.  D leaves a stage of slack
// to the release of the stage that is refilled.  With one warp staging every group
// all others waited for it (stalls on the full barrier 1.9 cycles per issue in stage
// 1, 3.8 in stage 2): 4096 channels of 8 bits, 2^20 samples, 6001 trials took 66.2 +
// 40.1 ms (stages 1 and 2) that way and 56.6 + 32.8 ms with turns; brute force over
// 1024 channels, 2^17 samples, 1001 trials 10.8 and 8.5 ms.
constexpr int kModePlain = 0, kModeTwin = 1, kModeWords = 2, kModePhase = 3, kModeDwords = 4;
template <int SB, int QS, int MODE, bool SKIP, typename Setup, typename Body>
__device__ __forceinline__ bool run_pipeline(const SumLaunch& L, Geo& g, Pipe& P,
                                             uint32_t* sw, int tile, Setup&& setup, Body&& body) {
  static_assert(MODE == kModePlain || MODE == kModePhase ? QS == 2 : QS == 4 || (QS == 2 && MODE == kModeWords),
                "sources per stage");
  static_assert(kSumMaxStages <= kWarps, "each warp stages at most one group before the loop");
  constexpr int kWinPerSrc = MODE == kModeTwin ? 2 : 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ww = L.win_bytes >> 2;
  const int S = L.stages;
  const int D = max(1, S - 2);
  const int zero_q = kWinPerSrc * QS * S * ww;
  if constexpr (SKIP) skip_empty_sources<QS>(L, g, P);
  const int ngroups = (g.nsrc + QS - 1) / QS;
  GroupDesc<QS> desc;
  desc.load(g, warp, lane);
  // stage 1: blocks past the last column of every row (the last row has the largest skew)
  if (g.skew && g.col >= g.ncols + __ldg(g.skew + g.nrows - 1)) return false;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&P.full[s], 1);
      mbar_init(&P.empty[s], kWarps);
    }
    P.failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  // order earlier generic accesses to the windows (a previous task of a persistent
  // block) before the bulk copies that refill them
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  if (SKIP || g.nsrc % QS)  // a source may be missing, or past the chunk
    for (int i = threadIdx.x; i < ww; i += kThreads) sw[zero_q + i] = 0u;
  __syncthreads();
  volatile int* failed = &P.failed;
  int next = warp;  // the next group this warp stages
  int phase = 0;
  if constexpr (MODE == kModePhase) phase = desc.phase(g, next, lane);
  auto stage_next = [&](int s) {
    if constexpr (MODE == kModeTwin)
      produce_twin(g, P, sw, ww, zero_q, tile, L.twin_off, desc, next, s, lane);
    else if constexpr (MODE == kModeWords || MODE == kModeDwords)
      produce_words<MODE == kModeDwords ? 2 : 1, QS>(g, P, sw, ww, zero_q, tile, desc, next, s, lane);
    else if constexpr (MODE == kModePhase)
      produce_phases<SB>(L, g, P, sw, ww, zero_q, tile, desc, phase, next, s, lane);
    else
      produce<SB>(g, P, sw, ww, zero_q, tile, desc, next, s, lane);
    next += kWarps;
    desc.load(g, next, lane);
    if constexpr (MODE == kModePhase) phase = desc.phase(g, next, lane);
  };
  if (next < min(D, ngroups)) stage_next(next);
  setup();
  int s_cur = 0, p = 0;
  uint32_t ph_cur = 0;
  for (; p < ngroups; ++p) {
    int code = 0;
    if (next == p + D && next < ngroups) {
      const int s = next % S;
      if (next >= S && !mbar_wait(&P.empty[s], ((next / S) - 1) & 1, failed, L.err)) code = kErrWaitEmpty;
      if (__any_sync(0xffffffffu, code)) code = kErrWaitEmpty;
      else stage_next(s);
    }
    if (!code && !mbar_wait(&P.full[s_cur], ph_cur, failed, L.err)) code = kErrWaitFull;
    if (__any_sync(0xffffffffu, code)) {
      if (code && !*failed) {
        atomicCAS(L.err, 0, code);
        *failed = 1;
      }
      break;
    }
    body(s_cur, sw);
    __syncwarp();
    if (lane == 0) mbar_arrive(&P.empty[s_cur]);
    if (++s_cur == S) {
      s_cur = 0;
      ph_cur ^= 1u;
    }
  }
  if (lane == 0 && *failed) {
    // let the copies this warp issued land before the block's shared memory goes away:
    // its groups next - kWarps, ... that it has not waited for
    for (int q = next - kWarps; q >= p && q >= 0; q -= kWarps) {
      const long long t0 = clock64();
      while (!mbar_try_wait(&P.full[q % S], (q / S) & 1) && clock64() - t0 < kWaitCycles) {
      }
    }
  }
  // every phase has completed: retire the barriers so the next task of a
  // persistent block can initialise them again
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int st = 0; st < S; ++st) {
      asm volatile("mbarrier.inval.shared::cta.b64 [%0];\n" ::"r"(smem_addr(&P.full[st])) : "memory");
      asm volatile("mbarrier.inval.shared::cta.b64 [%0];\n" ::"r"(smem_addr(&P.empty[st])) : "memory");
    }
  }
  return !P.failed;
}

// A block's rows are dealt to its warp groups in turn (group i has rows i, i + groups,
// ...), so that blocks in which some rows have no columns still keep every warp busy.
// Rows of this thread's warp group that have columns in the block, as a bit mask: skews
// move rows in and out of the first and last blocks of a launch, and the last row group
// may hold fewer rows.
template <int RB, int T, int ROWS = kSumRows>
__device__ __forceinline__ uint32_t active_rows(const Geo& g, int rbase) {
  constexpr int kGroups = ROWS / RB;
  uint32_t act = 0;
#pragma unroll
  for (int r = 0; r < RB; ++r)
    if (rbase + kGroups * r < g.nrows) {
      const int64_t c = row_col(g, rbase + kGroups * r);
      if (c < g.ncols && c + T > 0) act |= 1u << r;
    }
  return act;
}
// f(r) for the rows of `act`; with all rows active there is no branch between them,
// so that one row's loads can be issued under another's sums.
template <int RB, typename F>
__device__ __forceinline__ void for_rows(uint32_t act, F&& f) {
  if (act == (1u << RB) - 1u) {
#pragma unroll
    for (int r = 0; r < RB; ++r) f(r);
  } else {
#pragma unroll
    for (int r = 0; r < RB; ++r)
      if (act >> r & 1u) f(r);
  }
}

// ------------------------------------------------------------------ 8-bit samples
template <int RB, int NW, bool OUT16, int MODE = kModePlain, int ROWS = kSumRows>
__device__ __forceinline__ void sum_u8(const SumLaunch& L, uint3 blk, uint32_t* sw, Pipe& P) {
  static_assert(NW & 1, "an odd number of consecutive words per lane: conflict-free loads");
  // RB rows per thread: the block's ROWS rows are split over ROWS/RB
  // groups of warps, each group covering the whole tile for its RB rows
  constexpr int kGroups = ROWS / RB;
  constexpr int kWarpsPerTile = kWarps / kGroups;
  constexpr int T = kWarpsPerTile * 32 * NW * 4;
  Geo g = make_geo<MODE == kModePhase, ROWS>(L, T, blk);
  if (g.nrows <= 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rbase = warp / kWarpsPerTile, wt = warp % kWarpsPerTile;
  const int wbase = wt * 32 * NW + lane * NW;
  uint32_t act = 0;
  constexpr int kSeg = 32 * NW * 4;  // samples of a warp's segment
  uint32_t p01[RB][NW], p23[RB][NW];  // field sums of samples (4w, 4w+1) and (4w+2, 4w+3)
#pragma unroll
  for (int r = 0; r < RB; ++r)
#pragma unroll
    for (int k = 0; k < NW; ++k) p01[r][k] = p23[r][k] = 0;
  // 32-bit outputs: each warp adds its fields into the output through a slice of
  // shared memory past the ring (one row at a time, ordered by __syncwarp), as whole
  // 16-byte chunks: a read-add-write of the partial sums an earlier flush stored when
  // `add`.  Clears the fields.
  auto flush = [&](bool add) {
    uint32_t* st = sw + (2 * L.stages + 1) * (L.win_bytes >> 2) + warp * kSeg;
#pragma unroll
    for (int r = 0; r < RB; ++r) {
      if (!(act >> r & 1u)) continue;
#pragma unroll
      for (int k = 0; k < NW; ++k) {
        *reinterpret_cast<uint4*>(st + 4 * (lane * NW + k)) =
            make_uint4(p01[r][k] & 0x7fffu, p01[r][k] >> 15, p23[r][k] & 0x7fffu, p23[r][k] >> 15);
        p01[r][k] = p23[r][k] = 0;
      }
      __syncwarp();
      const int64_t c0 = row_col(g, rbase + kGroups * r) + static_cast<int64_t>(wt) * kSeg;  // multiple of 4
      uint32_t* out = reinterpret_cast<uint32_t*>(g.out + (rbase + kGroups * r) * g.out_pitch) + c0;
      for (int e = 4 * lane; e < kSeg; e += 128) {
        uint4 v = *reinterpret_cast<const uint4*>(st + e);
        if (c0 + e < 0) continue;
        if (c0 + e + 4 <= g.ncols && (reinterpret_cast<uintptr_t>(out + e) & 15) == 0) {
          if (add) {
            const uint4 o = *reinterpret_cast<const uint4*>(out + e);
            v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
          }
          *reinterpret_cast<uint4*>(out + e) = v;
        } else {
          const uint32_t a[4] = {v.x, v.y, v.z, v.w};
          for (int q = 0; q < 4; ++q)
            if (c0 + e + q < g.ncols) out[e + q] = add ? out[e + q] + a[q] : a[q];
        }
      }
      __syncwarp();
    }
  };
  int since = 0;       // sources summed in the fields since the last flush
  bool stored = false; // the output holds partial sums of an earlier flush
  const bool ok = run_pipeline<1, 2, MODE, true>(L, g, P, sw, T, [&] { act = active_rows<RB, T, ROWS>(g, rbase); }, [&](int s, const uint32_t* win) {
    for_rows<RB>(act, [&](int r) {
      const int4 rw = row_info(P, s, rbase + kGroups * r);
      const uint32_t* w0 = win + rw.x + wbase;
      const uint32_t* w1 = win + rw.z + wbase;
      uint32_t va[NW + 1], vb[NW + 1];
#pragma unroll
      for (int i = 0; i <= NW; ++i) { va[i] = w0[i]; vb[i] = w1[i]; }
#pragma unroll
      for (int k = 0; k < NW; ++k) {
        const uint32_t a = __funnelshift_r(va[k], va[k + 1], rw.y);
        const uint32_t b = __funnelshift_r(vb[k], vb[k + 1], rw.w);
        p01[r][k] = dot_lo(b, dot_lo(a, p01[r][k]));
        p23[r][k] = dot_hi(b, dot_hi(a, p23[r][k]));
      }
    });
    if constexpr (!OUT16) {  // (16-bit outputs hold at most 64 sources)
      since += 2;
      if (since >= kDotSources) {  // the fields are full: move them to the output
        flush(stored);
        stored = true;
        since = 0;
      }
    }
  });
  if (!ok) return;
  if constexpr (!OUT16) {
    if (since > 0 || !stored) flush(stored);
    return;
  }
  // 16-bit sums leave through shared memory as whole 16-byte chunks: the ring is
  // free once the pipeline has ended (every warp passed its final barrier), and
  // each warp stages one row of its segment at a time in a slice of its own, so
  // only __syncwarp orders the staging.  With a twin (twin[i] = sums[i - 1]) a
  // warp writes twin[1 .. seg] of its segment; twin[0] is the element before
  // the segment, written by the warp (or block) that holds it (the row's own twin[0]
  // is never read).
  uint16_t* st = reinterpret_cast<uint16_t*>(sw) + warp * kSeg;
#pragma unroll
  for (int r = 0; r < RB; ++r) {
    if (!(act >> r & 1u)) continue;
#pragma unroll
    for (int k = 0; k < NW; ++k)
      *reinterpret_cast<uint2*>(st + 4 * (lane * NW + k)) =
          make_uint2(dot_pack(p01[r][k]), dot_pack(p23[r][k]));
    __syncwarp();
    const int64_t c0 = row_col(g, rbase + kGroups * r) + static_cast<int64_t>(wt) * kSeg;  // multiple of 8
    char* row = g.out + (rbase + kGroups * r) * g.out_pitch;
    uint16_t* out = reinterpret_cast<uint16_t*>(row) + c0;
    uint16_t* tw = L.twin_off ? reinterpret_cast<uint16_t*>(row + L.twin_off) + c0 : nullptr;
    for (int e = 8 * lane; e < kSeg; e += 256) {
      if (c0 + e < 0) continue;
      const uint4 v = *reinterpret_cast<const uint4*>(st + e);
      if (c0 + e + 8 <= g.ncols && (reinterpret_cast<uintptr_t>(out + e) & 15) == 0) {
        *reinterpret_cast<uint4*>(out + e) = v;
      } else {
        for (int q = 0; q < 8; ++q)
          if (c0 + e + q < g.ncols) out[e + q] = st[e + q];
      }
      if (tw) {
        if (e > 0 && c0 + e + 7 <= g.ncols && (reinterpret_cast<uintptr_t>(tw + e) & 15) == 0) {
          const uint32_t p = st[e - 1];
          *reinterpret_cast<uint4*>(tw + e) =
              make_uint4(__byte_perm(p, v.x, 0x5410), __byte_perm(v.x, v.y, 0x5432),
                         __byte_perm(v.y, v.z, 0x5432), __byte_perm(v.z, v.w, 0x5432));
        } else {
          for (int q = e == 0 ? 1 : 0; q < 8; ++q)
            if (c0 + e + q <= g.ncols) tw[e + q] = st[e + q - 1];
        }
      }
    }
    // the first twin element of the next segment (its warp skips it)
    if (tw && lane == 31 && c0 + kSeg >= 1 && c0 + kSeg <= g.ncols) tw[kSeg] = st[kSeg - 1];
    __syncwarp();
  }
}

// ------------------------------------------------------------------ 16-bit samples
// 16-bit samples into 32-bit sums (stage 1 and brute force of 16-bit input).
// For output word k (samples 2k, 2k+1 of the block) a source whose offset is
// word-aligned gives the pair w[k] and one offset by a sample the pair
// (w[k] >> 16, w[k+1] & 0xffff), one byte permute of two words (selector 0x3210
// or 0x5432, so no branch separates a row's sources).  The aligned pairs are
// summed whole into a wrapping 32-bit word and their high halves into another
// (two sources per three-input add); the low samples' sums come out at the end
// as whole - (high << 16).  Three integer-pipe operations per word and source,
// where taking the halves apart by masks and offset-dependent selects took five.
template <int RB, int NW, int MODE = kModePlain, int ROWS = kSumRows>
__device__ __forceinline__ void sum_u16_wide(const SumLaunch& L, uint3 blk, uint32_t* sw, Pipe& P) {
  // RB rows per thread: the block's rows are split over ROWS/RB warp groups,
  // each covering the whole tile for its RB rows (as in sum_u8)
  constexpr int kGroups = ROWS / RB;
  constexpr int kWarpsPerTile = kWarps / kGroups;
  constexpr int T = kWarpsPerTile * 32 * NW * 2;
  Geo g = make_geo<MODE == kModePhase, ROWS>(L, T, blk);
  if (g.nrows <= 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rbase = warp / kWarpsPerTile, wt = warp % kWarpsPerTile;
  const int wbase = wt * 32 * NW + lane * NW;  // consecutive words, as in sum_u8
  uint32_t act = 0;
  uint32_t lo32[RB][NW], hi32[RB][NW];
#pragma unroll
  for (int r = 0; r < RB; ++r)
#pragma unroll
    for (int k = 0; k < NW; ++k) lo32[r][k] = hi32[r][k] = 0;
  const bool ok = run_pipeline<2, 2, MODE, true>(L, g, P, sw, 2 * T, [&] { act = active_rows<RB, T, ROWS>(g, rbase); }, [&](int s, const uint32_t* win) {
    for_rows<RB>(act, [&](int r) {
      const int4 rw = row_info(P, s, rbase + kGroups * r);
      const uint32_t* w0 = win + rw.x + wbase;
      const uint32_t* w1 = win + rw.z + wbase;
      uint32_t va[NW + 1], vb[NW + 1];
#pragma unroll
      for (int i = 0; i <= NW; ++i) { va[i] = w0[i]; vb[i] = w1[i]; }
      // rw.y / rw.w: 0 (word-aligned) or 16 (one sample in): one byte permute
      // aligns the pair; whole words are summed (wrapping) and high halves apart
      const uint32_t sa = rw.y ? 0x5432u : 0x3210u, sb = rw.w ? 0x5432u : 0x3210u;
#pragma unroll
      for (int k = 0; k < NW; ++k) {
        const uint32_t a = __byte_perm(va[k], va[k + 1], sa), b = __byte_perm(vb[k], vb[k + 1], sb);
        lo32[r][k] += a + b;
        hi32[r][k] += (a >> 16) + (b >> 16);
      }
    });
  });
  // lo32 holds sum(low) + 2^16 sum(high) mod 2^32 and sum(low) < 2^32 (at most
  // 65537 sources of 65535), so the low sums are lo32 - (hi32 << 16)
#pragma unroll
  for (int r = 0; r < RB; ++r)
#pragma unroll
    for (int k = 0; k < NW; ++k) lo32[r][k] -= hi32[r][k] << 16;
  if (!ok) return;
#pragma unroll
  for (int r = 0; r < RB; ++r) {
    if (!(act >> r & 1u)) continue;
    const int64_t c0 = row_col(g, rbase + kGroups * r);
    uint32_t* row = reinterpret_cast<uint32_t*>(g.out + (rbase + kGroups * r) * g.out_pitch);
#pragma unroll
    for (int k = 0; k < NW; ++k) {
      const int64_t c = c0 + static_cast<int64_t>(wbase + k) * 2;  // even
      if (c < 0 || c >= g.ncols) continue;
      uint32_t* dst = row + c;
      if (c + 2 <= g.ncols && (reinterpret_cast<uintptr_t>(dst) & 7) == 0) {
        *reinterpret_cast<uint2*>(dst) = make_uint2(lo32[r][k], hi32[r][k]);
      } else {
        dst[0] = lo32[r][k];
        if (c + 1 < g.ncols) dst[1] = hi32[r][k];
      }
    }
  }
}

// ------------------------------------------------------------------ folded samples
// A folded chunk holds in word s the samples s, s + H, s + 2H, s + 3H of a channel
// (8-bit samples, H a quarter of the output columns) or s, s + H (16-bit samples, H
// half of them): one word position stands for a column in each of those segments.  A
// delay moves all of them alike, so every row of every source reads whole aligned
// words whatever its delay: no shift, no neighbouring word.  Per word of four 8-bit
// samples that is one shared load and two dot products.  The subband sums keep the
// fold (segments 0, 1 and 2, 3 as two planes of packed 16-bit pairs, or one plane of
// 32-bit sums per segment), so stage 2 reads aligned words too and needs no twin.
// Lanes own interleaved words (lane l: l, l + 32, ...): a warp's loads and stores are
// 32 consecutive words.  Bound: shared loads and dot products both allow 128 sample
// additions per cycle and SM (3.7e13 per second); stage 1 runs 2.4e13 (first and last
// blocks of a time tile, whose rows are partly idle, cost it most: 2.7e13 with 8 GiB
// tiles), stage 2 (two bytes per addition: 64 per cycle) 1.5e13, its load pipe 85 %
// busy.  Against samples in time order: 4096 channels, 2^20 samples, 6001 trials 56.6 +
// 32.8 -> 34.4 + 27.3 ms.

// Columns of segment f that are stored, in launch columns: below ncols, and for sums
// into the output (L.seg > 0) inside the segment and the chunk.
__device__ __forceinline__ int64_t seg_cols(const SumLaunch& L, int f) {
  if (!L.seg) return L.ncols;
  return min(L.ncols, min(L.seg, L.nout - f * L.seg) - L.out_col0);
}

// Folded 8-bit samples into packed 16-bit planes (PACK) or 32-bit sums per segment.
template <int RB, int NW, bool PACK>
__device__ __forceinline__ void sum_fold8(const SumLaunch& L, uint3 blk, uint32_t* sw, Pipe& P) {
  constexpr int kGroups = kSumRows / RB;  // warp groups sharing the rows, as in sum_u8
  constexpr int kWarpsPerTile = kWarps / kGroups;
  constexpr int T = kWarpsPerTile * 32 * NW;
  Geo g = make_geo(L, T, blk);
  if (g.nrows <= 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rbase = warp / kWarpsPerTile;
  const int wbase = (warp % kWarpsPerTile) * 32 * NW + lane;
  uint32_t act = 0;
  uint32_t p01[RB][NW], p23[RB][NW];  // field sums of segments 0, 1 and 2, 3
#pragma unroll
  for (int r = 0; r < RB; ++r)
#pragma unroll
    for (int k = 0; k < NW; ++k) p01[r][k] = p23[r][k] = 0;
  // 32-bit outputs: adds the fields to what an earlier flush stored when `add`, and
  // clears them.  The block owns its outputs; the additions are reductions in L2, which
  // the warp does not wait for (128 consecutive bytes each).
  auto flush = [&](bool add) {
#pragma unroll
    for (int r = 0; r < RB; ++r) {
      if (!(act >> r & 1u)) continue;
      const int64_t c0 = row_col(g, rbase + kGroups * r) + wbase;
      char* row = g.out + (rbase + kGroups * r) * g.out_pitch;
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        uint32_t* out = reinterpret_cast<uint32_t*>(row + f * L.seg_stride) + c0;
        const int64_t lim = seg_cols(L, f) - c0;
#pragma unroll
        for (int k = 0; k < NW; ++k) {
          const uint32_t p = f < 2 ? p01[r][k] : p23[r][k];
          const uint32_t v = (f & 1) ? p >> 15 : p & 0x7fffu;
          if (32 * k >= lim || c0 + 32 * k < 0) continue;
          if (add) atomicAdd(out + 32 * k, v);
          else out[32 * k] = v;
        }
      }
#pragma unroll
      for (int k = 0; k < NW; ++k) p01[r][k] = p23[r][k] = 0;
    }
  };
  int since = 0;
  bool stored = false;
  const bool ok = run_pipeline<4, 4, kModeWords, true>(L, g, P, sw, T, [&] { act = active_rows<RB, T>(g, rbase); }, [&](int s, const uint32_t* win) {
    for_rows<RB>(act, [&](int r) {
      const int4 a = row_info(P, s, rbase + kGroups * r);
      const uint32_t* w0 = win + a.x + wbase;
      const uint32_t* w1 = win + a.y + wbase;
      const uint32_t* w2 = win + a.z + wbase;
      const uint32_t* w3 = win + a.w + wbase;
#pragma unroll
      for (int k = 0; k < NW; ++k) {
        const uint32_t v0 = w0[32 * k], v1 = w1[32 * k], v2 = w2[32 * k], v3 = w3[32 * k];
        p01[r][k] = dot_lo(v3, dot_lo(v2, dot_lo(v1, dot_lo(v0, p01[r][k]))));
        p23[r][k] = dot_hi(v3, dot_hi(v2, dot_hi(v1, dot_hi(v0, p23[r][k]))));
      }
    });
    if constexpr (!PACK) {  // (packed sums hold at most 64 sources)
      since += 4;
      if (since >= kDotSources) {
        flush(stored);
        stored = true;
        since = 0;
      }
    }
  });
  if (!ok) return;
  if constexpr (!PACK) {
    if (since > 0 || !stored) flush(stored);
    return;
  }
#pragma unroll
  for (int r = 0; r < RB; ++r) {
    if (!(act >> r & 1u)) continue;
    const int64_t c0 = row_col(g, rbase + kGroups * r) + wbase;
    char* row = g.out + (rbase + kGroups * r) * g.out_pitch;
    uint32_t* o0 = reinterpret_cast<uint32_t*>(row) + c0;
    uint32_t* o1 = reinterpret_cast<uint32_t*>(row + L.seg_stride) + c0;
#pragma unroll
    for (int k = 0; k < NW; ++k)
      if (c0 + 32 * k >= 0 && c0 + 32 * k < g.ncols) {
        o0[32 * k] = dot_pack(p01[r][k]);
        o1[32 * k] = dot_pack(p23[r][k]);
      }
  }
}

// Folded 16-bit samples into 32-bit sums per segment: words are summed whole
// (wrapping) beside their high halves; the low samples' sums are whole - (high << 16)
// (at most 65537 sources of 65535 each: no wrap of the low sums).
template <int RB, int NW>
__device__ __forceinline__ void sum_fold16(const SumLaunch& L, uint3 blk, uint32_t* sw, Pipe& P) {
  constexpr int kGroups = kSumRows / RB;
  constexpr int kWarpsPerTile = kWarps / kGroups;
  constexpr int T = kWarpsPerTile * 32 * NW;
  Geo g = make_geo(L, T, blk);
  if (g.nrows <= 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rbase = warp / kWarpsPerTile;
  const int wbase = (warp % kWarpsPerTile) * 32 * NW + lane;
  uint32_t act = 0;
  uint32_t all[RB][NW], hi[RB][NW];
#pragma unroll
  for (int r = 0; r < RB; ++r)
#pragma unroll
    for (int k = 0; k < NW; ++k) all[r][k] = hi[r][k] = 0;
  const bool ok = run_pipeline<4, 4, kModeWords, true>(L, g, P, sw, T, [&] { act = active_rows<RB, T>(g, rbase); }, [&](int s, const uint32_t* win) {
    for_rows<RB>(act, [&](int r) {
      const int4 a = row_info(P, s, rbase + kGroups * r);
      const uint32_t* w0 = win + a.x + wbase;
      const uint32_t* w1 = win + a.y + wbase;
      const uint32_t* w2 = win + a.z + wbase;
      const uint32_t* w3 = win + a.w + wbase;
#pragma unroll
      for (int k = 0; k < NW; ++k) {
        const uint32_t v0 = w0[32 * k], v1 = w1[32 * k], v2 = w2[32 * k], v3 = w3[32 * k];
        all[r][k] += v0 + v1;
        all[r][k] += v2 + v3;
        hi[r][k] = high_add(v3, high_add(v2, high_add(v1, high_add(v0, hi[r][k]))));
      }
    });
  });
  if (!ok) return;
  const int64_t lim0 = seg_cols(L, 0), lim1 = seg_cols(L, 1);
#pragma unroll
  for (int r = 0; r < RB; ++r) {
    if (!(act >> r & 1u)) continue;
    const int64_t c0 = row_col(g, rbase + kGroups * r) + wbase;
    char* row = g.out + (rbase + kGroups * r) * g.out_pitch;
    uint32_t* o0 = reinterpret_cast<uint32_t*>(row) + c0;
    uint32_t* o1 = reinterpret_cast<uint32_t*>(row + L.seg_stride) + c0;
#pragma unroll
    for (int k = 0; k < NW; ++k) {
      const int64_t c = c0 + 32 * k;
      if (c < 0) continue;
      if (c < lim0) o0[32 * k] = all[r][k] - (hi[r][k] << 16);
      if (c < lim1) o1[32 * k] = hi[r][k];
    }
  }
}

// Stage 2 of packed 16-bit planes: grid z = plane p, holding segments 2p (low halves)
// and 2p + 1.  Four words (each half <= 64 x 255) are added before the halves part.
template <int RB, int NW>
__device__ __forceinline__ void sum_plane16(const SumLaunch& L, uint3 blk, uint32_t* sw, Pipe& P) {
  constexpr int kGroups = kSumRows / RB;
  constexpr int kWarpsPerTile = kWarps / kGroups;
  constexpr int T = kWarpsPerTile * 32 * NW;
  Geo g = make_geo(L, T, blk);
  if (g.nrows <= 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rbase = warp / kWarpsPerTile;
  const int wbase = (warp % kWarpsPerTile) * 32 * NW + lane;
  uint32_t act = 0;
  uint32_t all[RB][NW], hi[RB][NW];
#pragma unroll
  for (int r = 0; r < RB; ++r)
#pragma unroll
    for (int k = 0; k < NW; ++k) all[r][k] = hi[r][k] = 0;
  const bool ok = run_pipeline<4, 4, kModeWords, false>(L, g, P, sw, T, [&] { act = active_rows<RB, T>(g, rbase); }, [&](int s, const uint32_t* win) {
    for_rows<RB>(act, [&](int r) {
      const int4 a = row_info(P, s, rbase + kGroups * r);
      const uint32_t* w0 = win + a.x + wbase;
      const uint32_t* w1 = win + a.y + wbase;
      const uint32_t* w2 = win + a.z + wbase;
      const uint32_t* w3 = win + a.w + wbase;
#pragma unroll
      for (int k = 0; k < NW; ++k) {
        const uint32_t q = (w0[32 * k] + w1[32 * k] + w2[32 * k]) + w3[32 * k];
        all[r][k] += q;
        hi[r][k] = high_add(q, hi[r][k]);
      }
    });
  });
  if (!ok) return;
  const int f = 2 * static_cast<int>(blk.z);
  const int64_t c0 = g.col + wbase, lim0 = seg_cols(L, f) - c0, lim1 = seg_cols(L, f + 1) - c0;
#pragma unroll
  for (int r = 0; r < RB; ++r) {
    if (!(act >> r & 1u)) continue;
    uint32_t* o0 = reinterpret_cast<uint32_t*>(g.out + (rbase + kGroups * r) * g.out_pitch) + f * L.seg + c0;
    uint32_t* o1 = o0 + L.seg;
#pragma unroll
    for (int k = 0; k < NW; ++k) {
      if (32 * k < lim0) o0[32 * k] = all[r][k] - (hi[r][k] << 16);
      if (32 * k < lim1) o1[32 * k] = hi[r][k];
    }
  }
}

// Stage 2 of 32-bit subband sums (grid z = plane = segment; one plane when the sums
// are not folded).  Sums wrap modulo 2^32 like the reference's uint32 accumulators.
// Blocks of eight rows have two sources per stage, for windows twice as wide.
template <int RB, int NW, int ROWS = kSumRows>
__device__ __forceinline__ void sum_plane32(const SumLaunch& L, uint3 blk, uint32_t* sw, Pipe& P) {
  constexpr int kGroups = ROWS / RB;
  constexpr int kWarpsPerTile = kWarps / kGroups;
  constexpr int T = kWarpsPerTile * 32 * NW;
  constexpr int QS = ROWS == kSumRows ? 4 : 2;
  Geo g = make_geo<false, ROWS>(L, T, blk);
  if (g.nrows <= 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rbase = warp / kWarpsPerTile;
  const int wbase = (warp % kWarpsPerTile) * 32 * NW + lane;
  uint32_t act = 0;
  uint32_t acc[RB][NW];
#pragma unroll
  for (int r = 0; r < RB; ++r)
#pragma unroll
    for (int k = 0; k < NW; ++k) acc[r][k] = 0;
  const bool ok = run_pipeline<4, QS, kModeWords, false>(L, g, P, sw, T, [&] { act = active_rows<RB, T, ROWS>(g, rbase); }, [&](int s, const uint32_t* win) {
    for_rows<RB>(act, [&](int r) {
      const int4 a = row_info(P, s, rbase + kGroups * r);
      const uint32_t* w0 = win + a.x + wbase;
      const uint32_t* w1 = win + a.y + wbase;
#pragma unroll
      for (int k = 0; k < NW; ++k) acc[r][k] += w0[32 * k] + w1[32 * k];
      if constexpr (QS == 4) {
        const uint32_t* w2 = win + a.z + wbase;
        const uint32_t* w3 = win + a.w + wbase;
#pragma unroll
        for (int k = 0; k < NW; ++k) acc[r][k] += w2[32 * k] + w3[32 * k];
      }
    });
  });
  if (!ok) return;
  const int f = static_cast<int>(blk.z);
  const int64_t c0 = g.col + wbase, lim = seg_cols(L, f) - c0;
#pragma unroll
  for (int r = 0; r < RB; ++r) {
    if (!(act >> r & 1u)) continue;
    uint32_t* out = reinterpret_cast<uint32_t*>(g.out + (rbase + kGroups * r) * g.out_pitch) + f * L.seg + c0;
#pragma unroll
    for (int k = 0; k < NW; ++k)
      if (32 * k < lim) out[32 * k] = acc[r][k];
  }
}

// ------------------------------------------------------------------ 32-bit samples
// Stage 1 and brute force of 32-bit samples into 64-bit sums (the reference's output type
// for them), and stage 2 of those: words and dwords in time order, lanes own interleaved
// elements.  Bound by the shared loads (4 or 8 bytes per addition).  1024 channels, 2^15
// samples, 501 trials, whole run: 1784 us with direct loads of every row, 391 us staged.
template <int RB, int NW, bool WIDE>
__device__ __forceinline__ void sum_to64(const SumLaunch& L, uint3 blk, uint32_t* sw, Pipe& P) {
  constexpr int kGroups = kSumRows / RB;
  constexpr int kWarpsPerTile = kWarps / kGroups;
  constexpr int T = kWarpsPerTile * 32 * NW;
  Geo g = make_geo(L, T, blk);
  if (g.nrows <= 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rbase = warp / kWarpsPerTile;
  const int wbase = (warp % kWarpsPerTile) * 32 * NW + lane;
  uint32_t act = 0;
  unsigned long long acc[RB][NW];
#pragma unroll
  for (int r = 0; r < RB; ++r)
#pragma unroll
    for (int k = 0; k < NW; ++k) acc[r][k] = 0;
  const bool ok = run_pipeline<4, 4, WIDE ? kModeDwords : kModeWords, !WIDE>(
      L, g, P, sw, T, [&] { act = active_rows<RB, T>(g, rbase); }, [&](int s, const uint32_t* win) {
    for_rows<RB>(act, [&](int r) {
      const int4 a = row_info(P, s, rbase + kGroups * r);
      const int at[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if constexpr (WIDE) {
          const unsigned long long* w = reinterpret_cast<const unsigned long long*>(win + at[i]) + wbase;
#pragma unroll
          for (int k = 0; k < NW; ++k) acc[r][k] += w[32 * k];
        } else {
          const uint32_t* w = win + at[i] + wbase;
#pragma unroll
          for (int k = 0; k < NW; ++k) acc[r][k] += w[32 * k];
        }
      }
    });
  });
  if (!ok) return;
#pragma unroll
  for (int r = 0; r < RB; ++r) {
    if (!(act >> r & 1u)) continue;
    const int64_t c0 = row_col(g, rbase + kGroups * r) + wbase;
    unsigned long long* out =
        reinterpret_cast<unsigned long long*>(g.out + (rbase + kGroups * r) * g.out_pitch) + c0;
#pragma unroll
    for (int k = 0; k < NW; ++k)
      if (c0 + 32 * k >= 0 && c0 + 32 * k < g.ncols) out[32 * k] = acc[r][k];
  }
}

// ------------------------------------------------------------------ 16-bit sums with a shifted twin
// Stage 2 of 8-bit input when stage 1 also wrote the one-sample-shifted twin of
// its sums (SumLaunch::twin_off): a row whose offset for a source is odd reads
// that source's twin, so every source word a row needs is one aligned shared
// load, with no permute.  Four sources per stage are added in packed 16-bit
// lanes (each <= 64 x 255, four <= 65280) and folded into two 32-bit sums; lanes own
// interleaved words (lane l: l, l + 32, ...), so the loads of a warp are 32
// consecutive words for any words per lane.  It waits on its shared loads
// (long-scoreboard stalls 3.3 per issue at two blocks per SM), so it is built for
// three blocks per SM: 36.7 ms for 4096 channels, 2^20 samples, 6001 trials against
// 43.2 at two blocks (with four rows per warp and turns 32.8).  Chunks that fold take
// sum_plane16 instead.
#ifndef DD_SUM16T_MINB
#define DD_SUM16T_MINB 3
#endif
template <int RB, int NW, int ROWS = kSumRows>
__device__ __forceinline__ void sum_u16_twin(const SumLaunch& L, uint3 blk, uint32_t* sw, Pipe& P) {
  constexpr int kGroups = ROWS / RB;  // warp groups sharing the rows, as in sum_u8
  constexpr int kWarpsPerTile = kWarps / kGroups;
  constexpr int T = kWarpsPerTile * 32 * NW * 2;
  Geo g = make_geo<false, ROWS>(L, T, blk);
  if (g.nrows <= 0) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rbase = warp / kWarpsPerTile;
  const int wbase = (warp % kWarpsPerTile) * 32 * NW + lane;
  uint32_t act = 0;
  uint32_t lo[RB][NW], hi[RB][NW];
#pragma unroll
  for (int r = 0; r < RB; ++r)
#pragma unroll
    for (int k = 0; k < NW; ++k) lo[r][k] = hi[r][k] = 0;
  const bool ok = run_pipeline<2, 4, kModeTwin, false>(L, g, P, sw, 2 * T, [&] { act = active_rows<RB, T, ROWS>(g, rbase); }, [&](int s, const uint32_t* win) {
    for_rows<RB>(act, [&](int r) {
      const int4 a = row_info(P, s, rbase + kGroups * r);
      const uint32_t* w0 = win + a.x + wbase;
      const uint32_t* w1 = win + a.y + wbase;
      const uint32_t* w2 = win + a.z + wbase;
      const uint32_t* w3 = win + a.w + wbase;
#pragma unroll
      for (int k = 0; k < NW; ++k) {
        const uint32_t q = (w0[32 * k] + w1[32 * k] + w2[32 * k]) + w3[32 * k];
        lo[r][k] += q;
        hi[r][k] = high_add(q, hi[r][k]);
      }
    });
  });
  if (!ok) return;
#pragma unroll
  for (int r = 0; r < RB; ++r) {
    if (!(act >> r & 1u)) continue;
    uint32_t* row = reinterpret_cast<uint32_t*>(g.out + (rbase + kGroups * r) * g.out_pitch) + g.col;
#pragma unroll
    for (int k = 0; k < NW; ++k) {
      const int64_t t = static_cast<int64_t>(wbase + 32 * k) * 2;
      if (g.col + t >= g.ncols) continue;
      const uint32_t s0 = lo[r][k] - (hi[r][k] << 16), s1 = hi[r][k];
      uint32_t* dst = row + t;
      if (g.col + t + 2 <= g.ncols && (reinterpret_cast<uintptr_t>(dst) & 7) == 0) {
        *reinterpret_cast<uint2*>(dst) = make_uint2(s0, s1);
      } else {
        dst[0] = s0;
        if (g.col + t + 1 < g.ncols) dst[1] = s1;
      }
    }
  }
}

template <int RB, int NW, bool OUT16, int MODE = kModePlain, int ROWS = kSumRows>
__global__ void __launch_bounds__(kThreads, DD_SUM8_MINB) k_sum_u8(SumLaunch L) {
  extern __shared__ __align__(128) uint32_t sw[];
  __shared__ Pipe P;
  sum_u8<RB, NW, OUT16, MODE, ROWS>(L, blockIdx, sw, P);
}
template <int RB, int NW, int MODE = kModePlain, int ROWS = kSumRows>
__global__ void __launch_bounds__(kThreads, DD_SUM16W_MINB) k_sum_u16w(SumLaunch L) {
  extern __shared__ __align__(128) uint32_t sw[];
  __shared__ Pipe P;
  sum_u16_wide<RB, NW, MODE, ROWS>(L, blockIdx, sw, P);
}
template <int RB, int NW, int ROWS = kSumRows>
__global__ void __launch_bounds__(kThreads, DD_SUM16T_MINB) k_sum_u16t(SumLaunch L) {
  extern __shared__ __align__(128) uint32_t sw[];
  __shared__ Pipe P;
  sum_u16_twin<RB, NW, ROWS>(L, blockIdx, sw, P);
}
template <int RB, int NW, bool PACK>
__global__ void __launch_bounds__(kThreads, DD_FOLD8_MINB) k_sum_fold8(SumLaunch L) {
  extern __shared__ __align__(128) uint32_t sw[];
  __shared__ Pipe P;
  sum_fold8<RB, NW, PACK>(L, blockIdx, sw, P);
}
template <int RB, int NW>
__global__ void __launch_bounds__(kThreads, DD_FOLD16_MINB) k_sum_fold16(SumLaunch L) {
  extern __shared__ __align__(128) uint32_t sw[];
  __shared__ Pipe P;
  sum_fold16<RB, NW>(L, blockIdx, sw, P);
}
template <int RB, int NW>
__global__ void __launch_bounds__(kThreads, DD_PLANE16_MINB) k_sum_plane16(SumLaunch L) {
  extern __shared__ __align__(128) uint32_t sw[];
  __shared__ Pipe P;
  sum_plane16<RB, NW>(L, blockIdx, sw, P);
}
template <int RB, int NW, bool WIDE>
__global__ void __launch_bounds__(kThreads, 2) k_sum_to64(SumLaunch L) {
  extern __shared__ __align__(128) uint32_t sw[];
  __shared__ Pipe P;
  sum_to64<RB, NW, WIDE>(L, blockIdx, sw, P);
}
template <int RB, int NW, int ROWS = kSumRows>
__global__ void __launch_bounds__(kThreads, DD_PLANE32_MINB) k_sum_plane32(SumLaunch L) {
  extern __shared__ __align__(128) uint32_t sw[];
  __shared__ Pipe P;
  sum_plane32<RB, NW, ROWS>(L, blockIdx, sw, P);
}

// ------------------------------------------------------------------ batched launches
// Block-to-group search: the last group whose first block is <= b.
__device__ __forceinline__ int find_group(const SumBatchGroup* groups, int ngroups, long long b) {
  int lo = 0, hi = ngroups - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(&groups[mid].first) <= b) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// The group's launch description, once per block, into shared memory.
__device__ __forceinline__ void load_launch(const SumBatchGroup* g, SumLaunch& s_L) {
  const uint32_t* src = reinterpret_cast<const uint32_t*>(&g->L);
  uint32_t* dst = reinterpret_cast<uint32_t*>(&s_L);
  for (int i = threadIdx.x; i < static_cast<int>(sizeof(SumLaunch) / 4); i += kThreads)
    dst[i] = __ldg(src + i);
}

__device__ __forceinline__ uint3 group_block(long long local, unsigned gx, unsigned gy) {
  uint3 blk;
  blk.x = static_cast<unsigned>(local % gx);
  local /= gx;
  blk.y = static_cast<unsigned>(local % gy);
  blk.z = static_cast<unsigned>(local / gy);
  return blk;
}

template <int KIND>
__device__ __forceinline__ void run_one(const SumLaunch& L, uint3 blk, uint32_t* sw, Pipe& P) {
  if constexpr (KIND == kSumKindU8Out16) sum_u8<kSumRowsPT8, DD_SUM8_NW, true>(L, blk, sw, P);
  else if constexpr (KIND == kSumKindU8Flush) sum_u8<kSumRowsPT8, DD_SUM8_NW, false>(L, blk, sw, P);
  else if constexpr (KIND == kSumKindU16Wide) sum_u16_wide<kSumRowsPTW, DD_SUM16W_NW>(L, blk, sw, P);
  else if constexpr (KIND == kSumKindU16Twin) sum_u16_twin<kSumRowsPTT, kSum16TNW>(L, blk, sw, P);
  else if constexpr (KIND == kSumKindU8Phase) sum_u8<kSumRowsPT8, kPhase8NW, false, kModePhase>(L, blk, sw, P);
  else if constexpr (KIND == kSumKindU16Phase) sum_u16_wide<kSumRowsPTW, DD_SUM16W_NW, kModePhase>(L, blk, sw, P);
  else if constexpr (KIND == kSumKindFold8) sum_fold8<kFold8RB, kFold8NW, true>(L, blk, sw, P);
  else if constexpr (KIND == kSumKindFold8W) sum_fold8<kFold8WRB, kFold8WNW, false>(L, blk, sw, P);
  else if constexpr (KIND == kSumKindFold16) sum_fold16<kFold16RB, kFold16NW>(L, blk, sw, P);
  else if constexpr (KIND == kSumKindPlane16) sum_plane16<kPlane16RB, kPlane16NW>(L, blk, sw, P);
  else if constexpr (KIND == kSumKindFold8S) sum_fold8<kFold8RB, kFold8NW / 2, true>(L, blk, sw, P);
  else if constexpr (KIND == kSumKindFold8WS) sum_fold8<kFold8WRB, kFold8WNW / 2, false>(L, blk, sw, P);
  else if constexpr (KIND == kSumKindFold16S) sum_fold16<kFold16RB, kFold16NW / 2>(L, blk, sw, P);
  else if constexpr (KIND == kSumKindPlane16S) sum_plane16<kPlane16RB, kPlane16NW / 2>(L, blk, sw, P);
  else if constexpr (KIND == kSumKindPlane32S) sum_plane32<kPlane32RB, kPlane32NW / 2>(L, blk, sw, P);
  else if constexpr (KIND == kSumKindU8Out16R8) sum_u8<kSumRowsPT8, DD_SUM8_NW, true, kModePlain, 8>(L, blk, sw, P);
  else if constexpr (KIND == kSumKindU8FlushR8) sum_u8<kSumRowsPT8, kFlush8R8NW, false, kModePlain, 8>(L, blk, sw, P);
  else if constexpr (KIND == kSumKindU16WideR8) sum_u16_wide<kSumRowsPTW, DD_SUM16W_NW, kModePlain, 8>(L, blk, sw, P);
  else if constexpr (KIND == kSumKindU16TwinR8) sum_u16_twin<kSumRowsPTT, kSum16TNW, 8>(L, blk, sw, P);
  else if constexpr (KIND == kSumKindPlane32R8) sum_plane32<kPlane32RB, kPlane32NW, 8>(L, blk, sw, P);
  else sum_plane32<kPlane32RB, kPlane32NW>(L, blk, sw, P);
}

// Static shared memory of the largest staged-sum kernel (k_sum_batch).
static_assert(sizeof(Pipe) + sizeof(SumLaunch) + 64 <= kSumStaticSmem, "window_bytes counts it");

// Grouped launch: one grid over the blocks of several staged sums of the same
// variant (the same stage of many plans), none of which reads another's output.
template <int KIND>
__global__ void __launch_bounds__(kThreads, 2) k_sum_grouped(const SumBatchGroup* groups,
                                                            int ngroups) {
  extern __shared__ __align__(128) uint32_t sw[];
  __shared__ Pipe P;
  __shared__ SumLaunch s_L;
  __shared__ int s_group;
  const long long b = blockIdx.x;
  if (threadIdx.x == 0) s_group = find_group(groups, ngroups, b);
  __syncthreads();
  const SumBatchGroup* G = groups + s_group;
  load_launch(G, s_L);
  __syncthreads();
  run_one<KIND>(s_L, group_block(b - __ldg(&G->first), __ldg(&G->gx), s_L.grid_y), sw, P);
}

// Persistent launch over the blocks of many staged sums, dependent stages
// included.  Blocks are handed out in order by an atomic counter; a group whose
// input is produced by an earlier group waits (bounded) until that group's
// blocks have all signalled completion.  Every block of an earlier group has
// already been handed to a running block, so the waits always end.
__device__ __forceinline__ void run_kind(int kind, const SumLaunch& L, uint3 blk, uint32_t* sw,
                                         Pipe& P) {
  switch (kind) {
    case kSumKindU8Out16: run_one<kSumKindU8Out16>(L, blk, sw, P); break;
    case kSumKindU8Flush: run_one<kSumKindU8Flush>(L, blk, sw, P); break;
    case kSumKindU16Wide: run_one<kSumKindU16Wide>(L, blk, sw, P); break;
    case kSumKindU16Twin: run_one<kSumKindU16Twin>(L, blk, sw, P); break;
    case kSumKindFold8: run_one<kSumKindFold8>(L, blk, sw, P); break;
    case kSumKindFold8W: run_one<kSumKindFold8W>(L, blk, sw, P); break;
    case kSumKindFold16: run_one<kSumKindFold16>(L, blk, sw, P); break;
    case kSumKindPlane16: run_one<kSumKindPlane16>(L, blk, sw, P); break;
    case kSumKindFold8S: run_one<kSumKindFold8S>(L, blk, sw, P); break;
    case kSumKindFold8WS: run_one<kSumKindFold8WS>(L, blk, sw, P); break;
    case kSumKindFold16S: run_one<kSumKindFold16S>(L, blk, sw, P); break;
    case kSumKindPlane16S: run_one<kSumKindPlane16S>(L, blk, sw, P); break;
    case kSumKindPlane32S: run_one<kSumKindPlane32S>(L, blk, sw, P); break;
    default: run_one<kSumKindPlane32>(L, blk, sw, P); break;
  }
}

__global__ void __launch_bounds__(kThreads, 2) k_sum_batch(const SumBatchGroup* groups,
                                                          int ngroups, long long total,
                                                          int* ctrs, unsigned long long* next,
                                                          int* err) {
  extern __shared__ __align__(128) uint32_t sw[];
  __shared__ Pipe P;
  __shared__ SumLaunch s_L;
  __shared__ long long s_blk;
  __shared__ int s_group, s_ok;
  // the next block is taken while the current one runs, so the atomic's latency
  // overlaps work (the hand-out order is unchanged)
  long long b_next = 0;
  if (threadIdx.x == 0) b_next = static_cast<long long>(atomicAdd(next, 1ull));
  for (;;) {
    if (threadIdx.x == 0) {
      const long long b = b_next;
      s_blk = b;
      s_ok = 1;
      if (b < total) {
        b_next = static_cast<long long>(atomicAdd(next, 1ull));
        const int g = find_group(groups, ngroups, b);
        s_group = g;
        const int wc = groups[g].wait_ctr;
        if (wc >= 0) {
          const int need = groups[g].wait_need;
          const long long t0 = clock64();
          for (;;) {
            int v;
            asm volatile("ld.acquire.gpu.global.s32 %0, [%1];\n" : "=r"(v) : "l"(ctrs + wc) : "memory");
            if (v >= need) break;
            if (*reinterpret_cast<volatile int*>(err) || clock64() - t0 > kWaitCycles) {
              atomicCAS(err, 0, kErrWaitGroup);
              s_ok = 0;
              break;
            }
            __nanosleep(128);
          }
          // the bulk copies that follow read what the other blocks wrote
          asm volatile("fence.proxy.async.global;\n" ::: "memory");
        }
      }
    }
    __syncthreads();
    const long long b = s_blk;
    if (b >= total) break;
    const SumBatchGroup* G = groups + s_group;
    load_launch(G, s_L);
    __syncthreads();
    if (s_ok) run_kind(G->kind, s_L, group_block(b - G->first, G->gx, s_L.grid_y), sw, P);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(ctrs + G->done_ctr, 1);
  }
}

template <typename K>
void launch_k(K kernel, dim3 grid, size_t smem, const SumLaunch& L, cudaStream_t st) {
  allow_dynamic_smem(kernel, smem);
  kernel<<<grid, kThreads, smem, st>>>(L);
  DD_LAUNCHED();
}

}  // namespace

int sum_tile_samples(int src_bytes, int nw) { return kWarps * 32 * nw * (4 / src_bytes); }

// Ring of `stages` groups of qs windows plus one zeroed window.
size_t sum_smem_bytes(int win_bytes, int stages, int qs) {
  return static_cast<size_t>(qs * stages + 1) * win_bytes;
}

size_t sum_kind_extra_smem(int kind) {
  // the flush staging of the 8-bit kernel with 32-bit outputs: one segment of
  // 32-bit sums per warp
  const int nw = kind == kSumKindU8Flush ? DD_SUM8_NW : kind == kSumKindU8Phase ? kPhase8NW
                 : kind == kSumKindU8FlushR8 ? kFlush8R8NW : 0;
  return static_cast<size_t>(kWarps) * 32 * nw * 4 * sizeof(uint32_t);
}

size_t sum_launch_smem(const SumLaunch& L) {
  const int kind = sum_kind(L);
  return sum_smem_bytes(L.win_bytes, L.stages, sum_kind_qs(kind)) + sum_kind_extra_smem(kind);
}

// Stages (groups of sources) for a window size: as many as fit DD_SUM_SMEM_KB of shared
// memory (two blocks per SM at the default), at least two.
// The twin-window stage-2 kernel (eight windows per stage) is limited by the
// latency of its shared loads rather than by issue: it takes at most
// DD_SUM16T_SMEM_KB so that three blocks fit an SM.
#ifndef DD_SUM16T_SMEM_KB
#define DD_SUM16T_SMEM_KB 68
#endif
int sum_stages(int win_bytes, int qs, size_t extra, int cap_kb) {
  const size_t cap = static_cast<size_t>(cap_kb > 0 ? cap_kb : DD_SUM_SMEM_KB) * 1024;
  int s = kSumMaxStages;
  while (s > 2 && sum_smem_bytes(win_bytes, s, qs) + extra > cap) --s;
  return s;
}

int sum_kind_stages(int kind, int win_bytes) {
  return sum_stages(win_bytes, sum_kind_qs(kind), sum_kind_extra_smem(kind),
                    kind == kSumKindU16Twin || kind == kSumKindU16TwinR8 ? DD_SUM16T_SMEM_KB : DD_SUM_SMEM_KB);
}

std::vector<SumDesc> build_sum_desc(const std::vector<int32_t>& tab, int64_t nrows,
                                    int64_t ncols, int64_t group, int* spread, int rows) {
  const int64_t blk = group > 0 ? group : nrows;
  const int64_t per = (blk + rows - 1) / rows;  // row groups per block of rows
  const int64_t nblk = (nrows + blk - 1) / blk;
  std::vector<SumDesc> d(static_cast<size_t>(nblk * per * ncols));
  int32_t most = 0;
  std::vector<int32_t> lo(static_cast<size_t>(ncols)), hi(static_cast<size_t>(ncols));
  for (int64_t b = 0; b < nblk; ++b) {
    const int64_t b0 = b * blk, b1 = std::min(nrows, b0 + blk);
    for (int64_t gi = 0; gi < per; ++gi) {
      const int64_t r0 = b0 + gi * rows;
      const int64_t r1 = std::min(b1, r0 + rows);
      SumDesc* row = d.data() + (b * per + gi) * ncols;
      if (r0 >= r1) continue;
      const int32_t* first = tab.data() + r0 * ncols;
      std::copy(first, first + ncols, lo.begin());
      std::copy(first, first + ncols, hi.begin());
      for (int64_t r = r0 + 1; r < r1; ++r) {
        const int32_t* v = tab.data() + r * ncols;
        for (int64_t c = 0; c < ncols; ++c) {
          lo[c] = std::min(lo[c], v[c]);
          hi[c] = std::max(hi[c], v[c]);
        }
      }
      for (int64_t c = 0; c < ncols; ++c) {
        row[c].lo = lo[c];
        row[c].span = hi[c] - lo[c];
        most = std::max(most, row[c].span);
      }
      for (int64_t r = r0; r < r1; ++r)
        for (int64_t c = 0; c < ncols; ++c)
          row[c].rel[r - r0] = static_cast<uint16_t>(tab[r * ncols + c] - lo[c]);
    }
  }
  *spread = most;
  return d;
}

void launch_sum(const SumLaunch& L, cudaStream_t st) {
  dim3 grid(sum_grid_x(L), L.grid_y, L.grid_z);
  if (L.stages < 2 || L.stages > kSumMaxStages) throw Error{DD_ERR_RUNTIME, "bad stage count"};
  if (!L.desc || !L.err) throw Error{DD_ERR_RUNTIME, "staged sum without descriptors"};
  const size_t smem = sum_launch_smem(L);
  switch (sum_kind(L)) {
    case kSumKindU8Out16: launch_k(k_sum_u8<kSumRowsPT8, DD_SUM8_NW, true>, grid, smem, L, st); break;
    case kSumKindU8Flush: launch_k(k_sum_u8<kSumRowsPT8, DD_SUM8_NW, false>, grid, smem, L, st); break;
    case kSumKindU16Wide: launch_k(k_sum_u16w<kSumRowsPTW, DD_SUM16W_NW>, grid, smem, L, st); break;
    case kSumKindU16Twin: launch_k(k_sum_u16t<kSumRowsPTT, kSum16TNW>, grid, smem, L, st); break;
    case kSumKindU8Phase: launch_k(k_sum_u8<kSumRowsPT8, kPhase8NW, false, kModePhase>, grid, smem, L, st); break;
    case kSumKindU16Phase: launch_k(k_sum_u16w<kSumRowsPTW, DD_SUM16W_NW, kModePhase>, grid, smem, L, st); break;
    case kSumKindWord64: launch_k(k_sum_to64<kTo64RB, kTo64NW, false>, grid, smem, L, st); break;
    case kSumKindPlane64: launch_k(k_sum_to64<kTo64RB, kTo64NW, true>, grid, smem, L, st); break;
    case kSumKindFold8: launch_k(k_sum_fold8<kFold8RB, kFold8NW, true>, grid, smem, L, st); break;
    case kSumKindFold8W: launch_k(k_sum_fold8<kFold8WRB, kFold8WNW, false>, grid, smem, L, st); break;
    case kSumKindFold16: launch_k(k_sum_fold16<kFold16RB, kFold16NW>, grid, smem, L, st); break;
    case kSumKindPlane16: launch_k(k_sum_plane16<kPlane16RB, kPlane16NW>, grid, smem, L, st); break;
    case kSumKindFold8S: launch_k(k_sum_fold8<kFold8RB, kFold8NW / 2, true>, grid, smem, L, st); break;
    case kSumKindFold8WS: launch_k(k_sum_fold8<kFold8WRB, kFold8WNW / 2, false>, grid, smem, L, st); break;
    case kSumKindFold16S: launch_k(k_sum_fold16<kFold16RB, kFold16NW / 2>, grid, smem, L, st); break;
    case kSumKindPlane16S: launch_k(k_sum_plane16<kPlane16RB, kPlane16NW / 2>, grid, smem, L, st); break;
    case kSumKindPlane32S: launch_k(k_sum_plane32<kPlane32RB, kPlane32NW / 2>, grid, smem, L, st); break;
    case kSumKindU8Out16R8: launch_k(k_sum_u8<kSumRowsPT8, DD_SUM8_NW, true, kModePlain, 8>, grid, smem, L, st); break;
    case kSumKindU8FlushR8: launch_k(k_sum_u8<kSumRowsPT8, kFlush8R8NW, false, kModePlain, 8>, grid, smem, L, st); break;
    case kSumKindU16WideR8: launch_k(k_sum_u16w<kSumRowsPTW, DD_SUM16W_NW, kModePlain, 8>, grid, smem, L, st); break;
    case kSumKindU16TwinR8: launch_k(k_sum_u16t<kSumRowsPTT, kSum16TNW, 8>, grid, smem, L, st); break;
    case kSumKindPlane32R8: launch_k(k_sum_plane32<kPlane32RB, kPlane32NW, 8>, grid, smem, L, st); break;
    default: launch_k(k_sum_plane32<kPlane32RB, kPlane32NW>, grid, smem, L, st); break;
  }
}

int sum_kind(const SumLaunch& L) { return L.kind; }
unsigned sum_grid_x(const SumLaunch& L) {
  const int T = sum_kind_tile(sum_kind(L));
  return static_cast<unsigned>((L.ncols + L.max_skew + T - 1) / T);
}

int sum_batch_blocks_per_sm(size_t smem) {
  int n = 0;
  DD_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_sum_batch, kThreads, smem));
  return n;
}

void launch_sum_batch(const SumBatchGroup* d_groups, int ngroups, long long total, int* d_ctrs,
                      unsigned long long* d_next, int* d_err, size_t smem, unsigned grid,
                      cudaStream_t st) {
  allow_dynamic_smem(k_sum_batch, smem);
  k_sum_batch<<<grid, kThreads, smem, st>>>(d_groups, ngroups, total, d_ctrs, d_next, d_err);
  DD_LAUNCHED();
}

template <int KIND>
void launch_grouped_k(const SumBatchGroup* d_groups, int ngroups, long long total, size_t smem,
                      cudaStream_t st) {
  allow_dynamic_smem(k_sum_grouped<KIND>, smem);
  k_sum_grouped<KIND><<<static_cast<unsigned>(total), kThreads, smem, st>>>(d_groups, ngroups);
  DD_LAUNCHED();
}

void launch_sum_grouped(const SumBatchGroup* d_groups, int ngroups, long long total, int kind,
                        size_t smem, cudaStream_t st) {
  if (total <= 0) return;
  if (total >= (1LL << 31)) throw Error{DD_ERR_RUNTIME, "grouped launch too large"};
  switch (kind) {
    case kSumKindU8Out16: launch_grouped_k<kSumKindU8Out16>(d_groups, ngroups, total, smem, st); break;
    case kSumKindU8Flush: launch_grouped_k<kSumKindU8Flush>(d_groups, ngroups, total, smem, st); break;
    case kSumKindU16Wide: launch_grouped_k<kSumKindU16Wide>(d_groups, ngroups, total, smem, st); break;
    case kSumKindU16Twin: launch_grouped_k<kSumKindU16Twin>(d_groups, ngroups, total, smem, st); break;
    case kSumKindU8Phase: launch_grouped_k<kSumKindU8Phase>(d_groups, ngroups, total, smem, st); break;
    case kSumKindU16Phase: launch_grouped_k<kSumKindU16Phase>(d_groups, ngroups, total, smem, st); break;
    case kSumKindFold8: launch_grouped_k<kSumKindFold8>(d_groups, ngroups, total, smem, st); break;
    case kSumKindFold8W: launch_grouped_k<kSumKindFold8W>(d_groups, ngroups, total, smem, st); break;
    case kSumKindFold16: launch_grouped_k<kSumKindFold16>(d_groups, ngroups, total, smem, st); break;
    case kSumKindPlane16: launch_grouped_k<kSumKindPlane16>(d_groups, ngroups, total, smem, st); break;
    case kSumKindFold8S: launch_grouped_k<kSumKindFold8S>(d_groups, ngroups, total, smem, st); break;
    case kSumKindFold8WS: launch_grouped_k<kSumKindFold8WS>(d_groups, ngroups, total, smem, st); break;
    case kSumKindFold16S: launch_grouped_k<kSumKindFold16S>(d_groups, ngroups, total, smem, st); break;
    case kSumKindPlane16S: launch_grouped_k<kSumKindPlane16S>(d_groups, ngroups, total, smem, st); break;
    case kSumKindPlane32S: launch_grouped_k<kSumKindPlane32S>(d_groups, ngroups, total, smem, st); break;
    case kSumKindU8Out16R8: launch_grouped_k<kSumKindU8Out16R8>(d_groups, ngroups, total, smem, st); break;
    case kSumKindU8FlushR8: launch_grouped_k<kSumKindU8FlushR8>(d_groups, ngroups, total, smem, st); break;
    case kSumKindU16WideR8: launch_grouped_k<kSumKindU16WideR8>(d_groups, ngroups, total, smem, st); break;
    case kSumKindU16TwinR8: launch_grouped_k<kSumKindU16TwinR8>(d_groups, ngroups, total, smem, st); break;
    case kSumKindPlane32R8: launch_grouped_k<kSumKindPlane32R8>(d_groups, ngroups, total, smem, st); break;
    default: launch_grouped_k<kSumKindPlane32>(d_groups, ngroups, total, smem, st); break;
  }
}

}  // namespace dd
