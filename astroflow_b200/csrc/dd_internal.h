// Internal declarations of the B200 dedispersion library (not part of the ABI).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <vector>

#include "../../include/astroflow_dd.h"

namespace dd {

// ---------------------------------------------------------------- errors
void set_error(const std::string& msg);
struct Error {
  int code;
  std::string msg;
};
#define DD_CUDA_TRY(call)                                                          \
  do {                                                                             \
    cudaError_t e_ = (call);                                                       \
    if (e_ != cudaSuccess) {                                                       \
      cudaGetLastError(); /* reported here: the thread's next check must not see it */ \
      throw ::dd::Error{DD_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)}; \
    }                                                                              \
  } while (0)

// Kernel launches made by this library on the calling thread (monotonic).
long long& launch_count();
#define DD_COUNT_LAUNCH() (++::dd::launch_count())
// After a kernel launch: count it and surface launch errors.
#define DD_LAUNCHED()                           \
  do {                                          \
    DD_COUNT_LAUNCH();                          \
    DD_CUDA_TRY(cudaGetLastError());            \
  } while (0)

// ---------------------------------------------------------------- device buffer
struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  ~DevBuf() { release(); }
  void alloc(size_t n);
  void release();
  template <typename T> T* as() const { return static_cast<T*>(p); }
};

// Geometry of one IQRM segment: the samples [t0, t1) are covered by the same
// set of IQRM windows, whose masks are OR-ed into seg_mask[segment][nchans].
struct IqrmSeg {
  uint32_t t0, t1;
};

}  // namespace dd

struct dd_plan {
  dd_header hdr{};
  dd_plan_params p{};
  dd_rfi_config rfi{};
  int device = 0;
  int nbits = 8;
  int elem = 1;  // bytes per input sample

  std::vector<double> freq;  // channel frequencies (ascending)
  int64_t cs = 0, ce = 0;    // band: [cs, ce] subband, [cs, ce) brute force
  int64_t dm_steps = 0;
  int64_t nin = 0;           // input samples
  int64_t nbin = 0;          // binned samples (subband) / input samples (brute)
  int64_t nout = 0;          // subband: output columns (nbin, or fewer for a stream's plan)
  float ref_freq = 0.f;
  double tsamp = 0;          // sampling time as the reference path uses it

  // subband geometry
  int64_t dch = 0, nsb = 0, ndm_nom = 0;
  int sbw = 32, ndm0 = 32;
  int max_delay = 0, max_res = 0;
  int inter16 = 0;           // stage-1 sums stored as uint16 (8-bit input, narrow subbands)
  // Folded layout (dd_sumsmem.cu): samples per word (4 or 2; 1: not folded), output
  // columns per segment (all of them when not folded), planes of subband sums.  The
  // time tiles, and x and subband-sum pitches of a folded plan count words.
  int fold = 1;
  bool may_fold = true;      // false: the folded layout's buffers did not fit the device
  int64_t seg = 0;
  int planes = 1;
  int twin = 0;              // stage 1 also writes the one-sample-shifted twin of its uint16 sums
  int64_t tile = 0;          // time tile of the stage-1 -> stage-2 pipeline
  int64_t tile_pitch = 0;    // row pitch of the inter tile (elements)
  int64_t xpitch = 0;        // row pitch of the channel-major prepared input (elements)
  int win1 = 0, win2 = 0;    // staged window bytes of the shared-memory sums (0: not used)
  bool small1 = false, small2 = false, smallb = false;  // half tiles (sum_kind_small): stages, brute force
  bool few1 = false, few2 = false, fewb = false;        // eight rows a block (sum_kind_rows8)
  int64_t max_skew1 = 0;     // largest row skew of stage 1
  int64_t reach1 = 0;        // largest offset a stage-1 window reads past its column
  int64_t spread1 = 0;       // largest spread of a stage-1 window
  int64_t max_off1 = 0;      // largest skewed stage-1 offset

  // brute-force geometry (CPU path semantics)
  int64_t nc = 0;            // channels summed, [cs, ce)
  int64_t sps = 0;           // samples per slice
  int64_t nslices = 0;
  int64_t cols0 = 0;         // columns of a full slice
  std::vector<int64_t> slice_cols;
  int64_t out_cols = 0;
  int64_t phase_len = 0;     // padded length of one phase row of the brute-force layout
  bool phases_merge = true;  // slices share one phase pattern (sps % ds == 0)
  int winb = 0;              // staged window bytes of the brute-force sums (0: not used)
  int subb = 0;              // ... of one phase row of a window (downsampled)
  int64_t pattern_descs = 0; // descriptors per slice pattern (downsampled)

  // tables (host copies)
  std::vector<int32_t> h_delay;  // [ndm_nom][dch] (subband) or [dm_steps][nc] (brute)
  std::vector<int32_t> h_res;    // [dm_steps][nsb]
  int64_t table_mismatch_fp64 = 0;

  // IQRM
  std::vector<uint32_t> win_t0, win_t1;
  std::vector<int32_t> lags;
  std::vector<dd::IqrmSeg> segs;
  int iqrm_variant = 0;
  std::vector<int32_t> bad;

  // device state
  dd::DevBuf d_delay, d_res, d_lags, d_bad_keep, d_win, d_seg_t0;
  dd::DevBuf d_binned;   // binned / working copy of the input [nbin][nchans]
  dd::DevBuf d_x;        // prepared channel-major input
  dd::DevBuf d_xlimit;   // PrepArgs::limit (empty: the sums read all of d_x)
  dd::DevBuf d_host_in, d_host_out;  // device side of dd_run_host (kept across calls)
  cudaStream_t copy_stream = nullptr; // dd_run_host: output copies overlapping the sums
  cudaEvent_t host_done = nullptr;    // the last host-path output copy enqueued
  bool host_pending = false;          // host_done marks copies a later run must wait for
  std::vector<cudaEvent_t> host_tile_copied;  // per time tile: its output copy of the last run
  int64_t host_tile = 0;                      // the time tile those copies were made with
  dd::DevBuf d_inter;    // stage-1 tile, then its twin
  dd::DevBuf d_bin_lut;  // full-bin values of the time binning (8/16-bit samples, ds > 1)
  int64_t inter_bytes = 0; // bytes of one buffer
  int64_t inter_budget = 0; // subband-sum bytes per time tile the tiling was set for
  int stages_override = 0;  // staged source pairs in flight (0: as many as fit)
  dd::DevBuf d_stats;    // IQRM sums [nwin][2][csub] uint64
  dd::DevBuf d_iqrm_scratch;
  dd::DevBuf d_masks;    // IQRM window masks [nwin][nchans]
  dd::DevBuf d_segmask;  // [nseg][nchans]
  dd::DevBuf d_zdm;      // per-sample zero-DM offsets [nbin]
  dd::DevBuf d_skew1;                    // row skews of stage 1 (SumLaunch::skew)
  dd::DevBuf d_desc1, d_desc2, d_descb;  // staging descriptors: stage 1, stage 2, brute force
  dd::DevBuf d_err;      // device error word of the staged sums (0: no error)
  double adds = 0;
  int64_t generation = 0;  // bumped whenever device tables are replaced
  std::vector<cudaEvent_t> events;  // timing events of dd_run_profiled
  ~dd_plan() {
    for (cudaEvent_t e : events) cudaEventDestroy(e);
    if (copy_stream) {
      cudaStreamSynchronize(copy_stream);
      cudaStreamDestroy(copy_stream);
    }
    if (host_done) cudaEventDestroy(host_done);
    for (cudaEvent_t e : host_tile_copied) cudaEventDestroy(e);
  }
};

namespace dd {

// ---- fast-math translation unit (dd_fastmath.cu) ----
void launch_subband_tables(const double* d_freq, int64_t cs, int64_t ce, float dm_low,
                           float dm_step, int64_t dm_steps, int sbw, int ndm0, float ref_freq,
                           double tsamp, int ds, int32_t* d_delay1, int32_t* d_res,
                           cudaStream_t st);
// mean_ws: device workspace of chan_end floats.
void launch_zero_dm_callsite(void* data, int nbits, size_t chan_start, size_t chan_end,
                             size_t down_ndata, float* mean_ws, cudaStream_t st);
// Per-sample float mean of the non-zero (after the IQRM segment masks) values of
// channels [cs, ce), in the arithmetic of the reference's range kernels.
void launch_zdm_range_mean(const void* x, int nbits, int64_t nsamp, int64_t nchans, int64_t cs,
                           int64_t ce, const uint8_t* d_segmask, const uint32_t* d_seg_t0,
                           int nseg, float* d_mean, cudaStream_t st);

// ---- RFI and layout (dd_rfi.cu) ----
// Time binning (dedispered.cu:337-376).  lut: the plan's table of full-bin values
// (launch_binning_lut; nullptr evaluates every bin directly).
void launch_time_binning(const void* in, void* out, int nbits, int64_t ndata, int64_t nchans,
                         int ds, const void* lut, cudaStream_t st);
// Entries of the full-bin table for these samples and bin width (0: no table).
int64_t binning_lut_entries(int nbits, int ds);
// Fills the full-bin table: lut[sum] for every sum of ds samples.
void launch_binning_lut(void* lut, int nbits, int ds, cudaStream_t st);
// d_win: [nwin][2] (t0, t1); d_sums: [nwin][2][csub] (sum, sum of squares).
void launch_iqrm_stats(const void* x, int nbits, int64_t nsamp, int64_t nchans, int64_t cs,
                       int64_t csub, const uint32_t* d_win, int nwin,
                       unsigned long long* d_sums, cudaStream_t st);
size_t iqrm_scratch_bytes(int nwin, int64_t csub, int nlags);
// Throws DD_ERR_INVALID when csub channels exceed what the statistics and votes of
// one window may hold in shared memory on the current device.
void check_iqrm_channels(int64_t csub);
void launch_iqrm_decide(const unsigned long long* d_sums, int nwin, const uint32_t* d_win,
                        int64_t nchans, int64_t cs, int64_t csub, int mode, float nsigma,
                        const int32_t* d_lags, int nlags, int variant, void* scratch,
                        uint8_t* d_masks, cudaStream_t st);
void launch_segment_masks(const uint8_t* d_masks, int nwin, const uint32_t* d_win,
                          const uint32_t* d_seg_t0, int nseg, int64_t nchans,
                          uint8_t* d_segmask, cudaStream_t st);
void launch_apply_masks_inplace(void* x, int nbits, int64_t nsamp, int64_t nchans,
                                const uint8_t* d_segmask, const uint32_t* d_seg_t0, int nseg,
                                cudaStream_t st);
void launch_zdm_offsets(const void* x, int nbits, int64_t nsamp, int64_t nchans, int64_t cs,
                        int64_t ce_excl, const uint8_t* d_segmask, const uint32_t* d_seg_t0,
                        int nseg, uint32_t* d_off, cudaStream_t st);
struct PrepArgs {
  const void* x;           // [nsamp][nchans] input (binned)
  int nbits;
  int64_t nsamp, nchans;
  const uint8_t* segmask;  // nullptr: no IQRM masking in this pass
  const uint32_t* seg_t0;
  int nseg;
  const uint32_t* zdm_off; // nullptr: no zero-DM subtraction in this pass
  const float* zdm_mean;   // per-sample float mean (DD_ZDM_RANGE_REF), or nullptr
  int64_t zdm_cs, zdm_ce;  // channel range the zero-DM offset applies to
  const uint8_t* keep;     // nullptr: no static mask
  // channel-major output: out[(c - c0) * rows_per_chan + phase][q] with
  // q = t / ds, phase = t % ds (ds = 1 for the subband layout)
  void* out;
  int64_t c0, c1;          // channels [c0, c1)
  int ds;
  int64_t pitch;           // elements per output row
  // folded layout (fold 4 or 2): out[(c - c0)][s] = the samples s, s + seg, ... of the
  // channel in one 32-bit word, words [0, nwords)
  int fold;
  int64_t seg, nwords;
  // per 64 channels from c0 & ~3 on: positions from here on are read by no sum and may be
  // left out (nullptr: write them all)
  const int64_t* limit;
  void* full_out;          // optional [nsamp][nchans] copy after all stages
};
void launch_prep(const PrepArgs& a, cudaStream_t st);

// ---- dedispersion sums (dd_dedisp.cu) ----
struct Stage1Args {
  const void* x;           // channel-major input, row pitch xpitch (elements)
  int64_t xpitch;
  int nbits;
  const int32_t* delay1;   // [ndm_nom][dch]
  int64_t dch, nsb, ndm_nom;
  int sbw;
  int64_t t0;              // absolute start sample of the tile
  int64_t ncols;           // columns of inter to compute
  void* inter;             // [ndm_nom][nsb][tile_pitch]
  int64_t tile_pitch;
  int inter16;
};
void launch_stage1(const Stage1Args& a, cudaStream_t st);
struct Stage2Args {
  const void* inter;
  int64_t tile_pitch;
  int inter16;
  const int32_t* res;      // [dm_steps][nsb]
  int64_t nsb, dm_steps;
  int ndm0;
  int64_t ncols;           // output columns of this tile
  void* out;               // row m at out + m*out_pitch + col0
  int64_t out_pitch, col0;
  int out64;
  int sbw;
  int src_max;             // largest value one inter element can hold
};
void launch_stage2(const Stage2Args& a, cudaStream_t st);
struct BruteArgs {
  const void* x;           // phase layout [nc][ds][phase_len]
  int64_t phase_len;
  int ds;
  int nbits;
  const int32_t* delay;    // [dm_steps][nc]
  int64_t nc, dm_steps;
  int64_t start;           // first input sample of the slice
  int64_t ncols;           // columns of this slice
  void* out;
  int64_t out_pitch, col0;
  int out64;
};
void launch_brute(const BruteArgs& a, cudaStream_t st);

// Allows `kernel` `dynamic_smem` bytes of dynamic shared memory: above 48 KB per
// block, counting the kernel's static shared memory, a launch needs the opt-in.
template <typename K>
inline void allow_dynamic_smem(K kernel, size_t dynamic_smem) {
  if (dynamic_smem == 0) return;
  cudaFuncAttributes fa{};
  DD_CUDA_TRY(cudaFuncGetAttributes(&fa, reinterpret_cast<const void*>(kernel)));
  if (dynamic_smem + fa.sharedSizeBytes > 48 * 1024)
    DD_CUDA_TRY(cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel),
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     static_cast<int>(dynamic_smem)));
}

// ---- shared-memory staged sums (dd_sumsmem.cu) ----
// Output rows per block.  A staged window serves all of them, so the traffic from L2
// into shared memory falls with their number; rows are split over warp groups that
// each cover the whole tile (kSumRowsPT* rows per thread).
constexpr int kSumRows = 16;
constexpr int kSumRowsPT8 = 4, kSumRowsPTW = 8, kSumRowsPTT = 4;
// Staging descriptor of one (row group, source) pair of a staged sum: the
// smallest offset of the group's rows for that source, the spread of their
// offsets, and each row's offset relative to the smallest.  Built on the host
// from the plan's tables; the kernels read one per source and row group.
struct SumDesc {
  int32_t lo;
  int32_t span;
  uint16_t rel[kSumRows];
  uint32_t phase[2];  // downsampled brute force: four bits per row, its delay's phase
};
static_assert(sizeof(SumDesc) == 48, "bulk copies move whole 16-byte units");
struct SumLaunch {
  enum Mode { kStage1 = 0, kStage2 = 1, kBrute = 2 };
  int mode;
  int kind;                // SumKind
  const char* src;         // byte address of source row 0
  int64_t src_pitch;       // bytes between source rows
  int64_t base;            // element index added to every offset
  int64_t valid;           // source elements from here on are zero: windows starting there are skipped
  int64_t max_off;         // largest offset of any row and source
  int64_t nsrc_total;      // stage 1: channels of the band; stage 2: subbands; brute: channels
  int64_t nrows_total;     // stage 1: nominal DMs; stage 2 and brute: DM trials
  int group;               // stage 1: subband width; stage 2: fine DMs per nominal DM
  int64_t nsb_out;         // stage 1: subbands (inter rows are (j, sb))
  char* out;               // byte address of output row 0, column 0
  int64_t out_pitch;       // bytes between output rows (stage 1: between (j, sb) rows)
  int64_t out_col0;        // first output column of the launch (elements)
  int out_elem;            // bytes per output element
  int64_t ncols;           // columns of the launch
  int win_bytes;           // bytes of one staged source window
  // Folded sums: bytes between the segments' (or packed planes') outputs of stage 1
  // and brute force; bytes between the planes stage 2 reads; columns per segment and
  // of the chunk where the sums go to the output (seg 0: into planes).
  int64_t seg_stride, plane_bytes, seg, nout;
  unsigned grid_y, grid_z;
  const SumDesc* desc;     // [grid_y][desc_pitch] staging descriptors
  int64_t desc_pitch;      // descriptors per row group (= columns of the offset table)
  // Stage 1: row r of group y and subband sb computes column u - skew of its row at
  // position u of the launch, skew[(y * nsb_out + sb) * kSumRows + r] (see
  // skew_stage1); the launch spans ncols + max_skew positions.
  const int32_t* skew;
  int64_t max_skew;
  // Downsampled brute force (ds > 1): grid z = slice of sps samples of the chunk's nin;
  // a source is ds phase rows (samples ph, ph + ds, ... of the channel) phase_pitch bytes
  // apart, staged in parts of sub_bytes; desc has a table of desc_pattern descriptors for
  // every first sample of a slice modulo ds.
  int ds, sub_bytes;
  int64_t sps, nin, phase_pitch, desc_pattern;
  int stages;              // groups of sources in flight (2..kSumMaxStages)
  int* err;                // device error word: set when a bounded wait gives up
  // 16-bit subband sums with a one-sample-shifted twin (0: none): the twin of the
  // element at byte address a sits at a + twin_off and holds the element before
  // it, twin[i] = sums[i - 1].  Stage 1 writes both; stage 2 reads a source whose
  // offset is odd from the twin, so every read is a whole aligned word.
  int64_t twin_off;
};
#ifndef DD_SUM_MAX_STAGES
#define DD_SUM_MAX_STAGES 8
#endif
// Shared memory (KB) the staged sums stay within by default: two blocks per SM.
#ifndef DD_SUM_SMEM_KB
#define DD_SUM_SMEM_KB 100
#endif
constexpr int kSumMaxStages = DD_SUM_MAX_STAGES;  // groups of sources in flight, at most
// Shared memory a block may have (227 KB on sm_100), and an upper bound of what the
// staged-sum kernels declare statically (checked in dd_sumsmem.cu).
constexpr size_t kSumBlockSmem = 227 * 1024;
constexpr size_t kSumStaticSmem = 3072;
void launch_sum(const SumLaunch& L, cudaStream_t st);
int sum_tile_samples(int src_bytes, int nw);
// Shared memory of a staged sum with `stages` pairs in flight.
// qs: source windows per pipeline stage.
size_t sum_smem_bytes(int win_bytes, int stages, int qs = 2);
// Pairs in flight that fit the shared memory of two blocks per SM (at least 2),
// next to `extra` bytes the kernel needs besides its ring (cap_kb: the shared
// memory to stay within, 0 for the default).
int sum_stages(int win_bytes, int qs = 2, size_t extra = 0, int cap_kb = 0);
// Stages of a kernel variant for a window size (its windows per stage, staging
// and shared-memory cap).
int sum_kind_stages(int kind, int win_bytes);
// Descriptors of a [nrows][ncols] offset table for row groups of `rows` rows,
// grouped within blocks of `group` rows (0: one block), in the launch's
// blockIdx.y order, and the largest spread of a group's offsets (a window that holds
// more than 65535 never fits shared memory, window_bytes).
std::vector<SumDesc> build_sum_desc(const std::vector<int32_t>& tab, int64_t nrows,
                                    int64_t ncols, int64_t group, int* spread, int rows = kSumRows);
// Device error codes of the staged sums.
constexpr int kErrWaitFull = 1;   // a consumer gave up waiting for a staged window
constexpr int kErrWaitEmpty = 2;  // the producer gave up waiting for a free stage
// Words per lane of the staged sums (an odd number of consecutive words for 8- and
// 16-bit samples, interleaved words for the others) and blocks per SM they are
// compiled for (register budget).
#ifndef DD_SUM8_NW
#define DD_SUM8_NW 9
#endif
#ifndef DD_SUM8_MINB
#define DD_SUM8_MINB 2
#endif
#ifndef DD_SUM16W_NW
#define DD_SUM16W_NW 5
#endif
#ifndef DD_SUM16W_MINB
#define DD_SUM16W_MINB 2
#endif
#ifndef DD_SUM16T_NW
#define DD_SUM16T_NW 6
#endif
constexpr int kSum16TNW = DD_SUM16T_NW;
#ifndef DD_PHASE8_NW
#define DD_PHASE8_NW 7
#endif
// Downsampled brute force: slices of half a second are a few thousand columns, so a block
// tile takes fewer words than the chunk-long sums (1000 channels, 61,441 samples, bins of
// two, 501 trials: 5 / 7 / 9 words 1.31 / 1.19 / 1.46 ms).
constexpr int kPhase8NW = DD_PHASE8_NW;
constexpr int kFlush8R8NW = 7;
// Folded sums: rows per thread, words per lane and blocks per SM.  Few rows of many
// words: a row of a stage costs one load of its offsets and four addresses whatever its
// words.  Measured (4096 channels, 2^17 samples, 6001 trials, stage 1 / stage 2, ms; and
// brute force, 1024 channels, 1001 trials): rows x words 8 x 5 4.83 / 3.61, 5.81;
// 4 x 10 4.52 / 3.46, 5.40; 2 x 20 4.44 / 3.41, 5.54; 2 x 12 at three blocks per SM
// 4.86 / 3.49, 7.04.  16-bit samples (8192 channels, 2001 trials): 8 x 5 and 8 x 8
// 10.2 / 8.11, 2 x 20 and 2 x 32 9.36 / 7.81.
#ifndef DD_FOLD8_RB
#define DD_FOLD8_RB 2
#endif
#ifndef DD_FOLD8_NW
#define DD_FOLD8_NW 20
#endif
#ifndef DD_FOLD8W_RB
#define DD_FOLD8W_RB 4
#endif
#ifndef DD_FOLD8W_NW
#define DD_FOLD8W_NW 10
#endif
#ifndef DD_FOLD8_MINB
#define DD_FOLD8_MINB 2
#endif
#ifndef DD_FOLD16_RB
#define DD_FOLD16_RB 2
#endif
#ifndef DD_FOLD16_NW
#define DD_FOLD16_NW 20
#endif
#ifndef DD_FOLD16_MINB
#define DD_FOLD16_MINB 2
#endif
#ifndef DD_PLANE16_RB
#define DD_PLANE16_RB 2
#endif
#ifndef DD_PLANE16_NW
#define DD_PLANE16_NW 20
#endif
#ifndef DD_PLANE16_MINB
#define DD_PLANE16_MINB 2
#endif
#ifndef DD_PLANE32_RB
#define DD_PLANE32_RB 2
#endif
#ifndef DD_PLANE32_NW
#define DD_PLANE32_NW 32
#endif
#ifndef DD_PLANE32_MINB
#define DD_PLANE32_MINB 2
#endif
constexpr int kFold8RB = DD_FOLD8_RB, kFold8NW = DD_FOLD8_NW;
constexpr int kFold8WRB = DD_FOLD8W_RB, kFold8WNW = DD_FOLD8W_NW;
constexpr int kFold16RB = DD_FOLD16_RB, kFold16NW = DD_FOLD16_NW;
constexpr int kPlane16RB = DD_PLANE16_RB, kPlane16NW = DD_PLANE16_NW;
constexpr int kTo64RB = 2, kTo64NW = 16;
constexpr int kPlane32RB = DD_PLANE32_RB, kPlane32NW = DD_PLANE32_NW;
// Kernel variants of the staged sums.  Samples in time order: 8-bit into 16-bit sums
// (U8Out16) or 32-bit sums (U8Flush), 16-bit into 32-bit sums (U16Wide), 16-bit subband
// sums with their one-sample-shifted twin (U16Twin), and the phase rows of downsampled
// brute force (U8Phase, U16Phase).  Folded samples: 8-bit into
// packed 16-bit planes (Fold8) or 32-bit sums (Fold8W), 16-bit into 32-bit sums
// (Fold16), and stage 2 of packed planes (Plane16).  Stage 2 of 32-bit sums, folded or
// not (Plane32).  32-bit samples into 64-bit sums and stage 2 of those (Word64, Plane64;
// not in batched launches).
enum SumKind { kSumKindU8Out16, kSumKindU8Flush, kSumKindU16Wide, kSumKindU16Twin,
               kSumKindU8Phase, kSumKindU16Phase, kSumKindFold8,
               kSumKindFold8W, kSumKindFold16, kSumKindPlane16, kSumKindPlane32,
               kSumKindFold8S, kSumKindFold8WS, kSumKindFold16S, kSumKindPlane16S, kSumKindPlane32S,
               kSumKindWord64, kSumKindPlane64,
               kSumKindU8Out16R8, kSumKindU8FlushR8, kSumKindU16WideR8, kSumKindU16TwinR8,
               kSumKindPlane32R8, kSumKinds };
// The folded variants and Plane32 have a second form with tiles of half the words (S) for
// launches that do not fill the GPU: a launch of fewer blocks than four per SM is bound by
// the latency of one block.  336 channels, 5120 samples, 591 trials: 32.9 -> 24.8 us a
// run (quarter tiles 27.0); at 4096 channels, 2^17 samples whole tiles are 5 % faster.
inline int sum_kind_small(int kind) {
  return kind >= kSumKindFold8 && kind <= kSumKindPlane32 ? kind + (kSumKindFold8S - kSumKindFold8) : kind;
}
constexpr long long kSumSmallBlocks = 4 * 148;
// Time-order variants of eight rows a block (R8), on tiles twice as long (U8FlushR8: seven
// words a lane, so that its staging past the ring leaves room for wider windows).  A
// window holds the spread of its rows' delays, which grows with the trial step, and half the
// rows spread half as far: where sixteen rows' windows pass shared memory these serve
// instead of the direct kernels.  1024 channels, 2^17 samples, 96 brute-force trials:
// 8 bits, 16-row spread 37,300 samples 10.4 -> 1.23 ms; 16 bits, 19,400 samples 11.9 -> 2.0
// ms; stage 2 of 16-bit samples, 512 trials spreading over 4,900 samples per 16 2.10 -> 0.31
// ms.  Stage 2 takes them already where 16 rows spread over more than two tiles: both
// forms then stage as many bytes per addition, and wide windows leave fewer blocks per SM
// (16 rows / 8 rows: twin, 2,820 samples 0.55 / 0.32 ms; 32-bit sums 0.38 / 0.30).
inline int sum_kind_rows8(int kind) {
  switch (kind) {
    case kSumKindU8Out16: return kSumKindU8Out16R8;
    case kSumKindU8Flush: return kSumKindU8FlushR8;
    case kSumKindU16Wide: return kSumKindU16WideR8;
    case kSumKindU16Twin: return kSumKindU16TwinR8;
    case kSumKindPlane32: case kSumKindPlane32S: return kSumKindPlane32R8;
    default: return kind;
  }
}
// Output rows of a block.
inline int sum_kind_rows(int kind) { return kind >= kSumKindU8Out16R8 ? 8 : kSumRows; }
int sum_kind(const SumLaunch& L);
// Tile of a kernel variant: samples per block, or words for the folded sums and Plane32.
inline int sum_kind_tile(int kind) {
  const auto words = [](int rb, int nw) { return sum_tile_samples(4, nw) * rb / kSumRows; };
  switch (kind) {
    case kSumKindU8Phase: return sum_tile_samples(1, kPhase8NW) * kSumRowsPT8 / kSumRows;
    case kSumKindU8Out16: case kSumKindU8Flush:
      return sum_tile_samples(1, DD_SUM8_NW) * kSumRowsPT8 / kSumRows;
    case kSumKindU16Wide: case kSumKindU16Phase: return sum_tile_samples(2, DD_SUM16W_NW) * kSumRowsPTW / kSumRows;
    case kSumKindU16Twin: return sum_tile_samples(2, kSum16TNW) * kSumRowsPTT / kSumRows;
    case kSumKindFold8: return words(kFold8RB, kFold8NW);
    case kSumKindFold8W: return words(kFold8WRB, kFold8WNW);
    case kSumKindFold16: return words(kFold16RB, kFold16NW);
    case kSumKindPlane16: return words(kPlane16RB, kPlane16NW);
    case kSumKindFold8S: return words(kFold8RB, kFold8NW / 2);
    case kSumKindFold8WS: return words(kFold8WRB, kFold8WNW / 2);
    case kSumKindFold16S: return words(kFold16RB, kFold16NW / 2);
    case kSumKindPlane16S: return words(kPlane16RB, kPlane16NW / 2);
    case kSumKindPlane32S: return words(kPlane32RB, kPlane32NW / 2);
    case kSumKindWord64: case kSumKindPlane64: return words(kTo64RB, kTo64NW);
    case kSumKindU8Out16R8: return sum_tile_samples(1, DD_SUM8_NW) * kSumRowsPT8 / 8;
    case kSumKindU8FlushR8: return sum_tile_samples(1, kFlush8R8NW) * kSumRowsPT8 / 8;
    case kSumKindU16WideR8: return sum_tile_samples(2, DD_SUM16W_NW) * kSumRowsPTW / 8;
    case kSumKindU16TwinR8: return sum_tile_samples(2, kSum16TNW) * kSumRowsPTT / 8;
    case kSumKindPlane32R8: return sum_tile_samples(4, kPlane32NW) * kPlane32RB / 8;
    default: return words(kPlane32RB, kPlane32NW);
  }
}
// Source windows per pipeline stage of a kernel variant.
inline int sum_kind_qs(int kind) {
  if (kind == kSumKindU16Twin || kind == kSumKindU16TwinR8) return 8;
  return kind >= kSumKindFold8 && kind < kSumKindU8Out16R8 ? 4 : 2;
}
// Bytes of a source element: samples, 16-bit sums or words.
inline int sum_kind_elem(int kind) {
  switch (kind) {
    case kSumKindU8Out16: case kSumKindU8Flush: case kSumKindU8Phase:
    case kSumKindU8Out16R8: case kSumKindU8FlushR8: return 1;
    case kSumKindU16Wide: case kSumKindU16Twin: case kSumKindU16Phase:
    case kSumKindU16WideR8: case kSumKindU16TwinR8: return 2;
    case kSumKindPlane64: return 8;
    default: return 4;
  }
}
// Shared memory of a launch (its variant's windows per stage, plus the variant's
// staging past the ring, sum_kind_extra_smem).
size_t sum_launch_smem(const SumLaunch& L);
size_t sum_kind_extra_smem(int kind);
unsigned sum_grid_x(const SumLaunch& L);
// One group of a batched (persistent) launch: all blocks of one staged sum.
struct SumBatchGroup {
  SumLaunch L;
  int kind;
  unsigned gx;           // blocks along x (time tiles)
  long long first;       // index of the group's first block in the batch
  int wait_ctr;          // counter to wait for (-1: none)
  int wait_need;         // ... until it reaches this value
  int done_ctr;          // counter each finished block increments
  int pad;
};
constexpr int kErrWaitGroup = 3;  // a batched group gave up waiting for its inputs
int sum_batch_blocks_per_sm(size_t smem);
// Persistent launch over groups (dependent stages ordered by counters).
void launch_sum_batch(const SumBatchGroup* d_groups, int ngroups, long long total, int* d_ctrs,
                      unsigned long long* d_next, int* d_err, size_t smem, unsigned grid,
                      cudaStream_t st);
// Grouped launch: one grid over independent groups of one variant (`kind`).
void launch_sum_grouped(const SumBatchGroup* d_groups, int ngroups, long long total, int kind,
                        size_t smem, cudaStream_t st);

// ---- brute-force table in the reference's host arithmetic (dd_hosttable.cpp) ----
void brute_delay_table_fastmath(const double* freq, size_t chan_start, size_t chan_end,
                                float dm_low, float dm_step, size_t dm_steps,
                                float ref_freq_value, double tsamp, int32_t* table);

// ---- probes (dd_probe.cu) ----
double measure_int_add_rate(int device);

}  // namespace dd
