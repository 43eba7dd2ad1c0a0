// Host-side launchers for the frontier-DP kernels (dispatch on index width and
// on K = residues interleaved per state).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "fdp_item.cuh"

namespace fdp {

constexpr int kMaxLanes = 16;  // K = 1..16 residues interleaved per state
constexpr int kCarryItems = 16;  // default states per lane of a grouped chunk with carry-over queues

// Where the streaming cells of a span of K lanes go run by run (cell_run_kernel)
// instead of item by item: from `from` to below `below` items per resident thread.
// A run shares one decode and one closure scan among its items, but three CTAs per
// SM hold less in flight than the item kernel's four to six, and a chunk of one or
// two items a lane has nothing to share.  Cells p >= 9 of a row, item by item and
// run by run, in ms:
//   lanes      n = 14        16          18          20           22
//   1       0.071 0.090  0.320 0.339  1.82 1.62  11.7 10.1   99.3  83.2
//   2       0.074 0.090  0.336 0.389  2.14 2.30  14.0 15.3  118   127
//   3       0.086 0.089  0.492 0.434  3.35 2.91  21.4 21.2  177   184
//   4       0.077 0.087  0.456 0.515  2.81 3.12  20.4 22.8  178   196
//   5       0.091 0.090  0.735 0.592  3.90 3.38  29.8 25.8  262   228
//   6       0.091 0.092  0.738 0.658  3.89 3.71  29.8 29.1  270   264
//   7       0.095 0.100  0.815 0.831  4.47 4.75  35.7 36.2  329   324
//   8       0.094 0.096  0.803 0.786  4.53 4.58  36.6 36.2  331   326
// 64-bit ranks (n = 23), where a decode costs twice the instructions: 1 lane 385
// 238, 2 428 390, 3 585 553, 4 572 590, 5 714 684; six lanes do not fit a device.
// 7 lanes stay with items: equal at n = 21 (106.8 106.7), ahead by runs at 22 alone.
struct RunsRange {
  uint64_t from, below;
};
constexpr RunsRange runs_range(bool u64, int K) {
  constexpr uint64_t all = ~uint64_t(0);
  if (u64) return K == 1 || K == 2 || K == 3 || K == 5 ? RunsRange{0, all} : RunsRange{0, 0};
  switch (K) {
    case 1: return {16, all};   // n >= 17 (0.682 0.622 there)
    case 3: return {0, 1024};   // n <= 20 (n = 21 59.8 61.4)
    case 5:
    case 6: return {0, all};
    case 8: return {8, all};    // n >= 16 (n = 15 0.196 0.204)
    default: return {0, 0};
  }
}

// Per-(width, height cap) device table blob.
struct DevTables {
  void *ptr = nullptr;
  bool u64 = false;
  int W = 0;
  int cap = 1000;  // FDP_FULL_CAP: the full space
};
cudaError_t upload_tables(int W, int cap, DevTables *out);
void free_tables(DevTables *t);

struct LaunchCfg {
  int block = 256;
  int grid = 0;              // 0: sized from occupancy (a multiple of the SM count)
  bool split_panels = false; // several panels: one single-panel launch per panel
  bool bounded_prefix = true;  // first rows in height-bounded spaces
  int lane_items = 8;        // items per lane of a warp chunk of the cell kernel
  int share_min = 4;         // share the chunk's prefix decode when it walks >= this many positions
  int compact_max_p = 7;     // cells p <= this update a chunk's items grouped by centre type (-1: never)
  int compact_items = 0;     // states per lane of a compacted chunk (without carry-over 1..FDP_REC_MAX_ITEMS;
                             // 0: 4 for one span, 2 when closure sources are staged, which leaves L1
                             // room; with carry-over 1..16, 0: kCarryItems)
  int compact_carry = 0;     // grouped cells queue heads across chunks so every update runs 32 items
                             // (1 on, -1 off, 0 automatic: on when the lanes fit one span)
  int row_init = 0;          // strip rows filled directly by the row-k initialiser (0: automatic, -1: never)
  bool row_init_tensor = true;  // the initialiser's products on the tensor cores (else the CUDA cores)
  int split_spans_min_p = 1;    // cells p >= this run each span of a several-span lane count as its own launch
  bool tail = true;  // cells s-1..1 of a full-space row as one fused pass where escape memory is at hand (fdp_tail.h)
  bool span_chains = true;  // with every cell split, each span's row sweeps run as a chain of launches of
                            // their own, concurrent with the other span's (n=22, 14 lanes: pass 17.20 -> 16.83 s)
};

template <typename Idx, int K>
cudaError_t launch_cell_t(const CellArgs &a, const LaunchCfg &cfg, cudaStream_t s);
template <typename Idx, int K>
cudaError_t launch_first_row_t(const FirstRowArgs &a, bool dot, cudaStream_t s);

// One cell p on [M][K] / [D][K] arrays: one kernel launch, or one per lane
// span or panel when the configuration splits them; *kernels (if given) is
// increased by the launches made.
cudaError_t launch_cell(const DevTables &t, int K, const uint32_t *mods, uint32_t *main, uint32_t *blk, int p,
                        bool blk_in_zero, bool blk_out_p1, const LaunchCfg &cfg, cudaStream_t s,
                        uint64_t *kernels = nullptr);
// main[rank(first-row state)] = 1 for every first-row mask.
cudaError_t launch_first_row_init(const DevTables &t, int K, uint32_t *main, cudaStream_t s);
// acc[k] += sum over first-row states of main[.][k]; then residues[k] = acc[k] mod p_k.
cudaError_t launch_first_row_dot(const DevTables &t, int K, const uint32_t *mods, const uint32_t *main,
                                 unsigned long long *acc, uint32_t *residues, cudaStream_t s);

// Every word of the K lanes of the first N states set to 1 (row 0 in the
// height-1 space: every such word is a first-row state with coefficient 1).
cudaError_t launch_fill_ones(uint32_t *a, uint64_t words, cudaStream_t s);
// Move a K-lane state vector, in place, from the space `from` to the larger
// space `to` of the same width (ranks only grow), staging through `tmp`
// (tmp_words words, not overlapping `a`); words of `to` outside the image are
// zeroed.
cudaError_t enqueue_expand(const DevTables &from, const DevTables &to, int K, uint32_t *a, uint32_t *tmp,
                           uint64_t tmp_words, cudaStream_t s, uint64_t *launches = nullptr);

// Upload (once per device) the count tables enqueue_expand uses for these caps;
// must run outside stream capture.
cudaError_t prepare_expand_tables(const std::vector<int> &caps);

// Operator-surface helpers.
cudaError_t launch_rank_words(int width, const uint64_t *words, uint64_t *ranks, uint64_t count, cudaStream_t s);
cudaError_t launch_unrank_words(int width, const uint64_t *ranks, uint64_t *words, uint64_t count, cudaStream_t s);
cudaError_t launch_ternary_index(const uint32_t *codes, uint32_t *index, uint64_t count, cudaStream_t s);
cudaError_t launch_ternary_index_chunked(int chunk, const uint32_t *codes, uint32_t *index, uint64_t count,
                                         cudaStream_t s);

int device_sm_count();

// While it lives, this thread's allocations, blocking copies, event queries and
// loads of kernels do not invalidate a capture that runs on another stream (of any
// thread, in any mode): what a call sets up on first use must not depend on who
// captures meanwhile.
struct BesideCaptures {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  BesideCaptures() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~BesideCaptures() { cudaThreadExchangeStreamCaptureMode(&mode); }
  BesideCaptures(const BesideCaptures &) = delete;
  BesideCaptures &operator=(const BesideCaptures &) = delete;
};

#if defined(__CUDACC__)
// Small launches of one chain overlap at their seams: a kernel launched with
// `overlap` starts once the CTAs of the one before it have all started, if there
// is room, sets up what no kernel writes (tables), and waits with chain_wait for
// the one before it to end before it touches a state.  Every CTA of a chained
// kernel calls both.  The line is a grid of three quarters of the resident CTAs,
// where the next one's first CTAs find room: width 14 x 16 lanes, cells 13..6,
// 159 -> 114 us; a full grid's early successors only hold room that its own CTAs
// and other streams could use (n = 20 x 4 409 -> 458 ms).
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename Kernel, typename Args>
cudaError_t launch_chained(Kernel kernel, unsigned grid, unsigned block, size_t smem, cudaStream_t s, const Args &args,
                           bool overlap) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args);
}
#endif

}  // namespace fdp
