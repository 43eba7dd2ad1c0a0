// Context object behind the opaque fdp_ctx handle.
#pragma once
#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <vector>

#include "../../include/oneesan_fdp.h"
#include "fdp_launch.h"

// A window of fdp_apply_cells that took escape words: they are free for other
// streams when `done` has been reached.
struct WindowUse {
  cudaStream_t stream;
  cudaEvent_t done;
  size_t bytes;
};

struct fdp_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  std::map<int, fdp::DevTables> tables;  // per frontier width
  uint32_t *d_main = nullptr;            // run_sync state, [M][lanes]
  uint32_t *d_blk = nullptr;             // run_sync state, [D][lanes]
  char *d_side = nullptr;                // what a synchronous call takes beside its state
  size_t cap_main = 0, cap_blk = 0, cap_side = 0;
  cudaMemPool_t pool = nullptr;          // escape words of windows, large side memory; stream-ordered
  std::vector<WindowUse> windows;        // those whose pool memory may still be in use
  unsigned long long *d_acc = nullptr;   // first-row dot accumulators
  uint32_t *d_res = nullptr;             // residues on the device
  uint32_t *h_res = nullptr;             // residues, pinned host
  unsigned int *d_err = nullptr;         // run_sync pass error word (device)
  unsigned int *h_err = nullptr;         // its copy after the pass (pinned host)
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  // A second stream for the sweep of the second lane span (lanes 8..): the
  // spans touch disjoint panels, so their cell launches run as two chains.
  cudaStream_t span_stream = nullptr;
  cudaEvent_t span_fork = nullptr, span_join = nullptr;
  // fdp_run_multi_sync's pinned results and the streams and events of its problems.
  uint32_t *h_multi = nullptr;
  size_t cap_hmulti = 0;  // words
  std::vector<cudaStream_t> multi_streams;
  std::vector<cudaEvent_t> multi_events;
  fdp::LaunchCfg cfg;
  std::mutex mu;         // serialises run_sync / apply_cells / time_cells / tuning
  std::mutex tables_mu;  // guards `tables` (also used by the serving thread)
  struct fdp_server *server = nullptr;  // request loop (fdp_server_start)
  ~fdp_ctx();
};

fdp_status fdp_ctx_tables(fdp_ctx *c, int W, const fdp::DevTables **out);
fdp_status fdp_ctx_tables_cap(fdp_ctx *c, int W, int cap, const fdp::DevTables **out);
cudaError_t fdp_ctx_malloc(fdp_ctx *c, void **p, size_t bytes);
fdp_status fdp_prepare_pass(fdp_ctx *c, int W, const fdp::DevTables **full);
// One residue pass of L lanes on stream s.  esc: fdp::tail_escape_words(W) x L
// words for the fused row tail, or null to run every cell as its own launch.  With span_stream (and fork /
// join events) given, a pass of more than 8 lanes sweeps its second lane span
// on that stream, concurrently with the first on s.
fdp_status fdp_enqueue_pass(fdp_ctx *c, const fdp::DevTables &t, int L, const uint32_t *mods, uint32_t *main,
                            uint32_t *blk, uint32_t *esc, unsigned long long *acc, uint32_t *d_res, uint32_t *h_res,
                            unsigned int *d_err, cudaStream_t s, uint64_t *launches,
                            cudaStream_t span_stream = nullptr, cudaEvent_t fork = nullptr,
                            cudaEvent_t join = nullptr);
// Residues a pass of fdp_run_sync holds when `lanes` are asked for.
int fdp_pass_lanes(fdp_ctx *c, int n, int lanes);
// Whether its pass is one launch, which reads no tuning of the cell kernels.
bool fdp_pass_is_whole(fdp_ctx *c, int n);
// Every cell its own launch, whatever the width and the memory.
void fdp_pass_single_cells(fdp_ctx *c, bool on);
// Time of a row of one pass of pr->lanes residues as fdp_run_sync runs it: from a
// graph, the low cells fused where that pass would fuse them, after an untimed run.
// A pass of one launch counts as sweep_rows rows.
fdp_status fdp_time_pass_row(fdp_ctx *c, const fdp_problem *pr, double *row_ms);
// A computation's error word: a kernel that gives up on a bounded wait writes
// a nonzero value to it.  Each computation (a run_sync graph, one problem of a
// run_multi_sync graph, one served request) owns its word in its own buffers;
// the reset is enqueued before its passes and the read-back after them, on the
// same stream, so concurrent computations never see each other's failures.
cudaError_t fdp_enqueue_err_reset(unsigned int *d_err, cudaStream_t s);
cudaError_t fdp_enqueue_err_read(unsigned int *h_err, const unsigned int *d_err, cudaStream_t s);
void fdp_set_last_error(const char *msg);
fdp_status fdp_cuda_status(cudaError_t e, const char *what);
void fdp_server_shutdown(fdp_ctx *c);
