// C ABI of the frontier-DP engine (include/oneesan_fdp.h).
#include <atomic>
#include <chrono>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/oneesan_fdp.h"
#include "fdp_api_internal.h"
#include "fdp_host.h"
#include "fdp_launch.h"
#include "fdp_rowinit_dev.h"
#include "fdp_tail_dev.h"

using fdp::DevTables;

static thread_local std::string g_last_error;

#define FDP_RUN_MAX_MODULI 64

// Device memory a synchronous call leaves free beside its escape words.
static constexpr size_t kEscapeMargin = size_t(1) << 30;
// Device memory the pool keeps mapped, and the most that a synchronous call leaves
// behind outside it, for the next one.
static constexpr size_t kPoolKeep = size_t(20) << 30;
static constexpr size_t kSideKeep = size_t(4) << 30;
// Windows of a context that hold pool memory at a time.
static constexpr size_t kWindows = 64;

static fdp_status cuda_status(cudaError_t e, const char *what) {
  if (e == cudaSuccess) return FDP_OK;
  g_last_error = std::string(what) + ": " + cudaGetErrorString(e);
  cudaGetLastError();  // clear a sticky-free error so the context stays usable
  return e == cudaErrorMemoryAllocation ? FDP_ERR_HBM : FDP_ERR_CUDA;
}

#define FDP_CK(expr, what)                                  \
  do {                                                      \
    fdp_status _s = cuda_status((expr), (what));            \
    if (_s != FDP_OK) return _s;                            \
  } while (0)

extern "C" const char *fdp_version(void) { return "oneesan-fdp-b200 0.1 (sm_100a)"; }
extern "C" const char *fdp_last_error(void) { return g_last_error.c_str(); }

extern "C" uint64_t fdp_main_states(int width) { return fdp::main_states(width); }
extern "C" uint64_t fdp_blocked_states(int width) { return fdp::blocked_states(width); }
extern "C" uint64_t fdp_cell_bytes(int width, int p) {
  if (width < 2 || width > FDP_MAXW || p < 1 || p >= width) return 0;
  return fdp::cell_bytes(width, p);
}

static fdp_status check_problem(const fdp_problem *pr) {
  if (!pr || pr->n < 1 || pr->n > FDP_MAX_N || pr->k < 1 || !pr->moduli) {
    g_last_error = "problem: need 1 <= n <= 27, k >= 1 and a moduli array";
    return FDP_ERR_ARGS;
  }
  if (pr->lanes < 1 || pr->lanes > FDP_MAX_LANES) {
    g_last_error = "problem: lanes must be in 1..16";
    return FDP_ERR_ARGS;
  }
  for (int i = 0; i < pr->k; ++i)
    if (pr->moduli[i] < 2) {
      g_last_error = "problem: modulus must be in [2, 2^32-1]";
      return FDP_ERR_MODULUS;
    }
  return FDP_OK;
}

static int fit_row_init(int W, int R, bool bounded, int *cap);

extern "C" fdp_status fdp_plan(const fdp_problem *pr, uint64_t budget, fdp_plan_out *out) {
  fdp_status s = check_problem(pr);
  if (s != FDP_OK) return s;
  if (!out) return FDP_ERR_ARGS;
  const int W = pr->n + 1;
  const int lanes = pr->lanes < pr->k ? pr->lanes : pr->k;
  fdp_plan_out o{};
  o.n = pr->n;
  o.width = W;
  o.k = pr->k;
  o.lanes = lanes;
  o.passes = (pr->k + lanes - 1) / lanes;
  o.index_bits = fdp::needs_u64(W) ? 64 : 32;
  o.main_states = fdp::main_states(W);
  o.blocked_states = fdp::blocked_states(W);
  o.state_bytes = 4ull * (o.main_states + o.blocked_states) * uint64_t(lanes);
  o.scratch_bytes = 0;
  o.table_bytes = o.index_bits == 64 ? sizeof(fdp::WidthTables<uint64_t>) : sizeof(fdp::WidthTables<uint32_t>);
  o.total_bytes = o.state_bytes + o.table_bytes + (1u << 20);
  o.rows = fdp::sweep_rows(W);
  o.cells_per_row = W - 1;
  // Rows run in height-bounded spaces first (fdp_set_tuning bounded_prefix),
  // then in the full space.
  // The first init_rows - 1 sweep rows are replaced by the row-k initialiser
  // (default tuning, when its scratch fits).
  std::vector<int> caps;
  if (W >= 4) caps = fdp::bounded_prefix_caps(W);
  int R = fdp::auto_row_init_rows(W), rcap = 0;
  if (R >= 2) R = fit_row_init(W, R, true, &rcap);
  o.init_rows = R;
  const int first_row = R >= 2 ? R : 1;
  o.bounded_rows = 0;
  o.alg_bytes_per_residue = 0;
  o.transitions_per_residue = 0;
  for (int row = first_row; row <= o.rows; ++row) {
    const int cap = row <= int(caps.size()) ? caps[size_t(row - 1)] : FDP_FULL_CAP;
    if (cap < FDP_FULL_CAP) ++o.bounded_rows;
    o.alg_bytes_per_residue += fdp::row_bytes(W, cap);
    o.transitions_per_residue += uint64_t(o.cells_per_row) * fdp::cell_transitions(W, cap);
  }
  // Width tables a pass uploads: the full space, each bounded space and the
  // height-1 space of row 0; the expansion tables fit in the 1 MiB margin.
  const uint64_t ntables = 1 + (caps.empty() ? 0 : caps.size() + 1);
  o.sweep_peak_bytes = o.state_bytes + ntables * o.table_bytes + (1u << 20);
  o.init_peak_bytes = o.sweep_peak_bytes + (R >= 2 ? fdp::row_init_tables(W, R, rcap) : 0);
  o.total_bytes = o.init_peak_bytes > o.sweep_peak_bytes ? o.init_peak_bytes : o.sweep_peak_bytes;
  o.fits = o.total_bytes <= budget ? 1 : 0;
  *out = o;
  return FDP_OK;
}

extern "C" fdp_status fdp_create(fdp_ctx **out, int device) {
  if (!out) return FDP_ERR_ARGS;
  *out = nullptr;
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || count < 1) {
    cudaGetLastError();
    g_last_error = "no CUDA device visible";
    return FDP_ERR_GPU_COUNT;
  }
  if (device < 0 || device >= count) {
    g_last_error = "device index out of range";
    return FDP_ERR_GPU_COUNT;
  }
  FDP_CK(cudaSetDevice(device), "cudaSetDevice");
  auto *c = new fdp_ctx();
  c->device = device;
  fdp_status s = cuda_status(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking), "stream");
  if (s == FDP_OK) s = cuda_status(cudaMalloc(&c->d_acc, sizeof(unsigned long long) * FDP_MAX_LANES), "acc");
  if (s == FDP_OK) s = cuda_status(cudaMalloc(&c->d_res, sizeof(uint32_t) * FDP_MAX_LANES), "res");
  if (s == FDP_OK) s = cuda_status(cudaMallocHost(&c->h_res, sizeof(uint32_t) * FDP_RUN_MAX_MODULI), "pinned res");
  if (s == FDP_OK) s = cuda_status(cudaMalloc(&c->d_err, sizeof(unsigned int)), "error word");
  if (s == FDP_OK) s = cuda_status(cudaMallocHost(&c->h_err, sizeof(unsigned int)), "pinned error word");
  if (s == FDP_OK) s = cuda_status(cudaEventCreate(&c->ev0), "event");
  if (s == FDP_OK) s = cuda_status(cudaEventCreate(&c->ev1), "event");
  if (s == FDP_OK) s = cuda_status(cudaStreamCreateWithFlags(&c->span_stream, cudaStreamNonBlocking), "span stream");
  if (s == FDP_OK) s = cuda_status(cudaEventCreateWithFlags(&c->span_fork, cudaEventDisableTiming), "span event");
  if (s == FDP_OK) s = cuda_status(cudaEventCreateWithFlags(&c->span_join, cudaEventDisableTiming), "span event");
  if (s != FDP_OK) {
    fdp_destroy(c);
    return s;
  }
  *out = c;
  return FDP_OK;
}

fdp_ctx::~fdp_ctx() {
  fdp_server_shutdown(this);
  cudaSetDevice(device);
  if (stream) cudaStreamSynchronize(stream);
  for (auto &kv : tables) fdp::free_tables(&kv.second);
  if (d_main) cudaFree(d_main);
  if (d_blk) cudaFree(d_blk);
  if (d_side) cudaFree(d_side);
  if (h_multi) cudaFreeHost(h_multi);
  for (cudaStream_t x : multi_streams) cudaStreamDestroy(x);
  for (cudaEvent_t x : multi_events) cudaEventDestroy(x);
  if (d_acc) cudaFree(d_acc);
  if (d_res) cudaFree(d_res);
  if (h_res) cudaFreeHost(h_res);
  if (d_err) cudaFree(d_err);
  if (h_err) cudaFreeHost(h_err);
  if (ev0) cudaEventDestroy(ev0);
  if (ev1) cudaEventDestroy(ev1);
  if (span_fork) cudaEventDestroy(span_fork);
  if (span_join) cudaEventDestroy(span_join);
  for (WindowUse &w : windows) cudaEventDestroy(w.done);
  if (pool) cudaMemPoolDestroy(pool);
  if (span_stream) cudaStreamDestroy(span_stream);
  if (stream) cudaStreamDestroy(stream);
}

extern "C" void fdp_destroy(fdp_ctx *ctx) { delete ctx; }

fdp_status fdp_ctx_tables_cap(fdp_ctx *c, int W, int cap, const DevTables **out) {
  std::lock_guard<std::mutex> lk(c->tables_mu);
  const int key = W * 4096 + (cap >= FDP_FULL_CAP ? 4095 : cap);
  auto it = c->tables.find(key);
  if (it == c->tables.end()) {
    DevTables t;
    const fdp::BesideCaptures beside;
    FDP_CK(fdp::upload_tables(W, cap, &t), "upload tables");
    it = c->tables.emplace(key, t).first;
  }
  *out = &it->second;
  return FDP_OK;
}

fdp_status fdp_ctx_tables(fdp_ctx *c, int W, const DevTables **out) {
  return fdp_ctx_tables_cap(c, W, FDP_FULL_CAP, out);
}

// Strip rows R the row-k initialiser fills directly for width W (0: the pass
// starts from row 0), and the height cap of the space row R runs in.  Used
// when the fill's scratch fits the blocked buffer (D words per lane, dead
// before the first sweep).
// The largest strip of at most R rows whose fill fits the blocked buffer.
static int fit_row_init(int W, int R, bool bounded, int *cap) {
  if (R > W - 1) R = W - 1;  // the state after row R-1 <= the last sweep row
  if (R > 7) R = 7;
  const std::vector<int> caps = (bounded && W >= 4) ? fdp::bounded_prefix_caps(W) : std::vector<int>{};
  for (; R >= 2; --R) {
    *cap = R <= int(caps.size()) ? caps[size_t(R - 1)] : FDP_FULL_CAP;
    if (fdp::row_init_scratch(W, R, *cap) <= fdp::blocked_states(W)) return R;
  }
  return 0;
}

static int row_init_rows(const fdp_ctx *c, int W, int *cap) {
  int R = c->cfg.row_init;
  if (R == 0) R = fdp::auto_row_init_rows(W);
  if (R < 2) return 0;
  return fit_row_init(W, R, c->cfg.bounded_prefix, cap);
}

// Whether a pass of width W is one launch with the state in shared memory: small
// widths, unless the tuning asks for a particular way through the first rows.
static bool whole_pass(const fdp_ctx *c, int W) {
  return c->cfg.tail && fdp::solves_whole(W) && c->cfg.row_init == 0 && c->cfg.bounded_prefix;
}

// Every device table a residue pass of width W reads, uploaded before any
// stream capture starts (allocation and blocking copies cannot be captured).
fdp_status fdp_prepare_pass(fdp_ctx *c, int W, const DevTables **full) {
  const fdp::BesideCaptures beside;
  fdp_status s = fdp_ctx_tables(c, W, full);
  if (s != FDP_OK) return s;
  int rcap = 0;
  if (const int R = row_init_rows(c, W, &rcap)) FDP_CK(fdp::prepare_row_init(W, R, rcap), "row-k initialiser tables");
  if (whole_pass(c, W)) {
    FDP_CK(fdp::prepare_whole(W), "whole-solve tables");
    return FDP_OK;
  }
  if (c->cfg.tail) FDP_CK(fdp::prepare_tail(W), "row tail tables");
  if (!c->cfg.bounded_prefix || W < 4) return s;
  std::vector<int> caps = fdp::bounded_prefix_caps(W);
  caps.push_back(1);
  const DevTables *t = nullptr;
  for (int cap : caps)
    if ((s = fdp_ctx_tables_cap(c, W, cap, &t)) != FDP_OK) return s;
  caps.push_back(FDP_FULL_CAP);
  FDP_CK(fdp::prepare_expand_tables(caps), "expand tables");
  return FDP_OK;
}

// cudaMalloc for what a call cannot do without: where it fails, once more after
// the windows in flight have handed their words back and without what the context
// keeps for later calls.
cudaError_t fdp_ctx_malloc(fdp_ctx *c, void **p, size_t bytes) {
  const fdp::BesideCaptures beside;
  cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaErrorMemoryAllocation || (!c->pool && !c->d_side)) return e;
  cudaGetLastError();
  if ((e = cudaDeviceSynchronize()) != cudaSuccess) return e;
  if (c->pool) cudaMemPoolTrimTo(c->pool, 0);
  if (c->d_side) cudaFree(c->d_side);
  c->d_side = nullptr;
  c->cap_side = 0;
  return cudaMalloc(p, bytes);
}

// The pool of the windows' escape words and of large side memory (SideMemory), kept
// mapped up to kPoolKeep bytes.  What
// lies idle in it stands in nobody's way: cudaMalloc of this process gets it from
// the driver.
static cudaError_t pool_take(fdp_ctx *c, void **p, size_t bytes, cudaStream_t st) {
  if (!c->pool) {
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = c->device;
    uint64_t keep = kPoolKeep;
    int off = 0;  // a window never waits for another stream's to get its words
    cudaError_t e = cudaMemPoolCreate(&c->pool, &props);
    if (e != cudaSuccess) {
      c->pool = nullptr;
      return e;
    }
    cudaMemPoolSetAttribute(c->pool, cudaMemPoolAttrReleaseThreshold, &keep);
    cudaMemPoolSetAttribute(c->pool, cudaMemPoolReuseAllowInternalDependencies, &off);
  }
  return cudaMallocFromPoolAsync(p, bytes, c->pool, st);
}

// Bytes the pool holds mapped that stream st can have.  The pool counts a window's
// words as unused from the call that frees them on; until its stream gets there
// they serve that stream alone.
static size_t pool_idle(fdp_ctx *c, cudaStream_t st) {
  uint64_t mapped = 0, used = 0;
  if (!c->pool || cudaMemPoolGetAttribute(c->pool, cudaMemPoolAttrReservedMemCurrent, &mapped) != cudaSuccess ||
      cudaMemPoolGetAttribute(c->pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess)
    return 0;
  for (size_t i = 0; i < c->windows.size();) {
    WindowUse &w = c->windows[i];
    if (cudaEventQuery(w.done) == cudaErrorNotReady) {
      cudaGetLastError();
      if (w.stream != st) used += w.bytes;
      ++i;
    } else {
      cudaEventDestroy(w.done);
      w = c->windows.back();
      c->windows.pop_back();
    }
  }
  return mapped > used ? size_t(mapped - used) : 0;
}

// Device memory that one synchronous call (the context locked) takes beside its
// state.  Up to kSideKeep bytes stay with the context for the next such call.  More
// comes from the windows' pool, where other allocators can get it after the call:
// the pool maps 10 GiB in 73 ms, once, and a call pays nothing for it after that
// (cudaMalloc and cudaFree in each call: 10 ms of 1.38 s at n = 20, 14 lanes, and
// the free waits for everything on the device, served requests too).  What exceeds
// the pool as well is allocated and freed by the call (40 GiB 30 ms, below 0.5 % of
// a pass that needs so much).
struct SideMemory {
  fdp_ctx *c;
  char *p = nullptr;
  bool pooled = false;
  explicit SideMemory(fdp_ctx *ctx) : c(ctx) {}
  SideMemory(const SideMemory &) = delete;
  SideMemory &operator=(const SideMemory &) = delete;
  ~SideMemory() {
    if (pooled) {
      cudaFreeAsync(p, c->stream);
      cudaStreamSynchronize(c->stream);  // the call has waited; only now does the driver hand it on
    }
    if (c->cap_side > kSideKeep) drop();
  }
  void drop() {
    const fdp::BesideCaptures beside;
    if (c->d_side) cudaFree(c->d_side);
    c->d_side = nullptr;
    c->cap_side = 0;
  }
  cudaError_t take(size_t bytes) {
    if (c->cap_side < bytes) {
      void *q = nullptr;
      if (bytes > kSideKeep && bytes <= kPoolKeep) {
        pooled = pool_take(c, &q, bytes, c->stream) == cudaSuccess;
        if (pooled) {
          p = static_cast<char *>(q);
          return cudaSuccess;
        }
        cudaGetLastError();
      }
      drop();
      const cudaError_t e = fdp_ctx_malloc(c, &q, bytes);
      if (e != cudaSuccess) return e;
      c->d_side = static_cast<char *>(q);
      c->cap_side = bytes;
    }
    p = c->d_side;
    return cudaSuccess;
  }
  // Bytes the call can do without: p stays null unless `leave` bytes remain free.
  bool take_optional(size_t bytes, size_t leave) {
    size_t free_b = 0, total_b = 0;
    if ((c->cap_side >= bytes || (cudaMemGetInfo(&free_b, &total_b) == cudaSuccess &&
                                  free_b + c->cap_side + pool_idle(c, c->stream) > bytes + leave)) &&
        take(bytes) == cudaSuccess)
      return true;
    cudaGetLastError();
    return false;
  }
};

static fdp_status ensure_buffer(fdp_ctx *c, uint32_t **buf, size_t *cap, size_t bytes, const char *what) {
  if (*cap >= bytes && *buf) return FDP_OK;
  if (*buf) cudaFree(*buf);
  *buf = nullptr;
  *cap = 0;
  FDP_CK(fdp_ctx_malloc(c, reinterpret_cast<void **>(buf), bytes ? bytes : 4), what);
  *cap = bytes;
  return FDP_OK;
}

// The context's state buffers for `lanes` lanes of width W.  Where a call that
// also wants `beside` bytes could have them but for the buffers of a larger
// problem, exact buffers take their place.
static fdp_status ensure_state(fdp_ctx *c, int W, int lanes, size_t beside) {
  const size_t mb = size_t(fdp::main_states(W)) * lanes * 4, bb = size_t(fdp::blocked_states(W)) * lanes * 4;
  size_t free_b = 0, total_b = 0;
  if (beside > c->cap_side && c->cap_main >= mb && c->cap_blk >= bb && cudaMemGetInfo(&free_b, &total_b) == cudaSuccess) {
    free_b += c->cap_side + pool_idle(c, c->stream);
    if (free_b <= beside + kEscapeMargin &&
        free_b + (c->cap_main - mb) + (c->cap_blk - bb) > beside + kEscapeMargin) {
      cudaFree(c->d_main);
      cudaFree(c->d_blk);
      c->d_main = c->d_blk = nullptr;
      c->cap_main = c->cap_blk = 0;
    }
  }
  fdp_status s = ensure_buffer(c, &c->d_main, &c->cap_main, mb, "main state");
  if (s == FDP_OK) s = ensure_buffer(c, &c->d_blk, &c->cap_blk, bb, "blocked state");
  return s;
}

// Whether passes of more than 8 lanes are large enough (32 GiB with the fused row
// tail's escape words) to be split where memory asks for it.
static bool may_split(int W, int lanes) {
  const uint64_t esc = fdp::tail_escape_words(W), lane = fdp::main_states(W) + fdp::blocked_states(W) + esc;
  return lanes > 8 && esc && lane * 4 * uint64_t(lanes) >= uint64_t(32) << 30;
}

// Residues a pass of fdp_run_sync really holds: `lanes`, or one span of 8 where, of
// `have` bytes, the escape words fit beside 8 lanes but not beside all of them
// (n = 22, 14 lanes: 16.4 s in one pass of single cells, 13.4 s as passes of 8 and 6).
static int pass_lanes(int W, int lanes, uint64_t have) {
  const uint64_t lane = (fdp::main_states(W) + fdp::blocked_states(W) + fdp::tail_escape_words(W)) * 4;
  const bool all = lane * uint64_t(lanes) + kEscapeMargin <= have, eight = lane * 8 + kEscapeMargin <= have;
  return may_split(W, lanes) && eight && !all ? 8 : lanes;
}

static int lanes_with_escapes(fdp_ctx *c, int W, int lanes) {
  size_t free_b = 0, total_b = 0;
  if (!c->cfg.tail || whole_pass(c, W) || !may_split(W, lanes) || cudaMemGetInfo(&free_b, &total_b) != cudaSuccess)
    return lanes;
  return pass_lanes(W, lanes, free_b + pool_idle(c, c->stream) + c->cap_side + c->cap_main + c->cap_blk);
}

extern "C" int fdp_test_pass_lanes(int n, int lanes, uint64_t have_bytes) {
  if (n < 1 || n > FDP_MAX_N || lanes < 1 || lanes > FDP_MAX_LANES) return 0;
  return pass_lanes(n + 1, lanes, have_bytes);
}

extern "C" fdp_status fdp_test_single_cells(fdp_ctx *c, int on) {
  if (!c) return FDP_ERR_ARGS;
  fdp_pass_single_cells(c, on != 0);
  return FDP_OK;
}

// Enqueue one whole residue pass on `s`: the row-0 state, the row sweeps, the
// first-row dot product and the residue copy to pinned host memory.  With the
// bounded prefix (c->cfg.bounded_prefix) row 0 is the height-1 space with every
// coefficient 1 and row r runs in the space of height cap r + 1 while that
// space is small; the state grows in place between them (the blocked buffer,
// dead at row boundaries, stages the move).  `blk` must hold D x L words of
// the full space.
// Test hook: the next `count` error-word resets write a nonzero value, as if
// a kernel had given up on a bounded wait (fdp_test_inject_pass_errors).
static std::atomic<int> g_injected_errors{0};

cudaError_t fdp_enqueue_err_reset(unsigned int *d_err, cudaStream_t s) {
  int v = g_injected_errors.load();
  while (v > 0 && !g_injected_errors.compare_exchange_weak(v, v - 1)) {
  }
  return cudaMemsetAsync(d_err, v > 0 ? 1 : 0, sizeof(unsigned int), s);
}

cudaError_t fdp_enqueue_err_read(unsigned int *h_err, const unsigned int *d_err, cudaStream_t s) {
  return cudaMemcpyAsync(h_err, d_err, sizeof(unsigned int), cudaMemcpyDeviceToHost, s);
}

extern "C" fdp_status fdp_test_inject_pass_errors(int count) {
  if (count < 0) return FDP_ERR_ARGS;
  g_injected_errors.store(count);
  return FDP_OK;
}

// `rows` row sweeps in the full space: each row's cells one launch each, or, given
// escape words, cells s-1..1 of it as one fused pass.
static fdp_status enqueue_full_rows(fdp_ctx *c, const DevTables &t, int L, const uint32_t *mods, uint32_t *main,
                                    uint32_t *blk, uint32_t *esc, int rows, cudaStream_t s, uint64_t *n,
                                    cudaStream_t span_stream, cudaEvent_t fork, cudaEvent_t join) {
  const int W = t.W;
  const bool fused = esc && c->cfg.tail && fdp::tail_symbols(W);
  auto cells = [&](int lanes, const uint32_t *m, uint32_t *mn, uint32_t *bk, int last, cudaStream_t ss) {
    cudaError_t e = cudaSuccess;
    for (int p = W - 1; p >= last && e == cudaSuccess; --p)
      e = fdp::launch_cell(t, lanes, m, mn, bk, p, p == W - 1, false, c->cfg, ss, n);
    return e;
  };
  // Span chains overlap the tails of single-cell launches; with the fused row
  // tail one chain is faster (n = 20, 14 lanes: 1.40 against 1.53 s), as its CTAs
  // take whole SMs and hold back the other chain's.
  if (!fused && span_stream && fork && join && c->cfg.span_chains && L > 8 && !c->cfg.split_panels &&
      c->cfg.split_spans_min_p <= 1 && rows > 0) {
    // Each lane span is laid out as a lane count of its own at its first
    // panel's offset and no cell reads another span's panels, so the spans'
    // row sweeps run as two chains of launches, joined before the read-out.
    FDP_CK(cudaEventRecord(fork, s), "span fork");
    FDP_CK(cudaStreamWaitEvent(span_stream, fork, 0), "span fork");
    for (int l0 = 0, i = 0; l0 < L; ++i) {
      const int le = fdp::span_end_of(L, l0);
      for (int row = 0; row < rows; ++row)
        FDP_CK(cells(le - l0, mods + l0, main + size_t(l0) * fdp::main_states(W),
                     blk + size_t(l0) * fdp::blocked_states(W), 1, i == 0 ? s : span_stream),
               "cell");
      l0 = le;
    }
    FDP_CK(cudaEventRecord(join, span_stream), "span join");
    FDP_CK(cudaStreamWaitEvent(s, join, 0), "span join");
    return FDP_OK;
  }
  for (int row = 0; row < rows; ++row) {
    FDP_CK(cells(L, mods, main, blk, fused ? fdp::tail_symbols(W) : 1, s), "cell");
    if (fused) FDP_CK(fdp::launch_tail(t, L, mods, main, blk, esc, s, n), "row tail");
  }
  return FDP_OK;
}

fdp_status fdp_enqueue_pass(fdp_ctx *c, const DevTables &t, int L, const uint32_t *mods, uint32_t *main,
                            uint32_t *blk, uint32_t *esc, unsigned long long *acc, uint32_t *d_res, uint32_t *h_res,
                            unsigned int *d_err, cudaStream_t s, uint64_t *launches, cudaStream_t span_stream,
                            cudaEvent_t fork, cudaEvent_t join) {
  const int W = t.W;
  if (whole_pass(c, W)) {
    FDP_CK(fdp::launch_whole(W, L, mods, d_res, s), "whole solve");
    if (h_res) FDP_CK(cudaMemcpyAsync(h_res, d_res, sizeof(uint32_t) * L, cudaMemcpyDeviceToHost, s), "residue copy");
    if (launches) ++*launches;
    return FDP_OK;
  }
  const uint64_t M = fdp::main_states(W), D = fdp::blocked_states(W);
  uint64_t n = 0;
  fdp_status st = FDP_OK;
  // Rows 1..B run in height-bounded spaces (caps[r-1] for row r), the rest in
  // the full space.
  const std::vector<int> caps = (c->cfg.bounded_prefix && W >= 4) ? fdp::bounded_prefix_caps(W) : std::vector<int>{};
  const int B = int(caps.size());
  auto space = [&](int cap, const DevTables **out) -> fdp_status {
    if (cap >= FDP_FULL_CAP) {
      *out = &t;
      return FDP_OK;
    }
    return fdp_ctx_tables_cap(c, W, cap, out);
  };
  const DevTables *prev = nullptr;
  int next_row = 1;
  int rcap = 0;
  if (const int R = row_init_rows(c, W, &rcap)) {
    // Rows 0..R-1 at once: the state after row R-1, filled into row R's space
    // (the blocked buffer is the fill's scratch).
    if ((st = space(rcap, &prev)) != FDP_OK) return st;
    FDP_CK(fdp::enqueue_row_init(W, R, rcap, L, mods, main, blk, D * uint64_t(L), c->cfg.row_init_tensor, d_err, s,
                                 &n),
           "row-k initialiser");
    next_row = R;
  } else if (B > 0) {
    // Row 0 in the height-1 space: every word is a first-row state, coefficient 1.
    if ((st = space(1, &prev)) != FDP_OK) return st;
    FDP_CK(fdp::launch_fill_ones(main, fdp::main_states_capped(W, 1) * uint64_t(L), s), "row-0 fill");
    ++n;
  } else {
    FDP_CK(cudaMemsetAsync(main, 0, size_t(M) * L * 4, s), "zero main");
    FDP_CK(fdp::launch_first_row_init(t, L, main, s), "row-0 init");
    prev = &t;
    ++n;
  }
  for (int row = next_row; row <= B && row <= fdp::sweep_rows(W); ++row) {
    const DevTables *cur = nullptr;
    if ((st = space(caps[size_t(row - 1)], &cur)) != FDP_OK) return st;
    if (cur != prev) FDP_CK(fdp::enqueue_expand(*prev, *cur, L, main, blk, D * uint64_t(L), s, &n), "grow state");
    for (int p = W - 1; p >= 1; --p) {
      FDP_CK(fdp::launch_cell(*cur, L, mods, main, blk, p, p == W - 1, false, c->cfg, s, &n), "bounded cell");
    }
    prev = cur;
  }
  if (prev != &t) FDP_CK(fdp::enqueue_expand(*prev, t, L, main, blk, D * uint64_t(L), s, &n), "grow state");
  const int row0 = next_row > B + 1 ? next_row : B + 1;
  if ((st = enqueue_full_rows(c, t, L, mods, main, blk, esc, fdp::sweep_rows(W) - row0 + 1, s, &n, span_stream, fork,
                              join)) != FDP_OK)
    return st;
  FDP_CK(fdp::launch_first_row_dot(t, L, mods, main, acc, d_res, s), "first-row dot");
  n += 2;
  if (h_res) FDP_CK(cudaMemcpyAsync(h_res, d_res, sizeof(uint32_t) * L, cudaMemcpyDeviceToHost, s), "residue copy");
  if (launches) *launches += n;
  return FDP_OK;
}

extern "C" fdp_status fdp_run_sync(fdp_ctx *c, const fdp_problem *pr, uint32_t *residues_out, fdp_run_stats *st) {
  if (!c || !residues_out) return FDP_ERR_ARGS;
  fdp_status s = check_problem(pr);
  if (s != FDP_OK) return s;
  if (pr->k > FDP_RUN_MAX_MODULI) {
    g_last_error = "run_sync: at most 64 moduli per call";
    return FDP_ERR_ARGS;
  }
  std::lock_guard<std::mutex> lk(c->mu);
  auto t0 = std::chrono::steady_clock::now();
  FDP_CK(cudaSetDevice(c->device), "cudaSetDevice");
  const int W = pr->n + 1;
  const DevTables *t = nullptr;
  if ((s = fdp_prepare_pass(c, W, &t)) != FDP_OK) return s;
  const int lanes = lanes_with_escapes(c, W, pr->lanes < pr->k ? pr->lanes : pr->k);
  // The state, and, where memory allows, the escape words of the fused row tail;
  // a pass without them runs every cell as its own launch.
  SideMemory esc(c);
  if (!whole_pass(c, W)) {
    const size_t eb = c->cfg.tail ? size_t(fdp::tail_escape_words(W)) * lanes * 4 : 0;
    if ((s = ensure_state(c, W, lanes, eb)) != FDP_OK) return s;
    if (eb) esc.take_optional(eb, kEscapeMargin);
  }
  // Every pass (lanes residues each) is captured into ONE graph, run with one launch.
  fdp_run_stats acc{};
  auto c0 = std::chrono::steady_clock::now();
  cudaGraph_t g = nullptr;
  cudaGraphExec_t ge = nullptr;
  FDP_CK(cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal), "begin capture");
  uint64_t launches = 0;
  fdp_status es = cuda_status(fdp_enqueue_err_reset(c->d_err, c->stream), "error word");
  for (int done = 0; done < pr->k && es == FDP_OK; done += lanes) {
    const int L = (pr->k - done) < lanes ? (pr->k - done) : lanes;
    es = fdp_enqueue_pass(c, *t, L, pr->moduli + done, c->d_main, c->d_blk, reinterpret_cast<uint32_t *>(esc.p),
                          c->d_acc, c->d_res, c->h_res + done, c->d_err, c->stream, &launches, c->span_stream, c->span_fork, c->span_join);
  }
  if (es == FDP_OK) es = cuda_status(fdp_enqueue_err_read(c->h_err, c->d_err, c->stream), "error word");
  cudaError_t ce = cudaStreamEndCapture(c->stream, &g);
  if (es != FDP_OK) {
    if (g) cudaGraphDestroy(g);
    return es;
  }
  FDP_CK(ce, "end capture");
  ce = cudaGraphInstantiate(&ge, g, 0);
  cudaGraphDestroy(g);
  FDP_CK(ce, "graph instantiate");
  acc.capture_s = std::chrono::duration<double>(std::chrono::steady_clock::now() - c0).count();
  cudaEventRecord(c->ev0, c->stream);
  ce = cudaGraphLaunch(ge, c->stream);
  cudaEventRecord(c->ev1, c->stream);
  cudaError_t se = cudaStreamSynchronize(c->stream);
  cudaGraphExecDestroy(ge);
  FDP_CK(ce, "graph launch");
  FDP_CK(se, "residue pass");
  if (*c->h_err) {
    g_last_error = "residue pass: a bounded wait on the device gave up; the residues are invalid";
    return FDP_ERR_CUDA;
  }
  float ms = 0;
  cudaEventElapsedTime(&ms, c->ev0, c->ev1);
  acc.device_s = ms * 1e-3;
  acc.kernel_launches = launches;
  for (int i = 0; i < pr->k; ++i) residues_out[i] = c->h_res[i];
  fdp_plan_out po{};
  fdp_plan(pr, ~0ull, &po);
  acc.alg_bytes = po.alg_bytes_per_residue * uint64_t(pr->k);
  acc.transitions = po.transitions_per_residue * uint64_t(pr->k);
  acc.wall_s = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  if (st) *st = acc;
  return FDP_OK;
}

int fdp_pass_lanes(fdp_ctx *c, int n, int lanes) {
  std::lock_guard<std::mutex> lk(c->mu);
  return cudaSetDevice(c->device) == cudaSuccess ? lanes_with_escapes(c, n + 1, lanes) : lanes;
}

bool fdp_pass_is_whole(fdp_ctx *c, int n) {
  std::lock_guard<std::mutex> lk(c->mu);
  return whole_pass(c, n + 1);
}

void fdp_pass_single_cells(fdp_ctx *c, bool on) {
  std::lock_guard<std::mutex> lk(c->mu);
  c->cfg.tail = !on;
}

fdp_status fdp_time_pass_row(fdp_ctx *c, const fdp_problem *pr, double *row_ms) {
  fdp_status s = check_problem(pr);
  if (s != FDP_OK) return s;
  std::lock_guard<std::mutex> lk(c->mu);
  FDP_CK(cudaSetDevice(c->device), "cudaSetDevice");
  const int W = pr->n + 1, L = pr->lanes < pr->k ? pr->lanes : pr->k;
  if (W < 3) return FDP_ERR_ARGS;
  const DevTables *t = nullptr;
  if ((s = fdp_prepare_pass(c, W, &t)) != FDP_OK) return s;
  const bool whole = whole_pass(c, W);
  SideMemory esc(c);
  if (!whole) {
    const size_t eb = c->cfg.tail ? size_t(fdp::tail_escape_words(W)) * L * 4 : 0;
    if ((s = ensure_state(c, W, L, eb)) != FDP_OK) return s;
    if (eb) esc.take_optional(eb, kEscapeMargin);
  }
  const int rows = whole ? fdp::sweep_rows(W) : (W < 19 ? 8 : 1);  // some ms together
  cudaGraph_t g = nullptr;
  cudaGraphExec_t ge = nullptr;
  uint64_t n = 0;
  FDP_CK(cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal), "begin capture");
  fdp_status es = whole ? cuda_status(fdp::launch_whole(W, L, pr->moduli, c->d_res, c->stream), "whole solve")
                        : enqueue_full_rows(c, *t, L, pr->moduli, c->d_main, c->d_blk,
                                            reinterpret_cast<uint32_t *>(esc.p), rows, c->stream, &n, c->span_stream,
                                            c->span_fork, c->span_join);
  cudaError_t e = cudaStreamEndCapture(c->stream, &g);
  if (es == FDP_OK) es = cuda_status(e, "end capture");
  if (es == FDP_OK) es = cuda_status(cudaGraphInstantiate(&ge, g, 0), "graph instantiate");
  if (g) cudaGraphDestroy(g);
  for (int i = 0; i < 2 && es == FDP_OK; ++i) {  // the first one untimed
    cudaEventRecord(c->ev0, c->stream);
    es = cuda_status(cudaGraphLaunch(ge, c->stream), "graph launch");
    cudaEventRecord(c->ev1, c->stream);
    const cudaError_t se = cudaStreamSynchronize(c->stream);
    if (es == FDP_OK) es = cuda_status(se, "timed rows");
  }
  if (ge) cudaGraphExecDestroy(ge);
  if (es != FDP_OK) return es;
  float ms = 0;
  cudaEventElapsedTime(&ms, c->ev0, c->ev1);
  *row_ms = double(ms) / rows;
  return FDP_OK;
}

// Escape words for one window of fdp_apply_cells, or null: allocated and freed
// in the order of the caller's stream, so windows on other streams get words of
// their own.  A pool that would have to grow leaves at least half of what is free
// to others, however many windows are in flight (at most kWindows; events say which
// are).  A window that needs more than the pool keeps (mapping fresh memory
// for each window costs more than the fused tail gives), or a stream under capture
// (the captured work must not depend on an allocation of this context), runs cell
// by cell.
static uint32_t *window_escapes(fdp_ctx *c, int W, int lanes, cudaStream_t st) {
  const size_t bytes = size_t(fdp::tail_escape_words(W)) * lanes * 4;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (!bytes || bytes > kPoolKeep || !c->cfg.tail || cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
    cudaGetLastError();
    return nullptr;
  }
  void *p = nullptr;
  const size_t idle = pool_idle(c, st);
  bool ok = c->windows.size() < kWindows && fdp::prepare_tail(W) == cudaSuccess;
  if (ok && bytes > idle) {
    size_t free_b = 0, total_b = 0;
    ok = cudaMemGetInfo(&free_b, &total_b) == cudaSuccess && free_b / 2 > bytes - idle;
  }
  if (!ok || pool_take(c, &p, bytes, st) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return static_cast<uint32_t *>(p);
}

// Gives a window's words back in the order of its stream.
static cudaError_t window_done(fdp_ctx *c, int W, int lanes, uint32_t *esc, cudaStream_t st) {
  cudaError_t e = cudaFreeAsync(esc, st);
  WindowUse w{st, nullptr, size_t(fdp::tail_escape_words(W)) * lanes * 4};
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&w.done, cudaEventDisableTiming);
  if (e != cudaSuccess) return e;
  c->windows.push_back(w);
  return cudaEventRecord(w.done, st);
}

extern "C" fdp_status fdp_apply_cells(fdp_ctx *c, int width, int p_hi, int p_lo, int lanes, const uint32_t *moduli,
                                      uint32_t *d_main, uint32_t *d_block, void *stream) {
  // Checked first, before anything that needs a context or a device.
  if (!fdp::panel_aligned(lanes, d_main) || !fdp::panel_aligned(lanes, d_block)) {
    g_last_error = "apply_cells: d_main and d_block must be aligned to one word of the widest lane panel "
                   "(32 bytes for 8 or more lanes, 16 for 4-7, 8 for 2-3)";
    return FDP_ERR_ARGS;
  }
  if (!c || !moduli || !d_main || !d_block) return FDP_ERR_ARGS;
  if (width < 2 || width > FDP_MAXW || p_lo < 1 || p_hi >= width || p_lo > p_hi || lanes < 1 ||
      lanes > FDP_MAX_LANES) {
    g_last_error = "apply_cells: need 2 <= width <= 28, 1 <= p_lo <= p_hi < width, 1 <= lanes <= 16";
    return FDP_ERR_ARGS;
  }
  for (int i = 0; i < lanes; ++i)
    if (moduli[i] < 2) return FDP_ERR_MODULUS;
  std::lock_guard<std::mutex> lk(c->mu);
  const fdp::BesideCaptures beside;  // a kernel's first launch loads it, too
  FDP_CK(cudaSetDevice(c->device), "cudaSetDevice");
  const DevTables *t = nullptr;
  fdp_status s = fdp_ctx_tables(c, width, &t);
  if (s != FDP_OK) return s;
  cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : c->stream;
  // A window that reaches down to cell 1 runs its low cells as one fused pass
  // where the escape words can be had.
  uint32_t *esc = p_lo == 1 && p_hi >= fdp::tail_symbols(width) - 1 ? window_escapes(c, width, lanes, st) : nullptr;
  const int last = esc ? fdp::tail_symbols(width) : p_lo;
  cudaError_t e = cudaSuccess;
  for (int p = p_hi; p >= last && e == cudaSuccess; --p)
    e = fdp::launch_cell(*t, lanes, moduli, d_main, d_block, p, false, true, c->cfg, st);
  if (esc) {
    if (e == cudaSuccess) e = fdp::launch_tail(*t, lanes, moduli, d_main, d_block, esc, st, nullptr);
    if (e == cudaSuccess) e = cudaMemsetAsync(d_block, 0, size_t(fdp::blocked_states(width)) * lanes * 4, st);
    const cudaError_t fe = window_done(c, width, lanes, esc, st);
    if (e == cudaSuccess) e = fe;
  }
  FDP_CK(e, "cell");
  return FDP_OK;
}

extern "C" fdp_status fdp_rank_words(fdp_ctx *c, int width, const uint64_t *d_words, uint64_t *d_ranks,
                                     uint64_t count, void *stream) {
  if (!c || width < 1 || width > FDP_MAXW || (count && (!d_words || !d_ranks))) return FDP_ERR_ARGS;
  FDP_CK(cudaSetDevice(c->device), "cudaSetDevice");
  FDP_CK(fdp::launch_rank_words(width, d_words, d_ranks, count, stream ? (cudaStream_t)stream : c->stream), "rank");
  return FDP_OK;
}

extern "C" fdp_status fdp_unrank_words(fdp_ctx *c, int width, const uint64_t *d_ranks, uint64_t *d_words,
                                       uint64_t count, void *stream) {
  if (!c || width < 1 || width > FDP_MAXW || (count && (!d_words || !d_ranks))) return FDP_ERR_ARGS;
  FDP_CK(cudaSetDevice(c->device), "cudaSetDevice");
  FDP_CK(fdp::launch_unrank_words(width, d_ranks, d_words, count, stream ? (cudaStream_t)stream : c->stream),
         "unrank");
  return FDP_OK;
}

extern "C" fdp_status fdp_ternary_index(fdp_ctx *c, const uint32_t *d_codes, uint32_t *d_index, uint64_t count,
                                        void *stream) {
  if (!c || (count && (!d_codes || !d_index))) return FDP_ERR_ARGS;
  FDP_CK(cudaSetDevice(c->device), "cudaSetDevice");
  FDP_CK(fdp::launch_ternary_index(d_codes, d_index, count, stream ? (cudaStream_t)stream : c->stream), "ternary");
  return FDP_OK;
}

extern "C" fdp_status fdp_ternary_index_chunked(fdp_ctx *c, int chunk, const uint32_t *d_codes, uint32_t *d_index,
                                                uint64_t count, void *stream) {
  if (!c || (chunk != 4 && chunk != 7) || (count && (!d_codes || !d_index))) {
    g_last_error = "ternary_index_chunked: chunk must be 4 or 7";
    return FDP_ERR_ARGS;
  }
  FDP_CK(cudaSetDevice(c->device), "cudaSetDevice");
  FDP_CK(fdp::launch_ternary_index_chunked(chunk, d_codes, d_index, count, stream ? (cudaStream_t)stream : c->stream),
         "ternary chunked");
  return FDP_OK;
}

extern "C" fdp_status fdp_time_cells(fdp_ctx *c, const fdp_problem *pr, int rows, double *cell_ms) {
  if (!c || !cell_ms || rows < 1) return FDP_ERR_ARGS;
  fdp_status s = check_problem(pr);
  if (s != FDP_OK) return s;
  std::lock_guard<std::mutex> lk(c->mu);
  FDP_CK(cudaSetDevice(c->device), "cudaSetDevice");
  const int W = pr->n + 1;
  if (W < 3) return FDP_ERR_ARGS;
  const DevTables *t = nullptr;
  if ((s = fdp_ctx_tables(c, W, &t)) != FDP_OK) return s;
  const int L = pr->lanes < pr->k ? pr->lanes : pr->k;
  if ((s = ensure_state(c, W, L, 0)) != FDP_OK) return s;
  std::vector<cudaEvent_t> ev(size_t(rows) * W * 2);
  for (auto &e : ev) FDP_CK(cudaEventCreate(&e), "event");
  // One untimed launch first: the first launch of a kernel variant also loads
  // its module and sets its shared-memory limit.
  fdp_status rs = cuda_status(
      fdp::launch_cell(*t, L, pr->moduli, c->d_main, c->d_blk, W - 1, true, false, c->cfg, c->stream), "cell");
  for (int r = 0; r < rows && rs == FDP_OK; ++r)
    for (int p = W - 1; p >= 1 && rs == FDP_OK; --p) {
      cudaEventRecord(ev[(size_t(r) * W + p) * 2], c->stream);
      rs = cuda_status(fdp::launch_cell(*t, L, pr->moduli, c->d_main, c->d_blk, p, p == W - 1, false, c->cfg,
                                        c->stream), "cell");
      cudaEventRecord(ev[(size_t(r) * W + p) * 2 + 1], c->stream);
    }
  cudaError_t se = cudaStreamSynchronize(c->stream);
  if (rs == FDP_OK) rs = cuda_status(se, "timed cells");
  if (rs == FDP_OK) {
    for (int p = 0; p < W; ++p) cell_ms[p] = 0;
    for (int r = 0; r < rows; ++r)
      for (int p = W - 1; p >= 1; --p) {
        float ms = 0;
        cudaEventElapsedTime(&ms, ev[(size_t(r) * W + p) * 2], ev[(size_t(r) * W + p) * 2 + 1]);
        cell_ms[p] += ms / rows;
      }
  }
  for (auto &e : ev) cudaEventDestroy(e);
  return rs;
}

fdp_status fdp_cuda_status(cudaError_t e, const char *what) { return cuda_status(e, what); }

// Lets other translation units of the library report a message through
// fdp_last_error().
void fdp_set_last_error(const char *msg) { g_last_error = msg ? msg : ""; }

extern "C" fdp_status fdp_set_tuning(fdp_ctx *c, const fdp_tuning *t) {
  if (!c || !t) return FDP_ERR_ARGS;
  if (t->block < 64 || t->block > 256 || t->block % 32 || t->grid < 0 || t->lane_items < 0 || t->lane_items > 64 ||
      t->share_min < 0 || t->compact_max_p < -1 || t->compact_carry < -1 || t->compact_carry > 1 ||
      t->compact_items < 0 || t->compact_items > (t->compact_carry < 0 ? FDP_REC_MAX_ITEMS : 16) ||
      t->row_init_rows < -1 || t->row_init_rows > 7 || t->row_init_product < 0 || t->row_init_product > 1 ||
      t->split_spans_min_p < 0) {
    g_last_error =
        "tuning: block must be a multiple of 32 in 64..256, grid >= 0, lane_items 0..64, share_min >= 0, "
        "compact_max_p >= -1, compact_carry -1..1, compact_items 0..16 (0..4 with compact_carry -1; "
        "a value above 4 is used only where heads carry over), "
        "row_init_rows -1..7, row_init_product 0..1";
    return FDP_ERR_ARGS;
  }
  std::lock_guard<std::mutex> lk(c->mu);
  c->cfg.block = t->block;
  c->cfg.grid = t->grid;
  c->cfg.split_panels = t->split_panels != 0;
  c->cfg.bounded_prefix = t->bounded_prefix != 0;
  c->cfg.lane_items = t->lane_items > 0 ? t->lane_items : fdp::LaunchCfg{}.lane_items;
  c->cfg.share_min = t->share_min > 0 ? t->share_min : fdp::LaunchCfg{}.share_min;
  c->cfg.compact_max_p = t->compact_max_p != 0 ? t->compact_max_p : fdp::LaunchCfg{}.compact_max_p;
  c->cfg.compact_items = t->compact_items;
  c->cfg.compact_carry = t->compact_carry;
  c->cfg.row_init = t->row_init_rows;
  c->cfg.row_init_tensor = t->row_init_product == 0;
  c->cfg.split_spans_min_p = t->split_spans_min_p > 0 ? t->split_spans_min_p : fdp::LaunchCfg{}.split_spans_min_p;
  return FDP_OK;
}

extern "C" fdp_status fdp_get_tuning(fdp_ctx *c, fdp_tuning *t) {
  if (!c || !t) return FDP_ERR_ARGS;
  std::lock_guard<std::mutex> lk(c->mu);
  t->block = c->cfg.block;
  t->grid = c->cfg.grid;
  t->split_panels = c->cfg.split_panels ? 1 : 0;
  t->bounded_prefix = c->cfg.bounded_prefix ? 1 : 0;
  t->lane_items = c->cfg.lane_items;
  t->share_min = c->cfg.share_min;
  t->compact_max_p = c->cfg.compact_max_p;
  t->compact_items = c->cfg.compact_items;
  t->compact_carry = c->cfg.compact_carry;
  t->row_init_rows = c->cfg.row_init;
  t->row_init_product = c->cfg.row_init_tensor ? 0 : 1;
  t->split_spans_min_p = c->cfg.split_spans_min_p;
  return FDP_OK;
}

// One problem of fdp_run_multi_sync: its buffers and its forked stream.
struct MultiPart {
  const DevTables *t = nullptr;
  int lanes = 1;
  uint32_t *main = nullptr, *blk = nullptr, *esc = nullptr, *res = nullptr;
  unsigned long long *acc = nullptr;
  unsigned int *err = nullptr;  // this problem's error word
  cudaStream_t s = nullptr;
  cudaEvent_t done = nullptr;
  cudaStream_t span_s = nullptr;  // the second lane span's sweep
  cudaEvent_t span_fork = nullptr, span_join = nullptr;
};

extern "C" fdp_status fdp_run_multi_sync(fdp_ctx *c, const fdp_problem *probs, int count, uint32_t *residues_out,
                                         fdp_run_stats *st) {
  if (!c || !probs || count < 1 || count > 64 || !residues_out) return FDP_ERR_ARGS;
  int total_k = 0;
  for (int i = 0; i < count; ++i) {
    fdp_status s = check_problem(&probs[i]);
    if (s != FDP_OK) return s;
    total_k += probs[i].k;
  }
  std::lock_guard<std::mutex> lk(c->mu);
  auto t0 = std::chrono::steady_clock::now();
  FDP_CK(cudaSetDevice(c->device), "cudaSetDevice");
  std::vector<MultiPart> parts(static_cast<size_t>(count));
  SideMemory mem(c);
  cudaGraph_t g = nullptr;
  cudaGraphExec_t ge = nullptr;
  fdp_status rs = FDP_OK;
  uint64_t launches = 0;
  auto cleanup = [&]() {
    if (ge) cudaGraphExecDestroy(ge);
    if (g) cudaGraphDestroy(g);
  };
#define MULTI_CK(expr, what)                   \
  do {                                         \
    rs = cuda_status((expr), (what));          \
    if (rs != FDP_OK) { cleanup(); return rs; } \
  } while (0)
  // Residues of every problem, then one error word per problem.
  if (c->cap_hmulti < size_t(total_k + count)) {
    if (c->h_multi) cudaFreeHost(c->h_multi);
    c->h_multi = nullptr;
    c->cap_hmulti = 0;
    MULTI_CK(cudaMallocHost(&c->h_multi, sizeof(uint32_t) * size_t(total_k + count)), "pinned residues");
    c->cap_hmulti = size_t(total_k + count);
  }
  uint32_t *const pinned = c->h_multi;
  // Two streams and three events a problem, and the fork event.
  while (c->multi_streams.size() < size_t(2 * count)) {
    cudaStream_t x = nullptr;
    MULTI_CK(cudaStreamCreateWithFlags(&x, cudaStreamNonBlocking), "multi stream");
    c->multi_streams.push_back(x);
  }
  while (c->multi_events.size() < size_t(3 * count + 1)) {
    cudaEvent_t x = nullptr;
    MULTI_CK(cudaEventCreateWithFlags(&x, cudaEventDisableTiming), "multi event");
    c->multi_events.push_back(x);
  }
  const cudaEvent_t fork = c->multi_events[size_t(3 * count)];
  for (int i = 0; i < count; ++i) {
    MultiPart &p = parts[size_t(i)];
    if ((rs = fdp_prepare_pass(c, probs[i].n + 1, &p.t)) != FDP_OK) { cleanup(); return rs; }
    p.lanes = probs[i].lanes < probs[i].k ? probs[i].lanes : probs[i].k;
    p.s = c->multi_streams[size_t(2 * i)];
    p.done = c->multi_events[size_t(3 * i)];
    if (p.lanes > 8) {
      p.span_s = c->multi_streams[size_t(2 * i + 1)];
      p.span_fork = c->multi_events[size_t(3 * i + 1)];
      p.span_join = c->multi_events[size_t(3 * i + 2)];
    }
  }
  // One allocation for every problem's buffers: states, small words and, where
  // memory allows, the escape words of the fused row tail.
  auto carve = [&](bool escapes) {
    size_t at = 0;
    auto take = [&](size_t bytes) -> char * {
      char *p = mem.p ? mem.p + at : nullptr;
      at += (bytes + 255) / 256 * 256;
      return p;
    };
    for (int i = 0; i < count; ++i) {
      MultiPart &p = parts[size_t(i)];
      const int W = probs[i].n + 1;
      const size_t l4 = size_t(p.lanes) * 4;
      const bool whole = whole_pass(c, W);
      p.main = reinterpret_cast<uint32_t *>(take(whole ? 4 : size_t(fdp::main_states(W)) * l4));
      p.blk = reinterpret_cast<uint32_t *>(take(whole ? 4 : size_t(fdp::blocked_states(W)) * l4 + 4));
      const size_t eb = escapes && c->cfg.tail ? size_t(fdp::tail_escape_words(W)) * l4 : 0;
      p.esc = eb ? reinterpret_cast<uint32_t *>(take(eb)) : nullptr;
      p.acc = reinterpret_cast<unsigned long long *>(take(sizeof(unsigned long long) * FDP_MAX_LANES));
      p.res = reinterpret_cast<uint32_t *>(take(sizeof(uint32_t) * FDP_MAX_LANES));
      p.err = reinterpret_cast<unsigned int *>(take(sizeof(unsigned int)));
    }
    return at;
  };
  const bool escapes = mem.take_optional(carve(true), kEscapeMargin);
  if (!escapes) MULTI_CK(mem.take(carve(false)), "multi states");
  carve(escapes);
  auto c0 = std::chrono::steady_clock::now();
  MULTI_CK(cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal), "begin capture");
  cudaEventRecord(fork, c->stream);
  int off = 0;
  for (int i = 0; i < count && rs == FDP_OK; ++i) {
    MultiPart &p = parts[size_t(i)];
    cudaStreamWaitEvent(p.s, fork, 0);
    rs = cuda_status(fdp_enqueue_err_reset(p.err, p.s), "error word");
    for (int done = 0; done < probs[i].k && rs == FDP_OK; done += p.lanes) {
      const int L = (probs[i].k - done) < p.lanes ? (probs[i].k - done) : p.lanes;
      rs = fdp_enqueue_pass(c, *p.t, L, probs[i].moduli + done, p.main, p.blk, p.esc, p.acc, p.res, pinned + off + done,
                            p.err, p.s, &launches, p.span_s, p.span_fork, p.span_join);
    }
    if (rs == FDP_OK)
      rs = cuda_status(fdp_enqueue_err_read(reinterpret_cast<unsigned int *>(pinned + total_k + i), p.err, p.s),
                       "error word");
    cudaEventRecord(p.done, p.s);
    cudaStreamWaitEvent(c->stream, p.done, 0);
    off += probs[i].k;
  }
  cudaError_t ce = cudaStreamEndCapture(c->stream, &g);
  if (rs != FDP_OK) { cleanup(); return rs; }
  MULTI_CK(ce, "end capture");
  MULTI_CK(cudaGraphInstantiate(&ge, g, 0), "graph instantiate");
  const double cap_s = std::chrono::duration<double>(std::chrono::steady_clock::now() - c0).count();
  cudaEventRecord(c->ev0, c->stream);
  MULTI_CK(cudaGraphLaunch(ge, c->stream), "graph launch");
  cudaEventRecord(c->ev1, c->stream);
  MULTI_CK(cudaStreamSynchronize(c->stream), "multi pass");
  float ms = 0;
  cudaEventElapsedTime(&ms, c->ev0, c->ev1);
  for (int i = 0; i < count; ++i)
    if (pinned[total_k + i]) {
      g_last_error = "multi pass: a bounded wait on the device gave up in problem " + std::to_string(i) +
                     "; the residues are invalid";
      cleanup();
      return FDP_ERR_CUDA;
    }
  for (int i = 0; i < total_k; ++i) residues_out[i] = pinned[i];
  if (st) {
    fdp_run_stats acc{};
    acc.device_s = ms * 1e-3;
    acc.capture_s = cap_s;
    acc.kernel_launches = launches;
    for (int i = 0; i < count; ++i) {
      fdp_plan_out po{};
      fdp_plan(&probs[i], ~0ull, &po);
      acc.alg_bytes += po.alg_bytes_per_residue * uint64_t(probs[i].k);
      acc.transitions += po.transitions_per_residue * uint64_t(probs[i].k);
    }
    acc.wall_s = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    *st = acc;
  }
  cleanup();
  return FDP_OK;
#undef MULTI_CK
}
