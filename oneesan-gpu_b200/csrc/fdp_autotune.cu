// Autotuner: memory admission from the plan, timed row sweeps per candidate
// (1 warm-up + `repeats`, median), estimated device seconds per residue, and a
// known-residue check of the winner at the problem's own n when the reference
// publishes a residue mod 4294967291 for it (else n = 9, 2674633373,
// scripts/test/groupbatch-runtime.py:17; its passes are one launch that reads no
// tuning, so the check runs them cell by cell).  A row is timed as a pass runs it
// (fdp_time_pass_row): with the low cells fused where memory allows, and with the
// residues such a pass really holds; a last pass of fewer residues counts with its
// own time.
//
// Stage 1 searches how the k moduli split into passes (lanes), one launch vs
// one launch per lane panel, and the CTA size.  Stage 2 (not where a pass is one
// launch) then tunes the cell
// kernel's scheduling knobs of the winner one at a time (coordinate descent,
// a change kept only when the row is at least 0.5 % faster): the warp chunk
// (lane_items), the shortest shared prefix decode (share_min), the highest
// cell updated grouped by centre type (compact_max_p), whether grouped heads
// carry over between chunks (compact_carry), the states per lane of a grouped
// chunk (compact_items) and, for lane counts above 8, the lowest
// cell that runs each lane span as its own launch (split_spans_min_p).
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <string>
#include <vector>

#include "../../include/oneesan_fdp.h"
#include "fdp_api_internal.h"
#include "fdp_host.h"

namespace {

double median(std::vector<double> v) {
  std::sort(v.begin(), v.end());
  const size_t n = v.size();
  return n % 2 ? v[n / 2] : 0.5 * (v[n / 2 - 1] + v[n / 2]);
}

// Residues the reference publishes mod 4294967291 (n, residue): the
// known-answer check of the tuned configuration runs at the problem's own n
// when it is listed.
struct Known {
  int n;
  uint32_t residue;
};
const Known kKnown[] = {
    {9, 2674633373u},   // scripts/test/groupbatch-runtime.py:17
    {18, 503411004u},   // docs/results/reverse-algorithm-2026-09-05.md:53
    {20, 2308006916u},  // scripts/test/groupbatch-scratch.py:17
    {21, 998035516u},   // docs/b300-hbm32.md:554
    {22, 1245069298u},  // docs/results/groupbatch-interleaved-2026-09-05.json:1027
    {23, 2762394459u},  // docs/b300-hbm32.md:382-385
};

int panel_count(int lanes) {
  int n = 0;
  for (int l = 0; l < lanes; ++n) l += (lanes - l >= 8) ? 8 : (lanes - l >= 4) ? 4 : (lanes - l >= 2) ? 2 : 1;
  return n;
}

}  // namespace

extern "C" fdp_status fdp_autotune(fdp_ctx *c, const fdp_problem *pr, uint64_t budget, int repeats,
                                   fdp_autotune_result *out, char *json_out, size_t json_cap) {
  if (!c || !pr || !out || pr->n < 3 || pr->n > FDP_MAX_N || pr->k < 1 || !pr->moduli) return FDP_ERR_ARGS;
  if (repeats < 1) repeats = 1;
  const int max_lanes = std::max(1, std::min({pr->lanes > 0 ? pr->lanes : FDP_MAX_LANES, pr->k, FDP_MAX_LANES}));
  // Candidate residues-per-pass values.
  std::vector<int> lane_opts;
  for (int L : {1, 2, 4, 7, 8, 12, 14, 16})
    if (L <= max_lanes) lane_opts.push_back(L);
  if (std::find(lane_opts.begin(), lane_opts.end(), max_lanes) == lane_opts.end()) lane_opts.push_back(max_lanes);
  const int k = pr->k;
  for (int L = 1; L <= max_lanes; ++L)  // an even split of k into passes
    if ((k + L - 1) / L * L == k && std::find(lane_opts.begin(), lane_opts.end(), L) == lane_opts.end() && L >= 4)
      lane_opts.push_back(L);
  std::sort(lane_opts.begin(), lane_opts.end());
  fdp_tuning saved{};
  fdp_get_tuning(c, &saved);
  const int W = pr->n + 1, rows = fdp::sweep_rows(W);
  std::string js = "{\"n\":" + std::to_string(pr->n) + ",\"k\":" + std::to_string(k) + ",\"candidates\":[";
  bool first = true;
  fdp_autotune_result best{};
  best.s_per_residue = INFINITY;
  int tried = 0, rejected = 0;
  // Time of one row in every pass of the k moduli at L residues a pass (`all`), and
  // in the first of them (`row`): medians of `repeats`, after one not counted.
  auto sample = [&](int L, double *row, double *all) -> fdp_status {
    const int last = k - (k - 1) / L * L;
    const fdp_problem full{pr->n, L, pr->moduli, L}, rest{pr->n, last, pr->moduli, last};
    std::vector<double> rows_ms, alls;
    for (int r = 0; r <= repeats; ++r) {
      double a = 0, b = 0;
      fdp_status s = fdp_time_pass_row(c, &full, &a);
      b = a;
      if (s == FDP_OK && last != L) s = fdp_time_pass_row(c, &rest, &b);
      if (s != FDP_OK) return s;
      if (r > 0) {
        rows_ms.push_back(a);
        alls.push_back(a * ((k - 1) / L) + b);
      }
    }
    *row = median(rows_ms);
    *all = median(alls);
    return FDP_OK;
  };
  double best_all = 0;
  for (int L : lane_opts) {
    fdp_problem cand{pr->n, L, pr->moduli, L};
    fdp_plan_out plan{};
    if (fdp_plan(&cand, budget, &plan) != FDP_OK || !plan.fits) {
      ++rejected;
      char buf[160];
      snprintf(buf, sizeof(buf), "%s{\"lanes\":%d,\"status\":\"memory-rejected\",\"state_bytes\":%llu}",
               first ? "" : ",", L, (unsigned long long)plan.state_bytes);
      js += buf;
      first = false;
      continue;
    }
    if (const int held = fdp_pass_lanes(c, pr->n, L); held != L) {  // a candidate of its own
      js += std::string(first ? "" : ",") + "{\"lanes\":" + std::to_string(L) + ",\"status\":\"runs as " +
            std::to_string(held) + "\"}";
      first = false;
      continue;
    }
    const int npanels = panel_count(L);
    for (int split = 0; split <= (npanels > 1 ? 1 : 0); ++split)
      for (int block : {128, 256}) {
        fdp_tuning t = saved;
        t.block = block;
        t.grid = 0;
        t.split_panels = split;
        fdp_status s = fdp_set_tuning(c, &t);
        double row = 0, all = 0;
        if (s == FDP_OK) s = sample(L, &row, &all);
        ++tried;
        char buf[320];
        if (s != FDP_OK) {
          snprintf(buf, sizeof(buf), "%s{\"lanes\":%d,\"split_panels\":%d,\"block\":%d,\"status\":\"failed\"}",
                   first ? "" : ",", L, split, block);
          js += buf;
          first = false;
          if (s == FDP_ERR_HBM) continue;
          fdp_set_tuning(c, &saved);
          return s;
        }
        const int passes = (k + L - 1) / L;
        // Each pass sweeps the rows the row-k initialiser does not fill
        // (its own fill is left out of the estimate); spread over k residues.
        const int swept = rows - (plan.init_rows >= 2 ? plan.init_rows - 1 : 0);
        const double spr = all * 1e-3 * swept / k;
        snprintf(buf, sizeof(buf),
                 "%s{\"lanes\":%d,\"split_panels\":%d,\"block\":%d,\"status\":\"ok\",\"row_ms\":%.4f,"
                 "\"s_per_residue\":%.6f,\"passes\":%d}",
                 first ? "" : ",", L, split, block, row, spr, passes);
        js += buf;
        first = false;
        if (spr < best.s_per_residue) {
          best.lanes = L;
          best.passes = passes;
          best.tuning = t;
          best.row_ms = row;
          best.s_per_residue = spr;
          best_all = all;
        }
      }
  }
  if (!std::isfinite(best.s_per_residue)) {
    fdp_set_tuning(c, &saved);
    fdp_set_last_error("autotune: no candidate fits the HBM budget");
    return FDP_ERR_HBM;
  }
  fdp_status s = fdp_set_tuning(c, &best.tuning);
  // Stage 2: the cell kernel's scheduling knobs of the winner.
  struct Knob {
    const char *name;
    int fdp_tuning::*field;
    std::vector<int> values;
  };
  const Knob knobs[] = {{"lane_items", &fdp_tuning::lane_items, {4, 8, 16}},
                        {"share_min", &fdp_tuning::share_min, {2, 4, 6}},
                        {"compact_max_p", &fdp_tuning::compact_max_p, {5, 7, 9}},
                        {"compact_carry", &fdp_tuning::compact_carry, {-1, 1}},
                        {"compact_items", &fdp_tuning::compact_items, {1, 2, 4, 8}},
                        {"split_spans_min_p", &fdp_tuning::split_spans_min_p, {1, 8, 1000}}};
  if (!fdp_pass_is_whole(c, pr->n)) {
    fdp_problem cand{pr->n, best.lanes, pr->moduli, best.lanes};
    fdp_tuning cur{};
    fdp_get_tuning(c, &cur);  // the winner with its defaults resolved
    fdp_plan_out plan{};
    fdp_plan(&cand, budget, &plan);
    const int swept = rows - (plan.init_rows >= 2 ? plan.init_rows - 1 : 0);
    for (const Knob &kb : knobs) {
      // Span splitting only applies to lane counts of two spans (above 8).
      if (kb.field == &fdp_tuning::split_spans_min_p && best.lanes <= 8) continue;
      const int keep = cur.*kb.field;
      for (int v : kb.values) {
        if (s != FDP_OK || v == keep) continue;
        fdp_tuning t = cur;
        t.*kb.field = v;
        if (fdp_set_tuning(c, &t) != FDP_OK) continue;
        double row = 0, all = 0;
        if ((s = sample(best.lanes, &row, &all)) != FDP_OK) break;
        ++tried;
        const double spr = all * 1e-3 * swept / k;
        char buf[320];
        snprintf(buf, sizeof(buf), ",{\"lanes\":%d,\"%s\":%d,\"status\":\"ok\",\"row_ms\":%.4f,\"s_per_residue\":%.6f}",
                 best.lanes, kb.name, v, row, spr);
        js += buf;
        if (all < best_all * 0.995) {
          best.tuning = t;
          best_all = all;
          best.row_ms = row;
          best.s_per_residue = spr;
          cur = t;
        }
      }
      if (s == FDP_OK) s = fdp_set_tuning(c, &cur);
    }
  }
  // Known-residue check of the chosen configuration: every lane mod 4294967291
  // at the problem's n when the reference publishes that residue, else n = 9.
  if (s == FDP_OK) {
    const uint32_t m = 4294967291u;
    Known chk_known = kKnown[0];
    for (const Known &kn : kKnown)
      if (kn.n == pr->n) chk_known = kn;
    std::vector<uint32_t> mods(size_t(best.lanes), m), res(size_t(best.lanes));
    fdp_problem chk{chk_known.n, best.lanes, mods.data(), best.lanes};
    fdp_run_stats st{};
    const bool cells = fdp_pass_is_whole(c, chk_known.n);
    if (cells) fdp_pass_single_cells(c, true);
    s = fdp_run_sync(c, &chk, res.data(), &st);
    if (cells) fdp_pass_single_cells(c, false);
    if (s == FDP_OK)
      for (uint32_t r : res)
        if (r != chk_known.residue) {
          fdp_set_tuning(c, &saved);
          fdp_set_last_error("autotune: WRONG RESIDUE in the known-answer check");
          return FDP_ERR_CUDA;
        }
    best.check_n = chk_known.n;
  }
  if (s != FDP_OK) {
    fdp_set_tuning(c, &saved);
    return s;
  }
  best.residues_per_hour = 3600.0 / best.s_per_residue;
  best.candidates = tried;
  best.rejected_memory = rejected;
  char tail[512];
  snprintf(tail, sizeof(tail),
           "],\"best\":{\"lanes\":%d,\"passes\":%d,\"split_panels\":%d,\"block\":%d,\"lane_items\":%d,"
           "\"share_min\":%d,\"compact_max_p\":%d,\"compact_carry\":%d,\"compact_items\":%d,"
           "\"split_spans_min_p\":%d,\"row_ms\":%.4f,"
           "\"s_per_residue\":%.6f,\"residues_per_hour\":%.3f},\"known_residue_check\":{\"n\":%d,\"status\":\"ok\"}}",
           best.lanes, best.passes, best.tuning.split_panels, best.tuning.block, best.tuning.lane_items,
           best.tuning.share_min, best.tuning.compact_max_p, best.tuning.compact_carry, best.tuning.compact_items,
           best.tuning.split_spans_min_p, best.row_ms,
           best.s_per_residue, best.residues_per_hour, best.check_n);
  js += tail;
  if (json_out && json_cap) {
    const size_t n = std::min(json_cap - 1, js.size());
    memcpy(json_out, js.data(), n);
    json_out[n] = 0;
  }
  *out = best;
  return FDP_OK;
}
