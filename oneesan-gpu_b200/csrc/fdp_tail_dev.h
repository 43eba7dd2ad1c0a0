// Device half of the fused row tail (fdp_tail.h).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "fdp_launch.h"

namespace fdp {

// Bottom symbols s of the fused tail for a frontier of width W in the full
// space: cells s-1..1 of a row run as one pass (0: the width has no tail).
int tail_symbols(int W);
// Escape words one lane of a width-W tail needs beside its state (0: no tail).
uint64_t tail_escape_words(int W);
// Upload (once per device) the tables launch_tail uses; outside stream capture.
cudaError_t prepare_tail(int W);
// Cells tail_symbols(W)-1 .. 1 on K lanes, in place.  blk holds the blocked
// output of cell tail_symbols(W) on entry and is left as it was; the blocked
// output of cell 1 is all zero.  esc: tail_escape_words(W) x K words.
cudaError_t launch_tail(const DevTables &t, int K, const uint32_t *mods, uint32_t *main, const uint32_t *blk,
                        uint32_t *esc, cudaStream_t s, uint64_t *launches);

// Small widths: the whole residue computation of K lanes in one launch, each
// lane's state in the shared memory of one CTA; residues[l] is the result.
bool solves_whole(int W);
cudaError_t prepare_whole(int W);  // tables, once per device; outside stream capture
cudaError_t launch_whole(int W, int K, const uint32_t *mods, uint32_t *residues, cudaStream_t s);

}  // namespace fdp
