// gpp_far.h -- unoccupied bands with per-band frequencies through a series
// for the frequencies away from wtilde (gpp_far.cu).
#pragma once

#include <cuda_runtime.h>

#include "gpp_gb300.h"
#include "gpp_kernels.h"

namespace gpp {

// Whether a call of these sizes takes the series (the device still decides
// from wtilde and wx whether it pays, and runs the per-term kernel where it
// does not): the same rule for every entry point, so that a state gives the
// same bits through all of them.
bool far_eligible(const Problem &p, int bands, bool mixed);

size_t far_bytes(const Problem &p, int bands, bool mixed);

// Unoccupied bands [b0, b1): writes their total into the first unoccupied
// slot of each frequency (part.ach_tile0) and band (part.n1, when set), all
// other slots being zero, or leaves them untouched.  *active is the device
// word that says which: the per-term launch takes it as its `skip`.  split_ws:
// the split planes of the bands and rows (mixed), or null (FP64).
cudaError_t far_unoccupied(const Problem &p, const Partials &part, void *ws, void *split_ws, int b0,
                           int b1, cudaStream_t s, const int **active);

// The near list's per-term sums in mixed precision (gpp_mixed.cu).
cudaError_t launch_near_mixed(const Problem &p, const Partials &part, void *split_ws,
                              const FarNear &near, int cap, cudaStream_t s);

}  // namespace gpp
