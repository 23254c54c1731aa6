// Small-order transmission (n <= 32): one CTA (or two, one per contact) solves one
// (E, k) point from the lead blocks to the Caroli trace in a single launch, every block in
// shared memory or registers.
#pragma once
#include "mixed.cuh"

namespace negf {

constexpr int kSmallMax = 32;      // largest order of the small-order kernel

// The 2-contact transmission of a.npts points of order a.n <= kSmallMax (one
// shape for all; a.slices is not used): T, ncyc, status as mixed_run leaves
// them.  A point's result does not depend on the other points of the call.
// One stream operation, no workspace.
cudaError_t launch_small_points(const MixedArgs& a, cudaStream_t s);

}  // namespace negf
