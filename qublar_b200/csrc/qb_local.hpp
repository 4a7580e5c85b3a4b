// The residual sweep of a problem whose branch fits one CTA's shared memory
// (qb_local.cu), in the lockstep or the cluster sweep's arithmetic as planned.
#pragma once

#include <cuda_runtime.h>

#include "qb_internal.hpp"
#include "qb_kernels.hpp"

namespace qb {

// Whether a problem's branch (residual pairs, bits) fits.
bool resid_local_fit(int n, int n_rays, int n_colours);
// The work table of the local sweep (host): per class, warp items of 16 lane
// pairs, a pair per 16-entry segment, a bit's pairs side by side.
void resid_local_plan(ResidualPlan& P);
// Whether a solve of R branches takes the local sweep: a plan that has it and
// whose estimated sweep time is the shorter one, unless the lockstep kernel is
// asked for (QB_RESID_KERNEL=lockstep, its phase times, or its barrier's test
// hook; QB_RESID_KERNEL=local asks for the local one).
bool resid_local_route(const ResidualPlan& p, int R);
// Branches seed0 .. seed0 + R - 1; the buffers of launch_resid_lockstep (no scratch).
qb_status launch_resid_local(const ResidualPlan& p, const SolveBuffers& b, int R, int sweeps, int refresh, uint64_t seed0,
                             cudaStream_t st);

}  // namespace qb
