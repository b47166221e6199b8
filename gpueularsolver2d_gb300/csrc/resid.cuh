// resid.cuh -- the end of an iteration's residual, shared by the residual
// kernels (resid.cu) and the small-mesh kernel (small32.cuh).
#pragma once

#include "dev_types.h"

namespace e2d {

// drou -> Resd = sqrt((drou + 1e-32) / EPSM) with EPSM = drou of iteration 1
// unless the caller fixed it.  Sets halt when the loop condition of
// gpu_solver.cu:2200 (step < MAXSTEP && Resd > EPSL) fails or the state went
// unphysical.  One thread.
__device__ __forceinline__ void resid_finish(const double drou, Ctl *ctl, double *hist, int hist_cap) {
    const int step = ctl->step + 1;
    if (step == 1 && !ctl->fixed_norm) ctl->epsm = drou;
    const double resd = sqrt((drou + 1.0E-32) / ctl->epsm);
    if (step - 1 < hist_cap) hist[step - 1] = resd;
    ctl->step = step;
    ctl->resd = resd;
    for (int k = 0; k < 8; k++) ctl->dtmin[k] = kDtNone;  // global time-step slots for the next iteration
    if ((ctl->freeze_after > 0 && step >= ctl->freeze_after) || (ctl->freeze_resd > 0.0 && resd <= ctl->freeze_resd))
        ctl->frozen = 1;
    if (ctl->nbad) ctl->halt = 2;
    else if (ctl->check_epsl && !(resd > ctl->epsl)) ctl->halt = 1;
    else if (step >= ctl->target) ctl->halt = 1;
}

}  // namespace e2d
