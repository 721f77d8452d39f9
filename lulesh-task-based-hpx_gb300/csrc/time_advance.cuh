// Device-side TimeIncrement, shared by the time kernels and by the material
// kernel, whose last block advances the time of the graph form's next cycle.
// Units compile it with and without contraction. The one product that could
// reach a sum, olddt * deltatimemultub, is rounded by itself (__dmul_rn; the
// others are exact or divided), so all round as the host TimeIncrement does,
// and the graph forms and the host loop pick identical time steps.
#pragma once

#include "lulesh_dev.h"

namespace lulesh {

// Loop condition of hpx_main (lulesh.cc:2374-2375) followed by
// TimeIncrement (lulesh.cc:182-229). Returns false when the loop has ended
// (or an error stopped it) and marks the state inactive.
static __device__ __forceinline__ bool advance_time(DevTime* t, const StepResult* r) {
    if (t->max_cycles < 0 || r->err != 0 || !(t->time < t->stoptime && t->cycle < t->max_cycles)) {
        t->active = 0;
        return false;
    }
    t->active = 1;
    double targetdt = t->stoptime - t->time;
    if ((t->dtfixed <= 0.0) && (t->cycle != 0)) {
        const double olddt = t->deltatime;
        double gnewdt = 1.0e+20;
        if (t->dtcourant < gnewdt) gnewdt = t->dtcourant / 2.0;
        if (t->dthydro < gnewdt) gnewdt = t->dthydro * 2.0 / 3.0;
        double newdt = gnewdt;
        const double ratio = newdt / olddt;
        if (ratio >= 1.0) {
            if (ratio < t->deltatimemultlb) newdt = olddt;
            else if (ratio > t->deltatimemultub) newdt = __dmul_rn(olddt, t->deltatimemultub);
        }
        if (newdt > t->dtmax) newdt = t->dtmax;
        t->deltatime = newdt;
    }
    if ((targetdt > t->deltatime) && (targetdt < (4.0 * t->deltatime / 3.0)))
        targetdt = 2.0 * t->deltatime / 3.0;
    if (targetdt < t->deltatime) t->deltatime = targetdt;
    t->time += t->deltatime;
    ++t->cycle;
    return true;
}

// Stores the cycle's dt minima (lulesh.cc:2229-2236) and stops the loop on a
// device error.
static __device__ __forceinline__ void finish_time(DevTime* t, const StepResult* r) {
    t->dtcourant = r->dtcourant;
    t->dthydro = r->dthydro;
    if (r->err != 0) t->active = 0;
}

}  // namespace lulesh
