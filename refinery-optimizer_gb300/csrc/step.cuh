// Scalars and controller of one PDHG step, shared by the step forms.
#pragma once

#include "mixed.h"

namespace sihg {

__device__ __forceinline__ float* pick(float* a, float* b, int sel) { return sel ? b : a; }
__device__ __forceinline__ bool fin(float v) { return !isinf(v); }

// Scalars of an instance for the elementwise passes (computed once per chunk).
struct StepScalars {
    int cur, avg, flag;
    float w, tau;
};

__device__ __forceinline__ StepScalars step_scalars(const Inst& S) {
    return StepScalars{S.cur, S.avg_pending, S.restart_flag, (float)S.avg_w, (float)(S.eta / S.omega)};
}

// The step-size schedule factors of the current attempt: from the table, or pow
// beyond it (the table holds the same pow results).
__device__ __forceinline__ void schedule_pows(Inst& S, const Vecs& V) {
    const long long k = S.attempts + 2;
    if (k < V.pow_n) {
        const double2 p = V.pow_tab[k];
        S.pow06 = p.x;
        S.pow03 = p.y;
    } else {
        S.pow06 = pow((double)k, -0.6);
        S.pow03 = pow((double)k, -0.3);
    }
}

// Step-size controller of one instance (PDLP adaptive step), one thread.
__device__ __forceinline__ void step_controller(Inst& S, double dx2, double inter) {
    const double om = S.omega;
    const double movement = om * dx2 + S.dy2 / om;
    const double ai = fabs(inter);
    const double eta_bar = ai > 0.0 ? movement / (2.0 * ai) : INFINITY;
    // PDLP counts iterations from 1: the base k = attempts + 2 is at least 2;
    // k^-0.6 and k^-0.3 were computed by the A x kernel of this step
    const double eta = S.eta;
    const double grow = (1.0 + S.pow06) * eta;
    const double eta_next = isinf(eta_bar) ? grow : fmin((1.0 - S.pow03) * eta_bar, grow);
    S.attempts += 1;
    if (!(movement == movement) || !(inter == inter)) {  // NaN: stop as a numerical failure
        S.done = 3;
        return;
    }
    if (eta <= eta_bar) {
        S.cur ^= 1;
        S.steps += 1;
        S.since_restart += 1;
        S.W += eta;
        S.avg_w = eta / S.W;
        S.avg_pending = 1;
    } else {
        S.rejections += 1;
        S.avg_pending = 0;
    }
    S.eta = eta_next;
}

}  // namespace sihg
