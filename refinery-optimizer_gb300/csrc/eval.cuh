// Evaluation of the current and the average point: epilogues of the two SpMVs
// and the restart / termination controller, shared by the step forms.
#pragma once

#include "step.cuh"
#include "warp.cuh"

namespace sihg {

// a - (s + e) for a float a and a float-float s + e, without losing the low part
__device__ __forceinline__ float diff_ff(float a, float s, float e) {
    float h, l;
    two_sum(a, -s, h, l);
    return __fadd_rn(h, __fsub_rn(l, e));
}

// Bound violation of the float-float row activity s + e (0 inside [rl, ru]).
__device__ __forceinline__ float row_violation(float s, float e, float rl, float ru) {
    float v = 0.f;
    if (fin(rl)) v = fmaxf(v, diff_ff(rl, s, e));
    if (fin(ru)) v = fmaxf(v, -diff_ff(ru, s, e));
    return v;
}

// dual objective contribution of a row (scaling invariant), PDHG sign y
__device__ __forceinline__ void row_dual_term(Acc& acc, float y, float rl, float ru) {
    if (y < 0.f && fin(rl)) acc.add_prod(-y, rl);
    if (y > 0.f && fin(ru)) acc.add_prod(-y, ru);
}

// Row evaluation of both candidates (0 = current, 1 = average): primal
// residual of K x_c against the row bounds (scaled 2-norm^2 and original
// inf-norm), row part of the dual objective, |y_c - y_last|^2.
struct EvalRowsEpi {
    Vecs V;
    const float *xg[2], *yc;
    Acc p2[2], dterm[2], dyl2[2];
    float pinf[2];
    struct Pre { float rl, ru, dr, yc, ya, yl; };
    __device__ Pre pre(int i) const { return Pre{V.rl[i], V.ru[i], V.drow[i], yc[i], V.y_avg[i], V.y_last[i]}; }
    __device__ void begin(const Inst& S) {
        xg[0] = pick(V.x0, V.x1, S.cur);
        xg[1] = V.x_avg;
        yc = pick(V.y0, V.y1, S.cur);
    }
    __device__ const float* gather(int v) const { return xg[v]; }
    __device__ void apply(int i, const SegDot<2>& d, const Pre& p) {
        V.kx_eval[i] = d.f(1);
        const float yv[2] = {p.yc, p.ya};
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const float res = row_violation(d.s[c], d.e[c], p.rl, p.ru);
            p2[c].add(res * res);
            pinf[c] = fmaxf(pinf[c], res / p.dr);
            row_dual_term(dterm[c], yv[c], p.rl, p.ru);
            const float dy = yv[c] - p.yl;
            dyl2[c].add(dy * dy);
        }
    }
    __device__ void values(Acc (&q)[8]) {
        q[0] = p2[0];
        q[1] = p2[1];
        q[2].s = pinf[0];
        q[2].c = 0.f;
        q[3].s = pinf[1];
        q[3].c = 0.f;
        q[4] = dterm[0];
        q[5] = dterm[1];
        q[6] = dyl2[0];
        q[7] = dyl2[1];
        for (int c = 0; c < 2; ++c) {
            p2[c].reset();
            dterm[c].reset();
            dyl2[c].reset();
            pinf[c] = 0.f;
        }
    }
    __device__ void finish(Inst& S, const double* tot) {
        for (int k = 0; k < 8; ++k) S.row_eval[k] = tot[k];
    }
};

// Restart / termination controller of one instance after an evaluation.
__device__ __forceinline__ void eval_controller(Inst& S, const double* cq, unsigned* done_count) {
    const double* rq = S.row_eval;
    double kkt[2], relp[2], reld[2], relg[2];
    const bool have_avg = S.W > 0.0;
    for (int c = 0; c < 2; ++c) {
        const double pobj = cq[4 + c];
        const double dobj = rq[4 + c] + cq[6 + c];
        const double gap = fabs(pobj - dobj);
        relp[c] = rq[2 + c] / (1.0 + S.b_inf);
        reld[c] = cq[2 + c] / (1.0 + S.c_inf);
        relg[c] = gap / (1.0 + fabs(pobj) + fabs(dobj));
        kkt[c] = sqrt(S.omega * rq[0 + c] + cq[0 + c] / S.omega + gap * gap);
        S.pobj[c] = pobj;
        S.dobj[c] = dobj;
        S.rel_p[c] = relp[c];
        S.rel_d[c] = reld[c];
        S.rel_g[c] = relg[c];
    }
    if (!have_avg) kkt[1] = INFINITY;
    S.evals += 1;
    S.avg_pending = 0;
    S.restart_flag = 0;
    if (!(kkt[0] == kkt[0])) {
        S.done = 3;
        S.out_sel = 0;
        atomicAdd(done_count, 1u);
        return;
    }
    // termination: current first, then the average
    for (int c = 0; c < 2; ++c) {
        if (c == 1 && !have_avg) break;
        if (relp[c] <= S.tol_p && reld[c] <= S.tol_d && relg[c] <= S.tol_g) {
            S.done = 1;
            S.out_sel = c;
            atomicAdd(done_count, 1u);
            return;
        }
    }
    const int cand = kkt[1] < kkt[0] ? 1 : 0;
    if (S.attempts >= S.max_attempts) {
        S.done = 2;
        S.out_sel = cand;
        atomicAdd(done_count, 1u);
        return;
    }
    const double worst = fmax(relp[cand] / S.tol_p, fmax(reld[cand] / S.tol_d, relg[cand] / S.tol_g));
    if (S.compensated == 2 || (S.compensated == 1 && worst < 100.0)) S.refine = 1;
    const double kc = kkt[cand];
    if (S.evals == 1) {  // initial point: record it as the last restart point
        S.kkt_last = kc;
        S.kkt_prev = kc;
        S.restart_flag = 1;
        return;
    }
    if (!S.enable_restart) return;
    const bool restart = kc <= S.beta_suff * S.kkt_last ||
                         (kc <= S.beta_nec * S.kkt_last && kc > S.kkt_prev) ||
                         (double)S.since_restart >= S.beta_art * (double)S.steps;
    S.kkt_prev = kc;
    if (!restart) return;
    const double dxn = sqrt(S.col_eval_dist[cand]), dyn = sqrt(S.row_eval[6 + cand]);
    if (dxn > 1e-10 && dyn > 1e-10) {
        const double th = S.weight_smoothing;
        S.omega = exp(th * log(dyn / dxn) + (1.0 - th) * log(S.omega));
    }
    S.kkt_last = kc;
    S.restart_flag = cand == 1 ? 2 : 1;
    S.restarts += 1;
    S.since_restart = 0;
    S.W = 0.0;
}

// Column evaluation of both candidates: reduced cost lambda = c + K^T y_c,
// dual residual (the parts no finite bound carries; scaled 2-norm^2 and
// original inf-norm), primal objective, column part of the dual objective,
// |x_c - x_last|^2.  The warp completing an instance runs its controller.
struct EvalColsEpi {
    Vecs V;
    unsigned* done_count;
    const float *yg[2], *xc;
    Acc d2[2], pobj[2], dterm[2], dxl2[2];
    float dinf[2];
    struct Pre { float c, l, u, dc, xc, xa, xl; };
    __device__ Pre pre(int j) const {
        return Pre{V.c[j], V.l[j], V.u[j], V.dcol[j], xc[j], V.x_avg[j], V.x_last[j]};
    }
    __device__ void begin(const Inst& S) {
        yg[0] = pick(V.y0, V.y1, S.cur);
        yg[1] = V.y_avg;
        xc = pick(V.x0, V.x1, S.cur);
    }
    __device__ const float* gather(int v) const { return yg[v]; }
    __device__ void apply(int j, const SegDot<2>& d, const Pre& p) {
        V.kty_eval[j] = d.f(1);
        const float xv[2] = {p.xc, p.xa};
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            float h, lo;  // lambda = c + (s + e) as the float-float h + lo
            two_sum(p.c, d.s[k], h, lo);
            lo = __fadd_rn(lo, d.e[k]);
            const float lam = __fadd_rn(h, lo);
            float rd = 0.f;
            if (lam > 0.f) {
                if (fin(p.l)) { dterm[k].add_prod(h, p.l); dterm[k].add(lo * p.l); } else rd = lam;
            } else if (lam < 0.f) {
                if (fin(p.u)) { dterm[k].add_prod(h, p.u); dterm[k].add(lo * p.u); } else rd = -lam;
            }
            d2[k].add(rd * rd);
            dinf[k] = fmaxf(dinf[k], rd / p.dc);
            pobj[k].add_prod(p.c, xv[k]);
            const float dx = xv[k] - p.xl;
            dxl2[k].add(dx * dx);
        }
    }
    __device__ void values(Acc (&q)[10]) {
        q[0] = d2[0];
        q[1] = d2[1];
        q[2].s = dinf[0];
        q[2].c = 0.f;
        q[3].s = dinf[1];
        q[3].c = 0.f;
        q[4] = pobj[0];
        q[5] = pobj[1];
        q[6] = dterm[0];
        q[7] = dterm[1];
        q[8] = dxl2[0];
        q[9] = dxl2[1];
        for (int k = 0; k < 2; ++k) {
            d2[k].reset();
            pobj[k].reset();
            dterm[k].reset();
            dxl2[k].reset();
            dinf[k] = 0.f;
        }
    }
    __device__ void finish(Inst& S, const double* tot) {
        S.col_eval_dist[0] = tot[8];
        S.col_eval_dist[1] = tot[9];
        eval_controller(S, tot, done_count);
    }
};

}  // namespace sihg
