/*
 * ias15_warm.cuh -- the learned warm start of a group's step, shared by the
 * block-cooperative kernels (ias15_coop.cuh, kernels_fast.cu).
 */
#ifndef ASSIST_GB300_IAS15_WARM_CUH
#define ASSIST_GB300_IAS15_WARM_CUH

#include "ias15_common.cuh"
#include "internal.h"
#include "mlp.cuh"

/* Shared buffers of the learned warm start (dynamic shared memory, present
 * only when a network is loaded or steps are logged). */
struct AgWarmSmem {
    AgMlpSmem M;
    double corr[7][3][32];          /* (br - er)_kc of each lane */
    float bpa[7][3][32];            /* |b_pred_kc| */
    float tgt[7][3][32];            /* logged targets */
    float xf[32][AG_MLP_IN + 1];    /* features of this step (logged with the target) */
    double kappa[7][32];
    int valid[32];
};

/* Node-0 part of the learned warm start for one group (all threads of the
 * block call it): owners publish (br - er) and |b_pred| of the particle's
 * x, y, z (variational particles keep the plain prediction), warp 0 forms
 * the features, the block runs the network, owners add kappa_k y_kc to b.
 * Every 8th step of a group is a plain probe (no inference).  Returns whether
 * the network ran (block-uniform).  pc: the position component of this warp (or
 * -1); nearest(x, y, z): distance to the nearest planet at the step's start.  Kept out of line so the plain kernel's
 * register allocation is not shaped by it. */
template <int C, class Nearest>
__device__ __noinline__ bool ag_warm_start(const AgBatchArgs& A, double* ws, int nslots, int slot, int pc, AgWarmSmem& WS,
                                           const Nearest& nearest, int lane, int wid, bool live, bool warm, bool wl_on,
                                           double hstep, double dtls, long long steps, bool& w_applied,
                                           bool& w_probe, unsigned long long& n_wused,
                                           unsigned long long& n_wfall) {
    const Ws<C> W{ws, nslots, slot};
    if (live && pc >= 0)
        for (int k = 0; k < 7; k++) {
            WS.corr[k][pc][lane] = W(W_BR + k, pc) - W(W_ER + k, pc);
            WS.bpa[k][pc][lane] = (float)fabs(W(W_B + k, pc));
        }
    __syncthreads();
    if (wid == 0) {
        bool ok = false;
        if (live) {
            double corr[7][3], kap[7];
            float bpa[7][3], x[AG_MLP_IN];
            for (int k = 0; k < 7; k++)
                for (int c = 0; c < 3; c++) { corr[k][c] = WS.corr[k][c][lane]; bpa[k][c] = WS.bpa[k][c][lane]; }
            const double x0 = W(W_X0, 0), y0 = W(W_X0, 1), z0 = W(W_X0, 2);
            const double rx = sqrt(fma(x0, x0, fma(y0, y0, z0 * z0)));
            ok = ag_warm_features(corr, bpa, hstep, dtls, rx, nearest(x0, y0, z0), x, kap);
            for (int k = 0; k < 7; k++) WS.kappa[k][lane] = kap[k];
            for (int i = 0; i < AG_MLP_IN; i++) { WS.xf[lane][i] = x[i]; WS.M.X[lane][i] = __float2bfloat16_rn(x[i]); }
        } else {
            for (int i = 0; i < AG_MLP_IN; i++) WS.M.X[lane][i] = __float2bfloat16_rn(0.0f);
        }
        WS.valid[lane] = ok ? 1 : 0;
    }
    __syncthreads();
    const bool valid = live && WS.valid[lane];
    w_probe = warm && valid && wl_on && (steps & 7) == 7;
    const bool want = warm && valid && wl_on && !w_probe;
    const bool ran = __syncthreads_or(want);
    if (ran) {
        ag_mlp_infer_block(*A.mlp, WS.M, wid, lane);
        if (want) {
            bool ok_y = true;
            for (int o = 0; o < AG_MLP_OUT; o++) {
                const float y = WS.M.Y[lane][o];
                ok_y = ok_y && isfinite(y) && fabsf(y) <= AG_MLP_YCLIP;
            }
            if (ok_y) {
                w_applied = true;
                if (pc >= 0)
                    for (int k = 0; k < 7; k++)
                        W(W_B + k, pc) = fma(WS.kappa[k][lane], (double)WS.M.Y[lane][3 * k + pc], W(W_B + k, pc));
                if (wid == 0) n_wused++;
            } else if (wid == 0) {
                n_wfall++;
            }
        }
    }
    return ran;
}

/* The logged pair of an accepted step: target = (b_conv - b_pred) / kappa with
 * b_pred = e + (br - er), the plain prediction (every thread of the block calls
 * it; lg: this lane logs). */
template <int C>
__device__ __noinline__ void ag_warm_log(const AgBatchArgs& A, double* ws, int nslots, int slot, int pc, AgWarmSmem& WS,
                                         int lane, int wid, bool lg) {
    const Ws<C> W{ws, nslots, slot};
    if (lg && pc >= 0)
        for (int k = 0; k < 7; k++) {
            const double bp = W(W_E + k, pc) + (W(W_BR + k, pc) - W(W_ER + k, pc));
            WS.tgt[k][pc][lane] = (float)((W(W_B + k, pc) - bp) / WS.kappa[k][lane]);
        }
    __syncthreads();
    if (lg && wid == 0) {
        bool fin = true;
        for (int k = 0; k < 7; k++)
            for (int c = 0; c < 3; c++) fin = fin && isfinite(WS.tgt[k][c][lane]) && fabsf(WS.tgt[k][c][lane]) < 1e6f;
        if (fin) {
            const int row = atomicAdd(A.log_count, 1);
            if (row < A.log_cap) {
                for (int i = 0; i < AG_MLP_IN; i++) A.log_x[(size_t)row * AG_MLP_IN + i] = WS.xf[lane][i];
                for (int k = 0; k < 7; k++)
                    for (int c = 0; c < 3; c++) A.log_t[(size_t)row * AG_MLP_OUT + 3 * k + c] = WS.tgt[k][c][lane];
            }
        }
    }
}

#endif
