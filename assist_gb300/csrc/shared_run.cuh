/*
 * shared_run.cuh -- state and control of a shared-step simulation's run
 * kernels (kernels_shared.cu, kernels_var.cu).
 */
#ifndef ASSIST_GB300_SHARED_RUN_CUH
#define ASSIST_GB300_SHARED_RUN_CUH

#include <cstddef>

#include "ias15_fast.cuh"
#include "run_ctl.h"

/* field layout: f*(3*stride) + k*stride + i */
enum { S_X0 = 0, S_V0, S_A0, S_XC, S_VC, S_AT, S_XP, S_VP, S_B, S_G = S_B + 7, S_E = S_G + 7, S_BR = S_E + 7, S_ER = S_BR + 7,
       S_PX = S_ER + 7, S_PV, S_PA, S_NF };

struct ShView {
    double* w;
    int stride;
    __device__ __forceinline__ double& operator()(int f, int k, int i) const { return w[((size_t)f * 3 + k) * stride + i]; }
};

struct ShRunArgs {
    ShView W;
    int n;
    const double* params;        /* 3 n, or null */
    double tmax, epsilon, min_dt;
    long long max_steps;         /* accepted steps after which to stop short of tmax (0: none) */
    int limit;                   /* steps of this launch */
    const ShCtl* in;
    ShCtl* out;
    unsigned long long* red;     /* ShRunMem's */
    unsigned *bar, *gave_up;
};

/* Steps of one launch (a year of 1,024 main-belt particles is 65): the device
 * is not held for longer than some tens of milliseconds at a time. */
#define SH_RUN_STEPS 256

#define SH_RUN_POLLS (1 << 22)
/* Grid barrier of one thread a block; false when its polls run out (the block
 * then leaves, and the others at their own limits). */
__device__ __forceinline__ bool sh_run_barrier(unsigned* bar) {
    volatile unsigned* vgen = bar + 1;
    const unsigned gen = *vgen;
    __threadfence();
    if (atomicAdd(&bar[0], 1u) == gridDim.x - 1) {
        atomicExch(&bar[0], 0u);
        __threadfence();
        atomicAdd(&bar[1], 1u);
        return true;
    }
    for (int k = 0; k < SH_RUN_POLLS; k++)
        if (*vgen != gen) {
            __threadfence();
            return true;
        }
    return false;
}

/* The last iteration's measures. */
struct ShMeasure {
    double db, a;
};

/* What the control warp decides at the end of an iteration. */
enum { SH_ACCEPT = 0, SH_REJECT, SH_ITERATE, SH_LEAVE };

/* An iteration's maxima over all blocks, by a block's control warp: buffer
 * round % 3 collects them, block 0 clears the next one (last read two barriers
 * ago).  False when the barrier was given up. */
__device__ __forceinline__ bool sh_run_maxima(const ShRunArgs& A, int round, int lane, double& mdb, double& ma, double& mb) {
    unsigned long long* rb = A.red + 3 * (round % 3);
    if (lane < 3) atomicMax(&rb[lane], (unsigned long long)__double_as_longlong(lane == 0 ? mdb : (lane == 1 ? ma : mb)));
    if (blockIdx.x == 0 && lane < 3) A.red[3 * ((round + 1) % 3) + lane] = 0ull;
    __threadfence();
    __syncwarp();
    bool ok = true;
    if (lane == 0) ok = sh_run_barrier(A.bar);
    ok = __shfl_sync(AG_FULL, ok ? 1 : 0, 0) != 0;
    const double r = lane < 3 ? __longlong_as_double((long long)atomicOr(&rb[lane], 0ull)) : 0.0;
    mdb = __shfl_sync(AG_FULL, r, 0);
    ma = __shfl_sync(AG_FULL, r, 1);
    mb = __shfl_sync(AG_FULL, r, 2);
    return ok;
}

/* Convergence and, once converged, acceptance and the next step's size, from
 * the maxima over all real particles, by a block's control warp (the same in
 * every block): K advanced; the decision, the step and the next one's ratio in
 * S, with S.fin set when the launch ends here. */
__device__ __forceinline__ int sh_run_decide(const ShRunArgs& A, ShCtl& K, AgFastStep& S, bool ok, double mdb, double ma, double mb,
                                             double hstep, bool last, int iters, ShMeasure& before, int lane) {
    const bool conv = ag_fast_converged(mdb, ma, iters, before.db, before.a);
    int cmd = SH_ITERATE;
    if (!ok) {
        cmd = SH_LEAVE;
    } else if (conv) {
        double dt_new = hstep;
        cmd = SH_ACCEPT;
        if (A.epsilon > 0.0) {
            const double err = mb / ma, safety = 0.25, ahs = fabs(hstep);
            if (ag_isnormal_pos(err)) dt_new = ag_inv_root7(err / A.epsilon) * hstep;
            else dt_new = hstep / safety;
            if (fabs(dt_new) < A.min_dt) dt_new = copysign(A.min_dt, dt_new);
            if (fabs(dt_new) < safety * ahs) cmd = SH_REJECT;
            else if (fabs(dt_new) > ahs / safety) dt_new = hstep / safety;
        }
        K.iterations += iters;
        if (lane == 0) {
            S.ah = hstep;
            S.aratio = cmd == SH_REJECT ? (K.dtls != 0.0 ? dt_new / K.dtls : 0.0) : dt_new / hstep;
        }
        K.dt = dt_new;
        if (cmd == SH_REJECT) {
            K.rejected++;
        } else {
            const double y = hstep + K.tc, s = K.t + y;
            K.tc = y - (s - K.t);
            K.t = s;
            K.dtls = hstep;
            K.dt_done = hstep;
            K.accepted++;
            if (last) { K.t = A.tmax; K.tc = 0.0; }
        }
    }
    if (lane == 0) {
        S.cmd = cmd;
        /* the launch ends: tmax, the steps asked for, or a barrier given up */
        S.fin = cmd == SH_LEAVE || (cmd == SH_ACCEPT && (K.t == A.tmax || (A.max_steps > 0 && K.accepted >= A.max_steps)));
    }
    return cmd;
}

#endif
