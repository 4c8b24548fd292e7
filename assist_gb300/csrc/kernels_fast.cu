/*
 * kernels_fast.cu -- K4f: the batched persistent IAS15 on the evaluation of
 * fast_forces.cuh (the default batched path; ag_fast_covers says which force
 * configurations it takes, the block-cooperative kernel of ias15_coop.cuh has
 * the others and the variational particles).
 *
 * A group of up to 32 particles that share their step times is integrated by
 * one block, as in ias15_coop.cuh, with the same step rules and statuses.
 * What differs is where the work goes: eight warps with the shares of
 * ag_fast_force and ias15_fast.cuh, of which warp 1 controls the steps (sizes,
 * times, convergence, retirement: lane masks the other warps read); the
 * step's eight tables are built together at its start; the quadratures
 * multiply by reciprocals and the step-size root is a Newton iteration (a
 * warp's FP64 division is 8.5 instructions, its pow 100).
 */
#include <cuda_runtime.h>

#include <type_traits>

#include "device_forces.cuh"
#include "internal.h"
#include "ias15_fast.cuh"
#include "ias15_warm.cuh"

enum { AG_CMD_STEP = 0, AG_CMD_DONE };

struct AgFastSmem {
    AgFastStep S;
    int g, stop, stage_fail, rot;
    int wg_off;                     /* learned warm start switched off for this group */
    double dtls;                    /* what the warm start reads of the control warp's state */
    long long steps;
};

/* Dynamic shared memory: the group's IAS15 state (40 fields x 3 components x
 * 32 lanes, 30 KB), the staged record (STAGE), the warm start's buffers
 * (WARM), the eight tables. */
template <bool STAGE, bool WARM>
struct AgFastDyn {
    static constexpr size_t ws = sizeof(double) * W_NF * 3 * 32;
    static constexpr size_t stage = STAGE ? (sizeof(AgRecStage) + 15) / 16 * 16 : 0;
    static constexpr size_t warm_off = ws + stage;
    static constexpr size_t tab_off = warm_off + (WARM ? (sizeof(AgWarmSmem) + 15) / 16 * 16 : 0);
    __host__ __device__ static size_t bytes(int n_ast) { return tab_off + 8 * (size_t)AgFastLayout(n_ast).stride; }
};

/* Dense output of component c: the states at the output times this step
 * covers, by ASSIST's interpolation (src/assist.c:556-597). */
static __device__ __noinline__ int ag_fast_dense(const AgBatchArgs& A, const Ws<3>& W, int c, int on, int on_end, double dir,
                                                 double t, double tc, double hstep, bool last, double tend) {
    const double tstep_end = (t + tc) + hstep;
    while (on < on_end && dir * (A.out_t[on] - tstep_end) <= 0.0 && !(last && A.out_t[on] == tend)) {
        if (c >= 0) {
            const double h = ((A.out_t[on] - t) - tc) / hstep;
            double s[9], sv[8];
            s[0] = hstep * h;
            s[1] = s[0] * s[0] / 2.;
            s[2] = s[1] * h / 3.;
            s[3] = s[2] * h / 2.;
            s[4] = 3. * s[3] * h / 5.;
            s[5] = 2. * s[4] * h / 3.;
            s[6] = 5. * s[5] * h / 7.;
            s[7] = 3. * s[6] * h / 4.;
            s[8] = 7. * s[7] * h / 9.;
            sv[0] = hstep * h;
            sv[1] = sv[0] * h / 2.;
            sv[2] = 2. * sv[1] * h / 3.;
            sv[3] = 3. * sv[2] * h / 4.;
            sv[4] = 4. * sv[3] * h / 5.;
            sv[5] = 5. * sv[4] * h / 6.;
            sv[6] = 6. * sv[5] * h / 7.;
            sv[7] = 7. * sv[6] * h / 8.;
            const double b0 = W(W_B + 0, c), b1 = W(W_B + 1, c), b2 = W(W_B + 2, c), b3 = W(W_B + 3, c),
                         b4 = W(W_B + 4, c), b5 = W(W_B + 5, c), b6 = W(W_B + 6, c);
            const double a0 = W(W_A0, c), v0 = W(W_V0, c);
            A.out_state[6 * (size_t)on + c] = W(W_X0, c) + (s[8] * b6 + s[7] * b5 + s[6] * b4 + s[5] * b3 + s[4] * b2 +
                                                            s[3] * b1 + s[2] * b0 + s[1] * a0 + s[0] * v0);
            A.out_state[6 * (size_t)on + 3 + c] =
                v0 + sv[7] * b6 + sv[6] * b5 + sv[5] * b4 + sv[4] * b3 + sv[3] * b2 + sv[2] * b1 + sv[1] * b0 + sv[0] * a0;
        }
        on++;
    }
    return on;
}

/* Distance to the nearest of the eleven planets at table 0. */
struct AgFastNearest {
    const AgFastView& V;
    __device__ __forceinline__ double operator()(double x, double y, double z) const {
        double m = 1e300;
        for (int k = -2; k < AG_PAIR_PL; k++) {
            const double* o = k == -2 ? V.node(0).rs : (k == -1 ? V.node(0).rj : V.rel(0) + 3 * k);
            const double dx = x + o[0], dy = y + o[1], dz = z + o[2];
            m = fmin(m, fma(dx, dx, fma(dy, dy, dz * dz)));
        }
        return sqrt(m);
    }
};

/* OCC: resident blocks per SM; STAGE: the active .440 record staged in shared
 * memory; WARM: the learned warm start and the logging of its pairs.  The
 * arithmetic is the same in all. */
template <int OCC, bool STAGE, bool WARM>
__global__ void __launch_bounds__(AG_FAST_THREADS, OCC) ag_k_fast(const DevEphem* __restrict__ Ep, ForceCfg cf, AgBatchArgs A) {
    const DevEphem& E = *Ep;
    __shared__ AgFastSmem M;
    AgFastStep& S = M.S;
    /* role rotation, as in ias15_coop.cuh: blocks sharing an SM put different
     * roles on each sub-partition */
    if (threadIdx.x == 0) {
        int r = 0;
        if (A.sm_slots) {
            unsigned smid;
            asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
            r = atomicAdd(&A.sm_slots[smid & (AG_SM_SLOTS - 1)], 1) & 3;
        }
        M.rot = r;
        M.stop = 0;
        M.stage_fail = 0;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = ((threadIdx.x >> 5) + M.rot) & 7, tid = (wid << 5) | lane;
    const int pc = ag_fast_comp(wid), hc = ag_fast_help(wid);
    const bool ctl = wid == 1;
    extern __shared__ __align__(16) unsigned char ag_dyn_smem[];
    const Ws<3> W{reinterpret_cast<double*>(ag_dyn_smem), 32, lane};
    AgRecStage* const R = STAGE ? reinterpret_cast<AgRecStage*>(ag_dyn_smem + AgFastDyn<STAGE, WARM>::ws) : nullptr;
    const AgFastView V(ag_dyn_smem + AgFastDyn<STAGE, WARM>::tab_off, E.n_ast);
    AgWarmSmem& WS = *reinterpret_cast<AgWarmSmem*>(ag_dyn_smem + AgFastDyn<STAGE, WARM>::warm_off);
    const bool warm = WARM && A.mlp != nullptr, logp = WARM && A.log_x != nullptr;
    AgStageCursor cur;
    if (STAGE && tid == 0) ag_mbar_init(&R->bar);
    ag_fast_masses(E, cf, S.F, tid);
    const long long clk0 = clock64();
    unsigned long long n_acc = 0, n_rej = 0, n_ev = 0, n_it = 0, n_tab = 0, n_wused = 0, n_wfall = 0;
    const unsigned bit = 1u << lane;
    const bool dense = A.out_start != nullptr;
    const double nan = __longlong_as_double(0x7ff8000000000000LL);

    while (true) {
        __syncthreads();
        if (tid == 0) M.g = atomicAdd(A.queue, 1);
        __syncthreads();
        const int g = M.g;
        if (g >= A.n_groups) break;
        const int gs = A.grp_size[g], g0 = A.grp_start[g];
        if (M.stop || M.stage_fail) {
            /* run-time budget spent (or a record copy lost): groups still
             * queued are not integrated (state untouched) and say so */
            if (wid == 0 && lane < gs) {
                const int p = A.order[g0 + lane];
                if (A.status) A.status[p] = AG_ST_TIMEOUT;
                if (dense)
                    for (int q = A.out_start[p]; q < A.out_start[p + 1]; q++)
                        for (int k = 0; k < 6; k++) A.out_state[6 * (size_t)q + k] = nan;
            }
            continue;
        }
        const int pid = lane < gs ? A.order[g0 + lane] : -1;
        const double ts = A.t0[A.order[g0]];
        const double tend = pid >= 0 ? A.t_end[pid] : ts;
        double dir;
        {
            const double d = tend - ts;
            const unsigned fwd = __ballot_sync(AG_FULL, d > 0.0), bwd = __ballot_sync(AG_FULL, d < 0.0);
            dir = fwd ? 1.0 : (bwd ? -1.0 : 1.0);
        }
        double prm[3] = {0.0, 0.0, 0.0};
        if (pid >= 0) {
            if (pc >= 0) {
                const double* s0 = A.state + 6 * (size_t)pid;
                W(W_X0, pc) = s0[pc]; W(W_V0, pc) = s0[3 + pc]; W(W_XC, pc) = 0.0; W(W_VC, pc) = 0.0;
                for (int k = 0; k < 7; k++) {
                    W(W_B + k, pc) = 0.0; W(W_E + k, pc) = 0.0; W(W_BR + k, pc) = 0.0; W(W_ER + k, pc) = 0.0;
                }
            }
            if (ctl && A.params)
                for (int k = 0; k < 3; k++) prm[k] = A.params[3 * (size_t)pid + k];
        }
        int on = 0, on_end = 0;                 /* dense output cursor (times sorted along the integration) */
        if (dense && pid >= 0) { on = A.out_start[pid]; on_end = A.out_start[pid + 1]; }
        /* the control warp's state of the group and of its lane */
        double t = ts, tc = 0.0, dt = dir * fabs(A.dt0), dtls = 0.0, hstep = 0.0;
        long long steps = 0;
        int pstat = AG_ST_OK;
        /* the learned start runs in a group until its learned steps take longer
         * than its plain probes (every 8th step), timed by thread 0 from the
         * step's tables to its converged corrector, and for a member until its
         * learned starts converge in more iterations than its probes */
        long long wg_t_l = 0, wg_t_p = 0, clk_step = 0;
        int wg_n_l = 0, wg_n_p = 0, wl_sum_l = 0, wl_n_l = 0, wl_sum_p = 0, wl_n_p = 0;
        bool wl_on = warm;
        if (WARM && tid == 0) M.wg_off = 0;
        bool clive = pid >= 0, cfin = clive && tend == ts, clast = false, last_group = false;
        while (true) {
            /* ---- control: who retires, the watchdog, the next step */
            if (ctl) {
                const unsigned live = __ballot_sync(AG_FULL, clive);
                unsigned fin = __ballot_sync(AG_FULL, clive && cfin);
                if (live & ~fin) {
                    /* a spent budget retires everyone */
                    const bool out = M.stage_fail || (A.watchdog_cycles > 0 && clock64() - clk0 > A.watchdog_cycles);
                    if (__any_sync(AG_FULL, out)) {
                        if (clive && !cfin) { pstat = AG_ST_TIMEOUT; cfin = true; }
                        fin = live;
                        if (lane == 0) M.stop = 1;
                    }
                }
                const bool go = clive && !cfin;
                const double rem = go ? fabs((tend - t) - tc) : 1e300;
                const double rem_min = ag_warp_min_nonneg(rem);
                last_group = fabs(dt) >= rem_min;
                hstep = last_group ? dir * rem_min : dt;
                clast = go && last_group && rem == rem_min;
                const unsigned lastm = __ballot_sync(AG_FULL, clast);
                if (live & ~fin) ag_fast_nodes(S, lane, t, tc, hstep);
                if (lane == 0) {
                    S.live = live & ~fin; S.fin = fin; S.last = lastm;
                    S.hstep = hstep; S.t = t; S.tc = tc;
                    if (WARM) { M.dtls = dtls; M.steps = steps; }
                }
            }
            __syncthreads();
            /* ---- retire lanes whose particle is complete */
            const unsigned fin = S.fin, livem = S.live;
            if (fin) {
                bool finite = true;
                if ((fin & bit) && pc >= 0) {
                    const double x1 = W(W_X0, pc) + W(W_XC, pc), v1 = W(W_V0, pc) + W(W_VC, pc);
                    double* s0 = A.state + 6 * (size_t)pid;
                    s0[pc] = x1; s0[3 + pc] = v1;
                    finite = isfinite(x1) && isfinite(v1);
                }
                const unsigned nf = __ballot_sync(AG_FULL, !finite);
                if (lane == 0 && pc >= 0) S.nf[pc] = nf;
                if (ctl && lane == 0) S.cmd = 0;
                __syncthreads();
                if (fin & bit) {
                    if (ctl) {
                        if (pstat == AG_ST_OK && ((S.nf[0] | S.nf[1] | S.nf[2]) & bit)) pstat = AG_ST_NONFINITE;
                        if (A.status) A.status[pid] = pstat;
                        clive = false;
                        cfin = false;
                    }
                }
                if (dense) {
                    /* times left at a completed particle are its t_end: the end
                     * state; a particle stopped early leaves NaN at the times it
                     * did not reach */
                    const unsigned okm = __ballot_sync(AG_FULL, (fin & bit) && pstat != AG_ST_OK &&
                                                                     pstat != AG_ST_NONFINITE);
                    if (ctl && lane == 0) S.cmd = (int)okm;
                    __syncthreads();
                    if ((fin & bit) && pc >= 0) {
                        const bool done_ok = !((unsigned)S.cmd & bit);
                        const double x1 = W(W_X0, pc) + W(W_XC, pc), v1 = W(W_V0, pc) + W(W_VC, pc);
                        for (int q = on; q < on_end; q++) {
                            A.out_state[6 * (size_t)q + pc] = done_ok ? x1 : nan;
                            A.out_state[6 * (size_t)q + 3 + pc] = done_ok ? v1 : nan;
                        }
                    }
                    __syncthreads();
                }
            }
            if (!livem) break;
            const bool live = (livem & bit) != 0;

            /* ---- the step's eight tables */
            const double* srec = nullptr;
            const double* ssrc = nullptr;
            if constexpr (STAGE) {
                double tf;
                if (!E.pl_spk && E.pl_rec_len <= AG_STAGE_MAX_REC && ag_planet_record(E, S.ptn[0], &ssrc, &tf) == AG_OK) {
                    int fail = 0;
                    srec = ag_stage_record(E, ssrc, *R, tid, cur, &fail);
                    if (fail) { M.stage_fail = 1; srec = nullptr; }
                }
            }
            if (live) ag_fast_predict(W, S, pc, hc, lane, 0);
            n_tab += 8;
            if (WARM && tid == 0) clk_step = clock64();
            if (ag_fast_tables(E, cf, 8, S.ptn, V, S.F, tid, srec, ssrc)) {
                if (clive) { pstat = M.stage_fail ? AG_ST_TIMEOUT : AG_ST_COVERAGE; cfin = true; }
                continue;
            }
            /* ---- node 0 */
            const double* Ap = A.params ? prm : nullptr;
            ag_fast_force(wid, lane, live, E, cf, V, 0, S.F, Ap);
            if (ctl && live) n_ev++;
            __syncthreads();
            bool w_applied = false, w_probe = false, w_ran = false;
            long long wsteps = 0;
            if (live && pc >= 0) W(W_A0, pc) = ag_fast_sum(S.F, pc, lane);
            if constexpr (WARM) {
                wsteps = M.steps;
                if (warm || logp)
                    w_ran = ag_warm_start<3>(A, W.w, W.ns, W.slot, pc, WS, AgFastNearest{V}, lane, wid, live, warm,
                                             wl_on && M.wg_off == 0, S.hstep, M.dtls, wsteps, w_applied, w_probe,
                                             n_wused, n_wfall);
                __syncthreads();        /* the owners' b for the helpers */
            }
            if (live) ag_fast_start(W, pc, hc);
            __syncthreads();            /* a0 for the velocity predictor's warps */
            /* ---- predictor-corrector iterations */
            int iters = 1, it_lane = 0;
            double last_db = 0.0, last_a = 0.0, ma7 = 0.0, mb6 = 0.0;
            bool conv = !live;
            while (true) {
                for (int n = 1; n < 8; n++) {
                    if (!conv) ag_fast_predict(W, S, pc, hc, lane, n);
                    __syncthreads();
                    ag_fast_force(wid, lane, !conv, E, cf, V, n, S.F, Ap);
                    if (ctl && !conv) n_ev++;
                    __syncthreads();
                    if (!conv && pc >= 0) ag_fast_correct(W, S, pc, lane, n);
                    __syncthreads();
                }
                if (ctl) {
                    /* one warp judges */
                    bool c = conv;
                    if (!c) {
                        ma7 = ag_max3(S.ra, lane);
                        mb6 = ag_max3(S.rb6, lane);
                        c = ag_fast_converged(ag_max3(S.rdb, lane), ma7, iters, last_db, last_a);
                        if (c) n_it += (unsigned long long)iters;
                    }
                    const unsigned m = __ballot_sync(AG_FULL, c);
                    if (lane == 0) S.conv = m;
                }
                __syncthreads();
                const unsigned done = S.conv;
                if (!conv && (done & bit)) { conv = true; it_lane = iters; }
                if (done == 0xffffffffu) break;
                iters++;
            }
            if (WARM && warm && live) {
                if (w_applied) { wl_sum_l += it_lane; wl_n_l++; }
                else if (w_probe) {
                    wl_sum_p += it_lane; wl_n_p++;
                    if (wl_n_p >= 4 && wl_n_l >= 8 && (long long)wl_sum_l * wl_n_p > (long long)wl_sum_p * wl_n_l) {
                        wl_on = false;
                        if (wid == 0) n_wfall++;
                    }
                }
            }
            if (WARM && warm && !A.warm_no_time_fallback && tid == 0 && M.wg_off == 0) {
                const long long dt_clk = clock64() - clk_step;
                if (w_ran) { wg_t_l += dt_clk; wg_n_l++; }
                else if ((wsteps & 7) == 7) { wg_t_p += dt_clk; wg_n_p++; }
                if (wg_n_p >= 3 && wg_n_l >= 12 && (double)wg_t_l / wg_n_l > (double)wg_t_p / wg_n_p) {
                    M.wg_off = 1;
                    n_wfall++;
                }
            }
            /* ---- step-size control: each lane's choice, the group takes the smallest */
            bool skip = false, reject = false;
            double dt_new = dt;
            if (ctl) {
                double dn_l = 1e300, nocap_l = 1e300;
                bool rej_l = false;
                if (A.epsilon > 0.0 && live) {
                    const double err = mb6 / ma7, safety = 0.25;
                    double dn;
                    if (ag_isnormal_pos(err)) dn = ag_inv_root7(err / A.epsilon) * hstep;
                    else dn = hstep / safety;
                    if (fabs(dn) < A.min_dt) dn = copysign(A.min_dt, dn);
                    nocap_l = fabs(dn);
                    const double ahs = fabs(hstep);
                    if (nocap_l < safety * ahs) rej_l = true;
                    else if (nocap_l > ahs / safety) dn = hstep / safety;
                    dn_l = fabs(dn);
                }
                if (live && !last_group && A.epsilon > 0.0 && A.dt_floor > 0.0 && nocap_l < A.dt_floor) {
                    /* step underflow: this lane's particle is hitting a body; it stops
                     * and the group goes on without it.  Not tested on a step cut short
                     * to land on a member's t_end: the proposals scale with that step */
                    pstat = AG_ST_UNDERFLOW;
                    cfin = true;
                    rej_l = false;
                    dn_l = 1e300;
                    nocap_l = 1e300;
                }
                /* only underflowing lanes left: no step */
                skip = __any_sync(AG_FULL, cfin) && !__any_sync(AG_FULL, live && !cfin);
                if (A.epsilon > 0.0) {
                    dt_new = dir * ag_warp_min_nonneg(dn_l);
                    /* a step shortened to land on a lane's t_end does not shrink the
                     * group's step beyond what the error control asks for */
                    const double nc = ag_warp_min_nonneg(nocap_l);
                    if (last_group) dt_new = dir * fmin(fabs(dt), fmax(fabs(dt_new), nc));
                }
                reject = __any_sync(AG_FULL, rej_l);
                if (lane == 0) {
                    S.cmd = skip ? 2 : (reject ? 1 : 0);
                    S.ah = hstep;
                    /* rejected: over the last accepted step (0: none yet) */
                    S.aratio = reject ? (dtls != 0.0 ? dt_new / dtls : 0.0) : dt_new / hstep;
                }
            }
            __syncthreads();
            const int cmd = S.cmd;
            if (cmd == 2) continue;
            if (cmd == 1) {
                if (live) ag_fast_retry(W, pc, hc, S.aratio);
                if (ctl) {
                    if (live) n_rej++;
                    dt = dt_new;
                }
                continue;
            }
            if constexpr (WARM) {
                if (logp)
                    ag_warm_log<3>(A, W.w, W.ns, W.slot, pc, WS, lane, wid,
                                   live && WS.valid[lane] && (wsteps % A.log_every) == 0);
            }
            /* ---- accept */
            if (dense && live) on = ag_fast_dense(A, W, pc, on, on_end, dir, S.t, S.tc, S.ah, (S.last & bit) != 0, tend);
            ag_fast_accept(W, pc, hc, live, S.ah, S.aratio);
            if (ctl) {
                if (live) n_acc++;
                const double y = hstep + tc, s = t + y;
                tc = y - (s - t);
                t = s;
                dtls = hstep;
                dt = dt_new;
                steps++;
                if (clast) cfin = true;
                if (last_group && live && !clast && fabs((tend - t) - tc) == 0.0) cfin = true;
                if (A.max_steps > 0 && steps >= A.max_steps && live && !cfin) { pstat = AG_ST_BUDGET; cfin = true; }
            }
            /* dense output reads this step's t and tc before the control warp writes the next's */
            if (dense) __syncthreads();
        }
    }
    if (ctl) {
        atomicAdd(&A.counters[0], n_acc);
        atomicAdd(&A.counters[1], n_rej);
        atomicAdd(&A.counters[2], n_ev);
        atomicAdd(&A.counters[3], n_it);
    }
    if (WARM && wid == 0) {
        atomicAdd(&A.counters[4], n_wused);
        atomicAdd(&A.counters[5], n_wfall);
    }
    if (tid == 0) atomicAdd(&A.counters[6], n_tab);
    /* a copy that did not complete in time: wait for it once more (bounded)
     * before the block's shared memory is released */
    if (STAGE && tid == 0 && M.stage_fail) ag_mbar_wait(&R->bar, cur.phase ^ 1u);
}

/* Opt the kernel in to its dynamic shared memory (above the 48 KB default). */
template <int OCC, bool STAGE, bool WARM>
static int ag_fast_attr() {
    return (int)cudaFuncSetAttribute(ag_k_fast<OCC, STAGE, WARM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)AgFastDyn<STAGE, WARM>::bytes(AG_MAX_AST));
}

template <int OCC, bool STAGE, bool WARM>
static int ag_fast_blocks_per_sm(int n_ast) {
    int bps = 0;
    if (ag_fast_attr<OCC, STAGE, WARM>() == 0)
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, ag_k_fast<OCC, STAGE, WARM>, AG_FAST_THREADS,
                                                      AgFastDyn<STAGE, WARM>::bytes(n_ast));
    return bps;
}

/* Slots (32 per resident block) of a build (occ 2 or 3, stage only with 2, or
 * the learned warm start) with n_ast asteroids on the current device. */
int ag_fast_max_slots(int occ, int stage, int warm, int n_ast) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int bps = warm ? ag_fast_blocks_per_sm<2, false, true>(n_ast)
              : occ == 3 ? ag_fast_blocks_per_sm<3, false, false>(n_ast)
                         : (stage ? ag_fast_blocks_per_sm<2, true, false>(n_ast) : ag_fast_blocks_per_sm<2, false, false>(n_ast));
    if (bps < 1) bps = 1;
    return sms * bps * 32;
}

template <int OCC, bool STAGE, bool WARM>
static int ag_fast_go(const DevEphem& E, const ForceCfg& c, const AgBatchArgs& a, cudaStream_t s) {
    const int e = ag_fast_attr<OCC, STAGE, WARM>();
    if (e) return e;
    ag_k_fast<OCC, STAGE, WARM><<<(a.nslots + 31) / 32, AG_FAST_THREADS, AgFastDyn<STAGE, WARM>::bytes(E.n_ast), s>>>(E.self_dev, c, a);
    return (int)cudaGetLastError();
}

int ag_launch_fast(const DevEphem& E, const ForceCfg& c, const AgBatchArgs& a, int occ, int stage, cudaStream_t s) {
    const int e = ag_ias_tables_init();
    if (e) return e;
    if (a.mlp || a.log_x) return ag_fast_go<2, false, true>(E, c, a, s);
    if (occ == 3) return ag_fast_go<3, false, false>(E, c, a, s);
    return stage ? ag_fast_go<2, true, false>(E, c, a, s) : ag_fast_go<2, false, false>(E, c, a, s);
}

/* What a launch sets up on its first use on a device, ahead of a stream capture. */
int ag_fast_ready(void) {
    int e = ag_ias_tables_init();
    if (!e) e = ag_fast_attr<2, false, false>();
    if (!e) e = ag_fast_attr<3, false, false>();
    if (!e) e = ag_fast_attr<2, true, false>();
    if (!e) e = ag_fast_attr<2, false, true>();
    return e;
}
