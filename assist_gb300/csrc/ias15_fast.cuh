/*
 * ias15_fast.cuh -- device pieces of IAS15 shared by the two integrators that
 * use the evaluation of fast_forces.cuh: the batched kernel (kernels_fast.cu)
 * and the shared-step kernel (kernels_shared.cu).  A block of eight warps holds
 * up to 32 particles, lane l of every warp working on particle l.  The
 * components x, y, z of the IAS15 state belong to warps 0, 2 and 3 (position
 * predictor, corrector, position update) with warps 5, 6 and 7 beside them
 * (velocity predictor and update, half of the b and g arithmetic); warp 1
 * controls the steps.
 */
#ifndef ASSIST_GB300_IAS15_FAST_CUH
#define ASSIST_GB300_IAS15_FAST_CUH

#include "fast_forces.cuh"
#include "ias15_common.cuh"

/* Component that warp w owns, or that it helps with (-1: none). */
__device__ __forceinline__ int ag_fast_comp(int w) { return w == 0 ? 0 : (w == 2 || w == 3 ? w - 1 : -1); }
__device__ __forceinline__ int ag_fast_help(int w) { return w >= 5 ? w - 5 : -1; }

/* Shared arrays of a block's steps. */
struct AgFastStep {
    AgFastShared F;
    double ra[3][32], rdb[3][32], rb6[3][32];   /* |a|, |delta b6|, |b6| of x, y, z at node 7 */
    double pcx[8][9], pcv[8][8], ptn[8];        /* predictor coefficients and times of the nodes */
    double hstep, t, tc;                        /* this step */
    double ah, aratio;                          /* the accepted (or rejected) step and the next one's size over it */
    unsigned live, fin, last;                   /* lanes integrating, to be retired, ending with this step */
    unsigned nf[3];                             /* lanes with a non-finite x, y, z */
    unsigned conv;                              /* lanes whose corrector has converged (or that do not integrate) */
    int cmd;
};

/* Predictor coefficients and times of the nodes of a step of size h from
 * t + tc, by lanes 1..7 of a warp (lane 0: the start). */
__device__ __forceinline__ void ag_fast_nodes(AgFastStep& S, int lane, double t, double tc, double h) {
    if (lane == 0) S.ptn[0] = t;
    if (lane < 1 || lane > 7) return;
    const double s0 = h * ag_ias.h[lane];
    /* the product rounded on its own, as the oracle forms a node time */
    S.ptn[lane] = t + (tc + __dmul_rn(h, ag_ias.h[lane]));
    double x = __dmul_rn(s0, s0) * 0.5, v = s0;
    S.pcx[lane][0] = s0; S.pcx[lane][1] = x; S.pcv[lane][0] = v;
#pragma unroll
    for (int k = 2; k < 9; k++) { x = x * ag_ias.fx[lane][k]; S.pcx[lane][k] = x; }
#pragma unroll
    for (int k = 1; k < 8; k++) { v = v * ag_ias.fv[lane][k]; S.pcv[lane][k] = v; }
}

/* The position (VEL: velocity) of component c at node n into the evaluation's arrays. */
template <bool VEL>
__device__ __forceinline__ void ag_fast_predict(const Ws<3>& W, AgFastStep& S, int c, int lane, int n) {
    double x = W(VEL ? W_V0 : W_X0, c);
    if (n != 0) {
        const double* s = VEL ? S.pcv[n] : S.pcx[n] + 1;
        double p = s[7] * W(W_B + 6, c);
#pragma unroll
        for (int j = 5; j >= 0; j--) p = fma(s[j + 1], W(W_B + j, c), p);
        p = fma(s[0], W(W_A0, c), p);
        if (!VEL) p = fma(S.pcx[n][0], W(W_V0, c), p);
        x += p + W(VEL ? W_VC : W_XC, c);
    }
    if (VEL) {
        S.F.vs[c][lane] = x;
        S.F.vf[c][lane] = ag_f2_of(x);
    } else {
        S.F.xs[c][lane] = x;
        S.F.xf[c][lane] = ag_f2_of(x);
    }
}
__device__ __forceinline__ void ag_fast_predict(const Ws<3>& W, AgFastStep& S, int pc, int hc, int lane, int n) {
    if (pc >= 0) ag_fast_predict<false>(W, S, pc, lane, n);
    if (hc >= 0) ag_fast_predict<true>(W, S, hc, lane, n);
}

/* Start of a step: g from the predicted b (g0, g1 by the owner, the others by
 * its helper: eleven and ten multiply-adds). */
template <int J0, int J1>
__device__ __forceinline__ void ag_fast_start(const Ws<3>& W, int c) {
    double b[7];
#pragma unroll
    for (int k = J0; k < 7; k++) b[k] = W(W_B + k, c);
#pragma unroll
    for (int j = J0; j < J1; j++) {
        double s = b[j];
#pragma unroll
        for (int k = j + 1; k < 7; k++) s = fma(b[k], ag_ias.d[j][k], s);
        W(W_G + j, c) = s;
    }
}
__device__ __forceinline__ void ag_fast_start(const Ws<3>& W, int pc, int hc) {
    if (pc >= 0) ag_fast_start<0, 2>(W, pc);
    if (hc >= 0) ag_fast_start<2, 7>(W, hc);
}

/* Corrector of component c at node n; node 7 leaves the error measures. */
__device__ __forceinline__ void ag_fast_correct(const Ws<3>& W, AgFastStep& S, int c, int lane, int n) {
    const double at = ag_fast_sum(S.F, c, lane);
    double gn = (at - W(W_A0, c)) * ag_ias.rrinv[n][0];
    for (int j = 1; j < n; j++) gn = (gn - W(W_G + j - 1, c)) * ag_ias.rrinv[n][j];
    const double delta = gn - W(W_G + n - 1, c);
    W(W_G + n - 1, c) = gn;
    for (int k = 0; k < n - 1; k++) W(W_B + k, c) = fma(delta, ag_ias.c[n - 1][k], W(W_B + k, c));
    const double bn = W(W_B + n - 1, c) + delta;
    W(W_B + n - 1, c) = bn;
    if (n == 7) {
        const double aa = fabs(at), db = fabs(delta), bb = fabs(bn);
        S.ra[c][lane] = ag_isnormal_pos(aa) ? aa : 0.0;
        S.rdb[c][lane] = ag_isnormal_pos(db) ? db : 0.0;
        S.rb6[c][lane] = ag_isnormal_pos(bb) ? bb : 0.0;
    }
}

/* The larger of a lane's three measures. */
__device__ __forceinline__ double ag_max3(const double (*r)[32], int lane) {
    return ag_max_nonneg(ag_max_nonneg(r[0][lane], r[1][lane]), r[2][lane]);
}

/* IAS15's convergence test on the error e = maxdb / maxa (non-negative): below
 * 1e-16, or no smaller than the last iteration's.  As products in FP64, one
 * rounding like the quotients' (a division is 600 cycles of the one warp that
 * judges, three products 200); the quotients where a product could leave the
 * range.  db, a: the last iteration's measures, updated. */
__device__ __forceinline__ bool ag_fast_converged(double maxdb, double maxa, int iters, double& db, double& a) {
    /* in 2^-300 .. 2^300 */
    auto mid = [](double x) { return ag_hi_word(x) - (723u << 20) < (600u << 20); };
    bool below, stalled = false;
    if (mid(maxa) && (iters == 1 || mid(a)) && ag_hi_word(maxdb) < (1323u << 20)) {
        below = __double_as_longlong(maxdb) < __double_as_longlong(1e-16 * maxa);
        if (iters > 2) stalled = __double_as_longlong(db * maxa) <= __double_as_longlong(maxdb * a);
    } else {
        const double e = maxdb / maxa;
        below = e < 1e-16;
        if (iters > 2) stalled = db / a <= e;
    }
    db = maxdb;
    a = maxa;
    return below || stalled || iters >= 12;
}

/* x^(-1/7): an FP32 estimate (1e-6) and two Newton steps
 * z <- z + z (1 - x z^7) / 7, each squaring the relative error (times 4):
 * full precision from 14 FP64 instructions, where pow takes about a hundred. */
__device__ __forceinline__ double ag_inv_root7(double x) {
    if (!(x > 1e-30 && x < 1e30)) return pow(x, -1.0 / 7.0);
    double z = ag_f2d_int(exp2f(log2f(ag_d2f_int(x)) * (-1.0f / 7.0f)));
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const double z2 = z * z, z4 = z2 * z2, z7 = z4 * z2 * z;
        z = fma(__dmul_rn(z, fma(-x, z7, 1.0)), 1.0 / 7.0, z);
    }
    return z;
}

/* b_j, e_j (J0 <= j < J1) of component c for a next step of ratio times the
 * last accepted one (the shift of the acceleration polynomial), from that
 * step's b (br) and e (er). */
template <int J0, int J1>
__device__ __forceinline__ void ag_fast_shift(const Ws<3>& W, int c, double ratio, const double* br, const double* er) {
    if (ratio > 20.0) {
#pragma unroll
        for (int k = J0; k < J1; k++) { W(W_E + k, c) = 0.0; W(W_B + k, c) = 0.0; }
        return;
    }
    constexpr double binom[8][8] = {
        {1, 0, 0, 0, 0, 0, 0, 0}, {1, 1, 0, 0, 0, 0, 0, 0}, {1, 2, 1, 0, 0, 0, 0, 0}, {1, 3, 3, 1, 0, 0, 0, 0},
        {1, 4, 6, 4, 1, 0, 0, 0}, {1, 5, 10, 10, 5, 1, 0, 0}, {1, 6, 15, 20, 15, 6, 1, 0}, {1, 7, 21, 35, 35, 21, 7, 1}};
    double q = 1.0;
#pragma unroll
    for (int j = 0; j < J0; j++) q *= ratio;
#pragma unroll
    for (int j = J0; j < J1; j++) {
        double s = 0.0;
#pragma unroll
        for (int k = 6; k >= j; k--) s = k == j ? s + br[k] : fma(br[k], binom[k + 1][j + 1], s);
        q *= ratio;
        /* rounded apart in every build */
        const double e = __dmul_rn(q, s), d = br[j] - er[j];
        W(W_E + j, c) = e;
        W(W_B + j, c) = __dadd_rn(e, d);
    }
}

/* A rejected step's retry: b and e from the last accepted step, zero when
 * there is none (ratio 0). */
template <int J0, int J1>
__device__ __forceinline__ void ag_fast_retry(const Ws<3>& W, int c, double ratio) {
    if (ratio == 0.0) {
#pragma unroll
        for (int k = J0; k < J1; k++) { W(W_B + k, c) = 0.0; W(W_E + k, c) = 0.0; }
        return;
    }
    double br[7], er[7];
#pragma unroll
    for (int k = J0; k < 7; k++) { br[k] = W(W_BR + k, c); er[k] = W(W_ER + k, c); }
    ag_fast_shift<J0, J1>(W, c, ratio, br, er);
}
__device__ __forceinline__ void ag_fast_retry(const Ws<3>& W, int pc, int hc, double ratio) {
    if (pc >= 0) ag_fast_retry<0, 2>(W, pc, ratio);
    if (hc >= 0) ag_fast_retry<2, 7>(W, hc, ratio);
}

/* Accepted step of size h, the whole block (live: this lane counts; one
 * barrier): x by the owner and v by its helper advanced by the step's
 * quadratures with compensated sums; b and e for the next step of ratio times
 * this one. */
__device__ __forceinline__ void ag_fast_accept(const Ws<3>& W, int pc, int hc, bool live, double h, double ratio) {
    const int c = pc >= 0 ? pc : hc;
    double b[7], e[7], a0 = 0.0, v0 = 0.0;
    if (live && c >= 0) {
#pragma unroll
        for (int k = 0; k < 7; k++) { b[k] = W(W_B + k, c); e[k] = W(W_E + k, c); }
        a0 = W(W_A0, c);
        v0 = W(W_V0, c);
    }
    __syncthreads();                /* the helper's b, e and v change the owner's inputs */
    if (!live || c < 0) return;
    if (pc >= 0) {
        double ix = b[6] * (1.0 / 72.0);
        ix = fma(b[5], 1.0 / 56.0, ix);
        ix = fma(b[4], 1.0 / 42.0, ix);
        ix = fma(b[3], 1.0 / 30.0, ix);
        ix = fma(b[2], 1.0 / 20.0, ix);
        ix = fma(b[1], 1.0 / 12.0, ix);
        ix = fma(b[0], 1.0 / 6.0, ix);
        ix = fma(a0, 0.5, ix);
        ix = fma(ix, __dmul_rn(h, h), __dmul_rn(v0, h));
        const double x0 = W(W_X0, c), y = ix + W(W_XC, c), s = x0 + y;
        W(W_XC, c) = y - (s - x0);
        W(W_X0, c) = s;
#pragma unroll
        for (int k = 0; k < 2; k++) { W(W_ER + k, c) = e[k]; W(W_BR + k, c) = b[k]; }
        ag_fast_shift<0, 2>(W, c, ratio, b, e);
    } else {
        double iv = b[6] * (1.0 / 8.0);
        iv = fma(b[5], 1.0 / 7.0, iv);
        iv = fma(b[4], 1.0 / 6.0, iv);
        iv = fma(b[3], 1.0 / 5.0, iv);
        iv = fma(b[2], 1.0 / 4.0, iv);
        iv = fma(b[1], 1.0 / 3.0, iv);
        iv = fma(b[0], 1.0 / 2.0, iv);
        iv = __dmul_rn(iv + a0, h);
        const double y = __dadd_rn(iv, W(W_VC, c)), s = v0 + y;
        W(W_VC, c) = y - (s - v0);
        W(W_V0, c) = s;
#pragma unroll
        for (int k = 2; k < 7; k++) { W(W_ER + k, c) = e[k]; W(W_BR + k, c) = b[k]; }
        ag_fast_shift<2, 7>(W, c, ratio, b, e);
    }
}

/* The smallest and the largest of the warp's non-negative doubles, whose bit
 * patterns order as integers do: the high words' extreme, then the low words'
 * among the lanes that have it. */
__device__ __forceinline__ double ag_warp_min_nonneg(double v) {
    const unsigned h = (unsigned)__double2hiint(v), l = (unsigned)__double2loint(v);
    const unsigned mh = __reduce_min_sync(AG_FULL, h), ml = __reduce_min_sync(AG_FULL, h == mh ? l : ~0u);
    return __hiloint2double((int)mh, (int)ml);
}
__device__ __forceinline__ double ag_warp_max_nonneg(double v) {
    const unsigned h = (unsigned)__double2hiint(v), l = (unsigned)__double2loint(v);
    const unsigned mh = __reduce_max_sync(AG_FULL, h), ml = __reduce_max_sync(AG_FULL, h == mh ? l : 0u);
    return __hiloint2double((int)mh, (int)ml);
}

#endif
