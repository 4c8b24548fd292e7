/*
 * kernels_var.cu -- the run kernel of shared-step simulations with six
 * first-order variational particles a particle, on the evaluation of
 * fast_forces.cuh: whole IAS15 steps on the device (kernels_shared.cu has the
 * one without variational particles).
 *
 * A block of eight warps holds up to L = 16 or 8 particles with their
 * variational ones.  An evaluation needs the particle's 3 x 6 Jacobian once
 * and IAS15's predictor and corrector for 21 components: with 32 particles a
 * block the components were 700 of 2,000 FP64 warp instructions a node, and 70
 * particles had three blocks.  Here the components are tasks over the block's
 * threads (full warps for any L), x, v, a, b, g in shared memory (56 KB for
 * L = 16, so that two blocks share an SM; e and the last accepted step's b, e,
 * used once a step, in global memory), and the warps' upper lanes, which have
 * no particle of their own, share the terms: a role's lanes are 32 / L copies
 * of the L particles, each with other packs (sub), summed by shuffles.
 *
 *   role 1               Sun (sub 0) and Jupiter (sub 1) with Jacobians, FP64;
 *                        GR terms; step control
 *   role 4               relativity with its Jacobian, FP64
 *   roles 0, 2, 3, 5..7  the pair terms' packs with Jacobians; 2 and 3 the
 *                        harmonics in FP32
 *
 * What bounds it is the latency of a node (role 4's FP64 Jacobian and the
 * components' two tasks a thread); 70 near-Earth particles over 60 days, 9
 * blocks: 22.0 ms with a launch a step and 32 particles a block in FP64, 6.5
 * here.  The step rules are those of kernels_shared.cu's run kernel
 * (variational particles never enter the error measures).
 */
#include <cuda_runtime.h>

#include "device_forces.cuh"
#include "ias15_fast.cuh"
#include "internal.h"
#include "shared_run.cuh"

enum { V_X0 = 0, V_V0, V_A0, V_XC, V_VC, V_B, V_G = V_B + 7, V_PX = V_G + 7, V_PV, V_NF };
#define AG_VAR_SLOTS 6

template <int L>
struct AgVarSmem {
    AgFastStep S;
    double J[18][L], Je[18][L];                     /* FP64 parts of the Jacobian (roles 1 and 4); J then the whole */
    AgF2 pj[AG_VAR_SLOTS][7][L];                    /* pair parts: symmetric part and trace sum */
    AgF2 pf[AG_VAR_SLOTS + 1][3][L];                /* pair accelerations; the last: relativity */
    double pa[3][L], acc[3][L];                     /* role 1's acceleration without the Sun's; the sum */
    double ss[3][L], gs[L];                         /* separation from the Sun and -GM / r^3 there */
    unsigned long long close[L];                    /* pair bodies left to FP64; bit 62 Earth's, 63 the Sun's harmonics */
    int any;
    int pidx[7][L];                                 /* particle of each (variational, lane) */
};

template <int L>
__host__ __device__ constexpr size_t ag_var_state_bytes() { return sizeof(double) * V_NF * 21 * L; }
template <int L>
__host__ __device__ inline size_t ag_var_bytes(int n_ast) {
    return ag_var_state_bytes<L>() + 8 * (size_t)AgFastLayout(n_ast).stride;
}

/* Pair slot of role w (0, 2, 3, 5, 6, 7), or -1. */
__device__ __forceinline__ int ag_var_slot(int w) { return w == 0 ? 0 : (w == 2 || w == 3 ? w - 1 : (w >= 5 ? w - 2 : -1)); }

/* FP64 terms of what the pairs leave out at the lane's particle: added to a, J. */
static __device__ __noinline__ void ag_var_close(const DevEphem& E, const ForceCfg& c, const double* rel, const AgFastNode* H,
                                                 unsigned long long m, const double* x, double* a, double (*J)[6]) {
    double ax = 0.0, ay = 0.0, az = 0.0;
    AgSymJac Y = {{0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, 0.0};
    const bool earth = (m >> 62) & 1, sun = (m >> 63) & 1;
    m &= ~(3ull << 62);
    while (m) {
        const int k = __ffsll((long long)m) - 1;
        m &= m - 1;
        const double gm = k < AG_PAIR_PL ? E.gm[ag_pair_planet(k)] : E.ast_gm[k - AG_PAIR_PL];
        const double dx = x[0] + rel[3 * k], dy = x[1] + rel[3 * k + 1], dz = x[2] + rel[3 * k + 2];
        const double ri = rsqrt(fma(dx, dx, fma(dy, dy, dz * dz))), g = gm * ri * ri * ri;
        ax = fma(-g, dx, ax); ay = fma(-g, dy, ay); az = fma(-g, dz, az);
        ag_symjac_term(Y, g, ri, dx, dy, dz);
    }
    ag_symjac_add(Y, J);
    if (earth) {
        const double dx = x[0] + rel[6], dy = x[1] + rel[7], dz = x[2] + rel[8];
        ag_term_earth_h<true>(E, c, dx, dy, dz, rsqrt(fma(dx, dx, fma(dy, dy, dz * dz))), ax, ay, az, J);
    }
    if (sun) {
        const double dx = x[0] + H->rs[0], dy = x[1] + H->rs[1], dz = x[2] + H->rs[2];
        ag_term_sun_h<true>(E, c, dx, dy, dz, rsqrt(fma(dx, dx, fma(dy, dy, dz * dz))), ax, ay, az, J);
    }
    a[0] += ax; a[1] += ay; a[2] += az;
}

/* The planets' pull on the Sun and their potential there in FP64 (a particle
 * beyond 200 AU, where they are no small part of the relativistic term). */
static __device__ __noinline__ void ag_var_sun_pull(const DevEphem& E, const double* rel, const AgFastNode* H, double* af, double* ut) {
    double s[3] = {0.0, 0.0, 0.0}, u = 0.0;
    for (int k = -1; k < AG_PAIR_PL; k++) {
        const double* o = k < 0 ? H->rj : rel + 3 * k;
        const double px = o[0] - H->rs[0], py = o[1] - H->rs[1], pz = o[2] - H->rs[2];
        const double ri = rsqrt(fma(px, px, fma(py, py, pz * pz)));
        const double gr = E.gm[k < 0 ? AG_JUP : ag_pair_planet(k)] * ri, f = gr * ri * ri;
        u += gr;
        s[0] = fma(-f, px, s[0]); s[1] = fma(-f, py, s[1]); s[2] = fma(-f, pz, s[2]);
    }
    af[0] = s[0]; af[1] = s[1]; af[2] = s[2];
    *ut = u;
}

/* Role w's share of the evaluation with Jacobian at table n; on: this lane's
 * particle counts.  The caller synchronises before and after. */
template <int L>
__device__ __forceinline__ void ag_var_force(int w, int lane, bool on, const DevEphem& E, const ForceCfg& c, const AgFastView& V,
                                             int n, AgVarSmem<L>& M) {
    constexpr int SUBS = 32 / L;
    AgFastShared& F = M.S.F;
    const AgFastNode& H = V.node(n);
    const int l = lane & (L - 1), sub = lane / L;
    if (w == 1) {
        const double x[3] = {F.xs[0][l], F.xs[1][l], F.xs[2][l]};
        const double* o = sub == 1 ? H.rj : H.rs;
        const double s[3] = {x[0] + o[0], x[1] + o[1], x[2] + o[2]};
        const double ri = rsqrt(fma(s[0], s[0], fma(s[1], s[1], s[2] * s[2])));
        double a[3] = {0.0, 0.0, 0.0}, J[3][6];
#pragma unroll
        for (int q = 0; q < 18; q++) J[q / 6][q % 6] = 0.0;
        if (on && sub == 0 && (c.forces & (AG_F_GR_POT | AG_F_GR_SIMPLE))) {
            const double dv[3] = {F.vs[0][l] - H.sv[0], F.vs[1][l] - H.sv[1], F.vs[2][l] - H.sv[2]};
            if (c.forces & AG_F_GR_POT) ag_term_gr_pot<true>(E, s, ri, a[0], a[1], a[2], J);
            if (c.forces & AG_F_GR_SIMPLE) ag_term_gr_simple<true>(E, s, ri, dv, a[0], a[1], a[2], J);
        }
        AgSymJac Y = {{0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, 0.0};
        const double g = (sub == 1 ? E.gm[AG_JUP] : E.gm[AG_SUN]) * ri * ri * ri;
        if (sub == 0) {
            /* the Sun's term goes into the last sum unrounded */
            M.gs[l] = -g;
            M.ss[0][l] = s[0]; M.ss[1][l] = s[1]; M.ss[2][l] = s[2];
        } else {
            a[0] = -g * s[0]; a[1] = -g * s[1]; a[2] = -g * s[2];
        }
        ag_symjac_term(Y, g, ri, s[0], s[1], s[2]);
        /* Jupiter's to the Sun's lanes */
#pragma unroll
        for (int k = 0; k < 3; k++) a[k] += __shfl_down_sync(AG_FULL, a[k], L);
#pragma unroll
        for (int k = 0; k < 6; k++) Y.s[k] += __shfl_down_sync(AG_FULL, Y.s[k], L);
        Y.g += __shfl_down_sync(AG_FULL, Y.g, L);
        if (sub == 0) {
            ag_symjac_add(Y, J);
#pragma unroll
            for (int q = 0; q < 18; q++) M.J[q][l] = J[q / 6][q % 6];
            M.pa[0][l] = a[0]; M.pa[1][l] = a[1]; M.pa[2][l] = a[2];
        }
        return;
    }
    const AgF2 xf[3] = {F.xf[0][l], F.xf[1][l], F.xf[2][l]};
    const AgPkRel* R = V.packs(n);
    const float big = fmaxf(fabsf(xf[0].h), fmaxf(fabsf(xf[1].h), fabsf(xf[2].h)));
    if (w == 4) {
        /* the planets' potential and pull at the particle: a share of them on
         * each copy of the lane */
        float up = 0.0f, gp[3] = {0.0f, 0.0f, 0.0f};
        for (int k = sub; k < AG_PAIR_PL + 1; k += SUBS) {
            float q[3], gm;
            if (k < AG_PAIR_PL) {
                const float* pk = reinterpret_cast<const float*>(R[k >> 1].c) + (k & 1);
                gm = (k & 1) ? F.gm[k >> 1].gb : F.gm[k >> 1].ga;
                for (int m = 0; m < 3; m++) q[m] = pk[4 * m] + xf[m].h;
            } else {
                gm = E.pv.gm_jup;
                for (int m = 0; m < 3; m++) q[m] = H.jf[m] + xf[m].h;
            }
            const float ri = rsqrtf(fmaf(q[0], q[0], fmaf(q[1], q[1], q[2] * q[2]))), f = gm * ri * ri * ri;
            up = fmaf(gm, ri, up);
            for (int m = 0; m < 3; m++) gp[m] = fmaf(f, q[m], gp[m]);
        }
#pragma unroll
        for (int o = L; o < 32; o <<= 1) {
            up += __shfl_xor_sync(AG_FULL, up, o);
            for (int m = 0; m < 3; m++) gp[m] += __shfl_xor_sync(AG_FULL, gp[m], o);
        }
        double a[3] = {0.0, 0.0, 0.0}, J[3][6];
#pragma unroll
        for (int q = 0; q < 18; q++) J[q / 6][q % 6] = 0.0;
        if (sub == 0 && (c.forces & AG_F_EIH)) {
            const double v[3] = {F.vs[0][l], F.vs[1][l], F.vs[2][l]};
            const double d[3] = {F.xs[0][l] + H.rs[0], F.xs[1][l] + H.rs[1], F.xs[2][l] + H.rs[2]};
            double aj[3] = {ag_f2d_int(H.af[0]), ag_f2d_int(H.af[1]), ag_f2d_int(H.af[2])}, ut = ag_f2d_int(H.ut);
            if (!(big < 200.0f)) ag_var_sun_pull(E, V.rel(n), &H, aj, &ut);
            const double g[3] = {ag_f2d_int(gp[0]), ag_f2d_int(gp[1]), ag_f2d_int(gp[2])};
            ag_fast_eih_jac(E, d, rsqrt(fma(d[0], d[0], fma(d[1], d[1], d[2] * d[2]))), v, H.sv, aj, ut, ag_f2d_int(up), g, a, J);
        }
        if (sub == 0) {
#pragma unroll
            for (int q = 0; q < 18; q++) M.Je[q][l] = J[q / 6][q % 6];
#pragma unroll
            for (int k = 0; k < 3; k++) M.pf[AG_VAR_SLOTS][k][l] = ag_f2_of(a[k]);
        }
        return;
    }
    const int slot = ag_var_slot(w);
    const float sx = xf[0].h + H.sp[0].h, sy = xf[1].h + H.sp[1].h, sz = xf[2].h + H.sp[2].h;
    const float rs2 = fmaf(sx, sx, fmaf(sy, sy, sz * sz));
    const bool wild = !(big < 1e6f);
    AgPkSum P;
    AgPkJac PJ;
    AgPk xh[3], xl[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        xh[k] = ag_pk(xf[k].h, xf[k].h);
        xl[k] = ag_pk(xf[k].l, xf[k].l);
        P.h[k] = P.l[k] = ag_pk(0.0f, 0.0f);
    }
    ag_pk_jac_clear(PJ);
    unsigned long long near = 0;
    /* packs dealt to (copy, role), the roles without harmonics first */
    const int order = w >= 5 ? w - 5 : (w == 0 ? 3 : w + 2);
#pragma unroll 1
    for (int p = order + AG_VAR_SLOTS * sub; p < V.L.packs; p += AG_VAR_SLOTS * SUBS)
        near |= (unsigned long long)ag_pk_term<true>(R[p], F.gm[p], xh, xl, rs2, P, &PJ) << (2 * p);
    AgF2 s[3], j[7];
#pragma unroll
    for (int k = 0; k < 3; k++)
        s[k] = ag_f2_add({ag_pk_a(P.h[k]), ag_pk_a(P.l[k])}, {ag_pk_b(P.h[k]), ag_pk_b(P.l[k])});
#pragma unroll
    for (int k = 0; k < 7; k++) {
        AgF2 a, b;
        ag_pk_jac_get(PJ, k, 0, a.h, a.l);
        ag_pk_jac_get(PJ, k, 1, b.h, b.l);
        j[k] = ag_f2_add(a, b);
    }
    if (sub == 0 && w == 3 && (c.forces & AG_F_EARTH_H)) {
        /* the Jacobian's share is larger than the term's by r / d: FP64 within 0.1 AU */
        float q[3], hj[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int k = 0; k < 3; k++) q[k] = ag_f2_sep(xf[k], ag_pk_a(R[1].c[k].h), ag_pk_a(R[1].c[k].l));
        const float r2 = fmaf(q[0], q[0], fmaf(q[1], q[1], q[2] * q[2]));
        if (!(r2 >= 1.0e-2f && r2 < 1e30f)) near |= 1ull << 62;
        else {
            ag_fast_earth_h(E.pv, c, q, r2, s);
            ag_fast_earth_hj(E.pv, c, q, r2, hj);
#pragma unroll
            for (int k = 0; k < 6; k++) j[k].l += hj[k];
        }
    }
    if (sub == 0 && w == 2 && (c.forces & AG_F_SUN_H)) {
        float hj[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        if (!(rs2 >= 1.0e-2f && rs2 < 1e30f)) near |= 1ull << 63;
        else if (rs2 < AG_SUN_H_FAR2) {
            const AgF2 d[3] = {ag_q_add(xf[0], H.sp[0]), ag_q_add(xf[1], H.sp[1]), ag_q_add(xf[2], H.sp[2])};
            ag_fast_sun_near<true>(E.pv, c, d, s, j);
        } else {
            const float q[3] = {sx, sy, sz};
            ag_fast_sun_h(E.pv, c, sx, sy, sz, rs2, s);
            ag_fast_sun_hj(E.pv, c, q, rs2, hj);
#pragma unroll
            for (int k = 0; k < 6; k++) j[k].l += hj[k];
        }
    }
    if (wild) {
        near |= (1ull << V.L.bodies) - 1;
#pragma unroll
        for (int k = 0; k < 3; k++) s[k] = {0.0f, 0.0f};
#pragma unroll
        for (int k = 0; k < 7; k++) j[k] = {0.0f, 0.0f};
    }
    near &= 3ull << 62 | ((1ull << V.L.bodies) - 1);     /* not the last pack's empty half (a NaN state) */
    if (on && near) {
        atomicOr(&M.close[l], near);
        M.any = 1;
    }
#pragma unroll
    for (int o = L; o < 32; o <<= 1) {
#pragma unroll
        for (int k = 0; k < 3; k++)
            s[k] = ag_f2_add(s[k], {__shfl_xor_sync(AG_FULL, s[k].h, o), __shfl_xor_sync(AG_FULL, s[k].l, o)});
#pragma unroll
        for (int k = 0; k < 7; k++)
            j[k] = ag_f2_add(j[k], {__shfl_xor_sync(AG_FULL, j[k].h, o), __shfl_xor_sync(AG_FULL, j[k].l, o)});
    }
    if (sub == 0) {
#pragma unroll
        for (int k = 0; k < 3; k++) M.pf[slot][k][l] = s[k];
#pragma unroll
        for (int k = 0; k < 7; k++) M.pj[slot][k][l] = j[k];
    }
}

/* After the roles have met: the whole Jacobian in M.J and the acceleration in
 * M.acc (element by element over the threads).  Ends with a block barrier. */
template <int L>
__device__ __forceinline__ void ag_var_assemble(const DevEphem& E, const ForceCfg& c, const AgFastView& V, int n, AgVarSmem<L>& M,
                                                int tid, int wid, int lane) {
    if (M.any) {
        if (wid == 1 && lane < L && M.close[lane]) {
            const AgFastShared& F = M.S.F;
            const double x[3] = {F.xs[0][lane], F.xs[1][lane], F.xs[2][lane]};
            double a[3] = {M.pa[0][lane], M.pa[1][lane], M.pa[2][lane]}, J[3][6];
            for (int q = 0; q < 18; q++) J[q / 6][q % 6] = 0.0;
            ag_var_close(E, c, V.rel(n), &V.node(n), M.close[lane], x, a, J);
            M.pa[0][lane] = a[0]; M.pa[1][lane] = a[1]; M.pa[2][lane] = a[2];
            for (int q = 0; q < 18; q++) M.J[q][lane] += J[q / 6][q % 6];
            M.close[lane] = 0ull;
        }
        __syncthreads();
        if (tid == 0) M.any = 0;
    }
    for (int t = tid; t < 21 * L; t += AG_FAST_THREADS) {
        const int q = t / L, l = t - q * L;
        if (q < 18) {
            const int a = q / 6, b = q - 6 * a;
            double s = M.Je[q][l];
            if (b < 3) {
                const int lo = a < b ? a : b, hi = a < b ? b : a, e = lo == 0 ? hi : lo + hi + 1;
                AgF2 p = M.pj[0][e][l];
#pragma unroll
                for (int k = 1; k < AG_VAR_SLOTS; k++) p = ag_f2_add(p, M.pj[k][e][l]);
                if (a == b) {
                    AgF2 g = M.pj[0][6][l];
#pragma unroll
                    for (int k = 1; k < AG_VAR_SLOTS; k++) g = ag_f2_add(g, M.pj[k][6][l]);
                    p = ag_f2_add(p, ag_f2_neg(g));
                }
                s += ag_f2_to(p);
            }
            M.J[q][l] += s;
        } else {
            const int k = q - 18;
            AgF2 p = M.pf[0][k][l];
#pragma unroll
            for (int m = 1; m <= AG_VAR_SLOTS; m++) p = ag_f2_add(p, M.pf[m][k][l]);
            M.acc[k][l] = fma(M.gs[l], M.ss[k][l], ag_f2_to(p) + M.pa[k][l]);
        }
    }
    __syncthreads();
}

/* A task's acceleration: component c of lane l (a variational one: the
 * Jacobian's row times its predicted state). */
template <int L>
__device__ __forceinline__ double ag_var_acc(const AgVarSmem<L>& M, const double* w, int c, int l) {
    if (c < 3) return M.acc[c][l];
    constexpr int T = 21 * L;
    const int q = 3 * (c / 3), a = c - q;
    const double *x = w + V_PX * T + q * L + l, *v = w + V_PV * T + q * L + l;
    double s = M.J[6 * a][l] * x[0];
    s = fma(M.J[6 * a + 1][l], x[L], s); s = fma(M.J[6 * a + 2][l], x[2 * L], s);
    s = fma(M.J[6 * a + 3][l], v[0], s); s = fma(M.J[6 * a + 4][l], v[L], s); s = fma(M.J[6 * a + 5][l], v[2 * L], s);
    return s;
}

/* L: particles a block. */
template <int L>
__global__ void __launch_bounds__(AG_FAST_THREADS, 2) ag_k_var_run(const DevEphem* __restrict__ Ep, ForceCfg cf, ShRunArgs R,
                                                                   const int* __restrict__ vmap) {
    constexpr int T = 21 * L;
    extern __shared__ __align__(16) unsigned char ag_var_dyn[];
    __shared__ AgVarSmem<L> M;
    AgFastStep& S = M.S;
    const DevEphem& E = *Ep;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, ll = lane & (L - 1);
    const bool ctl = wid == 1;
    double* const w = reinterpret_cast<double*>(ag_var_dyn);
    const AgFastView V(ag_var_dyn + ag_var_state_bytes<L>(), E.n_ast);
    /* fields S_E, S_BR, S_ER + k of task t */
    auto G = [&](int f, int t) -> double& {
        const int c = t / L, l = t - c * L, v = c / 3;
        return R.W(f, c - 3 * v, M.pidx[v][l]);
    };
    if (tid == 0) M.any = 0;
    if (tid < L) M.close[tid] = 0ull;
    ag_fast_masses<true>(E, cf, S.F, tid);
    ShCtl K = *R.in;
    const int gs = min(L, R.n - L * (int)blockIdx.x);
    for (int q = tid; q < 7 * L; q += AG_FAST_THREADS) {
        const int v = q / L, l = q - v * L, i = L * blockIdx.x + l;
        M.pidx[v][l] = l < gs ? (v == 0 ? i : vmap[6 * i + v - 1]) : 0;
    }
    const bool on = ll < gs;
    __syncthreads();
    /* state in */
    for (int t = tid; t < T; t += AG_FAST_THREADS) {
        const int c = t / L, l = t - c * L, v = c / 3, k = c - 3 * v;
        if (l >= gs) continue;
        const int p = M.pidx[v][l];
        w[V_X0 * T + t] = R.W(S_X0, k, p); w[V_V0 * T + t] = R.W(S_V0, k, p);
        w[V_XC * T + t] = R.W(S_XC, k, p); w[V_VC * T + t] = R.W(S_VC, k, p);
        for (int f = 0; f < 7; f++) w[(V_B + f) * T + t] = R.W(S_B + f, k, p);
    }
    /* states at node n of the step */
    auto predict = [&](int n) {
        const double *sx = S.pcx[n], *sv = S.pcv[n];
        for (int q = tid; q < T; q += AG_FAST_THREADS) {
            const int c = q / L, l = q - c * L;
            if (l >= gs) continue;
            double x = w[V_X0 * T + q], v = w[V_V0 * T + q];
            if (n != 0) {
                const double a0 = w[V_A0 * T + q], v0 = v;
                double b = w[(V_B + 6) * T + q];
                double px = sx[8] * b, pv = sv[7] * b;
#pragma unroll
                for (int f = 5; f >= 0; f--) {
                    b = w[(V_B + f) * T + q];
                    px = fma(sx[f + 2], b, px);
                    pv = fma(sv[f + 1], b, pv);
                }
                px = fma(sx[1], a0, px);
                px = fma(sx[0], v0, px);
                x += px + w[V_XC * T + q];
                pv = fma(sv[0], a0, pv);
                v += pv + w[V_VC * T + q];
            }
            if (c < 3) {
                S.F.xs[c][l] = x; S.F.vs[c][l] = v;
                S.F.xf[c][l] = ag_f2_of(x);
            } else {
                w[V_PX * T + q] = x; w[V_PV * T + q] = v;
            }
        }
    };
    int round = 0, run_steps = 0;
    double hstep = 0.0;
    bool last = false, gave_up = false;
    while (true) {
        if (ctl) {
            const double rem = (R.tmax - K.t) - K.tc;
            last = fabs(K.dt) >= fabs(rem);
            hstep = last ? rem : K.dt;
            ag_fast_nodes(S, lane, K.t, K.tc, hstep);
        }
        __syncthreads();
        /* ---- the step's tables and node 0 */
        predict(0);
        if (ag_fast_tables(E, cf, 8, S.ptn, V, S.F, tid)) {
            K.status = AG_ERR_COVERAGE;
            break;
        }
        ag_var_force<L>(wid, lane, on, E, cf, V, 0, M);
        __syncthreads();
        ag_var_assemble<L>(E, cf, V, 0, M, tid, wid, lane);
        for (int q = tid; q < T; q += AG_FAST_THREADS) {
            const int c = q / L, l = q - c * L;
            if (l >= gs) continue;
            w[V_A0 * T + q] = ag_var_acc<L>(M, w, c, l);
            double b[7];
#pragma unroll
            for (int k = 0; k < 7; k++) b[k] = w[(V_B + k) * T + q];
#pragma unroll
            for (int j = 0; j < 7; j++) {
                double s = b[j];
#pragma unroll
                for (int k = j + 1; k < 7; k++) s = fma(b[k], ag_ias.d[j][k], s);
                w[(V_G + j) * T + q] = s;
            }
        }
        __syncthreads();         /* the variational states at node 0 have been read */
        /* ---- predictor-corrector iterations */
        int iters = 1, cmd;
        ShMeasure before = {0.0, 0.0};
        while (true) {
            for (int n = 1; n < 8; n++) {
                predict(n);
                __syncthreads();
                ag_var_force<L>(wid, lane, on, E, cf, V, n, M);
                __syncthreads();
                ag_var_assemble<L>(E, cf, V, n, M, tid, wid, lane);
                for (int q = tid; q < T; q += AG_FAST_THREADS) {
                    const int c = q / L, l = q - c * L;
                    if (l >= gs) continue;
                    const double at = ag_var_acc<L>(M, w, c, l);
                    double gn = (at - w[V_A0 * T + q]) * ag_ias.rrinv[n][0];
                    for (int j = 1; j < n; j++) gn = (gn - w[(V_G + j - 1) * T + q]) * ag_ias.rrinv[n][j];
                    const double delta = gn - w[(V_G + n - 1) * T + q];
                    w[(V_G + n - 1) * T + q] = gn;
                    for (int k = 0; k < n - 1; k++) w[(V_B + k) * T + q] = fma(delta, ag_ias.c[n - 1][k], w[(V_B + k) * T + q]);
                    const double bn = w[(V_B + n - 1) * T + q] + delta;
                    w[(V_B + n - 1) * T + q] = bn;
                    if (n == 7 && c < 3) {
                        const double aa = fabs(at), db = fabs(delta), bb = fabs(bn);
                        S.ra[c][l] = ag_isnormal_pos(aa) ? aa : 0.0;
                        S.rdb[c][l] = ag_isnormal_pos(db) ? db : 0.0;
                        S.rb6[c][l] = ag_isnormal_pos(bb) ? bb : 0.0;
                    }
                }
                __syncthreads();
            }
            if (ctl) {
                double ma = ag_warp_max_nonneg(lane < gs ? ag_max3(S.ra, lane) : 0.0);
                double mdb = ag_warp_max_nonneg(lane < gs ? ag_max3(S.rdb, lane) : 0.0);
                double mb = ag_warp_max_nonneg(lane < gs ? ag_max3(S.rb6, lane) : 0.0);
                bool ok = true;
                if (gridDim.x > 1) {
                    ok = sh_run_maxima(R, round, lane, mdb, ma, mb);
                    round++;
                }
                gave_up = !ok;
                sh_run_decide(R, K, S, ok, mdb, ma, mb, hstep, last, iters, before, lane);
            }
            __syncthreads();
            cmd = S.cmd;
            if (cmd != SH_ITERATE) break;
            iters++;
        }
        const bool leave = S.fin != 0;
        const double h = S.ah, ratio = S.aratio;
        __syncthreads();             /* read before the control warp writes the next step's */
        if (cmd == SH_ACCEPT || cmd == SH_REJECT) {
            for (int q = tid; q < T; q += AG_FAST_THREADS) {
                const int c = q / L, l = q - c * L;
                if (l >= gs) continue;
                double b[7], e[7];
                if (cmd == SH_ACCEPT) {
#pragma unroll
                    for (int k = 0; k < 7; k++) { b[k] = w[(V_B + k) * T + q]; e[k] = G(S_E + k, q); }
                    const double a0 = w[V_A0 * T + q], x0 = w[V_X0 * T + q], v0 = w[V_V0 * T + q];
                    const int v = c / 3, k = c - 3 * v, p = M.pidx[v][l];
                    R.W(S_PX, k, p) = x0 + w[V_XC * T + q];
                    R.W(S_PV, k, p) = v0 + w[V_VC * T + q];
                    R.W(S_PA, k, p) = a0;
                    double ix = b[6] * (1.0 / 72.0), iv = b[6] * (1.0 / 8.0);
                    ix = fma(b[5], 1.0 / 56.0, ix); iv = fma(b[5], 1.0 / 7.0, iv);
                    ix = fma(b[4], 1.0 / 42.0, ix); iv = fma(b[4], 1.0 / 6.0, iv);
                    ix = fma(b[3], 1.0 / 30.0, ix); iv = fma(b[3], 1.0 / 5.0, iv);
                    ix = fma(b[2], 1.0 / 20.0, ix); iv = fma(b[2], 1.0 / 4.0, iv);
                    ix = fma(b[1], 1.0 / 12.0, ix); iv = fma(b[1], 1.0 / 3.0, iv);
                    ix = fma(b[0], 1.0 / 6.0, ix);  iv = fma(b[0], 1.0 / 2.0, iv);
                    ix = fma(a0, 0.5, ix);
                    iv = __dmul_rn(iv + a0, h);
                    ix = fma(ix, __dmul_rn(h, h), __dmul_rn(v0, h));
                    double y = ix + w[V_XC * T + q], s = x0 + y;
                    w[V_XC * T + q] = y - (s - x0);
                    w[V_X0 * T + q] = s;
                    y = __dadd_rn(iv, w[V_VC * T + q]);
                    s = v0 + y;
                    w[V_VC * T + q] = y - (s - v0);
                    w[V_V0 * T + q] = s;
#pragma unroll
                    for (int k = 0; k < 7; k++) { G(S_BR + k, q) = b[k]; G(S_ER + k, q) = e[k]; }
                } else {
#pragma unroll
                    for (int k = 0; k < 7; k++) { b[k] = G(S_BR + k, q); e[k] = G(S_ER + k, q); }
                }
                if (ratio == 0.0 || ratio > 20.0) {
                    for (int k = 0; k < 7; k++) { w[(V_B + k) * T + q] = 0.0; G(S_E + k, q) = 0.0; }
                } else {
                    constexpr double binom[8][8] = {
                        {1, 0, 0, 0, 0, 0, 0, 0}, {1, 1, 0, 0, 0, 0, 0, 0}, {1, 2, 1, 0, 0, 0, 0, 0}, {1, 3, 3, 1, 0, 0, 0, 0},
                        {1, 4, 6, 4, 1, 0, 0, 0}, {1, 5, 10, 10, 5, 1, 0, 0}, {1, 6, 15, 20, 15, 6, 1, 0}, {1, 7, 21, 35, 35, 21, 7, 1}};
                    double r = 1.0;
#pragma unroll
                    for (int j = 0; j < 7; j++) {
                        double s = 0.0;
#pragma unroll
                        for (int k = 6; k >= j; k--) s = k == j ? s + b[k] : fma(b[k], binom[k + 1][j + 1], s);
                        r *= ratio;
                        const double en = __dmul_rn(r, s), d = b[j] - e[j];
                        G(S_E + j, q) = en;
                        w[(V_B + j) * T + q] = __dadd_rn(en, d);
                    }
                }
            }
        }
        if (leave || ++run_steps >= R.limit) break;
    }
    __syncthreads();
    /* state out */
    for (int q = tid; q < T; q += AG_FAST_THREADS) {
        const int c = q / L, l = q - c * L, v = c / 3, k = c - 3 * v;
        if (l >= gs) continue;
        const int p = M.pidx[v][l];
        R.W(S_X0, k, p) = w[V_X0 * T + q]; R.W(S_V0, k, p) = w[V_V0 * T + q];
        R.W(S_XC, k, p) = w[V_XC * T + q]; R.W(S_VC, k, p) = w[V_VC * T + q];
        for (int f = 0; f < 7; f++) R.W(S_B + f, k, p) = w[(V_B + f) * T + q];
    }
    if (ctl && lane == 0) sh_run_report(K, gave_up, blockIdx.x, R.out, R.gave_up);
}

template <int L>
static int ag_var_attr() {
    return (int)cudaFuncSetAttribute(ag_k_var_run<L>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)ag_var_bytes<L>(AG_MAX_AST));
}

template <int L>
static int ag_var_fit(int n_ast) {
    int dev = 0, sms = 0, bps = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (ag_var_attr<L>() ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, ag_k_var_run<L>, AG_FAST_THREADS, ag_var_bytes<L>(n_ast)) !=
            cudaSuccess)
        return 0;
    return bps * sms;
}

/* Particles a block for a simulation of n with six variational particles
 * each, or 0 when its blocks do not fit on the device at once (coop: blocks
 * may meet in a cooperative launch). */
int ag_var_run_lanes(int n, int n_ast, bool coop) {
    for (int lanes = 8; lanes <= 16; lanes += 8) {
        const int blocks = (n + lanes - 1) / lanes;
        const int fit = lanes == 16 ? ag_var_fit<16>(n_ast) : ag_var_fit<8>(n_ast);
        if (blocks <= (coop ? fit : 1)) return lanes;
    }
    return 0;
}

cudaError_t ag_launch_var_run(const DevEphem& E, const ForceCfg& c, const ShRunArgs& r, const int* vmap, int lanes, cudaStream_t s) {
    int e = ag_ias_tables_init();
    if (e) return (cudaError_t)e;
    const int blocks = (r.n + lanes - 1) / lanes;
    const DevEphem* ep = E.self_dev;
    ForceCfg cc = c;
    ShRunArgs rr = r;
    void* args[] = {(void*)&ep, (void*)&cc, (void*)&rr, (void*)&vmap};
    const void* f = lanes == 16 ? (const void*)ag_k_var_run<16> : (const void*)ag_k_var_run<8>;
    const size_t bytes = lanes == 16 ? ag_var_bytes<16>(E.n_ast) : ag_var_bytes<8>(E.n_ast);
    if (blocks > 1) return cudaLaunchCooperativeKernel(f, blocks, AG_FAST_THREADS, args, bytes, s);
    return cudaLaunchKernel(f, dim3(1), dim3(AG_FAST_THREADS), args, bytes, s);
}
