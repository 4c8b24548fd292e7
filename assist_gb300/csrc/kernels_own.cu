/*
 * kernels_own.cu -- K2f: the accelerations of n particles, each at its own
 * time (assist_gb300_forces_device), for .440 planets and the force
 * configurations of fast_forces.cuh.
 *
 * A block of four warps takes 32 particles, lane l of each warp particle l.
 * Every particle has a body table of its own, so the ephemeris is most of the
 * work: 3,180 FP64 instructions a warp when one thread did it all.  Here the
 * bodies of the pair terms are evaluated as float pairs from a float-pair
 * image of the files (43 FP32 instructions a coefficient and its three
 * components; the sums' error of a few 2^-48 is of the size the terms'
 * thresholds allow for, and those are doubled here), Jupiter in the
 * reference's exact operations, the Sun in FP64 with fused multiply-adds (its
 * distance from the particles makes an ulp of its 0.01 AU 1e-18), and a body
 * close to the particle again in the exact operations.  About 300 FP64
 * instructions a block without variational particles.  33 particles 125 -> 27
 * to 29 us, 100,003 674 -> 231 to 239 us, 20,011 with six variational particles
 * each 312 -> 123 to 132 us (by the population drawn).
 *
 *   before the barrier   role 1: the Sun; role 0: Jupiter, Earth and Moon,
 *                        an eighth of the asteroids; role 2: the other
 *                        planets, a quarter; role 3: the rest
 *   after it             role 1: Sun, Jupiter, FP64 terms; roles 0, 2: pair terms;
 *                        role 3: the rest of them, relativity, harmonics
 */
#include <cuda_runtime.h>

#include "fast_forces.cuh"
#include "internal.h"

__global__ void ag_k_pair_image(const double* __restrict__ x, float2* __restrict__ out, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const double v = x[i];
        const float h = (float)v;
        out[i] = make_float2(h, (float)(v - (double)h));
    }
}

/* out[i] = x[i] as a float pair (hi, lo). */
int ag_launch_pair_image(const double* x, float2* out, size_t n, cudaStream_t s) {
    if (n == 0) return 0;
    const size_t blocks = (n + 255) / 256;
    ag_k_pair_image<<<(unsigned)(blocks < 4096 ? blocks : 4096), 256, 0, s>>>(x, out, n);
    return (int)cudaGetLastError();
}

/* Chebyshev sums of three components (ncf coefficients each, one after the
 * other from P on) at tau, as float pairs: x and y packed, z beside them. */
__device__ __forceinline__ void ag_cheb_pair(const float2* __restrict__ P, int ncf, AgF2 tau, AgF2* out) {
    const AgF2 two = {2.0f * tau.h, 2.0f * tau.l};
    AgF2 T0 = {1.0f, 0.0f}, T1 = tau;
    float2 a = P[0], b = P[ncf], c = P[2 * ncf];
    AgPk hxy = ag_pk(a.x, b.x), lxy = ag_pk(a.y, b.y), hz = ag_pk(c.x, 0.0f), lz = ag_pk(c.y, 0.0f);
    for (int p = 1; p < ncf; p++) {
        a = P[p]; b = P[ncf + p]; c = P[2 * ncf + p];
        const AgPk th = ag_pk(T1.h, T1.h), tl = ag_pk(T1.l, T1.l);
        ag_pk_acc(ag_pk(a.x, b.x), ag_pk(a.y, b.y), th, tl, hxy, lxy);
        ag_pk_acc(ag_pk(c.x, 0.0f), ag_pk(c.y, 0.0f), th, tl, hz, lz);
        const AgF2 T2 = ag_f2_add(ag_f2_mul(two, T1), ag_f2_neg(T0));
        T0 = T1; T1 = T2;
    }
    out[0] = ag_f2_fast(ag_pk_a(hxy), ag_pk_a(lxy));
    out[1] = ag_f2_fast(ag_pk_b(hxy), ag_pk_b(lxy));
    out[2] = ag_f2_fast(ag_pk_a(hz), ag_pk_a(lz));
}

struct AgOwnSmem {
    double xs[3][32], vs[3][32];
    AgF2 xf[3][32], vf[3][32];
    double rs[3][32], rj[3][32], sv[3][32];     /* origin minus Sun, minus Jupiter; the Sun's velocity */
    AgF2 sp[3][32];                             /* rs as float pairs */
    double pa[3][32];                           /* role 1's FP64 sums without the Sun */
    double ss[3][32], gs[32];                   /* separation from the Sun and -GM / r^3 there */
    AgF2 pf[3][3][32];                          /* pair sums of roles 0, 2, 3 */
    unsigned near[3][32];                       /* bodies left to FP64 */
    unsigned char flag[32];                     /* role 3: harmonics and relativity left to FP64 */
    int any, bad[32];
    AgPkGm gm[AG_MAX_PACKS];
};
struct AgOwnJac {
    double j[18][32];                           /* FP64 parts, then the whole Jacobian */
    double e[18][32];                           /* role 3's */
    AgF2 p[3][7][32];                           /* pair parts: symmetric part and trace sum */
};

/* The packs [p0, p1) of role w (0, 2 or 3; role 3 has relativity and the
 * harmonics too). */
__device__ __forceinline__ void ag_own_range(int packs, int w, int& p0, int& p1) {
    const int n3 = packs > 3 ? (packs - 3) / 3 : 0, h = (packs - n3 + 1) / 2;
    p0 = w == 0 ? 0 : (w == 2 ? h : packs - n3);
    p1 = w == 0 ? h : (w == 2 ? packs - n3 : packs);
}

/* A .440 column as float pairs (km). */
__device__ __forceinline__ void ag_own_column(const DevEphem& E, const float2* __restrict__ pl_pair, size_t rec, int col, double tf,
                                              AgF2* u) {
    const int ncf = E.col_ncf[col], niv = E.col_niv[col];
    const double tt = tf * (double)niv;
    double fl;
    const int b = ag_subinterval(tt, niv, &fl);
    ag_cheb_pair(pl_pair + rec + E.col_off[col] + ncf * 3 * b, ncf, ag_f2_of(fma(2.0, tt - fl, -1.0)), u);
}

/* Bodies close to the particle, or all of them far out, in FP64 from the
 * ephemeris in the reference's operations; and the terms of role 3 that FP32
 * does not cover.  Adds to a and, with JAC, to the Jacobian J. */
template <bool JAC>
static __device__ __noinline__ void ag_own_close(const DevEphem& E, const ForceCfg& c, double t, const AgOwnSmem& S, int lane,
                                                 double* a, double (*J)[6]) {
    const double x[3] = {S.xs[0][lane], S.xs[1][lane], S.xs[2][lane]}, v[3] = {S.vs[0][lane], S.vs[1][lane], S.vs[2][lane]};
    const double rs[3] = {S.rs[0][lane], S.rs[1][lane], S.rs[2][lane]};
    const double* rec = nullptr;
    double tf = 0.0, ax = 0.0, ay = 0.0, az = 0.0;
    ag_planet_record(E, t, &rec, &tf);
    AgSymJac Y = {{0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, 0.0};
    const int packs = E.pv.n_packs;
    for (int r = 0; r < 3; r++) {
        int p0, p1;
        ag_own_range(packs, r == 0 ? 0 : r + 1, p0, p1);
        unsigned m = S.near[r][lane];
        while (m) {
            const int k = 2 * p0 + __ffs(m) - 1;
            m &= m - 1;
            const float gh = (k & 1) ? ag_pk_b(S.gm[k >> 1].h) : ag_pk_a(S.gm[k >> 1].h);
            if (gh == 0.0f) continue;          /* left out by the configuration */
            double b[3], gm;
            if (k < AG_PAIR_PL) {
                gm = E.gm[ag_pair_planet(k)];
                ag_planet_exact<false>(E, rec, tf, ag_pair_planet(k), b, nullptr);
            } else {
                gm = E.ast_gm[k - AG_PAIR_PL];
                ag_asteroid_exact(E, k - AG_PAIR_PL, t, b);
                b[0] -= rs[0]; b[1] -= rs[1]; b[2] -= rs[2];
            }
            const double dx = x[0] + (0.0 - b[0]), dy = x[1] + (0.0 - b[1]), dz = x[2] + (0.0 - b[2]);
            const double ri = rsqrt(fma(dx, dx, fma(dy, dy, dz * dz))), g = gm * ri * ri * ri;
            ax = fma(-g, dx, ax); ay = fma(-g, dy, ay); az = fma(-g, dz, az);
            if (JAC) ag_symjac_term(Y, g, ri, dx, dy, dz);
        }
    }
    if (JAC) ag_symjac_add(Y, J);
    const unsigned f = S.flag[lane];
    if (f & 1) {
        double b[3];
        ag_planet_exact<false>(E, rec, tf, AG_EAR, b, nullptr);
        const double dx = x[0] + (0.0 - b[0]), dy = x[1] + (0.0 - b[1]), dz = x[2] + (0.0 - b[2]);
        ag_term_earth_h<JAC>(E, c, dx, dy, dz, rsqrt(fma(dx, dx, fma(dy, dy, dz * dz))), ax, ay, az, J);
    }
    const double d[3] = {x[0] + rs[0], x[1] + rs[1], x[2] + rs[2]};
    const double ri = rsqrt(fma(d[0], d[0], fma(d[1], d[1], d[2] * d[2])));
    if (f & 2) ag_term_sun_h<JAC>(E, c, d[0], d[1], d[2], ri, ax, ay, az, J);
    if (f & 4) {
        /* relativity far out, where the planets' sums are no small parts of it */
        double af[3] = {0.0, 0.0, 0.0}, gp[3] = {0.0, 0.0, 0.0}, ut = 0.0, up = 0.0;
        for (int k = 1; k < AG_NPL; k++) {
            double b[3];
            ag_planet_exact<false>(E, rec, tf, k, b, nullptr);
            const double sx = (0.0 - rs[0]) - b[0], sy = (0.0 - rs[1]) - b[1], sz = (0.0 - rs[2]) - b[2];
            const double si = rsqrt(fma(sx, sx, fma(sy, sy, sz * sz))), gr = E.gm[k] * si, q = gr * si * si;
            ut += gr;
            af[0] = fma(-q, sx, af[0]); af[1] = fma(-q, sy, af[1]); af[2] = fma(-q, sz, af[2]);
            const double px = x[0] - b[0], py = x[1] - b[1], pz = x[2] - b[2];
            const double pi = rsqrt(fma(px, px, fma(py, py, pz * pz)));
            up = fma(E.gm[k], pi, up);
            if (JAC) {
                const double g = E.gm[k] * pi * pi * pi;
                gp[0] = fma(g, px, gp[0]); gp[1] = fma(g, py, gp[1]); gp[2] = fma(g, pz, gp[2]);
            }
        }
        const double w[3] = {S.sv[0][lane], S.sv[1][lane], S.sv[2][lane]};
        if (JAC) {
            double ea[3];
            ag_fast_eih_jac(E, d, ri, v, w, af, ut, up, gp, ea, J);
            ax += ea[0]; ay += ea[1]; az += ea[2];
        } else {
            double v2 = 0.0, w2 = 0.0, vw = 0.0, dw = 0.0, da = 0.0, g = 0.0;
            for (int k = 0; k < 3; k++) {
                v2 = fma(v[k], v[k], v2); w2 = fma(w[k], w[k], w2); vw = fma(v[k], w[k], vw);
                dw = fma(d[k], w[k], dw); da = fma(d[k], af[k], da); g = fma(d[k], 4.0 * v[k] - 3.0 * w[k], g);
            }
            const double gr = E.gm[AG_SUN] * ri, pre = E.over_c_squared * gr * ri * ri, ga = 3.5 * E.over_c_squared * gr;
            const double fac = v2 - 4.0 * (gr + up) - ut + 2.0 * w2 - 4.0 * vw - 1.5 * (dw * ri) * (dw * ri) - 0.5 * da;
            ax += -pre * fac * d[0] + pre * g * (v[0] - w[0]) + ga * af[0];
            ay += -pre * fac * d[1] + pre * g * (v[1] - w[1]) + ga * af[1];
            az += -pre * fac * d[2] + pre * g * (v[2] - w[2]) + ga * af[2];
        }
    }
    a[0] += ax; a[1] += ay; a[2] += az;
}

template <bool JAC>
__global__ void __launch_bounds__(128, JAC ? 2 : 4) ag_k_forces_own(const DevEphem* __restrict__ Ep, const float2* __restrict__ pl_pair,
                                                                    const float2* __restrict__ spk_pair, ForceCfg c, int n,
                                                                    const double* __restrict__ t, const double* __restrict__ state,
                                                                    const double* __restrict__ params,
                                                                    const double* __restrict__ var_state, double* __restrict__ acc,
                                                                    double* __restrict__ var_acc, int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char ag_own_dyn[];
    __shared__ AgOwnSmem S;
    const DevEphem& E = *Ep;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, tid = threadIdx.x, i = 32 * blockIdx.x + lane;
    const bool on = i < n;
    const size_t ii = on ? i : 32 * (size_t)blockIdx.x;
    AgOwnJac& JS = *reinterpret_cast<AgOwnJac*>(ag_own_dyn);
    /* positions of the pair bodies as float pairs: planets barycentric,
     * asteroids heliocentric (AU): pos[(3 k + comp) * 32 + lane] */
    AgF2* pos = reinterpret_cast<AgF2*>(ag_own_dyn + (JAC ? sizeof(AgOwnJac) : 0));
    const int bodies = AG_PAIR_PL + E.n_ast, packs = E.pv.n_packs;
    const double ti = t[ii];
    if (tid == 0) S.any = 0;
    if (tid < 32) S.bad[tid] = AG_OK;
    {
        const bool pl = (c.forces & AG_F_PLANETS) != 0, as = (c.forces & AG_F_AST) != 0;
        if (tid < packs) {
            AgPkGm g = E.pv.gm[tid];
            const bool a = 2 * tid < AG_PAIR_PL ? pl : as, b = 2 * tid + 1 < AG_PAIR_PL ? pl : as;
            g.h = ag_pk(a ? ag_pk_a(g.h) : 0.0f, b ? ag_pk_b(g.h) : 0.0f);
            g.l = ag_pk(a ? ag_pk_a(g.l) : 0.0f, b ? ag_pk_b(g.l) : 0.0f);
            g.ta = a ? fmaxf(2.0f * g.ta, JAC ? E.pv.jac_thr[2 * tid] : 0.0f) : 0.0f;
            g.tb = b ? fmaxf(2.0f * g.tb, JAC ? E.pv.jac_thr[2 * tid + 1] : 0.0f) : 0.0f;
            S.gm[tid] = g;
        }
    }
    __syncthreads();
    /* ---- positions */
    const double* rec = nullptr;
    double tf = 0.0;
    const int pst = ag_planet_record(E, ti, &rec, &tf);
    if (pst != AG_OK) S.bad[lane] = pst;
    else {
        const size_t ro = (size_t)(rec - E.pl_data);
        const AgF2 icau = {E.pv.inv_cau_h, E.pv.inv_cau_l};
        auto put = [&](int k, const AgF2* u) {
#pragma unroll
            for (int m = 0; m < 3; m++) pos[(3 * k + m) * 32 + lane] = ag_f2_mul(u[m], icau);
        };
        if (wid == 1) {
            /* the Sun */
#pragma unroll
            for (int m = 0; m < 3; m++) {
                double v;
                const double x = 0.0 - ag_col1v(E, rec, AG_C_SUN, m, tf, &v) * E.inv_cau;
                S.rs[m][lane] = x;
                S.sv[m][lane] = v;
                S.sp[m][lane] = ag_f2_of(x);
            }
        } else if (wid == 0) {
            double b[3];
            ag_planet_exact<false>(E, rec, tf, AG_JUP, b, nullptr);
            for (int m = 0; m < 3; m++) S.rj[m][lane] = 0.0 - b[m];
            AgF2 e[3], l[3], u[3];
            ag_own_column(E, pl_pair, ro, AG_C_EMB, tf, e);
            ag_own_column(E, pl_pair, ro, AG_C_LUN, tf, l);
            for (int m = 0; m < 3; m++) u[m] = ag_f2_add(e[m], ag_f2_mul(l[m], {E.pv.f_earth_h, E.pv.f_earth_l}));
            put(2, u);
            for (int m = 0; m < 3; m++) u[m] = ag_f2_add(e[m], ag_f2_mul(l[m], {E.pv.f_moon_h, E.pv.f_moon_l}));
            put(3, u);
        } else if (wid == 2) {
            /* Mercury, Venus, Mars, Saturn .. Pluto */
#pragma unroll 1
            for (int q = 0; q < 7; q++) {
                AgF2 u[3];
                const int k = q < 2 ? q : q + 2;
                ag_own_column(E, pl_pair, ro, k < 2 ? k : (k == 4 ? AG_C_MAR : k), tf, u);
                put(k, u);
            }
        }
    }
    if (wid != 1) {
        const int m0 = wid == 0 ? 0 : (wid == 2 ? E.n_ast / 8 : E.n_ast / 8 + E.n_ast / 4);
        const int m1 = wid == 0 ? E.n_ast / 8 : (wid == 2 ? E.n_ast / 8 + E.n_ast / 4 : E.n_ast);
        const AgF2 km = {(float)(1.0 / 149597870.7), (float)(1.0 / 149597870.7 - (double)(float)(1.0 / 149597870.7))};
        const double jd = E.jd_ref + ti;
        const bool need = (c.forces & AG_F_AST) != 0;
        const bool inside = jd >= E.ast_beg_max && jd <= E.ast_end_min;      /* every asteroid's span */
        long long seg_key0 = 0, seg_key1 = 0;
        int b = 0;
        double mid = 0.0, rad = 0.0;
        AgF2 z = {0.0f, 0.0f};
#pragma unroll 1
        for (int m = m0; m < m1; m++) {
            AgF2 u[3] = {{0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}};
            if (inside || (jd >= E.ast_beg[m] && jd <= E.ast_end[m])) {      /* false for NaN */
                int k = 0;
                if (E.ast_nseg[m] > 1) {
                    k = (int)((jd - E.ast_beg[m]) / E.ast_res[m]);
                    if (k >= E.ast_nseg[m]) k = E.ast_nseg[m] - 1;
                }
                const AgSpkSeg sg = E.segs[E.ast_seg0[m] + k];
                const long long k0 = __double_as_longlong(sg.init_jd), k1 = __double_as_longlong(sg.inv_intlen_days);
                if (k0 != seg_key0 || k1 != seg_key1) {
                    /* record of the segment's grid: the asteroids usually share it */
                    b = (int)(((E.jd_ref - sg.init_jd) + ti) * sg.inv_intlen_days);
                    seg_key0 = k0;
                    seg_key1 = k1;
                }
                const int bb = b >= sg.nrec ? sg.nrec - 1 : (b < 0 ? 0 : b);
                const AgRecMeta meta = E.rec_meta[sg.meta_off + bb];
                if (__double_as_longlong(meta.x) != __double_as_longlong(mid) ||
                    __double_as_longlong(meta.z) != __double_as_longlong(rad)) {
                    z = ag_f2_of(((E.jd_ref - meta.x) + ti) * meta.z);
                    mid = meta.x;
                    rad = meta.z;
                }
                ag_cheb_pair(spk_pair + sg.data_off + (size_t)bb * sg.R + 2, sg.P, z, u);
            } else if (need) {
                S.bad[lane] = AG_ERR_COVERAGE;
            }
            for (int q = 0; q < 3; q++) pos[(3 * (AG_PAIR_PL + m) + q) * 32 + lane] = ag_f2_mul(u[q], km);
        }
    }
    double prm[3] = {0.0, 0.0, 0.0};
    if (wid == 1) {
        if (params)
            for (int k = 0; k < 3; k++) prm[k] = params[3 * ii + k];
    } else {
        const int k = wid == 0 ? 0 : wid - 1;
        const double x = state[6 * ii + k], v = state[6 * ii + 3 + k];
        S.xs[k][lane] = x; S.vs[k][lane] = v;
        S.xf[k][lane] = ag_f2_of(x); S.vf[k][lane] = ag_f2_of(v);
    }
    __syncthreads();
    /* ---- terms */
    const bool direct = (c.forces & AG_F_PLANETS) != 0;
    if (wid == 1) {
        double J[3][6], JA[3][3];
        if (JAC)
            for (int a = 0; a < 3; a++)
                for (int b = 0; b < 6; b++) J[a][b] = 0.0;
        const double x[3] = {S.xs[0][lane], S.xs[1][lane], S.xs[2][lane]};
        const double s[3] = {x[0] + S.rs[0][lane], x[1] + S.rs[1][lane], x[2] + S.rs[2][lane]};
        const double ri = rsqrt(fma(s[0], s[0], fma(s[1], s[1], s[2] * s[2])));
        double ax = 0.0, ay = 0.0, az = 0.0;
        const bool ng = (c.forces & AG_F_NONGRAV) && params && (prm[0] != 0.0 || prm[1] != 0.0 || prm[2] != 0.0);
        if (ng || (c.forces & (AG_F_GR_POT | AG_F_GR_SIMPLE))) {
            const double dv[3] = {S.vs[0][lane] - S.sv[0][lane], S.vs[1][lane] - S.sv[1][lane], S.vs[2][lane] - S.sv[2][lane]};
            bool has_ng;
            if (ng) ag_term_nongrav<JAC>(c, s, ri, dv, prm, ax, ay, az, J, JA, &has_ng);
            if (c.forces & AG_F_GR_POT) ag_term_gr_pot<JAC>(E, s, ri, ax, ay, az, J);
            if (c.forces & AG_F_GR_SIMPLE) ag_term_gr_simple<JAC>(E, s, ri, dv, ax, ay, az, J);
        }
        AgSymJac Y = {{0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, 0.0};
        if (direct) {
            const double j[3] = {x[0] + S.rj[0][lane], x[1] + S.rj[1][lane], x[2] + S.rj[2][lane]};
            const double rj = rsqrt(fma(j[0], j[0], fma(j[1], j[1], j[2] * j[2])));
            ag_term_planet<JAC>(E, true, AG_JUP, j[0], j[1], j[2], rj, ax, ay, az, &Y);
        }
        /* the Sun's term goes into the last sum unrounded */
        const double gs = E.gm[AG_SUN] * ri * ri * ri;
        S.gs[lane] = -gs;
        S.ss[0][lane] = s[0]; S.ss[1][lane] = s[1]; S.ss[2][lane] = s[2];
        if (JAC) {
            ag_symjac_term(Y, gs, ri, s[0], s[1], s[2]);
            ag_symjac_add(Y, J);
#pragma unroll
            for (int a = 0; a < 3; a++)
#pragma unroll
                for (int b = 0; b < 6; b++) JS.j[6 * a + b][lane] = J[a][b];
        }
        S.pa[0][lane] = ax; S.pa[1][lane] = ay; S.pa[2][lane] = az;
    } else {
        const int out = wid == 0 ? 0 : wid - 1;
        const AgF2 xf[3] = {S.xf[0][lane], S.xf[1][lane], S.xf[2][lane]};
        const AgF2 sp[3] = {S.sp[0][lane], S.sp[1][lane], S.sp[2][lane]};
        const float sx = xf[0].h + sp[0].h, sy = xf[1].h + sp[1].h, sz = xf[2].h + sp[2].h;
        const float rs2 = fmaf(sx, sx, fmaf(sy, sy, sz * sz));
        /* origin minus body k, component m */
        auto rel = [&](int k, int m) -> AgF2 {
            if (k >= bodies) return {1e6f, 0.0f};
            const AgF2 p = pos[(3 * k + m) * 32 + lane];
            return k < AG_PAIR_PL ? ag_f2_neg(p) : ag_f2_add(sp[m], ag_f2_neg(p));
        };
        AgPkSum P;
        AgPkJac PJ;
        AgPk xh[3], xl[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            xh[k] = ag_pk(xf[k].h, xf[k].h);
            xl[k] = ag_pk(xf[k].l, xf[k].l);
            P.h[k] = P.l[k] = ag_pk(0.0f, 0.0f);
        }
        if (JAC) ag_pk_jac_clear(PJ);
        unsigned near = 0;
        int p0, p1;
        ag_own_range(packs, wid, p0, p1);
#pragma unroll 1
        for (int p = p0; p < p1; p++) {
            AgPkRel R;
#pragma unroll
            for (int m = 0; m < 3; m++) {
                const AgF2 a = rel(2 * p, m), b = rel(2 * p + 1, m);
                R.c[m].h = ag_pk(a.h, b.h);
                R.c[m].l = ag_pk(a.l, b.l);
            }
            near |= ag_pk_term<JAC>(R, S.gm[p], xh, xl, rs2, P, &PJ) << (2 * (p - p0));
        }
        AgF2 s[3];
#pragma unroll
        for (int k = 0; k < 3; k++)
            s[k] = ag_f2_add({ag_pk_a(P.h[k]), ag_pk_a(P.l[k])}, {ag_pk_b(P.h[k]), ag_pk_b(P.l[k])});
        const float big = fmaxf(fabsf(xf[0].h), fmaxf(fabsf(xf[1].h), fabsf(xf[2].h)));
        const bool wild = !(big < 1e6f);
        unsigned flag = 0;
        double J[3][6];
        double ea[3];
        /* harmonics' Jacobian, xx xy xz yy yz zz: FP32 and, of a Sun nearer than 0.5 AU, float pairs */
        float hj[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        AgF2 nj[6] = {{0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}};
        if (wid == 3) {
            if (JAC)
                for (int a = 0; a < 3; a++)
                    for (int b = 0; b < 6; b++) J[a][b] = 0.0;
            if (c.forces & AG_F_EIH) {
                /* planets' pull on the Sun and their potentials there and at the
                 * particle (1e-3 of the term's factor: FP32) */
                float af[3] = {0.0f, 0.0f, 0.0f}, ut = 0.0f, up = 0.0f, gp[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll 1
                for (int k = 0; k < AG_NPL - 1; k++) {
                    float q[3], gm;
                    if (k < AG_PAIR_PL) {
                        gm = (k & 1) ? S.gm[k >> 1].gb : S.gm[k >> 1].ga;
                        for (int m = 0; m < 3; m++) q[m] = -pos[(3 * k + m) * 32 + lane].h;
                    } else {
                        gm = E.pv.gm_jup;
                        for (int m = 0; m < 3; m++) q[m] = ag_d2f_int(S.rj[m][lane]);
                    }
                    const float a[3] = {q[0] - sp[0].h, q[1] - sp[1].h, q[2] - sp[2].h};
                    const float b[3] = {q[0] + xf[0].h, q[1] + xf[1].h, q[2] + xf[2].h};
                    const float ia = rsqrtf(fmaf(a[0], a[0], fmaf(a[1], a[1], a[2] * a[2])));
                    const float ib = rsqrtf(fmaf(b[0], b[0], fmaf(b[1], b[1], b[2] * b[2])));
                    const float fa = gm * ia * ia * ia, fb = gm * ib * ib * ib;
                    ut = fmaf(gm, ia, ut);
                    up = fmaf(gm, ib, up);
                    for (int m = 0; m < 3; m++) { af[m] = fmaf(-fa, a[m], af[m]); gp[m] = fmaf(fb, b[m], gp[m]); }
                }
                const bool far = !(big < 200.0f);
                if (JAC && !far) {
                    const double x[3] = {S.xs[0][lane], S.xs[1][lane], S.xs[2][lane]};
                    const double v[3] = {S.vs[0][lane], S.vs[1][lane], S.vs[2][lane]};
                    const double w[3] = {S.sv[0][lane], S.sv[1][lane], S.sv[2][lane]};
                    const double d[3] = {x[0] + S.rs[0][lane], x[1] + S.rs[1][lane], x[2] + S.rs[2][lane]};
                    const double aj[3] = {ag_f2d_int(af[0]), ag_f2d_int(af[1]), ag_f2d_int(af[2])};
                    const double g[3] = {ag_f2d_int(gp[0]), ag_f2d_int(gp[1]), ag_f2d_int(gp[2])};
                    ag_fast_eih_jac(E, d, rsqrt(fma(d[0], d[0], fma(d[1], d[1], d[2] * d[2]))), v, w, aj, ag_f2d_int(ut),
                                   ag_f2d_int(up), g, ea, J);
                    for (int k = 0; k < 3; k++) s[k] = ag_f2_add(s[k], ag_f2_of(ea[k]));
                } else if (!far) {
                    const AgF2 d[3] = {ag_f2_add(xf[0], sp[0]), ag_f2_add(xf[1], sp[1]), ag_f2_add(xf[2], sp[2])};
                    const AgF2 v[3] = {S.vf[0][lane], S.vf[1][lane], S.vf[2][lane]};
                    const float w[3] = {ag_d2f_int(S.sv[0][lane]), ag_d2f_int(S.sv[1][lane]), ag_d2f_int(S.sv[2][lane])};
                    AgF2 e[3];
                    ag_fast_eih(E.pv, w, af, ut, d, v, up, e);
                    for (int k = 0; k < 3; k++) s[k] = ag_f2_add(s[k], e[k]);
                }
                if (far) flag |= 4;
            }
            if (c.forces & AG_F_EARTH_H) {
                float q[3];
                for (int m = 0; m < 3; m++) {
                    const AgF2 p = pos[(3 * 2 + m) * 32 + lane];
                    q[m] = ag_f2_sep(xf[m], -p.h, -p.l);
                }
                const float r2 = fmaf(q[0], q[0], fmaf(q[1], q[1], q[2] * q[2]));
                /* the Jacobian's share is larger by r / d: FP64 within 0.1 AU */
                if (!(r2 >= (JAC ? 1.0e-2f : 4.0e-4f) && r2 < 1e30f)) flag |= 1;
                else {
                    ag_fast_earth_h(E.pv, c, q, r2, s);
                    if (JAC) ag_fast_earth_hj(E.pv, c, q, r2, hj);
                }
            }
            if (c.forces & AG_F_SUN_H) {
                if (!(rs2 >= 1.0e-2f && rs2 < 1e30f)) flag |= 2;
                else if (rs2 < AG_SUN_H_FAR2) {
                    const AgF2 d[3] = {ag_q_add(xf[0], sp[0]), ag_q_add(xf[1], sp[1]), ag_q_add(xf[2], sp[2])};
                    ag_fast_sun_near<JAC>(E.pv, c, d, s, nj);
                } else {
                    ag_fast_sun_h(E.pv, c, sx, sy, sz, rs2, s);
                    const float q[3] = {sx, sy, sz};
                    if (JAC) ag_fast_sun_hj(E.pv, c, q, rs2, hj);
                }
            }
        }
        if (wild) {
            near = (1u << (2 * (p1 - p0))) - 1u;
            for (int k = 0; k < 3; k++) s[k] = {0.0f, 0.0f};
        }
        S.near[out][lane] = near;
        if (wid == 3) S.flag[lane] = (unsigned char)flag;
        if (near | flag) S.any = 1;
#pragma unroll
        for (int k = 0; k < 3; k++) S.pf[out][k][lane] = s[k];
        if (JAC) {
#pragma unroll
            for (int k = 0; k < 7; k++) {
                float ah, al, bh, bl;
                ag_pk_jac_get(PJ, k, 0, ah, al);
                ag_pk_jac_get(PJ, k, 1, bh, bl);
                if (k < 6) bl += hj[k];
                AgF2 p = ag_f2_add({ah, al}, {bh, bl});
                if (wid == 3 && k < 6) p = ag_f2_add(p, nj[k]);
                JS.p[out][k][lane] = wild ? AgF2{0.0f, 0.0f} : p;
            }
            if (wid == 3) {
#pragma unroll
                for (int a = 0; a < 3; a++) {
#pragma unroll
                    for (int b = 0; b < 6; b++) JS.e[6 * a + b][lane] = J[a][b];
                }
            }
        }
    }
    __syncthreads();
    if (S.any) {
        if (wid == 1 && (S.near[0][lane] | S.near[1][lane] | S.near[2][lane] | S.flag[lane]) && S.bad[lane] == AG_OK) {
            double a[3] = {S.pa[0][lane], S.pa[1][lane], S.pa[2][lane]}, J[3][6];
            for (int q = 0; q < 18; q++) J[q / 6][q % 6] = 0.0;
            ag_own_close<JAC>(E, c, ti, S, lane, a, J);
            S.pa[0][lane] = a[0]; S.pa[1][lane] = a[1]; S.pa[2][lane] = a[2];
            if (JAC)
                for (int q = 0; q < 18; q++) JS.j[q][lane] += J[q / 6][q % 6];
        }
        __syncthreads();
    }
    if (on && wid != 1) {
        const int k = wid == 0 ? 0 : wid - 1;
        const AgF2 s = ag_f2_add(ag_f2_add(S.pf[2][k][lane], S.pf[1][k][lane]), S.pf[0][k][lane]);
        if (S.bad[lane] == AG_OK) acc[3 * (size_t)i + k] = fma(S.gs[lane], S.ss[k][lane], ag_f2_to(s) + S.pa[k][lane]);
        if (k == 0 && status) status[i] = S.bad[lane];
    }
    if constexpr (JAC) {
        /* the Jacobian, its elements over the warps, then its six products */
        constexpr int sym[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
#pragma unroll
        for (int q = 0; q < 18; q++) {
            const int a = q / 6, b = q % 6;
            if ((q & 3) != wid) continue;
            double s = JS.e[q][lane];
            if (b < 3) {
                AgF2 p = ag_f2_add(ag_f2_add(JS.p[0][sym[a][b % 3]][lane], JS.p[1][sym[a][b % 3]][lane]),
                                   JS.p[2][sym[a][b % 3]][lane]);
                if (a == b)
                    p = ag_f2_add(p, ag_f2_neg(ag_f2_add(ag_f2_add(JS.p[0][6][lane], JS.p[1][6][lane]), JS.p[2][6][lane])));
                s += ag_f2_to(p);
            }
            JS.j[q][lane] += s;
        }
        __syncthreads();
        if (on && S.bad[lane] == AG_OK) {
            double J[18];
#pragma unroll
            for (int q = 0; q < 18; q++) J[q] = JS.j[q][lane];
            for (int q = wid; q < 6; q += 4) {
                const double* vs = var_state + ((size_t)i * 6 + q) * 6;
                double d[6];
#pragma unroll
                for (int k = 0; k < 6; k++) d[k] = vs[k];
#pragma unroll
                for (int a = 0; a < 3; a++) {
                    double o = J[6 * a] * d[0];
#pragma unroll
                    for (int k = 1; k < 6; k++) o = fma(J[6 * a + k], d[k], o);
                    var_acc[((size_t)i * 6 + q) * 3 + a] = o;
                }
            }
        }
    }
}

/* Whether ag_launch_forces_own takes the configuration (with variational
 * particles also every direct term on: the variational equations keep bodies
 * whose force is off, src/forces.c:352-432). */
bool ag_forces_own_covers(const DevEphem& E, const ForceCfg& c, int nv) {
    const int all = AG_F_PLANETS | AG_F_AST;
    return !E.pl_spk && ag_fast_covers(c) && (nv == 0 || (c.forces & all) == all);
}

int ag_launch_forces_own(const DevEphem& E, const float2* pl_pair, const float2* spk_pair, const ForceCfg& c, int n,
                         const double* t, const double* state, const double* params, int nv, const double* var_state,
                         double* acc, double* var_acc, int* status, cudaStream_t s) {
    const int blocks = (n + 31) / 32;
    auto bytes = [](int n_ast) { return sizeof(AgF2) * 3 * 32 * (AG_PAIR_PL + (size_t)n_ast); };
    if (nv) {
        /* the limit is the kernel's, shared by every thread of the process: always the largest */
        const cudaError_t e = cudaFuncSetAttribute(ag_k_forces_own<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)(bytes(AG_MAX_AST) + sizeof(AgOwnJac)));
        if (e != cudaSuccess) return (int)e;
        ag_k_forces_own<true><<<blocks, 128, bytes(E.n_ast) + sizeof(AgOwnJac), s>>>(E.self_dev, pl_pair, spk_pair, c, n, t, state, params, var_state, acc, var_acc, status);
    } else {
        ag_k_forces_own<false><<<blocks, 128, bytes(E.n_ast), s>>>(E.self_dev, pl_pair, spk_pair, c, n, t, state, params, nullptr, acc, nullptr, status);
    }
    return (int)cudaGetLastError();
}
