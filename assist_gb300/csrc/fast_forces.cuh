/*
 * fast_forces.cuh -- the block-cooperative force evaluation of the default
 * frame (barycentric, the Sun's gravity on, relativity with the Sun as its
 * source) with FP64 kept for what needs it: the Sun's and Jupiter's direct
 * terms, the non-gravitational term and any body close to the particle.  The
 * other planets and the asteroids, whose terms are below 1e-3 of the Sun's,
 * are float pairs two at a time (pair_terms.cuh); the relativistic term (below
 * 1e-6 of the Sun's) is a float pair with its small parts in FP32; the
 * harmonics are FP32 where they are below 1.1e-10 (the Earth's beyond 0.02 AU,
 * the Sun's beyond 0.5 AU), the Sun's float pairs down to 0.1 AU and FP64
 * nearer.  The evaluation's error is what it is with every term in FP64
 * (ag_pair_thr2's comment has the figures).
 *
 * Eight warps (roles) share an evaluation, lane l of each working on particle l:
 *   role 0       Jupiter, FP64           role 1   Sun, non-gravitational, GR, FP64
 *   roles 2, 3   a few of the pair terms' packs; the Sun's, the Earth's harmonics
 *   role 4       relativity              roles 5, 6, 7   the other packs
 * An SM does one FP64 warp instruction in 19 cycles over its four
 * sub-partitions (64 to 76 on one warp): about 150 a group and evaluation with
 * IAS15's own, against 515 with every term but the asteroids' in FP64.  Two
 * warps a sub-partition, because the FP32 streams are chains of dependent
 * instructions (7 cycles an instruction with one).
 *
 * The tables of up to eight times are built together (ag_fast_tables): a
 * lane forms one body's three components at one time, so a step's eight
 * tables take about 60 FP64 instructions on each warp, where eight separate
 * tables with a lane a component took 1,700 over four.
 */
#ifndef ASSIST_GB300_FAST_FORCES_CUH
#define ASSIST_GB300_FAST_FORCES_CUH

#include "coop_forces.cuh"

/* The force configurations this evaluation covers (the general one,
 * coop_forces.cuh, has the rest). */
__host__ __device__ __forceinline__ bool ag_fast_covers(const ForceCfg& c) {
    return c.geocentric == 0 && (c.forces & AG_F_SUN) != 0 && (!(c.forces & AG_F_EIH) || c.gr_eih_sources == 1);
}

/* One time's table: this header, then n_packs AgPkRel, then the FP64 origin
 * minus body of the pair terms' bodies (for a particle close to one). */
struct alignas(16) AgFastNode {
    double rs[3], rj[3];            /* origin minus Sun, minus Jupiter */
    double sv[3];                   /* the Sun's velocity */
    AgF2 sp[3];                     /* rs as a float pair */
    float jf[3], vf[3];             /* rj, sv in FP32 */
    float af[3], ut;                /* the planets' pull on the Sun and their potential there */
};

/* Sizes of the tables in dynamic shared memory. */
struct AgFastLayout {
    int packs, bodies, rel_off, stride;
    __host__ __device__ explicit AgFastLayout(int n_ast) {
        bodies = AG_PAIR_PL + n_ast;
        packs = (bodies + 1) / 2;
        rel_off = (int)sizeof(AgFastNode) + packs * (int)sizeof(AgPkRel);
        stride = (rel_off + bodies * 24 + 15) / 16 * 16;
    }
};

struct AgFastView {
    unsigned char* base;
    AgFastLayout L;
    __device__ __forceinline__ AgFastView(unsigned char* b, int n_ast) : base(b), L(n_ast) {}
    __device__ __forceinline__ AgFastNode& node(int n) const { return *reinterpret_cast<AgFastNode*>(base + n * L.stride); }
    __device__ __forceinline__ AgPkRel* packs(int n) const {
        return reinterpret_cast<AgPkRel*>(base + n * L.stride + sizeof(AgFastNode));
    }
    __device__ __forceinline__ double* rel(int n) const {
        return reinterpret_cast<double*>(base + n * L.stride + L.rel_off);
    }
};

/* A block's shared arrays of the evaluation. */
#define AG_FAST_WARPS 8
#define AG_FAST_THREADS (32 * AG_FAST_WARPS)
#define AG_FAST_SLOTS 6             /* roles 2..7 */
struct AgFastShared {
    double xs[3][32], vs[3][32];    /* particle states at the node */
    AgF2 xf[3][32], vf[3][32];      /* and as float pairs */
    double pa[2][3][32];            /* roles 0 and 1: FP64 partial accelerations without the Sun's */
    double ss[3][32], gs[32];       /* separation from the Sun and -GM / r^3 there */
    AgF2 pf[AG_FAST_SLOTS][3][32];  /* roles 2..7: pair sums */
    double pn[AG_FAST_SLOTS][3][32];            /* their FP64 parts, where near[] says so */
    int near[AG_FAST_SLOTS];
    double sun[8][3];               /* the Sun's raw position sums of the tables */
    AgPkGm gm[AG_MAX_PACKS];        /* masses; zero where the configuration leaves the body out */
};

/* Masses and thresholds (JAC: for terms with Jacobian) of the pair terms for
 * configuration c (whole block; the caller synchronises). */
template <bool JAC = false>
__device__ __forceinline__ void ag_fast_masses(const DevEphem& E, const ForceCfg& c, AgFastShared& F, int tid) {
    const bool pl = (c.forces & AG_F_PLANETS) != 0, as = (c.forces & AG_F_AST) != 0;
    if (tid < E.pv.n_packs) {
        AgPkGm g = E.pv.gm[tid];
        if (JAC) { g.ta = E.pv.jac_thr[2 * tid]; g.tb = E.pv.jac_thr[2 * tid + 1]; }
        const bool a = 2 * tid < AG_PAIR_PL ? pl : as, b = 2 * tid + 1 < AG_PAIR_PL ? pl : as;
        g.h = ag_pk(a ? ag_pk_a(g.h) : 0.0f, b ? ag_pk_b(g.h) : 0.0f);
        g.l = ag_pk(a ? ag_pk_a(g.l) : 0.0f, b ? ag_pk_b(g.l) : 0.0f);
        if (!a) g.ta = 0.0f;
        if (!b) g.tb = 0.0f;
        F.gm[tid] = g;
    }
}

/* ------------------------------------------------------------------ tables */

/* The position sums of a .440 column's three components (km). */
__device__ __forceinline__ void ag_col3(const DevEphem& E, const double* rec, int col, double tf, double* u) {
    const int ncf = E.col_ncf[col], niv = E.col_niv[col];
    const double tt = tf * (double)niv;
    double fl;
    const int b = ag_subinterval(tt, niv, &fl);
    const double t0 = fma(2.0, tt - fl, -1.0), two_t0 = 2.0 * t0;
    const double* P = rec + E.col_off[col] + ncf * 3 * b;
    double x = fma(t0, P[1], P[0]), y = fma(t0, P[ncf + 1], P[ncf]), z = fma(t0, P[2 * ncf + 1], P[2 * ncf]);
    double T0 = 1.0, T1 = t0;
#pragma unroll 2
    for (int p = 2; p < ncf; p++) {
        const double T2 = fma(two_t0, T1, -T0);
        x = fma(T2, P[p], x); y = fma(T2, P[ncf + p], y); z = fma(T2, P[2 * ncf + p], z);
        T0 = T1; T1 = T2;
    }
    u[0] = x; u[1] = y; u[2] = z;
}

/* One component of a .440 column: position (km) and velocity (AU/day). */
__device__ __forceinline__ double ag_col1v(const DevEphem& E, const double* rec, int col, int comp, double tf, double* v) {
    const int ncf = E.col_ncf[col], niv = E.col_niv[col];
    const double tt = tf * (double)niv;
    double fl;
    const int b = ag_subinterval(tt, niv, &fl);
    const double t0 = fma(2.0, tt - fl, -1.0), two_t0 = 2.0 * t0;
    const double* P = rec + E.col_off[col] + ncf * (3 * b + comp);
    double u = fma(t0, P[1], P[0]), w = P[1], T0 = 1.0, T1 = t0, S0 = 0.0, S1 = 1.0;
#pragma unroll 2
    for (int p = 2; p < ncf; p++) {
        const double T2 = fma(two_t0, T1, -T0), S2 = fma(two_t0, S1, fma(2.0, T1, -S0));
        u = fma(T2, P[p], u);
        w = fma(S2, P[p], w);
        T0 = T1; T1 = T2; S0 = S1; S1 = S2;
    }
    *v = w * E.col_vscale[col];
    return u;
}

/* An SPK segment's record at time t: the first X coefficient, the normalised
 * time z and the coefficients per component. */
__device__ __forceinline__ const double* ag_spk_record(const DevEphem& E, const AgSpkSeg& sg, const AgRecMeta* meta,
                                                       const double* data, double t, double* z, double* rate) {
    int b = (int)(((E.jd_ref - sg.init_jd) + t) * sg.inv_intlen_days);
    if (b >= sg.nrec) b = sg.nrec - 1;
    if (b < 0) b = 0;
    const AgRecMeta m = meta[sg.meta_off + b];
    *z = ((E.jd_ref - m.x) + t) * m.z;
    *rate = m.z;
    return data + sg.data_off + (size_t)b * sg.R + 2;
}

/* Position sums (km) of an SPK record's three components. */
__device__ __forceinline__ void ag_spk3(const double* X, int P, double z, double* u) {
    const double two_z = 2.0 * z;
    double x = X[0], y = X[P], w = X[2 * P], T0 = 1.0, T1 = z;
    if (P > 1) { x = fma(X[1], z, x); y = fma(X[P + 1], z, y); w = fma(X[2 * P + 1], z, w); }
#pragma unroll 2
    for (int q = 2; q < P; q++) {
        const double T2 = fma(two_z, T1, -T0);
        x = fma(X[q], T2, x); y = fma(X[P + q], T2, y); w = fma(X[2 * P + q], T2, w);
        T0 = T1; T1 = T2;
    }
    u[0] = x; u[1] = y; u[2] = w;
}

/* The same for one component with its velocity (km per day). */
__device__ __forceinline__ double ag_spk1v(const double* X, int P, double z, double rate, double* v) {
    const double two_z = 2.0 * z;
    double u = X[0], w = 0.0, T0 = 1.0, T1 = z, S0 = 0.0, S1 = 1.0;
    if (P > 1) { u = fma(X[1], z, u); w = X[1]; }
    for (int q = 2; q < P; q++) {
        const double T2 = fma(two_z, T1, -T0), S2 = fma(two_z, S1, fma(2.0, T1, -S0));
        u = fma(X[q], T2, u);
        w = fma(X[q], S2, w);
        T0 = T1; T1 = T2; S0 = S1; S1 = S2;
    }
    *v = w * rate;
    return u;
}

/* Planets-SPK slot at time t (its segment chosen as src/spk.c:492-548 does),
 * or a coverage error. */
__device__ __forceinline__ int ag_spk_slot(const DevEphem& E, int slot, double t, const double** X, int* P, double* z,
                                           double* rate) {
    const double jd = E.jd_ref + t;
    if (E.ps_nseg[slot] <= 0) return AG_ERR_NEPHEM;
    if (slot < AG_NPL && !(jd >= E.ps_beg[slot] && jd <= E.ps_end[slot])) return AG_ERR_COVERAGE;   /* NaN too */
    int n = 0;
    if (E.ps_nseg[slot] > 1) {
        n = (int)((jd - E.ps_beg[slot]) / E.ps_res[slot]);
        if (n >= E.ps_nseg[slot]) n = E.ps_nseg[slot] - 1;
        if (n < 0) n = 0;
    }
    const AgSpkSeg sg = E.psegs[E.ps_seg0[slot] + n];
    *X = ag_spk_record(E, sg, E.pmeta, E.pspk, t, z, rate);
    *P = sg.P;
    return AG_OK;
}

/* The raw sums (km; asteroids AU) go where the finished values will stand:
 * Jupiter's in the header, the pair bodies' in rel (EMB in Earth's place,
 * geocentric Moon in the Moon's), the Sun's in F.sun. */
__device__ __forceinline__ double* ag_fast_place(const AgFastView& V, int n, int planet) {
    if (planet == AG_JUP) return V.node(n).rj;
    const int k = planet < AG_JUP ? planet - 1 : planet - 2;
    return V.rel(n) + 3 * k;
}

/* Tables of the nn times tn[0..nn-1] (nn <= 8) by the whole block; ends with
 * a block barrier.  Returns 1 (in every thread) when a time is outside the
 * ephemeris.  srec/ssrc: the record ssrc staged at srec, or null. */
__device__ __forceinline__ int ag_fast_tables(const DevEphem& E, const ForceCfg& c, int nn, const double* tn,
                                              const AgFastView& V, AgFastShared& F, int tid, const double* srec = nullptr,
                                              const double* ssrc = nullptr) {
    const int lane = tid & 31, wid = tid >> 5;
    int bad = 0;
    /* pieces of up to 32 lanes, the longest first, dealt to the warps in turn:
     * planets (a lane a column and time, columns by falling length), the Sun
     * (a lane a component and time), asteroids (a lane a body and time) */
    const int n_pl = (10 * nn + 31) / 32, n_as = (E.n_ast * nn + 31) / 32;
    for (int piece = wid; piece < n_pl + 1 + n_as; piece += AG_FAST_WARPS) {
        if (piece < n_pl) {
            const int q = piece * 32 + lane, col = q / nn, n = q - col * nn;
            if (col < 10) {
                double u[3];
                if (E.pl_spk) {
                    /* planets Mercury .. Pluto without the Earth and Moon, then EMB and Moon */
                    const double* X;
                    int P;
                    double z, rate;
                    const int body = col < 2 ? col + 1 : (col < 8 ? col + 3 : (col == 8 ? AG_EAR : AG_MOO));
                    if (ag_spk_slot(E, body, tn[n], &X, &P, &z, &rate) != AG_OK) bad = 1;
                    else {
                        ag_spk3(X, P, z, u);
                        if (body == AG_EAR || body == AG_MOO) {
                            /* about the Earth-Moon barycentre */
                            double w[3];
                            if (ag_spk_slot(E, AG_NPL, tn[n], &X, &P, &z, &rate) != AG_OK) bad = 1;
                            else {
                                ag_spk3(X, P, z, w);
                                u[0] += w[0]; u[1] += w[1]; u[2] += w[2];
                            }
                        }
                        double* o = ag_fast_place(V, n, body);
                        o[0] = u[0]; o[1] = u[1]; o[2] = u[2];
                    }
                } else {
                    const double* rec;
                    double tf;
                    if (ag_planet_record(E, tn[n], &rec, &tf) != AG_OK) bad = 1;
                    else {
                        const int cs = E.pv.col_sorted[col];
                        if (srec && rec == ssrc) rec = srec;
                        ag_col3(E, rec, cs, tf, u);
                        /* MER VEN EMB MAR JUP SAT URA NEP PLU LUN */
                        const int body = cs < 2 ? cs + 1 : (cs == AG_C_EMB ? AG_EAR : (cs == AG_C_LUN ? AG_MOO : cs + 2));
                        double* o = ag_fast_place(V, n, body);
                        o[0] = u[0]; o[1] = u[1]; o[2] = u[2];
                    }
                }
            }
        } else if (piece == n_pl) {
            const int comp = lane / nn, n = lane - comp * nn;
            if (comp < 3) {
                double v;
                if (E.pl_spk) {
                    const double* X;
                    int P;
                    double z, rate;
                    if (ag_spk_slot(E, AG_SUN, tn[n], &X, &P, &z, &rate) != AG_OK) bad = 1;
                    else {
                        F.sun[n][comp] = ag_spk1v(X + comp * P, P, z, rate, &v);
                        V.node(n).sv[comp] = v * (1.0 / E.au_km);
                    }
                } else {
                    const double* rec;
                    double tf;
                    if (ag_planet_record(E, tn[n], &rec, &tf) != AG_OK) bad = 1;
                    else {
                        if (srec && rec == ssrc) rec = srec;
                        F.sun[n][comp] = ag_col1v(E, rec, AG_C_SUN, comp, tf, &v);
                        V.node(n).sv[comp] = v;
                    }
                }
            }
        } else {
            const int q = (piece - n_pl - 1) * 32 + lane, m = q / nn, n = q - m * nn;
            if (m < E.n_ast) {
                const double t = tn[n], jd = E.jd_ref + t;
                double* o = V.rel(n) + 3 * (AG_PAIR_PL + m);
                if (!(jd >= E.ast_beg[m] && jd <= E.ast_end[m])) {        /* NaN too */
                    bad = 1;
                    o[0] = o[1] = o[2] = 0.0;
                } else {
                    int k = 0;
                    if (E.ast_nseg[m] > 1) {
                        k = (int)((jd - E.ast_beg[m]) / E.ast_res[m]);
                        if (k >= E.ast_nseg[m]) k = E.ast_nseg[m] - 1;
                    }
                    const AgSpkSeg sg = E.segs[E.ast_seg0[m] + k];
                    double z, rate, u[3];
                    const double* X = ag_spk_record(E, sg, E.rec_meta, E.spk, t, &z, &rate);
                    ag_spk3(X, sg.P, z, u);
                    o[0] = u[0]; o[1] = u[1]; o[2] = u[2];
                }
            }
        }
    }
    if (__syncthreads_or(bad)) return 1;
    /* origin minus body in AU, and its float pair */
    const double icau = E.pl_spk ? 1.0 / E.au_km : E.inv_cau;
    const int per = 3 * nn;
    for (int q = tid; q < per * (2 + V.L.bodies); q += AG_FAST_THREADS) {
        const int body = q / per, r = q - body * per, n = r / 3, comp = r - 3 * n;
        AgFastNode& H = V.node(n);
        if (body == 0) {
            const double x = 0.0 - F.sun[n][comp] * icau;
            H.rs[comp] = x;
            H.sp[comp] = ag_f2_of(x);
            H.vf[comp] = ag_d2f_int(H.sv[comp]);
        } else if (body == 1) {
            const double x = 0.0 - H.rj[comp] * icau;
            H.rj[comp] = x;
            H.jf[comp] = ag_d2f_int(x);
        } else {
            const int k = body - 2;
            double* o = V.rel(n) + 3 * k + comp;
            float* pk = reinterpret_cast<float*>(&V.packs(n)[k >> 1].c[comp]) + (k & 1);
            auto put = [](double* d, float* p, double x) {
                const AgF2 f = ag_f2_of(x);
                *d = x;
                p[0] = f.h;
                p[2] = f.l;
            };
            if (k >= AG_PAIR_PL) {
                /* heliocentric, with ASSIST's kilometres per AU */
                put(o, pk, 0.0 - fma(*o, 1.0 / 149597870.7, F.sun[n][comp] * icau));
            } else if (!E.pl_spk && (k == 2 || k == 3)) {
                /* Earth (with the Moon: the two places are pack 1's) */
                if (k == 2) {
                    const double emb = o[0], lun = o[3];
                    float* pm = reinterpret_cast<float*>(&V.packs(n)[1].c[comp]) + 1;
                    float* pe = reinterpret_cast<float*>(&V.packs(n)[1].c[comp]);
                    put(o, pe, 0.0 - fma(lun, E.f_earth, emb) * icau);
                    put(o + 3, pm, 0.0 - fma(lun, E.f_moon, emb) * icau);
                }
            } else {
                put(o, pk, 0.0 - *o * icau);
            }
        }
    }
    if ((V.L.bodies & 1) && tid < 3 * nn) {
        /* the last pack's empty half: massless, far away */
        float* pk = reinterpret_cast<float*>(&V.packs(tid / 3)[V.L.packs - 1].c[tid % 3]) + 1;
        pk[0] = 1e6f;
        pk[2] = 0.0f;
    }
    __syncthreads();
    if ((c.forces & AG_F_EIH) && wid == 4) {
        /* the planets' pull on the Sun and their potential there (1e-3 of the
         * relativistic term's factor: FP32), four lanes a time */
        const int n = lane >> 2;
        float ax = 0.0f, ay = 0.0f, az = 0.0f, u = 0.0f;
        if (n < nn) {
            const AgFastNode& H = V.node(n);
            for (int k = lane & 3; k < 10; k += 4) {
                float d[3], gm;
                if (k == 9) {
                    for (int a = 0; a < 3; a++) d[a] = H.jf[a] - H.sp[a].h;
                    gm = E.pv.gm_jup;
                } else {
                    const float* pk = reinterpret_cast<const float*>(V.packs(n)[k >> 1].c) + (k & 1);
                    for (int a = 0; a < 3; a++) d[a] = pk[4 * a] - H.sp[a].h;
                    gm = (k & 1) ? F.gm[k >> 1].gb : F.gm[k >> 1].ga;
                }
                const float ri = rsqrtf(fmaf(d[0], d[0], fmaf(d[1], d[1], d[2] * d[2]))), gr = gm * ri, f = gr * ri * ri;
                u += gr;
                ax = fmaf(-f, d[0], ax); ay = fmaf(-f, d[1], ay); az = fmaf(-f, d[2], az);
            }
        }
        for (int o = 1; o < 4; o <<= 1) {
            u += __shfl_xor_sync(AG_FULL, u, o);
            ax += __shfl_xor_sync(AG_FULL, ax, o);
            ay += __shfl_xor_sync(AG_FULL, ay, o);
            az += __shfl_xor_sync(AG_FULL, az, o);
        }
        if (n < nn && (lane & 3) == 0) {
            AgFastNode& H = V.node(n);
            H.af[0] = ax; H.af[1] = ay; H.af[2] = az; H.ut = u;
        }
        __syncwarp();
    }
    return 0;
}

/* ------------------------------------------------------------------ terms */

/* Pair operations without the final renormalisation (the low part may grow to
 * a few units of the high part's last place): enough for the relativistic
 * term, which needs about 30 bits. */
__device__ __forceinline__ AgF2 ag_q_mul(AgF2 a, AgF2 b) {
    const float h = __fmul_rn(a.h, b.h);
    return {h, __fmaf_rn(a.l, b.h, __fmaf_rn(a.h, b.l, __fmaf_rn(a.h, b.h, -h)))};
}
__device__ __forceinline__ AgF2 ag_q_add(AgF2 a, AgF2 b) {
    const float s = __fadd_rn(a.h, b.h), bb = __fsub_rn(s, a.h);
    const float e = __fadd_rn(__fsub_rn(a.h, __fsub_rn(s, bb)), __fsub_rn(b.h, bb));
    return {s, __fadd_rn(e, __fadd_rn(a.l, b.l))};
}
__device__ __forceinline__ AgF2 ag_q_dot(const AgF2* a, const AgF2* b) {
    return ag_q_add(ag_q_mul(a[0], b[0]), ag_q_add(ag_q_mul(a[1], b[1]), ag_q_mul(a[2], b[2])));
}

/* The Sun's J2 between 0.1 and 0.5 AU, in float pairs: there it is up to 1.5e-9
 * of the acceleration, and its FP32 form's error was 2.5e-16 rms of it at 0.11
 * AU, as much as the whole FP64 sum's (1.2e-17 at 0.5 AU).  With the pole n,
 * z = d.n, c = z / |d|, k = GM 3/2 J2 R^2 / |d|^5: k ((5 c^2 - 1) d - 2 z n)
 * added to acc; JAC: its Jacobian, k ((5 c^2 - 1) I + 10 z (d n^T + n d^T) /
 * |d|^2 - 2 n n^T - 5 (7 c^2 - 1) d d^T / |d|^2), to j.  Out of line: few
 * particles are there. */
#define AG_SUN_H_FAR2 0.25f
template <bool JAC>
static __device__ __noinline__ void ag_fast_sun_near(const AgPairView& PV, const ForceCfg& c, const AgF2* d, AgF2* acc, AgF2* j) {
    const AgF2 n[3] = {{c.f_sun[0], c.f_sun[3]}, {c.f_sun[1], c.f_sun[4]}, {c.f_sun[2], c.f_sun[5]}};
    const AgF2 r2 = ag_q_dot(d, d), z = ag_q_dot(d, n);
    /* 1/|d|^2 = y^2 (1 - delta), 1/|d|^5 = y^5 (1 - 5/2 delta), delta = r2 y^2 - 1 */
    const float y = rsqrtf(r2.h);
    const AgF2 q = ag_q_mul({y, 0.0f}, {y, 0.0f}), t = ag_q_mul(r2, q);
    const float del = __fadd_rn(__fsub_rn(t.h, 1.0f), t.l);
    const AgF2 r2i = {q.h, __fmaf_rn(-q.h, del, q.l)};
    AgF2 k = ag_q_mul({PV.sk2, PV.sk2_l}, ag_q_mul(ag_q_mul(q, q), {y, 0.0f}));
    k.l = __fmaf_rn(k.h, __fmul_rn(-2.5f, del), k.l);
    const AgF2 zr = ag_q_mul(z, r2i), c2 = ag_q_mul(z, zr);
    const AgF2 f = ag_q_add(ag_q_mul({5.0f, 0.0f}, c2), {-1.0f, 0.0f}), z2 = {-2.0f * z.h, -2.0f * z.l};
    for (int a = 0; a < 3; a++)
        acc[a] = ag_f2_add(acc[a], ag_q_mul(k, ag_q_add(ag_q_mul(f, d[a]), ag_q_mul(z2, n[a]))));
    if (JAC) {
        const AgF2 h = ag_q_mul({10.0f, 0.0f}, zr);
        const AgF2 g = ag_q_mul(r2i, ag_q_add(ag_q_mul({-35.0f, 0.0f}, c2), {5.0f, 0.0f}));
        AgF2 A[3], B[3];
        for (int a = 0; a < 3; a++) {
            A[a] = ag_q_add(ag_q_mul(g, d[a]), ag_q_mul(h, n[a]));
            B[a] = ag_q_add(ag_q_mul(h, d[a]), {-2.0f * n[a].h, -2.0f * n[a].l});
        }
        int at = 0;
        for (int a = 0; a < 3; a++)
            for (int b = a; b < 3; b++, at++) {
                AgF2 s = ag_q_add(ag_q_mul(d[a], A[b]), ag_q_mul(n[a], B[b]));
                if (a == b) s = ag_q_add(s, f);
                j[at] = ag_f2_add(j[at], ag_q_mul(k, s));
            }
    }
}

/* Bodies close to the particle (bit k of near: pair body k0 + k), and the
 * harmonics of a body close by, in FP64 (the Sun's beyond 0.1 AU in pairs).  Out of line: a rare path whose
 * registers the evaluation should not carry. */
static __device__ __noinline__ void ag_fast_close(const DevEphem& E, const ForceCfg& c, const AgFastView* V,
                                                  const AgFastNode* H, int n, int k0, unsigned near, bool earth,
                                                  bool sun, bool eih, const double* x, const double* v, double* a) {
    const double* rel = V->rel(n);
    double ax = 0.0, ay = 0.0, az = 0.0;
    while (near) {
        const int k = k0 + __ffs(near) - 1;
        near &= near - 1;
        const double gm = k < AG_PAIR_PL ? E.gm[ag_pair_planet(k)] : E.ast_gm[k - AG_PAIR_PL];
        const double dx = x[0] + rel[3 * k], dy = x[1] + rel[3 * k + 1], dz = x[2] + rel[3 * k + 2];
        const double ri = rsqrt(fma(dx, dx, fma(dy, dy, dz * dz))), g = gm * ri * ri * ri;
        ax = fma(-g, dx, ax); ay = fma(-g, dy, ay); az = fma(-g, dz, az);
    }
    if (earth) {
        const double dx = x[0] + rel[6], dy = x[1] + rel[7], dz = x[2] + rel[8];
        ag_term_earth_h<false>(E, c, dx, dy, dz, rsqrt(fma(dx, dx, fma(dy, dy, dz * dz))), ax, ay, az, nullptr);
    }
    if (sun) {
        const double dx = x[0] + H->rs[0], dy = x[1] + H->rs[1], dz = x[2] + H->rs[2], r2 = fma(dx, dx, fma(dy, dy, dz * dz));
        if (r2 >= 1.0e-2 && r2 < 1e30) {
            const AgF2 d[3] = {ag_f2_of(dx), ag_f2_of(dy), ag_f2_of(dz)};
            AgF2 o[3] = {{0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}};
            ag_fast_sun_near<false>(E.pv, c, d, o, nullptr);
            ax += ag_f2_to(o[0]); ay += ag_f2_to(o[1]); az += ag_f2_to(o[2]);
        } else {
            ag_term_sun_h<false>(E, c, dx, dy, dz, rsqrt(r2), ax, ay, az, nullptr);
        }
    }
    if (eih) {
        /* relativity far out: ag_fast_eih's formula */
        const double gs = E.gm[AG_SUN], oc2 = E.over_c_squared;
        double af[3] = {0.0, 0.0, 0.0}, ut = 0.0;
        for (int k = -1; k < AG_PAIR_PL; k++) {
            /* the planets' pull on the Sun and their potential there */
            const double* o = k < 0 ? H->rj : rel + 3 * k;
            const double px = o[0] - H->rs[0], py = o[1] - H->rs[1], pz = o[2] - H->rs[2];
            const double ri = rsqrt(fma(px, px, fma(py, py, pz * pz)));
            const double gr = E.gm[k < 0 ? AG_JUP : ag_pair_planet(k)] * ri, f = gr * ri * ri;
            ut += gr;
            af[0] = fma(-f, px, af[0]); af[1] = fma(-f, py, af[1]); af[2] = fma(-f, pz, af[2]);
        }
        double d[3], rel_v[3], up = 0.0, r2 = 0.0, v2 = 0.0, w2 = 0.0, vw = 0.0, dw = 0.0, da = 0.0, f = 0.0;
        for (int k = 0; k < 3; k++) {
            const double w = H->sv[k];
            d[k] = x[k] + H->rs[k];
            rel_v[k] = v[k] - w;
            r2 = fma(d[k], d[k], r2); v2 = fma(v[k], v[k], v2); w2 = fma(w, w, w2); vw = fma(v[k], w, vw);
            dw = fma(d[k], w, dw); da = fma(d[k], af[k], da); f = fma(d[k], 4.0 * v[k] - 3.0 * w, f);
        }
        for (int k = -1; k < AG_PAIR_PL; k++) {
            const double* o = k < 0 ? H->rj : rel + 3 * k;
            const double px = x[0] + o[0], py = x[1] + o[1], pz = x[2] + o[2];
            up = fma(E.gm[k < 0 ? AG_JUP : ag_pair_planet(k)], rsqrt(fma(px, px, fma(py, py, pz * pz))), up);
        }
        const double ri = rsqrt(r2), gr = gs * ri, pre = oc2 * gr * ri * ri;
        const double fac = v2 - 4.0 * (gr + up) - ut + 2.0 * w2 - 4.0 * vw - 1.5 * (dw * ri) * (dw * ri) - 0.5 * da;
        const double ga = 3.5 * oc2 * gr;
        ax += -pre * fac * d[0] + pre * f * rel_v[0] + ga * af[0];
        ay += -pre * fac * d[1] + pre * f * rel_v[1] + ga * af[1];
        az += -pre * fac * d[2] + pre * f * rel_v[2] + ga * af[2];
    }
    a[0] = ax; a[1] = ay; a[2] = az;
}

/* EIH relativity with the Sun as its source (src/forces.c:1288-1983): the
 * Sun's part in float pairs, the planets' and the Sun's motion (1e-3 of it)
 * in FP32.  w: the Sun's velocity; af, ut: the planets' pull on the Sun and
 * their potential there; d: pair separation from the Sun; up: the planets'
 * potential at the particle. */
__device__ __forceinline__ void ag_fast_eih(const AgPairView& PV, const float* w, const float* af, float ut,
                                            const AgF2* d, const AgF2* v, float up, AgF2* out) {
    const AgF2 r2 = ag_q_dot(d, d);
    /* 1/r = y (1 - delta / 2 + 3/8 delta^2), delta = r2 y^2 - 1 */
    const float y = rsqrtf(r2.h);
    const AgF2 q = ag_q_mul({y, 0.0f}, {y, 0.0f}), t = ag_q_mul(r2, q);
    const float del = __fadd_rn(__fsub_rn(t.h, 1.0f), t.l);
    const AgF2 ri = {y, __fmul_rn(y, __fmul_rn(del, fmaf(0.375f, del, -0.5f)))}, ri2 = ag_q_mul(ri, ri);
    const AgF2 gr = ag_q_mul({PV.gm_sun_h, PV.gm_sun_l}, ri), v2 = ag_q_dot(v, v);
    const float w2 = fmaf(w[0], w[0], fmaf(w[1], w[1], w[2] * w[2]));
    const float vw = fmaf(v[0].h, w[0], fmaf(v[1].h, w[1], v[2].h * w[2]));
    const float dw = __fmul_rn(fmaf(d[0].h, w[0], fmaf(d[1].h, w[1], d[2].h * w[2])), ri.h);
    const float da = fmaf(d[0].h, af[0], fmaf(d[1].h, af[1], d[2].h * af[2]));
    const float rest = fmaf(-4.0f, up, fmaf(2.0f, w2, fmaf(-4.0f, vw, fmaf(-1.5f, __fmul_rn(dw, dw), fmaf(-0.5f, da, -ut)))));
    const AgF2 fac = ag_q_add(ag_q_add(v2, {-4.0f * gr.h, -4.0f * gr.l}), {rest, 0.0f});
    AgF2 fv[3], rel[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        fv[k] = ag_q_add({4.0f * v[k].h, 4.0f * v[k].l}, {-3.0f * w[k], 0.0f});
        rel[k] = ag_q_add(v[k], {-w[k], 0.0f});
    }
    const AgF2 pre = ag_q_mul({PV.oc2_h, PV.oc2_l}, ag_q_mul(gr, ri2));
    const AgF2 pf = ag_q_mul(pre, ag_q_dot(d, fv)), pd = ag_f2_neg(ag_q_mul(pre, fac));
    const float ga = 3.5f * PV.oc2_h * gr.h;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const AgF2 o = ag_q_add(ag_q_mul(pd, d[k]), ag_q_mul(pf, rel[k]));
        out[k] = ag_q_add(o, {ga * af[k], 0.0f});
    }
}

/* Relativity with its Jacobian in FP64 (the formulas of ag_term_eih_core for
 * the Sun as the source): d, ri the separation from the Sun, w the Sun's
 * velocity, aj the planets' pull on the Sun, ut their potential there, up and
 * gp their potential and the sum of GM d / r^3 at the particle. */
__device__ __forceinline__ void ag_fast_eih_jac(const DevEphem& E, const double* d, double ri, const double* v, const double* w,
                                               const double* aj, double ut, double up, const double* gp, double* acc,
                                               double (*J)[6]) {
    const double oc2 = E.over_c_squared, gs = E.gm[AG_SUN], r2i = ri * ri, gr = gs * ri, pre = gr * r2i;
    const double vi2 = fma(v[0], v[0], fma(v[1], v[1], v[2] * v[2])), vj2 = fma(w[0], w[0], fma(w[1], w[1], w[2] * w[2]));
    const double vivj = fma(v[0], w[0], fma(v[1], w[1], v[2] * w[2]));
    const double rdvj = fma(d[0], w[0], fma(d[1], w[1], d[2] * w[2]));
    const double rdaj = fma(d[0], aj[0], fma(d[1], aj[1], d[2] * aj[2]));
    const double fac = oc2 * (vi2 - 4.0 * (gr + up) - ut + 2.0 * vj2 - 4.0 * vivj - 1.5 * rdvj * rdvj * r2i - 0.5 * rdaj);
    double fv[3], rel[3];
    for (int k = 0; k < 3; k++) {
        fv[k] = 4.0 * v[k] - 3.0 * w[k];
        rel[k] = v[k] - w[k];
    }
    const double f = fma(d[0], fv[0], fma(d[1], fv[1], d[2] * fv[2]));
    const double pf = pre * fac, pq = oc2 * pre * f, ga = 3.5 * oc2 * gr;
    const double dpre = -3.0 * pre * r2i, t5 = 3.0 * oc2 * rdvj * r2i;
    const double sdu = -dpre * fac, swd = oc2 * dpre * f, swf = oc2 * pre, sy = -ga * r2i, sq = 4.0 * oc2 * pre;
    double u[3], ww[3], y[3], p[3], q[3];
    for (int b = 0; b < 3; b++) {
        acc[b] = fma(-pf, d[b], fma(pq, rel[b], ga * aj[b]));
        /* the factor's derivatives by position and velocity */
        const double dx = 4.0 * oc2 * fma(pre, d[b], gp[b]) - t5 * (w[b] - rdvj * d[b] * r2i) - 0.5 * oc2 * aj[b];
        const double dv = oc2 * (2.0 * v[b] - 4.0 * w[b]);
        u[b] = fma(sdu, d[b], -pre * dx);
        ww[b] = fma(swd, d[b], swf * fv[b]);
        y[b] = sy * d[b];
        p[b] = -pre * dv;
        q[b] = sq * d[b];
    }
    for (int a = 0; a < 3; a++)
        for (int b = 0; b < 3; b++) {
            J[a][b] += fma(d[a], u[b], fma(rel[a], ww[b], aj[a] * y[b])) - (a == b ? pf : 0.0);
            J[a][3 + b] += fma(d[a], p[b], rel[a] * q[b]) + (a == b ? pq : 0.0);
        }
}

/* x + h + l in FP32 for pairs that nearly cancel: the high parts' sum is then
 * exact.  (Of the high parts alone it is off by 6e-8 AU, which close to the
 * Earth was 2e-16 of the acceleration in the harmonics.) */
__device__ __forceinline__ float ag_f2_sep(AgF2 x, float h, float l) { return __fadd_rn(__fadd_rn(x.h, h), __fadd_rn(x.l, l)); }

/* The Earth's J2, J3, J4 in FP32 at separation q (r2 = |q|^2), added to the
 * low parts of the pair sums. */
__device__ __forceinline__ void ag_fast_earth_h(const AgPairView& PV, const ForceCfg& c, const float* q, float r2, AgF2* acc) {
    /* explicit roundings: every build of a kernel computes the same bits */
    const float sa = c.f_pole[0], ca = c.f_pole[1], sd = c.f_pole[2], cd = c.f_pole[3];
    const float cs = __fmul_rn(ca, sd), ss = __fmul_rn(sa, sd), cc = __fmul_rn(ca, cd), sc = __fmul_rn(sa, cd);
    const float p0 = fmaf(-q[0], sa, __fmul_rn(q[1], ca)), p1 = fmaf(-q[0], cs, fmaf(-q[1], ss, __fmul_rn(q[2], cd))),
                p2 = fmaf(q[0], cc, fmaf(q[1], sc, __fmul_rn(q[2], sd)));
    const float ri = rsqrtf(r2), r2i = __fmul_rn(ri, ri), c2 = __fmul_rn(__fmul_rn(p2, p2), r2i),
                r5 = __fmul_rn(__fmul_rn(r2i, r2i), ri);
    const float k2 = __fmul_rn(PV.ek2, r5), k3 = __fmul_rn(PV.ek3, r5), k4 = __fmul_rn(__fmul_rn(PV.ek4, r5), r2i);
    const float f2 = fmaf(5.0f, c2, -1.0f), f3 = fmaf(-7.0f, c2, 3.0f), f4 = fmaf(fmaf(63.0f, c2, -42.0f), c2, 3.0f);
    const float xy = fmaf(k2, f2, fmaf(k4, f4, -__fmul_rn(__fmul_rn(k3, r2i), __fmul_rn(f3, p2))));
    const float o0 = __fmul_rn(xy, p0), o1 = __fmul_rn(xy, p1);
    const float o2 = fmaf(__fmul_rn(k2, f2 - 2.0f), p2,
                          fmaf(-k3, fmaf(fmaf(-7.0f, c2, 6.0f), c2, -0.6f),
                               __fmul_rn(__fmul_rn(k4, fmaf(-28.0f, c2, f4 + 12.0f)), p2)));
    acc[0].l = __fadd_rn(acc[0].l, fmaf(-o0, sa, fmaf(-o1, cs, __fmul_rn(o2, cc))));
    acc[1].l = __fadd_rn(acc[1].l, fmaf(o0, ca, fmaf(-o1, ss, __fmul_rn(o2, sc))));
    acc[2].l = __fadd_rn(acc[2].l, fmaf(o1, cd, __fmul_rn(o2, sd)));
}

/* The Sun's J2, likewise. */
__device__ __forceinline__ void ag_fast_sun_h(const AgPairView& PV, const ForceCfg& c, float qx, float qy, float qz, float r2,
                                              AgF2* acc) {
    const float nx = __fmul_rn(c.f_pole[5], c.f_pole[7]), ny = __fmul_rn(c.f_pole[4], c.f_pole[7]), nz = c.f_pole[6];
    const float z = fmaf(qx, nx, fmaf(qy, ny, __fmul_rn(qz, nz)));
    const float ri = rsqrtf(r2), r2i = __fmul_rn(ri, ri), k2 = __fmul_rn(__fmul_rn(PV.sk2, __fmul_rn(r2i, r2i)), ri);
    const float f2 = fmaf(__fmul_rn(5.0f, z), __fmul_rn(z, r2i), -1.0f), zz = -2.0f * z;
    acc[0].l = fmaf(k2, fmaf(f2, qx, __fmul_rn(zz, nx)), acc[0].l);
    acc[1].l = fmaf(k2, fmaf(f2, qy, __fmul_rn(zz, ny)), acc[1].l);
    acc[2].l = fmaf(k2, fmaf(f2, qz, __fmul_rn(zz, nz)), acc[2].l);
}

/* R^T M R of a symmetric M (pole frame) added to the six elements J. */
__device__ __forceinline__ void ag_fast_rot_sym(const float* pole, const float M[3][3], float* J) {
    const float sa = pole[0], ca = pole[1], sd = pole[2], cd = pole[3];
    const float R[3][3] = {{-sa, ca, 0.0f}, {-ca * sd, -sa * sd, cd}, {ca * cd, sa * cd, sd}};
    int at = 0;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        float v[3];
#pragma unroll
        for (int k = 0; k < 3; k++) v[k] = M[0][k] * R[0][a] + M[1][k] * R[1][a] + M[2][k] * R[2][a];
#pragma unroll
        for (int b = a; b < 3; b++, at++) J[at] += v[0] * R[0][b] + v[1] * R[1][b] + v[2] * R[2][b];
    }
}

/* Jacobians of the harmonics in FP32 (the formulas of ag_term_earth_h and
 * ag_term_sun_h), added to the six elements J. */
__device__ __forceinline__ void ag_fast_earth_hj(const AgPairView& PV, const ForceCfg& c, const float* q, float r2, float* J) {
    const float sa = c.f_pole[0], ca = c.f_pole[1], sd = c.f_pole[2], cd = c.f_pole[3];
    const float p[3] = {-q[0] * sa + q[1] * ca, -q[0] * ca * sd - q[1] * sa * sd + q[2] * cd,
                        q[0] * ca * cd + q[1] * sa * cd + q[2] * sd};
    const float ri = rsqrtf(r2), r2i = ri * ri, c2 = p[2] * p[2] * r2i, r5 = r2i * r2i * ri;
    const float k2 = PV.ek2 * r5, k3 = PV.ek3 * r5, k4 = PV.ek4 * r5 * r2i;
    const float f2 = 5.0f * c2 - 1.0f, f3 = 3.0f - 7.0f * c2, f4 = (63.0f * c2 - 42.0f) * c2 + 3.0f;
    const float g2 = 7.0f * c2 - 1.0f, g3 = (35.0f * c2 - 30.0f) * c2 + 3.0f, ct = p[2] * ri;
    const float h2 = 21.0f * (1.0f - 3.0f * c2) * r2i, h3 = 3.0f * ((-21.0f * c2 + 14.0f) * c2 - 1.0f) * r2i;
    const float h4 = ((-63.0f * c2 + 70.0f) * c2 - 15.0f) * ct * ri;
    const float q2 = (33.0f * c2 - 18.0f) * c2 + 1.0f, q3 = (33.0f * c2 - 30.0f) * c2 + 5.0f;
    const float q4 = ((231.0f * c2 - 315.0f) * c2 + 105.0f) * c2 - 5.0f;
    float M[3][3];
#pragma unroll
    for (int a = 0; a < 2; a++) {
        M[a][a] = k2 * (f2 - 5.0f * g2 * p[a] * p[a] * r2i) + k3 * ct * (h2 * p[a] * p[a] - f3) * ri +
                  k4 * (f4 - 21.0f * q2 * p[a] * p[a] * r2i);
        M[a][2] = M[2][a] = -5.0f * k2 * (g2 - 2.0f) * p[a] * p[2] * r2i + k3 * h3 * p[a] - 21.0f * k4 * q3 * p[a] * p[2] * r2i;
    }
    M[0][1] = M[1][0] = -5.0f * k2 * g2 * p[0] * p[1] * r2i + k3 * h2 * ct * p[0] * p[1] * ri - 21.0f * k4 * q2 * p[0] * p[1] * r2i;
    M[2][2] = -k2 * g3 + k3 * h4 - 3.0f * k4 * q4;
    ag_fast_rot_sym(c.f_pole, M, J);
}
__device__ __forceinline__ void ag_fast_sun_hj(const AgPairView& PV, const ForceCfg& c, const float* q, float r2, float* J) {
    const float sa = c.f_pole[4], ca = c.f_pole[5], sd = c.f_pole[6], cd = c.f_pole[7];
    const float p[3] = {-q[0] * sa + q[1] * ca, -q[0] * ca * sd - q[1] * sa * sd + q[2] * cd,
                        q[0] * ca * cd + q[1] * sa * cd + q[2] * sd};
    const float ri = rsqrtf(r2), r2i = ri * ri, c2 = p[2] * p[2] * r2i, k2 = PV.sk2 * r2i * r2i * ri;
    const float f2 = 5.0f * c2 - 1.0f, g2 = 7.0f * c2 - 1.0f, g3 = (35.0f * c2 - 30.0f) * c2 + 3.0f;
    float M[3][3];
    M[0][0] = k2 * (f2 - 5.0f * g2 * p[0] * p[0] * r2i);
    M[1][1] = k2 * (f2 - 5.0f * g2 * p[1] * p[1] * r2i);
    M[2][2] = -k2 * g3;
    M[0][1] = M[1][0] = -5.0f * k2 * g2 * p[0] * p[1] * r2i;
    M[1][2] = M[2][1] = -5.0f * k2 * (g2 - 2.0f) * p[1] * p[2] * r2i;
    M[0][2] = M[2][0] = -5.0f * k2 * (g2 - 2.0f) * p[0] * p[2] * r2i;
    ag_fast_rot_sym(c.f_pole + 4, M, J);
}

/* The packs [p0, p1) of role w: dealt to roles 5, 6, 7, 2, 3, the remainder
 * to the first of them. */
__device__ __forceinline__ void ag_fast_range(int packs, int w, int& p0, int& p1) {
    const int at = w >= 5 ? w - 5 : w + 1, q = packs / 5, r = packs % 5;
    p0 = w == 4 ? 0 : at * q + min(at, r);
    p1 = w == 4 ? 0 : p0 + q + (at < r ? 1 : 0);
}

/* Role w's share of the evaluation at table n: FP64 partial sums to F.pa
 * (roles 0, 1), float pairs to F.pf and, with near[] set, FP64 sums to F.pn
 * (roles 2..7).  Every lane of the warp calls it; `on` lanes count.  The
 * caller synchronises the block before (states) and after (sums). */
__device__ __forceinline__ void ag_fast_force(int w, int lane, bool on, const DevEphem& E, const ForceCfg& c,
                                              const AgFastView& V, int n, AgFastShared& F, const double* A) {
    const AgFastNode& H = V.node(n);
    if (w < 2) {
        if (!on) return;
        const double x[3] = {F.xs[0][lane], F.xs[1][lane], F.xs[2][lane]};
        const double* o = w == 0 ? H.rj : H.rs;
        const double s[3] = {x[0] + o[0], x[1] + o[1], x[2] + o[2]};
        const double ri = rsqrt(fma(s[0], s[0], fma(s[1], s[1], s[2] * s[2])));
        double ax = 0.0, ay = 0.0, az = 0.0;
        if (w == 1) {
            const bool ng = (c.forces & AG_F_NONGRAV) && A != nullptr && (A[0] != 0.0 || A[1] != 0.0 || A[2] != 0.0);
            if (ng || (c.forces & (AG_F_GR_POT | AG_F_GR_SIMPLE))) {
                const double dv[3] = {F.vs[0][lane] - H.sv[0], F.vs[1][lane] - H.sv[1], F.vs[2][lane] - H.sv[2]};
                if (ng) {
                    double JA[3][3];
                    bool has_ng;
                    ag_term_nongrav<false>(c, s, ri, dv, A, ax, ay, az, nullptr, JA, &has_ng);
                }
                if (c.forces & (AG_F_GR_POT | AG_F_GR_SIMPLE)) {
                    double a[3] = {ax, ay, az};
                    ag_coop_gr_cold(E, c, s, ri, dv, a);
                    ax = a[0]; ay = a[1]; az = a[2];
                }
            }
        }
        const double gm = w == 1 ? E.gm[AG_SUN] : ((c.forces & AG_F_PLANETS) ? E.gm[AG_JUP] : 0.0);
        const double g = gm * ri * ri * ri;
        if (w == 0) {
            F.pa[0][0][lane] = -g * s[0]; F.pa[0][1][lane] = -g * s[1]; F.pa[0][2][lane] = -g * s[2];
        } else {
            /* the Sun's term goes into the last sum unrounded */
            F.gs[lane] = -g;
            F.ss[0][lane] = s[0]; F.ss[1][lane] = s[1]; F.ss[2][lane] = s[2];
            F.pa[1][0][lane] = ax; F.pa[1][1][lane] = ay; F.pa[1][2][lane] = az;
        }
        return;
    }
    const int slot = w - 2;
    const AgF2 xf[3] = {F.xf[0][lane], F.xf[1][lane], F.xf[2][lane]};
    const AgPkRel* R = V.packs(n);
    const float sx = xf[0].h + H.sp[0].h, sy = xf[1].h + H.sp[1].h, sz = xf[2].h + H.sp[2].h;
    const float rs2 = fmaf(sx, sx, fmaf(sy, sy, sz * sz));
    /* beyond 200 AU the planets' pull on the Sun, FP32 in the pair form, is no
     * longer a small part of the relativistic term: that is FP64 there; beyond
     * 1e6 AU, where the products' small parts approach FP32's smallest numbers,
     * every term is */
    const float big = fmaxf(fabsf(xf[0].h), fmaxf(fabsf(xf[1].h), fabsf(xf[2].h)));
    const bool wild = !(big < 1e6f);
    bool eih = false, ce = false, cs = false;
    unsigned near = 0;
    int p0, p1;
    ag_fast_range(V.L.packs, w, p0, p1);
    AgF2 acc[3];
    if (w == 4) {
        acc[0] = acc[1] = acc[2] = {0.0f, 0.0f};
        if (c.forces & AG_F_EIH) {
            eih = !(big < 200.0f);
            /* the planets' potential at the particle */
            float up;
            {
                const float jx = xf[0].h + H.jf[0], jy = xf[1].h + H.jf[1], jz = xf[2].h + H.jf[2];
                up = E.pv.gm_jup * rsqrtf(fmaf(jx, jx, fmaf(jy, jy, jz * jz)));
            }
#pragma unroll
            for (int p = 0; p < (AG_PAIR_PL + 1) / 2; p++) {
                AgPk q[3];
#pragma unroll
                for (int k = 0; k < 3; k++) q[k] = ag_pk_add(R[p].c[k].h, ag_pk(xf[k].h, xf[k].h));
                const AgPk r2 = ag_pk_fma(q[0], q[0], ag_pk_fma(q[1], q[1], ag_pk_mul(q[2], q[2])));
                up = fmaf(F.gm[p].ga, rsqrtf(ag_pk_a(r2)), up);
                if (2 * p + 1 < AG_PAIR_PL) up = fmaf(F.gm[p].gb, rsqrtf(ag_pk_b(r2)), up);
            }
            const AgF2 d[3] = {ag_f2_add(xf[0], H.sp[0]), ag_f2_add(xf[1], H.sp[1]), ag_f2_add(xf[2], H.sp[2])};
            const AgF2 v[3] = {F.vf[0][lane], F.vf[1][lane], F.vf[2][lane]};
            AgF2 e[3];
            ag_fast_eih(E.pv, H.vf, H.af, H.ut, d, v, up, e);
            if (!eih) { acc[0] = e[0]; acc[1] = e[1]; acc[2] = e[2]; }
        }
    } else {
        AgPkSum S;
        AgPk xh[3], xl[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            xh[k] = ag_pk(xf[k].h, xf[k].h);
            xl[k] = ag_pk(xf[k].l, xf[k].l);
            S.h[k] = S.l[k] = ag_pk(0.0f, 0.0f);
        }
#pragma unroll 1
        for (int p = p0; p < p1; p++) near |= ag_pk_term(R[p], F.gm[p], xh, xl, rs2, S) << (2 * (p - p0));
#pragma unroll
        for (int k = 0; k < 3; k++)
            acc[k] = ag_f2_add({ag_pk_a(S.h[k]), ag_pk_a(S.l[k])}, {ag_pk_b(S.h[k]), ag_pk_b(S.l[k])});
        if (w == 3 && (c.forces & AG_F_EARTH_H)) {
            /* J2, J3, J4: below 1.1e-10 of the acceleration beyond 0.02 AU */
            float q[3];
#pragma unroll
            for (int k = 0; k < 3; k++) q[k] = ag_f2_sep(xf[k], ag_pk_a(R[1].c[k].h), ag_pk_a(R[1].c[k].l));
            const float r2 = fmaf(q[0], q[0], fmaf(q[1], q[1], q[2] * q[2]));
            ce = !(r2 >= 4.0e-4f && r2 < 1e30f);
            if (!ce) ag_fast_earth_h(E.pv, c, q, r2, acc);
        }
        if (w == 2 && (c.forces & AG_F_SUN_H)) {
            /* J2: below 6e-11 of the acceleration beyond 0.5 AU */
            cs = !(rs2 >= AG_SUN_H_FAR2 && rs2 < 1e30f);
            if (!cs) ag_fast_sun_h(E.pv, c, sx, sy, sz, rs2, acc);
        }
        if (wild) {
            near = (1u << (2 * (p1 - p0))) - 1u;
#pragma unroll
            for (int k = 0; k < 3; k++) acc[k] = {0.0f, 0.0f};
        }
    }
    const bool mine = on && (near != 0 || ce || cs || eih);
    const bool any = __any_sync(AG_FULL, mine);
    if (any) {
        double a[3] = {0.0, 0.0, 0.0};
        if (mine) {
            /* a body that the configuration leaves out has no mass in the table */
            unsigned m = near;
            for (int p = p0; p < p1; p++) {
                if (ag_pk_a(F.gm[p].h) == 0.0f) m &= ~(1u << (2 * (p - p0)));
                if (ag_pk_b(F.gm[p].h) == 0.0f) m &= ~(2u << (2 * (p - p0)));
            }
            const double x[3] = {F.xs[0][lane], F.xs[1][lane], F.xs[2][lane]};
            const double v[3] = {F.vs[0][lane], F.vs[1][lane], F.vs[2][lane]};
            ag_fast_close(E, c, &V, &H, n, 2 * p0, m, ce, cs, eih, x, v, a);
        }
        F.pn[slot][0][lane] = a[0]; F.pn[slot][1][lane] = a[1]; F.pn[slot][2][lane] = a[2];
    }
    if (lane == 0) F.near[slot] = any ? 1 : 0;
    if (on) { F.pf[slot][0][lane] = acc[0]; F.pf[slot][1][lane] = acc[1]; F.pf[slot][2][lane] = acc[2]; }
}

/* Component k of the acceleration of lane l's particle, after the block has met. */
__device__ __forceinline__ double ag_fast_sum(const AgFastShared& F, int k, int lane) {
    const AgF2 s = ag_f2_add(ag_f2_add(ag_f2_add(F.pf[0][k][lane], F.pf[1][k][lane]), F.pf[2][k][lane]),
                             ag_f2_add(F.pf[3][k][lane], ag_f2_add(F.pf[4][k][lane], F.pf[5][k][lane])));
    double a = (ag_f2_to(s) + F.pa[0][k][lane]) + F.pa[1][k][lane];
    int any = 0;
#pragma unroll
    for (int w = 0; w < AG_FAST_SLOTS; w++) any |= F.near[w];
    if (any)
        for (int w = 0; w < AG_FAST_SLOTS; w++)
            if (F.near[w]) a += F.pn[w][k][lane];
    return fma(F.gs[lane], F.ss[k][lane], a);
}

#endif
