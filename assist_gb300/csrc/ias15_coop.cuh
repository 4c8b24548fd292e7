/*
 * ias15_coop.cuh -- block-cooperative grouped batched IAS15 (included by
 * kernels_coop.cu).
 *
 * A group of up to 32 particles that share their step times (the same
 * grouping as the warp-grouped kernel) is integrated by one 128-thread block:
 * lane l of every warp works on particle l, and the four warps split the
 * work of each force evaluation so that it runs on all four SM sub-partitions
 * (each has its own FP64 pipe):
 *
 *   warp 0  planets' direct gravity (ASSIST's order, Sun last), Marsden
 *           non-gravitational term, Earth J2-J4, geocentric indirect term
 *   warp 1  EIH/PPN relativity (its per-source sums too), GR potential/simple
 *   warp 2  first half of the asteroids
 *   warp 3  second half of the asteroids, Sun J2
 * (with variational particles, whose Jacobians fill warp 0's registers,
 * Earth J2-J4 stays on warp 2).  Batches are grouped so that particles with
 * non-gravitational parameters share groups: a group whose members have none
 * skips warp 0's costliest term.
 * Warps 0 and 1 both need the eleven particle-planet separations: each forms
 * half and they exchange them through shared memory at a named barrier
 * (without Jacobians; with them each warp forms all eleven).
 *
 * With variational particles the forces are on pair terms where those apply
 * (PAIRS, ag_coop_force_pairs), and a group of up to sixteen may put each
 * particle on two lanes that share its components (HALF).
 *
 * The partial accelerations (and partial Jacobians) meet in shared memory and
 * are summed in a fixed order ((w3 + w2) + w1) + w0, so the planets' terms,
 * the largest, come last as in ASSIST's sum.  The body table of each
 * substep time is built by the whole block, once a step: column components of
 * the .440 record and asteroid components of the SPK records on different
 * threads, with fused multiply-adds.  Each IAS15 state component has an owner
 * warp that predicts it, forms its acceleration from the partials and
 * updates its g, b and e: x, y, z belong to warps 0, 2, 3 (warps 1, 2, 3
 * with variational particles); the three
 * components of a variational particle share one warp (its J.dx product reads
 * only its own predicted values).
 * Per-particle control values (t, dt, convergence, retirement) are computed
 * identically by all four warps from shared data, so every branch around a
 * block barrier is uniform.
 *
 * Per evaluation this cuts the FP64 instructions on one sub-partition to
 * roughly a third of the warp-grouped kernel's, which is what bounds the
 * longest groups (the tail of a batch).
 *
 * Memory: without variational particles the block keeps the eight node
 * tables of a step (the node times do not change while the predictor-
 * corrector iterates, so each table is built once per step), each with the
 * origin-minus-body half of every separation formed once, and the group's
 * IAS15 state (40 fields x 3 components x 32 lanes) in dynamic shared
 * memory.  The plain kernel is built for two resident blocks per SM (236
 * registers) and for three (168); the host picks three only for batches
 * with many groups per block.
 */

#include "coop_forces.cuh"
#include "fast_forces.cuh"
#include "ias15_warm.cuh"

/* b, e of one component from the last accepted step's br, er (the shift of
 * the acceleration polynomial to the new step). */
template <class WsT>
__device__ __forceinline__ void ag_predict_next_comp(const WsT& W, int comp, double ratio) {
    if (ratio > 20.0) {
        for (int k = 0; k < 7; k++) { W(W_E + k, comp) = 0.0; W(W_B + k, comp) = 0.0; }
        return;
    }
    double q[8];
    q[1] = ratio;
    for (int k = 2; k < 8; k++) q[k] = q[k - 1] * ratio;
    constexpr double binom[8][8] = {
        {1, 0, 0, 0, 0, 0, 0, 0}, {1, 1, 0, 0, 0, 0, 0, 0}, {1, 2, 1, 0, 0, 0, 0, 0}, {1, 3, 3, 1, 0, 0, 0, 0},
        {1, 4, 6, 4, 1, 0, 0, 0}, {1, 5, 10, 10, 5, 1, 0, 0}, {1, 6, 15, 20, 15, 6, 1, 0}, {1, 7, 21, 35, 35, 21, 7, 1}};
    double br[7], er[7];
#pragma unroll
    for (int k = 0; k < 7; k++) { br[k] = W(W_BR + k, comp); er[k] = W(W_ER + k, comp); }
#pragma unroll
    for (int j = 0; j < 7; j++) {
        double s = 0.0;
#pragma unroll
        for (int k = 6; k >= j; k--) s = fma(br[k], binom[k + 1][j + 1], s);
        const double e = q[j + 1] * s;
        W(W_E + j, comp) = e;
        W(W_B + j, comp) = e + (br[j] - er[j]);
    }
}

/* Owner warp of IAS15 component comp: x, y, z -> warps 0, 2, 3 (warps
 * 1..3 with variational particles, which go to warps 0, 0, 1, 2, 3, 1). */
template <int NV>
__device__ __forceinline__ int ag_coop_owner(int comp) {
    if (comp < 3) return NV == 0 ? (comp == 0 ? 0 : comp + 1) : comp + 1;
    const int q = (comp - 3) / 3;
    return q < 2 ? 0 : ((q == 2 || q == 5) ? 1 : (q == 3 ? 2 : 3));
}

/* Position component owned by warp w (-1: none). */
template <int NV>
__device__ __forceinline__ int ag_coop_pcomp(int w) {
    return NV == 0 ? (w == 0 ? 0 : (w == 1 ? -1 : w - 1)) : w - 1;
}

/* Component ci of a warp, or -1.  HALF: a group of up to 16 particles, each
 * on two lanes that share its components, two of them to an instruction: x, y
 * and z on warps 1, 1 (other half) and 2, a variational particle's three on one
 * warp. */
template <int NV, bool HALF>
__device__ __forceinline__ int ag_coop_comp(int ci, int wid, int half) {
    if (!HALF) return ag_coop_owner<NV>(ci) == wid ? ci : -1;
    const int k = 2 * ci + half;                    /* of warp 0: 3..8, 3: 9..14, 1: 0 1 15 16 17, 2: 2 18 19 20 */
    if (wid == 0) return 3 + k;
    if (wid == 3) return 9 + k;
    if (wid == 1) return k < 2 ? k : (k < 5 ? 13 + k : -1);
    return k == 0 ? 2 : (k < 4 ? 17 + k : -1);
}

/* IAS15's fields of a block: the fields below W_E (the state, its
 * compensations, a0, b and g, used at every node) in shared memory, the others
 * (used once a step) in the global workspace. */
template <int C, int LANES>
struct WsSplit {
    double *s, *w;
    int ns, slot;
    __device__ __forceinline__ double& operator()(int f, int comp) const {
        return f < W_E ? s[(f * C + comp) * LANES] : w[((size_t)f * C + comp) * ns + slot];
    }
};

template <int NV, bool DYN_TABS = false>
struct AgCoopShared {
    static constexpr int C = 3 * (1 + NV);
    typename std::conditional<DYN_TABS, char, AgCoopTab[NV == 0 ? 8 : 1]>::type tab;
                                    /* body tables, one per node, kept through the predictor-corrector
                                       iterations of a step (the node times do not change while it
                                       iterates); with variational particles in dynamic shared memory
                                       (learned start: a single one, built anew) */
    AgCoopScratch scr;
    double xs[C][32], vs[C][32];                    /* state at the current node */
    double pa[4][3][32];                            /* partial accelerations */
    typename std::conditional<NV == 0, AgCoopSeps, char>::type seps;   /* warp 0 <-> warp 1 separations */
    double pj[NV > 0 ? 4 : 1][NV > 0 ? 18 : 1][32]; /* partial Jacobians */
    double ra[3][32], rdb[3][32];                   /* |a|, |delta b6| of x, y, z at node 7 */
    double rb6[3][32];                              /* |b6| of x, y, z after convergence */
    double pcx[8][9], pcv[8][8];                    /* predictor coefficients of nodes 1..7 of the step */
    double ptn[8];                                  /* and the node times */
    AgF2 xsf[NV == 0 ? 3 : 1][32];                  /* the state's position as float pairs (asteroid terms) */
    double sdn[32], sdc[32];                        /* each lane's next-step proposal, capped and uncapped */
    int srej[32];                                   /* and whether it rejects the step */
    int fin[3][32];
    int g, stop;
    int stage_fail;                                 /* a staged record copy did not complete */
    int wg_off;                                     /* learned warm start switched off for this group */
    int rot;                                        /* role rotation of this block */
};

/* The warps' parts of the Jacobian summed once, in S.pj[0] (each of the 18
 * variational components had summed its row: 324 FP64 instructions a node in
 * place of 54).  Ends with a block barrier. */
template <class Sh>
__device__ __forceinline__ void ag_coop_sum_jac(Sh& S, int wid, int lane, bool on) {
    if (on)
        for (int q = wid; q < 18; q += 4)
            S.pj[0][q][lane] = ((S.pj[3][q][lane] + S.pj[2][q][lane]) + S.pj[1][q][lane]) + S.pj[0][q][lane];
    __syncthreads();
}

/* Float pairs of a table's origin minus body: the pair terms' planets, then
 * the Sun and Jupiter (the asteroids' are in the table). */
#define AG_PREL (AG_PAIR_PL + 2)
typedef AgF2 AgPairRow[3];
__device__ __forceinline__ void ag_coop_pair_rows(const AgCoopTab& CT, AgPairRow* PR, int tid) {
    if (tid < 3 * AG_PREL) {
        const int k = tid / 3, comp = tid - 3 * k;
        PR[k][comp] = ag_f2_of(CT.rel[k < AG_PAIR_PL ? ag_pair_planet(k) : (k == AG_PAIR_PL ? AG_SUN : AG_JUP)][comp]);
    }
}

/* Warp w's share of the evaluation with Jacobian on pair terms (the bodies,
 * thresholds and precisions of fast_forces.cuh, every direct term on):
 *
 *   warp 0      Sun and Jupiter, non-gravitational terms (FP64), a third of the packs
 *   warp 1      relativity (FP64, with FP32 sums over the planets), GR terms
 *   warps 2, 3  a third of the packs each, the Earth's and the Sun's harmonics (FP32)
 *
 * It replaces ag_coop_force_part<true>, whose busiest warp has some 450 FP64
 * instructions a node; here 200 (warp 1). */
__device__ __forceinline__ void ag_coop_force_pairs(int w, const AgCoopTab& CT, const AgPairRow* PR, const DevEphem& E, const ForceCfg& c,
                                                    const double* x, const double* v, const double* A, double* acc, double (*J)[6]) {
#pragma unroll
    for (int q = 0; q < 18; q++) J[q / 6][q % 6] = 0.0;
    acc[0] = acc[1] = acc[2] = 0.0;
    const AgF2 xf[3] = {ag_f2_of(x[0]), ag_f2_of(x[1]), ag_f2_of(x[2])};
    if (w == 1) {
        double d[3], ri;
        ag_coop_sep(CT, x, AG_SUN, d[0], d[1], d[2], ri);
        const PlanetState& P = CT.T.P;
        const double sv[3] = {P.vx[AG_SUN], P.vy[AG_SUN], P.vz[AG_SUN]};
        if (c.forces & AG_F_EIH) {
            float up = 0.0f, gp[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll 1
            for (int k = 0; k < AG_PAIR_PL + 1; k++) {
                const AgPairRow& o = PR[k < AG_PAIR_PL ? k : AG_PAIR_PL + 1];
                const float gm = k < AG_PAIR_PL ? ((k & 1) ? E.pv.gm[k >> 1].gb : E.pv.gm[k >> 1].ga) : E.pv.gm_jup;
                const float q[3] = {o[0].h + xf[0].h, o[1].h + xf[1].h, o[2].h + xf[2].h};
                const float r = rsqrtf(fmaf(q[0], q[0], fmaf(q[1], q[1], q[2] * q[2]))), f = gm * r * r * r;
                up = fmaf(gm, r, up);
                for (int m = 0; m < 3; m++) gp[m] = fmaf(f, q[m], gp[m]);
            }
            const double g[3] = {ag_f2d_int(gp[0]), ag_f2d_int(gp[1]), ag_f2d_int(gp[2])};
            ag_fast_eih_jac(E, d, ri, v, sv, CT.T.eih_a[AG_SUN], CT.T.eih_t1[AG_SUN], ag_f2d_int(up), g, acc, J);
        }
        if (c.forces & AG_F_GR_POT) ag_term_gr_pot<true>(E, d, ri, acc[0], acc[1], acc[2], J);
        if (c.forces & AG_F_GR_SIMPLE) {
            const double pv[3] = {v[0] - sv[0], v[1] - sv[1], v[2] - sv[2]};
            ag_term_gr_simple<true>(E, d, ri, pv, acc[0], acc[1], acc[2], J);
        }
        return;
    }
    const AgPairRow& sun = PR[AG_PAIR_PL];
    const float big = fmaxf(fabsf(xf[0].h), fmaxf(fabsf(xf[1].h), fabsf(xf[2].h)));
    const bool wild = !(big < 1e6f);
    const float sx = xf[0].h + sun[0].h, sy = xf[1].h + sun[1].h, sz = xf[2].h + sun[2].h;
    const float rs2 = fmaf(sx, sx, fmaf(sy, sy, sz * sz));
    const int bodies = AG_PAIR_PL + E.n_ast, packs = (bodies + 1) / 2, slot = w == 0 ? 0 : w - 1;
    AgPkSum S;
    AgPkJac PJ;
    AgPk xh[3], xl[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        xh[k] = ag_pk(xf[k].h, xf[k].h);
        xl[k] = ag_pk(xf[k].l, xf[k].l);
        S.h[k] = S.l[k] = ag_pk(0.0f, 0.0f);
    }
    ag_pk_jac_clear(PJ);
    unsigned long long near = 0;
#pragma unroll 1
    for (int p = slot; p < packs; p += 3) {
        const int ka = 2 * p, kb = 2 * p + 1;
        const AgF2* a = ka < AG_PAIR_PL ? PR[ka] : CT.arel[ka - AG_PAIR_PL];
        const bool two = kb < bodies;
        const AgF2* b = !two ? a : (kb < AG_PAIR_PL ? PR[kb] : CT.arel[kb - AG_PAIR_PL]);
        AgPkRel R;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            /* the last pack's empty half: massless, far away */
            R.c[k].h = ag_pk(a[k].h, two ? b[k].h : 1e6f);
            R.c[k].l = ag_pk(a[k].l, two ? b[k].l : 0.0f);
        }
        AgPkGm G = E.pv.gm[p];
        G.ta = E.pv.jac_thr[ka];
        G.tb = E.pv.jac_thr[kb];
        const unsigned n = ag_pk_term<true>(R, G, xh, xl, rs2, S, &PJ);
        near |= (unsigned long long)(two ? n : n & 1u) << ka;
    }
    AgF2 s[3], j[7];
#pragma unroll
    for (int k = 0; k < 3; k++)
        s[k] = ag_f2_add({ag_pk_a(S.h[k]), ag_pk_a(S.l[k])}, {ag_pk_b(S.h[k]), ag_pk_b(S.l[k])});
#pragma unroll
    for (int k = 0; k < 7; k++) {
        AgF2 a, b;
        ag_pk_jac_get(PJ, k, 0, a.h, a.l);
        ag_pk_jac_get(PJ, k, 1, b.h, b.l);
        j[k] = ag_f2_add(a, b);
    }
    bool earth = false, sunh = false;          /* harmonics left to FP64 */
    if (w == 2 && (c.forces & AG_F_EARTH_H)) {
        float hj[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        float q[3];
#pragma unroll
        for (int k = 0; k < 3; k++) q[k] = ag_f2_sep(xf[k], PR[2][k].h, PR[2][k].l);
        const float r2 = fmaf(q[0], q[0], fmaf(q[1], q[1], q[2] * q[2]));
        earth = wild || !(r2 >= 1.0e-2f && r2 < 1e30f);
        if (!earth) {
            ag_fast_earth_h(E.pv, c, q, r2, s);
            ag_fast_earth_hj(E.pv, c, q, r2, hj);
#pragma unroll
            for (int k = 0; k < 6; k++) j[k].l += hj[k];
        }
    }
    if (w == 3 && (c.forces & AG_F_SUN_H)) {
        float hj[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        sunh = wild || !(rs2 >= 1.0e-2f && rs2 < 1e30f);
        if (!sunh && rs2 < AG_SUN_H_FAR2) {
            const AgF2 d[3] = {ag_q_add(xf[0], sun[0]), ag_q_add(xf[1], sun[1]), ag_q_add(xf[2], sun[2])};
            ag_fast_sun_near<true>(E.pv, c, d, s, j);
        } else if (!sunh) {
            const float q[3] = {sx, sy, sz};
            ag_fast_sun_h(E.pv, c, sx, sy, sz, rs2, s);
            ag_fast_sun_hj(E.pv, c, q, rs2, hj);
#pragma unroll
            for (int k = 0; k < 6; k++) j[k].l += hj[k];
        }
    }
    AgSymJac Y = {{0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, 0.0};
    double ax = 0.0, ay = 0.0, az = 0.0;
    if (wild) {
        near = 0;
        for (int p = slot; p < packs; p += 3) near |= (2 * p + 1 < bodies ? 3ull : 1ull) << (2 * p);
    } else {
        ax = ag_f2_to(s[0]); ay = ag_f2_to(s[1]); az = ag_f2_to(s[2]);
#pragma unroll
        for (int a = 0, e = 0; a < 3; a++)
#pragma unroll
            for (int b = a; b < 3; b++, e++) {
                const double t = ag_f2_to(j[e]);
                J[a][b] = t;
                if (b != a) J[b][a] = t;
            }
        const double g = ag_f2_to(j[6]);
        J[0][0] -= g; J[1][1] -= g; J[2][2] -= g;
    }
    while (near) {
        const int k = __ffsll((long long)near) - 1;
        near &= near - 1;
        double r[3];
        if (k < AG_PAIR_PL) {
            const double* o = CT.rel[ag_pair_planet(k)];
            r[0] = o[0]; r[1] = o[1]; r[2] = o[2];
        } else ag_coop_ast_rel(CT, false, k - AG_PAIR_PL, r);
        const double gm = k < AG_PAIR_PL ? E.gm[ag_pair_planet(k)] : E.ast_gm[k - AG_PAIR_PL];
        const double dx = x[0] + r[0], dy = x[1] + r[1], dz = x[2] + r[2];
        const double ri = rsqrt(fma(dx, dx, fma(dy, dy, dz * dz))), g = gm * ri * ri * ri;
        ax = fma(-g, dx, ax); ay = fma(-g, dy, ay); az = fma(-g, dz, az);
        ag_symjac_term(Y, g, ri, dx, dy, dz);
    }
    if (earth) {
        double dx, dy, dz, ri;
        ag_coop_sep(CT, x, AG_EAR, dx, dy, dz, ri);
        ag_term_earth_h<true>(E, c, dx, dy, dz, ri, ax, ay, az, J);
    }
    if (sunh) {
        double dx, dy, dz, ri;
        ag_coop_sep(CT, x, AG_SUN, dx, dy, dz, ri);
        ag_term_sun_h<true>(E, c, dx, dy, dz, ri, ax, ay, az, J);
    }
    if (w == 0) {
        double d[3], ri;
        ag_coop_sep(CT, x, AG_SUN, d[0], d[1], d[2], ri);
        if ((c.forces & AG_F_NONGRAV) && A != nullptr && (A[0] != 0.0 || A[1] != 0.0 || A[2] != 0.0)) {
            const PlanetState& P = CT.T.P;
            const double dv[3] = {v[0] - P.vx[AG_SUN], v[1] - P.vy[AG_SUN], v[2] - P.vz[AG_SUN]};
            double JA[3][3];
            bool has_ng;
            ag_term_nongrav<true>(c, d, ri, dv, A, ax, ay, az, J, JA, &has_ng);
        }
        double jx, jy, jz, rj;
        ag_coop_sep(CT, x, AG_JUP, jx, jy, jz, rj);
        const double gj = E.gm[AG_JUP] * rj * rj * rj, gs = E.gm[AG_SUN] * ri * ri * ri;
        ax = fma(-gj, jx, ax); ay = fma(-gj, jy, ay); az = fma(-gj, jz, az);
        ag_symjac_term(Y, gj, rj, jx, jy, jz);
        ax = fma(-gs, d[0], ax); ay = fma(-gs, d[1], ay); az = fma(-gs, d[2], az);
        ag_symjac_term(Y, gs, ri, d[0], d[1], d[2]);
    }
    ag_symjac_add(Y, J);
    acc[0] = ax; acc[1] = ay; acc[2] = az;
}

/* Distance from (x, y, z) to the nearest of the eleven planets in the table. */
struct AgTableNearest {
    const AgTable& T;
    __device__ __forceinline__ double operator()(double x, double y, double z) const {
        double m = 1e300;
#pragma unroll
        for (int k = 0; k < AG_NPL; k++) {
            const double dx = x - T.P.x[k], dy = y - T.P.y[k], dz = z - T.P.z[k];
            m = fmin(m, fma(dx, dx, fma(dy, dy, dz * dz)));
        }
        return sqrt(m);
    }
};

/* Dynamic shared memory of a block: the warm-start buffers (when present);
 * or, in the plain kernel without variational particles, the group's IAS15
 * state (40 fields x 3 components x 32 lanes, 30 KB); or, with them, the
 * eight body tables with the planets' float pairs and, in the build for one block a multiprocessor, the
 * state's fields below W_E (19 x 21 x 32, 102 KB; with HALF, for two blocks,
 * half of that).  What is not there stays in
 * the global workspace, indexed by slot. */
template <int NV, bool WARM, bool STAGE = false, int OCC = 2, bool HALF = false>
struct AgCoopDyn {
    static constexpr bool ws_shared = NV == 0 && !WARM;
    static constexpr bool ws_split = NV > 0 && !WARM && (OCC == 1 || HALF);
    static constexpr bool tabs = NV > 0 && !WARM;
    static constexpr size_t warm = WARM ? (sizeof(AgWarmSmem) + 15) / 16 * 16 : 0;
    static constexpr size_t ws = ws_shared ? sizeof(double) * W_NF * 3 * 32
                                           : (ws_split ? sizeof(double) * W_E * 3 * (1 + NV) * (HALF ? 16 : 32) : 0);
    static constexpr size_t stage_off = warm + ws;        /* the staged .440 record (STAGE) */
    static constexpr size_t stage = STAGE ? (sizeof(AgRecStage) + 15) / 16 * 16 : 0;
    static constexpr size_t tab_off = stage_off + stage;
    static constexpr size_t prel_off = tab_off + (tabs ? 8 * sizeof(AgCoopTab) : 0);
    static constexpr size_t bytes = prel_off + (tabs ? 8 * AG_PREL * sizeof(AgPairRow) : 0);
};

/* OCC: resident blocks per SM the kernel is compiled for.  The plain kernel
 * comes in three builds: 2 (242 registers), 3 (168 registers, a few
 * spills: faster on batches with many groups per block, slower on small
 * batches whose longest groups set the time), and 2 with the active .440
 * record staged in shared memory by bulk copies (STAGE; its 8 KB buffer does
 * not fit beside three blocks); the warm-start instantiations have only 2
 * (their network buffers would not fit).  The variational kernel comes in 1
 * and 2: a block alone keeps the state in shared memory.  It is bound by the
 * FP64 pipes' latency, about 2,500 FP64 warp instructions a block and node
 * (3,200 with a table and the 18 components' Jacobian sums at every node):
 * 2,053 mixed particles over 730 days 268.6 ms before, 218.1 so.  PAIRS: the
 * forces on pair terms, 1,300 a node, 168.2 ms.  HALF: a particle on two
 * lanes, 800 a node and 115 KB a block: 98.4 ms. */
template <int NV, bool WARM, int OCC = 2, bool STAGE = false, bool PAIRS = false, bool HALF = false>
__global__ void __launch_bounds__(128, OCC) ag_k_coop(const DevEphem* __restrict__ Ep, ForceCfg cf, AgBatchArgs A) {
    constexpr int C = 3 * (1 + NV);
    const DevEphem& E = *Ep;
    __shared__ AgCoopShared<NV, (NV > 0 && !WARM)> S;
    /* Role rotation: warp w of a block runs on sub-partition w % 4 of its SM,
     * and the four roles (planets / relativity / asteroids / asteroids and
     * Sun J2) do unequal FP64 work.  Blocks sharing an SM take successive
     * rotations (a per-SM counter) so that each sub-partition's FP64 pipe
     * serves a mix of roles; within a block everything below uses the
     * logical warp index wid and thread index tid. */
    if (threadIdx.x == 0) {
        int r = 0;
        if (A.sm_slots) {
            unsigned smid;
            asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
            r = atomicAdd(&A.sm_slots[smid & (AG_SM_SLOTS - 1)], 1) & 3;
        }
        S.rot = r;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = ((threadIdx.x >> 5) + S.rot) & 3, tid = (wid << 5) | lane;
    /* the lane's particle in the group, and which of the particle's lanes it is */
    const int pl = HALF ? lane & 15 : lane, half = HALF ? lane >> 4 : 0;
    constexpr int n_ci = HALF ? 3 : C;
    const int slot = blockIdx.x * 32 + pl;
    extern __shared__ __align__(16) unsigned char ag_dyn_smem[];
    using Dyn = AgCoopDyn<NV, WARM, STAGE, OCC, HALF>;
    constexpr bool tab8 = NV == 0 || Dyn::tabs;
    AgCoopTab* tabs;
    if constexpr (Dyn::tabs) tabs = reinterpret_cast<AgCoopTab*>(ag_dyn_smem + Dyn::tab_off);
    else tabs = S.tab;
    AgCoopTab& Tab = tabs[0];
    AgPairRow* const prel = PAIRS ? reinterpret_cast<AgPairRow*>(ag_dyn_smem + Dyn::prel_off) : nullptr;
    AgRecStage* const R =
        STAGE ? reinterpret_cast<AgRecStage*>(ag_dyn_smem + Dyn::stage_off) : nullptr;
    AgStageCursor cur;
    constexpr bool wss = Dyn::ws_shared;
    typename std::conditional<Dyn::ws_split, WsSplit<C, HALF ? 16 : 32>, Ws<C>>::type W;
    if constexpr (Dyn::ws_split) W.s = reinterpret_cast<double*>(ag_dyn_smem) + pl;
    W.w = wss ? reinterpret_cast<double*>(ag_dyn_smem + Dyn::warm) : A.ws;
    W.ns = wss ? 32 : A.nslots;
    W.slot = wss ? lane : slot;
    const long long clk0 = clock64();
    unsigned long long n_acc = 0, n_rej = 0, n_ev = 0, n_it = 0, n_wused = 0, n_wfall = 0, n_tab = 0;
    if (tid == 0) {
        for (int k = 0; k < (tab8 ? 8 : 1); k++) tabs[k].T.status = AG_OK;
        S.stop = 0;
        S.stage_fail = 0;
        if (STAGE) ag_mbar_init(&R->bar);
    }
    /* learned warm start and step logging */
    AgWarmSmem& WS = *reinterpret_cast<AgWarmSmem*>(ag_dyn_smem);
    const bool warm = WARM && A.mlp != nullptr;
    const bool logp = WARM && A.log_x != nullptr;

    while (true) {
        __syncthreads();
        if (tid == 0) S.g = atomicAdd(A.queue, 1);
        __syncthreads();
        const int g = S.g;
        if (g >= A.n_groups) break;
        const int gs = A.grp_size[g], g0 = A.grp_start[g];
        if (S.stop || S.stage_fail) {
            /* run-time budget spent (or a record copy lost): groups still
             * queued are not integrated (state untouched) and say so */
            if (wid == 0 && lane < gs) {
                const int p = A.order[g0 + lane];
                if (A.status) A.status[p] = AG_ST_TIMEOUT;
                if (NV == 0 && A.out_start != nullptr)
                    for (int q = A.out_start[p]; q < A.out_start[p + 1]; q++)
                        for (int k = 0; k < 6; k++) A.out_state[6 * (size_t)q + k] = __longlong_as_double(0x7ff8000000000000LL);
            }
            continue;
        }
        const int pid = pl < gs ? A.order[g0 + pl] : -1;
        double t = A.t0[A.order[g0]], tc = 0.0, dtls = 0.0;
        const double tend = pid >= 0 ? A.t_end[pid] : t;
        double dir;
        {
            const double d = pid >= 0 ? (tend - t) : 0.0;
            const unsigned fwd = __ballot_sync(AG_FULL, d > 0.0), bwd = __ballot_sync(AG_FULL, d < 0.0);
            dir = fwd ? 1.0 : (bwd ? -1.0 : 1.0);
        }
        double dt = dir * fabs(A.dt0);
        double prm[3] = {0.0, 0.0, 0.0};
        bool has_prm = false;
        int pstat = AG_ST_OK;
        bool live = pid >= 0;
        if (live) {
            const double* s0 = A.state + 6 * (size_t)pid;
            for (int ci = 0; ci < n_ci; ci++) {
                    const int comp = ag_coop_comp<NV, HALF>(ci, wid, half);
                    if (comp < 0) continue;
                double x0, v0;
                if (comp < 3) { x0 = s0[comp]; v0 = s0[3 + comp]; }
                else {
                    const double* vs = A.var_state + ((size_t)pid * NV + (comp - 3) / 3) * 6;
                    x0 = vs[(comp - 3) % 3]; v0 = vs[3 + (comp - 3) % 3];
                }
                W(W_X0, comp) = x0; W(W_V0, comp) = v0; W(W_XC, comp) = 0.0; W(W_VC, comp) = 0.0;
                for (int k = 0; k < 7; k++) {
                    W(W_B + k, comp) = 0.0; W(W_E + k, comp) = 0.0; W(W_BR + k, comp) = 0.0; W(W_ER + k, comp) = 0.0;
                }
            }
            if (A.params) {
                prm[0] = A.params[3 * (size_t)pid]; prm[1] = A.params[3 * (size_t)pid + 1]; prm[2] = A.params[3 * (size_t)pid + 2];
                has_prm = true;
            }
        }
        bool finish_now = live && (tend == t);
        long long steps = 0;
        /* dense output cursor (times sorted along the integration) */
        const bool dense = NV == 0 && A.out_start != nullptr;
        int on = 0, on_end = 0;
        if (dense && live) { on = A.out_start[pid]; on_end = A.out_start[pid + 1]; }
        /* warm start per group: on until its learned steps take longer than
         * its plain probes (every 8th step), timed by thread 0 with clock64
         * from the step's first body table to its converged corrector: the
         * inference's cost against the iterations it saves, where the group
         * iterates until its slowest member has converged */
        long long wg_t_l = 0, wg_t_p = 0, clk_step = 0;
        int wg_n_l = 0, wg_n_p = 0;
        if (tid == 0) S.wg_off = 0;
        /* and per member: on until its learned starts converge in more
         * iterations than its plain probes */
        bool wl_on = warm;
        int wl_sum_l = 0, wl_n_l = 0, wl_sum_p = 0, wl_n_p = 0;
        while (true) {
            /* ---- retire lanes whose particle is complete */
            if (__any_sync(AG_FULL, finish_now)) {
                if (finish_now) {
                    for (int ci = 0; ci < n_ci; ci++) {
                    const int comp = ag_coop_comp<NV, HALF>(ci, wid, half);
                    if (comp < 0) continue;
                        const double x1 = W(W_X0, comp) + W(W_XC, comp), v1 = W(W_V0, comp) + W(W_VC, comp);
                        if (dense && comp < 3) {
                            /* times left at a completed particle are its t_end: the end
                             * state; a particle stopped early leaves NaN at the times it
                             * did not reach */
                            const bool done_ok = pstat == AG_ST_OK;
                            const double nan = __longlong_as_double(0x7ff8000000000000LL);
                            for (int q = on; q < on_end; q++) {
                                A.out_state[6 * (size_t)q + comp] = done_ok ? x1 : nan;
                                A.out_state[6 * (size_t)q + 3 + comp] = done_ok ? v1 : nan;
                            }
                        }
                        if (comp < 3) {
                            double* s0 = A.state + 6 * (size_t)pid;
                            s0[comp] = x1; s0[3 + comp] = v1;
                            S.fin[comp][pl] = isfinite(x1) && isfinite(v1);
                        } else {
                            double* vs = A.var_state + ((size_t)pid * NV + (comp - 3) / 3) * 6;
                            vs[(comp - 3) % 3] = x1; vs[3 + (comp - 3) % 3] = v1;
                        }
                    }
                }
                __syncthreads();
                if (finish_now) {
                    const bool finite = S.fin[0][pl] && S.fin[1][pl] && S.fin[2][pl];
                    if (pstat == AG_ST_OK && !finite) pstat = AG_ST_NONFINITE;
                    if (wid == 0 && A.status) A.status[pid] = pstat;
                    live = false;
                    finish_now = false;
                }
            }
            if (!__any_sync(AG_FULL, live)) break;
            /* ---- watchdog (thread 0 decides for the block) */
            if (tid == 0 && (S.stage_fail || (A.watchdog_cycles > 0 && clock64() - clk0 > A.watchdog_cycles))) S.stop = 1;
            __syncthreads();
            if (S.stop) {
                pstat = AG_ST_TIMEOUT;
                finish_now = live;
                continue;
            }
            /* ---- step size: no further than the nearest unfinished end */
            const double rem = live ? fabs((tend - t) - tc) : 1e300;
            const double rem_min = warp_min(rem);
            double hstep;
            bool last_group = false;
            if (fabs(dt) >= rem_min) { hstep = dir * rem_min; last_group = true; }
            else hstep = dt;
            const bool last = live && last_group && rem == rem_min;
            /* the predictor's coefficients of nodes 1..7, (h_n hstep)^(k+1) over
             * the factorial-like products of IAS15's quadrature, once per step
             * (the group's step is the block's) rather than by every warp at
             * every node of every iteration; read after the next barrier */
            if (tid >= 1 && tid < 8) {
                /* the product rounded on its own, as the oracle forms a node time */
                S.ptn[tid] = t + (tc + __dmul_rn(hstep, ag_ias.h[tid]));
                const double s0 = hstep * ag_ias.h[tid];
                double x = s0 * s0 * 0.5, v = s0;
                S.pcx[tid][0] = s0; S.pcx[tid][1] = x; S.pcv[tid][0] = v;
#pragma unroll
                for (int k = 2; k < 9; k++) { x = x * ag_ias.fx[tid][k]; S.pcx[tid][k] = x; }
#pragma unroll
                for (int k = 1; k < 8; k++) { v = v * ag_ias.fv[tid][k]; S.pcv[tid][k] = v; }
            }

            /* ---- node 0: accelerations at the step start, g from the predicted b */
            if (WARM && tid == 0) clk_step = clock64();
            int bad = ag_coop_table_pass1<STAGE>(E, cf, t, S.scr, Tab, tid, R, cur, &S.stage_fail);
            n_tab++;
            if (live)
                for (int ci = 0; ci < n_ci; ci++) {
                    const int comp = ag_coop_comp<NV, HALF>(ci, wid, half);
                    if (comp < 0) continue;
                    S.xs[comp][pl] = W(W_X0, comp); S.vs[comp][pl] = W(W_V0, comp);
                    if constexpr (NV == 0 && !WARM) S.xsf[comp][lane] = ag_f2_of(W(W_X0, comp));
                }
            bad = __syncthreads_or(bad);
            if (bad) { pstat = S.stage_fail ? AG_ST_TIMEOUT : AG_ST_COVERAGE; finish_now = live; continue; }
            ag_coop_table_pass2(E, cf, t, Tab, S.scr, tid);
            __syncthreads();
            if (cf.geocentric == 1) { ag_coop_rel_geo(E, Tab, tid); __syncthreads(); }
            if constexpr (PAIRS) { ag_coop_pair_rows(Tab, prel, tid); __syncthreads(); }
            if (wid == 1 && (cf.forces & AG_F_EIH)) ag_coop_eih_sources(E, cf, Tab.T, lane);
            int fst = AG_OK;
            {
                const double xp[3] = {S.xs[0][pl], S.xs[1][pl], S.xs[2][pl]};
                const double vp[3] = {S.vs[0][pl], S.vs[1][pl], S.vs[2][pl]};
                double acc[3] = {0.0, 0.0, 0.0};
                if (NV > 0) {
                    if (live) {
                        double J[3][6];
                        if constexpr (PAIRS) ag_coop_force_pairs(wid, Tab, prel, E, cf, xp, vp, has_prm ? prm : nullptr, acc, J);
                        else fst = ag_coop_force_part<true>(wid, Tab, E, cf, xp, vp, has_prm ? prm : nullptr, acc, J);
                        for (int a = 0; a < 3; a++)
                            for (int b = 0; b < 6; b++) S.pj[wid][6 * a + b][lane] = J[a][b];
                    }
                } else if (wid < 2) {
                    if constexpr (NV == 0)
                        ag_coop_force_split01(wid, live, S.seps, lane, Tab, E, cf, xp, vp, has_prm ? prm : nullptr, acc);
                } else if (live) {
                    AgF2 xf3[3];
                    const AgF2* xfp = nullptr;          /* the float-pair position, where it was split */
                    if constexpr (NV == 0 && !WARM) {
                        xf3[0] = S.xsf[0][lane]; xf3[1] = S.xsf[1][lane]; xf3[2] = S.xsf[2][lane];
                        xfp = xf3;
                    }
                    fst = ag_coop_force_part<false, !WARM>(wid, Tab, E, cf, xp, vp, has_prm ? prm : nullptr, acc, nullptr,
                                                           nullptr, nullptr, xfp);
                }
                if (live) {
                    S.pa[wid][0][lane] = acc[0]; S.pa[wid][1][lane] = acc[1]; S.pa[wid][2][lane] = acc[2];
                    if (wid == 0 && half == 0) n_ev++;
                }
            }
            bad = __syncthreads_or(fst != AG_OK);
            if (bad) { pstat = AG_ST_COVERAGE; finish_now = live; continue; }
            if constexpr (NV > 0) ag_coop_sum_jac(S, wid, lane, live);
            if (live) {
                for (int ci = 0; ci < n_ci; ci++) {
                    const int comp = ag_coop_comp<NV, HALF>(ci, wid, half);
                    if (comp < 0) continue;
                    double at;
                    if (comp < 3) {
                        at = ((S.pa[3][comp][lane] + S.pa[2][comp][lane]) + S.pa[1][comp][lane]) + S.pa[0][comp][lane];
                    } else {
                        const int q = (comp - 3) / 3, a = (comp - 3) % 3;
                        double Jr[6];
                        for (int b = 0; b < 6; b++) Jr[b] = S.pj[0][6 * a + b][lane];
                        const double* dxq = &S.xs[3 + 3 * q][0];
                        const double* dvq = &S.vs[3 + 3 * q][0];
                        double s = Jr[0] * dxq[pl];
                        s = fma(Jr[1], dxq[32 + pl], s); s = fma(Jr[2], dxq[64 + pl], s);
                        s = fma(Jr[3], dvq[pl], s); s = fma(Jr[4], dvq[32 + pl], s); s = fma(Jr[5], dvq[64 + pl], s);
                        at = s;
                    }
                    W(W_A0, comp) = at;
                }
            }
            if (HALF) __syncwarp();
            /* ---- learned warm start: features, BF16 inference, b += kappa y */
            bool w_applied = false, w_probe = false, w_ran = false;
            if constexpr (WARM) {
                if (warm || logp)
                    w_ran = ag_warm_start<C>(A, W.w, W.ns, W.slot, ag_coop_pcomp<NV>(wid), WS, AgTableNearest{Tab.T}, lane,
                                             wid, live, warm, wl_on && S.wg_off == 0, hstep, dtls, steps, w_applied,
                                             w_probe, n_wused, n_wfall);
            }
            if (live) {
                for (int ci = 0; ci < n_ci; ci++) {
                    const int comp = ag_coop_comp<NV, HALF>(ci, wid, half);
                    if (comp < 0) continue;
                    double b[7];
#pragma unroll
                    for (int k = 0; k < 7; k++) b[k] = W(W_B + k, comp);
#pragma unroll
                    for (int j = 0; j < 7; j++) {
                        double s = b[j];
#pragma unroll
                        for (int k = j + 1; k < 7; k++) s = fma(b[k], ag_ias.d[j][k], s);
                        W(W_G + j, comp) = s;
                    }
                }
            }
            /* ---- predictor-corrector iterations */
            int iters = 1, it_lane = 0;
            double pc_last = 1e300, ma7 = 0.0;
            bool conv = !live;
            bool cov = false;
            while (true) {
                for (int n = 1; n < 8; n++) {
                    const double tn = S.ptn[n];
                    AgCoopTab& TabN = tabs[tab8 ? n : 0];
                    const bool build = !tab8 || iters == 1;     /* block-uniform */
                    bad = build ? ag_coop_table_pass1<STAGE>(E, cf, tn, S.scr, TabN, tid, R, cur, &S.stage_fail) : 0;
                    n_tab += build ? 1 : 0;
                    if (!conv) {
                        const double* sx = S.pcx[n];
                        const double* sv = S.pcv[n];
                        for (int ci = 0; ci < n_ci; ci++) {
                    const int comp = ag_coop_comp<NV, HALF>(ci, wid, half);
                    if (comp < 0) continue;
                            double px = sx[8] * W(W_B + 6, comp);
#pragma unroll
                            for (int j = 5; j >= 0; j--) px = fma(sx[j + 2], W(W_B + j, comp), px);
                            px = fma(sx[1], W(W_A0, comp), px);
                            px = fma(sx[0], W(W_V0, comp), px);
                            const double xn = W(W_X0, comp) + (px + W(W_XC, comp));
                            S.xs[comp][pl] = xn;
                            if constexpr (NV == 0 && !WARM) S.xsf[comp][lane] = ag_f2_of(xn);
                            double pv = sv[7] * W(W_B + 6, comp);
#pragma unroll
                            for (int j = 5; j >= 0; j--) pv = fma(sv[j + 1], W(W_B + j, comp), pv);
                            pv = fma(sv[0], W(W_A0, comp), pv);
                            S.vs[comp][pl] = W(W_V0, comp) + (pv + W(W_VC, comp));
                        }
                    }
                    bad = __syncthreads_or(bad);
                    if (bad) { cov = true; break; }
                    if (build) {
                        ag_coop_table_pass2(E, cf, tn, TabN, S.scr, tid);
                        __syncthreads();
                        if (cf.geocentric == 1) { ag_coop_rel_geo(E, TabN, tid); __syncthreads(); }
                        if constexpr (PAIRS) { ag_coop_pair_rows(TabN, prel + AG_PREL * n, tid); __syncthreads(); }
                        if (wid == 1 && (cf.forces & AG_F_EIH)) ag_coop_eih_sources(E, cf, TabN.T, lane);
                    }
                    {
                        const double xp[3] = {S.xs[0][pl], S.xs[1][pl], S.xs[2][pl]};
                        const double vp[3] = {S.vs[0][pl], S.vs[1][pl], S.vs[2][pl]};
                        double acc[3] = {0.0, 0.0, 0.0};
                        if (NV > 0) {
                            if (!conv) {
                                double J[3][6];
                                if constexpr (PAIRS)
                                    ag_coop_force_pairs(wid, TabN, prel + AG_PREL * n, E, cf, xp, vp, has_prm ? prm : nullptr, acc, J);
                                else ag_coop_force_part<true>(wid, TabN, E, cf, xp, vp, has_prm ? prm : nullptr, acc, J);
                                for (int a = 0; a < 3; a++)
                                    for (int b = 0; b < 6; b++) S.pj[wid][6 * a + b][lane] = J[a][b];
                            }
                        } else if (wid < 2) {
                            if constexpr (NV == 0)
                                ag_coop_force_split01(wid, !conv, S.seps, lane, TabN, E, cf, xp, vp, has_prm ? prm : nullptr, acc);
                        } else if (!conv) {
                            AgF2 xf3[3];
                            const AgF2* xfp = nullptr;
                            if constexpr (NV == 0 && !WARM) {
                                xf3[0] = S.xsf[0][lane]; xf3[1] = S.xsf[1][lane]; xf3[2] = S.xsf[2][lane];
                                xfp = xf3;
                            }
                            ag_coop_force_part<false, !WARM>(wid, TabN, E, cf, xp, vp, has_prm ? prm : nullptr, acc, nullptr,
                                                             nullptr, nullptr, xfp);
                        }
                        if (!conv) {
                            S.pa[wid][0][lane] = acc[0]; S.pa[wid][1][lane] = acc[1]; S.pa[wid][2][lane] = acc[2];
                            if (wid == 0 && half == 0) n_ev++;
                        }
                    }
                    __syncthreads();
                    if constexpr (NV > 0) ag_coop_sum_jac(S, wid, lane, !conv);
                    if (!conv) {
                        for (int ci = 0; ci < n_ci; ci++) {
                    const int comp = ag_coop_comp<NV, HALF>(ci, wid, half);
                    if (comp < 0) continue;
                            double at;
                            if (comp < 3) {
                                at = ((S.pa[3][comp][lane] + S.pa[2][comp][lane]) + S.pa[1][comp][lane]) + S.pa[0][comp][lane];
                            } else {
                                const int q = (comp - 3) / 3, a = (comp - 3) % 3;
                                double Jr[6];
                                for (int b = 0; b < 6; b++) Jr[b] = S.pj[0][6 * a + b][lane];
                                const double* dxq = &S.xs[3 + 3 * q][0];
                                const double* dvq = &S.vs[3 + 3 * q][0];
                                double s = Jr[0] * dxq[pl];
                                s = fma(Jr[1], dxq[32 + pl], s); s = fma(Jr[2], dxq[64 + pl], s);
                                s = fma(Jr[3], dvq[pl], s); s = fma(Jr[4], dvq[32 + pl], s); s = fma(Jr[5], dvq[64 + pl], s);
                                at = s;
                            }
                            double gn = (at - W(W_A0, comp)) * ag_ias.rrinv[n][0];
                            for (int j = 1; j < n; j++) gn = (gn - W(W_G + j - 1, comp)) * ag_ias.rrinv[n][j];
                            const double delta = gn - W(W_G + n - 1, comp);
                            W(W_G + n - 1, comp) = gn;
                            for (int k = 0; k < n - 1; k++) W(W_B + k, comp) = fma(delta, ag_ias.c[n - 1][k], W(W_B + k, comp));
                            W(W_B + n - 1, comp) += delta;
                            if (n == 7 && comp < 3) {
                                const double aa = fabs(at), db = fabs(delta);
                                S.ra[comp][pl] = ag_isnormal_pos(aa) ? aa : 0.0;
                                S.rdb[comp][pl] = ag_isnormal_pos(db) ? db : 0.0;
                            }
                        }
                    }
                    if (HALF) __syncwarp();      /* the other half has read this node's states */
                }
                if (cov) break;
                __syncthreads();
                if (!conv) {
                    double maxa = 0.0, maxdb = 0.0;
                    for (int k = 0; k < 3; k++) {
                        maxa = ag_max_nonneg(maxa, S.ra[k][pl]);
                        maxdb = ag_max_nonneg(maxdb, S.rdb[k][pl]);
                    }
                    ma7 = maxa;
                    const double pc_err = maxdb / maxa;
                    conv = (pc_err < 1e-16) || (iters > 2 && pc_last <= pc_err) || (iters >= 12);
                    if (conv) { it_lane = iters; if (wid == 0 && half == 0) n_it += (unsigned long long)iters; }
                    else pc_last = pc_err;
                }
                if (__all_sync(AG_FULL, conv)) break;
                iters++;
            }
            if (cov) { pstat = S.stage_fail ? AG_ST_TIMEOUT : AG_ST_COVERAGE; finish_now = live; continue; }
            if (warm && live) {
                if (w_applied) { wl_sum_l += it_lane; wl_n_l++; }
                else if (w_probe) {
                    wl_sum_p += it_lane; wl_n_p++;
                    /* the plain predictor converges faster for this member: fall back */
                    if (wl_n_p >= 4 && wl_n_l >= 8 && (long long)wl_sum_l * wl_n_p > (long long)wl_sum_p * wl_n_l) {
                        wl_on = false;
                        if (wid == 0) n_wfall++;
                    }
                }
            }
            if (warm && !A.warm_no_time_fallback && tid == 0 && S.wg_off == 0) {
                /* the step so far: body tables, forces, the start, the corrector */
                const long long dt_clk = clock64() - clk_step;
                const bool probe = (steps & 7) == 7;
                if (w_ran) { wg_t_l += dt_clk; wg_n_l++; }
                else if (probe) { wg_t_p += dt_clk; wg_n_p++; }
                /* the group's learned steps take longer than its plain probes: the
                 * plain predictor for the rest of the group */
                if (wg_n_p >= 3 && wg_n_l >= 12 && (double)wg_t_l / wg_n_l > (double)wg_t_p / wg_n_p) {
                    S.wg_off = 1;
                    n_wfall++;
                }
            }
            /* ---- step-size control: each lane's choice, the group takes the smallest */
            const int pc = HALF ? (wid == 1 ? half : (wid == 2 && half == 0 ? 2 : -1)) : ag_coop_pcomp<NV>(wid);
            if (live && pc >= 0) {
                const double bb = fabs(W(W_B + 6, pc));
                S.rb6[pc][pl] = ag_isnormal_pos(bb) ? bb : 0.0;
            }
            __syncthreads();
            double dt_new_l = 1e300, dt_nocap_l = 1e300;
            bool rej_l = false;
            /* warp 0 forms each lane's proposal (the power and the divisions
             * are FP64 work that every warp would repeat); the others read it */
            if (wid == 0) {
                if (A.epsilon > 0.0 && live) {
                    double mb = 0.0;
                    for (int k = 0; k < 3; k++) mb = ag_max_nonneg(mb, S.rb6[k][pl]);
                    const double err = mb / ma7;
                    const double safety = 0.25;
                    double dn;
                    if (ag_isnormal_pos(err)) dn = pow(A.epsilon / err, 1.0 / 7.0) * hstep;
                    else dn = hstep / safety;
                    if (fabs(dn) < A.min_dt) dn = copysign(A.min_dt, dn);
                    dt_nocap_l = fabs(dn);
                    const double ratio = dn / hstep;
                    if (fabs(ratio) < safety) rej_l = true;
                    else if (fabs(ratio) > 1.0 / safety) dn = hstep / safety;
                    dt_new_l = fabs(dn);
                }
                S.sdn[lane] = dt_new_l; S.sdc[lane] = dt_nocap_l; S.srej[lane] = rej_l ? 1 : 0;
            }
            __syncthreads();
            if (wid != 0) { dt_new_l = S.sdn[lane]; dt_nocap_l = S.sdc[lane]; rej_l = S.srej[lane] != 0; }
            if (live && !last_group && A.epsilon > 0.0 && A.dt_floor > 0.0 && dt_nocap_l < A.dt_floor) {
                /* step underflow: this lane's particle is hitting a body; it stops
                 * (state of the step start) and the group goes on without it.  Not
                 * tested on a step cut short to land on a member's t_end: the
                 * proposals scale with that short step */
                pstat = AG_ST_UNDERFLOW;
                finish_now = true;
                rej_l = false;
                dt_new_l = 1e300;
                dt_nocap_l = 1e300;
            }
            if (__any_sync(AG_FULL, finish_now && pstat == AG_ST_UNDERFLOW)) {
                if (!__any_sync(AG_FULL, live && !finish_now)) continue;   /* only underflowing lanes left */
            }
            double dt_new;
            if (A.epsilon > 0.0) {
                dt_new = dir * warp_min(dt_new_l);
                /* a step shortened to land on a lane's t_end does not shrink the
                 * group's step beyond what the error control asks for */
                if (last_group) dt_new = dir * fmin(fabs(dt), fmax(fabs(dt_new), warp_min(dt_nocap_l)));
            } else {
                dt_new = dt;            /* fixed step */
            }
            const bool reject = __any_sync(AG_FULL, rej_l);
            if (reject) {
                if (live) {
                    if (wid == 0 && half == 0) n_rej++;
                    for (int ci = 0; ci < n_ci; ci++) {
                    const int comp = ag_coop_comp<NV, HALF>(ci, wid, half);
                    if (comp < 0) continue;
                        if (dtls != 0.0) ag_predict_next_comp(W, comp, dt_new / dtls);
                        else
                            for (int k = 0; k < 7; k++) { W(W_B + k, comp) = 0.0; W(W_E + k, comp) = 0.0; }
                    }
                }
                dt = dt_new;
                continue;
            }
            /* ---- log (features, target) pairs of accepted steps: target =
             * (b_conv - b_pred) / kappa with b_pred = e + (br - er), the plain prediction */
            if (logp)
                ag_warm_log<C>(A, W.w, W.ns, W.slot, ag_coop_pcomp<NV>(wid), WS, lane, wid,
                               live && WS.valid[lane] && (steps % A.log_every) == 0);
            /* ---- dense output: states at the output times this step covers,
             * from the step's polynomial (the interpolation of ASSIST's
             * assist_interpolate, src/assist.c:556-597: s- and sv-coefficients
             * built by the same recurrences, x from the step-start x, v, a, b) */
            if (dense && live) {
                const double tstep_end = (t + tc) + hstep;
                while (on < on_end && dir * (A.out_t[on] - tstep_end) <= 0.0 && !(last && A.out_t[on] == tend)) {
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
                    if (ag_coop_pcomp<NV>(wid) >= 0) {
                        const int c = ag_coop_pcomp<NV>(wid);
                        const double b0 = W(W_B + 0, c), b1 = W(W_B + 1, c), b2 = W(W_B + 2, c), b3 = W(W_B + 3, c),
                                     b4 = W(W_B + 4, c), b5 = W(W_B + 5, c), b6 = W(W_B + 6, c);
                        const double a0 = W(W_A0, c), v0 = W(W_V0, c);
                        A.out_state[6 * (size_t)on + c] =
                            W(W_X0, c) + (s[8] * b6 + s[7] * b5 + s[6] * b4 + s[5] * b3 + s[4] * b2 + s[3] * b1 +
                                          s[2] * b0 + s[1] * a0 + s[0] * v0);
                        A.out_state[6 * (size_t)on + 3 + c] = v0 + sv[7] * b6 + sv[6] * b5 + sv[5] * b4 + sv[4] * b3 +
                                                              sv[3] * b2 + sv[2] * b1 + sv[1] * b0 + sv[0] * a0;
                    }
                    on++;
                }
            }
            /* ---- accept */
            if (live) {
                if (wid == 0 && half == 0) n_acc++;
                const double h2 = hstep * hstep;
                for (int ci = 0; ci < n_ci; ci++) {
                    const int comp = ag_coop_comp<NV, HALF>(ci, wid, half);
                    if (comp < 0) continue;
                    double b[7];
#pragma unroll
                    for (int k = 0; k < 7; k++) b[k] = W(W_B + k, comp);
                    const double a0 = W(W_A0, comp);
                    double ix = b[6] / 72. + b[5] / 56. + b[4] / 42. + b[3] / 30. + b[2] / 20. + b[1] / 12. + b[0] / 6. + a0 / 2.;
                    ix = fma(ix, h2, W(W_V0, comp) * hstep);
                    double y = ix + W(W_XC, comp);
                    const double x0 = W(W_X0, comp);
                    double s = x0 + y;
                    W(W_XC, comp) = y - (s - x0);
                    W(W_X0, comp) = s;
                    double iv = b[6] / 8. + b[5] / 7. + b[4] / 6. + b[3] / 5. + b[2] / 4. + b[1] / 3. + b[0] / 2. + a0;
                    iv = iv * hstep;
                    y = iv + W(W_VC, comp);
                    const double v0 = W(W_V0, comp);
                    s = v0 + y;
                    W(W_VC, comp) = y - (s - v0);
                    W(W_V0, comp) = s;
#pragma unroll
                    for (int k = 0; k < 7; k++) { W(W_ER + k, comp) = W(W_E + k, comp); W(W_BR + k, comp) = b[k]; }
                    ag_predict_next_comp(W, comp, dt_new / hstep);
                }
            }
            {
                const double y = hstep + tc;
                const double s = t + y;
                tc = y - (s - t);
                t = s;
            }
            dtls = hstep;
            dt = dt_new;
            steps++;
            if (last) finish_now = true;
            if (last_group && live && !last && fabs((tend - t) - tc) == 0.0) finish_now = true;
            if (A.max_steps > 0 && steps >= A.max_steps && live && !finish_now) { pstat = AG_ST_BUDGET; finish_now = true; }
        }
    }
    if (wid == 0) {
        atomicAdd(&A.counters[0], n_acc);
        atomicAdd(&A.counters[1], n_rej);
        atomicAdd(&A.counters[2], n_ev);
        atomicAdd(&A.counters[3], n_it);
        atomicAdd(&A.counters[4], n_wused);
        atomicAdd(&A.counters[5], n_wfall);
        if (tid == 0) atomicAdd(&A.counters[6], n_tab);   /* body tables, one per block and node time */
    }
    /* a copy that did not complete in time: wait for it once more (bounded)
     * before the block's shared memory is released */
    if (STAGE && tid == 0 && S.stage_fail) ag_mbar_wait(&R->bar, cur.phase ^ 1u);
}

/* Dynamic shared memory that leaves no room on a multiprocessor (228 KB) for
 * another such block or one of the pair-term kernel (60 KB and more). */
#define AG_COOP_ALONE (165 * 1024)

/* Opt the kernel in to its dynamic shared memory (above the 48 KB default). */
template <int NV, bool WARM, int OCC, bool STAGE = false, bool PAIRS = false, bool HALF = false>
static int ag_coop_dyn_attr() {
    constexpr size_t own = AgCoopDyn<NV, WARM, STAGE, OCC, HALF>::bytes;
    constexpr size_t bytes = (NV == 0 && !WARM && OCC == 2 && !STAGE) || HALF ? (size_t)AG_COOP_ALONE : own;
    if (bytes == 0) return 0;
    return (int)cudaFuncSetAttribute(ag_k_coop<NV, WARM, OCC, STAGE, PAIRS, HALF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

template <int NV, bool WARM, int OCC, bool STAGE = false, bool PAIRS = false, bool HALF = false>
static int ag_coop_blocks_per_sm() {
    int bps = 0;
    if (ag_coop_dyn_attr<NV, WARM, OCC, STAGE, PAIRS, HALF>() == 0)
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, ag_k_coop<NV, WARM, OCC, STAGE, PAIRS, HALF>, 128,
                                                      AgCoopDyn<NV, WARM, STAGE, OCC, HALF>::bytes);
    return bps;
}

/* Slots (32 per resident block) of the plain (nv = 0: occ 2 or 3, stage
 * only with occ 2) or variational (nv = 6: occ 1 or 2) kernel, or of their learned
 * warm-start builds (warm), on the current device. */
int ag_coop_max_slots(int nv, int occ, int stage, int warm, int pairs) {
    int dev = 0, sms = 0, bps = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (nv == 6 && pairs == 16) bps = occ == 1 ? 1 : ag_coop_blocks_per_sm<6, false, 2, false, true, true>();
    else if (nv == 6)
        bps = warm ? ag_coop_blocks_per_sm<6, true, 2>()
                   : (occ == 1 ? ag_coop_blocks_per_sm<6, false, 1>() : ag_coop_blocks_per_sm<6, false, 2>());
    else if (warm) bps = ag_coop_blocks_per_sm<0, true, 2>();
    else if (occ == 3) bps = ag_coop_blocks_per_sm<0, false, 3>();
    else if (stage) bps = ag_coop_blocks_per_sm<0, false, 2, true>();
    else bps = ag_coop_blocks_per_sm<0, false, 2>();
    if (bps < 1) bps = 1;
    return sms * bps * 32;
}

int ag_launch_coop(const DevEphem& E, const ForceCfg& c, const AgBatchArgs& a, int nv, int occ, int stage,
                   cudaStream_t s, int pairs) {
    int e = ag_ias_tables_init();
    if (e) return e;
    const int blocks = (a.nslots + 31) / 32;
    if (nv == 6 && (a.mlp || a.log_x)) {
        if ((e = ag_coop_dyn_attr<6, true, 2>())) return e;
        ag_k_coop<6, true, 2><<<blocks, 128, AgCoopDyn<6, true>::bytes, s>>>(E.self_dev, c, a);
    } else if (nv == 6 && pairs == 16) {
        if ((e = ag_coop_dyn_attr<6, false, 2, false, true, true>())) return e;
        ag_k_coop<6, false, 2, false, true, true>
            <<<blocks, 128, occ == 1 ? (size_t)AG_COOP_ALONE : AgCoopDyn<6, false, false, 2, true>::bytes, s>>>(E.self_dev, c, a);
    } else if (nv == 6 && pairs) {
        if ((e = ag_coop_dyn_attr<6, false, 2, false, true>())) return e;
        ag_k_coop<6, false, 2, false, true><<<blocks, 128, AgCoopDyn<6, false>::bytes, s>>>(E.self_dev, c, a);
    } else if (nv == 6 && occ == 1) {
        if ((e = ag_coop_dyn_attr<6, false, 1>())) return e;
        ag_k_coop<6, false, 1><<<blocks, 128, AgCoopDyn<6, false, false, 1>::bytes, s>>>(E.self_dev, c, a);
    } else if (nv == 6) {
        if ((e = ag_coop_dyn_attr<6, false, 2>())) return e;
        ag_k_coop<6, false, 2><<<blocks, 128, AgCoopDyn<6, false>::bytes, s>>>(E.self_dev, c, a);
    } else if (a.mlp || a.log_x) {
        if ((e = ag_coop_dyn_attr<0, true, 2>())) return e;
        ag_k_coop<0, true, 2><<<blocks, 128, AgCoopDyn<0, true>::bytes, s>>>(E.self_dev, c, a);
    } else if (occ == 1) {
        /* the plain build for two, each block with a multiprocessor to itself */
        if ((e = ag_coop_dyn_attr<0, false, 2>())) return e;
        ag_k_coop<0, false, 2><<<blocks, 128, AG_COOP_ALONE, s>>>(E.self_dev, c, a);
    } else if (occ == 3) {
        if ((e = ag_coop_dyn_attr<0, false, 3>())) return e;
        ag_k_coop<0, false, 3><<<blocks, 128, AgCoopDyn<0, false>::bytes, s>>>(E.self_dev, c, a);
    } else if (stage) {
        if ((e = ag_coop_dyn_attr<0, false, 2, true>())) return e;
        ag_k_coop<0, false, 2, true><<<blocks, 128, AgCoopDyn<0, false, true>::bytes, s>>>(E.self_dev, c, a);
    } else {
        if ((e = ag_coop_dyn_attr<0, false, 2>())) return e;
        ag_k_coop<0, false, 2><<<blocks, 128, AgCoopDyn<0, false>::bytes, s>>>(E.self_dev, c, a);
    }
    return (int)cudaGetLastError();
}

/* What a launch of this kernel sets up on its first use on a device (the
 * IAS15 tables, the shared-memory opt-ins of every build), done ahead of a
 * stream capture. */
int ag_coop_ready(void) {
    int e = ag_ias_tables_init();
    if (!e) e = ag_coop_dyn_attr<0, false, 2>();
    if (!e) e = ag_coop_dyn_attr<0, false, 3>();
    if (!e) e = ag_coop_dyn_attr<0, false, 2, true>();
    if (!e) e = ag_coop_dyn_attr<0, true, 2>();
    if (!e) e = ag_coop_dyn_attr<6, true, 2>();
    if (!e) e = ag_coop_dyn_attr<6, false, 1>();
    if (!e) e = ag_coop_dyn_attr<6, false, 2>();
    if (!e) e = ag_coop_dyn_attr<6, false, 2, false, true, true>();
    if (!e) e = ag_coop_dyn_attr<6, false, 2, false, true>();
    return e;
}
