/*
 * kernels_forces.cu -- ephemeris and force kernels (K1, K2) and their launchers.
 *
 *   ag_k_bodies_tile,
 *   ag_k_bodies_one   : full body states (GM, x, v, a) at n times; the device
 *                       side of assist_all_ephem / assist_get_particle
 *                       (src/forces.c:175-263).  ag_k_bodies is the form for
 *                       planets from an SPK file, one thread per (time, body).
 *   ag_k_forces_table : every particle at ONE shared time (the REBOUND callback
 *                       assist_additional_forces, src/forces.c:49-173).  Each block
 *                       evaluates the body table for that time into shared
 *                       memory (11 planet threads, one thread per asteroid, one
 *                       per EIH source), then one thread per real particle
 *                       computes its acceleration and, if it has variational
 *                       particles, their accelerations from its Jacobian.
 *   ag_k_forces_each  : every particle at its OWN time (batched API); bodies are
 *                       evaluated per thread.
 */
#include <cuda_runtime.h>
#include <cstdio>

#include "device_forces.cuh"
#include "internal.h"
#include "table_forces.cuh"

/* All particles at one time.  Particle arrays are SoA (x[3][n]). */
__global__ void __launch_bounds__(128) ag_k_forces_table(const DevEphem* __restrict__ Ep, ForceCfg c, double t, AgForceIO io) {
    const DevEphem& E = *Ep;
    __shared__ AgTable T;
    ag_block_table(E, c, t, T);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= io.n_real) return;
    ag_table_force_particle(E, c, T, io, i);
}

/* Every particle at its own time; nv (0 or 6) variational particles per real
 * particle stored right after it: state arrays are [n][6], var [n][nv][6]. */
template <int NV>
__global__ void __launch_bounds__(128) ag_k_forces_each(const DevEphem* __restrict__ Ep, ForceCfg c, int n, const double* __restrict__ t,
                                                        const double* __restrict__ state, const double* __restrict__ params,
                                                        const double* __restrict__ var_state, double* __restrict__ acc,
                                                        double* __restrict__ var_acc, int* __restrict__ status) {
    const DevEphem& E = *Ep;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double x[3] = {state[6 * (size_t)i], state[6 * (size_t)i + 1], state[6 * (size_t)i + 2]};
    const double v[3] = {state[6 * (size_t)i + 3], state[6 * (size_t)i + 4], state[6 * (size_t)i + 5]};
    double Ab[3] = {0.0, 0.0, 0.0};
    const double* A = nullptr;
    if (params) { Ab[0] = params[3 * (size_t)i]; Ab[1] = params[3 * (size_t)i + 1]; Ab[2] = params[3 * (size_t)i + 2]; A = Ab; }
    ThreadBodies B(E, t[i]);
    double a[3];
    int st;
    if (NV > 0) {
        double J[3][6], JA[3][3];
        bool has_ng;
        st = ag_forces<ThreadBodies, true>(B, E, c, x, v, A, a, J, JA, &has_ng);
#pragma unroll 1
        for (int q = 0; q < NV; q++) {
            const double* vs = var_state + ((size_t)i * NV + q) * 6;
            double out[3];
            ag_apply_jac(J, JA, has_ng, vs, vs + 3, nullptr, out);
            double* va = var_acc + ((size_t)i * NV + q) * 3;
            va[0] = out[0]; va[1] = out[1]; va[2] = out[2];
        }
    } else {
        st = ag_forces<ThreadBodies, false>(B, E, c, x, v, A, a, nullptr, nullptr, nullptr);
    }
    acc[3 * (size_t)i] = a[0]; acc[3 * (size_t)i + 1] = a[1]; acc[3 * (size_t)i + 2] = a[2];
    if (status) status[i] = st;
}

/* Full body states: out[(ti * nb + b) * 10 + ...] = GM, x, y, z, vx, vy, vz, ax, ay, az. */
__global__ void ag_k_bodies(const DevEphem* __restrict__ Ep, int n, const double* __restrict__ t, double* __restrict__ out,
                            int* __restrict__ status) {
    const DevEphem& E = *Ep;
    const int nb = AG_NPL + E.n_ast;
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n * nb) return;
    const int ti = g / nb, b = g % nb;
    double* o = out + (size_t)g * 10;
    int st;
    if (b < AG_NPL) {
        st = ag_planet_full(E, b, t[ti], o);
    } else {
        const int m = b - AG_NPL;
        double h[3], sun[10];
        o[0] = E.ast_gm[m];
        st = ag_asteroid_exact(E, m, t[ti], h);
        if (st == AG_OK) st = ag_planet_full(E, AG_SUN, t[ti], sun);
        o[1] = __dadd_rn(h[0], sun[1]); o[2] = __dadd_rn(h[1], sun[2]); o[3] = __dadd_rn(h[2], sun[3]);
        for (int k = 4; k < 10; k++) o[k] = __longlong_as_double(0x7ff8000000000000LL);
    }
    if (status) atomicMax(&status[ti], st);
}

/* a / b correctly rounded, y = 1 / b rounded to nearest: the product and two
 * residual corrections (Markstein 1990: with y correctly rounded the last one
 * gives the rounded quotient), five FP64 instructions where the compiler's
 * division takes 8.5 of the FP64 pipe's time.  For a and b far from the ends
 * of the exponent range. */
__device__ __forceinline__ double ag_div_by(double a, double b, double y) {
    double q = a * y;
    q = fma(fma(-q, b, a), y, q);
    return fma(fma(-q, b, a), y, q);
}

/* Position, velocity and acceleration sums of a .440 column in the operations
 * and order of src/ascii_ephem.c:27-65: NC components ncf apart from P on.
 * The recurrences run beside the sums (no arrays), and the products by 2 and
 * 4, which are exact, are fused. */
template <int NC>
__device__ __forceinline__ void ag_pva(const double* P, int ncf, double t0, double c, double* u, double* v, double* w) {
    const double two = __dmul_rn(2.0, t0);
    double T0 = 1.0, T1 = t0, S0 = 0.0, S1 = 1.0, U0 = 0.0, U1 = 0.0;
#pragma unroll
    for (int m = 0; m < NC; m++) {
        u[m] = __dadd_rn(__dadd_rn(0.0, P[m * ncf]), __dmul_rn(t0, P[m * ncf + 1]));
        v[m] = __dmul_rn(P[m * ncf + 1], c);
        w[m] = 0.0;
    }
    for (int p = 2; p < ncf; p++) {
        const double T2 = __dsub_rn(__dmul_rn(two, T1), T0);
        const double S2 = __dsub_rn(fma(2.0, T1, __dmul_rn(two, S1)), S0);
        const double U2 = p == 2 ? 4.0 : __dsub_rn(fma(4.0, S1, __dmul_rn(two, U1)), U0);
#pragma unroll
        for (int m = 0; m < NC; m++) {
            const double cf = P[m * ncf + p];
            u[m] = __dadd_rn(u[m], __dmul_rn(T2, cf));
            v[m] = __dadd_rn(v[m], __dmul_rn(__dmul_rn(S2, cf), c));
            w[m] = __dadd_rn(w[m], __dmul_rn(__dmul_rn(__dmul_rn(U2, cf), c), c));
        }
        T0 = T1; T1 = T2; S0 = S1; S1 = S2; U0 = U1; U1 = U2;
    }
}

/* A column's sub-interval at record fraction tf: its coefficients, Chebyshev
 * time and derivative factor. */
__device__ __forceinline__ const double* ag_col_at(const DevEphem& E, const double* rec, int col, double tf, double* t0,
                                                   double* c) {
    const int ncf = E.col_ncf[col], niv = E.col_niv[col];
    const double tt = __dmul_rn(tf, (double)niv);
    double fl;
    const int b = ag_subinterval(tt, niv, &fl);
    *t0 = __dsub_rn(__dmul_rn(2.0, __dsub_rn(tt, fl)), 1.0);
    *c = E.col_rate[col];
    return rec + E.col_off[col] + ncf * 3 * b;
}

/* The SPK record of an asteroid at time t, as ag_asteroid_exact chooses it:
 * first X coefficient, normalised time and coefficients per component.  The
 * two divisions are skipped when the asteroid's segment and record have the
 * epochs of the one before (key: init_jd, intlen_days, MID, RADIUS). */
struct AgAstRec {
    double init_jd = 0.0, intlen = 0.0, mid = 0.0, rad = 0.0, z = 0.0;
    int b = 0;
};
__device__ __forceinline__ int ag_ast_at(const DevEphem& E, int m, double t, AgAstRec& R, const double** X, int* P) {
    const double jd = E.jd_ref + t;
    if (!(jd >= E.ast_beg[m] && jd <= E.ast_end[m])) return AG_ERR_COVERAGE;   /* NaN too */
    int n = 0;
    if (E.ast_nseg[m] > 1) {
        n = (int)((E.jd_ref + t - E.ast_beg[m]) / E.ast_res[m]);
        if (n >= E.ast_nseg[m]) n = E.ast_nseg[m] - 1;
    }
    const AgSpkSeg sg = E.segs[E.ast_seg0[m] + n];
    auto same = [](double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); };
    if (!same(sg.init_jd, R.init_jd) || !same(sg.intlen_days, R.intlen)) {
        R.b = (int)(__ddiv_rn(__dadd_rn(__dsub_rn(E.jd_ref, sg.init_jd), t), sg.intlen_days));
        R.init_jd = sg.init_jd;
        R.intlen = sg.intlen_days;
    }
    int b = R.b;
    if (b >= sg.nrec) b = sg.nrec - 1;
    if (b < 0) b = 0;
    const AgRecMeta meta = E.rec_meta[sg.meta_off + b];
    if (!same(meta.x, R.mid) || !same(meta.y, R.rad)) {
        R.z = __ddiv_rn(__dadd_rn(__dsub_rn(E.jd_ref, meta.x), t), meta.y);
        R.mid = meta.x;
        R.rad = meta.y;
    }
    *X = E.spk + sg.data_off + (size_t)b * sg.R + 2;
    *P = sg.P;
    return AG_OK;
}

/* Heliocentric position (AU) of NC components from the record, in the order
 * of src/spk.c:428-474. */
template <int NC>
__device__ __forceinline__ void ag_ast_sum(const double* X, int P, double z, double* h) {
    const double two = __dmul_rn(2.0, z);
    double T0 = 1.0, T1 = z;
#pragma unroll
    for (int m = 0; m < NC; m++) {
        h[m] = __dadd_rn(0.0, X[m * P]);
        if (P > 1) h[m] = __dadd_rn(h[m], __dmul_rn(X[m * P + 1], z));
    }
    for (int q = 2; q < P; q++) {
        const double T2 = __dsub_rn(__dmul_rn(two, T1), T0);
#pragma unroll
        for (int m = 0; m < NC; m++) h[m] = __dadd_rn(h[m], __dmul_rn(X[m * P + q], T2));
        T0 = T1; T1 = T2;
    }
#pragma unroll
    for (int m = 0; m < NC; m++) h[m] = ag_div_by(h[m], 149597870.7, 1.0 / 149597870.7);
}

/* Full states of all bodies, lane = time: a block of four warps takes 32
 * times and each warp a share of the bodies of about equal FP64 work (1,250
 * to 1,550 warp instructions: 35 a coefficient of a planet, 8 of an
 * asteroid), so every lane works (one thread per time and body had 7 of 32
 * active and formed the Sun again for each asteroid).  A body's ten values go
 * through shared memory so that a store covers whole 80-byte rows.
 * Bound by the FP64 pipe: 30,011 times 3,053 -> 367 us. */
#define AG_TILE_PAD 11
/* Up to here a block a time: its 33 + 48 busy threads take 3.3 times the FP64
 * instructions a time, but a tile's warps run 1,500 of them one after the
 * other (50 us) where a single time takes 240. */
#define AG_BODIES_ONE 1024
__global__ void __launch_bounds__(128) ag_k_bodies_tile(const DevEphem* __restrict__ Ep, int n, const double* __restrict__ t,
                                                        double* __restrict__ out, int* __restrict__ status) {
    const DevEphem& E = *Ep;
    __shared__ double buf[4][32 * AG_TILE_PAD];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nb = AG_NPL + E.n_ast;
    const int i0 = 32 * blockIdx.x, i = i0 + lane, rows = min(32, n - i0);
    const bool on = i < n;
    const double ti = on ? t[i] : t[i0];
    double* row = buf[wid] + lane * AG_TILE_PAD;
    const double* rec = nullptr;
    double tf = 0.0;
    const int pst = ag_planet_record(E, ti, &rec, &tf);
    if (on && pst != AG_OK && status && wid == 0) atomicMax(&status[i], pst);
    auto flush = [&](int body, int k0) {
        /* values k0.. of the body's rows; rows whose record is missing keep
         * everything but GM as it was */
        __syncwarp();
        const unsigned okm = __ballot_sync(0xffffffffu, pst == AG_OK);
        for (int q = lane; q < 10 * rows; q += 32) {
            const int r = q / 10, k = q - 10 * r;
            if (k >= k0 && (k == 0 || ((okm >> r) & 1) || body >= AG_NPL))
                out[((size_t)(i0 + r) * nb + body) * 10 + k] = buf[wid][r * AG_TILE_PAD + k];
        }
        __syncwarp();
    };
    const double icau = E.inv_cau, ivel = E.inv_cau_per_day, adiv = E.pl_cau / (86400. * 86400.), iadiv = 1.0 / adiv;
    auto put = [&](int body, const double* u, const double* v, const double* w) {
        row[0] = E.gm[body];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            row[1 + k] = ag_div_by(u[k], E.pl_cau, icau);
            row[4 + k] = ag_div_by(v[k], E.cau_per_day, ivel);
            row[7 + k] = ag_div_by(w[k], adiv, iadiv);
        }
        flush(body, 0);
    };
    if (wid == 3) {
        /* the asteroids, about the Sun */
        double sun[3] = {0.0, 0.0, 0.0};
        if (pst == AG_OK) {
            double v[3], t0, c;
            const double* P = ag_col_at(E, rec, AG_C_SUN, tf, &t0, &c);
            (void)v;
            const int ncf = E.col_ncf[AG_C_SUN];
            const double two = __dmul_rn(2.0, t0);
            double T0 = 1.0, T1 = t0;
            for (int m = 0; m < 3; m++) sun[m] = __dadd_rn(__dadd_rn(0.0, P[m * ncf]), __dmul_rn(t0, P[m * ncf + 1]));
            for (int p = 2; p < ncf; p++) {
                const double T2 = __dsub_rn(__dmul_rn(two, T1), T0);
                for (int m = 0; m < 3; m++) sun[m] = __dadd_rn(sun[m], __dmul_rn(T2, P[m * ncf + p]));
                T0 = T1; T1 = T2;
            }
            for (int m = 0; m < 3; m++) sun[m] = ag_div_by(sun[m], E.pl_cau, icau);
        }
        AgAstRec R;
        int bad = AG_OK;
        for (int m = 0; m < E.n_ast; m++) {
            const double* X;
            int P;
            double h[3] = {0.0, 0.0, 0.0};
            const int st = ag_ast_at(E, m, ti, R, &X, &P);
            if (st != AG_OK) bad = st;
            else ag_ast_sum<3>(X, P, R.z, h);
            row[0] = E.ast_gm[m];
            for (int k = 0; k < 3; k++) row[1 + k] = __dadd_rn(h[k], sun[k]);
            for (int k = 4; k < 10; k++) row[k] = __longlong_as_double(0x7ff8000000000000LL);
            flush(AG_NPL + m, 0);
        }
        if (on && bad != AG_OK && status) atomicMax(&status[i], bad);
        return;
    }
    double u[3], v[3], w[3];
    auto column = [&](int col) {
        if (pst != AG_OK) return;
        double t0, c;
        const double* P = ag_col_at(E, rec, col, tf, &t0, &c);
        ag_pva<3>(P, E.col_ncf[col], t0, c, u, v, w);
    };
    if (wid == 0) {
        /* Earth and Moon from their barycentre and the geocentric Moon, Mars */
        double eu[3], ev[3], ew[3];
        column(AG_C_EMB);
        for (int k = 0; k < 3; k++) { eu[k] = u[k]; ev[k] = v[k]; ew[k] = w[k]; }
        column(AG_C_LUN);
        for (int e = 0; e < 2; e++) {
            const double f = e == 0 ? E.f_earth : E.f_moon;
            double a[3], b[3], c[3];
            for (int k = 0; k < 3; k++) {
                a[k] = __dadd_rn(eu[k], __dmul_rn(u[k], f));
                b[k] = __dadd_rn(ev[k], __dmul_rn(v[k], f));
                c[k] = __dadd_rn(ew[k], __dmul_rn(w[k], f));
            }
            put(e == 0 ? AG_EAR : AG_MOO, a, b, c);
        }
        column(AG_C_MAR);
        put(AG_MAR, u, v, w);
    } else {
        /* warp 1: Sun, Mercury, Venus; warp 2: Jupiter .. Pluto */
        const int b0 = wid == 1 ? AG_SUN : AG_JUP, b1 = wid == 1 ? AG_VEN : AG_PLU;
        for (int body = b0; body <= b1; body++) {
            column(ag_col_of(body));
            put(body, u, v, w);
        }
    }
}

/* The same for few times: a block a time, a thread a component of a column
 * (threads 0..32) or of an asteroid (64..), whose longest chain is 14
 * coefficients of 17 FP64 instructions. */
__global__ void __launch_bounds__(128) ag_k_bodies_one(const DevEphem* __restrict__ Ep, const double* __restrict__ t,
                                                       double* __restrict__ out, int* __restrict__ status) {
    const DevEphem& E = *Ep;
    __shared__ double col[11][3][3], sun[3];
    const int tid = threadIdx.x, ti = blockIdx.x, nb = AG_NPL + E.n_ast;
    const double tt = t[ti];
    double* o = out + (size_t)ti * nb * 10;
    const double* rec = nullptr;
    double tf = 0.0;
    const int pst = ag_planet_record(E, tt, &rec, &tf);
    if (tid == 0 && pst != AG_OK && status) atomicMax(&status[ti], pst);
    if (tid < 33 && pst == AG_OK) {
        const int c = tid / 3, m = tid - 3 * c, ncf = E.col_ncf[c];
        double t0, rate;
        const double* P = ag_col_at(E, rec, c, tf, &t0, &rate);
        ag_pva<1>(P + m * ncf, ncf, t0, rate, &col[c][m][0], &col[c][m][1], &col[c][m][2]);
        if (c == AG_C_SUN) sun[m] = ag_div_by(col[c][m][0], E.pl_cau, E.inv_cau);
    }
    double h = 0.0;
    int ast = -1;
    if (tid >= 64) {
        /* each thread holds its first asteroid component over the barrier */
        const int q = tid - 64;
        if (q < 3 * E.n_ast) {
            AgAstRec R;
            const double* X;
            int P;
            ast = q;
            const int st = ag_ast_at(E, q / 3, tt, R, &X, &P);
            if (st != AG_OK) { if (status) atomicMax(&status[ti], st); }
            else ag_ast_sum<1>(X + (q % 3) * P, P, R.z, &h);
        }
    }
    __syncthreads();
    if (tid < 33) {
        const int b = tid / 3, k = tid - 3 * b;
        if (k == 0) o[b * 10] = E.gm[b];
        if (pst == AG_OK) {
            double x[3];
            for (int d = 0; d < 3; d++) {
                if (b == AG_EAR || b == AG_MOO)
                    x[d] = __dadd_rn(col[AG_C_EMB][k][d], __dmul_rn(col[AG_C_LUN][k][d], b == AG_EAR ? E.f_earth : E.f_moon));
                else x[d] = col[ag_col_of(b)][k][d];
            }
            const double adiv = E.pl_cau / (86400. * 86400.);
            o[b * 10 + 1 + k] = ag_div_by(x[0], E.pl_cau, E.inv_cau);
            o[b * 10 + 4 + k] = ag_div_by(x[1], E.cau_per_day, E.inv_cau_per_day);
            o[b * 10 + 7 + k] = ag_div_by(x[2], adiv, 1.0 / adiv);
        }
    } else if (tid >= 64) {
        const double nan = __longlong_as_double(0x7ff8000000000000LL);
        for (int q = tid - 64; q < 3 * E.n_ast; q += 64) {
            const int m = q / 3, k = q - 3 * m;
            if (q != ast) {
                /* more than 21 asteroids: the rest after the barrier */
                AgAstRec R;
                const double* X;
                int P;
                h = 0.0;
                const int st = ag_ast_at(E, m, tt, R, &X, &P);
                if (st != AG_OK) { if (status) atomicMax(&status[ti], st); }
                else ag_ast_sum<1>(X + k * P, P, R.z, &h);
            }
            double* r = o + (AG_NPL + m) * 10;
            if (k == 0) r[0] = E.ast_gm[m];
            r[1 + k] = __dadd_rn(h, pst == AG_OK ? sun[k] : 0.0);
            r[4 + k] = nan;
            r[7 + k] = nan;
        }
    }
}

/* ------------------------------------------------------------------ launchers */

int ag_launch_forces_table(const DevEphem& E, const ForceCfg& c, double t, const AgForceIO& io, cudaStream_t s) {
    if (io.n_real <= 0) return 0;
    const int tpb = 128;
    const int blocks = (io.n_real + tpb - 1) / tpb;
    ag_k_forces_table<<<blocks, tpb, 0, s>>>(E.self_dev, c, t, io);
    return (int)cudaGetLastError();
}

int ag_launch_forces_each(const DevEphem& E, const ForceCfg& c, int n, const double* t, const double* state,
                          const double* params, int nv, const double* var_state, double* acc, double* var_acc,
                          int* status, cudaStream_t s) {
    if (n <= 0) return 0;
    const int tpb = 128;
    const int blocks = (n + tpb - 1) / tpb;
    if (nv == 6) ag_k_forces_each<6><<<blocks, tpb, 0, s>>>(E.self_dev, c, n, t, state, params, var_state, acc, var_acc, status);
    else ag_k_forces_each<0><<<blocks, tpb, 0, s>>>(E.self_dev, c, n, t, state, params, var_state, acc, var_acc, status);
    return (int)cudaGetLastError();
}

int ag_launch_bodies(const DevEphem& E, int n, const double* t, double* out, int* status, cudaStream_t s) {
    const int nb = AG_NPL + E.n_ast;
    const int total = n * nb;
    if (total <= 0) return 0;
    if (E.pl_spk) ag_k_bodies<<<(total + 127) / 128, 128, 0, s>>>(E.self_dev, n, t, out, status);
    else if (n <= AG_BODIES_ONE) ag_k_bodies_one<<<n, 128, 0, s>>>(E.self_dev, t, out, status);
    else ag_k_bodies_tile<<<(n + 31) / 32, 128, 0, s>>>(E.self_dev, n, t, out, status);
    return (int)cudaGetLastError();
}
