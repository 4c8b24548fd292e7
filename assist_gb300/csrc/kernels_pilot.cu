/*
 * kernels_pilot.cu -- expected close-encounter cost of each particle, which
 * orders the grouped batched kernels' work queue, and its deep passes, which
 * choose a group's kernel (below).
 *
 * A group of particles steps at the smallest step any member needs, and a
 * member passing close to a planet needs many small steps: such a group runs
 * several times longer than its orbit class suggests.  Queued late, it is
 * still running after every other block has gone idle.  This pilot
 * estimates, per particle, the extra steps of its encounters from a
 * two-body (heliocentric Kepler) propagation sampled on a time grid against
 * the planets' ephemeris positions.  With the local dynamical rate
 * w = sqrt(GM / d^3) of the Sun (heliocentric distance) and of each planet
 * (distance to it),
 *     base  = sum over samples of w_sun,
 *     extra = sum over samples of max(0, max_k w_k - w_sun),
 * and the result is extra / base: the fraction of steps the encounters add.
 * The grouping multiplies a particle's cost estimate by (1 + extra / base).
 * Integration results do not depend on the queue order, only the time the
 * batch takes does.  The arithmetic is FP32 (a ranking, not a trajectory);
 * the orbital elements are formed in FP64.
 *
 * For a particle that may come close to a planet the pilot then looks for a
 * deep pass: whether its path comes within AG_DEEP of a planet's radius of
 * influence, r_k (GM_k / GM_sun)^(1/3) (ag_k_deep).  Such a pass amplifies
 * rounding until the end state hangs on every operation's last bit; the batch
 * keeps groups with such a particle on the kernel with all terms in FP64, so
 * that this part of the pilot does choose their arithmetic.
 */
#include <cuda_runtime.h>

#include "device_ephem.cuh"
#include "internal.h"

/* Bodies sampled on the grid: the Sun (barycentric, to make the particles
 * heliocentric) and the planets except the Moon (its pull is a 1/81 share of
 * the Earth's, at the same place). */
#define AG_PILOT_NB 10
__constant__ int ag_pilot_body[AG_PILOT_NB] = {AG_SUN, AG_MER, AG_VEN, AG_EAR, AG_MAR,
                                               AG_JUP, AG_SAT, AG_URA, AG_NEP, AG_PLU};

/* grid[i * NB + b]: body b at time tmin + i * dtg; the Sun barycentric
 * (x, y, z, and vx in w; vy, vz follow in sunv), planets heliocentric. */
__global__ void ag_k_pilot_grid(const DevEphem* __restrict__ Ep, double tmin, double dtg, int G, float4* grid,
                                float2* sunv) {
    const DevEphem& E = *Ep;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= G) return;
    const double t = tmin + dtg * q;
    double s[10] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, o[10];
    const bool ok = ag_planet_full(E, AG_SUN, t, s) == AG_OK;
    grid[(size_t)q * AG_PILOT_NB] = make_float4((float)s[1], (float)s[2], (float)s[3], (float)s[4]);
    sunv[q] = make_float2((float)s[5], (float)s[6]);
    for (int b = 1; b < AG_PILOT_NB; b++) {
        float4 p = make_float4(1e30f, 1e30f, 1e30f, 0.0f);       /* off the ephemeris: far away */
        if (ok && ag_planet_full(E, ag_pilot_body[b], t, o) == AG_OK)
            p = make_float4((float)(o[1] - s[1]), (float)(o[2] - s[2]), (float)(o[3] - s[3]), 0.0f);
        grid[(size_t)q * AG_PILOT_NB + b] = p;
    }
}

/* ---------------------------------------------------------------- deep passes
 *
 * The path under the Sun and the planets, by Runge-Kutta steps in FP32 with
 * compensated sums, four lanes a particle with two or three planets each.
 * Barycentric, with the ephemeris's Sun, as the integrators have it.  The
 * samples are at most AG_DEEP_DAYS apart whatever the batch spans, with
 * velocities (cubic Hermite between them: 4e-7 AU for Mercury, the worst); a
 * step is short enough to see every approach (a quarter of the time to reach a
 * planet at the present rate). */

/* Distance over the radius of influence below which a pass is deep.  Of 20
 * million particle-years of a main-belt/NEO/Trojan/TNO mixture, the particles
 * whose end states move by more than 1e4 times a change of their start came
 * within 0.025 (all of them plunging into Jupiter); the rest is for the path's
 * own error: 0.035 of the radius is 5e-4 AU at the Earth, where the path of a
 * near-Earth orbit is off by up to 3e-5 AU after a year and 2e-4 after thirty.
 * 5 to 15 in 65,536 of the mixture come within 0.06 in a year, by the system
 * drawn. */
#define AG_DEEP 0.06f
#define AG_DEEP_DAYS 2.0
#define AG_DEEP_MAX_G 65536
#define AG_DEEP_LANES 4

int ag_pilot_deep_samples(double span) {
    const double g = ceil(fabs(span) / AG_DEEP_DAYS) + 1.0;
    return g < 2.0 ? 2 : (g < (double)AG_DEEP_MAX_G ? (int)g : AG_DEEP_MAX_G);
}

/* grid[2 (q NB + b)], + 1: body b, barycentric, at time tmin + q dt as
 * (x, y, z, vx), (vy, vz), velocities per sample. */
__global__ void ag_k_deep_grid(const DevEphem* __restrict__ Ep, double tmin, double dt, int G, float4* grid) {
    const DevEphem& E = *Ep;
    const int at = blockIdx.x * blockDim.x + threadIdx.x;
    if (at >= G * AG_PILOT_NB) return;
    const int q = at / AG_PILOT_NB, b = at - q * AG_PILOT_NB;
    double o[10];
    float4 p = make_float4(1e30f, 1e30f, 1e30f, 0.0f), v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);   /* off the ephemeris: far away */
    if (ag_planet_full(E, ag_pilot_body[b], tmin + dt * q, o) == AG_OK) {
        p = make_float4((float)o[1], (float)o[2], (float)o[3], (float)(dt * o[4]));
        v = make_float4((float)(dt * o[5]), (float)(dt * o[6]), 0.0f, 0.0f);
    }
    grid[2 * (size_t)at] = p;
    grid[2 * (size_t)at + 1] = v;
}

/* Body b at sample j + u: position and velocity (per sample). */
__device__ __forceinline__ void ag_deep_body(const float4* __restrict__ grid, int b, int j, float u, float* P, float* V) {
    const float4* g = grid + 2 * ((size_t)j * AG_PILOT_NB + b);
    const float4 a = g[0], va = g[1], c = g[2 * AG_PILOT_NB], vc = g[2 * AG_PILOT_NB + 1];
    const float A[3] = {a.x, a.y, a.z}, B[3] = {c.x, c.y, c.z}, W[3] = {a.w, va.x, va.y}, Y[3] = {c.w, vc.x, vc.y};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float d = B[k] - A[k];
        P[k] = fmaf(u, fmaf(u, fmaf(u, W[k] + Y[k] - 2.0f * d, 3.0f * d - 2.0f * W[k] - Y[k]), W[k]), A[k]);
        V[k] = fmaf(u, Y[k] - W[k], W[k]);
    }
}

/* Acceleration at p, sample j + u, by the Sun and all planets, from the lane's
 * own and its neighbours' (every lane of the warp calls it).  END: with the
 * velocity w also the largest GM / d^3 of any body, the smallest time to reach
 * a planet at the present rate and the smallest distance to one over its
 * radius of influence. */
template <bool END>
__device__ __forceinline__ void ag_deep_acc(const float4* __restrict__ grid, int G, float idt, const float* gm, float mu, int sub,
                                            const float* p, const float* w, int j, float u, float* a, float& w2, float& reach,
                                            float& q) {
    constexpr int MINE = (AG_PILOT_NB - 1 + AG_DEEP_LANES - 1) / AG_DEEP_LANES;
    const float* isoi = gm + MINE;                 /* (GM_sun / GM_k)^(1/3) */
    const int jj = j < 0 ? 0 : (j > G - 2 ? G - 2 : j);
    const float uu = u + (float)(j - jj);
    float S[3], V[3], s[3] = {0.0f, 0.0f, 0.0f};
    ag_deep_body(grid, 0, jj, uu, S, V);
    const float r[3] = {S[0] - p[0], S[1] - p[1], S[2] - p[2]};
    const float ri = rsqrtf(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]), ws = mu * ri * ri * ri;
    if (END) { w2 = ws; reach = 1e30f; q = 1e30f; }
#pragma unroll
    for (int m = 0; m < MINE; m++) {
        const int b = 1 + sub + m * AG_DEEP_LANES;
        if (b >= AG_PILOT_NB) continue;
        float P[3];
        ag_deep_body(grid, b, jj, uu, P, V);
        const float d[3] = {P[0] - p[0], P[1] - p[1], P[2] - p[2]};
        const float d2 = fmaxf(d[0] * d[0] + d[1] * d[1] + d[2] * d[2], 1e-10f);
        const float di = rsqrtf(d2), fd = gm[m] * di * di * di;
#pragma unroll
        for (int k = 0; k < 3; k++) s[k] += fd * d[k];
        if (END) {
            const float e[3] = {V[0] * idt - w[0], V[1] * idt - w[1], V[2] * idt - w[2]};
            const float h[3] = {P[0] - S[0], P[1] - S[1], P[2] - S[2]};
            w2 = fmaxf(w2, fd);
            reach = fminf(reach, d2 * di * rsqrtf(e[0] * e[0] + e[1] * e[1] + e[2] * e[2]));
            q = fminf(q, d2 * di * rsqrtf(h[0] * h[0] + h[1] * h[1] + h[2] * h[2]) * isoi[m]);
        }
    }
#pragma unroll
    for (int o = 1; o < AG_DEEP_LANES; o <<= 1) {
#pragma unroll
        for (int k = 0; k < 3; k++) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
        if (END) {
            w2 = fmaxf(w2, __shfl_xor_sync(0xffffffffu, w2, o));
            reach = fminf(reach, __shfl_xor_sync(0xffffffffu, reach, o));
            q = fminf(q, __shfl_xor_sync(0xffffffffu, q, o));
        }
    }
#pragma unroll
    for (int k = 0; k < 3; k++) a[k] = fmaf(ws, r[k], s[k]);
}

/* x += d with the rounding kept in c. */
__device__ __forceinline__ void ag_deep_sum(float& x, float& c, float d) {
    const float y = __fsub_rn(d, c), t = __fadd_rn(x, y);
    c = __fsub_rn(__fsub_rn(t, x), y);
    x = t;
}

/* deep[i] of the particles list[1 .. list[0]]: whether the path from t0 to te
 * passes a planet deep inside its sphere of influence; 1 too when the step
 * limit ends the search (a satellite's orbit). */
__global__ void __launch_bounds__(128) ag_k_deep(const DevEphem* __restrict__ Ep, const double* __restrict__ t0,
                                                 const double* __restrict__ te, const double* __restrict__ state,
                                                 const float4* __restrict__ grid, int G, double tmin, double dt,
                                                 const int* __restrict__ list, unsigned char* deep) {
    constexpr int MINE = (AG_PILOT_NB - 1 + AG_DEEP_LANES - 1) / AG_DEEP_LANES;
    const DevEphem& E = *Ep;
    const int at = (int)((blockIdx.x * blockDim.x + threadIdx.x) / AG_DEEP_LANES), sub = threadIdx.x & (AG_DEEP_LANES - 1);
    const int count = list[0];
    if (at - (int)(threadIdx.x & 31) / AG_DEEP_LANES >= count) return;         /* the whole warp */
    bool run = at < count;
    const int i = list[1 + (run ? at : count - 1)];
    const float mu = (float)E.gm[AG_SUN], idt = (float)(1.0 / dt);
    float gm[2 * MINE];
    for (int m = 0; m < MINE; m++) {
        const int b = 1 + sub + m * AG_DEEP_LANES, body = b < AG_PILOT_NB ? ag_pilot_body[b] : AG_PLU;
        gm[m] = (float)(E.gm[body] + (body == AG_EAR ? E.gm[AG_MOO] : 0.0));
        gm[MINE + m] = cbrtf(mu / gm[m]);
    }
    /* times as sample and fraction */
    const double ta = t0[i], tb = te[i], fa = (ta - tmin) / dt, fb = (tb - tmin) / dt;
    int j = (int)floor(fa);
    const int jb = (int)floor(fb);
    float u = (float)(fa - j);
    const float ub = (float)(fb - jb), sgn = tb >= ta ? 1.0f : -1.0f, span = (float)fabs(tb - ta);
    float x[3], w[3], cx[3], cw[3], a[3], w2, reach, q;
    for (int k = 0; k < 3; k++) {
        const double xk = state[6 * (size_t)i + k], wk = state[6 * (size_t)i + 3 + k];
        x[k] = (float)xk; cx[k] = (float)((double)x[k] - xk);
        w[k] = (float)wk; cw[k] = (float)((double)w[k] - wk);
    }
    /* the path's error grows with its length: shorter steps beyond three years */
    const float c = 0.1f * fminf(1.0f, cbrtf(1000.0f / fmaxf(span, 1.0f)));
    const int limit = 1000 + (int)fminf(2.0f * span, 60000.0f);
    int found = 0;
    ag_deep_acc<true>(grid, G, idt, gm, mu, sub, x, w, j, u, a, w2, reach, q);
    /* the warp's lanes leave the loop together (its shuffles are the whole warp's) */
    for (int s = 0;; s++) {
        if (run && (s == limit || q < AG_DEEP)) { found = 1; run = false; }
        const float rem = sgn * ((float)(jb - j) + (ub - u)) * (float)dt, h = fminf(fminf(c * rsqrtf(w2), 0.25f * reach), rem);
        if (!(h > 0.0f)) run = false;
        if (!__any_sync(0xffffffffu, run)) break;
        const float hs = run ? sgn * h : 0.0f;
        float k2[3], k3[3], k4[3], p[3], v2[3], v3[3], v4[3], n0, n1, n2;
        auto when = [&](float f, int& jj) {        /* u + f hs, j carried along */
            const float y = fmaf(f * hs, idt, u), fl = floorf(y);
            jj = j + (int)fl;
            return y - fl;
        };
        int jm, je;
        const float um = when(0.5f, jm);
        float ue = when(1.0f, je);
        if (run && !(h < rem)) { je = jb; ue = ub; }
        for (int k = 0; k < 3; k++) { p[k] = x[k] + 0.5f * hs * w[k]; v2[k] = w[k] + 0.5f * hs * a[k]; }
        ag_deep_acc<false>(grid, G, idt, gm, mu, sub, p, v2, jm, um, k2, n0, n1, n2);
        for (int k = 0; k < 3; k++) { p[k] = x[k] + 0.5f * hs * v2[k]; v3[k] = w[k] + 0.5f * hs * k2[k]; }
        ag_deep_acc<false>(grid, G, idt, gm, mu, sub, p, v3, jm, um, k3, n0, n1, n2);
        for (int k = 0; k < 3; k++) { p[k] = x[k] + hs * v3[k]; v4[k] = w[k] + hs * k3[k]; }
        ag_deep_acc<false>(grid, G, idt, gm, mu, sub, p, v4, je, ue, k4, n0, n1, n2);
        for (int k = 0; k < 3; k++) {
            ag_deep_sum(x[k], cx[k], hs / 6.0f * (w[k] + 2.0f * v2[k] + 2.0f * v3[k] + v4[k]) - hs * cw[k]);
            ag_deep_sum(w[k], cw[k], hs / 6.0f * (a[k] + 2.0f * k2[k] + 2.0f * k3[k] + k4[k]));
        }
        j = je;
        u = ue;
        ag_deep_acc<true>(grid, G, idt, gm, mu, sub, x, w, j, u, a, w2, reach, q);
    }
    if (found && sub == 0) deep[i] = 1;
}

/* The ratios; DEEP: also list[1 .. list[0]] (list[0] zero before), the
 * particles that ag_k_deep looks at: every one but those whose two-body path
 * stays clear of the planets by what the samples' spacing and the planets'
 * pull may hide. */
template <bool DEEP>
__global__ void ag_k_pilot(const DevEphem* __restrict__ Ep, int n, const double* __restrict__ t0,
                           const double* __restrict__ te, const double* __restrict__ state, const float4* __restrict__ grid,
                           const float2* __restrict__ sunv, int G, double tmin, double dtg, float* ratio,
                           unsigned char* deep, int* list) {
    const DevEphem& E = *Ep;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    ratio[i] = 0.0f;
    if (DEEP) deep[i] = 0;
    auto look = [&] {
        if (DEEP) list[1 + atomicAdd(&list[0], 1)] = i;
    };
    const double ta = t0[i], tb = te[i];
    /* the Sun at t0, linear between grid points */
    double f = (ta - tmin) / dtg;
    int g0 = (int)floor(f);
    g0 = g0 < 0 ? 0 : (g0 > G - 2 ? G - 2 : g0);
    f -= g0;
    const float4 sa = grid[(size_t)g0 * AG_PILOT_NB], sb = grid[(size_t)(g0 + 1) * AG_PILOT_NB];
    const float2 va = sunv[g0], vb = sunv[g0 + 1];
    const double sx = sa.x + f * (sb.x - sa.x), sy = sa.y + f * (sb.y - sa.y), sz = sa.z + f * (sb.z - sa.z);
    const double svx = sa.w + f * (sb.w - sa.w), svy = va.x + f * (vb.x - va.x), svz = va.y + f * (vb.y - va.y);
    const double* s0 = state + 6 * (size_t)i;
    const double r[3] = {s0[0] - sx, s0[1] - sy, s0[2] - sz};
    const double v[3] = {s0[3] - svx, s0[4] - svy, s0[5] - svz};
    const double mu = E.gm[AG_SUN];
    /* elliptic elements; other orbits keep the plain estimate */
    const double rn = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
    const double v2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
    const double rv = r[0] * v[0] + r[1] * v[1] + r[2] * v[2];
    const double inv_a = 2.0 / rn - v2 / mu;
    const float musun = (float)mu;
    float gmk[AG_PILOT_NB];
    for (int b = 1; b < AG_PILOT_NB; b++) gmk[b] = (float)E.gm[ag_pilot_body[b]];
    /* not an ellipse about the Sun: perhaps bound to a planet */
    if (!(inv_a > 0.0) || !(rn > 0.0)) return look();
    const double a = 1.0 / inv_a;
    double ev[3];
    for (int k = 0; k < 3; k++) ev[k] = ((v2 - mu / rn) * r[k] - rv * v[k]) / mu;
    const double e = sqrt(ev[0] * ev[0] + ev[1] * ev[1] + ev[2] * ev[2]);
    if (!(e < 0.98)) return look();
    const double h[3] = {r[1] * v[2] - r[2] * v[1], r[2] * v[0] - r[0] * v[2], r[0] * v[1] - r[1] * v[0]};
    const double hn = sqrt(h[0] * h[0] + h[1] * h[1] + h[2] * h[2]);
    if (!(hn > 0.0)) return look();
    /* perifocal frame: P toward pericentre (toward r for a circular orbit), Q = h x P / |h| */
    double P[3];
    if (e > 1e-8) { for (int k = 0; k < 3; k++) P[k] = ev[k] / e; }
    else { for (int k = 0; k < 3; k++) P[k] = r[k] / rn; }
    const double Q[3] = {(h[1] * P[2] - h[2] * P[1]) / hn, (h[2] * P[0] - h[0] * P[2]) / hn,
                         (h[0] * P[1] - h[1] * P[0]) / hn};
    /* eccentric and mean anomaly at t0 (from the perifocal coordinates of r) */
    const double xp = r[0] * P[0] + r[1] * P[1] + r[2] * P[2], yp = r[0] * Q[0] + r[1] * Q[1] + r[2] * Q[2];
    const double be = sqrt(1.0 - e * e);
    const double E0 = atan2(yp / (a * be), xp / a + e);
    const double M0 = E0 - e * sin(E0);
    const double nmot = sqrt(mu * inv_a) * inv_a;
    /* grid samples inside the integration interval */
    const double lo = fmin(ta, tb), hi = fmax(ta, tb);
    int i0 = (int)ceil((lo - tmin) / dtg), i1 = (int)floor((hi - tmin) / dtg);
    i0 = i0 < 0 ? 0 : i0;
    i1 = i1 > G - 1 ? G - 1 : i1;
    if (i1 < i0) return look();
    /* twice a planet's radius of influence, its distance from the Sun at most
     * half as large again as at the first sample */
    bool near = false;
    float rb[AG_PILOT_NB];
    if (DEEP)
        for (int b = 1; b < AG_PILOT_NB; b++) {
            const float4 pb = grid[(size_t)i0 * AG_PILOT_NB + b];
            rb[b] = 3.0f * sqrtf(pb.x * pb.x + pb.y * pb.y + pb.z * pb.z) * cbrtf(gmk[b] / musun);
        }
    const float fa = (float)a, fe = (float)e, fb = (float)(a * be);
    const float Pf[3] = {(float)P[0], (float)P[1], (float)P[2]}, Qf[3] = {(float)Q[0], (float)Q[1], (float)Q[2]};
    float base = 0.0f, extra = 0.0f;
    /* mean anomaly at the first sample in FP64, then FP32 increments (the
     * loop stays off the FP64 pipe) */
    const double twopi = 6.283185307179586;
    double Ms = M0 + nmot * ((tmin + dtg * i0) - ta);
    Ms -= twopi * floor(Ms / twopi);
    const float Mstart = (float)Ms, dM = (float)(nmot * dtg), tpf = 6.2831853f, itpf = 1.0f / 6.2831853f;
    for (int q = i0; q <= i1; q++) {
        float Mf = fmaf((float)(q - i0), dM, Mstart);
        Mf -= tpf * floorf(Mf * itpf);
        float Ea = Mf + fe * __sinf(Mf);
        for (int it = 0; it < 6; it++) {
            float sE, cE;
            __sincosf(Ea, &sE, &cE);
            Ea -= (Ea - fe * sE - Mf) / (1.0f - fe * cE);
        }
        float sE, cE;
        __sincosf(Ea, &sE, &cE);
        const float xo = fa * (cE - fe), yo = fb * sE;
        const float px = xo * Pf[0] + yo * Qf[0], py = xo * Pf[1] + yo * Qf[1], pz = xo * Pf[2] + yo * Qf[2];
        const float r2 = px * px + py * py + pz * pz;
        const float wsun = sqrtf(musun / (r2 * sqrtf(r2)));
        float wmax = 0.0f;
        const float4* gq = grid + (size_t)q * AG_PILOT_NB;
        /* what the spacing hides: the escape and the circular speed there
         * together, for one spacing (the ends lie off the samples); what the
         * planets' pull moves the path by: 2.8e-7 AU/day^2, Jupiter's at 1 AU */
        const float ago = fabsf((float)((tmin + dtg * q) - ta));
        const float hide = 2.42f * wsun * sqrtf(r2) * (float)dtg + 1.4e-7f * ago * ago;
#pragma unroll
        for (int b = 1; b < AG_PILOT_NB; b++) {
            const float4 pb = gq[b];
            const float dx = px - pb.x, dy = py - pb.y, dz = pz - pb.z;
            const float d2 = fmaxf(dx * dx + dy * dy + dz * dz, 1e-16f);
            wmax = fmaxf(wmax, sqrtf(gmk[b] / (d2 * sqrtf(d2))));
            if (DEEP) near = near || d2 < (rb[b] + hide) * (rb[b] + hide);
        }
        base += wsun;
        extra += fmaxf(0.0f, wmax - wsun);
    }
    if (base > 0.0f && isfinite(extra)) ratio[i] = extra / base;
    if (near) look();
}

int ag_pilot_encounters(const DevEphem& E, int n, const double* d_t0, const double* d_te, const double* d_state,
                        double tmin, double tmax, const AgPilotBuf& B, cudaStream_t s) {
    if (n <= 0) return 0;
    const int G = AG_PILOT_G, GD = ag_pilot_deep_samples(tmax - tmin);
    const double dtg = (tmax - tmin) / (G - 1), dtd = (tmax - tmin) / (GD - 1);
    if (!(dtg > 0.0)) {
        if (B.deep) cudaMemsetAsync(B.deep, 0, (size_t)n, s);
        return (int)cudaMemsetAsync(B.ratio, 0, sizeof(float) * (size_t)n, s);
    }
    ag_k_pilot_grid<<<(G + 127) / 128, 128, 0, s>>>(E.self_dev, tmin, dtg, G, B.grid, B.sunv);
    if (!B.deep) {
        ag_k_pilot<false><<<(n + 127) / 128, 128, 0, s>>>(E.self_dev, n, d_t0, d_te, d_state, B.grid, B.sunv, G, tmin, dtg, B.ratio,
                                                          nullptr, nullptr);
        return (int)cudaGetLastError();
    }
    cudaMemsetAsync(B.list, 0, sizeof(int), s);
    ag_k_pilot<true><<<(n + 127) / 128, 128, 0, s>>>(E.self_dev, n, d_t0, d_te, d_state, B.grid, B.sunv, G, tmin, dtg, B.ratio, B.deep,
                                                     B.list);
    ag_k_deep_grid<<<(GD * AG_PILOT_NB + 127) / 128, 128, 0, s>>>(E.self_dev, tmin, dtd, GD, B.dgrid);
    const int per = 128 / AG_DEEP_LANES;
    ag_k_deep<<<(n + per - 1) / per, 128, 0, s>>>(E.self_dev, d_t0, d_te, d_state, B.dgrid, GD, tmin, dtd, B.list, B.deep);
    return (int)cudaGetLastError();
}
