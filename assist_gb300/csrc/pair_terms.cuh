/*
 * pair_terms.cuh -- direct gravity of two bodies at a time in float-pair
 * arithmetic on packed FP32 instructions.
 *
 * A float pair is an unevaluated sum hi + lo of two floats (about 48
 * significant bits).  sm_103a's packed instructions (fma/add/mul.rn.f32x2)
 * do two FP32 operations each, so one instruction stream computes the terms
 * of two bodies: a warp's FP64 instruction holds the SM's FP64 pipe for 64 to
 * 76 cycles (measured), a packed FP32 one its issue slot for two, and a term
 * is 20 FP64 instructions or 68 packed ones.  The methods are Knuth's two-sum
 * and the product error from a fused multiply-add (Dekker 1971); packed
 * operations are written as PTX with explicit rounding, which is neither
 * contracted nor reordered.
 *
 * The term of a body, -GM d / |d|^3, from y0 (the FP32 estimate of 1/|d|):
 * with delta = |d|^2 y0^2 - 1 (about 2^-21, formed from the exact products'
 * errors), 1/|d|^3 = y0^3 (1 - 3/2 delta + 15/8 delta^2).  A term's
 * relative error is at most 8e-14 where the positions' own pairs play no part
 * (bound 1.5e-13, tests/test_pair_terms.py), so below 1e-16 of the acceleration,
 * an FP64 sum's rounding, for a term of 1e-3 of the Sun's pull (the body's
 * threshold, ag_pair_thr2; nearer bodies take the FP64 term) and less for all
 * smaller ones.
 *
 * Plain C++ without CUDA (the packed operations are then two scalar ones), for
 * the test.
 */
#ifndef ASSIST_GB300_PAIR_TERMS_CUH
#define ASSIST_GB300_PAIR_TERMS_CUH

#include <cmath>

#include "ieee_convert.cuh"

/* Two floats in one 64-bit register: a (low half) and b. */
struct AgPk {
#ifdef __CUDACC__
    unsigned long long v;
#else
    float a, b;
#endif
};

#ifdef __CUDACC__
__device__ __forceinline__ AgPk ag_pk(float a, float b) {
    AgPk r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float ag_pk_a(AgPk p) {
    float a;
    asm("mov.b64 {%0, _}, %1;" : "=f"(a) : "l"(p.v));
    return a;
}
__device__ __forceinline__ float ag_pk_b(AgPk p) {
    float b;
    asm("mov.b64 {_, %0}, %1;" : "=f"(b) : "l"(p.v));
    return b;
}
__device__ __forceinline__ AgPk ag_pk_add(AgPk x, AgPk y) {
    AgPk r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(x.v), "l"(y.v));
    return r;
}
__device__ __forceinline__ AgPk ag_pk_mul(AgPk x, AgPk y) {
    AgPk r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(x.v), "l"(y.v));
    return r;
}
__device__ __forceinline__ AgPk ag_pk_fma(AgPk x, AgPk y, AgPk z) {
    AgPk r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(x.v), "l"(y.v), "l"(z.v));
    return r;
}
__device__ __forceinline__ float ag_rsqrt_est(float x) { return rsqrtf(x); }
#define AG_PT __device__ __forceinline__
#else
inline AgPk ag_pk(float a, float b) { return {a, b}; }
inline float ag_pk_a(AgPk p) { return p.a; }
inline float ag_pk_b(AgPk p) { return p.b; }
inline AgPk ag_pk_add(AgPk x, AgPk y) { return {x.a + y.a, x.b + y.b}; }
inline AgPk ag_pk_mul(AgPk x, AgPk y) { return {x.a * y.a, x.b * y.b}; }
inline AgPk ag_pk_fma(AgPk x, AgPk y, AgPk z) { return {std::fma(x.a, y.a, z.a), std::fma(x.b, y.b, z.b)}; }
inline float ag_rsqrt_est(float x) { return 1.0f / std::sqrt(x); }
#define AG_PT inline
#endif

/* x - y, exactly rounded (a fused multiply-add by -1). */
AG_PT AgPk ag_pk_sub(AgPk x, AgPk y) { return ag_pk_fma(y, ag_pk(-1.0f, -1.0f), x); }
AG_PT AgPk ag_pk_neg(AgPk x) { return ag_pk_mul(x, ag_pk(-1.0f, -1.0f)); }

/* s + e = x + y exactly. */
AG_PT AgPk ag_pk_two_sum(AgPk x, AgPk y, AgPk& e) {
    const AgPk s = ag_pk_add(x, y), bb = ag_pk_sub(s, x);
    e = ag_pk_add(ag_pk_sub(x, ag_pk_sub(s, bb)), ag_pk_sub(y, bb));
    return s;
}

/* One component of two bodies' positions relative to the origin, hi and lo
 * parts packed (a 16-byte load). */
struct alignas(16) AgPkComp {
    AgPk h, l;
};
/* Two bodies: origin minus body, and their GM and threshold (ag_pair_thr2). */
struct AgPkRel {
    AgPkComp c[3];
};
struct alignas(16) AgPkGm {
    AgPk h, l;
    float ta, tb;
    float ga, gb;          /* GM in FP32 (the potential of the relativistic term) */
};

/* The smallest squared distance, over the particle's squared heliocentric
 * distance, at which a body of mass m (in solar masses) takes the pair term.
 * The pair's relative error (at most 8e-14) asks for a share m (r/d)^2 of the
 * Sun's pull below 1e-3; the separation's absolute error, about 3e-15 r rms with
 * the term's slope, for m (r/d)^3 below 1/150: 2e-17 of the acceleration rms.
 * The whole evaluation's error is no larger than with every term in FP64:
 * over 16 distances from the Sun and 49 from the planets, each 200 to 300
 * particles, 0.98 of it for shared times and 1.00 for own times (rms against
 * double-double; tests/test_gpu_rounding.py holds the single terms). */
inline float ag_pair_thr2(double m) {
    const double a = m / 1e-3, b = std::pow(150.0 * m, 2.0 / 3.0);
    return (float)(a > b ? a : b);
}

/* The same with its Jacobian, whose share m (r/d)^3 of the Sun's is larger: at
 * most 1/400 for the term's relative error, m (r/d)^4 at most 1/120 for the
 * separation's (1.5e-15 r rms with a slope of 4), each then 5e-17 rms of the
 * Jacobian, whose FP64 rounding is 3e-16.  With the acceleration's limits alone
 * it was 9e-16 at 0.6 AU of Pluto. */
inline float ag_pair_thr2_jac(double m) {
    const double a = std::pow(400.0 * m, 2.0 / 3.0), b = std::sqrt(120.0 * m), c = (double)ag_pair_thr2(m);
    return (float)(a > b ? (a > c ? a : c) : (b > c ? b : c));
}

/* Running sum of packed pair terms: hi and lo per component. */
struct AgPkSum {
    AgPk h[3], l[3];
};

/* Running sum of the terms' Jacobian (src/forces.c: 3 GM d d^T / r^5 - GM I /
 * r^3): its symmetric part xx, xy, xz, yy, yz, zz, times 2^40 (the low parts of
 * GM / r^5 far from a light body would leave FP32's normal range), and the sum
 * of GM / r^3. */
#define AG_PK_JSCALE 0x1p40f
struct AgPkJac {
    AgPk h[7], l[7];
};
AG_PT void ag_pk_jac_clear(AgPkJac& J) {
#pragma unroll
    for (int k = 0; k < 7; k++) J.h[k] = J.l[k] = ag_pk(0.0f, 0.0f);
}
/* Element k of half a (0) or b (1) without the factor. */
AG_PT void ag_pk_jac_get(const AgPkJac& J, int k, int half, float& h, float& l) {
    const float s = k < 6 ? 1.0f / AG_PK_JSCALE : 1.0f;
    h = s * (half ? ag_pk_b(J.h[k]) : ag_pk_a(J.h[k]));
    l = s * (half ? ag_pk_b(J.l[k]) : ag_pk_a(J.l[k]));
}

/* (h, l) += x y for the pairs x = xh + xl, y = yh + yl. */
AG_PT void ag_pk_acc(AgPk xh, AgPk xl, AgPk yh, AgPk yl, AgPk& h, AgPk& l) {
    const AgPk p = ag_pk_mul(xh, yh);
    AgPk pe = ag_pk_fma(xh, yh, ag_pk_neg(p));
    pe = ag_pk_fma(xh, yl, pe);
    pe = ag_pk_fma(xl, yh, pe);
    AgPk e;
    h = ag_pk_two_sum(h, p, e);
    l = ag_pk_add(l, ag_pk_add(e, pe));
}

/* Adds the terms of the two bodies of R to S at the position xh + xl
 * (packed: the same value in both halves); rs2: squared heliocentric distance
 * (FP32).  Returns bit 0 / bit 1 set for a body below its threshold (or not
 * finite), whose term is left out.  JAC: their Jacobian into J too. */
template <bool JAC = false>
AG_PT unsigned ag_pk_term(const AgPkRel& R, const AgPkGm& G, const AgPk* xh, const AgPk* xl, float rs2, AgPkSum& S,
                          AgPkJac* J = nullptr) {
    const AgPk m1 = ag_pk(-1.0f, -1.0f);
    AgPk dh[3], dl[3], p[3], ne[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const AgPkComp c = R.c[k];
        AgPk e;
        const AgPk s = ag_pk_two_sum(xh[k], c.h, e);
        e = ag_pk_add(e, ag_pk_add(xl[k], c.l));
        dh[k] = ag_pk_add(s, e);
        dl[k] = ag_pk_sub(e, ag_pk_sub(dh[k], s));
        /* d^2 = p - ne */
        const AgPk nd = ag_pk_mul(dh[k], m1);
        p[k] = ag_pk_mul(dh[k], dh[k]);
        ne[k] = ag_pk_fma(ag_pk_add(nd, nd), dl[k], ag_pk_fma(dh[k], nd, p[k]));
    }
    AgPk t1, t2;
    const AgPk r2 = ag_pk_two_sum(ag_pk_two_sum(p[0], p[1], t1), p[2], t2);
    const AgPk r2l = ag_pk_sub(ag_pk_add(t1, t2), ag_pk_add(ag_pk_add(ne[0], ne[1]), ne[2]));
    const float ra = ag_pk_a(r2), rb = ag_pk_b(r2);
    const bool na = !(ra >= G.ta * rs2 && ra < 1e30f), nb = !(rb >= G.tb * rs2 && rb < 1e30f);
    const AgPk y = ag_pk(ag_rsqrt_est(ra), ag_rsqrt_est(rb)), ny = ag_pk_mul(y, m1);
    /* y^2 = q - nqe, r2 q = th - nte, delta = |d|^2 y^2 - 1 */
    const AgPk q = ag_pk_mul(y, y), nqe = ag_pk_fma(y, ny, q), nq = ag_pk_mul(q, m1);
    const AgPk th = ag_pk_mul(r2, q), nte = ag_pk_fma(r2, nq, th);
    AgPk del = ag_pk_sub(ag_pk_add(th, m1), nte);
    del = ag_pk_fma(r2, ag_pk_mul(nqe, m1), del);
    del = ag_pk_fma(r2l, q, del);
    const AgPk corr = ag_pk_mul(del, ag_pk_fma(del, ag_pk(1.875f, 1.875f), ag_pk(-1.5f, -1.5f)));
    /* GM y = w - nwe, GM y^3 = g - ne3, both with the correction: G = -GM / |d|^3 = gh + gl */
    const AgPk w = ag_pk_mul(G.h, y);
    const AgPk nwe = ag_pk_sub(ag_pk_fma(G.h, ny, w), ag_pk_mul(G.l, y));
    const AgPk g = ag_pk_mul(w, q);
    AgPk gl = ag_pk_fma(w, nq, g);
    gl = ag_pk_fma(w, nqe, gl);
    gl = ag_pk_fma(nwe, q, gl);
    AgPk gh = ag_pk_mul(g, m1);
    gl = ag_pk_fma(gh, corr, gl);
    gh = ag_pk(na ? 0.0f : ag_pk_a(gh), nb ? 0.0f : ag_pk_b(gh));
    gl = ag_pk(na ? 0.0f : ag_pk_a(gl), nb ? 0.0f : ag_pk_b(gl));
#pragma unroll
    for (int k = 0; k < 3; k++) ag_pk_acc(gh, gl, dh[k], dl[k], S.h[k], S.l[k]);
    if (JAC) {
        /* f = -3 G / |d|^2 with 1 / |d|^2 = y^2 (1 - delta + delta^2); e = f d */
        const AgPk m3 = ag_pk(-3.0f, -3.0f);
        const AgPk c2 = ag_pk_mul(del, ag_pk_sub(del, ag_pk(1.0f, 1.0f)));
        const AgPk sc = ag_pk(AG_PK_JSCALE, AG_PK_JSCALE);
        const AgPk ih = ag_pk_mul(q, sc), il = ag_pk_mul(ag_pk_sub(ag_pk_mul(q, c2), nqe), sc);
        const AgPk g3h = ag_pk_mul(gh, m3), g3l = ag_pk_fma(gl, m3, ag_pk_fma(gh, m3, ag_pk_neg(g3h)));
        const AgPk fh = ag_pk_mul(g3h, ih);
        AgPk fl = ag_pk_fma(g3h, ih, ag_pk_neg(fh));
        fl = ag_pk_fma(g3h, il, fl);
        fl = ag_pk_fma(g3l, ih, fl);
        int at = 0;
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const AgPk eh = ag_pk_mul(fh, dh[a]);
            AgPk el = ag_pk_fma(fh, dh[a], ag_pk_neg(eh));
            el = ag_pk_fma(fh, dl[a], el);
            el = ag_pk_fma(fl, dh[a], el);
#pragma unroll
            for (int b = a; b < 3; b++, at++) ag_pk_acc(eh, el, dh[b], dl[b], J->h[at], J->l[at]);
        }
        AgPk e;
        J->h[6] = ag_pk_two_sum(J->h[6], ag_pk_neg(gh), e);
        J->l[6] = ag_pk_add(J->l[6], ag_pk_sub(e, gl));
    }
    return (na ? 1u : 0u) | (nb ? 2u : 0u);
}

#endif
