"""The packed float-pair gravity terms (assist_gb300/csrc/pair_terms.cuh)
against long double on the CPU: the header is plain C++ without CUDA, so g++
compiles the check.  Bound of a term's relative error: the correction's
rounding, 1.5 x four roundings at 2^-21 x 2^-24, and those of the products'
low parts, together below 1.5e-13; the positions' pairs, 2^-48 of the
positions' size R each way, times the term's slope of 3 over d."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include "pair_terms.cuh"
#include <cstdio>
#include <random>
int main() {
    std::mt19937_64 rng(1);
    std::uniform_real_distribution<double> U(-1, 1);
    int bad = 0;
    long n = 0;
    const double dist[] = {0.02, 0.1, 1.0, 7.0, 40.0, 500.0}, size[] = {0.3, 2.5, 30.0}, mass[] = {1e-19, 3e-15, 8e-10, 8.5e-8};
    for (double D : dist) for (double R : size) for (double gm : mass) for (int i = 0; i < 4000; i++) {
        AgPkRel A;
        AgPk xh[3], xl[3];
        AgPkSum S;
        double x[3], b[2][3];
        float h[2], l[2];
        for (int k = 0; k < 3; k++) x[k] = R * U(rng);
        for (int j = 0; j < 2; j++) {
            double u[3], nu = 0;
            for (int k = 0; k < 3; k++) { u[k] = U(rng); nu += u[k] * u[k]; }
            for (int k = 0; k < 3; k++) b[j][k] = x[k] - (j ? 3.0 : 1.0) * D * u[k] / std::sqrt(nu);
        }
        for (int k = 0; k < 3; k++) {
            for (int j = 0; j < 2; j++) { h[j] = (float)-b[j][k]; l[j] = (float)(-b[j][k] - h[j]); }
            A.c[k].h = ag_pk(h[0], h[1]); A.c[k].l = ag_pk(l[0], l[1]);
            h[0] = (float)x[k]; l[0] = (float)(x[k] - h[0]);
            xh[k] = ag_pk(h[0], h[0]); xl[k] = ag_pk(l[0], l[0]);
            S.h[k] = S.l[k] = ag_pk(0.0f, 0.0f);
        }
        AgPkGm G;
        h[0] = (float)gm; l[0] = (float)(gm - h[0]);
        G.h = ag_pk(h[0], h[0]); G.l = ag_pk(l[0], l[0]);
        G.ta = G.tb = 0.0f;
        AgPkJac J;
        ag_pk_jac_clear(J);
        if (ag_pk_term<true>(A, G, xh, xl, 1.0f, S, &J) != 0) bad++;
        for (int j = 0; j < 2; j++) {
            /* Jacobian: the term's bound with its slope of 5 over d, per element over its norm */
            {
                long double d[3], r2 = 0, t[7], e2 = 0, t2 = 0;
                for (int k = 0; k < 3; k++) { d[k] = (long double)x[k] - b[j][k]; r2 += d[k] * d[k]; }
                const long double g = (long double)gm / (r2 * sqrtl(r2));
                int at = 0;
                for (int a = 0; a < 3; a++) for (int c = a; c < 3; c++) t[at++] = 3 * g * d[a] * d[c] / r2;
                t[6] = g;
                for (int k = 0; k < 7; k++) {
                    float jh, jl;
                    ag_pk_jac_get(J, k, j, jh, jl);
                    const long double v = (long double)jh + jl;
                    e2 += (v - t[k]) * (v - t[k]); t2 += t[k] * t[k];
                }
                const double far = R + (j ? 3.0 : 1.0) * D;
                if (!((double)sqrtl(e2 / t2) < 2.5e-13 + 5.0 * 2.0 * 0x1p-48 * far / ((j ? 3.0 : 1.0) * D))) { std::printf("jacobian d %g: %g\n", D, (double)sqrtl(e2 / t2)); bad++; }
            }
            long double d[3], r2 = 0, e2 = 0, t2 = 0;
            for (int k = 0; k < 3; k++) { d[k] = (long double)x[k] - b[j][k]; r2 += d[k] * d[k]; }
            for (int k = 0; k < 3; k++) {
                const long double t = -(long double)gm * d[k] / (r2 * sqrtl(r2));
                const long double g = j ? (long double)ag_pk_b(S.h[k]) + ag_pk_b(S.l[k]) : (long double)ag_pk_a(S.h[k]) + ag_pk_a(S.l[k]);
                e2 += (g - t) * (g - t); t2 += t * t;
            }
            const double err = (double)sqrtl(e2 / t2), far = R + (j ? 3.0 : 1.0) * D;
            const double lim = 1.5e-13 + 3.0 * 2.0 * 0x1p-48 * far / ((j ? 3.0 : 1.0) * D);
            n++;
            if (!(err < lim)) { if (bad < 5) std::printf("d %g R %g gm %g: %g > %g\n", D, R, gm, err, lim); bad++; }
        }
        /* a body below its threshold, or out of FP32's range, is left out and says so */
        G.ta = 1e30f;
        const AgPk before = S.h[0];
        if (ag_pk_term(A, G, xh, xl, 1.0f, S) != 1u || ag_pk_a(S.h[0]) != ag_pk_a(before)) bad++;
    }
    /* the thresholds: 1e-3 of the Sun's pull for heavy bodies, the separation's rounding for light ones */
    if (!(std::fabs(ag_pair_thr2(2.86e-4) / 0.286 - 1) < 1e-6) || !(std::fabs(ag_pair_thr2(5e-10) / std::pow(7.5e-8, 2.0 / 3.0) - 1) < 1e-6)) bad++;
    std::printf("checked %ld bad %d\n", n, bad);
    return bad != 0;
}
"""


def test_pair_terms_against_long_double(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    src = tmp_path / "pair.cpp"
    src.write_text(HARNESS)
    exe = tmp_path / "pair"
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "assist_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
