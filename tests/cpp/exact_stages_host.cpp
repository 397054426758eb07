// Host build of the reference-exact sweep stages (cosmos_gb300/csrc/physics_exact.cuh): the integer-pipe form
// (xd) against the hardware form (double) of the half-step evolution and the FORCE flux, Newtonian and
// special-relativistic, on ordinary states and on ones at and beyond the ends of the integer pipes' range.
// Wherever the integer form's results are finite they have to be the hardware form's bits (elsewhere the
// kernels form the stage again in hardware FP64).  Prints what differs; exits non-zero if anything does.
#include "cuda_runtime.h"

#include <cstdio>
#include <cstdlib>
#include <random>

#include "../../cosmos_gb300/csrc/physics_exact.cuh"

using namespace cg;

static std::mt19937_64 gen(5);
static double uniform(double a, double b) { return a + (b - a) * ((gen() >> 11) * 0x1p-53); }

static void extremes(double* q) {
    switch (gen() % 12) {
        case 0: q[1] = q[2] = q[3] = 0.0; break;
        case 1: for (int f = 1; f < 4; f++) q[f] *= 1e-90; break;
        case 2: q[2] = 5e-324; break;
        case 3: q[3] = -1e-200; break;
        case 4: { const double e = std::pow(10.0, uniform(-85, 0)); q[0] *= e; q[4] *= e; break; }
        case 5: q[0] *= 1e90; q[4] *= 1e90; break;
        case 6: q[1 + gen() % 3] *= std::pow(10.0, uniform(-60, 0)); break;
        case 7: q[0] *= std::pow(10.0, uniform(-45, 35)); break;
        case 8: q[4] *= std::pow(10.0, uniform(-45, 35)); break;
        default: break;
    }
}

static long differ = 0, compared = 0;
static void same(const char* what, const xd* a, const double* b) {
    if (any_nonfinite(a, 5)) return;
    compared++;
    for (int f = 0; f < 5; f++)
        if (std::memcmp(&a[f].v, &b[f], 8) && differ++ < 10) printf("%s field %d: %a, not %a\n", what, f, a[f].v, b[f]);
}

template <class Sys>
static void stages(const Sys& S, const double (*c)[5], int axis, const StepRatio& st, const Bias& w, int lim) {
    const Pt z{0.0, 0.0, 0.0};
    xd xu[3][5], xl[5], xr_[5], xp[5];
    double du[3][5], dl[5], dr[5], dp[5];
    bool all = true;
    for (int k = 0; k < 3; k++) {
        for (int f = 0; f < 5; f++) xp[f] = xd(c[k][f]);
        S.cons(xp, z, xu[k]);
        S.cons(c[k], z, du[k]);
        same("cons", xu[k], du[k]);
        all = all && !any_nonfinite(xu[k], 5);
    }
    if (!all) return;
    evolve_half_cons(S, xu[0], xu[1], xu[2], z, axis, 0.0, st, w, lim, xl, xr_);
    evolve_half_cons(S, du[0], du[1], du[2], z, axis, 0.0, st, w, lim, dl, dr);
    const bool fine = !any_nonfinite(xl, 5) && !any_nonfinite(xr_, 5);  // one stage: both faces or neither
    if (fine) {
        same("left face", xl, dl);
        same("right face", xr_, dr);
    }
    xd xf[5];
    double df[5];
    force_cons(S, xu[0], xu[1], z, axis, 0.0, st, xf);
    force_cons(S, du[0], du[1], z, axis, 0.0, st, df);
    same("force", xf, df);
}

int main(int argc, char** argv) {
    const long n = argc > 1 ? atol(argv[1]) : 100000;
    const NewtonExact newton(1.4);
    const SRExact sr(5.0 / 3.0);
    const StepRatio st = make_ratio(0.002, 1.0 / 64);
    const double biases[] = {0.0, 0.0, 0.0, -0.7, 0.4, 1.0};
    for (long i = 0; i < n; i++) {
        double c[3][5];
        for (auto& q : c) {
            q[0] = uniform(0.1, 1.5);
            q[1] = uniform(-0.5, 0.5);
            q[2] = uniform(-0.5, 0.5);
            q[3] = uniform(-0.2, 0.2);
            q[4] = uniform(0.03, 1.5);
            extremes(q);
        }
        const Bias w = make_bias(biases[gen() % 6]);
        const int lim = (int)(gen() % 3), axis = (int)(gen() & 1);
        if (i & 1) stages(sr, c, axis, st, w, lim);
        else stages(newton, c, axis, st, w, lim);
    }
    printf("%ld compared, %ld differ\n", compared, differ);
    return differ != 0 || compared < n;
}
