// Host build of the reference-exact primitive recovery and black-hole state functions
// (cosmos_gb300/csrc/physics_exact.cuh) on conserved states taken as they come: physical ones, ones without a
// root, and ones whose sums cancel to an exact zero (tau = -D: no energy; S = 0 at rest; tau = S = 0: no internal
// energy).  The hardware form (double) has to be the reference's iteration written out below, status included,
// for every gamma > 1; wherever the integer-pipe form's (xd) results are finite they have to be the hardware
// form's bits.  Prints what differs; exits non-zero if anything does.
#include "cuda_runtime.h"

#include <cstdio>
#include <cstdlib>
#include <random>

#include "../../cosmos_gb300/csrc/physics_exact.cuh"

using namespace cg;

static std::mt19937_64 gen(7);
static double uniform(double a, double b) { return a + (b - a) * ((gen() >> 11) * 0x1p-53); }
static double spread(double lo, double hi) { return std::pow(10.0, uniform(lo, hi)); }

static long differ = 0, compared = 0;
static bool equal(double a, double b) { return std::memcmp(&a, &b, 8) == 0 || (std::isnan(a) && std::isnan(b)); }
static void same(const char* what, const double* a, const double* b, int n) {
    for (int f = 0; f < n; f++)
        if (!equal(a[f], b[f]) && differ++ < 10) printf("%s %d: %a, not %a\n", what, f, a[f], b[f]);
}
static void finite_same(const char* what, const xd* a, const double* b, int n) {
    if (any_nonfinite(a, n)) return;
    compared++;
    double v[16];
    for (int f = 0; f < n; f++) v[f] = a[f].v;
    same(what, v, b, n);
}

// RelativisticEuler/RelativisticEulerStateVector.cpp:30-101: rho, vx, vy, vz, p, W, h
static void reference(const double* u, double g, double tol, double* o, int* status) {
    const double D = u[0], tau = u[4];
    const double q = ((tau + D) * (tau + D)) - (((u[1] * u[1]) + (u[2] * u[2])) + (u[3] * u[3]));
    double dc = D / std::sqrt(q), ec = (D + tau) / std::sqrt(q);
    if (q < 1e-8) {
        dc = D / std::sqrt(1e-8);
        ec = (D + tau) / std::sqrt(1e-8);
    }
    const double c0 = -1.0 / (g * g), c1 = (-2.0 * dc) * ((g - 1.0) / (g * g));
    const double c2 = ((((g - 2.0) / g) * ((ec * ec) - 1.0)) + 1.0) - (((dc * dc) * ((g - 1.0) / g)) * ((g - 1.0) / g));
    const double c4 = (ec * ec) - 1.0, eta = (2.0 * dc) * ((g - 1.0) / g);
    double x = 1.0;
    bool found = false;
    for (int it = 0; it < 1000 && !found; it++) {
        const double f = ((((c4 * ((x * x) * x)) * (x - eta)) + (c2 * (x * x))) + (c1 * x)) + c0;
        const double fp = ((c1 + ((2.0 * c2) * x)) + ((4.0 * c4) * ((x * x) * x))) - (((3.0 * eta) * c4) * (x * x));
        const double nx = x - (f / fp);
        found = std::fabs(x - nx) < tol;
        if (!found) x = nx;
    }
    if (!found) *status |= ST_NEWTON_CAP;
    const double W = ((0.5 * ec) * x) * (1.0 + std::sqrt(1.0 + ((4.0 * ((g - 1.0) / g)) * ((1.0 - (dc * x)) / ((ec * ec) * (x * x))))));
    const double h = 1.0 / (dc * x), rho = D / W, rhw = (rho * h) * (W * W), p = (rhw - D) - tau;
    o[0] = rho < 1e-8 ? 1e-8 : rho;
    for (int k = 0; k < 3; k++) o[1 + k] = u[1 + k] / rhw;
    o[4] = p < 1e-8 ? 1e-8 : p;
    o[5] = W;
    o[6] = h;
}

// A conserved state: of a physical gas (special-relativistic, rho W etc.), or of anything
static void state(double* u) {
    const double rho = spread(-8, 1), p = rho * spread(-8, 3), v = uniform(0, 1) < 0.3 ? 0.0 : uniform(0, 0.99);
    const double ct = uniform(-1, 1), ph = uniform(0, 6.283185307179586), st = std::sqrt(1 - ct * ct);
    const double W = 1 / std::sqrt(1 - v * v), rhw = (rho + p * 2.5) * W * W;
    u[0] = rho * W;
    u[1] = rhw * v * st * std::cos(ph);
    u[2] = rhw * v * st * std::sin(ph);
    u[3] = rhw * v * ct;
    u[4] = rhw - p - u[0];
    switch (gen() % 10) {
        case 0: u[4] = -u[0]; break;
        case 1: u[0] = -u[0]; break;
        case 2: u[4] = -u[4]; break;
        case 3: u[1] = u[2] = u[3] = 0.0; break;
        case 4: u[1] = u[2] = u[3] = u[4] = 0.0; break;
        case 5: for (int f = 1; f < 4; f++) u[f] *= uniform(0, 20); break;
        case 6: u[0] = 0.0; break;
        case 7: u[gen() % 5] *= spread(-60, 60); break;
        default: break;
    }
}

static void recoveries(double gamma) {
    const GammaConst k(gamma);
    double u[5], want[7];
    state(u);
    const double tol = gen() & 1 ? 1e-8 : 1e-10;
    int s_want = 0, s_hw = 0, s_int = 0;
    reference(u, gamma, tol, want, &s_want);
    const C2P<double> d = con2prim_exact(five(u), k, tol, &s_hw);
    const double hw[7] = {d.rho, d.vx, d.vy, d.vz, d.p, d.W, d.h};
    same("hardware recovery", hw, want, 7);
    if (s_hw != s_want && differ++ < 10) printf("hardware recovery: status %d, not %d\n", s_hw, s_want);
    xd a[5];
    for (int f = 0; f < 5; f++) a[f] = xd(u[f]);
    const C2P<xd> x = con2prim_exact(five(a), k, tol, &s_int);
    const xd got[7] = {x.rho, x.vx, x.vy, x.vz, x.p, x.W, x.h};
    finite_same("integer recovery", got, want, 7);
    if (!any_nonfinite(got, 7) && s_int != s_want && differ++ < 10) printf("integer recovery: status %d, not %d\n", s_int, s_want);
    // as the sweeps use it
    const SRExact S(gamma);
    const Pt z{0.0, 0.0, 0.0};
    xd xo[5];
    double o[5];
    for (int axis = 0; axis < 2; axis++) {
        S.flux(a, axis, z, xo);
        S.flux(u, axis, z, o);
        finite_same("flux", xo, o, 5);
    }
    S.prim(a, z, xo);
    S.prim(u, z, o);
    finite_same("prim", xo, o, 5);
    // and of primitives: a state whose enthalpy vanishes among them (p / rho = -(gamma - 1) / gamma)
    double pr[5] = {u[0], u[1], u[2], u[3], u[4]};
    if (gen() % 4 == 0) {
        pr[4] = -(gamma - 1.0) / gamma * pr[0];
        pr[1] = pr[2] = pr[3] = 0.0;
    }
    for (int f = 0; f < 5; f++) a[f] = xd(pr[f]);
    S.cons(a, z, xo);
    S.cons(pr, z, o);
    finite_same("cons", xo, o, 5);
    const xd ws = S.wavespeed(a, 2, z);
    const double wd = S.wavespeed(pr, 2, z);
    finite_same("wavespeed", &ws, &wd, 1);
}

// the black-hole state functions in and around the horizon of a hole in the middle of the unit square
static void black_hole(const GRExact& S) {
    double u[5];
    state(u);
    Pt q{0.5, 0.5, 0.0};
    if (gen() % 50) {
        const double r = uniform(0, 1) < 0.5 ? uniform(0, 0.3) : spread(-6, 0), ph = uniform(0, 6.283185307179586);
        q = Pt{0.5 + r * std::cos(ph), 0.5 + r * std::sin(ph), 0.0};
    }
    xd a[5], xo[5];
    double o[5];
    for (int f = 0; f < 5; f++) a[f] = xd(u[f]);
    S.prim(a, q, xo);
    S.prim(u, q, o);
    finite_same("black-hole prim", xo, o, 5);
    for (int axis = 0; axis < 2; axis++) {
        S.flux(a, axis, q, xo);
        S.flux(u, axis, q, o);
        finite_same("black-hole flux", xo, o, 5);
    }
    S.source(a, q, xo);
    S.source(u, q, o);
    finite_same("black-hole source", xo, o, 5);
    double p[5] = {spread(-8, 1), 0, 0, 0, spread(-8, 1)};
    for (int f = 1; f < 4; f++) p[f] = uniform(0, 1) < 0.3 ? 0.0 : uniform(-0.7, 0.7);
    for (int f = 0; f < 5; f++) a[f] = xd(p[f]);
    S.cons(a, q, xo);
    S.cons(p, q, o);
    finite_same("black-hole cons", xo, o, 5);
    const xd cs = S.sound_speed(a, q);
    const double cd = S.sound_speed(p, q);
    finite_same("black-hole speed", &cs, &cd, 1);
}

int main(int argc, char** argv) {
    const long n = argc > 1 ? atol(argv[1]) : 20000;
    const double gammas[] = {5.0 / 3.0, 4.0 / 3.0, 1.4, 2.0, 1.1, 3.0, 1.0 + 0x1p-52, 1e20};
    for (long i = 0; i < n; i++) recoveries(gammas[gen() % 8]);
    const double hole[] = {0.05, 0.0, 0.5, 0.5, 0.0}, spinning[] = {0.05, 0.9, 0.5, 0.5, 0.0};
    const GRExact still(4.0 / 3.0, hole, 1.0 / 150), spun(5.0 / 3.0, spinning, 1.0 / 64);
    for (long i = 0; i < n; i++) black_hole(i & 1 ? still : spun);
    printf("%ld compared, %ld differ\n", compared, differ);
    return differ != 0 || compared < n;
}
