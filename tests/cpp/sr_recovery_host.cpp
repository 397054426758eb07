// Host build of the FP32 special-relativistic primitive recovery (cosmos_gb300/csrc/physics_sr_fast.cuh): the
// sweeps' form (Halley's iteration from the state at rest for a gas's states) and the black hole's form (the
// reference's iteration in FP32 throughout) against the reference's recovery in FP64 of the same conserved
// states.  Classes of states: a gas's (W to 7 and to 50, p / rho 1e-8 .. 1e3), and states that are none (negative
// D, E or tau, |S| beyond E, extrapolations across a jump, densities of 1e-8 to 1e-2), where the results follow the
// iteration.  For each class and gamma, the sweeps' form may be off by more than 1 % in no more states than the
// other form (beyond three standard deviations of the count), and its errors below that may sum to no more than
// 1.1 times the other's.  Prints the table; exits non-zero where a bound is broken.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "cuda_runtime.h"

struct float2 { float x, y; };
inline float2 make_float2(float a, float b) { return float2{a, b}; }
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fmaf_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
inline float2 __fadd2_rn(float2 a, float2 b) { return {a.x + b.x, a.y + b.y}; }
inline float2 __fmul2_rn(float2 a, float2 b) { return {a.x * b.x, a.y * b.y}; }
inline float2 __ffma2_rn(float2 a, float2 b, float2 c) { return {std::fmaf(a.x, b.x, c.x), std::fmaf(a.y, b.y, c.y)}; }
static float flush(float x) { return std::fabs(x) < 1.17549435e-38f ? std::copysign(0.0f, x) : x; }
// rcp / sqrt / rsqrt .approx.ftz by the name in the instruction, correctly rounded
static float approximate(const char* instruction, float x) {
    x = flush(x);
    if (instruction[0] == 's') return flush(std::sqrt(x));
    if (instruction[1] == 'c') return flush(1.0f / x);
    return flush((float)(1.0 / std::sqrt((double)x)));
}
static unsigned __float_as_uint(float x) {
    unsigned u;
    memcpy(&u, &x, 4);
    return u;
}
#define asm(...) r = approximate(&#__VA_ARGS__[1], x)  // the header's wrappers: float r; asm("..." : "=f"(r) : "f"(x));
#include "../../cosmos_gb300/csrc/physics_sr_fast.cuh"
#undef asm

using namespace cg;

static std::mt19937_64 gen(3);
static double uniform(double a, double b) { return a + (b - a) * ((gen() >> 11) * 0x1p-53); }
static double spread(double lo, double hi) { return std::pow(10.0, uniform(lo, hi)); }

static void gas(double* u, double g, double top, double lo, double hi, double range) {
    const double rho = spread(-range, range), p = rho * spread(lo, hi), r = uniform(0, 1), W = 1 + (top - 1) * r * r;
    const double v = std::sqrt(1 - 1 / (W * W)), ct = uniform(-1, 1), st = std::sqrt(1 - ct * ct), ph = uniform(0, 6.283185307179586);
    const double rhw = (rho + p * g / (g - 1)) * W * W;
    u[0] = rho * W;
    u[1] = rhw * v * st * std::cos(ph);
    u[2] = rhw * v * st * std::sin(ph);
    u[3] = rhw * v * ct;
    u[4] = rhw - p - u[0];
}

enum { kGas, kFast, kNoEnergy, kNegativeE, kNegativeTau, kNegativeD, kSuperluminal, kJump, kFloor, kClasses };
static const char* names[] = {"gas", "gas, W to 50", "E = 0", "E < 0", "tau < 0", "D < 0", "|S| to 3 |S|", "across a jump", "thin gas"};

static void state(int c, double g, float* o) {
    double u[5], b[5];
    gas(u, g, c == kFast ? 50 : 7, -8, 3, 2);
    switch (c) {
        case kNoEnergy: u[0] = (float)u[0]; u[4] = -u[0]; break;
        case kNegativeE: u[4] = -u[0] * uniform(1, 3); break;
        case kNegativeTau: u[4] *= -uniform(0, 1); break;
        case kNegativeD: u[0] = -u[0]; break;
        case kSuperluminal: { const double f = uniform(1, 3); for (int k = 1; k < 4; k++) u[k] *= f; break; }
        case kJump:
            gas(u, g, 2, -1, 1, 1);
            gas(b, g, 2, -1, 1, 1);
            for (int k = 0; k < 5; k++) u[k] += 0.5 * (u[k] - b[k]);
            break;
        case kFloor: { const double f = spread(-8, -2) / u[0]; for (int k = 0; k < 5; k++) u[k] *= f; break; }
        default: break;
    }
    for (int k = 0; k < 5; k++) o[k] = (float)u[k];
}

// The reference's recovery in FP64; false where its iteration or its result is no number
static bool reference(const float* uf, double g, double* o) {
    double u[5];
    for (int k = 0; k < 5; k++) u[k] = uf[k];
    const double D = u[0], E = u[4] + D;
    double q = E * E - (u[1] * u[1] + u[2] * u[2] + u[3] * u[3]);
    if (q < 1e-8) q = 1e-8;
    const double dc = D / std::sqrt(q), ec = E / std::sqrt(q), gr = (g - 1) / g;
    const double c0 = -1 / (g * g), c1 = -2 * dc * gr / g, c2 = (g - 2) / g * (ec * ec - 1) + 1 - dc * dc * gr * gr;
    const double c4 = ec * ec - 1, eta = 2 * dc * gr;
    double x = 1;
    for (int it = 0;; it++) {
        if (it == 200) return false;  // (the reference goes on to 1000; such states have no root)
        const double f = c4 * x * x * x * (x - eta) + c2 * x * x + c1 * x + c0;
        const double nx = x - f / (c1 + 2 * c2 * x + 4 * c4 * x * x * x - 3 * eta * c4 * x * x);
        if (!(std::fabs(nx) < 1e30)) return false;
        if (std::fabs(nx - x) < 1e-8) break;
        x = nx;
    }
    const double W = 0.5 * ec * x * (1 + std::sqrt(1 + 4 * gr * (1 - dc * x) / (ec * ec * x * x)));
    const double rho = D / W, rhw = rho / (dc * x) * W * W, p = rhw - D - u[4];
    o[0] = std::max(rho, 1e-8);
    for (int k = 0; k < 3; k++) o[1 + k] = u[1 + k] / rhw;
    o[4] = std::max(p, 1e-8);
    // and inside FP32's range as the recovery draws it
    return std::fabs(W) + o[0] + o[4] + std::fabs(o[1]) + std::fabs(o[2]) + std::fabs(o[3]) + std::fabs(1 / (dc * x)) < 1e30;
}

static double error(const SRPrim32& r, const double* w) {
    const double got[5] = {r.rho, r.vx, r.vy, r.vz, r.p};
    double e = 0;
    for (int k = 0; k < 5; k++) {
        const double d = std::fabs(got[k] - w[k]) / (std::fabs(w[k]) + 1e-3 * std::fabs(k == 0 || k == 4 ? w[0] + w[4] : 1.0) + 1e-3);
        e = std::isfinite(d) ? std::max(e, d) : 1e30;
    }
    return e;
}

int main(int argc, char** argv) {
    const long n = argc > 1 ? atol(argv[1]) : 20000;
    long broken = 0;
    for (const double gamma : {1.1, 4.0 / 3.0, 1.4, 5.0 / 3.0, 2.0, 2.5, 3.0})
        for (int c = 0; c < kClasses; c++)
            for (const float above : {2.0f, 0.0f}) {
                SRFastParams P{};
                sr_fast_constants(P, gamma);
                P.w64 = above;
                long seen = 0, off[2] = {0, 0}, flags[2] = {0, 0};
                double sum[2] = {0, 0};
                for (long i = 0; i < n; i++) {
                    float u[5];
                    double w[5];
                    int f[2] = {0, 0};
                    state(c, gamma, u);
                    const SRPrim32 r[2] = {sr_c2p_fast<true>(P, u, &f[0]), sr_c2p_fast<false>(P, u, &f[1])};
                    for (int m = 0; m < 2; m++) flags[m] += f[m];
                    if (!reference(u, gamma, w)) continue;
                    seen++;
                    for (int m = 0; m < 2; m++) {
                        const double e = error(r[m], w);
                        if (e > 1e-2) off[m]++;
                        else sum[m] += e;
                    }
                }
                const bool ok = off[0] <= off[1] + 3 * std::sqrt((double)off[1] + 1) && sum[0] <= 1.1 * sum[1] + 1e-12 &&
                                (c != kNoEnergy || flags[0] == n);
                broken += !ok;
                printf("gamma %.3f %-14s FP64 above %.0f: %ld states, off %ld and %ld, mean error %.2e and %.2e, not converged %ld and %ld%s\n",
                       gamma, names[c], above, seen, off[0], off[1], sum[0] / std::max(seen, 1l), sum[1] / std::max(seen, 1l),
                       flags[0], flags[1], ok ? "" : "  <--");
            }
    return broken != 0;
}
