// Host build of the integer-pipe FP64 operations (cosmos_gb300/csrc/exact_math.cuh) against the
// machine's own IEEE division, square root and product: significands at the edges of every digit and
// random ones, the whole error range of the FP32 estimates, and operands outside the fast range.
// Prints the number of results that differ from the machine's, and exits non-zero if any does.
#include <cstdio>
#include <cstdlib>

#include "../../cosmos_gb300/csrc/exact_math.cuh"

using namespace cg::xm;

static uint64_t state = 88172645463325252ull;
static uint64_t rnd() {
    state ^= state << 13;
    state ^= state >> 7;
    state ^= state << 17;
    return state;
}
// a significand of one of several shapes (53 bits, leading one dropped)
static uint64_t frac(int kind) {
    const uint64_t full = (1ull << 52) - 1, r = rnd() & full;
    const int k = (int)(rnd() % 53);
    switch (kind) {
        case 0: return r;
        case 1: return rnd() % 16;                        // just above a power of two
        case 2: return full - rnd() % 16;                 // just below the next
        case 3: return (1ull << k) & full;                // one bit
        case 4: return full ^ ((1ull << k) & full);       // one bit missing
        case 5: return r & ~((1ull << (k % 52)) - 1);     // short significands
        default: return (r >> 29 << 29) + rnd() % 4 - 2 & full;  // at the estimate's truncation
    }
}
static double make(uint64_t f, int e, int neg) { return double_of(((uint64_t)neg << 63) | ((uint64_t)e << 52) | f); }
static int exponent(int kind) {
    if (kind < 6) return 1023 + (int)(rnd() % 61) - 30;
    if (kind < 8) return 766 + (int)(rnd() % 516);  // the fast range and just outside
    return (int)(rnd() % 2048);  // the whole range: subnormals, infinities, NaN
}
// whether an operation may give NaN where the machine gives something else: an operand outside the fast range
static bool excused(double a) {
    const double m = __builtin_fabs(a);
    return a != 0.0 && !(m >= 0x1p-255 && m < 0x1p257);
}

int main(int argc, char** argv) {
    const long n = argc > 1 ? atol(argv[1]) : 1000000;
    long bad = 0;
    auto check = [&](const char* what, double a, double b, double got, double want, bool may) {
        const bool nan = got != got;
        if (may ? nan || bits_of(got) == bits_of(want) : nan ? want != want : bits_of(got) == bits_of(want)) return;
        if (bad++ < 10) printf("%s %a %a: %a, not %a\n", what, a, b, got, want);
    };
    auto truth = [&](const char* what, double a, double b, bool got, bool want) {
        if (got != want && bad++ < 10) printf("%s %a %a: %d\n", what, a, b, got);
    };
    auto all = [&](double a, double b, int ulps) {
        const bool ea = excused(a), eb = excused(b);
        check("div", a, b, div(a, make_divisor(b, ulps)), a / b, ea || eb || b == 0.0);
        check("mul", a, b, mul(a, b), a * b, ea || eb);
        check("root", a, 0.0, root(a, ulps), __builtin_sqrt(a), ea || a < 0.0);
        check("half", a, 0.0, scale2<-1>(a), a * 0.5, ea);
        check("twice", a, 0.0, scale2<1>(a), a * 2.0, ea);
        const double c = __builtin_fabs(b);
        if (c > 0.0 && c < __builtin_inf()) {
            truth("abs_less", a, c, abs_less(a, c), __builtin_fabs(a) < c);
            if (a != -__builtin_inf()) truth("less", a, c, less(a, c), a < c);
        }
        truth("positive", a, 0.0, plain_positive(a), a > 0.0 && !ea);
        truth("negative", a, 0.0, plain_negative(a), a < 0.0 && !ea);
        truth("finite", a, 0.0, cg::xm::finite(a), __builtin_isfinite(a));
    };
    const double special[] = {0.0, -0.0, 1.0, -1.0, 5e-324, 2.2250738585072014e-308, 1.7976931348623157e308,
                              1e-5, 0x1p-255, 0x1p257, __builtin_inf(), -__builtin_inf(), __builtin_nan("")};
    for (double a : special)
        for (double b : special) all(a, b, 0);
    for (long i = 0; i < n; i++) {
        const int fa = (int)(rnd() % 7), fb = (int)(rnd() % 7), k = (int)(rnd() % 10);
        const double a = make(frac(fa), exponent(k), (int)(rnd() & 1)), b = make(frac(fb), exponent(k), (int)(rnd() & 1));
        const int ulps = (int)(rnd() % 3) - 1;  // the device's estimates are within one unit
        all(a, b, ulps);
        const double sq = b * b;
        check("root", sq, 0.0, root(sq, ulps), __builtin_sqrt(sq), excused(sq));
    }
    printf("%ld differ\n", bad);
    return bad != 0;
}
