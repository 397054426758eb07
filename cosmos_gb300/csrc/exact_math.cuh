// Correctly rounded FP64 division, square root, product and comparisons on the integer and FP32
// pipes.  GB300 issues one FP64 warp instruction per 19 cycles and SM (latency 64), and a hardware
// division or square root is seven to eight of them (141-153 cycles per warp and SM, measured),
// while a 32 x 32 -> 64 bit multiply-add takes 1.2 and an add, logic or funnel shift 0.3-0.6.  The
// reference-exact kernels are bound by the FP64 pipe, half of it divisions, so the quotients, roots
// and part of the products are formed here from 53-bit significands: same results, bit for bit
// (round to nearest even of the exact value), on pipes that would otherwise idle.
//
// The operations have no slow path of their own (a branch per operation costs as much as the operation,
// and an FP64 instruction predicated off still takes its 19 cycles of the pipe, measured).  An operand
// outside the fast range that is not zero (subnormal, huge, infinite, NaN) makes the result NaN; a NaN
// goes through every later sum and operation, so whoever uses the type `xd` tests the results of a whole
// stage (any_nonfinite) and forms the stage again in hardware FP64 where one is not finite.
//
// The algorithms are digit-by-digit with exact integer remainders: a reciprocal (root) estimate good
// to about 28 bits gives two quotient (root) digits of 31 and 22+ bits, each from the exact remainder
// the one before left, and the sign of the final remainder against half an ulp decides the rounding.
// Neither a quotient nor a root of 53-bit operands can be a tie.  Host and device code: host builds
// (the tests) take the estimates from an argument, so that their whole error range can be checked.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define XM_HD __host__ __device__ __forceinline__
#else
#define XM_HD inline
#endif

namespace cg {
namespace xm {

XM_HD uint32_t hi32(uint64_t x) { return (uint32_t)(x >> 32); }
XM_HD uint32_t lo32(uint64_t x) { return (uint32_t)x; }
XM_HD uint64_t pack(uint32_t hi, uint32_t lo) { return ((uint64_t)hi << 32) | lo; }
XM_HD uint32_t mulhi(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
XM_HD int32_t mulhi_s(int32_t a, int32_t b) {
#ifdef __CUDA_ARCH__
    return __mulhi(a, b);
#else
    return (int32_t)(((int64_t)a * b) >> 32);
#endif
}
// high word of (hi:lo) << s, 0 <= s < 32
XM_HD uint32_t shl_hi(uint32_t lo, uint32_t hi, uint32_t s) {
#ifdef __CUDA_ARCH__
    return __funnelshift_l(lo, hi, s);
#else
    return (uint32_t)((pack(hi, lo) << s) >> 32);
#endif
}
// low word of (hi:lo) >> s, 0 <= s < 32
XM_HD uint32_t shr_lo(uint32_t lo, uint32_t hi, uint32_t s) {
#ifdef __CUDA_ARCH__
    return __funnelshift_r(lo, hi, s);
#else
    return (uint32_t)(pack(hi, lo) >> s);
#endif
}
XM_HD uint64_t bits_of(double x) {
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t u;
    memcpy(&u, &x, 8);
    return u;
#endif
}
XM_HD double double_of(uint64_t u) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double x;
    memcpy(&x, &u, 8);
    return x;
#endif
}
XM_HD float float_of(uint32_t u) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float x;
    memcpy(&x, &u, 4);
    return x;
#endif
}
XM_HD uint32_t bits_of(float x) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(x);
#else
    uint32_t u;
    memcpy(&u, &x, 4);
    return u;
#endif
}

constexpr uint32_t kExpMask = 0x7ff00000u, kFracMask = 0x000fffffu, kOne = 0x00100000u;
// Fast range of an operand: magnitudes in [2^-255, 2^257) (biased exponent 768 .. 1279), so that no
// product or quotient of two operands comes near the ends of the normal range.
XM_HD bool out_of_range(uint32_t hi) { return (hi & 0x7fffffffu) - 0x30000000u >= 0x20000000u; }
XM_HD bool is_zero(uint32_t hi, uint32_t lo) { return ((hi << 1) | lo) == 0; }
// the result of an operation: NaN, a signed zero, or the number formed
XM_HD double result(bool bad, bool zero, uint32_t sign, uint64_t q) {
    const uint32_t h = zero ? 0u : hi32(q), l = zero ? 0u : lo32(q);
    return double_of(pack(bad ? 0x7ff80000u : h | sign, l));
}

// FP32 estimates (relative error at most 2^-22.9 on the device: one ulp) of 1/x, x in [1, 2), and of
// 1/sqrt(x), x in [1, 4).  Host builds add `ulps` to the correctly rounded value instead.
XM_HD float est_rcp(float x, int ulps) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return float_of(bits_of(1.0f / x) + (uint32_t)ulps);
#endif
}
XM_HD float est_rsqrt(float x, int ulps) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return float_of(bits_of((float)(1.0 / __builtin_sqrt((double)x))) + (uint32_t)ulps);
#endif
}

// ---- division
// A divisor b prepared for any number of quotients: |b| = m 2^(e - 1075), m in [2^52, 2^53), and
// r = (2^32 / (m 2^-52)) (1 - l) with 0 < l < 2^-27.9 (proof at make_divisor).
struct Divisor {
    uint32_t mh, ml, r, eh;  // eh: exponent field in place (bits 20..30) with b's sign
    bool bad;                // outside the fast range (zero included)
};

XM_HD Divisor make_divisor(double b, int ulps = 0) {
    const uint64_t u = bits_of(b);
    const uint32_t h = hi32(u), l = lo32(u);
    Divisor d;
    d.mh = (h & kFracMask) | kOne;
    d.ml = l;
    d.eh = h & 0xfff00000u;
    // x = the significand truncated to 23 fraction bits, y = 1/x (1 + t1), |t1| <= 2^-22.9; with the
    // truncation y = 1/m (1 + t), |t| < 2^-21.9.  Clamped below one ulp under 1, R = y 2^32 is exact.
    float y = est_rcp(float_of(0x3f800000u | (shl_hi(l, h, 3) & 0x007fffffu)), ulps);
    const float below_one = float_of(0x3f7fffffu);
    y = y < below_one ? y : below_one;
    const uint32_t R = (bits_of(y) << 8) + 0x80000000u;  // y = 1.f 2^-1 or, at its end, f = 0: 0x3f000000 << 8 = 0
    // one Newton step: D = 2^31 (m y - 1) - k, k in [0, 2) from the two truncations, |D| < 2^10;
    // R - R D 2^-31 = (2^32 / m)(1 - t^2 + k 2^-31) + (0, 1], t^2 < 2^-43: at most 3.1 2^-31
    // relative too large, 6.2 units at m = 1; minus 8 units it is below 2^32 / m by at most 8 + 2^-11
    // units of at most 2^-31 relative: 0 < l < 2^-27.9, and it fits 32 bits.
    const int32_t D = (int32_t)(mulhi(shl_hi(l, d.mh, 11), R) - 0x80000000u);
    d.r = R - 8u - (uint32_t)mulhi_s((int32_t)(R >> 1), D << 2);
    d.bad = out_of_range(h);
    return d;
}

// magnitude of the quotient, both operands in the fast range (anything otherwise)
XM_HD uint64_t div_fast(uint32_t ah, uint32_t al, const Divisor& d) {
    const uint32_t mh = (ah & kFracMask) | kOne;
    // q = a / b scaled into [1, 2): shift the dividend when its significand is the smaller one
    const uint32_t s = pack(mh, al) < pack(d.mh, d.ml) ? 1u : 0u;
    // first digit, units of 2^-30: x = floor(a 2^30), q1 <= q 2^30, short by less than
    // 2^31 (2^-27.9 + 2^-30) + 1 < 12
    const uint32_t q1 = mulhi(shl_hi(al, mh, 10u + s), d.r);
    // remainder a 2^(30+s) - q1 b in [0, 12 b) < 2^57, exact modulo 2^64
    const uint64_t ra = pack(shl_hi(al, mh, 30u + s), al << (30u + s));
    const uint64_t b = pack(d.mh, d.ml);
    const uint64_t rem = ra - (uint64_t)q1 * b;
    // second digit, units of 2^-52: floor(rem 2^-25) < 2^32; short by less than 1.4 (2^25.6 2^-27.9 from
    // r, 2^-4.9 from the truncated remainder, 1 from the shift), never above
    const uint32_t q2 = mulhi((uint32_t)(rem >> 25), d.r) >> 5;
    const uint64_t left = (rem << 22) - (uint64_t)q2 * b;  // [0, 1.4 b)
    const uint64_t up = (b - 2 * left) >> 63;              // nearest: one more when left > b / 2
    const uint64_t q = ((uint64_t)q1 << 22) + q2 + up;     // [2^52, 2^53]
    const uint32_t e = (ah & kExpMask) - (d.eh & kExpMask) + ((1022u - s) << 20);
    return pack((uint32_t)(q >> 32) + e, (uint32_t)q);
}

XM_HD double div(double a, const Divisor& d) {
    const uint64_t u = bits_of(a);
    const uint32_t h = hi32(u), l = lo32(u);
    const bool zero = is_zero(h, l);
    return result(d.bad | (out_of_range(h) & !zero), zero, (h ^ d.eh) & 0x80000000u, div_fast(h, l, d));
}
XM_HD double div(double a, double b) { return div(a, make_divisor(b)); }

// ---- square root
XM_HD double root(double a, int ulps = 0) {
    const uint64_t u = bits_of(a);
    const uint32_t h = hi32(u), l = lo32(u);
    // A = the significand, twice it for an even biased exponent: a = A 2^-52 4^k, A in [2^52, 2^54)
    const uint32_t s = ((h >> 20) & 1u) ^ 1u;
    const uint32_t mh = (h & kFracMask) | kOne;
    const uint32_t x = shl_hi(l, mh, 10u + s);  // floor(A 2^-22): units of 2^-30, in [2^30, 2^32)
    // y = (A 2^-52)^-1/2 (1 + t), |t| < 2^-21.9, from A's top 24 bits; R = y 2^32
    float y = est_rsqrt(float_of((0x3f800000u + (s << 23)) | (shl_hi(l, mh, 3) & 0x007fffffu)), ulps);
    const float below_one = float_of(0x3f7fffffu);
    y = y < below_one ? y : below_one;
    const uint32_t R = (bits_of(y) << 8) + 0x80000000u;
    // one Newton step: E = 2^30 (A y^2 - 1) - k, k in [0, 3) from the three truncations; y - y E / 2 is
    // too large by less than 7 units, so minus 8 it is below the inverse root, by at most 8 units
    const int32_t E = (int32_t)(mulhi(mulhi(x, R), R) - 0x40000000u);
    const uint32_t r = R - 8u - (uint32_t)mulhi_s((int32_t)(R >> 1), E << 2);
    // first digit, units of 2^-30: short of the root by less than 12
    const uint32_t s1 = mulhi(x, r);
    const uint64_t A = pack(shl_hi(l, mh, s), l << s);
    const uint64_t rem = (A << 8) - (uint64_t)s1 * s1;  // A 2^8 < 2^62, remainder below 2^35.6
    // second digit rem 2^22 / (2 root), 1 / root = r 2^-62: short by less than 1.5 in all (0.2 from r, 0.13
    // from root for s1, 2^-5 from the truncated remainder, 1 from the shift), never above
    const uint32_t s2 = mulhi((uint32_t)(rem >> 4), r) >> 5;
    const uint64_t S = ((uint64_t)s1 << 22) + s2;
    const uint64_t left = (A << 52) - S * S;                // A 2^52 - S^2 < 3 S, exact modulo 2^64
    const uint64_t q = S + (uint64_t)(left > S ? 1u : 0u);  // up when the root exceeds S + 1/2
    const uint32_t e = (((h >> 20) + 1023u - s) >> 1) - 1u;  // the leading bit of q adds the one back
    const bool zero = is_zero(h, l);
    return result(h - 0x30000000u >= 0x20000000u && !zero, zero, h & 0x80000000u, pack((uint32_t)(q >> 32) + (e << 20), (uint32_t)q));
}

// ---- product
// magnitude of the product, both operands in the fast range (anything otherwise)
XM_HD uint64_t mul_fast(double a, double b) {
    const uint64_t ua = bits_of(a), ub = bits_of(b);
    const uint32_t ah = hi32(ua), bh = hi32(ub);
    const uint32_t al = lo32(ua), bl = lo32(ub), am = (ah & kFracMask) | kOne, bm = (bh & kFracMask) | kOne;
    // the 106-bit product in words w3:w2:w1:w0; the partial sums stay below 2^55
    const uint64_t p0 = (uint64_t)al * bl;
    uint64_t p1 = (uint64_t)al * bm + (p0 >> 32);
    p1 = (uint64_t)am * bl + p1;
    const uint64_t p2 = (uint64_t)am * bm + (p1 >> 32);
    const uint32_t w0 = lo32(p0), w1 = lo32(p1), w2 = lo32(p2), w3 = hi32(p2);
    const uint32_t n = w3 >> 9;  // 1 when the product of the significands is at least 2
    const uint32_t ql = shr_lo(w1, w2, 20u + n), qh = shr_lo(w2, w3, 20u + n);
    // the bits below: up when they exceed half, or equal it and the quotient is odd
    const uint32_t below = (w1 << (12u - n)) | (w0 < 1u ? w0 : 1u) | (ql & 1u);
    const uint64_t q = pack(qh, ql) + (uint64_t)(below > 0x80000000u ? 1u : 0u);
    const uint32_t e = (ah & kExpMask) + (bh & kExpMask) - ((1024u - n) << 20);
    return pack((uint32_t)(q >> 32) + e, (uint32_t)q);
}
XM_HD double mul(double a, double b) {
    const uint64_t ua = bits_of(a), ub = bits_of(b);
    const uint32_t ah = hi32(ua), bh = hi32(ub);
    const bool za = is_zero(ah, lo32(ua)), zb = is_zero(bh, lo32(ub));
    return result((out_of_range(ah) & !za) | (out_of_range(bh) & !zb), za | zb, (ah ^ bh) & 0x80000000u, mul_fast(a, b));
}

// a 2^K
template <int K>
XM_HD double scale2(double a) {
    const uint64_t u = bits_of(a);
    const uint32_t h = hi32(u), l = lo32(u);
    const bool zero = is_zero(h, l);
    const uint32_t s = h + (uint32_t)(K * (int)kOne);
    return double_of(pack(zero ? h : out_of_range(h) ? 0x7ff80000u : s, l));
}

// ---- comparisons on the bit patterns
XM_HD bool abs_less(double a, double c) {  // |a| < c, c a positive constant; false for NaN
    return (bits_of(a) & 0x7fffffffffffffffull) < bits_of(c);
}
// a < c, c a positive constant; false for NaN, and for -infinity (which the stage's test then finds)
XM_HD bool less(double a, double c) {
    const uint64_t u = bits_of(a);
    return (int64_t)u < (int64_t)bits_of(c) && hi32(u) < 0xfff00000u;
}
// a is positive (negative) with a magnitude in the fast range
XM_HD bool plain_positive(double a) { return hi32(bits_of(a)) - 0x30000000u < 0x20000000u; }
XM_HD bool plain_negative(double a) { return hi32(bits_of(a)) - 0xb0000000u < 0x20000000u; }
XM_HD bool finite(double a) { return (hi32(bits_of(a)) & 0x7fffffffu) < 0x7ff00000u; }

}  // namespace xm

// ---- a double whose products, quotients and roots run on the integer pipes and whose sums run on the
// FP64 pipe; see the note on NaN at the top
struct xd {
    double v;
    XM_HD xd() {}
    XM_HD xd(double x) : v(x) {}
    XM_HD explicit operator double() const { return v; }
};
XM_HD xd operator+(xd a, xd b) { return xd(a.v + b.v); }
XM_HD xd operator-(xd a, xd b) { return xd(a.v - b.v); }
XM_HD xd operator-(xd a) { return xd(xm::double_of(xm::bits_of(a.v) ^ 0x8000000000000000ull)); }
XM_HD xd operator*(xd a, xd b) { return xd(xm::mul(a.v, b.v)); }
XM_HD xd operator/(xd a, xd b) { return xd(xm::div(a.v, b.v)); }

// ---- a double as `xd` whose operations do not look at exponents: for operands that are zero or so far
// inside the normal range that no result leaves it (a zero is told by its high word).  A function that
// computes in xr tests its inputs (clean5) and what else its bounds need, states the bounds, and gives NaN
// back where a test failed.  Half of an `xd` product's instructions are such tests: without them the
// special-relativistic sweeps take 2256 -> 1874 us per step at 512^2, the Newtonian ones 1688 -> 1613 at 1024^2.
struct xr {
    double v;
    XM_HD xr() {}
    XM_HD xr(double x) : v(x) {}
    XM_HD explicit xr(xd x) : v(x.v) {}
};
namespace xm {
XM_HD bool zero_hi(double a) { return (hi32(bits_of(a)) & 0x7fffffffu) == 0; }
// |a| is neither zero nor in [2^LO, 2^HI)
template <int LO, int HI> XM_HD bool outside(double a) {
    const uint32_t l = lo32(bits_of(a)), h = (hi32(bits_of(a)) & 0x7fffffffu) | (l < 1u ? l : 1u);  // 0 for a zero only
    return h - 1u < ((uint32_t)(1023 + LO) << 20) - 1u || h >= ((uint32_t)(1023 + HI) << 20);
}
XM_HD double unless(bool zero, uint32_t sign, uint64_t q) {
    return double_of(pack((zero ? 0u : hi32(q)) | sign, zero ? 0u : lo32(q)));
}
XM_HD double raw_mul(double a, double b) {
    return unless(zero_hi(a) | zero_hi(b), (hi32(bits_of(a)) ^ hi32(bits_of(b))) & 0x80000000u, mul_fast(a, b));
}
XM_HD double raw_div(double a, const Divisor& d) {
    const uint64_t u = bits_of(a);
    return unless(zero_hi(a), (hi32(u) ^ d.eh) & 0x80000000u, div_fast(hi32(u), lo32(u), d));
}
template <int K> XM_HD double raw_scale2(double a) {
    const uint32_t h = hi32(bits_of(a));
    return double_of(pack(zero_hi(a) ? h : h + (uint32_t)(K * (int)kOne), lo32(bits_of(a))));
}
}  // namespace xm
XM_HD xr operator+(xr a, xr b) { return xr(a.v + b.v); }
XM_HD xr operator-(xr a, xr b) { return xr(a.v - b.v); }
XM_HD xr operator-(xr a) { return xr(xm::double_of(xm::bits_of(a.v) ^ 0x8000000000000000ull)); }
XM_HD xr operator*(xr a, xr b) { return xr(xm::raw_mul(a.v, b.v)); }
XM_HD xr operator/(xr a, const xm::Divisor& d) { return xr(xm::raw_div(a.v, d)); }
XM_HD xr operator/(xr a, xr b) { return xr(xm::raw_div(a.v, xm::make_divisor(b.v))); }
XM_HD xm::Divisor divisor(xr b) { return xm::make_divisor(b.v); }
XM_HD xr half(xr a) { return xr(xm::raw_scale2<-1>(a.v)); }
XM_HD xr twice(xr a) { return xr(xm::raw_scale2<1>(a.v)); }
XM_HD xr fourfold(xr a) { return xr(xm::raw_scale2<2>(a.v)); }
XM_HD xr root(xr a) { return xr(xm::root(a.v)); }

// The type a function computes in, its inputs and its results: double as is; xd as xr.
template <class T> struct Raw { using type = T; };
template <> struct Raw<xd> { using type = xr; };
// inputs of a state function: zero or in [2^-140, 2^100), the first (a density) not zero
XM_HD bool clean5(const double* a, double* o) {
#pragma unroll
    for (int k = 0; k < 5; k++) o[k] = a[k];
    return true;
}
XM_HD bool clean5(const xd* a, xr* o) {
    bool bad = xm::zero_hi(a[0].v);
#pragma unroll
    for (int k = 0; k < 5; k++) {
        o[k] = xr(a[k].v);
        bad |= xm::outside<-140, 100>(a[k].v);
    }
    return !bad;
}
template <int LO, int HI> XM_HD bool within(double) { return true; }
template <int LO, int HI> XM_HD bool within(xr a) { return !xm::outside<LO, HI>(a.v); }  // or zero
XM_HD bool nonzero(double) { return true; }
XM_HD bool nonzero(xr a) { return !xm::zero_hi(a.v); }
XM_HD bool bounded(double, bool) { return true; }  // whether a bound that only the unchecked arithmetic needs holds
XM_HD bool bounded(xr, bool holds) { return holds; }
XM_HD double given(double a, bool) { return a; }
XM_HD xd given(xr a, bool ok) { return xd(ok ? a.v : xm::double_of(0x7ff8000000000000ull)); }

// The same names on plain doubles are the hardware operations, so that one source gives both forms.
struct HwDivisor { double b; };
XM_HD HwDivisor divisor(double b) { return HwDivisor{b}; }
XM_HD double operator/(double a, HwDivisor d) { return a / d.b; }
XM_HD xm::Divisor divisor(xd b) { return xm::make_divisor(b.v); }
XM_HD xd operator/(xd a, const xm::Divisor& d) { return xd(xm::div(a.v, d)); }
XM_HD double half(double a) { return 0.5 * a; }
XM_HD xd half(xd a) { return xd(xm::scale2<-1>(a.v)); }
XM_HD double twice(double a) { return 2.0 * a; }
XM_HD xd twice(xd a) { return xd(xm::scale2<1>(a.v)); }
XM_HD double fourfold(double a) { return 4.0 * a; }
XM_HD xd fourfold(xd a) { return xd(xm::scale2<2>(a.v)); }
XM_HD double root(double a) { return ::sqrt(a); }
XM_HD xd root(xd a) { return xd(xm::root(a.v)); }
XM_HD double magnitude(double a) { return ::fabs(a); }
XM_HD xd magnitude(xd a) { return xd(xm::double_of(xm::bits_of(a.v) & 0x7fffffffffffffffull)); }
XM_HD bool below(double a, double c) { return a < c; }  // c positive (as in the next three)
XM_HD bool below(xd a, double c) { return xm::less(a.v, c); }
XM_HD bool below(xr a, double c) { return xm::less(a.v, c); }
XM_HD bool nearer_zero(double a, double c) { return ::fabs(a) < c; }
XM_HD bool nearer_zero(xd a, double c) { return xm::abs_less(a.v, c); }
XM_HD bool nearer_zero(xr a, double c) { return xm::abs_less(a.v, c); }
XM_HD bool above(double a, double c) { return a > c; }  // c positive
XM_HD bool above(xd a, double c) {
    const uint64_t u = xm::bits_of(a.v);
    return (int64_t)u > (int64_t)xm::bits_of(c) && xm::hi32(u) < 0x7ff00000u;
}
XM_HD bool above(xr a, double c) { return above(xd(a.v), c); }
XM_HD bool exceeds(double a, double b) { return a > b; }
XM_HD bool exceeds(xd a, xd b) { return a.v > b.v; }
XM_HD double times_zero(double a) { return a * 0.0; }  // a zero of a's sign, NaN where a is not finite
XM_HD xd times_zero(xd a) { return xm::finite(a.v) ? xd(xm::double_of(xm::bits_of(a.v) & 0x8000000000000000ull)) : a; }
// std::max as the reference uses it
XM_HD double larger(double a, double b) { return (a < b) ? b : a; }
XM_HD xd larger(xd a, xd b) { return (a.v < b.v) ? b : a; }
// whether an iteration may stop because its values are no numbers any more (xd: the stage is formed again)
XM_HD bool hopeless(double) { return false; }
XM_HD bool hopeless(xd a) { return !xm::finite(a.v); }
XM_HD bool hopeless(xr a) { return xm::outside<-60, 60>(a.v) || xm::zero_hi(a.v); }

XM_HD bool any_nonfinite(const xd* v, int n) {
    uint32_t m = 0;
#pragma unroll
    for (int k = 0; k < n; k++) {
        const uint32_t h = xm::hi32(xm::bits_of(v[k].v)) & 0x7fffffffu;
        m = h > m ? h : m;
    }
    return m >= 0x7ff00000u;
}

// a quotient whose operands may be anything, NaN where an integer-pipe one has none
XM_HD double checked_quotient(double a, double b) { return a / b; }
XM_HD xr checked_quotient(xr a, xr b) { return xr(xm::div(a.v, b.v)); }
// a / b: the integer pipes' quotient, the hardware's where that has none
XM_HD double quotient(double a, double b) {
    const double q = xm::div(a, b);
    if (xm::finite(q)) return q;
    return a / b;
}

}  // namespace cg
