// Reference-exact device physics.  Every expression keeps the reference's evaluation order
// (left-to-right C++ semantics of the cited lines), so that a translation unit compiled with
// --fmad=false produces the reference's FP64 results bit for bit.  The functions are generic over
// the number type T: double (hardware FP64) or xd (exact_math.cuh: products, quotients and roots on
// the integer pipes, NaN where an operand leaves their range).  A stage whose xd results are not all
// finite is formed again in double; both give the reference's bits.
#pragma once
#include "device_common.cuh"
#include "exact_math.cuh"

namespace cg {

// ============================================================== slope limiters
// Solvers/SlopeLimiters.cpp:3-6
template <class T> CG_D T gradient_ratio(T r, T w) { return T(2.0) / ((T(1.0) - w) + ((T(1.0) + w) * r)); }

// Solvers/SlopeLimiters.cpp:8-69 (0 SuperBee, 1 van Leer, otherwise MinBee)
template <class T> CG_D T limiter_exact(T r, T w, int lim) {
    if (lim == 0) {
        if (r < T(0.0)) return T(0.0);
        else if (r >= T(0.0) && r < T(0.5)) return T(2.0) * r;
        else if (r >= T(0.5) && r < T(1.0)) return T(1.0);
        return mn(mn(r, gradient_ratio(r, w)), T(2.0));
    } else if (lim == 1) {
        if (r < T(0.0)) return T(0.0);
        return mn((T(2.0) * r) / (T(1.0) + r), gradient_ratio(r, w));
    }
    if (r < T(0.0)) return T(0.0);
    else if (r >= T(0.0) && r < T(1.0)) return r;
    return mn(T(1.0), gradient_ratio(r, w));
}

// The bias w and what the slopes take from it, formed once on the host (or per item).
struct Bias {
    double w, a, b;  // w, 0.5 (1 + w), 0.5 (1 - w)
};
CG_HD Bias make_bias(double w) { return Bias{w, 0.5 * (1.0 + w), 0.5 * (1.0 - w)}; }

// One component of the slope vector, Solvers/SlopeLimiters.cpp:71-101: numerator and denominator each
// clamped to +1e-5.
CG_D double limited_slope(double dl, double dr, const Bias& w, int lim) {
    const double s = (w.a * dl) + (w.b * dr);
    double num = dl, den = dr;
    if (fabs(num) < 1e-5) num = 1e-5;
    if (fabs(den) < 1e-5) den = 1e-5;
    return s * limiter_exact(num / den, w.w, lim);
}
// The same value with the limiter's comparisons on bit patterns and, for bias 0 (every driver's), at
// most one quotient after r = num / den: with w = 0 both candidates of a minimum have the denominator
// 1 + r, and rounding is monotone, so the minimum of the rounded quotients is the rounded quotient of
// the smaller numerator (van Leer 2 min(r, 1) / (1 + r); SuperBee and MinBee 2 / (1 + r) from r = 1
// on).  Both differences inside the clamp (uniform flow, a velocity that is zero everywhere) give
// r = 1 and a limiter of 1.
// Bounds: differences zero or in [2^-200, 2^101) (tested); r in [2^-118, 2^118] after the clamp; the
// candidates in [2^-120, 2^120]; the slope zero or at least 2^-320.
CG_D xd limited_slope(xd dl, xd dr, const Bias& w, int lim) {
    const xr l = xr(dl.v), r_ = xr(dr.v);
    const bool plain = w.w == 0.0, ok = within<-200, 101>(l) & within<-200, 101>(r_);
    const bool tl = nearer_zero(l, 1e-5), tr = nearer_zero(r_, 1e-5);
    if (plain && ok) {
        const xr s = half(l) + half(r_);
        if (tl && tr) return xd(s.v);
        const xr r = (tl ? xr(1e-5) : l) / (tr ? xr(1e-5) : r_);
        if (xm::bits_of(r.v) >> 63) return xd(xm::double_of(xm::bits_of(s.v) & 0x8000000000000000ull));
        const bool lt1 = below(r, 1.0);
        xr phi = xr(2.0);
        bool quotient = true;
        if (lim == 1) {
            if (lt1) phi = twice(r);
        } else if (lt1) {
            quotient = false;
            phi = lim == 0 ? (below(r, 0.5) ? twice(r) : xr(1.0)) : r;
        }
        if (quotient) phi = phi / (xr(1.0) + r);
        return xd((s * phi).v);
    }
    const xd nan = xd(xm::double_of(0x7ff8000000000000ull));
    if (!ok) return nan;
    const xd s = (xd(w.a) * dl) + (xd(w.b) * dr);
    const xd r = (tl ? xd(1e-5) : dl) / (tr ? xd(1e-5) : dr);
    if (xm::plain_negative(r.v)) return xm::finite(s.v) ? xd(xm::double_of(xm::bits_of(s.v) & 0x8000000000000000ull)) : s;
    if (!xm::plain_positive(r.v)) return nan;
    const bool lt1 = below(r, 1.0);
    const xd xi = xd(2.0) / (xd(1.0 - w.w) + (xd(1.0 + w.w) * r));
    if (!xm::finite(xi.v)) return xi;  // a comparison would lose the NaN
    xd phi;
    if (lim == 1) phi = twice(r) / (xd(1.0) + r);
    else if (lt1) return s * (lim == 0 ? (below(r, 0.5) ? twice(r) : xd(1.0)) : r);
    else phi = lim == 0 ? r : xd(1.0);
    if (xi.v < phi.v) phi = xi;
    if (lim == 0 && 2.0 < phi.v) phi = xd(2.0);
    return s * phi;
}
// half of it, one copy for the integer pipes (300 instructions, five times per evolution)
CG_D double half_slope(double dl, double dr, const Bias& w, int lim) { return half(limited_slope(dl, dr, w, lim)); }
static __device__ __noinline__ xd half_slope(xd dl, xd dr, Bias w, int lim) { return half(limited_slope(dl, dr, w, lim)); }
template <class T> CG_D void slope_exact(const T* ul, const T* uc, const T* ur, const Bias& w, int lim, T* s) {
#pragma unroll
    for (int k = 0; k < 5; k++) s[k] = limited_slope(uc[k] - ul[k], ur[k] - uc[k], w, lim);
}

template <class T> CG_D V5<T> five(const T* a) { return V5<T>{{a[0], a[1], a[2], a[3], a[4]}}; }
template <class T> CG_D void give(const V5<T>& a, T* o) {
#pragma unroll
    for (int k = 0; k < 5; k++) o[k] = a.v[k];
}

// ============================================================== Newtonian Euler
// Velocities, two of their squares, specific total energy and pressure of a conserved state: what prim and
// flux share.
template <class T> struct NewtonParts { typename Raw<T>::type vx, vy, vz, xx, yy, et, pr; bool ok; };
template <class T> CG_D NewtonParts<T> newton_parts(V5<T> in, double g1, bool fits) {
    using R = typename Raw<T>::type;
    R u[5];
    NewtonParts<T> o;
    o.ok = clean5(in.v, u) & fits;
    const auto d = divisor(u[0]);
    o.vx = u[1] / d;
    o.vy = u[2] / d;
    o.vz = u[3] / d;
    o.et = u[4] / d;
    o.xx = o.vx * o.vx;
    o.yy = o.vy * o.vy;
    const R v2 = (o.xx + o.yy) + (o.vz * o.vz);
    o.pr = ((o.et - half(v2)) * R(g1)) * u[0];
    return o;
}

// Bounds of the xr arithmetic, for inputs zero or in [2^-140, 2^100) (clean5), density not zero and
// gamma - 1 in [2^-50, 2^50]: velocities in [2^-240, 2^240], their squares and products in [2^-480, 2^482],
// a difference of such terms zero or at least one of their units, 2^-533; pressures in [2^-733, 2^633],
// fluxes in [2^-973, 2^874].
struct NewtonExact {
    double g, g1;  // gamma, gamma - 1
    bool fits;     // gamma - 1 within the bounds
    static constexpr bool kCoords = false;
    NewtonExact() = default;
    explicit NewtonExact(double gamma, int* = nullptr)
        : g(gamma), g1(gamma - 1.0), fits(gamma - 1.0 >= 0x1p-50 && gamma - 1.0 <= 0x1p50) {}
    // Euler/EulerStateVector.cpp:55-66, computeTotalEnergy :129-134, EoS Euler/EulerEquationOfState.cpp:3-8
    template <class T> CG_D void cons(const T* in, Pt, T* u) const {
        using R = typename Raw<T>::type;
        R p[5];
        const bool ok = clean5(in, p) & fits;
        const R rho = p[0], vx = p[1], vy = p[2], vz = p[3];
        const R v2 = ((vx * vx) + (vy * vy)) + (vz * vz);
        const R e = p[4] / (R(g1) * rho);
        u[0] = given(rho, ok);
        u[1] = given(rho * vx, true);
        u[2] = given(rho * vy, true);
        u[3] = given(rho * vz, true);
        u[4] = given(rho * (half(v2) + e), true);
    }
    // Euler/EulerStateVector.cpp:30-40, computePressure Euler/EulerEquationOfState.cpp:10-15
    template <class T> CG_D void prim(const T* u, Pt, T* p) const {
        const NewtonParts<T> c = newton_parts(five(u), g1, fits);
        using R = typename Raw<T>::type;
        p[0] = given(R(u[0]), c.ok);
        p[1] = given(c.vx, true);
        p[2] = given(c.vy, true);
        p[3] = given(c.vz, true);
        p[4] = given(c.pr, true);
    }
    // Euler/EulerStateVector.cpp:68-89 (x) and :96-117 (y)
    template <class T> CG_D void flux(const T* u, int axis, Pt, T* f) const {
        using R = typename Raw<T>::type;
        const NewtonParts<T> c = newton_parts(five(u), g1, fits);
        const R rho = R(u[0]);
        // products of two velocities commute exactly, so one form serves both axes
        const R vn = axis == 0 ? c.vx : c.vy;
        f[0] = given(rho * vn, c.ok);
        const R nn = (rho * (axis == 0 ? c.xx : c.yy)) + c.pr, xy = rho * (c.vx * c.vy);
        f[1] = given(axis == 0 ? nn : xy, true);
        f[2] = given(axis == 0 ? xy : nn, true);
        f[3] = given(rho * (vn * c.vz), true);
        f[4] = given((rho * (vn * c.et)) + (vn * c.pr), true);
    }
    // Solvers/EulerSolvers.cpp:87-128 with Euler/EulerEquationOfState.cpp:17-22;
    // 2D is max(|vx|, |vy| + c) exactly as written at :117-118.
    template <class T> CG_D T wavespeed(const T* p, int dims, Pt) const {
        T c = magnitude(root((T(g) * p[4]) / p[0]));
        if (hopeless(c)) return c;  // a maximum would drop it
        if (dims == 1) return magnitude(p[1]) + c;
        return larger(magnitude(p[1]), magnitude(p[2]) + c);
    }
};

// ============================================================== SR con2prim (FP64)
// RelativisticEuler/RelativisticEulerStateVector.cpp:30-101; the same solve appears in its flux
// functions (:138-309) and, on densitised variables, BlackHoleEuler/BlackHoleEulerStateVector.cpp
// (:30-103, :159-350 with tol 1e-10 in the x flux at :205, :359-430).  Newton from x = 1 on the
// quartic in x, stop when |x - x_new| < tol keeping the previous iterate, at most 1000 steps.
template <class T> struct C2P { T rho, vx, vy, vz, p, W, h; };
template <class T> CG_D void give_prim(const C2P<T>& c, T* p) {
    p[0] = c.rho; p[1] = c.vx; p[2] = c.vy; p[3] = c.vz; p[4] = c.p;
}
// what the solve takes from gamma, formed once on the host
struct GammaConst {
    double g, cst, lin, quad, gm, gm4, hg;
    bool fits;  // gamma in [1 + 2^-50, 2^50]: the constants are zero or in [2^-101, 2^51]
    GammaConst() = default;
    // hg: gamma / (gamma - 1), the enthalpy's factor
    explicit GammaConst(double g_) : g(g_), cst(-1.0 / (g_ * g_)), lin((g_ - 1.0) / (g_ * g_)), quad((g_ - 2.0) / g_),
                                     gm((g_ - 1.0) / g_), gm4(4.0 * ((g_ - 1.0) / g_)), hg(g_ / (g_ - 1.0)),
                                     fits(g_ >= 1.0 + 0x1p-50 && g_ <= 0x1p50) {}
};

// One copy per number type (out of line): a sweep recovers eight states per cell, and the iteration
// is thousands of cycles long.  status: ST_NEWTON_CAP is set there when the cap is reached (may be null).
// Bounds of the xr arithmetic, for inputs zero or in [2^-140, 2^100): E in [2^-192, 2^101] (or zero), q
// after its floor in [2^-27, 2^203], dc in [2^-242, 2^114], ec in [2^-295, 2^115], ec^2 in [2^-590, 2^230];
// x in [2^-60, 2^60) at every iteration (tested), so that every term of f and fp lies within 2^-800 .. 2^580;
// the step's quotient is an `xd` one; W in [2^-60, 2^60) (tested, and that it is not zero: an E of exactly zero,
// tau = -D, makes it so, where the root's NaN is lost in the product), so rho h W^2 lies within 2^-560 .. 2^640
// and the velocities within 2^-780 .. 2^660.
// (Two states in one instruction stream were 7 % slower on the relativistic sweeps: their code does not fit
// the instruction caches.)
template <class T>
__device__ __noinline__ C2P<T> con2prim_exact(V5<T> in, GammaConst k, double tol, int* status) {
    using R = typename Raw<T>::type;
    R u[5];
    bool ok = clean5(in.v, u) & bounded(R(), k.fits);  // always in double
    const R D = u[0], Sx = u[1], Sy = u[2], Sz = u[3], tau = u[4];
    const R E = tau + D;
    const R q = (E * E) - (((Sx * Sx) + (Sy * Sy)) + (Sz * Sz));
    const bool tiny = below(q, 1e-8);
    const auto dq = divisor(root(tiny ? R(1e-8) : q));
    const R dc = D / dq, ec = E / dq;
    const R ec2 = ec * ec;
    const R linear = -(twice(dc) * R(k.lin));
    const R quartic = ec2 - R(1.0);
    const R quadratic = ((R(k.quad) * quartic) + R(1.0)) - (((dc * dc) * R(k.gm)) * R(k.gm));
    const R eta = twice(dc) * R(k.gm);
    const R quad2 = twice(quadratic), quart4 = fourfold(quartic), eta3 = (R(3.0) * eta) * quartic;
    R x = R(1.0);
    int it = 0;
    bool conv = false;
    while (it < 1000 && ok) {
        const R x2 = x * x, x3 = x2 * x;
        const R f = ((((quartic * x3) * (x - eta)) + (quadratic * x2)) + (linear * x)) + R(k.cst);
        const R fp = ((linear + (quad2 * x)) + (quart4 * x3)) - (eta3 * x2);
        const R nx = x - checked_quotient(f, fp);
        if (nearer_zero(x - nx, tol)) { conv = true; break; }
        it += 1;
        x = nx;
        ok = !hopeless(nx);
    }
    if (!conv && ok && status) atomicOr(status, ST_NEWTON_CAP);
    C2P<T> r;
    const R dx = dc * x;
    const R rt = root(R(1.0) + (R(k.gm4) * ((R(1.0) - dx) / (ec2 * (x * x)))));
    const R W = (half(ec) * x) * (R(1.0) + rt);
    ok = ok & within<-60, 60>(W) & nonzero(W);
    const R h = R(1.0) / dx;
    R rho = D / W;
    const R rhw = (rho * h) * (W * W);
    const auto dr = divisor(rhw);
    R p = (rhw - D) - tau;
    if (below(rho, 1e-8)) rho = R(1e-8);
    if (below(p, 1e-8)) p = R(1e-8);
    r.rho = given(rho, ok);
    r.vx = given(Sx / dr, ok);
    r.vy = given(Sy / dr, ok);
    r.vz = given(Sz / dr, ok);
    r.p = given(p, ok);
    r.W = given(W, ok);
    r.h = given(h, ok);
    return r;
}

// RelativisticEuler/RelativisticEulerEquationOfState.cpp:3-18
template <class T> CG_D T sr_enthalpy(T rho, T p, const GammaConst& k) { return T(1.0) + ((p / rho) * T(k.hg)); }
template <class T> CG_D T sr_sound(T rho, T p, const GammaConst& k) {
    const auto d = divisor(rho);
    T num = (T(k.g) * p) / d;
    T den = T(1.0) + ((p / d) * T(k.hg));
    return root(num / den);
}
// 1 / sqrt(1 - v2), capped (RelativisticEuler/RelativisticEulerStateVector.cpp:116-136)
template <class T> CG_D T lorentz(T v2) {
    const bool fast = above(v2, 1.0 - 1e-8);
    return T(1.0) / root(fast ? T(1.0 - 1e-8) : T(1.0) - v2);
}

// ============================================================== SR Euler (FP64)
struct SRExact {
    GammaConst k;
    int* status;  // optional: gets ST_NEWTON_CAP when a Newton solve hits its cap
    static constexpr bool kCoords = false;
    SRExact() = default;
    explicit SRExact(double gamma, int* st = nullptr) : k(gamma), status(st) {}
    // RelativisticEuler/RelativisticEulerStateVector.cpp:116-136.  Bounds: W in [1, 2^14], the enthalpy in
    // [2^-53, 2^341] (p / rho within 2^-240 .. 2^240), rho h W^2 in [2^-193, 2^469].
    template <class T> CG_D void cons(const T* in, Pt, T* u) const {
        using R = typename Raw<T>::type;
        R p[5];
        const bool ok = clean5(in, p) & k.fits;
        const R rho = p[0], vx = p[1], vy = p[2], vz = p[3], pr = p[4];
        const R v2 = ((vx * vx) + (vy * vy)) + (vz * vz);
        const R W = lorentz(v2);
        const R h = sr_enthalpy(rho, pr, k);
        const R rhw = (rho * h) * (W * W), D = rho * W;
        u[0] = given(D, ok);
        u[1] = given(rhw * vx, true);
        u[2] = given(rhw * vy, true);
        u[3] = given(rhw * vz, true);
        u[4] = given((rhw - pr) - D, true);
    }
    template <class T> CG_D void prim(const T* u, Pt, T* p) const {
        give_prim(con2prim_exact(five(u), k, 1e-8, status), p);
    }
    // RelativisticEuler/RelativisticEulerStateVector.cpp:138-220 (x), :227-309 (y).  Bounds beyond the
    // recovery's: velocities zero or in [2^-200, 2^100) (tested), so the terms lie within 2^-960 .. 2^840.
    template <class T> CG_D void flux_of(const C2P<T>& c, int axis, T* f) const {
        using R = typename Raw<T>::type;
        const R rho = R(c.rho), vx = R(c.vx), vy = R(c.vy), vz = R(c.vz), p = R(c.p), W = R(c.W), h = R(c.h);
        const bool ok = within<-60, 200>(rho) & within<-200, 100>(vx) & within<-200, 100>(vy) & within<-200, 100>(vz);
        const R rhw = (rho * h) * (W * W);
        const R vn = axis == 0 ? vx : vy;
        const R rw = rho * W;
        f[0] = given(rw * vn, ok);
        const R nn = (rhw * (vn * vn)) + p, xy = rhw * (vx * vy);
        f[1] = given(axis == 0 ? nn : xy, true);
        f[2] = given(axis == 0 ? xy : nn, true);
        f[3] = given(rhw * (vz * vn), true);
        f[4] = given((((rhw - p) - rw) * vn) + (p * vn), true);
    }
    template <class T> CG_D void flux(const T* u, int axis, Pt, T* f) const {
        flux_of(con2prim_exact(five(u), k, 1e-8, status), axis, f);
    }
    // Solvers/RelativisticEulerSolvers.cpp:87-128 (2D: max(|vx|, |vy|) + c)
    template <class T> CG_D T wavespeed(const T* p, int dims, Pt) const {
        T c = magnitude(sr_sound(p[0], p[4], k));
        if (dims == 1) return magnitude(p[1]) + c;
        return larger(magnitude(p[1]), magnitude(p[2])) + c;
    }
};

// ============================================================== Kerr-Schild spacetime (FP64)
struct BHExact {
    double M, a, bx, by, bz;
    double ma2, am, horizon;  // M^2 a^2, a M, M (1 + sqrt(1 - a^2))
    BHExact() = default;
    BHExact(double mass, double spin, double x, double y, double z) : M(mass), a(spin), bx(x), by(y), bz(z) {
        ma2 = (M * M) * (a * a);
        am = a * M;
        volatile double aa = a * a;  // rounded before the subtraction: host compilers may contract the two
        horizon = M * (1.0 + ::sqrt(1.0 - aa));
    }
    // BlackHoleSpacetime.cpp:54-68
    template <class T> CG_D T radius(T dx, T dy, T dz) const {
        const T zz = dz * dz;
        const T n2 = ((dx * dx) + (dy * dy)) + zz;
        const T d = n2 - T(ma2);
        return root(half(d + root((d * d) + fourfold(T(ma2) * zz))));
    }
    template <class T> CG_D T H(double x, double y, double z) const {
        T dx = x - bx, dy = y - by, dz = z - bz;
        T r = radius(dx, dy, dz);
        const T r3 = (r * r) * r;
        return -(T(M) * r3) / ((r3 * r) + (T(ma2) * (dz * dz)));
    }
    // BlackHoleSpacetime.cpp:70-90
    template <class T> CG_D void l(double x, double y, double z, T* o) const {
        T dx = x - bx, dy = y - by, dz = z - bz;
        T r = radius(dx, dy, dz);
        const auto d = divisor((r * r) + T(ma2));
        o[0] = -((r * dx) + (T(am) * dy)) / d;
        o[1] = -((r * dy) - (T(am) * dx)) / d;
        o[2] = -dz / r;
    }
    // H and l together (same arithmetic as the two separate calls)
    template <class T> CG_D void Hl(double x, double y, double z, T& h, T* o) const {
        T dx = x - bx, dy = y - by, dz = z - bz;
        T r = radius(dx, dy, dz);
        const T r2 = r * r, r3 = r2 * r;
        h = -(T(M) * r3) / ((r3 * r) + (T(ma2) * (dz * dz)));
        const auto d = divisor(r2 + T(ma2));
        o[0] = -((r * dx) + (T(am) * dy)) / d;
        o[1] = -((r * dy) - (T(am) * dx)) / d;
        o[2] = -dz / r;
    }
    // BlackHoleSpacetime.cpp:92-113 with "r + (y - y_BH)" of :108 as written
    template <class T> CG_D void L4(double x, double y, double z, T* o) const {
        T dx = x - bx, dy = y - by, dz = z - bz;
        T r = radius(dx, dy, dz);
        const auto d = divisor((r * r) + T(ma2));
        o[0] = T(-1.0);
        o[1] = -((r * dx) + (T(am) * dy)) / d;
        o[2] = -((r + dy) - (T(am) * dx)) / d;
        o[3] = -dz / r;
    }
    // BlackHoleSpacetime.cpp:153-186
    template <class T> CG_D void gamma(double x, double y, double z, T* m) const {
        T h, v[3];
        Hl(x, y, z, h, v);
        gamma_of(h, v, m);
    }
    template <class T> CG_D void gamma_of(T h, const T* v, T* m) const {
        const T h2 = twice(h);
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) m[3 * i + j] = T(i == j ? 1.0 : 0.0) - ((h2 * v[i]) * v[j]);
    }
    // BlackHoleSpacetime.cpp:188-228
    template <class T> CG_D void g4(double x, double y, double z, T* m) const {
        T h = H<T>(x, y, z), v[4];
        L4(x, y, z, v);
        const T h2 = twice(h);
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const double eta = (i == j) ? ((i == 0) ? -1.0 : 1.0) : 0.0;
                m[4 * i + j] = T(eta) - ((h2 * v[i]) * v[j]);
            }
    }
    // lapse and shift from one H/l evaluation
    template <class T> CG_D void lapse_shift(double x, double y, double z, T& al, T* b) const {
        T h, v[3];
        Hl(x, y, z, h, v);
        lapse_shift_of(h, v, al, b);
    }
    template <class T> CG_D void lapse_shift_of(T h, const T* v, T& al, T* b) const {
        const T h2 = twice(h), d = T(1.0) - h2;
        al = T(1.0) / root(d);
        const T f = h2 / d;
#pragma unroll
        for (int i = 0; i < 3; i++) b[i] = f * v[i];
    }
    // BlackHoleSpacetime.cpp:372-386
    CG_D bool excised(double x, double y, double z) const {
        const xd dx = x - bx, dy = y - by, dz = z - bz;
        double r = root(((dx * dx) + (dy * dy)) + (dz * dz)).v;
        if (!xm::finite(r)) r = ::sqrt((((x - bx) * (x - bx)) + ((y - by) * (y - by))) + ((z - bz) * (z - bz)));
        return r <= horizon;
    }
};

// Mathematics/MatrixAlgebra.cpp:106-149: cofactor expansion along row 0 down to 2x2.
template <class T> CG_D T det2(T a00, T a01, T a10, T a11) { return (a00 * a11) - (a10 * a01); }
template <class T> CG_D T det3(const T* m) {
    T d = T(0.0);
    d = d + (m[0] * det2(m[4], m[5], m[7], m[8]));
    d = d - (m[1] * det2(m[3], m[5], m[6], m[8]));
    d = d + (m[2] * det2(m[3], m[4], m[6], m[7]));
    return d;
}
// (the 4x4 algebra keeps its outer loops: it runs once per cell and step, and unrolled it is thousands
// of instructions)
template <class T> CG_D T det4(const T* m) {
    T d = T(0.0);
#pragma unroll 1
    for (int i = 0; i < 4; i++) {
        T c[9];
#pragma unroll
        for (int j = 0; j < 3; j++)
#pragma unroll
            for (int k = 0; k < 3; k++) c[3 * j + k] = (k < i) ? m[4 * (j + 1) + k] : m[4 * (j + 1) + k + 1];
        if (i % 2 == 0) d = d + (m[i] * det3(c));
        else d = d - (m[i] * det3(c));
    }
    return d;
}
template <int N, class T> CG_D void matmul_n(const T* a, const T* b, T* c) {
#pragma unroll N < 4 ? N : 1
    for (int i = 0; i < N; i++)
#pragma unroll
        for (int j = 0; j < N; j++) {
            T s = T(0.0);
#pragma unroll
            for (int k = 0; k < N; k++) s = s + (a[N * i + k] * b[N * k + j]);
            c[N * i + j] = s;
        }
}
template <int N, class T> CG_D T trace_n(const T* m) {
    T t = T(0.0);
#pragma unroll
    for (int i = 0; i < N; i++) t = t + m[N * i + i];
    return t;
}
// Mathematics/MatrixAlgebra.cpp:151-194 (Cayley-Hamilton)
template <class T> CG_D void inverse3(const T* m, T* o) {
    T d = det3(m), tr = trace_n<3>(m), m2[9];
    matmul_n<3>(m, m, m2);
    T tr2 = trace_n<3>(m2);
    T s = half((tr * tr) - tr2);
    T inv = T(1.0) / d;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) o[3 * i + j] = inv * (((i == j ? s : times_zero(s)) - (tr * m[3 * i + j])) + m2[3 * i + j]);
}
template <class T> CG_D void inverse4(const T* m, T* o) {
    T d = det4(m), tr = trace_n<4>(m), m2[16], m3[16];
    matmul_n<4>(m, m, m2);
    matmul_n<4>(m2, m, m3);
    T tr2 = trace_n<4>(m2), tr3 = trace_n<4>(m3);
    T c0 = T(1.0 / 6.0) * ((((tr * tr) * tr) - ((T(3.0) * tr) * tr2)) + twice(tr3));
    T c1 = half((tr * tr) - tr2);
    T inv = T(1.0) / d;
#pragma unroll 1
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
            o[4 * i + j] = inv * ((((i == j ? c0 : times_zero(c0)) - (c1 * m[4 * i + j])) + (tr * m2[4 * i + j])) - m3[4 * i + j]);
}

// ============================================================== GR Euler (FP64)
// The metric at one point, as the state functions take it: spatial metric, sqrt(det gamma), lapse, shift.
template <class T> struct Metric { T gm[9], sg, al, be[3]; };
// What the source term takes beyond it: inverse 4-metric, centred derivatives of the lapse, shift and
// spatial metric, extrinsic curvature.
template <class T> struct SourceMetric { T gi[16], da[3], db[9], dgm[27], K[9]; };

struct GRExact {
    GammaConst k;
    BHExact bh;
    double h, ih, hs;  // finite-difference spacing of the metric derivatives (the cell spacing), 1 / h, h / 2
    int* status;       // as in SRExact
    static constexpr bool kCoords = true;
    GRExact() = default;
    GRExact(double gamma, const double* hole, double spacing, int* st = nullptr)
        : k(gamma), bh(hole[0], hole[1], hole[2], hole[3], hole[4]), h(spacing), ih(1.0 / spacing), hs(0.5 * spacing),
          status(st) {}

    template <class T> CG_D void metric(Pt q, Metric<T>& o) const {
        T hh, l[3];
        bh.Hl(q.x, q.y, q.z, hh, l);
        bh.gamma_of(hh, l, o.gm);
        o.sg = root(det3(o.gm));
        bh.lapse_shift_of(hh, l, o.al, o.be);
    }
    // gamma_ij v^i v^j in the reference's order
    template <class T> CG_D T square(const T* m, const T* v) const {
        T v2 = T(0.0);
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) v2 = v2 + ((m[3 * i + j] * v[i]) * v[j]);
        return v2;
    }
    // BlackHoleEuler/BlackHoleEulerStateVector.cpp:118-157 (energy with W, not W^2, at :154)
    template <class T> CG_D void cons_in(const Metric<T>& g, const T* p, T* u) const {
        const T W = lorentz(square(g.gm, p + 1));
        const T hh = sr_enthalpy(p[0], p[4], k);
        const T sr = g.sg * p[0];
        u[0] = sr * W;
        const T srhw = (sr * hh) * (W * W);
#pragma unroll
        for (int f = 0; f < 3; f++) u[1 + f] = srhw * p[1 + f];
        u[4] = g.sg * ((((p[0] * hh) * W) - p[4]) - (p[0] * W));
    }
    template <class T> CG_D V5<T> undensitised(const T* u, T sg) const {
        const auto d = divisor(sg);
        return V5<T>{{u[0] / d, u[1] / d, u[2] / d, u[3] / d, u[4] / d}};
    }
    template <class T> CG_D C2P<T> c2p(const T* u, T sg, double tol) const {
        return con2prim_exact(undensitised(u, sg), k, tol, status);
    }
    // BlackHoleEuler/BlackHoleEulerStateVector.cpp:30-103
    template <class T> CG_D void prim_in(const Metric<T>& g, const T* u, T* p) const {
        give_prim(c2p(u, g.sg, 1e-8), p);
    }
    // BlackHoleEuler/BlackHoleEulerStateVector.cpp:159-250 (x, tol 1e-10) and :259-350 (y)
    template <class T> CG_D void flux_of(const Metric<T>& g, const C2P<T>& c, int axis, T* f) const {
        const T as = g.al * g.sg;
        const T rhw = (c.rho * c.h) * (c.W * c.W);
        const T vn = axis == 0 ? c.vx : c.vy;
        const T w = vn - ((axis == 0 ? g.be[0] : g.be[1]) / g.al);
        const T rw = c.rho * c.W;
        f[0] = as * (rw * w);
        const T x = rhw * (c.vx * w), y = rhw * (c.vy * w);
        f[1] = as * (axis == 0 ? x + c.p : x);
        f[2] = as * (axis == 0 ? y : y + c.p);
        f[3] = as * (rhw * (c.vz * w));
        f[4] = as * ((((rhw - c.p) - rw) * w) + (c.p * vn));
    }
    template <class T> CG_D void flux_in(const Metric<T>& g, const T* u, int axis, T* f) const {
        flux_of(g, c2p(u, g.sg, axis == 0 ? 1e-10 : 1e-8), axis, f);
    }
    // ---- metric derivatives (BlackHoleSpacetime.cpp:115-151, :250-334), centred with spacing h
    CG_D Pt off(Pt q, int d, double s) const {
        if (d == 0) q.x = q.x + s; else if (d == 1) q.y = q.y + s; else q.z = q.z + s;
        return q;
    }
    // BlackHoleSpacetime.cpp:336-370 from H, l at the point (Hs, v) and its centred differences
    template <class T> CG_D void Kij_of(T al, T Hs, const T* v, const T* dh, const T* dv, T* K) const {
        const T al2 = twice(al), a2hh = al2 * (Hs * Hs), a2h = al2 * Hs;
#pragma unroll 1
        for (int i = 0; i < 3; i++)
#pragma unroll 1
            for (int j = 0; j < 3; j++) {
                T kk = al * (((-(v[i] * dh[j]) - (v[j] * dh[i])) - (Hs * dv[3 * j + i])) - (Hs * dv[3 * i + j]));
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    kk = kk + (a2hh * (((v[i] * v[c]) * dv[3 * c + j]) + ((v[j] * v[c]) * dv[3 * c + i])));
                    kk = kk + ((((a2h * v[i]) * v[j]) * v[c]) * dh[c]);
                }
                K[3 * i + j] = kk;
            }
    }
    // The metric part of the source term at q: inverse 4-metric, centred derivatives of the lapse,
    // shift and spatial metric (spacing h), extrinsic curvature (BlackHoleSpacetime.cpp:115-151,
    // :230-370).  H and l are evaluated once per point; every quantity there comes from them.
    template <class T> CG_D void source_metric(Pt q, T al, T* gi, T* da, T* db, T* dgm, T* K) const {
        T g4m[16];
        bh.g4(q.x, q.y, q.z, g4m);
        inverse4(g4m, gi);
        const auto dh_ = divisor(T(h));
        T dH[3], dl[9], Hs, v[3];
#pragma unroll 1
        for (int d = 0; d < 3; d++) {
            Pt p1 = off(q, d, hs), p0 = off(q, d, -hs);
            T h1, h0, l1[3], l0[3], a1, a0, b1[3], b0[3], g1[9], g0[9];
            bh.Hl(p1.x, p1.y, p1.z, h1, l1);
            bh.Hl(p0.x, p0.y, p0.z, h0, l0);
            bh.lapse_shift_of(h1, l1, a1, b1);
            bh.lapse_shift_of(h0, l0, a0, b0);
            bh.gamma_of(h1, l1, g1);
            bh.gamma_of(h0, l0, g0);
            da[d] = (a1 - a0) / dh_;
            dH[d] = (h1 - h0) / dh_;
#pragma unroll
            for (int c = 0; c < 3; c++) db[3 * d + c] = T(ih) * (b1[c] - b0[c]);
#pragma unroll
            for (int c = 0; c < 3; c++) dl[3 * d + c] = T(ih) * (l1[c] - l0[c]);
#pragma unroll
            for (int c = 0; c < 9; c++) dgm[9 * d + c] = T(ih) * (g1[c] - g0[c]);
        }
        bh.Hl(q.x, q.y, q.z, Hs, v);
        Kij_of(al, Hs, v, dH, dl, K);
    }
    // BlackHoleEuler/BlackHoleEulerStateVector.cpp:359-510
    template <class T> CG_D void source_in(const Metric<T>& g, const SourceMetric<T>& sm, const T* u, T* s) const {
        C2P<T> c = c2p(u, g.sg, 1e-8);
        const T al = g.al, sg = g.sg;
        const T *be = g.be, *gm = g.gm, *gi = sm.gi, *da = sm.da, *db = sm.db, *dgm = sm.dgm, *K = sm.K;
        T uu[4];
        uu[0] = c.W / al;
        const T au = al * uu[0];
        uu[1] = (au * c.vx) - (be[0] * uu[0]);
        uu[2] = (au * c.vy) - (be[1] * uu[0]);
        uu[3] = (au * c.vz) - (be[2] * uu[0]);
        T E[16];
        const T rh = c.rho * c.h;
#pragma unroll 1
        for (int i = 0; i < 4; i++)
#pragma unroll 1
            for (int j = 0; j < 4; j++) E[4 * i + j] = ((rh * uu[i]) * uu[j]) + (c.p * gi[4 * i + j]);
        T S[5] = {T(0.0), T(0.0), T(0.0), T(0.0), T(0.0)};
        T vc[3];
#pragma unroll
        for (int i = 0; i < 3; i++) vc[i] = ((gm[3 * i + 0] * c.vx) + (gm[3 * i + 1] * c.vy)) + (gm[3 * i + 2] * c.vz);
        const T rhw = rh * (c.W * c.W);
#pragma unroll 1
        for (int i = 0; i < 3; i++) {
#pragma unroll 1
            for (int j = 0; j < 3; j++) {
                const T hb = half(be[j]);
#pragma unroll
                for (int m = 0; m < 3; m++) {
                    const T dgijk = dgm[9 * i + 3 * j + m];
                    S[i + 1] = S[i + 1] + (E[0] * ((hb * be[m]) * dgijk));
                    S[i + 1] = S[i + 1] + ((E[j + 1] * be[m]) * dgijk);
                    S[i + 1] = S[i + 1] + half(E[4 * (j + 1) + (m + 1)] * dgijk);
                }
                S[i + 1] = S[i + 1] + (((rhw * vc[j]) / al) * db[3 * i + j]);
            }
            S[i + 1] = S[i + 1] - ((E[0] * al) * da[i]);
        }
#pragma unroll 1
        for (int i = 0; i < 3; i++) {
#pragma unroll 1
            for (int j = 0; j < 3; j++) {
                S[4] = S[4] + (E[0] * ((be[i] * be[j]) * K[3 * i + j]));
                S[4] = S[4] + (E[i + 1] * (twice(be[j]) * K[3 * i + j]));
                S[4] = S[4] + (E[4 * (i + 1) + (j + 1)] * K[3 * i + j]);
            }
            S[4] = S[4] - (E[0] * (be[i] * da[i]));
            S[4] = S[4] - (E[i + 1] * da[i]);
        }
        const T f = al * sg;
#pragma unroll
        for (int i = 0; i < 5; i++) s[i] = f * S[i];
    }
    // BlackHoleEuler/BlackHoleEulerStateVector.cpp:519-549, eigenvalues
    // BlackHoleEuler/BlackHoleEulerEigenvalues.cpp:3-96 (largest signed eigenvalue)
    template <class T> CG_D T sound_speed(const T* p, Pt q) const {
        T hh, l[3], al, be[3], gm[9], gs[9];
        bh.Hl(q.x, q.y, q.z, hh, l);
        bh.lapse_shift_of(hh, l, al, be);
        bh.gamma_of(hh, l, gm);
        inverse3(gm, gs);
        const T cs = sr_sound(p[0], p[4], k), c2 = cs * cs;
        const T* v = p + 1;
        const T v2 = square(gm, v);
        const T o1 = T(1.0) - (v2 * c2), o2 = T(1.0) - c2, o3 = T(1.0) - v2;
        const T pre = al / o1;
        T s = T(0.0);
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const T mat = (al * v[i]) - be[i];
            const T rt = root(o3 * ((gs[3 * i + i] * o1) - ((v[i] * v[i]) * o2)));
            const T fast = (pre * ((v[i] * o2) + (cs * rt))) - be[i];
            const T slow = (pre * ((v[i] * o2) - (cs * rt))) - be[i];
            // not finite here: every eigenvalue must show in the result (a comparison would drop it)
            if (hopeless(mat) || hopeless(fast) || hopeless(slow)) return fast + slow + mat;
            if (exceeds(mat, s)) s = mat;
            if (exceeds(fast, s)) s = fast;
            if (exceeds(slow, s)) s = slow;
        }
        return s;
    }
    // the state functions at a point (state-level and per-interface calls)
    template <class T> CG_D void cons(const T* p, Pt q, T* u) const;
    template <class T> CG_D void prim(const T* u, Pt q, T* p) const;
    template <class T> CG_D void flux(const T* u, int axis, Pt q, T* f) const;
    template <class T> CG_D void source(const T* u, Pt q, T* s) const;
};

// One copy per number type: the functions are thousands of cycles long and used at many places.  S is a
// kernel's parameter (__grid_constant__) or the copy of it that a slow path holds; the metrics lie in local
// memory, formed once per point and shared by every state converted there.
template <class T> __device__ __noinline__ void gr_metric(const GRExact* S, Pt q, Metric<T>* o) { S->metric(q, *o); }
template <class T> __device__ __noinline__ V5<T> gr_cons(const GRExact* S, const Metric<T>* g, V5<T> p) {
    V5<T> o;
    S->cons_in(*g, p.v, o.v);
    return o;
}
template <class T> __device__ __noinline__ V5<T> gr_prim(const GRExact* S, const Metric<T>* g, V5<T> u) {
    V5<T> o;
    S->prim_in(*g, u.v, o.v);
    return o;
}
template <class T> __device__ __noinline__ V5<T> gr_flux(const GRExact* S, const Metric<T>* g, V5<T> u, int axis) {
    V5<T> o;
    S->flux_in(*g, u.v, axis, o.v);
    return o;
}
template <class T> __device__ __noinline__ void gr_source_metric(const GRExact* S, Pt q, T al, SourceMetric<T>* o) {
    S->source_metric(q, al, o->gi, o->da, o->db, o->dgm, o->K);
}
template <class T>
__device__ __noinline__ V5<T> gr_source(const GRExact* S, const Metric<T>* g, const SourceMetric<T>* sm, V5<T> u) {
    V5<T> o;
    S->source_in(*g, *sm, u.v, o.v);
    return o;
}
template <class T> CG_D void GRExact::cons(const T* p, Pt q, T* u) const {
    Metric<T> g;
    gr_metric(this, q, &g);
    give(gr_cons(this, &g, five(p)), u);
}
template <class T> CG_D void GRExact::prim(const T* u, Pt q, T* p) const {
    Metric<T> g;
    gr_metric(this, q, &g);
    give(gr_prim(this, &g, five(u)), p);
}
template <class T> CG_D void GRExact::flux(const T* u, int axis, Pt q, T* f) const {
    Metric<T> g;
    gr_metric(this, q, &g);
    give(gr_flux(this, &g, five(u), axis), f);
}
template <class T> CG_D void GRExact::source(const T* u, Pt q, T* s) const {
    Metric<T> g;
    SourceMetric<T> sm;
    gr_metric(this, q, &g);
    gr_source_metric(this, q, g.al, &sm);
    give(gr_source(this, &g, &sm, five(u)), s);
}

// ============================================================== generic evolution pieces
// The sums of the stages: half (a + c b), and a + c b.
template <class T> CG_D T half_mix(T a, T b, T c) { return half(a + (c * b)); }
template <class T> CG_D T plus_times(T a, T b, T c) { return a + (c * b); }

// Half-step evolution (Solvers/EulerSolvers.cpp:174-223; SR Solvers/RelativisticEulerSolvers.cpp:148-199;
// GR Solvers/BlackHoleEulerSolvers.cpp:234-307) from the conserved states of the cell and its two
// neighbours.  Produces the left- and/or right-face state as primitives (the reference's evolved
// EulerStateVector).
template <class Sys, class T>
CG_D void evolve_half_cons(const Sys& S, const T* ul, const T* um, const T* ur, Pt xc, int axis, double dx,
                           const StepRatio& st, const Bias& w, int lim, T* left_face, T* right_face) {
    T UL[5], UR[5], FL[5], FR[5];
#pragma unroll
    for (int k = 0; k < 5; k++) {
        const T hs = half_slope(um[k] - ul[k], ur[k] - um[k], w, lim);
        UL[k] = um[k] - hs;
        UR[k] = um[k] + hs;
    }
    const Pt pl = shift_pt(xc, axis, -(dx * 0.5)), pr = shift_pt(xc, axis, dx * 0.5);
    S.flux(UL, axis, pl, FL);
    S.flux(UR, axis, pr, FR);
    const T s = half(T(st.d));
#pragma unroll
    for (int k = 0; k < 5; k++) {
        T ev = s * (FL[k] - FR[k]);
        UL[k] = UL[k] + ev;
        UR[k] = UR[k] + ev;
    }
    if (left_face) S.prim(UL, pl, left_face);
    if (right_face) S.prim(UR, pr, right_face);
}
// ... from their primitive states
template <class Sys, class T>
CG_D void evolve_half_exact(const Sys& S, const T* l, const T* m, const T* r, Pt xc, int axis, double dx,
                            const StepRatio& st, const Bias& w, int lim, T* left_face, T* right_face) {
    T ul[5], um[5], ur[5];
    S.cons(l, shift_pt(xc, axis, -dx), ul);
    S.cons(m, xc, um);
    S.cons(r, shift_pt(xc, axis, dx), ur);
    evolve_half_cons(S, ul, um, ur, xc, axis, dx, st, w, lim, left_face, right_face);
}

// FORCE flux of two conserved states at interface xf (Solvers/EulerFirstOrderSolver.cpp:3-59;
// GR Solvers/BlackHoleEulerFirstOrderSolver.cpp:3-47).
template <class Sys, class T>
CG_D void force_cons(const Sys& S, const T* uL, const T* uR, Pt xf, int axis, double dx, const StepRatio& st, T* F) {
    T fL[5], fR[5], us[5], fs[5];
    S.flux(uL, axis, shift_pt(xf, axis, -(dx * 0.5)), fL);
    S.flux(uR, axis, shift_pt(xf, axis, dx * 0.5), fR);
    const T c = T(st.c), d = T(st.d);
#pragma unroll
    for (int k = 0; k < 5; k++) {
        us[k] = half_mix(uL[k] + uR[k], fL[k] - fR[k], d);
        F[k] = half_mix(fL[k] + fR[k], uL[k] - uR[k], c);
    }
    S.flux(us, axis, xf, fs);
#pragma unroll
    for (int k = 0; k < 5; k++) F[k] = half(F[k] + fs[k]);
}
// ... of two primitive states
template <class Sys, class T>
CG_D void force_exact(const Sys& S, const T* L, const T* R, Pt xf, int axis, double dx, const StepRatio& st, T* F) {
    T uL[5], uR[5];
    S.cons(L, shift_pt(xf, axis, -(dx * 0.5)), uL);
    S.cons(R, shift_pt(xf, axis, dx * 0.5), uR);
    force_cons(S, uL, uR, xf, axis, dx, st, F);
}

// ============================================================== GR sweep and source step (FP64)
// One interface flux of a black-hole sweep (Solvers/BlackHoleEulerSecondOrderSolver.cpp:3-37): the left
// cell's right face from the evolution centred at xf - dx/2, the right cell's left face from that
// centred at xf + dx/2, then FORCE at xf.  c: the four cells around the interface; order 1 takes the
// two middle cells themselves.  The metric is formed once per point; the evolutions' centres are the
// points where FORCE converts the face states.
// One side of it: from the three cells around the left (side 0) or right (1) cell, its face state at xf,
// conserved at the cell's centre as FORCE has it, and its flux.
template <class T>
CG_D void gr_interface_side(const GRExact* S, const V5<T>* c, int side, int order, Pt xf, int axis, double dx,
                            const StepRatio& st, const Bias& w, int lim, V5<T>& u, V5<T>& f) {
    Metric<T> gc;
    const Pt xc = shift_pt(xf, axis, side == 0 ? -(dx * 0.5) : dx * 0.5);
    gr_metric(S, xc, &gc);
    V5<T> face = c[1];
    if (order == 2) {
        Metric<T> go;
        const V5<T> um = gr_cons(S, &gc, c[1]);
        gr_metric(S, shift_pt(xc, axis, -dx), &go);
        const V5<T> ul = gr_cons(S, &go, c[0]);
        gr_metric(S, shift_pt(xc, axis, dx), &go);
        const V5<T> ur = gr_cons(S, &go, c[2]);
        V5<T> UL, UR;
#pragma unroll
        for (int k = 0; k < 5; k++) {
            const T hs = half_slope(um.v[k] - ul.v[k], ur.v[k] - um.v[k], w, lim);
            UL.v[k] = um.v[k] - hs;
            UR.v[k] = um.v[k] + hs;
        }
        // the face wanted lies at xc + dx/2 (left cell) or xc - dx/2 (right cell)
        const T s = half(T(st.d));
        gr_metric(S, shift_pt(xc, axis, side == 0 ? -(dx * 0.5) : dx * 0.5), &go);
        const V5<T> V = side == 0 ? UL : UR;
        V5<T> X = side == 0 ? UR : UL;
        const V5<T> fo = gr_flux(S, &go, V, axis);
        gr_metric(S, shift_pt(xc, axis, side == 0 ? dx * 0.5 : -(dx * 0.5)), &go);
        const V5<T> fi = gr_flux(S, &go, X, axis);
#pragma unroll
        for (int k = 0; k < 5; k++)
            X.v[k] = X.v[k] + (s * (side == 0 ? fo.v[k] - fi.v[k] : fi.v[k] - fo.v[k]));
        face = gr_prim(S, &go, X);
    }
    u = gr_cons(S, &gc, face);
    f = gr_flux(S, &gc, u, axis);
}
// ... and FORCE of the two sides
template <class T>
CG_D void gr_interface_force(const GRExact* S, const V5<T>& uL, const V5<T>& uR, const V5<T>& fL, const V5<T>& fR,
                             Pt xf, int axis, const StepRatio& st, T* F) {
    Metric<T> g;
    V5<T> us;
    const T cc = T(st.c), d = T(st.d);
#pragma unroll
    for (int k = 0; k < 5; k++) {
        us.v[k] = half_mix(uL.v[k] + uR.v[k], fL.v[k] - fR.v[k], d);
        F[k] = half_mix(fL.v[k] + fR.v[k], uL.v[k] - uR.v[k], cc);
    }
    gr_metric(S, xf, &g);
    const V5<T> fs = gr_flux(S, &g, us, axis);
#pragma unroll
    for (int k = 0; k < 5; k++) F[k] = half(F[k] + fs.v[k]);
}
template <class T>
CG_D void gr_interface(const GRExact* S, const V5<T>* c, int order, Pt xf, int axis, double dx, const StepRatio& st,
                       const Bias& w, int lim, T* F) {
    V5<T> u[2], f[2];
#pragma unroll 1
    for (int side = 0; side < 2; side++)
        gr_interface_side(S, c + side, side, order, xf, axis, dx, st, w, lim, u[side], f[side]);
    gr_interface_force(S, u[0], u[1], f[0], f[1], xf, axis, st, F);
}

// computeFORCEUpdate (Solvers/EulerFirstOrderSolver.cpp:96-101) of a black-hole cell at q.
template <class T>
CG_D void gr_update(const GRExact* S, const V5<T>& c, const T* FL, const T* FR, Pt q, double d, T* out) {
    Metric<T> g;
    gr_metric(S, q, &g);
    V5<T> u = gr_cons(S, &g, c);
#pragma unroll
    for (int k = 0; k < 5; k++) u.v[k] = u.v[k] + (T(d) * (FL[k] - FR[k]));
    give(gr_prim(S, &g, u), out);
}

// Fractional evolution on frozen neighbours, Solvers/BlackHoleEulerSolvers.cpp:159-232: slopes
// from the neighbours at xc -/+ dx, face fluxes evaluated at xc -/+ dx (not dx/2), the middle
// state advanced by frac * dt/dx and converted back at xc.  ul, ur: the neighbours' conserved
// states, gl, gr_, gm the metrics there and at xc.
template <class T>
CG_D V5<T> evolve_fraction_in(const GRExact* S, double frac, const V5<T>& ul, const V5<T>& m, const V5<T>& ur,
                              const Metric<T>* gl, const Metric<T>* gm, const Metric<T>* gr_, int axis,
                              const StepRatio& st, const Bias& w, int lim) {
    V5<T> um = gr_cons(S, gm, m), UL, UR;
#pragma unroll
    for (int k = 0; k < 5; k++) {
        const T hs = half_slope(um.v[k] - ul.v[k], ur.v[k] - um.v[k], w, lim);
        UL.v[k] = um.v[k] - hs;
        UR.v[k] = um.v[k] + hs;
    }
    UL = gr_flux(S, gl, UL, axis);
    UR = gr_flux(S, gr_, UR, axis);
    const T s = T(frac) * T(st.d);
#pragma unroll
    for (int k = 0; k < 5; k++) um.v[k] = um.v[k] + (s * (UL.v[k] - UR.v[k]));
    return gr_prim(S, gm, um);
}
template <class T>
CG_D void evolve_fraction_exact(const GRExact& S, double frac, const T* l, const T* m, const T* r, Pt xc, int axis,
                                double dx, const StepRatio& st, const Bias& w, int lim, T* out) {
    Metric<T> gl, gm, gr_;
    gr_metric(&S, shift_pt(xc, axis, -dx), &gl);
    gr_metric(&S, xc, &gm);
    gr_metric(&S, shift_pt(xc, axis, dx), &gr_);
    give(evolve_fraction_in(&S, frac, gr_cons(&S, &gl, five(l)), five(m), gr_cons(&S, &gr_, five(r)), &gl, &gm, &gr_,
                            axis, st, w, lim), out);
}

// Classical RK4 on the source with interleaved fractional sweeps,
// Solvers/BlackHoleEulerForcingSolver.cpp:3-70 (1D: X fractions 1/2, 1/2, 1) and :72-185
// (2D: X 1/4, Y 1/2, X 1/4 for stages 1-2; X 1/2, Y 1, X 1/2 for stage 3).
// u: conserved states of the left, right, top and bottom neighbours and (u[4]) of the cell itself
// (cell-centred); q the cell's coordinate; returns the updated conserved state.  The neighbours are
// frozen and the spacetime is static: the neighbours' states as the fractional sweeps read them
// (conserved again from their recovered primitives), the metrics and the source term's metric part
// are formed once for the four stages.
// Team::sync() is called before the parts of a stage: threads that run in lockstep fetch the code together.
struct OneThread { CG_D void sync() const {} };
template <class Team, class T>
CG_D V5<T> rk_cell_exact(const Team& team, const GRExact* S, int dims, const V5<T>* u, Pt q, double dx, double dt,
                         const StepRatio& sr, const Bias& w, int lim, Metric<T>* gq) {
    Metric<T> gn[4];
    SourceMetric<T> sm;
    V5<T> un[4];
#pragma unroll 1
    for (int n = 0; n < (dims == 2 ? 4 : 2); n++) {
        team.sync();
        gr_metric(S, shift_pt(q, n >> 1, n & 1 ? dx : -dx), &gn[n]);
        un[n] = gr_cons(S, &gn[n], gr_prim(S, &gn[n], u[n]));
    }
    gr_metric(S, q, gq);
    gr_source_metric(S, q, gq->al, &sm);
    const V5<T> cm = u[4];
    // out = cm + (k0 + (2 k1 + (2 k2 + k3))) / 6; the stages share one copy of the code
    V5<T> k0, k1, k2, k = gr_source(S, gq, &sm, cm);
#pragma unroll
    for (int i = 0; i < 5; i++) k0.v[i] = k1.v[i] = k2.v[i] = k.v[i] = T(dt) * k.v[i];
#pragma unroll 1
    for (int stage = 0; stage < 3; stage++) {
        V5<T> p;
#pragma unroll
        for (int i = 0; i < 5; i++) p.v[i] = cm.v[i] + (stage < 2 ? half(k.v[i]) : k.v[i]);
        team.sync();
        p = gr_prim(S, gq, p);
        const double fx = dims == 1 ? (stage < 2 ? 0.5 : 1.0) : (stage < 2 ? 0.25 : 0.5), fy = stage < 2 ? 0.5 : 1.0;
#pragma unroll 1
        for (int part = 0; part < (dims == 1 ? 1 : 3); part++) {
            const int y = part == 1;
            team.sync();
            p = evolve_fraction_in(S, y ? fy : fx, un[2 * y], p, un[2 * y + 1], &gn[2 * y], gq, &gn[2 * y + 1], y, sr, w,
                                   lim);
        }
        k = gr_source(S, gq, &sm, gr_cons(S, gq, p));
#pragma unroll
        for (int i = 0; i < 5; i++) {
            k.v[i] = T(dt) * k.v[i];
            if (stage == 0) k1.v[i] = twice(k.v[i]);
            else if (stage == 1) k2.v[i] = twice(k.v[i]);
        }
    }
    V5<T> o;
#pragma unroll
    for (int i = 0; i < 5; i++) o.v[i] = cm.v[i] + (T(1.0 / 6.0) * (k0.v[i] + (k1.v[i] + (k2.v[i] + k.v[i]))));
    return o;
}

}  // namespace cg
