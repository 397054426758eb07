// Physics policies plugged into the generic sweep kernels (sweep_kernels.cuh).
#pragma once
#include "physics_exact.cuh"
#include "physics_fast.cuh"
#include "physics_sr_fast.cuh"
#include "sweep_kernels.cuh"

namespace cg {

// Cell position helpers shared by the policies.  A sweep line is a row (axis 0) or a column
// (axis 1); k indexes cells along it.  Cell (i, j) sits at (x, y) = (j dx, i dx)
// (Solvers/BlackHoleEulerSecondOrderSolver.cpp:88-100); 1D grids are row i = 0, so y = 0 as in
// the reference's 1D solvers.
struct LineMap {
    int axis, nx;
    CG_D void ij(int line, int k, int& i, int& j) const {
        if (axis == 0) { i = line; j = k; } else { i = k; j = line; }
    }
    CG_D bool mask_on(const unsigned char* mask, int line, int k) const {
        if (!mask) return true;
        int i, j;
        ij(line, k, i, j);
        return mask[(size_t)i * nx + j] != 0;
    }
};

// ------------------------------------------------------------------ reference-exact, FP64
// The stages of a sweep in hardware FP64, out of line: taken where a stage's integer-pipe results are
// not all finite (exact_math.cuh).  Arguments go by value, so that the callers' stay in registers.
template <class Sys>
__device__ __noinline__ V5<double> slow_cons(Sys S, V5<double> p) {
    V5<double> u;
    S.cons(p.v, Pt{0.0, 0.0, 0.0}, u.v);
    return u;
}
template <class Sys>
__device__ __noinline__ V5<double> slow_prim(Sys S, V5<double> u) {
    V5<double> o;
    S.prim(u.v, Pt{0.0, 0.0, 0.0}, o.v);
    return o;
}
struct FacePair { V5<double> L, R; };
template <class Sys>
__device__ __noinline__ FacePair slow_faces(Sys S, V5<double> l, V5<double> m, V5<double> r, int axis, StepRatio st,
                                            Bias w, int lim) {
    const Pt z{0.0, 0.0, 0.0};
    double a[5], b[5];
    FacePair o;
    evolve_half_cons(S, l.v, m.v, r.v, z, axis, 0.0, st, w, lim, a, b);
    S.cons(a, z, o.L.v);
    S.cons(b, z, o.R.v);
    return o;
}
template <class Sys>
__device__ __noinline__ V5<double> slow_force(Sys S, V5<double> uL, V5<double> uR, int axis, StepRatio st) {
    V5<double> o;
    force_cons(S, uL.v, uR.v, Pt{0.0, 0.0, 0.0}, axis, 0.0, st, o.v);
    return o;
}
template <class Sys>
__device__ __noinline__ V5<double> slow_update(Sys S, V5<double> u, V5<double> FL, V5<double> FR, double d) {
    V5<double> o;
    for (int f = 0; f < 5; f++) u.v[f] = u.v[f] + (d * (FL.v[f] - FR.v[f]));
    S.prim(u.v, Pt{0.0, 0.0, 0.0}, o.v);
    return o;
}
template <class Sys>
__device__ __noinline__ double slow_wavespeed(Sys S, V5<double> c, int dims, Pt q) {
    if constexpr (Sys::kCoords) return S.sound_speed(c.v, q);
    else return S.wavespeed(c.v, dims, q);
}

CG_D void load5(const double* a, xd* o) {
#pragma unroll
    for (int f = 0; f < 5; f++) o[f] = xd(a[f]);
}
CG_D void store5(const xd* a, double* o) {
#pragma unroll
    for (int f = 0; f < 5; f++) o[f] = a[f].v;
}

// The state functions on the integer pipes, one copy each: a sweep evaluates five fluxes and three of each
// conversion per cell; all inlined they are 9000 instructions (140 KB) in a row, and waiting for
// instructions was the largest stall (3.2 of 9.5 cycles per instruction at 389 x 509).  Out of line: 421 -> 364
// us per step there, 31.7 -> 21.5 for 1000 cells in 1D, 122 registers instead of 139.  Splitting further
// (what prim and flux share, the stages' sums) measured 1-8 % slower.
template <class Sys> __device__ __noinline__ V5<xd> x_cons(Sys S, V5<xd> p) {
    V5<xd> o;
    S.cons(p.v, Pt{0.0, 0.0, 0.0}, o.v);
    return o;
}
template <class Sys> __device__ __noinline__ V5<xd> x_prim(Sys S, V5<xd> u) {
    V5<xd> o;
    S.prim(u.v, Pt{0.0, 0.0, 0.0}, o.v);
    return o;
}
template <class Sys> __device__ __noinline__ V5<xd> x_flux(Sys S, V5<xd> u, int axis) {
    V5<xd> o;
    S.flux(u.v, axis, Pt{0.0, 0.0, 0.0}, o.v);
    return o;
}
// The same functions for the generic evolution pieces (evolve_half_cons, force_cons).
template <class Sys>
struct OutOfLine {
    Sys S;
    CG_D void cons(const xd* p, Pt, xd* u) const { give(x_cons(S, five(p)), u); }
    CG_D void prim(const xd* u, Pt, xd* p) const { give(x_prim(S, five(u)), p); }
    CG_D void flux(const xd* u, int axis, Pt, xd* f) const { give(x_flux(S, five(u), axis), f); }
};

struct FaceOf { V5<double> u; bool bad; };

// The stages of a coordinate-free sweep on conserved states (Newtonian, SR).
template <class Sys>
struct ExactStages {
    Sys sys;
    Bias w;
    int lim;
    // conserved state of a cell
    CG_D V5<double> cons(const V5<double>& p) const {
        xd a[5], u[5];
        V5<double> o;
        load5(p.v, a);
        OutOfLine<Sys>{sys}.cons(a, Pt{0.0, 0.0, 0.0}, u);
        store5(u, o.v);
        if (any_nonfinite(u, 5)) o = slow_cons(sys, p);
        return o;
    }
    CG_D V5<double> prim(const V5<double>& u) const {
        xd a[5], p[5];
        V5<double> o;
        load5(u.v, a);
        OutOfLine<Sys>{sys}.prim(a, Pt{0.0, 0.0, 0.0}, p);
        store5(p, o.v);
        if (any_nonfinite(p, 5)) o = slow_prim(sys, u);
        return o;
    }
    // conserved face states of the cell m after its half-step evolution (each through its primitives, as
    // the reference's evolved states are)
    CG_D void faces(const V5<double>& l, const V5<double>& m, const V5<double>& r, int axis, const StepRatio& st,
                    V5<double>& L, V5<double>& R) const {
        const Pt z{0.0, 0.0, 0.0};
        xd a[5], b[5], c[5], fl[5], fr[5];
        load5(l.v, a);
        load5(m.v, b);
        load5(r.v, c);
        evolve_half_cons(OutOfLine<Sys>{sys}, a, b, c, z, axis, 0.0, st, w, lim, fl, fr);
        OutOfLine<Sys>{sys}.cons(fl, z, a);
        OutOfLine<Sys>{sys}.cons(fr, z, b);
        store5(a, L.v);
        store5(b, R.v);
        if (any_nonfinite(a, 5) || any_nonfinite(b, 5)) {
            const FacePair o = slow_faces(sys, l, m, r, axis, st, w, lim);
            L = o.L;
            R = o.R;
        }
    }
    CG_D V5<double> force(const V5<double>& uL, const V5<double>& uR, int axis, const StepRatio& st) const {
        xd a[5], b[5], f[5];
        V5<double> o;
        load5(uL.v, a);
        load5(uR.v, b);
        force_cons(OutOfLine<Sys>{sys}, a, b, Pt{0.0, 0.0, 0.0}, axis, 0.0, st, f);
        store5(f, o.v);
        if (any_nonfinite(f, 5)) o = slow_force(sys, uL, uR, axis, st);
        return o;
    }
    // ---- the same stages in the pieces that two threads of a cell, or two interfaces, share
    CG_D double half_slope_of(double dl, double dr) const { return half_slope(xd(dl), xd(dr), w, lim).v; }
    // flux of a conserved state; not finite where the integer pipes have none (the stage that uses it then
    // forms it again)
    CG_D V5<double> flux(const V5<double>& u, int axis) const {
        xd a[5], f[5];
        V5<double> o;
        load5(u.v, a);
        OutOfLine<Sys>{sys}.flux(a, axis, Pt{0.0, 0.0, 0.0}, f);
        store5(f, o.v);
        return o;
    }
    // the face state that the extrapolated state V evolves to, FL and FR the fluxes of the cell's two
    CG_D FaceOf face_of_side(const V5<double>& V, const V5<double>& FL, const V5<double>& FR, int axis,
                             const StepRatio& st) const {
        const Pt z{0.0, 0.0, 0.0};
        const xd s = half(xd(st.d));
        xd a[5], b[5];
        FaceOf o;
#pragma unroll
        for (int k = 0; k < 5; k++) a[k] = xd(V.v[k]) + (s * (xd(FL.v[k]) - xd(FR.v[k])));
        OutOfLine<Sys>{sys}.prim(a, z, b);
        OutOfLine<Sys>{sys}.cons(b, z, a);
        store5(a, o.u.v);
        o.bad = any_nonfinite(a, 5);
        return o;
    }
    // FORCE of two conserved states whose fluxes are at hand
    CG_D V5<double> force_of(const V5<double>& uL, const V5<double>& uR, const V5<double>& fL, const V5<double>& fR,
                             int axis, const StepRatio& st) const {
        xd us[5], F[5], fs[5];
        V5<double> o;
#pragma unroll
        for (int k = 0; k < 5; k++) {
            us[k] = half_mix(xd(uL.v[k] + uR.v[k]), xd(fL.v[k] - fR.v[k]), xd(st.d));
            F[k] = half_mix(xd(fL.v[k] + fR.v[k]), xd(uL.v[k] - uR.v[k]), xd(st.c));
        }
        OutOfLine<Sys>{sys}.flux(us, axis, Pt{0.0, 0.0, 0.0}, fs);
#pragma unroll
        for (int k = 0; k < 5; k++) F[k] = half(F[k] + fs[k]);
        store5(F, o.v);
        if (any_nonfinite(F, 5)) o = slow_force(sys, uL, uR, axis, st);
        return o;
    }
    // computeFORCEUpdate, Solvers/EulerFirstOrderSolver.cpp:96-101, then setConservedVariableVector
    CG_D V5<double> update(const V5<double>& u, const V5<double>& FL, const V5<double>& FR, double d) const {
        xd a[5], p[5];
        V5<double> o;
#pragma unroll
        for (int f = 0; f < 5; f++) a[f] = plus_times(xd(u.v[f]), xd(FL.v[f] - FR.v[f]), xd(d));
        OutOfLine<Sys>{sys}.prim(a, Pt{0.0, 0.0, 0.0}, p);
        store5(p, o.v);
        if (any_nonfinite(p, 5)) o = slow_update(sys, u, FL, FR, d);
        return o;
    }
    CG_D double wavespeed(const V5<double>& c, int dims) const {
        xd p[5];
        load5(c.v, p);
        double s = sys.wavespeed(p, dims, Pt{0.0, 0.0, 0.0}).v;
        if (!xm::finite(s)) s = slow_wavespeed(sys, c, dims, Pt{0.0, 0.0, 0.0});
        return speed_or_inf(c.v[0], c.v[4], s);
    }
};

// Primitive storage exactly like the reference's grids, for the generic kernels: the FP64 batch's tiles
// (Newtonian) and the CFL reduction of every system.  The single grids' sweeps are in exact_tiles.cuh.
template <class Sys>
struct ExactPolicy {
    using S = double;
    using X = double;
    using W = double;  // wavespeed reduction type
    using Cell = V5<double>;
    using Face = V5<double>;  // conserved
    struct Coef { double dt; StepRatio r; };
    static constexpr bool kMasked = false;
    static constexpr bool kHasDx = true;
    ExactStages<Sys> st;
    LineMap lm;
    int dims, ny;
    double dx, dt;
    StepRatio r;

    CG_D Coef make_coef(const DtSrc& ds, double d) const { return Coef{d, ds.ratio(d, dx)}; }
    CG_D void use_coef(const Coef& c) { dt = c.dt; r = c.r; }
    CG_D void recon(const Cell& l, const Cell& m, const Cell& rr, int, int, Face& L, Face& R) const {
        st.faces(st.cons(l), st.cons(m), st.cons(rr), lm.axis, r, L, R);
    }
    CG_D void face_of(const Cell& c, Face& f) const { f = st.cons(c); }
    CG_D void flux(const Face& L, const Face& R, int, int, V5<double>& F) const { F = st.force(L, R, lm.axis, r); }
    CG_D Cell update(const Cell& c, const V5<double>& FL, const V5<double>& FR, int, int) const {
        return st.update(st.cons(c), FL, FR, r.d);
    }
    CG_D bool active(int, int, const unsigned char*) const { return true; }
    CG_D double wavespeed(const Cell& c, int line, int k) const;
    CG_D void flush_status(int*) const {}
};

template <class Sys>
CG_D double ExactPolicy<Sys>::wavespeed(const Cell& c, int, int) const { return st.wavespeed(c, dims); }

// GR CFL speed, Solvers/BlackHoleEulerSolvers.cpp:87-131: coordinates use spacing 1/N, and in 2D
// the excision test reads (j/ncol, i/nrow) while the speed is evaluated at (i/nrow, j/ncol).
template <>
CG_D double ExactPolicy<GRExact>::wavespeed(const Cell& c, int line, int k) const {
    int i, j;
    lm.ij(line, k, i, j);
    const double cs = quotient(1.0, (double)lm.nx), rs = dims == 1 ? 0.0 : quotient(1.0, (double)ny);
    const double x = j * cs, y = i * rs;
    const GRExact& sys = st.sys;
    if (sys.bh.excised(x, y, 0.0)) return 0.0;
    const Pt q = dims == 1 ? Pt{x, 0.0, 0.0} : Pt{y, x, 0.0};
    xd p[5];
    load5(c.v, p);
    double s = sys.sound_speed(p, q).v;
    if (!xm::finite(s)) s = slow_wavespeed(sys, c, dims, q);
    return speed_or_inf(c.v[0], c.v[4], fabs(s));
}

// ------------------------------------------------------------------ Newtonian FP32 bulk
// Conserved FP32 storage; see physics_fast.cuh for the reformulations.  AXIS and LIM are fixed at
// compile time; MASKED selects whether the AMR update mask is consulted at all.
template <int AXIS, int LIM, bool MASKED>
struct NewtonFastPolicy {
    using S = float;
    using X = float;
    using W = float;
    using Cell = V5<float>;
    using Face = V5<float>;
    using Coef = FastCoef;
    static constexpr bool kMasked = MASKED;
    static constexpr bool kHasDx = false;  // dx enters through the precomputed coefficients
    NewtonFastParams P;
    LineMap lm;
    int dims;
    float dtdx, half_dtdx, q_dxdt;

    // FP32 coefficients come precomputed (device step controller or host), so no FP64
    // instruction runs in the FP32 sweeps
    CG_D Coef make_coef(const DtSrc& ds, double) const { return ds.fast_coef(); }
    CG_D void use_coef(const Coef& c) {
        dtdx = c.dtdx;
        half_dtdx = c.half_dtdx;
        q_dxdt = c.q_dxdt;
    }
    CG_D void recon(const Cell& l, const Cell& m, const Cell& r, int, int, Face& L, Face& R) const {
        nf_recon<AXIS, LIM>(P, l.v, m.v, r.v, half_dtdx, L.v, R.v);
    }
    CG_D void face_of(const Cell& c, Face& f) const { f = c; }
    CG_D void flux(const Face& L, const Face& R, int, int, V5<float>& F) const {
        nf_force<AXIS>(P, L.v, R.v, half_dtdx, q_dxdt, F.v);
    }
    CG_D Cell update(const Cell& c, const V5<float>& FL, const V5<float>& FR, int, int) const {
        Cell o;
        nf_update(dtdx, c.v, FL.v, FR.v, o.v);
        return o;
    }
    CG_D bool active(int line, int k, const unsigned char* mask) const {
        return MASKED ? lm.mask_on(mask, line, k) : true;
    }
    CG_D float wavespeed(const Cell& c, int, int) const { return nf_wavespeed(P, c.v, dims); }
    CG_D void flush_status(int*) const {}
};

// FP32 bulk policy of the special-relativistic system (physics_sr_fast.cuh): the sweep structure
// of NewtonFastPolicy with the relativistic flux, whose primitive recovery ends in FP64.
template <int AXIS, int LIM, bool MASKED>
struct SRFastPolicy {
    using S = float;
    using X = float;
    using W = float;
    using Cell = V5<float>;
    using Face = V5<float>;
    using Coef = FastCoef;
    static constexpr bool kMasked = MASKED;
    static constexpr bool kHasDx = false;
    NewtonFastParams NP;  // limiter and bias factors
    SRFastParams P;
    LineMap lm;
    int dims;
    float dtdx, half_dtdx, q_dxdt;
    int flags;  // bit 0: a primitive recovery did not converge

    CG_D Coef make_coef(const DtSrc& ds, double) const { return ds.fast_coef(); }
    CG_D void use_coef(const Coef& c) {
        dtdx = c.dtdx;
        half_dtdx = c.half_dtdx;
        q_dxdt = c.q_dxdt;
    }
    CG_D void recon(const Cell& l, const Cell& m, const Cell& r, int, int, Face& L, Face& R) {
        sr_recon_fast<AXIS, LIM>(P, NP, l.v, m.v, r.v, half_dtdx, L.v, R.v, &flags);
    }
    CG_D void face_of(const Cell& c, Face& f) const { f = c; }
    CG_D void flux(const Face& L, const Face& R, int, int, V5<float>& F) {
        sr_force_fast<AXIS>(P, L.v, R.v, half_dtdx, q_dxdt, F.v, &flags);
    }
    CG_D Cell update(const Cell& c, const V5<float>& FL, const V5<float>& FR, int, int) const {
        Cell o;
#pragma unroll
        for (int f = 0; f < 5; f++) o.v[f] = fmaf(dtdx, FL.v[f] - FR.v[f], c.v[f]);
        return o;
    }
    CG_D bool active(int line, int k, const unsigned char* mask) const {
        return MASKED ? lm.mask_on(mask, line, k) : true;
    }
    CG_D float wavespeed(const Cell& c, int, int) { return sr_wavespeed_fast(P, c.v, dims, &flags); }
    CG_D void flush_status(int* st) const {
        if (st && flags) atomicOr(st, ST_NEWTON_CAP);
    }
};

template <int AXIS, int LIM, bool MASKED>
inline SRFastPolicy<AXIS, LIM, MASKED> make_sr_fast(double gamma, double bias, int nx, int dims, double c2p64_above) {
    SRFastPolicy<AXIS, LIM, MASKED> p;
    const float w = (float)bias;
    p.NP.g1 = p.NP.hg1 = p.NP.gam = 0.0f;
    p.NP.wa = 0.5f * (1.0f + w);
    p.NP.wb = 0.5f * (1.0f - w);
    p.NP.hom = 0.5f * (1.0f - w);
    p.NP.hop = 0.5f * (1.0f + w);
    p.P.wa = p.NP.wa;
    p.P.wb = p.NP.wb;
    p.P.hom = p.NP.hom;
    p.P.hop = p.NP.hop;
    sr_fast_constants(p.P, gamma);
    p.P.w64 = c2p64_above > 0.0 ? (float)c2p64_above : 0.0f;  // W >= 1 > 0: threshold 0 always runs FP64
    p.lm.axis = AXIS;
    p.lm.nx = nx;
    p.dims = dims;
    p.dtdx = p.half_dtdx = p.q_dxdt = 0.0f;
    p.flags = 0;
    return p;
}

template <int AXIS, int LIM, bool MASKED>
inline NewtonFastPolicy<AXIS, LIM, MASKED> make_newton_fast(double gamma, double bias, int nx, int dims) {
    NewtonFastPolicy<AXIS, LIM, MASKED> p;
    const float g = (float)gamma, w = (float)bias;
    p.P.g1 = g - 1.0f;
    p.P.hg1 = 0.5f * (g - 1.0f);
    p.P.gam = g;
    p.P.wa = 0.5f * (1.0f + w);
    p.P.wb = 0.5f * (1.0f - w);
    p.P.hom = 0.5f * (1.0f - w);
    p.P.hop = 0.5f * (1.0f + w);
    p.lm.axis = AXIS;
    p.lm.nx = nx;
    p.dims = dims;
    p.dtdx = p.half_dtdx = p.q_dxdt = 0.0f;
    return p;
}

}  // namespace cg
