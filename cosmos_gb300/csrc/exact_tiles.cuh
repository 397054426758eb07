// FP64 reference-exact sweeps of single grids, in tiles: one thread per cell, both axes by one kernel.
//
// A block owns LC lines x P = NT / LC positions along the sweep; thread t has line t % LC, position t / LC.
// X sweeps take one line (a row) of 32 or 128 cells, Y sweeps four columns of 32 (a warp's loads are
// then whole 32-byte sectors).  What bounds these kernels is the FP64 pipe and the integer pipes that
// stand in for it (physics_exact.cuh), never memory, so the layout only has to give every SM the same
// number of warps: a marching thread per column (the form before this one) left a 389 x 509 grid with
// 400 warps on 152 SMs.  Each cell's conserved state is formed once and read by its neighbours from
// shared memory (before: three times in registers), each half-step evolution and each interface flux once
// per tile.  Measured with the integer-pipe arithmetic (GB300, whole solves against the marching,
// hardware-FP64 form): 389 x 509 Newtonian SLIC 0.50 -> 0.10 ms per sweep, 200 x 200 FORCE 0.113 -> 0.017,
// 181 x 230 SR 0.88 -> 0.11, 150 x 150 black-hole step 9.0 -> 2.6 ms, 128^2 Level-1 AMR run 79.5 -> 13.8 ms.
#pragma once
#include "policies.cuh"

namespace cg {

struct TileArgs {
    Geom G;
    double dx;
    Bias w;
    int lim, order;
    const double* src;
    double* dst;
    DtSrc ds;
    SweepOut out;
};

// The time step and its ratios, read by every thread from the controller (one broadcast load each).
CG_D bool tile_step(const DtSrc& ds, double dx, double& dt, StepRatio& r) {
    if (!ds.get(dt)) return false;
    r = ds.ratio(dt, dx);
    return true;
}

// where cell k of a line lies in a field
template <int AXIS> CG_D size_t tile_at(const Geom& G, int line, int k) {
    return AXIS == 0 ? (size_t)line * G.pitch + k : (size_t)k * G.pitch + line;
}
template <int AXIS> CG_D V5<double> tile_load(const Geom& G, const double* src, int line, int k) {
    const size_t at = tile_at<AXIS>(G, line, ghost_index(k, AXIS == 0 ? G.nx : G.ny, G.bc));
    V5<double> c;
#pragma unroll
    for (int f = 0; f < 5; f++) c.v[f] = src[f * G.fstride + at];
    return c;
}
template <int AXIS> CG_D void tile_store(const Geom& G, double* dst, int line, int k, const V5<double>& c) {
    const size_t at = tile_at<AXIS>(G, line, k);
#pragma unroll
    for (int f = 0; f < 5; f++) dst[f * G.fstride + at] = c.v[f];
}
template <int N> CG_D V5<double> sm_get(const double (&a)[5][N], int t) {
    V5<double> c;
#pragma unroll
    for (int f = 0; f < 5; f++) c.v[f] = a[f][t];
    return c;
}
template <int N> CG_D void sm_set(double (&a)[5][N], int t, const V5<double>& c) {
#pragma unroll
    for (int f = 0; f < 5; f++) a[f][t] = c.v[f];
}

// ---- coordinate-free systems (Newtonian, SR).  Position p owns cell c = s0 - 1 + p: its conserved state,
// its half-step evolution and the flux at its right interface; positions 1 .. P - 2 update.  MASKED (AMR
// levels): cells whose flag is off are copied, and only what an updating cell needs is evaluated.
// Four blocks of 128 threads per SM (at most 128 registers): 3, 5 or 6 measured within 3 %, so occupancy is
// not what bounds them.
template <class Sys, int AXIS, int ORDER, int NT, int LC, bool MASKED>
__global__ void __launch_bounds__(NT, 512 / NT) exact_tile_kernel(const __grid_constant__ ExactStages<Sys> S, TileArgs A) {
    constexpr int P = NT / LC;
    __shared__ double sU[5][NT + 2 * LC];  // conserved states of cells s0 - 2 .. s0 + P - 1
    __shared__ double sL[5][NT];           // conserved left-face state of the thread's cell
    __shared__ double sF[5][NT];           // flux at the right interface of the thread's cell
    __shared__ unsigned char sa[MASKED ? NT + LC : 1];
    const Geom& G = A.G;
    const int t = threadIdx.x, l = t % LC, p = t / LC;
    const int n = AXIS == 0 ? G.nx : G.ny;
    const int line = AXIS == 0 ? (int)blockIdx.y : (int)blockIdx.x * LC + l;
    const int s0 = (AXIS == 0 ? (int)blockIdx.x : (int)blockIdx.y) * (P - 2);
    const int send = min(s0 + P - 2, n);
    const int c = s0 - 1 + p;
    const bool in = AXIS == 0 || line < G.nx;
    const bool live = in && c <= send;             // cells beyond send neither update nor feed an interface
    const bool own = in && p >= 1 && c < send;     // updates (or copies) its cell
    double dt;
    StepRatio r;
    if (!tile_step(A.ds, A.dx, dt, r)) {  // inactive step: keep the ping-pong buffers consistent
        if (own) tile_store<AXIS>(G, A.dst, line, c, tile_load<AXIS>(G, A.src, line, c));
        return;
    }
    bool act = own;
    if (MASKED) {
        act = own && A.out.mask[AXIS == 0 ? (size_t)line * G.nx + c : (size_t)c * G.nx + line] != 0;
        sa[t] = act ? 1 : 0;
        if (p == P - 1) sa[NT + l] = 0;  // the cell after belongs to the next tile
    }
    if (MASKED && !__syncthreads_or(act) && !A.out.slot_set()) {  // nothing of the tile updates
        if (own) tile_store<AXIS>(G, A.dst, line, c, tile_load<AXIS>(G, A.src, line, c));
        return;
    }
    if (live) sm_set(sU, t + LC, S.cons(tile_load<AXIS>(G, A.src, line, c)));
    if (in && p == 0) sm_set(sU, t, S.cons(tile_load<AXIS>(G, A.src, line, s0 - 2)));
    if ((live && p == P - 1) || (in && c == send))  // c + 1 <= send + 1 <= n + 1: a valid ghost
        sm_set(sU, t + 2 * LC, S.cons(tile_load<AXIS>(G, A.src, line, c + 1)));
    __syncthreads();
    const bool next = MASKED && sa[t + LC] != 0;
    const bool need_flux = !MASKED || act || next;
    const bool need_faces = need_flux || (MASKED && p >= 1 && sa[t - LC] != 0);
    V5<double> R;
    if (ORDER == 2) {
        if (live && need_faces) {
            V5<double> L;
            S.faces(sm_get(sU, t), sm_get(sU, t + LC), sm_get(sU, t + 2 * LC), AXIS, r, L, R);
            sm_set(sL, t, L);
        }
        __syncthreads();
    }
    V5<double> Fr;
    if (live && c < send && p < P - 1 && need_flux) {  // right interface of c, between c and c + 1
        if (ORDER == 2) Fr = S.force(R, sm_get(sL, t + LC), AXIS, r);
        else Fr = S.force(sm_get(sU, t + LC), sm_get(sU, t + 2 * LC), AXIS, r);
        sm_set(sF, t, Fr);
    }
    __syncthreads();
    double ws = 0.0;
    unsigned long long* const slot = A.out.slot();
    if (own) {
        V5<double> nc;
        if (act) nc = S.update(sm_get(sU, t + LC), sm_get(sF, t - LC), Fr, r.d);
        else nc = tile_load<AXIS>(G, A.src, line, c);
        tile_store<AXIS>(G, A.dst, line, c, nc);
        if (slot) ws = S.wavespeed(nc, G.dims);
    }
    if (slot) block_max_to<NT>(slot, ws);
}

// ---- black hole.  Position p evaluates interface s0 + p (between cells s0 + p - 1 and s0 + p), each side's
// evolution at its own, separately rounded coordinates as the reference does, and updates cell s0 + p
// (p < P - 1).  Excision: a cell updates when it and its neighbours up to `reach` cells along both axes lie
// outside the horizon (Solvers/BlackHoleEulerSecondOrderSolver.cpp:44-46 in 1D, :81-85 in 2D; reach 1 for
// FORCE, Solvers/BlackHoleEulerFirstOrderSolver.cpp:94-95, :131-133).
CG_D bool gr_excised_near(const BHExact& b, int dims, int i, int j, double dx, int reach) {
    const double x = j * dx, y = dims == 1 ? 0.0 : i * dx;
    // far from the horizon (by a cell more than the stencil's reach) nothing of the stencil is inside
    const double ex = x - b.bx, ey = y - b.by, far = b.horizon + (reach + 1) * dx;
    if (far > 0.0 && ((ex * ex) + (ey * ey)) + (b.bz * b.bz) > 1.000001 * (far * far)) return false;
    if (dims == 1) {
        for (int d = -reach; d <= reach; d++)
            if (b.excised((j + d) * dx, 0.0, 0.0)) return true;
        return false;
    }
    if (b.excised(x, y, 0.0)) return true;
    for (int d = 1; d <= reach; d++) {
        if (b.excised((j - d) * dx, y, 0.0) || b.excised((j + d) * dx, y, 0.0) || b.excised(x, (i - d) * dx, 0.0) ||
            b.excised(x, (i + d) * dx, 0.0))
            return true;
    }
    return false;
}

struct GRStencil { V5<double> c[4]; };
__device__ __noinline__ V5<double> slow_interface(GRExact S, GRStencil q, int order, Pt xf, int axis, double dx,
                                                  StepRatio st, Bias w, int lim) {
    V5<double> F;
    gr_interface<double>(&S, q.c, order, xf, axis, dx, st, w, lim, F.v);
    return F;
}
__device__ __noinline__ V5<double> slow_gr_update(GRExact S, V5<double> c, V5<double> FL, V5<double> FR, Pt q, double d) {
    V5<double> o;
    gr_update<double>(&S, c, FL.v, FR.v, q, d, o.v);
    return o;
}
CG_D V5<xd> as_xd(const V5<double>& a) {
    V5<xd> o;
    load5(a.v, o.v);
    return o;
}

template <int AXIS, int NT, int LC>
__global__ void __launch_bounds__(NT) gr_tile_kernel(const __grid_constant__ GRExact S, TileArgs A) {
    constexpr int P = NT / LC;
    __shared__ double sc[5][NT + 3 * LC];  // cells s0 - 2 .. s0 + P (primitives)
    __shared__ double sF[5][NT];           // flux at the thread's interface
    __shared__ unsigned char sa[NT + LC];  // whether the cell left of the thread's interface updates
    const Geom& G = A.G;
    const int t = threadIdx.x, l = t % LC, p = t / LC;
    const int n = AXIS == 0 ? G.nx : G.ny;
    const int line = AXIS == 0 ? (int)blockIdx.y : (int)blockIdx.x * LC + l;
    const int s0 = (AXIS == 0 ? (int)blockIdx.x : (int)blockIdx.y) * (P - 1);
    const int send = min(s0 + P - 1, n);
    const int k = s0 + p;
    const bool in = AXIS == 0 || line < G.nx;
    const bool own = in && p < P - 1 && k < send;
    double dt;
    StepRatio r;
    if (!tile_step(A.ds, A.dx, dt, r)) {
        if (own) tile_store<AXIS>(G, A.dst, line, k, tile_load<AXIS>(G, A.src, line, k));
        return;
    }
    const int ci = AXIS == 0 ? line : k, cj = AXIS == 0 ? k : line;
    bool act = own && (!A.out.mask || A.out.mask[(size_t)ci * G.nx + cj] != 0);
    act = act && !gr_excised_near(S.bh, G.dims, ci, cj, A.dx, A.order == 2 ? 2 : 1);
    if (in && p == 0) sa[t] = 0;
    sa[t + LC] = act ? 1 : 0;
    for (int q = p; q < P + 3; q += P) {
        const int m = s0 - 2 + q;
        if (in && m <= send + 1) sm_set(sc, q * LC + l, tile_load<AXIS>(G, A.src, line, m));
    }
    __syncthreads();
    const Pt xf = AXIS == 0 ? Pt{(k - 0.5) * A.dx, line * A.dx, 0.0} : Pt{line * A.dx, (k - 0.5) * A.dx, 0.0};
    if (in && k <= send && (act || sa[t])) {
        V5<xd> q[4];
        xd F[5];
        V5<double> o;
#pragma unroll
        for (int m = 0; m < 4; m++) q[m] = as_xd(sm_get(sc, t + m * LC));
        gr_interface<xd>(&S, q, A.order, xf, AXIS, A.dx, r, A.w, A.lim, F);
        store5(F, o.v);
        if (any_nonfinite(F, 5)) {
            GRStencil g;
            for (int m = 0; m < 4; m++) g.c[m] = sm_get(sc, t + m * LC);
            o = slow_interface(S, g, A.order, xf, AXIS, A.dx, r, A.w, A.lim);
        }
        sm_set(sF, t, o);
    }
    __syncthreads();
    if (own) {
        const V5<double> c = sm_get(sc, t + 2 * LC);
        V5<double> nc = c;
        if (act) {
            const Pt at{cj * A.dx, ci * A.dx, 0.0};
            const V5<double> FL = sm_get(sF, t), FR = sm_get(sF, t + LC);
            xd fl[5], fr[5], o[5];
            load5(FL.v, fl);
            load5(FR.v, fr);
            gr_update<xd>(&S, as_xd(c), fl, fr, at, r.d, o);
            store5(o, nc.v);
            if (any_nonfinite(o, 5)) nc = slow_gr_update(S, c, FL, FR, at, r.d);
        }
        tile_store<AXIS>(G, A.dst, line, k, nc);
    }
}

}  // namespace cg
