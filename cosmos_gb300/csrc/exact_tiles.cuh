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

// Threads of a block of the black-hole kernels at most: at 168 registers each they fill the SM's file.
constexpr int kLockThreads = 384;

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
CG_D V5<double> tile_get(const double* a, int m, int t) {  // of [5][m]
    V5<double> c;
#pragma unroll
    for (int f = 0; f < 5; f++) c.v[f] = a[f * m + t];
    return c;
}
CG_D void tile_set(double* a, int m, int t, const V5<double>& c) {
#pragma unroll
    for (int f = 0; f < 5; f++) a[f * m + t] = c.v[f];
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
    __shared__ double sL[5][NT];           // conserved left-face state of the thread's cell (order 1: its flux)
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
    if (ORDER == 1) {  // the cell's flux, for its two interfaces (FORCE takes it of the cells themselves)
        if (live && need_faces) {
            R = S.flux(sm_get(sU, t + LC), AXIS);
            sm_set(sL, t, R);
        }
        __syncthreads();
    }
    V5<double> Fr;
    if (live && c < send && p < P - 1 && need_flux) {  // right interface of c, between c and c + 1
        if (ORDER == 2) Fr = S.force(R, sm_get(sL, t + LC), AXIS, r);
        else Fr = S.force_of(sm_get(sU, t + LC), sm_get(sU, t + 2 * LC), R, sm_get(sL, t + LC), AXIS, r);
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

// ---- the same sweep with two threads per cell, for grids (or AMR levels) too small to give every SM's four
// schedulers a warp: there a tile's time is one warp's 9000 instructions in a row, not the pipes.  Threads
// 2 k and 2 k + 1 share cell k of the tile, one face each: the conserved states are formed by all threads at
// once (the even ones the cells, two odd ones the tile's outer neighbours), the five slopes three and three,
// each thread then takes its own face through flux, evolution, recovery and its FORCE flux; the odd thread
// evaluates the interface to the right and updates the cell.  Three fluxes, two recoveries and two
// conversions in a row instead of five, three and three to five.  Values that two threads of a cell exchange
// go through shuffles, so LC x 2 threads of a position stay in one warp.
struct ThreadPair {
    int side;
    unsigned mask;  // the warp's threads that take part (both of a cell or neither)
    CG_D V5<double> other(const V5<double>& a) const {
        V5<double> o;
#pragma unroll
        for (int f = 0; f < 5; f++) o.v[f] = __shfl_xor_sync(mask, a.v[f], 1);
        return o;
    }
    CG_D V5<xd> other(const V5<xd>& a) const {
        V5<xd> o;
#pragma unroll
        for (int f = 0; f < 5; f++) o.v[f] = xd(__shfl_xor_sync(mask, a.v[f].v, 1));
        return o;
    }
};
template <class Sys, int AXIS, int NT, int LC, bool MASKED>
__global__ void __launch_bounds__(NT) exact_pair_kernel(const __grid_constant__ ExactStages<Sys> S, TileArgs A) {
    constexpr int NC = NT / 2, P = NC / LC;
    __shared__ double sU[5][NC + 2 * LC];      // conserved states of cells s0 - 2 .. s0 + P - 1
    __shared__ double sG[5][NC], sH[5][NC];    // left-face state of the cell and its flux
    __shared__ double sF[5][NC];               // flux at the right interface of the cell
    __shared__ unsigned char sa[MASKED ? NC + LC : 1];
    const Geom& G = A.G;
    const int side = threadIdx.x & 1, t = threadIdx.x >> 1, l = t % LC, p = t / LC;
    const int n = AXIS == 0 ? G.nx : G.ny;
    const int line = AXIS == 0 ? (int)blockIdx.y : (int)blockIdx.x * LC + l;
    const int s0 = (AXIS == 0 ? (int)blockIdx.x : (int)blockIdx.y) * (P - 2);
    const int send = min(s0 + P - 2, n);
    const int c = s0 - 1 + p;
    const bool in = AXIS == 0 || line < G.nx;
    const bool live = in && c <= send;
    const bool own = in && p >= 1 && c < send;
    double dt;
    StepRatio r;
    const bool on = tile_step(A.ds, A.dx, dt, r);
    bool act = on && own;
    if (MASKED) {
        act = act && A.out.mask[AXIS == 0 ? (size_t)line * G.nx + c : (size_t)c * G.nx + line] != 0;
        if (side == 0) sa[t] = act ? 1 : 0;
        if (side == 0 && p == P - 1) sa[NC + l] = 0;  // the cell after belongs to the next tile
    }
    if (!on || (MASKED && !__syncthreads_or(act) && !A.out.slot_set())) {  // nothing of the tile updates
        if (own && side == 1) tile_store<AXIS>(G, A.dst, line, c, tile_load<AXIS>(G, A.src, line, c));
        return;
    }
    {
        // even threads: their cell; odd threads: the cell before the tile's first or after its last (the one
        // after `send` where the line ends inside the tile), else the even thread's again
        int k = c, at = t + LC;
        if (side == 1 && p == 0) {
            k = s0 - 2;
            at = t;
        } else if (side == 1 && (p == P - 1 || c == send)) {
            k = c + 1;
            at = t + 2 * LC;
        }
        if (live) {
            const V5<double> u = S.cons(tile_load<AXIS>(G, A.src, line, k));
            if (side == 0 || k != c) sm_set(sU, at, u);
        }
    }
    __syncthreads();
    const bool next = MASKED && sa[t + LC] != 0;
    const bool need_flux = !MASKED || act || next;
    const bool need_faces = live && (need_flux || (MASKED && p >= 1 && sa[t - LC] != 0));
    V5<double> u, f;  // the thread's face state and its flux
    const ThreadPair both{side, __ballot_sync(0xffffffffu, need_faces)};
    if (need_faces) {
        const V5<double> um = sm_get(sU, t + LC);
        V5<double> hs;
#pragma unroll
        for (int k = 0; k < 3; k++) {  // fields 0, 1, 2 or 2, 3, 4
            const int q = k + 2 * side;
            const double m = sU[q][t + LC], h = S.half_slope_of(m - sU[q][t], sU[q][t + 2 * LC] - m);
            const double o = __shfl_xor_sync(both.mask, h, 1);
            hs.v[k] = side == 0 ? h : o;
            hs.v[k + 2] = side == 0 ? o : h;
        }
        V5<double> V;
#pragma unroll
        for (int k = 0; k < 5; k++) V.v[k] = side == 0 ? um.v[k] - hs.v[k] : um.v[k] + hs.v[k];
        const V5<double> F = S.flux(V, AXIS), O = both.other(F);
        const FaceOf e = S.face_of_side(V, side == 0 ? F : O, side == 0 ? O : F, AXIS, r);
        u = e.u;
        if (__shfl_xor_sync(both.mask, (int)e.bad, 1) || e.bad) {  // as S.faces: both faces again in hardware FP64
            const FacePair o = slow_faces(S.sys, sm_get(sU, t), um, sm_get(sU, t + 2 * LC), AXIS, r, S.w, S.lim);
            u = side == 0 ? o.L : o.R;
        }
        f = S.flux(u, AXIS);
        if (side == 0) {
            sm_set(sG, t, u);
            sm_set(sH, t, f);
        }
    }
    __syncthreads();
    V5<double> Fr;
    if (side == 1 && live && c < send && p < P - 1 && need_flux) {
        Fr = S.force_of(u, sm_get(sG, t + LC), f, sm_get(sH, t + LC), AXIS, r);
        sm_set(sF, t, Fr);
    }
    __syncthreads();
    double ws = 0.0;
    unsigned long long* const slot = A.out.slot();
    if (own && side == 1) {
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
    gr_interface(&S, q.c, order, xf, axis, dx, st, w, lim, F.v);
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

// A block has LC lines of P interfaces each (one fewer cells update).  PAIR: threads 2 k and 2 k + 1 share interface k,
// one side each, and both evaluate FORCE of the two: six recoveries in a row instead of ten.
template <int AXIS, bool PAIR>
__global__ void __launch_bounds__(kLockThreads) gr_tile_kernel(const __grid_constant__ GRExact S, TileArgs A, int P, int LC) {
    extern __shared__ double smem[];
    double* const sc = smem;                    // [5][(P + 3) LC]: cells s0 - 2 .. s0 + P (primitives)
    double* const sF = sc + 5 * (P + 3) * LC;   // [5][P LC]: flux at the thread's interface
    unsigned char* const sa = (unsigned char*)(sF + 5 * P * LC);  // [(P + 1) LC]: whether the cell to its left updates
    const Geom& G = A.G;
    const int side = PAIR ? threadIdx.x & 1 : 0, x = PAIR ? threadIdx.x >> 1 : threadIdx.x;
    const int l = AXIS == 0 ? x / P : x % LC, p = AXIS == 0 ? x % P : x / LC, t = p * LC + l;
    const int n = AXIS == 0 ? G.nx : G.ny;
    const int line = (int)(AXIS == 0 ? blockIdx.y : blockIdx.x) * LC + l;
    const int s0 = (int)(AXIS == 0 ? blockIdx.x : blockIdx.y) * (P - 1);
    const int send = min(s0 + P - 1, n);
    const int k = s0 + p;
    const bool in = x < P * LC && line < (AXIS == 0 ? G.ny : G.nx);
    const bool own = in && p < P - 1 && k < send;  // (of a pair, side 0 updates)
    const int mc = (P + 3) * LC, mf = P * LC;
    double dt;
    StepRatio r;
    if (!tile_step(A.ds, A.dx, dt, r)) {
        if (own && side == 0) tile_store<AXIS>(G, A.dst, line, k, tile_load<AXIS>(G, A.src, line, k));
        return;
    }
    const int ci = AXIS == 0 ? line : k, cj = AXIS == 0 ? k : line;
    bool act = own && (!A.out.mask || A.out.mask[(size_t)ci * G.nx + cj] != 0);
    act = act && !gr_excised_near(S.bh, G.dims, ci, cj, A.dx, A.order == 2 ? 2 : 1);
    if (in && p == 0) sa[t] = 0;
    if (in) sa[t + LC] = act ? 1 : 0;
    for (int q = p + (PAIR ? side * P : 0); q < P + 3; q += P) {
        const int m = s0 - 2 + q;
        if (in && m <= send + 1) {
            tile_set(sc, mc, q * LC + l, tile_load<AXIS>(G, A.src, line, m));
        }
    }
    __syncthreads();
    const V5<double> c = in ? tile_get(sc, mc, t + 2 * LC) : V5<double>{};
    const bool need = in && k <= send && (act || sa[t]);
    if (own && !act && side == 0) tile_store<AXIS>(G, A.dst, line, k, c);
    const ThreadPair both{side, PAIR ? __ballot_sync(0xffffffffu, need) : 0u};
    if (!need) return;
    const Pt xf = AXIS == 0 ? Pt{(k - 0.5) * A.dx, line * A.dx, 0.0} : Pt{line * A.dx, (k - 0.5) * A.dx, 0.0};
    xd F[5];
    if (PAIR) {
        V5<xd> q[3], u, f;
#pragma unroll
        for (int m = 0; m < 3; m++) q[m] = as_xd(tile_get(sc, mc, t + (side + m) * LC));
        gr_interface_side(&S, q, side, A.order, xf, AXIS, A.dx, r, A.w, A.lim, u, f);
        const V5<xd> ou = both.other(u), of = both.other(f);
        gr_interface_force(&S, side == 0 ? u : ou, side == 0 ? ou : u, side == 0 ? f : of, side == 0 ? of : f, xf,
                           AXIS, r, F);
    } else {
        V5<xd> q[4];
#pragma unroll
        for (int m = 0; m < 4; m++) q[m] = as_xd(tile_get(sc, mc, t + m * LC));
        gr_interface(&S, q, A.order, xf, AXIS, A.dx, r, A.w, A.lim, F);
    }
    V5<double> o;
    store5(F, o.v);
    if (side == 0) {
        if (any_nonfinite(F, 5)) {
            GRStencil g;
            for (int m = 0; m < 4; m++) g.c[m] = tile_get(sc, mc, t + m * LC);
            o = slow_interface(S, g, A.order, xf, AXIS, A.dx, r, A.w, A.lim);
        }
        tile_set(sF, mf, t, o);
    }
    __syncthreads();
    if (!act || side != 0) return;
    const Pt at{cj * A.dx, ci * A.dx, 0.0};
    const V5<double> FR = tile_get(sF, mf, t + LC);
    xd fl[5], fr[5], un[5];
    load5(o.v, fl);
    load5(FR.v, fr);
    gr_update<xd>(&S, as_xd(c), fl, fr, at, r.d, un);
    V5<double> nc;
    store5(un, nc.v);
    if (any_nonfinite(un, 5)) nc = slow_gr_update(S, c, o, FR, at, r.d);
    tile_store<AXIS>(G, A.dst, line, k, nc);
}

}  // namespace cg
