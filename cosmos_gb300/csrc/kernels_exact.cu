// FP64 reference-exact kernels.  Compiled with --fmad=false so that every double operation is
// rounded exactly as the reference's (built with -ffp-contract=off) -- results are bit-identical.
#include <cstring>

#include "exact_tiles.cuh"
#include "launch.h"
#include "policies.cuh"

namespace cg {

namespace {

template <class Sys>
ExactPolicy<Sys> make_policy(const SweepArgs& a, const Sys& sys) {
    ExactPolicy<Sys> p;
    p.st = ExactStages<Sys>{sys, make_bias(a.bias), a.lim};
    p.lm.axis = a.G.axis;
    p.lm.nx = a.G.nx;
    p.dims = a.G.dims;
    p.ny = a.G.ny;
    p.dx = a.dx;
    p.dt = 0.0;
    p.r = StepRatio{0.0, 0.0};
    return p;
}

TileArgs tile_args(const SweepArgs& a) {
    return TileArgs{a.G, a.dx, make_bias(a.bias), a.lim, a.order, (const double*)a.src, (double*)a.dst, a.ds, a.out};
}

template <class Sys, int AXIS, int NT, int LC>
void run_tiles(const ExactStages<Sys>& S, const SweepArgs& a) {
    constexpr int T = NT / LC - 2;
    const Geom& G = a.G;
    const TileArgs A = tile_args(a);
    const dim3 grid = AXIS == 0 ? dim3((G.nx + T - 1) / T, G.ny) : dim3((G.nx + LC - 1) / LC, (G.ny + T - 1) / T);
    if (a.out.mask) {
        if (a.order == 2) exact_tile_kernel<Sys, AXIS, 2, NT, LC, true><<<grid, NT, 0, a.stream>>>(S, A);
        else exact_tile_kernel<Sys, AXIS, 1, NT, LC, true><<<grid, NT, 0, a.stream>>>(S, A);
    } else {
        if (a.order == 2) exact_tile_kernel<Sys, AXIS, 2, NT, LC, false><<<grid, NT, 0, a.stream>>>(S, A);
        else exact_tile_kernel<Sys, AXIS, 1, NT, LC, false><<<grid, NT, 0, a.stream>>>(S, A);
    }
}

template <class Sys, int AXIS, int NT, int LC>
void run_pairs(const ExactStages<Sys>& S, const SweepArgs& a) {
    constexpr int T = NT / 2 / LC - 2;
    const Geom& G = a.G;
    const TileArgs A = tile_args(a);
    const dim3 grid = AXIS == 0 ? dim3((G.nx + T - 1) / T, G.ny) : dim3((G.nx + LC - 1) / LC, (G.ny + T - 1) / T);
    if (a.out.mask) exact_pair_kernel<Sys, AXIS, NT, LC, true><<<grid, NT, 0, a.stream>>>(S, A);
    else exact_pair_kernel<Sys, AXIS, NT, LC, false><<<grid, NT, 0, a.stream>>>(S, A);
}

// SLIC sweeps of at most five warps of cells to an SM go two threads to a cell (1000 cells in 1D: 20.4 -> 15.9 us per
// step; 128^2 with a finer level, every launch this small: 12.5 -> 12.2 ms per run; at 9.5 warps to an SM, SR
// 181 x 230, the pairs' extra work costs more than it hides: 340 -> 398).  Masked sweeps count the cells of the
// whole level, of which few update, so up to twenty: a whole Level-1 run of a blast on 128^2 (5 % of the finer level
// refined) 2.79 ms with five, 2.76 with twenty (SR 5.74, 4.88); where the whole level is refined twenty costs what
// it costs unmasked (3.16, 3.80; SR 7.31, 8.99).
// Otherwise X sweeps take one-warp tiles (30 of 32 cells update) where they waste fewer threads on the row's end
// than the larger ones (126 of 128), or where those would not give every SM a block.  389 x 509 (544 threads a
// row instead of 640): 349 -> 305 us per step; 1024^2 (1120 against 1152): 1613 -> 1532; SR 512^2 1874 -> 1690.
// (Blocks of several lines shaped to fill whole waves, as the black hole's below, measured 303 -> 310 .. 341,
// 1532 -> 1456 .. 1655 and 1690 -> 1602 .. 1928 for caps of 64 to 512 threads: no shape was better at all three.)
template <class Sys>
cudaError_t run_sweep(const Sys& sys, const SweepArgs& a) {
    const ExactStages<Sys> S{sys, make_bias(a.bias), a.lim};
    const int wide = (a.G.nx + 125) / 126;
    const long long warps = (long long)((a.G.nx + 29) / 30) * a.G.ny;
    if (a.order == 2 && warps <= (long long)(a.out.mask ? 20 : 5) * device_sm_count()) {
        if (a.G.axis == 1) run_pairs<Sys, 1, 256, 4>(S, a);
        else run_pairs<Sys, 0, 64, 1>(S, a);
        count_launch();
        return cudaGetLastError();
    }
    if (a.G.axis == 1) run_tiles<Sys, 1, 128, 4>(S, a);
    else if ((a.G.nx + 29) / 30 * 32 <= wide * 128 || wide * (long long)a.G.ny < device_sm_count()) run_tiles<Sys, 0, 32, 1>(S, a);
    else run_tiles<Sys, 0, 128, 1>(S, a);
    count_launch();
    return cudaGetLastError();
}

// Black-hole sweeps of at most five warps of cells to an SM take two threads to an interface: 150^2 2196 -> 1835 us
// per step with the launch shapes below (200^2, at 8.2 warps: 2635 without, 2730 with).
bool gr_pairs(const Geom& G) { return (long long)G.nx * G.ny <= 5ll * 32 * device_sm_count(); }

// Shape of a black-hole sweep's blocks: `lines` lines by `points` interfaces (one fewer cells update), `each`
// threads to an interface.  Of the ways to cut a line into equal pieces and to put pieces together, the one whose
// waves of blocks cost least: a wave has its warps' work and about ten warps' worth of latency.  A fixed 64 or
// 128 threads left the last wave and the last tile of a line nearly empty, and blocks that run apart
// fetch the 100 KB of code apart: 400^2 13.7 -> 8.6 ms per step, with the source step's lockstep blocks.
struct TileShape { int points, lines, threads; size_t bytes; };
TileShape tile_shape(int n, int lines, int each) {
    constexpr int kWaveWarps = 10, kWarps = kLockThreads / 32;
    TileShape best{0, 0, 0, 0};
    long long cost = 0;
    const long long sms = device_sm_count();
    const int most = kLockThreads / each;
    int m = (n + most - 2) / (most - 1);
    for (int tried = 0; tried < 24 && m <= n; tried++, m++) {
        const int P = (n + m - 1) / m + 1;
        if (best.points && P < 17) break;
        for (int lc = 1; lc * P <= most && lc <= lines; lc++) {
            const size_t bytes = (size_t)lc * (5 * (2 * P + 3) * sizeof(double) + P + 1);
            if (bytes > 48 * 1024) break;
            const int warps = (P * lc * each + 31) / 32, resident = kWarps / warps;
            const long long blocks = (long long)((n + P - 2) / (P - 1)) * ((lines + lc - 1) / lc);
            const long long slots = sms * resident, waves = (blocks + slots - 1) / slots;
            const long long per_sm = waves == 1 ? (blocks + sms - 1) / sms : resident;
            const long long c = waves * (kWaveWarps + per_sm * warps);
            if (!best.points || c < cost) {
                best = TileShape{P, lc, warps * 32, bytes};
                cost = c;
            }
        }
    }
    return best;
}

GRExact make_gr(const SweepArgs& a, int* status = nullptr) { return GRExact(a.gamma, a.bh, a.dx, status); }

}  // namespace

cudaError_t launch_sweep_exact(const SweepArgs& a) {
    if (a.system == 0) return run_sweep(NewtonExact(a.gamma), a);
    if (a.system == 1) return run_sweep(SRExact(a.gamma, a.out.status), a);
    const GRExact S = make_gr(a, a.out.status);
    const TileArgs A = tile_args(a);
    const Geom& G = a.G;
    const bool pair = gr_pairs(G);
    const int n = G.axis == 0 ? G.nx : G.ny, lines = G.axis == 0 ? G.ny : G.nx;
    const TileShape h = tile_shape(n, lines, pair ? 2 : 1);
    const int groups = (lines + h.lines - 1) / h.lines, tiles = (n + h.points - 2) / (h.points - 1);
    const dim3 grid(G.axis == 0 ? tiles : groups, G.axis == 0 ? groups : tiles);
    const auto kernel = G.axis == 0 ? (pair ? gr_tile_kernel<0, true> : gr_tile_kernel<0, false>)
                                    : (pair ? gr_tile_kernel<1, true> : gr_tile_kernel<1, false>);
    kernel<<<grid, h.threads, h.bytes, a.stream>>>(S, A, h.points, h.lines);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_wavespeed_exact(const SweepArgs& a, unsigned long long* slot) {
    constexpr int NT = 256;
    Geom G = a.G;
    SweepArgs b = a;
    b.G.axis = 0;
    SweepOut o = a.out;
    if (slot) { o.smax = slot; o.ws_ctl = nullptr; }
    const size_t n = (size_t)G.nx * G.ny;
    int blocks = (int)((n + NT - 1) / NT);
    if (blocks > device_sm_count() * 16) blocks = device_sm_count() * 16;
    const double* src = (const double*)a.src;
    if (a.system == 0) wavespeed_kernel<ExactPolicy<NewtonExact>, NT><<<blocks, NT, 0, a.stream>>>(make_policy(b, NewtonExact(a.gamma)), b.G, src, o);
    else if (a.system == 1) wavespeed_kernel<ExactPolicy<SRExact>, NT><<<blocks, NT, 0, a.stream>>>(make_policy(b, SRExact(a.gamma)), b.G, src, o);
    else wavespeed_kernel<ExactPolicy<GRExact>, NT><<<blocks, NT, 0, a.stream>>>(make_policy(b, make_gr(a)), b.G, src, o);
    count_launch();
    return cudaGetLastError();
}

// ------------------------------------------------------------------ GR RK4 source step
// Solvers/BlackHoleEulerForcingSolver.cpp:187-250: per cell away from the horizon (cell and its
// 2 (1D) or 4 (2D) neighbours outside), conserved neighbours from a 1-ghost transmissive copy,
// classical RK4 with interleaved fractional sweeps, converted back at the cell.
// Cell (j, i) of the grid and its neighbours' coordinates, each index times dx as the reference has them.
struct RkAt {
    int j, i;
    double dx;
    CG_D Pt at(int dj, int di) const { return Pt{(j + dj) * dx, (i + di) * dx, 0.0}; }
};
struct RkCell { V5<double> c[5]; };  // primitives of the left, right, top and bottom neighbours and of the cell
template <class T, class Team>
CG_D V5<T> rk_source_cell(const Team& team, const GRExact* S, int dims, const RkCell& c, RkAt a, double dt,
                          const StepRatio& sr, const Bias& w, int lim) {
    V5<T> u[5];
    Metric<T> g;
#pragma unroll 1
    for (int n = 0; n < 5; n++) {
        if (dims == 1 && (n == 2 || n == 3)) continue;
        V5<T> p;
#pragma unroll
        for (int f = 0; f < 5; f++) p.v[f] = T(c.c[n].v[f]);
        gr_metric(S, a.at(n == 0 ? -1 : n == 1 ? 1 : 0, n == 2 ? -1 : n == 3 ? 1 : 0), &g);
        u[n] = gr_cons(S, &g, p);
    }
    const V5<T> nc = rk_cell_exact(team, S, dims, u, a.at(0, 0), a.dx, dt, sr, w, lim, &g);
    return gr_prim(S, &g, nc);
}
__device__ __noinline__ V5<double> slow_rk(GRExact S, int dims, RkCell c, RkAt a, double dt, StepRatio sr, Bias w, int lim) {
    return rk_source_cell<double>(OneThread{}, &S, dims, c, a, dt, sr, w, lim);
}

// One thread per cell, 350 000 instructions a warp out of 100 KB of code: with a warp or two to a scheduler, the
// instruction fetches bound it (a third of a warp's time).  A block has all the cells that an SM gets
// (up to 384; whole waves of blocks), and its warps run the stages in lockstep, so that one fetch serves them:
// without the barriers 150^2 is 2020 instead of 1820 us per step and 400^2 9585 instead of 8570.  (Two threads
// per cell, one for each side's neighbours, have 0.7 of the instructions in a row, but twice the warps: 2000.)
struct Lockstep { CG_D void sync() const { __syncthreads(); } };  // threads that have left do not count
__global__ void __launch_bounds__(kLockThreads) rk_source_kernel(const __grid_constant__ GRExact sys, Geom G, double dx,
                                                                 Bias w, int lim, const double* __restrict__ src,
                                                                 double* __restrict__ dst, DtSrc ds) {
    const size_t cell = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int i = (int)(cell / G.nx), j = (int)(cell - (size_t)i * G.nx);
    const size_t idx = (size_t)i * G.pitch + j;
    double dt;
    const bool in = i < G.ny, act = in && ds.get(dt) && !gr_excised_near(sys.bh, G.dims, i, j, dx, 1);
    if (!act) {
        if (in) {
#pragma unroll
            for (int f = 0; f < 5; f++) dst[f * G.fstride + idx] = src[f * G.fstride + idx];
        }
        return;
    }
    auto ld = [&](int ii, int jj, V5<double>& p) {
        const size_t k = (size_t)ghost_index(ii, G.ny, 0) * G.pitch + ghost_index(jj, G.nx, 0);
#pragma unroll
        for (int f = 0; f < 5; f++) p.v[f] = src[f * G.fstride + k];
    };
    RkCell c;
    ld(i, j - 1, c.c[0]);
    ld(i, j + 1, c.c[1]);
    if (G.dims == 2) {
        ld(i - 1, j, c.c[2]);
        ld(i + 1, j, c.c[3]);
    }
    ld(i, j, c.c[4]);
    const RkAt at{j, G.dims == 1 ? 0 : i, dx};
    const StepRatio sr = ds.ratio(dt, dx);
    const V5<xd> nc = rk_source_cell<xd>(Lockstep{}, &sys, G.dims, c, at, dt, sr, w, lim);
    V5<double> o;
    store5(nc.v, o.v);
    if (any_nonfinite(nc.v, 5)) o = slow_rk(sys, G.dims, c, at, dt, sr, w, lim);
#pragma unroll
    for (int f = 0; f < 5; f++) dst[f * G.fstride + idx] = o.v[f];
}

cudaError_t launch_rk_source_exact(const SweepArgs& a) {
    const long long cells = (long long)a.G.nx * a.G.ny, sms = device_sm_count();
    const long long waves = (cells + sms * kLockThreads - 1) / (sms * kLockThreads);
    const int threads = (int)((cells + sms * waves - 1) / (sms * waves) + 31) / 32 * 32;
    rk_source_kernel<<<(unsigned)((cells + threads - 1) / threads), threads, 0, a.stream>>>(
        make_gr(a, a.out.status), a.G, a.dx, make_bias(a.bias), a.lim, (const double*)a.src, (double*)a.dst, a.ds);
    count_launch();
    return cudaGetLastError();
}

// ------------------------------------------------------------------ conversions
__global__ void prim_in_exact_kernel(const double* __restrict__ aos, double* __restrict__ soa, Geom G) {
    const size_t n = (size_t)G.nx * G.ny;
    for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) {
        const size_t i = c / G.nx, j = c % G.nx;
#pragma unroll
        for (int f = 0; f < 5; f++) soa[f * G.fstride + i * G.pitch + j] = aos[5 * c + f];
    }
}
__global__ void prim_out_exact_kernel(const double* __restrict__ soa, double* __restrict__ aos, Geom G) {
    const size_t n = (size_t)G.nx * G.ny;
    for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) {
        const size_t i = c / G.nx, j = c % G.nx;
#pragma unroll
        for (int f = 0; f < 5; f++) aos[5 * c + f] = soa[f * G.fstride + i * G.pitch + j];
    }
}
static int grid_for(size_t n) {
    size_t b = (n + 255) / 256;
    return (int)(b > device_sm_count() * 32 ? device_sm_count() * 32 : (b ? b : 1));
}
cudaError_t launch_prim_in_exact(const double* aos, void* soa, const Geom& G, cudaStream_t st) {
    prim_in_exact_kernel<<<grid_for((size_t)G.nx * G.ny), 256, 0, st>>>(aos, (double*)soa, G);
    count_launch();
    return cudaGetLastError();
}
cudaError_t launch_prim_out_exact(const void* soa, double* aos, const Geom& G, cudaStream_t st) {
    prim_out_exact_kernel<<<grid_for((size_t)G.nx * G.ny), 256, 0, st>>>((const double*)soa, aos, G);
    count_launch();
    return cudaGetLastError();
}

// ------------------------------------------------------------------ step controller
__global__ void dt_kernel(StepCtl* c) {
    if (threadIdx.x == 0 && blockIdx.x == 0) step_ctl_advance(c);
}
cudaError_t launch_dt_kernel(StepCtl* ctl, cudaStream_t st) {
    dt_kernel<<<1, 32, 0, st>>>(ctl);
    count_launch();
    return cudaGetLastError();
}

// ------------------------------------------------------------------ AMR flagging
// Conserved state of a cell for the flag passes: FP64 storage and the FP32 black-hole storage hold
// primitives (converted with the system's exact cons), FP32 Newtonian and SR storage holds
// conserved values already.
struct ConsLoader {
    int system, precision;
    Geom G;
    const void* state;
    NewtonExact nw;
    SRExact sr;
    GRExact gr;
    CG_D void get(int i, int j, Pt q, double* u) const {
        const size_t k = (size_t)ghost_index(i, G.ny, 0) * G.pitch + ghost_index(j, G.nx, 0);
        if (precision == 1 && system != 2) {  // FP32 Newtonian / SR storage is conserved
            const float* s = (const float*)state;
#pragma unroll
            for (int f = 0; f < 5; f++) u[f] = (double)s[f * G.fstride + k];
            return;
        }
        // primitives: FP64 storage, and the FP32 black-hole storage
        double p[5];
#pragma unroll
        for (int f = 0; f < 5; f++)
            p[f] = precision == 1 ? (double)((const float*)state)[f * G.fstride + k]
                                  : ((const double*)state)[f * G.fstride + k];
        cons_of(p, q, u);
    }
    // Newtonian and SR conversions on the integer pipes, as in the sweeps
    CG_D void cons_of(const double* p, Pt q, double* u) const {
        if (system == 0) give(ExactStages<NewtonExact>{nw, Bias{}, 0}.cons(five(p)), u);
        else if (system == 1) give(ExactStages<SRExact>{sr, Bias{}, 0}.cons(five(p)), u);
        else gr.cons(p, q, u);
    }
    CG_D void prim_of(const double* u, Pt q, double* p) const {
        if (system == 0) give(ExactStages<NewtonExact>{nw, Bias{}, 0}.prim(five(u)), p);
        else if (system == 1) give(ExactStages<SRExact>{sr, Bias{}, 0}.prim(five(u)), p);
        else gr.prim(u, q, p);
    }
};

// Whether |x / div| >= tol, 20 times per cell of the passes below: the quotient is formed only where |x| lies
// within 2^-50 of tol div, relatively, or that product is no ordinary number; elsewhere its rounding cannot
// matter.  Integer comparisons of the bit patterns (a quotient on the FP64 pipe is 141 cycles a warp).
struct Reach {
    double div, tol;
    long long lo, hi;  // |x| below lo: no; above hi: yes
    Reach(double d, double t) : div(d), tol(t), lo(0), hi(0x7ff0000000000000ll) {
        const double m = t * d;
        if (!(d > 0.0 && t > 1e-290 && t < 1e290 && m > 1e-290 && m < 1e290)) return;
        const double l = m * (1.0 - 0x1p-50), h = m * (1.0 + 0x1p-50);
        memcpy(&lo, &l, sizeof lo);
        memcpy(&hi, &h, sizeof hi);
    }
    CG_D bool operator()(double x) const {
        const long long a = __double_as_longlong(x) & 0x7fffffffffffffffll;
        if (a < lo) return false;
        if (a > hi && a <= 0x7ff0000000000000ll) return true;
        return fabs(x / div) >= tol;
    }
};

// Refinement pass, AMR/EulerAMR.cpp:207-229 (1D) and :400-431 (2D); the SR and GR Level-1 drivers
// read the bottom neighbour at [i+2][j+2] (AMR/RelativisticEulerAMR.cpp:422,
// AMR/BlackHoleEulerAMR.cpp:490), whose corner ghost keeps the default state (1,0,0,0,1).
// The Level-2 drivers' passes (AMR/EulerAMR.cpp:643-664 coarse, :699-722 intermediate, and the SR
// twins, whose coarse pass reads [i+2][j+1], AMR/RelativisticEulerAMR.cpp:1008) use `plain` (the
// Newtonian neighbours for every system), a threshold other than the tolerance, the coarse spacing
// as the divisor on a finer grid (`div`) and, for the intermediate pass, `need_on` (only cells
// whose own flag is on are tested).  dx places the cells (black-hole coordinates).
__global__ void amr_flags_kernel(ConsLoader L, double dx, Reach reach, int plain, int need_on, unsigned char* coarse,
                                 unsigned char* fine) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y;
    const Geom& G = L.G;
    if (j >= G.nx) return;
    if (need_on && !coarse[(size_t)i * G.nx + j]) return;
    double c[5], l[5], r[5], t[5], b[5];
    bool hit = false;
    if (G.dims == 1) {
        L.get(0, j - 1, Pt{(j - 1) * dx, 0.0, 0.0}, l);
        L.get(0, j, Pt{j * dx, 0.0, 0.0}, c);
        L.get(0, j + 1, Pt{(j + 1) * dx, 0.0, 0.0}, r);
#pragma unroll
        for (int k = 0; k < 5; k++)
            if (reach(c[k] - l[k]) || reach(r[k] - c[k])) hit = true;
    } else {
        L.get(i - 1, j, Pt{j * dx, (i - 1) * dx, 0.0}, t);
        L.get(i, j - 1, Pt{(j - 1) * dx, i * dx, 0.0}, l);
        L.get(i, j, Pt{j * dx, i * dx, 0.0}, c);
        L.get(i, j + 1, Pt{(j + 1) * dx, i * dx, 0.0}, r);
        if (L.system == 0 || plain) L.get(i + 1, j, Pt{j * dx, (i + 1) * dx, 0.0}, b);
        else if (i == G.ny - 1 && j == G.nx - 1) {
            const double dflt[5] = {1.0, 0.0, 0.0, 0.0, 1.0};
            if (L.precision == 1) {
                // FP32 grids hold conserved values; the default state in conserved form
                L.cons_of(dflt, Pt{(j + 1) * dx, (i + 1) * dx, 0.0}, b);
            } else {
                L.cons_of(dflt, Pt{(j + 1) * dx, (i + 1) * dx, 0.0}, b);
            }
        } else L.get(i + 1, j + 1, Pt{(j + 1) * dx, (i + 1) * dx, 0.0}, b);
#pragma unroll
        for (int k = 0; k < 5; k++)
            if (reach(c[k] - t[k]) || reach(b[k] - c[k]) || reach(c[k] - l[k]) ||
                reach(r[k] - c[k]))
                hit = true;
    }
    if (!hit) return;
    if (G.dims == 1) {
        coarse[j] = 0;
        fine[2 * j] = 1;
        fine[2 * j + 1] = 1;
    } else {
        coarse[(size_t)i * G.nx + j] = 0;
        const size_t fw = 2 * (size_t)G.nx;
        fine[(2 * i) * fw + 2 * j] = 1;
        fine[(2 * i) * fw + 2 * j + 1] = 1;
        fine[(2 * i + 1) * fw + 2 * j] = 1;
        fine[(2 * i + 1) * fw + 2 * j + 1] = 1;
    }
}

static ConsLoader make_loader(const SweepArgs& a, int precision, const void* state, const Geom& G) {
    ConsLoader L;
    L.system = a.system;
    L.precision = precision;
    L.G = G;
    L.state = state;
    L.nw = NewtonExact(a.gamma);
    L.sr = SRExact(a.gamma);
    L.gr = make_gr(a);
    return L;
}

cudaError_t launch_amr_flags(const SweepArgs& a, int precision, double tol, unsigned char* coarse, unsigned char* fine) {
    return launch_amr_flags_ex(a, precision, tol, a.dx, false, false, coarse, fine);
}
cudaError_t launch_amr_flags_ex(const SweepArgs& a, int precision, double thr, double div, bool plain, bool need_on,
                                unsigned char* coarse, unsigned char* fine) {
    dim3 grid((a.G.nx + 127) / 128, a.G.ny);
    amr_flags_kernel<<<grid, 128, 0, a.stream>>>(make_loader(a, precision, a.src, a.G), a.dx, Reach(div, thr),
                                                 plain ? 1 : 0, need_on ? 1 : 0, coarse, fine);
    count_launch();
    return cudaGetLastError();
}

// Derefinement pass, AMR/EulerAMR.cpp:310-345 (1D) and :538-586 (2D); GR coordinates
// AMR/BlackHoleEulerAMR.cpp:388-421 (1D fine cells read one fine cell to the left) and :632-686.
// Restriction writes the coarse state (FP64 storage only holds primitives, converted with the
// system's exact prim; FP32 storage receives the averaged conserved state).
// The Level-2 drivers' passes (AMR/EulerAMR.cpp:804-838 on the fine grid, :875-911 on the
// intermediate grid) take other thresholds and the coarse spacing as divisor (`div`), and are
// `strict`: they derefine only where every child is flagged (Level-1 tests the first child).
__global__ void amr_derefine_kernel(ConsLoader F, Geom CG, double dx, Reach reach, int strict,
                                    unsigned char* coarse, unsigned char* fine, void* coarse_state) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y;
    if (j >= CG.nx) return;
    const double fdx = dx * 0.5;
    bool marked = false;
    double c[5], l[5], r[5], t[5], b[5], avg[5];
    Pt qc;
    if (CG.dims == 1) {
        F.get(0, 2 * j, Pt{((j * 2) - 1) * fdx, 0.0, 0.0}, l);
        F.get(0, 2 * j + 1, Pt{(j * 2) * fdx, 0.0, 0.0}, c);
        F.get(0, 2 * j + 2, Pt{((j * 2) + 1) * fdx, 0.0, 0.0}, r);
#pragma unroll
        for (int k = 0; k < 5; k++)
            if (reach(c[k] - l[k]) || reach(r[k] - c[k])) marked = true;
        if (marked || !fine[2 * j] || (strict && !fine[2 * j + 1])) return;
        fine[2 * j] = 0;
        fine[2 * j + 1] = 0;
        coarse[j] = 1;
        double u0[5], u1[5];
        F.get(0, 2 * j, Pt{(j * 2) * fdx, 0.0, 0.0}, u0);
        F.get(0, 2 * j + 1, Pt{((j * 2) + 1) * fdx, 0.0, 0.0}, u1);
#pragma unroll
        for (int k = 0; k < 5; k++) avg[k] = 0.5 * (u0[k] + u1[k]);
        qc = Pt{j * dx, 0.0, 0.0};
    } else {
        F.get(2 * i, 2 * j + 1, Pt{((j * 2) + 1) * fdx, (i * 2) * fdx, 0.0}, t);
        F.get(2 * i + 1, 2 * j, Pt{(j * 2) * fdx, ((i * 2) + 1) * fdx, 0.0}, l);
        F.get(2 * i + 1, 2 * j + 1, Pt{((j * 2) + 1) * fdx, ((i * 2) + 1) * fdx, 0.0}, c);
        F.get(2 * i + 1, 2 * j + 2, Pt{((j * 2) + 2) * fdx, ((i * 2) + 1) * fdx, 0.0}, r);
        F.get(2 * i + 2, 2 * j + 1, Pt{((j * 2) + 1) * fdx, ((i * 2) + 2) * fdx, 0.0}, b);
#pragma unroll
        for (int k = 0; k < 5; k++)
            if (reach(c[k] - t[k]) || reach(b[k] - c[k]) || reach(c[k] - l[k]) ||
                reach(r[k] - c[k]))
                marked = true;
        const size_t fw = 2 * (size_t)CG.nx;
        if (marked || !fine[(2 * i) * fw + 2 * j]) return;
        if (strict && !(fine[(2 * i) * fw + 2 * j + 1] && fine[(2 * i + 1) * fw + 2 * j] &&
                        fine[(2 * i + 1) * fw + 2 * j + 1]))
            return;
        fine[(2 * i) * fw + 2 * j] = 0;
        fine[(2 * i) * fw + 2 * j + 1] = 0;
        fine[(2 * i + 1) * fw + 2 * j] = 0;
        fine[(2 * i + 1) * fw + 2 * j + 1] = 0;
        coarse[(size_t)i * CG.nx + j] = 1;
        double u0[5], u1[5], u2[5], u3[5];
        F.get(2 * i, 2 * j, Pt{(j * 2) * fdx, (i * 2) * fdx, 0.0}, u0);
        F.get(2 * i, 2 * j + 1, Pt{((j * 2) + 1) * fdx, (i * 2) * fdx, 0.0}, u1);
        F.get(2 * i + 1, 2 * j, Pt{(j * 2) * fdx, ((i * 2) + 1) * fdx, 0.0}, u2);
        F.get(2 * i + 1, 2 * j + 1, Pt{((j * 2) + 1) * fdx, ((i * 2) + 1) * fdx, 0.0}, u3);
#pragma unroll
        for (int k = 0; k < 5; k++) avg[k] = 0.25 * (((u0[k] + u1[k]) + u2[k]) + u3[k]);
        qc = Pt{j * dx, i * dx, 0.0};
    }
    if (!coarse_state) return;
    const size_t idx = (size_t)i * CG.pitch + j;
    if (F.precision == 1) {
        float* s = (float*)coarse_state;
#pragma unroll
        for (int k = 0; k < 5; k++) s[k * CG.fstride + idx] = (float)avg[k];
    } else {
        double p[5];
        F.prim_of(avg, qc, p);
        double* s = (double*)coarse_state;
#pragma unroll
        for (int k = 0; k < 5; k++) s[k * CG.fstride + idx] = p[k];
    }
}

cudaError_t launch_amr_derefine(const SweepArgs& a, int precision, const void* fine_state, const Geom& FG, double tol,
                                unsigned char* coarse, unsigned char* fine, void* coarse_state) {
    return launch_amr_derefine_ex(a, precision, fine_state, FG, tol * 0.5, a.dx, false, coarse, fine, coarse_state);
}
cudaError_t launch_amr_derefine_ex(const SweepArgs& a, int precision, const void* fine_state, const Geom& FG, double thr,
                                   double div, bool strict, unsigned char* coarse, unsigned char* fine,
                                   void* coarse_state) {
    dim3 grid((a.G.nx + 127) / 128, a.G.ny);
    amr_derefine_kernel<<<grid, 128, 0, a.stream>>>(make_loader(a, precision, fine_state, FG), a.G, a.dx, Reach(div, thr),
                                                    strict ? 1 : 0, coarse, fine, coarse_state);
    count_launch();
    return cudaGetLastError();
}

// End-of-step level exchange of the Level-1 drivers, AMR/EulerAMR.cpp:287-307 (1D) and :500-546
// (2D): a coarse cell whose flag is off takes the conserved average of its fine children
// (0.5 (a + b) in 1D, 0.25 (((a + b) + c) + d) in 2D, then the system's prim), and every fine
// child whose flag is off takes its parent's state.  One thread per coarse cell touches only
// that cell and its own children, in the reference's order (restriction, then injection).  The
// Level-2 drivers' exchange between the intermediate and fine levels (AMR/EulerAMR.cpp:780-801) is
// `strict`: restriction only where every child is flagged, injection only under a flagged parent.
// FP64 storage holds primitives; FP32 Newtonian/SR storage holds conserved values, which are
// averaged in FP64 and copied as stored.
__global__ void amr_sync_kernel(ConsLoader F, Geom CG, void* coarse_state, void* fine_state,
                                const unsigned char* coarse, const unsigned char* fine, int strict) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y;
    if (j >= CG.nx) return;
    const Geom& FG = F.G;
    const int nk = CG.dims == 1 ? 2 : 4;
    int ki[4], kj[4];
    for (int q = 0; q < nk; q++) {
        ki[q] = CG.dims == 1 ? 0 : 2 * i + (q >> 1);
        kj[q] = 2 * j + (q & 1);
    }
    const size_t cidx = (size_t)i * CG.pitch + j;
    const bool fp32 = F.precision == 1;
    const bool on = coarse[(size_t)i * CG.nx + j] != 0;
    bool all = true;
    for (int q = 0; q < nk; q++) all = all && fine[(size_t)ki[q] * FG.nx + kj[q]];
    if (!on && (!strict || all)) {
        double u[4][5], avg[5];
        for (int q = 0; q < nk; q++) F.get(ki[q], kj[q], Pt{0.0, 0.0, 0.0}, u[q]);
#pragma unroll
        for (int k = 0; k < 5; k++)
            avg[k] = nk == 2 ? 0.5 * (u[0][k] + u[1][k]) : 0.25 * (((u[0][k] + u[1][k]) + u[2][k]) + u[3][k]);
        if (fp32) {
#pragma unroll
            for (int k = 0; k < 5; k++) ((float*)coarse_state)[k * CG.fstride + cidx] = (float)avg[k];
        } else {
            double p[5];
            F.prim_of(avg, Pt{0.0, 0.0, 0.0}, p);
#pragma unroll
            for (int k = 0; k < 5; k++) ((double*)coarse_state)[k * CG.fstride + cidx] = p[k];
        }
    }
    for (int q = 0; q < nk; q++) {
        if (fine[(size_t)ki[q] * FG.nx + kj[q]] || (strict && !on)) continue;
        const size_t fidx = (size_t)ki[q] * FG.pitch + kj[q];
        if (fp32) {
#pragma unroll
            for (int k = 0; k < 5; k++)
                ((float*)fine_state)[k * FG.fstride + fidx] = ((const float*)coarse_state)[k * CG.fstride + cidx];
        } else {
#pragma unroll
            for (int k = 0; k < 5; k++)
                ((double*)fine_state)[k * FG.fstride + fidx] = ((const double*)coarse_state)[k * CG.fstride + cidx];
        }
    }
}

cudaError_t launch_amr_sync(const SweepArgs& a, int precision, void* coarse_state, void* fine_state, const Geom& FG,
                            const unsigned char* coarse, const unsigned char* fine, bool strict) {
    if (a.system == 2) return cudaErrorNotSupported;
    dim3 grid((a.G.nx + 127) / 128, a.G.ny);
    amr_sync_kernel<<<grid, 128, 0, a.stream>>>(make_loader(a, precision, fine_state, FG), a.G, coarse_state,
                                                fine_state, coarse, fine, strict ? 1 : 0);
    count_launch();
    return cudaGetLastError();
}

// Whether any of n flag bytes is set (the drivers' `refined` test, AMR/EulerAMR.cpp:241-249):
// ORs 1 into *out, which the caller zeroes first.
__global__ void amr_any_kernel(const unsigned char* __restrict__ f, size_t n, unsigned long long* out) {
    int hit = 0;
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x)
        hit |= f[k];
    if (__syncthreads_or(hit) && threadIdx.x == 0) atomicOr(out, 1ull);
}

cudaError_t launch_amr_any(const unsigned char* flags, size_t n, unsigned long long* out, cudaStream_t st) {
    size_t b = (n + 255) / 256;
    if (b > device_sm_count() * 4) b = device_sm_count() * 4;
    amr_any_kernel<<<(int)(b ? b : 1), 256, 0, st>>>(flags, n, out);
    count_launch();
    return cudaGetLastError();
}

// ------------------------------------------------------------------ state-level functions
// The reference's per-state functions (state vectors, equations of state, slope limiters, the
// black-hole eigenvalues) for n independent items, one thread per item, with the same arithmetic
// as the sweeps.  Item k reads in_stride doubles at in + k in_stride (and, for the black-hole
// system, its coordinates at xyz + 3k) and writes out_stride doubles at out + k out_stride.
template <class Sys>
CG_D void state_vector_op(const Sys& S, int op, const double* v, Pt q, double* o) {
    if (op == kStateCons) S.cons(v, q, o);
    else if (op == kStatePrim) S.prim(v, q, o);
    else S.flux(v, op == kStateFluxX ? 0 : 1, q, o);
}

// BlackHoleEuler/BlackHoleEulerEigenvalues.cpp:3-96: material, fast and slow acoustic eigenvalues
// along x, y, z (the terms whose largest value is GRExact::sound_speed).
CG_D void gr_eigenvalues(const GRExact& S, const double* p, Pt q, double* o) {
    double al, be[3];
    S.bh.lapse_shift(q.x, q.y, q.z, al, be);
    double gm[9], gs[9];
    S.bh.gamma(q.x, q.y, q.z, gm);
    inverse3(gm, gs);
    const double cs = sr_sound(p[0], p[4], S.k);
    const double v[3] = {p[1], p[2], p[3]};
    double v2 = 0.0;
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) v2 = v2 + ((gm[3 * i + j] * v[i]) * v[j]);
    for (int i = 0; i < 3; i++) {
        const double rt = sqrt((1.0 - v2) * ((gs[3 * i + i] * (1.0 - (v2 * (cs * cs)))) - ((v[i] * v[i]) * (1.0 - (cs * cs)))));
        const double pre = al / (1.0 - (v2 * (cs * cs)));
        o[i] = (al * v[i]) - be[i];
        o[3 + i] = (pre * ((v[i] * (1.0 - (cs * cs))) + (cs * rt))) - be[i];
        o[6 + i] = (pre * ((v[i] * (1.0 - (cs * cs))) - (cs * rt))) - be[i];
    }
}

__global__ void state_eval_kernel(StateEvalArgs a, NewtonExact nw, SRExact sr, const __grid_constant__ GRExact gr) {
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < a.n; k += (size_t)gridDim.x * blockDim.x) {
        const double* v = a.in + a.in_stride * k;
        double* o = a.out + a.out_stride * k;
        const Pt q = a.xyz ? Pt{a.xyz[3 * k], a.xyz[3 * k + 1], a.xyz[3 * k + 2]} : Pt{0.0, 0.0, 0.0};
        const double g = a.gamma;
        switch (a.op) {
            case kStateCons:
            case kStatePrim:
            case kStateFluxX:
            case kStateFluxY:
                if (a.system == 0) state_vector_op(nw, a.op, v, q, o);
                else if (a.system == 1) state_vector_op(sr, a.op, v, q, o);
                else state_vector_op(gr, a.op, v, q, o);
                break;
            case kStateSound:  // Euler/EulerEquationOfState.cpp:17-22; SR :10-18; black hole :519-549
                if (a.system == 0) o[0] = sqrt((g * v[4]) / v[0]);
                else if (a.system == 1) o[0] = sr_sound(v[0], v[4], sr.k);
                else o[0] = gr.sound_speed(v, q);
                break;
            case kStateInternalEnergy:  // Euler/EulerEquationOfState.cpp:3-8
                o[0] = v[4] / ((g - 1.0) * v[0]);
                break;
            case kStateTotalEnergy: {  // Euler/EulerStateVector.cpp:129-134 (the conserved energy)
                double u[5];
                nw.cons(v, q, u);
                o[0] = u[4];
                break;
            }
            case kStatePressure:  // Euler/EulerEquationOfState.cpp:10-15 from (rho, ., ., ., e)
                o[0] = (v[4] * (g - 1.0)) * v[0];
                break;
            case kStateEnthalpy:  // RelativisticEuler/RelativisticEulerEquationOfState.cpp:3-8
                o[0] = sr_enthalpy(v[0], v[4], sr.k);
                break;
            case kStateSource:  // BlackHoleEuler/BlackHoleEulerStateVector.cpp:359-510
                gr.source(v, q, o);
                break;
            case kStateEigenvalues:
                gr_eigenvalues(gr, v, q, o);
                break;
            case kStateGradientRatio:  // Solvers/SlopeLimiters.cpp:3-6
                o[0] = gradient_ratio(v[0], a.bias);
                break;
            case kStateLimiter:  // Solvers/SlopeLimiters.cpp:8-69
                o[0] = limiter_exact(v[0], a.bias, a.lim);
                break;
            case kStateSlope:  // Solvers/SlopeLimiters.cpp:71-101 on three conserved vectors
                slope_exact(v, v + 5, v + 10, make_bias(a.bias), a.lim, o);
                break;
            default:
                break;
        }
    }
}

cudaError_t launch_state_eval(const SweepArgs& s, const StateEvalArgs& a) {
    size_t b = (a.n + 127) / 128;
    if (b > device_sm_count() * 8) b = device_sm_count() * 8;
    state_eval_kernel<<<(int)(b ? b : 1), 128, 0, s.stream>>>(a, NewtonExact(s.gamma),
                                                                SRExact(s.gamma), make_gr(s));
    count_launch();
    return cudaGetLastError();
}

// ------------------------------------------------------------------ per-interface functions
// The reference's static building blocks, one item per thread, in the reference's operation order
// (this unit is compiled without FMA contraction):
//   0 computeLaxFriedrichsFlux, 1 computeRichtmyerFlux (the intermediate state), 2 computeFORCEFlux,
//   3 computeFORCEUpdate (Solvers/EulerFirstOrderSolver.cpp:3-24, :96-101), 4 computeFractional-
//   EvolutionVector, 5 computeEvolutionVector (Solvers/EulerSolvers.cpp:163-172);
//   6..11 computeX/Y{LaxFriedrichs,Richtmyer,FORCE}Flux of primitive states
//   (Solvers/EulerFirstOrderSolver.cpp:26-94 and the SR and black-hole twins; black hole: states
//   at x -/+ dx/2, the intermediate state's flux at x);
//   12/13 computeX/YSLICFlux (Solvers/EulerSecondOrderSolver.cpp:3-25; black hole
//   Solvers/BlackHoleEulerSecondOrderSolver.cpp:3-39: evolutions at x -/+ dx/2);
//   14/15 evolveStateByHalfX/YTimeStep of states, 16/17 evolveStateByHalfTimeStep of vectors
//   (Solvers/EulerSolvers.cpp:174-223; black hole Solvers/BlackHoleEulerSolvers.cpp:234-307);
//   black hole only: 18/19 evolveStateByFractionalX/YTimeStep, 20 evolveStateByFractionalTimeStep
//   (Solvers/BlackHoleEulerSolvers.cpp:159-232), 21/22 the forcing solver's
//   evolveConservedVariableVector / ...2D (Solvers/BlackHoleEulerForcingSolver.cpp:3-185).
template <class Sys>
CG_D void iface_item(const Sys& S, bool gr, const IfaceArgs& A, const double* a, Pt q, double* o) {
    const double* b = a + 5;
    const double* c = a + 10;
    const double* d = a + 15;
    const int op = A.op;
    const int axis = (op & 1) ? 1 : 0;
    const double dx = A.dx, dt = A.dt;
    const StepRatio sr = make_ratio(dt, dx);
    const Bias w = make_bias(A.bias);
    switch (op) {
        case 0: { const double r = dx / dt; for (int k = 0; k < 5; k++) o[k] = 0.5 * ((c[k] + d[k]) + (r * (a[k] - b[k]))); break; }
        case 1: { const double r = dt / dx; for (int k = 0; k < 5; k++) o[k] = 0.5 * ((a[k] + b[k]) + (r * (c[k] - d[k]))); break; }
        case 2: for (int k = 0; k < 5; k++) o[k] = 0.5 * (a[k] + b[k]); break;
        case 3: { const double r = dt / dx; for (int k = 0; k < 5; k++) o[k] = a[k] + (r * (b[k] - c[k])); break; }
        case 4: case 5: {
            const double r = (op == 4 ? A.frac : 0.5) * (dt / dx);
            for (int k = 0; k < 5; k++) o[k] = r * (a[k] - b[k]);
            break;
        }
        case 6: case 7: case 8: case 9: {
            double uL[5], uR[5], fL[5], fR[5];
            const Pt pl = shift_pt(q, axis, -(dx * 0.5)), pr = shift_pt(q, axis, dx * 0.5);
            S.cons(a, pl, uL);
            S.cons(b, pr, uR);
            S.flux(uL, axis, pl, fL);
            S.flux(uR, axis, pr, fR);
            if (op <= 7) {
                const double r = dx / dt;
                for (int k = 0; k < 5; k++) o[k] = 0.5 * ((fL[k] + fR[k]) + (r * (uL[k] - uR[k])));
                break;
            }
            const double r = dt / dx;
            double us[5];
            for (int k = 0; k < 5; k++) us[k] = 0.5 * ((uL[k] + uR[k]) + (r * (fL[k] - fR[k])));
            S.flux(us, axis, q, o);
            break;
        }
        case 10: case 11: force_exact(S, a, b, q, axis, dx, sr, o); break;
        case 12: case 13: {
            double eR[5], eL[5];
            evolve_half_exact(S, a, b, c, shift_pt(q, axis, -(dx * 0.5)), axis, dx, sr, w, A.lim, (double*)nullptr, eR);
            evolve_half_exact(S, b, c, d, shift_pt(q, axis, dx * 0.5), axis, dx, sr, w, A.lim, eL, (double*)nullptr);
            force_exact(S, eR, eL, q, axis, dx, sr, o);
            break;
        }
        case 14: case 15:
            evolve_half_exact(S, a, b, c, q, axis, dx, sr, w, A.lim, A.side == 0 ? o : nullptr,
                              A.side == 0 ? nullptr : o);
            break;
        case 16: case 17: {
            double u[5];
            const double* x = A.side == 0 ? a : b;
            for (int k = 0; k < 5; k++) u[k] = x[k] + c[k];
            S.prim(u, gr ? shift_pt(q, axis, A.side == 0 ? -(dx * 0.5) : dx * 0.5) : q, o);
            break;
        }
        default: break;
    }
}

__global__ void iface_kernel(IfaceArgs A, NewtonExact nw, SRExact sr, const __grid_constant__ GRExact gr) {
    const int w = A.width;
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < A.n; k += (size_t)gridDim.x * blockDim.x) {
        const double* a = A.in + (size_t)w * k;
        double* o = A.out + 5 * k;
        const Pt q = A.xyz ? Pt{A.xyz[3 * k], A.xyz[3 * k + 1], A.xyz[3 * k + 2]} : Pt{0.0, 0.0, 0.0};
        if (A.system == 0) iface_item(nw, false, A, a, q, o);
        else if (A.system == 1) iface_item(sr, false, A, a, q, o);
        else if (A.op <= 17) iface_item(gr, true, A, a, q, o);
        else if (A.op <= 19) evolve_fraction_exact(gr, A.frac, a, a + 5, a + 10, q, A.op - 18, A.dx, make_ratio(A.dt, A.dx), make_bias(A.bias), A.lim, o);
        else if (A.op == 20) {
            double u[5];
            for (int f = 0; f < 5; f++) u[f] = a[f] + a[5 + f];
            gr.prim(u, q, o);
        } else {  // 21: left, middle, right; 22: left, middle, right, top, bottom
            const int dims = A.op - 20;
            V5<double> u[5];
            Metric<double> g;
            for (int f = 0; f < 5; f++) {
                u[0].v[f] = a[f];
                u[4].v[f] = a[5 + f];
                u[1].v[f] = a[10 + f];
                u[2].v[f] = dims == 2 ? a[15 + f] : 0.0;
                u[3].v[f] = dims == 2 ? a[20 + f] : 0.0;
            }
            give(rk_cell_exact(OneThread{}, &gr, dims, u, q, A.dx, A.dt, make_ratio(A.dt, A.dx), make_bias(A.bias), A.lim, &g), o);
        }
    }
}

cudaError_t launch_interface_eval(const SweepArgs& s, const IfaceArgs& a) {
    size_t b = (a.n + 127) / 128;
    if (b > (size_t)device_sm_count() * 8) b = (size_t)device_sm_count() * 8;
    SweepArgs g = s;
    g.dx = a.dx;  // the black-hole metric derivatives take the cell spacing (the reference's h)
    iface_kernel<<<(int)(b ? b : 1), 128, 0, s.stream>>>(a, NewtonExact(s.gamma), SRExact(s.gamma),
                                                         make_gr(g));
    count_launch();
    return cudaGetLastError();
}

// ------------------------------------------------------------------ spacetime record
// Every public quantity of the reference's BlackHoleSpacetime (BlackHoleEuler/BlackHoleSpacetime.cpp:
// 54-386) at one point, metric derivatives by the reference's centred differences with spacing
// S.h, in the layout of the public COSMOS_ST_* offsets.
__global__ void spacetime_kernel(const __grid_constant__ GRExact S, size_t n, const double* __restrict__ xyz, double* __restrict__ out) {
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
        const Pt q{xyz[3 * k], xyz[3 * k + 1], xyz[3 * k + 2]};
        double* o = out + (size_t)kSpacetimeWidth * k;
        const BHExact& b = S.bh;
        o[0] = b.H<double>(q.x, q.y, q.z);                            // computeKerrSchildScalar
        b.l(q.x, q.y, q.z, o + 1);                            // computeKerrSchildVector
        b.L4(q.x, q.y, q.z, o + 4);                           // computeKerrSchildSpacetimeVector
        const double h = S.h, hs = 0.5 * h;
        for (int d = 0; d < 3; d++) {                         // the scalar and vector derivatives
            const Pt p1 = S.off(q, d, hs), p0 = S.off(q, d, -hs);
            double h1, h0, a1[3], a0[3];
            b.Hl(p1.x, p1.y, p1.z, h1, a1);
            b.Hl(p0.x, p0.y, p0.z, h0, a0);
            o[8 + d] = (h1 - h0) / h;
            for (int c = 0; c < 3; c++) o[11 + 3 * d + c] = (1.0 / h) * (a1[c] - a0[c]);
        }
        double m[9], g4m[16];
        b.gamma(q.x, q.y, q.z, m);
        b.g4(q.x, q.y, q.z, g4m);
        for (int i = 0; i < 9; i++) o[20 + i] = m[i];
        for (int i = 0; i < 16; i++) o[29 + i] = g4m[i];
        inverse3(m, o + 45);
        inverse4(g4m, o + 54);
        o[70] = det3(m);
        o[71] = det4(g4m);
        double al, gi[16];
        b.lapse_shift(q.x, q.y, q.z, al, o + 100);
        o[99] = al;
        // lapse, shift and spatial-metric derivatives and K_ij as the source term takes them
        S.source_metric(q, al, gi, o + 103, o + 106, o + 72, o + 115);
        o[124] = b.excised(q.x, q.y, q.z) ? 1.0 : 0.0;
    }
}

cudaError_t launch_spacetime_eval(const SweepArgs& s, size_t n, const double* xyz, double* out) {
    size_t blocks = (n + 127) / 128;
    if (blocks > (size_t)device_sm_count() * 8) blocks = (size_t)device_sm_count() * 8;
    spacetime_kernel<<<(int)(blocks ? blocks : 1), 128, 0, s.stream>>>(make_gr(s), n, xyz, out);
    count_launch();
    return cudaGetLastError();
}

// ------------------------------------------------------------------ conservation sums
// Sum of each stored field over the grid with Kahan-Babuska (Neumaier) compensation per thread,
// then compensated double atomics are avoided: per-block partials go to a small buffer summed by
// the last block in a fixed order, so the result is deterministic.
__global__ void field_sums_kernel(const void* __restrict__ state, Geom G, int precision, double* partial,
                                  unsigned int* counter, double* out5) {
    double s[5] = {0, 0, 0, 0, 0}, comp[5] = {0, 0, 0, 0, 0};
    const size_t n = (size_t)G.nx * G.ny;
    for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) {
        const size_t i = c / G.nx, j = c % G.nx, k = i * G.pitch + j;
#pragma unroll
        for (int f = 0; f < 5; f++) {
            const double v = precision == 1 ? (double)((const float*)state)[f * G.fstride + k]
                                            : ((const double*)state)[f * G.fstride + k];
            const double t = s[f] + v;
            comp[f] += (fabs(s[f]) >= fabs(v)) ? ((s[f] - t) + v) : ((v - t) + s[f]);
            s[f] = t;
        }
    }
    __shared__ double red[5][256];
#pragma unroll
    for (int f = 0; f < 5; f++) red[f][threadIdx.x] = s[f] + comp[f];
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int f = 0; f < 5; f++) {
            double a = 0.0, ca = 0.0;
            for (int q = 0; q < blockDim.x; q++) {
                const double v = red[f][q], t = a + v;
                ca += (fabs(a) >= fabs(v)) ? ((a - t) + v) : ((v - t) + a);
                a = t;
            }
            partial[blockIdx.x * 5 + f] = a + ca;
        }
        __threadfence();
        const unsigned int done = atomicAdd(counter, 1u);
        if (done == gridDim.x - 1) {
            __threadfence();
            for (int f = 0; f < 5; f++) {
                double a = 0.0, ca = 0.0;
                for (unsigned q = 0; q < gridDim.x; q++) {
                    const double v = ((volatile double*)partial)[q * 5 + f], t = a + v;
                    ca += (fabs(a) >= fabs(v)) ? ((a - t) + v) : ((v - t) + a);
                    a = t;
                }
                out5[f] = a + ca;
            }
            *counter = 0;
        }
    }
}

cudaError_t launch_field_sums(const void* soa, const Geom& G, int precision, double* out5, cudaStream_t st) {
    // scratch: 152*4 blocks * 5 partials + a counter, carved from out5's companion buffer
    constexpr int kBlocks = 152 * 4;
    double* partial = out5 + 8;
    unsigned int* counter = (unsigned int*)(out5 + 8 + kBlocks * 5);
    field_sums_kernel<<<kBlocks, 256, 0, st>>>(soa, G, precision, partial, counter, out5);
    count_launch();
    return cudaGetLastError();
}

}  // namespace cg
