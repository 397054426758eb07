// One whole FP32 Newtonian SLIC step, X(dt/2) Y(dt) X(dt/2) with its time step and CFL reduction, in one launch
// (small 2D grids).
//
// What bounds a step there is not its work but four launches in a row, each a few microseconds of start, one
// dependent pass and a drain: 193 x 257 took 18.6 us per step (dt kernel 3.7, X 5.6, Y 9.3, X 6.7 under the
// profiler) where its memory traffic is under one.  Here a block of 16 warps takes a tile of 56 x 12 cells with
// its halo (4 columns and 2 rows on each side) through the three sweeps in shared memory: warp w sweeps row
// w - 2 in X, owns row w - 1 in Y (its evolution, and the flux above it) and sweeps row w in X again.  The
// arithmetic is the single sweeps' (x_pair_compute, nf_recon, nf_force4, nf_update on the same pairs), so the
// results are theirs bit for bit; the price is the halo's repeated work, 1.33 x in the rows, which is why large
// grids keep the three sweeps.
//
// The times of both forms stand at kFusedStepCells (kernels_fast.cu): 193 x 257 18.6 -> 9.7 us per step.
// (Programmatic dependent launch of the next step's blocks measured no faster.)
//
// The time step: every block forms it itself (one thread, while the others load the tile) from the controller,
// which nobody writes meanwhile; the last block to finish enters it there.
#pragma once
#include "sweep_pairs.cuh"

namespace cg {

constexpr int kTileCols = 56, kTileRows = 12, kTileWarps = kTileRows + 4;
constexpr int kTileW = 68;  // floats per row in shared memory: columns x0 - 4 .. x0 + 59 and 4 more

struct StepTileSmem {
    float u[5][kTileRows + 4][kTileW];  // rows y0 - 2 .. y0 + 13
    float l[5][kTileRows + 2][64];      // lower-face states of rows y0 - 1 .. y0 + 12
    float f[5][kTileRows + 2][64];      // flux above rows y0 - 1 .. y0 + 11
    float red[kTileWarps];
    StepNow now;
    FastCoef full, halved;
    int it;
};

// Cell index of position k of a line of n >= 8 cells, k at most four outside: wrapped, or mirrored (positions
// more than two outside only feed values nobody reads).
CG_D int tile_index(int k, int n, int bc) {
    if (bc == 1) return k < 0 ? k + n : (k >= n ? (k - n < n ? k - n : n - 1) : k);
    return ghost_index(min(max(k, -2), n + 1), n, bc);
}

template <int LIM>
__global__ void __launch_bounds__(kTileWarps * 32, 2) step_tile_kernel(NewtonFastParams P, Geom G,
                                                                       const float* __restrict__ src,
                                                                       float* __restrict__ dst, StepCtl* ctl) {
    extern __shared__ __align__(16) unsigned char step_smem[];
    StepTileSmem& S = *reinterpret_cast<StepTileSmem*>(step_smem);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int x0 = blockIdx.x * kTileCols, y0 = blockIdx.y * kTileRows;
    // ---- the tile: warp w loads row y0 - 2 + w
    {
        const int row = tile_index(min(y0 - 2 + w, G.ny + 1), G.ny, G.bc);
        const float* s = src + (size_t)row * G.pitch;
        const int c = x0 - 4 + 2 * lane;
        const bool in = c >= 0 && c + 1 < G.nx;
        const int qa = tile_index(c, G.nx, G.bc), qb = tile_index(c + 1, G.nx, G.bc);
#pragma unroll
        for (int f = 0; f < 5; f++) {
            const float* p = s + f * G.fstride;
            const float2 v = in ? *reinterpret_cast<const float2*>(p + c) : make_float2(p[qa], p[qb]);
            *reinterpret_cast<float2*>(&S.u[f][w][2 * lane]) = v;
        }
    }
    if (threadIdx.x == 0) {
        S.now = step_now(ctl);
        S.it = ctl->it;
        S.full = S.now.full();
        S.halved = S.now.halved();
    }
    __syncthreads();
    const bool active = S.now.active;
    float ws = 0.0f;
    auto pair_at = [&](const float* row, Cell2& c) {
#pragma unroll
        for (int f = 0; f < 5; f++) c.v[f].v = *reinterpret_cast<const float2*>(row + f * ((kTileRows + 4) * kTileW));
    };
    if (active) {
        const FastCoef ch = S.halved;
        {  // ---- X(dt/2) of rows y0 - 2 .. y0 + 13: columns x0 - 2 .. x0 + 57, in place (the warp's own row)
            Cell2 m, nc;
            pair_at(&S.u[0][w][2 * lane], m);
            x_pair_compute<LIM>(P, m, ch, nc);
            __syncwarp();
            if (lane >= 1 && lane <= 30)
#pragma unroll
                for (int f = 0; f < 5; f++) *reinterpret_cast<float2*>(&S.u[f][w][2 * lane]) = nc.v[f].v;
            __syncwarp();
            // transmissive ghosts are mirrored again: a swept ghost is not the mirror of the swept cell
            if (G.bc != 1 && lane < 5) {
                float* r = S.u[lane][w];
                if (x0 == 0) {
                    r[3] = r[4];
                    r[2] = r[5];
                }
                const int e = G.nx - x0 + 4;  // the row's end in the tile
                if (e <= 61) {
                    r[e] = r[e - 1];
                    r[e + 1] = r[e - 2];
                }
            }
        }
        __syncthreads();
        // ---- Y(dt): warp w owns row y0 - 1 + w
        Cell2 m;
        f2 R[5], Fr[5];
        const FastCoef cf = S.full;
        const Force4Coef c4 = force4_coef(cf);
        if (w < kTileRows + 2) {
            Cell2 a, b;
            f2 L[5];
            pair_at(&S.u[0][w][2 * lane], a);
            pair_at(&S.u[0][w + 1][2 * lane], m);
            pair_at(&S.u[0][w + 2][2 * lane], b);
            nf_recon<1, LIM>(P, a.v, m.v, b.v, cf.half_dtdx, L, R);
#pragma unroll
            for (int f = 0; f < 5; f++) *reinterpret_cast<float2*>(&S.l[f][w][2 * lane]) = L[f].v;
        }
        __syncthreads();
        if (w < kTileRows + 1) {
            f2 Ln[5];
#pragma unroll
            for (int f = 0; f < 5; f++) Ln[f].v = *reinterpret_cast<const float2*>(&S.l[f][w + 1][2 * lane]);
            nf_force4<1>(P, R, Ln, c4.dtdx, c4.dxdt, Fr);
#pragma unroll
            for (int f = 0; f < 5; f++) *reinterpret_cast<float2*>(&S.f[f][w][2 * lane]) = Fr[f].v;
        }
        __syncthreads();
        if (w >= 1 && w <= kTileRows) {
            f2 Fl[5];
            Cell2 nc;
#pragma unroll
            for (int f = 0; f < 5; f++) Fl[f].v = *reinterpret_cast<const float2*>(&S.f[f][w - 1][2 * lane]);
            nf_update(c4.q_dtdx, m.v, Fl, Fr, nc.v);
#pragma unroll
            for (int f = 0; f < 5; f++) *reinterpret_cast<float2*>(&S.u[f][w + 1][2 * lane]) = nc.v[f].v;
        }
        __syncthreads();
        // ---- X(dt/2) of row y0 + w: columns x0 .. x0 + 55 are stored
        const int row = y0 + w;
        if (w < kTileRows && row < G.ny) {
            Cell2 c, nc;
            pair_at(&S.u[0][w + 2][2 + 2 * min(lane, 30)], c);
            x_pair_compute<LIM>(P, c, ch, nc);
            const int j = x0 - 2 + 2 * lane;
            if (lane >= 1 && lane <= kTileCols / 2 && j < G.nx) {
                const bool two = j + 1 < G.nx;
                float* d = dst + (size_t)row * G.pitch + j;
#pragma unroll
                for (int f = 0; f < 5; f++) {
                    if (two) *reinterpret_cast<float2*>(d + f * G.fstride) = nc.v[f].v;
                    else d[f * G.fstride] = nc.v[f].v.x;
                }
                const f2 s = nf_wavespeed(P, nc.v, 2);
                ws = fmaxf(ws, two ? fmaxf(s.v.x, s.v.y) : s.v.x);  // fmaxf drops a NaN
            }
        }
    } else if (w < kTileRows && y0 + w < G.ny) {  // the run has ended: keep the ping-pong buffers consistent
        const int j = x0 + 2 * lane;
        float* d = dst + (size_t)(y0 + w) * G.pitch + j;
        if (lane < kTileCols / 2 && j < G.nx)
#pragma unroll
            for (int f = 0; f < 5; f++) {
                d[f * G.fstride] = S.u[f][w + 2][4 + 2 * lane];
                if (j + 1 < G.nx) d[f * G.fstride + 1] = S.u[f][w + 2][5 + 2 * lane];
            }
    }
    ws = warp_max(ws);
    if (lane == 0) S.red[w] = ws;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < kTileWarps; k++) ws = fmaxf(ws, S.red[k]);
        // few blocks: the maximum goes out without a look at the slot first
        if (active && ws > 0.0f) atomicMax(&ctl->smax[(S.it + 1) & 1], (unsigned long long)__double_as_longlong((double)ws));
        __threadfence();
        if (atomicAdd(&ctl->done, 1u) == gridDim.x * gridDim.y - 1) {
            // every block has read the controller and reduced into the other slot: enter the step, empty the
            // slot it was taken from
            __threadfence();
            ctl->done = 0;
            step_enter(ctl, S.now, S.it & 1);
        }
    }
}

}  // namespace cg
