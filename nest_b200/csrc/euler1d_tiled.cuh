// Tiled multi-CTA 1D stage kernels, templated on the arithmetic type:
// instantiated for double in euler1d.cu (-fmad=false, nest's operation order,
// bit for bit with the OpenMP path) and for float in euler1d_f32.cu (the FP32
// form, fast reciprocal / square root).  Time, dt and the wave-speed maximum
// stay FP64 in both.
//
// One CTA of T1 + 32 threads owns T1 cells: primitives of its cells and a 2-cell
// halo into shared memory, one HLLE per face, the update with the ghost
// copies it feeds; stage 2 fuses the Heun average and the block's max
// |u|+c (one atomic per block).  dt is derived on the device from that
// maximum by the next stage 1, so a step is two launches and no host
// synchronisation.  k1d_step runs a whole step in one launch (out of place), a
// warp per 24 or 56 cells with nothing in shared memory.
#pragma once

#include "euler1d_arith.cuh"
#include "kernels.h"

namespace nestb {
namespace {

// cells per tile: 224 puts at most 448 cells on an SM at 65536 cells (293
// tiles over 148 SMs; 256 gave 512 on most SMs): FP64 step 8.76 -> 8.46 us
constexpr int T1 = 224;
// threads per block: at least one per extended cell (T1 + 4), so that no
// phase loops twice, in whole warps (the stage-2 reduction shuffles over
// full warps)
constexpr int NT1 = T1 + 32;

// Writes the ghost copies that the value of interior cell c (0-based) feeds.
template <typename T>
__device__ __forceinline__ void push_ghosts_1d(T* U, int nt, int k, int c, int n, int h, int bc, T v) {
    if (bc == BC_PERIODIC) {
        if (c < h) U[k * nt + h + n + c] = v;
        if (c >= n - h) U[k * nt + (c - (n - h))] = v;
    } else {
        if (c == 0) for (int g = 0; g < h; ++g) U[k * nt + g] = v;
        if (c == n - 1) for (int g = 0; g < h; ++g) U[k * nt + h + n + g] = v;
    }
}

// LIM (both kernels): the slope limiter fixed at compile time (LIM_MINMOD,
// nest's default) or -1 to read it from the loop parameters.
template <typename T, int STAGE, int LIM>
__global__ void __launch_bounds__(NT1)
k1d_stage(const T* __restrict__ Uin, const T* Un, T* Uout,
          int n, int h, double dx, double gamma_d, int bc, LoopParams lp, StepCtrl* ctrl, int p) {
    __shared__ T W[3][T1 + 4];
    __shared__ T F[3][T1 + 1];
    __shared__ double red[33];
    pdl_wait();
    pdl_trigger();
    int nt = n + 2 * h;
    const Gas<T> gas(gamma_d);
    double dt;
    if (STAGE == 1) {
        bool done = step_is_done(ctrl, p, lp);
        double ms = speed_1d(ctrl, p);
        double pd = done ? -1.0 : prescribed_dt(ctrl, p, lp);
        if (pd > 0.0) dt = pd;
        else {
            dt = lp.cfl * dx / ms;
            if (lp.t_final > 0.0) dt = smin(dt, lp.t_final - ctrl->time[p]);
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) publish_step_1d(ctrl, p, lp, done, dt, false);
        if (done) return;
    } else {
        if (!ctrl->active[p]) return;
        dt = ctrl->dt[p];
    }
    const T dtdx = (T)(dt / dx);
    int c0 = blockIdx.x * T1;  // first interior cell of the tile
    // primitives of extended cells c0-2 .. c0+T1+1 (clamped at the array end)
    for (int t = threadIdx.x; t < T1 + 4; t += NT1) {
        int e = min(h + c0 - 2 + t, nt - 1);
        T rho = Uin[e], mom = Uin[nt + e], erg = Uin[2 * nt + e];
        const Cell1<T> w = cell1d<false>(gas, rho, mom, erg);
        W[0][t] = rho;
        W[1][t] = w.u;
        W[2][t] = w.p;
    }
    __syncthreads();
    int nf = min(T1, n - c0) + 1;  // faces of this tile
    for (int f = threadIdx.x; f < nf; f += NT1) {
        const F3<T> q = plm_flux(gas, LIM >= 0 ? LIM : lp.lim, [&](int k, int t) { return W[k][t]; }, f, f + 1, f + 2, f + 3);
        F[0][f] = q.a; F[1][f] = q.b; F[2][f] = q.c;
    }
    __syncthreads();
    int c = c0 + threadIdx.x;
    double ms = 0.0;
    if (threadIdx.x < T1 && c < n) {
        int e = h + c;
        T v[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            T s = Uin[k * nt + e] - dtdx * (F[k][threadIdx.x + 1] - F[k][threadIdx.x]);
            v[k] = (STAGE == 1) ? s : T(0.5) * (Un[k * nt + e] + s);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            Uout[k * nt + e] = v[k];
            push_ghosts_1d(Uout, nt, k, c, n, h, bc, v[k]);
        }
        if (STAGE == 2) {
            const Cell1<T> w = cell1d<true>(gas, v[0], v[1], v[2]);
            ms = (double)(fabs(w.u) + w.cs);
            if (!(v[0] > T(0)) || !(w.p > T(0)))
                flag_cell(ctrl, ctrl->step[p] + 1, (double)v[0], (double)w.p, c, 0, errw_slot(p ^ 1));
        }
    }
    if (STAGE == 2) {
        ms = warp_max(ms);
        int w = threadIdx.x >> 5, l = threadIdx.x & 31;
        if (l == 0) red[w] = ms;
        __syncthreads();
        if (w == 0) {
            double x = (l < (NT1 + 31) / 32) ? red[l] : 0.0;
            x = warp_max(x);
            if (l == 0) {
                if (!(x == x) || x > 1.79e308) atomicOr(&ctrl->err, ERRW_NONFINITE | errw_slot(p ^ 1));
                atomic_max_speed(&ctrl->maxs[p ^ 1][0], x);
            }
        }
    }
}

// Interior cell whose value cell c holds (any c, ghost cells and beyond
// included): nest's periodic copy, or the zero-gradient copy of the nearest
// end cell.
__device__ __forceinline__ int source_cell_1d(int c, int n, int bc) {
    if (bc == BC_PERIODIC) {
        c %= n;
        return c < 0 ? c + n : c;
    }
    return min(max(c, 0), n - 1);
}

constexpr int STEP_WARPS = 4;  // warps per CTA of k1d_step
// output cells of a warp with CPL cells per lane: all but four at each end
__host__ __device__ constexpr int step_cells(int cpl) { return 32 * cpl - 8; }

// v[i] = u[i] - dtdx (right flux - left flux) of the lane's cells.
template <typename T, int CPL>
__device__ __forceinline__ void warp_update(const T (&u)[CPL][3], const F3<T> (&f)[CPL], T dtdx, T (&v)[CPL][3]) {
    const F3<T> l = { __shfl_up_sync(0xffffffffu, f[CPL - 1].a, 1), __shfl_up_sync(0xffffffffu, f[CPL - 1].b, 1),
                      __shfl_up_sync(0xffffffffu, f[CPL - 1].c, 1) };
#pragma unroll
    for (int i = 0; i < CPL; ++i) {
        const F3<T> q = i > 0 ? f[i > 0 ? i - 1 : 0] : l;
        v[i][0] = u[i][0] - dtdx * (f[i].a - q.a);
        v[i][1] = u[i][1] - dtdx * (f[i].b - q.b);
        v[i][2] = u[i][2] - dtdx * (f[i].c - q.c);
    }
}

// One whole RK2 (Heun) step in one launch, out of place (Un -> Unext; the
// caller alternates two buffers).  A warp owns 24 cells (56 with two per lane)
// and works alone: lane k holds cells c0 - 4 + CPL k .. (their U^n, primitives, U1
// and its primitives in registers), faces and neighbours' slopes come by
// shuffles.  The four cells at each end are the halo of the two stages,
// recomputed by the neighbouring warps instead of being exchanged.  Every value
// is computed by the same expression, on the same operands, as in the two stage
// kernels (and nest's loop): U1 of a ghost cell is U1 of the cell it copies, which
// the periodic wrap of the primitives gives directly and the zero-gradient case
// takes from that cell's lane.  The block's maximum goes to the next step's slot
// in one fire-and-forget atomic (publish_step_1d clears the words).  U1out
// (optional) receives U1 of the step with its ghosts.  A finished step (time,
// step count or error) copies Un to Unext so that the state ends in the buffer
// the caller expects.
// Bound: one chain of two stages and the launch.  us per step (FP64 5003 / 65536 /
// 200003 cells, FP32 50021): 4.2 / 5.2 / 10.3, 3.0, against 6.0 / 7.3 / 14.3, 5.5 with
// 224-cell CTAs that staged each phase through shared memory and moved the
// maximum with a counter of finished blocks.
template <typename T, int LIM, int CPL>
__global__ void __launch_bounds__(32 * STEP_WARPS)
k1d_step(const T* __restrict__ Un, T* __restrict__ Unext, T* __restrict__ U1out, int n, int h, double dx,
         double gamma_d, int bc, LoopParams lp, StepCtrl* ctrl, int p) {
    constexpr int CELLS = step_cells(CPL);
    __shared__ double red[STEP_WARPS];
    const Gas<T> gas(gamma_d);
    const int nt = n + 2 * h;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c0 = (blockIdx.x * STEP_WARPS + warp) * CELLS, c = c0 - 4 + CPL * lane;
    const int lim = LIM >= 0 ? LIM : lp.lim;
    const double rdx = lp.cfl * dx;
    auto own = [&](int i) {
        const int x = CPL * lane + i;
        return x >= 4 && x < 4 + CELLS && c + i < n;
    };
    auto store = [&](T* U, const T (&v)[3], int ci) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            U[k * nt + h + ci] = v[k];
            push_ghosts_1d(U, nt, k, ci, n, h, bc, v[k]);
        }
    };
    T u[CPL][3], v[CPL][3], w[CPL][3];
    int e[CPL];
#pragma unroll
    for (int i = 0; i < CPL; ++i) e[i] = h + source_cell_1d(c + i, n, bc);
    pdl_wait();
    pdl_trigger();
#pragma unroll
    for (int i = 0; i < CPL; ++i)
#pragma unroll
        for (int k = 0; k < 3; ++k) u[i][k] = Un[k * nt + e[i]];
    if (step_is_done(ctrl, p, lp, true)) {
        if (blockIdx.x == 0 && threadIdx.x == 0) publish_step_1d(ctrl, p, lp, true, 0.0, true);
        for (int i = 0; i < CPL; ++i)
            if (own(i)) store(Unext, u[i], c + i);
        return;
    }
    auto prims = [&](const T (&a)[CPL][3]) {
#pragma unroll
        for (int i = 0; i < CPL; ++i) {
            const Cell1<T> q = cell1d<false>(gas, a[i][0], a[i][1], a[i][2]);
            w[i][0] = a[i][0]; w[i][1] = q.u; w[i][2] = q.p;
        }
    };
    F3<T> f[CPL];
    prims(u);
    warp_flux(gas, lim, w, f);  // needs no dt
    const int sel = ctrl->sel[p];
    double dt;
    {
        const double pd = prescribed_dt(ctrl, p, lp);
        if (pd > 0.0) {
            dt = pd;
        } else {
            dt = div_rn(rdx, bits_speed(ctrl->maxs[p][sel & 1]));
            if (lp.t_final > 0.0) dt = smin(dt, lp.t_final - ctrl->time[p]);
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) publish_step_1d(ctrl, p, lp, false, dt, true);
    const T dtdx = (T)div_rn(dt, dx);

    warp_update(u, f, dtdx, v);
    if (bc != BC_PERIODIC && (c0 < 4 || c0 + CELLS + 4 > n)) {
        // zero-gradient ghosts: U1 of the end cell they copy, held by a lane of this
        // warp whenever the warp reaches past the domain
        T r[CPL][3];
#pragma unroll
        for (int i = 0; i < CPL; ++i) {
            const int x = (min(max(c + i, 0), n - 1) - (c0 - 4)) & (32 * CPL - 1);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                r[i][k] = __shfl_sync(0xffffffffu, v[0][k], x / CPL);
                if (CPL > 1) {
                    const T hi = __shfl_sync(0xffffffffu, v[CPL - 1][k], x / CPL);
                    if (x % CPL) r[i][k] = hi;
                }
            }
        }
#pragma unroll
        for (int i = 0; i < CPL; ++i)
#pragma unroll
            for (int k = 0; k < 3; ++k) v[i][k] = r[i][k];
    }
    prims(v);
    warp_flux(gas, lim, w, f);
    warp_update(v, f, dtdx, w);
    double ms = 0.0;
#pragma unroll
    for (int i = 0; i < CPL; ++i) {
        const T x[3] = { T(0.5) * (u[i][0] + w[i][0]), T(0.5) * (u[i][1] + w[i][1]), T(0.5) * (u[i][2] + w[i][2]) };
        const Cell1<T> q = cell1d<true>(gas, x[0], x[1], x[2]);
        if (own(i)) {
            store(Unext, x, c + i);
            if (U1out) store(U1out, v[i], c + i);
            // (a NaN is dropped here and flagged below)
            ms = smax(ms, (double)(fabs(q.u) + q.cs));
            if (!(x[0] > T(0)) || !(q.p > T(0)))
                flag_cell(ctrl, ctrl->step[p] + 1, (double)x[0], (double)q.p, c + i, 0, errw_slot(p ^ 1));
        }
    }
    ms = warp_max_speed(ms);
    if (lane == 0) red[warp] = ms;
    __syncthreads();
    if (threadIdx.x == 0) {
        double m = red[0];
        for (int i = 1; i < STEP_WARPS; ++i) m = smax(m, red[i]);
        if (m > 1.79e308) atomicOr(&ctrl->err, ERRW_NONFINITE | errw_slot(p ^ 1));
        atomic_max_speed(&ctrl->maxs[p ^ 1][sel >> 1], m);
    }
}

// Ghost fill + max |u|+c of the current state into slot p (used once after
// an upload, and by the standalone compute_dt entry point).
template <typename T>
__global__ void __launch_bounds__(T1)
k1d_prepare(T* U, int n, int h, double gamma_d, int bc, StepCtrl* ctrl, int p) {
    __shared__ double red[33];
    pdl_wait();
    pdl_trigger();
    int nt = n + 2 * h;
    const Gas<T> gas(gamma_d);
    int c = blockIdx.x * T1 + threadIdx.x;
    double ms = 0.0;
    if (c < n) {
        int e = h + c;
        T v0 = U[e], v1 = U[nt + e], v2 = U[2 * nt + e];
        push_ghosts_1d(U, nt, 0, c, n, h, bc, v0);
        push_ghosts_1d(U, nt, 1, c, n, h, bc, v1);
        push_ghosts_1d(U, nt, 2, c, n, h, bc, v2);
        const Cell1<T> w = cell1d<true>(gas, v0, v1, v2);
        ms = (double)(fabs(w.u) + w.cs);
    }
    ms = warp_max(ms);
    int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) red[w] = ms;
    __syncthreads();
    if (w == 0) {
        double x = (l < T1 / 32) ? red[l] : 0.0;
        x = warp_max(x);
        if (l == 0) atomic_max_speed(&ctrl->maxs[p][0], x);
    }
}

template <typename T>
cudaError_t launch_1d_prepare_t(T* U, int n, int h, double gamma, int bc, StepCtrl* ctrl, int p, cudaStream_t st) {
    int blocks = (n + T1 - 1) / T1;
    return launch_pdl(k1d_prepare<T>, dim3(blocks), dim3(T1), 0, st, U, n, h, gamma, bc, ctrl, p);
}

template <typename T>
cudaError_t launch_1d_step_t(T* U, T* U1, int n, int h, double dx, double gamma, int bc, const LoopParams& lp,
                             StepCtrl* ctrl, int p, int which, cudaStream_t st, T* Uout) {
    int blocks = (n + T1 - 1) / T1;
    const bool mm = lp.lim == LIM_MINMOD;
    cudaError_t e = cudaSuccess;
    if (which & 1)
        e = launch_pdl(mm ? k1d_stage<T, 1, LIM_MINMOD> : k1d_stage<T, 1, -1>, dim3(blocks), dim3(NT1), 0, st,
                       (const T*)U, (const T*)nullptr, U1, n, h, dx, gamma, bc, lp, ctrl, p);
    if ((which & 2) && e == cudaSuccess)
        e = launch_pdl(mm ? k1d_stage<T, 2, LIM_MINMOD> : k1d_stage<T, 2, -1>, dim3(blocks), dim3(NT1), 0, st,
                       (const T*)U1, (const T*)U, Uout ? Uout : U, n, h, dx, gamma, bc, lp, ctrl, p);
    return e;
}

// Cells from which k1d_step takes two per lane: fewer halo cells and more
// independent work per warp against a longer chain, and below half the blocks
// fit an SM beside those of the next launch, which wait there.  us per step, one /
// two per lane: FP64 30000 cells 4.36 / 4.87, 50021 5.91 / 5.27, 65536 6.04 / 5.13,
// 200003 12.4 / 10.8, 400000 22.8 / 19.2; FP32 50021 3.34 / 3.73, 65536 3.46 / 3.47,
// 100000 5.41 / 3.97, 400000 14.3 / 9.4.
template <typename T> constexpr int STEP_TWO_CELLS = sizeof(T) == 8 ? 40000 : 80000;

template <typename T>
cudaError_t launch_1d_fused_t(const T* Un, T* Unext, T* U1out, int n, int h, double dx, double gamma, int bc,
                              const LoopParams& lp, StepCtrl* ctrl, int p, cudaStream_t st) {
    const bool two = n >= STEP_TWO_CELLS<T>;
    const int cells = step_cells(two ? 2 : 1) * STEP_WARPS, blocks = (n + cells - 1) / cells;
    auto kern = lp.lim == LIM_MINMOD ? (two ? k1d_step<T, LIM_MINMOD, 2> : k1d_step<T, LIM_MINMOD, 1>)
                                     : (two ? k1d_step<T, -1, 2> : k1d_step<T, -1, 1>);
    return launch_pdl(kern, dim3(blocks), dim3(32 * STEP_WARPS), 0, st, Un, Unext, U1out, n, h, dx, gamma, bc, lp,
                      ctrl, p);
}

}  // namespace
}  // namespace nestb
