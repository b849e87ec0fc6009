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
// warp per 24 cells with nothing in shared memory.
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
            if (!(v[0] > T(0)) || !(w.p > T(0))) flag_cell(ctrl, ctrl->step[p] + 1, (double)v[0], (double)w.p, c, 0);
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
                if (!(x == x) || x > 1.79e308) atomicOr(&ctrl->err, ERRW_NONFINITE);
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

constexpr int STEP_CELLS = 24;  // output cells per warp of k1d_step
constexpr int STEP_WARPS = 4;   // warps per CTA

// Stage fluxes of a warp whose lane k holds the primitives w of cell k: lane k
// returns the face between cells k and k+1 (k = 1 .. 29 where all 32 cells are
// valid), in the expressions of plm_flux.
template <typename T>
__device__ __forceinline__ F3<T> warp_flux(const Gas<T>& g, int lim, const T (&w)[3]) {
    T P[3], M[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const T d = __shfl_down_sync(0xffffffffu, w[k], 1) - w[k];
        const T s = limit(__shfl_up_sync(0xffffffffu, d, 1), d, lim);
        P[k] = w[k] + T(0.5) * s;
        M[k] = __shfl_down_sync(0xffffffffu, w[k] - T(0.5) * s, 1);
    }
    return face_flux(g, P[0], P[1], P[2], M[0], M[1], M[2]);
}

// One whole RK2 (Heun) step in one launch, out of place (Un -> Unext; the
// caller alternates two buffers).  A warp owns 24 cells and works alone: lane k
// holds cell c0 - 4 + k (its U^n, primitives, U1 and its primitives in registers),
// faces and neighbours' slopes come by shuffles.  The four lanes at each side are
// the halo of the two stages, recomputed by the neighbouring warps instead of
// being exchanged.  Every value is computed by the same expression, on the
// same operands, as in the two stage kernels (and nest's loop): U1 of a ghost
// cell is U1 of the cell it copies, which the periodic wrap of the primitives
// gives directly and the zero-gradient case takes from that cell's lane.  The
// block's maximum goes to the next step's slot in one fire-and-forget atomic
// (publish_step_1d clears the words).  U1out (optional) receives U1 of the step
// with its ghosts.  A finished step (time, step count or error) copies Un to
// Unext so that the state ends in the buffer the caller expects.
// Bound: one chain of two stages and the launch.  us per step (FP64 5003 / 65536 /
// 200003 cells, FP32 50021): 4.10 / 6.03 / 12.5, 2.95, against 6.03 / 7.32 / 14.3, 5.52 with 224-cell
// CTAs that staged each phase through shared memory and moved the maximum with
// a counter of finished blocks.
template <typename T, int LIM>
__global__ void __launch_bounds__(32 * STEP_WARPS)
k1d_step(const T* __restrict__ Un, T* __restrict__ Unext, T* __restrict__ U1out, int n, int h, double dx,
         double gamma_d, int bc, LoopParams lp, StepCtrl* ctrl, int p) {
    __shared__ double red[STEP_WARPS];
    const Gas<T> gas(gamma_d);
    const int nt = n + 2 * h;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c0 = (blockIdx.x * STEP_WARPS + warp) * STEP_CELLS, c = c0 - 4 + lane;
    const bool own = lane >= 4 && lane < 4 + STEP_CELLS && c < n;
    const int e = h + source_cell_1d(c, n, bc);
    const int lim = LIM >= 0 ? LIM : lp.lim;
    const double rdx = lp.cfl * dx;
    auto store = [&](T* U, const T (&v)[3]) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            U[k * nt + h + c] = v[k];
            push_ghosts_1d(U, nt, k, c, n, h, bc, v[k]);
        }
    };
    pdl_wait();
    pdl_trigger();
    const T u[3] = { Un[e], Un[nt + e], Un[2 * nt + e] };
    if (step_is_done(ctrl, p, lp)) {
        if (blockIdx.x == 0 && threadIdx.x == 0) publish_step_1d(ctrl, p, lp, true, 0.0, true);
        if (own) store(Unext, u);
        return;
    }
    T w[3];
    {
        const Cell1<T> q = cell1d<false>(gas, u[0], u[1], u[2]);
        w[0] = u[0]; w[1] = q.u; w[2] = q.p;
    }
    const F3<T> f = warp_flux(gas, lim, w);  // needs no dt
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

    T v[3] = { u[0] - dtdx * (f.a - __shfl_up_sync(0xffffffffu, f.a, 1)),
               u[1] - dtdx * (f.b - __shfl_up_sync(0xffffffffu, f.b, 1)),
               u[2] - dtdx * (f.c - __shfl_up_sync(0xffffffffu, f.c, 1)) };
    if (bc != BC_PERIODIC && (c0 < 4 || c0 + STEP_CELLS + 4 > n)) {
        // zero-gradient ghosts: U1 of the end cell they copy, a lane of this warp
        // whenever the warp reaches past the domain
        const int src = min(max(c, 0), n - 1) - (c0 - 4);
#pragma unroll
        for (int k = 0; k < 3; ++k) v[k] = __shfl_sync(0xffffffffu, v[k], src & 31);
    }
    {
        const Cell1<T> q = cell1d<false>(gas, v[0], v[1], v[2]);
        w[0] = v[0]; w[1] = q.u; w[2] = q.p;
    }
    const F3<T> g = warp_flux(gas, lim, w);
    const T x[3] = { T(0.5) * (u[0] + (v[0] - dtdx * (g.a - __shfl_up_sync(0xffffffffu, g.a, 1)))),
                     T(0.5) * (u[1] + (v[1] - dtdx * (g.b - __shfl_up_sync(0xffffffffu, g.b, 1)))),
                     T(0.5) * (u[2] + (v[2] - dtdx * (g.c - __shfl_up_sync(0xffffffffu, g.c, 1)))) };
    const Cell1<T> q = cell1d<true>(gas, x[0], x[1], x[2]);
    double ms = 0.0;
    if (own) {
        store(Unext, x);
        if (U1out) store(U1out, v);
        ms = (double)(fabs(q.u) + q.cs);
        if (!(x[0] > T(0)) || !(q.p > T(0))) flag_cell(ctrl, ctrl->step[p] + 1, (double)x[0], (double)q.p, c, 0);
    }
    ms = warp_max_speed(ms);
    if (lane == 0) red[warp] = ms;
    __syncthreads();
    if (threadIdx.x == 0) {
        // as bit patterns, which order like the speeds (a NaN above them all)
        unsigned long long m = speed_bits(red[0]);
        for (int i = 1; i < STEP_WARPS; ++i) m = max(m, speed_bits(red[i]));
        if (!(bits_speed(m) <= 1.79e308)) atomicOr(&ctrl->err, ERRW_NONFINITE);
        atomicMax(&ctrl->maxs[p ^ 1][sel >> 1], m);
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

template <typename T>
cudaError_t launch_1d_fused_t(const T* Un, T* Unext, T* U1out, int n, int h, double dx, double gamma, int bc,
                              const LoopParams& lp, StepCtrl* ctrl, int p, cudaStream_t st) {
    const int cells = STEP_CELLS * STEP_WARPS, blocks = (n + cells - 1) / cells;
    return launch_pdl(lp.lim == LIM_MINMOD ? k1d_step<T, LIM_MINMOD> : k1d_step<T, -1>, dim3(blocks),
                      dim3(32 * STEP_WARPS), 0, st, Un, Unext, U1out, n, h, dx, gamma, bc, lp, ctrl, p);
}

}  // namespace
}  // namespace nestb
