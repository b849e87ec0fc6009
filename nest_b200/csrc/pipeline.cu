// Device pipeline executor over nest's per-patch storage.
//
// nest composes a time step from stages run over every patch in order
// (include/nest/pipeline.hpp:14-151): an Exchange stage fills the halos
// (fill_all_halos), a Compute stage maps each patch to a new patch
// (value(patch)), a Reduce stage folds a value over the patches and hands
// it back to each (init / reduce / finalize); execute() runs the stages of a
// pipeline in order.  nest's own examples drive the Euler solver this way
// from host loops over patches (examples/sod1d/sod1d.cpp:219-270).
//
// Here a pipeline is a list of stages, each one kernel launch over all
// patches of the storage an exchange plan describes (nest_exchange_*):
//   EXCHANGE   the plan's halo copies (the nest_exchange kernel),
//   EULER_RHS  compute: dst = src - (dt/dx) (F_{i+1/2} - F_{i-1/2}) on every
//              interior cell, nest's euler_rhs_t (examples/sod1d/
//              euler1d.hpp:279-397) including its one-sided reconstruction
//              at the first and last interior cell of each patch,
//   COPY       compute: dst = src on the interiors,
//   AVERAGE    compute: dst = 0.5 a + 0.5 b on the interiors (sod1d's SSPRK2
//              combine, sod1d.cpp:262-266),
//   CFL_DT     reduce: init 0, reduce the max |u| + c of each patch interior,
//              finalize dt = cfl dx / max, clipped to t_final - time
//              (compute_dt, sod1d.cpp:97-128 and :222-223),
//   CHECK      nest's positivity check every `k` steps (sod1d.cpp:279-301),
//   CLOCK      time += dt, step += 1.
// A 1D pipeline of up to 16384 cells runs whole, all stages and all steps, in one
// launch of one CTA or one thread-block cluster (k_pipe_loop); others run a
// launch per stage.  dt, time and the step count live in a device control block,
// so a step needs no host synchronisation and runs of per-stage steps are
// replayed from CUDA graphs.  A CFL_DT stage that finds time >= t_final marks the step
// inactive: the later stages of that execution do nothing.
//
// Compiled with -fmad=false: every formula keeps nest's operation order, so
// results equal nest's CPU code bit for bit.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <map>
#include <new>
#include <vector>

#include "euler1d_arith.cuh"
#include "solver_impl.h"

using namespace nestb;
using namespace nestb::rt;

namespace nestb {
namespace {

// One patch of the storage: element offset of its block, interior extents
// and extended extents (1D: n1 = ext1 = 1).
struct PatchInfo {
    long long off;
    int n0, n1, ext0, ext1;
};

// Device control block of a pipeline.
struct PipeCtrl {
    double time, dt, t_final;
    double maxs;          // CFL_DT: reduced max |u| + c (non-negative; bits compare like values)
    int step;
    int active;           // 0: the run is finished, stages after CFL_DT do nothing
    unsigned err;         // ERRW_* bits (CHECK)
    int bad_step, bad_cell, bad_patch;
    double bad_rho, bad_p;
};

__device__ __forceinline__ long long interior_at(const PatchInfo& P, int h, int dim, int v, int a, int b) {
    return P.off + (long long)v * P.ext0 * P.ext1 + (long long)(a + h) * P.ext1 + (dim == 2 ? b + h : 0);
}

// cons_to_prim, euler1d.hpp:69-84.
__device__ __forceinline__ void prim1d(const double* U, long long e, long long plane, double gm1, double& r, double& u,
                                       double& p) {
    r = U[e];
    const double m = U[plane + e];
    u = m / r;
    p = eos_pressure(gm1, r, m, U[2 * plane + e]);
}

// plm_reconstruct, euler1d.hpp:150-171: left and right face states of cell 0.
__device__ __forceinline__ void plm3(const double* Wm, const double* W0, const double* Wp, int lim, double* L,
                                     double* R) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double slope = limit(W0[k] - Wm[k], Wp[k] - W0[k], lim);
        L[k] = W0[k] - 0.5 * slope;
        R[k] = W0[k] + 0.5 * slope;
    }
}

// euler_rhs_t::operator() (euler1d.hpp:297-396) on every interior cell of
// every patch: grid.y = patch, one thread per cell.
__global__ void __launch_bounds__(128) k_pipe_rhs1d(const double* __restrict__ src, double* __restrict__ dst,
                                                     const PatchInfo* P, int h, double dx, double gamma, int lim,
                                                     const PipeCtrl* c) {
    if (!c->active) return;
    const PatchInfo pi = P[blockIdx.y];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= pi.n0) return;
    const double gm1 = gamma - 1.0, dt = c->dt;
    const long long plane = pi.ext0, e = pi.off + h + i;
    double W[5][3];  // cells i-2 .. i+2
#pragma unroll
    for (int q = 1; q <= 3; ++q) prim1d(src, e + q - 2, plane, gm1, W[q][0], W[q][1], W[q][2]);
    // one-sided at the patch edges: i-2 -> i-1 on the first cell, i+2 -> i+1 on the last
    if (i >= 1) prim1d(src, e - 2, plane, gm1, W[0][0], W[0][1], W[0][2]);
    else for (int k = 0; k < 3; ++k) W[0][k] = W[1][k];
    if (i < pi.n0 - 1) prim1d(src, e + 2, plane, gm1, W[4][0], W[4][1], W[4][2]);
    else for (int k = 0; k < 3; ++k) W[4][k] = W[3][k];
    double aL[3], aR[3], bL[3], bR[3], cL[3], cR[3];
    plm3(W[0], W[1], W[2], lim, aL, aR);
    plm3(W[1], W[2], W[3], lim, bL, bR);
    plm3(W[2], W[3], W[4], lim, cL, cR);
    double fl[3], fr[3];
    hlle1d(gamma, gm1, aR[0], aR[1], aR[2], bL[0], bL[1], bL[2], fl[0], fl[1], fl[2]);
    hlle1d(gamma, gm1, bR[0], bR[1], bR[2], cL[0], cL[1], cL[2], fr[0], fr[1], fr[2]);
#pragma unroll
    for (int k = 0; k < 3; ++k) dst[k * plane + e] = src[k * plane + e] - (dt / dx) * (fr[k] - fl[k]);
}

// dst = src (op 0) or dst = 0.5 a + 0.5 b (op 1) on every interior element.
__global__ void __launch_bounds__(256) k_pipe_interior(double* dst, const double* a, const double* b,
                                                        const PatchInfo* P, int h, int dim, int nvars, int op,
                                                        const PipeCtrl* c) {
    if (!c->active) return;
    const PatchInfo pi = P[blockIdx.y];
    const long long per = (long long)pi.n0 * pi.n1, total = per * nvars;
    for (long long t = blockIdx.x * 256ll + threadIdx.x; t < total; t += (long long)gridDim.x * 256) {
        const int v = (int)(t / per);
        const long long q = t - v * per;
        const int ia = (int)(q / pi.n1), ib = (int)(q - (long long)ia * pi.n1);
        const long long o = interior_at(pi, h, dim, v, ia, ib);
        dst[o] = op == 0 ? a[o] : 0.5 * a[o] + 0.5 * b[o];
    }
}

// CFL reduce: init (slot 0), reduce (one block per patch, atomic max on the
// bit pattern of the non-negative maximum), finalize (one thread).
__global__ void k_pipe_cfl_init(PipeCtrl* c) {
    if (c->t_final > 0.0) c->active = (c->time < c->t_final) && !(c->err & ERRW_STOP) ? 1 : 0;
    else c->active = (c->err & ERRW_STOP) ? 0 : 1;
    c->maxs = 0.0;
}

__global__ void __launch_bounds__(256) k_pipe_cfl_reduce(const double* U, const PatchInfo* P, int h, double gamma,
                                                          PipeCtrl* c) {
    if (!c->active) return;
    const PatchInfo pi = P[blockIdx.x];
    const double gm1 = gamma - 1.0;
    double ms = 0.0;
    for (int i = threadIdx.x; i < pi.n0; i += 256) {
        double r, u, p;
        prim1d(U, pi.off + h + i, pi.ext0, gm1, r, u, p);
        const double cs = sqrt(gamma * p / r);  // eos_t::sound_speed, euler1d.hpp:54-56
        ms = smax(ms, fabs(u) + cs);
    }
    ms = warp_max(ms);
    __shared__ double red[8];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ms;
    __syncthreads();
    if (threadIdx.x == 0) {
        double m = 0.0;
        for (int w = 0; w < 8; ++w) m = smax(m, red[w]);
        atomicMax(reinterpret_cast<unsigned long long*>(&c->maxs), speed_bits(m));
    }
}

__global__ void k_pipe_cfl_finalize(PipeCtrl* c, double cfl, double dx) {
    if (!c->active) return;
    double dt = cfl * dx / c->maxs;
    if (c->t_final > 0.0) dt = smin(dt, c->t_final - c->time);
    c->dt = dt;
}

// nest's positivity check (sod1d.cpp:279-301) on the interiors, when the
// completed step count is a multiple of `every`.
__global__ void __launch_bounds__(256) k_pipe_check(const double* U, const PatchInfo* P, int h, double gamma,
                                                     int every, PipeCtrl* c) {
    if (!c->active || (c->step + 1) % every != 0) return;
    const PatchInfo pi = P[blockIdx.x];
    const double gm1 = gamma - 1.0;
    for (int i = threadIdx.x; i < pi.n0; i += 256) {
        double r, u, p;
        prim1d(U, pi.off + h + i, pi.ext0, gm1, r, u, p);
        if (!(r > 0.0) || !(p > 0.0)) {
            const unsigned bit = (r == r && p == p) ? ERRW_NONPOSITIVE : ERRW_NONFINITE;
            if (!(atomicOr(&c->err, bit) & ERRW_STOP)) {
                c->bad_step = c->step + 1; c->bad_cell = i; c->bad_patch = blockIdx.x;
                c->bad_rho = r; c->bad_p = p;
            }
        }
    }
}

__global__ void k_pipe_clock(PipeCtrl* c) {
    if (!c->active) return;
    c->time = c->time + c->dt;
    c->step = c->step + 1;
}

struct Stage {
    int kind, src, dst, aux;
    double param;
};

// ---------------------------------------------------------------------------
// The whole pipeline in one launch (1D)
// ---------------------------------------------------------------------------

constexpr int LOOP_STAGES = 32, LOOP_BUFFERS = 17;
constexpr int LOOP_THREADS = 512, LOOP_K = 2;  // threads per CTA, cells per thread
constexpr size_t LOOP_SMEM = 160 << 10;        // most that the buffers of the one-CTA form take
constexpr int LOOP_SLOT = 28;                  // cells of a warp that shares faces
// One CTA (cheap barriers, buffers in shared memory) where its warps take the cells in
// two slots each or where there are few, else a cluster of 16, whose six barriers a
// step cost about 0.45 us each: us per step, one CTA / cluster, 100 cells in 2 patches
// 4.6 / 11.4, 400 in 4 6.3 / 12.5, 800 in 5 (30 slots) 8.9 / 12.6, 900 in 8 (40, no slots)
// 13.3 / 12.4.
constexpr int LOOP_ONE_CTA = 640, LOOP_ONE_SLOTS = LOOP_K * LOOP_THREADS / 32;

struct LoopArgs {
    int nstages;
    Stage st[LOOP_STAGES];
    unsigned sync_before;         // bit s: stage s needs a barrier before it
    double* buf[LOOP_BUFFERS];
    const PatchInfo* P;
    int npatch, ncells, h;
    const int2* copies;           // exchange: (destination, source) element offsets
    int ncopies;
    double dx, gamma;
    int lim;
    int share;                    // a warp per LOOP_SLOT cells of a patch, faces shared by shuffles
    int total, nbuf;              // elements of a buffer, buffers (SMEM)
    PipeCtrl* c;
    int steps;                    // executions of the stage list at most
    int max_steps, step0;         // > 0: stop at a multiple of 8 executions once step - step0 reaches it
    int once_more;                // a CFL stage has compute stages before it
};

// Executes the stage list up to `steps` times in one CTA or one cluster: a
// thread owns up to LOOP_K cells in every stage, so element-wise stages follow
// one another without a barrier, and only a stage that reads other threads'
// elements (EXCHANGE, EULER_RHS, the CFL maximum), or overwrites what others may
// still be reading, waits for one (LoopArgs::sync_before).  Every thread keeps the
// clock in registers; they all compute the same dt.  The formulas are those of
// the stage kernels above, with the branch-free division and square root.
// An execution whose CFL stage finds the run finished is the last one: its later halo
// exchanges still run, and further executions of the batch of eight would run nothing
// but exchanges.  They would change nothing either, unless compute stages come before the
// CFL stage in the list and so have changed what exchanges before it have copied; then one
// more execution of the batch (further ones repeat it) refreshes the halos.
// share: a warp takes up to 28 neighbouring cells of a patch and a halo of two on each side,
// and every primitive, slope and flux is computed once instead of by up to five cells.
// SMEM (one CTA): the buffers live in shared memory for the launch.
// Bound: the latency of the stages' chains and their barriers.  nest's sod1d step
// (ten stages, twelve launches), us per step against a launch per stage: 100 cells
// 4.6 (26), 400 6.2 (30), 1024 12.5 (31), 4000 12.6 (31), 16000 25 (38); with every cell
// computing both its faces and the buffers in global memory 100 cells 6.4, 400 9.8,
// 1024 14.1, 4000 14.4.
template <bool CLUSTER, bool SMEM>
__global__ void __launch_bounds__(LOOP_THREADS) k_pipe_loop(LoopArgs a) {
    namespace cg = cooperative_groups;
    extern __shared__ double pipe_buf[];
    __shared__ double red[2][16 * (LOOP_THREADS / 32)];
    const int NC = CLUSTER ? (int)cg::this_cluster().num_blocks() : 1;
    const int rank = CLUSTER ? (int)cg::this_cluster().block_rank() : 0;
    auto sync = [&]() {
        if (CLUSTER) cg::this_cluster().sync();
        else __syncthreads();
    };
    const int T = blockDim.x, nw = T >> 5, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int gt = rank * T + threadIdx.x, NT = NC * T;
    const Gas<double> gas(a.gamma);
    const double gm1 = a.gamma - 1.0;
    PipeCtrl* const c = a.c;

    // the thread's cells: element offset, plane stride, place in the patch (patch -1:
    // none; with shared faces a warp's lanes hold neighbouring cells, two of halo on each side, and
    // e is the element that a lane reads as its cell)
    struct Own {
        int e, plane, patch, i, n0;
    } own[LOOP_K];
#pragma unroll
    for (int k = 0; k < LOOP_K; ++k) {
        own[k] = { 0, 0, -1, 0, 0 };
        if (a.share) {
            int f = (gt + k * NT) >> 5, p = 0;
            while (p < a.npatch && f >= (a.P[p].n0 + LOOP_SLOT - 1) / LOOP_SLOT)
                f -= (a.P[p++].n0 + LOOP_SLOT - 1) / LOOP_SLOT;
            if (p < a.npatch) {
                // one-sided at the patch edges: the cell two outside reads as the one outside
                const int i = LOOP_SLOT * f - 2 + lane, n0 = a.P[p].n0;
                own[k] = { (int)a.P[p].off + a.h + min(max(i, -1), n0), a.P[p].ext0,
                           lane >= 2 && lane < 2 + LOOP_SLOT && i < n0 ? p : -1, i, n0 };
            }
        } else {
            int f = gt + k * NT;
            if (f < a.ncells) {
                int p = 0;
                while (f >= a.P[p].n0) f -= a.P[p++].n0;
                own[k] = { (int)a.P[p].off + a.h + f, a.P[p].ext0, p, f, a.P[p].n0 };
            }
        }
    }
    if (SMEM)
        for (int b = 0; b < a.nbuf; ++b)
            for (int q = threadIdx.x; q < a.total; q += T) pipe_buf[b * a.total + q] = a.buf[b][q];
    auto buf = [&](int b) { return SMEM ? pipe_buf + b * a.total : a.buf[b]; };
    double time = c->time, dt = c->dt;
    int step = c->step, active = c->active;
    const double t_final = c->t_final;
    int cfl_count = 0;
    // Whether a CHECK has failed, in an earlier launch (read before the barrier: no thread
    // has run a CHECK) or in this one, where the news travels with the wave-speed
    // maxima: a thread whose cell failed sends FAILED, above every speed, in the
    // place of its own, so that all threads stop at the same CFL stage.
    const double FAILED = __longlong_as_double(0x7fffffffffffffffll);
    bool stopped = (*reinterpret_cast<volatile unsigned*>(&c->err) & ERRW_STOP) != 0, failed = false;
    sync();  // the buffers are filled, and every CTA of a cluster runs before its memory is written

    bool ended = false;
    for (int n = 0; n < a.steps; ++n) {
        // batches of 8, as a launch per stage runs them
        if (n > 0 && (n & 7) == 0 && ((a.max_steps > 0 && step - a.step0 >= a.max_steps) || !(time < t_final))) break;
        bool finished = false;
        for (int s = 0; s < a.nstages; ++s) {
            const Stage& g = a.st[s];
            if ((a.sync_before >> s) & 1u) sync();
            double* const src = buf(g.src);
            double* const dst = buf(g.dst);
            if (g.kind == NEST_STAGE_CFL_DT) {
                double ms = 0.0;
#pragma unroll
                for (int k = 0; k < LOOP_K; ++k)
                    if (own[k].patch >= 0) {
                        const int e = own[k].e;
                        const int pl = own[k].plane;
                        const Cell1<double> w = cell1d<true>(gas, src[e], src[e + pl], src[e + 2 * pl]);
                        ms = smax(ms, fabs(w.u) + w.cs);
                    }
                ms = warp_max_speed(failed ? FAILED : ms);
                double* const r = red[cfl_count & 1];
                ++cfl_count;
                if (lane < NC)
                    (CLUSTER ? cg::this_cluster().map_shared_rank(r, lane) : r)[rank * nw + warp] = ms;
                sync();
                unsigned long long mb = 0;
                for (int q = lane; q < NC * nw; q += 32) mb = max(mb, speed_bits(r[q]));
                const double m = warp_max_speed(bits_speed(mb));
                stopped = stopped || m != m;
                active = (!(t_final > 0.0) || time < t_final) && !stopped ? 1 : 0;
                if (active) {
                    dt = div_rn(g.param * a.dx, m);
                    if (t_final > 0.0) dt = smin(dt, t_final - time);
                }
                finished = !active;
                continue;
            }
            if (g.kind == NEST_STAGE_EXCHANGE) {
                for (int q = gt; q < a.ncopies; q += NT) {
                    const int2 d = a.copies[q];
                    src[d.x] = src[d.y];
                }
                continue;
            }
            if (!active) continue;
            switch (g.kind) {
                case NEST_STAGE_EULER_RHS: {
                    const double dtdx = div_rn(dt, a.dx);
                    if (a.share) {
#pragma unroll
                        for (int k = 0; k < LOOP_K; ++k) {
                            const int e = own[k].e, pl = own[k].plane;
                            if (pl == 0) continue;  // the whole warp
                            const double U[1][3] = { { src[e], src[e + pl], src[e + 2 * pl] } };
                            const Cell1<double> q = cell1d<false>(gas, U[0][0], U[0][1], U[0][2]);
                            const double W[1][3] = { { U[0][0], q.u, q.p } };
                            F3<double> f[1];
                            warp_flux(gas, a.lim, W, f);
                            const double fa = __shfl_up_sync(0xffffffffu, f[0].a, 1);
                            const double fb = __shfl_up_sync(0xffffffffu, f[0].b, 1);
                            const double fc = __shfl_up_sync(0xffffffffu, f[0].c, 1);
                            if (own[k].patch < 0) continue;
                            dst[e] = U[0][0] - dtdx * (f[0].a - fa);
                            dst[e + pl] = U[0][1] - dtdx * (f[0].b - fb);
                            dst[e + 2 * pl] = U[0][2] - dtdx * (f[0].c - fc);
                        }
                        break;
                    }
#pragma unroll
                    for (int k = 0; k < LOOP_K; ++k) {
                        if (own[k].patch < 0) continue;
                        const int e = own[k].e;
                        const int pl = own[k].plane, i = own[k].i;
                        double U[3], W[5][3];  // cells i-2 .. i+2
#pragma unroll
                        for (int q = 0; q < 5; ++q) {
                            // one-sided at the patch edges: i-2 -> i-1 on the first cell, i+2 -> i+1 on the last
                            const int x = e + (q == 0 && i == 0 ? -1 : q == 4 && i == own[k].n0 - 1 ? 1 : q - 2);
                            const double r = src[x], m = src[x + pl], E = src[x + 2 * pl];
                            const Cell1<double> w = cell1d<false>(gas, r, m, E);
                            W[q][0] = r; W[q][1] = w.u; W[q][2] = w.p;
                            if (q == 2) { U[0] = r; U[1] = m; U[2] = E; }
                        }
                        double aL[3], aR[3], bL[3], bR[3], cL[3], cR[3];
                        plm3(W[0], W[1], W[2], a.lim, aL, aR);
                        plm3(W[1], W[2], W[3], a.lim, bL, bR);
                        plm3(W[2], W[3], W[4], a.lim, cL, cR);
                        const F3<double> fl = face_flux(gas, aR[0], aR[1], aR[2], bL[0], bL[1], bL[2]);
                        const F3<double> fr = face_flux(gas, bR[0], bR[1], bR[2], cL[0], cL[1], cL[2]);
                        dst[e] = U[0] - dtdx * (fr.a - fl.a);
                        dst[e + pl] = U[1] - dtdx * (fr.b - fl.b);
                        dst[e + 2 * pl] = U[2] - dtdx * (fr.c - fl.c);
                    }
                    break;
                }
                case NEST_STAGE_COPY:
                case NEST_STAGE_AVERAGE: {
                    const double* const aux = buf(g.aux);
#pragma unroll
                    for (int k = 0; k < LOOP_K; ++k)
                        if (own[k].patch >= 0)
                            for (int v = 0; v < 3; ++v) {
                                const int e = own[k].e + v * own[k].plane;
                                dst[e] = g.kind == NEST_STAGE_COPY ? src[e] : 0.5 * src[e] + 0.5 * aux[e];
                            }
                    break;
                }
                case NEST_STAGE_CHECK:
                    if ((step + 1) % (int)g.param == 0) {
#pragma unroll
                        for (int k = 0; k < LOOP_K; ++k)
                            if (own[k].patch >= 0) {
                                double r, u, p;
                                prim1d(src, own[k].e, own[k].plane, gm1, r, u, p);
                                if (!(r > 0.0) || !(p > 0.0)) {
                                    failed = true;
                                    const unsigned bit = (r == r && p == p) ? ERRW_NONPOSITIVE : ERRW_NONFINITE;
                                    if (!(atomicOr(&c->err, bit) & ERRW_STOP)) {
                                        c->bad_step = step + 1; c->bad_cell = own[k].i; c->bad_patch = own[k].patch;
                                        c->bad_rho = r; c->bad_p = p;
                                    }
                                }
                            }
                    }
                    break;
                case NEST_STAGE_CLOCK:
                    time = time + dt;
                    step = step + 1;
                    break;
            }
        }
        if (finished) {
            if (ended || !a.once_more || (n & 7) == 7) break;
            ended = true;
        }
    }
    if (SMEM) {
        __syncthreads();
        for (int b = 0; b < a.nbuf; ++b)
            for (int q = threadIdx.x; q < a.total; q += T) a.buf[b][q] = pipe_buf[b * a.total + q];
    }
    if (CLUSTER) sync();  // no CTA leaves while another's stores to it may be in flight
    if (gt == 0) { c->time = time; c->dt = dt; c->step = step; c->active = active; }
}

}  // namespace
}  // namespace nestb

struct nest_pipeline {
    nest_exchange* plan = nullptr;
    int dim = 1, nvars = 3, halo = 2, npatch = 0, nwork = 0, lim = LIM_MINMOD;
    double dx = 1.0, gamma = 1.4;
    long long total = 0;              // elements of one storage block (all patches)
    int max_n0 = 0;
    std::vector<PatchInfo> patches;
    PatchInfo* dpatches = nullptr;
    std::vector<double*> work;        // pipeline-owned buffers 1..nwork
    PipeCtrl* ctrl = nullptr;
    PipeCtrl* host_ctrl = nullptr;
    std::vector<Stage> stages;
    int ncells = 0;
    int2* dcopies = nullptr;          // 1D: the exchange plan's element pairs
    int ncopies = 0;
    int slots = 0;                    // 1D: groups of up to LOOP_SLOT cells of one patch
    size_t loop_smem = 0;             // shared memory that the one-CTA form may take for the buffers
    int loop_ctas = 0;                // CTAs of the one-launch form (0: a launch per stage)
    cudaStream_t own = nullptr;
    std::map<std::pair<void*, cudaStream_t>, cudaGraphExec_t> graphs;
};

namespace nestb {
namespace {

constexpr int PIPE_GRAPH_STEPS = 8;

void drop_pipe_graphs(nest_pipeline* p) {
    for (auto& kv : p->graphs) cudaGraphExecDestroy(kv.second);
    p->graphs.clear();
}

double* buffer(nest_pipeline* p, void* state, int b) { return b == 0 ? (double*)state : p->work[b - 1]; }

cudaError_t launch_stage(nest_pipeline* p, const Stage& s, void* state, cudaStream_t st) {
    double* src = buffer(p, state, s.src);
    const int h = p->halo;
    switch (s.kind) {
        case NEST_STAGE_EXCHANGE: {
            nest_status r = nest_exchange_execute(p->plan, src, NEST_F64, st);
            return r == NEST_OK ? cudaSuccess : cudaErrorLaunchFailure;
        }
        case NEST_STAGE_EULER_RHS: {
            dim3 gr((p->max_n0 + 127) / 128, p->npatch);
            k_pipe_rhs1d<<<gr, 128, 0, st>>>(src, buffer(p, state, s.dst), p->dpatches, h, p->dx, p->gamma, p->lim,
                                             p->ctrl);
            break;
        }
        case NEST_STAGE_COPY:
        case NEST_STAGE_AVERAGE: {
            long long per = 0;
            for (auto& q : p->patches) per = std::max(per, (long long)q.n0 * q.n1 * p->nvars);
            dim3 gr((unsigned)std::min<long long>((per + 255) / 256, 64), p->npatch);
            k_pipe_interior<<<gr, 256, 0, st>>>(buffer(p, state, s.dst), src,
                                                s.kind == NEST_STAGE_AVERAGE ? buffer(p, state, s.aux) : nullptr,
                                                p->dpatches, h, p->dim, p->nvars,
                                                s.kind == NEST_STAGE_AVERAGE ? 1 : 0, p->ctrl);
            break;
        }
        case NEST_STAGE_CFL_DT:
            k_pipe_cfl_init<<<1, 1, 0, st>>>(p->ctrl);
            k_pipe_cfl_reduce<<<p->npatch, 256, 0, st>>>(src, p->dpatches, h, p->gamma, p->ctrl);
            k_pipe_cfl_finalize<<<1, 1, 0, st>>>(p->ctrl, s.param, p->dx);
            break;
        case NEST_STAGE_CHECK:
            k_pipe_check<<<p->npatch, 256, 0, st>>>(src, p->dpatches, h, p->gamma, (int)s.param, p->ctrl);
            break;
        case NEST_STAGE_CLOCK:
            k_pipe_clock<<<1, 1, 0, st>>>(p->ctrl);
            break;
        default:
            return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

// Barriers of the one-launch form: what has happened to each buffer since the
// last one decides whether a stage must wait (the list repeats, so it starts from
// what its own end leaves behind).
unsigned loop_barriers(const std::vector<Stage>& st) {
    struct Seen {
        bool own_written = false;   // interiors, each element by its owner
        bool halo_written = false;
        bool read_across = false;   // by threads other than the owner
    };
    unsigned bits = 0;
    Seen b[LOOP_BUFFERS];
    for (int pass = 0; pass < 2; ++pass)
        for (size_t s = 0; s < st.size(); ++s) {
            const Stage& g = st[s];
            bool wait = false;
            switch (g.kind) {
                case NEST_STAGE_EXCHANGE: wait = b[g.src].own_written || b[g.src].read_across; break;
                case NEST_STAGE_EULER_RHS:
                    wait = b[g.src].own_written || b[g.src].halo_written || b[g.dst].read_across;
                    break;
                case NEST_STAGE_COPY:
                case NEST_STAGE_AVERAGE: wait = b[g.dst].read_across; break;
                default: break;
            }
            if (wait) {
                bits |= 1u << s;
                for (Seen& x : b) x = Seen{};
            }
            switch (g.kind) {
                case NEST_STAGE_EXCHANGE: b[g.src].read_across = b[g.src].halo_written = true; break;
                case NEST_STAGE_EULER_RHS: b[g.src].read_across = b[g.dst].own_written = true; break;
                case NEST_STAGE_COPY:
                case NEST_STAGE_AVERAGE: b[g.dst].own_written = true; break;
                case NEST_STAGE_CFL_DT:  // waits inside, after its own reads
                    for (Seen& x : b) x = Seen{};
                    break;
                default: break;
            }
        }
    return bits;
}

bool use_loop(const nest_pipeline* p) { return p->loop_ctas > 0 && p->stages.size() <= LOOP_STAGES; }

cudaError_t launch_loop(nest_pipeline* p, void* state, int steps, int max_steps, int step0, cudaStream_t st) {
    LoopArgs a{};
    a.nstages = (int)p->stages.size();
    for (int s = 0; s < a.nstages; ++s) a.st[s] = p->stages[s];
    // A caller may pass one of the work arrays as the state, or memory that overlaps them:
    // two indices then name the same elements, which the analysis by index cannot see, so
    // every stage waits for the one before, as with a launch per stage.
    bool apart = true;
    for (double* w : p->work) apart = apart && ((double*)state + p->total <= w || w + p->total <= (double*)state);
    a.sync_before = apart ? loop_barriers(p->stages) : ~0u;
    for (int b = 0; b <= p->nwork; ++b) a.buf[b] = buffer(p, state, b);
    a.P = p->dpatches;
    a.npatch = p->npatch; a.ncells = p->ncells; a.h = p->halo;
    a.copies = p->dcopies; a.ncopies = p->ncopies;
    a.dx = p->dx; a.gamma = p->gamma; a.lim = p->lim;
    a.c = p->ctrl;
    a.steps = steps; a.max_steps = max_steps; a.step0 = step0;
    bool computed = false;
    for (const Stage& g : p->stages) {
        if (g.kind == NEST_STAGE_CFL_DT && computed) a.once_more = 1;
        computed |= g.kind == NEST_STAGE_EULER_RHS || g.kind == NEST_STAGE_COPY || g.kind == NEST_STAGE_AVERAGE;
    }
    const int NC = p->loop_ctas;
    // shared faces where the slots take no more rounds of the warps than the cells do of the
    // threads (8000 cells in 16 patches, two rounds for one: 19.4 us a step for 16.9) and
    // short patches do not leave their lanes idle
    auto rounds = [&](int units, int per_cta) { return (units + NC * per_cta - 1) / (NC * per_cta); };
    const int cell_rounds = NC == 1 ? LOOP_K : rounds(p->ncells, LOOP_THREADS);
    a.share = rounds(p->slots, LOOP_THREADS / 32) <= cell_rounds && LOOP_SLOT * p->slots <= 2 * p->ncells;
    const int per = ((a.share ? 32 * p->slots : p->ncells) + NC - 1) / NC;  // lanes per CTA
    const int threads = std::min(LOOP_THREADS, (per + 31) / 32 * 32);
    if (NC == 1) {
        a.total = (int)p->total;
        a.nbuf = p->nwork + 1;
        const size_t smem = sizeof(double) * (size_t)a.total * a.nbuf;
        if (!apart || smem > p->loop_smem) k_pipe_loop<false, false><<<1, threads, 0, st>>>(a);
        else k_pipe_loop<false, true><<<1, threads, smem, st>>>(a);
        return cudaGetLastError();
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(NC, 1, 1);
    cfg.blockDim = dim3(threads, 1, 1);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = NC;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_pipe_loop<true, false>, a);
}

// CTAs of the one-launch form for a 1D pipeline: one for the smallest, else a
// cluster of 16 (or the 8 every device places), 0 where the cells do not fit.
int loop_ctas_for(int ncells, int slots) {
    if (ncells <= LOOP_ONE_CTA || (slots <= LOOP_ONE_SLOTS && LOOP_SLOT * slots <= 2 * ncells)) return 1;
    for (int NC : {16, 8}) {
        if (ncells > NC * LOOP_THREADS * LOOP_K) continue;
        if (NC > 8 &&
            cudaFuncSetAttribute(k_pipe_loop<true, false>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
            cudaGetLastError();
            continue;
        }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(NC, 1, 1);
        cfg.blockDim = dim3(LOOP_THREADS, 1, 1);
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = NC;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, k_pipe_loop<true, false>, &cfg) != cudaSuccess) {
            cudaGetLastError();
            continue;
        }
        if (clusters >= 1) return NC;
    }
    return 0;
}

cudaError_t launch_all(nest_pipeline* p, void* state, cudaStream_t st) {
    cudaError_t e = cudaSuccess;
    for (const Stage& s : p->stages)
        if ((e = launch_stage(p, s, state, st)) != cudaSuccess) break;
    return e;
}

nest_status read_pipe_ctrl(nest_pipeline* p, cudaStream_t st) {
    CK(cudaMemcpyAsync(p->host_ctrl, p->ctrl, sizeof(PipeCtrl), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    const PipeCtrl& c = *p->host_ctrl;
    if (c.err & ERRW_STOP) {
        char buf[256];
        const bool nan = !(c.bad_rho == c.bad_rho) || !(c.bad_p == c.bad_p);
        std::snprintf(buf, sizeof buf, "%s at step %d in patch %d, interior cell %d: rho = %.17g, p = %.17g",
                      nan ? "non-finite state (NaN)" : "positivity violation (rho <= 0 or p <= 0)", c.bad_step,
                      c.bad_patch, c.bad_cell, c.bad_rho, c.bad_p);
        return fail(NEST_ERR_NUMERIC, buf);
    }
    return NEST_OK;
}

nest_status pcheck(const nest_pipeline* p) {
    if (!p) return fail(NEST_ERR_INVALID, "null pipeline handle");
    return NEST_OK;
}

}  // namespace
}  // namespace nestb

extern "C" {

nest_status nest_pipeline_create(int dim, int nx, int ny, int npx, int npy, int halo, double dx, double gamma,
                                 int limiter, int nwork, nest_pipeline** out) {
    if (!out) return fail(NEST_ERR_INVALID, "null argument");
    *out = nullptr;
    if (dim != 1 && dim != 2) return fail(NEST_ERR_INVALID, "dim must be 1 or 2");
    if (!(dx > 0.0) || !(gamma > 1.0)) return fail(NEST_ERR_INVALID, "dx must be positive and gamma > 1");
    if (nwork < 0 || nwork > 16) return fail(NEST_ERR_INVALID, "work buffers must be 0..16");
    if (limiter != LIM_MINMOD && limiter != LIM_MC && limiter != LIM_NONE) return fail(NEST_ERR_INVALID, "bad limiter");
    auto* p = new (std::nothrow) nest_pipeline;
    if (!p) return fail(NEST_ERR_OOM, "host allocation failed");
    p->dim = dim; p->nvars = dim == 1 ? 3 : 4; p->halo = halo; p->dx = dx; p->gamma = gamma; p->lim = limiter;
    p->nwork = nwork;
    auto cleanup = [&](nest_status st) { nest_pipeline_destroy(p); return st; };
    nest_status r = nest_exchange_create_periodic(dim, nx, ny, npx, npy, p->nvars, halo, &p->plan);
    if (r != NEST_OK) return cleanup(r);
    p->npatch = dim == 2 ? npx * npy : npx;
    std::vector<long long> offs(p->npatch + 1);
    std::vector<int> boxes(4 * p->npatch);
    nest_exchange_layout(p->plan, offs.data(), boxes.data(), nullptr);
    p->total = offs[p->npatch];
    for (int q = 0; q < p->npatch; ++q) {
        PatchInfo pi;
        pi.off = offs[q];
        pi.n0 = boxes[4 * q + 2];
        pi.n1 = dim == 2 ? boxes[4 * q + 3] : 1;
        pi.ext0 = pi.n0 + 2 * halo;
        pi.ext1 = dim == 2 ? pi.n1 + 2 * halo : 1;
        p->patches.push_back(pi);
        p->max_n0 = std::max(p->max_n0, pi.n0);
        p->ncells += dim == 1 ? pi.n0 : 0;
        p->slots += dim == 1 ? (pi.n0 + LOOP_SLOT - 1) / LOOP_SLOT : 0;
    }
    cudaError_t e;
    if (dim == 1 && p->ncells <= 16 * LOOP_THREADS * LOOP_K && (p->loop_ctas = loop_ctas_for(p->ncells, p->slots)) > 0) {
        const size_t need = sizeof(double) * (size_t)p->total * (nwork + 1);
        if (p->loop_ctas == 1 && need <= LOOP_SMEM) {
            if (cudaFuncSetAttribute(k_pipe_loop<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)LOOP_SMEM) == cudaSuccess)
                p->loop_smem = LOOP_SMEM;
            else
                cudaGetLastError();
        }
        std::vector<int2> pairs;
        for (auto [d, src] : exchange_pairs_1d(p->plan)) pairs.push_back(make_int2((int)d, (int)src));
        p->ncopies = (int)pairs.size();
        if ((e = cudaMalloc(&p->dcopies, sizeof(int2) * pairs.size())) != cudaSuccess ||
            (e = cudaMemcpy(p->dcopies, pairs.data(), sizeof(int2) * pairs.size(), cudaMemcpyHostToDevice)) !=
                cudaSuccess)
            return cleanup(cuda_fail(e, "exchange pairs"));
    }
    if ((e = cudaMalloc(&p->dpatches, sizeof(PatchInfo) * p->npatch)) != cudaSuccess) return cleanup(cuda_fail(e, "cudaMalloc"));
    if ((e = cudaMemcpy(p->dpatches, p->patches.data(), sizeof(PatchInfo) * p->npatch, cudaMemcpyHostToDevice)) !=
        cudaSuccess)
        return cleanup(cuda_fail(e, "cudaMemcpy"));
    for (int w = 0; w < nwork; ++w) {
        double* b = nullptr;
        if ((e = cudaMalloc(&b, sizeof(double) * p->total)) != cudaSuccess) return cleanup(cuda_fail(e, "cudaMalloc(work)"));
        p->work.push_back(b);
        if ((e = cudaMemset(b, 0, sizeof(double) * p->total)) != cudaSuccess) return cleanup(cuda_fail(e, "memset"));
    }
    if ((e = cudaMalloc(&p->ctrl, sizeof(PipeCtrl))) != cudaSuccess) return cleanup(cuda_fail(e, "cudaMalloc(ctrl)"));
    if ((e = cudaMemset(p->ctrl, 0, sizeof(PipeCtrl))) != cudaSuccess) return cleanup(cuda_fail(e, "memset"));
    if ((e = cudaMallocHost(&p->host_ctrl, sizeof(PipeCtrl))) != cudaSuccess) return cleanup(cuda_fail(e, "cudaMallocHost"));
    if ((e = cudaStreamCreateWithFlags(&p->own, cudaStreamNonBlocking)) != cudaSuccess)
        return cleanup(cuda_fail(e, "cudaStreamCreate"));
    // a step that starts active until a CFL stage says otherwise
    PipeCtrl c{};
    c.active = 1;
    if ((e = cudaMemcpy(p->ctrl, &c, sizeof c, cudaMemcpyHostToDevice)) != cudaSuccess) return cleanup(cuda_fail(e, "cudaMemcpy"));
    // the copies above went to the legacy stream, which the callers' streams do not wait for
    if ((e = cudaStreamSynchronize(cudaStreamLegacy)) != cudaSuccess) return cleanup(cuda_fail(e, "sync"));
    *out = p;
    return NEST_OK;
}

nest_status nest_pipeline_destroy(nest_pipeline* p) {
    if (!p) return NEST_OK;
    if (p->own) cudaStreamSynchronize(p->own);
    drop_pipe_graphs(p);
    for (double* b : p->work) cudaFree(b);
    cudaFree(p->dpatches);
    cudaFree(p->dcopies);
    cudaFree(p->ctrl);
    if (p->host_ctrl) cudaFreeHost(p->host_ctrl);
    if (p->own) cudaStreamDestroy(p->own);
    nest_exchange_destroy(p->plan);
    delete p;
    return NEST_OK;
}

nest_status nest_pipeline_plan(nest_pipeline* p, nest_exchange** plan) {
    nest_status r = pcheck(p);
    if (r != NEST_OK) return r;
    if (plan) *plan = p->plan;
    return NEST_OK;
}

nest_status nest_pipeline_add(nest_pipeline* p, int kind, int src, int dst, int aux, double param) {
    nest_status r = pcheck(p);
    if (r != NEST_OK) return r;
    auto bad = [&](int b) { return b < 0 || b > p->nwork; };
    if (kind < NEST_STAGE_EXCHANGE || kind > NEST_STAGE_CLOCK) return fail(NEST_ERR_INVALID, "unknown stage kind");
    if (bad(src) || bad(dst) || bad(aux)) return fail(NEST_ERR_INVALID, "buffer index out of range");
    if ((kind == NEST_STAGE_EULER_RHS || kind == NEST_STAGE_CFL_DT || kind == NEST_STAGE_CHECK) && p->dim != 1)
        return fail(NEST_ERR_UNSUPPORTED, "Euler, CFL and positivity stages run nest's 1D patch scheme");
    if (kind == NEST_STAGE_EULER_RHS && src == dst) return fail(NEST_ERR_INVALID, "EULER_RHS needs dst != src");
    if (kind == NEST_STAGE_CFL_DT && !(param > 0.0)) return fail(NEST_ERR_INVALID, "CFL_DT needs cfl > 0");
    if (kind == NEST_STAGE_CHECK && !(param >= 1.0)) return fail(NEST_ERR_INVALID, "CHECK needs a period >= 1");
    p->stages.push_back(Stage{kind, src, dst, aux, param});
    drop_pipe_graphs(p);
    return NEST_OK;
}

nest_status nest_pipeline_execute(nest_pipeline* p, void* d_state, void* stream) {
    nest_status r = pcheck(p);
    if (r != NEST_OK) return r;
    if (!d_state) return fail(NEST_ERR_INVALID, "null state");
    cudaStream_t st = stream ? (cudaStream_t)stream : p->own;
    cudaError_t e = use_loop(p) ? launch_loop(p, d_state, 1, 0, 0, st) : launch_all(p, d_state, st);
    if (e != cudaSuccess) return cuda_fail(e, "pipeline stage launch");
    return NEST_OK;
}

nest_status nest_pipeline_run(nest_pipeline* p, void* d_state, double t_final, int max_steps, int* steps_out,
                              void* stream) {
    nest_status r = pcheck(p);
    if (r != NEST_OK) return r;
    if (!d_state || !(t_final > 0.0)) return fail(NEST_ERR_INVALID, "need a state and t_final > 0");
    bool has_cfl = false;
    for (auto& s : p->stages) has_cfl |= s.kind == NEST_STAGE_CFL_DT;
    if (!has_cfl) return fail(NEST_ERR_INVALID, "run needs a CFL_DT stage (it decides when to stop)");
    cudaStream_t st = stream ? (cudaStream_t)stream : p->own;
    if ((r = read_pipe_ctrl(p, st)) != NEST_OK) return r;
    const int start = p->host_ctrl->step;
    // t_final into the control block (the CFL stages read it)
    CK(cudaMemcpyAsync(&p->ctrl->t_final, &t_final, sizeof(double), cudaMemcpyHostToDevice, st));
    CK(cudaStreamSynchronize(st));
    const bool loop = use_loop(p);
    // executions per launch of the one-launch form (without a CLOCK stage no step
    // is counted, and the loop below gives up after two batches)
    bool has_clock = false;
    for (auto& s : p->stages) has_clock |= s.kind == NEST_STAGE_CLOCK;
    const int chunk = has_clock ? 512 * PIPE_GRAPH_STEPS : PIPE_GRAPH_STEPS;
    auto key = std::make_pair(d_state, st);
    auto it = p->graphs.find(key);
    if (!loop && it == p->graphs.end()) {
        cudaGraph_t g;
        CK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        cudaError_t e = cudaSuccess;
        for (int k = 0; k < PIPE_GRAPH_STEPS && e == cudaSuccess; ++k) e = launch_all(p, d_state, st);
        cudaError_t e2 = cudaStreamEndCapture(st, &g);
        if (e != cudaSuccess) {
            if (e2 == cudaSuccess) cudaGraphDestroy(g);
            return cuda_fail(e, "pipeline capture");
        }
        if (e2 != cudaSuccess) return cuda_fail(e2, "cudaStreamEndCapture");
        cudaGraphExec_t ge;
        cudaError_t e3 = cudaGraphInstantiate(&ge, g, 0);
        cudaGraphDestroy(g);
        if (e3 != cudaSuccess) return cuda_fail(e3, "cudaGraphInstantiate");
        it = p->graphs.emplace(key, ge).first;
    }
    int last = -1;
    for (;;) {
        if (loop) {
            cudaError_t e = launch_loop(p, d_state, chunk, max_steps, start, st);
            if (e != cudaSuccess) { r = cuda_fail(e, "pipeline launch"); break; }
        } else {
            CK(cudaGraphLaunch(it->second, st));
        }
        if ((r = read_pipe_ctrl(p, st)) != NEST_OK) break;
        const PipeCtrl& c = *p->host_ctrl;
        if (!(c.time < t_final) || !c.active) break;
        if (max_steps > 0 && c.step - start >= max_steps) break;
        if (c.step == last) { r = fail(NEST_ERR_NUMERIC, "time stopped advancing"); break; }
        last = c.step;
    }
    // later execute() calls run without a stopping time
    const double zero = 0.0;
    const int one = 1;
    cudaMemcpyAsync(&p->ctrl->t_final, &zero, sizeof zero, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(&p->ctrl->active, &one, sizeof one, cudaMemcpyHostToDevice, st);
    cudaStreamSynchronize(st);
    if (steps_out) *steps_out = p->host_ctrl->step - start;
    return r;
}

nest_status nest_pipeline_clock(nest_pipeline* p, double* time, double* dt, int* step) {
    nest_status r = pcheck(p);
    if (r != NEST_OK) return r;
    if ((r = read_pipe_ctrl(p, p->own)) != NEST_OK) return r;
    if (time) *time = p->host_ctrl->time;
    if (dt) *dt = p->host_ctrl->dt;
    if (step) *step = p->host_ctrl->step;
    return NEST_OK;
}

nest_status nest_pipeline_set_clock(nest_pipeline* p, double time, double dt, int step) {
    nest_status r = pcheck(p);
    if (r != NEST_OK) return r;
    PipeCtrl c{};
    c.time = time; c.dt = dt; c.step = step; c.active = 1;
    CK(cudaMemcpyAsync(p->ctrl, &c, sizeof c, cudaMemcpyHostToDevice, p->own));
    CK(cudaStreamSynchronize(p->own));
    return NEST_OK;
}

nest_status nest_pipeline_buffer(nest_pipeline* p, int index, void** dev) {
    nest_status r = pcheck(p);
    if (r != NEST_OK) return r;
    if (index < 1 || index > p->nwork) return fail(NEST_ERR_INVALID, "work buffer index out of range");
    if (dev) *dev = p->work[index - 1];
    return NEST_OK;
}

}  // extern "C"
