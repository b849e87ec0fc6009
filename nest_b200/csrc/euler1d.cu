// 1D Euler hot path for sm_100a: fused PLM-minmod + HLLE + flux divergence +
// RK2 stage, on-device ghost fill and CFL max-speed reduction.
//
// Compiled with -fmad=false: the FP64 arithmetic keeps the operation order
// of nest's OpenMP path (examples/benchmark/benchmark_euler1d.cpp:113-209)
// and matches it bit for bit.
//
// Two execution shapes:
//   * resident (k1d_loop): one CTA, or a thread-block cluster of 16 (8), holds
//     the whole domain on chip and runs the complete time loop (dt, ghost fill,
//     both stages, Heun average) with no kernel boundary and no host round-trip
//     per step, up to 4080 cells.  Where no cluster can be placed, one CTA with
//     several cells per thread (k1d_resident) takes up to about 2300.
//   * tiled (euler1d_tiled.cuh): a whole step per launch, a warp per 24 or 56 cells
//     (the stage-1 halo recomputed per warp), or the two stage kernels; stage
//     2 fuses the Heun average, the ghost fill of the new state and the
//     max-wave-speed reduction; dt is derived on the device from that
//     maximum, so steps need no host synchronisation (they are captured in
//     CUDA graphs by the host code).
#include <cooperative_groups.h>

#include <map>
#include <mutex>

#include "euler1d_arith.cuh"
#include "kernels.h"

namespace nestb {

// ---------------------------------------------------------------------------
// Resident single-CTA solver
// ---------------------------------------------------------------------------

__device__ __forceinline__ int ghost_src_1d(int e, int n, int h, int bc) {
    // extended index e of a ghost cell -> extended index of its source
    if (e < h) return bc == BC_PERIODIC ? n + e : h;
    return bc == BC_PERIODIC ? e - n : h + n - 1;
}

// Ghost copies fed by interior cell c (0-based) of a 3-variable SoA array
// over the extended range: nest's periodic copy or the zero-gradient copy.
__device__ __forceinline__ void ghost_copies_1d(double* A, int nt, int n, int h, int bc, int c, double v0, double v1,
                                                double v2) {
    auto put = [&](int e) { A[e] = v0; A[nt + e] = v1; A[2 * nt + e] = v2; };
    if (bc == BC_PERIODIC) {
        if (c >= n - h) put(c + h - n);
        if (c < h) put(h + n + c);
    } else {
        if (c == 0) for (int e = 0; e < h; ++e) put(e);
        if (c == n - 1) for (int e = h + n; e < nt; ++e) put(e);
    }
}

// Resident single-CTA solver for devices that cannot place a cluster (more
// cells than k1d_loop's one CTA takes): the whole extended domain lives in shared
// memory (U, U1, primitives W, face fluxes F) and the CTA runs the complete
// time loop.  A step is four phases separated by four barriers:
//   faces of stage 1 (PLM + HLLE from W)        | update U1, its primitives and ghost copies |
//   faces of stage 2 (from the primitives of U1) | Heun update of U, its primitives, ghost copies and max |u|+c
// Each thread handles K faces / cells per phase (K >= 2: independent
// chains of FP64 division / square root interleave).  The arithmetic of
// every face and cell is that of nest's OpenMP loop
// (examples/benchmark/benchmark_euler1d.cpp:113-209); primitives of a ghost
// cell are the primitives of its source cell, which is what nest computes
// from the copied conserved values.
// LIM (both resident kernels): the slope limiter fixed at compile time
// (LIM_MINMOD, nest's default) or -1 to read it from the loop parameters.
template <int K, int MAXT, int LIM>
__global__ void __launch_bounds__(MAXT)
k1d_resident(double* __restrict__ Ug, int n, int h, double dx, double gamma, int bc, LoopParams lp, StepCtrl* ctrl,
             int p) {
    extern __shared__ double sm[];
    const int nt = n + 2 * h, T = blockDim.x, tid = threadIdx.x;
    double* U = sm;
    double* U1 = U + 3 * nt;
    double* W = U1 + 3 * nt;
    double* F = W + 3 * nt;
    double* red = F + 3 * (n + 1);
    const double gm1 = gamma - 1.0;
    const int nw = (T + 31) >> 5;

    // primitives of cell value (r, m, e): u, p (cons_to_prim, euler1d.hpp:69-84)
    auto prims_of = [&](int c, double r, double m, double e, double* Wd) {
        const double u = m / r;
        const double pr = eos_pressure(gm1, r, m, e);
        const int x = h + c;
        Wd[x] = r; Wd[nt + x] = u; Wd[2 * nt + x] = pr;
        ghost_copies_1d(Wd, nt, n, h, bc, c, r, u, pr);
    };
    // max |u| + c over this thread's cells of A (benchmark_euler1d.cpp:168-180), warp maxima to red.
    // step_done > 0: the state after that step, checked for positivity; a
    // failing cell makes the maximum infinite, which ends the loop for the CTA
    auto speeds = [&](int step_done) {
        double ms = 0.0;
#pragma unroll
        for (int q = 0; q < K; ++q) {
            const int c = tid + q * T;
            if (c < n) {
                const int x = h + c;
                const double u = W[nt + x], pr = W[2 * nt + x], r = W[x];
                const double cs = sqrt(gamma * pr / r);
                ms = smax(ms, fabs(u) + cs);
                if (step_done > 0 && (!(r > 0.0) || !(pr > 0.0))) {
                    flag_cell(ctrl, step_done, r, pr, c, 0);
                    ms = __longlong_as_double(0x7ff0000000000000ll);
                }
            }
        }
        ms = warp_max(ms);
        if ((tid & 31) == 0) red[tid >> 5] = ms;
    };
    auto reduce_red = [&]() {
        double ms = 0.0;
        for (int w = 0; w < nw; ++w) ms = smax(ms, red[w]);
        return ms;
    };
    // face fluxes of the stage whose primitives are in W
    auto faces = [&]() {
#pragma unroll
        for (int q = 0; q < K; ++q) {
            const int f = tid + q * T;
            if (f <= n) {
                // face between extended cells a = h+f-1 and b = h+f
                const int a = h + f - 1, b = h + f;
                double sa[3], sb[3];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const double* w = W + k * nt;
                    sa[k] = limit(w[a] - w[a - 1], w[b] - w[a], LIM >= 0 ? LIM : lp.lim);
                    sb[k] = limit(w[b] - w[a], w[b + 1] - w[b], LIM >= 0 ? LIM : lp.lim);
                }
                const double rL = W[a] + 0.5 * sa[0], uL = W[nt + a] + 0.5 * sa[1], pL = W[2 * nt + a] + 0.5 * sa[2];
                const double rR = W[b] - 0.5 * sb[0], uR = W[nt + b] - 0.5 * sb[1], pR = W[2 * nt + b] - 0.5 * sb[2];
                double f0, f1, f2;
                hlle1d(gamma, gm1, rL, uL, pL, rR, uR, pR, f0, f1, f2);
                F[f] = f0; F[(n + 1) + f] = f1; F[2 * (n + 1) + f] = f2;
            }
        }
    };
    // stage update of this thread's cells: out = in - dtdx (F_{c+1} - F_c),
    // or U = 0.5 (U + that) in stage 2; then the new state's primitives and ghosts
    auto update = [&](const double* Uin, double* Uout, bool heun, double dtdx) {
#pragma unroll
        for (int q = 0; q < K; ++q) {
            const int c = tid + q * T;
            if (c < n) {
                const int x = h + c;
                double v[3];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    v[k] = Uin[k * nt + x] - dtdx * (F[k * (n + 1) + c + 1] - F[k * (n + 1) + c]);
                    if (heun) v[k] = 0.5 * (Uout[k * nt + x] + v[k]);
                    Uout[k * nt + x] = v[k];
                }
                ghost_copies_1d(Uout, nt, n, h, bc, c, v[0], v[1], v[2]);
                prims_of(c, v[0], v[1], v[2], W);
            }
        }
    };

    // prologue: state, ghosts, primitives and the first max wave speed
    for (int i = tid; i < 3 * nt; i += T) { U[i] = Ug[i]; U1[i] = 0.0; }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < K; ++q) {
        const int c = tid + q * T;
        if (c < n) {
            const int x = h + c;
            const double r = U[x], m = U[nt + x], e = U[2 * nt + x];
            ghost_copies_1d(U, nt, n, h, bc, c, r, m, e);
            prims_of(c, r, m, e, W);
        }
    }
    __syncthreads();
    speeds(0);
    __syncthreads();
    double ms = reduce_red();

    double time = ctrl->time[p];
    int step = ctrl->step[p];
    const bool stopped = (ctrl->err & ERRW_STOP) != 0;  // an earlier step failed: run nothing
    for (int it = 0;; ++it) {
        if (stopped) break;
        if (lp.step_budget > 0 && it >= lp.step_budget) break;
        if (lp.t_final > 0.0 && !(time < lp.t_final)) break;
        if (lp.max_steps > 0 && step >= lp.max_steps) break;
        if (lp.dts_in && step >= lp.dts_cap) break;
        double dt;
        if (lp.fixed_dt > 0.0) {
            dt = lp.fixed_dt;
        } else if (lp.dts_in) {
            dt = lp.dts_in[step];
        } else {
            dt = lp.cfl * dx / ms;
            if (lp.t_final > 0.0) dt = smin(dt, lp.t_final - time);
        }
        if (!(ms == ms) || ms > 1.79e308) { if (tid == 0) atomicOr(&ctrl->err, ERRW_NONFINITE); break; }
        if (tid == 0 && lp.dts_out && step < lp.dts_cap) lp.dts_out[step] = dt;
        const double dtdx = dt / dx;
        faces();                        // stage 1 fluxes from W = prims(U)
        __syncthreads();
        update(U, U1, false, dtdx);     // U1, W = prims(U1), ghosts
        __syncthreads();
        faces();                        // stage 2 fluxes
        __syncthreads();
        update(U1, U, true, dtdx);      // U = (U + U1 - dt L(U1)) / 2, W = prims(U), ghosts
        speeds(step + 1);
        __syncthreads();
        ms = reduce_red();
        time += dt;
        ++step;
    }
    for (int i = tid; i < 3 * nt; i += T) Ug[i] = U[i];
    if (tid == 0) {
        ctrl->time[p] = time; ctrl->step[p] = step;
        ctrl->time[p ^ 1] = time; ctrl->step[p ^ 1] = step;
    }
}

// Point-to-point messages between the CTAs of a cluster: a store into another
// CTA's shared memory that counts its bytes on an mbarrier there (st.async), so a
// receiver waits for its data alone and a sender for nothing.
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned peer_addr(unsigned a, int rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void send_f64(unsigned dst, double v, unsigned bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];"
                 ::"r"(dst), "l"(__double_as_longlong(v)), "r"(bar) : "memory");
}
__device__ __forceinline__ void bar_init(unsigned bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
// The one arrival of a phase, which then completes with its last byte.
__device__ __forceinline__ void bar_expect(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Waits for the phase of that parity; false where it has not come after `polls` looks.
__device__ __forceinline__ bool bar_wait(unsigned bar, unsigned parity, int polls) {
    for (int k = 0; k < polls; ++k) {
        unsigned done;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}

// Largest chunk of the resident loop: cells per CTA (9 warps of 31 cells).
constexpr int LOOP_WARPS = 9, LOOP_CELLS = 31 * LOOP_WARPS;

// The resident time loop: the NC CTAs of a thread-block cluster (one per SM), or
// one CTA, split the cells into contiguous chunks (of m at most) and run the
// complete loop.  One thread owns one cell: its U and U1 stay in registers, and
// only the primitives go through shared memory.  Lane k of a warp computes the
// face to the right of its cell, and takes the left face (k >= 1) from the lane
// below, so a warp computes 32 faces for 31 cells and a stage needs no barrier
// between its fluxes and its update.
// In a cluster a step has one exchange: at its end the threads of a chunk's first
// and last four cells send their new state to the neighbouring CTAs, which
// compute U1 of the two nearest cells themselves, and every warp sends its
// wave-speed maximum to every CTA, so dt comes from local shared memory while
// the stage-1 fluxes (which do not need it) are computed.
// What bounds it is one thread's chain of dependent FP64 operations (two face
// chains and two cell chains a step) and, in a cluster, the exchange.
// Sod tube, us per step (with IEEE divisions and square roots, state in shared
// memory and a barrier between fluxes and update): 100 cells 1.40 (5.87), 200 cells
// 1.82 (6.47), both one CTA; 1024 cells on 16 CTAs 2.01 (4.67), 4080 cells 2.94 (5.68).
// Two cluster barriers a step instead (about 0.45 us each): 2.46 and 3.40; messages
// for both stages 2.20 and 3.04; registers for two blocks an SM (96, spills) 2.13, 2.99.
// LIM: the slope limiter fixed at compile time (LIM_MINMOD, nest's default) or
// -1 to read it from the loop parameters.  SHORT: waits give up after lp.short_waits - 1
// looks, to test the way out of them (a limit read from the parameters costs the loop
// 1.5 %, so the instance that runs otherwise has its own).
constexpr int WAIT_POLLS = 1 << 24;  // a quarter of a second and more, which no message takes
template <bool CLUSTER, int LIM, bool SHORT = false>
__global__ void __launch_bounds__(32 * LOOP_WARPS, 1)
k1d_loop(double* __restrict__ Ug, int n, int h, int m, double dx, double gamma, int bc, LoopParams lp,
         StepCtrl* ctrl, int p) {
    namespace cg = cooperative_groups;
    extern __shared__ double sm[];
    const int NC = CLUSTER ? (int)cg::this_cluster().num_blocks() : 1;
    const int r = CLUSTER ? (int)cg::this_cluster().block_rank() : 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int nt = n + 2 * h;
    // this CTA's cells [c_lo, c_lo + mloc)
    const int mloc = n / NC + (r < n % NC ? 1 : 0), c_lo = r * (n / NC) + min(r, n % NC);
    constexpr int H = CLUSTER ? 4 : 2, X = CLUSTER ? 2 : 0;   // halo slots, recomputed cells on each side
    const int mw = m + 2 * H;
    double* const W = sm;             // [3][3][mw]: state of even / odd steps and U1, variable k, local cell l at H + l
    double* const Uh = W + 9 * mw;    // [2][4][2]: momentum and energy of the recomputed cells, by step
    double* const red = Uh + 16;      // [2][NC * nw]: wave-speed maxima of every warp, by step
    const Gas<double, ArithChain> gas(gamma);
    const int left = (r + NC - 1) % NC, right = (r + 1) % NC;
    const int mloc_left = n / NC + (left < n % NC ? 1 : 0);
    const bool per = bc == BC_PERIODIC;
    const bool has_left = CLUSTER && (per || r > 0), has_right = CLUSTER && (per || r < NC - 1);

    const int l = 31 * warp + lane - 1 - X;           // this lane's face is to the right of local cell l
    const bool own = lane >= 1 && l >= 0 && l < mloc; // and it owns cell l,
    const bool ext = lane >= 1 && ((has_left && l < 0) || (has_right && l >= mloc && l < mloc + X));  // or repeats its U1
    const int c = c_lo + l;
    // lanes past the faces that a stage needs repeat the last one
    const int ls1 = min(max(l, has_left ? -1 - X : -1), mloc - 1 + (has_right ? X : 0)), ls2 = min(max(l, -1), mloc - 1);
    const bool edge = CLUSTER && (warp == 0 || 31 * warp + 30 - X >= mloc - 2);  // reads halo slots

    // Message q (0 before the loop, it + 1 at the end of step it) is the halo of the state
    // and the maxima, with buffers and barriers by q & 1.  Thread 0 announces the bytes of
    // q + 2 when q has arrived: they cannot be sent before its own warp's maximum
    // q + 1, which it sends later.  For the same reason nothing of q is overwritten by
    // q + 2 before every warp here has read it.
    __shared__ unsigned long long bars[4];
    __shared__ volatile unsigned lost;        // a wait gave up
    const unsigned bar0 = smem_addr(bars);
    auto bar_halo = [&](int q) { return bar0 + 8 * (q & 1); };
    auto bar_max = [&](int q) { return bar0 + 16 + 8 * (q & 1); };
    const unsigned halo_bytes = 128u * ((has_left ? 1 : 0) + (has_right ? 1 : 0)), max_bytes = 8u * NC * nw;
    auto announce = [&](int q) { bar_expect(bar_halo(q), halo_bytes); bar_expect(bar_max(q), max_bytes); };

    // stores the primitives of the lane's cell into buffer b, with the ghosts they feed
    auto put = [&](int b, double v0, double v1, double v2) {
        double* const w = W + b * 3 * mw + H;
        auto to = [&](int x) { w[x] = v0; w[mw + x] = v1; w[2 * mw + x] = v2; };
        to(l);
        if (!per) {
            if (c == 0) { to(-1); to(-2); }
            if (c == n - 1) { to(mloc); to(mloc + 1); }
        } else if (!CLUSTER) {
            if (l < 2) to(mloc + l);
            if (l >= mloc - 2) to(l - mloc);
        }
    };
    // sends the own cell, four from an end of the chunk or less, to the neighbour there
    auto send_halo = [&](int q, double v0, double v1, double v2, double m1, double e2) {
        auto send = [&](int rank, int x, int xu) {
            const unsigned bar = peer_addr(bar_halo(q), rank);
            const unsigned a = peer_addr(smem_addr(W + (q & 1) * 3 * mw + H + x), rank);
            send_f64(a, v0, bar); send_f64(a + 8 * mw, v1, bar); send_f64(a + 16 * mw, v2, bar);
            if (xu >= 0) {
                const unsigned u = peer_addr(smem_addr(Uh + (q & 1) * 8 + 2 * xu), rank);
                send_f64(u, m1, bar); send_f64(u + 8, e2, bar);
            }
        };
        if (l < 4 && has_left) send(left, mloc_left + l, l < 2 ? 2 + l : -1);
        if (l >= mloc - 4 && has_right) send(right, l - mloc, l >= mloc - 2 ? l - (mloc - 2) : -1);
    };
    auto faces = [&](int b, int ls) {
        const double* w = W + b * 3 * mw + H + ls - 1;
        return plm_flux(gas, LIM >= 0 ? LIM : lp.lim, [&](int k, int s) { return w[k * mw + s]; }, 0, 1, 2, 3);
    };
    auto send_max = [&](double s, int q) {
        s = warp_max_speed(s);
        double* const d = red + (CLUSTER ? (q & 1) * NC * nw : 0) + r * nw + warp;
        if (CLUSTER) {
            if (lane < NC) send_f64(peer_addr(smem_addr(d), lane), s, peer_addr(bar_max(q), lane));
        } else if (lane == 0) {
            *d = s;
        }
    };
    auto read_max = [&](int q) {
        const double* const d = red + (CLUSTER ? (q & 1) * NC * nw : 0);
        double s = 0.0;
        for (int k = lane; k < NC * nw; k += 32) s = smax(s, d[k]);
        return warp_max_speed(s);
    };
    double u0 = 1.0, u1 = 0.0, u2 = 1.0;
    // waits for message q and takes the state of a recomputed cell from it.  (Waiting for the
    // maxima after the stage-1 fluxes took dt's division out of their shadow: 2.13 -> 2.25
    // us a step at 1024 cells.)
    auto receive = [&](int q) {
        if (!CLUSTER) return;
        const unsigned parity = (q >> 1) & 1;
        const int polls = SHORT ? lp.short_waits - 1 : WAIT_POLLS;
        const bool ok = (!edge || bar_wait(bar_halo(q), parity, polls)) && bar_wait(bar_max(q), parity, polls);
        if (!ok) {
            lost = 1u;
            if (lane == 0) atomicOr(&ctrl->err, ERRW_LOST);
        } else if (threadIdx.x == 0) {
            announce(q + 2);
        }
        if (ext) {
            const double* const u = Uh + (q & 1) * 8 + 2 * (l < 0 ? l + 2 : 2 + l - mloc);
            u0 = W[(q & 1) * 3 * mw + H + l]; u1 = u[0]; u2 = u[1];
        }
    };

    // prologue: the own cell, its primitives and the first wave speeds
    if (own) { u0 = Ug[h + c]; u1 = Ug[nt + h + c]; u2 = Ug[2 * nt + h + c]; }
    if (CLUSTER) {
        if (threadIdx.x == 0) {
            for (int k = 0; k < 4; ++k) bar_init(bar0 + 8 * k);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            announce(0);
            announce(1);
            lost = 0u;
        }
        cg::this_cluster().sync();  // every CTA of the cluster runs, its barriers announced
    }
    double time = ctrl->time[p];
    int step = ctrl->step[p];
    // an earlier step failed: run nothing.  (Read before the first maximum is sent, which
    // depends on it: other CTAs may flag a cell once they have that.)
    const bool stopped = (*reinterpret_cast<volatile unsigned*>(&ctrl->err) & ERRW_STOP) != 0;
    {
        const Cell1<double> w = cell1d<true>(gas, u0, u1, u2);
        if (own) {
            put(0, u0, w.u, w.p);
            if (CLUSTER) send_halo(0, u0, w.u, w.p, u1, u2);
        }
        send_max(own && !stopped ? smax(0.0, fabs(w.u) + w.cs) : 0.0, 0);
    }
    __syncthreads();
    receive(0);

    for (int it = 0;; ++it) {
        if (stopped) break;
        if (lp.step_budget > 0 && it >= lp.step_budget) break;
        if (lp.t_final > 0.0 && !(time < lp.t_final)) break;
        if (lp.max_steps > 0 && step >= lp.max_steps) break;
        if (lp.dts_in && step >= lp.dts_cap) break;
        const double ms = read_max(it);
        const F3<double> f = faces(CLUSTER ? it & 1 : 0, ls1);
        double dt;
        if (lp.fixed_dt > 0.0) {
            dt = lp.fixed_dt;
        } else if (lp.dts_in) {
            dt = lp.dts_in[step];
        } else {
            dt = div_rn(lp.cfl * dx, ms);
            if (lp.t_final > 0.0) dt = smin(dt, lp.t_final - time);
        }
        const bool bad = !(ms == ms) || ms > 1.79e308;
        if (!CLUSTER && bad) { if (threadIdx.x == 0) atomicOr(&ctrl->err, ERRW_NONFINITE); break; }
        if (r == 0 && threadIdx.x == 0 && lp.dts_out && step < lp.dts_cap && !bad) lp.dts_out[step] = dt;
        const double dtdx = div_rn(dt, dx);
        // stage 1: U1 = U - dtdx (F_right - F_left)
        const double v0 = u0 - dtdx * (f.a - __shfl_up_sync(0xffffffffu, f.a, 1));
        const double v1 = u1 - dtdx * (f.b - __shfl_up_sync(0xffffffffu, f.b, 1));
        const double v2 = u2 - dtdx * (f.c - __shfl_up_sync(0xffffffffu, f.c, 1));
        {
            const Cell1<double> w = cell1d<false>(gas, v0, v1, v2);
            if (own || ext) put(2, v0, w.u, w.p);
        }
        __syncthreads();
        if (CLUSTER) {
            // (the same in all threads: lost was written before the barrier, and unless it
            // was, all of them have the same maximum)
            if (lost) break;
            if (bad) { if (r == 0 && threadIdx.x == 0) atomicOr(&ctrl->err, ERRW_NONFINITE); break; }
        }
        // stage 2: U = (U + U1 - dtdx (F_right - F_left)) / 2, its wave speed
        // and positivity (a failing cell makes the maximum infinite, which
        // ends the loop on every CTA)
        const F3<double> e = faces(2, ls2);
        u0 = 0.5 * (u0 + (v0 - dtdx * (e.a - __shfl_up_sync(0xffffffffu, e.a, 1))));
        u1 = 0.5 * (u1 + (v1 - dtdx * (e.b - __shfl_up_sync(0xffffffffu, e.b, 1))));
        u2 = 0.5 * (u2 + (v2 - dtdx * (e.c - __shfl_up_sync(0xffffffffu, e.c, 1))));
        {
            const Cell1<double> w = cell1d<true>(gas, u0, u1, u2);
            double s = 0.0;
            if (own) {
                put(CLUSTER ? (it + 1) & 1 : 0, u0, w.u, w.p);
                if (CLUSTER) send_halo(it + 1, u0, w.u, w.p, u1, u2);
                s = smax(0.0, fabs(w.u) + w.cs);
                if (!(u0 > 0.0) || !(w.p > 0.0)) {
                    flag_cell(ctrl, step + 1, u0, w.p, c, 0);
                    s = __longlong_as_double(0x7ff0000000000000ll);
                }
            }
            send_max(s, it + 1);
        }
        __syncthreads();
        receive(it + 1);
        time += dt;
        ++step;
    }
    // state and the domain's ghost cells back to global memory
    if (own) {
        const double v[3] = { u0, u1, u2 };
        for (int k = 0; k < 3; ++k) {
            Ug[k * nt + h + c] = v[k];
            if (bc == BC_PERIODIC) {
                if (c >= n - h) Ug[k * nt + c + h - n] = v[k];
                if (c < h) Ug[k * nt + h + n + c] = v[k];
            } else {
                if (c == 0) for (int g = 0; g < h; ++g) Ug[k * nt + g] = v[k];
                if (c == n - 1) for (int g = h + n; g < nt; ++g) Ug[k * nt + g] = v[k];
            }
        }
    }
    if (r == 0 && threadIdx.x == 0) {
        ctrl->time[p] = time; ctrl->step[p] = step;
        ctrl->time[p ^ 1] = time; ctrl->step[p ^ 1] = step;
    }
    if (CLUSTER) {
        // No CTA leaves while stores to it may be in flight.  All that were sent have been
        // waited for, unless a wait gave up.  A store then was sent before its receiver gave
        // up, which gives it 0.1 ms, or by a CTA that finds the news here and gives its own.
        if (threadIdx.x == 0 && (lost || (*reinterpret_cast<volatile unsigned*>(&ctrl->err) & ERRW_LOST)))
            for (int k = 0; k < 100; ++k) __nanosleep(1000);
        cg::this_cluster().sync();
    }
}

size_t resident_smem_bytes(int n, int h) {
    int nt = n + 2 * h;
    return sizeof(double) * (size_t)(9 * nt + 3 * (n + 1) + 33);
}

// Launch of the resident loop with a cluster of NC CTAs (1: a plain launch).
struct LoopShape {
    int m, threads;
    size_t smem;
};
// Chunk and block size for n cells on NC CTAs; false where they do not fit
// (every CTA of a cluster needs four cells for its neighbours' halos).
static bool loop_shape(int n, int NC, LoopShape& s) {
    s.m = (n + NC - 1) / NC;
    const int lanes = s.m + (NC > 1 ? 4 : 0);
    if (lanes > LOOP_CELLS || (NC > 1 && n / NC < 4)) return false;
    s.threads = (lanes + 30) / 31 * 32;
    s.smem = sizeof(double) * (size_t)(9 * (s.m + 8) + 16 + 2 * NC * (s.threads / 32));
    return true;
}

template <class K>
static cudaError_t cluster_config(K kern, int NC, const LoopShape& s, cudaLaunchConfig_t& cfg,
                                  cudaLaunchAttribute* at, int& clusters) {
    cudaError_t e;
    clusters = 0;
    if (NC > 8 && (e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)) != cudaSuccess)
        return e;
    cfg = {};
    cfg.gridDim = dim3(NC, 1, 1);
    cfg.blockDim = dim3(s.threads, 1, 1);
    cfg.dynamicSmemBytes = s.smem;
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = NC;
    at->val.clusterDim.y = 1;
    at->val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if ((e = cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg)) != cudaSuccess) {
        cudaGetLastError();
        clusters = 0;
    }
    return cudaSuccess;
}

// Returns cudaErrorNotSupported (nothing launched) when the chunk sizes or the
// device's cluster occupancy do not allow that cluster size.
static cudaError_t launch_1d_cluster(double* U, int n, int h, double dx, double gamma, int bc, const LoopParams& lp,
                                     StepCtrl* ctrl, int p, cudaStream_t st, int NC) {
    LoopShape s;
    if (!loop_shape(n, NC, s)) return cudaErrorNotSupported;
    auto kern = lp.short_waits > 0 ? k1d_loop<true, -1, true>
                : lp.lim == LIM_MINMOD ? k1d_loop<true, LIM_MINMOD> : k1d_loop<true, -1>;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at;
    int clusters;
    cudaError_t e = cluster_config(kern, NC, s, cfg, &at, clusters);
    if (e != cudaSuccess) return e;
    if (clusters < 1) return cudaErrorNotSupported;
    cfg.stream = st;
    return cudaLaunchKernelEx(&cfg, kern, U, n, h, s.m, dx, gamma, bc, lp, ctrl, p);
}

// Whether launch_1d_cluster can place a cluster of 16 or 8 CTAs for n cells
// on the current device (the chunk-size rules and the cluster occupancy query
// of launch_1d_cluster, with nothing launched); remembered per device and n.
bool cluster_1d_available(int n, int h) {
    if (n < 256 || n > 4080) return false;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    static std::mutex mu;
    static std::map<std::pair<int, int>, bool> known;
    std::lock_guard<std::mutex> lk(mu);
    auto it = known.find({dev, n});
    if (it != known.end()) return it->second;
    bool ok = false;
    for (int NC : {16, 8}) {
        LoopShape s;
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at;
        int clusters = 0;
        if (!loop_shape(n, NC, s)) continue;
        // both limiter instances use the same threads and shared memory; the
        // minmod one stands for both
        if (cluster_config(k1d_loop<true, LIM_MINMOD>, NC, s, cfg, &at, clusters) != cudaSuccess) {
            cudaGetLastError();
            continue;
        }
        if (clusters >= 1) { ok = true; break; }
    }
    known[{dev, n}] = ok;
    return ok;
}

cudaError_t launch_1d_resident(double* U, int n, int h, double dx, double gamma, int bc,
                               const LoopParams& lp, StepCtrl* ctrl, int p, cudaStream_t st) {
    const bool mm = lp.lim == LIM_MINMOD;
    // fewer than 256 cells: one CTA, whose barrier is cheap (us a step on one CTA / a
    // cluster: 200 cells 1.83 / 2.16, 248 1.84 / 2.17, 256 2.28 / 2.03)
    if (n < 256) {
        LoopShape s;
        loop_shape(n, 1, s);
        (mm ? k1d_loop<false, LIM_MINMOD> : k1d_loop<false, -1>)<<<1, s.threads, s.smem, st>>>(U, n, h, s.m, dx, gamma,
                                                                                         bc, lp, ctrl, p);
        return cudaGetLastError();
    }
    // a cluster of 16 (else 8) CTAs, one per SM
    for (int NC : {16, 8}) {
        cudaError_t e = launch_1d_cluster(U, n, h, dx, gamma, bc, lp, ctrl, p, st, NC);
        if (e != cudaErrorNotSupported) return e;
    }
    size_t smem = resident_smem_bytes(n, h);
    // K faces per thread: at least two (independent FP64 chains per thread),
    // more when n + 1 faces exceed 2 * 1024
    const int K = (n + 1 <= 2048) ? 2 : 3;
    if (n + 1 > 3 * 1024) return cudaErrorInvalidValue;
    int threads = ((n + 1 + K - 1) / K + 31) / 32 * 32;
    cudaError_t e;
    // the thread bound sets the register budget: 640 threads (n < 1280, up to
    // 102 registers) or 1024 (64 registers)
    auto go = [&](auto kern) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess) kern<<<1, threads, smem, st>>>(U, n, h, dx, gamma, bc, lp, ctrl, p);
    };
    if (K == 2 && threads <= 640) mm ? go(k1d_resident<2, 640, LIM_MINMOD>) : go(k1d_resident<2, 640, -1>);
    else if (K == 2) mm ? go(k1d_resident<2, 1024, LIM_MINMOD>) : go(k1d_resident<2, 1024, -1>);
    else mm ? go(k1d_resident<3, 1024, LIM_MINMOD>) : go(k1d_resident<3, 1024, -1>);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

}  // namespace nestb

// Tiled multi-CTA stage kernels (FP64 instantiation; euler1d_f32.cu holds the
// FP32 one).
#include "euler1d_tiled.cuh"

namespace nestb {

cudaError_t launch_1d_prepare(double* U, int n, int h, double gamma, int bc, StepCtrl* ctrl, int p,
                              cudaStream_t st) {
    return launch_1d_prepare_t<double>(U, n, h, gamma, bc, ctrl, p, st);
}

cudaError_t launch_1d_step(double* U, double* U1, int n, int h, double dx, double gamma, int bc,
                           const LoopParams& lp, StepCtrl* ctrl, int p, int which, cudaStream_t st, double* Uout) {
    return launch_1d_step_t<double>(U, U1, n, h, dx, gamma, bc, lp, ctrl, p, which, st, Uout);
}

cudaError_t launch_1d_fused(const double* Un, double* Unext, double* U1out, int n, int h, double dx, double gamma,
                            int bc, const LoopParams& lp, StepCtrl* ctrl, int p, cudaStream_t st) {
    return launch_1d_fused_t<double>(Un, Unext, U1out, n, h, dx, gamma, bc, lp, ctrl, p, st);
}

}  // namespace nestb
