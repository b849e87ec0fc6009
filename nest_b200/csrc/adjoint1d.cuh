// Discrete adjoint of the 1D fused stage, sm_100a, templated on the
// arithmetic type: double (adjoint1d.cu, IEEE arithmetic) and float
// (adjoint1d_f32.cu, fast reciprocal / square root) for the FP32 form.
//
// Forward stage (nest's OpenMP path, examples/benchmark/benchmark_euler1d.cpp:113-165):
//   W_c   = prim(U_c)                          (euler1d.hpp:69-84, p clamped at 0)
//   s_c   = minmod(W_c - W_{c-1}, W_{c+1} - W_c)
//   F_f   = HLLE(W_a + s_a/2, W_b - s_b/2)     (face f between cells a = b-1 and b)
//   U'_i  = U_i - lambda (F_{i+1/2} - F_{i-1/2}),  lambda = dt/dx (dt read from device memory)
// Adjoint (dt frozen), for a given adjoint Ubar' of the stage output:
//   Fbar_f   = lambda (Ubar'_b - Ubar'_a)
//   WLbar_f, WRbar_f = HLLE Jacobians^T Fbar_f   (branch of the forward: S_L >= 0,
//              S_R <= 0 or the HLLE average, with the active argument of each Davis min/max)
//   sbar_c   = WLbar_{c+1/2}/2 - WRbar_{c-1/2}/2
//   Wbar_i   = WRbar_{i-1/2} + WLbar_{i+1/2}
//              + sbar_i ([d1 active] - [d2 active]) + sbar_{i-1} [d2 active at i-1]
//              - sbar_{i+1} [d1 active at i+1]          (minmod subgradient; 0 if d1 d2 <= 0)
//   Ubar_i   = Ubar'_i + (dW/dU)_i^T Wbar_i
// Each lane gathers one cell (no atomics).  Periodic indices wrap modulo n,
// which is exactly the transpose of the periodic ghost fill
// (benchmark_euler1d.cpp:102-110): a ghost cell's adjoint lands on its source.
// A Heun step reverses both stages in one launch (k1d_adjoint_step): a warp owns
// 22 or 54 cells and a halo of five on each side, one or two cells a lane, and
// everything between neighbours goes by shuffles.
#pragma once

#include "common.cuh"
#include "f64div.cuh"
#include "kernels.h"

namespace nestb {
namespace {

constexpr int ADJ_WARPS = 4;  // warps per CTA
// output cells of a warp with CPL cells per lane: all but five at each end
__host__ __device__ constexpr int adj_cells(int cpl) { return 32 * cpl - 10; }

template <typename T>
struct St3 { T r, u, p; };

// What a reversed face divides for: the sound speeds as the forward computes
// them, 1 / (S_R - S_L) and 1 / (2 r c) of each side (not used where c = 0).  FP64
// takes the branch-free forms of f64div.cuh and repeats with the IEEE ones,
// out of line, where a range test fails.
template <typename T> struct FaceDiv { T cL, cR, iD, qL, qR; };

template <typename T>
__device__ __forceinline__ T face_spread(const St3<T>& L, const St3<T>& R, T cL, T cR) {
    return smax(L.u + cL, R.u + cR) - smin(L.u - cL, R.u - cR);
}

template <typename T>
__device__ __forceinline__ FaceDiv<T> face_div_plain(T gamma, St3<T> L, St3<T> R) {
    FaceDiv<T> d;
    d.cL = sqrt(gamma * L.p / L.r);
    d.cR = sqrt(gamma * R.p / R.r);
    d.iD = T(1) / face_spread(L, R, d.cL, d.cR);
    d.qL = T(0.5) / (L.r * d.cL);
    d.qR = T(0.5) / (R.r * d.cR);
    return d;
}
__device__ __noinline__ FaceDiv<double> face_div_ieee(double gamma, St3<double> L, St3<double> R) {
    return face_div_plain(gamma, L, R);
}
__device__ __forceinline__ FaceDiv<float> face_div(float gamma, St3<float> L, St3<float> R) {
    return face_div_plain(gamma, L, R);
}
__device__ __forceinline__ FaceDiv<double> face_div(double gamma, St3<double> L, St3<double> R) {
    ArithFast m;
    FaceDiv<double> d;
    m.pos(L.r); m.pos(L.p); m.pos(R.r); m.pos(R.p);
    d.cL = m.root_quot(gamma * L.p, L.r);
    d.cR = m.root_quot(gamma * R.p, R.r);
    const double spread = face_spread(L, R, d.cL, d.cR);
    m.pos(spread); m.pos(gamma);
    d.iD = m.inverse(spread);
    d.qL = 0.5 * m.inverse(L.r * d.cL);
    d.qR = 0.5 * m.inverse(R.r * d.cR);
    if (m.ok()) return d;
    return face_div_ieee(gamma, L, R);
}

// Primitives of a cell, 1 / rho and whether the pressure clamp is open.  The
// FP64 velocity and pressure are rounded as the forward rounds them (its unit
// does not contract), so every comparison below sees the forward's values.
template <typename T> struct CellAdj { T u, p, ir, act; };

__device__ __forceinline__ CellAdj<float> cell_adj(float gm1, float r, float m, float e) {
    const float u = m / r, praw = gm1 * (e - 0.5f * r * u * u);
    return { u, smax(praw, 0.f), 1.f / r, praw < 0.f ? 0.f : 1.f };
}
__device__ __forceinline__ CellAdj<double> cell_adj_p(double gm1, double r, double u, double ir, double e) {
    const double ke = __dmul_rn(__dmul_rn(__dmul_rn(0.5, r), u), u), praw = __dmul_rn(gm1, __dsub_rn(e, ke));
    return { u, smax(praw, 0.0), ir, praw < 0.0 ? 0.0 : 1.0 };
}
__device__ __noinline__ CellAdj<double> cell_adj_ieee(double gm1, double r, double m, double e) {
    return cell_adj_p(gm1, r, m / r, 1.0 / r, e);
}
__device__ __forceinline__ CellAdj<double> cell_adj(double gm1, double r, double m, double e) {
    ArithFast a;
    const auto ir = a.recip(r);
    const CellAdj<double> c = cell_adj_p(gm1, r, a.quot(m, ir), ir.y, e);
    a.pos(r); a.pos(c.p); a.num(m);
    if (a.ok()) return c;
    return cell_adj_ieee(gm1, r, m, e);
}

// Reverse of hlle1d (common.cuh) for one face: Wbar of the left and right
// face states for the flux adjoint fb.  igm1 = 1 / (gamma - 1).
template <typename T>
__device__ __forceinline__ void hlle1d_adj(T gamma, T igm1, St3<T> L, St3<T> R, const T fb[3], T wl[3], T wr[3]) {
    const FaceDiv<T> dv = face_div(gamma, L, R);
    const T cL = dv.cL, cR = dv.cR;
    T EL = L.p * igm1 + T(0.5) * L.r * L.u * L.u, ER = R.p * igm1 + T(0.5) * R.r * R.u * R.u;
    T aL = L.u - cL, aR = R.u - cR;
    T bL = L.u + cL, bR = R.u + cR;
    T SL = smin(aL, aR), SR = smax(bL, bR);
    bool slR = aR < aL;   // std::min picks the right argument only when it is smaller
    bool srR = bL < bR;   // std::max picks the right argument when the left is smaller
    T FL[3] = { L.r * L.u, L.r * L.u * L.u + L.p, (EL + L.p) * L.u };
    T FR[3] = { R.r * R.u, R.r * R.u * R.u + R.p, (ER + R.p) * R.u };
    T UL[3] = { L.r, L.r * L.u, EL }, UR[3] = { R.r, R.r * R.u, ER };
    T fLb[3] = {0, 0, 0}, fRb[3] = {0, 0, 0}, uLb[3] = {0, 0, 0}, uRb[3] = {0, 0, 0};
    T SLb = T(0), SRb = T(0);
    if (SL >= T(0)) {
        for (int k = 0; k < 3; ++k) fLb[k] = fb[k];
    } else if (SR <= T(0)) {
        for (int k = 0; k < 3; ++k) fRb[k] = fb[k];
    } else {
        // one reciprocal per face: the adjoint needs the derivative, not the
        // forward's rounding
        const T iD = dv.iD;
        for (int k = 0; k < 3; ++k) {
            T dU = UR[k] - UL[k];
            T F = (SR * FL[k] - SL * FR[k] + SL * SR * dU) * iD;
            T g = fb[k] * iD;
            fLb[k] = g * SR;
            fRb[k] = -g * SL;
            uRb[k] = g * SL * SR;
            uLb[k] = -uRb[k];
            SLb += g * (-FR[k] + SR * dU + F);
            SRb += g * (FL[k] + SL * dU - F);
        }
    }
    // Davis speeds -> u and c of the active side
    T uLb_ = T(0), uRb_ = T(0), cLb = T(0), cRb = T(0);
    if (slR) { uRb_ += SLb; cRb -= SLb; } else { uLb_ += SLb; cLb -= SLb; }
    if (srR) { uRb_ += SRb; cRb += SRb; } else { uLb_ += SRb; cLb += SRb; }
    // one side: fluxes, conserved state, energy, sound speed -> (rho, u, p)
    auto side = [&](St3<T> S, T E, T c, T q, const T* fb_, const T* ub_, T ubar, T cbar, T* wo) {
        T rb = T(0), ub = ubar, pb = T(0), Eb = T(0);
        // F0 = r u
        rb += fb_[0] * S.u; ub += fb_[0] * S.r;
        // F1 = (r u) u + p
        rb += fb_[1] * S.u * S.u; ub += fb_[1] * T(2) * S.r * S.u; pb += fb_[1];
        // F2 = (E + p) u
        Eb += fb_[2] * S.u; pb += fb_[2] * S.u; ub += fb_[2] * (E + S.p);
        // U = (r, r u, E)
        rb += ub_[0]; rb += ub_[1] * S.u; ub += ub_[1] * S.r; Eb += ub_[2];
        // E = p / (g-1) + 0.5 r u^2
        pb += Eb * igm1; rb += Eb * T(0.5) * S.u * S.u; ub += Eb * S.r * S.u;
        // c = sqrt(g p / r): dc/dp = g / (2 r c), dc/dr = -c / (2 r)
        if (c > T(0)) {  // q = 1 / (2 r c): dc/dr = -c^2 q
            pb += cbar * gamma * q;
            rb -= cbar * (c * c) * q;
        }
        wo[0] = rb; wo[1] = ub; wo[2] = pb;
    };
    side(L, EL, cL, dv.qL, fLb, uLb, uLb_, cLb, wl);
    side(R, ER, cR, dv.qR, fRb, uRb, uRb_, cRb, wr);
}

// One reverse stage of a warp whose lanes hold CPL neighbouring cells each:
// their conserved values U and output adjoints Lo.  out is the stage's
// Jacobian-transpose term of the cells (the caller adds Lo and any Extra), valid
// three cells inside the valid ones.
template <typename T, int CPL>
__device__ __forceinline__ void rev_stage(const T (&U)[CPL][3], const T (&Lo)[CPL][3], T lambda, T gamma, T gm1,
                                          T igm1, T (&out)[CPL][3]) {
    constexpr unsigned ALL = 0xffffffffu;
    // x of the cell to the right / left of the lane's cell i
    auto right = [&](const T (&x)[CPL], int i) { return i + 1 < CPL ? x[i + 1 < CPL ? i + 1 : 0] : __shfl_down_sync(ALL, x[0], 1); };
    auto left = [&](const T (&x)[CPL], int i) { return i > 0 ? x[i > 0 ? i - 1 : 0] : __shfl_up_sync(ALL, x[CPL - 1], 1); };
    CellAdj<T> q[CPL];
    T P[CPL][3], M[CPL][3], fb[CPL][3];
    int br[CPL];  // minmod branches, two bits a variable: 0 none, 1 d1, 2 d2
#pragma unroll
    for (int i = 0; i < CPL; ++i) {
        q[i] = cell_adj(gm1, U[i][0], U[i][1], U[i][2]);
        br[i] = 0;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        T W[CPL], L[CPL], d[CPL], m[CPL];
#pragma unroll
        for (int i = 0; i < CPL; ++i) {
            W[i] = k == 0 ? U[i][0] : k == 1 ? q[i].u : q[i].p;
            L[i] = Lo[i][k];
        }
#pragma unroll
        for (int i = 0; i < CPL; ++i) d[i] = right(W, i) - W[i];
#pragma unroll
        for (int i = 0; i < CPL; ++i) {
            const T d2 = d[i], d1 = left(d, i);
            T s;
            if (d1 * d2 <= T(0)) s = T(0);
            else if (fabs(d1) < fabs(d2)) { s = d1; br[i] |= 1 << (2 * k); }
            else { s = d2; br[i] |= 2 << (2 * k); }
            P[i][k] = W[i] + T(0.5) * s;
            m[i] = W[i] - T(0.5) * s;
        }
#pragma unroll
        for (int i = 0; i < CPL; ++i) {
            M[i][k] = right(m, i);
            fb[i][k] = lambda * (right(L, i) - L[i]);
        }
    }
    T wl[CPL][3], wr[CPL][3];  // adjoints of the face to the right: of the cell's state, of the next cell's
#pragma unroll
    for (int i = 0; i < CPL; ++i)
        hlle1d_adj(gamma, igm1, St3<T>{ P[i][0], P[i][1], P[i][2] }, St3<T>{ M[i][0], M[i][1], M[i][2] }, fb[i], wl[i],
                   wr[i]);
    T wb[CPL][3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        T r[CPL], v[CPL], t1[CPL], t2[CPL];
#pragma unroll
        for (int i = 0; i < CPL; ++i) r[i] = wr[i][k];
#pragma unroll
        for (int i = 0; i < CPL; ++i) {
            const T wq = left(r, i);                           // the cell's state at the face to its left
            const T sb = T(0.5) * wl[i][k] - T(0.5) * wq;      // its slope adjoint
            const int b = (br[i] >> (2 * k)) & 3;
            t1[i] = b == 1 ? sb : T(0);
            t2[i] = b == 2 ? sb : T(0);
            v[i] = wq + wl[i][k];
            if (b == 1) v[i] += sb;
            else if (b == 2) v[i] -= sb;
        }
#pragma unroll
        for (int i = 0; i < CPL; ++i) wb[i][k] = (v[i] + left(t2, i)) - right(t1, i);
    }
    // (rho, u, p) = prim(rho, m, E): transpose of its Jacobian at the cell
#pragma unroll
    for (int i = 0; i < CPL; ++i) {
        const T u = q[i].u, ir = q[i].ir, act = q[i].act;
        out[i][0] = wb[i][0] - wb[i][1] * u * ir + act * wb[i][2] * gm1 * T(0.5) * u * u;
        out[i][1] = wb[i][1] * ir - act * wb[i][2] * gm1 * u;
        out[i][2] = act * wb[i][2] * gm1;
    }
}

// Output of a reverse stage into the solver layout, with the adjoint's ghost
// cells kept consistent with the periodic wrap.
template <typename T>
__device__ __forceinline__ void put_global(T* Lin, int n, int h, int i, const T v[3]) {
    const int nt = n + 2 * h, e = h + i;
    for (int k = 0; k < 3; ++k) {
        Lin[k * nt + e] = v[k];
        if (i < h) Lin[k * nt + h + n + i] = v[k];
        if (i >= n - h) Lin[k * nt + (i - (n - h))] = v[k];
    }
}

// One reverse Heun step in one launch: tmp = S'(U1)^T lam / 2, then
// lam_new = S'(Un)^T tmp + lam / 2.  The lanes of a warp hold CPL cells each from
// c0 - 5 on; tmp is valid three cells inside them and the result five, the cells
// that the warp writes (the halo's tmp is recomputed by the neighbouring warps,
// bit for bit the same).  Bound: the latency of two reversed stages, and with many
// cells the FP64 pipe.  us of backward per step of a checkpointed sweep, the
// recomputed forward step included (FP64 65536 / 5000 cells, FP32 65536 / 5000):
// 13.1 / 7.3, 8.6 / 5.5, against 15.6 / 10.3, 10.7 / 7.9 with CTAs of 112 cells that
// staged ten phases through shared memory and IEEE divisions.
template <typename T, int CPL>
__global__ void __launch_bounds__(32 * ADJ_WARPS)
k1d_adjoint_step(const T* __restrict__ Un, const T* __restrict__ U1, const T* __restrict__ lam,
                 T* __restrict__ lam_new, int n, int h, const double* dtp, double dx, double gamma_d) {
    const int lane = threadIdx.x & 31;
    const int c = (blockIdx.x * ADJ_WARPS + (threadIdx.x >> 5)) * adj_cells(CPL) - 5 + CPL * lane;
    const int nt = n + 2 * h;
    int e[CPL];
#pragma unroll
    for (int i = 0; i < CPL; ++i) {
        e[i] = (c + i) % n;
        e[i] = (e[i] < 0 ? e[i] + n : e[i]) + h;
    }
    const T gamma = (T)gamma_d, gm1 = (T)(gamma_d - 1.0), igm1 = T(1) / gm1;
    pdl_wait();
    pdl_trigger();
    const T lambda = (T)(*dtp / dx);
    T a[CPL][3], b[CPL][3], lo[CPL][3], j[CPL][3];
#pragma unroll
    for (int i = 0; i < CPL; ++i)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            lo[i][k] = T(0.5) * lam[k * nt + e[i]];
            a[i][k] = U1[k * nt + e[i]];
            b[i][k] = Un[k * nt + e[i]];
        }
    rev_stage<T, CPL>(a, lo, lambda, gamma, gm1, igm1, j);
#pragma unroll
    for (int i = 0; i < CPL; ++i)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            a[i][k] = lo[i][k];  // lam / 2
            lo[i][k] += j[i][k];
        }
    rev_stage<T, CPL>(b, lo, lambda, gamma, gm1, igm1, j);
#pragma unroll
    for (int i = 0; i < CPL; ++i) {
        const int x = CPL * lane + i;
        if (x >= 5 && x < 5 + adj_cells(CPL) && c + i < n) {
            T v[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) v[k] = (lo[i][k] + j[i][k]) + a[i][k];
            put_global(lam_new, n, h, c + i, v);
        }
    }
}

// Cells from which a lane takes two (a longer chain, fewer halo cells): us of
// backward per step, one / two per lane: FP64 50000 cells 11.3 / 13.2, 65536 13.7 /
// 13.7, 200000 28.5 / 27.4; FP32 50000 8.05 / 8.23, 65536 9.33 / 8.61, 200000 16.0 / 15.0.
template <typename T> constexpr int ADJ_TWO_CELLS = sizeof(T) == 8 ? 100000 : 60000;

template <typename T>
cudaError_t launch_1d_adjoint_step_t(const T* Un, const T* U1, const T* lam, T* lam_new, int n, int h,
                                     const double* dtp, double dx, double gamma, cudaStream_t st) {
    const bool two = n >= ADJ_TWO_CELLS<T>;
    const int cells = adj_cells(two ? 2 : 1) * ADJ_WARPS, blocks = (n + cells - 1) / cells;
    return launch_pdl(two ? k1d_adjoint_step<T, 2> : k1d_adjoint_step<T, 1>, dim3(blocks), dim3(32 * ADJ_WARPS), 0, st,
                      Un, U1, lam, lam_new, n, h, dtp, dx, gamma);
}

}  // namespace
}  // namespace nestb
