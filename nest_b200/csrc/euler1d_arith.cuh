// 1D cell and face arithmetic of the FP64 plain form with the branch-free
// division and square root of f64div.cuh (hlle1d, eos_pressure and the sound
// speed of common.cuh: the same expressions in the same order, so the same
// values), and the FP32 form's under the same names.
//
// The 1D kernels are bound by the latency of one thread's chain, and a face has
// ten divisions and square roots.  With nvcc's IEEE forms each of them is a
// branch that the next has to wait for; here they interleave, and a value whose
// range tests fail (rare) is computed again, out of line, with the IEEE ones.
// In the resident loop the square root's approximation runs beside the quotient it
// is taken of (ArithChain), and the pressure takes neither clamp nor halving on its chain (Sod's tube, with the
// host's copies: 100 cells to t = 0.1 169 -> 163 us, 1024 cells to 0.2 2880 -> 2800).
#pragma once

#include "common.cuh"
#include "f64div.cuh"

namespace nestb {
namespace {

template <typename T> struct F3 { T a, b, c; };

// Constants of a launch: gamma, gamma - 1 and, for FP64, its reciprocal (in
// range: else `fast` is false and everything takes the IEEE forms).
// A: the branch-free policy that FP64 takes.
template <typename T, class A = ArithFast> struct Gas {
    T gamma, gm1;
    __device__ __forceinline__ explicit Gas(double g) : gamma((T)g), gm1((T)(g - 1.0)) {}
};
template <class A> struct Gas<double, A> {
    double gamma, gm1;
    ArithFast::Recip ig;
    bool fast;
    __device__ __forceinline__ explicit Gas(double g)
        : gamma(g), gm1(g - 1.0), ig{ g - 1.0, recip_f64(g - 1.0) }, fast(g < 1024.0 && g - 1.0 > 0x1p-20) {}
};

// hlle_flux, euler1d.hpp:178-242.  Tested: rho and p of both sides (2^-128 to
// 2^128), dS = SR - SL in the same range, which bounds the velocities where the
// average is taken, and the mass and energy flux numerators from below (the
// momentum one holds SR p - SL p).
template <class A>
__device__ __forceinline__ F3<double> hlle1d_fast(A& m, double gamma, const typename A::Recip& ig, double rL, double uL,
                                                  double pL, double rR, double uR, double pR) {
    m.pos(rL); m.pos(pL); m.pos(rR); m.pos(pR);
    const double cL = m.root_quot(gamma * pL, rL);
    const double cR = m.root_quot(gamma * pR, rR);
    const double EL = m.quot(pL, ig) + 0.5 * rL * uL * uL;
    const double ER = m.quot(pR, ig) + 0.5 * rR * uR * uR;
    const double SL = smin(uL - cL, uR - cR);
    const double SR = smax(uL + cL, uR + cR);
    const double mL = rL * uL, mR = rR * uR;
    const double FL1 = mL * uL + pL, FL2 = (EL + pL) * uL;
    const double FR1 = mR * uR + pR, FR2 = (ER + pR) * uR;
    const double SLR = SL * SR, dS = SR - SL;
    const double n0 = SR * mL - SL * mR + SLR * (rR - rL);
    const double n1 = SR * FL1 - SL * FR1 + SLR * (mR - mL);
    const double n2 = SR * FL2 - SL * FR2 + SLR * (ER - EL);
    m.pos(dS); m.num(n0); m.num(n2);
    const auto id = m.recip(dS);
    const bool l = SL >= 0.0, r = SR <= 0.0;
    return { l ? mL : r ? mR : m.quot(n0, id), l ? FL1 : r ? FR1 : m.quot(n1, id), l ? FL2 : r ? FR2 : m.quot(n2, id) };
}

__device__ __noinline__ F3<double> hlle1d_ieee(double gamma, double gm1, double rL, double uL, double pL, double rR,
                                               double uR, double pR) {
    F3<double> f;
    hlle1d(gamma, gm1, rL, uL, pL, rR, uR, pR, f.a, f.b, f.c);
    return f;
}

template <class A>
__device__ __forceinline__ F3<double> face_flux(const Gas<double, A>& g, double rL, double uL, double pL, double rR,
                                                double uR, double pR) {
    A m;
    const F3<double> f = hlle1d_fast(m, g.gamma, g.ig, rL, uL, pL, rR, uR, pR);
    if (m.ok() && g.fast) return f;
    return hlle1d_ieee(g.gamma, g.gm1, rL, uL, pL, rR, uR, pR);
}
__device__ __forceinline__ F3<float> face_flux(const Gas<float>& g, float rL, float uL, float pL, float rR, float uR,
                                               float pR) {
    F3<float> f;
    hlle1d(g.gamma, g.gm1, rL, uL, pL, rR, uR, pR, f.a, f.b, f.c);
    return f;
}

// Velocity, pressure (clamped at 0) and, where CS, the sound speed of a
// conserved cell (cons_to_prim and sound_speed, euler1d.hpp:31-84).  A finite
// velocity follows from the pressure's range.
template <typename T> struct Cell1 { T u, p, cs; };

template <bool CS>
__device__ __noinline__ Cell1<double> cell1d_ieee(double gamma, double gm1, double r, double m, double e) {
    const double u = m / r, p = eos_pressure(gm1, r, m, e);
    return { u, p, CS ? sqrt(gamma * p / r) : 0.0 };
}

template <bool CS, class A>
__device__ __forceinline__ Cell1<double> cell1d(const Gas<double, A>& g, double r, double m, double e) {
    A a;
    const auto ir = a.recip(r);
    const double u = a.quot(m, ir);
    // (a p that the clamp would change fails its test; halving is exact, and a
    // subnormal product is far below the energy's rounding)
    const double p = g.gm1 * fma(-0.5, r * u * u, e);
    const double cs = CS ? a.root_quot(g.gamma * p, r) : 0.0;
    a.pos(r); a.pos(p); a.num(m);
    if (a.ok() && g.fast) return { u, p, cs };
    return cell1d_ieee<CS>(g.gamma, g.gm1, r, m, e);
}
template <bool CS>
__device__ __forceinline__ Cell1<float> cell1d(const Gas<float>& g, float r, float m, float e) {
    const float u = m / r, p = eos_pressure(g.gm1, r, m, e);
    return { u, p, CS ? sqrt(g.gamma * p / r) : 0.f };
}

// PLM face states and flux between cells a and b, with their outer neighbours
// am and bp (each (rho, u, p) through w(k, cell)).
template <typename T, class A, class W>
__device__ __forceinline__ F3<T> plm_flux(const Gas<T, A>& g, int lim, W w, int am, int a, int b, int bp) {
    T L[3], R[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const T wa = w(k, a), wb = w(k, b), d = wb - wa;
        L[k] = wa + T(0.5) * limit(wa - w(k, am), d, lim);
        R[k] = wb - T(0.5) * limit(d, w(k, bp) - wb, lim);
    }
    return face_flux(g, L[0], L[1], L[2], R[0], R[1], R[2]);
}

// Stage fluxes of a warp whose lanes hold the primitives w of CPL neighbouring
// cells each: f[i] is the face to the right of the lane's cell i, in the
// expressions of plm_flux (valid two cells inside the valid ones).
template <typename T, int CPL>
__device__ __forceinline__ void warp_flux(const Gas<T>& g, int lim, const T (&w)[CPL][3], F3<T> (&f)[CPL]) {
    T P[CPL][3], M[CPL + 1][3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        T d[CPL];
#pragma unroll
        for (int i = 0; i < CPL; ++i)
            d[i] = (i + 1 < CPL ? w[i + 1 < CPL ? i + 1 : 0][k] : __shfl_down_sync(0xffffffffu, w[0][k], 1)) - w[i][k];
        const T dm = __shfl_up_sync(0xffffffffu, d[CPL - 1], 1);
#pragma unroll
        for (int i = 0; i < CPL; ++i) {
            const T s = limit(i > 0 ? d[i > 0 ? i - 1 : 0] : dm, d[i], lim);
            P[i][k] = w[i][k] + T(0.5) * s;
            M[i][k] = w[i][k] - T(0.5) * s;
        }
        M[CPL][k] = __shfl_down_sync(0xffffffffu, M[0][k], 1);
    }
#pragma unroll
    for (int i = 0; i < CPL; ++i)
        f[i] = face_flux(g, P[i][0], P[i][1], P[i][2], M[i + 1][0], M[i + 1][1], M[i + 1][2]);
}

}  // namespace
}  // namespace nestb
