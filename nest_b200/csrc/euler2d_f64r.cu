// FP64 plain form of the 2D stage kernels as a staged row march (sm_100a).
//
// Same scheme, operation order and results (bit for bit) as stage2d_body in
// euler2d_kernels.cuh, compiled with -fmad=false; what changes is how a warp
// keeps its work fed:
//   * input rows reach the warp through shared-memory rings filled by 16-byte
//     cp.async copies issued three rows ahead (U^n one row ahead in stage 2),
//     so loads in flight hold no registers and the update's re-read of its
//     own row is a shared-memory hit;
//   * the row window is the primitives of rows q and q+1, the upper x-face
//     state of row q and the x-flux of face q-1/2 (16 doubles), and the first
//     rows of the tile are computed before the loop, so the loop body is one
//     block with the x-face and the y-face fluxes of a row side by side,
//     free to interleave their division and square-root chains.
// A warp owns a strip of 32 columns j0-2 .. j0+29 (j0 = 28 strip) and
// writes lanes 2..29, like stage2d_body.
#include "euler2d_kernels.cuh"
#include "f64div.cuh"
#include "kernels.h"

#include <algorithm>
#include <cstdlib>
#include <string>

namespace nestb {
namespace {

constexpr int LOOKD = 3;                   // stage-input rows in flight ahead of the march
constexpr int RING_UD = 4, RING_ND = 2;    // ring slots: stage input, U^n (stage 2)
__host__ __device__ constexpr int ring_d_per_warp(int stage) { return (RING_UD + (stage == 2 ? RING_ND : 0)) * 4 * 32; }
extern __shared__ __align__(16) double f64r_ring[];

__device__ __forceinline__ void cp16d(double* smem_dst, const double* gsrc) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cpd_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cpd_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

using W4 = Win4<double>;

// A row runs with ArithFast (f64div.cuh); one in which a range test fails for a
// lane that can reach an output is computed again with ArithIeee before anything
// of it is stored.
//
// What the tests rest on.  prim() tests rho and p of every cell the row adds to
// the window (and the two momenta as numerators); a finite u or v follows, with
// |u| < 2^181, because 2^-128 <= p = (gamma - 1) (E - ke) < 2^128 needs
// ke < 2^233.  A row whose window holds a cell that failed runs with the IEEE
// policy as a whole (`hold` below).  A minmod face state w -+ s/2 lies between w
// and half way to a neighbour, so rho and p of a face need no test of their own
// (with the other limiters, which can reach or pass the neighbour's value, they
// get one).  dS = SR - SL is at least about the smaller sound speed where the
// average flux is taken, and its numerators stay under 2^880; the mass,
// transverse and energy ones, which can be tiny, are tested (the normal one
// holds SR p - SL p, which cannot).
// Face states w + s/2 and w - s/2.
template <class A>
__device__ __forceinline__ W4 face_up(const A& m, const W4& w, const W4& s) {
    return { m.half(w.a, 0.5, s.a), m.half(w.b, 0.5, s.b), m.half(w.c, 0.5, s.c), m.half(w.d, 0.5, s.d) };
}
template <class A>
__device__ __forceinline__ W4 face_dn(const A& m, const W4& w, const W4& s) {
    return { m.half(w.a, -0.5, s.a), m.half(w.b, -0.5, s.b), m.half(w.c, -0.5, s.c), m.half(w.d, -0.5, s.d) };
}

// cons2prim, hlle4 and cell_speeds_p of euler2d_kernels.cuh for the FP64
// plain form (the same expressions in the same order, so the same values),
// with their divisions and square roots taken from a policy.  The checked policy
// also takes the halves out of the kinetic energies: ((0.5 r) u) u is 0.5 ((r u) u)
// and so on, exactly, unless a product is subnormal, and there it is far below
// the rounding of the energy (at least 2^-130) it is added to.

// (r u) u + (r v) v, twice ke2(r, u, v).
__device__ __forceinline__ double twice_ke(double r, double u, double v) { return r * u * u + r * v * v; }

template <class A>
__device__ __forceinline__ W4 prim_d(A& m, const W4& c, double gm1) {
    const auto ir = m.recip(c.a);
    const double u = m.quot(c.b, ir), v = m.quot(c.c, ir);
    // (a p that the clamp would change fails its test)
    const double p = A::checked ? gm1 * fma(-0.5, twice_ke(c.a, u, v), c.d) : smax(gm1 * (c.d - ke2(c.a, u, v)), 0.0);
    m.pos(c.a); m.pos(p); m.num(c.b); m.num(c.c);
    return { c.a, u, v, p };
}

// ig: reciprocal of gamma - 1; FACE: test the face states.
template <bool FACE, class A>
__device__ __forceinline__ void hlle4_d(A& m, double gamma, const typename A::Recip& ig, double rL, double nL,
                                        double tL, double pL, double rR, double nR, double tR, double pR, double& f0,
                                        double& f1, double& f2, double& f3) {
    const double cL = m.root(m.quot(gamma * pL, m.recip(rL)));
    const double cR = m.root(m.quot(gamma * pR, m.recip(rR)));
    // (r n) n, r t and (r t) t below are shared with the fluxes
    const double EL = A::checked ? fma(0.5, twice_ke(rL, nL, tL), m.quot(pL, ig)) : m.quot(pL, ig) + ke2(rL, nL, tL);
    const double ER = A::checked ? fma(0.5, twice_ke(rR, nR, tR), m.quot(pR, ig)) : m.quot(pR, ig) + ke2(rR, nR, tR);
    const double SL = smin(nL - cL, nR - cR);
    const double SR = smax(nL + cL, nR + cR);
    const double mL = rL * nL, mR = rR * nR;
    const double FL0 = mL, FL1 = mL * nL + pL, FL2 = mL * tL, FL3 = (EL + pL) * nL;
    const double FR0 = mR, FR1 = mR * nR + pR, FR2 = mR * tR, FR3 = (ER + pR) * nR;
    if (FACE) { m.pos(rL); m.pos(pL); m.pos(rR); m.pos(pR); }
    if (A::checked) {
        // the average flux in every lane, then the regime's selection
        const double SLR = SL * SR, dS = SR - SL;
        const auto id = m.recip(dS);
        const double a0 = SR * FL0 - SL * FR0 + SLR * (rR - rL), a1 = SR * FL1 - SL * FR1 + SLR * (mR - mL);
        const double a2 = SR * FL2 - SL * FR2 + SLR * (rR * tR - rL * tL), a3 = SR * FL3 - SL * FR3 + SLR * (ER - EL);
        m.num(a0); m.num(a2); m.num(a3);
        // SL >= 0 and SR <= 0 from the bits (c > 0, so neither is -0)
        const bool l = __double2hiint(SL) >= 0, r = __double_as_longlong(SR) <= 0;
        f0 = l ? FL0 : r ? FR0 : m.quot(a0, id);
        f1 = l ? FL1 : r ? FR1 : m.quot(a1, id);
        f2 = l ? FL2 : r ? FR2 : m.quot(a2, id);
        f3 = l ? FL3 : r ? FR3 : m.quot(a3, id);
    } else if (SL >= 0.0) {
        f0 = FL0; f1 = FL1; f2 = FL2; f3 = FL3;
    } else if (SR <= 0.0) {
        f0 = FR0; f1 = FR1; f2 = FR2; f3 = FR3;
    } else {
        const double SLR = SL * SR;
        const auto id = m.recip(SR - SL);
        f0 = m.quot(SR * FL0 - SL * FR0 + SLR * (rR - rL), id);
        f1 = m.quot(SR * FL1 - SL * FR1 + SLR * (mR - mL), id);
        f2 = m.quot(SR * FL2 - SL * FR2 + SLR * (rR * tR - rL * tL), id);
        f3 = m.quot(SR * FL3 - SL * FR3 + SLR * (ER - EL), id);
    }
}

template <class A>
__device__ __forceinline__ double speeds_d(A& m, double U0, double U1, double U2, double U3, double gamma,
                                           double gm1, double& sx, double& sy) {
    const double rho = smax(U0, 1e-10);
    const auto ir = m.recip(rho);
    const double u = m.quot(U1, ir), v = m.quot(U2, ir);
    const double uv = u * u + v * v;
    const double p = smax(gm1 * (A::checked ? fma(-0.5, rho * uv, U3) : U3 - 0.5 * rho * uv), 1e-10);
    const double c = m.root(m.quot(gamma * p, ir));
    sx = fabs(u) + c;
    sy = fabs(v) + c;
    // p is at least 1e-10, and at most a few pc where pc > 0; the test of pc also
    // takes cells to be flagged and states that are not finite to the IEEE forms
    const double pc = A::checked ? gm1 * fma(-0.5, twice_ke(rho, u, v), U3) : gm1 * (U3 - ke2(rho, u, v));
    m.pos(rho); m.pos(pc); m.num(U1); m.num(U2);
    return pc;
}

// LIM: the slope limiter fixed at compile time (LIM_MINMOD, nest's default),
// or -1 to read it from the loop parameters; a fixed limiter leaves no
// limiter branch in the row loop.
template <int STAGE, bool TOT, int LIM, class Args>
__device__ __forceinline__ void f64r_body(const Args& a, int strip, int tile_row) {
    const Geo2D& g = a.g;
    const int lane = threadIdx.x & 31;
    const double gamma = g.gamma;
    const double gm1 = g.gamma - 1.0;

    const int lim = LIM >= 0 ? LIM : a.lp.lim;

    const int nx = g.nx, ny = g.ny, pitch = g.pitch;
    const int j0 = strip * STRIP;
    if (j0 >= ny) return;                  // whole warp idle
    const int j = j0 - 2 + lane;           // this lane's column
    const bool out_col = lane >= 2 && lane < 30 && j < ny;
    const bool edge_col = j < 2 || j >= ny - 2;
    const int i0 = tile_row * a.tx;
    if (i0 >= nx) return;
    const int rows = min(a.tx, nx - i0);
    const int last_row = nx + 1;           // staged rows past it are clamped to it
    const long long vs = g.vstride;
    const double* __restrict__ Ui = a.Uin;
    const double* Unp = a.Un;
    double* const Uo = a.Uout;

    // this warp's rings: RING_UD slots of the stage input, then RING_ND of U^n;
    // a slot is [var][32 columns]
    double* const ringw = f64r_ring + threadIdx.y * ring_d_per_warp(STAGE);
    // 16-byte chunk copies: lane l moves columns j0-2+2(l & 15) .. +1 of
    // variables l >> 4 and (l >> 4) + 2.  Chunk starts are 16-byte aligned
    // (j0 = 28 strip, pitch a multiple of 16); chunks past the row end re-read
    // the row's last two columns, which feed only discarded lanes.
    const int part = lane & 15, cvar = lane >> 4;
    const long long cseg = min(j0 + 2 * part, pitch - 2) + (long long)cvar * vs;
    const int cofs = cvar * 32 + 2 * part;
    auto stage_rows = [&](const double* base, int i, double* slot) {
        const double* q = base + (long long)(min(i, last_row) + 2) * pitch + cseg;
        cp16d(slot + cofs, q);
        cp16d(slot + cofs + 64, q + 2 * vs);
    };
    auto stage_row = [&](int i) { stage_rows(Ui, i, ringw + (i & (RING_UD - 1)) * 128); };
    auto stage_un = [&](int i) { stage_rows(Unp, i, ringw + RING_UD * 128 + (i & (RING_ND - 1)) * 128); };
    auto ring_row = [&](int i) -> W4 {
        const double* d = ringw + (i & (RING_UD - 1)) * 128 + lane;
        return { d[0], d[32], d[64], d[96] };
    };
    auto ring_un = [&](int i) -> W4 {
        const double* d = ringw + RING_UD * 128 + (i & (RING_ND - 1)) * 128 + lane;
        return { d[0], d[32], d[64], d[96] };
    };
    auto load = [&](int i) -> W4 {
        const long long o = g.at(i, min(j, ny + 1));
        return { __ldg(Ui + o), __ldg(Ui + vs + o), __ldg(Ui + 2 * vs + o), __ldg(Ui + 3 * vs + o) };
    };

    // gamma and gamma - 1 inside the range tests' assumptions; else every row
    // takes the IEEE policy.  `hold`: rows still to run with it because the
    // window holds a cell that failed a test (a cell enters as row i+2 and
    // leaves with the upper face state of row i, three rows later).
    const int hold_all = gamma < 1024.0 && gm1 > 0x1p-20 ? 0 : 1 << 30;
    int hold = hold_all;
    constexpr bool FACE = LIM != LIM_MINMOD;
    const typename ArithFast::Recip igf{ gm1, recip_f64(gm1) };
    const typename ArithIeee::Recip igi{ gm1 };

    // prologue: rows i0-2 .. i0+1, the x-flux of face i0-1/2 and the upper
    // x-face state of row i0
    W4 Wq, Wq1, Pq, Fm;
    double dtdx, dtdy;
    {
        const W4 c0 = load(i0 - 2), c1 = load(i0 - 1);
        for (int r = 0; r < LOOKD; ++r) stage_row(i0 + r);
        if (STAGE == 2)
            for (int r = 0; r < LOOKD - 2; ++r) stage_un(i0 + r);
        cpd_commit();
        // the step's dt while the first rows are on their way
        double dt;
        const bool run = stage_dt<STAGE>(a, strip == 0 && tile_row == 0 && lane == 0, dt);
        cpd_wait<0>();
        __syncwarp();
        if (!run) return;
        dtdx = div_rn(dt, g.dx);
        dtdy = div_rn(dt, g.dy);
        auto pro = [&](auto& m, auto& mp, const auto& ig) {
            const W4 Wa = prim_d(mp, c0, gm1), Wb = prim_d(mp, c1, gm1);
            Wq = prim_d(mp, ring_row(i0), gm1);
            Wq1 = prim_d(mp, ring_row(i0 + 1), gm1);
            const W4 Sb = limit4(Wa, Wb, Wq, lim), Sq = limit4(Wb, Wq, Wq1, lim);
            const W4 L = face_up(m, Wb, Sb), R = face_dn(m, Wq, Sq);
            hlle4_d<FACE>(m, gamma, ig, L.a, L.b, L.c, L.d, R.a, R.b, R.c, R.d, Fm.a, Fm.b, Fm.c, Fm.d);
            Pq = face_up(m, Wq, Sq);
        };
        // columns up to the last ghost column can reach an output; lanes past
        // it read the row padding
        ArithFast m, mp;
        pro(m, mp, igf);
        const bool badp = __any_sync(0xffffffffu, !mp.ok() && j <= ny + 1);
        if (badp) hold = max(hold, 3);
        if (badp || hold || __any_sync(0xffffffffu, !m.ok() && j <= ny + 1)) {
            ArithIeee mi;
            pro(mi, mi, igi);
        }
    }

    double smx = 0.0, smy = 0.0;
    double t0 = 0.0, t1 = 0.0, t2 = 0.0, t3 = 0.0;
#pragma unroll 1
    for (int k = 0; k < rows; ++k) {
        const int i = i0 + k;
        // refill the slots of row i-1 once every lane has read them; then
        // wait for rows up to i+2 (and U^n row i)
        __syncwarp();
        stage_row(i + LOOKD);
        if (STAGE == 2) stage_un(i + LOOKD - 2);
        cpd_commit();
        cpd_wait<LOOKD - 2>();
        __syncwarp();

        // The row's arithmetic, with the divisions of a policy: the x-face
        // i+1/2 from rows i .. i+2, the y-faces of row i (face j+1/2, normal v,
        // transverse u; the left face from the left neighbour), the update of
        // every lane's cell of row i and, in stage 2, its wave speeds.
        struct RowOut {
            W4 W2, P1, Fc, s;  // P1: upper x-face state of row i+1
            double sx, sy, pc;
        };
        auto row = [&](auto& mp, auto& mf, const auto& ig) {
            RowOut o;
            o.W2 = prim_d(mp, ring_row(i + 2), gm1);
            const W4 S1 = limit4(Wq, Wq1, o.W2, lim);
            const W4 M1 = face_dn(mf, Wq1, S1);
            o.P1 = face_up(mf, Wq1, S1);
            hlle4_d<FACE>(mf, gamma, ig, Pq.a, Pq.b, Pq.c, Pq.d, M1.a, M1.b, M1.c, M1.d, o.Fc.a, o.Fc.b, o.Fc.c,
                          o.Fc.d);
            const W4 sy = limit4(shfl_up4(Wq), Wq, shfl_dn4(Wq), lim);
            const W4 Rq = shfl_dn4(face_dn(mf, Wq, sy));
            const W4 Ly = face_up(mf, Wq, sy);
            W4 Gy;
            hlle4_d<FACE>(mf, gamma, ig, Ly.a, Ly.c, Ly.b, Ly.d, Rq.a, Rq.c, Rq.b, Rq.d, Gy.a, Gy.c, Gy.b, Gy.d);
            const W4 Gl = shfl_up4(Gy);
            const W4 C0 = ring_row(i);
            o.s.a = C0.a - (dtdx * (o.Fc.a - Fm.a) + dtdy * (Gy.a - Gl.a));
            o.s.b = C0.b - (dtdx * (o.Fc.b - Fm.b) + dtdy * (Gy.b - Gl.b));
            o.s.c = C0.c - (dtdx * (o.Fc.c - Fm.c) + dtdy * (Gy.c - Gl.c));
            o.s.d = C0.d - (dtdx * (o.Fc.d - Fm.d) + dtdy * (Gy.d - Gl.d));
            if (STAGE == 2) {
                const W4 N0 = ring_un(i);
                o.s.a = 0.5 * (N0.a + o.s.a);
                o.s.b = 0.5 * (N0.b + o.s.b);
                o.s.c = 0.5 * (N0.c + o.s.c);
                o.s.d = 0.5 * (N0.d + o.s.d);
                o.pc = speeds_d(mf, o.s.a, o.s.b, o.s.c, o.s.d, gamma, gm1, o.sx, o.sy);
            }
            return o;
        };
        // The branch-free arithmetic first; if a range test of something that
        // can reach an output failed, the whole row again with the IEEE
        // operations.  Either way the stored values are those of the IEEE
        // arithmetic.  What reaches an output: the primitives of every lane
        // up to the last ghost column (y-slopes of the lanes two away), and
        // the fluxes and wave speeds of lanes 1..29 inside the domain (lane
        // j-1's y-face is lane j's left face); lanes past the ghost columns
        // read the row padding.
        ArithFast mp, mf;
        RowOut o = row(mp, mf, igf);
        const bool badp = __any_sync(0xffffffffu, !mp.ok() && j <= ny + 1);
        const bool badf = __any_sync(0xffffffffu, !mf.ok() && lane >= 1 && lane < 30 && j < ny);
        if (badp) hold = max(hold, 4);
        if (badf || hold > 0) {
            ArithIeee mi;
            o = row(mi, mi, igi);
            if (hold > 0) --hold;
        }

        if (out_col) {
            const double s0 = o.s.a, s1 = o.s.b, s2 = o.s.c, s3 = o.s.d;
            if (STAGE == 2) {
                const double pc = o.pc;
                if (!(s0 >= 1e-10) || !(pc > 0.0)) {
                    double pe = pc;
                    if (s0 > 0.0 && s0 < 1e-10) pe = gm1 * (s3 - ke2(s0, s1 / s0, s2 / s0));
                    if (!(s0 > 0.0) || !(pe > 0.0) || !(pe == pe))
                        flag_cell(a.ctrl, a.ctrl->step[a.p] + 1, s0, pe, i, j);
                }
                smx = smax(smx, o.sx);
                smy = smax(smy, o.sy);
                if (TOT) { t0 += s0; t1 += s1; t2 += s2; t3 += s3; }
            }
            const long long oo = g.at(i, j);
            Uo[oo] = s0; Uo[vs + oo] = s1; Uo[2 * vs + oo] = s2; Uo[3 * vs + oo] = s3;
            if (edge_col || i < 2 || i >= nx - 2) {
                store_ghosts(Uo, g, 0, i, j, s0);
                store_ghosts(Uo, g, 1, i, j, s1);
                store_ghosts(Uo, g, 2, i, j, s2);
                store_ghosts(Uo, g, 3, i, j, s3);
            }
        }
        Fm = o.Fc;
        Pq = o.P1;
        Wq = Wq1;
        Wq1 = o.W2;
    }
    // no copy may land in shared memory after the warp has left
    cpd_wait<0>();
    __syncwarp();
    if (STAGE == 2) {
        smx = warp_max_speed(smx);
        smy = warp_max_speed(smy);
        if (lane == 0) {
            if (!(smx == smx) || !(smy == smy) || smx > 1.79e308 || smy > 1.79e308)
                atomicOr(&a.ctrl->err, ERRW_NONFINITE);
            atomic_max_speed(&a.ctrl->maxs[a.p ^ 1][0], smx);
            atomic_max_speed(&a.ctrl->maxs[a.p ^ 1][1], smy);
        }
        if (TOT) {
            t0 = warp_sum(t0); t1 = warp_sum(t1); t2 = warp_sum(t2); t3 = warp_sum(t3);
            if (lane == 0) {
                long long wid = ((long long)tile_row * ((ny + STRIP - 1) / STRIP) + strip) * 4;
                a.partials[wid + 0] = t0; a.partials[wid + 1] = t1;
                a.partials[wid + 2] = t2; a.partials[wid + 3] = t3;
            }
        }
    }
}

// Register budget: 168 a thread, 12 warps per SM.  The kernels are bound by the
// FP64 pipe (about 360 / 410 FP64 instructions a row, two issue cycles each,
// put a 4096^2 step at 0.81 ms) and by the latency of its division and square
// root chains, and with no branch in them the compiler interleaves the x- and
// y-face chains of a row: more registers a warp pay off against fewer warps.
// 4096^2 diagonal Riemann problem, ms per step over 64 steps (24-row tiles):
// budget 128 (16 warps, spills) 1.313, 144 (14) 1.328, ptxas's own choice (158,
// 12) 1.297, 168 (12) 1.261, 192 (10) 1.421, unrolled by 2 1.429.  With the
// quotients tested one by one by an exact residual and the IEEE square root the
// step took 2.090 ms, 1000 steps of the 2048^2 periodic Kelvin-Helmholtz state
// 576 -> 349 ms.  Tile rows now: 16 1.286, 24 1.261, 32 1.265, 48 1.283.
// Dependent launch, and dt worked out while the first rows are on their way:
// 4096^2 1.256 -> 1.229, 2048^2 Kelvin-Helmholtz 0.348 -> 0.339, 256 x 192 25.5 -> 22.9 us.
// Halves of the kinetic energies fused, Goldschmidt's square root, regimes and
// numerator tests from integer words: 4096^2 1.233 -> 1.164, 2048^2 Kelvin-
// Helmholtz 0.339 -> 0.322 (then: budget 160 1.176, 176 1.166).
#ifndef NEST_F64R_REGS
#define NEST_F64R_REGS 168
#endif

template <int STAGE, bool TOT, int LIM>
__global__ void __maxnreg__(NEST_F64R_REGS) k2d_f64r(StageArgs<double> a) {
    pdl_wait();
    pdl_trigger();
    f64r_body<STAGE, TOT, LIM>(a, blockIdx.x * blockDim.y + threadIdx.y, blockIdx.y);
}

// Arguments of one batched work item: the arrays of its problem, whose geometry
// stays in global memory (the body copies the fields its row loop needs).
struct F64View {
    const double* Uin;
    const double* Un;
    double* Uout;
    const Geo2D& g;
    const LoopParams& lp;
    StepCtrl* ctrl;
    double* partials;
    int p;
    int tx;
};

// Batched stage (bit for bit the single-domain solver's result per
// problem): every warp walks the work list (problem, strip, tile row) with the
// grid's warp count as stride (one item each by default).
// Us per step with TOTALS, against the register-window march with IEEE
// divisions in 32-row items: 4 problems of 64..128 a side 24 (216), 48 of 64..256
// 182 (258), 64 of 48..320 312 (508; before the fused halves).
template <int STAGE, bool TOT>
__global__ void __maxnreg__(NEST_F64R_REGS) kbatch_f64(BatchArgs<double> b) {
    pdl_wait();
    pdl_trigger();
    const int nw = gridDim.x * blockDim.y;
    for (int it = blockIdx.x * blockDim.y + threadIdx.y; it < b.nitems; it += nw) {
        const int4 w = b.items[it];
        const BatchProblem& P = b.probs[w.x];
        const F64View v{STAGE == 1 ? b.U + P.off : b.U1 + P.off, STAGE == 2 ? b.U + P.off : nullptr,
                        STAGE == 1 ? b.U1 + P.off : b.U + P.off, P.g, b.lp, b.ctrls + w.x,
                        TOT ? b.partials + 4ll * P.item0 : nullptr, b.p, b.tx};
        f64r_body<STAGE, TOT, LIM_MINMOD>(v, w.y, w.z);
    }
}

template <int LIM>
cudaError_t launch_f64r_lim(const StageArgs<double>& a1, const StageArgs<double>& a2, dim3 gr, dim3 b, size_t sm1,
                            size_t sm2, int which, bool tot, cudaStream_t st) {
    cudaError_t e = cudaSuccess;
    if (which & 1) e = launch_pdl(k2d_f64r<1, false, LIM>, gr, b, sm1, st, a1);
    if ((which & 2) && e == cudaSuccess)
        e = launch_pdl(tot ? k2d_f64r<2, true, LIM> : k2d_f64r<2, false, LIM>, gr, b, sm2, st, a2);
    return e;
}

size_t f64r_ring_bytes(int stage, int warps) { return (size_t)warps * ring_d_per_warp(stage) * sizeof(double); }

}  // namespace

cudaError_t launch_2d_step_f64r(double* U, double* U1, const Geo2D& g, const LoopParams& lp, StepCtrl* ctrl,
                                double* partials, int p, int tx, int warps, int which, cudaStream_t st,
                                double* Uout) {
    const int nstrips = (g.ny + STRIP - 1) / STRIP;
    dim3 b(32, warps), gr((nstrips + warps - 1) / warps, (g.nx + tx - 1) / tx);
    StageArgs<double> a1{U, nullptr, U1, g, lp, ctrl, nullptr, p, tx};
    StageArgs<double> a2{U1, U, Uout ? Uout : U, g, lp, ctrl, partials, p, tx};
    const size_t sm1 = f64r_ring_bytes(1, warps), sm2 = f64r_ring_bytes(2, warps);
    return lp.lim == LIM_MINMOD ? launch_f64r_lim<LIM_MINMOD>(a1, a2, gr, b, sm1, sm2, which, partials != nullptr, st)
                                : launch_f64r_lim<-1>(a1, a2, gr, b, sm1, sm2, which, partials != nullptr, st);
}

cudaError_t launch_batch_f64(const BatchArgs<double>& b, int which, int blocks, int warps, cudaStream_t st) {
    const dim3 blk(32, warps);
    const size_t sm1 = f64r_ring_bytes(1, warps), sm2 = f64r_ring_bytes(2, warps);
    cudaError_t e = cudaSuccess;
    if (which & 1) e = launch_pdl(kbatch_f64<1, false>, dim3(blocks), blk, sm1, st, b);
    if ((which & 2) && e == cudaSuccess)
        e = launch_pdl(b.partials ? kbatch_f64<2, true> : kbatch_f64<2, false>, dim3(blocks), blk, sm2, st, b);
    return e;
}

// Resident blocks per SM of the batched stages (6 KB of rings a warp: no
// opt-in shared memory up to the 8 warps a block may have).
int batch_max_blocks_f64(int warps) {
    int nb = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kbatch_f64<2, true>, 32 * warps, f64r_ring_bytes(2, warps));
    return nb;
}

namespace {
// The policies' quotient, its sign set for a divisor of either sign, and
// whether the kernels would keep it.
__global__ void k_div_selftest(const double* a, const double* b, double* q, int* ok, int n) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) {
        const double d = fabs(b[t]), v = copysign(1.0, b[t]) * a[t];
        q[t] = quot_f64(v, d, recip_f64(d));
        ok[t] = quot_in_range(v, d, q[t]) ? 1 : 0;
    }
}
__global__ void k_sqrt_selftest(const double* a, double* r, int* ok, int n) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) {
        r[t] = sqrt_f64(a[t]);
        ok[t] = a[t] >= 0x1p-257 && a[t] < 0x1p268 ? 1 : 0;
    }
}
__global__ void k_sqrt_quot_selftest(const double* a, const double* b, double* r, int* ok, int n) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) {
        double q;
        F64Range m;
        r[t] = sqrt_quot_f64(a[t], b[t], q);
        m.root(q);
        ok[t] = m.ok() && a[t] >= 0x1p-128 && a[t] < 0x1p138 && b[t] >= 0x1p-128 && b[t] < 0x1p128 ? 1 : 0;
    }
}
}  // namespace

}  // namespace nestb

namespace {
template <class Launch>
nest_status selftest(const void* d_a, const void* d_q, const void* d_ok, int n, const char* what, Launch launch) {
    if (!d_a || !d_q || !d_ok || n < 0) return nestb::record_error(NEST_ERR_INVALID, "null array or n < 0");
    if (n == 0) return NEST_OK;
    launch((n + 255) / 256);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) return nestb::record_error(NEST_ERR_CUDA, std::string(what) + cudaGetErrorString(e));
    return NEST_OK;
}
}  // namespace

extern "C" nest_status nest_selftest_div_f64(const double* d_a, const double* d_b, double* d_q, int* d_ok, int n) {
    if (!d_b) return nestb::record_error(NEST_ERR_INVALID, "null array or n < 0");
    return selftest(d_a, d_q, d_ok, n, "division self-test: ",
                    [&](int blocks) { nestb::k_div_selftest<<<blocks, 256>>>(d_a, d_b, d_q, d_ok, n); });
}

extern "C" nest_status nest_selftest_sqrt_f64(const double* d_x, double* d_r, int* d_ok, int n) {
    return selftest(d_x, d_r, d_ok, n, "square root self-test: ",
                    [&](int blocks) { nestb::k_sqrt_selftest<<<blocks, 256>>>(d_x, d_r, d_ok, n); });
}

extern "C" nest_status nest_selftest_sqrt_quot_f64(const double* d_a, const double* d_b, double* d_r, int* d_ok, int n) {
    if (!d_b) return nestb::record_error(NEST_ERR_INVALID, "null array or n < 0");
    return selftest(d_a, d_r, d_ok, n, "square root of a quotient self-test: ",
                    [&](int blocks) { nestb::k_sqrt_quot_selftest<<<blocks, 256>>>(d_a, d_b, d_r, d_ok, n); });
}
