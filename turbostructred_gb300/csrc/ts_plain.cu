// Plain FP64 path: the drop-in for ExplicitRungeKuttaFVM<R>::IterationStep
// (src/Methods/ExplicitRungeKuttaFVM.h:1440-1491) on one GB300.
//
// This translation unit is compiled with --fmad=false and IEEE division and
// square root, and every expression keeps the reference's operation order, so
// results match the reference's FP64 CPU path bit for bit (up to the sign of
// exact zeros: products with the zero components of axis normals, which the
// reference evaluates, are dropped here).
//
// One step, on the handle's stream:
//   k_ghost<A>   ghost layers per axis: periodic copy or boundary condition
//                (Kernel::ExchangeValues + ComputeDummyCellValues, kernel.h:334-915)
//   k_recon      per-cell slopes and limiter (ComputeSolutionReconstruction, :879-925)
//   k_flux<A>    one kernel per face direction: face states, EOS, Riemann flux
//                and max eigenvalue (ComputeResidual face loops, :1182-1419)
//   k_dt         spectral radius per cell, V/SR, warp-shuffle min, last block
//                finalises dt (ComputeTimeStep, :1427-1437)
//   k_update     flux divergence fused with the stage update
//                (residual accumulation :1232 + Kernel::UpdateSolution,
//                kernel.h:319-331); the last block closes the step: time,
//                iteration and the Kernel::Run termination rules
//
// What bounds it: the FP64 pipe.  GB300 takes 19 clocks per SM for an FP64
// warp instruction of any kind, comparisons, min/max and |x| included, while
// the issue slots are 85 % idle.  So everything but the additions and
// multiplications themselves runs on the integer pipe: divisions and square
// roots (ts_exact64.cuh), comparisons, sign changes and halvings; terms that
// are exact zeros are skipped where a whole warp agrees (transverse momentum
// of 1D and 2D flows, constant neighbourhoods, equal fluxes); the slope
// projections lim * (slope * h/2) are formed once per cell instead of at each
// of its faces; and the residual norms are summed per thread over many
// cells before the block's reduction.  The results are bit for bit the same.
// Measured on one GB300, time per step before and after: 3D blast 192^3 (Roe,
// Barth-Jespersen) 28.4 -> 9.98 ms (k_recon 8.1 -> 0.69, each k_flux 5.9 ->
// 2.7, k_update 3.0 -> 0.72); 2D shear layer 1024^2 (HLLC) 3.27 -> 0.70 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "ts_exact64.cuh"
#include "ts_plain.h"

namespace ts {

namespace {

typedef unsigned long long u64;

__device__ __forceinline__ long long vidx(const Layout& L, int v) { return (long long)v * L.plane; }

// ---------------------------------------------------------------------------
// Boundary conditions (BCGeneral.h:186-268) for a normal sgn*e_A; `side` is
// the BC table entry (the domain side, or the kind a marker selected).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void bc_values(const Phys& ph, int side, int A, double sgn, const double in[NV],
                                          double out[NV]) {
    const int t = ph.bc.type[side];
#pragma unroll
    for (int v = 0; v < NV; ++v) out[v] = in[v];
    if (t == TS_BC_SYMMETRY) {
        // rVinNormal = (n.rVin) n ; res -= 2 rVinNormal (BCGeneral.h:214-226)
        const double m = in[1 + A];
        const double s = sgn * m;
        const double rn = s * sgn;
        out[1 + A] = m - 2.0 * rn;
    } else if (t == TS_BC_WALL) {
        out[1] = in[1] * (-1.0);
        out[2] = in[2] * (-1.0);
        out[3] = in[3] * (-1.0);
    } else if (t == TS_BC_MOVING_WALL) {
        const double rho = in[0];
        const double ux = in[1] / rho, uy = in[2] / rho, uz = in[3] / rho;
        const double rhoe = in[4] - 0.5 * rho * (ux * ux + uy * uy + uz * uz);
        const double dx = 2.0 * ph.bc.vel[side][0] - ux;
        const double dy = 2.0 * ph.bc.vel[side][1] - uy;
        const double dz = 2.0 * ph.bc.vel[side][2] - uz;
        out[1] = rho * dx;
        out[2] = rho * dy;
        out[3] = rho * dz;
        out[4] = rhoe + 0.5 * rho * (dx * dx + dy * dy + dz * dz);
    } else if (t == TS_BC_SUBSONIC_INLET) {
        const double r = ph.bc.density[side];
        const double vx = ph.bc.vel[side][0], vy = ph.bc.vel[side][1], vz = ph.bc.vel[side][2];
        out[0] = r;
        out[1] = r * vx;
        out[2] = r * vy;
        out[3] = r * vz;
        double eint = ph.bc.pstatic[side] / (ph.gamma - 1);
        if (ph.eos == TS_EOS_STIFFENED_GAS) eint = eint + ph.gamma * ph.p_inf / (ph.gamma - 1);
        out[4] = eint + 0.5 * r * (vx * vx + vy * vy + vz * vz);
    }
    // Natural and SubsonicOutlet copy the inner state (BCGeneral.h:200-211).
}

// Comparisons of doubles on the integer pipe.  GB300 executes FP64 at about
// 1.7 operations per clock per SM, and half of k_recon's FP64-pipe
// instructions were comparisons (measured with ncu).  dkey is monotone in the
// value and gives -0 and +0 the same key, so dkey(a) < dkey(b) is exactly
// a < b, and the sign tests below are exactly x > 0 and x < 0, for every
// non-NaN a, b, x (a NaN only arises in a run whose health flags stop it).
__device__ __forceinline__ long long dkey(double x) {
    const long long b = __double_as_longlong(x);
    return b < 0 ? (b ^ 0x7FFFFFFFFFFFFFFFLL) + 1 : b;
}
__device__ __forceinline__ bool dlt(double a, double b) { return dkey(a) < dkey(b); }
__device__ __forceinline__ bool dpos(double x) { return __double_as_longlong(x) > 0; }
__device__ __forceinline__ bool dneg(double x) {
    const long long b = __double_as_longlong(x);
    return b < 0 && b != (long long)0x8000000000000000ULL;
}
__device__ __forceinline__ bool dzero(double x) { return x64::is_zero(x64::hi_of(x), x64::lo_of(x)); }
// |x| and -x on the integer pipe
__device__ __forceinline__ double dabs(double x) { return x64::of_words(x64::hi_of(x) & 0x7FFFFFFFu, x64::lo_of(x)); }
__device__ __forceinline__ double dneg_of(double x) { return x64::of_words(x64::hi_of(x) ^ 0x80000000u, x64::lo_of(x)); }
// |a| < |b|: the magnitudes' bit patterns order like their values
__device__ __forceinline__ bool dabs_lt(double a, double b) {
    return (__double_as_longlong(a) & 0x7FFFFFFFFFFFFFFFLL) < (__double_as_longlong(b) & 0x7FFFFFFFFFFFFFFFLL);
}

// ---------------------------------------------------------------------------
// Arithmetic of the two instances of every heavy routine
// ---------------------------------------------------------------------------
// Fast: divisions, square roots and halvings on the integer pipe
// (ts_exact64.cuh), correctly rounded like the hardware's, for operands in the
// ranges stated there; anything else sets `bad` and the result is discarded.
// Plain: the hardware operations, for the faces and cells where Fast gave up
// (zero, subnormal, infinite or NaN divisors and the like).  Both perform the
// same additions and multiplications in the same order.
struct Fast {
    typedef x64::Divisor Div;
    bool bad = false;
    __device__ __forceinline__ Div divisor(double b) { return x64::divisor(b, bad); }
    __device__ __forceinline__ double over(double a, const Div& d) { return x64::quotient(a, d, bad); }
    __device__ __forceinline__ double div(double a, double b) { return x64::div(a, b, bad); }
    __device__ __forceinline__ double root(double a) { return x64::root(a, bad); }
    __device__ __forceinline__ double half(double a) { return x64::half(a, bad); }
    __device__ __forceinline__ double mul(double a, double b) { return a * b; }
    __device__ __forceinline__ double min(double a, double b) { return dlt(a, b) ? a : b; }
    __device__ __forceinline__ double max(double a, double b) { return dlt(a, b) ? b : a; }
    __device__ __forceinline__ bool lt(double a, double b) { return dlt(a, b); }
    __device__ __forceinline__ bool ge0(double a) { return !dneg(a); }
    __device__ __forceinline__ bool le0(double a) { return !dpos(a); }
};
// FastMul: also the products written o.mul on the integer pipe (the 56 of the
// Roe flux's closing sums, of its 106).  An integer product takes 14.4 clocks
// per warp and SM, beside the FP64 pipe's 19 for the rest of the flux, so about
// half of them balances the two; with all of them there the code no longer fits the
// instruction cache.  One step of the 3D blast 192^3: none 9.96 ms, these 56
// 8.6 ms, the other 50 9.4 ms, all 9.8 ms.
struct FastMul : Fast {
    __device__ __forceinline__ double mul(double a, double b) {
        bool rare;
        const double r = x64::mul(a, b, rare);
        bad |= rare;
        return r;
    }
};
// 3D Roe faces use it: those grids keep the pipes full.  A grid of 1D or 2D
// ends in latency instead, which the integer products lengthen (2D box
// 203x157: 2741 -> 2763 us, 1D tube of 1000 cells: 40.0 -> 44.1 ms), and HLLC
// has too few products for it (2D shear layer 1024^2: 10.8 -> 10.3 ms with all).
template <int ND, int SOLVER>
using FaceArith = std::conditional_t<ND == 3 && SOLVER == TS_RS_ROE_PIKE, FastMul, Fast>;
struct Plain {
    typedef double Div;
    __device__ __forceinline__ Div divisor(double b) { return b; }
    __device__ __forceinline__ double over(double a, Div d) { return a / d; }
    __device__ __forceinline__ double div(double a, double b) { return a / b; }
    __device__ __forceinline__ double root(double a) { return sqrt(a); }
    __device__ __forceinline__ double half(double a) { return a * 0.5; }
    __device__ __forceinline__ double mul(double a, double b) { return a * b; }
    __device__ __forceinline__ double min(double a, double b) { return fmin(a, b); }
    __device__ __forceinline__ double max(double a, double b) { return fmax(a, b); }
    __device__ __forceinline__ bool lt(double a, double b) { return a < b; }
    __device__ __forceinline__ bool ge0(double a) { return a >= 0.0; }
    __device__ __forceinline__ bool le0(double a) { return a <= 0.0; }
};

// ---------------------------------------------------------------------------
// Riemann solvers
// ---------------------------------------------------------------------------
// Momentum components NC.. of both states are exact zeros (NC < 3: 1D and 2D
// flows without transverse momentum, checked by the caller): every term they
// enter is an exact zero and is left out, and their flux is zero.

__device__ __forceinline__ double pressure(const Phys& ph, double ro, double vx, double vy, double vz, double roE) {
    double p = (ph.gamma - 1.0) * (roE - ro * (vx * vx + vy * vy + vz * vz) / 2.0);
    if (ph.eos == TS_EOS_STIFFENED_GAS) p = p - ph.gamma * ph.p_inf;
    return p;
}

template <class O>
__device__ __forceinline__ double harten(double z, double eps, O& o) {
    z = dabs(z);
    if (o.lt(z, eps)) z = o.half(o.div(z * z, eps) + eps);
    return z;
}

template <int NC>
__device__ __forceinline__ double dot(const double a[3], const double b[3]) {
    double s = a[0] * b[0];
    if (NC > 1) s = s + a[1] * b[1];
    if (NC > 2) s = s + a[2] * b[2];
    return s;
}

// Velocity, |u|^2 and pressure of a face state (the pressure of
// RoeSolverPerfectGasEOS.h:41-58, shared by the solvers below).
template <int NC, class O>
struct Side {
    typename O::Div ro;
    double v[3], q, p;
    __device__ __forceinline__ Side(const Phys& ph, const double U[NV], O& o) {
        ro = o.divisor(U[0]);
        v[1] = v[2] = 0.0;
#pragma unroll
        for (int b = 0; b < NC; ++b) v[b] = o.over(U[1 + b], ro);
        q = dot<NC>(v, v);
        p = ph.gm1 * (U[4] - o.half(U[0] * q));
        if (ph.eos == TS_EOS_STIFFENED_GAS) p = p - ph.gpinf;
    }
    // F(U).e_A (RoeSolverPerfectGasEOS.h:41-58)
    template <int A>
    __device__ __forceinline__ void flux(const double U[NV], double res[NV]) const {
        const double rvn = U[0] * v[A];
        res[0] = rvn;
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            res[1 + b] = b < NC ? rvn * v[b] : 0.0;
            if (b == A) res[1 + b] = res[1 + b] + p;
        }
        res[4] = v[A] * (U[4] + p);
    }
};

// RoeSolverPerfectGasEOS::ComputeFlux (RoeSolverPerfectGasEOS.h:74-160) with
// fn = e_A; dn = 1 so dn*c = c and 1/(dn*dn) = 1 exactly.
template <int A, int NC, class O>
__device__ __forceinline__ double roe_flux(const Phys& ph, const double UL[NV], const double UR[NV], double flux[NV],
                                           O& o) {
    const double g = ph.gamma;
    const Side<NC, O> l(ph, UL, o), r(ph, UR, o);
    {
        double FL[NV], FR[NV];
        l.template flux<A>(UL, FL);
        r.template flux<A>(UR, FR);
#pragma unroll
        for (int i = 0; i < NV; ++i) flux[i] = FL[i] + FR[i];
    }
    const double ro_l = UL[0], ro_r = UR[0];
    const double e_l = o.over(UL[4], l.ro), e_r = o.over(UR[4], r.ro);
    double k = o.half(l.q);
    double h_l = (e_l - k) * g + k;
    k = o.half(r.q);
    double h_r = (e_r - k) * g + k;
    if (ph.eos == TS_EOS_STIFFENED_GAS) {
        h_l = h_l - o.over(ph.gpinf, l.ro);
        h_r = h_r - o.over(ph.gpinf, r.ro);
    }
    const double sl = o.root(ro_l), sr = o.root(ro_r);
    const typename O::Div ss = o.divisor(sl + sr);
    const double ql = o.over(sl, ss);
    const double qr = o.over(sr, ss);
    double vel[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int b = 0; b < NC; ++b) vel[b] = ql * l.v[b] + qr * r.v[b];
    const double h = ql * h_l + qr * h_r;
    const double phi2 = ph.hgm1 * dot<NC>(vel, vel);
    const double c = o.root(ph.gm1 * h - phi2);
    const double uw = vel[A];
    const double eig_max = dabs(uw) + c;
    double AA1 = dabs(uw), AA3 = dabs(uw + c), AA4 = dabs(uw - c);
    if (ph.eps != 0.0) {
        const double he = ph.eps * eig_max;
        AA1 = harten(AA1, he, o);
        AA3 = harten(AA3, he, o);
        AA4 = harten(AA4, he, o);
    }
    const double Eig1 = AA1;
    const double Eiga = o.div(o.half(AA3 - AA4), c);
    const double Eigb = o.half(AA3 + AA4) - AA1;
    const double R1 = phi2 * ro_r - ph.gm1 * ro_r * (dot<NC>(vel, r.v) - e_r);
    const double D1 = ro_r * (r.v[A] - vel[A]);
    const double R2 = phi2 * ro_l - ph.gm1 * ro_l * (dot<NC>(vel, l.v) - e_l);
    const double D2 = ro_l * (l.v[A] - vel[A]);
    const double C2 = o.div(1.0, c * c);
    // Qa = (0, e_A, uw), Qb = (1, vel, h); terms multiplying a zero Qa entry
    // are exact zeros and are left out.
    {
        const double t = o.mul(Eig1, UL[0]) + o.mul(Eiga, D2) + o.mul(Eigb, o.mul(R2, C2)) - o.mul(Eig1, UR[0]) -
                         o.mul(Eiga, D1) - o.mul(Eigb, o.mul(R1, C2));
        flux[0] = o.half(flux[0] + t);
    }
#pragma unroll
    for (int b = 0; b < 3; ++b) {
        if (b >= NC) continue;
        double t;
        if (b == A)
            t = o.mul(Eig1, UL[1 + b]) + o.mul(Eiga, R2 + o.mul(D2, vel[b])) +
                o.mul(Eigb, o.mul(o.mul(R2, vel[b]), C2) + D2) - o.mul(Eig1, UR[1 + b]) -
                o.mul(Eiga, R1 + o.mul(D1, vel[b])) - o.mul(Eigb, o.mul(o.mul(R1, vel[b]), C2) + D1);
        else
            t = o.mul(Eig1, UL[1 + b]) + o.mul(Eiga, o.mul(D2, vel[b])) +
                o.mul(Eigb, o.mul(o.mul(R2, vel[b]), C2)) - o.mul(Eig1, UR[1 + b]) -
                o.mul(Eiga, o.mul(D1, vel[b])) - o.mul(Eigb, o.mul(o.mul(R1, vel[b]), C2));
        flux[1 + b] = o.half(flux[1 + b] + t);
    }
    {
        const double t = o.mul(Eig1, UL[4]) + o.mul(Eiga, o.mul(R2, uw) + o.mul(D2, h)) +
                         o.mul(Eigb, o.mul(o.mul(R2, h), C2) + o.mul(D2, uw)) - o.mul(Eig1, UR[4]) -
                         o.mul(Eiga, o.mul(R1, uw) + o.mul(D1, h)) -
                         o.mul(Eigb, o.mul(o.mul(R1, h), C2) + o.mul(D1, uw));
        flux[4] = o.half(flux[4] + t);
    }
    return eig_max;
}

// HLLC (Toro ch. 10.4) with Einfeldt-type speeds from Roe averages; same
// operation order as the oracle's restatement.  Not in the reference.  The
// flux and star state of the side that S* selects are formed once, from the
// selected operands.
template <int A, int NC, class O>
__device__ __forceinline__ double hllc_flux(const Phys& ph, const double UL[NV], const double UR[NV], double flux[NV],
                                            O& o) {
    const double g = ph.gamma;
    const bool stiff = ph.eos == TS_EOS_STIFFENED_GAS;
    const double pinf = stiff ? ph.p_inf : 0.0;
    const double rl = UL[0], rr = UR[0];
    const Side<NC, O> l(ph, UL, o), r(ph, UR, o);
    const double ul = l.v[A], ur = r.v[A];
    // p + 0 = p for every p but -0, whose sound speed is zero either way
    const double cl = o.root(o.over(g * (stiff ? l.p + pinf : l.p), l.ro));
    const double cr = o.root(o.over(g * (stiff ? r.p + pinf : r.p), r.ro));
    const double hl = o.over(UL[4] + l.p, l.ro);
    const double hr = o.over(UR[4] + r.p, r.ro);
    const double sl = o.root(rl), sr = o.root(rr);
    const typename O::Div ss = o.divisor(sl + sr);
    const double wl = o.over(sl, ss), wr = o.over(sr, ss);
    double vt[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int b = 0; b < NC; ++b) vt[b] = wl * l.v[b] + wr * r.v[b];
    const double ut = vt[A];
    const double ht = wl * hl + wr * hr;
    const double ct = o.root(ph.gm1 * (ht - o.half(dot<NC>(vt, vt))));
    const double a0 = ul - cl, a1 = ut - ct, b0 = ur + cr, b1 = ut + ct;
    const double SL = o.min(a0, a1), SR = o.max(b0, b1);
    const double lam = o.max(dabs(SL), dabs(SR));
    const double ml = rl * (SL - ul), mr = rr * (SR - ur);
    const double sstar = o.div(r.p - l.p + ul * ml - ur * mr, ml - mr);
    // F_L if S_L >= 0, F_R if S_R <= 0, else the star state on the side of S*
    const bool supl = o.ge0(SL), supr = !supl && o.le0(SR);
    const bool left = supl || (!supr && o.ge0(sstar));
    double U[NV], v[3];
#pragma unroll
    for (int i = 0; i < NV; ++i) U[i] = left ? UL[i] : UR[i];
#pragma unroll
    for (int b = 0; b < 3; ++b) v[b] = left ? l.v[b] : r.v[b];
    const double p = left ? l.p : r.p;
    const double rvn = U[0] * v[A];
    flux[0] = rvn;
#pragma unroll
    for (int b = 0; b < 3; ++b) {
        flux[1 + b] = b < NC ? rvn * v[b] : 0.0;
        if (b == A) flux[1 + b] = flux[1 + b] + p;
    }
    flux[4] = v[A] * (U[4] + p);
    if (!supl && !supr) {
        const double S = left ? SL : SR, m = left ? ml : mr;
        const double coef = o.div(m, S - sstar);
        const double Er = o.over(U[4], left ? l.ro : r.ro);
        double us[NV];
        us[0] = coef;
#pragma unroll
        for (int b = 0; b < 3; ++b) us[1 + b] = b < NC ? coef * (b == A ? sstar : v[b]) : 0.0;
        us[4] = coef * (Er + (sstar - v[A]) * (sstar + o.div(p, m)));
#pragma unroll
        for (int i = 0; i < NV; ++i)
            if (i < 1 + NC || i == 4) flux[i] = flux[i] + S * (us[i] - U[i]);
    }
    return lam;
}

// Exact (Godunov) flux, GodunovSolverPerfectGasEOS::ComputeFlux
// (GodunovSolverPerfectGasEOS.h:266-430), ideal gas.  p* solves
// fL(p) + fR(p) + (uR - uL) = 0 (f1/f2, :56-96).  The reference minimises the
// square of that function with alglib's Levenberg-Marquardt (stopping at a
// gradient below 1e-10, :143-187); here a bounded Newton-Raphson iteration
// on the root with the analytic derivative (Toro, sec. 4.3.1) from the
// primitive-variable guess (Toro eq. 4.47), to a relative change below 1e-14.
// Everything after p* keeps the reference's steps and operation order.
__device__ __forceinline__ double god_f(double g, double rk, double pk, double p) {
    double res;
    if (p > pk) {
        const double A = 2 / ((g + 1.0) * rk);
        const double B = pk * (g - 1.0) / (g + 1.0);
        res = (p - pk) * sqrt(A / (p + B));
    } else {
        const double a = sqrt(g * pk / rk);
        res = pow(p / pk, (g - 1.0) / (2 * g)) - 1.0;
        res *= 2 * a / (g - 1.0);
    }
    return res;
}

__device__ __forceinline__ double god_df(double g, double rk, double pk, double p) {
    if (p > pk) {
        const double A = 2 / ((g + 1.0) * rk);
        const double B = pk * (g - 1.0) / (g + 1.0);
        return sqrt(A / (B + p)) * (1.0 - (p - pk) / (2.0 * (B + p)));
    }
    return pow(p / pk, -(g + 1.0) / (2.0 * g)) / (rk * sqrt(g * pk / rk));
}

// Returns false when 60 iterations do not converge (the caller flags it).
__device__ bool god_pstar(double g, double rl, double ul, double pl, double rr, double ur, double pr, double& ps) {
    const double al = sqrt(g * pl / rl), ar = sqrt(g * pr / rr);
    const double du = ur - ul;
    // both pressure functions are finite above lo (a side with a negative
    // reconstructed pressure is on its shock branch, which needs p + B > 0)
    double lo = 0.0;
    if (pl < 0) lo = fmax(lo, -pl * (g - 1.0) / (g + 1.0));
    if (pr < 0) lo = fmax(lo, -pr * (g - 1.0) / (g + 1.0));
    const double floor_p = lo + 1e-12 * (fabs(pl) + fabs(pr));
    double p = 0.5 * (pl + pr) - 0.125 * du * (rl + rr) * (al + ar);
    if (!(p > floor_p)) p = 0.5 * (pl + pr);
    if (!(p > floor_p)) p = 2.0 * floor_p;
    for (int it = 0; it < 60; ++it) {
        const double f = god_f(g, rl, pl, p) + god_f(g, rr, pr, p) + du;
        const double d = god_df(g, rl, pl, p) + god_df(g, rr, pr, p);
        double pn = p - f / d;
        if (!(pn > floor_p)) pn = floor_p;
        const double ch = 2.0 * fabs(pn - p) / (pn + p);
        p = pn;
        if (ch < 1e-14) { ps = p; return true; }
    }
    ps = p;
    return false;
}

template <int A>
__device__ double godunov_flux(const Phys& ph, const double UL[NV], const double UR[NV], double flux[NV],
                               bool& converged) {
    const double g = ph.gamma;
    const double roL = UL[0], roR = UR[0];
    const double velL[3] = {UL[1] / UL[0], UL[2] / UL[0], UL[3] / UL[0]};
    const double velR[3] = {UR[1] / UR[0], UR[2] / UR[0], UR[3] / UR[0]};
    // GetPressure (:17-25)
    const double pL =
        (g - 1.0) * roL * (UL[4] / roL - (velL[0] * velL[0] + velL[1] * velL[1] + velL[2] * velL[2]) / 2.0);
    const double pR =
        (g - 1.0) * roR * (UR[4] / roR - (velR[0] * velR[0] + velR[1] * velR[1] + velR[2] * velR[2]) / 2.0);
    const double uL = velL[A], uR = velR[A];
    // ComputeStarVariables (:143-264)
    double pStar;
    converged = god_pstar(g, roL, uL, pL, roR, uR, pR, pStar);
    const double uStar = 0.5 * (uL + uR) + 0.5 * (god_f(g, roR, pR, pStar) - god_f(g, roL, pL, pStar));
    const double C = (g - 1.0) / (g + 1.0);
    double maxs = 0, roStarL, roStarR, SL = 0, SHL = 0, STL = 0, SR = 0, SHR = 0, STR = 0;
    bool shockL, shockR;
    const double pRatioL = pStar / pL, aL = sqrt(g * pL / roL);
    if (pStar > pL) {
        shockL = true;
        roStarL = pRatioL + C;
        roStarL /= C * pRatioL + 1.0;
        roStarL *= roL;
        SL = sqrt((g + 1) * pRatioL / (2 * g) + (g - 1) / (2 * g));
        SL = uL - aL * SL;
        maxs = fmax(maxs, fabs(SL));
    } else {
        shockL = false;
        roStarL = roL * pow(pRatioL, 1.0 / g);
        SHL = uL - aL;
        const double aStarL = aL * pow(pRatioL, (g - 1) / (2 * g));
        STL = uStar - aStarL;
        maxs = fmax(maxs, fabs(SHL));
    }
    const double pRatioR = pStar / pR, aR = sqrt(g * pR / roR);
    if (pStar > pR) {
        shockR = true;
        roStarR = pRatioR + C;
        roStarR /= C * pRatioR + 1.0;
        roStarR *= roR;
        SR = sqrt((g + 1) * pRatioR / (2 * g) + (g - 1) / (2 * g));
        SR = uR + aR * SR;
        maxs = fmax(maxs, fabs(SR));
    } else {
        shockR = false;
        roStarR = roR * pow(pRatioR, 1.0 / g);
        SHR = uR + aR;
        const double aStarR = aR * pow(pRatioR, (g - 1) / (2 * g));
        STR = uStar + aStarR;
        maxs = fmax(maxs, fabs(SHR));
    }
    // sampling at S = x/t = 0 (:299-393)
    const double S = 0;
    double ro, u, p;
    const double* vel;
    if (uStar >= S) {
        vel = velL;
        if (shockL) {
            if (SL >= S) { ro = roL; u = uL; p = pL; }
            else { ro = roStarL; u = uStar; p = pStar; }
        } else if (SHL > S) {
            ro = roL; u = uL; p = pL;
        } else if (S > STL) {
            ro = roStarL; u = uStar; p = pStar;
        } else {
            const double aL2 = sqrt(g * pL / roL);
            const double CL = 2.0 / (g + 1) + (g - 1) * (uL - S) / ((g + 1) * aL2);
            const double CLRo = pow(CL, 2.0 / (g - 1));
            const double CLP = pow(CL, 2.0 * g / (g - 1));
            ro = CLRo * roL;
            u = aL2 + 0.5 * (g - 1) * uL + S;
            u *= 2 / (g + 1);
            p = CLP * pL;
        }
    } else {
        vel = velR;
        if (shockR) {
            if (SR <= S) { ro = roR; u = uR; p = pR; }
            else { ro = roStarR; u = uStar; p = pStar; }
        } else if (SHR < S) {
            ro = roR; u = uR; p = pR;
        } else if (S < STR) {
            ro = roStarR; u = uStar; p = pStar;
        } else {
            const double aR2 = sqrt(g * pR / roR);
            const double CR = 2.0 / (g + 1) - (g - 1) * (uR - S) / ((g + 1) * aR2);
            const double CRRo = pow(CR, 2.0 / (g - 1));
            const double CRP = pow(CR, 2.0 * g / (g - 1));
            ro = CRRo * roR;
            u = -aR2 + 0.5 * (g - 1) * uR + S;
            u *= 2 / (g + 1);
            p = CRP * pR;
        }
    }
    // face state (:396-404): normal velocity u, tangential from the upwind side
    double Vf[3];
#pragma unroll
    for (int b = 0; b < 3; ++b) Vf[b] = (b == A) ? vel[b] + (u - vel[A]) : vel[b];
    double Uf[NV];
    Uf[0] = ro;
    Uf[1] = ro * Vf[0];
    Uf[2] = ro * Vf[1];
    Uf[3] = ro * Vf[2];
    Uf[4] = ro * (p / (ro * (g - 1.0)) + 0.5 * (Vf[0] * Vf[0] + Vf[1] * Vf[1] + Vf[2] * Vf[2]));
    // F(Uface, n) (:28-46)
    {
        const double r = Uf[0];
        const double vx = Uf[1] / r, vy = Uf[2] / r, vz = Uf[3] / r;
        const double roE = Uf[4];
        const double pp = (g - 1.0) * (roE - r * (vx * vx + vy * vy + vz * vz) / 2.0);
        const double v3[3] = {vx, vy, vz};
        const double vn = v3[A];
        flux[0] = r * vn;
#pragma unroll
        for (int b = 0; b < 3; ++b) flux[1 + b] = (b == A) ? r * vn * v3[b] + pp : r * vn * v3[b];
        flux[4] = vn * (roE + pp);
    }
    return maxs;
}

// ---------------------------------------------------------------------------
// Kernels
// ---------------------------------------------------------------------------

// Transverse (p,q) -> (i,j,k) for a line along axis A.
template <int A>
__device__ __forceinline__ void line_cell(int p, int q, int s, int& i, int& j, int& k) {
    if (A == 0) { i = s; j = p; k = q; }
    else if (A == 1) { i = p; j = s; k = q; }
    else { i = p; j = q; k = s; }
}

template <int A>
__global__ void k_ghost(PlainBufs b, Phys ph) {
    if (b.ctl->stop_req) return;
    const Layout& L = b.L;
    const int n1 = (A == 0) ? L.ny : L.nx;
    const int n2 = (A == 2) ? L.ny : L.nz;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n1 * n2) return;
    const int p = t % n1, q = t / n1;
    int i, j, k;
    line_cell<A>(p, q, 0, i, j, k);
    const long long c0 = L.at(i, j, k);
    const long long st = L.stride(A);
    const int n = L.n(A);
    double* U = b.U;
    if (ph.periodic[A]) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            double* u = U + vidx(L, v) + c0;
            u[-1 * st] = u[(long long)(n - 1) * st];
            u[(long long)n * st] = u[0];
            u[-2 * st] = u[(long long)(n - 2) * st];
            u[(long long)(n + 1) * st] = u[st];
        }
        return;
    }
    double in[NV], out[NV];
    // the BC of this row's boundary face on each side (its marker, if the
    // side is position-dependent: the same one for both ghost layers)
    const int idl = bc_id(ph.bc.mark, 2 * A, face_index(2 * A, i, j, k, L.nx, L.ny));
    const int idr = bc_id(ph.bc.mark, 2 * A + 1, face_index(2 * A + 1, i, j, k, L.nx, L.ny));
    // left side ghosts mirror cells 0 and 1; right side mirror n-1 and n-2
    // (ComputeDummyCellValues, kernel.h:731-765); faceNormalL on both sides.
    for (int layer = 1; layer <= GHOST; ++layer) {
#pragma unroll
        for (int v = 0; v < NV; ++v) in[v] = U[vidx(L, v) + c0 + (long long)(layer - 1) * st];
        bc_values(ph, idl, A, -1.0, in, out);
#pragma unroll
        for (int v = 0; v < NV; ++v) U[vidx(L, v) + c0 - (long long)layer * st] = out[v];
#pragma unroll
        for (int v = 0; v < NV; ++v) in[v] = U[vidx(L, v) + c0 + (long long)(n - layer) * st];
        bc_values(ph, idr, A, -1.0, in, out);
#pragma unroll
        for (int v = 0; v < NV; ++v) U[vidx(L, v) + c0 + (long long)(n - 1 + layer) * st] = out[v];
    }
}


// ---------------------------------------------------------------------------
// Viscous part (ExplicitRungeKuttaFVM.h:81-874), FP64 like the rest of the path
// ---------------------------------------------------------------------------

// Velocity component d of cell c (VariablesTransition.h:18-36).
__device__ __forceinline__ double velc(const PlainBufs& b, long long c, int d) {
    return b.U[vidx(b.L, 1 + d) + c] / b.U[vidx(b.L, 0) + c];
}

__device__ __forceinline__ double vgrad(const PlainBufs& b, long long c, int d, int e) {
    return b.VG[vidx(b.L, 3 * d + e) + c];
}

// Central-difference gradients of the three velocity components in every
// interior cell (Kernel::ComputeGradientNonUniformStructured, kernel.h:918-938).
__global__ void k_vgrad(PlainBufs b, Phys ph) {
    if (b.ctl->stop_req) return;
    const Layout& L = b.L;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y, k = blockIdx.z;
    if (i >= L.nx) return;
    const long long c = L.at(i, j, k);
    const int nd = ph.nd;
    for (int d = 0; d < 3; ++d) {
        const double dux = velc(b, c + L.stride(0), d) - velc(b, c - L.stride(0), d);
        const double gx = dux / (b.cx[0][i + 1 + L.gx] - b.cx[0][i - 1 + L.gx]);
        double gy = 0.0, gz = 0.0;
        if (nd > 1) {
            const double duy = velc(b, c + L.stride(1), d) - velc(b, c - L.stride(1), d);
            gy = duy / (b.cx[1][j + 1 + L.gy] - b.cx[1][j - 1 + L.gy]);
        }
        if (nd > 2) {
            const double duz = velc(b, c + L.stride(2), d) - velc(b, c - L.stride(2), d);
            gz = duz / (b.cx[2][k + 1 + L.gz] - b.cx[2][k - 1 + L.gz]);
        }
        b.VG[vidx(L, 3 * d) + c] = gx;
        b.VG[vidx(L, 3 * d + 1) + c] = gy;
        b.VG[vidx(L, 3 * d + 2) + c] = gz;
    }
}

__device__ __forceinline__ double det3(double a00, double a01, double a02, double a10, double a11, double a12,
                                       double a20, double a21, double a22) {
    return a00 * (a11 * a22 - a12 * a21) - a01 * (a10 * a22 - a12 * a20) + a02 * (a10 * a21 - a11 * a20);
}

// Least-squares gradient of GradientComputer::ExecuteByLeastSquares
// (GradientComputer.h:20-52) by the normal equations (A^T A) g = A^T rhs and
// Cramer's rule; the reference uses Eigen's JacobiSVD, which agrees to
// rounding.
__device__ void ls_gradient(int nd, int m, const double (*A)[3], const double* rhs, double* g) {
    double M[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}, bb[3] = {0, 0, 0};
    for (int r = 0; r < m; ++r)
        for (int a = 0; a < nd; ++a) {
            bb[a] += A[r][a] * rhs[r];
            for (int e = 0; e < nd; ++e) M[a][e] += A[r][a] * A[r][e];
        }
    g[0] = g[1] = g[2] = 0.0;
    if (nd == 1) {
        g[0] = bb[0] / M[0][0];
    } else if (nd == 2) {
        const double det = M[0][0] * M[1][1] - M[0][1] * M[1][0];
        g[0] = (bb[0] * M[1][1] - M[0][1] * bb[1]) / det;
        g[1] = (M[0][0] * bb[1] - bb[0] * M[1][0]) / det;
    } else {
        const double det = det3(M[0][0], M[0][1], M[0][2], M[1][0], M[1][1], M[1][2], M[2][0], M[2][1], M[2][2]);
        g[0] = det3(bb[0], M[0][1], M[0][2], bb[1], M[1][1], M[1][2], bb[2], M[2][1], M[2][2]) / det;
        g[1] = det3(M[0][0], bb[0], M[0][2], M[1][0], bb[1], M[1][2], M[2][0], bb[2], M[2][2]) / det;
        g[2] = det3(M[0][0], M[0][1], bb[0], M[1][0], M[1][1], bb[1], M[2][0], M[2][1], bb[2]) / det;
    }
}

// Ghost gradients beyond boundary cell (i, j, k) on side `side` of axis A
// (ComputeDummyCellGradients, ExplicitRungeKuttaFVM.h:318-680): least-squares
// gradient at the face centre from the face value (mean of the cell and its
// BC image, BCGeneral::getFaceValues) and the stencil of
// Stencil::InternalBorderStencil plus the ghost cell; ghost = 2 g_face - g_cell.
template <int A>
__device__ void dummy_gradient(const PlainBufs& b, const Phys& ph, int side, int i, int j, int k) {
    const Layout& L = b.L;
    const int nd = ph.nd;
    const int ix[3] = {i, j, k};
    const int go[3] = {L.gx, L.gy, L.gz};
    const long long inner = L.at(i, j, k);
    const long long ghost = inner + (side ? L.stride(A) : -L.stride(A));
    double fc[3] = {b.cx[0][i + L.gx], b.cx[1][j + L.gy], b.cx[2][k + L.gz]};
    const double xa = b.cx[A][ix[A] + go[A]], ha = b.ch[A][ix[A] + go[A]];
    fc[A] = side ? xa + 0.5 * ha : xa - 0.5 * ha;
    double Vin[NV], du[NV], Vf[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) Vin[v] = b.U[vidx(L, v) + inner];
    bc_values(ph, bc_id(ph.bc.mark, 2 * A + side, face_index(2 * A + side, i, j, k, L.nx, L.ny)), A,
              side ? 1.0 : -1.0, Vin, du);
#pragma unroll
    for (int v = 0; v < NV; ++v) Vf[v] = 0.5 * (Vin[v] + du[v]);
    // stencil: the cell, its neighbours along the other active axes (+ then -), the ghost
    int st[7][3];
    int m = 0;
    st[m][0] = i; st[m][1] = j; st[m][2] = k; ++m;
    for (int a = 0; a < nd; ++a) {
        if (a == A) continue;
        for (int sg = 1; sg >= -1; sg -= 2) {
            st[m][0] = i; st[m][1] = j; st[m][2] = k;
            st[m][a] += sg;
            ++m;
        }
    }
    st[m][0] = i; st[m][1] = j; st[m][2] = k;
    st[m][A] += side ? 1 : -1;
    ++m;
    double Am[7][3], rhs[7], g[3];
    for (int r = 0; r < m; ++r) {
        Am[r][0] = fc[0] - b.cx[0][st[r][0] + L.gx];
        Am[r][1] = fc[1] - b.cx[1][st[r][1] + L.gy];
        Am[r][2] = fc[2] - b.cx[2][st[r][2] + L.gz];
    }
    for (int d = 0; d < 3; ++d) {
        const double value = Vf[1 + d] / Vf[0];
        for (int r = 0; r < m; ++r) rhs[r] = value - velc(b, L.at(st[r][0], st[r][1], st[r][2]), d);
        ls_gradient(nd, m, Am, rhs, g);
        for (int e = 0; e < 3; ++e) b.VG[vidx(L, 3 * d + e) + ghost] = 2.0 * g[e] - vgrad(b, inner, d, e);
    }
}

// Gradients of the first ghost layer along axis A: the opposite interior
// cell's on a periodic axis (ExchangeGradients on one rank,
// ExplicitRungeKuttaFVM.h:136-316), least squares otherwise.
template <int A>
__global__ void k_vgrad_bc(PlainBufs b, Phys ph) {
    if (b.ctl->stop_req) return;
    const Layout& L = b.L;
    const int n1 = (A == 0) ? L.ny : L.nx;
    const int n2 = (A == 2) ? L.ny : L.nz;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n1 * n2) return;
    const int p = t % n1, q = t / n1;
    int i, j, k;
    line_cell<A>(p, q, 0, i, j, k);
    const long long c0 = L.at(i, j, k);
    const long long st = L.stride(A);
    const int n = L.n(A);
    if (ph.periodic[A]) {
        for (int pl = 0; pl < 9; ++pl) {
            double* g = b.VG + vidx(L, pl) + c0;
            g[(long long)n * st] = g[0];
            g[-st] = g[(long long)(n - 1) * st];
        }
        return;
    }
    int ih = i, jh = j, kh = k;
    if (A == 0) ih = n - 1; else if (A == 1) jh = n - 1; else kh = n - 1;
    dummy_gradient<A>(b, ph, 0, i, j, k);
    dummy_gradient<A>(b, ph, 1, ih, jh, kh);
}

// Viscous flux of the face along axis A between cells cl and cr, s the
// index of cr along A (ComputeViscousFluxes, ExplicitRungeKuttaFVM.h:683-874).
template <int A>
__device__ void visc_flux(const PlainBufs& b, const Phys& ph, long long cl, long long cr, int s, double fv[NV]) {
    const Layout& L = b.L;
    const int g0 = (A == 0) ? L.gx : (A == 1 ? L.gy : L.gz);
    const double dx = b.cx[A][s + g0] - b.cx[A][s - 1 + g0];
    const double l = b.ch[A][s - 1 + g0] / dx;
    const double r = b.ch[A][s + g0] / dx;
    double D[3][3], uu[3];
    for (int d = 0; d < 3; ++d) {
        for (int e = 0; e < 3; ++e) D[d][e] = 0.5 * (r * vgrad(b, cl, d, e) + l * vgrad(b, cr, d, e));
        D[d][A] = (velc(b, cr, d) - velc(b, cl, d)) / dx;
    }
    for (int d = 0; d < 3; ++d) uu[d] = 0.5 * (l * velc(b, cr, d) + r * velc(b, cl, d));
    const double mu = ph.visc;
    const double sv = (-2.0 / 3.0) * mu;
    const double td = sv * (D[0][0] + D[1][1] + D[2][2]);
    fv[0] = 0.0;
    if (A == 0) {
        const double txx = td + 2 * mu * D[0][0];
        const double txy = mu * (D[0][1] + D[1][0]);
        const double txz = mu * (D[0][2] + D[2][0]);
        fv[1] = txx; fv[2] = txy; fv[3] = txz;
        fv[4] = uu[0] * txx + uu[1] * txy + uu[2] * txz;
    } else if (A == 1) {
        const double tyy = td + 2 * mu * D[1][1];
        const double txy = mu * (D[0][1] + D[1][0]);
        const double tyz = mu * (D[1][2] + D[2][1]);
        fv[1] = txy; fv[2] = tyy; fv[3] = tyz;
        fv[4] = uu[0] * txy + uu[1] * tyy + uu[2] * tyz;
    } else {
        const double tzz = td + 2 * mu * D[2][2];
        const double txz = mu * (D[0][2] + D[2][0]);
        const double tyz = mu * (D[1][2] + D[2][1]);
        fv[1] = txz; fv[2] = tyz; fv[3] = tzz;
        fv[4] = uu[0] * txz + uu[1] * tyz + uu[2] * tzz;
    }
}

// Venkatakrishnan l-function (Limiters.h:102-115): um, ui, d2 already divided
// by un = (umax - umin) / 2.
template <class O>
__device__ __forceinline__ double venkat(double um, double ui, double d2, double eps2, O& o) {
    const double dm = um - ui;
    return o.div((dm * dm + eps2) + 2 * d2 * dm, dm * dm + 2 * d2 * d2 + dm * d2 + eps2);
}

// Reconstruction kinds (the limiter choice folded in).
enum { P_LINEAR = 1, P_ENO2 = 2, P_LIM_BJ = 3, P_LIM_VK = 4 };

// a1 / d1 < a2 / d2 as rounded quotients, for ratios too close for the FP32
// estimates in recon_var.
__device__ __noinline__ bool ratio_less(double a1, double d1, double a2, double d2) { return a1 / d1 < a2 / d2; }

// FP32 estimate (truncated, relative error 2^-23) of a positive double with
// an exponent field in [897, 1150].
__device__ __forceinline__ float est32(u64 b) { return __uint_as_float((unsigned)(b >> 29) - 0xC0000000u); }
__device__ __forceinline__ bool est32_ok(u64 b) { return (unsigned)(b >> 52) - 897u < 254u; }

// Slopes (Linear2PointsStencil.h:147-178 or ENO2PointsStencil.h:202-239) and,
// for Linear2psLim, the limiter (Linear2psLim.h:305-374, Limiters.h:28-119) of
// variable v in cell c.  d: divisors of the slopes (ENO2: left and right);
// hs: half cell sizes.  With b.fold the stored value is the projection
// lim * (slope * h/2) to the high face (its negative goes to the low face),
// otherwise slope and limiter.
template <int ND, int KIND, class O>
__device__ __forceinline__ void recon_var(const PlainBufs& b, int v, long long c, const typename O::Div* d,
                                          const double* hs, double eps2, O& o) {
    const Layout& L = b.L;
    const double* U = b.U + vidx(L, v) + c;
    const double val = U[0];
    double nm[ND], np[ND], g[ND], gs[ND];
#pragma unroll
    for (int a = 0; a < ND; ++a) {
        const long long st = L.stride(a);
        nm[a] = U[-st];
        np[a] = U[st];
    }
    // the largest and smallest of the cell and its neighbours
    long long kmax = dkey(val), kmin = kmax;
    double umax = val, umin = val;
    if (KIND == P_LIM_BJ || KIND == P_LIM_VK) {
#pragma unroll
        for (int f = 0; f < 2 * ND; ++f) {
            const double vn = (f & 1) ? np[f >> 1] : nm[f >> 1];
            const long long kv = dkey(vn);
            if (kmax < kv) { umax = vn; kmax = kv; }
            if (kmin > kv) { umin = vn; kmin = kv; }
        }
        // a constant neighbourhood (finite): slopes and projections are zero
        if (kmax == kmin && (__double2hiint(val) & 0x7FF00000) != 0x7FF00000) {
#pragma unroll
            for (int a = 0; a < ND; ++a) b.G[vidx(L, a * NV + v) + c] = 0.0;
            if (!b.fold) b.Lim[vidx(L, v) + c] = 1.0;
            return;
        }
    }
#pragma unroll
    for (int a = 0; a < ND; ++a) {
        if (KIND == P_ENO2) {
            const double gl = o.over(val - nm[a], d[2 * a]);
            const double gr = o.over(np[a] - val, d[2 * a + 1]);
            g[a] = dabs_lt(gl, gr) ? gl : gr;
        } else {
            g[a] = o.over(np[a] - nm[a], d[a]);
        }
        gs[a] = g[a] * hs[a];
    }
    double lmin = 1.0;
    if (KIND == P_LIM_BJ || KIND == P_LIM_VK) {
        // umax - umin < 3 DBL_MIN: for unequal values of magnitude 2^-960 or
        // more the difference is larger, no subtraction needed
        const bool big = ((__double2hiint(umax) & 0x7FF00000) >= 0x03F00000) ||
                         ((__double2hiint(umin) & 0x7FF00000) >= 0x03F00000);
        const bool flat = kmax == kmin || (!big && dlt(umax - umin, 3.0 * 2.2250738585072014e-308));
        if (!flat) {
            // differences (SampleSolution(+-h/2) - val) to the 2 ND faces
            const double am = umax - val, an = umin - val;
            if constexpr (KIND == P_LIM_VK) {
                const typename O::Div un = o.divisor(o.half(umax - umin));
                const double xm = o.over(umax, un), xn = o.over(umin, un), xu = o.over(val, un);
#pragma unroll
                for (int f = 0; f < 2 * ND; ++f) {
                    const double s = (f & 1) ? gs[f >> 1] : -gs[f >> 1];
                    const double d2 = (val + s) - val;
                    if (dzero(d2)) continue;
                    const double lv = venkat(dpos(d2) ? xm : xn, xu, o.over(d2, un), eps2, o);
                    if (o.lt(lv, lmin)) lmin = lv;
                }
            } else if constexpr (std::is_same_v<O, Plain>) {
#pragma unroll
                for (int f = 0; f < 2 * ND; ++f) {
                    const double s = (f & 1) ? gs[f >> 1] : -gs[f >> 1];
                    const double d2 = (val + s) - val;
                    double lv = 1.0;
                    if (d2 > 0) { const double r = am / d2; lv = r < 1.0 ? r : 1.0; }
                    if (d2 < 0) { const double r = an / d2; lv = r < 1.0 ? r : 1.0; }
                    if (lv < lmin) lmin = lv;
                }
            } else {
                // The limiter is the smallest of the rounded ratios a / d2
                // (a = umax - val or umin - val) below 1.  Rounding is
                // monotone, so only the smallest ratio is divided out: it is
                // found on FP32 estimates (error < 2^-20), and estimates
                // closer than 2^-18 are settled by their quotients.  A ratio
                // with |a| >= |d2| rounds to 1 or more and is dropped.
                const u64 ap = (u64)__double_as_longlong(am), aq = (u64)__double_as_longlong(dabs(an));
                u64 ba = 0, bd = 0;
                float br = 2.0f;
#pragma unroll
                for (int f = 0; f < 2 * ND; ++f) {
                    const double s = (f & 1) ? gs[f >> 1] : -gs[f >> 1];
                    const double d2 = (val + s) - val;
                    const u64 ad = (u64)__double_as_longlong(dabs(d2));
                    const u64 aa = __double2hiint(d2) < 0 ? aq : ap;
                    if (aa < ad) {
                        o.bad |= !est32_ok(ad);
                        const float r = est32_ok(aa) ? __fdividef(est32(aa), est32(ad)) : 0.0f;
                        bool take = r < br * (1.0f - 3.8e-6f);
                        // (a zero or the same ratio cannot be undercut: local extrema,
                        // and states that differ by a few ulps)
                        if (!take && r <= br * (1.0f + 3.8e-6f) && ba != 0 && !(aa == ba && ad == bd))
                            take = ratio_less(__longlong_as_double(aa), __longlong_as_double(ad),
                                              __longlong_as_double(ba), __longlong_as_double(bd));
                        if (take) { ba = aa; bd = ad; br = r; }
                    }
                }
                if (br < 2.0f) lmin = o.div(__longlong_as_double(ba), __longlong_as_double(bd));
            }
        }
    }
    if (b.fold) {
#pragma unroll
        for (int a = 0; a < ND; ++a)
            b.G[vidx(L, a * NV + v) + c] = (KIND == P_LIM_BJ || KIND == P_LIM_VK) ? lmin * gs[a] : gs[a];
    } else {
#pragma unroll
        for (int a = 0; a < ND; ++a) b.G[vidx(L, a * NV + v) + c] = g[a];
        if (KIND == P_LIM_BJ || KIND == P_LIM_VK) b.Lim[vidx(L, v) + c] = lmin;
    }
}

template <int ND, int KIND, class O>
__device__ __forceinline__ void recon_cell(const PlainBufs& b, int i, int j, int k, O& o) {
    const Layout& L = b.L;
    const long long c = L.at(i, j, k);
    const int ix[3] = {i, j, k};
    typename O::Div d[KIND == P_ENO2 ? 2 * ND : ND];
    double hs[ND];
#pragma unroll
    for (int a = 0; a < ND; ++a) {
        const int at = ix[a] + (a == 0 ? L.gx : (a == 1 ? L.gy : L.gz));
        const double* X = b.cx[a];
        if (KIND == P_ENO2) {
            d[2 * a] = o.divisor(X[at] - X[at - 1]);
            d[2 * a + 1] = o.divisor(X[at + 1] - X[at]);
        } else {
            d[a] = o.divisor(X[at + 1] - X[at - 1]);
        }
        hs[a] = o.half(b.ch[a][at]);
    }
    const double eps2 = KIND == P_LIM_VK ? b.eps2[c] : 0.0;
#pragma unroll 1
    for (int v = 0; v < NV; ++v) recon_var<ND, KIND, O>(b, v, c, d, hs, eps2, o);
}

template <int ND, int KIND>
__device__ __noinline__ void recon_plain(const PlainBufs& b, int i, int j, int k) {
    Plain o;
    recon_cell<ND, KIND, Plain>(b, i, j, k, o);
}

// Cell t of the interior in storage order (one flat index over all rows: no
// warp holds the end of a row alone).
__device__ __forceinline__ void cell_of(const Layout& L, unsigned t, int& i, int& j, int& k) {
    const unsigned row = t / (unsigned)L.nx;
    i = (int)(t - row * (unsigned)L.nx);
    k = (int)(row / (unsigned)L.ny);
    j = (int)(row - (unsigned)k * (unsigned)L.ny);
}

// Per interior cell: slopes and limiter (ComputeSolutionReconstruction).
template <int ND, int KIND>
__global__ void __launch_bounds__(kPlainBlock) k_recon(const __grid_constant__ PlainBufs b) {
    if (b.ctl->stop_req) return;
    const unsigned t = blockIdx.x * kPlainBlock + threadIdx.x;
    if (t >= (unsigned)b.L.cells()) return;
    int i, j, k;
    cell_of(b.L, t, i, j, k);
    Fast o;
    recon_cell<ND, KIND, Fast>(b, i, j, k, o);
    if (o.bad) recon_plain<ND, KIND>(b, i, j, k);
}

__device__ __forceinline__ double face_area(const PlainBufs& b, int nd, int a, int i, int j, int k) {
    const Layout& L = b.L;
    const double hx = b.ch[0][i + L.gx], hy = b.ch[1][j + L.gy], hz = b.ch[2][k + L.gz];
    if (a == 0) return nd == 1 ? 1.0 : (nd == 2 ? hy : hy * hz);
    if (a == 1) return nd == 2 ? hx : hx * hz;
    return hx * hy;
}

// Face-centred sample of a cell's reconstruction (SampleSolution) at its high
// (HI) or low face along axis a; h is the cell size the reference samples
// with.
template <bool HI>
__device__ __forceinline__ void sample(const PlainBufs& b, const Phys& ph, long long c, int a, double h,
                                       double out[NV]) {
    const Layout& L = b.L;
#pragma unroll
    for (int v = 0; v < NV; ++v) out[v] = b.U[vidx(L, v) + c];
    if (ph.recon == TS_RECON_PIECEWISE_CONSTANT) return;
    if (b.fold) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const double d = b.G[vidx(L, a * NV + v) + c];
            out[v] = HI ? out[v] + d : out[v] - d;
        }
        return;
    }
    const double s = (HI ? 0.5 : -0.5) * h;
    if (ph.recon == TS_RECON_LINEAR_2POINTS_LIMITED) {
#pragma unroll
        for (int v = 0; v < NV; ++v) out[v] = out[v] + b.Lim[vidx(L, v) + c] * (b.G[vidx(L, a * NV + v) + c] * s);
    } else {
#pragma unroll
        for (int v = 0; v < NV; ++v) out[v] = out[v] + b.G[vidx(L, a * NV + v) + c] * s;
    }
}

// The Riemann flux and eigenvalue of one face.  1D and 2D problems whose
// transverse momentum is zero in every state of the warp take the instance
// without its terms.
template <int A, int SOLVER, int NC, class O>
__device__ __forceinline__ double riemann(const Phys& ph, const double UL[NV], const double UR[NV], double F[NV], O& o) {
    if (SOLVER == TS_RS_HLLC) return hllc_flux<A, NC, O>(ph, UL, UR, F, o);
    return roe_flux<A, NC, O>(ph, UL, UR, F, o);
}

template <int A, int SOLVER>
__device__ __noinline__ double riemann_plain(const Phys& ph, const double* UL, const double* UR, double* F) {
    Plain o;
    return riemann<A, SOLVER, 3, Plain>(ph, UL, UR, F, o);
}

template <int A, int ND, int SOLVER>
__device__ __forceinline__ double face_flux(const Phys& ph, const double UL[NV], const double UR[NV], double F[NV]) {
    typedef FaceArith<ND, SOLVER> O;
    O o;
    double lam;
    bool z = false;
    if (ND < 3) {
        bool mine = true;
#pragma unroll
        for (int b = ND; b < 3; ++b) mine = mine && dzero(UL[1 + b]) && dzero(UR[1 + b]);
        z = __all_sync(__activemask(), mine);
    }
    if (ND < 3 && z) lam = riemann<A, SOLVER, ND, O>(ph, UL, UR, F, o);
    else lam = riemann<A, SOLVER, 3, O>(ph, UL, UR, F, o);
    if (o.bad) {
        double l[NV], r[NV], f[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) { l[v] = UL[v]; r[v] = UR[v]; }
        lam = riemann_plain<A, SOLVER>(ph, l, r, f);
#pragma unroll
        for (int v = 0; v < NV; ++v) F[v] = f[v];
    }
    return lam;
}

// One face per thread along axis A; faces are stored at their right cell.
template <int A, int ND, int SOLVER>
__global__ void __launch_bounds__(kPlainBlock, ND == 3 ? 4 : 1) k_flux(const __grid_constant__ PlainBufs b,
                                                      const __grid_constant__ Phys ph) {
    if (b.ctl->stop_req) return;
    const Layout& L = b.L;
    // one flat index over the faces of all rows
    const unsigned t = blockIdx.x * kPlainBlock + threadIdx.x;
    const unsigned mx = L.nx + (A == 0), my = L.ny + (A == 1), mz = L.nz + (A == 2);
    const unsigned row = t / mx;
    const int i = (int)(t - row * mx), k = (int)(row / my), j = (int)(row - (unsigned)k * my);
    if (k >= (int)mz) return;
    const int s = (A == 0) ? i : (A == 1 ? j : k);
    const int n = L.n(A);
    const long long st = L.stride(A);
    const long long cf = L.at(i, j, k);  // cell to the right of the face
    const double* H = b.ch[A];
    const int g0 = (A == 0) ? L.gx : (A == 1 ? L.gy : L.gz);
    double UL[NV], UR[NV];
    if (s == 0 && !ph.periodic[A]) {
        sample<false>(b, ph, cf, A, H[s + g0], UR);
        bc_values(ph, bc_id(ph.bc.mark, 2 * A, face_index(2 * A, i, j, k, L.nx, L.ny)), A, 1.0, UR, UL);
    } else if (s == n && !ph.periodic[A]) {
        sample<true>(b, ph, cf - st, A, H[s - 1 + g0], UL);
        bc_values(ph, bc_id(ph.bc.mark, 2 * A + 1, face_index(2 * A + 1, i, j, k, L.nx, L.ny)), A, 1.0, UL, UR);
    } else {
        // A ghost reconstruction on a periodic axis is the opposite interior
        // cell's object sampled with the ghost's own h (ExchangeReconstructions).
        const long long cl = (s == 0) ? cf + (long long)(n - 1) * st : cf - st;
        const long long cr = (s == n) ? cf - (long long)n * st : cf;
        sample<true>(b, ph, cl, A, H[s - 1 + g0], UL);
        sample<false>(b, ph, cr, A, H[s + g0], UR);
    }
    double F[NV];
    double lam;
    if (SOLVER == TS_RS_GODUNOV) {
        bool ok;
        lam = godunov_flux<A>(ph, UL, UR, F, ok);
        if (!ok) atomicOr(&b.ctl->health, (unsigned)TS_HEALTH_RIEMANN);
    } else {
        lam = face_flux<A, ND, SOLVER>(ph, UL, UR, F);
    }
    // viscous flux subtracted from the convective one (ExplicitRungeKuttaFVM.h:1220-1222);
    // the cell values and gradients of the ghost cells serve the domain faces
    if (ph.viscous) {
        double fv[NV];
        visc_flux<A>(b, ph, cf - st, cf, s, fv);
#pragma unroll
        for (int v = 0; v < NV; ++v) F[v] -= fv[v];
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) b.F[A][vidx(L, v) + cf] = F[v];
    b.Lam[A][cf] = lam;
    // viscous spectral-radius term of the face for its left cell (:1239-1248),
    // Prandtl number 1, only for faces whose left cell is interior
    if (ph.visc != 0.0 && s > 0) {
        const double roFace = sqrt(UL[0] * UR[0]);
        const double t1 = 4.0 / (3.0 * roFace), t2 = ph.gamma / roFace;
        double vsr = (t1 < t2) ? t2 : t1;
        vsr *= ph.visc / 1.0;
        const double fS = face_area(b, ph.nd, A, i, j, k);
        vsr *= fS * fS;
        int il = i, jl = j, kl = k;
        if (A == 0) il -= 1; else if (A == 1) jl -= 1; else kl -= 1;
        const double Vl = b.ch[0][il + L.gx] * b.ch[1][jl + L.gy] * b.ch[2][kl + L.gz];
        vsr /= Vl;
        b.VSR[A][cf] = vsr;
    }
}

// Minimum of the warp's values of V/SR.  They are not negative (a NaN of
// either sign has a larger pattern than +inf), so they order like their bits.
__device__ __forceinline__ u64 umin64(u64 a, u64 b) { return a < b ? a : b; }
__device__ __forceinline__ u64 warp_min(u64 v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = umin64(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
constexpr u64 kInfBits = 0x7FF0000000000000ULL;

// Bits of V / sr.
__device__ __forceinline__ u64 ratio_bits(double V, double sr) {
    bool bad = false;
    double r = x64::div(V, sr, bad);
    if (bad) r = V / sr;
    return (u64)__double_as_longlong(r);
}

// Spectral radius per cell in the reference's accumulation order (x-left,
// x-right, y-left, ...), V/SR, block min by warp shuffles; the high-side
// ghost cells, whose SR is their single face term, join the min.  The last
// block to finish reduces the block minima and sets dt.
template <int ND>
__global__ void __launch_bounds__(kPlainBlock) k_dt(const __grid_constant__ PlainBufs b,
                                                    const __grid_constant__ Phys ph) {
    if (b.ctl->stop_req) return;
    const Layout& L = b.L;
    const unsigned cells = (unsigned)L.cells(), step = gridDim.x * kPlainBlock;
    u64 r = kInfBits;
    for (unsigned t = blockIdx.x * kPlainBlock + threadIdx.x; t < cells; t += step) {
        int i, j, k;
        cell_of(L, t, i, j, k);
        const long long c = L.at(i, j, k);
        const double hx = b.ch[0][i + L.gx], hy = b.ch[1][j + L.gy], hz = b.ch[2][k + L.gz];
        const double V = hx * hy * hz;
        double sr = 0.0;
        const int ix[3] = {i, j, k};
#pragma unroll
        for (int a = 0; a < ND; ++a) {
            const double fS = face_area(b, ND, a, i, j, k);
            const long long st = L.stride(a);
            const double lo = fS * b.Lam[a][c], hi = fS * b.Lam[a][c + st];
            sr = a == 0 ? lo : sr + lo;
            sr += hi;
            if (ph.visc != 0.0) sr += b.VSR[a][c + st];
            if (ix[a] == L.n(a) - 1) {
                double hg[3] = {hx, hy, hz};
                hg[a] = b.ch[a][L.n(a) + (a == 0 ? L.gx : (a == 1 ? L.gy : L.gz))];
                r = umin64(r, ratio_bits(hg[0] * hg[1] * hg[2], hi));
            }
        }
        r = umin64(r, ratio_bits(V, sr));
        if (step > cells - t) break;  // t + step would not fit 32 bits for the largest grids
    }
    __shared__ u64 wmin[kPlainBlock / 32];
    r = warp_min(r);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) wmin[wid] = r;
    __syncthreads();
    const int nblk = gridDim.x;
    __shared__ bool last;
    if (threadIdx.x == 0) {
        u64 m = wmin[0];
        for (int w = 1; w < kPlainBlock / 32; ++w) m = umin64(m, wmin[w]);
        b.partial[blockIdx.x] = __longlong_as_double((long long)m);
        __threadfence();
        last = (atomicAdd(&b.ctl->blocks_done, 1u) == (unsigned)(nblk - 1));
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    u64 m = kInfBits;
    for (int t = threadIdx.x; t < nblk; t += kPlainBlock)
        m = umin64(m, (u64)__double_as_longlong(((volatile double*)b.partial)[t]));
    m = warp_min(m);
    if (lane == 0) wmin[wid] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        m = wmin[0];
        for (int w = 1; w < kPlainBlock / 32; ++w) m = umin64(m, wmin[w]);
        const double least = __longlong_as_double((long long)m);
        Ctl* ctl = b.ctl;
        double dt = least * ph.cfl;
        if ((ctl->save_sol > 0) && (ctl->next_sol < ctl->time + dt)) dt = ctl->next_sol - ctl->time;
        if ((ctl->save_slice > 0) && (ctl->next_slice < ctl->time + dt)) dt = ctl->next_slice - ctl->time;
        ctl->dt_min_raw = least;
        ctl->dt = dt;
        for (int v = 0; v < NV; ++v) ctl->res[v] = 0.0;
        ctl->blocks_done = 0;
    }
}

// Health flags of an updated state.  The pressure test is settled in FP32
// where the pressure is a thousandth of the energy or more (the FP32 estimate
// is off by 1e-6 of the energy), and formed in FP64 otherwise.
__device__ __noinline__ unsigned int health_plain(const Phys& ph, double u0, double u1, double u2, double u3,
                                                  double u4) {
    unsigned int health = 0;
    const double ke = 0.5 * (u1 * u1 + u2 * u2 + u3 * u3) / u0;
    const double p = pressure(ph, u0, 0.0, 0.0, 0.0, u4 - ke);
    if (!(u0 == u0) || !(u4 == u4) || !(p == p)) health |= TS_HEALTH_NAN;
    if (u0 <= 0.0) health |= TS_HEALTH_NEG_DENSITY;
    if (p <= 0.0 && ph.eos == TS_EOS_IDEAL_GAS) health |= TS_HEALTH_NEG_PRESSURE;
    if (ph.eos == TS_EOS_STIFFENED_GAS && p + ph.p_inf <= 0.0) health |= TS_HEALTH_NEG_PRESSURE;
    return health;
}
// FP32 estimate of a double of either sign; false outside the normal range
// (zero gives 0).
__device__ __forceinline__ bool est32_signed(double x, float& f) {
    const u64 b = (u64)__double_as_longlong(dabs(x));
    f = est32(b);
    if (__double2hiint(x) < 0) f = -f;
    if (b < ((u64)897 << 52)) { f = 0.0f; return true; }  // below 2^-126: nothing beside the energy's tolerance
    return est32_ok(b);
}
__device__ __forceinline__ unsigned int health_of(const Phys& ph, const double u[NV]) {
    float r, m1, m2, m3, e;
    bool ok = est32_signed(u[0], r);
    ok = est32_signed(u[1], m1) && ok;
    ok = est32_signed(u[2], m2) && ok;
    ok = est32_signed(u[3], m3) && ok;
    ok = est32_signed(u[4], e) && ok;
    // p + p_inf = (g - 1) (E - kinetic - p_inf) for both equations of state
    const float pr = e - 0.5f * (m1 * m1 + m2 * m2 + m3 * m3) / r - (float)ph.p_inf;
    if (ok && r > 1e-30f && pr > 1e-3f * e && e > 1e-30f && pr < 1e37f) return 0u;
    return health_plain(ph, u[0], u[1], u[2], u[3], u[4]);
}

// U + dt (R / V) of one cell's variables; F = the face fluxes.
template <int ND, class O>
__device__ __forceinline__ void update_cell(const PlainBufs& b, const Phys& ph, int i, int j, int k, double dt,
                                            double u[NV], double nrm[NV], O& o) {
    const Layout& L = b.L;
    const long long c = L.at(i, j, k);
    const double hx = b.ch[0][i + L.gx], hy = b.ch[1][j + L.gy], hz = b.ch[2][k + L.gz];
    const double V = hx * hy * hz;
    double R[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) R[v] = 0.0;
#pragma unroll
    for (int a = 0; a < ND; ++a) {
        const double fS = face_area(b, ND, a, i, j, k);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const double* F = b.F[a] + vidx(L, v) + c;
            const double fh = F[L.stride(a)], fl = F[0];
            // equal (finite) fluxes: the difference is a zero
            if (__double_as_longlong(fh) == __double_as_longlong(fl) && (__double2hiint(fh) & 0x7FF00000) != 0x7FF00000)
                continue;
            const double d = (fh - fl) * fS;
            R[v] = a == 0 ? dneg_of(d) : R[v] - d;
        }
    }
    double uo[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) uo[v] = b.U[vidx(L, v) + c];
    // source terms after the face fluxes (ExplicitRungeKuttaFVM.h:1421-1423;
    // ProcessExternalForces and ProcessExternalAcceleration, kernel.h:941-989)
    if (ph.force || ph.accel) {
        const typename O::Div ro = o.divisor(uo[0]);
        const double vu = o.over(uo[1], ro), vv = o.over(uo[2], ro), vw = o.over(uo[3], ro);
        if (ph.force) {
            R[1] += V * ph.sigma[0];
            R[2] += V * ph.sigma[1];
            R[3] += V * ph.sigma[2];
            R[4] += (ph.sigma[0] * vu + ph.sigma[1] * vv + ph.sigma[2] * vw) * V;
        }
        if (ph.accel) {
            const double r0 = uo[0];
            R[1] += r0 * V * ph.g[0];
            R[2] += r0 * V * ph.g[1];
            R[3] += r0 * V * ph.g[2];
            R[4] += ((r0 * ph.g[0]) * vu + (r0 * ph.g[1]) * vv + (r0 * ph.g[2]) * vw) * V;
        }
    }
    const typename O::Div iv = o.divisor(V);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        u[v] = uo[v];
        nrm[v] = 0.0;
        if (dzero(R[v])) continue;
        u[v] = uo[v] + dt * o.over(R[v], iv);
        nrm[v] = V * dabs(R[v]);
    }
}
template <int ND>
__device__ __noinline__ void update_plain(const PlainBufs& b, const Phys& ph, int i, int j, int k, double dt,
                                          double* u, double* nrm) {
    Plain o;
    update_cell<ND, Plain>(b, ph, i, j, k, dt, u, nrm, o);
}

// Residual R = -sum_a (F_{a,+} - F_{a,-}) fS_a accumulated from zero in the
// reference's direction order, then U += dt*(R/V); residual norms and health.
// The last block closes the step: time += dt, iteration++ (IterationStep
// :1486-1487); under Run also the snapshot-time bookkeeping and termination
// test (kernel.h:1763-1846).
template <int ND>
__global__ void __launch_bounds__(kPlainBlock) k_update(const __grid_constant__ PlainBufs b,
                                                        const __grid_constant__ Phys ph) {
    if (b.ctl->stop_req) return;
    const Layout& L = b.L;
    const unsigned cells = (unsigned)L.cells(), step = gridDim.x * kPlainBlock;
    const double dt = b.ctl->dt;
    double sum[NV] = {0, 0, 0, 0, 0};
    unsigned int health = 0;
    for (unsigned t = blockIdx.x * kPlainBlock + threadIdx.x; t < cells; t += step) {
        int i, j, k;
        cell_of(L, t, i, j, k);
        const long long c = L.at(i, j, k);
        double u[NV], nrm[NV];
        Fast o;
        update_cell<ND, Fast>(b, ph, i, j, k, dt, u, nrm, o);
        if (o.bad) {
            double w[NV], m[NV];
            update_plain<ND>(b, ph, i, j, k, dt, w, m);
#pragma unroll
            for (int v = 0; v < NV; ++v) { u[v] = w[v]; nrm[v] = m[v]; }
        }
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            b.U[vidx(L, v) + c] = u[v];
            if (!dzero(nrm[v])) sum[v] += nrm[v];
        }
        health |= health_of(ph, u);
        if (step > cells - t) break;
    }
    // block sums of the diagnostic norms (accumulation order differs from the
    // reference's serial sum; the norms are reported, never fed back)
    __shared__ double red[NV][kPlainBlock / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        double s = sum[v];
        if (__any_sync(0xffffffffu, !dzero(s))) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        }
        if (lane == 0) red[v][wid] = s;
    }
    health = __reduce_or_sync(0xffffffffu, health);
    if (lane == 0 && health) atomicOr(&b.ctl->health, health);
    __syncthreads();
    if (threadIdx.x < NV) {
        double s = 0.0;
        for (int w = 0; w < kPlainBlock / 32; ++w) s += red[threadIdx.x][w];
        if (!dzero(s)) atomicAdd(&b.ctl->res[threadIdx.x], s);
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        Ctl* ctl = b.ctl;
        __threadfence();
        if (atomicAdd(&ctl->blocks_done, 1u) == gridDim.x - 1) {
            ctl->blocks_done = 0;
            ctl->time += ctl->dt;
            ctl->iteration += 1;
            if (ctl->run_mode) {
                if ((ctl->save_sol > 0) && (ctl->next_sol == ctl->time)) ctl->next_sol += ctl->save_sol;
                if ((ctl->save_slice > 0) && (ctl->next_slice == ctl->time)) ctl->next_slice += ctl->save_slice;
                if (ctl->iteration == ctl->max_iteration || ctl->time >= ctl->max_time) ctl->stop_req = 1;
            }
        }
    }
}

}  // namespace

// Blocks of k_dt and k_update: each thread takes several cells of a large
// grid, so that the block's closing reductions are a small part of its work.
static unsigned reduce_blocks(const Layout& L) {
    const long long full = (L.cells() + kPlainBlock - 1) / kPlainBlock;
    return (unsigned)std::min<long long>(full, kPlainReduceBlocks);
}

int plain_partial_blocks(const Layout& L) { return (int)reduce_blocks(L); }

template <int ND>
static void launch_recon(const PlainBufs& b, const Phys& ph, unsigned blocks, cudaStream_t st) {
    if (ph.recon == TS_RECON_LINEAR_2POINTS) k_recon<ND, P_LINEAR><<<blocks, kPlainBlock, 0, st>>>(b);
    else if (ph.recon == TS_RECON_ENO2_2POINTS) k_recon<ND, P_ENO2><<<blocks, kPlainBlock, 0, st>>>(b);
    else if (ph.limiter == TS_LIM_VENKATAKRISHNAN) k_recon<ND, P_LIM_VK><<<blocks, kPlainBlock, 0, st>>>(b);
    else k_recon<ND, P_LIM_BJ><<<blocks, kPlainBlock, 0, st>>>(b);
}

template <int A, int ND>
static void launch_flux(const PlainBufs& b, const Phys& ph, cudaStream_t st) {
    const Layout& L = b.L;
    const long long faces = (long long)(L.nx + (A == 0)) * (L.ny + (A == 1)) * (L.nz + (A == 2));
    const unsigned blocks = (unsigned)((faces + kPlainBlock - 1) / kPlainBlock);
    if (ph.solver == TS_RS_GODUNOV) k_flux<A, ND, TS_RS_GODUNOV><<<blocks, kPlainBlock, 0, st>>>(b, ph);
    else if (ph.solver == TS_RS_HLLC) k_flux<A, ND, TS_RS_HLLC><<<blocks, kPlainBlock, 0, st>>>(b, ph);
    else k_flux<A, ND, TS_RS_ROE_PIKE><<<blocks, kPlainBlock, 0, st>>>(b, ph);
}

cudaError_t plain_step(const PlainBufs& b, const Phys& ph, cudaStream_t st, cudaEvent_t* ev, int* n_launch,
                       const char** names) {
    const Layout& L = b.L;
    const dim3 blk(kPlainBlock);
    const dim3 cells((L.nx + kPlainBlock - 1) / kPlainBlock, L.ny, L.nz);
    auto ghost_grid = [&](int a) {
        const int n1 = (a == 0) ? L.ny : L.nx;
        const int n2 = (a == 2) ? L.ny : L.nz;
        return dim3((n1 * n2 + kPlainBlock - 1) / kPlainBlock);
    };
    int nl = 0;
    if (ev) cudaEventRecord(ev[0], st);
    auto mark = [&](const char* name) {
        if (names) names[nl] = name;
        ++nl;
        if (ev) cudaEventRecord(ev[nl], st);
    };
    k_ghost<0><<<ghost_grid(0), blk, 0, st>>>(b, ph);
    mark("k_ghost_x");
    if (ph.nd > 1) { k_ghost<1><<<ghost_grid(1), blk, 0, st>>>(b, ph); mark("k_ghost_y"); }
    if (ph.nd > 2) { k_ghost<2><<<ghost_grid(2), blk, 0, st>>>(b, ph); mark("k_ghost_z"); }
    if (ph.viscous) {
        k_vgrad<<<cells, blk, 0, st>>>(b, ph);
        mark("k_vgrad");
        k_vgrad_bc<0><<<ghost_grid(0), blk, 0, st>>>(b, ph);
        mark("k_vgrad_bc_x");
        if (ph.nd > 1) { k_vgrad_bc<1><<<ghost_grid(1), blk, 0, st>>>(b, ph); mark("k_vgrad_bc_y"); }
        if (ph.nd > 2) { k_vgrad_bc<2><<<ghost_grid(2), blk, 0, st>>>(b, ph); mark("k_vgrad_bc_z"); }
    }
    if (ph.recon != TS_RECON_PIECEWISE_CONSTANT) {
        const unsigned blocks = (unsigned)((L.cells() + kPlainBlock - 1) / kPlainBlock);
        if (ph.nd == 3) launch_recon<3>(b, ph, blocks, st);
        else if (ph.nd == 2) launch_recon<2>(b, ph, blocks, st);
        else launch_recon<1>(b, ph, blocks, st);
        mark("k_recon");
    }
    if (ph.nd == 3) launch_flux<0, 3>(b, ph, st);
    else if (ph.nd == 2) launch_flux<0, 2>(b, ph, st);
    else launch_flux<0, 1>(b, ph, st);
    mark("k_flux_x");
    if (ph.nd == 3) launch_flux<1, 3>(b, ph, st);
    else if (ph.nd == 2) launch_flux<1, 2>(b, ph, st);
    if (ph.nd > 1) mark("k_flux_y");
    if (ph.nd > 2) { launch_flux<2, 3>(b, ph, st); mark("k_flux_z"); }
    const unsigned rb = reduce_blocks(L);
    if (ph.nd == 3) k_dt<3><<<rb, blk, 0, st>>>(b, ph);
    else if (ph.nd == 2) k_dt<2><<<rb, blk, 0, st>>>(b, ph);
    else k_dt<1><<<rb, blk, 0, st>>>(b, ph);
    mark("k_dt");
    if (ph.nd == 3) k_update<3><<<rb, blk, 0, st>>>(b, ph);
    else if (ph.nd == 2) k_update<2><<<rb, blk, 0, st>>>(b, ph);
    else k_update<1><<<rb, blk, 0, st>>>(b, ph);
    mark("k_update");
    if (n_launch) *n_launch = nl;
    return cudaGetLastError();
}

}  // namespace ts
