// Building blocks of the FP64 path shared by its kernels (ts_plain.cu,
// ts_tube64.cu): boundary conditions, the two kinds of arithmetic, the
// Riemann solvers, the reconstruction of one cell's variable, and the health
// flags.  The units that include it are compiled with --fmad=false.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

#include "ts_exact64.cuh"
#include "ts_internal.h"

namespace ts {

namespace {

typedef unsigned long long u64;
constexpr u64 kInfBits = 0x7FF0000000000000ULL;

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
// non-NaN a, b, x.  A NaN orders by its bits here.  Where one can come from
// physical cells (a face state of second order with a negative pressure: the
// root of its sound speed, or a neighbour that has left the physical states),
// Fast gives the face or the cell up and Safe tells it apart.
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
// a NaN that arithmetic made (its quiet bit is in the high word)
__device__ __forceinline__ bool dnan(double x) { return (x64::hi_of(x) & 0x7FFFFFFFu) > 0x7FF00000u; }
__device__ __forceinline__ bool dfinite(double x) { return (x64::hi_of(x) & 0x7FF00000u) != 0x7FF00000u; }
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
// ranges stated there (results that are subnormal, mostly); anything else sets `bad` and the result is discarded.
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
// Safe: Fast whose operations fall back one by one instead of giving up: for
// kernels in which a warp's latency is all that counts, and a subnormal result
// (in the tails of a wave, of cells that a perturbation has just reached) would send
// some warp through the second arithmetic at every step.
static __device__ __noinline__ double hw_div(double a, double b) { return a / b; }
static __device__ __noinline__ double hw_sqrt(double a) { return sqrt(a); }
static __device__ __noinline__ double hw_half(double a) { return a * 0.5; }
struct Safe : Fast {
    struct Div {
        x64::Divisor d;
        double b;
        bool bad;
    };
    __device__ __forceinline__ Div divisor(double b) {
        Div r;
        r.b = b;
        r.bad = false;
        r.d = x64::divisor(b, r.bad);
        return r;
    }
    __device__ __forceinline__ double over(double a, const Div& d) {
        bool no = d.bad;
        double q = x64::quotient(a, d.d, no);
        if (no) q = hw_div(a, d.b);
        return q;
    }
    __device__ __forceinline__ double div(double a, double b) { return over(a, divisor(b)); }
    __device__ __forceinline__ double root(double a) {
        bool no = false;
        double r = x64::root(a, no);
        if (no) r = hw_sqrt(a);
        return r;
    }
    __device__ __forceinline__ double half(double a) {
        bool no = false;
        double r = x64::half(a, no);
        if (no) r = hw_half(a);
        return r;
    }
    // fmin, fmax and the comparisons of Plain for NaN too: no face is solved again
    __device__ __forceinline__ double min(double a, double b) { return (dlt(a, b) && !dnan(a)) || dnan(b) ? a : b; }
    __device__ __forceinline__ double max(double a, double b) { return (dlt(a, b) || dnan(a)) && !dnan(b) ? b : a; }
    __device__ __forceinline__ bool lt(double a, double b) { return dlt(a, b) && !dnan(a) && !dnan(b); }
    __device__ __forceinline__ bool ge0(double a) { return !dneg(a) && !dnan(a); }
    __device__ __forceinline__ bool le0(double a) { return !dpos(a) && !dnan(a); }
};
// FaceArith: 3D Roe faces use FastMul: those grids keep the pipes full.  A grid of 1D or 2D
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

// ---------------------------------------------------------------------------
// Reconstruction
// ---------------------------------------------------------------------------
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
// estimates in recon_value.
__device__ __noinline__ bool ratio_less(double a1, double d1, double a2, double d2) { return a1 / d1 < a2 / d2; }

// FP32 estimate (truncated, relative error 2^-23) of a positive double with
// an exponent field in [897, 1150].
__device__ __forceinline__ float est32(u64 b) { return __uint_as_float((unsigned)(b >> 29) - 0xC0000000u); }
__device__ __forceinline__ bool est32_ok(u64 b) { return (unsigned)(b >> 52) - 897u < 254u; }

// recon_value as the reference states it: for the cells that Fast gives up.  A
// slope that is not finite enters the samples along the other axes too, times
// the zero component of their offset.
template <int ND, int KIND>
__device__ __forceinline__ void recon_stated(double val, const double nm[ND], const double np[ND], const double* d,
                                             const double* hs, double eps2, double g[ND], double& lmin,
                                             double proj[ND]) {
    double one[ND], gs[ND];
    lmin = 1.0;
#pragma unroll
    for (int a = 0; a < ND; ++a) {
        if (KIND == P_ENO2) {
            const double gl = (val - nm[a]) / d[2 * a], gr = (np[a] - val) / d[2 * a + 1];
            one[a] = fabs(gl) < fabs(gr) ? gl : gr;
        } else {
            one[a] = (np[a] - nm[a]) / d[a];
        }
    }
#pragma unroll
    for (int a = 0; a < ND; ++a) {
        g[a] = one[a];
#pragma unroll
        for (int b = 0; b < ND; ++b)
            if (b != a) g[a] += one[b] * 0.0;
        gs[a] = g[a] * hs[a];
    }
    if (KIND == P_LIM_BJ || KIND == P_LIM_VK) {
        double umax = val, umin = val;
#pragma unroll
        for (int f = 0; f < 2 * ND; ++f) {
            const double vn = (f & 1) ? np[f >> 1] : nm[f >> 1];
            if (umax < vn) umax = vn;
            if (umin > vn) umin = vn;
        }
        if (!(umax - umin < 3.0 * 2.2250738585072014e-308)) {
            Plain o;
            const double un = 0.5 * (umax - umin);
#pragma unroll
            for (int f = 0; f < 2 * ND; ++f) {
                const double d2 = (val + ((f & 1) ? gs[f >> 1] : -gs[f >> 1])) - val;
                if (!(d2 > 0 || d2 < 0)) continue;
                const double um = d2 > 0 ? umax : umin;
                double lv;
                if (KIND == P_LIM_VK) {
                    lv = venkat(um / un, val / un, d2 / un, eps2, o);
                } else {
                    const double r = (um - val) / d2;
                    lv = r < 1.0 ? r : 1.0;
                }
                if (lmin > lv) lmin = lv;
            }
        }
    }
#pragma unroll
    for (int a = 0; a < ND; ++a) proj[a] = (KIND == P_LIM_BJ || KIND == P_LIM_VK) ? lmin * gs[a] : gs[a];
}

// Whether dividing zero by the distances gives zeros (Fast gives up a cell with
// a distance of zero).
template <class O, int N>
__device__ __forceinline__ bool nonzero(const typename O::Div* d) {
    bool ok = true;
    if constexpr (std::is_same_v<O, Safe>) {
#pragma unroll
        for (int k = 0; k < N; ++k) ok = ok && !d[k].bad;
    }
    return ok;
}

// As Fast and Safe form them: slopes (Linear2PointsStencil.h:147-178 or
// ENO2PointsStencil.h:202-239) and, for Linear2psLim, the limiter
// (Linear2psLim.h:305-374, Limiters.h:28-119) of one variable of a cell from
// its value and its neighbours'.  d: divisors of
// the slopes (ENO2: left and right); hs: half cell sizes.  g: slopes, lmin:
// limiter, proj: the projections lim * (slope * h/2) to the high faces (their
// negatives go to the low faces).
template <int ND, int KIND, class O>
__device__ __forceinline__ void recon_value(double val, const double nm[ND], const double np[ND],
                                            const typename O::Div* d, const double* hs, double eps2, double g[ND],
                                            double& lmin, double proj[ND], O& o) {
    double gs[ND];
    lmin = 1.0;
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
        // a constant neighbourhood (finite): slopes and projections are zero, but
        // for a distance of zero (cells narrower than their coordinates' last bit)
        if (kmax == kmin && dfinite(val) && nonzero<O, KIND == P_ENO2 ? 2 * ND : ND>(d)) {
#pragma unroll
            for (int a = 0; a < ND; ++a) g[a] = proj[a] = 0.0;
            return;
        }
    }
#pragma unroll
    for (int a = 0; a < ND; ++a) {
        if (KIND == P_ENO2) {
            const double gl = o.over(val - nm[a], d[2 * a]);
            const double gr = o.over(np[a] - val, d[2 * a + 1]);
            g[a] = dabs_lt(gl, gr) && !dnan(gr) ? gl : gr;
        } else {
            g[a] = o.over(np[a] - nm[a], d[a]);
        }
        gs[a] = g[a] * hs[a];
    }
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
            } else if constexpr (std::is_same_v<O, Safe>) {
                // as below, with every ratio below 1 divided out
                const u64 ap = (u64)__double_as_longlong(am), aq = (u64)__double_as_longlong(dabs(an));
#pragma unroll
                for (int f = 0; f < 2 * ND; ++f) {
                    const double s = (f & 1) ? gs[f >> 1] : dneg_of(gs[f >> 1]);
                    const double d2 = (val + s) - val;
                    const u64 ad = (u64)__double_as_longlong(dabs(d2));
                    const u64 aa = __double2hiint(d2) < 0 ? aq : ap;
                    if (aa < ad && ad <= kInfBits) {
                        const double r = o.div(__longlong_as_double((long long)aa), __longlong_as_double((long long)ad));
                        if (dlt(r, lmin)) lmin = r;
                    }
                }
            } else {
                // The limiter is the smallest of the rounded ratios a / d2
                // (a = umax - val or umin - val) below 1.  Rounding is
                // monotone, so only the smallest ratio is divided out.  d2 is the
                // projection gs up to rounding: where no projection is
                // lost in the value's rounding (val < 2^25 max|gs|) and the FP32
                // estimates tell the smaller a from the larger and the largest
                // |gs| from the next (2^-17 apart; estimates are good to 2^-20),
                // the smallest ratio is that of these two, and only its d2 is formed (2
                // FP64 additions of 8 in 2D and 12 in 3D: shear layer 1024^2 10.50 -> 9.84
                // ms per pass).
                const u64 ap = (u64)__double_as_longlong(am), aq = (u64)__double_as_longlong(dabs(an));
                const u64 a1 = ap < aq ? ap : aq, a2 = ap < aq ? aq : ap;
                u64 s1 = (u64)__double_as_longlong(dabs(gs[0])), s2 = 0;
#pragma unroll
                for (int a = 1; a < ND; ++a) {
                    const u64 t = (u64)__double_as_longlong(dabs(gs[a]));
                    if (t > s1) { s2 = s1; s1 = t; }
                    else if (t > s2) s2 = t;
                }
                const int es = (int)(s1 >> 52);
                const bool clear = (unsigned)(es - 1) < 2046u && (int)(((unsigned)__double2hiint(val) >> 20) & 0x7FFu) - es <= 24;
                const u64 sc = ((u64)es - 1023u) << 52;  // the exponent of s1, taken out of all
                const float f1 = est32(s1 - sc);
                const float f2 = (long long)s2 > (long long)sc && est32_ok(s2 - sc) ? est32(s2 - sc) : 0.0f;
                const bool in = (a1 >> 52) != 0 && (long long)a1 > (long long)sc && est32_ok(a1 - sc) && est32_ok(a2 - sc);
                const float e1 = est32(a1 - sc), e2 = est32(a2 - sc);
                constexpr float kNear = 1.0f - 7.7e-6f;
                if (clear && a1 == 0) {
                    lmin = 0.0;  // a local extremum
                } else if (clear && in && e1 > f1 * (2.0f - kNear)) {
                    // every ratio is above 1
                } else if (clear && in && e1 < f1 * kNear && f2 < f1 * kNear && e1 < e2 * kNear) {
                    const double g1 = __longlong_as_double((long long)s1);
                    const double d2 = ap < aq ? (val + g1) - val : val - (val - g1);
                    lmin = o.div(__longlong_as_double((long long)a1), d2);
                } else {
                    // too close to tell: the same on every face's own d2, and
                    // estimates closer than 2^-18 settled by their quotients.  A ratio
                    // with |a| >= |d2| rounds to 1 or more and is dropped.
                    u64 ba = 0, bd = 0;
                    float br = 2.0f;
#pragma unroll
                    for (int f = 0; f < 2 * ND; ++f) {
                        const double s = (f & 1) ? gs[f >> 1] : -gs[f >> 1];
                        const double d2 = (val + s) - val;
                        const u64 ad = (u64)__double_as_longlong(dabs(d2));
                        const u64 aa = __double2hiint(d2) < 0 ? aq : ap;
                        if (aa < ad) {
                            // estimates with the exponent of d2 taken out of both (a
                            // subnormal a or d2 gives up)
                            const bool an = (aa >> 52) != 0;
                            o.bad |= (unsigned)(ad >> 52) - 1u >= 2046u || (!an && aa != 0);
                            const u64 sc = ((ad >> 52) - 1023u) << 52, as = aa - sc;
                            const float r = an && (long long)aa > (long long)sc && est32_ok(as)
                                                ? __fdividef(est32(as), est32(ad - sc)) : 0.0f;
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
    }
#pragma unroll
    for (int a = 0; a < ND; ++a) proj[a] = (KIND == P_LIM_BJ || KIND == P_LIM_VK) ? lmin * gs[a] : gs[a];
}

// ---------------------------------------------------------------------------
// Faces, time step and health
// ---------------------------------------------------------------------------
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

// Minimum of the warp's values of V/SR.  They are not negative (a NaN of
// either sign has a larger pattern than +inf), so they order like their bits.
__device__ __forceinline__ u64 umin64(u64 a, u64 b) { return a < b ? a : b; }
__device__ __forceinline__ u64 warp_min(u64 v) {
    // the least high word, then the least low word among its holders
    const unsigned hi = (unsigned)(v >> 32), least = __reduce_min_sync(0xffffffffu, hi);
    const unsigned lo = __reduce_min_sync(0xffffffffu, hi == least ? (unsigned)v : 0xffffffffu);
    return (u64)least << 32 | lo;
}

// Bits of V / sr.
__device__ __forceinline__ u64 ratio_bits(double V, double sr) {
    bool bad = false;
    double r = x64::div(V, sr, bad);
    if (bad) r = V / sr;
    return (u64)__double_as_longlong(r);
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

}  // namespace

}  // namespace ts
