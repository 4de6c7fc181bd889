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
// warp instruction of any kind, comparisons, min/max and |x| included.  So what
// need not be there runs on the integer pipe: divisions, square roots and about
// half of the products (ts_exact64.cuh), comparisons, sign changes and halvings;
// terms that are exact zeros are skipped where a whole warp agrees (transverse
// momentum of 1D and 2D flows, constant neighbourhoods, equal fluxes); the slope
// projections lim * (slope * h/2) are formed once per cell instead of at each
// of its faces, and the limiter forms the one difference that decides it; the
// residual norms are summed per thread over many cells before the block's
// reduction.  The results are bit for bit the same.  The ghost layers and the
// fluxes of the axes are branches of the captured step.
// Measured on one GB300, time per step before and after: 3D blast 192^3 (Roe,
// Barth-Jespersen) 28.4 -> 8.6 ms; 2D shear layer 1024^2 (HLLC) 3.27 -> 0.61 ms;
// 2D box 203x157 167 -> 63 us.  1D problems: ts_tube64.cu.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "ts_cell64.cuh"
#include "ts_plain.h"

namespace ts {

namespace {

__device__ __forceinline__ long long vidx(const Layout& L, int v) { return (long long)v * L.plane; }

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

// Slopes and limiter of variable v in cell c.  With b.fold the stored value is
// the projection, otherwise slope and limiter.
template <int ND, int KIND, class O>
__device__ __forceinline__ void recon_var(const PlainBufs& b, int v, long long c, const typename O::Div* d,
                                          const double* hs, double eps2, O& o) {
    const Layout& L = b.L;
    const double* U = b.U + vidx(L, v) + c;
    double nm[ND], np[ND], g[ND], proj[ND], lim;
#pragma unroll
    for (int a = 0; a < ND; ++a) {
        const long long st = L.stride(a);
        nm[a] = U[-st];
        np[a] = U[st];
    }
    if constexpr (std::is_same_v<O, Plain>) recon_stated<ND, KIND>(U[0], nm, np, d, hs, eps2, g, lim, proj);
    else recon_value<ND, KIND, O>(U[0], nm, np, d, hs, eps2, g, lim, proj, o);
#pragma unroll
    for (int a = 0; a < ND; ++a) b.G[vidx(L, a * NV + v) + c] = b.fold ? proj[a] : g[a];
    if (!b.fold && (KIND == P_LIM_BJ || KIND == P_LIM_VK)) b.Lim[vidx(L, v) + c] = lim;
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

template <class O>
__device__ __forceinline__ double face_area_of(int nd, int a, double hx, double hy, double hz, O& o) {
    if (a == 0) return nd == 1 ? 1.0 : (nd == 2 ? hy : o.mul(hy, hz));
    if (a == 1) return nd == 2 ? hx : o.mul(hx, hz);
    return o.mul(hx, hy);
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

// Bits of V/SR of a cell (the least of its own and of the high-side ghost
// cells', whose SR is their single face term), SR in the reference's
// accumulation order (x-left, x-right, y-left, ...).
template <int ND, class O>
__device__ __forceinline__ u64 dt_cell(const PlainBufs& b, const Phys& ph, int i, int j, int k, O& o) {
    const Layout& L = b.L;
    const long long c = L.at(i, j, k);
    const double hx = b.ch[0][i + L.gx], hy = b.ch[1][j + L.gy], hz = b.ch[2][k + L.gz];
    const double V = o.mul(o.mul(hx, hy), hz);
    double sr = 0.0;
    u64 r = kInfBits;
    const int ix[3] = {i, j, k};
#pragma unroll
    for (int a = 0; a < ND; ++a) {
        const double fS = face_area_of(ND, a, hx, hy, hz, o);
        const long long st = L.stride(a);
        const double lo = o.mul(fS, b.Lam[a][c]), hi = o.mul(fS, b.Lam[a][c + st]);
        sr = a == 0 ? lo : sr + lo;
        sr += hi;
        if (ph.visc != 0.0) sr += b.VSR[a][c + st];
        if (ix[a] == L.n(a) - 1) {
            double hg[3] = {hx, hy, hz};
            hg[a] = b.ch[a][L.n(a) + (a == 0 ? L.gx : (a == 1 ? L.gy : L.gz))];
            r = umin64(r, ratio_bits(hg[0] * hg[1] * hg[2], hi));
        }
    }
    return umin64(r, ratio_bits(V, sr));
}
template <int ND>
__device__ __noinline__ u64 dt_plain(const PlainBufs& b, const Phys& ph, int i, int j, int k) {
    Plain o;
    return dt_cell<ND, Plain>(b, ph, i, j, k, o);
}

// V/SR of every cell, block min by warp shuffles.  The last
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
        FastMul o;
        u64 mine = dt_cell<ND, FastMul>(b, ph, i, j, k, o);
        if (o.bad) mine = dt_plain<ND>(b, ph, i, j, k);
        r = umin64(r, mine);
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
        last = count_in(&b.ctl->blocks_done) == (unsigned)(nblk - 1);
    }
    __syncthreads();
    if (!last) return;
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

// U + dt (R / V) of one cell's variables; F = the face fluxes.
template <int ND, class O>
__device__ __forceinline__ void update_cell(const PlainBufs& b, const Phys& ph, int i, int j, int k, double dt,
                                            double u[NV], double nrm[NV], O& o) {
    const Layout& L = b.L;
    const long long c = L.at(i, j, k);
    const double hx = b.ch[0][i + L.gx], hy = b.ch[1][j + L.gy], hz = b.ch[2][k + L.gz];
    const double V = o.mul(o.mul(hx, hy), hz);
    double R[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) R[v] = 0.0;
#pragma unroll
    for (int a = 0; a < ND; ++a) {
        const double fS = face_area_of(ND, a, hx, hy, hz, o);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const double* F = b.F[a] + vidx(L, v) + c;
            const double fh = F[L.stride(a)], fl = F[0];
            // equal (finite) fluxes: the difference is a zero
            if (__double_as_longlong(fh) == __double_as_longlong(fl) && (__double2hiint(fh) & 0x7FF00000) != 0x7FF00000)
                continue;
            const double d = o.mul(fh - fl, fS);
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
        // (dt is infinite where no cell has a wave speed)
        if (dzero(R[v]) && dfinite(dt)) continue;
        u[v] = uo[v] + o.mul(dt, o.over(R[v], iv));
        nrm[v] = o.mul(V, dabs(R[v]));
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
        FastMul o;
        update_cell<ND, FastMul>(b, ph, i, j, k, dt, u, nrm, o);
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
    // reference's serial sum; the norms are reported, never fed back), added to
    // kNormSlots running sums each where there are many blocks: one sum of 2432
    // block sums loses more to rounding (blast 192^3: 1.8e-15 against 1.1e-15);
    // with few the closing pass over the slots would cost more than it gives
    // (2D box 203x157: 2.5 us of a 69 us step)
    const bool slots = gridDim.x > kNormDirectBlocks;
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
    __shared__ bool last;
    if (threadIdx.x < NV) {
        double s = 0.0;
        for (int w = 0; w < kPlainBlock / 32; ++w) s += red[threadIdx.x][w];
        double* to = slots ? &b.norms[threadIdx.x * kNormSlots + blockIdx.x % kNormSlots] : &b.ctl->res[threadIdx.x];
        if (!dzero(s)) atomicAdd(to, s);
    }
    __syncthreads();
    Ctl* ctl = b.ctl;
    if (threadIdx.x == 0) last = count_in(&ctl->blocks_done) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    // the slots of each norm, summed pairwise and cleared for the next step
    for (int v = wid; slots && v < NV; v += kPlainBlock / 32) {
        double s = __ldcg(&b.norms[v * kNormSlots + lane]);
        b.norms[v * kNormSlots + lane] = 0.0;
        if (__any_sync(0xffffffffu, !dzero(s))) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        }
        if (lane == 0) ctl->res[v] = s;
    }
    if (threadIdx.x == 0) {
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
                       const char** names, const PlainSide* side) {
    // axes 1 and 2 on their own branches
    const int branches = side ? ph.nd - 1 : 0;
    auto fork = [&] {
        if (branches) cudaEventRecord(side->fork, st);
        for (int k = 0; k < branches; ++k) cudaStreamWaitEvent(side->stream[k], side->fork, 0);
    };
    auto join = [&] {
        for (int k = 0; k < branches; ++k) {
            cudaEventRecord(side->join[k], side->stream[k]);
            cudaStreamWaitEvent(st, side->join[k], 0);
        }
    };
    const cudaStream_t st1 = branches > 0 ? side->stream[0] : st, st2 = branches > 1 ? side->stream[1] : st;
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
    fork();
    k_ghost<0><<<ghost_grid(0), blk, 0, st>>>(b, ph);
    mark("k_ghost_x");
    if (ph.nd > 1) { k_ghost<1><<<ghost_grid(1), blk, 0, st1>>>(b, ph); mark("k_ghost_y"); }
    if (ph.nd > 2) { k_ghost<2><<<ghost_grid(2), blk, 0, st2>>>(b, ph); mark("k_ghost_z"); }
    join();
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
    fork();
    if (ph.nd == 3) launch_flux<0, 3>(b, ph, st);
    else if (ph.nd == 2) launch_flux<0, 2>(b, ph, st);
    else launch_flux<0, 1>(b, ph, st);
    mark("k_flux_x");
    if (ph.nd == 3) launch_flux<1, 3>(b, ph, st1);
    else if (ph.nd == 2) launch_flux<1, 2>(b, ph, st1);
    if (ph.nd > 1) mark("k_flux_y");
    if (ph.nd > 2) { launch_flux<2, 3>(b, ph, st2); mark("k_flux_z"); }
    join();
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
