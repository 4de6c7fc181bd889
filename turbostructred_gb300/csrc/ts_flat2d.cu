// Mixed-precision stage of one small 2D problem: a CTA per 32 x 4 tile, every
// phase of the stage one pass over the CTA's threads, nothing marched.
//
// What bounds it: latency.  A small grid leaves most of the chip idle, and the
// marching kernel (k_mix_step) takes five dependent rows of loads and three
// passes of three barriers for the one row that each CTA then owns (10.4 us
// per stage at 128 x 128, in rows of 64 threads, against 6.1).  Here all 288 cells of the tile and its 2-cell halo
// are loaded at once, one per thread; the slopes of the 200 cells that the
// faces need, the 132 x faces (threads 0..131) and 160 y faces (threads
// 160..319), and the 128 residuals each take one pass, with a barrier between.  A
// tile converts 2.25 and reconstructs 1.6 cells per cell that it owns, where a
// row that marches far takes 1.1 of each; kFlatCells (ts_mixed.cu) has the line.
//
// The arithmetic is k_mix_step's: working copy, slopes and face states are explicitly
// rounded, and each is formed at one place of the code, so a cell's copies in
// neighbouring CTAs are the same bits.
#include <cuda_runtime.h>

#include "ts_flux32.cuh"
#include "ts_mixed.h"

namespace ts {
namespace {

using namespace mix32;

constexpr int HB2 = 2;
constexpr int FTX = 32, FTY = 4;                      // cells of a tile
constexpr int FBX = FTX + 2 * HB2, FBY = FTY + 2 * HB2;  // with the halo
constexpr int FRX = FTX + 2, FRY = FTY + 2;           // with the ring that is reconstructed
constexpr int FY0 = 160;                              // first thread with a y face
constexpr int FNT = FY0 + FTX * (FTY + 1);            // 320 threads
static_assert(FTY * (FTX + 1) <= FY0 && FBX * FBY <= FNT && FRX * FRY <= FNT, "one pass per phase");

// Shared memory (floats): working state, half-slopes along x and y, fluxes.
struct FlatMem {
    float w[NV][FBY][FBX];
    float d[2][NV][FRY][FRX];
    float fx[NV + 1][FTY][FTX + 1];
    float fy[NV + 1][FTY + 1][FTX];
    float wmax[FNT / 32];
    unsigned int whealth[FNT / 32];
};

enum { FK_PWC = 0, FK_LINEAR = 1, FK_ENO2 = 2, FK_LIM_BJ = 3, FK_LIM_VK = 4 };

int flat_kind(const MixPhys& mp) {
    if (mp.recon == TS_RECON_LINEAR_2POINTS) return FK_LINEAR;
    if (mp.recon == TS_RECON_ENO2_2POINTS) return FK_ENO2;
    if (mp.recon == TS_RECON_LINEAR_2POINTS_LIMITED)
        return mp.limiter == TS_LIM_VENKATAKRISHNAN ? FK_LIM_VK : FK_LIM_BJ;
    return FK_PWC;
}

// Limited half-slopes of one variable along x and y (Linear2PointsStencil.h:66-97,
// ENO2PointsStencil.h:20-58, Linear2psLim.h:63-132, Limiters.h:28-115).
template <int KIND>
__device__ __forceinline__ void slopes2(float w0, const float (&nm)[2], const float (&np)[2], const AxisGeo (&g)[2],
                                        float eps2, float top, float (&dd)[2]) {
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        if (KIND == FK_ENO2) {
            const float gl = (w0 - nm[a]) * g[a].il, gr = (np[a] - w0) * g[a].ir;
            dd[a] = __fmul_rn(fabsf(gl) < fabsf(gr) ? gl : gr, g[a].hh);
        } else {
            dd[a] = __fmul_rn(np[a] - nm[a], g[a].ks);
        }
    }
    if (KIND != FK_LIM_BJ && KIND != FK_LIM_VK) return;
    const float umax = fmaxf(fmaxf(w0, fmaxf(nm[0], np[0])), fmaxf(nm[1], np[1]));
    const float umin = fminf(fminf(w0, fminf(nm[0], np[0])), fminf(nm[1], np[1]));
    float lim = 1.0f;
    if (KIND == FK_LIM_BJ) {
        // the smallest admissible ratio over the four face projections; with
        // both slopes 0 the ratio is dropped by fminf
        lim = fminf(top, quot(fminf(umax - w0, w0 - umin), fmaxf(fabsf(dd[0]), fabsf(dd[1]))));
    } else if (umax - umin > 0.0f) {
        const float iun = 2.0f / (umax - umin);
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            const float d2 = (f & 1) ? -dd[f >> 1] : dd[f >> 1];
            if (d2 == 0.0f) continue;
            const float dm = ((d2 > 0.0f ? umax : umin) - w0) * iun;
            const float q = d2 * iun;
            lim = fminf(lim, ((dm * dm + eps2) + 2.0f * q * dm) / (dm * dm + 2.0f * q * q + dm * q + eps2));
        }
    }
    dd[0] = __fmul_rn(dd[0], lim);
    dd[1] = __fmul_rn(dd[1], lim);
}

// The flux through one face on axis A between the box cells (xl, yl) and
// (xr, yr); g: the face's index along the axis, n its last, f its index on a
// domain side.
template <int A, int SOLVER, int KIND>
__device__ __forceinline__ float flat_face(const MixPhys& mp, const FlatMem& s, int yl, int xl, int yr, int xr, int g,
                                           int n, int per, int f, float F[NV]) {
    float UL[NV], UR[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        UL[v] = s.w[v][yl][xl];
        UR[v] = s.w[v][yr][xr];
        if (KIND != FK_PWC) {
            UL[v] = __fadd_rn(UL[v], s.d[A][v][yl - 1][xl - 1]);
            UR[v] = __fadd_rn(UR[v], -s.d[A][v][yr - 1][xr - 1]);
        }
    }
    if (g == 0 && !per) {
#pragma unroll
        for (int v = 0; v < NV; ++v) UL[v] = UR[v];
        bc32(mp, bc_id32(mp, 2 * A, f), A, UL);
    } else if (g == n && !per) {
#pragma unroll
        for (int v = 0; v < NV; ++v) UR[v] = UL[v];
        bc32(mp, bc_id32(mp, 2 * A + 1, f), A, UR);
    }
    return flux32<SOLVER, A>(mp, UL, UR, F);
}

// finish_problem with every field read at once, beside the maximum: the block
// that closes a step is alone, and each dependent trip to L2 is 0.3 us (200
// stages of 128^2 1409 -> 1361 us).  (In k_mix_step it changes how the
// compiler contracts the 1D Roe flux, and with it the results' last bits.)
__device__ __forceinline__ void finish_at_once(Ctl* ctl, double cfl) {
    const float m = __uint_as_float(*(volatile unsigned int*)&ctl->srmax_bits);
    const double t0 = ctl->time, save_sol = ctl->save_sol, save_slice = ctl->save_slice, max_time = ctl->max_time;
    const double sol = ctl->next_sol, slice = ctl->next_slice;
    const int it = ctl->iteration + 1, par = ctl->parity ^ 1, run = ctl->run_mode, max_it = ctl->max_iteration;
    double res[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) res[v] = ctl->res_acc[v];
    // positive numbers have positive bit patterns (no comparison on the FP64 pipe)
    const bool sols = __double_as_longlong(save_sol) > 0, slices = __double_as_longlong(save_slice) > 0;
    double dt, raw;
    step_size(cfl, m, dt, raw);
    if (sols && (sol < t0 + dt)) dt = sol - t0;
    if (slices && (slice < t0 + dt)) dt = slice - t0;
    const double t1 = t0 + dt;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        ctl->res[v] = res[v];
        ctl->res_acc[v] = 0.0;
    }
    ctl->dt_min_raw = raw;
    ctl->dt = dt;
    ctl->dt_apply = dt;
    ctl->time = t1;
    ctl->iteration = it;
    ctl->parity = par;
    ctl->srmax_bits = 0u;
    ctl->blocks_done = 0u;
    if (run) {
        if (sols && (sol == t1)) ctl->next_sol = sol + save_sol;
        if (slices && (slice == t1)) ctl->next_slice = slice + save_slice;
        if (it == max_it || t1 >= max_time) ctl->stop_req = 1;
    }
}

template <int SOLVER, int KIND>
__global__ void __launch_bounds__(FNT, 3) k_flat2d(const __grid_constant__ ProbDesc d) {
    __shared__ FlatMem s;
    Ctl* const ctl = d.ctl;
    if (ctl->stop_req) return;
    const int par = ctl->parity;
    const float dtf = __double2float_rn(ctl->dt_apply);
    const MixPhys& mp = d.mp;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int nx = d.kn[0], ny = d.kn[2], perx = d.kper[0], pery = d.kper[2];
    const int i0 = (int)(blockIdx.x % d.ncx) * FTX, j0 = (int)(blockIdx.x / d.ncx) * FTY;
    const AxisGeo* const geox = d.kgeo[0] + d.kgoff[0];
    const AxisGeo* const geoy = d.kgeo[2] + d.kgoff[2];
    const AxisGeo gz = d.kgeo[1][d.kgoff[1]];  // the inactive axis
    const size_t plane = (size_t)d.L.plane;
    unsigned int health = 0;
    // the tile and its halo: pending update, working copy, U^{n+1} of the own cells
    if (tid < FBX * FBY) {
        const int by = tid / FBX, bx = tid - by * FBX;
        const int gi = i0 + bx - HB2, gj = j0 + by - HB2;
        if (gi < nx + HB2 && gj < ny + HB2) {
            int si, sj, xs, ys;
            resolve(gi, nx, perx, 0, si, xs);
            resolve(gj, ny, pery, 2, sj, ys);
            const size_t c = (size_t)(d.kbase + si + (long long)sj * d.kstr[2]);
            const double* U = d.U[par] + c;
            const float* R = d.R[par] + c;
            double u[NV];
            float inc[NV], w[NV];
#pragma unroll
            for (int v = 0; v < NV; ++v) u[v] = __ldcg(U + v * plane);
#pragma unroll
            for (int v = 0; v < NV; ++v) inc[v] = __ldcg(R + v * plane);
            const float cf = __ldg(&geox[si].ih) * gz.ih * (dtf * __ldg(&geoy[sj].ih));
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                const double e = v == 4 && mp.eos == TS_EOS_STIFFENED_GAS ? u[v] - mp.einf_d : u[v];
                w[v] = __fmaf_rn(cf, inc[v], f64_to_f32(e));
                inc[v] = __fmul_rn(cf, inc[v]);
            }
            if (xs >= 0) bc32(mp, bc_id32(mp, xs, sj), 0, w);
            if (ys >= 0) bc32(mp, bc_id32(mp, ys, si), 1, w);
#pragma unroll
            for (int v = 0; v < NV; ++v) s.w[v][by][bx] = w[v];
            if (bx >= HB2 && bx < FTX + HB2 && by >= HB2 && by < FTY + HB2 && gi < nx && gj < ny) {
                double* Uo = d.U[par ^ 1] + c;
                double un[NV];
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    un[v] = u[v] + f32_to_f64(inc[v]);
                    __stcg(Uo + v * plane, un[v]);
                }
                // rho > 0 tested on the bit pattern (no FP64 comparison)
                const long long b = __double_as_longlong(un[0]);
                if (b <= 0 || b > 0x7FF0000000000000LL)
                    health |= (b & 0x7FFFFFFFFFFFFFFFLL) > 0x7FF0000000000000LL ? TS_HEALTH_NAN : TS_HEALTH_NEG_DENSITY;
                if (!(w[4] == w[4])) health |= TS_HEALTH_NAN;
            }
        }
    }
    __syncthreads();
    if (KIND != FK_PWC) {
        if (tid < FRX * FRY) {
            const int ry = tid / FRX, rx = tid - ry * FRX;
            const int gi = i0 + rx - 1, gj = j0 + ry - 1;
            const bool corner = (rx == 0 || rx == FRX - 1) && (ry == 0 || ry == FRY - 1);
            // nothing is reconstructed beyond a non-periodic side
            if (!corner && gi <= nx && gj <= ny && (perx || (gi >= 0 && gi < nx)) && (pery || (gj >= 0 && gj < ny))) {
                int si, sj, side;
                resolve(gi, nx, 1, 0, si, side);
                resolve(gj, ny, 1, 0, sj, side);
                const AxisGeo g[2] = {geox[si], geoy[sj]};
                float eps2 = 0.0f;
                if (KIND == FK_LIM_VK) {
                    // eps^2 = (K (h1 h2)^(1/2))^3 with K = 5 (Limiters.h:93-96, Constants.h:11)
                    const float area = g[0].h * g[1].h;
                    eps2 = 125.0f * (area * sqrtf(area));
                }
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    const float nm[2] = {s.w[v][ry + 1][rx], s.w[v][ry][rx + 1]};
                    const float np[2] = {s.w[v][ry + 1][rx + 2], s.w[v][ry + 2][rx + 1]};
                    float dd[2];
                    slopes2<KIND>(s.w[v][ry + 1][rx + 1], nm, np, g, eps2, mp.lim_top, dd);
                    s.d[0][v][ry][rx] = dd[0];
                    s.d[1][v][ry][rx] = dd[1];
                }
            }
        }
        __syncthreads();
    }
    if (tid < FTY * (FTX + 1)) {
        const int y = tid / (FTX + 1), x = tid - y * (FTX + 1);
        if (i0 + x <= nx && j0 + y < ny) {
            float F[NV];
            const float lam = flat_face<0, SOLVER, KIND>(mp, s, y + HB2, x + 1, y + HB2, x + 2, i0 + x, nx, perx, j0 + y, F);
#pragma unroll
            for (int v = 0; v < NV; ++v) s.fx[v][y][x] = F[v];
            s.fx[NV][y][x] = lam;
        }
    } else if (tid >= FY0) {
        const int y = (tid - FY0) / FTX, x = (tid - FY0) % FTX;
        if (i0 + x < nx && j0 + y <= ny) {
            float F[NV];
            const float lam = flat_face<1, SOLVER, KIND>(mp, s, y + 1, x + HB2, y + 2, x + HB2, j0 + y, ny, pery, i0 + x, F);
#pragma unroll
            for (int v = 0; v < NV; ++v) s.fy[v][y][x] = F[v];
            s.fy[NV][y][x] = lam;
        }
    }
    __syncthreads();
    float srmax = 0.0f, nrm[NV] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    const int y = tid / FTX, x = tid % FTX, gi = i0 + x, gj = j0 + y;
    if (tid < FTX * FTY && gi < nx && gj < ny) {
        const AxisGeo gx = geox[gi], gy = geoy[gj];
        const float hx = gx.h, hy = gy.h;
        const float fsx = gz.h * hy, fsy = hx * gz.h, vol = fsy * hy;  // face areas, volume
        const float ixy = gx.ih * gz.ih, iv = ixy * gy.ih;
        const float kx = flux_scale<SOLVER>() * fsx, ky = flux_scale<SOLVER>() * fsy;
        const float lxl = s.fx[NV][y][x], lxr = s.fx[NV][y][x + 1], lyl = s.fy[NV][y][x], lyr = s.fy[NV][y + 1][x];
        float R[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            R[v] = -(s.fx[v][y][x + 1] - s.fx[v][y][x]) * kx;
            R[v] -= (s.fy[v][y + 1][x] - s.fy[v][y][x]) * ky;
        }
        const float sr = fsx * (lxl + lxr) + fsy * (lyl + lyr);
        // spectral radii of the ghost cells beyond the high sides
        if (gi == nx - 1) srmax = fmaxf(srmax, fsx * lxr * (geox[nx].ih * gz.ih) * gy.ih);
        if (gj == ny - 1) srmax = fmaxf(srmax, fsy * lyr * ixy * geoy[ny].ih);
        srmax = fmaxf(srmax, sr * iv);
        // source terms after the face fluxes (kernel.h:941-989), on the working state
        if (mp.force || mp.accel) {
            const float ro = s.w[0][y + HB2][x + HB2], iro = 1.0f / ro;
            const float vu = s.w[1][y + HB2][x + HB2] * iro, vv = s.w[2][y + HB2][x + HB2] * iro,
                        vw = s.w[3][y + HB2][x + HB2] * iro;
            if (mp.force) {
                R[1] += vol * mp.sigma[0];
                R[2] += vol * mp.sigma[1];
                R[3] += vol * mp.sigma[2];
                R[4] += (mp.sigma[0] * vu + mp.sigma[1] * vv + mp.sigma[2] * vw) * vol;
            }
            if (mp.accel) {
                R[1] += ro * vol * mp.g[0];
                R[2] += ro * vol * mp.g[1];
                R[3] += ro * vol * mp.g[2];
                R[4] += ((ro * mp.g[0]) * vu + (ro * mp.g[1]) * vv + (ro * mp.g[2]) * vw) * vol;
            }
        }
        float* Ro = d.R[par ^ 1] + (size_t)(d.kbase + gi + (long long)gj * d.kstr[2]);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            if (mp.norms) nrm[v] = vol * fabsf(R[v]);
            __stcg(Ro + v * plane, R[v]);
        }
    }
    // the tile's CFL maximum and health; the last tile closes the step
    if (mp.norms && wid < FTX * FTY / 32) add_norms(ctl, nrm, 0xffffffffu, lane, 32);
    const unsigned int mbits = __reduce_max_sync(0xffffffffu, __float_as_uint(srmax));
    health = __reduce_or_sync(0xffffffffu, health);
    if (lane == 0) {
        s.wmax[wid] = __uint_as_float(mbits);
        s.whealth[wid] = health;
    }
    __syncthreads();
    if (tid == 0) {
        float m = 0.0f;
        unsigned int hh = 0;
#pragma unroll
        for (int k = 0; k < FNT / 32; ++k) {
            m = fmaxf(m, s.wmax[k]);
            hh |= s.whealth[k];
        }
        if (m > 0.0f) atomicMax(&ctl->srmax_bits, __float_as_uint(m));
        if (hh) atomicOr(&ctl->health, hh);
        if (count_in(&ctl->blocks_done) == gridDim.x - 1) finish_at_once(ctl, mp.cfl);
    }
}

template <class F>
void with_flat(const MixPhys& mp, F&& f) {
    auto go = [&]<int S>() {
        switch (flat_kind(mp)) {
        case FK_PWC: f.template operator()<S, FK_PWC>(); break;
        case FK_LINEAR: f.template operator()<S, FK_LINEAR>(); break;
        case FK_ENO2: f.template operator()<S, FK_ENO2>(); break;
        case FK_LIM_VK: f.template operator()<S, FK_LIM_VK>(); break;
        default: f.template operator()<S, FK_LIM_BJ>(); break;
        }
    };
    if (mp.solver == TS_RS_HLLC) go.template operator()<TS_RS_HLLC>();
    else go.template operator()<TS_RS_ROE_PIKE>();
}

}  // namespace

int flat2d_tiles(const ProbDesc& d, int* ncx) {
    *ncx = (d.kn[0] + FTX - 1) / FTX;
    return *ncx * ((d.kn[2] + FTY - 1) / FTY);
}

void flat2d_launch(const ProbDesc& d, int tiles, cudaStream_t st) {
    with_flat(d.mp, [&]<int S, int K>() { k_flat2d<S, K><<<tiles, FNT, 0, st>>>(d); });
}

}  // namespace ts
