// Mixed-precision 1D problems: many stages per launch, one thread-block
// cluster per problem, the state on chip.  Serves a single 1D domain and the
// 1D problems of a batch.
//
// What bounds it: latency.  A stage launched by itself is 7 us at any size up
// to some thousand cells (launch, control word, loads, four barriers, the
// atomics that close the step), of which the arithmetic is a few hundred
// clocks.  Here each CTA of the cluster owns consecutive cells, one per
// thread, whose FP64 state and FP32 pending residual stay in registers; a stage
// needs two cluster barriers (390 clocks each):
//   1  the working copy of every cell in its CTA's shared memory, of the two
//      cells next to a CTA boundary also in the neighbour's (distributed shared
//      memory), and the boundary images at the ends.  The FP64 additions of
//      the pending update (64 clocks each) run between arrival and wait;
//   -  half-slopes of the own cells and of one cell beyond each end (two extra
//      threads), the faces (the one at the CTA's high end by the first extra
//      thread; both CTAs solve it, from the same bits), the residuals, and each warp's
//      CFL maximum to every CTA;
//   2  dt and the step's bookkeeping, repeated by every thread.
// The cells are dealt evenly, so every CTA has two at least and a halo cell is
// its neighbour's.  The arithmetic is that of k_mix_step and finish_with.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "ts_flux32.cuh"
#include "ts_mixed.h"

namespace ts {
namespace {

using namespace mix32;
namespace cg = cooperative_groups;

constexpr int kMaxThreads = 544;             // of a CTA
constexpr int kMaxOwn = kMaxThreads - 2;     // cells of a CTA
constexpr int kMaxWarps = kMaxThreads / 32;

// Shared memory of a CTA that owns up to `own` cells (floats).
struct Tube32Mem {
    int w, d, f, total;  // working copy, half-slopes, face fluxes
    TS_HD constexpr explicit Tube32Mem(int own)
        : w(0), d(w + NV * (own + 4)), f(d + NV * (own + 2)), total(f + (NV + 1) * (own + 1)) {}
};

enum { T_LINEAR = 1, T_ENO2 = 2, T_LIM_BJ = 3, T_LIM_VK = 4 };

// Limited half-slope of one variable (as recon_k of the stage kernel); h3 = h^3.
// The Venkatakrishnan ratio, ((dm^2 + eps^2) + 2 q dm) / (dm^2 + 2 q^2 + dm q +
// eps^2) with eps^2 = (K h)^3 and K = 5 (Limiters.h:93-115, Constants.h:11), has the
// FMAs that the compiler makes of it there, eps^2 among them.
__device__ __forceinline__ float half_slope(int kind, float nm, float w0, float np, const AxisGeo& g, float h3,
                                            float top) {
    float dd;
    if (kind == T_ENO2) {
        const float gl = (w0 - nm) * g.il, gr = (np - w0) * g.ir;
        dd = __fmul_rn(fabsf(gl) < fabsf(gr) ? gl : gr, g.hh);
    } else {
        dd = __fmul_rn(np - nm, g.ks);
    }
    if (kind != T_LIM_BJ && kind != T_LIM_VK) return dd;
    const float umax = fmaxf(w0, fmaxf(nm, np)), umin = fminf(w0, fminf(nm, np));
    float lim = 1.0f;
    if (kind == T_LIM_BJ) {
        lim = fminf(top, quot(fminf(umax - w0, w0 - umin), fabsf(dd)));
    } else if (umax - umin > 0.0f) {
        const float iun = 2.0f / (umax - umin);
#pragma unroll
        for (int sg = 0; sg < 2; ++sg) {
            const float d2 = sg ? -dd : dd;
            if (d2 == 0.0f) continue;
            const float dm = ((d2 > 0.0f ? umax : umin) - w0) * iun;
            const float q = d2 * iun;
            const float q2 = 2.0f * q, dm2 = __fmul_rn(dm, dm);
            const float num = __fmaf_rn(q2, dm, __fmaf_rn(125.0f, h3, dm2));
            const float den = __fmaf_rn(125.0f, h3, __fmaf_rn(dm, q, __fmaf_rn(q2, q, dm2)));
            lim = fminf(lim, num / den);
        }
    }
    return __fmul_rn(dd, lim);
}

// a >= b on the integer pipe: every warp forms it at every stage, and an FP64
// comparison of 16 of them is 300 clocks.
__device__ __forceinline__ bool at_least(double a, double b) {
    auto key = [](double x) {
        const long long k = __double_as_longlong(x);
        return k < 0 ? (long long)0x8000000000000000ULL - k : k;
    };
    const long long inf = 0x7FF0000000000000LL, x = key(a), y = key(b);
    return x >= y && x <= inf && y >= -inf && x >= -inf && y <= inf;
}

// ONE: a single domain, its descriptor a kernel parameter as in k_mix_step
// (with the descriptor in shared memory the compiler contracts the Roe
// flux's multiply-adds differently, as it does in the batched k_mix_step: each
// instance gives the bits of its counterpart).  Otherwise list holds the
// problems' descriptor indices, and with stop_unhealthy a non-physical state
// ends a problem's loop (the host stops it).
// WIDE, for CTAs of more than kWideThreads: each CTA sends its CFL maximum instead of
// each of its warps, a barrier more, but 16 values instead of up to 16 x 17 for
// every warp to send and read (one tube, batched, 7487 cells 6.07 -> 5.68 us per
// stage, with at_least; 480 cells would take 3.07 instead of 2.96).
constexpr int kWideThreads = 256;
template <int SOLVER, bool ONE, bool WIDE>
__global__ void __launch_bounds__(kMaxThreads, 1) k_tube32(const __grid_constant__ ProbDesc one,
                                                           const ProbDesc* __restrict__ probs,
                                                           const int* __restrict__ list, int budget,
                                                           int stop_unhealthy) {
    extern __shared__ float sm[];
    __shared__ ProbDesc sd;
    __shared__ unsigned int smax[kTailMaxCluster * kMaxWarps];
    __shared__ unsigned int shealth, wmax[kMaxWarps];
    cg::cluster_group cluster = cg::this_cluster();
    const int nblk = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, W = blockDim.x >> 5;
    if (!ONE) {
        const int* src = (const int*)(probs + list[blockIdx.x / nblk]);
        for (int k = tid; k < (int)(sizeof(ProbDesc) / sizeof(int)); k += blockDim.x) ((int*)&sd)[k] = src[k];
        if (tid == 0) shealth = 0u;
        __syncthreads();
    }
    const ProbDesc& d = ONE ? one : sd;
    // A finished problem that is still listed is left alone (the whole cluster
    // leaves here): it may be read back, and its memory given to another
    // problem, on other streams beside this launch.
    if (d.ctl->stop_req) return;
    const MixPhys& mp = d.mp;
    const int n = d.kn[0];
    const int C = min(nblk, max(1, n / 2));  // CTAs that own cells
    const int base = n / C, rem = n % C;
    const int m = rank < C ? base + (rank < rem) : 0, i0 = rank * base + min(rank, rem);
    const int own_max = base + (rem > 0);
    const Tube32Mem at(own_max);
    const int pw = own_max + 4, pd = own_max + 2, pf = own_max + 1;  // pitches
    const bool per = d.kper[0] != 0, own = tid < m;
    const AxisGeo* const geo = d.kgeo[0] + d.kgoff[0];
    const float h1 = d.kgeo[1][d.kgoff[1]].h, ih1 = d.kgeo[1][d.kgoff[1]].ih;
    const float hz = d.kgeo[2][d.kgoff[2]].h, ihz = d.kgeo[2][d.kgoff[2]].ih;
    const int kind = mp.recon == TS_RECON_LINEAR_2POINTS_LIMITED
                         ? (mp.limiter == TS_LIM_VENKATAKRISHNAN ? T_LIM_VK : T_LIM_BJ)
                         : (mp.recon == TS_RECON_LINEAR_2POINTS ? T_LINEAR : (mp.recon == TS_RECON_ENO2_2POINTS ? T_ENO2 : 0));
    const bool stiff = mp.eos == TS_EOS_STIFFENED_GAS;
    const long long plane = d.L.plane;
    const size_t cell = (size_t)(d.kbase + i0 + (own ? tid : 0));
    // the control word, kept by every thread
    const Ctl* const ctl = d.ctl;
    double time = ctl->time, next_sol = ctl->next_sol, next_slice = ctl->next_slice, dt = ctl->dt, raw = ctl->dt_min_raw;
    const double save_sol = ctl->save_sol, save_slice = ctl->save_slice, max_time = ctl->max_time;
    float dtf = __double2float_rn(ctl->dt_apply);
    int iteration = ctl->iteration, par = ctl->parity;
    const int max_iteration = ctl->max_iteration, run_mode = ctl->run_mode;
    const bool sols = save_sol > 0, slices = save_slice > 0;
    double u[NV];
    float r[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        u[v] = own ? __ldcg(d.U[par] + v * plane + cell) : 1.0;
        r[v] = own ? __ldcg(d.R[par] + v * plane + cell) : 0.0f;
    }
    // the cell this thread reconstructs (local index), and its geometry
    const int rl = own ? tid : (tid == m ? -1 : m);
    bool rec = kind != 0 && rank < C && tid <= m + 1;
    int ri = i0 + rl;
    if (ri < 0 || ri >= n) {
        rec = rec && per;  // beyond a non-periodic side nothing is reconstructed
        ri = ri < 0 ? ri + n : ri - n;
    }
    AxisGeo g{};
    if (rec) g = geo[ri];
    const float h3 = g.h * g.h * g.h;
    // the own cell's factors (k_mix_step: cell_geo, residual_of)
    const AxisGeo gx = geo[own ? i0 + tid : 0];
    const float cfx = gx.ih * ih1;
    const float fsx = h1 * hz, fsz = gx.h * h1, iv = (gx.ih * ih1) * ihz;
    const float kx = flux_scale<SOLVER>() * fsx;
    const float farx = own && i0 + tid == n - 1 ? geo[n].ih * ih1 : 0.0f;
    // where this cell's working copy also goes
    float *to_left = nullptr, *to_right = nullptr;
    if (rank < C) {
        const int left = rank > 0 ? rank - 1 : (per ? C - 1 : -1), right = rank < C - 1 ? rank + 1 : (per ? 0 : -1);
        if (own && tid < 2 && left >= 0)
            to_left = cluster.map_shared_rank(sm + at.w, left) + base + (left < rem) + 2 + tid;
        if (own && tid >= m - 2 && right >= 0) to_right = cluster.map_shared_rank(sm + at.w, right) + (tid - m + 2);
    }
    // boundary images beyond a non-periodic side: of cells 0, 1 and n-1, n-2
    const int lo_img = own && !per && i0 + tid < 2 ? i0 + tid : -1;
    const int hi_img = own && !per && n - 1 - (i0 + tid) < 2 ? n - 1 - (i0 + tid) : -1;
    const int sent = WIDE ? 1 : W;  // values of a CTA
    unsigned int* const remote_max =
        lane < nblk && (!WIDE || wid == 0) ? cluster.map_shared_rank(smax, lane) + rank * sent + (WIDE ? 0 : wid) : nullptr;
    unsigned int health = 0;
    bool stop = false;
    cluster.sync();  // every CTA has started: its shared memory may be written
#pragma unroll 1
    for (int st = 0; st < budget && !stop; ++st) {
        const float cf = cfx * (dtf * ihz);
        float w[NV], inc[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            inc[v] = __fmul_rn(cf, r[v]);
            const double e = v == 4 && stiff ? u[v] - mp.einf_d : u[v];
            w[v] = __fmaf_rn(cf, r[v], f64_to_f32(e));
        }
        if (own) {
#pragma unroll
            for (int v = 0; v < NV; ++v) sm[at.w + v * pw + tid + 2] = w[v];
            if (to_left) {
#pragma unroll
                for (int v = 0; v < NV; ++v) to_left[v * pw] = w[v];
            }
            if (to_right) {
#pragma unroll
                for (int v = 0; v < NV; ++v) to_right[v * pw] = w[v];
            }
#pragma unroll 1
            for (int side = 0; side < 2; ++side) {
                const int img = side ? hi_img : lo_img;
                if (img < 0) continue;
                float b[NV];
#pragma unroll
                for (int v = 0; v < NV; ++v) b[v] = w[v];
                bc32(mp, bc_id32(mp, side, 0), 0, b);
                const int to = side ? m + 2 + img : 1 - img;
#pragma unroll
                for (int v = 0; v < NV; ++v) sm[at.w + v * pw + to] = b[v];
            }
        }
        cg::cluster_group::arrival_token first = cluster.barrier_arrive();
        if (own) {
            // the pending update (its FP64 additions overlap the barrier)
#pragma unroll
            for (int v = 0; v < NV; ++v) u[v] = u[v] + f32_to_f64(inc[v]);
            const long long b = __double_as_longlong(u[0]);
            unsigned int now = 0;
            if (b <= 0 || b > 0x7FF0000000000000LL)
                now |= (b & 0x7FFFFFFFFFFFFFFFLL) > 0x7FF0000000000000LL ? TS_HEALTH_NAN : TS_HEALTH_NEG_DENSITY;
            if (!(w[4] == w[4])) now |= TS_HEALTH_NAN;
            health |= now;
        }
        cluster.barrier_wait(std::move(first));
        if (kind) {
            if (rec) {
                const float* s = sm + at.w + rl + 2;
                float* o = sm + at.d + rl + 1;
#pragma unroll
                for (int v = 0; v < NV; ++v)
                    o[v * pd] = half_slope(kind, s[v * pw - 1], s[v * pw], s[v * pw + 1], g, h3, mp.lim_top);
            }
            __syncthreads();
        }
        if (rank < C && tid <= m) {
            float UL[NV], UR[NV], F[NV];
            const int f = i0 + tid;
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                UL[v] = sm[at.w + v * pw + tid + 1];
                UR[v] = sm[at.w + v * pw + tid + 2];
                if (kind) {
                    UL[v] = __fadd_rn(UL[v], sm[at.d + v * pd + tid]);
                    UR[v] = __fadd_rn(UR[v], -sm[at.d + v * pd + tid + 1]);
                }
            }
            if (f == 0 && !per) {
#pragma unroll
                for (int v = 0; v < NV; ++v) UL[v] = UR[v];
                bc32(mp, bc_id32(mp, 0, 0), 0, UL);
            } else if (f == n && !per) {
#pragma unroll
                for (int v = 0; v < NV; ++v) UR[v] = UL[v];
                bc32(mp, bc_id32(mp, 1, 0), 0, UR);
            }
            const float lam = flux32<SOLVER, 0>(mp, UL, UR, F);
#pragma unroll
            for (int v = 0; v < NV; ++v) sm[at.f + v * pf + tid] = F[v];
            sm[at.f + NV * pf + tid] = lam;
        }
        __syncthreads();
        float srmax = 0.0f;
        if (own) {
            const float* F = sm + at.f + tid;
            const float lxl = F[NV * pf], lxr = F[NV * pf + 1];
            if (farx != 0.0f) srmax = fmaxf(srmax, fsx * lxr * farx * ihz);
            srmax = fmaxf(srmax, (fsx * (lxl + lxr)) * iv);
        }
        // srmax >= 0: its bits order like unsigned integers
        unsigned int mbits = __reduce_max_sync(0xffffffffu, __float_as_uint(srmax));
        if (WIDE) {
            if (lane == 0) wmax[wid] = mbits;
            __syncthreads();
            if (wid == 0) mbits = __reduce_max_sync(0xffffffffu, lane < W ? wmax[lane] : 0u);
        }
        if (remote_max) *remote_max = mbits;
        if (!ONE && stop_unhealthy && health) {  // rare
            for (int k = 0; k < nblk; ++k) atomicOr(cluster.map_shared_rank(&shealth, k), health);
        }
        cg::cluster_group::arrival_token second = cluster.barrier_arrive();
        if (own) {
            const float* F = sm + at.f + tid;
#pragma unroll
            for (int v = 0; v < NV; ++v) r[v] = -(F[v * pf + 1] - F[v * pf]) * kx;
            // source terms after the face fluxes (kernel.h:941-989), on the working state
            if (mp.force || mp.accel) {
                const float ro = w[0], iro = 1.0f / ro;
                const float vu = w[1] * iro, vv = w[2] * iro, vw = w[3] * iro;
                const float vol = fsz * hz;
                if (mp.force) {
                    r[1] += vol * mp.sigma[0];
                    r[2] += vol * mp.sigma[1];
                    r[3] += vol * mp.sigma[2];
                    r[4] += (mp.sigma[0] * vu + mp.sigma[1] * vv + mp.sigma[2] * vw) * vol;
                }
                if (mp.accel) {
                    r[1] += ro * vol * mp.g[0];
                    r[2] += ro * vol * mp.g[1];
                    r[3] += ro * vol * mp.g[2];
                    r[4] += ((ro * mp.g[0]) * vu + (ro * mp.g[1]) * vv + (ro * mp.g[2]) * vw) * vol;
                }
            }
        }
        cluster.barrier_wait(std::move(second));
        // dt and the step's bookkeeping (finish_with)
        unsigned int all = 0;
        for (int k = lane; k < nblk * sent; k += 32) all = max(all, smax[k]);
        all = __reduce_max_sync(0xffffffffu, all);
        step_size(mp.cfl, __uint_as_float(all), dt, raw);
        if (sols && (next_sol < time + dt)) dt = next_sol - time;
        if (slices && (next_slice < time + dt)) dt = next_slice - time;
        dtf = __double2float_rn(dt);
        time += dt;
        iteration += 1;
        par ^= 1;
        if (run_mode) {
            if (sols && (next_sol == time)) next_sol += save_sol;
            if (slices && (next_slice == time)) next_slice += save_slice;
            stop = iteration == max_iteration || at_least(time, max_time);
        }
        const bool finished = stop;
        if (!ONE && shealth) stop = true;
        if (rank == 0 && tid == 0 && (stop || st == budget - 1)) {
            Ctl* c = d.ctl;
            c->time = time;
            c->dt = dt;
            c->dt_min_raw = raw;
            c->dt_apply = dt;
            c->iteration = iteration;
            c->parity = par;
            c->next_sol = next_sol;
            c->next_slice = next_slice;
            c->stop_req = finished ? 1 : 0;
            c->srmax_bits = 0u;
            c->blocks_done = 0u;
        }
    }
    // the state and pending residual where the stage kernels expect them
    if (own) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            d.U[par][v * plane + cell] = u[v];
            d.R[par][v * plane + cell] = r[v];
        }
    }
    health = __reduce_or_sync(0xffffffffu, health);
    if (lane == 0 && health) atomicOr(&d.ctl->health, health);
    cluster.sync();  // no CTA leaves while another may still write to it
}

int own_cells(int cluster, int cells) {
    // (a problem with fewer than two cells per CTA leaves CTAs idle and has up
    // to three in the others)
    return std::max(3, (cells + cluster - 1) / cluster);
}
int block_threads(int cluster, int cells) { return (own_cells(cluster, cells) + 2 + 31) / 32 * 32; }

// Calls f.template operator()<SOLVER, WIDE>() for a launch.
template <class F>
auto with_instance(int solver, int threads, F&& f) {
    auto go = [&]<int S>() {
        return threads > kWideThreads ? f.template operator()<S, true>() : f.template operator()<S, false>();
    };
    return solver == TS_RS_HLLC ? go.template operator()<TS_RS_HLLC>() : go.template operator()<TS_RS_ROE_PIKE>();
}

// Static and dynamic shared memory of the largest CTA: within what needs no opt-in.
static_assert(sizeof(float) * Tube32Mem(kMaxOwn).total + sizeof(ProbDesc) + 4 * (kTailMaxCluster + 1) * kMaxWarps + 64 <=
              48 << 10);

void config(int cluster, int problems, int cells, cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr) {
    cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3((unsigned)(cluster * problems));
    cfg.blockDim = dim3((unsigned)block_threads(cluster, cells));
    cfg.dynamicSmemBytes = sizeof(float) * Tube32Mem(own_cells(cluster, cells)).total;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
}

}  // namespace

int tube32_max_cells() { return kTailMaxCluster * kMaxOwn; }

bool tube32_serves(const ProbDesc& d) {
    // no residual norms are formed
    return d.L.nd == 1 && d.kn[0] <= tube32_max_cells() && !d.mp.norms;
}

int tube32_at_once(int solver, bool one, int cluster, int problems, int cells, int* threads) {
    if (cluster < 1 || cluster > kTailMaxCluster || cells < 2 || (cells + cluster - 1) / cluster > kMaxOwn) return 0;
    const int nt = block_threads(cluster, cells);
    if (threads) *threads = nt;
    auto at_once = [&]<int S, bool ONE, bool WIDE>() {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[1];
        int active = 0;
        config(cluster, problems, cells, cfg, attr);
        // (clusters of more than 8 CTAs: allowed once per instance, before any launch)
        if ((cluster > 8 && cudaFuncSetAttribute(k_tube32<S, ONE, WIDE>, cudaFuncAttributeNonPortableClusterSizeAllowed,
                                                 1) != cudaSuccess) ||
            cudaOccupancyMaxActiveClusters(&active, k_tube32<S, ONE, WIDE>, &cfg) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        return active;
    };
    return with_instance(solver, nt, [&]<int S, bool WIDE>() {
        return one ? at_once.template operator()<S, true, WIDE>() : at_once.template operator()<S, false, WIDE>();
    });
}

cudaError_t tube32_launch_one(int cluster, const ProbDesc& d, int budget, cudaStream_t st) {
    if (budget <= 0) return cudaSuccess;
    return with_instance(d.mp.solver, block_threads(cluster, d.kn[0]), [&]<int S, bool WIDE>() {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[1];
        config(cluster, 1, d.kn[0], cfg, attr);
        cfg.stream = st;
        return cudaLaunchKernelEx(&cfg, k_tube32<S, true, WIDE>, d, (const ProbDesc*)nullptr, (const int*)nullptr, budget, 0);
    });
}

cudaError_t tube32_launch(int solver, int cluster, int problems, int cells, const ProbDesc* d_probs, const int* d_list,
                          int budget, bool stop_unhealthy, cudaStream_t st) {
    if (problems <= 0 || budget <= 0) return cudaSuccess;
    ProbDesc none;
    std::memset(&none, 0, sizeof none);
    return with_instance(solver, block_threads(cluster, cells), [&]<int S, bool WIDE>() {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[1];
        config(cluster, problems, cells, cfg, attr);
        cfg.stream = st;
        return cudaLaunchKernelEx(&cfg, k_tube32<S, false, WIDE>, none, d_probs, d_list, budget, stop_unhealthy ? 1 : 0);
    });
}

}  // namespace ts
