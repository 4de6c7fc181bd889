// FP64 path of 1D problems: many steps per launch, one thread-block cluster,
// the state on chip.  The arithmetic is that of the stage kernels of
// ts_plain.cu, operation by operation (ts_cell64.cuh; --fmad=false), so the
// results are the same bits.
//
// What bounds it: latency.  A 1D step is a chain of about 150 FP64
// instructions, and a warp waits 64 clocks for each of them, whatever it has
// in parallel; the stage kernels add four or five launches with a few
// dependent trips to L2 each (20 to 25 us per step at any size below some
// thousand cells).  Here each CTA of the cluster owns up to 254
// consecutive cells, one per thread, in registers; a step needs two cluster barriers
// (390 clocks each, measured):
//   1  every cell's state in its CTA's shared memory, the two cells next to a
//      CTA boundary also in the neighbour's (distributed shared memory), the
//      ghost cells at the ends;
//   -  slopes of the own cells and of one cell beyond each end, the faces of
//      the own cells (those on a CTA boundary are solved by both CTAs, from
//      the same bits), V/SR and its minimum over the warp, written
//      to every CTA;
//   2  the minimum over the cluster: dt and the step's bookkeeping, repeated
//      by every thread on its own copy, and the update.
// The residuals are formed between a warp's arrival at the second barrier
// and the wait for it.  Two extra threads per CTA reconstruct the cells beyond
// its ends; the first of them also solves the face at its high end.
//
// Measured on one GB300, whole passes, stage kernels -> here: shock tube of
// 1000 cells to its end time (Roe, first order, 1736 steps) 40.0 -> 15.7 ms;
// 397 cells, HLLC, Barth-Jespersen, 64 steps 1650 -> 757 us.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "ts_cell64.cuh"
#include "ts_plain.h"

namespace ts {

namespace {

namespace cg = cooperative_groups;

constexpr int kMaxCtas = 16;       // CTAs of the cluster
constexpr int kMaxThreads = 256;
constexpr int kMaxOwn = kMaxThreads - 2;  // cells of a CTA
constexpr int kMaxWarps = kMaxThreads / 32;

// Shared memory of a CTA that owns up to `own` cells (doubles).
struct TubeMem {
    int u, hi, lo, f, total;  // state, high and low face states, face fluxes
    TS_HD explicit TubeMem(int own) {
        u = 0;
        hi = u + NV * (own + 4);
        lo = hi + NV * (own + 2);
        f = lo + NV * (own + 2);
        total = f + (NV + 1) * (own + 1);
    }
};

template <int SOLVER, int KIND>
__global__ void __launch_bounds__(kMaxThreads, 1) k_tube64(const __grid_constant__ PlainBufs b,
                                                           const __grid_constant__ Phys ph, int budget) {
    extern __shared__ double sm[];
    __shared__ u64 smin[kMaxCtas * kMaxWarps];
    __shared__ double snorm[NV][kMaxWarps], sall[NV][kMaxCtas];
    cg::cluster_group cluster = cg::this_cluster();
    if (b.ctl->stop_req) return;  // the same answer in every CTA
    const Layout& L = b.L;
    const int C = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int n = L.nx, base = n / C, rem = n % C;
    const int i0 = rank * base + min(rank, rem), m = base + (rank < rem);
    const int own_max = base + (rem > 0);
    const TubeMem at(own_max);
    const int pu = own_max + 4, ph_ = own_max + 2, pf = own_max + 1;  // pitches
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, W = blockDim.x >> 5;
    const bool own = tid < m;
    const bool per = ph.periodic[0];
    const int g0 = L.gx;
    Safe o;
    double u[NV], R[NV];
    double* const gu = b.U + L.at(i0 + tid, 0, 0);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        u[v] = own ? gu[v * L.plane] : 1.0;
        R[v] = 0.0;
    }
    // the cell this thread reconstructs (local index), and its geometry
    int rl = own ? tid : (tid == m ? -1 : m);
    bool rec = KIND != 0 && tid <= m + 1;
    int ri = i0 + rl;
    if (ri < 0 || ri >= n) {
        rec = rec && per;  // beyond a non-periodic side nothing is reconstructed
        ri = ri < 0 ? ri + n : ri - n;
    }
    typename Safe::Div sd[2];
    double hs = 0.0, eps2 = 0.0;
    if (rec) {
        const double* X = b.cx[0] + ri + g0;
        if (KIND == P_ENO2) {
            sd[0] = o.divisor(X[0] - X[-1]);
            sd[1] = o.divisor(X[1] - X[0]);
        } else {
            sd[0] = o.divisor(X[1] - X[-1]);
        }
        hs = o.half(b.ch[0][ri + g0]);
        if (KIND == P_LIM_VK) eps2 = b.eps2[L.at(ri, 0, 0)];
    }
    const double hy = b.ch[1][0], hz = b.ch[2][0];
    const double V = b.ch[0][min(i0 + tid, n - 1) + g0] * hy * hz;
    const double Vend = b.ch[0][n + g0] * hy * hz;  // of the ghost cell beyond the high side
    const typename Safe::Div iv = o.divisor(V);
    const bool last_cell = own && i0 + tid == n - 1;
    // ghost layers: of cells 0, 1 and n-1, n-2 (four cells at least).  Written when
    // the launch ends: a store to global memory in a step has to complete before
    // the barrier that follows it.
    const bool at_hi = own && n - 1 - (i0 + tid) < GHOST;
    const int layer = at_hi ? n - 1 - (i0 + tid) : (own && i0 + tid < GHOST ? i0 + tid : -1);
    double ghost[NV] = {1.0, 0.0, 0.0, 0.0, 1.0};
    const int idl = bc_id(ph.bc.mark, 0, 0), idr = bc_id(ph.bc.mark, 1, 0);
    // where this cell's state also goes: the neighbours' halo cells
    double *to_left = nullptr, *to_right = nullptr;
    {
        const int left = rank > 0 ? rank - 1 : (per ? C - 1 : -1), right = rank < C - 1 ? rank + 1 : (per ? 0 : -1);
        if (own && tid < 2 && left >= 0)
            to_left = cluster.map_shared_rank(sm + at.u, left) + base + (left < rem) + 2 + tid;
        if (own && tid >= m - 2 && right >= 0) to_right = cluster.map_shared_rank(sm + at.u, right) + (tid - m + 2);
    }
    u64* const remote_min = lane < C ? cluster.map_shared_rank(smin, lane) + rank * W + wid : nullptr;
    // the control word, kept by every thread
    double time = b.ctl->time, next_sol = b.ctl->next_sol, next_slice = b.ctl->next_slice, dt = 0.0, least = 0.0;
    const double save_sol = b.ctl->save_sol, save_slice = b.ctl->save_slice, max_time = b.ctl->max_time;
    int iteration = b.ctl->iteration;
    const int max_iteration = b.ctl->max_iteration;
    const bool run_mode = b.ctl->run_mode != 0;
    bool stop = false;
    unsigned int health = 0;
    cluster.sync();  // every CTA has started: its shared memory may be written
#pragma unroll 1
    for (int step = 0; step < budget && !stop; ++step) {
        // states and ghosts (k_ghost<0>)
        if (own) {
#pragma unroll
            for (int v = 0; v < NV; ++v) sm[at.u + v * pu + tid + 2] = u[v];
            if (to_left) {
#pragma unroll
                for (int v = 0; v < NV; ++v) to_left[v * pu] = u[v];
            }
            if (to_right) {
#pragma unroll
                for (int v = 0; v < NV; ++v) to_right[v * pu] = u[v];
            }
            if (layer >= 0) {
                // the ghost cell beyond the side (kept for the state's ghost layers)
#pragma unroll
                for (int v = 0; v < NV; ++v) ghost[v] = u[v];
                if (!per) {
                    bc_values(ph, at_hi ? idr : idl, 0, -1.0, u, ghost);
                    const int to = at_hi ? m + 2 + layer : 1 - layer;
#pragma unroll
                    for (int v = 0; v < NV; ++v) sm[at.u + v * pu + to] = ghost[v];
                }
            }
        }
        cluster.sync();
        // slopes (k_recon) as face states
        if constexpr (KIND != 0) {
            if (rec) {
                const double* s = sm + at.u + rl + 2;
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    const double val = s[v * pu];
                    double g, lim, proj;
                    const double nm = s[v * pu - 1], np = s[v * pu + 1];
                    recon_value<1, KIND, Safe>(val, &nm, &np, sd, &hs, eps2, &g, lim, &proj, o);
                    sm[at.hi + v * ph_ + rl + 1] = val + proj;
                    sm[at.lo + v * ph_ + rl + 1] = val - proj;
                }
            }
            __syncthreads();
        }
        // the face at the cell's low side (k_flux<0>); thread m: the CTA's high end
        if (tid <= m) {
            double UL[NV], UR[NV], F[NV];
            const int s = i0 + tid;
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                UL[v] = KIND != 0 ? sm[at.hi + v * ph_ + tid] : sm[at.u + v * pu + tid + 1];
                UR[v] = KIND != 0 ? sm[at.lo + v * ph_ + tid + 1] : sm[at.u + v * pu + tid + 2];
            }
            if (s == 0 && !per) bc_values(ph, idl, 0, 1.0, UR, UL);
            if (s == n && !per) bc_values(ph, idr, 0, 1.0, UL, UR);
            const bool thin = dzero(UL[2]) && dzero(UR[2]) && dzero(UL[3]) && dzero(UR[3]);
            double lam;
            bool full = !__all_sync(__activemask(), thin);
            if (!full) {
                lam = riemann<0, SOLVER, 1, Safe>(ph, UL, UR, F, o);
                // an infinity or NaN times a zero momentum is no zero (every factor of
                // a transverse term is one of the mass flux's too)
                full = !dfinite(F[0]);
            }
            if (full) lam = riemann<0, SOLVER, 3, Safe>(ph, UL, UR, F, o);
#pragma unroll
            for (int v = 0; v < NV; ++v) sm[at.f + v * pf + tid] = F[v];
            sm[at.f + NV * pf + tid] = lam;
        }
        __syncthreads();
        // V / SR (k_dt); the area of a 1D face is 1
        u64 r = kInfBits;
        if (own) {
            const double lo = sm[at.f + NV * pf + tid], hi = sm[at.f + NV * pf + tid + 1];
            r = ratio_bits(V, lo + hi);
            if (last_cell) r = umin64(r, ratio_bits(Vend, hi));
        }
        r = warp_min(r);
        if (remote_min) *remote_min = r;
        cg::cluster_group::arrival_token token = cluster.barrier_arrive();
        // R and R / V (k_update)
        double rv[NV];
        if (own) {
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                const double fh = sm[at.f + v * pf + tid + 1], fl = sm[at.f + v * pf + tid];
                const bool same = __double_as_longlong(fh) == __double_as_longlong(fl) &&
                                  (__double2hiint(fh) & 0x7FF00000) != 0x7FF00000;
                R[v] = same ? 0.0 : dneg_of(fh - fl);
            }
            if (ph.force || ph.accel) {
                const typename Safe::Div ro = o.divisor(u[0]);
                const double vu = o.over(u[1], ro), vv = o.over(u[2], ro), vw = o.over(u[3], ro);
                if (ph.force) {
                    R[1] += V * ph.sigma[0];
                    R[2] += V * ph.sigma[1];
                    R[3] += V * ph.sigma[2];
                    R[4] += (ph.sigma[0] * vu + ph.sigma[1] * vv + ph.sigma[2] * vw) * V;
                }
                if (ph.accel) {
                    const double r0 = u[0];
                    R[1] += r0 * V * ph.g[0];
                    R[2] += r0 * V * ph.g[1];
                    R[3] += r0 * V * ph.g[2];
                    R[4] += ((r0 * ph.g[0]) * vu + (r0 * ph.g[1]) * vv + (r0 * ph.g[2]) * vw) * V;
                }
            }
#pragma unroll
            for (int v = 0; v < NV; ++v) rv[v] = dzero(R[v]) ? 0.0 : o.over(R[v], iv);
        }
        cluster.barrier_wait(std::move(token));
        u64 all = kInfBits;
        for (int k = lane; k < C * W; k += 32) all = umin64(all, smin[k]);
        least = __longlong_as_double((long long)warp_min(all));
        dt = least * ph.cfl;
        if ((save_sol > 0) && (next_sol < time + dt)) dt = next_sol - time;
        if ((save_slice > 0) && (next_slice < time + dt)) dt = next_slice - time;
        if (own) {
            // (dt is infinite where no cell has a wave speed)
#pragma unroll
            for (int v = 0; v < NV; ++v)
                if (!dzero(R[v]) || !dfinite(dt)) u[v] = u[v] + dt * rv[v];
            health |= health_of(ph, u);
        }
        time += dt;
        iteration += 1;
        if (run_mode) {
            if ((save_sol > 0) && (next_sol == time)) next_sol += save_sol;
            if ((save_slice > 0) && (next_slice == time)) next_slice += save_slice;
            stop = iteration == max_iteration || time >= max_time;
        }
    }
    // state, health and the last step's norms V |R| (pairwise sums)
    if (own) {
#pragma unroll
        for (int v = 0; v < NV; ++v) gu[v * L.plane] = u[v];
    }
    if (layer >= 0) {
        double* dst = b.U + L.at(at_hi == !per ? n + layer : -1 - layer, 0, 0);
#pragma unroll
        for (int v = 0; v < NV; ++v) dst[v * L.plane] = ghost[v];
    }
    health = __reduce_or_sync(0xffffffffu, health);
    if (lane == 0 && health) atomicOr(&b.ctl->health, health);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        double s = own ? V * dabs(R[v]) : 0.0;
        for (int k = 16; k > 0; k >>= 1) s += __shfl_xor_sync(0xffffffffu, s, k);
        if (lane == 0) snorm[v][wid] = s;
    }
    __syncthreads();
    if (tid < NV) {
        double s = 0.0;
        for (int w = 0; w < W; ++w) s += snorm[tid][w];
        cluster.map_shared_rank(&sall[0][0], 0)[tid * kMaxCtas + rank] = s;
    }
    cluster.sync();
    if (rank == 0 && tid < NV) {
        double s = 0.0;
        for (int k = 0; k < C; ++k) s += sall[tid][k];
        b.ctl->res[tid] = s;
    }
    if (rank == 0 && tid == 0) {
        Ctl* c = b.ctl;
        c->time = time;
        c->dt = dt;
        c->dt_min_raw = least;
        c->next_sol = next_sol;
        c->next_slice = next_slice;
        c->iteration = iteration;
        c->stop_req = stop;
    }
}

template <class F>
bool with_tube(const Phys& ph, F&& f) {
    auto go = [&]<int S>() {
        if (ph.recon == TS_RECON_PIECEWISE_CONSTANT) return f.template operator()<S, 0>();
        if (ph.recon == TS_RECON_LINEAR_2POINTS) return f.template operator()<S, P_LINEAR>();
        if (ph.recon == TS_RECON_ENO2_2POINTS) return f.template operator()<S, P_ENO2>();
        if (ph.limiter == TS_LIM_VENKATAKRISHNAN) return f.template operator()<S, P_LIM_VK>();
        return f.template operator()<S, P_LIM_BJ>();
    };
    return ph.solver == TS_RS_HLLC ? go.template operator()<TS_RS_HLLC>() : go.template operator()<TS_RS_ROE_PIKE>();
}

template <int S, int K>
cudaError_t tube_config(const Layout& L, int ctas, cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr) {
    const int own = (L.nx + ctas - 1) / ctas;
    cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3((own + 2 + 31) / 32 * 32);
    cfg.dynamicSmemBytes = sizeof(double) * TubeMem(own).total;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaSuccess;
    if (ctas > 8) e = cudaFuncSetAttribute(k_tube64<S, K>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}

}  // namespace

int tube64_ctas(const Layout& L, const Phys& ph, int fold) {
    if (L.nd != 1 || L.nx < 4 || !fold || ph.viscous || ph.visc != 0.0) return 0;
    if (ph.solver != TS_RS_ROE_PIKE && ph.solver != TS_RS_HLLC) return 0;
    // about 30 cells, a warp, per CTA while the cluster has CTAs left
    int ctas = std::min(kMaxCtas, std::max(1, L.nx / 30));
    if ((L.nx + ctas - 1) / ctas > kMaxOwn) return 0;
    const bool ok = with_tube(ph, [&]<int S, int K>() {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[1];
        int active = 0;
        if (tube_config<S, K>(L, ctas, cfg, attr) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&active, k_tube64<S, K>, &cfg) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        return active > 0;
    });
    return ok ? ctas : 0;
}

cudaError_t tube64_steps(const PlainBufs& b, const Phys& ph, int ctas, int steps, cudaStream_t st) {
    cudaError_t e = cudaSuccess;
    with_tube(ph, [&]<int S, int K>() {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[1];
        e = tube_config<S, K>(b.L, ctas, cfg, attr);
        cfg.stream = st;
        if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, k_tube64<S, K>, b, ph, steps);
        return true;
    });
    return e;
}

}  // namespace ts
