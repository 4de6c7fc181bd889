// Plain FP64 path (bit-for-bit with the reference's CPU step): device buffers
// and the per-step launch sequence.  See ts_plain.cu.
#pragma once

#include <cuda_runtime.h>

#include "ts_internal.h"

namespace ts {

constexpr int kPlainBlock = 128;
// Most blocks of k_dt and k_update: 16 per SM of 152, whose threads then take
// up to 23 cells each at 192^3 (k_update 3.0 -> 0.72 ms there, with its
// divisions on the integer pipe).
constexpr int kPlainReduceBlocks = 152 * 16;

// Running sums that the blocks of k_update add each norm to (one per lane of
// the warp that sums them up).
constexpr int kNormSlots = 32;
constexpr unsigned kNormDirectBlocks = 512;

struct PlainBufs {
    Layout L;
    double* U;           // NV planes: conserved state
    // With `fold`, G holds the (limited) projections lim * (slope * h/2) to the
    // cell's high faces, and the low faces take their negatives.  Without it
    // (a periodic axis whose ghost cells differ in size from the cells they
    // repeat, so a face samples with another h) G holds slopes, Lim limiters.
    int fold;
    double* G;           // nd*NV planes, plane a*NV+v
    double* Lim;         // NV planes: limiter values (null with fold)
    double* F[3];        // NV planes per axis: face fluxes stored at the face's right cell
    double* Lam[3];      // 1 plane per axis: face max eigenvalue
    const double* cx[3]; // cell centres per axis, index i + ghost width
    const double* ch[3]; // cell sizes per axis
    const double* eps2;  // Venkatakrishnan eps^2 per cell (one plane) or null
    double* partial;     // per-block minima of V/SR
    double* norms;       // NV x kNormSlots running sums of V |R| (zero between steps)
    Ctl* ctl;
    double* VG;          // viscous flow: 9 planes, d(velocity d)/d(axis e) at plane 3d+e
    double* VSR[3];      // viscosity > 0: 1 plane per axis, the face's viscous
                         // spectral-radius term, stored at the face's right cell
};

int plain_partial_blocks(const Layout& L);

// Enqueues one step.  With `ev` non-null, records ev[0] before the first
// launch and ev[i+1] after launch i (ev needs kPlainMaxLaunches+1 events);
// *n_launch receives the launch count and names[i] the kernel names.
// With `side`, the ghost layers and the fluxes of the axes are launched beside
// one another (the step is then captured into a graph).
constexpr int kPlainMaxLaunches = 14;
struct PlainSide {
    cudaStream_t stream[2] = {nullptr, nullptr};
    cudaEvent_t fork = nullptr, join[2] = {nullptr, nullptr};
};
cudaError_t plain_step(const PlainBufs& b, const Phys& ph, cudaStream_t st, cudaEvent_t* ev = nullptr,
                       int* n_launch = nullptr, const char** names = nullptr, const PlainSide* side = nullptr);

// 1D problems: many steps per launch by one thread-block cluster that keeps
// the state on chip (ts_tube64.cu).  The CTAs of the cluster, or 0 when the
// problem takes the stage kernels.
int tube64_ctas(const Layout& L, const Phys& ph, int fold);
// `steps` steps (fewer when a Run ends) in one launch.
cudaError_t tube64_steps(const PlainBufs& b, const Phys& ph, int ctas, int steps, cudaStream_t st);

}  // namespace ts
