// Whole-grid FP64 kernels that are not stencils: the ghost fill applied in
// place, the CFL max-wavespeed reductions (WENO and DG semantics) and the
// primitive recovery.  Compiled with --fmad=false (reference arithmetic).
#include "batch.cuh"
#include "zk_common.cuh"
#include "zk_kernels.h"
#include "zuikaku.h"

namespace zk {
namespace {

// Ghost fill in place: U[g] = U[src(g)] for every filled cell, all nvar
// planes, with the slip-wall sign flips of src_DG/fluid.cpp:600-607,625-632.
// Sources are never filled cells, so the gather has no write/read hazard.
__global__ void fill_ghosts_kernel(double* U, const int8_t* kind, const int32_t* gsrc, Grid g,
                                   int nvar, int nm) {
    const size_t total = (size_t)g.ny * g.pitch;
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < total;
         k += (size_t)gridDim.x * blockDim.x) {
        const int8_t kd = kind[k] & KIND_MASK;
        if (kd < KIND_COPY) continue;
        const size_t s = (size_t)gsrc[k];
        for (int v = 0; v < nvar; ++v) {
            const int c = v / nm;  // conserved variable of plane v ([variable][mode] order)
            const bool neg = (kd == KIND_SLIP_X && c == 1) || (kd == KIND_SLIP_Y && c == 2);
            const double x = U[v * g.plane + s];
            U[v * g.plane + k] = neg ? -x : x;
        }
    }
}

__device__ __forceinline__ double warp_max(double m) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double x = __shfl_xor_sync(0xffffffffu, m, o);
        m = (x > m) ? x : m;
    }
    return m;
}

// Block max -> one atomicMax on the bit pattern.  Values are >= +0 and never
// NaN here, and the IEEE order of non-negative doubles is the integer order
// of their bits, so the integer max is the double max.
__device__ __forceinline__ void block_max_commit(double m, unsigned long long* out) {
    __shared__ double part[32];
    m = warp_max(m);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) part[warp] = m;
    __syncthreads();
    if (warp == 0) {
        m = (lane < (int)(blockDim.x >> 5)) ? part[lane] : 0.0;
        m = warp_max(m);
        if (lane == 0) atomicMax(out, (unsigned long long)__double_as_longlong(m));
    }
}

// The grid's max delivered to the host: like block_max_commit, and the last
// CTA to arrive stores the result in `host` (mapped host memory) and leaves
// the accumulator and ticket 0 for the next reduction.  A call is then one
// launch and a synchronise; clearing the accumulator and copying the result
// back were two more operations on the stream (64^2 WENO step with its wave
// speed: 53 -> 46 us).
__device__ __forceinline__ void block_max_deliver(double m, MaxSlot* slot, unsigned long long* host) {
    block_max_commit(m, &slot->max);
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&slot->ticket, 1u) == gridDim.x - 1) {
            *static_cast<volatile unsigned long long*>(host) = atomicExch(&slot->max, 0ull);
            slot->ticket = 0u;
        }
    }
}

// computeMaxSpeed, src_WENO/fluid.cpp:539-553: all cells, no floors; a NaN
// speed never wins (spd > umax is false), umax starts at 0.
//
// Bound: HBM (32 B per cell).  A thread takes two neighbouring cells per
// 16-byte load of each plane (rows are whole 256-byte lines, so pairs never
// straddle a row) and finds their column from one 32-bit remainder; with a
// 64-bit division and 8-byte loads per cell the 2048^2 reduction took 58 us
// (2.3 TB/s), it takes 34 us
// in this form, the FP64 divisions and square roots alongside.
__global__ void __launch_bounds__(256) max_speed_weno_kernel(const double* __restrict__ U, Grid g, double gamma,
                                                             MaxSlot* slot, unsigned long long* host) {
    double umax = 0.0;
    const uint32_t half = (uint32_t)g.pitch / 2, n = (uint32_t)g.ny * half;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int j = 2 * (int)(t % half);
        if (j >= g.nx) continue;
        const size_t k = 2 * (size_t)t;
        const double2 r = *reinterpret_cast<const double2*>(U + k);
        const double2 mx = *reinterpret_cast<const double2*>(U + g.plane + k);
        const double2 my = *reinterpret_cast<const double2*>(U + 2 * g.plane + k);
        const double2 E = *reinterpret_cast<const double2*>(U + 3 * g.plane + k);
        const double s0 = weno_cell_speed(r.x, mx.x, my.x, E.x, gamma);
        if (s0 > umax) umax = s0;
        if (j + 1 < g.nx) {
            const double s1 = weno_cell_speed(r.y, mx.y, my.y, E.y, gamma);
            if (s1 > umax) umax = s1;
        }
    }
    block_max_deliver(umax, slot, host);
}

// Largest corner wave speed of the DG cell at k, or umax
// (computeMaxSpeedDG_omp, src_DG/solver.cpp:26-64): the state at the corners
// (xi, eta) = (-1,-1), (+1,-1), (-1,+1), (+1,+1), summed over the modes in
// increasing order.  P_n(+1) = 1 and P_n(-1) = (-1)^n exactly, so a mode's
// corner values are +-1 times its coefficient: every coefficient is read once
// and enters the four sums by additions alone.
template <int P>
__device__ __forceinline__ double dg_corner_speed(const double* __restrict__ dof, size_t plane, size_t k,
                                                  double gamma, double umax) {
    constexpr int NQ = P + 1, NM = NQ * NQ;
    double cs[4][4] = {};
#pragma unroll
    for (int m = 0; m < NM; ++m)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const double x = dof[(size_t)(c * NM + m) * plane + k];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                cs[q][c] += corner_odd<NQ>(m, q) ? -x : x;
            }
        }
    return dg_cell_speed(cs, gamma, umax);
}

// computeMaxSpeedDG_omp over the bctype-0 cells of the whole grid.  Bound: HBM
// (32 NM B per cell, read once; with the corners in an outer loop each
// coefficient was read four times and P=3 at 2048^2 took 975 us, now 323 us).
template <int P>
__global__ void __launch_bounds__(256) max_speed_dg_kernel(const double* __restrict__ dof,
                                                           const int8_t* __restrict__ kind, Grid g, double gamma,
                                                           MaxSlot* slot, unsigned long long* host) {
    double umax = 0.0;
    const uint32_t pitch = (uint32_t)g.pitch, n = (uint32_t)g.ny * pitch;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        if ((int)(k % pitch) >= g.nx || !(kind[k] & KIND_FLUID)) continue;
        umax = dg_corner_speed<P>(dof, g.plane, k, gamma, umax);
    }
    block_max_deliver(umax, slot, host);
}

// recoverPrimitives, src_WENO/fluid.cpp:500-515 (mode-0 planes for DG).
// U points at variable 0 (mode 0 for DG); vs = plane stride between variables.
__global__ void recover_kernel(const double* U, Grid g, size_t vs, double gamma, double* prim) {
    const size_t n = (size_t)g.ny * g.nx;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n;
         t += (size_t)gridDim.x * blockDim.x) {
        const size_t i = t / g.nx, j = t - i * g.nx, k = i * g.pitch + j;
        double rho = U[k], ux = U[vs + k] / rho, vy = U[2 * vs + k] / rho;
        prim[k] = rho;
        prim[g.plane + k] = ux;
        prim[2 * g.plane + k] = vy;
        prim[3 * g.plane + k] = (gamma - 1.0) * (U[3 * vs + k] - 0.5 * rho * (ux * ux + vy * vy));
    }
}

// Mach number and speed of the cell averages, the plot notebook's
// compute_mach (plot.ipynb cell 0): |u| / sqrt(gamma p / rho), p recovered as
// recoverPrimitives does.  U points at variable 0 (mode 0 for DG); vs = plane
// stride between variables.
__global__ void mach_kernel(const double* U, Grid g, size_t vs, double gamma, double* mach, double* speed) {
    const size_t n = (size_t)g.ny * g.nx;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n;
         t += (size_t)gridDim.x * blockDim.x) {
        const size_t i = t / g.nx, j = t - i * g.nx, k = i * g.pitch + j;
        const double rho = U[k], ux = U[vs + k] / rho, vy = U[2 * vs + k] / rho;
        const double p = (gamma - 1.0) * (U[3 * vs + k] - 0.5 * rho * (ux * ux + vy * vy));
        const double vel = sqrt(ux * ux + vy * vy);
        speed[k] = vel;
        mach[k] = vel / sqrt(gamma * p / rho);
    }
}

// ---- batched runner: per-problem CFL reductions and step control ---------------

constexpr int kRedChunk = 2048;  // cells per reduction tile of the batched runner

// Max wave speed of every listed problem of a batch group that is not finished
// and whose speed the previous step's stage 3 did not already leave (first
// step after admission), committed to its control block (same per-cell semantics as the kernels
// above; the max is exact, so the tiling does not change the result).
__global__ void __launch_bounds__(256) max_speed_batch_kernel(const void* __restrict__ items, int method,
                                                              const int* __restrict__ dir, int cap) {
    const int total = __ldg(dir + 1);
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
        const DirHit h = dir_lookup(dir, cap, t);
        double umax = 0.0;
        BatchCtl* ctl;
        if (method == ZK_METHOD_DG) {
            const DgItem& it = static_cast<const DgItem*>(items)[h.item];
            ctl = it.ctl;
            if (ctl->state >= BATCH_DONE || ctl->lam_ready) continue;
            const Grid g = it.g;
            const size_t n = (size_t)g.ny * g.nx, c1 = min(n, (size_t)(h.local + 1) * kRedChunk);
            for (size_t c = (size_t)h.local * kRedChunk + threadIdx.x; c < c1; c += blockDim.x) {
                const size_t i = c / g.nx, j = c - i * g.nx, k = i * g.pitch + j;
                if (!(it.kind[k] & KIND_FLUID)) continue;
                switch (it.nm) {
                    case 4: umax = dg_corner_speed<1>(it.U[0], g.plane, k, it.gamma, umax); break;
                    case 9: umax = dg_corner_speed<2>(it.U[0], g.plane, k, it.gamma, umax); break;
                    default: umax = dg_corner_speed<3>(it.U[0], g.plane, k, it.gamma, umax); break;
                }
            }
        } else {
            const WenoItem& it = static_cast<const WenoItem*>(items)[h.item];
            ctl = it.ctl;
            if (ctl->state >= BATCH_DONE || ctl->lam_ready) continue;
            const Grid g = it.g;
            const double* U = it.U[0];
            const double gamma = it.gamma;
            const size_t n = (size_t)g.ny * g.nx, c1 = min(n, (size_t)(h.local + 1) * kRedChunk);
            for (size_t c = (size_t)h.local * kRedChunk + threadIdx.x; c < c1; c += blockDim.x) {
                const size_t i = c / g.nx, j = c - i * g.nx, k = i * g.pitch + j;
                const double spd =
                    weno_cell_speed(U[k], U[g.plane + k], U[2 * g.plane + k], U[3 * g.plane + k], gamma);
                if (spd > umax) umax = spd;
            }
        }
        block_max_commit(umax, &ctl->lam);
        __syncthreads();
    }
}

// End of a step (post): count it, log its dt, finish or fail the problem.
__device__ __forceinline__ void batch_ctl_post(BatchCtl& c) {
    if (!c.stepping) return;
    c.stepping = 0;
    c.dtlog[c.steps_done] = c.dt;
    c.steps_done += 1;
    c.t += c.dt;
    if (c.status & (STATUS_NAN | STATUS_TIMEOUT)) {
        c.state = BATCH_FAILED;
        c.t_done = global_ns();
    } else if (c.steps_done >= c.steps_target) {
        c.state = BATCH_DONE;
        c.t_done = global_ns();
    } else {
        c.lam_ready = 1;  // stage 3 left the new state's wave speed in lam
    }
}

// Start of a step (pre): admitted problems that are not finished take a time
// step from their CFL rule -- WENO dt = cfl da / lambda (the per-step form of
// src_WENO/solver.cpp:159-171), DG dt = cfl * dgSafeDt (src_DG/solver.cpp:19-23)
// -- and reset the speed accumulator.  A non-finite or non-positive dt fails
// the problem.
__device__ __forceinline__ void batch_ctl_pre(BatchCtl& c, bool admitted) {
    c.stepping = 0;
    if (!admitted || c.state >= BATCH_DONE) return;
    c.state = BATCH_RUNNING;
    const double lam = __longlong_as_double((long long)c.lam);
    c.lam = 0ull;
    c.lam_ready = 0;
    double dt;
    if (c.method == ZK_METHOD_DG) dt = c.cfl * (0.9 / (2.0 * (2 * c.order + 1)) * c.da / ref_max(lam, 1e-7));
    else dt = c.cfl * c.da / lam;
    if (!(dt > 0.0) || isinf(dt)) {
        c.state = BATCH_FAILED;
        c.status |= STATUS_NAN;
        c.t_done = global_ns();
        return;
    }
    c.dt = dt;
    c.dtdx = dt / c.da;
    c.dtdy = dt / c.da;
    c.stepping = 1;
}

// One thread per problem of the group: the end of a step and/or the start of
// the next.
__global__ void batch_ctl_kernel(BatchCtl* ctl, const int* __restrict__ members, int n,
                                 const int* __restrict__ admitted, bool post, bool pre) {
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
        const int id = members[s];
        if (post) batch_ctl_post(ctl[id]);
        if (pre) batch_ctl_pre(ctl[id], admitted[id]);
    }
}

__global__ void batch_clock_kernel(unsigned long long* t) { *t = global_ns(); }

int grid_for(size_t n, int threads, int sms) {
    size_t b = (n + threads - 1) / threads;
    size_t cap = (size_t)sms * 8;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (int)b;
}

}  // namespace

cudaError_t launch_fill_ghosts(double* U, const int8_t* kind, const int32_t* gsrc, const Grid& g,
                               int nvar, int nm, int sms, cudaStream_t s) {
    fill_ghosts_kernel<<<grid_for((size_t)g.ny * g.pitch, 256, sms), 256, 0, s>>>(U, kind, gsrc, g, nvar, nm);
    return cudaGetLastError();
}

cudaError_t launch_max_speed_weno(const double* U, const Grid& g, double gamma, MaxSlot* slot,
                                  unsigned long long* host, int sms, cudaStream_t s) {
    max_speed_weno_kernel<<<grid_for(g.plane / 2, 256, sms), 256, 0, s>>>(U, g, gamma, slot, host);
    return cudaGetLastError();
}

cudaError_t launch_max_speed_dg(const double* dof, const int8_t* kind, const Grid& g, int nm, double gamma,
                                MaxSlot* slot, unsigned long long* host, int sms, cudaStream_t s) {
    const int grid = grid_for(g.plane, 256, sms);
    switch (nm) {
        case 4: max_speed_dg_kernel<1><<<grid, 256, 0, s>>>(dof, kind, g, gamma, slot, host); break;
        case 9: max_speed_dg_kernel<2><<<grid, 256, 0, s>>>(dof, kind, g, gamma, slot, host); break;
        case 16: max_speed_dg_kernel<3><<<grid, 256, 0, s>>>(dof, kind, g, gamma, slot, host); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_recover(const double* U, const Grid& g, int nm, double gamma, double* prim,
                           int sms, cudaStream_t s) {
    recover_kernel<<<grid_for((size_t)g.ny * g.nx, 256, sms), 256, 0, s>>>(U, g, (size_t)nm * g.plane, gamma, prim);
    return cudaGetLastError();
}

cudaError_t launch_mach(const double* U, const Grid& g, int nm, double gamma, double* mach, double* speed, int sms,
                        cudaStream_t s) {
    mach_kernel<<<grid_for((size_t)g.ny * g.nx, 256, sms), 256, 0, s>>>(U, g, (size_t)nm * g.plane, gamma, mach, speed);
    return cudaGetLastError();
}

int batch_red_tiles(int ny, int nx) { return (int)(((size_t)ny * nx + kRedChunk - 1) / kRedChunk); }

cudaError_t launch_batch_max_speed(int method, const void* items, const int* dir, int cap, int grid, cudaStream_t s) {
    max_speed_batch_kernel<<<grid, 256, 0, s>>>(items, method, dir, cap);
    return cudaGetLastError();
}

cudaError_t launch_batch_ctl(bool post, bool pre, BatchCtl* ctl, const int* members, int n, const int* admitted,
                             cudaStream_t s) {
    batch_ctl_kernel<<<(n + 127) / 128, 128, 0, s>>>(ctl, members, n, admitted, post, pre);
    return cudaGetLastError();
}

cudaError_t launch_batch_clock(unsigned long long* t, cudaStream_t s) {
    batch_clock_kernel<<<1, 1, 0, s>>>(t);
    return cudaGetLastError();
}

}  // namespace zk
