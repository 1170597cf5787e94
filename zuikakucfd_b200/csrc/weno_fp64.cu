// WENO5 + HLLC + SSP-RK3 stage, FP64, the reference's arithmetic op for op.
//
// This file is compiled with --fmad=false: every multiply and add rounds on
// its own, as the reference built with -ffp-contract=off does, so the result
// is bit-identical to it.  It is also the plain FP64 GPU path the mixed
// precision kernel is measured against.
//
// One CTA owns a tile of 32 columns and 2, 8 or 16 rows (launch_stage chooses
// by grid size).  It stages the tile plus a 3-cell halo of the stage input in
// shared memory (ghost cells already replaced by their fill source),
// reconstructs both face values of every cell and direction, computes every x
// and y interface flux of the tile ONCE (the reference computes each interface
// twice, from both neighbours; both evaluations see the same six inputs in the
// same order and give the same bits), then forms dU and the Shu-Osher combine
// for every cell of the tile, ghosts included, exactly as the reference's
// whole-array Eigen expressions do.
//
// Bound: the FP64 pipe.  A cell's smoothness indicators in one direction serve
// its left-biased value on one face and its right-biased value on the other
// (the same expressions of the same cells), so the reconstruction runs per
// cell: 3 indicators, 3 reciprocals and 5 weights where a face evaluates 6, 6
// and 6; and every division is branch-free (fp64_div.cuh).  About 1,070 FP64
// instructions per interface become 805: 177 -> 159 us a stage at 1024^2 (FP64
// pipe 65%; the staging, combine and barrier phases of three CTAs per SM leave
// the rest).
#include "batch.cuh"
#include "chain.cuh"
#include "context_id.h"
#include "fp64_div.cuh"
#include "zk_common.cuh"
#include "zk_kernels.h"

// Built twice: with --fmad=false as the reference-arithmetic path (namespace
// zk), and with -DZK_FP64_FMA, fused multiply-adds contracted, as the
// ZK_PREC_FP64_FMA path (namespace zk_fma).
#ifdef ZK_FP64_FMA
#define ZK_FP64_NS zk_fma
#else
#define ZK_FP64_NS zk
#endif

namespace ZK_FP64_NS {
using namespace zk;
namespace {

// A tile is 32 x TY cells; NW warps (TY + 1 by default) take the 2 TY + 2
// face-row tasks (TY + 1 x-face rows, TY + 1 y-face rows) in turn.
constexpr int TX = 32, HX = TX + 6;
template <int TY, int NW = TY + 1>
struct Tile {
    static constexpr int HY = TY + 6, NTHREAD = NW * 32;
};

// weno5_reconstruct, src_WENO/fluid.cpp:230-263, of one cell: from cells
// i-2 .. i+2 (A B C D E) the left-biased value on its face i+1/2 (UL there)
// and the right-biased value on its face i-1/2 (UR there).  Products by powers
// of two are exact, so an explicit fma with one rounds as the reference's
// separate multiply and add do.
//
// PLAIN: every stencil cell's values are plain (see stage_tile), which bounds
// the squared indicators by 1e-12 and 2^250 and the weights' sums likewise.
template <bool PLAIN>
__device__ __forceinline__ void weno5_weights(double t0, double t1, double t2, double (&a)[3], double (&e)[3],
                                              double& ia, double& ie) {
    const double q0 = t0 * t0, q1 = t1 * t1, q2 = t2 * t2;
    if (PLAIN && !ones_low(q0, q1, q2)) {
        const double y0 = recip(q0), y1 = recip(q1), y2 = recip(q2);
        a[0] = quot(0.1, q0, y0);
        a[1] = e[1] = quot(0.6, q1, y1);
        a[2] = quot(0.3, q2, y2);
        e[0] = quot(0.1, q2, y2);
        e[2] = quot(0.3, q0, y0);
        const double sa = a[0] + a[1] + a[2], se = e[0] + e[1] + e[2];
        if (!ones_low(sa, se)) {
            ia = recip(sa);
            ie = recip(se);
            return;
        }
    }
    a[0] = 0.1 / q0; a[1] = e[1] = 0.6 / q1; a[2] = 0.3 / q2;
    e[0] = 0.1 / q2; e[2] = 0.3 / q0;
    ia = 1.0 / (a[0] + a[1] + a[2]);
    ie = 1.0 / (e[0] + e[1] + e[2]);
}
template <bool PLAIN>
__device__ __forceinline__ void weno5_cell(double A, double B, double C, double D, double E, double& left,
                                           double& right) {
    const double eps = 1e-6, C1 = 13.0 / 12.0;
    const double C3 = 3 * C;
    const double d0 = __fma_rn(-2.0, B, A) + C, d1 = __fma_rn(-4.0, B, A) + C3;
    const double d2 = __fma_rn(-2.0, C, B) + D, d3 = B - D;
    const double d4 = __fma_rn(-2.0, D, C) + E, d5 = __fma_rn(-4.0, D, C3) + E;
    const double t0 = eps + __fma_rn(0.25, d1 * d1, C1 * d0 * d0);
    const double t1 = eps + __fma_rn(0.25, d3 * d3, C1 * d2 * d2);
    const double t2 = eps + __fma_rn(0.25, d5 * d5, C1 * d4 * d4);
    double a[3], e[3], ia, ie;
    weno5_weights<PLAIN>(t0, t1, t2, a, e, ia, ie);
    const double qL0 = (1.0 / 3.0) * A - (7.0 / 6.0) * B + (11.0 / 6.0) * C;
    const double qL1 = -(1.0 / 6.0) * B + (5.0 / 6.0) * C + (1.0 / 3.0) * D;
    const double qL2 = (1.0 / 3.0) * C + (5.0 / 6.0) * D - (1.0 / 6.0) * E;
    left = (a[0] * qL0 + a[1] * qL1 + a[2] * qL2) * ia;
    const double qR0 = (11.0 / 6.0) * C - (7.0 / 6.0) * D + (1.0 / 3.0) * E;
    const double qR1 = (1.0 / 3.0) * B + (5.0 / 6.0) * C - (1.0 / 6.0) * D;
    const double qR2 = -(1.0 / 6.0) * A + (5.0 / 6.0) * B + (1.0 / 3.0) * C;
    right = (e[0] * qR0 + e[1] * qR1 + e[2] * qR2) * ie;
}

// muscl_reconstruct, src_WENO/fluid.cpp:203-225 (not called by the reference's
// solvers; the ZK_RECON_MUSCL_* options): cells UL2, UL1 | UR1, UR2 around the
// face, slopes through minmod (LIM 0), van Leer (1) or superbee (2).
__device__ __forceinline__ double minmod2(double a, double b) {
    return a * b <= 0.0 ? 0.0 : (fabs(a) < fabs(b) ? a : b);
}
template <int LIM>
__device__ __forceinline__ double muscl_slope(double a, double b) {
    if constexpr (LIM == 0) {
        return minmod2(a, b);
    } else if constexpr (LIM == 1) {
        const double ab = a * b;
        return ab <= 0.0 ? 0.0 : 2.0 * ab / (a + b);
    } else {
        const double s1 = minmod2(a, 2.0 * b), s2 = minmod2(2.0 * a, b);
        return s1 * s2 <= 0.0 ? 0.0 : (fabs(s1) > fabs(s2) ? s1 : s2);
    }
}
// Both values of the face between u[1] and u[2] of four cells `st` apart.
template <int LIM>
__device__ __forceinline__ void muscl_face(const double* u, int st, double& left, double& right) {
    const double dL = u[st] - u[0], dC = u[2 * st] - u[st], dR = u[3 * st] - u[2 * st];
    left = u[st] + 0.5 * muscl_slope<LIM>(dL, dC);
    right = u[2 * st] - 0.5 * muscl_slope<LIM>(dC, dR);
}

// hllcFlux (WENO variant), src_WENO/fluid.cpp:268-317, with plain divisions:
// for operands outside fp64_div.cuh's ranges.
__device__ __noinline__ void hllc_any(const double* L, const double* R, double gamma, double* F) {
    const double eps = 1e-12;
    double rhoL = ref_max(L[0], eps), uL = L[1] / rhoL, vL = L[2] / rhoL, EL = L[3] / rhoL;
    double pL = ref_max((gamma - 1.0) * (L[3] - 0.5 * rhoL * (uL * uL + vL * vL)), eps);
    double aL = sqrt(gamma * pL / rhoL);
    double rhoR = ref_max(R[0], eps), uR = R[1] / rhoR, vR = R[2] / rhoR, ER = R[3] / rhoR;
    double pR = ref_max((gamma - 1.0) * (R[3] - 0.5 * rhoR * (uR * uR + vR * vR)), eps);
    double aR = sqrt(gamma * pR / rhoR);

    double sqL = sqrt(rhoL), sqR = sqrt(rhoR), den = sqL + sqR;
    double u_roe = (sqL * uL + sqR * uR) / den;
    double h_roe = (sqL * (EL + pL / rhoL) + sqR * (ER + pR / rhoR)) / den;
    double c_roe = sqrt(ref_max((gamma - 1.0) * (h_roe - 0.5 * u_roe * u_roe), eps));
    double SL = ref_min(uL - aL, u_roe - c_roe);
    double SR = ref_max(uR + aR, u_roe + c_roe);

    if (SL >= 0.0) {
        F[0] = rhoL * uL; F[1] = rhoL * uL * uL + pL; F[2] = rhoL * uL * vL; F[3] = (L[3] + pL) * uL;
        return;
    }
    if (SR <= 0.0) {
        F[0] = rhoR * uR; F[1] = rhoR * uR * uR + pR; F[2] = rhoR * uR * vR; F[3] = (R[3] + pR) * uR;
        return;
    }
    double num = pR - pL + rhoL * uL * (SL - uL) - rhoR * uR * (SR - uR);
    double den2 = rhoL * (SL - uL) - rhoR * (SR - uR);
    if (fabs(den2) < 1e-12) den2 = (den2 >= 0 ? 1e-12 : -1e-12);
    double Ss = num / den2;
    // star state of the upwind side (the reference's star_state lambda)
    const bool left = (Ss >= 0.0);
    const double rho = left ? rhoL : rhoR, u = left ? uL : uR, v = left ? vL : vR;
    const double E = left ? EL : ER, p = left ? pL : pR, S = left ? SL : SR;
    const double* Us = left ? L : R;
    double c = rho * (S - u) / (S - Ss);
    double s0 = c, s1 = c * Ss, s2 = c * v, s3 = c * (E + (Ss - u) * (Ss + p / (rho * (S - u))));
    double F0 = rho * u, F1 = rho * u * u + p, F2 = rho * u * v, F3 = (Us[3] + p) * u;
    F[0] = F0 + S * (s0 - Us[0]);
    F[1] = F1 + S * (s1 - Us[1]);
    F[2] = F2 + S * (s2 - Us[2]);
    F[3] = F3 + S * (s3 - Us[3]);
}

// The same flux for plain tiles: the same values formed in the same order,
// quotients over a common denominator sharing its reciprocal.  Plain cells
// reconstruct to values below 2^63 that are 0 or above 2^-620, so every
// quotient and remainder below is normal unless a difference underflows or
// vanishes: den2, r and d are tested.
__device__ __forceinline__ void hllc_plain(const double (&L)[4], const double (&R)[4], double gamma, double (&F)[4]) {
    const double eps = 1e-12;
    const double rhoL = ref_max(L[0], eps), rhoR = ref_max(R[0], eps);
    const double sqL = sqrt(rhoL), sqR = sqrt(rhoR), den = sqL + sqR;
    bool ok = !ones_low(rhoL, rhoR, den);
    {
        const double yL = recip(rhoL), yR = recip(rhoR);
        const double uL = quot(L[1], rhoL, yL), vL = quot(L[2], rhoL, yL), EL = quot(L[3], rhoL, yL);
        const double pL = ref_max((gamma - 1.0) * (L[3] - 0.5 * rhoL * (uL * uL + vL * vL)), eps);
        const double aL = sqrt(quot(gamma * pL, rhoL, yL));
        const double uR = quot(R[1], rhoR, yR), vR = quot(R[2], rhoR, yR), ER = quot(R[3], rhoR, yR);
        const double pR = ref_max((gamma - 1.0) * (R[3] - 0.5 * rhoR * (uR * uR + vR * vR)), eps);
        const double aR = sqrt(quot(gamma * pR, rhoR, yR));
        const double yd = recip(den);
        const double u_roe = quot(sqL * uL + sqR * uR, den, yd);
        const double h_roe =
            quot(sqL * (EL + quot(pL, rhoL, yL)) + sqR * (ER + quot(pR, rhoR, yR)), den, yd);
        const double c_roe = sqrt(ref_max((gamma - 1.0) * (h_roe - 0.5 * u_roe * u_roe), eps));
        const double SL = ref_min(uL - aL, u_roe - c_roe);
        const double SR = ref_max(uR + aR, u_roe + c_roe);
        if (SL >= 0.0) {
            F[0] = rhoL * uL; F[1] = rhoL * uL * uL + pL; F[2] = rhoL * uL * vL; F[3] = (L[3] + pL) * uL;
        } else if (SR <= 0.0) {
            F[0] = rhoR * uR; F[1] = rhoR * uR * uR + pR; F[2] = rhoR * uR * vR; F[3] = (R[3] + pR) * uR;
        } else {
            const double num = pR - pL + rhoL * uL * (SL - uL) - rhoR * uR * (SR - uR);
            double den2 = rhoL * (SL - uL) - rhoR * (SR - uR);
            if (fabs(den2) < 1e-12) den2 = (den2 >= 0 ? 1e-12 : -1e-12);
            const double Ss = divide(num, den2);
            const bool left = (Ss >= 0.0);
            const double rho = left ? rhoL : rhoR, u = left ? uL : uR, v = left ? vL : vR;
            const double E = left ? EL : ER, p = left ? pL : pR, S = left ? SL : SR;
            const double U0 = left ? L[0] : R[0], U1 = left ? L[1] : R[1], U2 = left ? L[2] : R[2],
                         U3 = left ? L[3] : R[3];
            const double r = rho * (S - u), d = S - Ss;
            ok = ok && in_range(den2) && in_range(r) && in_range(d);
            const double c = divide(r, d);
            const double s3 = c * (E + (Ss - u) * (Ss + divide(p, r)));
            F[0] = rho * u + S * (c - U0);
            F[1] = rho * u * u + p + S * (c * Ss - U1);
            F[2] = rho * u * v + S * (c * v - U2);
            F[3] = (U3 + p) * u + S * (s3 - U3);
        }
    }
    if (!ok) {
        double l[4], r[4], f[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            l[q] = L[q];
            r[q] = R[q];
        }
        hllc_any(l, r, gamma, f);
#pragma unroll
        for (int q = 0; q < 4; ++q) F[q] = f[q];
    }
}

struct StageArgs {
    const double* Ucur;  // stage input (ghosts unfilled)
    const double* Un;    // state at the start of the step
    double* Uout;        // stage output (may alias Un at stage 3: read-before-write per cell)
    const int8_t* kind;
    const int32_t* gsrc;
    Grid g;
    double dtdx, dtdy, gamma;
    int stage;  // 0: write dU only, 1..3: Shu-Osher stage
    uint32_t* status;
    int want_lam;  // 1: return the max wave speed of the cells written
};

template <int TY>
struct Smem {
    double sU[4][TY + 6][HX];
    // states left and right of each x / y face; the flux replaces the left one
    double xl[4][TY][TX + 1], xr[4][TY][TX + 1];
    double yl[4][TY + 1][TX], yr[4][TY + 1][TX];
    int8_t sK[TY + 6][HX];
};

// Both values of every face of a staged tile (WENO5), into S: one variable of
// a row of cells per warp task, TY x rows (columns 0 .. 31), the columns -1 and
// 32 of all x rows, TY + 2 y rows (rows -1 .. TY).
template <int TY, int NW, bool PLAIN>
__device__ __forceinline__ void weno5_faces(Smem<TY>& S, bool edge) {
    auto& sU = S.sU;
    auto& sK = S.sK;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int task = warp; task < 4 * (2 * TY + 3); task += NW) {
        const int q = task & 3, row = task >> 2;
        double left, right;
        if (row <= TY) {
            int r = row, c = lane;
            if (row == TY) {
                if (lane >= 2 * TY) continue;
                r = lane >> 1;
                c = (lane & 1) ? TX : -1;
            }
            if (edge) {
                const int8_t* k = &sK[r + 3][c + 3];
                if (k[-1] != KIND_UPDATED && k[0] != KIND_UPDATED && k[1] != KIND_UPDATED) continue;
            }
            const double* u = &sU[q][r + 3][c + 3];
            weno5_cell<PLAIN>(u[-2], u[-1], u[0], u[1], u[2], left, right);
            if (c < TX) S.xl[q][r][c + 1] = left;
            if (c >= 0) S.xr[q][r][c] = right;
        } else {
            const int r = row - TY - 2, c = lane;
            if (edge) {
                const int8_t* k = &sK[r + 3][c + 3];
                if (k[-HX] != KIND_UPDATED && k[0] != KIND_UPDATED && k[HX] != KIND_UPDATED) continue;
            }
            const double* u = &sU[q][r + 3][c + 3];
            weno5_cell<PLAIN>(u[-2 * HX], u[-HX], u[0], u[HX], u[2 * HX], left, right);
            if (r < TY) S.yl[q][r + 1][c] = left;
            if (r >= 0) S.yr[q][r][c] = right;
        }
    }
    __syncthreads();
}

// The interface fluxes of a staged tile, each computed once, left in S.xl and
// S.yl, a row of faces per warp task.  RECON 0: WENO5, the reference's scheme,
// from its own pass over the cells; else MUSCL with limiter RECON - 1, whose
// slopes are too few operations to pay for that pass and its barrier (a step
// with minmod, by cells / by faces: 192^2 30.1 / 18.9 us, 1024^2 271 / 233).
template <int TY, int NW, int RECON, bool PLAIN>
__device__ __forceinline__ void tile_fluxes(Smem<TY>& S, double gamma, bool edge) {
    auto& sU = S.sU;
    auto& sK = S.sK;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if constexpr (RECON == 0) weno5_faces<TY, NW, PLAIN>(S, edge);
    for (int task = warp; task < 2 * TY + 2; task += NW) {
        if (task <= TY) {
            // x face on the left of tile cell (r, c)
            int r, c;
            if (task < TY) { r = task; c = lane; }
            else { if (lane >= TY) continue; r = lane; c = TX; }
            if (edge && sK[r + 3][c + 2] != KIND_UPDATED && sK[r + 3][c + 3] != KIND_UPDATED) continue;
            double L[4], R[4], F[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if constexpr (RECON == 0) {
                    L[q] = S.xl[q][r][c];
                    R[q] = S.xr[q][r][c];
                } else {
                    muscl_face<RECON - 1>(&sU[q][r + 3][c + 1], 1, L[q], R[q]);
                }
            }
            if constexpr (PLAIN) hllc_plain(L, R, gamma, F);
            else hllc_any(L, R, gamma, F);
#pragma unroll
            for (int q = 0; q < 4; ++q) S.xl[q][r][c] = F[q];
        } else {
            // y face above tile cell (r, c); normal momentum swapped in
            const int r = task - TY - 1, c = lane;
            if (edge && sK[r + 2][c + 3] != KIND_UPDATED && sK[r + 3][c + 3] != KIND_UPDATED) continue;
            double L[4], R[4], F[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int v = q == 1 ? 2 : q == 2 ? 1 : q;
                if constexpr (RECON == 0) {
                    L[q] = S.yl[v][r][c];
                    R[q] = S.yr[v][r][c];
                } else {
                    muscl_face<RECON - 1>(&sU[v][r + 1][c + 3], HX, L[q], R[q]);
                }
            }
            if constexpr (PLAIN) hllc_plain(L, R, gamma, F);
            else hllc_any(L, R, gamma, F);
#pragma unroll
            for (int q = 0; q < 4; ++q) S.yl[q][r][c] = F[q];
        }
    }
}

// One tile whose top-left cell is (i0, j0).  Ends with every thread past its
// last shared-memory read, so a persistent caller may reuse S after a barrier.
// Returns the thread's max wave speed of the cells it wrote (want_lam), else 0.
template <int TY, int NW = TY + 1, int RECON = 0>
__device__ __forceinline__ double stage_tile(const StageArgs& a, int j0, int i0, Smem<TY>& S) {
    constexpr int HY = Tile<TY, NW>::HY, NTHREAD = Tile<TY, NW>::NTHREAD;
    auto& sU = S.sU;
    auto& sFx = S.xl;
    auto& sFy = S.yl;
    auto& sK = S.sK;
    const int ny = a.g.ny, nx = a.g.nx, pitch = a.g.pitch;
    const size_t plane = a.g.plane;

    // 1. tile + halo of the stage input, ghosts replaced by their source.
    //    Plain tiles hold |rho| < 2^60 and momenta and energies that are 0 or
    //    within 2^-200 .. 2^60 (fp64_div.cuh); edge tiles have cells in or
    //    beside the tile that are not updated, whose faces may not be needed.
    bool odd = false, border = false;
    for (int t = threadIdx.x; t < HY * HX; t += NTHREAD) {
        const int r = t / HX, c = t - r * HX;
        const int gi = i0 - 3 + r, gj = j0 - 3 + c;
        int8_t kd = KIND_PASSIVE;
        double v0 = 0.0, v1 = 0.0, v2 = 0.0, v3 = 0.0;
        if (gi >= 0 && gi < ny && gj >= 0 && gj < nx) {
            const size_t k = (size_t)gi * pitch + gj;
            kd = a.kind[k] & KIND_MASK;
            v0 = a.Ucur[k];  // beside the kind's load; ghosts load again
            v1 = a.Ucur[plane + k];
            v2 = a.Ucur[2 * plane + k];
            v3 = a.Ucur[3 * plane + k];
            if (kd >= KIND_COPY) {
                const size_t ks = (size_t)a.gsrc[k];
                v0 = a.Ucur[ks];
                v1 = a.Ucur[plane + ks];
                v2 = a.Ucur[2 * plane + ks];
                v3 = a.Ucur[3 * plane + ks];
            }
        }
        sU[0][r][c] = v0; sU[1][r][c] = v1; sU[2][r][c] = v2; sU[3][r][c] = v3;
        sK[r][c] = kd;
        odd |= !(fabs(v0) < 0x1p60 && plain_value(v1) && plain_value(v2) && plain_value(v3));
        border |= kd != KIND_UPDATED && r >= 2 && r < TY + 4 && c >= 2 && c < TX + 4;
    }
    const bool edge = __syncthreads_or(border);
    if (!__syncthreads_or(odd)) tile_fluxes<TY, NW, RECON, true>(S, a.gamma, edge);
    else tile_fluxes<TY, NW, RECON, false>(S, a.gamma, edge);
    __syncthreads();
    const int lane = threadIdx.x & 31;

    // 2. dU and the stage combine for every cell of the tile
    uint32_t flags = 0;
    double umax = 0.0;
    for (int t = threadIdx.x; t < TY * TX; t += NTHREAD) {
        const int r = t / TX, c = t - r * TX;
        const int gi = i0 + r, gj = j0 + c;
        if (gi >= ny || gj >= nx) continue;
        const size_t k = (size_t)gi * pitch + gj;
        const int8_t kd = sK[r + 3][c + 3];
        double d[4] = {0.0, 0.0, 0.0, 0.0};
        if (kd == KIND_UPDATED) {
            // src_WENO/fluid.cpp:454-460; y-face fluxes carry the momentum swap
            d[0] = -(a.dtdx * (sFx[0][r][c + 1] - sFx[0][r][c]) + a.dtdy * (sFy[0][r + 1][c] - sFy[0][r][c]));
            d[1] = -(a.dtdx * (sFx[1][r][c + 1] - sFx[1][r][c]) + a.dtdy * (sFy[2][r + 1][c] - sFy[2][r][c]));
            d[2] = -(a.dtdx * (sFx[2][r][c + 1] - sFx[2][r][c]) + a.dtdy * (sFy[1][r + 1][c] - sFy[1][r][c]));
            d[3] = -(a.dtdx * (sFx[3][r][c + 1] - sFx[3][r][c]) + a.dtdy * (sFy[3][r + 1][c] - sFy[3][r][c]));
        }
        double o[4];
        if (a.stage == 0) {
#pragma unroll
            for (int q = 0; q < 4; ++q) o[q] = d[q];
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const double un = a.Un[q * plane + k];
                const double v = sU[q][r + 3][c + 3];
                if (a.stage == 1) o[q] = un + d[q];
                else if (a.stage == 2) o[q] = 0.75 * un + 0.25 * (v + d[q]);
                else o[q] = (1.0 / 3.0) * un + (2.0 / 3.0) * (v + d[q]);
            }
            if (kd == KIND_UPDATED) {
                if (isnan(o[0]) || isnan(o[1]) || isnan(o[2]) || isnan(o[3])) flags |= STATUS_NAN;
                if (!(o[0] > 0.0)) flags |= STATUS_RHO;
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) a.Uout[q * plane + k] = o[q];
        if (a.want_lam) {
            const double spd = weno_cell_speed(o[0], o[1], o[2], o[3], a.gamma);
            if (spd > umax) umax = spd;
        }
    }
    flags = __reduce_or_sync(0xffffffffu, flags);
    if (flags && lane == 0) atomicOr(a.status, flags);
    return umax;
}

// Tiles of TY rows worked by NW warps, CTAS of them resident per SM.
template <int RECON, int TY, int NW, int CTAS>
__global__ void __launch_bounds__(NW * 32, CTAS) weno_stage_fp64_kernel(StageArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    chain_wait();
    stage_tile<TY, NW, RECON>(a, blockIdx.x * TX, blockIdx.y * TY, *reinterpret_cast<Smem<TY>*>(smem));
}

// Persistent stage over every listed problem of a batch group: CTA b takes
// global tiles b, b + gridDim.x, ...; stage s reads U[s-1] (U^n at stage 1)
// and writes U[s % 3].  Stage 3 also leaves the max wave speed of the new
// state (computeMaxSpeed over all cells) in the problem's control block.
// Tile variant V (batch.cuh); the register share is that of 864 threads per
// SM (72 registers).
template <int V, int TY = weno_variant_rows(V), int NW = weno_variant_warps(V)>
__global__ void __launch_bounds__(NW * 32, batch_min_blocks(NW * 32, 864, sizeof(Smem<TY>)))
    weno_stage_fp64_batch_kernel(const WenoItem* __restrict__ items, const int* __restrict__ dir, int cap,
                                 int stage) {
    extern __shared__ __align__(16) unsigned char smem[];
    Smem<TY>& S = *reinterpret_cast<Smem<TY>*>(smem);
    __shared__ StageArgs sa;  // the current tile's problem, kept out of registers
    __shared__ int s_org[3];  // tile origin x, y; 0 when the problem is not stepping
    __shared__ unsigned long long* s_lam;
    const int total = __ldg(dir + 1);
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
        if (threadIdx.x == 0) {
            const DirHit h = dir_lookup(dir, cap, t);
            const WenoItem& it = items[h.item];
            BatchCtl* ctl = it.ctl;
            s_org[2] = ctl->stepping;
            if (s_org[2]) {
                const int tiles_x = (it.g.nx + TX - 1) / TX;
                const int ty = h.local / tiles_x;
                s_org[0] = (h.local - ty * tiles_x) * TX;
                s_org[1] = ty * TY;
                sa = StageArgs{it.U[stage - 1], it.U[0], it.U[stage % 3], it.kind, it.gsrc, it.g,
                               ctl->dtdx, ctl->dtdy, it.gamma, stage, &ctl->status, stage == 3};
                s_lam = &ctl->lam;
            }
        }
        __syncthreads();
        if (s_org[2]) {
            const double m = stage_tile<TY, NW>(sa, s_org[0], s_org[1], S);
            if (stage == 3) block_max_commit_to(m, s_lam);  // the next step's wave speed
        }
        __syncthreads();
    }
}

}  // namespace

namespace {
template <auto kernel>
cudaError_t set_smem(size_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}
template <int V>
constexpr size_t batch_smem() { return sizeof(Smem<weno_variant_rows(V)>); }
template <int V>
cudaError_t batch_ready() {
    static PerContext attributes;
    return attributes.once([] { return set_smem<weno_stage_fp64_batch_kernel<V>>(batch_smem<V>()); });
}
template <int V>
cudaError_t launch_batch_v(const WenoItem* items, const int* dir, int cap, int stage, int grid, cudaStream_t s) {
    const cudaError_t e = batch_ready<V>();
    if (e != cudaSuccess) return e;
    weno_stage_fp64_batch_kernel<V><<<grid, weno_variant_warps(V) * 32, batch_smem<V>(), s>>>(items, dir, cap, stage);
    return cudaGetLastError();
}
template <int V>
int occupancy_v() {
    int n = 0;
    if (batch_ready<V>() != cudaSuccess) return 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, weno_stage_fp64_batch_kernel<V>, weno_variant_warps(V) * 32,
                                                  batch_smem<V>());
    return n;
}
template <int RECON, int TY, int NW, int CTAS>
cudaError_t launch_tiles(const StageArgs& a, cudaStream_t s) {
    const dim3 grid((a.g.nx + TX - 1) / TX, (a.g.ny + TY - 1) / TY);
    return launch_chained(weno_stage_fp64_kernel<RECON, TY, NW, CTAS>, grid, NW * 32, sizeof(Smem<TY>), s, a);
}

// Tile by the number of tiles.  Throughput favours 8 rows at 9 warps, 3 CTAs
// per SM at 72 registers (smaller tiles recompute more halo values per cell,
// larger ones leave one CTA per SM between its barriers), but a small grid is
// bound by one tile's latency on a chip mostly idle.  Stage times in us on 148
// SMs (graph replay; rows/warps x CTAs per SM; tiles of 8 rows):
//            8/9x3  2/14x2  8/18x1  16/26x1
//   64^2     11.8     5.4     9.8    14.2       16 tiles
//   128^2    12.0     7.3    10.1    14.6       64
//   192^2    12.3    13.1    10.1    14.6      144
//   256^2    16.8    21.7    18.0    14.6      256
//   300^2    21.4    29.7    25.7    27.1      380
//   1024^2  158     331     246     188       4096
// so the 2-row tile while two per SM are all resident, then one wider tile of
// 8, then of 16 rows per SM while that suffices, else 8/9.  Tile rows of ghosts
// alone do not count (33 x 1024: 9.8 us with 8/18, 13.4 with 16/26), and a grid
// just above one 8-row tile per SM stays with 8/9 while its updated rows would
// fit one (39 x 960: 12.1 against 14.5; 163 x 250, which does not: 16.2, 14.6).
template <int RECON>
cudaError_t launch_stage(const StageArgs& a, cudaStream_t s) {
    // every tile height at once: a later call with another grid may be inside a
    // stream capture, where no kernel should be loaded for the first time
    static PerContext attributes;
    const cudaError_t e = attributes.once([] {
        cudaError_t r = set_smem<weno_stage_fp64_kernel<RECON, 8, 9, 3>>(sizeof(Smem<8>));
        if constexpr (RECON == 0) {
            if (r == cudaSuccess) r = set_smem<weno_stage_fp64_kernel<0, 2, 14, 2>>(sizeof(Smem<2>));
            if (r == cudaSuccess) r = set_smem<weno_stage_fp64_kernel<0, 8, 18, 1>>(sizeof(Smem<8>));
            if (r == cudaSuccess) r = set_smem<weno_stage_fp64_kernel<0, 16, 26, 1>>(sizeof(Smem<16>));
        }
        return r;
    });
    if (e != cudaSuccess) return e;
    if constexpr (RECON == 0) {
        int dev = 0, sms = 0;
        cudaError_t q = cudaGetDevice(&dev);
        if (q == cudaSuccess) q = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (q != cudaSuccess) return q;
        const long long cols = (a.g.nx + TX - 1) / TX;
        auto tiles = [&](int rows) { return cols * ((a.g.ny - 3 + rows - 1) / rows); };
        if (tiles(2) <= 2 * sms) return launch_tiles<RECON, 2, 14, 2>(a, s);
        if (tiles(8) <= sms) return launch_tiles<RECON, 8, 18, 1>(a, s);
        if (cols * (a.g.ny - 6) > 8 * sms && tiles(16) <= sms) return launch_tiles<RECON, 16, 26, 1>(a, s);
    }
    return launch_tiles<RECON, 8, 9, 3>(a, s);
}
}  // namespace

cudaError_t launch_weno_stage_fp64_batch(int variant, const WenoItem* items, const int* dir, int cap, int stage,
                                         int grid, cudaStream_t s) {
    static_assert(kWenoVariants == 6, "one case per tile variant");
    switch (variant) {
        case 0: return launch_batch_v<0>(items, dir, cap, stage, grid, s);
        case 1: return launch_batch_v<1>(items, dir, cap, stage, grid, s);
        case 2: return launch_batch_v<2>(items, dir, cap, stage, grid, s);
        case 3: return launch_batch_v<3>(items, dir, cap, stage, grid, s);
        case 4: return launch_batch_v<4>(items, dir, cap, stage, grid, s);
        case 5: return launch_batch_v<5>(items, dir, cap, stage, grid, s);
        default: return cudaErrorInvalidValue;
    }
}

int weno_fp64_batch_occupancy(int variant) {
    switch (variant) {
        case 0: return occupancy_v<0>();
        case 1: return occupancy_v<1>();
        case 2: return occupancy_v<2>();
        case 3: return occupancy_v<3>();
        case 4: return occupancy_v<4>();
        case 5: return occupancy_v<5>();
        default: return 0;
    }
}

cudaError_t launch_weno_stage_fp64(const double* Ucur, const double* Un, double* Uout,
                                   const int8_t* kind, const int32_t* gsrc, const Grid& g,
                                   double dtdx, double dtdy, double gamma, int stage,
                                   uint32_t* status, cudaStream_t s, int recon) {
    StageArgs a{Ucur, Un, Uout, kind, gsrc, g, dtdx, dtdy, gamma, stage, status};
    switch (recon) {
        case 0: return launch_stage<0>(a, s);
        case 1: return launch_stage<1>(a, s);
        case 2: return launch_stage<2>(a, s);
        case 3: return launch_stage<3>(a, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace ZK_FP64_NS
