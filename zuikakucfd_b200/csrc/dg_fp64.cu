// Discontinuous Galerkin P=1..3 stage, FP64, the reference's arithmetic op
// for op (compiled with --fmad=false, like weno_fp64.cu).
//
// Per RK stage two kernels, both on segments of 32 columns of a row:
//   dg_face_kernel<P>   every x and y interface flux ONCE: traces of both cells
//                       at the NQ Gauss points of the face (ghost neighbours
//                       gathered through the fill source map), HLLC or HLL; the
//                       reference computes each face twice from identical
//                       inputs.
//   dg_cell_kernel<P>   P + 1 threads per cell: volume quadrature, the four
//                       face integrals in the reference's order (right, left,
//                       bottom, top), inverse-mass scaling, the Shu-Osher
//                       combine and the Persson + Zhang-Shu limiter; ghosts get
//                       the combine of their filled value, exactly as the
//                       whole-array reference does.
// Basis values are tabulated on the host (no FMA contraction) with the
// reference's own expressions and kept in __constant__ memory, one table set
// per P.
#include <cmath>
#include <cstring>
#include <mutex>

#include "batch.cuh"
#include "chain.cuh"
#include "context_id.h"
#include "dg_common.cuh"
#include "fp64_div.cuh"
#include "zk_internal.h"

// Built twice: with --fmad=false as the reference-arithmetic path (namespace
// zk), and with -DZK_FP64_FMA, fused multiply-adds contracted and the cell
// integrals sum-factorised, as the ZK_PREC_FP64_FMA path (namespace zk_fma).
#ifdef ZK_FP64_FMA
#define ZK_FP64_NS zk_fma
#else
#define ZK_FP64_NS zk
#endif

namespace ZK_FP64_NS {
using namespace zk;

#ifdef ZK_FP64_FMA
constexpr bool kFma = true;
#else
constexpr bool kFma = false;
#endif

__constant__ DGTab c_dgtab[3];

namespace {

// legP / legD, src_DG/fluid.cpp:34-55 (host; this translation unit's host code
// is compiled without FMA contraction)
double legP_h(int n, double x) {
    switch (n) {
        case 0: return 1.0;
        case 1: return x;
        case 2: return 0.5 * (3.0 * x * x - 1.0);
        case 3: return 0.5 * (5.0 * x * x * x - 3.0 * x);
        case 4: return 0.125 * (35.0 * x * x * x * x - 30.0 * x * x + 3.0);
        default: return 0.0;
    }
}
double legD_h(int n, double x) {
    switch (n) {
        case 0: return 0.0;
        case 1: return 1.0;
        case 2: return 3.0 * x;
        case 3: return 0.5 * (15.0 * x * x - 3.0);
        case 4: return 0.5 * (35.0 * x * x * x - 15.0 * x);
        default: return 0.0;
    }
}

// Gauss-Legendre nodes and weights, the decimal literals of
// src_DG/fluid.cpp:94-111 for NQ = 2..4.
const double kGLPt[5][4] = {{0}, {0},
                            {-0.5773502691896257, 0.5773502691896257, 0, 0},
                            {-0.7745966692414834, 0.0, 0.7745966692414834, 0},
                            {-0.8611363115940526, -0.3399810435848563, 0.3399810435848563, 0.8611363115940526}};
const double kGLWt[5][4] = {{0}, {0},
                            {1.0, 1.0, 0, 0},
                            {0.5555555555555556, 0.8888888888888888, 0.5555555555555556, 0},
                            {0.3478548451374538, 0.6521451548625461, 0.6521451548625461, 0.3478548451374538}};

}  // namespace

void dg_make_tables(int P, DGTab* T) {
    std::memset(T, 0, sizeof(DGTab));
    const int NQ = P + 1, NM = NQ * NQ;
    const double* PT = kGLPt[NQ];
    const double* WT = kGLWt[NQ];
    auto phi2 = [&](int m, double xi, double eta) { return legP_h(m / (P + 1), xi) * legP_h(m % (P + 1), eta); };
    for (int qa = 0; qa < NQ; ++qa)
        for (int qb = 0; qb < NQ; ++qb) {
            const int p = qa * NQ + qb;
            const double xi = PT[qa], eta = PT[qb];
            T->vw[p] = WT[qa] * WT[qb];
            for (int m = 0; m < NM; ++m) {
                T->vphi[p][m] = phi2(m, xi, eta);
                T->vdxi[p][m] = legD_h(m / (P + 1), xi) * legP_h(m % (P + 1), eta);
                T->vdet[p][m] = legP_h(m / (P + 1), xi) * legD_h(m % (P + 1), eta);
            }
        }
    for (int q = 0; q < NQ; ++q)
        for (int m = 0; m < NM; ++m) {
            // traces: right side (xi=+1), left (xi=-1), bottom (eta=+1), top (eta=-1)
            T->tr[0][q][m] = phi2(m, +1.0, PT[q]);
            T->tr[1][q][m] = phi2(m, -1.0, PT[q]);
            T->tr[2][q][m] = phi2(m, PT[q], +1.0);
            T->tr[3][q][m] = phi2(m, PT[q], -1.0);
            // face weights bv = phi2(m, face point) * w (src_DG/fluid.cpp:740,756,776,792)
            for (int f = 0; f < 4; ++f) T->bv[f][q][m] = T->tr[f][q][m] * WT[q];
        }
    // Zhang-Shu basis at 4x4 Gauss points, cubic factors dropped
    // (src_DG/fluid.cpp:808-823, :892-895)
    const double* G4 = kGLPt[4];
    for (int a = 0; a < 4; ++a)
        for (int b = 0; b < 4; ++b)
            for (int m = 0; m < NM; ++m) {
                const int px = m / (P + 1), py = m % (P + 1);
                const double x = G4[a], y = G4[b];
                const double fa = (px == 0) ? 1.0 : (px == 1) ? x : (px == 2) ? 0.5 * (3.0 * x * x - 1.0) : 0.0;
                const double fb = (py == 0) ? 1.0 : (py == 1) ? y : (py == 2) ? 0.5 * (3.0 * y * y - 1.0) : 0.0;
                T->zs[a * 4 + b][m] = fa * fb;
            }
}

void dg_make_sep(int P, DGSep* S) {
    std::memset(S, 0, sizeof(DGSep));
    const int NQ = P + 1;
    for (int n = 0; n < NQ; ++n) {
        for (int q = 0; q < NQ; ++q) {
            S->L[n][q] = legP_h(n, kGLPt[NQ][q]);
            S->D[n][q] = legD_h(n, kGLPt[NQ][q]);
        }
        S->E[n][0] = legP_h(n, +1.0);
        S->E[n][1] = legP_h(n, -1.0);
        for (int a = 0; a < 4; ++a) {
            const double x = kGLPt[4][a];
            S->Z[n][a] = (n == 0) ? 1.0 : (n == 1) ? x : (n == 2) ? 0.5 * (3.0 * x * x - 1.0) : 0.0;
        }
    }
    for (int q = 0; q < NQ; ++q) S->W[q] = kGLWt[NQ][q];
}

int dg_upload_tables(int P, const DGTab& T) {
    // __constant__ memory is per CUDA context: upload once per (context, P)
    static std::mutex mu;
    static PerContext uploaded[DG_MAXNQ];
    std::lock_guard<std::mutex> lock(mu);
    const cudaError_t e = uploaded[P].once(
        [&] { return cudaMemcpyToSymbol(c_dgtab, &T, sizeof(DGTab), sizeof(DGTab) * (P - 1)); });
    return e == cudaSuccess ? ZK_OK : ZK_ERR_CUDA;
}

namespace {

// Whether quotients of the momenta (and, whole, the energy) of state U by its
// floored density may take the shared reciprocal (fp64_div.cuh).
__device__ __forceinline__ bool momenta_plain(double rho, const double U[4]) {
    return in_range(rho) && rho < 0x1p100 && num_ok(U[1]) && num_ok(U[2]);
}
__device__ __forceinline__ bool state_plain(double rho, const double U[4]) {
    return momenta_plain(rho, U) && num_ok(U[3]);
}

// eulerFluxX / eulerFluxY, src_DG/fluid.cpp:123-143 (floors 1e-3)
__device__ __forceinline__ void euler_flux(const double U[4], double gam, double F[4], double G[4]) {
    const double eps = 1e-3;
    double rho = ref_max(U[0], eps), u, v;
    if (momenta_plain(rho, U)) {
        const double y = recip(rho);
        u = quot(U[1], rho, y);
        v = quot(U[2], rho, y);
    } else {
        u = U[1] / rho;
        v = U[2] / rho;
    }
    double p = ref_max((gam - 1.0) * (U[3] - 0.5 * rho * (u * u + v * v)), eps);
    F[0] = rho * u; F[1] = rho * u * u + p; F[2] = rho * u * v; F[3] = (U[3] + p) * u;
    G[0] = rho * v; G[1] = rho * u * v; G[2] = rho * v * v + p; G[3] = (U[3] + p) * v;
}

// hllcFlux, DG variant, src_DG/fluid.cpp:450-520, with plain divisions: for
// states outside fp64_div.cuh's ranges.
__device__ __noinline__ void hllc_dg_any(const double* L, const double* R, double gamma, double* F) {
    const double eps = 1e-5;
    double rhoL = ref_max(L[0], eps), uL = L[1] / rhoL, vL = L[2] / rhoL, EL = L[3] / rhoL;
    double pL = ref_max((gamma - 1.0) * (L[3] - 0.5 * rhoL * (uL * uL + vL * vL)), eps);
    double aL = sqrt(ref_max(gamma * pL / rhoL, eps));
    double rhoR = ref_max(R[0], eps), uR = R[1] / rhoR, vR = R[2] / rhoR, ER = R[3] / rhoR;
    double pR = ref_max((gamma - 1.0) * (R[3] - 0.5 * rhoR * (uR * uR + vR * vR)), eps);
    double aR = sqrt(ref_max(gamma * pR / rhoR, eps));
    double sqL = sqrt(rhoL), sqR = sqrt(rhoR);
    double den = sqL + sqR;
    if (den < eps) den = eps;
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
    if (fabs(den2) < eps) den2 = (den2 >= 0 ? eps : -eps);
    double Ss = num / den2;
    const bool left = (Ss >= 0.0);
    const double rho = left ? rhoL : rhoR, u = left ? uL : uR, v = left ? vL : vR;
    const double E = left ? EL : ER, p = left ? pL : pR, S = left ? SL : SR;
    const double* Us = left ? L : R;
    double denom = S - Ss;
    if (fabs(denom) < eps) denom = (denom >= 0 ? eps : -eps);
    double c = rho * (S - u) / denom;
    double term = (Ss - u) * (Ss + p / (rho * (S - u)));
    if (isnan(term) || isinf(term)) term = 0.0;
    double s1 = c * Ss, s2 = c * v, s3 = c * (E + term);
    F[0] = (rho * u) + S * (c - Us[0]);
    F[1] = (rho * u * u + p) + S * (s1 - Us[1]);
    F[2] = (rho * u * v) + S * (s2 - Us[2]);
    F[3] = ((Us[3] + p) * u) + S * (s3 - Us[3]);
}

// The same flux, quotients over a common denominator sharing its reciprocal:
// the same values formed in the same order.  Its 15 divisions and 6 square
// roots are over half of an interface's FP64 work (face pass with plain
// division: P=3 1024^2 419 us, now 373; contracted build 768^2 269, now 207).
__device__ __forceinline__ void hllc_dg(const double (&L)[4], const double (&R)[4], double gamma, double (&F)[4]) {
    const double eps = 1e-5;
    const double rhoL = ref_max(L[0], eps), rhoR = ref_max(R[0], eps);
    const double sqL = sqrt(rhoL), sqR = sqrt(rhoR);
    double den = sqL + sqR;
    if (den < eps) den = eps;
    bool ok = state_plain(rhoL, L) && state_plain(rhoR, R) && in_range(den);
    if (ok) {
        const double yL = recip(rhoL), yR = recip(rhoR), yd = recip(den);
        const double uL = quot(L[1], rhoL, yL), vL = quot(L[2], rhoL, yL), EL = quot(L[3], rhoL, yL);
        const double pL = ref_max((gamma - 1.0) * (L[3] - 0.5 * rhoL * (uL * uL + vL * vL)), eps);
        const double aL = sqrt(ref_max(quot(gamma * pL, rhoL, yL), eps));
        const double uR = quot(R[1], rhoR, yR), vR = quot(R[2], rhoR, yR), ER = quot(R[3], rhoR, yR);
        const double pR = ref_max((gamma - 1.0) * (R[3] - 0.5 * rhoR * (uR * uR + vR * vR)), eps);
        const double aR = sqrt(ref_max(quot(gamma * pR, rhoR, yR), eps));
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
            if (fabs(den2) < eps) den2 = (den2 >= 0 ? eps : -eps);
            const double Ss = divide(num, den2);
            const bool left = (Ss >= 0.0);
            const double rho = left ? rhoL : rhoR, u = left ? uL : uR, v = left ? vL : vR;
            const double E = left ? EL : ER, p = left ? pL : pR, S = left ? SL : SR;
            const double U0 = left ? L[0] : R[0], U1 = left ? L[1] : R[1], U2 = left ? L[2] : R[2],
                         U3 = left ? L[3] : R[3];
            double denom = S - Ss;
            if (fabs(denom) < eps) denom = (denom >= 0 ? eps : -eps);
            const double r = rho * (S - u);
            ok = in_range(den2) && in_range(denom) && in_range(r);
            const double c = divide(r, denom);
            const double term = (Ss - u) * (Ss + divide(p, r));  // finite: every factor is in range
            F[0] = rho * u + S * (c - U0);
            F[1] = rho * u * u + p + S * (c * Ss - U1);
            F[2] = rho * u * v + S * (c * v - U2);
            F[3] = (U3 + p) * u + S * (c * (E + term) - U3);
        }
    }
    if (!ok) {
        double l[4], r[4], f[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            l[c] = L[c];
            r[c] = R[c];
        }
        hllc_dg_any(l, r, gamma, f);
#pragma unroll
        for (int c = 0; c < 4; ++c) F[c] = f[c];
    }
}

// hlleFlux, src_DG/fluid.cpp:525-580 (the reference defines it, never calls it)
__device__ __forceinline__ void hlle_dg(const double L[4], const double R[4], double gamma, double F[4]) {
    const double eps = 1e-6;
    double rhoL = ref_max(L[0], eps), uL = L[1] / rhoL, vL = L[2] / rhoL, EL = L[3];
    double pL = ref_max((gamma - 1.0) * (EL - 0.5 * rhoL * (uL * uL + vL * vL)), eps);
    double aL = sqrt(ref_max(gamma * pL / rhoL, eps));
    double HL = (EL + pL) / rhoL;
    double rhoR = ref_max(R[0], eps), uR = R[1] / rhoR, vR = R[2] / rhoR, ER = R[3];
    double pR = ref_max((gamma - 1.0) * (ER - 0.5 * rhoR * (uR * uR + vR * vR)), eps);
    double aR = sqrt(ref_max(gamma * pR / rhoR, eps));
    double HR = (ER + pR) / rhoR;
    double sqL = sqrt(rhoL), sqR = sqrt(rhoR);
    double invDen = 1.0 / ref_max(sqL + sqR, eps);
    double u_roe = (sqL * uL + sqR * uR) * invDen;
    double v_roe = (sqL * vL + sqR * vR) * invDen;
    double h_roe = (sqL * HL + sqR * HR) * invDen;
    double c_roe = sqrt(ref_max((gamma - 1.0) * (h_roe - 0.5 * (u_roe * u_roe + v_roe * v_roe)), eps));
    double SL = ref_min(uL - aL, u_roe - c_roe);
    double SR = ref_max(uR + aR, u_roe + c_roe);
    double FL[4] = {rhoL * uL, rhoL * uL * uL + pL, rhoL * uL * vL, (EL + pL) * uL};
    double FR[4] = {rhoR * uR, rhoR * uR * uR + pR, rhoR * uR * vR, (ER + pR) * uR};
    if (SL >= 0.0) {
        for (int c = 0; c < 4; ++c) F[c] = FL[c];
    } else if (SR <= 0.0) {
        for (int c = 0; c < 4; ++c) F[c] = FR[c];
    } else {
        double invDiff = 1.0 / ref_max(SR - SL, eps);
        for (int c = 0; c < 4; ++c) F[c] = (SR * FL[c] - SL * FR[c] + SL * SR * (R[c] - L[c])) * invDiff;
    }
}

// Gathered dof read: the fill source of ghost cells, slip walls negating
// the normal momentum (src_DG/fluid.cpp:600-607, 625-632).
struct CellRef {
    size_t k;  // index to read
    int neg;   // conserved variable to negate (-1 = none)
};
__device__ __forceinline__ CellRef cell_ref(const DGArgs& a, size_t k) {
    const int8_t kd = a.kind[k] & KIND_MASK;
    if (kd < KIND_COPY) return {k, -1};
    return {(size_t)a.gsrc[k], kd == KIND_SLIP_X ? 1 : (kd == KIND_SLIP_Y ? 2 : -1)};
}

__device__ __forceinline__ void copy8_async(double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// ---- interface fluxes --------------------------------------------------------------
// One CTA takes the 32 x faces on the left of cells (i, j0 .. j0+31) and the
// 32 y faces above them; a warp takes one direction and QP of the NQ Gauss
// points of its 32 faces.  Both rows of cells are staged in shared memory once
// and serve both directions (a thread per face and direction read each cell
// twice from L2, and its 4 NQ traces took 128-146 registers: 4 CTAs of 4 warps
// per SM, FP64 pipe 40-45%).

// Gauss points per thread (a throughput choice: P = 3, 1024^2: 2 373 us, 1 475,
// 4 495).  A grid of few CTAs is bound by the latency of a thread's interface
// fluxes instead and takes one point per thread, see launch_stage.
constexpr int face_points(int P) { return P == 3 ? 2 : P + 1; }

template <int P, int QPT = face_points(P)>
struct FaceTile {
    static constexpr int NQ = P + 1, NM = NQ * NQ;
    static constexpr int QP = QPT;       // Gauss points per thread
    static constexpr int NWD = NQ / QP;  // warps per direction
    static constexpr int NTHREAD = 64 * NWD;
    double lo[4 * NM][34];  // row i, columns j0-1 .. j0+31
    double up[4 * NM][32];  // row i-1, columns j0 .. j0+31
};

template <int P, int QPT>
__device__ __forceinline__ void face_tile(const DGArgs& a, int j0, int i, FaceTile<P, QPT>& S) {
    using F = FaceTile<P, QPT>;
    constexpr int NM = F::NM, QP = F::QP, NW = F::NTHREAD / 32;
    const DGTab& T = c_dgtab[P - 1];
    const int ny = a.g.ny, nx = a.g.nx, pitch = a.g.pitch;
    const size_t plane = a.g.plane;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int j = j0 + lane;                      // < pitch: the padding columns are passive cells
    const size_t k = (size_t)i * pitch + j;
    const size_t kl = j > 0 ? k - 1 : k;          // j = 0 has no x face
    const bool cu = (a.kind[k] & KIND_MASK) == KIND_UPDATED;
    const bool need_x = j > 0 && j < nx && (cu || (a.kind[kl] & KIND_MASK) == KIND_UPDATED);
    const bool need_y = j < nx && (cu || (a.kind[k - pitch] & KIND_MASK) == KIND_UPDATED);
    if (!__any_sync(0xffffffffu, need_x || need_y)) return;  // the same cells in every warp
    const CellRef rc = cell_ref(a, k), ru = cell_ref(a, k - pitch);
    for (int v = w; v < 4 * NM; v += NW) {
        copy8_async(&S.lo[v][lane + 1], a.cur + (size_t)v * plane + rc.k);
        copy8_async(&S.up[v][lane], a.cur + (size_t)v * plane + ru.k);
    }
    const CellRef rl = cell_ref(a, j0 > 0 ? k - lane - 1 : k - lane);  // the column left of the tile
    for (int v = threadIdx.x; v < 4 * NM; v += F::NTHREAD) copy8_async(&S.lo[v][0], a.cur + (size_t)v * plane + rl.k);
    copy_commit();
    copy_wait<0>();
    // slip walls: each thread negates what it copied
    if (rc.neg >= 0 || ru.neg >= 0)
        for (int v = w; v < 4 * NM; v += NW) {
            if (rc.neg == v / NM) S.lo[v][lane + 1] = -S.lo[v][lane + 1];
            if (ru.neg == v / NM) S.up[v][lane] = -S.up[v][lane];
        }
    if (rl.neg >= 0)
        for (int v = threadIdx.x; v < 4 * NM; v += F::NTHREAD)
            if (rl.neg == v / NM) S.lo[v][0] = -S.lo[v][0];
    __syncthreads();

    const bool ydir = w >= F::NWD;
    const int q0 = (ydir ? w - F::NWD : w) * QP;
    if (!(ydir ? need_y : need_x)) return;
    const double* pl = ydir ? &S.up[0][lane] : &S.lo[0][lane];
    const int sl = ydir ? 32 : 34;
    const double* pr = &S.lo[0][lane + 1];
    const double(*tl)[DG_MAXNM] = T.tr[ydir ? 2 : 0];
    const double(*tr)[DG_MAXNM] = T.tr[ydir ? 3 : 1];
    double UL[QP][4], UR[QP][4];
#pragma unroll
    for (int u = 0; u < QP; ++u)
#pragma unroll
        for (int c = 0; c < 4; ++c) UL[u][c] = UR[u][c] = 0.0;
#pragma unroll
    for (int m = 0; m < NM; ++m)
#pragma unroll
        for (int u = 0; u < QP; ++u) {
            const double bl = tl[q0 + u][m], br = tr[q0 + u][m];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                UL[u][c] += pl[(c * NM + m) * sl] * bl;
                UR[u][c] += pr[(c * NM + m) * 34] * br;
            }
        }
    const size_t qstride = ydir ? (size_t)(ny + 1) * pitch : (size_t)ny * a.xpitch;
    double* out = ydir ? a.fy + k : a.fx + (size_t)i * a.xpitch + j;
#pragma unroll
    for (int u = 0; u < QP; ++u) {
        // y faces: normal momentum into slot 1, and back (src_DG/fluid.cpp:772-774)
        const double l[4] = {UL[u][0], ydir ? UL[u][2] : UL[u][1], ydir ? UL[u][1] : UL[u][2], UL[u][3]};
        const double r[4] = {UR[u][0], ydir ? UR[u][2] : UR[u][1], ydir ? UR[u][1] : UR[u][2], UR[u][3]};
        double f[4];
        if (a.hll) hlle_dg(l, r, a.gamma, f);
        else hllc_dg(l, r, a.gamma, f);
        double* o = out + (size_t)((q0 + u) * 4) * qstride;
        o[0] = f[0];
        o[qstride] = ydir ? f[2] : f[1];
        o[2 * qstride] = ydir ? f[1] : f[2];
        o[3 * qstride] = f[3];
    }
}

// Rows 3 .. ny-3 hold every face of an updated cell; TALL: from row `row0`, a
// variant of its own since the addition alone made the pass 1 to 4% longer.
template <int P, bool TALL, int QPT = face_points(P)>
__global__ void __launch_bounds__(FaceTile<P, QPT>::NTHREAD) dg_face_kernel(DGArgs a, int row0) {
    __shared__ FaceTile<P, QPT> S;
    chain_wait();
    face_tile(a, blockIdx.x * 32, (TALL ? row0 : 3) + blockIdx.y, S);
}

// ---- cells ---------------------------------------------------------------------------
// One CTA takes 32 cells of a row with one thread per cell and px: thread
// (lane, w) holds the 4 NQ modes m = w NQ .. w NQ + NQ - 1 of cell lane.
// Each mode's sum over the quadrature points, faces and limiter points keeps
// the reference's order, so the split changes no bit; what a thread needs from
// the others (the Euler fluxes at a point, each evaluated once, by warp
// w = its eta index) goes through shared memory.  A warp's global accesses are
// whole 256-byte row segments, its table reads are warp-uniform.  With one
// thread per cell the 64 accumulators of P = 3 spilled 656 bytes and the face
// fluxes arrived in 16 dependent rounds of loads (P=3 1024^2: 2,093 us, FP64
// pipe 28%); now 727 us (FP64 pipe 68%).  The same layout at P=2 203x331: 69 ->
// 29 us.
template <int P>
struct CellTile {
    static constexpr int NQ = P + 1, NM = NQ * NQ, NTHREAD = 32 * NQ;
    static constexpr int CH = P == 3 ? 2 : NQ;  // quadrature rows per round of point fluxes
    double sd[4 * NM][32];      // filled stage input; later the limiter's view of the result
    double fg[CH * NQ][8][32];  // F and G at the round's points; later the limiter's exchange
    double fx[4 * NQ][33], fyu[4 * NQ][32], fyd[4 * NQ][32];  // interface fluxes
    int bad[NQ][32];  // by eta index: variables with an F (bit c) or G (bit 4 + c) that is not finite
    // mode of thread (lane, w)'s n-th accumulator: px = w in the reference's
    // summation order, py = w where the sums are factorised
    static __device__ __forceinline__ int mode(int w, int n) { return kFma ? n * NQ + w : w * NQ + n; }
};

// applyLimiter (src_DG/fluid.cpp:824-992) on the tile: Persson modal filter
// (cells with persson set) then Zhang-Shu positivity, on the cells with `in`
// set.  o = the thread's modes.  Variable c's filter is evaluated by warp
// c mod NQ, point pt of the 16 positivity points by warp pt mod NQ; minima
// over the points are exact in any order.  A positivity pass whose outcome is
// known is skipped: |factor| <= 1, so point values lie within mean +- sum
// |modes|, and when that lower bound (less a 1e-12 relative margin, 500 times
// the rounding of a 16-term sum) clears the floor the pass returns exactly 1.
// Every thread of the CTA calls it; ends with every thread past its reads of S.
template <int P>
__device__ __forceinline__ void limit_tile(CellTile<P>& S, double (&o)[4][P + 1], bool in, bool persson,
                                           const DGTab& T, double gamma, double s0) {
    constexpr int NQ = P + 1, NM = NQ * NQ, NZ = NQ < 3 ? NQ : 3;
    const double kappa = 1.0, RHO_MIN = 1e-5, P_MIN = 1e-5, EPS = 1e-5;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double(*ex)[32] = S.fg[0];  // exchange rows of 32 lanes, through the flux buffer
    constexpr int FAC = 0, SPR = 4, THR = SPR + 4 * NQ, THP = THR + NQ;
    static_assert((THP + NQ) * 32 * sizeof(double) <= sizeof(S.fg), "the exchange rows fit the flux buffer");
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int n = 0; n < NQ; ++n) S.sd[c * NM + CellTile<P>::mode(w, n)][lane] = o[c][n];
    __syncthreads();
    for (int c = w; c < 4; c += NQ) {
        double f = 1.0;
        if (in && persson) {
            double Etot = 0.0, Ep = 0.0;
#pragma unroll
            for (int m = 0; m < NM; ++m) {
                const double x = S.sd[c * NM + m][lane];
                Etot += x * x;
                if (m / NQ == P || m % NQ == P) Ep += x * x;
            }
            const double s = log10(Ep / (Etot + EPS));
            if (s > s0) {
                double eps;
                if (s > s0 + kappa) eps = 1.0;
                else {
                    const double r = (s - s0) / kappa;
                    eps = 0.5 * (1.0 + sin(M_PI * (r - 0.5)));
                }
                f = 1.0 - eps;
            }
        }
        ex[FAC + c][lane] = f;
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const double f = ex[FAC + c][lane];
        double spread = 0.0;
#pragma unroll
        for (int n = 0; n < NQ; ++n) {
            if (w == P || n == P) {
                o[c][n] *= f;
                S.sd[c * NM + CellTile<P>::mode(w, n)][lane] = o[c][n];
            }
            if (w < NZ && n < NZ && (w || n)) spread += fabs(o[c][n]);
        }
        ex[SPR + c * NQ + w][lane] = spread;
    }
    __syncthreads();
    // means: density floor, pressure floor through the energy (every warp)
    const double rho0 = ref_max(S.sd[0][lane], RHO_MIN), mx0 = S.sd[NM][lane], my0 = S.sd[2 * NM][lane];
    double E0 = S.sd[3 * NM][lane];
    const double p0 = (gamma - 1.0) * (E0 - 0.5 * (mx0 * mx0 + my0 * my0) / rho0);
    if (p0 < P_MIN) E0 = P_MIN / (gamma - 1.0) + 0.5 * (mx0 * mx0 + my0 * my0) / rho0;
    if (in && w == 0) {
        o[0][0] = rho0;
        o[3][0] = E0;
    }
    double sp[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        sp[c] = ex[SPR + c * NQ][lane];
#pragma unroll
        for (int n = 1; n < NQ; ++n) sp[c] += ex[SPR + c * NQ + n][lane];
    }
    double theta_rho = 1.0;
    const bool rho_pass = in && !(rho0 - sp[0] - 1e-12 * (fabs(rho0) + sp[0]) > RHO_MIN);
    if (__syncthreads_or(rho_pass)) {
        double th = 1.0;
        if (rho_pass)
#pragma unroll 1
            for (int pt = w; pt < 16; pt += NQ) {
                asm volatile("" ::: "memory");  // the modes stay in shared memory
                double rho = 0.0 + rho0 * T.zs[pt][0];
#pragma unroll
                for (int m = 1; m < NM; ++m) rho += S.sd[m][lane] * T.zs[pt][m];
                if (rho < RHO_MIN) th = ref_min(th, (rho0 - RHO_MIN) / (rho0 - rho + EPS));
            }
        ex[THR + w][lane] = th;
        __syncthreads();
#pragma unroll
        for (int n = 0; n < NQ; ++n) theta_rho = ref_min(theta_rho, ex[THR + n][lane]);
        if (theta_rho < 1.0)
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
                for (int n = 0; n < NQ; ++n)
                    if (w || n) {
                        o[c][n] *= theta_rho;
                        S.sd[c * NM + CellTile<P>::mode(w, n)][lane] = o[c][n];
                    }
    }
    const double p_avg = (gamma - 1.0) * (E0 - 0.5 * (mx0 * mx0 + my0 * my0) / rho0);
    bool p_pass = in;
    {
        const double rlo = rho0 - sp[0] - 1e-12 * (fabs(rho0) + sp[0]);
        if (rlo > RHO_MIN) {  // theta_rho is 1 here
            const double mx = fabs(mx0) + sp[1], my = fabs(my0) + sp[2];
            const double ke = 0.5 * (mx * mx + my * my) / rlo;
            const double plo =
                (gamma - 1.0) * (E0 - sp[3] - ke) - 1e-12 * (gamma - 1.0) * (fabs(E0) + sp[3] + ke);
            if (plo > P_MIN) p_pass = false;
        }
    }
    double theta_p = 1.0;
    if (__syncthreads_or(p_pass)) {
        double th = 1.0;
        if (p_pass)
#pragma unroll 1
            for (int pt = w; pt < 16; pt += NQ) {
                asm volatile("" ::: "memory");
                const double f0 = T.zs[pt][0];
                double rho = 0.0 + rho0 * f0, mx = 0.0 + mx0 * f0, my = 0.0 + my0 * f0, E = 0.0 + E0 * f0;
#pragma unroll
                for (int m = 1; m < NM; ++m) {
                    const double phi = T.zs[pt][m];
                    rho += S.sd[m][lane] * phi;
                    mx += S.sd[NM + m][lane] * phi;
                    my += S.sd[2 * NM + m][lane] * phi;
                    E += S.sd[3 * NM + m][lane] * phi;
                }
                if (rho <= RHO_MIN) continue;
                const double u = mx / rho, v = my / rho;
                const double p = (gamma - 1.0) * (E - 0.5 * rho * (u * u + v * v));
                if (p < P_MIN) th = ref_min(th, (p_avg - P_MIN) / (p_avg - p + EPS));
            }
        ex[THP + w][lane] = th;
        __syncthreads();
#pragma unroll
        for (int n = 0; n < NQ; ++n) theta_p = ref_min(theta_p, ex[THP + n][lane]);
    }
    if (theta_p < 1.0)
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int n = 0; n < NQ; ++n)
                if (w || n) o[c][n] *= theta_p;
}

// The volume and face integrals of cell `lane` in the reference's order of
// operations (thread px = w), added to o.
template <int P>
__device__ __forceinline__ void integrals(const DGTab& T, CellTile<P>& S, double gamma, double (&o)[4][P + 1]) {
    constexpr int NQ = P + 1, NM = NQ * NQ, CH = CellTile<P>::CH;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int bad = 0;
    // volume integral (src_DG/fluid.cpp:698-718), CH rows of points at a time
#pragma unroll 1
    for (int qa0 = 0; qa0 < NQ; qa0 += CH) {
        double U[CH][4];
#pragma unroll
        for (int u = 0; u < CH; ++u)
#pragma unroll
            for (int c = 0; c < 4; ++c) U[u][c] = S.sd[c * NM][lane];  // phi_0 = 1
#pragma unroll
        for (int m = 1; m < NM; ++m)
#pragma unroll
            for (int u = 0; u < CH; ++u) {
                const double b = T.vphi[(qa0 + u) * NQ + w][m];
#pragma unroll
                for (int c = 0; c < 4; ++c) U[u][c] += S.sd[c * NM + m][lane] * b;
            }
#pragma unroll
        for (int u = 0; u < CH; ++u) {
            double F[4], G[4];
            euler_flux(U[u], gamma, F, G);
            int top = 0;  // the largest exponent
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                S.fg[u * NQ + w][c][lane] = F[c];
                S.fg[u * NQ + w][4 + c][lane] = G[c];
                top = max(top, max(__double2hiint(F[c]) & 0x7fffffff, __double2hiint(G[c]) & 0x7fffffff));
            }
            if (top >= 0x7ff00000)
#pragma unroll
                for (int c = 0; c < 4; ++c) bad |= (isfinite(F[c]) ? 0 : 1 << c) | (isfinite(G[c]) ? 0 : 16 << c);
        }
        __syncthreads();
        // terms whose basis derivative is 0 identically (d/dxi at px = 0,
        // d/deta at py = 0) add +-0 and are left out, or NaN for a flux that is
        // not finite: those are added at the end, from `bad`
#pragma unroll 1
        for (int pt = 0; pt < CH * NQ; ++pt) {
            const int p = qa0 * NQ + pt;
            const double coeff = T.vw[p];
            double F[4], G[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                F[c] = S.fg[pt][c][lane];
                G[c] = S.fg[pt][4 + c][lane];
            }
            if (w == 0) {
#pragma unroll
                for (int n = 1; n < NQ; ++n) {
                    const double det = T.vdet[p][n];
#pragma unroll
                    for (int c = 0; c < 4; ++c) o[c][n] += coeff * (G[c] * det);
                }
            } else {
                const double dx0 = T.vdxi[p][w * NQ];
#pragma unroll
                for (int c = 0; c < 4; ++c) o[c][0] += coeff * (F[c] * dx0);
#pragma unroll
                for (int n = 1; n < NQ; ++n) {
                    const double dxi = T.vdxi[p][w * NQ + n], det = T.vdet[p][w * NQ + n];
#pragma unroll
                    for (int c = 0; c < 4; ++c) o[c][n] += coeff * (F[c] * dxi + G[c] * det);
                }
            }
        }
        if (qa0 + CH < NQ) __syncthreads();
    }
    S.bad[w][lane] = bad;
    copy_wait<0>();
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NQ; ++q) bad |= S.bad[q][lane];
    if (bad)
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int n = 0; n < NQ; ++n)
                if ((w == 0 && (bad >> c & 1)) || (n == 0 && (bad >> (4 + c) & 1))) o[c][n] = NAN;
    // face integrals: right (-), left (+), bottom (-), top (+)
    // (src_DG/fluid.cpp:731-796).  P_n(+1) = 1 and P_n(-1) = (-1)^n exactly,
    // so an x face's weights are those of px = 0 up to sign, and a y face's
    // weight is one per thread: its product serves all NQ modes.
    const bool odd = w & 1;
#pragma unroll
    for (int q = 0; q < NQ; ++q)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const double f = S.fx[q * 4 + c][lane + 1];
#pragma unroll
            for (int n = 0; n < NQ; ++n) o[c][n] -= T.bv[0][q][n] * f;
        }
#pragma unroll
    for (int q = 0; q < NQ; ++q)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const double x = S.fx[q * 4 + c][lane], f = odd ? -x : x;
#pragma unroll
            for (int n = 0; n < NQ; ++n) o[c][n] += T.bv[0][q][n] * f;
        }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const double b = T.bv[2][q][w * NQ];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const double t = b * S.fyd[q * 4 + c][lane];
#pragma unroll
            for (int n = 0; n < NQ; ++n) o[c][n] -= t;
        }
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const double b = T.bv[2][q][w * NQ];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const double t = b * S.fyu[q * 4 + c][lane];
#pragma unroll
            for (int n = 0; n < NQ; ++n) o[c][n] += (n & 1) ? -t : t;
        }
    }
}

// The same integrals by sum factorisation (ZK_PREC_FP64_FMA; thread py = w):
// phi_m = P_px(xi) P_py(eta), so the state at a point contracts px first (own
// modes only) and py at the point, and the projection back contracts eta at
// fixed xi, then xi: 384 multiply-adds per thread at P=3 where the direct sums
// take 768.  With one fused launch per stage (two threads per cell, tile and
// interface fluxes in one CTA: 208 registers, 8 warps per SM, FP64 pipe 23%)
// the P=3 stage at 768^2 took 1,077 us, this pass and the face pass take
// 535.
template <int P>
__device__ __forceinline__ void integrals_factored(const DGTab& T, CellTile<P>& S, double gamma,
                                                   double (&o)[4][P + 1]) {
    constexpr int NQ = P + 1, NM = NQ * NQ, CH = CellTile<P>::CH;
    static_assert(NQ * NQ * 4 <= CH * NQ * 8, "the xi-contracted modes fit the flux buffer");
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // one-dimensional factors at Gauss point q: P_n, P_n', and P_n w_q
    auto L = [&](int n, int q) { return T.vphi[q * NQ][n * NQ]; };
    auto D = [&](int n, int q) { return T.vdxi[q * NQ][n * NQ]; };
    auto WL = [&](int n, int q) { return T.bv[2][q][n * NQ]; };
    double(*ex)[32] = S.fg[0];  // [py][qa][c]: own modes contracted over px
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        double v[NQ];
#pragma unroll
        for (int n = 0; n < NQ; ++n) v[n] = S.sd[c * NM + n * NQ + w][lane];
#pragma unroll
        for (int qa = 0; qa < NQ; ++qa) {
            double e = v[0];
#pragma unroll
            for (int n = 1; n < NQ; ++n) e += v[n] * L(n, qa);
            ex[(w * NQ + qa) * 4 + c][lane] = e;
        }
    }
    __syncthreads();
    double U[NQ][4];  // the state at the points (qa, qb = w)
#pragma unroll
    for (int qa = 0; qa < NQ; ++qa)
#pragma unroll
        for (int c = 0; c < 4; ++c) U[qa][c] = ex[qa * 4 + c][lane];
#pragma unroll
    for (int n = 1; n < NQ; ++n) {
        const double b = L(n, w);
#pragma unroll
        for (int qa = 0; qa < NQ; ++qa)
#pragma unroll
            for (int c = 0; c < 4; ++c) U[qa][c] += ex[(n * NQ + qa) * 4 + c][lane] * b;
    }
    __syncthreads();
#pragma unroll
    for (int qa0 = 0; qa0 < NQ; qa0 += CH) {
#pragma unroll
        for (int u = 0; u < CH; ++u) {
            double F[4], G[4];
            euler_flux(U[qa0 + u], gamma, F, G);
            const double coeff = T.vw[(qa0 + u) * NQ + w];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                S.fg[u * NQ + w][c][lane] = F[c] * coeff;
                S.fg[u * NQ + w][4 + c][lane] = G[c] * coeff;
            }
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < CH; ++u) {
            double f[4] = {0.0, 0.0, 0.0, 0.0}, g[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int qb = 0; qb < NQ; ++qb) {
                const double l = L(w, qb), d = D(w, qb);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    f[c] += S.fg[u * NQ + qb][c][lane] * l;
                    g[c] += S.fg[u * NQ + qb][4 + c][lane] * d;
                }
            }
#pragma unroll
            for (int n = 0; n < NQ; ++n)
#pragma unroll
                for (int c = 0; c < 4; ++c) o[c][n] += D(n, qa0 + u) * f[c] + L(n, qa0 + u) * g[c];
        }
        if (qa0 + CH < NQ) __syncthreads();
    }
    copy_wait<0>();
    __syncthreads();
    // face integrals: x faces weigh P_py = w's factor (one sum for all px),
    // y faces P_px's; P_n(+1) = 1, P_n(-1) = (-1)^n
    const bool odd = w & 1;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        double r = 0.0, l = 0.0, y[NQ];
#pragma unroll
        for (int n = 0; n < NQ; ++n) y[n] = 0.0;
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const double b = WL(w, q), u = S.fyu[q * 4 + c][lane];
            r += b * S.fx[q * 4 + c][lane + 1];
            l += b * S.fx[q * 4 + c][lane];
            const double t = (odd ? -u : u) - S.fyd[q * 4 + c][lane];
#pragma unroll
            for (int n = 0; n < NQ; ++n) y[n] += WL(n, q) * t;
        }
#pragma unroll
        for (int n = 0; n < NQ; ++n) o[c][n] += (((n & 1) ? -l : l) - r) + y[n];
    }
}

// Cells (i, j0 .. j0+31).  Returns the thread's max corner wave speed of the
// fluid cells written when want_lam (computeMaxSpeedDG_omp), else 0.  Ends with
// every thread past its reads of S, except for a caller's barrier.
template <int P>
__device__ __forceinline__ double cell_tile(const DGArgs& a, int j0, int i, CellTile<P>& S) {
    using C = CellTile<P>;
    constexpr int NQ = C::NQ, NM = C::NM;
    const DGTab& T = c_dgtab[P - 1];
    const int ny = a.g.ny, nx = a.g.nx;
    const size_t plane = a.g.plane;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int j = j0 + lane;  // < pitch: the padding columns are passive cells
    const size_t k = (size_t)i * a.g.pitch + j;
    const int8_t kd = a.kind[k] & KIND_MASK;
    const bool upd = kd == KIND_UPDATED;
    const bool work = __any_sync(0xffffffffu, upd);  // the same in every warp
    const CellRef r = cell_ref(a, k);

    for (int v = w; v < 4 * NM; v += NQ) copy8_async(&S.sd[v][lane], a.cur + (size_t)v * plane + r.k);
    copy_commit();
    if (work) {
        const size_t xq = (size_t)ny * a.xpitch, yq = (size_t)(ny + 1) * a.g.pitch;
        const double* fx = a.fx + (size_t)i * a.xpitch + j;
        for (int e = w; e < 4 * NQ; e += NQ) {
            copy8_async(&S.fx[e][lane], fx + e * xq);
            if (lane == 31) copy8_async(&S.fx[e][32], fx + e * xq + 1);
            copy8_async(&S.fyu[e][lane], a.fy + e * yq + k);
            copy8_async(&S.fyd[e][lane], a.fy + e * yq + k + a.g.pitch);
        }
    }
    copy_commit();
    if (a.stage > 0) {  // U^n towards L2; read by the combine
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int n = 0; n < NQ; ++n)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(a.un + (size_t)(c * NM + CellTile<P>::mode(w, n)) * plane + k));
    }
    copy_wait<1>();
    if (r.neg >= 0)  // slip walls: each thread negates what it copied
        for (int v = w; v < 4 * NM; v += NQ)
            if (v / NM == r.neg) S.sd[v][lane] = -S.sd[v][lane];
    __syncthreads();

    double o[4][NQ];
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int n = 0; n < NQ; ++n) o[c][n] = 0.0;
    if (work) {
        if constexpr (kFma) integrals_factored<P>(T, S, a.gamma, o);
        else integrals<P>(T, S, a.gamma, o);
        // inverse mass: (2px+1)(2py+1) * 0.5 / h (src_DG/fluid.cpp:800-804)
#pragma unroll
        for (int n = 0; n < NQ; ++n) {
            const double scale = (double)((2 * w + 1) * (2 * n + 1)) * a.inv2h;
#pragma unroll
            for (int c = 0; c < 4; ++c) o[c][n] = upd ? o[c][n] * scale : 0.0;
        }
    }

    if (a.stage == 0) {
        if (j < nx)
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
                for (int n = 0; n < NQ; ++n) a.out[(size_t)(c * NM + CellTile<P>::mode(w, n)) * plane + k] = o[c][n];
        return 0.0;
    }
    // Shu-Osher combine with dt applied (src_DG/fluid.cpp:1024-1026, 1036-1038, 1046-1048)
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int n = 0; n < NQ; ++n) {
            const int v = c * NM + CellTile<P>::mode(w, n);
            const double dn = a.un[(size_t)v * plane + k];
            const double dd = a.dt * o[c][n];
            const double x = S.sd[v][lane];
            if (a.stage == 1) o[c][n] = dn + dd;
            else if (a.stage == 2) o[c][n] = 0.75 * dn + 0.25 * (x + dd);
            else o[c][n] = (1.0 / 3.0) * dn + (2.0 / 3.0) * (x + dd);
        }
    if (a.limiter == ZK_LIMITER_REFERENCE && i >= 3 && i < ny - 3)
        limit_tile<P>(S, o, j >= 3 && j < nx - 3, upd, T, a.gamma, a.s0);
    if (upd && w == 0) {
        uint32_t flags = 0;
        if constexpr (kFma) {
            const double rho = o[0][0], mx = o[1][0], my = o[2][0], E = o[3][0];
            if (!isfinite(rho) || !isfinite(E)) flags |= STATUS_NAN;
            if (!((a.gamma - 1.0) * (E - 0.5 * (mx * mx + my * my) / rho) > 0.0)) flags |= STATUS_P;
        } else {
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (isnan(o[c][0])) flags |= STATUS_NAN;
        }
        if (!(o[0][0] > 0.0)) flags |= STATUS_RHO;
        if (flags) atomicOr(a.status, flags);
    }
    if (j < nx)
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int n = 0; n < NQ; ++n) a.out[(size_t)(c * NM + CellTile<P>::mode(w, n)) * plane + k] = o[c][n];
    if (!a.want_lam) return 0.0;
    // corner q by warp q mod NQ; corner values of the basis are +-1 (reduce_fp64.cu)
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int n = 0; n < NQ; ++n) S.sd[c * NM + CellTile<P>::mode(w, n)][lane] = o[c][n];
    __syncthreads();
    double umax = 0.0;
    if (j < nx && (a.kind[k] & KIND_FLUID))
        for (int q = w; q < 4; q += NQ) {
            double cs[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int m = 0; m < NM; ++m) {
                const bool neg = corner_odd<NQ>(m, q);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const double x = S.sd[c * NM + m][lane];
                    cs[c] += neg ? -x : x;
                }
            }
            umax = dg_state_speed(cs, a.gamma, umax);
        }
    return umax;
}

// CTAs per SM of the cell kernels: 128, 104 and 80 registers, no spills (P=2:
// 6 over 5 CTAs +1.2%; P=3: 5 CTAs at 100 registers the same time).
constexpr int cell_ctas(int P) { return P == 3 ? 4 : P == 2 ? 6 : 12; }

template <int P, bool TALL>  // TALL: as dg_face_kernel
__global__ void __launch_bounds__(CellTile<P>::NTHREAD, cell_ctas(P)) dg_cell_kernel(DGArgs a, int row0) {
    __shared__ CellTile<P> S;
    chain_wait();
    cell_tile<P>(a, blockIdx.x * 32, TALL ? row0 + blockIdx.y : blockIdx.y, S);
}

#ifndef ZK_FP64_FMA  // the batched runner has no FP64_FMA groups
// Stage-s arguments of batch item `it` (stage s reads U[s-1], writes U[s % 3]).
__device__ __forceinline__ DGArgs batch_args(const DgItem& it, int stage) {
    const BatchCtl* ctl = it.ctl;
    DGArgs a;
    a.cur = it.U[stage - 1];
    a.un = it.U[0];
    a.out = it.U[stage % 3];
    a.kind = it.kind;
    a.gsrc = it.gsrc;
    a.fx = it.fx;
    a.fy = it.fy;
    a.g = it.g;
    a.xpitch = it.xpitch;
    a.dt = ctl->dt;
    a.inv2h = it.inv2h;
    a.gamma = it.gamma;
    a.stage = stage;
    a.limiter = it.limiter;
    a.hll = it.hll;
    a.s0 = it.s0;
    a.status = &it.ctl->status;
    a.want_lam = stage == 3;
    return a;
}

// Persistent face pass of a batch group: a problem's tiles are its rows
// 3 .. ny-3 in segments of 32 columns.
template <int P>
__global__ void __launch_bounds__(FaceTile<P>::NTHREAD, P == 3 ? 5 : 8) dg_faces_fp64_batch_kernel(
    const DgItem* __restrict__ items, const int* __restrict__ dir, int cap, int stage) {
    __shared__ FaceTile<P> S;
    __shared__ DGArgs sa;
    __shared__ int s_job[3];  // stepping, row, segment start
    const int total = __ldg(dir + 1);
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
        if (threadIdx.x == 0) {
            const DirHit h = dir_lookup(dir, cap, t);
            const DgItem& it = items[h.item];
            s_job[0] = it.ctl->stepping;
            if (s_job[0]) {
                const int segs = (it.g.nx + 31) / 32, r = h.local / segs;
                s_job[1] = 3 + r;
                s_job[2] = (h.local - r * segs) * 32;
                sa = batch_args(it, stage);
            }
        }
        __syncthreads();
        if (s_job[0]) face_tile(sa, s_job[2], s_job[1], S);
        __syncthreads();
    }
}

// Persistent cell pass of a batch group: tiles are row segments of 32 cells.
template <int P>
__global__ void __launch_bounds__(CellTile<P>::NTHREAD, cell_ctas(P)) dg_cell_fp64_batch_kernel(
    const DgItem* __restrict__ items, const int* __restrict__ dir, int cap, int stage) {
    __shared__ CellTile<P> S;
    __shared__ DGArgs sa;
    __shared__ int s_job[3];  // stepping, row, segment start
    __shared__ unsigned long long* s_lam;
    const int total = __ldg(dir + 1);
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
        if (threadIdx.x == 0) {
            const DirHit h = dir_lookup(dir, cap, t);
            const DgItem& it = items[h.item];
            s_job[0] = it.ctl->stepping;
            if (s_job[0]) {
                const int segs = (it.g.nx + 31) / 32;
                s_job[1] = h.local / segs;
                s_job[2] = (h.local - s_job[1] * segs) * 32;
                sa = batch_args(it, stage);
                s_lam = &it.ctl->lam;
            }
        }
        __syncthreads();
        if (s_job[0]) {
            const double m = cell_tile<P>(sa, s_job[2], s_job[1], S);
            if (stage == 3) block_max_commit_to(m, s_lam);  // the next step's wave speed
        }
        __syncthreads();
    }
}

#endif

// applyLimiter alone, in place on the state (src_DG/fluid.cpp:824-992).
template <int P>
__global__ void __launch_bounds__(CellTile<P>::NTHREAD) dg_limit_kernel(DGArgs a) {
    constexpr int NQ = P + 1, NM = NQ * NQ;
    __shared__ CellTile<P> S;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int j = blockIdx.x * 32 + lane, i = 3 + blockIdx.y;
    const bool in = j >= 3 && j < a.g.nx - 3;
    const size_t plane = a.g.plane, k = (size_t)i * a.g.pitch + j;
    double o[4][NQ];
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int n = 0; n < NQ; ++n) o[c][n] = a.out[(size_t)(c * NM + CellTile<P>::mode(w, n)) * plane + k];
    limit_tile<P>(S, o, in, (a.kind[k] & KIND_MASK) == KIND_UPDATED, c_dgtab[P - 1], a.gamma, a.s0);
    if (in)
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int n = 0; n < NQ; ++n) a.out[(size_t)(c * NM + CellTile<P>::mode(w, n)) * plane + k] = o[c][n];
}

// One Gauss point per thread while the face pass has at most two CTAs per SM
// (a step on 148 SMs, us, several points and one; FP64 and FP64_FMA):
//             CTAs   P=1                    P=2                    P=3
//   64^2       118   31.3 27.4  28.5 25.1   43.9 36.0  38.2 31.1   51.7 47.9  40.2 37.3
//   96^2       273   31.1 27.7  28.7 25.6   46.1 39.2  39.8 33.8   56.7 55.9  45.7 45.1
//   128^2      492   32.5 31.1  30.7 29.6   50.4 49.4  45.6 48.6   85.1 86.6  65.9 71.4
//   192^2     1122   42.0 43.4  41.0 43.2   84.0 86.2  73.0 81.2   151  157   117  134
template <int P>
cudaError_t launch_stage(const DGArgs& a, cudaStream_t s) {
    constexpr int kRows = 65535;  // gridDim.y
    const int segs = (a.g.nx + 31) / 32, ny = a.g.ny, faces = ny - 5;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    if (ny <= kRows) {
        const dim3 grid(segs, faces);
        if ((long long)segs * faces <= 2 * sms)
            e = launch_chained(dg_face_kernel<P, false, 1>, grid, FaceTile<P, 1>::NTHREAD, 0, s, a, 0);
        else
            e = launch_chained(dg_face_kernel<P, false>, grid, FaceTile<P>::NTHREAD, 0, s, a, 0);
        if (e != cudaSuccess) return e;
        return launch_chained(dg_cell_kernel<P, false>, dim3(segs, ny), CellTile<P>::NTHREAD, 0, s, a, 0);
    }
    for (int r = 0; r < faces && e == cudaSuccess; r += kRows)
        e = launch_chained(dg_face_kernel<P, true>, dim3(segs, faces - r < kRows ? faces - r : kRows),
                           FaceTile<P>::NTHREAD, 0, s, a, 3 + r);
    for (int r = 0; r < ny && e == cudaSuccess; r += kRows)
        e = launch_chained(dg_cell_kernel<P, true>, dim3(segs, ny - r < kRows ? ny - r : kRows),
                           CellTile<P>::NTHREAD, 0, s, a, r);
    return e;
}

template <int P>
cudaError_t launch_limit(const DGArgs& a, cudaStream_t s) {
    dg_limit_kernel<P><<<dim3((a.g.nx + 31) / 32, a.g.ny - 6), CellTile<P>::NTHREAD, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_dg_stage_fp64(int P, const DGArgs& a, cudaStream_t s) {
    switch (P) {
        case 1: return launch_stage<1>(a, s);
        case 2: return launch_stage<2>(a, s);
        case 3: return launch_stage<3>(a, s);
        default: return cudaErrorInvalidValue;
    }
}

#ifndef ZK_FP64_FMA
// Batch tiles per problem: face pass (ny - 5) ceil(nx/32), cell pass ny ceil(nx/32).
int dg_fp64_batch_tiles(int pass, int ny, int nx) { return (pass == 0 ? ny - 5 : ny) * ((nx + 31) / 32); }

template <int P>
cudaError_t launch_batch_p(const DgItem* items, const int* dir_face, const int* dir_cell, int cap, int stage,
                           int grid_face, int grid_cell, cudaStream_t s) {
    dg_faces_fp64_batch_kernel<P><<<grid_face, FaceTile<P>::NTHREAD, 0, s>>>(items, dir_face, cap, stage);
    dg_cell_fp64_batch_kernel<P><<<grid_cell, CellTile<P>::NTHREAD, 0, s>>>(items, dir_cell, cap, stage);
    return cudaGetLastError();
}

// One FP64 DG stage of a batch group (face pass, then cell pass).
cudaError_t launch_dg_stage_fp64_batch(int P, const DgItem* items, const int* dir_face, const int* dir_cell, int cap,
                                       int stage, int grid_face, int grid_cell, cudaStream_t s) {
    switch (P) {
        case 1: return launch_batch_p<1>(items, dir_face, dir_cell, cap, stage, grid_face, grid_cell, s);
        case 2: return launch_batch_p<2>(items, dir_face, dir_cell, cap, stage, grid_face, grid_cell, s);
        case 3: return launch_batch_p<3>(items, dir_face, dir_cell, cap, stage, grid_face, grid_cell, s);
        default: return cudaErrorInvalidValue;
    }
}

// Resident CTAs per SM of the batch face (pass 0) and cell (pass 1) kernels.
int dg_fp64_batch_occupancy(int P, int pass) {
    int n = 0;
    switch (P * 2 + pass) {
        case 2: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, dg_faces_fp64_batch_kernel<1>, FaceTile<1>::NTHREAD, 0); break;
        case 3: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, dg_cell_fp64_batch_kernel<1>, CellTile<1>::NTHREAD, 0); break;
        case 4: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, dg_faces_fp64_batch_kernel<2>, FaceTile<2>::NTHREAD, 0); break;
        case 5: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, dg_cell_fp64_batch_kernel<2>, CellTile<2>::NTHREAD, 0); break;
        case 6: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, dg_faces_fp64_batch_kernel<3>, FaceTile<3>::NTHREAD, 0); break;
        case 7: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, dg_cell_fp64_batch_kernel<3>, CellTile<3>::NTHREAD, 0); break;
        default: break;
    }
    return n;
}

#endif

cudaError_t launch_dg_limit_fp64(int P, const DGArgs& a, cudaStream_t s) {
    switch (P) {
        case 1: return launch_limit<1>(a, s);
        case 2: return launch_limit<2>(a, s);
        case 3: return launch_limit<3>(a, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace ZK_FP64_NS
