// Equation: quadrature geometry on the device, DG residual (Equation::assemble),
// block Jacobian (Equation::jacobian) fused with the Newton-matrix update
// B = scale*J + M, mass matrix apply/solve, L2 norms and the projection of
// analytic fields (MeshFn::interp).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <new>

#include "internal.hpp"
#include "quadrature.hpp"

using namespace cpg;

namespace {

constexpr int nqf_of(int p) { return (2 * p <= 2) ? 2 : ((2 * p <= 4) ? 4 : 6); }

// ---------------------------------------------------------------------------
// Residual (Equation.cpp:152-191), a CTA of four warps per four cells, in two
// phases that alternate over chunks of the cells' quadrature points:
//
//  1. a thread per point, whatever cell it belongs to: state, flux, weight.
//     The weighted flux and the Legendre values P_1..P_p(xi), P_1..P_p(eta)
//     go to the point's row in shared memory.
//  2. a warp per cell: a lane takes every 16th point and half the components
//     with all test functions (every 32nd point of a scalar equation), with
//     gradients from P_1' = 1, P_2' = 3 P_1, P_3' = 5 P_2 + 1.  The lanes'
//     sums meet in a reduce-scatter.
//
// Bound by latency: the loads of a point's geometry and its neighbour's
// coefficients, and the barriers that wait for them (p = 3 Euler: FP64 units
// 26%, shared memory 31% busy; 96 registers, the point phase spills 176 bytes
// a thread, 5% of the loads and stores of L1).  So a point's loads are issued
// together, six CTAs share an SM (five at p = 3; one more or less costs 3-17%
// at either degree; eight of a scalar equation), and a row of 14 doubles
// serves 40 multiply-adds of a lane, which keeps shared memory's bandwidth out
// of the way.
// 50,000 p=3 Euler cells: 285 us; one warp per cell with a lane per point and
// all nb*nc sums in every lane (255 registers, 8 warps an SM) took 601 us,
// rows contracted by one lane per test function 359 us (63% of the shared-
// memory bandwidth), two points a thread 290 us (but 10% more at p=2).
// ---------------------------------------------------------------------------
// What follows a cell's residual R in a Runge-Kutta stage (each cell's own
// coefficients only, so no other cell's input is touched):
//   RES_PLAIN  out = R
//   RES_STAGE  k = dt M^{-1} R -> out; next = u0 + a k
//   RES_RK2    u0 += (k1 + k) / 2
//   RES_RK4    u0 += (k1 + 2 k2 + 2 k3 + k) / 6
enum { RES_PLAIN = 0, RES_STAGE = 1, RES_RK2 = 2, RES_RK4 = 3 };

constexpr int RES_T = 128, RES_CAP = 256;  // threads and chunk of points per CTA
// CTAs an SM: a scalar equation's rows are short
__host__ __device__ constexpr int res_ctas(int components, int degree) {
    return components == 1 ? 8 : (degree > 2 ? 5 : 6);
}

// u_c = sum_k U_c,k psi_k, the coefficients in pairs where they are 16-byte
// aligned
template <int P, int NC, bool VEC>
__device__ __forceinline__ void eval_state(const double (&psi)[nbasis<P>()], const double *U, double (&out)[NC]) {
    constexpr int NB = nbasis<P>();
#pragma unroll
    for (int e = 0; e < NC; e++) {
        double s = 0.0;
        if constexpr (VEC) {
#pragma unroll
            for (int m = 0; m < NB; m += 2) {
                const double2 v = *reinterpret_cast<const double2 *>(U + e * NB + m);
                s += v.x * psi[m];
                s += v.y * psi[m + 1];
            }
        } else {
#pragma unroll
            for (int m = 0; m < NB; m++) s += U[e * NB + m] * psi[m];
        }
        out[e] = s;
    }
}
template <int P>
__device__ __forceinline__ void basis_of(const double (&lx)[P + 1], const double (&ly)[P + 1],
                                         double (&psi)[nbasis<P>()]) {
    int k = 0;
#pragma unroll
    for (int a = 0; a <= P; a++)
#pragma unroll
        for (int d = 0; d <= P - a; d++) psi[k++] = lx[a] * ly[d];
}

// the Legendre values of a row, P_0 = 1 included
template <int P>
__device__ __forceinline__ void row_values(const double *row, double (&lx)[P + 1], double (&ly)[P + 1]) {
    double pl[2 * P];
#pragma unroll
    for (int l = 0; l < 2 * P; l += 2) {
        const double2 v = *reinterpret_cast<const double2 *>(row + l);
        pl[l] = v.x;
        pl[l + 1] = v.y;
    }
    lx[0] = ly[0] = 1.0;
#pragma unroll
    for (int l = 0; l < P; l++) {
        lx[l + 1] = pl[l];
        ly[l + 1] = pl[P + l];
    }
}
template <int N>
__device__ __forceinline__ void load_group(const double *p, double (&v)[N]) {
    if constexpr (N == 2) {
        const double2 t = *reinterpret_cast<const double2 *>(p);
        v[0] = t.x;
        v[1] = t.y;
    } else {
        v[0] = p[0];
    }
}

// Sums v[0..N) over the lanes that differ in the bits OFF, OFF/2, .. 1, each
// lane keeping the sums [base, base + lim) in v[0..lim): half of the values
// change hands at each step instead of all of them.
template <int N, int OFF>
__device__ __forceinline__ void reduce_scatter(double *v, int lane, int &base, int &lim) {
    constexpr int H = (N + 1) / 2;
    const bool hi = lane & OFF;
#pragma unroll
    for (int t = 0; t < H; t++) {
        const double a = v[t], b = t + H < N ? v[t + H] : 0.0;
        v[t] = (hi ? b : a) + __shfl_xor_sync(0xffffffffu, hi ? a : b, OFF);
    }
    base += hi ? H : 0;
    lim = hi ? max(lim - H, 0) : min(lim, H);
    if constexpr (OFF > 1) reduce_scatter<H, OFF / 2>(v, lane, base, lim);
}

// A state that is not admissible (Euler: density or pressure <= 0, or not
// finite) at any of the cell's quadrature points records the cell in
// *nonphys (cell + 1, first writer wins) for the host to report.
template <class Phys, int P, int MODE, int RES_CELLS>
__global__ void __launch_bounds__(RES_T, res_ctas(Phys::NC, P))
    k_residual(Geo g, Phys ph, BCParams bc, const double *__restrict__ u, double t, int *__restrict__ nonphys,
               double *out, cpg::RkStage rk) {
    constexpr int NB = nbasis<P>(), NC = Phys::NC, BL = NB * NC, NQF = nqf_of(P);
    constexpr int T = RES_T;
    static_assert(RES_CELLS <= T / 32, "a warp per cell");
    // a point's row: weighted fluxes, P_1..P_p(xi), P_1..P_p(eta), an odd
    // multiple of 16 bytes so that 8 rows' 16-byte accesses fall in distinct banks
    constexpr int XO = 2 * NC, WS = ((XO + 2 * P) / 2 | 1) * 2;
    constexpr bool VEC = NB % 2 == 0;  // a component's coefficients are whole pairs
    constexpr int NG = NC == 4 ? 2 : 1, CG = NC / NG, LG = 32 / NG;  // component groups, lanes of a group
    __shared__ __align__(16) double sW[RES_CAP][WS];
    __shared__ __align__(16) double sU[RES_CELLS][BL];
    __shared__ double2 sbox[RES_CELLS];  // 2 / width, 2 / height
    __shared__ int sv[RES_CELLS + 1], sf[RES_CELLS + 1];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int cell0 = blockIdx.x * RES_CELLS, nc = min(RES_CELLS, g.n - cell0);
    for (int r = tid; r < nc * BL; r += T) (&sU[0][0])[r] = u[(size_t)cell0 * BL + r];
    if (tid <= nc) {
        sv[tid] = g.vq_ptr[cell0 + tid];
        sf[tid] = g.f_ptr[cell0 + tid];
    }
    if (tid >= 32 && tid < 32 + nc) {
        const double4 box = g.bb[cell0 + tid - 32];
        sbox[tid - 32] = make_double2(2.0 / box.z, 2.0 / box.w);
    }
    const bool pairs = VEC && (reinterpret_cast<uintptr_t>(u) & 15) == 0;
    __syncthreads();
    const int v0 = sv[0], nv = sv[nc] - v0, nvp = (nv + 31) & ~31;  // faces start at a warp
    const int f0 = sf[0], total = nvp + (sf[nc] - f0) * NQF;
    const int grp = lane / LG, share = lane % LG;
    double acc[CG * NB];
#pragma unroll
    for (int e = 0; e < CG * NB; e++) acc[e] = 0.0;

    for (int base = 0; base < total; base += RES_CAP) {
        if (base) __syncthreads();
        for (int it = tid; it < RES_CAP && base + it < total; it += T) {
            const int idx = base + it;
            const bool vol = idx < nvp;
            if (vol && idx >= nv) continue;
            const int f = vol ? 0 : f0 + (idx - nvp) / NQF, q = vol ? v0 + idx : f0 * NQF + (idx - nvp);
            int c = 0;  // the point's cell
#pragma unroll
            for (int m = 1; m < RES_CELLS; m++) c += m < nc && (vol ? q >= sv[m] : f >= sf[m]) ? 1 : 0;
            // everything the point needs is loaded up front
            const double xi = (vol ? g.vxi : g.qxi)[q], eta = (vol ? g.veta : g.qeta)[q];
            const double wq = (vol ? g.vw : g.qw)[q], x = (vol ? g.vx : g.qx)[q], y = (vol ? g.vy : g.qy)[q];
            int nbr = 0;
            double nx = 0.0, ny = 0.0, xin = 0.0, etan = 0.0;
            if (!vol) {
                nbr = g.f_nbr[f];
                nx = g.f_nx[f];
                ny = g.f_ny[f];
                xin = g.qxin[q];
                etan = g.qetan[q];
            }
            double *row = sW[it], um[NC];
            {
                double lx[P + 1], ly[P + 1], pl[2 * P], psi[NB];
                legendre_v<P>(xi, lx);
                legendre_v<P>(eta, ly);
#pragma unroll
                for (int l = 0; l < P; l++) {
                    pl[l] = lx[l + 1];
                    pl[P + l] = ly[l + 1];
                }
#pragma unroll
                for (int l = 0; l < 2 * P; l += 2)
                    *reinterpret_cast<double2 *>(row + XO + l) = make_double2(pl[l], pl[l + 1]);
                basis_of<P>(lx, ly, psi);
                eval_state<P, NC, VEC>(psi, sU[c], um);
            }
            const auto pm = ph.prim(um);
            if (!ph.admissible(um, pm)) atomicCAS(nonphys, 0, cell0 + c + 1);
            if (vol) {
                double Fx[NC], Fy[NC];
                ph.flux(um, pm, x, y, Fx, Fy);
                const double wx = wq * sbox[c].x, wy = wq * sbox[c].y;
                if constexpr (NC == 1) {
                    *reinterpret_cast<double2 *>(row) = make_double2(wx * Fx[0], wy * Fy[0]);
                } else {
#pragma unroll
                    for (int e = 0; e < NC; e += 2) {
                        *reinterpret_cast<double2 *>(row + e) = make_double2(wx * Fx[e], wx * Fx[e + 1]);
                        *reinterpret_cast<double2 *>(row + NC + e) = make_double2(wy * Fy[e], wy * Fy[e + 1]);
                    }
                }
            } else {
                double up[NC], F[NC];
                if (nbr >= 0) {
                    double lx[P + 1], ly[P + 1], psi[NB];
                    legendre_v<P>(xin, lx);
                    legendre_v<P>(etan, ly);
                    basis_of<P>(lx, ly, psi);
                    const double *Un = u + (size_t)nbr * BL;
                    if (pairs) eval_state<P, NC, VEC>(psi, Un, up);
                    else eval_state<P, NC, false>(psi, Un, up);
                } else {
                    boundary_state(ph, bc, nbr, um, x, y, t, nx, ny, up);
                }
                ph.numflux(um, pm, up, x, y, nx, ny, F);
                const double w = -wq;
                if constexpr (NC == 1) {
                    row[0] = w * F[0];
                } else {
#pragma unroll
                    for (int e = 0; e < NC; e += 2)
                        *reinterpret_cast<double2 *>(row + e) = make_double2(w * F[e], w * F[e + 1]);
                }
            }
        }
        __syncthreads();
        if (wid < nc) {
            const int qa = max(sv[wid] - v0 - base, 0), qb = min(sv[wid + 1] - v0 - base, RES_CAP);
            for (int q = qa + share; q < qb; q += LG) {
                const double *row = sW[q];
                double lx[P + 1], ly[P + 1], dx[P + 1], dy[P + 1], wx[CG], wy[CG];
                row_values<P>(row + XO, lx, ly);
                dx[0] = dy[0] = 0.0;
                dx[1] = dy[1] = 1.0;
                if constexpr (P >= 2) dx[2] = 3.0 * lx[1], dy[2] = 3.0 * ly[1];
                if constexpr (P >= 3) dx[3] = 5.0 * lx[2] + 1.0, dy[3] = 5.0 * ly[2] + 1.0;
                load_group<CG>(row + grp * CG, wx);
                if constexpr (NC == 1) wy[0] = row[1];
                else load_group<CG>(row + NC + grp * CG, wy);
                int k = 0;
#pragma unroll
                for (int a = 0; a <= P; a++)
#pragma unroll
                    for (int d = 0; d <= P - a; d++, k++) {
                        if (a > 0) {
                            const double gx = d > 0 ? dx[a] * ly[d] : dx[a];
#pragma unroll
                            for (int e = 0; e < CG; e++) acc[e * NB + k] += wx[e] * gx;
                        }
                        if (d > 0) {
                            const double gy = a > 0 ? lx[a] * dy[d] : dy[d];
#pragma unroll
                            for (int e = 0; e < CG; e++) acc[e * NB + k] += wy[e] * gy;
                        }
                    }
            }
            const int off = nvp - f0 * NQF - base;
            const int fa = max(sf[wid] * NQF + off, 0), fb = min(sf[wid + 1] * NQF + off, RES_CAP);
            for (int q = fa + share; q < fb; q += LG) {
                const double *row = sW[q];
                double lx[P + 1], ly[P + 1], w[CG];
                row_values<P>(row + XO, lx, ly);
                load_group<CG>(row + grp * CG, w);
                int k = 0;
#pragma unroll
                for (int a = 0; a <= P; a++)
#pragma unroll
                    for (int d = 0; d <= P - a; d++, k++) {
                        const double psi = a == 0 ? ly[d] : (d == 0 ? lx[a] : lx[a] * ly[d]);
#pragma unroll
                        for (int e = 0; e < CG; e++) acc[e * NB + k] += w[e] * psi;
                    }
            }
        }
    }
    if (wid >= nc) return;
    const int cell = cell0 + wid;
    double *R = sU[wid];  // the cell's coefficients are needed no more (every warp is past the last barrier)
    int at0 = 0, lim = CG * NB;
    reduce_scatter<CG * NB, LG / 2>(acc, lane, at0, lim);
    constexpr int LEFT = (CG * NB + LG - 1) / LG + 1;  // at most this many sums stay in a lane
#pragma unroll
    for (int e = 0; e < LEFT; e++)
        if (e < lim) R[grp * CG * NB + at0 + e] = acc[e];
    __syncwarp();
    const size_t at = (size_t)cell * BL;
    for (int r = lane; r < BL; r += 32) {
        if constexpr (MODE == RES_PLAIN) {
            out[at + r] = R[r];
        } else {
            const double *Mi = rk.mass_inv + (size_t)cell * NB * NB;
            const int c = r / NB, kk = r % NB;
            double sum = 0.0;
#pragma unroll
            for (int m = 0; m < NB; m++) sum += Mi[m * NB + kk] * R[c * NB + m];
            const double kv = rk.dt * sum;
            if constexpr (MODE == RES_STAGE) {
                out[at + r] = kv;
                rk.next[at + r] = rk.u0[at + r] + rk.a * kv;
            } else if constexpr (MODE == RES_RK2) {
                rk.u0[at + r] = rk.u0[at + r] + 0.5 * (rk.k1[at + r] + kv);
            } else {
                rk.u0[at + r] = rk.u0[at + r] +
                                (((rk.k1[at + r] + 2 * rk.k2[at + r]) + 2 * rk.k3[at + r]) + kv) * (1.0 / 6.0);
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Jacobian: one CTA per cell.  Quadrature-point data (basis values, flux
// Jacobians) is staged in shared memory in chunks; owner thread (h, k, j0)
// sums the entries of test function k, trial functions j0 and j0 + 1 and the
// component couplings (c, c2) of half the rows c, in the diagonal block and
// the neighbour blocks.
//   diagonal  +=  sum_q w phi_j (Ax dpsi_k/dx + Ay dpsi_k/dy)
//             -=  sum_faces sum_q w psi_k phi_j dFhat(u, u2, n, +1)
//   neighbour  =  - sum_q w psi_k phi_j^nbr dFhat(u, u2, n, -1)
// (Equation.cpp:193-279, computeVolumeJacobian :59-73,
//  computeBoundaryJacobian :75-112).  Output: scale * J (+ M on the diagonal).
//
// Bound by the loads from shared memory; the staging code, which holds two
// states and two 4x4 flux Jacobians, spills (p = 3 Euler: 1,296 bytes stored,
// 820 loaded a thread at 128 registers).  An owner's 2 x 8 entries take 20
// doubles a volume point for 52 FP64 operations; one trial function and all
// 16 couplings took 35 for 50.  100,000 p = 3 Euler cells: 8.0 -> 6.9 ms.
// Each entry's sum stays one thread's, point after point in order: a p = 3
// stage matrix's factors amplify its rounding by cond(D_i), up to 1e9, and
// regrouped sums (8x8 DMMA tiles, 5.8 ms) moved P^{-1} A x by 1e-7 at 100,000
// cells.
// ---------------------------------------------------------------------------
constexpr int JT = 128;  // threads per CTA
// points per chunk: one thread stages a volume point or one side of a face
// point; the two kinds share their shared memory (40 KB at p = 3, four CTAs an
// SM).  72 and 48 points take a six-sided p = 3 cell in one chunk each.
constexpr int VQC = 72, FQC = 48;

// s + (a x + b y), its roundings spelled out: left to the compiler, the
// contraction depends on the code around it
__device__ __forceinline__ double volume_sum(double s, double a, double x, double b, double y) {
    return __dadd_rn(s, __fma_rn(a, x, __dmul_rn(b, y)));
}

template <class Phys, int P, class TOut>
// four CTAs share an SM at 128 registers a thread (three or five: 6-14% slower)
__global__ void __launch_bounds__(JT, 4) k_jacobian(Geo g, Phys ph, BCParams bc, const double *__restrict__ u,
                                                 double t, double scale, int add_mass,
                                                 const double *__restrict__ mass, const int *__restrict__ rowptr,
                                                 TOut *__restrict__ J) {
    constexpr int NB = nbasis<P>(), NC = Phys::NC, BL = NB * NC, NQF = nqf_of(P), NC2 = NC * NC;
    constexpr int FPC = FQC / NQF;  // faces per chunk
    // the nc x nc flux-Jacobian rows are staged and read as double2 (16-byte
    // aligned) and padded by two doubles: with rows of 16 doubles (128 bytes)
    // every staging thread's store fell in the same bank; at 144 bytes a
    // quarter-warp's 16-byte stores cover distinct banks
    constexpr bool V2 = NC2 % 2 == 0;
    constexpr int NC2P = V2 ? NC2 + 2 : NC2;
    // basis rows at an odd stride: a half-warp's staging stores (one row per
    // thread) then fall in distinct banks
    constexpr int NBP = NB % 2 == 0 ? NB + 1 : NB;
    const int cell = blockIdx.x;
    const int tid = threadIdx.x;
    __shared__ double sU[BL];
    __shared__ __align__(16) double sA[2 * VQC][NC2P];  // volume: Ax, Ay; faces: M+, M-
    __shared__ double sB[3 * VQC][NBP];  // w phi, dphi/dx, dphi/dy; w psi, psi, the neighbour's basis
    double(*sAx)[NC2P] = sA, (*sAy)[NC2P] = sA + VQC, (*fMp)[NC2P] = sA, (*fMm)[NC2P] = sA + VQC;
    double(*sPW)[NBP] = sB, (*sDX)[NBP] = sB + VQC, (*sDY)[NBP] = sB + 2 * VQC;
    double(*fPsiW)[NBP] = sB, (*fPhiO)[NBP] = sB + VQC, (*fPhiN)[NBP] = sB + 2 * VQC;

    for (int r = tid; r < BL; r += JT) sU[r] = u[(size_t)cell * BL + r];
    const double4 box = g.bb[cell];
    const double sx = 2.0 / box.z, sy = 2.0 / box.w;
    constexpr int H = NC == 4 ? 2 : 1, JW = NC == 4 ? 2 : 1;  // halves of the rows, trial functions of an owner
    constexpr int JG = (NB + JW - 1) / JW, PAIRS = NC2 / H, CR = NC / H;
    static_assert(H * NB * JG <= JT, "an owner per thread");
    const bool owner = tid < H * NB * JG;
    const int kk = tid % NB, j0 = tid / NB % JG * JW, h = tid / (NB * JG);
    double acc[JW][PAIRS];
#pragma unroll
    for (int w = 0; w < JW; w++)
#pragma unroll
        for (int e = 0; e < PAIRS; e++) acc[w][e] = 0.0;
    __syncthreads();

    // ---- volume
    const int v0 = g.vq_ptr[cell], v1 = g.vq_ptr[cell + 1];
    for (int c0 = v0; c0 < v1; c0 += VQC) {
        const int cnt = min(VQC, v1 - c0);
        for (int q = tid; q < cnt; q += JT) {
            const int qq = c0 + q;
            double psi[NB], dx[NB], dy[NB];
            basis_grad<P>(g.vxi[qq], g.veta[qq], sx, sy, psi, dx, dy);
            double uu[NC];
#pragma unroll
            for (int c = 0; c < NC; c++) {
                double s = 0.0;
#pragma unroll
                for (int k = 0; k < NB; k++) s += sU[c * NB + k] * psi[k];
                uu[c] = s;
            }
            double Ax[NC2], Ay[NC2];
            ph.fluxjac(uu, g.vx[qq], g.vy[qq], Ax, Ay);
            const double w = g.vw[qq];
#pragma unroll
            for (int k = 0; k < NB; k++) {
                sPW[q][k] = w * psi[k];
                sDX[q][k] = dx[k];
                sDY[q][k] = dy[k];
            }
            if constexpr (V2) {
#pragma unroll
                for (int e = 0; e < NC2 / 2; e++) {
                    reinterpret_cast<double2 *>(sAx[q])[e] = make_double2(Ax[2 * e], Ax[2 * e + 1]);
                    reinterpret_cast<double2 *>(sAy[q])[e] = make_double2(Ay[2 * e], Ay[2 * e + 1]);
                }
            } else {
#pragma unroll
                for (int e = 0; e < NC2; e++) {
                    sAx[q][e] = Ax[e];
                    sAy[q][e] = Ay[e];
                }
            }
        }
        __syncthreads();
        if (owner) {
            for (int q = 0; q < cnt; q++) {
                double ax[JW], ay[JW];
#pragma unroll
                for (int w = 0; w < JW; w++) {
                    const double pw = sPW[q][j0 + w];
                    ax[w] = sDX[q][kk] * pw;
                    ay[w] = sDY[q][kk] * pw;
                }
                if constexpr (V2) {
                    const double2 *Ax2 = reinterpret_cast<const double2 *>(sAx[q] + h * PAIRS);
                    const double2 *Ay2 = reinterpret_cast<const double2 *>(sAy[q] + h * PAIRS);
#pragma unroll
                    for (int e = 0; e < PAIRS / 2; e++) {
                        const double2 a = Ax2[e], b = Ay2[e];
#pragma unroll
                        for (int w = 0; w < JW; w++) {
                            acc[w][2 * e] = volume_sum(acc[w][2 * e], a.x, ax[w], b.x, ay[w]);
                            acc[w][2 * e + 1] = volume_sum(acc[w][2 * e + 1], a.y, ax[w], b.y, ay[w]);
                        }
                    }
                } else {
                    acc[0][0] = volume_sum(acc[0][0], sAx[q][0], ax[0], sAy[q][0], ay[0]);
                }
            }
        }
        __syncthreads();
    }

    // ---- faces, in chunks of whole faces
    const int fa = g.f_ptr[cell], fb = g.f_ptr[cell + 1];
    const int diag = rowptr[cell];
    const size_t bl2 = (size_t)BL * BL;
    for (int fc = fa; fc < fb; fc += FPC) {
        const int nfc = min(FPC, fb - fc);
        const int rows = nfc * NQF;
        // psi and M+, or the neighbour's basis and M-; a scalar equation's two
        // sides are one thread's, as its basis values cost more than its fluxes
        // (50,000 cells, p = 1 and 2: 330 and 388 us; a thread a side 363 and 408)
        constexpr int SIDES = NC == 1 ? 1 : 2;
        for (int it = tid; it < SIDES * rows; it += JT) {
            const bool plus = SIDES == 1 || it < rows;
            const int q = plus ? it : it - rows, f = fc + q / NQF;
            const int fq = fc * NQF + q;
            double psi[NB], phin[NB];
            basis<P>(g.qxi[fq], g.qeta[fq], psi);
            double um[NC], u2[NC];
#pragma unroll
            for (int c = 0; c < NC; c++) {
                double s = 0.0;
#pragma unroll
                for (int k = 0; k < NB; k++) s += sU[c * NB + k] * psi[k];
                um[c] = s;
            }
            const int nbr = g.f_nbr[f];
            const double nx = g.f_nx[f], ny = g.f_ny[f], x = g.qx[fq], y = g.qy[fq], w = g.qw[fq];
            if (nbr >= 0) {
                basis<P>(g.qxin[fq], g.qetan[fq], phin);
                const double *Un = u + (size_t)nbr * BL;
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    double s = 0.0;
#pragma unroll
                    for (int k = 0; k < NB; k++) s += __ldg(Un + c * NB + k) * phin[k];
                    u2[c] = s;
                }
            } else {
                boundary_state(ph, bc, nbr, um, x, y, t, nx, ny, u2);
#pragma unroll
                for (int k = 0; k < NB; k++) phin[k] = 0.0;
            }
            double M[NC2];
            if (plus) {
                ph.numfluxjac(um, u2, x, y, nx, ny, 1, M);
                if (nbr == CPG_BC_WALL || nbr == CPG_BC_OUTFLOW) {
                    // chain rule through the state-dependent exterior value
                    double Mm[NC2], R[NC2];
                    ph.numfluxjac(um, u2, x, y, nx, ny, -1, Mm);
                    if (nbr == CPG_BC_WALL) {
                        ph.wall_deriv(nx, ny, R);
                    } else {
#pragma unroll
                        for (int e = 0; e < NC2; e++) R[e] = (e % (NC + 1) == 0) ? 1.0 : 0.0;
                    }
#pragma unroll
                    for (int r = 0; r < NC; r++)
#pragma unroll
                        for (int c = 0; c < NC; c++) {
                            double s = 0.0;
#pragma unroll
                            for (int m = 0; m < NC; m++) s += Mm[r * NC + m] * R[m * NC + c];
                            M[r * NC + c] += s;
                        }
                }
#pragma unroll
                for (int k = 0; k < NB; k++) {
                    fPsiW[q][k] = w * psi[k];
                    fPhiO[q][k] = psi[k];
                }
                if constexpr (SIDES == 1) {
                    ph.numfluxjac(um, u2, x, y, nx, ny, -1, fMm[q]);
#pragma unroll
                    for (int k = 0; k < NB; k++) fPhiN[q][k] = phin[k];
                }
            } else {
                ph.numfluxjac(um, u2, x, y, nx, ny, -1, M);
#pragma unroll
                for (int k = 0; k < NB; k++) fPhiN[q][k] = phin[k];
            }
            double *row = plus ? fMp[q] : fMm[q];
            if constexpr (V2) {
#pragma unroll
                for (int e = 0; e < NC2 / 2; e++)
                    reinterpret_cast<double2 *>(row)[e] = make_double2(M[2 * e], M[2 * e + 1]);
            } else {
                row[0] = M[0];
            }
        }
        __syncthreads();
        if (owner) {
            for (int fl = 0; fl < nfc; fl++) {
                const int f = fc + fl;
                double nacc[JW][PAIRS];
#pragma unroll
                for (int w = 0; w < JW; w++)
#pragma unroll
                    for (int e = 0; e < PAIRS; e++) nacc[w][e] = 0.0;
                for (int q = fl * NQF; q < (fl + 1) * NQF; q++) {
                    const double pwk = fPsiW[q][kk];
                    double dg[JW], nb[JW];
#pragma unroll
                    for (int w = 0; w < JW; w++) {
                        dg[w] = pwk * fPhiO[q][j0 + w];
                        nb[w] = pwk * fPhiN[q][j0 + w];
                    }
                    if constexpr (V2) {
                        const double2 *Mp2 = reinterpret_cast<const double2 *>(fMp[q] + h * PAIRS);
                        const double2 *Mm2 = reinterpret_cast<const double2 *>(fMm[q] + h * PAIRS);
#pragma unroll
                        for (int e = 0; e < PAIRS / 2; e++) {
                            const double2 a = Mp2[e], b = Mm2[e];
#pragma unroll
                            for (int w = 0; w < JW; w++) {
                                acc[w][2 * e] -= dg[w] * a.x;
                                acc[w][2 * e + 1] -= dg[w] * a.y;
                                nacc[w][2 * e] -= nb[w] * b.x;
                                nacc[w][2 * e + 1] -= nb[w] * b.y;
                            }
                        }
                    } else {
                        acc[0][0] -= dg[0] * fMp[q][0];
                        nacc[0][0] -= nb[0] * fMm[q][0];
                    }
                }
                const int blk = g.f_blk[f];
                if (blk >= 0) {
                    TOut *B = J + (size_t)blk * bl2;
#pragma unroll
                    for (int w = 0; w < JW; w++)
#pragma unroll
                        for (int e = 0; e < PAIRS; e++)
                            if (j0 + w < NB)
                                B[(size_t)(e % NC * NB + j0 + w) * BL + ((h * CR + e / NC) * NB + kk)] =
                                    (TOut)(scale * nacc[w][e]);
                }
            }
        }
        __syncthreads();
    }
    if (owner) {
        TOut *B = J + (size_t)diag * bl2;
#pragma unroll
        for (int w = 0; w < JW; w++) {
            const int j = j0 + w;
            if (j >= NB) break;
            const double mkj = add_mass ? mass[(size_t)cell * NB * NB + j * NB + kk] : 0.0;
#pragma unroll
            for (int e = 0; e < PAIRS; e++) {
                const int c = h * CR + e / NC, c2 = e % NC;
                const double v = c == c2 ? __fma_rn(scale, acc[w][e], mkj) : scale * acc[w][e];
                B[(size_t)(c2 * NB + j) * BL + (c * NB + kk)] = (TOut)v;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// mass matrix: y = alpha * Mi x + beta * z  (Mi = M or M^{-1} per cell,
// replicated over components)
// ---------------------------------------------------------------------------
template <int NB>
__global__ void k_mass(int n, int nc, const double *__restrict__ Mi, const double *__restrict__ x, double alpha,
                       const double *__restrict__ z, double beta, double *__restrict__ y, const int *skip) {
    if (skip && *skip) return;  // a Krylov solve that has converged
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int BL = NB * nc;
    if (idx >= (int64_t)n * BL) return;
    const int cell = (int)(idx / BL), r = (int)(idx % BL), c = r / NB, k = r % NB;
    const double *M = Mi + (size_t)cell * NB * NB;
    const double *xc = x + (size_t)cell * BL + c * NB;
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < NB; j++) s += M[j * NB + k] * xc[j];
    double v = alpha * s;
    if (z) v = v + beta * z[idx];
    y[idx] = v;
}

// per-CTA partial sums of u_c^T M u_c; fixed grid for deterministic results
constexpr int RED_CTAS = 256;
template <int NB>
__global__ void k_l2_partial(int n, int nc, const double *__restrict__ M, const double *__restrict__ u,
                             double *__restrict__ part) {
    __shared__ double sh[4][256];
    double acc[4] = {0, 0, 0, 0};
    const int BL = NB * nc;
    for (int cell = blockIdx.x * blockDim.x + threadIdx.x; cell < n; cell += gridDim.x * blockDim.x) {
        const double *Mc = M + (size_t)cell * NB * NB;
        for (int c = 0; c < nc; c++) {
            const double *uc = u + (size_t)cell * BL + c * NB;
            double s = 0.0;
            for (int j = 0; j < NB; j++) {
                double mj = 0.0;
                for (int k = 0; k < NB; k++) mj += Mc[j * NB + k] * uc[k];
                s += uc[j] * mj;
            }
            acc[c] += s;
        }
    }
    for (int c = 0; c < 4; c++) sh[c][threadIdx.x] = acc[c];
    __syncthreads();
    for (int off = blockDim.x / 2; off > 0; off >>= 1) {
        if ((int)threadIdx.x < off)
            for (int c = 0; c < 4; c++) sh[c][threadIdx.x] += sh[c][threadIdx.x + off];
        __syncthreads();
    }
    if (threadIdx.x < 4) part[blockIdx.x * 4 + threadIdx.x] = sh[threadIdx.x][0];
}
// per-CTA partial sums of sum_q w_q (u_h(x_q) - exact(x_q))^2 over the cells'
// volume quadrature points (MeshFn::L2Error); fixed grid, deterministic
template <int P, int NC>
__global__ void k_l2_error_partial(Geo g, int kind, BCParams prm, double t, const double *__restrict__ u,
                                   double *__restrict__ part) {
    constexpr int NB = nbasis<P>(), BL = NB * NC;
    __shared__ double sh[4][256];
    double acc[4] = {0, 0, 0, 0};
    for (int cell = blockIdx.x * blockDim.x + threadIdx.x; cell < g.n; cell += gridDim.x * blockDim.x) {
        const double *uc = u + (size_t)cell * BL;
        double cs[NC];
#pragma unroll
        for (int c = 0; c < NC; c++) cs[c] = 0.0;
        for (int q = g.vq_ptr[cell]; q < g.vq_ptr[cell + 1]; q++) {
            double psi[NB], ex[NC];
            basis<P>(g.vxi[q], g.veta[q], psi);
            field_eval<NC>(kind, prm.dparams, g.vx[q], g.vy[q], t, ex);
#pragma unroll
            for (int c = 0; c < NC; c++) {
                double v = 0.0;
#pragma unroll
                for (int k = 0; k < NB; k++) v += uc[c * NB + k] * psi[k];
                const double d = v - ex[c];
                cs[c] += g.vw[q] * (d * d);
            }
        }
#pragma unroll
        for (int c = 0; c < NC; c++) acc[c] += cs[c];
    }
    for (int c = 0; c < 4; c++) sh[c][threadIdx.x] = acc[c];
    __syncthreads();
    for (int off = blockDim.x / 2; off > 0; off >>= 1) {
        if ((int)threadIdx.x < off)
            for (int c = 0; c < 4; c++) sh[c][threadIdx.x] += sh[c][threadIdx.x + off];
        __syncthreads();
    }
    if (threadIdx.x < 4) part[blockIdx.x * 4 + threadIdx.x] = sh[threadIdx.x][0];
}
__global__ void k_l2_final(int nparts, const double *__restrict__ part, double *__restrict__ out) {
    const int c = threadIdx.x;
    if (c >= 4) return;
    double s = 0.0;
    for (int p = 0; p < nparts; p++) s += part[p * 4 + c];
    out[c] = s;
}

// MeshFn::interp: coefficients = pinv * f(tensor Gauss points of the box)
template <int NC>
__global__ void k_interp(int n, int nb, int m, const double4 *__restrict__ bb, const double *__restrict__ gl,
                         const double *__restrict__ pinv, int kind, BCParams prm, double t,
                         double *__restrict__ u) {
    const int cell = blockIdx.x * blockDim.x + threadIdx.x;
    if (cell >= n) return;
    const double4 box = bb[cell];
    const int nq = m * m, BL = nb * NC;
    double cf[NC][15];
    for (int c = 0; c < NC; c++)
        for (int k = 0; k < nb; k++) cf[c][k] = 0.0;
    for (int i = 0; i < m; i++)
        for (int j = 0; j < m; j++) {
            double o[4];
            field_eval<NC>(kind, prm.dparams, (gl[i] + 1) * box.z / 2.0 + box.x, (gl[j] + 1) * box.w / 2.0 + box.y,
                           t, o);
            const int e = i * m + j;
            for (int k = 0; k < nb; k++) {
                const double p = pinv[k * nq + e];
                for (int c = 0; c < NC; c++) cf[c][k] += p * o[c];
            }
        }
    for (int c = 0; c < NC; c++)
        for (int k = 0; k < nb; k++) u[(size_t)cell * BL + c * nb + k] = cf[c][k];
}

// dispatch on physics and degree
template <class F>
cpg_status with_physics(const cpg_equation *eq, F &&f) {
    auto by_deg = [&](auto ph) -> cpg_status {
        switch (eq->degree) {
            case 1: return f(ph, std::integral_constant<int, 1>{});
            case 2: return f(ph, std::integral_constant<int, 2>{});
            case 3: return f(ph, std::integral_constant<int, 3>{});
        }
        return fail(eq->ctx, CPG_ERR_UNSUPPORTED, "degree must be 1..3");
    };
    switch (eq->physics) {
        case CPG_ADVECTION_CONST: {
            Advection<false> ph;
            ph.bx = eq->beta[0];
            ph.by = eq->beta[1];
            return by_deg(ph);
        }
        case CPG_ADVECTION_ROTATING: {
            Advection<true> ph;
            ph.bx = ph.by = 0;
            return by_deg(ph);
        }
        case CPG_EULER: {
            Euler ph;
            ph.gamma = eq->gamma;
            ph.exact = eq->exact_jacobian;
            return by_deg(ph);
        }
    }
    return fail(eq->ctx, CPG_ERR_INVALID_ARG, "unknown physics");
}

// dense inverse by Gauss-Jordan with partial pivoting (host, small blocks)
bool host_inverse(int n, const double *A, double *Ainv) {
    std::vector<double> a(A, A + (size_t)n * n);
    std::vector<double> b((size_t)n * n, 0.0);
    for (int i = 0; i < n; i++) b[(size_t)i * n + i] = 1.0;
    for (int p = 0; p < n; p++) {
        int piv = p;
        for (int r = p + 1; r < n; r++)
            if (std::fabs(a[(size_t)p * n + r]) > std::fabs(a[(size_t)p * n + piv])) piv = r;
        if (a[(size_t)p * n + piv] == 0.0) return false;
        if (piv != p)
            for (int c = 0; c < n; c++) {
                std::swap(a[(size_t)c * n + p], a[(size_t)c * n + piv]);
                std::swap(b[(size_t)c * n + p], b[(size_t)c * n + piv]);
            }
        const double d = a[(size_t)p * n + p];
        for (int c = 0; c < n; c++) {
            a[(size_t)c * n + p] /= d;
            b[(size_t)c * n + p] /= d;
        }
        for (int r = 0; r < n; r++) {
            if (r == p) continue;
            const double f = a[(size_t)p * n + r];
            if (f == 0.0) continue;
            for (int c = 0; c < n; c++) {
                a[(size_t)c * n + r] -= f * a[(size_t)c * n + p];
                b[(size_t)c * n + r] -= f * b[(size_t)c * n + p];
            }
        }
    }
    std::memcpy(Ainv, b.data(), sizeof(double) * n * n);
    return true;
}

// Gauss-Legendre nodes of order m, ascending (Newton on P_m)
std::vector<double> gauss_nodes(int m) {
    std::vector<double> x(m);
    for (int i = 0; i < m; i++) {
        long double z = std::cos(M_PI * (i + 0.75) / (m + 0.5));
        for (int it = 0; it < 60; it++) {
            long double p0 = 1, p1 = z;
            for (int k = 2; k <= m; k++) {
                long double p2 = ((2 * k - 1) * z * p1 - (k - 1) * p0) / k;
                p0 = p1;
                p1 = p2;
            }
            const long double dp = m * (z * p1 - p0) / (z * z - 1);
            const long double dz = p1 / dp;
            z -= dz;
            if (std::fabs((double)dz) < 1e-18) break;
        }
        x[m - 1 - i] = (double)z;
    }
    for (int i = 0; i < m / 2; i++) {
        const double a = 0.5 * (x[m - 1 - i] - x[i]);
        x[m - 1 - i] = a;
        x[i] = -a;
    }
    if (m % 2) x[m / 2] = 0.0;
    return x;
}

template <int P>
void host_basis(double xi, double eta, double *psi) {
    basis<P>(xi, eta, psi);
}
void host_basis_dyn(int p, double xi, double eta, double *psi) {
    if (p == 1) host_basis<1>(xi, eta, psi);
    else if (p == 2) host_basis<2>(xi, eta, psi);
    else host_basis<3>(xi, eta, psi);
}

void free_equation(cpg_equation *eq) {
    void *ptrs[] = {eq->bb, eq->vq_ptr, eq->f_ptr, eq->f_nbr, eq->f_blk, eq->vx, eq->vy, eq->vxi, eq->veta,
                    eq->vw, eq->f_nx, eq->f_ny, eq->qx, eq->qy, eq->qxi, eq->qeta, eq->qxin, eq->qetan,
                    eq->qw, eq->mass, eq->mass_inv, eq->interp_pinv, eq->rowptr_d, eq->colidx_d};
    for (void *p : ptrs) dfree(p);
}

}  // namespace

extern "C" {

cpg_status cpg_equation_create(cpg_ctx *ctx, const cpg_mesh *mm, const cpg_equation_desc *d, cpg_equation **out) {
    if (!ctx || !mm || !d || !out) return CPG_ERR_INVALID_ARG;
    *out = nullptr;
    if (d->degree < 1 || d->degree > 3) return fail(ctx, CPG_ERR_UNSUPPORTED, "degree must be 1..3");
    if (d->physics < 0 || d->physics > 2) return fail(ctx, CPG_ERR_INVALID_ARG, "unknown physics");
    const Mesh &m = cpg_mesh_ref(mm);
    cpg_equation *eq = new (std::nothrow) cpg_equation();
    if (!eq) return fail(ctx, CPG_ERR_OOM, "host allocation");
    eq->ctx = ctx;
    eq->physics = d->physics;
    eq->degree = d->degree;
    eq->nb = (d->degree + 1) * (d->degree + 2) / 2;
    eq->nc = d->physics == CPG_EULER ? 4 : 1;
    eq->bl = eq->nb * eq->nc;
    eq->n = m.n;
    eq->nqf = nqf_of(d->degree);
    eq->gamma = d->gamma;
    eq->beta[0] = d->beta[0];
    eq->beta[1] = d->beta[1];
    eq->exact_jacobian = d->exact_jacobian ? 1 : 0;
    eq->bc.dkind = d->dirichlet_kind;
    for (int q = 0; q < 8; q++) eq->bc.dparams[q] = d->dirichlet_params[q];
    for (int q = 0; q < 4; q++) eq->bc.inflow[q] = d->inflow_state[q];

    const int n = m.n, p = d->degree, nb = eq->nb, nqf = eq->nqf;
    const quad::TriRule tr = quad::tri_rule(2 * p);
    const quad::LineRule lr = quad::line_rule(2 * p);
    std::vector<double4> bb(n);
    std::vector<int> vq_ptr(n + 1, 0), f_ptr(n + 1, 0), f_nbr, f_blk;
    std::vector<double> vx, vy, vxi, veta, vw, fnx, fny, qx, qy, qxi, qeta, qxin, qetan, qw;
    std::vector<double> mass((size_t)n * nb * nb, 0.0), minv((size_t)n * nb * nb, 0.0);
    eq->rowptr.assign(1, 0);
    eq->colidx.clear();
    for (int i = 0; i < n; i++) bb[i] = make_double4(m.bb[4 * i], m.bb[4 * i + 1], m.bb[4 * i + 2], m.bb[4 * i + 3]);
    for (int i = 0; i < n; i++) {
        const double x0 = m.bb[4 * i], y0 = m.bb[4 * i + 1], w = m.bb[4 * i + 2], h = m.bb[4 * i + 3];
        // volume qp: Quadrature::polygonIntegral (Quadrature.cpp:13-57)
        for (int t = m.tri_ptr[i]; t < m.tri_ptr[i + 1]; t++) {
            const double *T = &m.tri[6 * (size_t)t];
            const double x1 = T[0], y1 = T[1], x2 = T[2], y2 = T[3], x3 = T[4], y3 = T[5];
            const double area = 0.5 * std::fabs(x1 * y2 + x2 * y3 + x3 * y1 - x1 * y3 - x3 * y2 - x2 * y1);
            for (int k = 0; k < tr.n; k++) {
                const double a = tr.p[k][0], b = tr.p[k][1];
                const double x = x1 * (1 - a - b) + x2 * a + x3 * b;
                const double y = y1 * (1 - a - b) + y2 * a + y3 * b;
                vx.push_back(x);
                vy.push_back(y);
                vxi.push_back(2.0 * (x - x0) / w - 1);
                veta.push_back(2.0 * (y - y0) / h - 1);
                vw.push_back(tr.p[k][2] * area);
            }
        }
        vq_ptr[i + 1] = (int)vx.size();
        // mass block M(k, j) = sum_q w psi_k psi_j (MassMatrix.cpp:30-94)
        double *Mi = mass.data() + (size_t)i * nb * nb;
        for (int q = vq_ptr[i]; q < vq_ptr[i + 1]; q++) {
            double psi[15];
            host_basis_dyn(p, vxi[q], veta[q], psi);
            for (int j = 0; j < nb; j++)
                for (int k = 0; k < nb; k++) Mi[j * nb + k] += vw[q] * psi[k] * psi[j];
        }
        if (!host_inverse(nb, Mi, minv.data() + (size_t)i * nb * nb)) {
            free_equation(eq);
            delete eq;
            return fail(ctx, CPG_ERR_SINGULAR_BLOCK, "singular mass block at cell " + std::to_string(i));
        }
        // Jacobian pattern row (Jacobian.cpp:7-47)
        eq->colidx.push_back(i);
        // faces: getOutwardNormal (PolyMesh.cpp:248-273) and lineIntegral
        // points (Quadrature.cpp:67-101)
        const int s = m.cell_ptr[i], nv = m.cell_ptr[i + 1] - s;
        double cx = 0, cy = 0;
        for (int k = 0; k < nv; k++) {
            cx += m.vxy[2 * (s + k)];
            cy += m.vxy[2 * (s + k) + 1];
        }
        cx /= nv;
        cy /= nv;
        for (int e = 0; e < nv; e++) {
            const int a = s + e, b = s + (e + 1) % nv;
            const double ax = m.vxy[2 * a], ay = m.vxy[2 * a + 1], bx = m.vxy[2 * b], by = m.vxy[2 * b + 1];
            const double dx = ax - bx, dy = ay - by;
            const double length = std::sqrt(dx * dx + dy * dy);
            const double sv = -dy * (ax - cx) + dx * (ay - cy);
            const int sg = (0.0 < sv) - (sv < 0.0);
            fnx.push_back(-sg * dy / length);
            fny.push_back(sg * dx / length);
            const int nbr = m.nbr[a];
            f_nbr.push_back(nbr);
            if (nbr >= 0) {
                f_blk.push_back((int)eq->colidx.size());
                eq->colidx.push_back(nbr);
            } else {
                f_blk.push_back(-1);
            }
            const double sx = m.shift[2 * a], sy = m.shift[2 * a + 1];
            const double len = std::sqrt((bx - ax) * (bx - ax) + (by - ay) * (by - ay));
            for (int k = 0; k < lr.n; k++) {
                const double xi = lr.p[k][0];
                const double x = ax + 0.5 * (xi + 1) * (bx - ax);
                const double y = ay + 0.5 * (xi + 1) * (by - ay);
                qx.push_back(x);
                qy.push_back(y);
                qxi.push_back(2.0 * (x - x0) / w - 1);
                qeta.push_back(2.0 * (y - y0) / h - 1);
                if (nbr >= 0) {
                    const double nx0 = m.bb[4 * nbr], ny0 = m.bb[4 * nbr + 1];
                    const double nw = m.bb[4 * nbr + 2], nh = m.bb[4 * nbr + 3];
                    qxin.push_back(2.0 * ((x + sx) - nx0) / nw - 1);
                    qetan.push_back(2.0 * ((y + sy) - ny0) / nh - 1);
                } else {
                    qxin.push_back(0.0);
                    qetan.push_back(0.0);
                }
                qw.push_back(lr.p[k][1] * 0.5 * len);
            }
        }
        f_ptr[i + 1] = (int)f_nbr.size();
        eq->rowptr.push_back((int)eq->colidx.size());
    }
    (void)nqf;
    eq->n_vqp = (int)vx.size();
    eq->n_faces = (int)f_nbr.size();
    // Dirichlet faces read the boundary field at time t; nothing else does
    eq->time_dependent_bc = std::count(f_nbr.begin(), f_nbr.end(), (int)CPG_BC_DIRICHLET) > 0 ? 1 : 0;
    // interpolation pseudo-inverse (MeshFn::interp, MeshFn.cpp:56-145)
    const int mq = p + 1, nq = mq * mq;
    eq->gl_nodes = gauss_nodes(mq);
    std::vector<double> G((size_t)nq * nb), pinv((size_t)nb * nq);
    for (int i = 0; i < mq; i++)
        for (int j = 0; j < mq; j++) {
            double psi[15];
            host_basis_dyn(p, eq->gl_nodes[i], eq->gl_nodes[j], psi);
            for (int k = 0; k < nb; k++) G[(size_t)(i * mq + j) * nb + k] = psi[k];
        }
    {
        // normal equations in long double: pinv = (G^T G)^{-1} G^T
        std::vector<long double> N((size_t)nb * nb, 0.0L), Ni((size_t)nb * nb, 0.0L);
        for (int a = 0; a < nb; a++)
            for (int b = 0; b < nb; b++) {
                long double s = 0;
                for (int e = 0; e < nq; e++) s += (long double)G[(size_t)e * nb + a] * G[(size_t)e * nb + b];
                N[a * nb + b] = s;
            }
        for (int a = 0; a < nb; a++) Ni[a * nb + a] = 1.0L;
        for (int c = 0; c < nb; c++) {  // SPD: Gauss-Jordan without pivoting
            const long double d = N[c * nb + c];
            for (int k = 0; k < nb; k++) {
                N[c * nb + k] /= d;
                Ni[c * nb + k] /= d;
            }
            for (int r = 0; r < nb; r++) {
                if (r == c) continue;
                const long double f = N[r * nb + c];
                for (int k = 0; k < nb; k++) {
                    N[r * nb + k] -= f * N[c * nb + k];
                    Ni[r * nb + k] -= f * Ni[c * nb + k];
                }
            }
        }
        for (int k = 0; k < nb; k++)
            for (int e = 0; e < nq; e++) {
                long double s = 0;
                for (int a = 0; a < nb; a++) s += Ni[k * nb + a] * G[(size_t)e * nb + a];
                pinv[(size_t)k * nq + e] = (double)s;
            }
    }
    cpg_status st = CPG_OK;
    auto up = [&](auto **dst, const auto &src) {
        if (st == CPG_OK) st = upload(ctx, dst, src);
    };
    up(&eq->bb, bb);
    up(&eq->vq_ptr, vq_ptr);
    up(&eq->f_ptr, f_ptr);
    up(&eq->f_nbr, f_nbr);
    up(&eq->f_blk, f_blk);
    up(&eq->vx, vx);
    up(&eq->vy, vy);
    up(&eq->vxi, vxi);
    up(&eq->veta, veta);
    up(&eq->vw, vw);
    up(&eq->f_nx, fnx);
    up(&eq->f_ny, fny);
    up(&eq->qx, qx);
    up(&eq->qy, qy);
    up(&eq->qxi, qxi);
    up(&eq->qeta, qeta);
    up(&eq->qxin, qxin);
    up(&eq->qetan, qetan);
    up(&eq->qw, qw);
    up(&eq->mass, mass);
    up(&eq->mass_inv, minv);
    up(&eq->interp_pinv, pinv);
    up(&eq->rowptr_d, eq->rowptr);
    up(&eq->colidx_d, eq->colidx);
    if (st != CPG_OK) {
        free_equation(eq);
        delete eq;
        return st;
    }
    // ILU(0) level counts of the pattern (for information)
    {
        std::vector<int> lv(n, 0), uv(n, 0);
        int nl = 0, nu = 0;
        for (int j = 0; j < n; j++) {
            int l = 0;
            for (int k = eq->rowptr[j]; k < eq->rowptr[j + 1]; k++)
                if (eq->colidx[k] < j) l = std::max(l, lv[eq->colidx[k]] + 1);
            lv[j] = l;
            nl = std::max(nl, l + 1);
        }
        for (int i = n - 1; i >= 0; i--) {
            int l = 0;
            for (int k = eq->rowptr[i]; k < eq->rowptr[i + 1]; k++)
                if (eq->colidx[k] > i) l = std::max(l, uv[eq->colidx[k]] + 1);
            uv[i] = l;
            nu = std::max(nu, l + 1);
        }
        eq->levels_lower = nl;
        eq->levels_upper = nu;
    }
    *out = eq;
    return CPG_OK;
}

void cpg_equation_destroy(cpg_equation *eq) {
    if (!eq) return;
    // cudaFree synchronizes the device; the context may already be gone
    free_equation(eq);
    delete eq;
}

cpg_status cpg_equation_get_info(const cpg_equation *eq, cpg_equation_info *info) {
    if (!eq || !info) return CPG_ERR_INVALID_ARG;
    info->n_cells = eq->n;
    info->nb = eq->nb;
    info->nc = eq->nc;
    info->bl = eq->bl;
    info->n_dof = (int64_t)eq->n * eq->bl;
    info->nnzb = (int64_t)eq->colidx.size();
    info->n_vqp = eq->n_vqp;
    info->n_faces = eq->n_faces;
    info->nqf = eq->nqf;
    info->levels_lower = eq->levels_lower;
    info->levels_upper = eq->levels_upper;
    return CPG_OK;
}

// Equation::assemble (Equation.cpp:152-191) as seen from the C ABI: the
// residual, then -- outside stream capture -- a read of the state word, so
// that a non-physical state is reported by the call that met it.  The
// steppers launch the kernel alone (assemble_raw) and read the word at the
// synchronisation their Newton norms make anyway.
cpg_status cpg_assemble(cpg_ctx *ctx, const cpg_equation *eq, const double *u, double t, double *b) {
    if (!ctx || !eq || !u || !b) return CPG_ERR_INVALID_ARG;
    CPG_TRY(assemble_raw(ctx, eq, u, t, b));
    if (ctx->deferred_checks) return CPG_OK;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    CPG_CUDA(ctx, cudaStreamIsCapturing(ctx->stream, &cs));
    if (cs != cudaStreamCaptureStatusNone) return CPG_OK;
    return check_state(ctx, "residual");
}

cpg_status cpg_jacobian(cpg_ctx *ctx, const cpg_equation *eq, const double *u, double t, double scale, int add_mass,
                        cpg_bsr *J) {
    if (!ctx || !eq || !u || !J) return CPG_ERR_INVALID_ARG;
    if (J->n_rows != eq->n || J->bl != eq->bl || J->nnzb != (int64_t)eq->colidx.size())
        return fail(ctx, CPG_ERR_INVALID_ARG, "Jacobian matrix does not have the equation's pattern");
    return with_physics(eq, [&](auto ph, auto pc) -> cpg_status {
        constexpr int P = decltype(pc)::value;
        auto launch = [&](auto *vals) {
            using TOut = std::remove_pointer_t<decltype(vals)>;
            k_jacobian<decltype(ph), P, TOut><<<eq->n, JT, 0, ctx->stream>>>(
                eq->geo(), ph, eq->bc, u, t, scale, add_mass, eq->mass, eq->rowptr_d, vals);
            return launched(ctx, "jacobian kernel");
        };
        const cpg_status st = J->precision == CPG_F32 ? launch((float *)J->vals) : launch((double *)J->vals);
        bsr_touch(J);
        return st;
    });
}

static cpg_status mass_op(cpg_ctx *ctx, const cpg_equation *eq, const double *Mi, const double *x, double alpha,
                          const double *z, double beta, double *y) {
    const int64_t N = (int64_t)eq->n * eq->bl;
    const int T = 256;
    const int grid = (int)((N + T - 1) / T);
    switch (eq->nb) {
        case 3: k_mass<3><<<grid, T, 0, ctx->stream>>>(eq->n, eq->nc, Mi, x, alpha, z, beta, y, ctx->skip_dev); break;
        case 6: k_mass<6><<<grid, T, 0, ctx->stream>>>(eq->n, eq->nc, Mi, x, alpha, z, beta, y, ctx->skip_dev); break;
        case 10: k_mass<10><<<grid, T, 0, ctx->stream>>>(eq->n, eq->nc, Mi, x, alpha, z, beta, y, ctx->skip_dev); break;
        default: return fail(ctx, CPG_ERR_UNSUPPORTED, "basis size");
    }
    return launched(ctx, "mass kernel");
}

cpg_status cpg_mass_apply(cpg_ctx *ctx, const cpg_equation *eq, const double *x, double *y) {
    if (!ctx || !eq || !x || !y) return CPG_ERR_INVALID_ARG;
    return mass_op(ctx, eq, eq->mass, x, 1.0, nullptr, 0.0, y);
}

cpg_status cpg_mass_solve(cpg_ctx *ctx, const cpg_equation *eq, const double *x, double *y) {
    if (!ctx || !eq || !x || !y) return CPG_ERR_INVALID_ARG;
    return mass_op(ctx, eq, eq->mass_inv, x, 1.0, nullptr, 0.0, y);
}

cpg_status cpg_mass_export(cpg_ctx *ctx, const cpg_equation *eq, double *mass_host) {
    if (!ctx || !eq || !mass_host) return CPG_ERR_INVALID_ARG;
    CPG_CUDA(ctx, cudaMemcpyAsync(mass_host, eq->mass, sizeof(double) * eq->n * eq->nb * eq->nb,
                                  cudaMemcpyDeviceToHost, ctx->stream));
    CPG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return CPG_OK;
}

cpg_status cpg_l2norm(cpg_ctx *ctx, const cpg_equation *eq, const double *u, double *out_host) {
    if (!ctx || !eq || !u || !out_host) return CPG_ERR_INVALID_ARG;
    double *part, *hp;
    CPG_TRY(scratch(ctx, RED_CTAS * 4 + 4, &part));
    CPG_TRY(pinned(ctx, 4, &hp));
    switch (eq->nb) {
        case 3: k_l2_partial<3><<<RED_CTAS, 256, 0, ctx->stream>>>(eq->n, eq->nc, eq->mass, u, part); break;
        case 6: k_l2_partial<6><<<RED_CTAS, 256, 0, ctx->stream>>>(eq->n, eq->nc, eq->mass, u, part); break;
        case 10: k_l2_partial<10><<<RED_CTAS, 256, 0, ctx->stream>>>(eq->n, eq->nc, eq->mass, u, part); break;
        default: return fail(ctx, CPG_ERR_UNSUPPORTED, "basis size");
    }
    CPG_TRY(launched(ctx, "l2 partial kernel"));
    k_l2_final<<<1, 32, 0, ctx->stream>>>(RED_CTAS, part, part + RED_CTAS * 4);
    CPG_TRY(launched(ctx, "l2 final kernel"));
    CPG_CUDA(ctx, cudaMemcpyAsync(hp, part + RED_CTAS * 4, 4 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    CPG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    for (int c = 0; c < eq->nc; c++) {
        if (!std::isfinite(hp[c])) return fail(ctx, CPG_ERR_NONFINITE, "non-finite L2 norm");
        out_host[c] = std::sqrt(std::max(0.0, hp[c]));
    }
    return CPG_OK;
}

cpg_status cpg_l2error(cpg_ctx *ctx, const cpg_equation *eq, const double *u, int kind, const double *params,
                       double t, double *out_host) {
    if (!ctx || !eq || !u || !out_host || kind < 0 || kind > 3) return CPG_ERR_INVALID_ARG;
    BCParams prm{};
    for (int q = 0; q < 8; q++) prm.dparams[q] = params ? params[q] : 0.0;
    double *part, *hp;
    CPG_TRY(scratch(ctx, RED_CTAS * 4 + 4, &part));
    CPG_TRY(pinned(ctx, 4, &hp));
    const Geo g = eq->geo();
    auto launch = [&](auto pc) {
        constexpr int P = decltype(pc)::value;
        if (eq->nc == 4) k_l2_error_partial<P, 4><<<RED_CTAS, 256, 0, ctx->stream>>>(g, kind, prm, t, u, part);
        else k_l2_error_partial<P, 1><<<RED_CTAS, 256, 0, ctx->stream>>>(g, kind, prm, t, u, part);
    };
    switch (eq->degree) {
        case 1: launch(std::integral_constant<int, 1>{}); break;
        case 2: launch(std::integral_constant<int, 2>{}); break;
        case 3: launch(std::integral_constant<int, 3>{}); break;
        default: return fail(ctx, CPG_ERR_UNSUPPORTED, "degree must be 1..3");
    }
    CPG_TRY(launched(ctx, "l2 error kernel"));
    k_l2_final<<<1, 32, 0, ctx->stream>>>(RED_CTAS, part, part + RED_CTAS * 4);
    CPG_TRY(launched(ctx, "l2 final kernel"));
    CPG_CUDA(ctx, cudaMemcpyAsync(hp, part + RED_CTAS * 4, 4 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    CPG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    for (int c = 0; c < eq->nc; c++) {
        if (!std::isfinite(hp[c])) return fail(ctx, CPG_ERR_NONFINITE, "non-finite L2 error");
        out_host[c] = std::sqrt(std::max(0.0, hp[c]));
    }
    return CPG_OK;
}

cpg_status cpg_interp(cpg_ctx *ctx, const cpg_equation *eq, int kind, const double *params, double t, double *u) {
    if (!ctx || !eq || !u || kind < 0 || kind > 3) return CPG_ERR_INVALID_ARG;
    BCParams prm{};
    for (int q = 0; q < 8; q++) prm.dparams[q] = params ? params[q] : 0.0;
    // node table lives in the scratch buffer
    double *gl;
    CPG_TRY(scratch(ctx, 16, &gl));
    CPG_CUDA(ctx, cudaMemcpyAsync(gl, eq->gl_nodes.data(), sizeof(double) * eq->gl_nodes.size(),
                                  cudaMemcpyHostToDevice, ctx->stream));
    const int T = 128, grid = (eq->n + T - 1) / T;
    if (eq->nc == 4)
        k_interp<4><<<grid, T, 0, ctx->stream>>>(eq->n, eq->nb, eq->degree + 1, eq->bb, gl, eq->interp_pinv, kind,
                                                 prm, t, u);
    else
        k_interp<1><<<grid, T, 0, ctx->stream>>>(eq->n, eq->nb, eq->degree + 1, eq->bb, gl, eq->interp_pinv, kind,
                                                 prm, t, u);
    CPG_TRY(launched(ctx, "interp kernel"));
    // the node table copy above is asynchronous from pageable memory of a
    // long-lived vector; synchronize so the scratch buffer may be reused
    CPG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return CPG_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// L2 norm without any allocation.
//
// cpg_l2norm keeps its partial sums in the context's scratch buffer and reads
// the result back through a pinned host buffer; both are allocated (or grown)
// on demand.  A caller that hands all of the device memory to its own pool --
// the serving loop, for instance, admits each solve against a fixed memory
// budget -- or that may not allocate inside its Newton loop can use
// cpg_l2norm_noalloc instead: its partial sums live in the file-scope device
// array below, which every GPU that loads this library holds until the
// process exits, and the result is copied straight into the caller's host
// array.
// ---------------------------------------------------------------------------
namespace {
constexpr int L2_NOALLOC_MAX_NC = 4;  // components a call may reduce
// 4 partial-sum slots per reduction CTA (k_l2_partial) plus the 4 totals
constexpr int L2_NOALLOC_DOUBLES = RED_CTAS * 4 + 4;  // 1028 doubles, 8224 bytes
static __device__ __align__(256) double g_l2_noalloc[L2_NOALLOC_DOUBLES];
std::mutex g_l2_noalloc_mu;
double *g_l2_noalloc_addr[128] = {};  // device address of the array, per device
}  // namespace

extern "C" cpg_status cpg_l2norm_noalloc(cpg_ctx *ctx, const cpg_equation *eq, const double *u, double *out_host) {
    if (!ctx || !eq || !u || !out_host) return CPG_ERR_INVALID_ARG;
    const size_t need = (size_t)RED_CTAS * 4 + (size_t)eq->nc;
    if (eq->nc > L2_NOALLOC_MAX_NC || need > (size_t)L2_NOALLOC_DOUBLES)
        return fail(ctx, CPG_ERR_INVALID_ARG,
                    "cpg_l2norm_noalloc: " + std::to_string(eq->nc) + " components need " + std::to_string(need) +
                        " doubles of static scratch; the maximum is " + std::to_string(L2_NOALLOC_DOUBLES) +
                        " doubles (" + std::to_string(L2_NOALLOC_MAX_NC) + " components)");
    if (eq->nb != 3 && eq->nb != 6 && eq->nb != 10) return fail(ctx, CPG_ERR_UNSUPPORTED, "basis size");
    int dev = -1;
    CPG_CUDA(ctx, cudaGetDevice(&dev));
    if (dev != ctx->device || dev < 0 || dev >= 128)
        return fail(ctx, CPG_ERR_INVALID_ARG, "cpg_l2norm_noalloc: make the context's device current");
    double *part = nullptr;
    {
        // set-up, once per device, with that device current: the host-side
        // name of the array is not a device address
        std::lock_guard<std::mutex> lock(g_l2_noalloc_mu);
        if (!g_l2_noalloc_addr[dev]) {
            void *p = nullptr;
            const cudaError_t e = cudaGetSymbolAddress(&p, g_l2_noalloc);
            if (e != cudaSuccess) return cuda_fail(ctx, e, "cudaGetSymbolAddress of the static norm scratch");
            g_l2_noalloc_addr[dev] = (double *)p;
        }
        part = g_l2_noalloc_addr[dev];
    }
    // every slot read below is written earlier in the same call, so nothing
    // needs clearing; calls that overlap on the GPU share the array and race
    switch (eq->nb) {
        case 3: k_l2_partial<3><<<RED_CTAS, 256, 0, ctx->stream>>>(eq->n, eq->nc, eq->mass, u, part); break;
        case 6: k_l2_partial<6><<<RED_CTAS, 256, 0, ctx->stream>>>(eq->n, eq->nc, eq->mass, u, part); break;
        default: k_l2_partial<10><<<RED_CTAS, 256, 0, ctx->stream>>>(eq->n, eq->nc, eq->mass, u, part); break;
    }
    CPG_TRY(launched(ctx, "l2 partial kernel (static scratch)"));
    k_l2_final<<<1, 32, 0, ctx->stream>>>(RED_CTAS, part, part + RED_CTAS * 4);
    CPG_TRY(launched(ctx, "l2 final kernel (static scratch)"));
    double sums[L2_NOALLOC_MAX_NC];
    CPG_CUDA(ctx, cudaMemcpyAsync(sums, part + RED_CTAS * 4, sizeof(double) * eq->nc, cudaMemcpyDeviceToHost,
                                  ctx->stream));
    CPG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    for (int c = 0; c < eq->nc; c++) {
        if (!std::isfinite(sums[c])) return fail(ctx, CPG_ERR_NONFINITE, "non-finite L2 norm");
        out_host[c] = std::sqrt(std::max(0.0, sums[c]));
    }
    return CPG_OK;
}

namespace {
// Four cells a CTA fill its threads' rounds of points; one or two are done
// sooner, which is what counts while all CTAs fit on the SMs at once: so one
// cell a CTA up to as many cells as CTAs are resident (148 SMs: 740 for p = 3
// Euler, 888 for p = 2, 1,184 for a scalar), two up to twice as many.  At
// p = 1 a cell has about 30 points, a quarter of the CTA's threads, and two
// are as soon done as one.  RK4 step with one, two and four cells a CTA, us:
//   Euler p = 3     700 cells 37.1 43.8 57.8   1,480 cells 66.0 51.2 63.6   1,600 cells 81.7 72.5 63.8
//   Euler p = 2     800 cells 29.0 29.0 37.3   1,776 cells 51.6 35.1 41.2   2,000 cells 65.9 51.5 42.5
//   scalar p = 3  1,184 cells 25.1 29.2 37.2   2,368 cells 43.3 35.0 41.2   2,500 cells 51.3 46.6 41.7
//   scalar p = 2  1,184 cells 20.9 20.7 26.8   2,368 cells 35.1 23.0 28.4   2,500 cells 41.4 33.1 28.9
//   scalar p = 1    700 cells 18.6 16.8 18.8   2,368 cells 31.9 18.8 20.7   2,500 cells 39.3 27.1 20.8
// (lines at 740 and 1,480 cells for all of them cost up to 29% in between).
template <int MODE>
cpg_status launch_residual(cpg_ctx *ctx, const cpg_equation *eq, const double *u, double t, double *out,
                           const RkStage &rk) {
    return with_physics(eq, [&](auto ph, auto pc) -> cpg_status {
        constexpr int P = decltype(pc)::value;
        auto launch = [&](auto cells) {
            constexpr int C = decltype(cells)::value;
            k_residual<decltype(ph), P, MODE, C><<<(eq->n + C - 1) / C, RES_T, 0, ctx->stream>>>(
                eq->geo(), ph, eq->bc, u, t, ctx->flag_dev + FLAG_NONPHYS, out, rk);
        };
        const int resident = res_ctas(decltype(ph)::NC, P) * ctx->num_sms;
        constexpr int FEW = P > 1 ? 1 : 2;
        if (eq->n <= resident) launch(std::integral_constant<int, FEW>{});
        else if (eq->n <= 2 * resident) launch(std::integral_constant<int, 2>{});
        else launch(std::integral_constant<int, 4>{});
        return launched(ctx, "residual kernel");
    });
}
}  // namespace

namespace cpg {
cpg_status assemble_raw(cpg_ctx *ctx, const cpg_equation *eq, const double *u, double t, double *b) {
    return launch_residual<RES_PLAIN>(ctx, eq, u, t, b, RkStage{});
}
cpg_status rk_stage(cpg_ctx *ctx, const cpg_equation *eq, const double *u, double t, double *k, RkStage rk) {
    rk.mass_inv = eq->mass_inv;
    if (rk.next) return launch_residual<RES_STAGE>(ctx, eq, u, t, k, rk);
    return rk.k2 ? launch_residual<RES_RK4>(ctx, eq, u, t, nullptr, rk)
                 : launch_residual<RES_RK2>(ctx, eq, u, t, nullptr, rk);
}
// y = alpha * M x + beta * z (Newton residual r = M k - dt b)
cpg_status mass_apply_axpy(cpg_ctx *ctx, const cpg_equation *eq, const double *x, double alpha, const double *z,
                           double beta, double *y) {
    return mass_op(ctx, eq, eq->mass, x, alpha, z, beta, y);
}
// y = alpha * M^{-1} x
cpg_status mass_solve_scaled(cpg_ctx *ctx, const cpg_equation *eq, const double *x, double alpha, double *y) {
    return mass_op(ctx, eq, eq->mass_inv, x, alpha, nullptr, 0.0, y);
}
}  // namespace cpg
