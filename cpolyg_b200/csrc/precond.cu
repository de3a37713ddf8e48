// Preconditioners: block ILU(0) (BlockILU0, src/Preconditioners.cpp:49-158)
// and block Jacobi (BlockJacobi, src/Preconditioners.cpp:8-47).
//
// Storage mirrors the reference's three BlockMatrix objects:
//   L  : strictly lower blocks L_ji = A_ji D_i^{-1}, row order of A;
//   DU : per row [D_i^{-1}, U_ij = D_i^{-1} A_ij ...], row order of A;
// Block Jacobi keeps only the D_i^{-1} rows.  Pivot blocks are inverted in
// FP64 (partial pivoting); factors may be stored in FP32.
//
// Factorisation is level scheduled over the lower dependency graph of the
// natural row order (row j depends on its lower neighbours i < j), which
// reproduces the reference's sequential result; each level is one launch
// with one CTA per row.  Application runs the forward sweep and the backward
// sweep (fused with D^{-1}) either as one sync-free launch each (rows claimed
// in level order; block sizes 6, 10, 24, 40) or as one
// launch per level (other block sizes, or CPG_ILU_SWEEP=levels).
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <type_traits>

#include "internal.hpp"
#include "tcgen05.cuh"

using namespace cpg;

namespace cpg {
cpg_status rows_op(cpg_ctx *ctx, int precision, int bl, int nrows, const int *rows, const int *rowptr,
                   const int *col, const void *vals, const double *x, double *y, int mode);
}

namespace {

enum { MODE_MATVEC = 0, MODE_FORWARD = 1, MODE_BACKWARD = 2 };

// C = A * B or C -= A * B, column-major BL x BL blocks in shared memory.
// Each thread owns a 2 x 4 register tile (rows r0, r0+1; columns c0..c0+3);
// row tiles vary fastest across a warp, so the B reads are broadcasts and the
// A reads are consecutive doubles.
__device__ __forceinline__ void smem_gemm(int BL, const double *A, const double *B, double *C, bool sub) {
    const int tr_n = (BL + 1) / 2, tc_n = (BL + 3) / 4;
    for (int t = threadIdx.x; t < tr_n * tc_n; t += blockDim.x) {
        const int r0 = 2 * (t % tr_n), c0 = 4 * (t / tr_n);
        const bool r1ok = r0 + 1 < BL;
        const int nc = min(4, BL - c0);
        double acc[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
        const double *b0 = B + c0 * BL;
        for (int m = 0; m < BL; m++) {
            const double a0 = A[m * BL + r0], a1 = r1ok ? A[m * BL + r0 + 1] : 0.0;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const double bv = j < nc ? b0[j * BL + m] : 0.0;
                acc[0][j] += a0 * bv;
                acc[1][j] += a1 * bv;
            }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (j >= nc) break;
            double *cc = C + (c0 + j) * BL + r0;
            if (sub) {
                cc[0] = cc[0] - acc[0][j];
                if (r1ok) cc[1] = cc[1] - acc[1][j];
            } else {
                cc[0] = acc[0][j];
                if (r1ok) cc[1] = acc[1][j];
            }
        }
    }
}

// The same product on the FP64 tensor-core path (DMMA, mma.sync m8n8k4 f64;
// the 5th-generation tcgen05 MMA has no FP64 kind), for block sizes that are
// multiples of 8.  Each warp owns 8x8 output tiles and walks k in steps of
// four.  Fragments: A(g, t), B(t, g), C(g, 2t) and C(g, 2t+1) with
// g = lane / 4, t = lane % 4.
__device__ __forceinline__ void dmma_m8n8k4(double &d0, double &d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}
__device__ __forceinline__ void smem_gemm_dmma(int BL, const double *A, const double *B, double *C, bool sub) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int nt = BL >> 3;
    for (int tile = warp; tile < nt * nt; tile += nw) {  // warp-uniform: all lanes issue the MMA
        const int r0 = (tile % nt) * 8, c0 = (tile / nt) * 8;
        double d0 = 0.0, d1 = 0.0;
        for (int k = 0; k < BL; k += 4)
            dmma_m8n8k4(d0, d1, A[(k + t) * BL + r0 + g], B[(c0 + g) * BL + k + t]);
        double *cc = C + (size_t)(c0 + 2 * t) * BL + r0 + g;
        if (sub) {
            cc[0] = cc[0] - d0;
            cc[BL] = cc[BL] - d1;
        } else {
            cc[0] = d0;
            cc[BL] = d1;
        }
    }
}
__device__ __forceinline__ void block_gemm(int BL, const double *A, const double *B, double *C, bool sub) {
    if ((BL & 7) == 0) smem_gemm_dmma(BL, A, B, C, sub);
    else smem_gemm(BL, A, B, C, sub);
}

template <class T>
__device__ __forceinline__ void load_blk(int BL, const T *src, double *dst) {
    for (int o = threadIdx.x; o < BL * BL; o += blockDim.x) dst[o] = (double)src[o];
}
template <class T>
__device__ __forceinline__ void store_blk(int BL, const double *src, T *dst) {
    for (int o = threadIdx.x; o < BL * BL; o += blockDim.x) dst[o] = (T)src[o];
}

constexpr int FT = 320;  // threads per factor CTA: 8 columns x 40 rows of a 40x40 block at a time

// ---------------------------------------------------------------------------
// Pivot-block inverses, one warp per block (the batched kernel below runs a
// level's blocks side by side).  Gauss-Jordan with partial pivoting: pivot
// = largest magnitude, lowest index on ties (LAPACK's idamax rule); the
// column swaps that undo the pivoting are composed into perm, so column c of
// the inverse is column perm[c] of the result.  Both return false on a zero
// pivot.
// ---------------------------------------------------------------------------
// Shared-memory layout of the blocked form: column-major blocks with leading
// dimension inv_ld(BL) = BL + d, d making inv_ld = 10 (mod 16) (42 for 40x40),
// and the panel scratch S at 12 doubles per column: the DMMA accumulator
// accesses and S-fragment loads are conflict-free and the lane-per-column
// reads of S's rows 2-way.
__host__ __device__ constexpr int inv_ld(int bl) { return bl + (10 - bl % 16 + 16) % 16; }
constexpr int INV_SLD = 12;

__device__ __forceinline__ int warp_argmax_col(const double *A, int BL, int ld, int p, double &best_out) {
    const int lane = threadIdx.x & 31;
    double best = -1.0;
    int bi = p;
    for (int r = p + lane; r < BL; r += 32) {
        const double a = fabs(A[p * ld + r]);
        if (a > best) {
            best = a;
            bi = r;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, off);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
        if (ob > best || (ob == best && oi < bi)) {
            best = ob;
            bi = oi;
        }
    }
    best_out = best;
    return bi;
}

__device__ __forceinline__ void warp_compose_perm(int BL, const int *piv, int *perm) {
    if ((threadIdx.x & 31) == 0) {
        for (int c = 0; c < BL; c++) perm[c] = c;
        for (int p = BL - 1; p >= 0; p--) {
            const int q = piv[p], t = perm[p];
            perm[p] = perm[q];
            perm[q] = t;
        }
    }
    __syncwarp();
}

// Blocked form for BL % 8 == 0, in panels of 8 pivot columns, without moving
// rows: pivot column p is eliminated with row q_p, the largest among the rows
// not used yet, which stays where it is.  Ties go to the lowest position that
// the rows would have with LAPACK's swaps (rows p and q_p trade positions), so
// the pivots, and with them the result's bits, are those of the elimination
// that swaps.  The panel is
// eliminated in registers, a lane holding the 8 panel columns of its one or
// two rows; the pivot is found with three 32-bit warp reductions (the bits of
// a non-negative double order as it does) and its row reaches the other lanes
// in shuffles.  The other columns X then take the block update
// A_X <- [0 on the panel's pivot rows; A_X elsewhere] + panel * A_X(q, :), a
// rank-8 product on DMMA.  In the end (A^{-1})(p, q_s) = T(q_p, s) for the
// array T left in A.  S holds INV_SLD x (BL - 8) doubles of scratch.
//
// A pivot step is a chain of about 250 cycles, and 13 blocks share an SM; with
// the panel in shared memory and rows swapped it was 4,400 cycles (rows of a
// column hit by serial load-store pairs), 186 us a level of 3,300 40x40
// blocks (level average) against 93 us now.
template <int BL, int LD, int SLD>
__device__ bool warp_inverse_panel(double *A, double *S, int *row_of) {
    static_assert(BL % 8 == 0 && BL <= 64, "panel inverse shape");
    constexpr unsigned ALL = 0xffffffffu;
    constexpr int NX = BL - 8, RT = BL / 8, XT = NX / 8;
    constexpr bool TWO = BL > 32;  // lanes below BL - 32 hold a second row
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const bool has0 = lane < BL, has1 = TWO && lane + 32 < BL;
    bool free0 = has0, free1 = has1, ok = true;  // rows not used as a pivot yet
    int pos0 = lane, pos1 = lane + 32;           // their positions
    for (int K = 0; K < BL; K += 8) {
        double c[8], d[8];  // rows lane and lane + 32 of the panel
        int q[8];
        unsigned pm0 = 0, pm1 = 0;  // the panel's pivot rows
#pragma unroll
        for (int k = 0; k < 8; k++) {
            c[k] = has0 ? A[(K + k) * LD + lane] : 0.0;
            d[k] = has1 ? A[(K + k) * LD + lane + 32] : 0.0;
        }
#pragma unroll
        for (int p = 0; p < 8; p++) {
            // 0 for a used row and for NaN (never a pivot unless nothing else is left)
            const double m0 = fabs(c[p]), m1 = fabs(d[p]);
            const unsigned long long b0 = free0 && m0 >= 0.0 ? __double_as_longlong(m0) : 0ull;
            const unsigned long long b1 = TWO && free1 && m1 >= 0.0 ? __double_as_longlong(m1) : 0ull;
            const bool second = TWO && free1 && (!free0 || b1 > b0 || (b1 == b0 && pos1 < pos0));
            const unsigned long long bits = b1 > b0 ? b1 : b0;
            const unsigned hi = (unsigned)(bits >> 32), lo = (unsigned)bits;
            const unsigned mhi = __reduce_max_sync(ALL, hi);
            const unsigned mlo = __reduce_max_sync(ALL, hi == mhi ? lo : 0u);
            const bool best = (free0 || free1) && hi == mhi && lo == mlo;
            const unsigned chosen =
                __reduce_min_sync(ALL, best ? (unsigned)(second ? pos1 << 8 | (lane + 32) : pos0 << 8 | lane) : ~0u);
            const int row = chosen & 255, pos = chosen >> 8;
            ok = ok && (mhi | mlo) != 0u;
            if (pos0 == K + p) pos0 = pos;
            if (pos1 == K + p) pos1 = pos;
            q[p] = row;
            double rp[8];  // the pivot row, scaled
#pragma unroll
            for (int k = 0; k < 8; k++) rp[k] = __shfl_sync(ALL, TWO && row >= 32 ? d[k] : c[k], row & 31);
            const double pv = rp[p], inv = pv != 0.0 ? 1.0 / pv : 0.0;
#pragma unroll
            for (int k = 0; k < 8; k++) rp[k] = (k == p ? 1.0 : rp[k]) * inv;
            const double f0 = c[p], f1 = d[p];
            const bool is0 = row == lane, is1 = TWO && row == lane + 32;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                c[k] = is0 ? rp[k] : (k == p ? 0.0 : c[k]) - f0 * rp[k];
                if constexpr (TWO) d[k] = is1 ? rp[k] : (k == p ? 0.0 : d[k]) - f1 * rp[k];
            }
            free0 = free0 && !is0;
            free1 = free1 && !is1;
            if (row < 32) pm0 |= 1u << row;
            else pm1 |= 1u << (row & 31);
        }
#pragma unroll
        for (int k = 0; k < 8; k++) {
            if (has0) A[(K + k) * LD + lane] = c[k];
            if (has1) A[(K + k) * LD + lane + 32] = d[k];
            if (lane == k) row_of[K + k] = q[k];
        }
        for (int x = lane; x < NX; x += 32) {  // S = A_X(q, :)
            const double *col = A + (x < K ? x : x + 8) * LD;
#pragma unroll
            for (int k = 0; k < 8; k++) S[x * SLD + k] = col[q[k]];
        }
        __syncwarp();
        double s0[XT], s1[XT];
#pragma unroll
        for (int x = 0; x < XT; x++) {
            s0[x] = S[(8 * x + g) * SLD + t];
            s1[x] = S[(8 * x + g) * SLD + 4 + t];
        }
#pragma unroll 1
        for (int rt = 0; rt < RT; rt++) {
            const int r = 8 * rt + g;
            const bool pivot = ((r < 32 ? pm0 >> r : pm1 >> (r & 31)) & 1u) != 0u;
            const double a0 = A[(K + t) * LD + r], a1 = A[(K + 4 + t) * LD + r];
#pragma unroll
            for (int x = 0; x < XT; x++) {
                double *cc = A + (size_t)((8 * x < K ? 8 * x : 8 * x + 8) + 2 * t) * LD + r;
                double d0 = pivot ? 0.0 : cc[0], d1 = pivot ? 0.0 : cc[LD];
                dmma_m8n8k4(d0, d1, a0, s0[x]);
                dmma_m8n8k4(d0, d1, a1, s1[x]);
                cc[0] = d0;
                cc[LD] = d1;
            }
        }
        __syncwarp();
    }
    return ok;
}

// Unblocked form for any block size: the update ping-pongs between A and B
// with the row swap folded into the reads (rows p and q trade places), so
// no element is read after it is overwritten.  Returns the result buffer.
__device__ double *warp_inverse_gj(int BL, double *A, double *B, int *piv, int *perm, bool &ok) {
    const int lane = threadIdx.x & 31;
    ok = true;
    double *src = A, *dst = B;
    for (int p = 0; p < BL; p++) {
        double best;
        const int q = warp_argmax_col(src, BL, BL, p, best);
        ok = ok && best > 0.0;
        if (lane == 0) piv[p] = q;
        const double pv = src[p * BL + q];
        const double inv = (pv != 0.0) ? 1.0 / pv : 0.0;
        for (int o = lane; o < BL * BL; o += 32) {
            const int r = o % BL, c = o / BL;
            const double rp = (c == p ? 1.0 : src[c * BL + q]) * inv;
            if (r == p) {
                dst[o] = rp;
            } else {
                const int rs = (r == q) ? p : r;
                dst[o] = (c == p ? 0.0 : src[c * BL + rs]) - src[p * BL + rs] * rp;
            }
        }
        __syncwarp();
        double *tt = src;
        src = dst;
        dst = tt;
    }
    warp_compose_perm(BL, piv, perm);
    return src;
}

// block -> registers (PER elements per thread, element o = tid + k*FT)
template <int PER, class T>
__device__ __forceinline__ void fetch_blk(int BL2, const T *src, double (&v)[PER]) {
#pragma unroll
    for (int k = 0; k < PER; k++) {
        const int o = threadIdx.x + k * FT;
        v[k] = o < BL2 ? (double)src[o] : 0.0;
    }
}
template <int PER>
__device__ __forceinline__ void stash_blk(int BL2, const double (&v)[PER], double *dst) {
#pragma unroll
    for (int k = 0; k < PER; k++) {
        const int o = threadIdx.x + k * FT;
        if (o < BL2) dst[o] = v[k];
    }
}

// Padded shared-memory blocks for the DMMA path: column-major with leading
// dimension LD = BL + 4 doubles.  With LD = BL the fragment loads of the
// m8n8k4 products hit the same banks 2-way (A operand) and 4-way (B
// operand); the padding staggers the columns so a half-warp's sixteen
// 8-byte loads fall in distinct banks.
template <int BL>
struct Pad {
    static constexpr int LD = BL + 4;
    static __device__ __forceinline__ int at(int o) { return (o / BL) * LD + o % BL; }  // dense index -> padded
};
template <int BL, int PER>
__device__ __forceinline__ void stash_pad(const double (&v)[PER], double *dst) {
#pragma unroll
    for (int k = 0; k < PER; k++) {
        const int o = threadIdx.x + k * FT;
        if (o < BL * BL) dst[Pad<BL>::at(o)] = v[k];
    }
}
template <int BL, class T>
__device__ __forceinline__ void load_pad(const T *src, double *dst) {
    for (int o = threadIdx.x; o < BL * BL; o += FT) dst[Pad<BL>::at(o)] = (double)src[o];
}
template <int BL, class T>
__device__ __forceinline__ void store_pad(const double *src, T *dst) {
    for (int o = threadIdx.x; o < BL * BL; o += FT) dst[o] = (T)src[Pad<BL>::at(o)];
}
// One 8-row strip of a product on padded blocks: tiles [c0, c0 + 8 NTC) of
// rows r0..r0+7, the tiles' accumulators in registers.  Each A fragment is
// loaded once for the strip's NTC products (1 + NTC shared loads per NTC
// MMAs, against 2 per MMA for single tiles); every tile still accumulates
// its k steps in ascending order.
template <int BL, int NTC>
__device__ __forceinline__ void strip_mma(const double *A, const double *B, int r0, int c0, double (&d)[NTC][2]) {
    constexpr int LD = Pad<BL>::LD;
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int c = 0; c < NTC; c++) d[c][0] = d[c][1] = 0.0;
#pragma unroll 2
    for (int k = 0; k < BL; k += 4) {
        const double a = A[(k + t) * LD + r0 + g];
#pragma unroll
        for (int c = 0; c < NTC; c++) dmma_m8n8k4(d[c][0], d[c][1], a, B[(c0 + 8 * c + g) * LD + k + t]);
    }
}
// The three products of one lower neighbour (L_ji = A_ji D_i^{-1} into T,
// U_ij = D_i^{-1} A_ij straight to global, then Ahat_jj -= L_ji A_ij), by
// strips: the two independent products run side by side on the two halves
// of the CTA's warps, and the update splits each strip in two.
template <int BL, class TS>
__device__ __forceinline__ void neighbour_products(const double *Xp, const double *Dp, const double *Yp, double *Tp,
                                                   double *Ap, TS *U) {
    constexpr int LD = Pad<BL>::LD, NT = BL / 8, NW = FT / 32, HALF = NW / 2;
    constexpr int NH = (NT + 1) / 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    if (warp < HALF) {
        for (int st = warp; st < NT; st += HALF) {  // T = X D
            double d[NT][2];
            strip_mma<BL, NT>(Xp, Dp, 8 * st, 0, d);
#pragma unroll
            for (int c = 0; c < NT; c++) {
                double *cc = Tp + (8 * c + 2 * t) * LD + 8 * st + g;
                cc[0] = d[c][0];
                cc[LD] = d[c][1];
            }
        }
    } else {
        for (int st = warp - HALF; st < NT; st += HALF) {  // U = D Y
            double d[NT][2];
            strip_mma<BL, NT>(Dp, Yp, 8 * st, 0, d);
#pragma unroll
            for (int c = 0; c < NT; c++) {
                TS *cc = U + (size_t)(8 * c + 2 * t) * BL + 8 * st + g;
                cc[0] = (TS)d[c][0];
                cc[BL] = (TS)d[c][1];
            }
        }
    }
    __syncthreads();
    for (int u = warp; u < 2 * NT; u += NW) {  // Ahat -= T Y, half a strip per unit
        const int st = u >> 1;
        if ((u & 1) == 0) {
            double d[NH][2];
            strip_mma<BL, NH>(Tp, Yp, 8 * st, 0, d);
#pragma unroll
            for (int c = 0; c < NH; c++) {
                double *cc = Ap + (8 * c + 2 * t) * LD + 8 * st + g;
                cc[0] = cc[0] - d[c][0];
                cc[LD] = cc[LD] - d[c][1];
            }
        } else if constexpr (NT - NH > 0) {
            double d[NT - NH][2];
            strip_mma<BL, NT - NH>(Tp, Yp, 8 * st, 8 * NH, d);
#pragma unroll
            for (int c = 0; c < NT - NH; c++) {
                double *cc = Ap + (8 * (NH + c) + 2 * t) * LD + 8 * st + g;
                cc[0] = cc[0] - d[c][0];
                cc[LD] = cc[LD] - d[c][1];
            }
        }
    }
}

// One CTA per row j of the level:
//   for each lower neighbour i < j (ascending):
//       L_ji = A_ji D_i^{-1}; Ahat_jj -= L_ji A_ij; U_ij = D_i^{-1} A_ij
// then k_block_inverse forms D_j^{-1} = inv(Ahat_jj) for the whole level.
// BLC > 0 compiles the block size in: the three blocks of the next lower
// neighbour are then fetched into registers while the current products run,
// and with BLC % 8 == 0 the products run on DMMA with U_ij stored straight
// from the fragments.  BLC == 0 is the generic path (any block size).
template <class TA, class TS, int BLC>
__global__ void __launch_bounds__(FT, 3) k_ilu_factor(int bl_rt, const int *__restrict__ rows, const TA *__restrict__ A,
                                                   const int *__restrict__ diag_a, const int *__restrict__ lp_ptr,
                                                   const int *__restrict__ lp_i, const int *__restrict__ lp_aji,
                                                   const int *__restrict__ lp_aij, const int *__restrict__ lp_l,
                                                   const int *__restrict__ lp_u, TS *__restrict__ Lv,
                                                   TS *Uv, const int *__restrict__ U_rowptr,
                                                   double *dinv, const int *__restrict__ dinv_idx, int *flag,
                                                   double *__restrict__ Eout) {
    extern __shared__ double sm[];
    const int BL = BLC ? BLC : bl_rt;
    const int BL2 = BL * BL;
    const size_t b2 = (size_t)BL2;
    double *Ah = sm, *D = sm + b2, *X = sm + 2 * b2, *Y = sm + 3 * b2, *T = sm + 4 * b2;
    const int j = rows ? rows[blockIdx.x] : blockIdx.x;
    const int p0 = lp_ptr[j], p1 = lp_ptr[j + 1];
    if constexpr (BLC > 0 && BLC % 8 == 0) {  // DMMA on padded blocks
        constexpr int PER = (BLC * BLC + FT - 1) / FT;
        constexpr int PB = BLC * Pad<BLC>::LD;   // doubles per padded block
        double *Ap = sm, *Dp = sm + PB, *Xp = sm + 2 * PB, *Yp = sm + 3 * PB, *Tp = sm + 4 * PB;
        double rd[PER], rx[PER], ry[PER];
        if (p0 < p1) {
            fetch_blk<PER>(BL2, dinv + (size_t)dinv_idx[lp_i[p0]] * b2, rd);
            fetch_blk<PER>(BL2, A + (size_t)lp_aji[p0] * b2, rx);
            fetch_blk<PER>(BL2, A + (size_t)lp_aij[p0] * b2, ry);
        }
        load_pad<BLC>(A + (size_t)diag_a[j] * b2, Ap);
        for (int p = p0; p < p1; p++) {
            stash_pad<BLC, PER>(rd, Dp);
            stash_pad<BLC, PER>(rx, Xp);
            stash_pad<BLC, PER>(ry, Yp);
            __syncthreads();
            if (p + 1 < p1) {  // next neighbour's blocks in flight during the products
                fetch_blk<PER>(BL2, dinv + (size_t)dinv_idx[lp_i[p + 1]] * b2, rd);
                fetch_blk<PER>(BL2, A + (size_t)lp_aji[p + 1] * b2, rx);
                fetch_blk<PER>(BL2, A + (size_t)lp_aij[p + 1] * b2, ry);
            } else if (Eout) {  // last neighbour: A_jj again, for E_j below
                fetch_blk<PER>(BL2, A + (size_t)diag_a[j] * b2, rx);
            }
            neighbour_products<BLC, TS>(Xp, Dp, Yp, Tp, Ap, Uv + (size_t)lp_u[p] * b2);
            store_pad<BLC>(Tp, Lv + (size_t)lp_l[p] * b2);
            __syncthreads();
        }
        __syncthreads();
        // Ahat_jj goes to its D^{-1} slot; k_block_inverse inverts it in place
        store_pad<BLC>(Ap, dinv + (size_t)dinv_idx[j] * b2);
        if (Eout) {  // E_j = A_jj - Ahat_jj for the split form of P^{-1} A (0 without lower neighbours)
#pragma unroll
            for (int k = 0; k < PER; k++) {
                const int o = threadIdx.x + k * FT;
                if (o < BL2) Eout[(size_t)j * b2 + o] = p0 < p1 ? rx[k] - Ap[Pad<BLC>::at(o)] : 0.0;
            }
        }
        return;
    } else if constexpr (BLC > 0) {  // compiled-in sizes not divisible by 8: scalar products
        constexpr int PER = (BLC * BLC + FT - 1) / FT;
        double rd[PER], rx[PER], ry[PER];
        if (p0 < p1) {
            fetch_blk<PER>(BL2, dinv + (size_t)dinv_idx[lp_i[p0]] * b2, rd);
            fetch_blk<PER>(BL2, A + (size_t)lp_aji[p0] * b2, rx);
            fetch_blk<PER>(BL2, A + (size_t)lp_aij[p0] * b2, ry);
        }
        load_blk(BL, A + (size_t)diag_a[j] * b2, Ah);
        for (int p = p0; p < p1; p++) {
            stash_blk<PER>(BL2, rd, D);
            stash_blk<PER>(BL2, rx, X);
            stash_blk<PER>(BL2, ry, Y);
            __syncthreads();
            if (p + 1 < p1) {  // next neighbour's blocks in flight during the products
                fetch_blk<PER>(BL2, dinv + (size_t)dinv_idx[lp_i[p + 1]] * b2, rd);
                fetch_blk<PER>(BL2, A + (size_t)lp_aji[p + 1] * b2, rx);
                fetch_blk<PER>(BL2, A + (size_t)lp_aij[p + 1] * b2, ry);
            }
            smem_gemm(BL, X, D, T, false);  // L_ji
            __syncthreads();
            store_blk(BL, T, Lv + (size_t)lp_l[p] * b2);
            smem_gemm(BL, T, Y, Ah, true);   // Ahat_jj -= L_ji A_ij
            smem_gemm(BL, D, Y, X, false);   // U_ij
            __syncthreads();
            store_blk(BL, X, Uv + (size_t)lp_u[p] * b2);
            __syncthreads();
        }
    } else {
        load_blk(BL, A + (size_t)diag_a[j] * b2, Ah);
        for (int p = p0; p < p1; p++) {
            load_blk(BL, dinv + (size_t)dinv_idx[lp_i[p]] * b2, D);
            load_blk(BL, A + (size_t)lp_aji[p] * b2, X);
            load_blk(BL, A + (size_t)lp_aij[p] * b2, Y);
            __syncthreads();
            block_gemm(BL, X, D, T, false);  // L_ji
            __syncthreads();
            store_blk(BL, T, Lv + (size_t)lp_l[p] * b2);
            block_gemm(BL, T, Y, Ah, true);   // Ahat_jj -= L_ji A_ij
            block_gemm(BL, D, Y, X, false);   // U_ij
            __syncthreads();
            store_blk(BL, X, Uv + (size_t)lp_u[p] * b2);
            __syncthreads();
        }
    }
    __syncthreads();
    // Ahat_jj goes to its D^{-1} slot; k_block_inverse inverts it in place
    double *dj = dinv + (size_t)dinv_idx[j] * b2;
    for (int o = threadIdx.x; o < BL2; o += FT) dj[o] = Ah[o];
    if (Eout) {  // E_j = A_jj - Ahat_jj for the split form of P^{-1} A
        const TA *ajj = A + (size_t)diag_a[j] * b2;
        for (int o = threadIdx.x; o < BL2; o += FT) Eout[(size_t)j * b2 + o] = (double)ajj[o] - Ah[o];
    }
}

// max over rows of sum_c |B(r, c)| for a column-major BL x BL block
// (leading dimension ld) in shared memory (lanes over rows: consecutive addresses), on every lane
__device__ __forceinline__ double warp_norm_inf(int BL, int ld, const double *B) {
    double m = 0.0;
    for (int r = threadIdx.x & 31; r < BL; r += 32) {
        double sum = 0.0;
        for (int c = 0; c < BL; c++) sum += fabs(B[(size_t)c * ld + r]);
        m = fmax(m, sum);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, off));
    return m;
}

// The level's pivot blocks, one warp each: Ahat_jj (FP64, in its D^{-1}
// slot) -> D_j^{-1} in place, and into the DU row's first block when the
// factors are stored in FP32.  WPB warps per CTA, each with its own shared
// block (plus a second one or the panel scratch).
template <class TS, int BLC>
__global__ void __launch_bounds__(128) k_block_inverse(int bl_rt, int nrows, const int *__restrict__ rows,
                                                       TS *Uv, const int *__restrict__ U_rowptr, double *dinv,
                                                       const int *__restrict__ dinv_idx, int *flag,
                                                       unsigned long long *cond_max) {
    extern __shared__ double sm[];
    const int BL = BLC ? BLC : bl_rt;
    const size_t b2 = (size_t)BL * BL;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    const int k = blockIdx.x * wpb + warp;  // this warp's row of the level
    if (k >= nrows) return;                 // warp-uniform; no block-wide barriers below
    constexpr bool PANEL = BLC > 0 && BLC % 8 == 0;
    constexpr int BLP = BLC > 0 ? BLC : 8;
    // doubles per warp: the block (leading dimension ld), then the panel
    // scratch (INV_SLD x (BL-8)) or a second block, then piv + perm (ints)
    const int ld = PANEL ? inv_ld(BL) : BL;
    const size_t blk = (size_t)ld * BL;
    const size_t second = PANEL ? (size_t)INV_SLD * (BL - 8) : b2;
    const size_t per_warp = blk + second + BL;
    double *A = sm + warp * per_warp, *B = A + blk;
    int *piv = (int *)(B + second), *perm = piv + BL;
    const int j = rows ? rows[k] : k;
    double *dj = dinv + (size_t)dinv_idx[j] * b2;
    for (int o = lane; o < (int)b2; o += 32) A[(o / BL) * ld + o % BL] = dj[o];
    __syncwarp();
    const double nrm_a = warp_norm_inf(BL, ld, A);  // before the inversion overwrites A
    bool ok;
    const double *Di;
    if constexpr (PANEL) {
        ok = warp_inverse_panel<BLP, inv_ld(BLP), INV_SLD>(A, B, perm);
        Di = A;
    } else {
        Di = warp_inverse_gj(BL, A, B, piv, perm, ok);
    }
    if (!ok && lane == 0) {
        atomicExch(flag, 1);
        atomicMin(flag + 1, j);
    }
    // cond_inf(Ahat_jj) = |Ahat_jj|_inf |Ahat_jj^{-1}|_inf (the inverse's row
    // sums do not depend on the column order perm); the largest over all
    // pivot blocks, by the ordering of non-negative doubles' bit patterns
    const double cond = nrm_a * warp_norm_inf(BL, ld, Di);
    if (ok && lane == 0 && cond_max) atomicMax(cond_max, (unsigned long long)__double_as_longlong(cond));
    TS *uj = Uv + (size_t)U_rowptr[j] * b2;
    const bool both = (void *)uj != (void *)dj;
    for (int c = 0; c < BL; c++) {
        // unblocked: column c is column perm[c] of the result; blocked: the
        // result's column c belongs to column perm[c], its rows to rows perm[r]
        const double *src = Di + (size_t)(PANEL ? c : perm[c]) * ld;
        const size_t to = (size_t)(PANEL ? perm[c] : c) * BL;
        for (int r = lane; r < BL; r += 32) {
            const double v = src[PANEL ? perm[r] : r];
            dj[to + r] = v;
            if (both) uj[to + r] = (TS)v;
        }
    }
}

// ---------------------------------------------------------------------------
// FP32 factors of 40x40 blocks on the 5th-generation tensor cores.  The same
// three products per lower neighbour as k_ilu_factor (L_ji = A_ji D_i^{-1},
// U_ij = D_i^{-1} A_ij, Ahat_jj -= L_ji A_ij), each a 64 x 40 x 40
// tcgen05.mma of kind::tf32 (M padded from 40 to 64 with zero rows, five K
// steps of 8) with the FP32 accumulator in TMEM.  SPLIT = 3 carries each FP32
// operand as two TF32 parts and sums three products per K step, for about
// FP32 accuracy; SPLIT = 1 is plain TF32.  One CTA (one warpgroup) per row:
// all threads stage the operands into shared memory (core-matrix layout),
// thread 0 issues the MMAs and commits them to an mbarrier, warps 0-2 read
// the accumulators back (row m of an M = 64 accumulator sits in TMEM lane
// m % 16 + 32 (m / 16)).  Ahat_jj = A_jj - sum L A is formed in FP64 in the
// pivot's D^{-1} slot, which k_block_inverse then inverts in FP64 as before.
// Every mbarrier wait is bounded; one that runs out sets flag[6], and the CTA
// frees its TMEM and returns (the factorisation reports CPG_ERR_TIMEOUT).
// ---------------------------------------------------------------------------
namespace tcf {
constexpr int BL = 40, M = 64, NT = 128, KSTEPS = BL / 8;
constexpr int LBO = 128;                    // bytes between the 4-wide K chunks of a row group
constexpr int SBO = (BL / 4) * LBO;         // bytes between 8-row groups (the whole K extent)
constexpr int A_TILE = (M / 8) * SBO;       // 64 x 40 TF32: rows 40..63 stay zero
constexpr int B_TILE = (BL / 8) * SBO;      // 40 x 40 TF32
constexpr int PER = (BL * BL + NT - 1) / NT;
constexpr uint32_t TMEM_COLS = 128;         // L at column 0, U at 40, sum(L A) at 80
constexpr long long MAX_SPINS = 1LL << 24;  // mbarrier polls (>= 32 ns apart): > 0.5 s
__host__ __device__ constexpr size_t smem_bytes(int split) {
    return (size_t)(split == 3 ? 2 : 1) * (3 * A_TILE + 2 * B_TILE) + 64;
}
// byte offset of element (row r, K index k) in a K-major core-matrix tile
__device__ __forceinline__ int off(int r, int k) { return (r >> 3) * SBO + (k >> 2) * LBO + (r & 7) * 16 + (k & 3) * 4; }
__device__ __forceinline__ void put(unsigned char *hi, unsigned char *lo, int o, float x) {
    if (lo) {
        float h, l;
        tc::split_tf32(x, h, l);
        *(float *)(hi + o) = h;
        *(float *)(lo + o) = l;
    } else {
        *(float *)(hi + o) = x;
    }
}
// C (TMEM) = A * B over the five K steps; acc0: add to C's content
template <int SPLIT>
__device__ __forceinline__ void product(uint32_t c, const unsigned char *Ah, const unsigned char *Al,
                                        const unsigned char *Bh, const unsigned char *Bl, bool acc0) {
    constexpr uint32_t idesc = tc::idesc_tf32(M, BL);
#pragma unroll
    for (int s = 0; s < KSTEPS; s++) {
        const uint32_t ko = (uint32_t)s * 2 * LBO;
        const uint64_t ah = tc::sdesc(tc::saddr(Ah) + ko, LBO, SBO), bh = tc::sdesc(tc::saddr(Bh) + ko, LBO, SBO);
        tc::mma_tf32(c, ah, bh, idesc, (acc0 || s > 0) ? 1u : 0u);
        if (SPLIT == 3) {
            const uint64_t al = tc::sdesc(tc::saddr(Al) + ko, LBO, SBO), bl = tc::sdesc(tc::saddr(Bl) + ko, LBO, SBO);
            tc::mma_tf32(c, ah, bl, idesc, 1u);
            tc::mma_tf32(c, al, bh, idesc, 1u);
        }
    }
}
// thread 0 waits (bounded) for the committed MMAs; the barrier hands the
// outcome to every thread
__device__ __forceinline__ bool wait_mma(uint64_t *bar, uint32_t parity, volatile int *s_ok) {
    if (threadIdx.x == 0) {
        long long spins = 0;
        while (!tc::mbar_test(bar, parity)) {
            if (++spins > MAX_SPINS) {
                *s_ok = 0;
                break;
            }
            if (spins > 64) __nanosleep(32);
        }
    }
    __syncthreads();
    return *s_ok != 0;
}
}  // namespace tcf

template <int SPLIT>
__global__ void __launch_bounds__(tcf::NT) k_ilu_factor_tc(const int *__restrict__ rows, const float *__restrict__ A,
                                                          const int *__restrict__ diag_a, const int *__restrict__ lp_ptr,
                                                          const int *__restrict__ lp_i, const int *__restrict__ lp_aji,
                                                          const int *__restrict__ lp_aij, const int *__restrict__ lp_l,
                                                          const int *__restrict__ lp_u, float *__restrict__ Lv,
                                                          float *__restrict__ Uv, double *dinv,
                                                          const int *__restrict__ dinv_idx, int *flag) {
    using namespace tcf;
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr int H = SPLIT == 3 ? 2 : 1;  // tiles per operand
    unsigned char *XA = smem, *DA = XA + H * A_TILE, *LA = DA + H * A_TILE;
    unsigned char *DB = LA + H * A_TILE, *YB = DB + H * B_TILE;
    uint64_t *bar = (uint64_t *)(YB + H * B_TILE);
    uint32_t *s_tmem = (uint32_t *)(bar + 1);
    volatile int *s_ok = (volatile int *)(s_tmem + 1);
    auto lo = [&](unsigned char *t, int tile) -> unsigned char * { return SPLIT == 3 ? t + tile : nullptr; };
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int j = rows[blockIdx.x];
    const int p0 = lp_ptr[j], p1 = lp_ptr[j + 1];
    constexpr int BL2 = BL * BL;
    // zero the A-operand tiles once: their rows 40..63 are never written
    for (int o = tid; o < 3 * H * A_TILE / 16; o += NT) ((uint4 *)smem)[o] = make_uint4(0u, 0u, 0u, 0u);
    if (tid == 0) {
        tc::mbar_init(bar, 1);
        *s_ok = 1;
    }
    if (warp == 0) tc::tmem_alloc(s_tmem, TMEM_COLS);
    tc::fence_smem_async();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tbase = *s_tmem;
    const uint32_t tL = tbase, tU = tbase + 40, tS = tbase + 80;
    const uint32_t lrow = (uint32_t)(32 * warp) << 16;  // this warp's TMEM lane base
    const int m = 16 * warp + lane;                      // accumulator row held by this thread
    const bool row_ok = warp < 3 && lane < 16 && m < BL;
    uint32_t parity = 0;
    bool ok = true;
    double rd[PER];
    float rx[PER], ry[PER];
    auto fetch = [&](int p) {
        const double *d = dinv + (size_t)dinv_idx[lp_i[p]] * BL2;
        const float *x = A + (size_t)lp_aji[p] * BL2, *y = A + (size_t)lp_aij[p] * BL2;
#pragma unroll
        for (int k = 0; k < PER; k++) {
            const int o = tid + k * NT;
            rd[k] = o < BL2 ? d[o] : 0.0;
            rx[k] = o < BL2 ? x[o] : 0.0f;
            ry[k] = o < BL2 ? y[o] : 0.0f;
        }
    };
    if (p0 < p1) fetch(p0);
    for (int p = p0; p < p1 && ok; p++) {
        // operands: X = A_ji and D = D_i^{-1} as A tiles (row, K), D and
        // Y = A_ij as B tiles (column, K); blocks are column-major
#pragma unroll
        for (int k = 0; k < PER; k++) {
            const int o = tid + k * NT;
            if (o < BL2) {
                const int r = o % BL, c = o / BL;
                const float dv = (float)rd[k];
                put(XA, lo(XA, A_TILE), off(r, c), rx[k]);
                put(DA, lo(DA, A_TILE), off(r, c), dv);
                put(DB, lo(DB, B_TILE), off(c, r), dv);
                put(YB, lo(YB, B_TILE), off(c, r), ry[k]);
            }
        }
        tc::fence_smem_async();
        tc::fence_before();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after();
            product<SPLIT>(tL, XA, lo(XA, A_TILE), DB, lo(DB, B_TILE), false);  // L_ji = A_ji D_i^{-1}
            product<SPLIT>(tU, DA, lo(DA, A_TILE), YB, lo(YB, B_TILE), false);  // U_ij = D_i^{-1} A_ij
            tc::commit(bar);
        }
        if (p + 1 < p1) fetch(p + 1);  // the next neighbour's blocks in flight during the products
        ok = wait_mma(bar, parity, s_ok);
        parity ^= 1;
        if (!ok) break;
        tc::fence_after();
        if (warp < 3) {
            float* Lg = Lv + (size_t)lp_l[p] * BL2;
            float* Ug = Uv + (size_t)lp_u[p] * BL2;
#pragma unroll
            for (int cb = 0; cb < BL / 8; cb++) {
                float v[8], w[8];
                tc::tmem_ld8(tL + lrow + 8 * cb, v);
                tc::tmem_ld8(tU + lrow + 8 * cb, w);
                tc::tmem_wait_ld();
                if (row_ok) {
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        const int n = 8 * cb + q;
                        Lg[(size_t)n * BL + m] = v[q];
                        Ug[(size_t)n * BL + m] = w[q];
                        put(LA, lo(LA, A_TILE), off(m, n), v[q]);  // L_ji as the A operand of the update
                    }
                }
            }
        }
        tc::fence_smem_async();
        tc::fence_before();
        __syncthreads();
        if (tid == 0) {
            tc::fence_after();
            product<SPLIT>(tS, LA, lo(LA, A_TILE), YB, lo(YB, B_TILE), p > p0);  // sum_i L_ji A_ij
            tc::commit(bar);
        }
        ok = wait_mma(bar, parity, s_ok);  // the tiles are free again
        parity ^= 1;
    }
    // Ahat_jj = A_jj - sum_i L_ji A_ij, FP64, into the pivot's D^{-1} slot
    double *dj = dinv + (size_t)dinv_idx[j] * BL2;
    const float *ajj = A + (size_t)diag_a[j] * BL2;
    if (ok && p0 == p1) {
        for (int o = tid; o < BL2; o += NT) dj[o] = (double)ajj[o];
    } else if (ok) {
        tc::fence_after();
        if (warp < 3) {
#pragma unroll
            for (int cb = 0; cb < BL / 8; cb++) {
                float v[8];
                tc::tmem_ld8(tS + lrow + 8 * cb, v);
                tc::tmem_wait_ld();
                if (row_ok) {
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        const size_t o = (size_t)(8 * cb + q) * BL + m;
                        dj[o] = (double)ajj[o] - (double)v[q];
                    }
                }
            }
        }
    }
    tc::fence_before();
    __syncthreads();
    if (warp == 0) {
        tc::fence_after();
        tc::tmem_dealloc(tbase, TMEM_COLS);
    }
    if (!ok && tid == 0) atomicExch(flag + 6, 1);
}

// The tensor-core factor applies to FP32 matrices and factors of 40x40
// blocks, on request: CPG_FACTOR_TC=3 (three TF32 passes) or =1 (one pass).
// The default keeps the FP64-DMMA products: the pivot update Ahat_jj -=
// sum L_ji A_ij of the stiff Newton matrix cancels heavily, and TF32-class
// products with an FP32 accumulator leave pivots that double FGMRES's
// iterations (three passes) or stall it (one pass).
int factor_tc_mode() {
    const char *e = std::getenv("CPG_FACTOR_TC");
    if (!e) return 0;
    const int v = std::atoi(e);
    return v == 0 ? 0 : (v == 1 ? 1 : 3);
}

template <int SPLIT>
cpg_status launch_factor_tc(cpg_ctx *ctx, cpg_precond *P, const cpg_bsr *A, int nrows, const int *rows) {
    // dynamic shared memory of at least 57 KB keeps at most 4 CTAs (4 x 128
    // TMEM columns) on an SM, so no TMEM allocation ever waits for another CTA
    const size_t smem = std::max<size_t>(tcf::smem_bytes(SPLIT), 57 * 1024);
    CPG_TRY(smem_limit_once(ctx, (const void *)k_ilu_factor_tc<SPLIT>, (int)smem));
    k_ilu_factor_tc<SPLIT><<<nrows, tcf::NT, smem, ctx->stream>>>(
        rows, (const float *)A->vals, P->diag_a_d, P->lp_ptr_d, P->lp_i_d, P->lp_aji_d, P->lp_aij_d, P->lp_l_d,
        P->lp_u_d, (float *)P->L_vals, (float *)P->U_vals, P->dinv64, P->dinv_idx_d, ctx->flag_dev);
    CPG_TRY(launched(ctx, "ilu factor kernel (tcgen05 tf32)"));
    // pivot-block inverses in FP64, as on the other paths
    constexpr int BL = tcf::BL;
    const size_t per_warp = ((size_t)inv_ld(BL) * BL + (size_t)INV_SLD * (BL - 8) + BL) * sizeof(double);
    const int wpb = 1;
    const size_t ismem = per_warp * wpb;
    CPG_TRY(smem_limit_once(ctx, (const void *)k_block_inverse<float, 40>, (int)ismem));
    k_block_inverse<float, 40><<<(nrows + wpb - 1) / wpb, 32 * wpb, ismem, ctx->stream>>>(
        BL, nrows, rows, (float *)P->U_vals, P->U_rowptr_d, P->dinv64, P->dinv_idx_d, ctx->flag_dev, P->cond_d);
    return launched(ctx, "pivot block inverse kernel");
}

template <class TA, class TS, int BLC>
cpg_status launch_factor_bl(cpg_ctx *ctx, cpg_precond *P, const cpg_bsr *A, int nrows, const int *rows) {
    if constexpr (std::is_same<TA, float>::value && std::is_same<TS, float>::value && BLC == 40) {
        const int mode = factor_tc_mode();
        if (mode == 3) return launch_factor_tc<3>(ctx, P, A, nrows, rows);
        if (mode == 1) return launch_factor_tc<1>(ctx, P, A, nrows, rows);
    }
    const int BL = P->bl;
    const int ld = (BLC > 0 && BLC % 8 == 0) ? BL + 4 : BL;  // padded blocks on the DMMA path
    const size_t smem = 5 * (size_t)BL * ld * sizeof(double) + 16;
    // compiled-in block sizes have one size; the generic kernel gets the
    // whole shared memory of a CTA, so its limit is raised once for any size
    CPG_TRY(smem_limit_once(ctx, (const void *)k_ilu_factor<TA, TS, BLC>,
                            BLC > 0 ? (int)smem : (smem > 48 * 1024 ? 227 * 1024 : 0)));
    if (smem > 227 * 1024) return fail(ctx, CPG_ERR_UNSUPPORTED, "block too large for the factor kernel");
    double *dinv = P->precision == CPG_F64 ? (double *)P->U_vals : P->dinv64;
    // E_j for the split form: FP64 values and FP64 factors only
    constexpr bool F64 = std::is_same<TA, double>::value && std::is_same<TS, double>::value;
    double *E = (F64 && P->split_capable) ? P->E_vals : nullptr;
    k_ilu_factor<TA, TS, BLC><<<nrows, FT, smem, ctx->stream>>>(
        BL, rows, (const TA *)A->vals, P->diag_a_d, P->lp_ptr_d, P->lp_i_d, P->lp_aji_d, P->lp_aij_d, P->lp_l_d,
        P->lp_u_d, (TS *)P->L_vals, (TS *)P->U_vals, P->U_rowptr_d, dinv, P->dinv_idx_d, ctx->flag_dev, E);
    CPG_TRY(launched(ctx, "ilu factor kernel"));
    // pivot-block inverses: else up to 4 warps per CTA within 110 KB of shared memory
    constexpr bool PANEL = BLC > 0 && BLC % 8 == 0;
    const size_t b2 = (size_t)BL * BL;
    const size_t per_warp =
        ((PANEL ? (size_t)inv_ld(BL) * BL + (size_t)INV_SLD * (BL - 8) : 2 * b2) + BL) * sizeof(double);
    // a warp per CTA in the blocked form: as many blocks share an SM as its shared memory holds
    const int wpb = PANEL ? 1 : (int)std::max<size_t>(1, std::min<size_t>(4, (110 * 1024) / per_warp));
    const size_t ismem = per_warp * wpb;
    if (ismem > 227 * 1024) return fail(ctx, CPG_ERR_UNSUPPORTED, "pivot block too large for shared memory");
    CPG_TRY(smem_limit_once(ctx, (const void *)k_block_inverse<TS, BLC>,
                            BLC > 0 ? (int)ismem : (ismem > 48 * 1024 ? 227 * 1024 : 0)));
    k_block_inverse<TS, BLC><<<(nrows + wpb - 1) / wpb, 32 * wpb, ismem, ctx->stream>>>(
        BL, nrows, rows, (TS *)P->U_vals, P->U_rowptr_d, dinv, P->dinv_idx_d, ctx->flag_dev, P->cond_d);
    return launched(ctx, "pivot block inverse kernel");
}

template <class TA, class TS>
cpg_status launch_factor(cpg_ctx *ctx, cpg_precond *P, const cpg_bsr *A, int nrows, const int *rows) {
    if (P->bl > FT) return fail(ctx, CPG_ERR_UNSUPPORTED, "block size above the factor kernel's thread count");
    switch (P->bl) {
        case 6: return launch_factor_bl<TA, TS, 6>(ctx, P, A, nrows, rows);
        case 10: return launch_factor_bl<TA, TS, 10>(ctx, P, A, nrows, rows);
        case 24: return launch_factor_bl<TA, TS, 24>(ctx, P, A, nrows, rows);
        case 40: return launch_factor_bl<TA, TS, 40>(ctx, P, A, nrows, rows);
        case 48: return launch_factor_bl<TA, TS, 48>(ctx, P, A, nrows, rows);
        default: return launch_factor_bl<TA, TS, 0>(ctx, P, A, nrows, rows);
    }
}

cpg_status factor_level(cpg_ctx *ctx, cpg_precond *P, const cpg_bsr *A, int nrows, const int *rows) {
    if (nrows <= 0) return CPG_OK;
    if (A->precision == CPG_F64 && P->precision == CPG_F64) return launch_factor<double, double>(ctx, P, A, nrows, rows);
    if (A->precision == CPG_F64 && P->precision == CPG_F32) return launch_factor<double, float>(ctx, P, A, nrows, rows);
    if (A->precision == CPG_F32 && P->precision == CPG_F32) return launch_factor<float, float>(ctx, P, A, nrows, rows);
    return launch_factor<float, double>(ctx, P, A, nrows, rows);
}

void free_precond(cpg_precond *P) {
    void *ptrs[] = {P->lrows_d, P->urows_d, P->L_rowptr_d, P->L_col_d, P->L_vals, P->U_rowptr_d, P->U_col_d,
                    P->U_vals, P->dinv64, P->dinv_idx_d, P->lp_ptr_d, P->lp_i_d, P->lp_aji_d, P->lp_aij_d,
                    P->lp_l_d, P->lp_u_d, P->diag_a_d, P->sweep.rows, P->E_vals, P->u2a_d, P->cond_d,
                    P->tune_tmp};
    for (void *p : ptrs) dfree(p);
    op_plan_free(P);
}

}  // namespace

namespace cpg {

namespace sweep_form {

cpg_status apply_syncfree(cpg_ctx *ctx, const cpg_precond *P, double *x, int kind) {
    int *err = ctx->flag_dev + 2;  // status word: a wait ran out
    if (!P->sweep.clean) CPG_TRY(sweep_workspace(ctx, P));  // a launch failed half way
    SweepState st = P->sweep;
    st.flags = P->row_flags_d;
    st.gen = 2 * ++P->generation - 1;
    P->sweep.clean = false;  // until the backward sweep has been launched as well
    CPG_TRY(sweep_op(ctx, P->precision, P->bl, P->n, P->lrows_d, P->L_rowptr_d, P->L_col_d, P->L_vals, x,
                     MODE_FORWARD, st, err, kind));
    st.gen++;
    CPG_TRY(sweep_op(ctx, P->precision, P->bl, P->n, P->urows_d, P->U_rowptr_d, P->U_col_d, P->U_vals, x,
                     MODE_BACKWARD, st, err, kind));
    P->sweep.clean = true;
    return CPG_OK;
}

cpg_status apply_levels(cpg_ctx *ctx, const cpg_precond *P, double *x, int variant, const double *addv) {
    if (P->kind == CPG_PC_ILU0) {
        const int nl = (int)P->lptr.size() - 1;
        for (int l = 0; l < nl; l++) {
            const int cnt = P->lptr[l + 1] - P->lptr[l];
            // rows without lower blocks pass through the forward sweep unchanged
            CPG_TRY(rows_op_v(ctx, P->precision, P->bl, cnt, P->lrows_d + P->lptr[l], P->L_rowptr_d, P->L_col_d,
                              P->L_vals, x, x, MODE_FORWARD, variant));
        }
    }
    const int nu = (int)P->uptr.size() - 1;
    for (int l = 0; l < nu; l++) {
        const int cnt = P->uptr[l + 1] - P->uptr[l];
        CPG_TRY(rows_op_v(ctx, P->precision, P->bl, cnt, P->urows_d + P->uptr[l], P->U_rowptr_d, P->U_col_d,
                          P->U_vals, x, x, MODE_BACKWARD, variant, addv));
    }
    return CPG_OK;
}

// addv (or null) is added to every row of the backward sweep: the split form
// in a level form (the sync-free ones have the two-launch operator)
cpg_status apply_form(cpg_ctx *ctx, const cpg_precond *P, double *x, int form, const double *addv) {
    if (form == 1) return apply_syncfree(ctx, P, x, 0);
    if (form >= 4) return apply_syncfree(ctx, P, x, form - 3);
    return apply_levels(ctx, P, x, form == 3 ? 2 : 0, addv);
}

// process-wide decisions, so every preconditioner of one kind, block size,
// precision, size class and candidate set takes the same form (and the same
// summation order)
std::mutex g_form_mu;
std::map<int, int> g_form;

// Picks the fastest sweep form on the preconditioner's own rows before its
// first application: each candidate runs twice on a scratch copy of the
// caller's vector, timed with events on the stream, and the fastest is kept
// for every preconditioner of the same class in the process.  The caller's
// vector only ever sees the decided form, so a solve's result does not
// depend on whether it was the one that timed the forms.
cpg_status apply_tuning(cpg_ctx *ctx, const cpg_precond *P, double *x, const double *addv) {
    const size_t N = (size_t)P->n * P->bl;
    // the scratch copy was allocated with the preconditioner, so the first
    // application neither allocates nor frees device memory
    double *tmp = P->tune_tmp;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    bool timed = tmp && cudaEventCreate(&e0) == cudaSuccess && cudaEventCreate(&e1) == cudaSuccess;
    float best_ms[8] = {1e30f, 1e30f, 1e30f, 1e30f, 1e30f, 1e30f, 1e30f, 1e30f};
    bool dropped[8] = {false, false, false, false, false, false, false, false};
    cpg_status st = CPG_OK;
    {
        const TimedLaunches launches(ctx);
        for (int rep = 0; rep < 2 && timed && st == CPG_OK; rep++)
            for (int c = 0; c < P->n_cand && st == CPG_OK; c++) {
                if (dropped[c]) continue;
                float ms = 1e30f;
                if (cudaMemcpyAsync(tmp, x, N * sizeof(double), cudaMemcpyDeviceToDevice, ctx->stream) != cudaSuccess ||
                    cudaEventRecord(e0, ctx->stream) != cudaSuccess) {
                    timed = false;
                    break;
                }
                st = apply_form(ctx, P, tmp, P->cand[c], addv);
                if (st == CPG_OK && cudaEventRecord(e1, ctx->stream) == cudaSuccess &&
                    cudaEventSynchronize(e1) == cudaSuccess && cudaEventElapsedTime(&ms, e0, e1) == cudaSuccess)
                    best_ms[c] = std::min(best_ms[c], ms);
                // a candidate whose bounded wait ran out (e.g. other work held its
                // SMs) is dropped; its status word must not fail the caller's solve
                if (st == CPG_OK && check_sweep_error(ctx, CPG_OK) != CPG_OK) {
                    dropped[c] = true;
                    best_ms[c] = 1e30f;
                }
            }
    }
    (void)cudaGetLastError();
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (st != CPG_OK) return st;
    int best = -1;
    for (int c = 0; c < P->n_cand; c++)
        if (!dropped[c] && best_ms[c] < 1e29f && (best < 0 || best_ms[c] < best_ms[best])) best = c;
    if (!timed || best < 0) {
        // nothing was timed (no scratch memory for the copy, or every
        // candidate gave up): apply the level form this once and decide at a
        // later application rather than record an untimed choice
        return apply_form(ctx, P, x, 2, addv);
    }
    {
        std::lock_guard<std::mutex> lk(g_form_mu);
        auto it = g_form.find(P->form_key);
        if (it == g_form.end()) g_form[P->form_key] = P->cand[best];
        P->sweep_mode = g_form[P->form_key];  // a concurrent first decision wins
    }
    return apply_form(ctx, P, x, P->sweep_mode, addv);
}

// the candidates of a new preconditioner, or its form when already decided;
// true if the environment forces a form
bool choose_form(cpg_precond *P, const char *env) {
    P->sweep_mode = 2;
    if (P->kind != CPG_PC_ILU0) return false;
    if (env && std::strcmp(env, "levels") == 0) return true;
    if (env && std::strcmp(env, "levels_wide") == 0) {
        P->sweep_mode = 3;
        return true;
    }
    if (env && std::strcmp(env, "syncfree") == 0 && P->syncfree) {
        P->sweep_mode = 1;
        return true;
    }
    if (env && std::strcmp(env, "syncfree_direct") == 0 && P->syncfree) {
        P->sweep_mode = 4;
        return true;
    }
    if (env && std::strncmp(env, "form", 4) == 0) {  // form1 .. form6
        const int f = std::atoi(env + 4);
        const bool needs_syncfree = f == 1 || f >= 4;
        if (f >= 1 && f <= 6 && (!needs_syncfree || P->syncfree)) {
            P->sweep_mode = f;
            return true;
        }
    }
    P->n_cand = 0;
    if (P->syncfree) {  // the TMA ring (1) and the widest direct rows (6) never won a size class
        P->cand[P->n_cand++] = 4;
        P->cand[P->n_cand++] = 5;
    }
    P->cand[P->n_cand++] = 2;
    if (rows_tunable(P->bl)) P->cand[P->n_cand++] = 3;
    if (P->n_cand < 2) return false;
    int size_class = 0;
    while ((1 << size_class) < P->n) size_class++;
    // with the candidates: a row too long for the sync-free forms keeps a
    // preconditioner out of them whatever others of its size have decided
    P->form_key = (((P->bl * 2 + (P->precision == CPG_F32)) * 2 + P->syncfree) << 6) | size_class;
    std::lock_guard<std::mutex> lk(g_form_mu);
    auto it = g_form.find(P->form_key);
    P->sweep_mode = it != g_form.end() ? it->second : 0;
    return false;
}

}  // namespace sweep_form

cpg_status precond_apply_raw(cpg_ctx *ctx, const cpg_precond *P, double *x, const double *addv) {
    if (!P || P->kind == CPG_PC_NONE) return CPG_OK;
    if (P->sweep_mode == 0) return sweep_form::apply_tuning(ctx, P, x, addv);
    return sweep_form::apply_form(ctx, P, x, P->sweep_mode, addv);
}

// Split form of P^{-1} A for P = (I + L) D (I + U') factored from A, where
// L = L_A D^{-1} and U' = D^{-1} U_A hold A's strictly lower and upper
// blocks.  Then A = (I + L) D + D U' + E with E_i = A_ii - Ahat_ii, and
//   P^{-1} A x = (I + U')^{-1} [x + D^{-1} (I + L)^{-1} (U_A + E) x],
// so one product reads A's upper blocks and E (split_rows_op), the forward
// sweep runs as usual and the backward sweep adds x to every row.  Per
// Krylov step that streams the upper part of A and E instead of all of A.
//
// The identity holds for the stored factors only up to their rounding:
// L D - L_A, D U' - U_A and E - (A_ii - D_i) are each of order
// eps * cond(D_i) |A|, so the split product is the plain one of a matrix
// perturbed by that much (measured: 0.01 to 0.08 eps * max cond_inf(D_i),
// relative).  A solve takes it only while that stays well below its
// tolerance: SPLIT_ROUNDING * eps * max cond_inf(D_i) <= tol.
constexpr double SPLIT_ROUNDING = 0.25;

bool split_ready(const cpg_precond *P, const cpg_bsr *A) {
    return P && A && P->kind == CPG_PC_ILU0 && P->split_capable && P->split_src == A &&
           P->split_version == A->version && A->precision == CPG_F64 && P->precision == CPG_F64;
}

bool fused_ready(const cpg_precond *P, const cpg_bsr *A) {
    return P && A && P->kind == CPG_PC_ILU0 && P->op_capable && P->split_src == A && P->split_version == A->version;
}

// The two-launch operator differs from the product followed by the sweeps by
// the rounding of the stored L and of z = D^{-1} y, which both carry on either
// side: measured up to 0.013 eps * max cond_inf(D_i) apart (p = 2, 3 Euler and
// advection stage matrices of 500 to 100,000 cells), as far as two sweep forms
// are from each other.  A single product takes it only where that is within
// the accuracy asked for; a Krylov solve needs no such bound, since its
// operator is as accurate either way.
constexpr double FUSED_ROUNDING = 0.02;

bool fused_allowed(const cpg_precond *P, const cpg_bsr *A, double accuracy) {
    return fused_ready(P, A) && P->split_capable && P->pivot_cond > 0.0 && std::isfinite(P->pivot_cond) &&
           FUSED_ROUNDING * DBL_EPSILON * P->pivot_cond <= accuracy;
}

bool split_allowed(const cpg_precond *P, const cpg_bsr *A, double tol) {
    return split_ready(P, A) && P->pivot_cond > 0.0 && std::isfinite(P->pivot_cond) &&
           SPLIT_ROUNDING * DBL_EPSILON * P->pivot_cond <= tol;
}

cpg_status split_apply_prec(cpg_ctx *ctx, const cpg_bsr *A, const cpg_precond *P, const double *x, double *y) {
    if (P->op_capable) return op_apply_prec(ctx, A, P, x, y, true);
    CPG_TRY(split_rows_op(ctx, A, P->U_rowptr_d, P->U_col_d, P->u2a_d, P->E_vals, x, y));
    return precond_apply_raw(ctx, P, y, x);
}

cpg_status check_sweep_error(cpg_ctx *ctx, cpg_status st) {
    if (st != CPG_OK && st != CPG_ERR_NONFINITE && st != CPG_ERR_NOT_CONVERGED) return st;
    int err = 0;
    cudaError_t e = cudaMemcpyAsync(&err, ctx->flag_dev + 2, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "sweep status");
    if (!err) return st;
    e = cudaMemsetAsync(ctx->flag_dev + 2, 0, sizeof(int), ctx->stream);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "sweep status reset");
    return fail(ctx, CPG_ERR_TIMEOUT, "a triangular sweep's bounded wait on a row ran out");
}

// One row of a sync-free sweep (0 TMA ring, 1 polled values, 2 flags) that
// waits for a row nobody publishes: rows 0 and 1 (6x6 blocks), row 1 reads
// row 0, and only row 1 is in the sweep's order.  Returns once it has ended.
static cpg_status sweep_wait_check(cpg_ctx *ctx, int which) {
    const int h_ints[16] = {0, 0, 1, 0, 1, 0, 0, 0, 0, 0, 0, 0, 1, 0, 1, 0};
    int *ibuf = nullptr;
    double *dbuf = nullptr;
    CPG_TRY(dmalloc(ctx, &ibuf, 16));
    cpg_status st = dmalloc(ctx, &dbuf, 36 + 12 + 12);
    if (st == CPG_OK) {
        cudaError_t e = cudaMemsetAsync(dbuf, 0, 48 * sizeof(double), ctx->stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(ibuf, h_ints, sizeof(h_ints), cudaMemcpyHostToDevice, ctx->stream);
        if (e != cudaSuccess) st = cuda_fail(ctx, e, "sweep check setup");
    }
    if (st == CPG_OK) {
        const int *rowptr = ibuf, *col = ibuf + 3, *order = ibuf + 4;
        cpg_precond rows;
        rows.n = 2;
        rows.bl = 6;
        rows.sweep.z = dbuf + 48;  // pending for good
        rows.sweep.claims = ibuf + 8;
        rows.sweep.rows = (int4 *)(ibuf + 12);  // {1, 0, 1, 0}
        rows.sweep.n = 1;
        rows.sweep.flags = ibuf + 5;  // never 1
        rows.sweep.gen = 1;
        st = sweep_workspace(ctx, &rows);
        const int kinds[3] = {0, 1, SWEEP_KIND_FLAGS};
        if (st == CPG_OK)
            st = sweep_op(ctx, CPG_F64, 6, 1, order, rowptr, col, dbuf, dbuf + 36, MODE_FORWARD, rows.sweep,
                          ctx->flag_dev + 2, kinds[which]);
    }
    cudaStreamSynchronize(ctx->stream);
    dfree(ibuf);
    dfree(dbuf);
    return st;
}

}  // namespace cpg

extern "C" {

cpg_status cpg_precond_create(cpg_ctx *ctx, const cpg_bsr *A, int kind, int precision, cpg_precond **out) {
    if (!ctx || !A || !out) return CPG_ERR_INVALID_ARG;
    if (kind != CPG_PC_NONE && kind != CPG_PC_ILU0 && kind != CPG_PC_BJACOBI)
        return fail(ctx, CPG_ERR_INVALID_ARG, "unknown preconditioner kind");
    if (precision != CPG_F64 && precision != CPG_F32) return fail(ctx, CPG_ERR_INVALID_ARG, "precision");
    *out = nullptr;
    cpg_precond *P = new (std::nothrow) cpg_precond();
    if (!P) return fail(ctx, CPG_ERR_OOM, "host allocation");
    P->ctx = ctx;
    P->kind = kind;
    P->precision = precision;
    P->n = A->n_rows;
    P->bl = A->bl;
    if (kind == CPG_PC_NONE) {
        *out = P;
        return CPG_OK;
    }
    const int n = A->n_rows;
    const std::vector<int> &rp = A->rowptr, &cl = A->colidx;
    std::vector<int> diag_a(n, -1), a2l(A->nnzb, -1), a2u(A->nnzb, -1), u2a;
    const bool ilu = kind == CPG_PC_ILU0;
    P->L_rowptr.assign(1, 0);
    P->U_rowptr.assign(1, 0);
    P->L_rowptr.reserve(n + 1);
    P->U_rowptr.reserve(n + 1);
    P->L_col.reserve(A->nnzb / 2);
    P->U_col.reserve(A->nnzb / 2 + n);
    u2a.reserve(A->nnzb / 2 + n);
    for (int i = 0; i < n; i++) {
        for (int k = rp[i]; k < rp[i + 1]; k++) {
            if (cl[k] == i) {
                if (diag_a[i] >= 0) {
                    free_precond(P);
                    delete P;
                    return fail(ctx, CPG_ERR_INVALID_ARG, "row " + std::to_string(i) + " has two diagonal blocks");
                }
                diag_a[i] = k;
            }
            for (int k2 = k + 1; k2 < rp[i + 1] && ilu; k2++)
                if (cl[k2] == cl[k]) {
                    free_precond(P);
                    delete P;
                    return fail(ctx, CPG_ERR_INVALID_ARG, "row " + std::to_string(i) + " repeats a column");
                }
        }
        if (diag_a[i] < 0) {
            free_precond(P);
            delete P;
            return fail(ctx, CPG_ERR_INVALID_ARG, "row " + std::to_string(i) + " has no diagonal block");
        }
        // DU row: D^{-1} first, then upper blocks in A's row order
        P->U_col.push_back(i);
        u2a.push_back(-1);
        if (ilu) {
            for (int k = rp[i]; k < rp[i + 1]; k++) {
                if (cl[k] < i) {
                    a2l[k] = (int)P->L_col.size();
                    P->L_col.push_back(cl[k]);
                } else if (cl[k] > i) {
                    a2u[k] = (int)P->U_col.size();
                    P->U_col.push_back(cl[k]);
                    u2a.push_back(k);
                }
            }
        }
        P->L_rowptr.push_back((int)P->L_col.size());
        P->U_rowptr.push_back((int)P->U_col.size());
    }
    P->nnzL = (int64_t)P->L_col.size();
    P->nnzU = (int64_t)P->U_col.size();
    // factor work lists: for row j, lower neighbours i ascending with the A
    // position of (i, j) (the reference searches row i for column j,
    // Preconditioners.cpp:78-80; structurally symmetric patterns required)
    std::vector<int> lp_i, lp_aji, lp_aij, lp_l, lp_u;
    P->lp_ptr.assign(1, 0);
    P->lp_ptr.reserve(n + 1);
    for (auto *v : {&lp_i, &lp_aji, &lp_aij, &lp_l, &lp_u}) v->reserve(P->nnzL);
    std::vector<std::pair<int, int>> low;  // (i, A index of (j, i))
    for (int j = 0; j < n; j++) {
        low.clear();
        if (ilu)
            for (int k = rp[j]; k < rp[j + 1]; k++)
                if (cl[k] < j) low.push_back({cl[k], k});
        std::sort(low.begin(), low.end());
        for (auto &pr : low) {
            const int i = pr.first;
            int kij = -1;
            for (int k = rp[i]; k < rp[i + 1]; k++)
                if (cl[k] == j) {
                    kij = k;
                    break;
                }
            if (kij < 0) {
                free_precond(P);
                delete P;
                return fail(ctx, CPG_ERR_INVALID_ARG,
                            "block pattern is not structurally symmetric at (" + std::to_string(i) + "," +
                                std::to_string(j) + ")");
            }
            lp_i.push_back(i);
            lp_aji.push_back(pr.second);
            lp_aij.push_back(kij);
            lp_l.push_back(a2l[pr.second]);
            lp_u.push_back(a2u[kij]);
        }
        P->lp_ptr.push_back((int)lp_i.size());
    }
    if (ilu) {
        level_sets(n, rp, cl, P->lptr, P->lrows, P->uptr, P->urows);
    } else {
        P->lptr = {0, n};
        P->uptr = {0, n};
        P->lrows.resize(n);
        for (int i = 0; i < n; i++) P->lrows[i] = i;
        P->urows = P->lrows;
    }
    std::vector<int> dinv_idx(n);
    for (int i = 0; i < n; i++) dinv_idx[i] = precision == CPG_F64 ? P->U_rowptr[i] : i;
    const char *sweep_env = std::getenv("CPG_ILU_SWEEP");
    const bool level_sweeps = sweep_env && std::strcmp(sweep_env, "levels") == 0;
    int longest = 0;
    for (int i = 0; i < n; i++)
        longest = std::max({longest, P->L_rowptr[i + 1] - P->L_rowptr[i], P->U_rowptr[i + 1] - P->U_rowptr[i]});
    P->syncfree = ilu && sweep_supported(P->bl) && !level_sweeps && longest <= SWEEP_MAX_ROW_BLOCKS;
    // the split form of P^{-1} A (FP64 values and factors); CPG_SPLIT_OPERATOR=0 turns it off
    const char *split_env = std::getenv("CPG_SPLIT_OPERATOR");
    P->split_capable = ilu && precision == CPG_F64 && A->precision == CPG_F64 && sweep_supported(P->bl) &&
                       longest <= SWEEP_MAX_ROW_BLOCKS && !(split_env && std::strcmp(split_env, "0") == 0);
    const bool forced = sweep_form::choose_form(P, sweep_env);
    // The two-launch operator is a sync-free form: a level form that the
    // environment asks for turns it off as well.  A level form that the class
    // was timed into does not: the operator was not what was timed, and its
    // bits must not depend on which preconditioner came first.
    int longest_a = 0;
    for (int i = 0; i < n; i++) longest_a = std::max(longest_a, rp[i + 1] - rp[i]);
    P->op_capable = P->syncfree && precision == CPG_F64 && A->precision == CPG_F64 && longest_a <= OP_MAX_ROW_BLOCKS &&
                    !(forced && (P->sweep_mode == 2 || P->sweep_mode == 3));
    cpg_status st = CPG_OK;
    // scratch for timing the sweep forms at the first application (an
    // undecided class only; a vector's worth, freed with the preconditioner)
    if (P->sweep_mode == 0) st = dmalloc(ctx, &P->tune_tmp, (size_t)n * P->bl);
    auto up = [&](int **dst, const std::vector<int> &src) {
        if (st == CPG_OK) st = upload(ctx, dst, src);
    };
    up(&P->lrows_d, P->lrows);
    up(&P->urows_d, P->urows);
    up(&P->L_rowptr_d, P->L_rowptr);
    up(&P->L_col_d, P->L_col);
    up(&P->U_rowptr_d, P->U_rowptr);
    up(&P->U_col_d, P->U_col);
    up(&P->lp_ptr_d, P->lp_ptr);
    up(&P->lp_i_d, lp_i);
    up(&P->lp_aji_d, lp_aji);
    up(&P->lp_aij_d, lp_aij);
    up(&P->lp_l_d, lp_l);
    up(&P->lp_u_d, lp_u);
    up(&P->diag_a_d, diag_a);
    up(&P->dinv_idx_d, dinv_idx);
    if (st == CPG_OK) st = dmalloc(ctx, &P->cond_d, 1);
    if (P->split_capable) {
        up(&P->u2a_d, u2a);
        if (st == CPG_OK) st = dmalloc(ctx, &P->E_vals, (size_t)n * P->bl * P->bl);
    }
    if (P->syncfree && st == CPG_OK) st = sweep_plan_create(ctx, P);
    if (P->op_capable && st == CPG_OK) st = op_plan_create(ctx, P, A);
    const size_t b2 = (size_t)P->bl * P->bl;
    if (st == CPG_OK && P->nnzL) {
        cudaError_t e = cudaMalloc(&P->L_vals, P->nnzL * b2 * P->elem());
        if (e != cudaSuccess) { (void)cudaGetLastError(); P->L_vals = nullptr; st = fail(ctx, CPG_ERR_OOM, "ILU L storage"); }
    }
    if (st == CPG_OK) {
        cudaError_t e = cudaMalloc(&P->U_vals, P->nnzU * b2 * P->elem());
        if (e != cudaSuccess) { (void)cudaGetLastError(); P->U_vals = nullptr; st = fail(ctx, CPG_ERR_OOM, "ILU DU storage"); }
    }
    if (st == CPG_OK && precision == CPG_F32) st = dmalloc(ctx, &P->dinv64, (size_t)n * b2);
    if (st == CPG_OK) st = cpg_precond_refactor(ctx, P, A);
    if (st != CPG_OK) {
        free_precond(P);
        delete P;
        return st;
    }
    *out = P;
    return CPG_OK;
}

cpg_status cpg_precond_refactor(cpg_ctx *ctx, cpg_precond *P, const cpg_bsr *A) {
    if (!ctx || !P || !A) return CPG_ERR_INVALID_ARG;
    if (P->kind == CPG_PC_NONE) return CPG_OK;
    if (A->n_rows != P->n || A->bl != P->bl) return fail(ctx, CPG_ERR_INVALID_ARG, "matrix does not fit preconditioner");
    P->split_src = nullptr;  // until this factorisation has succeeded
    const int init[2] = {0, INT_MAX};
    CPG_CUDA(ctx, cudaMemcpyAsync(ctx->flag_dev, init, sizeof(init), cudaMemcpyHostToDevice, ctx->stream));
    CPG_CUDA(ctx, cudaMemsetAsync(ctx->flag_dev + 6, 0, sizeof(int), ctx->stream));
    if (P->cond_d) CPG_CUDA(ctx, cudaMemsetAsync(P->cond_d, 0, sizeof(unsigned long long), ctx->stream));
    const int nlev = (int)P->lptr.size() - 1;
    for (int l = 0; l < nlev; l++)
        CPG_TRY(factor_level(ctx, P, A, P->lptr[l + 1] - P->lptr[l], P->lrows_d + P->lptr[l]));
    int flag[7];
    unsigned long long cond_bits = 0;
    CPG_CUDA(ctx, cudaMemcpyAsync(flag, ctx->flag_dev, sizeof(flag), cudaMemcpyDeviceToHost, ctx->stream));
    if (P->cond_d)
        CPG_CUDA(ctx, cudaMemcpyAsync(&cond_bits, P->cond_d, sizeof(cond_bits), cudaMemcpyDeviceToHost, ctx->stream));
    CPG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    std::memcpy(&P->pivot_cond, &cond_bits, sizeof(double));
    if (flag[6]) return fail(ctx, CPG_ERR_TIMEOUT, "a tensor-core product of the factorisation did not complete");
    if (flag[0]) return fail(ctx, CPG_ERR_SINGULAR_BLOCK, "singular pivot block at row " + std::to_string(flag[1]));
    if (A->precision == CPG_F64 && P->precision == CPG_F64) {
        P->split_src = A;  // the factors (and E = A_ii - Ahat_ii) are those of these values
        P->split_version = A->version;
    }
    return CPG_OK;
}

cpg_status cpg_precond_apply(cpg_ctx *ctx, const cpg_precond *P, double *x) {
    if (!ctx || !x) return CPG_ERR_INVALID_ARG;
    const cpg_status st = precond_apply_raw(ctx, P, x);
    if (ctx->deferred_checks) return st;
    return check_sweep_error(ctx, st);
}

cpg_status cpg_precond_apply_op(cpg_ctx *ctx, const cpg_precond *P, const cpg_bsr *A, const double *x, double *y,
                                double accuracy) {
    if (!ctx || !P || !A || !x || !y || x == y) return CPG_ERR_INVALID_ARG;
    if (A->n_rows != P->n || A->bl != P->bl) return fail(ctx, CPG_ERR_INVALID_ARG, "matrix does not fit preconditioner");
    cpg_status st;
    if (split_allowed(P, A, accuracy)) {
        st = split_apply_prec(ctx, A, P, x, y);
    } else if (fused_allowed(P, A, accuracy)) {
        st = op_apply_prec(ctx, A, P, x, y, false);
    } else {
        st = bsr_matvec_raw(ctx, A, x, y);
        if (st == CPG_OK) st = precond_apply_raw(ctx, P, y);
    }
    if (ctx->deferred_checks) return st;
    return check_sweep_error(ctx, st);
}

int cpg_precond_split_ready(const cpg_precond *P, const cpg_bsr *A) { return split_ready(P, A) ? 1 : 0; }

double cpg_precond_pivot_cond(const cpg_precond *P) { return P ? P->pivot_cond : 0.0; }

int cpg_precond_sweep_form(const cpg_precond *P) {
    if (!P || P->kind != CPG_PC_ILU0) return 0;
    return P->sweep_mode;
}

cpg_status cpg_debug_decide_sweep_form(const cpg_precond *P, int form) {
    if (!P || P->form_key < 0) return CPG_ERR_INVALID_ARG;
    bool known = form == 0;
    for (int c = 0; c < P->n_cand; c++) known = known || P->cand[c] == form;
    if (!known) return CPG_ERR_INVALID_ARG;
    std::lock_guard<std::mutex> lk(sweep_form::g_form_mu);
    if (form) sweep_form::g_form[P->form_key] = form;
    else sweep_form::g_form.erase(P->form_key);
    return CPG_OK;
}

cpg_status cpg_debug_wait_timeout(cpg_ctx *ctx, int kernel) {
    if (!ctx || kernel < 0 || kernel > 6) return CPG_ERR_INVALID_ARG;
    CPG_TRY(kernel < 3 ? sweep_wait_check(ctx, kernel) : op_wait_check(ctx, kernel >= 5, kernel % 2 == 0));
    if (ctx->deferred_checks) return CPG_OK;
    const cpg_status st = check_sweep_error(ctx, CPG_OK);
    return st == CPG_OK ? fail(ctx, CPG_ERR_INVALID_ARG, "a sweep wait did not report running out") : st;
}

cpg_status cpg_debug_sweep_timeout(cpg_ctx *ctx) {
    if (!ctx) return CPG_ERR_INVALID_ARG;
    cpg_status st = CPG_ERR_TIMEOUT;
    for (int kernel = 0; kernel < 7 && st == CPG_ERR_TIMEOUT; kernel++) st = cpg_debug_wait_timeout(ctx, kernel);
    return st;
}

void cpg_precond_destroy(cpg_precond *P) {
    if (!P) return;
    // cudaFree synchronizes the device; the context may already be gone
    free_precond(P);
    delete P;
}

cpg_status cpg_precond_levels(const cpg_precond *P, int *n_lower, int *lower_ptr, int *lower_rows, int *n_upper,
                              int *upper_ptr, int *upper_rows) {
    if (!P) return CPG_ERR_INVALID_ARG;
    if (n_lower) *n_lower = (int)P->lptr.size() - 1;
    if (n_upper) *n_upper = (int)P->uptr.size() - 1;
    if (lower_ptr) std::memcpy(lower_ptr, P->lptr.data(), sizeof(int) * P->lptr.size());
    if (lower_rows) std::memcpy(lower_rows, P->lrows.data(), sizeof(int) * P->lrows.size());
    if (upper_ptr) std::memcpy(upper_ptr, P->uptr.data(), sizeof(int) * P->uptr.size());
    if (upper_rows) std::memcpy(upper_rows, P->urows.data(), sizeof(int) * P->urows.size());
    return CPG_OK;
}

cpg_status cpg_precond_export(cpg_ctx *ctx, const cpg_precond *P, double *dinv_host, int *l_rowptr, int *l_col,
                              double *l_host, int *u_rowptr, int *u_col, double *u_host) {
    if (!ctx || !P || P->kind == CPG_PC_NONE) return CPG_ERR_INVALID_ARG;
    const size_t b2 = (size_t)P->bl * P->bl;
    std::vector<double> U((size_t)P->nnzU * b2), L((size_t)P->nnzL * b2);
    auto fetch = [&](const void *src, size_t nblk, double *dst) -> cpg_status {
        if (!nblk) return CPG_OK;
        if (P->precision == CPG_F64) {
            CPG_CUDA(ctx, cudaMemcpyAsync(dst, src, nblk * b2 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
            CPG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        } else {
            std::vector<float> f(nblk * b2);
            CPG_CUDA(ctx, cudaMemcpyAsync(f.data(), src, nblk * b2 * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
            CPG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
            for (size_t q = 0; q < f.size(); q++) dst[q] = f[q];
        }
        return CPG_OK;
    };
    CPG_TRY(fetch(P->U_vals, P->nnzU, U.data()));
    CPG_TRY(fetch(P->L_vals, P->nnzL, L.data()));
    // split DU rows into D^{-1} and the strictly upper part
    int nu = 0;
    if (u_rowptr) u_rowptr[0] = 0;
    for (int i = 0; i < P->n; i++) {
        const int k0 = P->U_rowptr[i];
        if (dinv_host) std::memcpy(dinv_host + (size_t)i * b2, U.data() + (size_t)k0 * b2, b2 * sizeof(double));
        for (int k = k0 + 1; k < P->U_rowptr[i + 1]; k++, nu++) {
            if (u_col) u_col[nu] = P->U_col[k];
            if (u_host) std::memcpy(u_host + (size_t)nu * b2, U.data() + (size_t)k * b2, b2 * sizeof(double));
        }
        if (u_rowptr) u_rowptr[i + 1] = nu;
    }
    if (l_rowptr) std::memcpy(l_rowptr, P->L_rowptr.data(), sizeof(int) * P->L_rowptr.size());
    if (l_col && P->nnzL) std::memcpy(l_col, P->L_col.data(), sizeof(int) * P->L_col.size());
    if (l_host && P->nnzL) std::memcpy(l_host, L.data(), sizeof(double) * L.size());
    return CPG_OK;
}

}  // extern "C"
