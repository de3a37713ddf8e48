// The left-preconditioned Krylov operator w = P^{-1} A x in two launches, for
// an FP64 block ILU(0) P = (I + L) D (I + U) factored from A's current values
// (BlockMatrix::gmres's matvec(vi1); pc.solve(vi1), src/BlockMatrix.cpp:121-122).
//
// The reference's BlockILU0 changes only the pivot blocks, so the strictly
// lower factor is L = A_L D^{-1}.  Written with z = D^{-1} y instead of y, the
// forward substitution of y = (I + L)^{-1} A x reads A's own lower blocks,
//   y_j = sum_{k >= j} A_jk x_k + sum_{i < j} A_ji (x_i - z_i),  z_j = D_j^{-1} y_j,
// and the backward one is w_i = z_i - sum_{j > i} U_ij w_j.  One application
// streams A, D^{-1} and U (11 blocks a row on a Voronoi mesh) where the product
// followed by the two sweeps streams A, L, D^{-1} and U (14): the same operator
// with the products of the lower blocks grouped differently, at the same
// rounding (against 80-bit arithmetic on p = 2, 3 Euler stage matrices, cond(D)
// 9e4 to 5e6: 0.95 to 1.07 of the error of the other order).
//
// Both sweeps are sync-free: a CTA claims rows in level order from a counter
// and a row waits for the rows it reads, each thread polling the values that
// it multiplies (poll.cuh).  The forward sweep leaves w pending (which only
// the backward sweep writes), the backward sweep z.
//
// Progress: every CTA takes its rows in claim order and a row only waits on
// rows claimed before it by CTAs that are running, so the earliest unfinished
// row can always proceed.  Every wait is bounded; one that runs out sets *err,
// after which no wait lasts (the solve reports CPG_ERR_TIMEOUT); the sweeps
// still visit every row, so z ends pending again.
//
// Bound by HBM on large meshes and by the level chain on small ones.  100,000
// rows of 40x40 blocks: forward 1,495 us (6.85 TB/s of blocks), backward 610 us
// (6.3 TB/s), against 3,060 us for the product and two sweeps; 18,500 rows in
// nine systems: 289 + 123 us.  GMRES step, 1,009 rows of 24x24: 24 us of 41.
#include <algorithm>
#include <atomic>
#include <vector>

#include "internal.hpp"
#include "poll.cuh"

using namespace cpg;

namespace {

constexpr long long OP_COPY_SPINS = 1LL << 24;                 // mbarrier polls, a backstop only

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Threads of a row: PB threads take one block, IT vector loads of two doubles
// each, so a thread keeps two rows of the block and advances by STEP columns;
// NB blocks are taken side by side where one block would not fill a few warps.
template <int BL>
struct OpShape;
template <> struct OpShape<6> { static constexpr int PB = 18, NB = 5, CTAS = 16; };
template <> struct OpShape<10> { static constexpr int PB = 50, NB = 3, CTAS = 8; };
template <> struct OpShape<24> { static constexpr int PB = 96, NB = 1, CTAS = 10; };
template <> struct OpShape<40> { static constexpr int PB = 160, NB = 1, CTAS = 6; };

template <int BL>
struct Op {
    static constexpr int PB = OpShape<BL>::PB, NB = OpShape<BL>::NB, CTAS = OpShape<BL>::CTAS;
    static constexpr int BL2 = BL * BL, IT = BL2 / (2 * PB), STEP = 2 * PB / BL, G = NB * STEP;
    static constexpr int TPR = (PB * NB + 31) / 32 * 32;
    static_assert(BL2 == 2 * PB * IT && 2 * PB == STEP * BL, "a block is a whole number of passes of whole columns");
    static_assert(TPR >= BL && TPR >= OP_MAX_ROW_BLOCKS, "one thread per row entry and per element of the result");
};

// The rows of a sweep, in claim order, and their blocks: {row, first entry,
// entries that wait for nothing | entries << 16, block of D^{-1}} and per
// entry {column, block}.  Warp 0 fetches the next row's while this one streams.
struct RowSlot {
    int4 m;
    int2 e[OP_MAX_ROW_BLOCKS];
};

// The forward sweep.  SPLIT: the split form's rows t_j = E_j x_j +
// sum_{k > j} A_jk x_k - sum_{i < j} L_ji t_i, with t in z and no product with
// D_j^{-1} (the backward sweep has it).
template <int BL, bool SPLIT>
__global__ void __launch_bounds__(Op<BL>::TPR, Op<BL>::CTAS)
    k_op_forward(int n, const int4 *__restrict__ meta, const int2 *__restrict__ ent, const double *__restrict__ A,
                 const double *__restrict__ DU, const double *__restrict__ E, const double *__restrict__ L,
                 const double *__restrict__ x, double *z, double *w, int *claim, int *other_claim, int *err,
                 const int *skip) {
    if (skip && *skip) return;  // a Krylov solve that has converged
    using S = Op<BL>;
    constexpr int IT = S::IT, STEP = S::STEP, G = S::G, BL2 = S::BL2, PB = S::PB, NB = S::NB;
    constexpr uint32_t D_BYTES = BL2 * sizeof(double);
    __shared__ __align__(128) double sD[SPLIT ? 2 : BL2];  // D_j^{-1}, copied while the row's blocks stream
    __shared__ RowSlot slot[2];
    __shared__ __align__(16) double red[G][BL], red2[SPLIT ? 1 : STEP][BL];
    __shared__ double ys[SPLIT ? 1 : BL];
    __shared__ int s_next;
    __shared__ __align__(8) uint64_t bar;
    const int tid = threadIdx.x;
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (blockIdx.x == 0) *other_claim = 0;
        s_next = atomicAdd(claim, 1);
    }
    __syncthreads();
    int q = s_next;
    if (q >= n) return;
    if (tid < OP_MAX_ROW_BLOCKS) {
        const int4 m = __ldg(meta + q);
        if (tid == 0) slot[0].m = m;
        if (tid < (m.z >> 16)) slot[0].e[tid] = __ldg(ent + m.y + tid);
    }
    __syncthreads();
    const int bs = tid / PB, lt = tid % PB;  // block side by side, place in it
    const bool works = bs < NB;
    const int r0 = (2 * lt) % BL, c0 = (2 * lt) / BL;
    const bool alone = gridDim.x >= (unsigned)n;  // a CTA for every row: nothing to claim ahead
    uint32_t phase = 0;
    for (int cur = 0;; cur ^= 1) {
        const RowSlot &row = slot[cur];
        const int i = row.m.x, nfree = row.m.z & 0xffff, nall = row.m.z >> 16;
        int qn = n;
        if (tid == 0) {
            if constexpr (!SPLIT) {
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(&bar)),
                             "r"(D_BYTES)
                             : "memory");
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                        smem_addr(sD)),
                    "l"(DU + (size_t)row.m.w * BL2), "r"(D_BYTES), "r"(smem_addr(&bar))
                    : "memory");
            }
            if (!alone) qn = atomicAdd(claim, 1);
        }
        // the blocks that wait for others come last; have them in L2 by then
        const double *dep = SPLIT ? L : A;
        if (tid >= S::TPR - 32) {
            const int b = nfree + tid - (S::TPR - 32);
            if (b < nall)
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(dep + (size_t)row.e[b].y * BL2),
                             "r"(D_BYTES)
                             : "memory");
        }
        double acc0 = 0.0, acc1 = 0.0;
        if (works) {
            for (int b = bs; b < nfree; b += NB) {
                const int2 e = row.e[b];
                const double *p = (SPLIT && b == 0 ? E : A) + (size_t)e.y * BL2 + 2 * lt;
                const double *xp = x + (size_t)e.x * BL + c0;
                double2 a[IT];
                double xv[IT];
#pragma unroll
                for (int k = 0; k < IT; k++) a[k] = __ldcs(reinterpret_cast<const double2 *>(p + k * 2 * PB));
#pragma unroll
                for (int k = 0; k < IT; k++) xv[k] = __ldg(xp + k * STEP);
#pragma unroll
                for (int k = 0; k < IT; k++) {
                    acc0 += a[k].x * xv[k];
                    acc1 += a[k].y * xv[k];
                }
            }
        }
        int4 mn = make_int4(0, 0, 0, 0);
        if (tid < 32) {  // the next row, while this one waits
            qn = __shfl_sync(0xffffffffu, qn, 0);
            if (qn < n) mn = __ldg(meta + qn);
        }
        if (works) {
            for (int b = nfree + bs; b < nall; b += NB) {
                const int2 e = row.e[b];
                const double *p = dep + (size_t)e.y * BL2 + 2 * lt;
                const double *xp = x + (size_t)e.x * BL + c0;
                double2 a[IT];
                double xv[IT], zv[IT];
#pragma unroll
                for (int k = 0; k < IT; k++) a[k] = __ldcs(reinterpret_cast<const double2 *>(p + k * 2 * PB));
#pragma unroll
                for (int k = 0; k < IT; k++) xv[k] = SPLIT ? 0.0 : __ldg(xp + k * STEP);
                poll_strided<IT, STEP>(z + (size_t)e.x * BL + c0, zv, err);
#pragma unroll
                for (int k = 0; k < IT; k++) {
                    const double d = xv[k] - zv[k];
                    acc0 += a[k].x * d;
                    acc1 += a[k].y * d;
                }
            }
            *reinterpret_cast<double2 *>(&red[bs * STEP + c0][r0]) = make_double2(acc0, acc1);
        }
        int2 en = make_int2(0, 0);
        if (tid < 32 && tid < (mn.z >> 16)) en = __ldg(ent + mn.y + tid);
        __syncthreads();
        if (tid < BL) {
            double s = 0.0;
#pragma unroll
            for (int g = 0; g < G; g++) s += red[g][tid];
            if constexpr (SPLIT) {
                publish_value(z + (size_t)i * BL + tid, s);
                set_pending(w + (size_t)i * BL + tid);
            } else {
                ys[tid] = s;
            }
        }
        if constexpr (!SPLIT) __syncthreads();
        if (!SPLIT && bs == 0) {  // z_j = D_j^{-1} y_j
            long long spins = 0;
            for (;;) {
                uint32_t ok;
                asm volatile(
                    "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                    : "=r"(ok)
                    : "r"(smem_addr(&bar)), "r"(phase)
                    : "memory");
                if (ok) break;
                // the row's copy is still in flight: reported, then waited for
                // as long again, so that none outlives its CTA
                if (++spins == OP_COPY_SPINS) atomicExch(err, 2);
                if (spins >= 2 * OP_COPY_SPINS) break;
            }
            acc0 = acc1 = 0.0;
#pragma unroll
            for (int k = 0; k < IT; k++) {
                const double2 a = *reinterpret_cast<const double2 *>(sD + 2 * lt + k * 2 * PB);
                const double yv = ys[c0 + k * STEP];
                acc0 += a.x * yv;
                acc1 += a.y * yv;
            }
            *reinterpret_cast<double2 *>(&red2[c0][r0]) = make_double2(acc0, acc1);
        }
        phase ^= 1;
        if (tid < 32) {
            if (tid == 0) {
                slot[cur ^ 1].m = mn;
                s_next = qn;
            }
            if (tid < (mn.z >> 16)) slot[cur ^ 1].e[tid] = en;
        }
        __syncthreads();
        if (!SPLIT && tid < BL) {
            double s = 0.0;
#pragma unroll
            for (int g = 0; g < STEP; g++) s += red2[g][tid];
            publish_value(z + (size_t)i * BL + tid, s);
            // the backward sweep publishes w_i here
            set_pending(w + (size_t)i * BL + tid);
        }
        if (s_next >= n) return;
    }
}

// The backward sweep w_i = z_i - sum_{j > i} U_ij w_j; SPLIT: w_i = x_i +
// D_i^{-1} t_i - sum_{j > i} U_ij w_j.  A row's first entry is D_i^{-1}.
template <int BL, bool SPLIT>
__global__ void __launch_bounds__(Op<BL>::TPR, Op<BL>::CTAS)
    k_op_backward(int n, const int4 *__restrict__ meta, const int2 *__restrict__ ent, const double *__restrict__ DU,
                  const double *__restrict__ x, double *z, double *w, int *claim, int *other_claim, int *err,
                  const int *skip) {
    if (skip && *skip) return;
    using S = Op<BL>;
    constexpr int IT = S::IT, STEP = S::STEP, G = S::G, BL2 = S::BL2, PB = S::PB, NB = S::NB;
    constexpr uint32_t B_BYTES = BL2 * sizeof(double);
    __shared__ RowSlot slot[2];
    __shared__ __align__(16) double red[2][G][BL];
    __shared__ int s_next[2];
    const int tid = threadIdx.x;
    if (tid == 0) {
        if (blockIdx.x == 0) *other_claim = 0;
        s_next[0] = atomicAdd(claim, 1);
    }
    __syncthreads();
    const int q = s_next[0];
    if (q >= n) return;
    if (tid < OP_MAX_ROW_BLOCKS) {
        const int4 m = __ldg(meta + q);
        if (tid == 0) slot[0].m = m;
        if (tid < (m.z >> 16)) slot[0].e[tid] = __ldg(ent + m.y + tid);
    }
    __syncthreads();
    const int bs = tid / PB, lt = tid % PB;
    const bool works = bs < NB;
    const int r0 = (2 * lt) % BL, c0 = (2 * lt) / BL;
    const bool alone = gridDim.x >= (unsigned)n;
    for (int cur = 0;; cur ^= 1) {
        const RowSlot &row = slot[cur];
        const int i = row.m.x, nall = row.m.z >> 16;
        int qn = n;
        if (tid == 0 && !alone) qn = atomicAdd(claim, 1);
        if (tid >= S::TPR - 32) {
            const int b = 2 + tid - (S::TPR - 32);  // every block but those that are loaded at once
            if (b < nall)
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(DU + (size_t)row.e[b].y * BL2),
                             "r"(B_BYTES)
                             : "memory");
        }
        double zi = 0.0;
        if (tid < BL) zi = SPLIT ? __ldg(x + (size_t)i * BL + tid) : __ldcg(z + (size_t)i * BL + tid);
        double acc0 = 0.0, acc1 = 0.0;
        if (works) {
            if (SPLIT && bs == 0) {
                const double *p = DU + (size_t)row.e[0].y * BL2 + 2 * lt;
                const double *zp = z + (size_t)i * BL + c0;
#pragma unroll
                for (int k = 0; k < IT; k++) {
                    const double2 a = __ldcs(reinterpret_cast<const double2 *>(p + k * 2 * PB));
                    const double zv = __ldcg(zp + k * STEP);
                    acc0 += a.x * zv;
                    acc1 += a.y * zv;
                }
            }
            for (int b = 1 + bs; b < nall; b += NB) {
                const int2 e = row.e[b];
                const double *p = DU + (size_t)e.y * BL2 + 2 * lt;
                double2 a[IT];
                double wv[IT];
#pragma unroll
                for (int k = 0; k < IT; k++) a[k] = __ldcs(reinterpret_cast<const double2 *>(p + k * 2 * PB));
                poll_strided<IT, STEP>(w + (size_t)e.x * BL + c0, wv, err);
#pragma unroll
                for (int k = 0; k < IT; k++) {
                    acc0 -= a[k].x * wv[k];
                    acc1 -= a[k].y * wv[k];
                }
            }
            *reinterpret_cast<double2 *>(&red[cur][bs * STEP + c0][r0]) = make_double2(acc0, acc1);
        }
        if (tid < 32) {
            qn = __shfl_sync(0xffffffffu, qn, 0);
            if (tid == 0) s_next[cur ^ 1] = qn;
            if (qn < n) {
                const int4 m = __ldg(meta + qn);
                if (tid == 0) slot[cur ^ 1].m = m;
                if (tid < (m.z >> 16)) slot[cur ^ 1].e[tid] = __ldg(ent + m.y + tid);
            }
        }
        // one barrier a row: this row's sums are read before the next row's
        // barrier, and their buffer is written again only after it
        __syncthreads();
        if (tid < BL) {
            double s = 0.0;
#pragma unroll
            for (int g = 0; g < G; g++) s += red[cur][g][tid];
            publish_value(w + (size_t)i * BL + tid, zi + s);
            set_pending(z + (size_t)i * BL + tid);
        }
        if (s_next[cur ^ 1] >= n) return;
    }
}

__global__ void k_fill_pending(int64_t n, unsigned long long *z) {
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x)
        z[q] = PENDING;
}

// {row, first block, blocks, 0} in the claim orders of the two sweeps
__global__ void k_sweep_rows(int n, const int *__restrict__ lrows, const int *__restrict__ urows,
                             const int *__restrict__ L_rowptr, const int *__restrict__ U_rowptr, int4 *rows) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const int f = lrows[q], b = urows[q];
    rows[q] = make_int4(f, L_rowptr[f], L_rowptr[f + 1] - L_rowptr[f], 0);
    rows[n + q] = make_int4(b, U_rowptr[b], U_rowptr[b + 1] - U_rowptr[b], 0);
}
// place of every row in the claim orders of the two sweeps
__global__ void k_places(int n, const int *__restrict__ lrows, const int *__restrict__ urows, int *lpos, int *upos) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    lpos[lrows[q]] = q;
    upos[urows[q]] = q;
}
// e into [first, first + count), ordered by the columns' places
__device__ __forceinline__ void insert_entry(int2 *first, int count, int2 e, const int *pos) {
    int2 *at = first + count;
    for (; at > first && pos[at[-1].x] > pos[e.x]; at--) *at = at[-1];
    *at = e;
}
// A thread per claim-order place q of both sweeps.  Entries lie where the
// row's blocks lie in A (forward) and DU (backward); L and DU rows hold A's
// lower and upper blocks in A's row order.
__global__ void k_op_plan(int n, const int *__restrict__ lrows, const int *__restrict__ urows, const int *lpos,
                          const int *upos, const int *__restrict__ rowptr, const int *__restrict__ col,
                          const int *__restrict__ L_rowptr, const int *__restrict__ U_rowptr, int4 *fmeta, int2 *fent,
                          int2 *sent, int4 *bmeta, int2 *bent) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    {
        const int i = lrows[q], k0 = rowptr[i], k1 = rowptr[i + 1];
        int nfree = 1;
        for (int k = k0; k < k1; k++) {
            if (col[k] == i) fent[k0] = make_int2(i, k);
            else if (col[k] > i) fent[k0 + nfree++] = make_int2(col[k], k);
        }
        int nall = nfree;
        for (int k = k0; k < k1; k++)
            if (col[k] < i) insert_entry(fent + k0 + nfree, nall++ - nfree, make_int2(col[k], k), lpos);
        fmeta[q] = make_int4(i, k0, nfree | nall << 16, U_rowptr[i]);
        if (sent) {  // the split form's rows: E, A's upper blocks and L
            sent[k0] = make_int2(i, i);
            for (int e = 1; e < nfree; e++) sent[k0 + e] = fent[k0 + e];
            int l = L_rowptr[i], count = 0;
            for (int k = k0; k < k1; k++)
                if (col[k] < i) insert_entry(sent + k0 + nfree, count++, make_int2(col[k], l++), lpos);
        }
    }
    {
        const int i = urows[q], u0 = U_rowptr[i];
        int u = u0, count = 0;
        bent[u0] = make_int2(i, u0);
        for (int k = rowptr[i]; k < rowptr[i + 1]; k++)
            if (col[k] > i) insert_entry(bent + u0 + 1, count++, make_int2(col[k], ++u), upos);
        bmeta[q] = make_int4(i, u0, 1 | (count + 1) << 16, 0);
    }
}

// CTAs that share an SM, per device and kernel, computed once
template <class K>
cpg_status ctas_per_sm(cpg_ctx *ctx, K kernel, int threads, std::atomic<int> *known, int *out) {
    const bool cacheable = ctx->device >= 0 && ctx->device < 64;
    int occ = cacheable ? known[ctx->device].load() : 0;
    if (!occ) {
        CPG_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, 0));
        occ = std::max(1, occ);
        if (cacheable) known[ctx->device].store(occ);
    }
    *out = occ;
    return CPG_OK;
}

template <int BL, bool SPLIT>
cpg_status launch_op(cpg_ctx *ctx, const cpg_bsr *A, const cpg_precond *P, const double *x, double *y) {
    static std::atomic<int> fwd_known[64], bwd_known[64];
    int fwd = 0, bwd = 0;
    CPG_TRY(ctas_per_sm(ctx, k_op_forward<BL, SPLIT>, Op<BL>::TPR, fwd_known, &fwd));
    CPG_TRY(ctas_per_sm(ctx, k_op_backward<BL, SPLIT>, Op<BL>::TPR, bwd_known, &bwd));
    const cpg_op_plan &pl = P->op;
    if (!P->sweep.clean) CPG_TRY(sweep_workspace(ctx, P));  // a launch failed half way
    int *err = ctx->flag_dev + 2;
    const int n = P->n;
    const double *DU = (const double *)P->U_vals;
    P->sweep.clean = false;  // until the backward sweep has been launched as well
    k_op_forward<BL, SPLIT><<<std::min(n, fwd * ctx->num_sms), Op<BL>::TPR, 0, ctx->stream>>>(
        n, pl.fmeta, SPLIT ? pl.sent : pl.fent, (const double *)A->vals, DU, P->E_vals, (const double *)P->L_vals, x,
        P->sweep.z, y, P->sweep.claims, P->sweep.claims + 1, err, ctx->skip_dev);
    CPG_TRY(launched(ctx, "operator forward sweep"));
    k_op_backward<BL, SPLIT><<<std::min(n, bwd * ctx->num_sms), Op<BL>::TPR, 0, ctx->stream>>>(
        n, pl.bmeta, pl.bent, DU, x, P->sweep.z, y, P->sweep.claims + 1, P->sweep.claims, err, ctx->skip_dev);
    CPG_TRY(launched(ctx, "operator backward sweep"));
    P->sweep.clean = true;
    return CPG_OK;
}

}  // namespace

namespace cpg {

cpg_status sweep_plan_create(cpg_ctx *ctx, cpg_precond *P) {
    const size_t n = P->n, N = n * P->bl;
    // the rows in claim order, z, the claims and the ring's flags
    CPG_TRY(dmalloc(ctx, &P->sweep.rows, 2 * n + (N + 1) / 2 + (n + 5) / 4));
    P->sweep.n = P->n;
    P->sweep.z = (double *)(P->sweep.rows + 2 * n);
    P->sweep.claims = (int *)(P->sweep.z + N);
    P->row_flags_d = P->sweep.claims + 2;
    CPG_CUDA(ctx, cudaMemsetAsync(P->row_flags_d, 0, sizeof(int) * n, ctx->stream));
    k_sweep_rows<<<(int)((n + 127) / 128), 128, 0, ctx->stream>>>(P->n, P->lrows_d, P->urows_d, P->L_rowptr_d,
                                                                 P->U_rowptr_d, P->sweep.rows);
    CPG_TRY(launched(ctx, "sweep plan kernel"));
    return sweep_workspace(ctx, P);
}

// z pending and the counters zero, as the forward sweeps expect them
cpg_status sweep_workspace(cpg_ctx *ctx, const cpg_precond *P) {
    const int64_t N = (int64_t)P->n * P->bl;
    CPG_CUDA(ctx, cudaMemsetAsync(P->sweep.claims, 0, 2 * sizeof(int), ctx->stream));
    k_fill_pending<<<(int)std::min<int64_t>((N + 255) / 256, (int64_t)ctx->num_sms * 16), 256, 0, ctx->stream>>>(
        N, reinterpret_cast<unsigned long long *>(P->sweep.z));
    CPG_TRY(launched(ctx, "sweep workspace kernel"));
    P->sweep.clean = true;
    return CPG_OK;
}

// The plan, from the patterns on the device.  A row's own block comes first,
// the entries that wait for others come last, by their place in claim order.
cpg_status op_plan_create(cpg_ctx *ctx, cpg_precond *P, const cpg_bsr *A) {
    const size_t n = P->n, nnz = A->nnzb, nu = P->nnzU, ns = P->split_capable ? nnz : 0;
    // one allocation: the rows of both sweeps, their entries, and the rows'
    // places in claim order
    const size_t ents_at = 2 * n * sizeof(int4), pos_at = ents_at + (nnz + ns + nu) * sizeof(int2);
    CPG_TRY(dmalloc(ctx, &P->op.base, pos_at + 2 * n * sizeof(int)));
    char *d = P->op.base;
    P->op.fmeta = (int4 *)d;
    P->op.bmeta = P->op.fmeta + n;
    P->op.fent = (int2 *)(d + ents_at);
    P->op.sent = P->op.fent + nnz;
    P->op.bent = P->op.sent + ns;
    int *pos = (int *)(d + pos_at);
    const int grid = (int)((n + 127) / 128);
    k_places<<<grid, 128, 0, ctx->stream>>>((int)n, P->lrows_d, P->urows_d, pos, pos + n);
    CPG_TRY(launched(ctx, "operator plan kernel"));
    k_op_plan<<<grid, 128, 0, ctx->stream>>>((int)n, P->lrows_d, P->urows_d, pos, pos + n, A->rowptr_d, A->colidx_d,
                                            P->L_rowptr_d, P->U_rowptr_d, P->op.fmeta, P->op.fent,
                                            ns ? P->op.sent : nullptr, P->op.bmeta, P->op.bent);
    return launched(ctx, "operator plan kernel");
}

// One row of the forward or the backward kernel that waits for a row nobody
// publishes (6x6 blocks, rows 0 and 1, one of them in the plan), and the
// other kernel on a row that waits for nothing.  Returns once both have ended.
cpg_status op_wait_check(cpg_ctx *ctx, bool split, bool backward) {
    constexpr int B2 = 36;
    // claims, padding | rows of both sweeps | their entries
    const int4 one = make_int4(backward ? 0 : 1, 0, 1 | 1 << 16, 0), two = make_int4(one.x, 0, 1 | 2 << 16, 0);
    const int4 h[5] = {make_int4(0, 0, 0, 0), backward ? one : two, backward ? two : one,
                       make_int4(one.x, one.x, 1 - one.x, 1 - one.x), make_int4(one.x, one.x, 1 - one.x, 1 - one.x)};
    int4 *meta = nullptr;
    double *buf = nullptr;
    CPG_TRY(dmalloc(ctx, &meta, 5));
    cpg_status st = dmalloc(ctx, &buf, 2 * B2 + 12 + 24);
    if (st == CPG_OK) {
        cudaError_t e = cudaMemcpyAsync(meta, h, sizeof(h), cudaMemcpyHostToDevice, ctx->stream);
        if (e == cudaSuccess) e = cudaMemsetAsync(buf, 0, (2 * B2 + 12) * sizeof(double), ctx->stream);
        if (e != cudaSuccess) st = cuda_fail(ctx, e, "operator check setup");
    }
    if (st == CPG_OK) {
        cpg_bsr A;
        cpg_precond P;
        A.vals = P.U_vals = P.L_vals = P.E_vals = buf;  // two zero blocks
        P.n = 2;
        P.bl = 12;  // z and w pending
        P.sweep.claims = (int *)meta;
        P.sweep.z = buf + 2 * B2 + 12;
        P.op.fmeta = meta + 1;
        P.op.bmeta = meta + 2;
        P.op.fent = P.op.sent = (int2 *)(meta + 3);
        P.op.bent = (int2 *)(meta + 4);
        st = sweep_workspace(ctx, &P);
        P.n = 1;
        P.bl = 6;
        const double *x = buf + 2 * B2;
        double *w = P.sweep.z + 12;
        if (st == CPG_OK) st = op_apply_prec(ctx, &A, &P, x, w, split);
    }
    cudaStreamSynchronize(ctx->stream);
    dfree(meta);
    dfree(buf);
    return st;
}

void op_plan_free(cpg_precond *P) { dfree(P->op.base); }

// y = P^{-1} A x; split: in the split form (the caller checked that it may)
cpg_status op_apply_prec(cpg_ctx *ctx, const cpg_bsr *A, const cpg_precond *P, const double *x, double *y,
                         bool split) {
#define CPG_OP(BLV) \
    case BLV: return split ? launch_op<BLV, true>(ctx, A, P, x, y) : launch_op<BLV, false>(ctx, A, P, x, y)
    switch (P->bl) {
        CPG_OP(6);
        CPG_OP(10);
        CPG_OP(24);
        CPG_OP(40);
        default: return fail(ctx, CPG_ERR_UNSUPPORTED, "block size of the two-launch operator");
    }
#undef CPG_OP
}

}  // namespace cpg
