// Krylov solvers and vector kernels: restarted GMRES with classical
// Gram-Schmidt (BlockMatrix::gmres, src/BlockMatrix.cpp:79-163), its flexible
// right-preconditioned variant (FGMRES), both also for a batch of independent
// systems, damped block Jacobi (BlockMatrix::jacobi, :51-77), and MeshFn
// arithmetic.
//
// The Krylov basis V lives on the device, column i at V + i*N.  One Arnoldi
// step is: the operator, h = V^T w (multi-dot), and w -= V h fused with |w|
// and the Givens update of the least-squares problem, all on the device; the
// host reads the systems' state once per restart cycle.  Reductions use a
// fixed grid and a fixed combination order, so results are reproducible run
// to run.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "internal.hpp"

using namespace cpg;

namespace {

constexpr int RED = 256;   // CTAs of a reduction (fixed for determinism)
constexpr int RT = 256;    // threads per reduction CTA

__device__ __forceinline__ double block_sum(double v, double *sh) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) sh[w] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int q = 0; q < (int)(blockDim.x >> 5); q++) s += sh[q];
    __syncthreads();
    return s;
}

// partial[l*RED + cta] = sum over this CTA's slice of V_l . w
__global__ void __launch_bounds__(RT) k_mdot(int64_t N, const double *__restrict__ V, const double *__restrict__ w,
                                             double *__restrict__ part) {
    __shared__ double sh[RT / 32];
    const int l = blockIdx.y;
    const double *v = V + (size_t)l * N;
    double s = 0.0;
    for (int64_t q = (int64_t)blockIdx.x * RT + threadIdx.x; q < N; q += (int64_t)RED * RT) s += v[q] * w[q];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) part[(size_t)l * RED + blockIdx.x] = s;
}
// out[l] = sum_cta partial[l*RED + cta]
__global__ void k_reduce_parts(int nv, const double *__restrict__ part, double *__restrict__ out) {
    const int l = blockIdx.x;
    __shared__ double sh[RT / 32];
    double s = 0.0;
    for (int q = threadIdx.x; q < RED; q += blockDim.x) s += part[(size_t)l * RED + q];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) out[l] = s;
}
// partial sums of |x|^2
__global__ void __launch_bounds__(RT) k_sumsq(int64_t N, const double *__restrict__ x, double *__restrict__ part) {
    __shared__ double sh[RT / 32];
    double s = 0.0;
    for (int64_t q = (int64_t)blockIdx.x * RT + threadIdx.x; q < N; q += (int64_t)RED * RT) s += x[q] * x[q];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}
// out[0] = sqrt(sum parts) ; out[1] = 1 / out[0]
__global__ void k_norm_final(const double *__restrict__ part, double *__restrict__ out) {
    __shared__ double sh[RT / 32];
    double s = 0.0;
    for (int q = threadIdx.x; q < RED; q += blockDim.x) s += part[q];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) {
        const double nr = sqrt(s);
        out[0] = nr;
        out[1] = 1. / nr;
    }
}
__global__ void k_axpby(int64_t N, double a, const double *__restrict__ x, double b, double *__restrict__ y) {
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < N; q += (int64_t)gridDim.x * blockDim.x)
        y[q] = a * x[q] + b * y[q];
}
__global__ void k_copy(int64_t N, const double *__restrict__ x, double *__restrict__ y, const int *skip) {
    if (skip && *skip) return;  // a Krylov solve that has converged
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < N; q += (int64_t)gridDim.x * blockDim.x)
        y[q] = x[q];
}
__global__ void k_fill(int64_t N, double v, double *__restrict__ y) {
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < N; q += (int64_t)gridDim.x * blockDim.x)
        y[q] = v;
}
// Jacobi update x = (omega*Dinvb + x) - omega*t
__global__ void k_jacobi_update(int64_t N, double omega, const double *__restrict__ dinvb,
                                const double *__restrict__ t, double *__restrict__ x) {
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < N; q += (int64_t)gridDim.x * blockDim.x)
        x[q] = (omega * dinvb[q] + x[q]) - omega * t[q];
}

int grid_for(cpg_ctx *ctx, int64_t N) {
    const int64_t g = (N + 255) / 256;
    return (int)std::min<int64_t>(g, (int64_t)ctx->num_sms * 16);
}

// Krylov workspace from the context (grow-only)
cpg_status kws(cpg_ctx *ctx, size_t n, double **out) {
    if (n > ctx->kws_cap) {
        if (ctx->kws) {
            CPG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
            cudaFree(ctx->kws);
            ctx->kws = nullptr;
            ctx->kws_cap = 0;
        }
        CPG_TRY(dmalloc(ctx, &ctx->kws, n));
        ctx->kws_cap = n;
    }
    *out = ctx->kws;
    return CPG_OK;
}

// device norm; result (norm, 1/norm) at out_dev[0..1]
cpg_status norm_dev(cpg_ctx *ctx, int64_t N, const double *x, double *part, double *out_dev) {
    k_sumsq<<<RED, RT, 0, ctx->stream>>>(N, x, part);
    CPG_TRY(launched(ctx, "sumsq kernel"));
    k_norm_final<<<1, RT, 0, ctx->stream>>>(part, out_dev);
    return launched(ctx, "norm kernel");
}

cpg_status read_host(cpg_ctx *ctx, const double *dev, int n, double *host) {
    double *hp;
    CPG_TRY(pinned(ctx, n, &hp));
    CPG_CUDA(ctx, cudaMemcpyAsync(hp, dev, n * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    CPG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    std::memcpy(host, hp, n * sizeof(double));
    return CPG_OK;
}

}  // namespace

namespace cpg {

cpg_status vec_axpby(cpg_ctx *ctx, int64_t n, double a, const double *x, double b, double *y) {
    if (n <= 0) return CPG_OK;
    k_axpby<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(n, a, x, b, y);
    return launched(ctx, "axpby kernel");
}
cpg_status vec_copy(cpg_ctx *ctx, int64_t n, const double *x, double *y) {
    if (n <= 0) return CPG_OK;
    k_copy<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(n, x, y, ctx->skip_dev);
    return launched(ctx, "copy kernel");
}
cpg_status vec_fill(cpg_ctx *ctx, int64_t n, double v, double *y) {
    if (n <= 0) return CPG_OK;
    k_fill<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(n, v, y);
    return launched(ctx, "fill kernel");
}
cpg_status vec_dot(cpg_ctx *ctx, int64_t n, const double *x, const double *y, double *out_host) {
    double *part;
    CPG_TRY(scratch(ctx, RED + 8, &part));
    k_mdot<<<dim3(RED, 1), RT, 0, ctx->stream>>>(n, x, y, part);
    CPG_TRY(launched(ctx, "dot kernel"));
    k_reduce_parts<<<1, RT, 0, ctx->stream>>>(1, part, part + RED);
    CPG_TRY(launched(ctx, "dot reduce kernel"));
    return read_host(ctx, part + RED, 1, out_host);
}

}  // namespace cpg

// BSR operator / preconditioner pair
struct KrylovOp : LinOp {
    const cpg_bsr *A;
    const cpg_precond *P;
    bool split;  // P^{-1} A in split form (an FP64 ILU(0) of A's current values, rounding well below tol)
    bool fused;  // or in two launches that share A's lower blocks (the same, at the plain product's rounding)
    KrylovOp(const cpg_bsr *a, const cpg_precond *p, double tol)
        : A(a), P(p), split(split_allowed(p, a, tol)), fused(!split && fused_ready(p, a)) {}
    cpg_status apply(cpg_ctx *ctx, const double *x, double *y) const override { return bsr_matvec_raw(ctx, A, x, y); }
    cpg_status prec(cpg_ctx *ctx, double *x) const override { return precond_apply_raw(ctx, P, x); }
    cpg_status apply_prec(cpg_ctx *ctx, const double *x, double *y) const override {
        if (split) return split_apply_prec(ctx, A, P, x, y);
        if (fused) return op_apply_prec(ctx, A, P, x, y, false);
        return LinOp::apply_prec(ctx, x, y);
    }
};

namespace {
// ---------------------------------------------------------------------------
// Segmented GMRES: K independent systems stacked along the vector (a block
// diagonal operator, segment k = dofs [off[k], off[k+1])), each with its own
// Krylov scalars.  One Arnoldi step is the operator and two launches: the dot
// products (k_seg_dots), and the update of w fused with its norm, the Givens
// rotation of the new Hessenberg column and the stopping test (k_seg_update).
// The last CTA of a system to finish a launch combines the partial sums, so a
// reduction and what depends on it need no launch of their own; six launches
// a step before, about 28 us of a 110 us step at 24,000 dofs.
//
// The basis is kept as the vectors w_l before normalisation and their factors
// s_l = 1 / |w_l| (v_l = s_l w_l): the operator is linear, so the factors go
// into the coefficients and no pass over a vector is spent on scaling it.
//
// Every reduction runs on a grid that depends on its own system's length
// only, so a system's result does not depend on what else is batched with
// it.  Once every system has converged, a device word makes the remaining
// launches of the cycle return at once; the host enqueues a whole restart
// cycle and reads the systems' state once per cycle.  The iteration is the
// reference's (BlockMatrix.cpp:79-163).
// ---------------------------------------------------------------------------

struct Seg {
    const int64_t *off;  // K + 1 dof offsets
    int K;
    int ctas;            // most CTAs of a segment's reductions (the stride of the partial sums)
};
__device__ __forceinline__ bool skipped(const int *done) { return done && *done; }

// A reduction over a segment takes its dofs in tiles, which its CTAs stride
// over.  At most SEG_CTAS CTAs (four an SM, one wave) take part, `groups` of
// them on the same tiles: a CTA's set-up and its share of the combination cost
// as much as two tiles, so one tile a CTA took twice the time at 10^6 dofs.
constexpr int SEG_CTAS = 592;
__host__ __device__ __forceinline__ int seg_ctas(int64_t len, int tile, int groups) {
    const int64_t c = (len + tile - 1) / tile, most = SEG_CTAS / groups;
    return (int)(c < 1 ? 1 : (c > most ? most : c));
}
struct Slice {
    int64_t lo, hi, step;  // this thread's first dof of each tile, the segment's end, the tiles' distance
    int ctas;              // CTAs that share the segment; this one is one of them if on
    bool on;
};
__device__ __forceinline__ Slice slice_of(const Seg &sg, int seg, int tile, int groups) {
    Slice s;
    s.hi = sg.off[seg + 1];
    s.ctas = seg_ctas(s.hi - sg.off[seg], tile, groups);
    s.on = (int)blockIdx.x < s.ctas;
    s.lo = sg.off[seg] + (int64_t)blockIdx.x * tile + threadIdx.x;
    s.step = (int64_t)s.ctas * tile;
    return s;
}
constexpr int PER = 4, DOT_TILE = PER * RT;  // dofs of a tile per thread in the dot products
constexpr int UPD_TILE = 2 * RT;             // tile of the update and of the norms
// whether this CTA is the last of `total` to come here, its stores of before
// visible to the one that is; the counter is left at zero
__device__ __forceinline__ bool last_cta(int *ticket, int total) {
    __shared__ int last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(ticket, 1) == total - 1;
        if (last) *ticket = 0;
        __threadfence();
    }
    __syncthreads();
    return last != 0;
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

constexpr int DOTS = 4, DOT_GROUPS = 16;  // dot products of a CTA; groups of them at the longest restart (62)

// Krylov scalars of the K systems (device)
struct KState {
    double *hcol;   // K x HS: h column of the step, then |w|
    double *sc;     // K x HS: factors s_l of the basis vectors
    double *H;      // K x HP: packed upper triangle (Givens-rotated Hessenberg)
    double *c, *s;  // K x m
    double *y;      // K x (m+1)
    double *cy;     // K x (m+1): solution-update coefficients
    double *nrm2b;  // K x 2: |P^{-1} b| (or |b|), residual estimate
    int *active;    // K: still iterating in this cycle
    int *nsteps;    // K: Arnoldi steps taken in this cycle
    int *finished;  // K: converged (stops for good)
    int *its;       // K: iterations as the reference counts them
    int *ticket;    // K x DOT_GROUPS + 1: CTAs that have finished a launch, per system (and group of dot
                    // products); systems
    int *n_active;  // systems still iterating
    int *done;      // 1: no system active
    int *x_zero;    // 1: the initial guess is the zero vector
    int *status;    // [0] a non-finite quantity (bit 0), [1] the sweeps' status word
    int HS, HP, m;
};

// the power of two below s (1 for zero, subnormal or non-finite s): scaling by it is exact
__device__ __forceinline__ double pow2_below(double s) {
    const unsigned long long e = (unsigned long long)__double_as_longlong(s) & 0x7ff0000000000000ULL;
    return e == 0 || e == 0x7ff0000000000000ULL ? 1.0 : __longlong_as_double((long long)e);
}

// h_l = v_l . w for the step's vectors l = 0..i, four of them per CTA (w is
// read once for the four; w has the factor s_i of the vector the operator was
// applied to, whose power of two is taken out of w first: w_l and w = A w_i
// both carry |w_i|, whose square would leave the exponent range long before
// |w_i| does).  HBM-bound: the vectors, and w a quarter as often.  A thread's
// 20 loads of a tile are independent, and each group of four has a last CTA
// of its own, so that the final sums run side by side.
__global__ void __launch_bounds__(RT, 4) k_seg_dots(Seg sg, const double *__restrict__ V, int64_t N,
                                                    const double *__restrict__ w, double *__restrict__ part, KState st,
                                                    int i) {
    if (skipped(st.done)) return;
    const int seg = blockIdx.z;
    if (!st.active[seg]) return;
    const Slice sl = slice_of(sg, seg, DOT_TILE, gridDim.y);
    if (!sl.on) return;
    __shared__ double sh[DOTS][RT / 32];
    const int l0 = blockIdx.y * DOTS, nl = min(DOTS, i + 1 - l0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const double *v[DOTS], *sc = st.sc + (size_t)seg * st.HS;
    const double si = sc[i], p2 = pow2_below(si);
    double acc[DOTS];
#pragma unroll
    for (int k = 0; k < DOTS; k++) {
        v[k] = V + (size_t)(l0 + (k < nl ? k : 0)) * N;
        acc[k] = 0.0;
    }
    for (int64_t q = sl.lo; q - threadIdx.x < sl.hi; q += sl.step) {
        double wq[PER], vq[DOTS][PER];
#pragma unroll
        for (int e = 0; e < PER; e++) {
            const bool in = q + e * RT < sl.hi;
            wq[e] = in ? __ldg(w + q + e * RT) * p2 : 0.0;
#pragma unroll
            for (int k = 0; k < DOTS; k++) vq[k][e] = in ? __ldg(v[k] + q + e * RT) : 0.0;
        }
#pragma unroll
        for (int e = 0; e < PER; e++)
#pragma unroll
            for (int k = 0; k < DOTS; k++) acc[k] += vq[k][e] * wq[e];
    }
#pragma unroll
    for (int k = 0; k < DOTS; k++) {
        acc[k] = warp_sum(acc[k]);
        if (lane == 0) sh[k][warp] = acc[k];
    }
    __syncthreads();
    if ((int)threadIdx.x < nl) {
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < RT / 32; q++) s += sh[threadIdx.x][q];
        part[((size_t)(l0 + threadIdx.x) * sg.K + seg) * sg.ctas + blockIdx.x] = s;
    }
    if (!last_cta(st.ticket + seg * DOT_GROUPS + blockIdx.y, sl.ctas)) return;
    constexpr int SHARE = RT / DOTS;  // threads that sum one dot product's partials
    const int k = threadIdx.x / SHARE, l = l0 + k;
    double s = 0.0;
    if (k < nl)
        for (int q = threadIdx.x % SHARE; q < sl.ctas; q += SHARE)
            s += __ldcg(part + ((size_t)l * sg.K + seg) * sg.ctas + q);
    s = warp_sum(s);
    if (lane == 0) sh[0][warp] = s;
    __syncthreads();
    if (k < nl && threadIdx.x % SHARE == 0) {
        double t = 0.0;
#pragma unroll
        for (int q = 0; q < SHARE / 32; q++) t += sh[0][warp + q];
        st.hcol[(size_t)seg * st.HS + l] = t * sc[l] * (si / p2);
    }
}

// sum of a CTA's values, then of the segment's CTAs: true on the last CTA,
// with the segment's sum in *total on every thread
__device__ __forceinline__ bool seg_total(double v, const Slice &sl, const Seg &sg, int seg, double *part, int *ticket,
                                          double *total) {
    __shared__ double sh[RT / 32], tot;
    const double s = block_sum(v, sh);
    if (threadIdx.x == 0) part[(size_t)seg * sg.ctas + blockIdx.x] = s;
    if (!last_cta(ticket + seg * DOT_GROUPS, sl.ctas)) return false;
    double t = 0.0;
    for (int q = threadIdx.x; q < sl.ctas; q += RT) t += __ldcg(part + (size_t)seg * sg.ctas + q);
    t = block_sum(t, sh);
    if (threadIdx.x == 0) tot = t;
    __syncthreads();
    *total = tot;
    return true;
}

// w <- s_i w - sum_l (h_l s_l) w_l per system (column order as dgemv 'N');
// the last CTA: |w|, the rotation of the new Hessenberg column, the new
// rotation, the residual estimate and the stopping test
__global__ void __launch_bounds__(RT, 4) k_seg_update(Seg sg, int64_t N, int i, const double *__restrict__ V,
                                                   double *__restrict__ w, double *__restrict__ part, KState st,
                                                   double tol) {
    if (skipped(st.done)) return;
    const int seg = blockIdx.y;
    if (!st.active[seg]) return;
    const Slice sl = slice_of(sg, seg, UPD_TILE, 1);
    if (!sl.on) return;
    __shared__ double sh_h[64], sh_c[64], sh_s[64];
    const double *hcol = st.hcol + (size_t)seg * st.HS;
    double *sc = st.sc + (size_t)seg * st.HS;
    if ((int)threadIdx.x <= i) sh_h[threadIdx.x] = -hcol[threadIdx.x] * sc[threadIdx.x];
    __syncthreads();
    const double si = sc[i];
    double ss = 0.0;
    // eight vectors' values of two dofs in flight at a time
    for (int64_t q = sl.lo; q < sl.hi; q += sl.step) {
        const int64_t q2 = q + RT;
        const bool two = q2 < sl.hi;
        const double *v = V + q, *v2 = V + (two ? q2 : q);
        double x = w[q] * si, x2 = two ? w[q2] * si : 0.0;
        for (int l0 = 0; l0 <= i; l0 += 8) {
            double a[8], b[8];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const bool in = l0 + k <= i;
                a[k] = in ? __ldg(v + (size_t)(l0 + k) * N) : 0.0;
                b[k] = in ? __ldg(v2 + (size_t)(l0 + k) * N) : 0.0;
            }
#pragma unroll
            for (int k = 0; k < 8; k++)
                if (l0 + k <= i) {
                    x += sh_h[l0 + k] * a[k];
                    x2 += sh_h[l0 + k] * b[k];
                }
        }
        w[q] = x;
        ss += x * x;
        if (two) {
            w[q2] = x2;
            ss += x2 * x2;
        }
    }
    double total;
    if (!seg_total(ss, sl, sg, seg, part, st.ticket, &total)) return;
    double *H = st.H + (size_t)seg * st.HP + i * (i + 1) / 2, *c = st.c + (size_t)seg * st.m,
           *s = st.s + (size_t)seg * st.m, *y = st.y + (size_t)seg * (st.m + 1);
    if ((int)threadIdx.x <= i) {
        sh_h[threadIdx.x] = hcol[threadIdx.x];
        sh_c[threadIdx.x] = (int)threadIdx.x < i ? c[threadIdx.x] : 0.0;
        sh_s[threadIdx.x] = (int)threadIdx.x < i ? s[threadIdx.x] : 0.0;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const double hnew = sqrt(total);
        sc[i + 1] = 1. / hnew;
        if (!isfinite(hnew)) atomicOr(st.status, 1);
        double h = sh_h[0];
        for (int k = 0; k < i; ++k) {
            const double h1 = sh_h[k + 1];
            sh_h[k] = __dsub_rn(__dmul_rn(sh_c[k], h), __dmul_rn(sh_s[k], h1));
            h = __dadd_rn(__dmul_rn(sh_s[k], h), __dmul_rn(sh_c[k], h1));
        }
        const double dd = __dsqrt_rn(__dadd_rn(__dmul_rn(h, h), __dmul_rn(hnew, hnew)));
        const double ci = __ddiv_rn(h, dd), sn = __ddiv_rn(-hnew, dd), yi = y[i];
        c[i] = ci;
        s[i] = sn;
        sh_h[i] = dd;
        const double ynew = __dmul_rn(sn, yi);
        y[i + 1] = ynew;
        y[i] = __dmul_rn(ci, yi);
        st.nsteps[seg] = i + 1;
        if (i + 1 >= st.m || fabs(ynew) < tol * st.nrm2b[2 * seg]) {
            st.active[seg] = 0;
            if (atomicSub(st.n_active, 1) == 1) *st.done = 1;
        }
    }
    __syncthreads();
    if ((int)threadIdx.x <= i) H[threadIdx.x] = sh_h[threadIdx.x];
}

// |r| per system: the norm of the right-hand side (start false), or the start
// of a cycle from the residual r = w_0: s_0, y_0 = |r| and which systems
// iterate
__global__ void __launch_bounds__(RT) k_seg_norm(Seg sg, const double *__restrict__ r, double *__restrict__ part,
                                                 KState st, bool start, double tol) {
    const int seg = blockIdx.y;
    const Slice sl = slice_of(sg, seg, UPD_TILE, 1);
    if (!sl.on) return;
    double ss = 0.0, total;
    for (int64_t q = sl.lo; q < sl.hi; q += sl.step) {
        ss += r[q] * r[q];
        if (q + RT < sl.hi) ss += r[q + RT] * r[q + RT];
    }
    if (!seg_total(ss, sl, sg, seg, part, st.ticket, &total) || threadIdx.x) return;
    const double nr = sqrt(total);
    if (!start) {
        st.nrm2b[2 * seg] = nr;
        return;
    }
    if (!isfinite(nr) || !isfinite(st.nrm2b[2 * seg])) atomicOr(st.status, 1);
    st.sc[(size_t)seg * st.HS] = 1. / nr;
    st.y[(size_t)seg * (st.m + 1)] = nr;
    st.nsteps[seg] = 0;
    const bool act = !st.finished[seg] && !(fabs(nr) < tol * st.nrm2b[2 * seg]);
    st.active[seg] = act ? 1 : 0;
    if (act) atomicAdd(st.n_active, 1);
    __threadfence();
    if (atomicAdd(st.ticket + sg.K * DOT_GROUPS, 1) == sg.K - 1) {  // the last system
        st.ticket[sg.K * DOT_GROUPS] = 0;
        __threadfence();
        *st.done = atomicAdd(st.n_active, 0) == 0 ? 1 : 0;
    }
}

// end of a cycle, one warp a system: R y = g (packed upper triangle, dtpsv
// 'U','N','N'), the update coefficients, and whether the system has converged
__global__ void __launch_bounds__(32) k_gmres_end(int j, KState st, double tol, int flexible, const int *sweep_err) {
    __shared__ double sh_H[62 * 63 / 2], sh_y[64];
    const int seg = blockIdx.x, lane = threadIdx.x;
    if (seg == 0 && lane == 0) {
        st.status[1] = *sweep_err;
        *st.n_active = 0;
    }
    if (st.finished[seg]) {
        if (lane == 0) st.nsteps[seg] = 0;  // leaves x alone
        return;
    }
    const int i = st.nsteps[seg];
    const double *H = st.H + (size_t)seg * st.HP, *y = st.y + (size_t)seg * (st.m + 1);
    for (int k = lane; k < i * (i + 1) / 2; k += 32) sh_H[k] = H[k];
    for (int k = lane; k <= i; k += 32) sh_y[k] = y[k];
    __syncwarp();
    for (int col = i - 1; col >= 0; col--) {
        const int kk = col * (col + 1) / 2;
        const double yc = __ddiv_rn(sh_y[col], sh_H[kk + col]);
        __syncwarp();
        for (int row = lane; row < col; row += 32) sh_y[row] = __dsub_rn(sh_y[row], __dmul_rn(yc, sh_H[kk + row]));
        if (lane == 0) sh_y[col] = yc;
        __syncwarp();
    }
    for (int l = lane; l < i; l += 32)
        st.cy[(size_t)seg * (st.m + 1) + l] = (flexible ? sh_y[l] : -sh_y[l]) * st.sc[(size_t)seg * st.HS + l];
    if (lane == 0) {
        st.its[seg] = st.m * j + i;
        const double r = fabs(sh_y[i]);
        st.nrm2b[2 * seg + 1] = r;
        if (r < tol * st.nrm2b[2 * seg]) st.finished[seg] = 1;
    }
}

// x += sum_{l < nsteps[seg]} cy[seg][l] * B_l over each segment
__global__ void k_seg_combine(Seg sg, int64_t N, const double *__restrict__ B, const double *__restrict__ cy,
                              int cstride, const int *__restrict__ nsteps, double *__restrict__ x) {
    __shared__ double sc[64];
    const int seg = blockIdx.y, nv = nsteps[seg];
    if (nv <= 0) return;
    for (int l = threadIdx.x; l < nv; l += blockDim.x) sc[l] = cy[(size_t)seg * cstride + l];
    __syncthreads();
    const int64_t a = sg.off[seg], b = sg.off[seg + 1];
    for (int64_t q = a + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < b; q += (int64_t)gridDim.x * blockDim.x) {
        double v = x[q];
#pragma unroll 4
        for (int l = 0; l < nv; l++) v += sc[l] * B[(size_t)l * N + q];
        x[q] = v;
    }
}

// clears *zero if any element of x is not zero
__global__ void k_zero_test(int64_t N, const double *__restrict__ x, int *zero) {
    bool any = false;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < N; q += (int64_t)gridDim.x * blockDim.x)
        any = any || !(x[q] == 0.0);
    if (__syncthreads_or(any) && threadIdx.x == 0) *zero = 0;
}
// r0 = a * b + r, or a * b where the initial guess is zero (r is not read)
__global__ void k_residual0(int64_t N, double a, const double *__restrict__ b, double rscale, double *__restrict__ r,
                            const int *x_zero) {
    const bool zero = x_zero && *x_zero;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < N; q += (int64_t)gridDim.x * blockDim.x)
        r[q] = zero ? a * b[q] : a * b[q] + rscale * r[q];
}
// r = -p where the initial guess is zero
__global__ void k_negate_if(int64_t N, const double *__restrict__ p, double *__restrict__ r, const int *x_zero) {
    if (!*x_zero) return;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < N; q += (int64_t)gridDim.x * blockDim.x)
        r[q] = -p[q];
}

int grid_seg(int64_t N, int K) {
    const int64_t per = (N / std::max(1, K) + 255) / 256;
    return (int)std::max<int64_t>(1, std::min<int64_t>(per, 512));
}

// sweep_err: the sweeps' status word as the last cycle left it
cpg_status gmres_seg_run(cpg_ctx *ctx, const LinOp &op, int K, const int64_t *off_host, const double *b, double *x,
                         int m, double tol, int maxit, int flexible, cpg_solve_stats *stats, int *sweep_err) {
    *sweep_err = -1;
    if (m < 1 || m > 62) return fail(ctx, CPG_ERR_INVALID_ARG, "GMRES restart must be 1..62");
    if (K < 1 || K > 1024) return fail(ctx, CPG_ERR_INVALID_ARG, "1..1024 systems per batched solve");
    const int64_t N = off_host[K];
    int64_t longest = 0;
    for (int k = 0; k < K; k++) longest = std::max(longest, off_host[k + 1] - off_host[k]);
    // workspace: V (m+1) N, r N, [Z m N]
    const size_t need = (size_t)(m + 2 + (flexible ? m : 0)) * N;
    double *ws;
    CPG_TRY(kws(ctx, need, &ws));
    double *V = ws, *r = ws + (size_t)(m + 1) * N, *Z = r + N;
    // scratch: partial sums, the systems' scalars, offsets and ints
    const int HS = m + 4, HP = m * (m + 1) / 2 + 1, ctas = seg_ctas(longest, UPD_TILE, 1);
    const size_t n_part = (size_t)ctas * K * (m + 2);
    const size_t n_dbl = n_part + (size_t)K * (2 * HS + HP + 2 * m + 2 * (m + 1) + 2);
    const size_t n_int = (4 + DOT_GROUPS) * (size_t)K + 6;
    double *sc;
    CPG_TRY(scratch(ctx, n_dbl + (size_t)(K + 1) + (n_int + 1) / 2, &sc));
    double *part = sc;
    KState st;
    st.m = m;
    st.HS = HS;
    st.HP = HP;
    st.hcol = part + n_part;
    st.sc = st.hcol + (size_t)K * HS;
    st.H = st.sc + (size_t)K * HS;
    st.c = st.H + (size_t)K * HP;
    st.s = st.c + (size_t)K * m;
    st.y = st.s + (size_t)K * m;
    st.cy = st.y + (size_t)K * (m + 1);
    int64_t *off_dev = (int64_t *)(st.cy + (size_t)K * (m + 1));
    // what the host reads after a cycle lies together: nrm2b, finished, its, status
    st.nrm2b = (double *)(off_dev + K + 1);
    st.finished = (int *)(st.nrm2b + 2 * (size_t)K);
    st.its = st.finished + K;
    st.status = st.its + K;
    st.active = st.status + 2;
    st.nsteps = st.active + K;
    st.ticket = st.nsteps + K;
    st.n_active = st.ticket + (size_t)K * DOT_GROUPS + 1;
    st.done = st.n_active + 1;
    st.x_zero = st.done + 1;
    const size_t read_bytes = 2 * (size_t)K * sizeof(double) + (2 * (size_t)K + 2) * sizeof(int);
    double *hbuf;
    CPG_TRY(pinned(ctx, read_bytes / sizeof(double) + 2 + (size_t)K, &hbuf));
    int64_t *hoff = (int64_t *)hbuf;  // on its way to the device before the first read-back
    std::memcpy(hoff, off_host, sizeof(int64_t) * (K + 1));
    CPG_CUDA(ctx, cudaMemcpyAsync(off_dev, hoff, sizeof(int64_t) * (K + 1), cudaMemcpyHostToDevice, ctx->stream));
    CPG_CUDA(ctx, cudaMemsetAsync(st.finished, 0, sizeof(int) * n_int, ctx->stream));
    CPG_CUDA(ctx, cudaMemsetAsync(st.x_zero, 1, sizeof(int), ctx->stream));
    const Seg sg{off_dev, K, ctas};
    const dim3 vgrid(grid_seg(N, K), K), rgrid(ctas, K);
    const int egrid = grid_for(ctx, N);

    // a zero initial guess (every Newton iteration of the DIRK steppers) has
    // the residual -P^{-1} b, which the norm of the right-hand side needs
    // anyway: the launches for it return at once then
    k_zero_test<<<egrid, 256, 0, ctx->stream>>>(N, x, st.x_zero);
    CPG_TRY(launched(ctx, "initial guess test kernel"));
    // nrm2b: |P^{-1} b| (left) or |b| (flexible), per system
    const double *rhs = b;
    if (!flexible) {
        CPG_TRY(vec_copy(ctx, N, b, r));
        CPG_TRY(op.prec(ctx, r));
        rhs = r;
    }
    k_seg_norm<<<rgrid, RT, 0, ctx->stream>>>(sg, rhs, part, st, false, tol);
    CPG_TRY(launched(ctx, "segmented norm kernel"));
    if (maxit % m > 0) maxit = (maxit / m + 1) * m;
    const int cycles = maxit / m;
    int j;
    cpg_status rc = CPG_OK;
    const double *hnb = hbuf;
    const int *hint = (const int *)(hbuf + 2 * (size_t)K);
    for (j = 0; j < cycles && rc == CPG_OK; j++) {
        // w_0 = P^{-1}(A x - b)   or   b - A x
        const int *zero = j == 0 ? st.x_zero : nullptr;
        ctx->skip_dev = zero;
        rc = op.apply(ctx, x, V);
        if (rc == CPG_OK) {
            k_residual0<<<egrid, 256, 0, ctx->stream>>>(N, flexible ? 1.0 : -1.0, b, flexible ? -1.0 : 1.0, V, zero);
            rc = launched(ctx, "initial residual kernel");
        }
        if (rc == CPG_OK && !flexible) rc = op.prec(ctx, V);
        if (rc == CPG_OK && !flexible && zero) {
            k_negate_if<<<egrid, 256, 0, ctx->stream>>>(N, r, V, zero);
            rc = launched(ctx, "initial residual kernel");
        }
        ctx->skip_dev = nullptr;
        if (rc != CPG_OK) break;
        k_seg_norm<<<rgrid, RT, 0, ctx->stream>>>(sg, V, part, st, true, tol);
        CPG_TRY(launched(ctx, "gmres start kernel"));
        // the cycle, with no host synchronisation: once every system has
        // converged the remaining launches return at once
        ctx->skip_dev = st.done;
        for (int i = 0; i < m && rc == CPG_OK; i++) {
            double *vi = V + (size_t)N * i, *vi1 = V + (size_t)N * (i + 1);
            if (!flexible) {
                rc = op.apply_prec(ctx, vi, vi1);
            } else {
                double *zi = Z + (size_t)N * i;
                rc = vec_copy(ctx, N, vi, zi);
                if (rc == CPG_OK) rc = op.prec(ctx, zi);
                if (rc == CPG_OK) rc = op.apply(ctx, zi, vi1);
            }
            if (rc != CPG_OK) break;
            const int groups = (i + DOTS) / DOTS;
            k_seg_dots<<<dim3(seg_ctas(longest, DOT_TILE, groups), groups, K), RT, 0, ctx->stream>>>(sg, V, N, vi1,
                                                                                                     part, st, i);
            rc = launched(ctx, "segmented multi-dot kernel");
            if (rc == CPG_OK) {
                k_seg_update<<<rgrid, RT, 0, ctx->stream>>>(sg, N, i, V, vi1, part, st, tol);
                rc = launched(ctx, "segmented gram-schmidt kernel");
            }
        }
        ctx->skip_dev = nullptr;
        if (rc != CPG_OK) break;
        k_gmres_end<<<K, 32, 0, ctx->stream>>>(j, st, tol, flexible, ctx->flag_dev + 2);
        CPG_TRY(launched(ctx, "gmres end kernel"));
        k_seg_combine<<<vgrid, 256, 0, ctx->stream>>>(sg, N, flexible ? Z : V, st.cy, m + 1, st.nsteps, x);
        CPG_TRY(launched(ctx, "solution update kernel"));
        // one read-back per cycle: which systems have converged, and status
        CPG_CUDA(ctx, cudaMemcpyAsync(hbuf, st.nrm2b, read_bytes, cudaMemcpyDeviceToHost, ctx->stream));
        CPG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        *sweep_err = hint[2 * K + 1];
        if (*sweep_err) return CPG_OK;  // gmres_checked reports it: nothing further is worth a cycle
        if (hint[2 * K]) return fail(ctx, CPG_ERR_NONFINITE, "non-finite GMRES quantity (right-hand side, residual or "
                                                             "Arnoldi vector)");
        bool all = true;
        for (int k = 0; k < K; k++) all = all && hint[k];
        if (all) break;
    }
    if (rc != CPG_OK) return rc;
    // iteration counts and residuals as the reference reports them
    // (BlockMatrix.cpp:157-158): its = m*j + i, |y_i| / |P^{-1} b|
    for (int k = 0; k < K && stats; k++) {
        const double res = hnb[2 * k] > 0 ? hnb[2 * k + 1] / hnb[2 * k] : 0.0;
        stats[k].iterations = hint[k] ? hint[K + k] : m * cycles + m;
        stats[k].residual = res;
        stats[k].converged = res < tol ? 1 : 0;
    }
    return CPG_OK;
}

// one status check per solve: a triangular sweep whose bounded wait ran out
// turns the whole solve into CPG_ERR_TIMEOUT.  A solve that read the status
// word with its last cycle and found it clear needs no read of its own.
cpg_status gmres_checked(cpg_ctx *ctx, const LinOp &op, int K, const int64_t *off, const double *b, double *x, int m,
                         double tol, int maxit, int flexible, cpg_solve_stats *stats) {
    int sweep_err;
    const cpg_status st = gmres_seg_run(ctx, op, K, off, b, x, m, tol, maxit, flexible, stats, &sweep_err);
    return sweep_err == 0 ? st : check_sweep_error(ctx, st);
}
}  // namespace

namespace cpg {
cpg_status gmres_op(cpg_ctx *ctx, const LinOp &op, int64_t N, const double *b, double *x, int m, double tol,
                    int maxit, int flexible, cpg_solve_stats *stats) {
    const int64_t off[2] = {0, N};
    return gmres_checked(ctx, op, 1, off, b, x, m, tol, maxit, flexible, stats);
}
}  // namespace cpg

extern "C" {

cpg_status cpg_gmres(cpg_ctx *ctx, const cpg_bsr *A, const cpg_precond *P, const double *b, double *x, int m,
                     double tol, int maxit, int flexible, cpg_solve_stats *stats) {
    if (!ctx || !A || !b || !x || maxit < 1) return CPG_ERR_INVALID_ARG;
    if (P && (P->n != A->n_rows || P->bl != A->bl)) return fail(ctx, CPG_ERR_INVALID_ARG, "preconditioner size");
    KrylovOp op(A, P, tol);
    return gmres_op(ctx, op, (int64_t)A->n_rows * A->bl, b, x, m, tol, maxit, flexible, stats);
}

cpg_status cpg_gmres_batched(cpg_ctx *ctx, const cpg_bsr *A, const cpg_precond *P, int nsys, const int *seg_rows,
                             const double *b, double *x, int m, double tol, int maxit, int flexible,
                             cpg_solve_stats *stats) {
    if (!ctx || !A || !b || !x || !seg_rows || maxit < 1 || nsys < 1) return CPG_ERR_INVALID_ARG;
    if (P && (P->n != A->n_rows || P->bl != A->bl)) return fail(ctx, CPG_ERR_INVALID_ARG, "preconditioner size");
    if (seg_rows[0] != 0 || seg_rows[nsys] != A->n_rows)
        return fail(ctx, CPG_ERR_INVALID_ARG, "system row ranges must start at 0 and end at the matrix's rows");
    std::vector<int64_t> off(nsys + 1);
    for (int k = 0; k <= nsys; k++) {
        if (k > 0 && seg_rows[k] <= seg_rows[k - 1])
            return fail(ctx, CPG_ERR_INVALID_ARG, "system row ranges must be increasing and non-empty");
        off[k] = (int64_t)seg_rows[k] * A->bl;
    }
    // the systems must be independent: every block of a row lies in the row's system
    for (int k = 0; k < nsys; k++)
        for (int i = seg_rows[k]; i < seg_rows[k + 1]; i++)
            for (int q = A->rowptr[i]; q < A->rowptr[i + 1]; q++)
                if (A->colidx[q] < seg_rows[k] || A->colidx[q] >= seg_rows[k + 1])
                    return fail(ctx, CPG_ERR_INVALID_ARG,
                                "block (" + std::to_string(i) + ", " + std::to_string(A->colidx[q]) +
                                    ") couples two systems");
    KrylovOp op(A, P, tol);
    return gmres_checked(ctx, op, nsys, off.data(), b, x, m, tol, maxit, flexible, stats);
}

}  // extern "C"

namespace {
cpg_status jacobi_run(cpg_ctx *ctx, const cpg_bsr *A, const cpg_precond *P, const double *b, double *x,
                      double tol, int maxit, cpg_solve_stats *stats) {
    const int64_t N = (int64_t)A->n_rows * A->bl;
    double *ws;
    CPG_TRY(kws(ctx, 3 * (size_t)N, &ws));
    double *dinvb = ws, *t = ws + N, *r = ws + 2 * N;
    double *sc;
    CPG_TRY(scratch(ctx, RED + 8, &sc));
    const double omega = 1.0;
    CPG_TRY(vec_copy(ctx, N, b, dinvb));
    CPG_TRY(precond_apply_raw(ctx, P, dinvb));
    int mm;
    double nr = 0.0;
    for (mm = 0; mm < maxit; mm++) {
        CPG_TRY(bsr_matvec_raw(ctx, A, x, t));
        CPG_TRY(vec_copy(ctx, N, t, r));
        CPG_TRY(vec_axpby(ctx, N, -1.0, b, 1.0, r));
        CPG_TRY(norm_dev(ctx, N, r, sc, sc + RED));
        CPG_TRY(read_host(ctx, sc + RED, 1, &nr));
        if (!std::isfinite(nr)) return fail(ctx, CPG_ERR_NONFINITE, "non-finite Jacobi residual");
        if (nr < tol) break;
        CPG_TRY(precond_apply_raw(ctx, P, t));
        k_jacobi_update<<<grid_for(ctx, N), 256, 0, ctx->stream>>>(N, omega, dinvb, t, x);
        CPG_TRY(launched(ctx, "jacobi update kernel"));
    }
    if (stats) {
        stats->iterations = mm;
        stats->residual = nr;
        stats->converged = nr < tol ? 1 : 0;
    }
    return CPG_OK;
}
}  // namespace

extern "C" {

cpg_status cpg_jacobi_solve(cpg_ctx *ctx, const cpg_bsr *A, const cpg_precond *P, const double *b, double *x,
                            double tol, int maxit, cpg_solve_stats *stats) {
    if (!ctx || !A || !P || !b || !x) return CPG_ERR_INVALID_ARG;
    return check_sweep_error(ctx, jacobi_run(ctx, A, P, b, x, tol, maxit, stats));
}

cpg_status cpg_axpby(cpg_ctx *ctx, int64_t n, double a, const double *x, double b, double *y) {
    if (!ctx || !x || !y || n < 0) return CPG_ERR_INVALID_ARG;
    return vec_axpby(ctx, n, a, x, b, y);
}

}  // extern "C"
