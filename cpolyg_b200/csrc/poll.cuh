// Values published by storing them.  A vector that is about to be published
// holds PENDING in every element, a signalling NaN: arithmetic produces only
// quiet NaNs, so no result is mistaken for it.  The reader of a value polls
// the value itself.  Publishing is one store, waiting one load, where a flag
// takes a fence, a release store, an acquire load and then the load of the
// value.  Every wait is bounded; one that runs out sets *err, after which no
// wait lasts.
#pragma once
#include <cuda_runtime.h>

namespace cpg {

constexpr unsigned long long PENDING = 0x7ff4c0deb200feedULL;
constexpr int POLL_NS = 64;
constexpr long long POLL_MAX = 1LL << 22;  // polls; a wait of that many took 1.4 s (__nanosleep may return at once)

__device__ __forceinline__ double poll_load(const double *p) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void publish_value(double *p, double v) {
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
__device__ __forceinline__ void set_pending(double *p) { *reinterpret_cast<unsigned long long *>(p) = PENDING; }
__device__ __forceinline__ bool is_pending(double v) {
    return (unsigned long long)__double_as_longlong(v) == PENDING;
}

// Loads the N values a thread multiplies (null: none) once all of them have
// been published.  A thread that has to wait polls one value until it is
// there, then loads all that are missing: thousands of rows may wait at a
// level's start, and polls of all N values took enough of L2 to slow the rows
// that they wait for (100,000 40x40 rows: 2.1 ms a sweep pair against 1.5 ms),
// while polling one value after the other adds a round trip for each
// (GMRES on 1,009 24x24 rows: 1.42 ms against 1.25).
template <int N>
__device__ __forceinline__ void poll_values(const double *const (&p)[N], double (&v)[N], int *err) {
#pragma unroll
    for (int k = 0; k < N; k++) v[k] = p[k] ? poll_load(p[k]) : 0.0;
    long long spins = 0;
    for (;;) {
        const double *missing = nullptr;
#pragma unroll
        for (int k = 0; k < N; k++)
            if (is_pending(v[k])) missing = p[k];
        if (!missing) return;
        do {
            if (++spins > POLL_MAX || ((spins & 255) == 0 && *(volatile int *)err != 0)) {
                atomicExch(err, 1);
                return;
            }
            __nanosleep(POLL_NS);
        } while (is_pending(poll_load(missing)));
#pragma unroll
        for (int k = 0; k < N; k++)
            if (is_pending(v[k])) v[k] = poll_load(p[k]);
    }
}
// the same for p, p + STEP, ...
template <int N, int STEP>
__device__ __forceinline__ void poll_strided(const double *p, double (&v)[N], int *err) {
    const double *q[N];
#pragma unroll
    for (int k = 0; k < N; k++) q[k] = p + k * STEP;
    poll_values<N>(q, v, err);
}

}  // namespace cpg
