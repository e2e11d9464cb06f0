// common.cuh -- shared helpers of the sm_100a monodomain library.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include <string>

#include "../../include/ep_gpu.h"

// cell-model code is host+device so the same source can be exercised on
// the host (tests, debugging) and compiled into the sm_100a kernels
#define EP_HD __host__ __device__ __forceinline__

namespace ep {

// ---- error reporting (thread-local message behind ep_last_error) ----
void set_error(const char *fmt, ...);
const char *last_error();

#define EP_CUDA(call)                                                          \
    do {                                                                       \
        cudaError_t e_ = (call);                                               \
        if (e_ != cudaSuccess) {                                               \
            ::ep::set_error("%s:%d %s: %s", __FILE__, __LINE__, #call,         \
                            cudaGetErrorString(e_));                           \
            return EP_ERR_CUDA;                                                \
        }                                                                      \
    } while (0)

#define EP_CHECK_ARG(cond, msg)                                                \
    do {                                                                       \
        if (!(cond)) { ::ep::set_error("%s", msg); return EP_ERR_ARG; }        \
    } while (0)

constexpr int kMaxTypes = 256;     // parameter sets per handle (uint8 node types)
constexpr int kMaxSub = 64;        // ionic sub-steps per global step
constexpr int kSlice = 32;         // SELL slice height (one warp)

// Device status word shared by all kernels of a handle.
struct DevStatus {
    unsigned long long newton_iters;
    unsigned int newton_cap_hits;
    unsigned int timeouts;
    unsigned int nonfinite;
    unsigned int cg_fail;
    unsigned long long fallback;
    unsigned int pad[8];
};

// Bounded sense-reversing grid barrier for cooperative (co-resident) grids.
// Returns false when the wait gave up; the caller must then leave the kernel
// (every block reaches the same conclusion through *err).  `limit` caps the
// polls of one wait (0: kGridPolls, a few seconds); a wait that runs out
// sets err, which the host reads as EP_ERR_TIMEOUT and then clears.
constexpr unsigned int kGridPolls = 1u << 24;
struct GridBarrier {
    unsigned int count;
    unsigned int gen;
    unsigned int err;
    unsigned int limit;
    unsigned long long seq;      // last tag of the solves so far (cg.cu group_reduce)
    unsigned long long pad;
};

__device__ __forceinline__ bool grid_sync(GridBarrier *b, unsigned int nblocks) {
    __shared__ int s_ok;
    // the CTA barrier orders every thread's writes before thread 0's
    // gpu-scope fence and arrival (fences are cumulative), as a cooperative
    // grid sync does: one fence per CTA, not one per thread
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        volatile unsigned int *vgen = &b->gen;
        volatile unsigned int *verr = &b->err;
        const unsigned int lim = *(volatile unsigned int *)&b->limit;
        const unsigned int max_polls = lim ? lim : kGridPolls;
        const unsigned int g = *vgen;
        __threadfence();
        // the last arrival wraps the count back to 0 in the same atomic (no
        // separate reset store for the release fence to wait on)
        const unsigned int arrived = atomicInc(&b->count, nblocks - 1u);
        if (arrived == nblocks - 1) {
            __threadfence();
            atomicAdd(&b->gen, 1u);
        } else {
            // at most max_polls polls with a short sleep, then give up
            unsigned int polls = 0;
            while (*vgen == g) {
                if (*verr) { ok = 0; break; }
                if (++polls > max_polls) { atomicExch(&b->err, 1u); ok = 0; break; }
                __nanosleep(64);
            }
        }
        __threadfence();
        if (*verr) ok = 0;
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// ---- arithmetic of the cell models ----
// a / b.  FP32 on the device: the hardware reciprocal estimate (1 ulp) and one
// correction of the quotient by its exact remainder (P. Markstein, IBM J.
// Res. Dev. 34 (1990) 111), four instructions without the special-case branch
// of the / operator, which the models' wide-ranging denominators take often
// enough to cost more than the arithmetic around them (Mahajan's FP32 kernel
// ran with 9 of 32 lanes active).  Within 0.51 ulp where b and the quotient
// are normal and |b| < 2^126; the callers keep their denominators there (a zero
// or infinite one gives NaN).  dvc: for denominators a caller's constants decide,
// zero and infinity as with / (a test and a select more: everywhere, they cost
// 5 to 13 % of the ionic phase).
EP_HD double dv(double a, double b) { return a / b; }
EP_HD float dv(float a, float b) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
    const float q = a * r;
    return fmaf(fmaf(-b, q, a), r, q);
#else
    return a / b;
#endif
}
EP_HD double dvc(double a, double b) { return a / b; }
EP_HD float dvc(float a, float b) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
    const float q = a * r, rem = fmaf(-b, q, a);
    return fabsf(rem) < INFINITY ? fmaf(rem, r, q) : q;
#else
    return a / b;
#endif
}
// x / d for a constant d: the reciprocal in two parts, the quotient rounded
// as a division's to within half an ulp more
template <typename R> EP_HD R over(R x, double d) {
    const R hi = (R)(1.0 / d);
    const R lo = sizeof(R) == 4 ? (R)(1.0 / d - (double)hi) : (R)(fma(-(double)hi, d, 1.0) / d);
    return fma(x, hi, x * lo);
}
// the smaller of x and a number; NaN stays NaN
EP_HD float cap(float x, float most) {
#ifdef __CUDA_ARCH__
    float y;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(x), "f"(most));
    return y;
#else
    return x > most ? most : x;
#endif
}
EP_HD double cap(double x, double most) { return x > most ? most : x; }
// exp(x), the argument capped where 1 + exp(x) is exp(x) to every digit and
// products of three such factors still fit the type
EP_HD float cexp(float x) { return expf(cap(x, 28.f)); }
EP_HD double cexp(double x) { return exp(cap(x, 200.0)); }
// exp(x) - 1, the argument capped as the reach of the type asks
EP_HD float cexpm1(float x) { return expm1f(cap(x, 80.f)); }
EP_HD double cexpm1(double x) { return expm1(cap(x, 600.0)); }

template <typename T> struct RealName;
template <> struct RealName<float> { static constexpr const char *s = "f32"; };
template <> struct RealName<double> { static constexpr const char *s = "f64"; };

inline int div_up(long long a, long long b) { return (int)((a + b - 1) / b); }

}  // namespace ep
