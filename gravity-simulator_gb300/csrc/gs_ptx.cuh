// gs_ptx.cuh -- inline-PTX helpers for sm_103a: mbarrier, TMA bulk copies,
// bounded waits.  Every wait has a time limit; on expiry the caller gets
// `false`, sets a status bit and leaves its loop (no trap, no endless spin).
#pragma once

#include <cstdint>

#include "gs_internal.h"

namespace gs {

// Time limit of one bounded wait (ns of %globaltimer).
constexpr unsigned long long kWaitLimitNs = 2000000000ull;

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
                 : "memory");
}

// Make barrier initialisation visible to the async (TMA) proxy.
__device__ __forceinline__ void mbar_fence_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, unsigned parity)
{
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return done != 0;
}

// Bounded wait for the phase with the given parity to complete.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, unsigned parity)
{
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = global_ns();
    for (;;) {
        if (mbar_try_wait(bar, parity)) return true;
        if (global_ns() - t0 > kWaitLimitNs) return false;
    }
}

// TMA bulk copy global -> shared (no tensor map), completing on `bar`.
// dst and src 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, unsigned bytes, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ float rsqrt_approx(float x)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Kahan-compensated accumulation: s + (-c) carries the running sum.
__device__ __forceinline__ void kahan_add(float &s, float &c, float v)
{
    const float y = v - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
}

// grav_sim's compensated update (src/integrator.c:1014-1016):
//   err += d*dt; y_new = y + err; err += y - y_new;  every op rounded alone.
__device__ __forceinline__ void comp_update(double &y, double &err, double d, double dt)
{
    const double y0 = y;
    err = __dadd_rn(err, __dmul_rn(d, dt));
    y = __dadd_rn(y0, err);
    err = __dadd_rn(err, __dsub_rn(y0, y));
}

// Element k of a force kernel's result: a[k], and the kick that follows it.
__device__ __forceinline__ void store_and_kick(double *__restrict__ a, size_t k, double value,
                                               const Kick &kick)
{
    a[k] = value;
    if (kick.v) {
        double v = kick.v[k], e = kick.ve[k];
        comp_update(v, e, value, kick.h);
        kick.v[k] = v;
        kick.ve[k] = e;
    }
}

}  // namespace gs
