// Values as their own flags (see flow.cu): a vector starts as 0xff bytes, a
// row's value is one relaxed store, a reader loads until it sees something
// else.  Waits are bounded (WaitBound).
#pragma once

#include "device_common.cuh"

namespace unapgpu {

// ---- values that say whether they are there -------------------------------
__device__ __forceinline__ float ld_flow(const float* p)
{
    float v;
    asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ double ld_flow(const double* p)
{
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ bool absent(float v) { return __float_as_uint(v) == 0xffffffffu; }
__device__ __forceinline__ bool absent(double v) { return __double_as_longlong(v) == -1ll; }
__device__ __forceinline__ void st_flow(float* p, float v)
{
    if (absent(v)) v = __uint_as_float(0x7fffffffu);
    asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}
__device__ __forceinline__ void st_flow(double* p, double v)
{
    if (absent(v)) v = __longlong_as_double(0x7ff8000000000000ll);
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}

// One more poll of a wait: true when the wait has to be given up.
__device__ __forceinline__ bool give_up(int& spins, int* err)
{
    if ((++spins & 0xfff) == 0) {
        if (spins >= kWaitPolls) *(volatile int*)err = 1;
        if (*(volatile int*)err) return true;
    }
    return false;
}

// Loads at(k) for the entries in `need` (one bit each) until every value is
// there; all lanes of the warp call it.
template <class T, int CK, class At>
__device__ __forceinline__ void wait_values(unsigned need, At&& at, T (&v)[CK], int* err)
{
    int spins = 0;
    for (;;) {
#pragma unroll
        for (int k = 0; k < CK; ++k)
            if (need >> k & 1u) v[k] = ld_flow(at(k));
#pragma unroll
        for (int k = 0; k < CK; ++k)
            if ((need >> k & 1u) && !absent(v[k])) need &= ~(1u << k);
        if (!__any_sync(0xffffffffu, need != 0)) return;
        if (give_up(spins, err)) return;
    }
}

// A task far ahead of the rows that are being computed would poll for long:
// until a row two wavefronts before its own is there, the whole warp polls
// that one address, with pauses.
template <class T>
__device__ __forceinline__ void wait_near(const T* p, WaitBound b)
{
    int spins = b.spent;
    while (absent(ld_flow(p))) {
        __nanosleep(64);
        if (give_up(spins, b.err)) return;
    }
}

}  // namespace unapgpu
