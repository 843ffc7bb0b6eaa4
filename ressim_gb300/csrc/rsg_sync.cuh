// Synchronisation helpers of the sync-free (flag-driven) kernels, shared by the device translation units
// (internal linkage in each): release stores and relaxed polls of per-row flags at GPU scope with one acquire
// fence per row, values that are their own flags, the bounded waits, and the warp's claim of consecutive positions from
// an atomic counter.
#pragma once
#include <cuda_runtime.h>

#include "rsg_impl.h"

namespace rsg {
namespace {

constexpr unsigned kSpinLimit = 1u << 22;   // x up to 256 ns back-off: about one second per wait

__device__ __forceinline__ void st_release(int* p, int v) {
    asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_relaxed(const int* p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void fence_acquire() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// Another round of a bounded wait: a short busy phase, then back-off up to 256 ns; false when the limit is reached
// (ERR_TIMEOUT is set) or another wait already gave up.
__device__ __forceinline__ bool poll_again(unsigned it, unsigned& ns, int* err) {
    if (it < 64) return true;
    __nanosleep(ns);
    ns = ns < 32 ? 32 : (ns < 256 ? 2 * ns : 256);
    if (it >= 64 + kSpinLimit) {
        atomicOr(err, ERR_TIMEOUT);
        return false;
    }
    return (it & 255u) != 255u || *(volatile int*)err == 0;
}

// Values that are their own flags. A word holds a value's bits, or all ones: not yet there. (All ones is a NaN; a value
// with those bits is stored as another NaN.) A 4- or 8-byte relaxed access is single-copy atomic, so a poll that finds the
// word filled has the whole value: a dependency costs one trip through L2. Whoever starts a sweep has cleared its words
// (by the launch before it).
template <class T>
struct Word;
template <>
struct Word<double> {
    using type = unsigned long long;
    static constexpr type empty = ~0ull;
    __device__ static __forceinline__ type make(double v) {
        const type b = static_cast<type>(__double_as_longlong(v));
        return b == empty ? 0x7ff8000000000000ull : b;
    }
    __device__ static __forceinline__ double value(type b) { return __longlong_as_double(static_cast<long long>(b)); }
};
template <>
struct Word<float> {
    using type = unsigned;
    static constexpr type empty = ~0u;
    __device__ static __forceinline__ type make(float v) {
        const type b = __float_as_uint(v);
        return b == empty ? 0x7fc00000u : b;
    }
    __device__ static __forceinline__ float value(type b) { return __uint_as_float(b); }
};
__device__ __forceinline__ unsigned long long ld_word(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned ld_word(const unsigned* p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_word(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void st_word(unsigned* p, unsigned v) {
    asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ int warp_claim(unsigned* ctr, int rows = 32) {
    unsigned base = 0;
    if ((threadIdx.x & 31) == 0) base = atomicAdd(ctr, unsigned(rows));
    return int(__shfl_sync(0xffffffffu, base, 0));
}

}  // namespace
}  // namespace rsg
