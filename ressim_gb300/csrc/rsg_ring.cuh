// Shared-memory ring of the block sweeps: mbarrier and bulk-copy helpers and the producer's byte ring (internal linkage in
// each translation unit that includes it). Every wait is bounded: when it runs out, ERR_TIMEOUT is set and the kernel
// runs on to its end.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#include "rsg_impl.h"

namespace rsg {
namespace {

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return ok != 0;
}
// Waits for the phase of the given parity to complete, for about a second at most (a try_wait suspends the thread for a time
// of the hardware's choosing, so the limit is in clocks). `dead`: an earlier wait of this thread ran out -- the later ones
// are not waited for, so that the kernel ends.
constexpr long long kBarClocks = 2000000000ll;
__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t parity, int& dead, int* err, int tag = 1) {
    if (dead || mbar_try(bar, parity)) return;
    const long long t0 = clock64();
    do {
        if (mbar_try(bar, parity)) return;
    } while (clock64() - t0 < kBarClocks);
    dead = tag;
    atomicOr(err, ERR_TIMEOUT);
}
// bytes (a multiple of 16) from global memory to shared memory, both 16-byte aligned; completes on the mbarrier
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(reinterpret_cast<unsigned long long>(src)), "r"(bytes), "r"(bar)
                 : "memory");
}
// the same bytes into L2 only, without waiting
__device__ __forceinline__ void bulk_prefetch(const void* src, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(reinterpret_cast<unsigned long long>(src)), "r"(bytes) : "memory");
}
// Ring offset of entry `entry` of a batch-wide list of which a step holds the part from `first` on, at offset `base`. The
// difference is taken before it is scaled: entry numbers of a whole batch times their bytes do not fit 32 bits.
__host__ __device__ constexpr uint32_t ring_entry(uint32_t base, int entry, int first, uint32_t entryBytes) {
    return base + uint32_t(entry - first) * entryBytes;
}
// Byte ring: allocations in order, freed in order; an allocation is contiguous (it wraps to the start when the end is too
// short). head == tail only when empty.
struct ByteRing {
    uint32_t cap, head = 0, tail = 0;
    int live = 0;
    __device__ __forceinline__ bool alloc(uint32_t n, uint32_t& at) {
        if (live == 0) head = tail = 0;
        if (live == 0 || head > tail) {
            if (cap - head >= n) at = head;
            else if (tail > n) at = 0;
            else return false;
        } else {
            if (tail - head <= n) return false;
            at = head;
        }
        head = at + n;
        ++live;
        return true;
    }
    // the oldest allocation ends; `next`: where the one after it starts (ignored when none is left)
    __device__ __forceinline__ void free_oldest(uint32_t next) {
        --live;
        tail = next;
    }
};

}  // namespace
}  // namespace rsg
