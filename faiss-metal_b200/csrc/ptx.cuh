// Thin inline-PTX wrappers shared by the kernels that use mbarriers and bulk copies.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace b200f {

constexpr long long kWaitLimitCycles = 2000000000LL;  // ~1 s: bound of every device-side wait

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// Programmatic dependent launch.  pdl_trigger: the next kernel of the stream, launched with the attribute, may
// take its place on the SMs; pdl_wait: everything earlier in the stream has completed and is visible
// (no effect in a kernel launched without the attribute).  A kernel that may be launched that way waits
// before its first access to memory, and triggers after it: its successor then overlaps with no
// other kernel than itself.  What its predecessor wrote it reads with coherent loads (no __ldg, no
// const __restrict__): the read-only path wants data that nobody writes while the kernel is resident.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Before TMA loads of what earlier kernels wrote with plain stores.
__device__ __forceinline__ void fence_proxy_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
            "{\n\t"
            ".reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t"
            "}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
    return done;
}

// Bounded wait.  Returns false when the wait ran out (status word gets `err_bit`, the CTA
// abort flag is raised) or another thread of the CTA already aborted; the caller must then
// leave its loop.
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity,
                                                  volatile int* abort_flag, int32_t* status,
                                                  int err_bit, long long limit_cycles = kWaitLimitCycles) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    int spins = 0;
    while (true) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((++spins & 255) == 0) {
            if (*abort_flag) return false;
            if (clock64() - t0 > limit_cycles) {
                *abort_flag = 1;
                if (status) atomicOr(status, err_bit);
                return false;
            }
        }
    }
}

// Untiled bulk copy global -> shared (both addresses 16-byte aligned, size a multiple of 16),
// completion counted in bytes on an mbarrier.  No multicast.
__device__ __forceinline__ void bulk_load(uint32_t dst_smem, const void* src, uint32_t bytes,
                                          uint32_t bar) {
    asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
            ::"r"(dst_smem), "l"(src), "r"(bytes), "r"(bar)
            : "memory");
}

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(addr));
    return v;
}

}  // namespace b200f
