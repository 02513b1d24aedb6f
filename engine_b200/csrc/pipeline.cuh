// mbarrier + bulk-copy (TMA, untiled) primitives for sm_100a, as inline PTX.
//
// Every wait is bounded: after kSpinLimit unsuccessful polls the caller gets
// `false`, records the failure in a status word and leaves the kernel instead
// of hanging the GPU.
#pragma once

#include <stdint.h>

namespace ribn {

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return done != 0;
}

// try_wait already suspends the thread for a hardware-defined interval per
// call, so a few million polls is on the order of seconds at worst.
constexpr uint32_t kSpinLimit = 1u << 22;

__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity) {
    for (uint32_t spin = 0; spin < kSpinLimit; ++spin) {
        if (mbar_try_wait(bar, parity)) return true;
        if (spin > 4096) __nanosleep(64);
    }
    return false;
}

// The same wait with an explicit suspend-time hint: the thread stays suspended for up to `hint_ns` per poll, so a
// warp that waits for data takes few issue slots from the warps that compute.
__device__ __forceinline__ bool mbar_try_wait_hint(uint64_t* bar, uint32_t parity, uint32_t hint_ns) {
    uint32_t done;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity), "r"(hint_ns)
        : "memory");
    return done != 0;
}
__device__ __forceinline__ bool mbar_wait_bounded_hint(uint64_t* bar, uint32_t parity, uint32_t hint_ns) {
    for (uint32_t spin = 0; spin < kSpinLimit; ++spin) {
        if (mbar_try_wait_hint(bar, parity, hint_ns)) return true;
    }
    return false;
}

// Bounded wait that polls without suspending: a thread that mbarrier.try_wait suspends is late by some hundred clocks, which the
// hand-overs of a K step cannot afford.  `polls`: how often at most, kPolls (about a second) or nothing once a wait has run out.
constexpr uint32_t kPolls = 1u << 26;
__device__ __forceinline__ bool mbar_spin(uint32_t bar, uint32_t parity, uint32_t polls) {
    uint32_t done;
    asm volatile(
        "{\n\t"
        ".reg .pred p, q;\n\t"
        ".reg .u32 left;\n\t"
        "mov.u32 left, %3;\n\t"
        "POLL:\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "@p bra DONE;\n\t"
        "sub.u32 left, left, 1;\n\t"
        "setp.gt.s32 q, left, 0;\n\t"
        "@q bra POLL;\n\t"
        "DONE:\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}"
        : "=r"(done)
        : "r"(bar), "r"(parity), "r"(polls)
        : "memory");
    return done != 0;
}
__device__ __forceinline__ bool mbar_spin(uint64_t* bar, uint32_t parity) { return mbar_spin(smem_addr(bar), parity, kPolls); }

// Untiled bulk copy global -> shared of `bytes` (a multiple of 16; both
// addresses 16-byte aligned), completion counted on `bar` in bytes.
__device__ __forceinline__ void bulk_copy_g2s(void* dst_smem, const void* src_global, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_addr(dst_smem)),
        "l"(src_global), "r"(bytes), "r"(smem_addr(bar))
        : "memory");
}

__device__ __forceinline__ void named_barrier_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Programmatic dependent launch: let the next kernel in the stream start its
// prologue, and wait for the previous kernel's memory before touching its output.
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait_prior() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

}  // namespace ribn
