// tcgen05 (fifth-generation tensor core) helpers shared by the kernels that use tensor memory, and the
// int8 peak probe.
#pragma once
#include "kernels_mma.cuh"

namespace pgb {

__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    // K-major, no swizzle: 8 rows x 16 bytes per core matrix; LBO = distance between the two
    // 16-byte K halves, SBO = distance between 8-row groups; bit 46 = descriptor version 1
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo_bytes >> 4) << 16) |
           ((uint64_t)(sbo_bytes >> 4) << 32) | (1ull << 46);
}
__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t"
        "}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
}
// One thread of a converged warp, chosen in the form that the compiler knows to be a single one: an MMA pair with its
// commits takes 34 cycles to issue in a block chosen by elect.sync and 165 under a condition like `lane == 0`
// (measured; bulk and tensor copies are of the same kind).
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// try_wait that lets the hardware park the thread for up to `ns` nanoseconds instead of
// returning at once (the peak probe, whose MMAs run for long)
__device__ __forceinline__ uint32_t mbar_try_wait_park(uint32_t bar, uint32_t parity, uint32_t ns) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(ns)
        : "memory");
    return ok;
}

// bounded wait that also gives up when another role has already failed
__device__ __forceinline__ bool um_wait(uint32_t bar, uint32_t parity, volatile int *fail) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (*fail) return false;
        if (clock64() - t0 > 2000000000LL) {
            *fail = 1;
            return false;
        }
    }
    return true;
}

// Arrival of lane 0 of a warp, without a branch
__device__ __forceinline__ void mbar_arrive_lane0(uint32_t bar, int lane) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.s32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(bar),
                 "r"(lane)
                 : "memory");
}
// The same for loops that go on after a failure: the waits that follow return at once (the flag is set), the
// accesses stay in bounds, the results are reported as bad.  Saves the vote of every single wait.
__device__ __forceinline__ void um_spin(uint32_t bar, uint32_t parity, volatile int *fail) {
    if (mbar_try_wait(bar, parity)) return;
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (*fail) return;
        if (clock64() - t0 > 2000000000LL) *fail = 1;
    }
}

// ---------------------------------------------------------------- int8 tensor peak probe
// The denominator of the prefill roofline, measured instead of quoted: one CTA per SM issues
// `iters` back-to-back 128 x 256 x 32 tcgen05.mma kind::i8 (s8 x u8 -> s32) on operands that stay
// in shared memory, alternating between two 256-column accumulators in tensor memory; nothing else
// runs.  ops = iters * 2 * 128 * 256 * 32 per CTA.
constexpr int kPeakABytes = 2 * 128 * 16, kPeakBBytes = 2 * 256 * 16;
constexpr uint32_t kPeakIdesc = (2u << 4) | (1u << 7) | (0u << 10) | ((256u >> 3) << 17) | ((128u >> 4) << 24);
__global__ void __launch_bounds__(128, 1) int8_peak_probe_kernel(int iters, int *err) {
    __shared__ __align__(128) uint8_t ops[kPeakABytes + kPeakBBytes];
    __shared__ __align__(8) unsigned long long bar;
    __shared__ uint32_t s_tmem;
    const int tid = threadIdx.x, warp = tid >> 5;
    for (int i = tid; i < kPeakABytes + kPeakBBytes; i += blockDim.x)
        ops[i] = i < kPeakABytes ? (uint8_t)(int8_t)(((i * 37 + 11) % 7) - 3) : (uint8_t)((i * 29 + 5) & 15);
    const uint32_t b = smem_u32(&bar);
    if (tid == 0) {
        mbar_init(b, 1);
        fence_mbar_init();
    }
    fence_proxy_async();  // operands written by threads, read by the tensor core
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const uint32_t tmem = s_tmem;
    if (tid == 0) {
        const uint64_t adesc = umma_desc(smem_u32(ops), 128 * 16, 128);
        const uint64_t bdesc = umma_desc(smem_u32(ops + kPeakABytes), 256 * 16, 128);
        for (int i = 0; i < iters; ++i) umma_i8(tmem + (i & 1) * 256, adesc, bdesc, kPeakIdesc, i >= 2 ? 1u : 0u);
        umma_commit(b);
        const long long t0 = clock64();
        while (!mbar_try_wait_park(b, 0u, 20000u))
            if (clock64() - t0 > 20000000000LL) {
                report_error(err, kErrBarrierTimeout);
                break;
            }
        tmem_fence_after();
    }
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

}  // namespace pgb
