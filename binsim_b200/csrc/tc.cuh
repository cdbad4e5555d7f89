// Barrier, descriptor and tensor-memory helpers of the tcgen05 kernels
// (sigma_tc.cu: TF32 products of the FP32-bulk sigma; sigma_split.cu: split products
// of the FP64 sigma).  The counters are per source file.
#pragma once
#include "common.cuh"

namespace bsim {

namespace {

constexpr unsigned long long kTcWaitNs = 20000000ull;   // a wait gives up after 20 ms
constexpr long kTcSpinCap = 1L << 26;                   // and after this many rounds in any case
constexpr long kTcCheck = 16;                            // the flags and the clock are read after so many rounds
constexpr long kTcMinSpins = 1000;                      // but not before this many: a preempted CTA's clock runs on
constexpr unsigned kTcSuspendNs = 20000;                // longest sleep in one test of a phase
constexpr uint32_t kCoreBytes = 128;      // one core matrix: 8 rows x 16 bytes

__device__ int g_tc_timeouts;   // waits that gave up
__device__ int g_tc_abort;      // set with the first of them: later CTAs do not start their waits

__host__ __device__ inline uint32_t align128(uint32_t x) { return (x + 127u) & ~127u; }

__device__ __forceinline__ void mbar_init(uint32_t a, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t a)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(a) : "memory");
}
// One arrival for the warp, after every lane got here (its shared-memory writes, or
// its tensor-memory reads, fenced by each lane).
__device__ __forceinline__ void warp_arrive(uint32_t a)
{
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(a);
}
// One test of the phase; the thread may sleep in it (up to kTcSuspendNs) until
// the phase completes, so a waiting warp takes no issue slots from the others.
__device__ __forceinline__ bool mbar_try(uint32_t a, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred P1;\n\tmbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2, %3;\n\t"
                 "selp.b32 %0, 1, 0, P1;\n\t}"
                 : "=r"(ok)
                 : "r"(a), "r"(parity), "n"(kTcSuspendNs)
                 : "memory");
    return ok != 0;
}

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Bounded wait for the phase of the given parity; false when the CTA aborts
// (its own wait gave up, another wait of the CTA did, or another CTA's did).
// The flags and the clock are read after every kTcCheck tests that came back without
// the phase.
__device__ bool mbar_wait(uint32_t a, uint32_t parity, volatile int *abort_flag)
{
    if (mbar_try(a, parity)) return true;
    const unsigned long long t0 = global_ns();
    for (long i = 1; i < kTcSpinCap; ++i) {
        if (mbar_try(a, parity)) return true;
        if (i % kTcCheck) continue;
        if (*abort_flag) return false;
        if (*(volatile int *)&g_tc_abort) { *abort_flag = 1; return false; }
        if (i >= kTcMinSpins && global_ns() - t0 > kTcWaitNs) break;
    }
    *abort_flag = 1;
    atomicExch(&g_tc_abort, 1);
    atomicAdd(&g_tc_timeouts, 1);
    return false;
}

// Bounded wait that ignores the abort flags: the wait for this CTA's own MMAs
// before its tensor memory is freed.
__device__ void mbar_wait_drain(uint32_t a, uint32_t parity)
{
    const unsigned long long t0 = global_ns();
    for (long i = 0; i < kTcSpinCap; ++i) {
        if (mbar_try(a, parity)) return;
        if (i >= kTcMinSpins && global_ns() - t0 > kTcWaitNs) break;
    }
    atomicExch(&g_tc_abort, 1);
    atomicAdd(&g_tc_timeouts, 1);
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Shared-memory matrix descriptor: no swizzle (canonical K-major core matrices),
// leading byte offset = next K chunk, stride byte offset = next 8-row group,
// descriptor version 1 (bits 46-47).
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
__device__ __forceinline__ void umma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}
}  // namespace

}  // namespace bsim
