// A CTA's own pipeline: mbarriers in shared memory and bulk copies that
// complete on them (the LU solve's producer warp, the wide update's).
#pragma once

#include "v2d_internal.cuh"

namespace v2d {
namespace {

__device__ __forceinline__ unsigned smem_addr(const void *p)
{
    return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long *b, int count)
{
    asm volatile("mbarrier.init.shared.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long *b)
{
    asm volatile("{\n.reg .b64 t;\nmbarrier.arrive.shared.b64 t, [%0];\n}" ::"r"(smem_addr(b))
                 : "memory");
}
// One arrival once the thread's earlier cp.async copies have landed.
__device__ __forceinline__ void mbar_arrive_copies(unsigned long long *b)
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];" ::"r"(smem_addr(b)) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned long long *b, unsigned bytes)
{
    asm volatile("{\n.reg .b64 t;\nmbarrier.arrive.expect_tx.shared.b64 t, [%0], %1;\n}" ::"r"(
                     smem_addr(b)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_test(unsigned long long *b, unsigned parity)
{
    unsigned ok;
    asm volatile("{\n.reg .pred p;\nmbarrier.test_wait.parity.shared.b64 p, [%1], %2;\n"
                 "selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok)
                 : "r"(smem_addr(b)), "r"(parity)
                 : "memory");
    return ok != 0;
}
// Waits between the threads of a CTA: they end when the CTA gives up (quit) or
// after 32 tests in a row and `limit` slower ones: false.  kPipeSpins of them
// take longer than kFlowSpins of the solve's waits on other CTAs, which a thread
// of this one may be in.
constexpr int kPipeSpins = 1 << 27;
__device__ __forceinline__ bool mbar_wait(unsigned long long *b, unsigned parity,
                                          volatile int *quit, int limit)
{
    for (int n = 0; n < 32; ++n)
        if (mbar_test(b, parity)) return true;
    for (int n = 0; n < limit && !(quit && *quit); ++n) {
        __nanosleep(32);
        if (mbar_test(b, parity)) return true;
    }
    return false;
}
// The same by a whole warp, with one answer for all of its lanes.
__device__ __forceinline__ bool mbar_wait_warp(unsigned long long *b, unsigned parity,
                                               volatile int *quit, int limit)
{
    return __all_sync(0xffffffffu, mbar_wait(b, parity, quit, limit));
}
// bytes (a multiple of 16) from src to dst, both 16-byte aligned; completes on b.
__device__ __forceinline__ void bulk_copy(void *dst, const void *src, unsigned bytes,
                                          unsigned long long *b)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_addr(dst)),
        "l"(src), "r"(bytes), "r"(smem_addr(b))
        : "memory");
}

}  // namespace
}  // namespace v2d
