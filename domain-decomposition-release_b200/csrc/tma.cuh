// tma.cuh -- device helpers of the TMA-fed kernels: shared-memory barriers
// with bounded waits, and bulk tensor loads.
#pragma once

#include <cuda.h>

#include <cstdint>

namespace jv {

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint32_t bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// true when the phase with this parity has completed, false after ~1 s
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity) {
    long long t0 = 0;
    for (;;) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
        if (t0 == 0) t0 = clock64();  // the clock is read only by a wait that has to wait
        if (clock64() - t0 > 2000000000LL) return false;
    }
}
// A thread's reads of shared memory come before the bulk copies that refill
// it: executed by the reader before it gives the buffer back.  The barrier
// alone orders only ordinary accesses; without the fence late reads met the
// next plane (migrations of 144^3 differed from run to run in 31 of 200, with
// two kernels on the chip in every one).
__device__ __forceinline__ void reads_before_bulk_copies() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, int x, int y, int z, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::
            "r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(bar)
        : "memory");
}

}  // namespace jv
