// tma_common.cuh -- Tensor Memory Accelerator helpers of the smoothing passes:
// mbarrier and copy wrappers with bounded waits, aligned shared memory and the
// tensor-map encoder.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>

namespace mhdproj {
namespace tma {

constexpr int WAIT_LIMIT = 1 << 22;

// ------------------------------------------------------------- PTX wrappers
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* b, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_barrier_init() { asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory"); }
// Orders this thread's (and, after a barrier, the block's) generic-proxy
// accesses of shared memory before the copies it issues next.
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* b, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* b, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait for the phase of the given parity; false when it ran out.
__device__ __forceinline__ bool mbar_wait(unsigned long long* b, unsigned parity) {
    for (int i = 0; i < WAIT_LIMIT; i++)
        if (mbar_try_wait(b, parity)) return true;
    return false;
}
__device__ __forceinline__ void tma_3d(void* dst, const CUtensorMap* tm, int x, int y, int z, unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];\n" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<unsigned long long>(tm)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void tma_4d(void* dst, const CUtensorMap* tm, int x, int h, int y, int z,
                                       unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
        "%5}], [%6];\n" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<unsigned long long>(tm)), "r"(x), "r"(h), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}

template <class SM>
__device__ __forceinline__ SM& aligned_smem(unsigned char* raw) {
    return *reinterpret_cast<SM*>(raw + ((128u - (smem_u32(raw) & 127u)) & 127u));
}

// cuTensorMapEncodeTiled, nullptr when the driver has none.
PFN_cuTensorMapEncodeTiled_v12000 encoder();

}  // namespace tma
}  // namespace mhdproj
