// Device primitives shared by the stacking kernels: mbarriers and TMA copies
// with a bounded wait, the order-preserving (S/N, motion) keys of a tile's
// shared maximum, and the tensor-map encoder of the host side.
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace ftb {

// cuTensorMapEncodeTiled from the driver (throws when it is not available)
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder();

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
            smem_addr(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_addr(bar))
        : "memory");
}

// The tensor maps of a launch lie in global memory, at an address that earlier launches
// used for other maps: a copy from the host wrote them, and the loads read them through
// the tensor-map proxy. One fence a map, by the CTA's threads in turn, orders the two; the
// CTA's barrier has to follow before the first load.
__device__ __forceinline__ void tensor_maps_acquire(const CUtensorMap* maps, int count) {
    for (int k = static_cast<int>(threadIdx.x); k < count; k += static_cast<int>(blockDim.x))
        asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(reinterpret_cast<uint64_t>(maps + k))
                     : "memory");
}

__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Bounded wait on the staging barrier: `limit` clock cycles (about two seconds
// by default), then the kernel records an error and gives up (the host turns it
// into an exception).
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, int* err, long long limit) {
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (clock64() - t0 > limit) {
            atomicExch(err, 1);
            return false;
        }
    }
    return true;
}

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_addr(dst)),
        "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_addr(bar))
        : "memory");
}

// A tile's shared maximum: key = (order-preserving bits of S/N) << 32 | (~index) << 1 |
// sign, so a larger S/N wins and equal S/N goes to the lower motion index. The two zeros
// are equal (+ 0.0f gives both the bits of +0); the winner's own sign is in the lowest bit.
__device__ __forceinline__ unsigned long long snr_key(float s, int j) {
    const uint32_t b = __float_as_uint(__fadd_rn(s, 0.0f));
    const uint32_t o = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
    return (static_cast<unsigned long long>(o) << 32) |
           __funnelshift_l(__float_as_uint(s), ~static_cast<uint32_t>(j), 1);
}

__device__ __forceinline__ void snr_unkey(unsigned long long k, float& s, int& j) {
    const uint32_t o = static_cast<uint32_t>(k >> 32), low = static_cast<uint32_t>(k);
    s = __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) | low << 31 : ~o);
    j = static_cast<int>(low >> 1 ^ 0x7fffffffu);
}

}  // namespace ftb
