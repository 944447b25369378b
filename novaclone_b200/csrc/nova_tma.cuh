// sm_100a primitives of the TMA-fed stage pipeline: mbarriers in shared
// memory and tiled bulk tensor loads (cp.async.bulk.tensor, no multicast).
//
// Every wait is bounded: after kWaitLimitNs (or 2^26 polls) without the phase
// completing, or when another thread has already raised the error word, the
// wait sets *err = 1 and returns false, and the caller leaves its pipeline.
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <cstdint>
#include <type_traits>

#include "nova_regsplit.h"

namespace nova {

constexpr unsigned long long kWaitLimitNs = 1000000000ull;  // 1 s

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

// makes the initialised barriers visible to the async (TMA) proxy
__device__ __forceinline__ void mbar_init_fence()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// wait for the phase of parity `parity` to complete; false on timeout or when
// *err is already raised (abandon = true: ignore *err, used while draining)
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int *err, bool abandon = false)
{
    if (mbar_test(bar, parity)) return true;
    const unsigned long long t0 = global_ns();
    for (unsigned it = 1; it < (1u << 26); it++) {
        if (mbar_test(bar, parity)) return true;
        if ((it & 255u) == 0) {
            if (!abandon && *(volatile int *)err) return false;
            if (global_ns() - t0 > kWaitLimitNs) break;
        }
    }
    atomicExch(err, 1);
    return false;
}

// 4-D tiled load of the tensor map's box at (c0..c3) into shared memory at
// dst; completion is signalled on bar as transaction bytes
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c0, int c1, int c2,
                                            int c3)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], "
        "[%2];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
        : "memory");
}

// the driver's cuTensorMapEncodeTiled, looked up once through the runtime
// (no link against libcuda); null when the driver does not export it
inline PFN_cuTensorMapEncodeTiled_v12000 tma_encode_tiled()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = []() -> PFN_cuTensorMapEncodeTiled_v12000 {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return nullptr;
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }();
    return fn;
}

// Registers of a warp-specialised kernel: CONSUMERS threads rise to INC, PRODUCERS
// (whole warpgroups) fall to DEC.
template <int CONSUMERS, int INC, int PRODUCERS, int DEC> struct RegSplit {
    static_assert(CONSUMERS % 128 == 0 && PRODUCERS % 128 == 0, "setmaxnreg is executed by whole warpgroups");
    static constexpr int kThreads = CONSUMERS + PRODUCERS;
    __device__ static void consumer() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(INC)); }
    __device__ static void producer() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(DEC)); }
};

// whether the registers the compiler gave `kern` cover the split (before its
// first launch: the consumers' wait for them has no bound)
template <int CONSUMERS, int INC, int PRODUCERS, int DEC, class Kern>
cudaError_t reg_split_ok(RegSplit<CONSUMERS, INC, PRODUCERS, DEC>, Kern kern)
{
    cudaFuncAttributes at;
    const cudaError_t e = cudaFuncGetAttributes(&at, kern);
    if (e != cudaSuccess) return e;
    return reg_split_fits(at.numRegs, CONSUMERS, INC, PRODUCERS, DEC) ? cudaSuccess : cudaErrorInvalidConfiguration;
}

// step(R, m, p) for the planes p = PERIOD m + R < n in order (R an integral_constant,
// so that ring slots and queue positions are compile-time constants), until one
// returns false
template <int PERIOD, int R, class Step> __device__ __forceinline__ bool march_period(int n, int m, int p, Step &step)
{
    if (!step(std::integral_constant<int, R>{}, m, p + R)) return false;
    if constexpr (R + 1 < PERIOD)
        return p + R + 1 >= n || march_period<PERIOD, R + 1>(n, m, p, step);
    else
        return true;
}
template <int PERIOD, class Step> __device__ __forceinline__ bool march_unrolled(int n, Step &step)
{
    bool ok = true;
    for (int m = 0, p = 0; ok && p < n; m++, p += PERIOD) ok = march_period<PERIOD, 0>(n, m, p, step);
    return ok;
}

// 3-D tiled load (a single component of a field: dims k, j, i)
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c0, int c1, int c2)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], "
        "[%2];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}

}  // namespace nova
