// Inline-PTX helpers for sm_103a: bulk (1-D) TMA copies between global and
// shared memory completed through an mbarrier, and bounded waits that give up
// with an error flag instead of spinning forever.
#pragma once
#include <cstdint>

namespace mhd {

// Device error bits (ORed into the context's error word).
enum : int {
    DEVERR_TIMEOUT = 1,   // a bounded mbarrier wait expired
    DEVERR_NONFINITE = 2, // the CFL reduction met a NaN speed
};

// About one second at 2 GHz; a TMA copy of a few KB completes in microseconds.
constexpr long long kWaitLimitCycles = 2000000000LL;

__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Programmatic dependent launch.  Every kernel of a step is launched with
// launch_after (below).  It begins with after_previous(), which waits until the
// kernel before it has completed and its writes are visible (at once in a plain
// launch); no global memory is touched before that.  Where a CTA has little left
// to do it calls before_next(): once all CTAs have (or have ended), the next
// kernel is brought in, so its launch overlaps this one's last stores.  Called
// at the start instead, the next kernel's CTAs fill the SMs that happen to be free
// first and a grid of less than a wave spreads unevenly.  Ten plain 64^3 steps / two
// EXACT 96^3 / four 100x72x72 / four corrected 64^3: 1.02, 1.15, 1.08, 1.52 ms
// without any of this, 1.11, 1.11, 1.02, 1.39 with before_next at the start, 1.02,
// 1.11, 1.03, 1.33 as it is.
__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void before_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// What a dependent kernel may read, and how: it is live while the kernels before it still
// write, so data that another kernel writes (state, side arrays, partials, flags,
// activations, weights, dt) is read after after_previous() through plain loads or
// asynchronous copies.  __ldg and __restrict__ promise the compiler and the read-only path
// that the data is constant for the kernel's lifetime; they are kept for constant tables.
// Loops therefore load what they need before they store (a store may alias a later load).

// src to dst by the whole grid, four loads in flight a thread (the compiler cannot
// move a load above a store that may alias it).
template <typename V>
__device__ __forceinline__ void copy_strided(const V* src, V* dst, size_t n)
{
    const size_t step = (size_t)gridDim.x * blockDim.x;
    size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (; e + 3 * step < n; e += 4 * step) {
        const V x0 = src[e], x1 = src[e + step], x2 = src[e + 2 * step], x3 = src[e + 3 * step];
        dst[e] = x0;
        dst[e + step] = x1;
        dst[e + 2 * step] = x2;
        dst[e + 3 * step] = x3;
    }
    for (; e < n; e += step)
        dst[e] = src[e];
}

// A launch that may start while the one before it in the stream drains; the
// kernel begins with after_previous().  Captured into a graph it becomes a
// programmatic edge.  Returns the launch's error.
template <typename... P, typename... A>
static cudaError_t launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args)
{
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
    if (e != cudaSuccess)
        (void)cudaGetLastError();  // it is the caller's: not left for whoever asks next
    return e;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Waits for the phase with the given parity; returns false (and records
// DEVERR_TIMEOUT) if it has not completed within `limit` SM cycles.
__device__ __forceinline__ bool mbar_wait_limit(uint64_t* bar, uint32_t parity, int* err, long long limit)
{
    if (mbar_try_wait(bar, parity))
        return true;
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (clock64() - t0 > limit) {
            if (err)
                atomicOr(err, DEVERR_TIMEOUT);
            return false;
        }
    }
    return true;
}

// The same with the kernels' limit, kWaitLimitCycles.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, int* err)
{
    return mbar_wait_limit(bar, parity, err, kWaitLimitCycles);
}

// Global -> shared bulk copy; dst, src 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void tma_load_1d(void* dst, const void* src, uint32_t bytes, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// Shared -> global bulk copy, tracked by the issuing thread's bulk group.
__device__ __forceinline__ void tma_store_1d(void* dst, const void* src, uint32_t bytes)
{
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
                 "r"(smem_u32(src)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }

// Wait until the committed bulk stores have finished reading shared memory.
__device__ __forceinline__ void tma_store_wait_read()
{
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

// Wait until the committed bulk stores are complete (visible in global memory).
__device__ __forceinline__ void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// Make generic-proxy writes to shared memory visible to the async (TMA) proxy.
__device__ __forceinline__ void fence_proxy_async_smem()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Tiled 3-D tensor copies (cp.async.bulk.tensor) through a tensor map that
// lives in kernel parameter space (a __grid_constant__ argument); coordinates
// are in elements, innermost first.  The load completes on an mbarrier, the
// store joins the issuing thread's bulk group.  The shared buffer is 128-byte
// aligned and the innermost coordinate times the element size a multiple of
// 16 bytes (checked by the callers' planners).
__device__ __forceinline__ void tma_load_3d(void* dst, const void* tmap, int c0, int c1, int c2, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(tmap)), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tma_load_2d(void* dst, const void* tmap, int c0, int c1, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
        "[%4];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(tmap)), "r"(c0), "r"(c1), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tma_store_3d(const void* tmap, int c0, int c1, int c2, const void* src)
{
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(
                     reinterpret_cast<uint64_t>(tmap)),
                 "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(src))
                 : "memory");
}

// 4- and 8-byte asynchronous global -> shared copies (per thread; completion through
// cp.async groups), used where a tile must be scattered element by element.
__device__ __forceinline__ void cp_async4(void* dst, const void* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
// 16-byte asynchronous global -> shared copy, not cached in L1 (both
// addresses 16-byte aligned).
__device__ __forceinline__ void cp_async16(void* dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

}  // namespace mhd
