// Launches that follow one another closely: programmatic dependent launch, table uploads and clears as kernels.
//
// A step of a small model is a chain of ten to twenty short launches.  A kernel launched with launch_next may start while the
// kernel before it in the stream still runs, as soon as all CTAs of that one are past await_launches() and leave room, and waits there
// itself until it has completed and its writes are visible: what a launch costs before its first instruction overlaps.  (A chain of
// kernels of 10 us with 888 CTAs: 14.3 us a kernel with plain launches, 11.8 at best.)  Every CTA calls await_launches() before it
// touches global memory, so that a kernel is complete only after all before it are, and whatever follows in the stream
// without the attribute (copies, events, other libraries' kernels) waits for it as always.  No more than two kernels overlap.
// These kernels read with ordinary loads alone.  A read-only load (__ldg, a const __restrict__ parameter) asks that nobody writes the
// memory during the reading kernel's lifetime, which begins here while the kernel before may still write it, and the compiler may move
// it in front of the wait.
//
// A table copied by the copy engine between two kernels holds them up for 13 us (6 below 1 KB); read from pinned memory by a kernel, before
// it waits, 1.5 to 4 us for 1 to 52 KB.  A memset costs 5 us there, a kernel that clears 2.
#pragma once

#include "common.cuh"

namespace af8 {

__device__ __forceinline__ void await_launches()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// An ordinary load that stores in between need not hold up, as a read-only one: what the kernels load a block or a row ahead, and what
// no thread writes before it was used.  (As *p the UF8/AL8 update spills 30 to 80 bytes and the sums over ragged rows take 94 us instead of 90;
// without `volatile` the general kernel's sums take 48 registers instead of 32, 638 -> 774 us for 67 M parameters.)
__device__ __forceinline__ float load_state(const float *p)
{
    float x;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(x) : "l"(p));
    return x;
}
__device__ __forceinline__ float4 load_state(const float4 *p)
{
    float4 x;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w) : "l"(p));
    return x;
}
__device__ __forceinline__ uint4 load_state(const uint4 *p)
{
    uint4 x;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w) : "l"(p));
    return x;
}

template <typename... Params, typename... Args>
inline cudaError_t launch_next(void (*kernel)(Params...), dim3 grid, int block, size_t smem, cudaStream_t st, const Args &...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

// MAPS: the table holds tensor maps.  They are read through a proxy of their own, which tensormap_acquire on the reading side orders behind
// a release on this one.
template <bool MAPS>
__global__ void __launch_bounds__(256)
upload_kernel(const uint2 *host, uint2 *dev, int n)         // n units of 8 bytes
{
    const int i = 2 * (blockIdx.x * 256 + threadIdx.x);
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (i + 1 < n) asm volatile("ld.global.cv.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(host + i));
    else if (i < n) asm volatile("ld.global.cv.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(host + i));
    await_launches();                                        // (kernels before this one may still read the table)
    if (i + 1 < n) *reinterpret_cast<uint4 *>(dev + i) = v;
    else if (i < n) dev[i] = make_uint2(v.x, v.y);
    if (MAPS) asm volatile("fence.proxy.tensormap::generic.release.sys;" ::: "memory");
}

// Enqueues the copy of a table.  `host` stays as it is until the copy has run.  Pinned tables on 16-byte boundaries that the device can
// read are copied by a kernel, any other memory by the copy engine.  (APOLLO's write-back table has 104 bytes a tensor: whole units of 8.)
template <bool MAPS = false>
inline int upload_table(void *dev, const void *host, size_t bytes, cudaStream_t st)
{
    cudaPointerAttributes a = {};
    const bool units = ((reinterpret_cast<uintptr_t>(dev) | reinterpret_cast<uintptr_t>(host)) & 15) == 0 && (bytes & 7) == 0 && bytes < (1u << 20);
    if (units && cudaPointerGetAttributes(&a, host) != cudaSuccess) {
        cudaGetLastError();                                  // (the question's own error, not one that is waiting for the caller)
        a = {};
    }
    if (units && a.type == cudaMemoryTypeHost && a.devicePointer != nullptr) {
        const int n = (int)(bytes / 8);
        AF8_CUDA_TRY(launch_next(upload_kernel<MAPS>, (n + 511) / 512, 256, 0, st, static_cast<const uint2 *>(a.devicePointer), static_cast<uint2 *>(dev), n));
        return AF8_OK;
    }
    AF8_CUDA_TRY(cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, st));
    return AF8_OK;
}

__global__ void __launch_bounds__(256)
clear_kernel(double *a, int64_t na, double *b, int64_t nb)
{
    await_launches();
    const int64_t stride = (int64_t)gridDim.x * 256, first = (int64_t)blockIdx.x * 256 + threadIdx.x;
    for (int64_t i = first; i < na; i += stride) a[i] = 0.0;
    for (int64_t i = first; i < nb; i += stride) b[i] = 0.0;
}
// zeros into one or two arrays of doubles
inline int clear_doubles(double *a, int64_t na, double *b, int64_t nb, cudaStream_t st)
{
    const int64_t most = na > nb ? na : nb, grid = (most + 1023) / 1024;
    AF8_CUDA_TRY(launch_next(clear_kernel, (unsigned)(grid < 1184 ? grid : 1184), 256, 0, st, a, na, b, nb));
    return AF8_OK;
}

}  // namespace af8
