// Work distribution of the kernels whose CTAs take many units in turn: cluster launch control (sm_100).
//
// A kernel is launched with one CTA per unit.  As many start as the GPU holds; each works on the unit of its own block index
// and then, instead of ending, cancels the launch of a CTA that has not started and takes that CTA's unit.  Against a grid of
// resident CTAs that walk the units with the grid's stride, the units at work stay a compact window that moves over the tensors
// whatever the speed of single CTAs: one that falls behind leaves no hole to be filled later, far behind the others.  DRAM
// serves that window faster.  Copies with the streams of a UF8/AL8 update (8 bytes read and 6 written per element; rings of two
// stages, six CTAs per SM) reached 5.9 and 6.2 TB/s over 64 M and 256 M elements with the stride, 6.5 and 6.8 this way; a
// counter in global memory that hands out the units does as well but has to be cleared before each launch.  Reads alone: 6.9
// and 7.1 TB/s.  A kernel bound by instruction issue gains nothing (the full-rank update: 1 to 3 %).
//
// One thread of the CTA asks and takes.  A request is answered in about a microsecond, so it is made a unit ahead.
#pragma once

#include "common.cuh"
#include "fullrank_fast.cuh"

namespace af8 {

constexpr int DEVERR_UNIT_TIMEOUT = 5;       // a request for the next unit was not answered

// A value that the whole warp read from the same place: the compiler takes what a shuffle broadcasts for uniform and keeps what
// follows from it (addresses, loop control) in uniform registers, as it does with block indices.
__device__ __forceinline__ int warp_uniform(int x) { return __shfl_sync(0xffffffffu, x, 0); }

struct __align__(16) UnitQueue {         // in shared memory, the asking thread's
    uint4 answer;
    uint64_t arrived;                    // mbarrier
    uint32_t phase;
    int32_t asked;                       // a request is on its way
};

__device__ __forceinline__ void unit_ask(UnitQueue &q)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], 16;\n\t"
                 "clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%1], [%0];"
                 ::"r"(smem_u32(&q.arrived)), "r"(smem_u32(&q.answer)) : "memory");
    q.asked = 1;
}
// the first request
__device__ __forceinline__ void unit_start(UnitQueue &q)
{
    mbar_init(&q.arrived, 1);
    q.phase = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    unit_ask(q);
}
// the unit that was asked for, or -1 when none is left
__device__ __forceinline__ int unit_read(const UnitQueue &q)
{
    uint32_t ok;
    int id;
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 lo, hi;\n\t.reg .b128 h;\n\t.reg .b32 y, z, w;\n\t"
                 "ld.shared.v2.b64 {lo, hi}, [%2];\n\tmov.b128 h, {lo, hi};\n\t"
                 "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\tmov.b32 %1, -1;\n\t"
                 "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%1, y, z, w}, h;\n\t}"
                 : "=r"(ok), "=r"(id) : "r"(smem_u32(&q.answer)) : "memory");
    return ok ? id : -1;
}
// The next unit of this CTA, or -1: none is left (and nothing is asked for after that).  The one after it is asked for.  An answer
// that does not come raises the error flag and counts as the last.
__device__ __forceinline__ int unit_take(UnitQueue &q)
{
    if (!q.asked) return -1;
    if (!mbar_wait_bounded(&q.arrived, q.phase)) {
        atomicExch(&g_device_error, DEVERR_UNIT_TIMEOUT);
        q.asked = 0;
        return -1;
    }
    q.asked = 0;
    q.phase ^= 1u;
    const int id = unit_read(q);
    if (id >= 0) {
        fence_proxy_async();                 // (the answer was read before it is written again)
        unit_ask(q);
    }
    return id;
}
// before the CTA leaves early: its request must not outlive its shared memory
__device__ __forceinline__ void unit_drain(UnitQueue &q)
{
    if (q.asked) mbar_wait_bounded(&q.arrived, q.phase);
    q.asked = 0;
}

}  // namespace af8
