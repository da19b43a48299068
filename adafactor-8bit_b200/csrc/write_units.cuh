// Write passes that need nothing of an element but its gradient, its parameter and factors of its row and column: units of
// 2048 consecutive elements of a table's tensors, taken by cluster launch control (schedule.cuh), through a ring of stages in shared
// memory.
//
// A fifth warp of the CTA takes the units, brings their gradients and parameters in (two bulk copies a unit, across tensors) and
// hands on with them what their tensor's elements need; the other four warps work.  (With requests made by one of those four, whose
// answers and descriptors it then waited for, the momentum-free Adafactor pass over 176 M parameters was 4 % slower than without any
// of this.)  A thread owns four groups of four elements, 512 apart, so that every access of a warp is one contiguous run.
#pragma once

#include "launch.cuh"
#include "schedule.cuh"

namespace af8 {

constexpr int WRITE_UNIT = 2048, WRITE_THREADS = 128, WRITE_STAGES = 3;
constexpr int DEVERR_WRITE_TIMEOUT = 6;
template <int GB, int PB> constexpr size_t write_smem_bytes() { return (size_t)WRITE_STAGES * WRITE_UNIT * (GB + PB); }

// A unit; kernels add what its tensor's elements need.
struct __align__(16) WriteUnit {
    int64_t base, row, col;          // flat index, row and column of its first element
    int64_t cols;
    void *param;
    const void *grad;
    int count;                       // elements; 0: no unit is left
    uint32_t magic;                  // floor(2^32 / cols) + 1: quotients by the column count
};
// row and column of the element o of a unit: a long row ends once in a unit at most, a short one has columns below 2^12 here
__device__ __forceinline__ void write_position(const WriteUnit &U, int o, int64_t &row, int64_t &col)
{
    const int64_t C = U.cols;
    col = U.col + o;
    row = U.row;
    if (C >= WRITE_UNIT) {
        if (col >= C) { col -= C; ++row; }
    } else {
        const uint32_t down = __umulhi((uint32_t)col, U.magic);
        row += down;
        col = (uint32_t)col - down * (uint32_t)C;
    }
}

template <typename Unit>
struct WriteShared {
    Unit unit[WRITE_STAGES];
    UnitQueue queue;
    uint64_t full[WRITE_STAGES], free[WRITE_STAGES];
    int abort;
};

// Tensors: first(t) the number of the first unit of tensor t (ascending), count() tensors, load(t, U) sets what does not depend on the
// unit (but magic) and returns the number of elements, a multiple of 8.
// work(U, stage, release): a unit whose copies have landed, gradients first, parameters after them; release() once the thread has read
// the stage and U (a warp's lanes together).
template <int GB, int PB, typename Unit, typename Tensors, typename Work>
__device__ __forceinline__ void write_units(const Tensors &tensors, WriteShared<Unit> &sh, unsigned char *ring, Work work)
{
    constexpr int P_OFF = WRITE_UNIT * GB, STAGE = WRITE_UNIT * (GB + PB), NS = WRITE_STAGES;
    const int tid = threadIdx.x;
    if (tid == WRITE_THREADS) {
        for (int k = 0; k < NS; ++k) { mbar_init(&sh.full[k], 1); mbar_init(&sh.free[k], WRITE_THREADS / 32); }
        sh.abort = 0;
        unit_start(sh.queue);
    }
    __syncthreads();
    await_launches();

    if (tid >= WRITE_THREADS) {
        if (tid != WRITE_THREADS) return;
        int t = -1;
        int64_t first = 0, end = 0, numel = 0;
        Unit U = {};
        int id = (int)blockIdx.x;
        for (uint32_t n = 0;; ++n) {
            const int sl = (int)(n % NS);
            if (n >= NS && !mbar_wait_bounded(&sh.free[sl], (n / NS + 1) & 1u)) { sh.abort = 1; atomicExch(&g_device_error, DEVERR_WRITE_TIMEOUT); }
            const bool given_up = *static_cast<volatile int *>(&sh.abort) != 0;
            if (id < 0 || given_up) {
                unit_drain(sh.queue);
                if (given_up)                                        // the copies in flight get a bounded chance to land before the CTA may end
                    for (uint32_t k = n > NS ? n - NS : 0; k < n; ++k) mbar_wait_bounded(&sh.full[k % NS], (k / NS) & 1u);
                sh.unit[sl].count = 0;
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&sh.full[sl])) : "memory");
                return;
            }
            if (t < 0 || id < first || id >= end) {
                if (t < 0 || id < first) {
                    int lo = 0, hi = tensors.count() - 1;
                    while (lo < hi) {
                        const int mid = (lo + hi + 1) >> 1;
                        if (tensors.first(mid) <= id) lo = mid; else hi = mid - 1;
                    }
                    t = lo;
                } else while (t + 1 < tensors.count() && tensors.first(t + 1) <= id) ++t;
                first = tensors.first(t);
                numel = tensors.load(t, U);
                end = first + (numel + WRITE_UNIT - 1) / WRITE_UNIT;
                U.magic = (uint32_t)(0x100000000ull / (uint64_t)U.cols) + 1u;
            }
            U.base = (id - first) * WRITE_UNIT;
            U.count = (int)min((int64_t)WRITE_UNIT, numel - U.base);
            U.row = (numel >> 32) == 0 ? (int64_t)((uint32_t)U.base / (uint32_t)U.cols) : U.base / U.cols;
            U.col = U.base - U.row * U.cols;
            sh.unit[sl] = U;
            fence_proxy_async();
            mbar_expect_tx(&sh.full[sl], (uint32_t)(U.count * (GB + PB)));
            bulk_g2s(ring + sl * STAGE + P_OFF, static_cast<const unsigned char *>(U.param) + U.base * PB, (uint32_t)(U.count * PB), &sh.full[sl]);
            bulk_g2s(ring + sl * STAGE, static_cast<const unsigned char *>(U.grad) + U.base * GB, (uint32_t)(U.count * GB), &sh.full[sl]);
            id = unit_take(sh.queue);
        }
    }

    for (uint32_t n = 0;; ++n) {
        const int sl = (int)(n % NS);
        const bool landed = mbar_wait_bounded(&sh.full[sl], (n / NS) & 1u);
        if (!landed) { sh.abort = 1; atomicExch(&g_device_error, DEVERR_WRITE_TIMEOUT); }
        const Unit &U = sh.unit[sl];
        if (warp_uniform(U.count) == 0) break;
        const auto release = [&]() {
            __syncwarp();
            if ((tid & 31) == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&sh.free[sl])) : "memory");
        };
        if (__all_sync(0xffffffffu, landed)) work(U, ring + sl * STAGE, release);
        else release();                                              // (nothing is written from a copy that never came)
    }
}

}  // namespace af8
