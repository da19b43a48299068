// APOLLO projection on the fifth-generation tensor cores.  "Right" case (rows >= cols):
//   g_low[M x N] = G[M x K] @ Pt[K x N],   M = rows, K = cols, N = rank
// "Left" case (rows < cols), as the transposed problem:
//   g_low^T[M x N] = G^T[M x K] @ P^T[K x N],   M = cols, K = rows
// with the same three-plane bf16 split of Pt as apollo_mma.cuh.  tcgen05.mma reads both
// operands from shared memory and accumulates in tensor memory (TMEM).
//
// Operands are K-major with the 64-byte swizzle: a stage holds 32 values of K, i.e. rows of
// 64 bytes, written by tiled bulk tensor copies (TMA) whose tensor maps use
// CU_TENSOR_MAP_SWIZZLE_64B; the matrix descriptors name the same swizzle, 512 bytes between
// 8-row groups, and advance by 32 bytes per 16 values of K.  The gradient already has K
// contiguous; the planes of Pt are written transposed ([3][N][K]) by the split kernel and
// arrive with one three-dimensional copy per stage.
// In the left case the gradient has M contiguous: a stage of it is two boxes of 32 rows (K) x 64 columns (128 bytes,
// 128-byte swizzle), an M-major operand.  (A separate transposition of such gradients, 52 us per Llama-3-8B layer, and
// their second trip through memory are gone with it.)
//
// Two SMs share a tile of 256 rows wherever the instruction allows it (cta_group::2, ranks of whole 32s; CG = 2 below): each holds its 128
// rows of the gradient, half of the columns of Pt and the totals of its rows; the first CTA of the pair issues the MMAs for both.  One SM
// alone reads 56 KB of operands a stage from L2 and 72 KB from shared memory, one of a pair 32 and 48.  That alone changed
// nothing (four Llama-3-8B layers, rank 256: 1308 -> 1307 us): the stage was as long as the workers' pass over it, a chain of a
// wait, loads, eight dependent sums, conversion and addition in binary64, 1170 of 1700 cycles.  They now read two
// stages at a time, whose chains overlap: 1164 us (four at a time spill registers: 1209; two in one SM alone, which has four stages: 1273).
// Without the pass 1106, without copies of the planes either 1030; at the 1.3 to 1.5 GHz that the power limit leaves the
// MMAs themselves, at the measured bf16 rate, take 800 (a burst) to 960 us.
//
// CTA = 320 threads, one CTA per SM, persistent over (task, M tile) pairs:
//   warps 0-7  read every gradient tile from shared memory before its MMAs: they add up the
//              squares of each row of M (the channel norms ||G_row||^2 that the scaling step needs,
//              so the gradient is read from memory once) and zero non-finite entries; then
//              drain the accumulator: warp w owns TMEM lanes 32 (w % 4) .. +31 and columns
//              128 (w / 4) .. +127, 128 totals per thread; then store g_low and the norms.
//   warp 8     allocates / frees TMEM; its lane 0 issues the MMAs and the commits
//   warp 9     lane 0 issues the copies
// Four 56 KB stages, of a pair seven of 32 KB; a "full" barrier completes on the copies' transaction bytes, a "clean"
// barrier of the issuing CTA when the worker warps (of both) have read (and, rarely, repaired) the gradient tile, an "empty"
// barrier (of both) on tcgen05.commit.
//
// The tensor cores add into their binary32 accumulators with truncation, whose error grows
// linearly with K (measured 1.4e-5 relative at K = 4096, as with mma.sync).  The accumulation
// is therefore cut into chunks of 256 values of K that alternate between two TMEM accumulators;
// while one is being filled the other is added, with rounding, into the workers' registers.
//
// Every wait is bounded (two seconds of %globaltimer); on a time-out the thread raises the
// device error flag and leaves; the others follow at their next wait or tile, and the tensor
// memory is freed after all have reported (or after a bounded wait).  After the start-up
// barrier no block-wide barrier is used, so a lost role cannot hang the others (a pair meets once more at the end, when every wait is over).  No copy
// uses cluster multicast.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>

#include "common.cuh"
#include "fullrank_fast.cuh"     // mbarrier helpers, g_device_error
#include "tensormap.cuh"         // tiled bulk tensor copies
#include "apollo_mma.cuh"        // ProjTask, clean_chunk

namespace af8 {

constexpr int UM_BM = 128, UM_BK = 32, UM_THREADS = 320, UM_WORKERS = 256, UM_MMA_WARP = 8, UM_TMA_WARP = 9;
template <int CG> __host__ __device__ constexpr int um_stages() { return CG == 2 ? 7 : 4; }
template <int CG> __host__ __device__ constexpr int um_scan() { return CG == 2 ? 2 : 1; }      // stages that the workers read at a time
constexpr int UM_PAIR_N = 32;      // a pair takes ranks that are multiples of this
constexpr int UM_FLUSH = 8;        // stages (256 values of K) per accumulator chunk
constexpr int UM_MAXN = 256;
constexpr int UM_ROW_BYTES = UM_BK * 2;                       // 64
constexpr int UM_A_BYTES = UM_BM * UM_ROW_BYTES;              // 8 KB (a multiple of 1024, like a stage: the 128-byte swizzle's period)
constexpr int UM_B_BYTES = UM_MAXN * UM_ROW_BYTES;            // 16 KB per plane at N = 256
template <int CG> __host__ __device__ constexpr int um_stage_bytes() { return UM_A_BYTES + 3 * UM_B_BYTES / CG; }   // 56 KB; of a pair: 32 KB in each SM
constexpr int UM_SBO = 8 * UM_ROW_BYTES;                      // 512 bytes between 8-row groups
constexpr int DEVERR_UMMA_TIMEOUT = 2;

// One projection of a tcgen05 launch: the mma.sync task plus the two tensor maps
struct __align__(64) UmmaTask {
    CUtensorMap map_a;       // right: G as [M][K], box 128 x 32; left: G as [K][M], box 32 x 64
    CUtensorMap map_b;       // planes as [3][N][K], box 3 x N x 32 (of a pair: 3 x N/2 x 32)
    ProjTask t;
    double *chan_g2;         // [M] sums of squares of the rows of G (non-finite entries count as zero)
    unsigned char pad[384 - 2 * sizeof(CUtensorMap) - sizeof(ProjTask) - sizeof(double *)];
};
static_assert(sizeof(CUtensorMap) == 128 && sizeof(UmmaTask) == 384, "task layout");

__device__ __forceinline__ uint64_t umma_smem_desc(uint32_t smem_addr)
{
    // start address and stride byte offset in units of 16 bytes (the leading byte offset is not
    // used by swizzled K-major layouts); descriptor version 1; layout type 4 = 64-byte swizzle
    return (uint64_t)((smem_addr >> 4) & 0x3fffu) | ((uint64_t)1 << 16) | ((uint64_t)(UM_SBO >> 4) << 32) |
           (1ull << 46) | (4ull << 61);
}
// M-major A with the 128-byte swizzle: blocks of 64 values of M x 8 of K (1024 bytes); 4096 bytes to the next 64 values
// of M (a box), 1024 bytes to the next 8 of K; layout type 2 = 128-byte swizzle
constexpr int UM_LEFT_BOX_M = 64, UM_LEFT_BOX_BYTES = UM_BK * UM_LEFT_BOX_M * 2;
__device__ __forceinline__ uint64_t umma_smem_desc_left(uint32_t smem_addr)
{
    return (uint64_t)((smem_addr >> 4) & 0x3fffu) | ((uint64_t)(UM_LEFT_BOX_BYTES >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) |
           (1ull << 46) | (2ull << 61);
}
// kind::f16 instruction descriptor: D = F32, A = B = BF16, B K-major, A K-major or (bit 15) M-major, M = 128 (a pair: 256), N = n
template <int CG>
__device__ __forceinline__ uint32_t umma_instr_desc(int n, bool a_m_major)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | (a_m_major ? 1u << 15 : 0u) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(CG * UM_BM >> 4) << 24);
}
template <int CG>
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    if (CG == 2)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                     ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                     ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// arrives on the barrier (of a pair: on that of both CTAs) when the MMAs issued so far are done
template <int CG>
__device__ __forceinline__ void umma_commit(uint64_t *bar)
{
    if (CG == 2)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                     ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
    else
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ uint32_t cluster_rank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// every thread of both CTAs
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
// Arrives on the same barrier of the pair's first CTA.  At the default scope: what the other side reads after it was written by copies
// that this thread has seen complete, in the SM that reads it; a generic write before it takes fence_cluster.  (With release and acquire at
// cluster scope each arrival waits for the thread's other accesses: 1.3 ms become 2.4.)
__device__ __forceinline__ void mbar_arrive_first(uint64_t *bar)
{
    asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %0, 0;\n\t"
                 "mbarrier.arrive.shared::cluster.b64 _, [a];\n\t}" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void fence_cluster() { asm volatile("fence.acq_rel.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// Pt[K][N] (fp32) -> three bf16 planes stored [N][K]
__global__ void __launch_bounds__(256)
apollo_split_transposed_kernel(const float *__restrict__ p, int K, int N, __nv_bfloat16 *__restrict__ planes)
{
    __shared__ float tile[32][33];
    const int k0 = blockIdx.x * 32, n0 = blockIdx.y * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;     // 32 x 8
    for (int r = ty; r < 32; r += 8) {
        const int k = k0 + r, n = n0 + tx;
        tile[r][tx] = (k < K && n < N) ? p[(int64_t)k * N + n] : 0.0f;
    }
    __syncthreads();
    const int64_t plane = (int64_t)K * N;
    for (int r = ty; r < 32; r += 8) {
        const int n = n0 + r, k = k0 + tx;
        if (n < N && k < K) {
            const float x = tile[tx][r];
            const __nv_bfloat16 h1 = __float2bfloat16_rn(x);
            const float r1 = __fsub_rn(x, __bfloat162float(h1));
            const __nv_bfloat16 h2 = __float2bfloat16_rn(r1);
            const float r2 = __fsub_rn(r1, __bfloat162float(h2));
            const int64_t o = (int64_t)n * K + k;
            planes[o] = h1;
            planes[plane + o] = h2;
            planes[2 * plane + o] = __float2bfloat16_rn(r2);
        }
    }
}

__device__ __forceinline__ int volatile_load(const int *p) { return *reinterpret_cast<const volatile int *>(p); }

// Sum of squares of the 8 bf16 values of a 16-byte chunk of a staged gradient tile.  The common
// case is eight binary32 multiply-adds; when that sum is not finite (a NaN or an infinity in the
// chunk, or squares beyond binary32) the non-finite entries are zeroed in shared memory, as the
// reference zeroes them in the gradient (optimizer.py:2606), and the sum is redone in binary64.
__device__ __forceinline__ float umma_chunk_sum(uint4 v)
{
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    float s = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float lo = __uint_as_float(w[i] << 16), hi = __uint_as_float(w[i] & 0xffff0000u);
        s = __fmaf_rn(lo, lo, s);
        s = __fmaf_rn(hi, hi, s);
    }
    return s;
}
__device__ __noinline__ double umma_chunk_sumsq(unsigned char *p, bool &wrote)
{
    const uint4 v = *reinterpret_cast<uint4 *>(p);
    uint32_t w[4] = {v.x, v.y, v.z, v.w};
    const float s = umma_chunk_sum(v);
    if (s <= 3.0e38f) return (double)s;                          // false for NaN and infinity
    bool changed = false;
    double d = 0.0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if ((w[i] & 0x7f80u) == 0x7f80u) { w[i] &= 0xffff0000u; changed = true; }
        if ((w[i] & 0x7f800000u) == 0x7f800000u) { w[i] &= 0x0000ffffu; changed = true; }
        const double lo = (double)__uint_as_float(w[i] << 16), hi = (double)__uint_as_float(w[i] & 0xffff0000u);
        d += lo * lo;
        d += hi * hi;
    }
    if (changed) {
        *reinterpret_cast<uint4 *>(p) = make_uint4(w[0], w[1], w[2], w[3]);
        wrote = true;
    }
    return d;
}

// Left case: the 4 values of half a 16-byte chunk belong to 4 rows of M.  Their squares are added to acc[4] in binary32 (the
// caller passes the sums on to binary64 after at most 8 values); where a magnitude from 2^60 up makes squares that might
// leave binary32, they go into wide[4] in binary64, and non-finite entries are zeroed in shared memory as above.
__device__ __forceinline__ void umma_quad_add(uint2 v, float (&acc)[4])
{
    const uint32_t w[2] = {v.x, v.y};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const float lo = __uint_as_float(w[i] << 16), hi = __uint_as_float(w[i] & 0xffff0000u);
        acc[2 * i] = __fmaf_rn(lo, lo, acc[2 * i]);
        acc[2 * i + 1] = __fmaf_rn(hi, hi, acc[2 * i + 1]);
    }
}
__device__ __forceinline__ void umma_quad_squares(unsigned char *p, float (&acc)[4], double (&wide)[4], bool &wrote)
{
    const uint2 v = *reinterpret_cast<const uint2 *>(p);
    uint32_t w[2] = {v.x, v.y};
    const uint32_t top = __vmaxu2(w[0] & 0x7fff7fffu, w[1] & 0x7fff7fffu);
    if ((top >> 16) < 0x5d80u && (top & 0xffffu) < 0x5d80u) {
        umma_quad_add(v, acc);
        return;
    }
    bool changed = false;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        if ((w[i] & 0x7f80u) == 0x7f80u) { w[i] &= 0xffff0000u; changed = true; }
        if ((w[i] & 0x7f800000u) == 0x7f800000u) { w[i] &= 0x0000ffffu; changed = true; }
        const double lo = (double)__uint_as_float(w[i] << 16), hi = (double)__uint_as_float(w[i] & 0xffff0000u);
        wide[2 * i] += lo * lo;
        wide[2 * i + 1] += hi * hi;
    }
    if (changed) {
        *reinterpret_cast<uint2 *>(p) = make_uint2(w[0], w[1]);
        wrote = true;
    }
}

template <int CG>
__global__ void __launch_bounds__(UM_THREADS, 1)
apollo_project_umma_kernel(const UmmaTask *__restrict__ tasks, int n_tasks, int total_tiles)
{
    constexpr int UM_STAGES = um_stages<CG>(), UM_STAGE_BYTES = um_stage_bytes<CG>(), UM_SCAN = um_scan<CG>();
    extern __shared__ __align__(1024) unsigned char um_smem[];
    __shared__ __align__(8) uint64_t s_full[UM_STAGES], s_clean[UM_STAGES], s_empty[UM_STAGES], s_acc_full[2], s_acc_empty[2], s_done;
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < UM_STAGES; ++s) { mbar_init(&s_full[s], 1); mbar_init(&s_clean[s], CG * UM_WORKERS / 32); mbar_init(&s_empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&s_acc_full[b], 1); mbar_init(&s_acc_empty[b], CG * UM_WORKERS / 32); }
        mbar_init(&s_done, UM_THREADS);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == UM_MMA_WARP) {   // all 512 columns of tensor memory: two 128 x 256 binary32 accumulators
        if (CG == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(512u) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(512u) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncthreads();             // the only block-wide barrier: after it the roles run on mbarriers alone
    if (CG == 2) cluster_sync(); // (the other CTA's barriers are set up, and both have allocated)
    tc_fence_after();
    const int cta = CG == 2 ? (int)cluster_rank() : 0;
    // one arrival of a warp, on the barrier of the CTA that issues the MMAs
    const auto arrive_issuer = [&](uint64_t *bar) {
        __syncwarp();
        if (lane == 0) { if (CG == 2) mbar_arrive_first(bar); else mbar_arrive(bar); }
    };
    const uint32_t tmem = s_tmem;
    const uint32_t smem_base = smem_u32(um_smem);

    // Running counters, advanced identically by every thread: stage fills and accumulator
    // chunks since the kernel started.  Use number n of a barrier = counter / ring size; the
    // consumer of use n waits for phase parity n & 1, the producer of use n >= 1 for (n-1) & 1.
    int fills = 0, gchunk = 0;
    int issued = 0;                 // producer only: stage fills issued so far
    int mapped = -1;                // producer only: task whose tensor maps it has acquired

    for (int tile = blockIdx.x / CG; tile < total_tiles; tile += gridDim.x / CG) {
        if (volatile_load(&s_abort)) break;
        int lo = 0, hi = n_tasks - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(&tasks[mid].t.first_tile) <= tile) lo = mid; else hi = mid - 1;
        }
        const UmmaTask *U = tasks + lo;
        const ProjTask *T = &U->t;
        const int M = __ldg(&T->M), N = __ldg(&T->N), K = __ldg(&T->K);
        const int m0 = (tile - __ldg(&T->first_tile)) * CG * UM_BM + cta * UM_BM;       // rows of this CTA
        const int ksteps = (K + UM_BK - 1) / UM_BK;
        const int nchunks = (ksteps + UM_FLUSH - 1) / UM_FLUSH;
        const int plane_bytes = N / CG * UM_ROW_BYTES;                     // (of a pair each CTA has half of the columns)
        const bool right = __ldg(&T->right) != 0;
        bool failed = false;

        if (warp < UM_MMA_WARP) {
            // ---------------- workers (256 threads) ----------------
            // this thread's part of the accumulator: TMEM lanes 32 (warp % 4) + lane, columns 128 (warp / 4) ...
            const int row = (warp & 3) * 32 + lane, col_half = warp >> 2;
            float total[128];
#pragma unroll
            for (int i = 0; i < 128; ++i) total[i] = 0.0f;

            // add accumulator chunk c of this tile into the totals, with rounding, and hand the buffer back
            auto flush = [&](int c) -> bool {
                const int g = gchunk + c, buf = g & 1;
                if (!__all_sync(0xffffffffu, mbar_wait_bounded(&s_acc_full[buf], (uint32_t)(g >> 1) & 1u))) return false;
                tc_fence_after();
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    if (col_half * 128 + j * 16 < N) {           // uniform over the warp
                        uint32_t v[16];
                        const uint32_t taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(buf * UM_MAXN + col_half * 128 + j * 16);
                        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                                       "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                                     : "r"(taddr));
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int e = 0; e < 16; ++e) total[j * 16 + e] = __fadd_rn(total[j * 16 + e], __uint_as_float(v[e]));
                    }
                }
                tc_fence_before();
                arrive_issuer(&s_acc_empty[buf]);
                return true;
            };
            // The 8 KB gradient tile of a stage is 512 chunks of 16 bytes, two per thread.  rs: this thread's share
            // of squared norms of rows of M, over all of K.  Right: chunk i lies in row i / 4 of the tile (the swizzle
            // permutes chunks within a row), rs[0] and rs[1] are of rows tid / 4 and 64 + tid / 4.  Left: warp w has the
            // 16 rows of M from 16 w on, a lane 4 of them (lane & 3) at 4 values of K: 2 (lane / 4 % 4) and the next one
            // of two of the four groups of 8.  The 128-byte swizzle puts chunk c of a box row k at c ^ (k & 7): the 16
            // lanes of an access hit 16 different pairs of banks.
            double rs[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) rs[i] = 0.0;
            const int lk = 2 * ((lane >> 2) & 3), lc = 2 * (warp & 3) + ((lane >> 1) & 1);
            const int lbase = (warp >> 2) * UM_LEFT_BOX_BYTES + (lane >> 4) * 2048 + (lane & 1) * 8;
            const int left0 = lbase + lk * 128 + ((lc ^ lk) << 4), left1 = lbase + (lk + 1) * 128 + ((lc ^ (lk + 1)) << 4);
            // NS stages from stage ks of the tile on
            const auto scan_stages = [&](int ks, auto count) -> bool {
                constexpr int NS = decltype(count)::value;
                unsigned char *st[NS];
                bool wrote = false;
#pragma unroll
                for (int i = 0; i < NS; ++i) {
                    const int f = fills + ks + i, slot = f % UM_STAGES;
                    if (!__all_sync(0xffffffffu, mbar_wait_bounded(&s_full[slot], (uint32_t)(f / UM_STAGES) & 1u))) return false;
                    st[i] = um_smem + slot * UM_STAGE_BYTES;
                }
                if (right) {
                    uint4 v[2 * NS];
                    float sum[2 * NS];
                    bool finite = true;
#pragma unroll
                    for (int i = 0; i < 2 * NS; ++i) v[i] = *reinterpret_cast<const uint4 *>(st[i >> 1] + (tid + (i & 1) * UM_WORKERS) * 16);
#pragma unroll
                    for (int i = 0; i < 2 * NS; ++i) { sum[i] = umma_chunk_sum(v[i]); finite = finite && sum[i] <= 3.0e38f; }
                    if (finite) {
#pragma unroll
                        for (int i = 0; i < 2 * NS; ++i) rs[i & 1] += (double)sum[i];
                    } else {
#pragma unroll 1
                        for (int i = 0; i < NS; ++i) {
                            unsigned char *const p = um_smem + ((fills + ks + i) % UM_STAGES) * UM_STAGE_BYTES + tid * 16;
                            rs[0] += umma_chunk_sumsq(p, wrote);
                            rs[1] += umma_chunk_sumsq(p + UM_WORKERS * 16, wrote);
                        }
                    }
                } else {
                    float rq[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                    uint2 v[4 * NS];
                    uint32_t top = 0;
#pragma unroll
                    for (int i = 0; i < 4 * NS; ++i) v[i] = *reinterpret_cast<const uint2 *>(st[i >> 2] + ((i & 1) ? left1 : left0) + ((i >> 1) & 1) * 1024);
#pragma unroll
                    for (int i = 0; i < 4 * NS; ++i) top = __vmaxu2(top, __vmaxu2(v[i].x & 0x7fff7fffu, v[i].y & 0x7fff7fffu));
                    if ((top >> 16) < 0x5d80u && (top & 0xffffu) < 0x5d80u) {
#pragma unroll
                        for (int i = 0; i < 4 * NS; ++i) umma_quad_add(v[i], rq);
                    } else {
#pragma unroll 1
                        for (int i = 0; i < 4 * NS; ++i)
                            umma_quad_squares(um_smem + ((fills + ks + (i >> 2)) % UM_STAGES) * UM_STAGE_BYTES + ((i & 1) ? left1 : left0) + ((i >> 1) & 1) * 1024, rq, rs, wrote);
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) rs[i] += (double)rq[i];      // (at most 8 values each)
                }
                if (wrote) {                                 // repaired entries must be visible to the MMAs
                    if (CG == 2) fence_cluster();
                    fence_proxy_async();
                }
#pragma unroll
                for (int i = 0; i < NS; ++i) arrive_issuer(&s_clean[(fills + ks + i) % UM_STAGES]);
                return true;
            };
            auto scan = [&](int c) -> bool {
                const int k_end = min(ksteps, (c + 1) * UM_FLUSH);
                int ks = c * UM_FLUSH;
                for (; ks + UM_SCAN <= k_end; ks += UM_SCAN)
                    if (!scan_stages(ks, std::integral_constant<int, UM_SCAN>())) return false;
                for (; ks < k_end; ++ks)
                    if (!scan_stages(ks, std::integral_constant<int, 1>())) return false;
                return true;
            };
            for (int c = 0; c < nchunks && !failed; ++c) {
                if (!scan(c)) { failed = true; break; }
                if (c >= 1 && !flush(c - 1)) failed = true;
            }
            if (!failed && !flush(nchunks - 1)) failed = true;
            failed = __any_sync(0xffffffffu, failed);            // uniform over the warp from here on
            // ---------------- epilogue: the totals to g_low ----------------
            if (!failed) {
                const int m = m0 + row;
                const float sgn = __ldg(&T->negate) ? -1.0f : 1.0f;
                float *__restrict__ out = T->out;
                if (m < M && right) {
#pragma unroll
                    for (int q = 0; q < 32; ++q) {
                        const int n = col_half * 128 + q * 4;
                        if (n < N)
                            *reinterpret_cast<float4 *>(out + (int64_t)m * N + n) =
                                make_float4(sgn * total[4 * q], sgn * total[4 * q + 1], sgn * total[4 * q + 2], sgn * total[4 * q + 3]);
                    }
                } else if (m < M) {
                    // left case computed as the transposed problem: g_low is [N][M]; a warp's 32
                    // rows are consecutive addresses of one output row
#pragma unroll
                    for (int e = 0; e < 128; ++e) {
                        const int n = col_half * 128 + e;
                        if (n < N) out[(int64_t)n * M + m] = sgn * total[e];
                    }
                }
                // the threads that share a row (four; left: eight) add their parts; one of them stores the norm
                double *__restrict__ chan = U->chan_g2;
                if (right) {
#pragma unroll
                    for (int o = 1; o < 4; o <<= 1) { rs[0] += __shfl_xor_sync(0xffffffffu, rs[0], o); rs[1] += __shfl_xor_sync(0xffffffffu, rs[1], o); }
                    if ((tid & 3) == 0 && chan != nullptr) {
                        const int ra = m0 + (tid >> 2), rb = ra + 64;
                        if (ra < M) chan[ra] = rs[0];
                        if (rb < M) chan[rb] = rs[1];
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
#pragma unroll
                        for (int o = 4; o < 32; o <<= 1) rs[i] += __shfl_xor_sync(0xffffffffu, rs[i], o);
                        const int r = m0 + 16 * warp + 4 * lane + i;
                        if (lane < 4 && r < M && chan != nullptr) chan[r] = rs[i];
                    }
                }
            }
        } else if (warp == UM_MMA_WARP && lane == 0 && cta == 0) {
            // ---------------- MMA issuer ----------------
            const uint32_t idesc = umma_instr_desc<CG>(N, !right);
            for (int ks = 0; ks < ksteps; ++ks) {
                const int g = gchunk + ks / UM_FLUSH, buf = g & 1;
                const bool chunk_start = (ks % UM_FLUSH) == 0;
                if (chunk_start && g >= 2) {                    // the workers have drained this buffer
                    if (!mbar_wait_bounded(&s_acc_empty[buf], (uint32_t)((g >> 1) - 1) & 1u)) { failed = true; break; }
                    tc_fence_after();
                }
                const int f = fills + ks, slot = f % UM_STAGES, use = f / UM_STAGES;
                // the workers have read this stage (which also means that its copies have landed)
                if (!mbar_wait_bounded(&s_clean[slot], (uint32_t)use & 1u)) { failed = true; break; }
                if (!mbar_wait_bounded(&s_full[slot], (uint32_t)use & 1u)) { failed = true; break; }   // complete already: orders the copies before the MMAs in this thread
                tc_fence_after();
                const uint32_t a0 = smem_base + slot * UM_STAGE_BYTES;
                const uint32_t d = tmem + (uint32_t)(buf * UM_MAXN);
#pragma unroll
                for (int k16 = 0; k16 < UM_BK / 16; ++k16) {
                    const uint64_t ad = right ? umma_smem_desc(a0 + k16 * 32) : umma_smem_desc_left(a0 + k16 * 2048);
#pragma unroll
                    for (int t = 2; t >= 0; --t) {              // smallest plane first
                        const uint64_t bd = umma_smem_desc(a0 + UM_A_BYTES + t * plane_bytes + k16 * 32);
                        umma_bf16<CG>(d, ad, bd, idesc, (!chunk_start || k16 > 0 || t < 2) ? 1u : 0u);
                    }
                }
                umma_commit<CG>(&s_empty[slot]);                    // frees the slot when these MMAs are done
                if ((ks % UM_FLUSH) == UM_FLUSH - 1 || ks == ksteps - 1) umma_commit<CG>(&s_acc_full[buf]);
            }
        } else if (warp == UM_TMA_WARP && lane == 0) {
            // ---------------- copies ----------------
            const uint32_t bytes = (uint32_t)(UM_A_BYTES + 3 * plane_bytes);
            if (lo != mapped) {
                tensormap_acquire(&U->map_a);
                tensormap_acquire(&U->map_b);
                mapped = lo;
            }
            for (int ks = 0; ks < ksteps; ++ks) {
                const int f = fills + ks, slot = f % UM_STAGES, use = f / UM_STAGES;
                if (use >= 1 && !mbar_wait_bounded(&s_empty[slot], (uint32_t)(use - 1) & 1u)) { failed = true; break; }
                unsigned char *st = um_smem + slot * UM_STAGE_BYTES;
                mbar_expect_tx(&s_full[slot], bytes);
                if (right) tma_load_2d(st, &U->map_a, ks * UM_BK, m0, &s_full[slot]);
                else {
                    tma_load_2d(st, &U->map_a, m0, ks * UM_BK, &s_full[slot]);
                    tma_load_2d(st + UM_LEFT_BOX_BYTES, &U->map_a, m0 + UM_LEFT_BOX_M, ks * UM_BK, &s_full[slot]);
                }
                tma_load_3d(st + UM_A_BYTES, &U->map_b, ks * UM_BK, cta * (N / CG), 0, &s_full[slot]);
                issued = f + 1;
            }
        }
        if (failed) {
            s_abort = 1;
            atomicExch(&g_device_error, DEVERR_UMMA_TIMEOUT);
        }
        if (failed || volatile_load(&s_abort)) {
            // a role gave up: the producer gives its copies still in flight a bounded chance to land
            // before the block may end
            if (warp == UM_TMA_WARP && lane == 0)
                for (int back = 0; back < UM_STAGES && back < issued; ++back) {
                    const int f = issued - 1 - back;
                    mbar_wait_bounded(&s_full[f % UM_STAGES], (uint32_t)(f / UM_STAGES) & 1u);
                }
            break;
        }
        fills += ksteps;
        gchunk += nchunks;
    }

    // every thread reports in; the allocating warp frees the tensor memory once all have
    // (or after a bounded wait, when a role was lost to a time-out)
    mbar_arrive(&s_done);
    if (warp == UM_MMA_WARP) {
        mbar_wait_bounded(&s_done, 0u);
        __syncwarp();
    }
    // (a pair: no CTA ends, or frees, while the other may still arrive on its barriers or use its memory; every wait before has an end)
    if (CG == 2) { __syncwarp(); cluster_sync(); }
    if (warp == UM_MMA_WARP) {
        if (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
    if (CG == 2) { __syncwarp(); cluster_sync(); }
}

template <int CG> constexpr size_t um_smem_bytes() { return (size_t)um_stages<CG>() * um_stage_bytes<CG>() + 1024; }

}  // namespace af8
