// Statistic pass of the specialised full-rank configurations (fullrank_fast.cuh): per V block, the
// sum of squares of the update u = m_new / (sqrt(v_new) + eps) that the APPLY pass is going to use
// (first pass of the NORM -> APPLY structure, optimizer.py:1048-1077).
//
// Nothing computed here reaches a stored state: the sums only produce the norm that
// feeds the Fira limiter and the RMS clip, i.e. fp32 parameters with a 1e-5 tolerance.
// So with UF8/AL8 this pass, unlike the update kernel, decodes the second moment with the
// hardware exp2 (relative error 2^-22) instead of the exact sequence; every other format takes
// the exact decode (AL16: within one unit in the last place) and correctly rounded updates, as
// in the general kernel, and adds a lane's squares in groups of eight.  One WARP owns one V block
// (8 sub-steps of 256 elements, 8 per lane), keeps its sum in registers and writes one
// float: no block-wide barrier, plain coalesced 64/128-bit loads.  The 256 possible values
// of the block's codes go into a per-warp shared-memory table first (8 exp2 per lane and
// block instead of 64; entry 0 is the exact zero), guarded by warp-level syncs only.
//
// Per element: 2 special-function operations (sqrt, reciprocal) plus 1/8 for the table; the
// special-function pipe was the busiest unit with the decode per element (3 operations,
// 70 % busy): the table took the pass from 1.04 to 0.93 ms on the TinyLlama set.
// (Replacing the reciprocal by rsqrt and a short series was measured slower; so were requests for the
// next block's lines in L2, 0.972 against 0.955 ms.)
//
// What it waits for then is its loads (8 of 13 stall cycles an instruction).  With bf16 gradients, UF8 and AL8 each lane copies what it will
// read into a ring of its own in shared memory (cp.async; no other thread reads it, so nothing but its own groups is waited for), three
// steps of 256 elements ahead and on into the warp's next block, whose ranges are loaded a block ahead as well.  The ring takes the
// place of load registers: 64 without spills at four CTAs of 256 threads.  270 M parameters 223 -> 204 us (5.3 TB/s); with four steps of a
// block unrolled instead of eight 220, with five CTAs 232 and more (spills), five CTAs without the ring 223 and four 227.
//
// AL16 has too many codes for a table: an element
// costs a polynomial more (176 M UF4/AL16 parameters: 0.30 ms; 0.55 with the binary64 sequence of exp2_lane).
#pragma once

#include "common.cuh"
#include "fullrank_fast.cuh"

namespace af8 {

constexpr int STAT_THREADS = 256;
#ifndef AF8_STAT_MIN_CTAS
#define AF8_STAT_MIN_CTAS 5
#endif
#ifndef AF8_STAT_MIN_CTAS16
#define AF8_STAT_MIN_CTAS16 3
#endif
#ifndef AF8_STAT_UNROLL
#define AF8_STAT_UNROLL 4
#endif
constexpr int STAT_RING = 4, STAT_SLOT = FAST_MBLOCK * 4;    // steps in flight; bytes of one: gradients, momentum and second-moment codes
template <typename GradT, int VB, int MF> __host__ __device__ constexpr bool stat_ring() { return std::is_same<GradT, bf16_tag>::value && VB == 8 && MF == AF8_M_UF8; }
#ifndef AF8_STAT_MIN_CTAS_RING
#define AF8_STAT_MIN_CTAS_RING 4
#endif
template <typename GradT, int VB, int MF> __host__ __device__ constexpr int stat_min_ctas()
{
    return stat_ring<GradT, VB, MF>() ? AF8_STAT_MIN_CTAS_RING : VB == 16 ? AF8_STAT_MIN_CTAS16 : AF8_STAT_MIN_CTAS;
}

__device__ __forceinline__ void copy_async16(void *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async8(void *dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int ROOT>
__device__ __forceinline__ float ex2_approx(float x)
{
    float y;
    if (ROOT == ROOT_FTZ) asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    else asm("ex2.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// AL16 decode of two codes (optimizer.py:341-349) of a block with min_log >= -125 and a finite scale: the exponent as
// al16_decode2 rounds it, 2^n times the Taylor polynomial of 2^f for f in [-1/2, 1/2] (truncation 2^-27), error below one
// unit in the last place.
__device__ __forceinline__ float2 al16_decode2_stat(uint32_t pair, float scale, float min_log)
{
    const uint32_t c0 = pair & 0xffffu, c1 = pair >> 16;
    const float2 c = __fadd2_rn(make_float2(__uint_as_float(0x4b000000u | c0), __uint_as_float(0x4b000000u | c1)), bc2(-8388609.0f));
    const float2 t = __fadd2_rn(div2_by(__fmul2_rn(c, bc2(scale)), bc2(1.0f / 65534.0f), bc2(-65534.0f)), bc2(min_log));
    const float2 z = __fadd2_rn(t, bc2(AF8_MAGIC_F));
    const float2 f = sub2(t, __fadd2_rn(z, bc2(-AF8_MAGIC_F)));
    float2 p = bc2(1.52527338e-5f);                       // ln(2)^7 / 7!
    p = __ffma2_rn(p, f, bc2((float)AF8_EXP2_C6));
    p = __ffma2_rn(p, f, bc2((float)AF8_EXP2_C5));
    p = __ffma2_rn(p, f, bc2((float)AF8_EXP2_C4));
    p = __ffma2_rn(p, f, bc2((float)AF8_EXP2_C3));
    p = __ffma2_rn(p, f, bc2((float)AF8_EXP2_C2));
    p = __ffma2_rn(p, f, bc2((float)AF8_EXP2_C1));
    p = __ffma2_rn(p, f, bc2(1.0f));
    // (the low bits of z hold n; code 0 decodes to zero)
    return make_float2(c0 ? __int_as_float(__float_as_int(p.x) + (__float_as_int(z.x) << 23)) : 0.0f,
                       c1 ? __int_as_float(__float_as_int(p.y) + (__float_as_int(z.y) << 23)) : 0.0f);
}

template <typename GradT>
__device__ __forceinline__ void stat_load_g(const void *grad, int64_t off, float (&g)[8]);

template <>
__device__ __forceinline__ void stat_load_g<float>(const void *grad, int64_t off, float (&g)[8])
{
    const float4 *p = reinterpret_cast<const float4 *>(static_cast<const float *>(grad) + off);
    const float4 a = __ldcs(p), b = __ldcs(p + 1);
    g[0] = a.x; g[1] = a.y; g[2] = a.z; g[3] = a.w; g[4] = b.x; g[5] = b.y; g[6] = b.z; g[7] = b.w;
}

__device__ __forceinline__ void stat_widen(uint4 a, float (&g)[8])
{
    g[0] = __uint_as_float(a.x << 16); g[1] = __uint_as_float(a.x & 0xffff0000u);
    g[2] = __uint_as_float(a.y << 16); g[3] = __uint_as_float(a.y & 0xffff0000u);
    g[4] = __uint_as_float(a.z << 16); g[5] = __uint_as_float(a.z & 0xffff0000u);
    g[6] = __uint_as_float(a.w << 16); g[7] = __uint_as_float(a.w & 0xffff0000u);
}
template <>
__device__ __forceinline__ void stat_load_g<bf16_tag>(const void *grad, int64_t off, float (&g)[8])
{
    stat_widen(__ldcs(reinterpret_cast<const uint4 *>(static_cast<const uint16_t *>(grad) + off)), g);
}

template <typename GradT, int VB, int MF>
__global__ void __launch_bounds__(STAT_THREADS, (stat_min_ctas<GradT, VB, MF>()))
fullrank_stat_kernel(const FullrankLaunch L)
{
    // per-warp decode table of the block's 256 second-moment codes: 8 exponentials per lane and block
    // instead of 64 (the special-function pipe is the busiest unit of this pass); entry 0 is exact zero
    constexpr bool TABLE = VB == 8;
    constexpr float M_UNIT = MF == AF8_M_UF4 ? 0.125f : 0.0078125f;
    constexpr bool EXACT = root_exact<VB, MF>;
    __shared__ float s_dec[STAT_THREADS / 32][TABLE ? 256 : 1];
    __shared__ double s_exp2[EXACT && TABLE ? 32 : 1];       // copy of the exp2 table of the exact decode
    constexpr bool RING = stat_ring<GradT, VB, MF>();
    constexpr int STEPS = FAST_VBLOCK / FAST_MBLOCK, UNROLL = RING ? STEPS : AF8_STAT_UNROLL;
    __shared__ __align__(16) unsigned char s_ring[STAT_THREADS / 32][RING ? STAT_RING * STAT_SLOT : 16];
    const int lane = threadIdx.x & 31;
    if (EXACT && TABLE) {
        if (threadIdx.x < 32) s_exp2[threadIdx.x] = c_exp2_tab[threadIdx.x];
        __syncthreads();
    }
    await_launches();
    float *const dec = s_dec[threadIdx.x >> 5];
    const int64_t warps = (int64_t)gridDim.x * (STAT_THREADS / 32);
    const int64_t w0 = (int64_t)blockIdx.x * (STAT_THREADS / 32) + (threadIdx.x >> 5);

    int t = -1;
    int64_t cur_first = 0, cur_end = 0, numel = 0;
    const void *grad = nullptr;
    const uint8_t *mq = nullptr, *vq = nullptr;
    const float *m_scale = nullptr, *v_scale = nullptr, *v_min_log = nullptr;
    float v_w = 0.f, m_w = 0.f, eps_d = 0.f, eps_g = 0.f;
    bool small_w = true;

    for (int64_t blk = w0; blk < L.total_blocks;) {
        // the next tensor (uniform over the warp)
        if (t < 0) t = find_tensor(L.tensors, L.n_tensors, blk);
        else while (t + 1 < L.n_tensors && L.tensors[t + 1].first_block <= blk) ++t;
        const af8_fullrank_tensor *T = L.tensors + t;
        numel = T->numel;
        cur_first = T->first_block;
        cur_end = cur_first + (numel + FAST_VBLOCK - 1) / FAST_VBLOCK;
        grad = T->grad;
        mq = T->m_q; vq = static_cast<const uint8_t *>(T->v_q);
        m_scale = T->m_scale; v_scale = T->v_scale; v_min_log = T->v_min_log;
        v_w = T->v_w; m_w = MF == AF8_M_NONE ? 0.0f : T->m_w;
        eps_d = T->eps_denom; eps_g = T->eps_gradsq;
        small_w = fabsf(v_w) < 0.5f && fabsf(m_w) < 0.5f;

        // The blocks of this warp in this tensor, in one of two copies of the loop (see ROOT_EXACT; TinyLlama-1.1B with UF8/AL8:
        // 0.95 and 1.24 ms).
        const int64_t stop = min(cur_end, L.total_blocks);
        const auto blocks = [&](auto root) {
            constexpr int ROOT = decltype(root)::value;
            // the ring: this lane's 8 elements of a step lie in its own 32 bytes of the step's slot
            unsigned char *const ring = s_ring[threadIdx.x >> 5];
            const auto request = [&](int64_t first, int step) {
                const int64_t o = first + step * FAST_MBLOCK + lane * 8;
                unsigned char *const r = ring + step % STAT_RING * STAT_SLOT;
                copy_async16(r + lane * 16, static_cast<const uint16_t *>(grad) + o);
                copy_async8(r + FAST_MBLOCK * 2 + lane * 8, mq + o);
                copy_async8(r + FAST_MBLOCK * 3 + lane * 8, vq + o);
            };
            bool ahead = false;                 // the first steps of the block at hand are requested, its ranges loaded
            [[maybe_unused]] float next_sc = 0.0f, next_ml = 0.0f, next_ms = 0.0f;
            for (; blk < stop; blk += warps) {
                const int64_t b = blk - cur_first;
                const int64_t base = b * FAST_VBLOCK;
                const int64_t rem = numel - base;
                // decode v = 2^((code-1)*scale/levels + min_log) as 2^(code*a + c)
                const bool requested = RING && ahead;
                const float sc = requested ? next_sc : load_state(v_scale + b), ml = requested ? next_ml : load_state(v_min_log + b);
                // (lane s: the momentum scale of step s)
                [[maybe_unused]] const float ms = requested ? next_ms : RING && rem >= FAST_VBLOCK ? load_state(m_scale + b * STEPS + (lane & (STEPS - 1))) : 0.0f;
                if (RING) {
                    const int64_t nb = b + warps;
                    ahead = blk + warps < stop && numel - nb * FAST_VBLOCK >= FAST_VBLOCK && small_w;
                    if (ahead) { next_sc = load_state(v_scale + nb); next_ml = load_state(v_min_log + nb); next_ms = load_state(m_scale + nb * STEPS + (lane & (STEPS - 1))); }
                }
                [[maybe_unused]] const float a = sc * (VB == 16 ? 1.0f / 65534.0f : 1.0f / 254.0f);
                [[maybe_unused]] const float c = ml - a;
                float acc = 0.0f;

                // (a block that decodes to NaN, or into the subnormals, takes the forms that hold there)
                const bool regular = !EXACT || (sc <= 3.402823466e38f && (VB == 8 || ml >= -125.0f));

                if (rem >= FAST_VBLOCK && small_w && regular) {
                    if (TABLE) {
                        __syncwarp();                                   // the previous block's look-ups are done
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            const int code = lane + 32 * k;
                            if (EXACT) dec[code] = al8_decode_fast<true>((uint32_t)code, sc, ml, s_exp2);
                            else dec[code] = code ? ex2_approx<ROOT>(__fmaf_rn((float)code, a, c)) : 0.0f;
                        }
                        __syncwarp();
                    }
                    if (RING && !requested) {
#pragma unroll
                        for (int q = 0; q < STAT_RING - 1; ++q) { request(base, q); copy_async_commit(); }
                    }
                    const float2 wv2 = bc2(v_w), wm2 = bc2(m_w), ed2 = bc2(eps_d);
                    float2 acc2 = make_float2(0.0f, 0.0f);
#pragma unroll UNROLL
                    for (int s = 0; s < STEPS; ++s) {
                        const int64_t off = base + s * FAST_MBLOCK + lane * 8;
                        float g[8];
                        [[maybe_unused]] const unsigned char *const slot = ring + s % STAT_RING * STAT_SLOT;
                        if (RING) {
                            const int q = s + STAT_RING - 1;         // (into the slot that the step before has left)
                            if (q < STEPS) request(base, q);
                            else if (ahead) request(base + warps * FAST_VBLOCK, q - STEPS);
                            copy_async_commit();
                            copy_async_wait<STAT_RING - 1>();
                            stat_widen(*reinterpret_cast<const uint4 *>(slot + lane * 16), g);
                        } else {
                            stat_load_g<GradT>(grad, off, g);
                        }
                        if (L.negate_grad) {                       // maximize (optimizer.py:1973-1974)
#pragma unroll
                            for (int j = 0; j < 8; ++j) g[j] = -g[j];
                        }
                        uint2 mw = make_uint2(0u, 0u);
                        uint32_t vw[VB / 4];
                        if (RING) mw = *reinterpret_cast<const uint2 *>(slot + FAST_MBLOCK * 2 + lane * 8);
                        else if (MF == AF8_M_UF8) mw = __ldcs(reinterpret_cast<const uint2 *>(mq + off));
                        if (MF == AF8_M_UF4) mw.x = __ldcs(reinterpret_cast<const uint32_t *>(mq + off / 2));
                        if (VB == 8) {
                            const uint2 w = RING ? *reinterpret_cast<const uint2 *>(slot + FAST_MBLOCK * 3 + lane * 8) : __ldcs(reinterpret_cast<const uint2 *>(vq + off));
                            vw[0] = w.x; vw[1] = w.y;
                        } else {
                            const uint4 w = __ldcs(reinterpret_cast<const uint4 *>(vq + off * 2));
                            vw[0] = w.x; vw[1] = w.y; vw[VB / 4 - 2] = w.z; vw[VB / 4 - 1] = w.w;
                        }
                        float2 sum8 = make_float2(0.0f, 0.0f);
                        const float2 mc2 = bc2(RING ? __shfl_sync(0xffffffffu, ms, s) * M_UNIT : MF == AF8_M_NONE ? 0.0f : load_state(m_scale + b * STEPS + s) * M_UNIT);
#pragma unroll
                        for (int j = 0; j < 8; j += 2) {
                            const float2 gj = make_float2(g[j], g[j + 1]);
                            float2 g2 = __fmul2_rn(gj, gj);
                            if (eps_g != 0.0f) g2 = __fadd2_rn(g2, bc2(eps_g));
                            float2 v_old;
                            if (VB == 8) {
                                v_old = make_float2(dec[TABLE ? __byte_perm(vw[j >> 2], 0u, 0x4440u | (uint32_t)(j & 3)) : 0u],
                                                    dec[TABLE ? __byte_perm(vw[j >> 2], 0u, 0x4440u | (uint32_t)((j + 1) & 3)) : 0u]);
                            } else {
                                v_old = al16_decode2_stat(vw[(j >> 1) & (VB / 4 - 1)], sc, ml);
                            }
                            const float2 vj = __ffma2_rn(wv2, sub2(g2, v_old), v_old);
                            float2 mj = gj;
                            if (MF == AF8_M_UF8) {
                                const uint32_t mword = (j < 4) ? mw.x : mw.y;
                                const float2 mb = make_float2(__uint_as_float(__byte_perm(mword, 0x4b000000u, 0x7540u | (uint32_t)(j & 3))),
                                                              __uint_as_float(__byte_perm(mword, 0x4b000000u, 0x7540u | (uint32_t)((j + 1) & 3))));
                                const float2 m_old = __fmul2_rn(__fadd2_rn(mb, bc2(-8388736.0f)), mc2);
                                mj = __ffma2_rn(wm2, sub2(gj, m_old), m_old);
                            } else if (MF == AF8_M_UF4) {                      // byte j / 2, the even element in its high nibble
                                const float2 mb = make_float2(__uint_as_float(0x4b000000u | ((mw.x >> (4 * j + 4)) & 15u)), __uint_as_float(0x4b000000u | ((mw.x >> (4 * j)) & 15u)));
                                const float2 m_old = __fmul2_rn(__fadd2_rn(mb, bc2(-8388616.0f)), mc2);
                                mj = __ffma2_rn(wm2, sub2(gj, m_old), m_old);
                            }
                            const float2 u = root_update2<MF, ROOT>(mj, vj, ed2);
                            if (EXACT) sum8 = __ffma2_rn(u, u, sum8);
                            else acc2 = __ffma2_rn(u, u, acc2);
                        }
                        if (EXACT) acc2 = __fadd2_rn(acc2, sum8);
                    }
                    acc = __fadd_rn(acc2.x, acc2.y);
                } else {
                    // tail block of a tensor, EMA weights >= 0.5, or an irregular block: element-wise with guards
                    for (int64_t i = lane; i < FAST_VBLOCK; i += 32) {
                        if (i >= rem) break;
                        const int64_t e = base + i;
                        float gj = GradLoad<GradT>::load1(grad, e);
                        if (L.negate_grad) gj = -gj;
                        const float g2 = __fadd_rn(__fmul_rn(gj, gj), eps_g);
                        const uint32_t code = VB == 16 ? reinterpret_cast<const uint16_t *>(vq)[e] : vq[e];
                        const float v_old = EXACT ? al_decode(code, sc, ml, VB == 16 ? 65534.0f : 254.0f) : code ? ex2_approx<ROOT>(__fmaf_rn((float)code, a, c)) : 0.0f;
                        const float vj = lerp_t(v_old, g2, v_w);
                        float mj = gj;
                        if (MF != AF8_M_NONE) {
                            const int k = MF == AF8_M_UF8 ? (int)mq[e] - 128 : (int)((e & 1) ? (mq[e >> 1] & 15u) : (mq[e >> 1] >> 4)) - 8;
                            mj = lerp_t(__fmul_rn((float)k, load_state(m_scale + e / FAST_MBLOCK) * M_UNIT), gj, m_w);
                        }
                        const float u = root_update2<MF, EXACT ? ROOT_EXACT : ROOT>(make_float2(mj, 0.0f), make_float2(vj, 0.0f), bc2(eps_d)).x;
                        acc = __fmaf_rn(u, u, acc);
                    }
                }
                acc = warp_sum(acc);
                if (lane == 0) L.block_sumsq[blk] = acc;
            }
        };
        if (eps_d >= EPS_HIDES) blocks(std::integral_constant<int, EXACT ? ROOT_REFINED : ROOT_FTZ>());
        else blocks(std::integral_constant<int, EXACT ? ROOT_EXACT : ROOT_FULL>());
    }
}

}  // namespace af8
