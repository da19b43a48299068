// Full-rank fused step, specialised kernel: AdamW- / RMSprop-style update (Adam denominator) with an
// AL8 or AL16 second moment (V block 2048) and a UF8 or UF4 momentum (M block 256) or none, fp32
// parameters with fp32 or bf16 gradients, or bf16 parameters (rounded to nearest or stochastically)
// with bf16 gradients.
//
// Reference semantics: _update_param_8bit full-rank branch with the Adam
// denominator (optimizer.py:2115-2123), _fallback_1d_update
// (optimizer.py:903-910), _m_ema_pytorch (optimizer.py:690-700), the AL codec
// (optimizer.py:299-353) and the uniform codecs (optimizer.py:504-532).
//
// Work decomposition.  The launch covers a table of tensors; the unit of work
// is one V block (2048 consecutive elements of one tensor).  A persistent grid
// walks the flat block space with a grid stride.  One CTA of 128 threads owns a
// block; warp w owns elements [512w, 512w+512), i.e. two M blocks, so a
// momentum absmax is a pure warp reduction.  Lane l owns the 4-element groups at
// 512w+4l, +128, +256 and +384: every shared-memory read and every global store
// of a warp is one contiguous run.  Sixteen elements per thread halve what a
// block costs besides its elements against eight (256 threads): 69 -> 56
// instructions per parameter, and a block-wide barrier joins four warps instead
// of eight.
//
// Data movement.  The parameter, gradient and code arrays of a full block
// are brought into a two-stage shared-memory ring by bulk asynchronous copies
// (cp.async.bulk, completion on an mbarrier).  While block i is being processed
// the copies of block i+1 of the same tensor are already in flight, and the
// 256-entry AL8 decode table of block i+1 is computed while warp 0 derives the
// range of block i.  A tail block (fewer than 2048 real elements) is copied into
// its slot by the threads.  Every wait on an
// mbarrier is bounded; a wait that runs out raises the device error flag that
// af8_device_status() reports, the threads skip the stores of that block and
// the CTA stops at its next block-wide barrier.
//
// What bounds it: instruction issue and the latency between dependent
// instructions (62 % of the issue slots with 22 warps resident; DRAM 64 % busy), so
// the hot loop is kept small (about 14 KB of code): what is rare - tail blocks, uncommon
// scalars, codes in doubt - is rolled up or handled by a compact general branch.  Inlined
// between the parts of the loop those copies had put instruction fetches at the top of the
// stall list.  Exact IEEE arithmetic is spent only where it decides a stored bit:
//   * the EMAs, the dequantisation and both requantisations are bit-exact
//     restatements of the torch ops;
//   * the block extrema are reduced on v itself (log2 is monotone) and the
//     exactly rounded log2 is taken of the two extreme values only;
//   * an AL8 code is first computed from the hardware log2
//     approximation; only when that estimate lies closer to a rounding
//     boundary than its own error bound is the exact sequence (binary64 log2,
//     IEEE division) evaluated, so the stored code is always the exact one;
//     AL16 codes, 257 times finer, are always computed exactly;
//   * the momentum division m/absmax uses the correctly rounded reciprocal of
//     the block's absmax with one residual correction, which yields the IEEE
//     quotient;
//   * the parameter update u = m / (sqrt(v) + eps) feeds nothing but the
//     parameter; with UF8/AL8 it uses the hardware approximations of sqrt and
//     reciprocal (relative error below 3e-7, for subnormal second moments too: see
//     EPS_HIDES), with every other format the correctly rounded operations.
//
// Measured on a B200, before -> after the split by sixteen elements (and, for the formats other
// than UF8/AL8, against the general kernel): TinyLlama-1.1B update pass 3.23 -> 2.8 ms (5.5 TB/s);
// bf16 parameters with stochastic rounding 5.0 -> 3.6 ms; UF4/AL16, 176 M parameters 4.17 -> 0.93 ms;
// AL8 without momentum, fp32 gradients, 110 M parameters 1.95 -> 0.32 ms (4.9 TB/s).  The correctly
// rounded update of these formats (ROOT_REFINED) costs 5 to 12 % against the hardware approximations
// (30 % with the IEEE functions), the tests for infinities and NaNs (STRICT) up to 4 %.
#pragma once

#include "common.cuh"
#include "launch.cuh"

namespace af8 {

constexpr int FAST_VBLOCK = 2048;
constexpr int FAST_MBLOCK = 256;
constexpr int FAST_THREADS = 128;
constexpr int FAST_EPT = 16;  // elements per thread
constexpr int FAST_WARPS = FAST_THREADS / 32;
// resident CTAs asked of the compiler (AL8: 5 -> 6 gave 1-3 %; AL16: see fast_stash)
#ifndef AF8_FAST_CTAS8
#define AF8_FAST_CTAS8 6
#endif
#ifndef AF8_FAST_CTAS16
#define AF8_FAST_CTAS16 5
#endif
template <int VB> constexpr int fast_min_ctas() { return VB == 8 ? AF8_FAST_CTAS8 : AF8_FAST_CTAS16; }

// Whether the new second moments wait for the block's range in the ring slot, in place of the consumed parameters, instead of
// in registers, and the two momentum blocks of a warp take turns in one copy of the code.  AL16: the binary64 sequences of
// sixteen elements at once took 144 registers, three CTAs per SM, and were bound by latency (55 % of the issue slots); eight at
// a time fit 96 registers and five CTAs (67 M UF4/AL16 parameters 383 -> 346 us; four
// CTAs 352, six 428).  The slot is then read until the block's
// last code is written, so that the last warp to leave it has it refilled.  With AL8, where registers suffice, the detour
// costs more than it gives (fp32 parameters 177 -> 188 us, bf16 ones 174 -> 196).
template <int VB> __host__ __device__ constexpr bool fast_stash() { return VB == 16; }

struct FullrankLaunch {
    const af8_fullrank_tensor *tensors;
    const af8_dyn_scalars *dyn;
    float *block_sumsq;
    int64_t total_blocks;
    int32_t n_tensors;
    int32_t negate_grad;
    float v_floor;
    int32_t param_dtype;    // AF8_F32 / AF8_BF16 / AF8_F16
    int32_t sr;             // stochastic rounding of 16-bit parameters
};

// Index of the tensor that owns flat block `blk` (first_block is ascending).
__device__ __forceinline__ int find_tensor(const af8_fullrank_tensor *tensors, int n, int64_t blk)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (tensors[mid].first_block <= blk) lo = mid; else hi = mid - 1;
    }
    return lo;
}

template <typename T> struct GradLoad;

template <> struct GradLoad<float> {
    static __device__ __forceinline__ float load1(const void *base, int64_t off)
    {
        return static_cast<const float *>(base)[off];
    }
};

struct bf16_tag {};
struct f16_tag {};
template <> struct GradLoad<f16_tag> {      // (general kernel only)
    static __device__ __forceinline__ float load1(const void *base, int64_t off)
    {
        return f16_bits_to_f32(static_cast<const uint16_t *>(base)[off]);
    }
};
template <> struct GradLoad<bf16_tag> {
    static __device__ __forceinline__ float load1(const void *base, int64_t off)
    {
        return bf16_bits_to_f32(static_cast<const uint16_t *>(base)[off]);
    }
};

// How the update m / (sqrt(v) + eps) is formed.  It feeds nothing but the parameter and the norm.
//   ROOT_EXACT    every operation correctly rounded, as in the general kernel; every format pair but UF8/AL8
//   ROOT_REFINED  the same numbers from the hardware approximations and one residual step each (Markstein 1990), in packed
//                 arithmetic: a third of the instructions of the IEEE functions.  Above EPS_HIDES (below) only: a residual
//                 of v < 2^-100 may be subnormal, but no bit of such a square root survives the addition of eps.  (The
//                 remainder of a gradient below 2^-100 may be, too: the last bit of a quotient below 2^-62)
//   ROOT_FTZ      hardware approximations in their flush-to-zero forms, one MUFU instruction each (UF8/AL8; relative error
//                 below 3e-7).  A second moment below 2^-126 has a square root below 2^-63, which an eps of 2^-38
//                 (EPS_HIDES) or more absorbs whole; below that eps the square root is the denominator and must not be
//                 flushed: with the constructor's eps of 1e-30 a first gradient of 1e-18 would otherwise give an update
//                 of 1e12 instead of 31.6
//   ROOT_FULL     the approximations without the flush, three more instructions each (UF8/AL8 below EPS_HIDES)
constexpr float EPS_HIDES = 0x1p-38f;
constexpr int ROOT_FTZ = 0, ROOT_FULL = 1, ROOT_EXACT = 2, ROOT_REFINED = 3;
template <int VB, int MF> constexpr bool root_exact = !(VB == 8 && MF == AF8_M_UF8);
template <int ROOT>
__device__ __forceinline__ float root_sqrt(float x)
{
    if (ROOT == ROOT_EXACT) return __fsqrt_rn(x);
    float y;
    if (ROOT == ROOT_FTZ) asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    else asm("sqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
template <int ROOT>
__device__ __forceinline__ float root_rcp(float x)
{
    if (ROOT == ROOT_EXACT) return __frcp_rn(x);
    float y;
    if (ROOT == ROOT_FULL) asm("rcp.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    else asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rsqrt_approx(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// the updates of two elements from the un-requantised m and v (optimizer.py:905, 909); without momentum m is the gradient
// and the reference divides (optimizer.py:911-917)
template <int MF, int ROOT>
__device__ __forceinline__ float2 root_update2(float2 m, float2 v, float2 eps)
{
    if (ROOT == ROOT_REFINED) {
        const float2 one = make_float2(1.0f, 1.0f), neg = make_float2(-1.0f, -1.0f);
        const float2 y = make_float2(rsqrt_approx(fmaxf(v.x, 0x1p-126f)), rsqrt_approx(fmaxf(v.y, 0x1p-126f)));     // (zero: s = 0)
        const float2 s = __fmul2_rn(v, y);
        const float2 root = __ffma2_rn(__ffma2_rn(s, s, __fmul2_rn(v, neg)), __fmul2_rn(y, make_float2(-0.5f, -0.5f)), s);
        float2 den = __fadd2_rn(root, eps);
        // (an infinite v has made it NaN: its reciprocal is zero, like that of the largest number, which is flushed)
        den = make_float2(fminf(den.x, 3.402823466e38f), fminf(den.y, 3.402823466e38f));
        const float2 nd = __fmul2_rn(den, neg), r = make_float2(root_rcp<ROOT>(den.x), root_rcp<ROOT>(den.y));
        const float2 inv = __ffma2_rn(__ffma2_rn(nd, r, one), r, r);
        const float2 u = __fmul2_rn(m, inv);
        return MF == AF8_M_NONE ? __ffma2_rn(__ffma2_rn(nd, u, m), inv, u) : u;
    }
    const float2 den = __fadd2_rn(make_float2(root_sqrt<ROOT>(v.x), root_sqrt<ROOT>(v.y)), eps);
    if (ROOT == ROOT_EXACT && MF == AF8_M_NONE) return make_float2(__fdiv_rn(m.x, den.x), __fdiv_rn(m.y, den.y));
    return __fmul2_rn(m, make_float2(root_rcp<ROOT>(den.x), root_rcp<ROOT>(den.y)));
}
__device__ __forceinline__ float lg2_approx(float x)
{
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// |lg2.approx(x) - log2(x)| <= 1.22e-7 |log2(x)| + 1.7e-7 for every normal x (all of them measured on a B200, and by
// tests/test_lg2_approx_gpu.py: 2.74e-7 for |log2| in [1, 2), 7.78e-6 in [64, 128))
constexpr float LG2_REL = 1.22e-7f, LG2_ABS = 1.7e-7f;

#define AF8_MAGIC_F 12582912.0f       /* 1.5 * 2^23: adding it rounds to an integer (half to even) */
#define AF8_MAGIC_I 0x4b400000

// (byte j of a packed word) - 128 as a float, without a conversion instruction:
// the byte becomes the low mantissa bits of 2^23 + byte
__device__ __forceinline__ float byte_minus_128(uint32_t word, int j)
{
    return __uint_as_float(__byte_perm(word, 0x4b000000u, 0x7540u | (uint32_t)j)) - 8388736.0f;
}

// block-wide constants of the second-moment requantisation, produced by warp 0
struct __align__(16) VRange {
    float min_log;   // stored range
    float scale;
    float k;         // 254 / scale (estimate path)
    float c;         // -min_log * k
    float thr;       // an estimate is trusted when |t - rint(t)| <= thr
    float pad[3];
};

// Blackwell packed binary32 arithmetic: one instruction works on a pair of floats held in
// a 64-bit register; each component rounds exactly like the scalar *_rn operation.
__device__ __forceinline__ float2 bc2(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(bc2(-1.0f), b, a); }   // a - b, one rounding

// two binary32 numbers rounded to nearest bf16, packed (first one in the low half)
__device__ __forceinline__ uint32_t bf16x2_rn(float lo, float hi)
{
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

// ---------------------------------------------------------------------------
// device error flag, mbarrier and bulk-copy helpers
// ---------------------------------------------------------------------------
// Set (never cleared by kernels) when a bounded wait ran out.  Read back by
// af8_device_status().
__device__ int g_device_error = 0;
constexpr int DEVERR_COPY_TIMEOUT = 1;

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t global_timer_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Wait for a phase of the barrier for at most `limit_ns` of wall time (two seconds unless told
// otherwise; a block's copies take microseconds).  Returns false when the time ran out.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity, uint64_t limit_ns = 2000000000ull)
{
    uint64_t t0 = 0;
    for (uint32_t i = 0;; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 0xffu) == 0xffu) {
            const uint64_t now = global_timer_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > limit_ns) return false;
        }
    }
}
// global -> shared bulk copy of `bytes` (multiple of 16, both addresses 16-byte
// aligned); completion is signalled on `bar` as transaction bytes.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ---------------------------------------------------------------------------
// second-moment codecs of the update kernel
// ---------------------------------------------------------------------------
// AL16 has 65536 codes, so there is no table of a block's values: every element is decoded and
// encoded with the binary64 sequences below.  Their small tables live one entry per lane in the
// warp's registers and are read with shuffles (a shared-memory table costs about ten cycles of the
// load pipe per look-up in bank conflicts, a shuffle one), and the operands enter binary64 through
// their bits where they can (conversions run at a quarter of the rate of the arithmetic).
struct LaneTables {
    double e2;          // 2^(lane/32)
    double l2;          // -log2(inv) of centre `lane`
    uint32_t inv_hi;    // high word of inv
};
struct LogLaneEntry { uint32_t inv_hi; double l2; };
__constant__ LogLaneEntry c_log2_lane[32] = {
#include "log2_lane_table.inc"
};

// exp2_cr_fast with the table in the lanes: |x| <= 150
__device__ __forceinline__ float exp2_lane(float x, const LaneTables &T)
{
    // n = rint(32 x) and the remainder x - n/32 are exact in binary32 (|32 x| < 2^13)
    const float z = __fadd_rn(__fmul_rn(x, 32.0f), 12582912.0f);
    const int n = __float_as_int(z);                                     // low bits hold n
    const double r = (double)__fmaf_rn(__fsub_rn(z, 12582912.0f), -0.03125f, x);
    const double t = __shfl_sync(0xffffffffu, T.e2, n & 31);
    double p = AF8_EXP2_C6;
    p = fma(p, r, AF8_EXP2_C5);
    p = fma(p, r, AF8_EXP2_C4);
    p = fma(p, r, AF8_EXP2_C3);
    p = fma(p, r, AF8_EXP2_C2);
    p = fma(p, r, AF8_EXP2_C1);
    p = fma(p, r, 1.0);
    const double y = t * p;                                              // in [1, 2.03)
    return __double2float_rn(__hiloint2double(__double2hiint(y) + (((n - 0x4b400000) >> 5) << 20), __double2loint(y)));
}

// Correctly rounded log2 of a positive normal x (up to the relative error 2^-52 of the sum before the last
// rounding): x = 2^e * m with m in [63/64, 127/64); the nearest of the 32 centres 1 + j/32 selects inv_j,
// r = m*inv_j - 1 is exact (24 + 21 bits) with |r| <= 2^-6, log2(1 + r) by its Taylor series through r^9 (truncation
// below 2^-57 of r).  Around x = 1 the centre is 1 itself, inv = 1 and the table entry 0, so that the result stays
// relatively accurate there.
__device__ __forceinline__ float log2_lane(float x, const LaneTables &T)
{
    const uint32_t b = __float_as_uint(x), near = b + 0x20000u;
    const int j = (near >> 18) & 31;
    const double m = __hiloint2double((int)((b >> 3) - ((near >> 23) << 20) + 0x3ff00000u), (int)(b << 29));
    const double inv = __hiloint2double((int)__shfl_sync(0xffffffffu, T.inv_hi, j), 0);
    const double tab = __shfl_sync(0xffffffffu, T.l2, j);
    const double e = __hiloint2double(0x43300000, (int)(near >> 23)) - (4503599627370496.0 + 127.0);
    const double r = fma(m, inv, -1.0);
    double p = 0x1.484b13d7c02a9p-3;        //  1/(9 ln 2)
    p = fma(p, r, -0x1.71547652b82fep-3);   // -1/(8 ln 2)
    p = fma(p, r, 0x1.a61762a7adedap-3);    //  1/(7 ln 2)
    p = fma(p, r, -0x1.ec709dc3a03fep-3);   // -1/(6 ln 2)
    p = fma(p, r, 0x1.2776c50ef9bfep-2);    //  1/(5 ln 2)
    p = fma(p, r, -0x1.71547652b82fep-2);   // -1/(4 ln 2)
    p = fma(p, r, 0x1.ec709dc3a03fep-2);    //  1/(3 ln 2)
    p = fma(p, r, -0x1.71547652b82fep-1);   // -1/(2 ln 2)
    p = fma(p, r, 0x1.71547652b82fep+0);    //  1/ln 2
    return __double2float_rn(fma(p, r, e + tab));
}

// x / d from the correctly rounded reciprocal of d and one residual step: the IEEE quotient (Markstein)
__device__ __forceinline__ float2 div2_by(float2 x, float2 rc, float2 nd)
{
    const float2 q = __fmul2_rn(x, rc);
    return __ffma2_rn(__ffma2_rn(q, nd, x), rc, q);
}

// false: the block held an infinite second moment
__device__ __forceinline__ bool range_finite(float scale, float min_log) { return scale <= 3.402823466e38f && min_log <= 3.402823466e38f; }

// AL16 decode of two codes (optimizer.py:341-349) of a block with a finite range; every lane of the warp takes part
__device__ __forceinline__ float2 al16_decode2(uint32_t pair, float scale, float min_log, const LaneTables &T)
{
    const uint32_t c0 = pair & 0xffffu, c1 = pair >> 16;
    // code - 1 as a float: the code becomes the low mantissa bits of 2^23 + code
    const float2 c = make_float2(__fsub_rn(__uint_as_float(0x4b000000u | c0), 8388609.0f), __fsub_rn(__uint_as_float(0x4b000000u | c1), 8388609.0f));
    const float2 x = __fmul2_rn(c, bc2(scale));
    const float2 t = __fadd2_rn(div2_by(x, bc2(1.0f / 65534.0f), bc2(-65534.0f)), bc2(min_log));
    // (code 0 decodes to zero; its t, just below min_log, only has to stay in range)
    const float y0 = exp2_lane(t.x, T), y1 = exp2_lane(t.y, T);
    return make_float2(c0 ? y0 : 0.0f, c1 ? y1 : 0.0f);
}

// ---------------------------------------------------------------------------
// stochastic rounding of a pair to bf16 (same bits as sr_bf16_bits of each)
// ---------------------------------------------------------------------------
// "r24 < low16 * 256" only depends on the top 16 of the 24 random bits, r24 / 256 < low16; and adding
// 65535 - r16 to the binary32 pattern carries into the upper half exactly then.  The last xor-shift of
// the generator (by 31) does not reach the top 24 bits.  Infinities, NaNs and steps into an infinity
// take the exact function.
//
// The counters z of a block, 2048 consecutive ones, nearly always share their bits 30 to 63.  Then z ^ (z >> 30) has the same
// high word for all of them, and its part of the first product is one number per block; an element takes two
// multiplications there instead of three and a shift less (67 M parameters 238 -> 229 us).
struct SrCounter {
    uint32_t lo, mix, high;      // low word of the first counter; what is xored into a low word; the high word's part of the product
    bool shared;                 // the block's counters do share their upper bits
};
__device__ __forceinline__ SrCounter sr_counter(uint64_t base, int64_t first, uint32_t n)
{
    const uint64_t z = base + (uint64_t)first + 0x9E3779B97F4A7C15ull;
    const uint32_t hi = (uint32_t)(z >> 32);
    SrCounter c;
    c.lo = (uint32_t)z;
    c.mix = (uint32_t)(z >> 30);
    c.high = (hi ^ (hi >> 30)) * 0x1CE4E5B9u;
    c.shared = (c.lo & 0x3fffffffu) <= 0x40000000u - n;
    return c;
}
// upper 32 bits of the generator's output for counter lo + j (if the block shares its upper bits)
__device__ __forceinline__ uint32_t sr_hi32(const SrCounter &c, uint32_t j)
{
    const uint32_t a = (c.lo + j) ^ c.mix;
    uint64_t z = (uint64_t)a * 0x1CE4E5B9u + ((uint64_t)c.high << 32);
    z += (uint64_t)(a * 0xBF58476Du) << 32;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return (uint32_t)(z >> 32);
}
__device__ __forceinline__ uint32_t sr_bf16x2(float a, float b, uint32_t ha, uint32_t hb)
{
    const uint32_t x = __float_as_uint(a) + (~ha >> 16), y = __float_as_uint(b) + (~hb >> 16);
    return __byte_perm(x, y, 0x7632);
}

// three-operand maximum, NaN if any operand is
__device__ __forceinline__ float max3_nan(float a, float b, float c)
{
    float d;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float max3(float a, float b, float c)
{
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float min3(float a, float b, float c)
{
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// ---------------------------------------------------------------------------
// the kernel
// ---------------------------------------------------------------------------
template <typename T> struct ParamElem { typedef float type; };
template <> struct ParamElem<bf16_tag> { typedef uint16_t type; };
template <typename T> struct GradBytes { static constexpr int value = 4; };
template <> struct GradBytes<bf16_tag> { static constexpr int value = 2; };

// the step's scalars of the current tensor, in shared memory
struct __align__(16) StepScalars {
    float decay, step_mul, fira, eps_d;
    float v_w, m_w, eps_g;
    int16_t plain;      // both EMA weights below 1/2 and no eps on g^2
    int16_t zero_upd;   // the limiter asked for a zero update
};

// Ring geometry of one kernel variant: byte offsets inside a slot and the slot count.
template <typename GradT, typename ParamT, int VB, int MF> struct FastRing {
    static constexpr int GB = GradBytes<GradT>::value;
    static constexpr int PB = GradBytes<ParamT>::value;     // bytes per parameter: 4 (float) or 2 (bf16_tag)
    static constexpr int MQ_BYTES = MF == AF8_M_UF8 ? FAST_VBLOCK : (MF == AF8_M_UF4 ? FAST_VBLOCK / 2 : 0);
    static constexpr int VQ_BYTES = FAST_VBLOCK * VB / 8;
    static constexpr int P_OFF = 0;
    static constexpr int G_OFF = FAST_VBLOCK * PB;
    static constexpr int VQ_OFF = G_OFF + FAST_VBLOCK * GB;
    static constexpr int MQ_OFF = VQ_OFF + VQ_BYTES;
    static constexpr int STAGE_BYTES = MQ_OFF + MQ_BYTES;
    static constexpr int NST = 2;
    static constexpr int SMEM_BYTES = NST * STAGE_BYTES;
};

// Eight elements (two groups of four) of one momentum block: EMAs, update, new parameter.
// PLAIN: the common scalars (see StepScalars::plain).  LAG: sumsq += u^2 over the elements whose bit is set in real.
// ROOT: see ROOT_EXACT.
template <int MF, bool PLAIN, bool ROUND_DECAY, bool LAG, int ROOT>
__device__ __forceinline__ void fast_ema8(const StepScalars &S, const float2 (&g)[4], const float2 (&v_old)[4], const float2 (&m_old)[4],
                                          float2 (&p)[4], float2 (&v)[4], float2 (&m)[4], uint32_t real, float &sumsq)
{
    const float2 w_v = bc2(S.v_w), w_m = bc2(S.m_w), eps_d2 = bc2(S.eps_d), decay2 = bc2(S.decay), step2 = bc2(S.step_mul), fira2 = bc2(S.fira);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        // second moment (optimizer.py:2117-2119)
        if (PLAIN) {
            v[j] = __ffma2_rn(w_v, sub2(__fmul2_rn(g[j], g[j]), v_old[j]), v_old[j]);
        } else {
            v[j] = make_float2(lerp_t(v_old[j].x, __fadd_rn(__fmul_rn(g[j].x, g[j].x), S.eps_g), S.v_w),
                               lerp_t(v_old[j].y, __fadd_rn(__fmul_rn(g[j].y, g[j].y), S.eps_g), S.v_w));
        }
        // momentum (optimizer.py:698); without one the gradient itself is normalised (optimizer.py:911-917)
        if (MF == AF8_M_NONE) m[j] = g[j];
        else if (PLAIN) m[j] = __ffma2_rn(w_m, sub2(g[j], m_old[j]), m_old[j]);
        else m[j] = make_float2(lerp_t(m_old[j].x, g[j].x, S.m_w), lerp_t(m_old[j].y, g[j].y, S.m_w));
        float2 u = root_update2<MF, ROOT>(m[j], v[j], eps_d2);
        if (LAG) {                                                // (padding may be 0 * inf)
            if ((real >> (2 * j)) & 1u) sumsq = __fmaf_rn(u.x, u.x, sumsq);
            if ((real >> (2 * j + 1)) & 1u) sumsq = __fmaf_rn(u.y, u.y, sumsq);
        }
        float2 x = __fmul2_rn(p[j], decay2);                      // optimizer.py:2039
        if (ROUND_DECAY) {                                        // Tensor.mul_ on a bf16 tensor rounds to bf16
            const uint32_t pk = bf16x2_rn(x.x, x.y);
            x = make_float2(__uint_as_float(pk << 16), __uint_as_float(pk & 0xffff0000u));
        }
        u = __fmul2_rn(u, fira2);                                 // optimizer.py:803 (1 without a limiter)
        if (!S.zero_upd) x = __ffma2_rn(step2, u, x);             // optimizer.py:874; non-finite norm: zero update (optimizer.py:798-800)
        p[j] = x;
    }
}

__device__ __forceinline__ void unpack_bf16x4(uint2 w, float2 &a, float2 &b)
{
    a = make_float2(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u));
    b = make_float2(__uint_as_float(w.y << 16), __uint_as_float(w.y & 0xffff0000u));
}

// low bytes of four words
__device__ __forceinline__ uint32_t pack4(uint32_t a, uint32_t b, uint32_t c, uint32_t d)
{
    return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}

// element j of a register array, for the rare paths that are kept rolled: the kernel's hot loop is about
// 14 KB of code, and unrolled copies of the exact sequences between its parts cost more in instruction
// fetches than anything else (a quarter of the stall cycles in an earlier version)
template <int N>
__device__ __forceinline__ float pick(const float (&x)[N], int j)
{
    float r = x[0];
#pragma unroll
    for (int k = 1; k < N; ++k) r = j == k ? x[k] : r;
    return r;
}
template <int N, typename T>
__device__ __forceinline__ void put(T (&x)[N], int j, T value)
{
#pragma unroll
    for (int k = 0; k < N; ++k) x[k] = j == k ? value : x[k];
}

// the inputs of a thread's eight elements of one momentum block (groups at oa and oa + 128) from a ring slot
// REGULAR: the block's range is finite
template <typename GradT, typename ParamT, int VB, int MF, bool REGULAR>
__device__ __forceinline__ void fast_load8(const unsigned char *st, int oa, const float *tab, float v_scale, float v_min_log, float m_scale,
                                           const LaneTables &LT, float2 (&p)[4], float2 (&g)[4], float2 (&v_old)[4], float2 (&m_old)[4])
{
    using Ring = FastRing<GradT, ParamT, VB, MF>;
    const int ob = oa + 128;
    if (Ring::PB == 4) {
        const float4 a = *reinterpret_cast<const float4 *>(st + Ring::P_OFF + oa * 4);
        const float4 c = *reinterpret_cast<const float4 *>(st + Ring::P_OFF + ob * 4);
        p[0] = make_float2(a.x, a.y); p[1] = make_float2(a.z, a.w); p[2] = make_float2(c.x, c.y); p[3] = make_float2(c.z, c.w);
    } else {
        unpack_bf16x4(*reinterpret_cast<const uint2 *>(st + Ring::P_OFF + oa * 2), p[0], p[1]);
        unpack_bf16x4(*reinterpret_cast<const uint2 *>(st + Ring::P_OFF + ob * 2), p[2], p[3]);
    }
    if (Ring::GB == 4) {
        const float4 a = *reinterpret_cast<const float4 *>(st + Ring::G_OFF + oa * 4);
        const float4 c = *reinterpret_cast<const float4 *>(st + Ring::G_OFF + ob * 4);
        g[0] = make_float2(a.x, a.y); g[1] = make_float2(a.z, a.w); g[2] = make_float2(c.x, c.y); g[3] = make_float2(c.z, c.w);
    } else {
        unpack_bf16x4(*reinterpret_cast<const uint2 *>(st + Ring::G_OFF + oa * 2), g[0], g[1]);
        unpack_bf16x4(*reinterpret_cast<const uint2 *>(st + Ring::G_OFF + ob * 2), g[2], g[3]);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int o = h ? ob : oa;
        if (VB == 8) {
            const uint32_t w = *reinterpret_cast<const uint32_t *>(st + Ring::VQ_OFF + o);
            v_old[2 * h] = make_float2(tab[w & 0xffu], tab[__byte_perm(w, 0u, 0x4441u)]);
            v_old[2 * h + 1] = make_float2(tab[__byte_perm(w, 0u, 0x4442u)], tab[w >> 24]);
        } else {
            const uint2 w = *reinterpret_cast<const uint2 *>(st + Ring::VQ_OFF + o * 2);
            v_old[2 * h] = al16_decode2(w.x, v_scale, v_min_log, LT);
            v_old[2 * h + 1] = al16_decode2(w.y, v_scale, v_min_log, LT);
            if (!REGULAR && !range_finite(v_scale, v_min_log)) {     // code 0 is zero, the others infinity or NaN
                const float x1 = al_decode(1u, v_scale, v_min_log, 65534.0f), x2 = al_decode(2u, v_scale, v_min_log, 65534.0f);
                const auto value = [=](uint32_t c) { return c == 0u ? 0.0f : c == 1u ? x1 : x2; };
                v_old[2 * h] = make_float2(value(w.x & 0xffffu), value(w.x >> 16));
                v_old[2 * h + 1] = make_float2(value(w.y & 0xffffu), value(w.y >> 16));
            }
        }
        if (MF == AF8_M_UF8) {
            // (byte - 128) * fl(scale / 128) (optimizer.py:528-531): a power-of-two divisor, and
            // m_scale >= 1e-12 keeps the quotient far from the subnormal range
            const float2 mc2 = bc2(__fmul_rn(m_scale, 0.0078125f));
            const uint32_t w = *reinterpret_cast<const uint32_t *>(st + Ring::MQ_OFF + o);
            const float2 x = make_float2(__uint_as_float(__byte_perm(w, 0x4b000000u, 0x7540u)), __uint_as_float(__byte_perm(w, 0x4b000000u, 0x7541u)));
            const float2 y = make_float2(__uint_as_float(__byte_perm(w, 0x4b000000u, 0x7542u)), __uint_as_float(__byte_perm(w, 0x4b000000u, 0x7543u)));
            m_old[2 * h] = __fmul2_rn(__fadd2_rn(x, bc2(-8388736.0f)), mc2);
            m_old[2 * h + 1] = __fmul2_rn(__fadd2_rn(y, bc2(-8388736.0f)), mc2);
        } else if (MF == AF8_M_UF4) {
            // (nibble - 8) * fl(scale / 8), the even element in the high nibble
            const float2 mc2 = bc2(__fmul_rn(m_scale, 0.125f));
            const uint32_t w = *reinterpret_cast<const uint16_t *>(st + Ring::MQ_OFF + o / 2);
            const float2 x = make_float2(__uint_as_float(0x4b000000u | ((w >> 4) & 15u)), __uint_as_float(0x4b000000u | (w & 15u)));
            const float2 y = make_float2(__uint_as_float(0x4b000000u | (w >> 12)), __uint_as_float(0x4b000000u | ((w >> 8) & 15u)));
            m_old[2 * h] = __fmul2_rn(__fadd2_rn(x, bc2(-8388616.0f)), mc2);
            m_old[2 * h + 1] = __fmul2_rn(__fadd2_rn(y, bc2(-8388616.0f)), mc2);
        } else {
            m_old[2 * h] = m_old[2 * h + 1] = make_float2(0.0f, 0.0f);
        }
    }
}

// Requantisation of one momentum block: 32 lanes of eight elements, groups at e and e + 128
// (optimizer.py:510, 518).  Writes the codes and the scale when `live`.  STRICT: infinities and NaNs as in the general
// kernel, which leaves NaNs out of the largest magnitude and gives both the code of zero.
template <int MF, bool STRICT>
__device__ __forceinline__ void fast_store_m(const float2 (&m)[4], uint8_t *m_q, float *m_scale, int64_t e, bool live, int lane)
{
    const auto top3 = [](float a, float b, float c) { return STRICT ? max3_nan(a, b, c) : max3(a, b, c); };
    float amx = fabsf(m[0].x);
    amx = top3(amx, fabsf(m[0].y), fabsf(m[1].x));
    amx = top3(amx, fabsf(m[1].y), fabsf(m[2].x));
    amx = top3(amx, fabsf(m[2].y), fabsf(m[3].x));
    amx = top3(amx, fabsf(m[3].y), 0.0f);
    // non-negative floats order like their bit patterns: one REDUX instead of a shuffle tree
    const uint32_t abits = __reduce_max_sync(0xffffffffu, __float_as_uint(amx));
    float am = fmaxf(__uint_as_float(abits), 1e-12f);
    const float2 ra2 = bc2(__frcp_rn(am)), nam2 = bc2(-am);
    // round(m / am * levels) (the product with the power of two is exact); |m / am| <= 1, so only
    // +levels needs the clamp to levels - 1
    constexpr float LEVELS = MF == AF8_M_UF4 ? 8.0f : 128.0f;
    constexpr int TOP = MF == AF8_M_UF4 ? 7 : 127;
    uint32_t raw[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 kf = __ffma2_rn(div2_by(m[j], ra2, nam2), bc2(LEVELS), bc2(AF8_MAGIC_F));
        raw[2 * j] = (uint32_t)min(__float_as_int(kf.x), AF8_MAGIC_I + TOP);
        raw[2 * j + 1] = (uint32_t)min(__float_as_int(kf.y), AF8_MAGIC_I + TOP);
    }
    if (STRICT && abits >= 0x7f800000u) {      // an infinity or a NaN in the block
        float x[8];
        amx = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; ++j) { x[j] = j & 1 ? m[j >> 1].y : m[j >> 1].x; amx = fmaxf(amx, fabsf(x[j])); }
        am = fmaxf(warp_max(amx), 1e-12f);
#pragma unroll
        for (int j = 0; j < 8; ++j) raw[j] = (uint32_t)AF8_MAGIC_I + (MF == AF8_M_UF4 ? uf4_encode(x[j], am) - 8u : uf8_encode(x[j], am) - 128u);
    }
    if (!live) return;
    if (MF == AF8_M_UF8) {
        // low bytes hold k mod 256; k + 128 is that byte with its top bit flipped
        *reinterpret_cast<uint32_t *>(m_q + e) = pack4(raw[0], raw[1], raw[2], raw[3]) ^ 0x80808080u;
        *reinterpret_cast<uint32_t *>(m_q + e + 128) = pack4(raw[4], raw[5], raw[6], raw[7]) ^ 0x80808080u;
    } else {
        // low nibbles hold k mod 16; the first element of a byte is its high nibble
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t b0 = ((raw[4 * h] & 15u) << 4) | (raw[4 * h + 1] & 15u), b1 = ((raw[4 * h + 2] & 15u) << 4) | (raw[4 * h + 3] & 15u);
            *reinterpret_cast<uint16_t *>(m_q + ((e + 128 * h) >> 1)) = (uint16_t)((b0 | (b1 << 8)) ^ 0x8888u);
        }
    }
    if (lane == 0) *m_scale = am;
}

// The 16-bit patterns of eight new bf16 parameters (elements o .. o + 3 and o + 4 + GAP .. of the run that starts at base): the
// last rounding, to nearest or stochastic (optimizer.py:873-881).
template <bool SR, int GAP = 124>
__device__ __forceinline__ void fast_round8(const float2 (&p)[4], uint64_t sr_base, int64_t base, int o, const SrCounter &counter, uint32_t (&w)[4])
{
    if (!SR) {
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = bf16x2_rn(p[j].x, p[j].y);
        return;
    }
    float top = 0.0f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t k = (uint32_t)(o + (j < 2 ? 0 : GAP) + 2 * j);
        w[j] = sr_bf16x2(p[j].x, p[j].y, sr_hi32(counter, k), sr_hi32(counter, k + 1u));
        top = max3_nan(top, fabsf(p[j].x), fabsf(p[j].y));
    }
    if (!(top < 3.3895314e38f) || !counter.shared) {      // an infinity, a NaN, a step into an infinity; or counters that do not share their upper bits
        const float x[8] = {p[0].x, p[0].y, p[1].x, p[1].y, p[2].x, p[2].y, p[3].x, p[3].y};
#pragma unroll 1
        for (int k = 0; k < 4; ++k) {
            const uint64_t i = (uint64_t)(base + o + (k < 2 ? 0 : GAP) + 2 * k);
            put(w, k, sr_bf16_bits(pick(x, 2 * k), sr_bits24(sr_base, i)) | (sr_bf16_bits(pick(x, 2 * k + 1), sr_bits24(sr_base, i + 1)) << 16));
        }
    }
}

// The four new second moments of the group at o, in place of its consumed inputs in the ring slot: 16 bytes of fp32
// parameters, or 8 of bf16 parameters and 8 of gradients.
template <int PB, int P_OFF, int G_OFF>
__device__ __forceinline__ void stash_put(unsigned char *st, int o, float a, float b, float c, float d)
{
    if (PB == 4) {
        *reinterpret_cast<float4 *>(st + P_OFF + o * 4) = make_float4(a, b, c, d);
    } else {
        *reinterpret_cast<float2 *>(st + P_OFF + o * 2) = make_float2(a, b);
        *reinterpret_cast<float2 *>(st + G_OFF + o * 2) = make_float2(c, d);
    }
}
template <int PB, int P_OFF, int G_OFF>
__device__ __forceinline__ float4 stash_get(const unsigned char *st, int o)
{
    if (PB == 4) return *reinterpret_cast<const float4 *>(st + P_OFF + o * 4);
    const float2 a = *reinterpret_cast<const float2 *>(st + P_OFF + o * 2), b = *reinterpret_cast<const float2 *>(st + G_OFF + o * 2);
    return make_float4(a.x, a.y, b.x, b.y);
}
template <int PB, int P_OFF, int G_OFF>
__device__ __forceinline__ float *stash_at(unsigned char *st, int e)
{
    if (PB == 4) return reinterpret_cast<float *>(st + P_OFF) + e;
    return reinterpret_cast<float *>(st + ((e & 2) ? G_OFF : P_OFF) + (e & ~3) * 2) + (e & 1);
}

// Bulk copies of the full blocks b + from * G .. b + (to - 1) * G into their ring slots (one thread).
template <typename Ring, int MF>
__device__ __forceinline__ void fast_issue(const af8_fullrank_tensor &sT, unsigned char *ring, uint64_t *full, int b, int G, int n, int from, int to)
{
    constexpr int VQ = Ring::VQ_BYTES / (FAST_VBLOCK / 8);       // bits per second-moment code
    const unsigned char *gp = static_cast<const unsigned char *>(sT.grad);
    const unsigned char *pp = static_cast<const unsigned char *>(sT.param);
    const unsigned char *vp = static_cast<const unsigned char *>(sT.v_q);
    fence_proxy_async();
    for (int k = from; k < to; ++k) {
        const int64_t nb = (int64_t)(b + k * G) * FAST_VBLOCK;
        const int sl = (n + k) % Ring::NST;
        unsigned char *dst = ring + sl * Ring::STAGE_BYTES;
        mbar_expect_tx(&full[sl], Ring::STAGE_BYTES);
        bulk_g2s(dst + Ring::P_OFF, pp + nb * Ring::PB, FAST_VBLOCK * Ring::PB, &full[sl]);
        bulk_g2s(dst + Ring::G_OFF, gp + nb * Ring::GB, FAST_VBLOCK * Ring::GB, &full[sl]);
        bulk_g2s(dst + Ring::VQ_OFF, vp + nb * (VQ / 8), Ring::VQ_BYTES, &full[sl]);
        if (MF != AF8_M_NONE)
            bulk_g2s(dst + Ring::MQ_OFF, sT.m_q + (MF == AF8_M_UF4 ? nb / 2 : nb), Ring::MQ_BYTES, &full[sl]);
    }
}

// SR: bf16 parameters rounded stochastically.  LAG: the scalars are those of the previous step and the
// sum of squares of this step's raw update goes to block_sumsq.  ROOT_FTZ: every eps of the table is at least EPS_HIDES.
// (A kernel of its own: chosen per tensor or per block inside one kernel, the two forms cost the common one 2 to 15 %
// in registers and instruction fetches.  TinyLlama-1.1B, UF8/AL8: 2.69 ms with ROOT_FTZ, 2.94 ms with ROOT_FULL.)
template <typename GradT, typename ParamT, int VB, int MF, bool SR, bool LAG, int ROOT>
__global__ void __launch_bounds__(FAST_THREADS, fast_min_ctas<VB>())
fullrank_fast_kernel(const FullrankLaunch L)
{
    using Ring = FastRing<GradT, ParamT, VB, MF>;
    using PElem = typename ParamElem<ParamT>::type;
    constexpr int GB = Ring::GB, PB = Ring::PB, NST = Ring::NST, STAGE_BYTES = Ring::STAGE_BYTES;
    constexpr int P_OFF = Ring::P_OFF, G_OFF = Ring::G_OFF, VQ_OFF = Ring::VQ_OFF, MQ_OFF = Ring::MQ_OFF;
    constexpr int MPB = FAST_VBLOCK / FAST_MBLOCK;                // momentum blocks per V block
    constexpr int QMAX = VB == 16 ? 65535 : 255;
    constexpr float QM1 = VB == 16 ? 65534.0f : 254.0f;
    constexpr bool TABLE = VB == 8;
    constexpr bool STASH = fast_stash<VB>();
    constexpr int MB_UNROLL = STASH ? 1 : 2;
    static_assert(!STASH || NST == 2, "a slot that is left is refilled for the block after the next one");
    // Infinities and NaNs in whole blocks as in the general kernel.  Not with UF8/AL8, where their tests cost 8 % of the
    // update pass: there a NaN is left out of the range and of the largest magnitude.
    constexpr bool STRICT = root_exact<VB, MF>;

    extern __shared__ __align__(128) unsigned char s_ring[];     // NST slots of STAGE_BYTES
    __shared__ __align__(8) uint64_t s_full[NST];
    __shared__ __align__(16) af8_fullrank_tensor sT;
    __shared__ StepScalars sS;
    __shared__ float s_tab[2][TABLE ? 256 : 1];
    __shared__ uint32_t s_redmin[FAST_WARPS];
    __shared__ uint32_t s_redmax[FAST_WARPS];
    __shared__ float s_usq[FAST_WARPS];
    __shared__ VRange s_vr;
    __shared__ int s_abort;
    __shared__ int s_left;                           // STASH: warps that have left a slot, a running count
    __shared__ double s_exp2[TABLE ? 32 : 1];        // copy of the exp2 table of the decode
    __shared__ double2 s_log2[97];                   // copy of the log2 table of the range computation

    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    const int ow = warp * (FAST_EPT * 32) + lane * 4;   // first group of four of this thread; the others follow at 128, 256, ...

    if (TABLE && tid < 32) s_exp2[tid] = c_exp2_tab[tid];
    if (tid < 97) s_log2[tid] = c_log2_tab[tid];
    LaneTables LT;
    if (!TABLE) { LT.e2 = c_exp2_tab[lane]; LT.l2 = c_log2_lane[lane].l2; LT.inv_hi = c_log2_lane[lane].inv_hi; }
    if (tid == 0) {
        for (int k = 0; k < NST; ++k) mbar_init(&s_full[k], 1);
        s_abort = 0;
        s_left = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    await_launches();

    int cur_t = -1;
    int64_t cur_first = 0, cur_end = 0;      // block range of the current tensor
    int nfull = 0;                           // number of full blocks of the current tensor
    const int G = (int)gridDim.x;
    uint32_t phase = 0;                      // bit k: parity to wait for on ring slot k
    int ahead = 0;                           // consecutive blocks from the current one whose copies are in flight
    bool staged = false;                     // this block's decode table and ranges were prepared last iteration
    float csc = 0.f, cml = 0.f;              // range of this block (AL16: the elements are decoded with it)
    float nsc = 0.f, nml = 0.f;              // prefetched range of the next block
    float cms[2] = {0.f, 0.f}, nms[2] = {0.f, 0.f};   // momentum scales of this warp's two blocks, and the next ones
    int n = 0;

    for (int64_t blk = blockIdx.x; blk < L.total_blocks; blk += gridDim.x, ++n) {
        // ---- tensor change (rare, uniform over the CTA) ----
        if (cur_t < 0 || blk >= cur_end) {
            int t = cur_t;
            if (t < 0) {
                t = find_tensor(L.tensors, L.n_tensors, blk);
            } else {
                while (t + 1 < L.n_tensors && L.tensors[t + 1].first_block <= blk) ++t;
            }
            __syncthreads();
            if (tid < (int)(sizeof(af8_fullrank_tensor) / 4))
                reinterpret_cast<uint32_t *>(&sT)[tid] =
                    reinterpret_cast<const uint32_t *>(L.tensors + t)[tid];
            __syncthreads();
            if (tid == 0) {
                StepScalars S;
                S.decay = sT.decay; S.step_mul = -sT.alpha; S.fira = 1.0f; S.eps_d = sT.eps_denom;
                S.v_w = sT.v_w; S.m_w = MF == AF8_M_NONE ? 0.0f : sT.m_w; S.eps_g = sT.eps_gradsq;
                S.zero_upd = 0;
                if (L.dyn != nullptr) {
                    const af8_dyn_scalars ds = L.dyn[t];
                    S.step_mul = ds.step; S.fira = ds.fira; S.zero_upd = ds.zero != 0.0f;
                }
                S.plain = fabsf(S.v_w) < 0.5f && fabsf(S.m_w) < 0.5f && S.eps_g == 0.0f;
                sS = S;
            }
            __syncthreads();
            cur_t = t;
            cur_first = sT.first_block;
            cur_end = cur_first + (sT.numel + FAST_VBLOCK - 1) / FAST_VBLOCK;
            nfull = (int)(sT.numel / FAST_VBLOCK);   // a tensor has fewer than 2^31 blocks (checked on the host)
            staged = false;                          // (ahead is 0 here: copies never cross a tensor)
        }
        const int b = (int)(blk - cur_first);         // V block index inside the tensor
        const int64_t base = (int64_t)b * FAST_VBLOCK;   // first element of the block
        const bool full = b < nfull;
        const int rem = full ? FAST_VBLOCK : (int)(sT.numel - base);   // real elements from base on (> 0)
        const int stage = n & 1;                      // decode-table buffer of this block
        const int slot = n % NST;                     // ring slot of this block
        const int b_next = b + G;
        // blocks blk, blk+G, ... that are full blocks of this tensor get their copies issued ahead
        int want = 0;
#pragma unroll
        for (int k = 0; k < NST; ++k)
            if (want == k && b + k * G < nfull) want = k + 1;
        const bool next_staged = want >= 2;           // the next block gets its table and ranges prepared here

        // ---- issue the bulk copies (one thread; STASH: the first ones of a tensor, the others when a slot is left) ----
        if (tid == 0 && ahead < want && (!STASH || ahead == 0)) fast_issue<Ring, MF>(sT, s_ring, s_full, b, G, n, ahead, want);
        const int in_flight = want;                   // copies outstanding now, this block included
        ahead = want > 0 ? want - 1 : 0;              // ... as seen from the next block
        // ---- ranges of this block (if not prefetched) and of the next one ----
        if (!staged) {
            csc = load_state(sT.v_scale + b);
            cml = load_state(sT.v_min_log + b);
            if (MF != AF8_M_NONE) {
#pragma unroll
                for (int k = 0; k < 2; ++k)           // (momentum blocks beyond the tensor are not allocated)
                    cms[k] = (2 * warp + k) * FAST_MBLOCK < rem ? load_state(sT.m_scale + (int64_t)b * MPB + 2 * warp + k) : 0.0f;
            }
            if (TABLE) {
                s_tab[stage][tid] = al8_decode_fast<STRICT>((uint32_t)tid, csc, cml, s_exp2);   // optimizer.py:341-349
                s_tab[stage][tid + 128] = al8_decode_fast<STRICT>((uint32_t)tid + 128u, csc, cml, s_exp2);
            }
            __syncthreads();
        }
        if (next_staged) {
            nsc = load_state(sT.v_scale + b_next);
            nml = load_state(sT.v_min_log + b_next);
            if (MF != AF8_M_NONE) {
                const float2 x = make_float2(load_state(sT.m_scale + (int64_t)b_next * MPB + 2 * warp), load_state(sT.m_scale + (int64_t)b_next * MPB + 2 * warp + 1));
                nms[0] = x.x; nms[1] = x.y;
            }
        }

        // ---- this block's inputs in its ring slot ----
        unsigned char *const st = s_ring + slot * STAGE_BYTES;
        bool bad = false;
        if (full) {
            if (!mbar_wait_bounded(&s_full[slot], (phase >> slot) & 1u)) {
                bad = true;      // this thread stores nothing for the block
                s_abort = 1;     // and the CTA stops at the next block-wide barrier
                atomicExch(&g_device_error, DEVERR_COPY_TIMEOUT);
            }
            phase ^= 1u << slot;
        } else {
            // Tail block: guarded plain loads into the slot.  Beyond the end the gradient and the parameter are
            // zero; the V state is padded to the block, the M state only to its own 256-element blocks.
#pragma unroll 1
            for (int e = tid; e < FAST_VBLOCK; e += FAST_THREADS) {
                const bool ok = e < rem;
                if (PB == 4) reinterpret_cast<float *>(st + P_OFF)[e] = ok ? static_cast<const float *>(sT.param)[base + e] : 0.0f;
                else reinterpret_cast<uint16_t *>(st + P_OFF)[e] = ok ? static_cast<const uint16_t *>(sT.param)[base + e] : (uint16_t)0;
                if (GB == 4) reinterpret_cast<float *>(st + G_OFF)[e] = ok ? static_cast<const float *>(sT.grad)[base + e] : 0.0f;
                else reinterpret_cast<uint16_t *>(st + G_OFF)[e] = ok ? static_cast<const uint16_t *>(sT.grad)[base + e] : (uint16_t)0;
                if (VB == 8) (st + VQ_OFF)[e] = static_cast<const uint8_t *>(sT.v_q)[base + e];
                else reinterpret_cast<uint16_t *>(st + VQ_OFF)[e] = static_cast<const uint16_t *>(sT.v_q)[base + e];
                const bool m_ok = (e & ~(FAST_MBLOCK - 1)) < rem;
                if (MF == AF8_M_UF8) (st + MQ_OFF)[e] = m_ok ? sT.m_q[base + e] : (uint8_t)128;
                if (MF == AF8_M_UF4 && (e & 1) == 0) (st + MQ_OFF)[e >> 1] = m_ok ? sT.m_q[(base + e) >> 1] : (uint8_t)0x88;
            }
            __syncthreads();
        }

        const StepScalars S = sS;
        SrCounter counter = {};
        if (SR) counter = sr_counter(sT.sr_base, base, FAST_VBLOCK);
        // (uniform over the CTA; a block that decodes to infinities or NaNs takes the general forms: ROOT_REFINED would lose a NaN)
        const bool hot = full && S.plain && (!root_exact<VB, MF> || range_finite(csc, cml));
        float v[STASH ? 8 : FAST_EPT];       // hot blocks: the new second moments (STASH: of one momentum block)
        float usq = 0.0f;                    // LAG: this thread's sum of squares of the raw update
        // Extrema of v.  v >= 0, so the bit patterns order like the values.  The minimum runs over the
        // non-zero elements (optimizer.py:312-313) and travels as bits - 1, which sends "none" to the top.
        uint32_t umin, umax;

        if (hot) {
            // ---- two momentum blocks per warp: EMAs, update, parameter, momentum codes ----
            float fmn = INFINITY, fmx = 0.0f;    // (STRICT: a NaN reaches fmx, else neither)
#pragma unroll (MB_UNROLL)
            for (int mb = 0; mb < 2; ++mb) {
                const int oa = ow + mb * FAST_MBLOCK;
                float2 g[4], p[4], v_old[4], m_old[4], vn[4], mn[4];
                fast_load8<GradT, ParamT, VB, MF, true>(st, oa, s_tab[stage], csc, cml, STASH ? (mb ? cms[1] : cms[0]) : cms[mb], LT, p, g, v_old, m_old);
                if (L.negate_grad) {                              // maximize (optimizer.py:1973-1974)
#pragma unroll
                    for (int j = 0; j < 4; ++j) g[j] = make_float2(-g[j].x, -g[j].y);
                }
                fast_ema8<MF, true, PB == 2 && !SR, LAG, ROOT>(S, g, v_old, m_old, p, vn, mn, 0xffu, usq);
#pragma unroll
                for (int j = 0; j < 4; ++j) { v[(STASH ? 0 : 8 * mb) + 2 * j] = vn[j].x; v[(STASH ? 0 : 8 * mb) + 2 * j + 1] = vn[j].y; }
                if constexpr (STASH) {
                    stash_put<PB, P_OFF, G_OFF>(st, oa, v[0], v[1], v[2], v[3]);
                    stash_put<PB, P_OFF, G_OFF>(st, oa + 128, v[4], v[5], v[6], v[7]);
#pragma unroll
                    for (int j = 0; j < 8; j += 2) {
                        fmn = min3(fmn, v[j], v[j + 1]);
                        fmx = STRICT ? max3_nan(fmx, v[j], v[j + 1]) : max3(fmx, v[j], v[j + 1]);
                    }
                }
                PElem *const pa = static_cast<PElem *>(sT.param) + base + oa;
                if (PB == 4) {
                    if (!bad) {
                        *reinterpret_cast<float4 *>(pa) = make_float4(p[0].x, p[0].y, p[1].x, p[1].y);
                        *reinterpret_cast<float4 *>(pa + 128) = make_float4(p[2].x, p[2].y, p[3].x, p[3].y);
                        if (sT.param_copy != nullptr) {           // bf16 compute copy
                            uint16_t *const ca = static_cast<uint16_t *>(sT.param_copy) + base + oa;
                            *reinterpret_cast<uint2 *>(ca) = make_uint2(bf16x2_rn(p[0].x, p[0].y), bf16x2_rn(p[1].x, p[1].y));
                            *reinterpret_cast<uint2 *>(ca + 128) = make_uint2(bf16x2_rn(p[2].x, p[2].y), bf16x2_rn(p[3].x, p[3].y));
                        }
                    }
                } else {
                    uint32_t w[4];
                    fast_round8<SR>(p, sT.sr_base, base, oa, counter, w);
                    if (!bad) {
                        *reinterpret_cast<uint2 *>(pa) = make_uint2(w[0], w[1]);
                        *reinterpret_cast<uint2 *>(pa + 128) = make_uint2(w[2], w[3]);
                    }
                }
                if (MF != AF8_M_NONE)
                    fast_store_m<MF, STRICT>(mn, sT.m_q, sT.m_scale + (int64_t)b * MPB + 2 * warp + mb, base + oa, !bad, lane);
            }
            if constexpr (!STASH) {
                fmn = fmx = v[0];
#pragma unroll
                for (int j = 1; j + 1 < FAST_EPT; j += 2) {
                    fmn = min3(fmn, v[j], v[j + 1]);
                    fmx = STRICT ? max3_nan(fmx, v[j], v[j + 1]) : max3(fmx, v[j], v[j + 1]);
                }
                fmn = fminf(fmn, v[FAST_EPT - 1]);
                fmx = STRICT ? max3_nan(fmx, v[FAST_EPT - 1], v[FAST_EPT - 1]) : fmaxf(fmx, v[FAST_EPT - 1]);
            }
            umin = __reduce_min_sync(0xffffffffu, __float_as_uint(fmn));
            umax = __reduce_max_sync(0xffffffffu, __float_as_uint(fmx));
            if (umin == 0u || (STRICT && umax > 0x7f800000u)) {      // the warp holds a zero (rare after the first steps, except in all-zero regions) or a NaN
                uint32_t um = 0xffffffffu, ux = 0u;
                if constexpr (STASH) {
#pragma unroll 1
                    for (int q = 0; q < FAST_EPT; ++q) {
                        float *const x = stash_at<PB, P_OFF, G_OFF>(st, ow + (q >> 2) * 128 + (q & 3));
                        if (!(*x >= 0.0f)) *x = AF8_TINY;                // (see al_log2)
                        um = min(um, __float_as_uint(*x) - 1u);
                        ux = max(ux, __float_as_uint(*x));
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < FAST_EPT; ++j) {
                        if (STRICT && !(v[j] >= 0.0f)) v[j] = AF8_TINY;
                        um = min(um, __float_as_uint(v[j]) - 1u);
                        if (STRICT) ux = max(ux, __float_as_uint(v[j]));
                    }
                }
                umin = __reduce_min_sync(0xffffffffu, um);
                if (STRICT) umax = __reduce_max_sync(0xffffffffu, ux);
            } else {
                umin -= 1u;
            }
        } else {
            // ---- a tail block, or uncommon scalars: the general forms, rolled, the new second moments in place of
            //      the consumed inputs in the ring slot ----
            umin = 0xffffffffu;
            umax = 0u;
#pragma unroll 1
            for (int mb = 0; mb < 2; ++mb) {
                const int oa = ow + mb * FAST_MBLOCK;
                float2 g[4], p[4], v_old[4], m_old[4], vn[4], mn[4];
                fast_load8<GradT, ParamT, VB, MF, false>(st, oa, s_tab[stage], csc, cml, mb ? cms[1] : cms[0], LT, p, g, v_old, m_old);
                if (L.negate_grad) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) g[j] = make_float2(-g[j].x, -g[j].y);
                }
                uint32_t real = 0u;                               // bit j: element j exists
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if ((j < 4 ? oa : oa + 124) + j < rem) real |= 1u << j;
                fast_ema8<MF, false, PB == 2 && !SR, LAG, root_exact<VB, MF> ? ROOT_EXACT : ROOT>(S, g, v_old, m_old, p, vn, mn, real, usq);
                float x[8], q[8];
                uint32_t w[4] = {0u, 0u, 0u, 0u};
                if (PB == 2) fast_round8<SR>(p, sT.sr_base, base, oa, counter, w);
#pragma unroll
                for (int j = 0; j < 4; ++j) {                     // padding re-enters both states as zero
                    if (!((real >> (2 * j)) & 1u)) { vn[j].x = 0.0f; mn[j].x = 0.0f; }
                    if (!((real >> (2 * j + 1)) & 1u)) { vn[j].y = 0.0f; mn[j].y = 0.0f; }
                    if (!(vn[j].x >= 0.0f)) vn[j].x = STRICT ? AF8_TINY : 0.0f;      // NaN (see al_log2)
                    if (!(vn[j].y >= 0.0f)) vn[j].y = STRICT ? AF8_TINY : 0.0f;
                    x[2 * j] = vn[j].x; x[2 * j + 1] = vn[j].y;
                    q[2 * j] = p[j].x; q[2 * j + 1] = p[j].y;
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    umin = min(umin, __float_as_uint(x[j]) - 1u);
                    umax = max(umax, __float_as_uint(x[j]));
                    const int e = (j < 4 ? oa : oa + 124) + j;
                    if (((real >> j) & 1u) && !bad) {
                        if (PB == 4) {
                            static_cast<float *>(sT.param)[base + e] = q[j];
                            if (sT.param_copy != nullptr) static_cast<uint16_t *>(sT.param_copy)[base + e] = (uint16_t)f32_to_bf16_rn_bits(q[j]);
                        } else {
                            static_cast<uint16_t *>(sT.param)[base + e] = (uint16_t)(w[j >> 1] >> (16 * (j & 1)));
                        }
                    }
                }
                if (MF != AF8_M_NONE)
                    fast_store_m<MF, STRICT>(mn, sT.m_q, sT.m_scale + (int64_t)b * MPB + 2 * warp + mb, base + oa,
                                     (2 * warp + mb) * FAST_MBLOCK < rem && !bad, lane);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int o = oa + 128 * h;
                    if (PB == 4) {
                        *reinterpret_cast<float4 *>(st + P_OFF + o * 4) = make_float4(x[4 * h], x[4 * h + 1], x[4 * h + 2], x[4 * h + 3]);
                    } else {
                        *reinterpret_cast<float2 *>(st + P_OFF + o * 2) = make_float2(x[4 * h], x[4 * h + 1]);
                        *reinterpret_cast<float2 *>(st + G_OFF + o * 2) = make_float2(x[4 * h + 2], x[4 * h + 3]);
                    }
                }
            }
            umin = __reduce_min_sync(0xffffffffu, umin);
            umax = __reduce_max_sync(0xffffffffu, umax);
        }
        if (lane == 0) { s_redmin[warp] = umin; s_redmax[warp] = umax; }
        if (LAG) {                           // the block's sum of squares travels with the extrema
            const float ws = warp_sum(usq);
            if (lane == 0) s_usq[warp] = ws;
        }
        // ---- D: only warp 0 consumes the extrema; the other warps signal and move on ----
        if (warp == 0) asm volatile("bar.sync 1, %0;" ::"n"(FAST_THREADS) : "memory");
        else asm volatile("bar.arrive 1, %0;" ::"n"(FAST_THREADS) : "memory");

        // ---- warp 0: exact log2 of the two extreme values only (optimizer.py:308-318) ----
        if (warp == 0) {
            umin = lane < FAST_WARPS ? s_redmin[lane] : 0xffffffffu;
            umax = lane < FAST_WARPS ? s_redmax[lane] : 0u;
            umin = __reduce_min_sync(0xffffffffu, umin);
            umax = __reduce_max_sync(0xffffffffu, umax);
            // lane 0 takes the log of the minimum, lane 1 of the maximum
            float lg = (lane == 0) ? ((umin == 0xffffffffu) ? INFINITY : al_log2_fast(__uint_as_float(umin + 1u), s_log2))
                                   : ((lane == 1) ? al_log2_fast(__uint_as_float(umax), s_log2) : 0.0f);
            const float mx_l = __shfl_sync(0xffffffffu, lg, 1);
            if (lane == 0) {
                const float mn = lg == 1024.0f ? INFINITY : lg;      // (infinite second moments)
                const float mx = mx_l == 1024.0f ? INFINITY : mx_l;
                VRange r;
                al_range(mn, mx, L.v_floor, r.min_log, r.scale);
                if (VB == 8) {
                    r.k = __fdiv_rn(254.0f, r.scale);
                    r.c = -__fmul_rn(r.min_log, r.k);
                    // Error bound of the estimate in code units.  In units of the logarithm, times k: the hardware log2, one
                    // rounding of min_log * k and one of the exact log2.  In codes (up to 254): the roundings of k and of the
                    // estimate, and the three of the exact sequence, 5 * 254 * 2^-24.  (With the bound twice as wide a warp redid a
                    // code in every third block instead of every sixth: 67 M parameters of one scale 177 us against 173, the
                    // RMSprop step of 110 M parameters 337 against 332.)
                    const float lmax = fmaxf(fmaxf(fabsf(r.min_log), fabsf(mx)), 1.0f);
                    const float err = __fmaf_rn(__fmaf_rn(lmax, LG2_REL + 1.22e-7f, LG2_ABS), r.k, 8.0e-5f);
                    r.thr = 0.5f - err;
                    // Exact path for every element of the block when the range is absurd (NaN / inf)
                    // or when some non-zero element lies below the floor (subnormal values with the
                    // default floor): the estimate path has no lower clamp and flushes subnormals.
                    if (!(r.k >= 1.0f) || L.v_floor < -126.0f || mn < L.v_floor) r.thr = -1.0f;
                } else {
                    r.k = __frcp_rn(r.scale);                    // for the quotient by the scale
                    r.c = 0.0f; r.thr = range_finite(r.scale, r.min_log) ? 0.0f : -1.0f;     // (negative: exact path)
                }
                s_vr = r;
                sT.v_scale[b] = r.scale;
                sT.v_min_log[b] = r.min_log;
                if (LAG) {
                    float s = 0.0f;
#pragma unroll
                    for (int w = 0; w < FAST_WARPS; ++w) s = __fadd_rn(s, s_usq[w]);
                    L.block_sumsq[blk] = s;
                }
            }
        }

        // ---- what does not need the range: the next block's decode table ----
        if (TABLE && next_staged) {
            s_tab[stage ^ 1][tid] = al8_decode_fast<STRICT>((uint32_t)tid, nsc, nml, s_exp2);
            s_tab[stage ^ 1][tid + 128] = al8_decode_fast<STRICT>((uint32_t)tid + 128u, nsc, nml, s_exp2);
        }
        __syncthreads();                     // ---- E ----
        if (s_abort) {       // a copy never completed: give the ones still in flight a bounded chance, then stop
            for (int k = 1; k < in_flight; ++k) mbar_wait_bounded(&s_full[(n + k) % NST], (phase >> ((n + k) % NST)) & 1u);
            break;
        }

        // ---- second-moment codes ----
        const VRange r = s_vr;
        if (!hot) {
            // the exact sequence for every element, from the values left in the ring slot
#pragma unroll 1
            for (int q = 0; q < FAST_EPT; ++q) {
                const int o = ow + (q >> 2) * 128, k = q & 3;
                const float x = PB == 4 ? reinterpret_cast<const float *>(st + P_OFF)[o + k]
                                        : reinterpret_cast<const float *>(st + (k < 2 ? P_OFF : G_OFF) + o * 2)[k & 1];
                const uint32_t c = al_encode(x, al_log2_fast(x, s_log2), r.min_log, r.scale, QM1, QMAX);
                if (VB == 8) static_cast<uint8_t *>(sT.v_q)[base + o + k] = (uint8_t)c;
                else static_cast<uint16_t *>(sT.v_q)[base + o + k] = (uint16_t)c;
            }
            __syncthreads();             // the slot may be refilled from the next iteration on
        } else if constexpr (VB == 8) {
            uint8_t *const vp = static_cast<uint8_t *>(sT.v_q) + base;
            const float2 k2 = bc2(r.k), c2 = bc2(r.c), mg2 = bc2(AF8_MAGIC_F + 1.0f), nmg2 = bc2(-(AF8_MAGIC_F + 1.0f));
#pragma unroll
            for (int mb = 0; mb < 2; ++mb) {
                float x[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) x[j] = v[8 * mb + j];
                uint32_t kk[8];
                float dd[8];
                float dmax = 0.0f;
#pragma unroll
                for (int j = 0; j < 8; j += 2) {
                    // An exact zero estimates as -inf: te and sm are -inf, whose low byte is 0, the
                    // reserved code, and d is NaN, which the tests below ignore.  Every other element
                    // of a block that takes this path is a normal number at or above min_log, so
                    // 0 <= t <= 254 up to the estimate's error and no clamp is needed.
                    const float2 le = make_float2(lg2_approx(x[j]), lg2_approx(x[j + 1]));
                    const float2 te = __ffma2_rn(le, k2, c2);
                    const float2 sm = __fadd2_rn(te, mg2);             // rint(te) + 1 in the low bits
                    const float2 rf = __fadd2_rn(sm, nmg2);
                    const float2 d = sub2(te, rf);                     // distance to the chosen integer
                    dd[j] = d.x; dd[j + 1] = d.y;
                    dmax = max3(dmax, fabsf(d.x), fabsf(d.y));         // (drops NaN)
                    kk[j] = __float_as_uint(sm.x); kk[j + 1] = __float_as_uint(sm.y);
                }
                if (dmax > r.thr) {
                    // rare: redo the codes in doubt with the exact sequence (an exact zero's distance is NaN and its code 0)
                    uint32_t odd = 0u;
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (!(fabsf(dd[j]) <= r.thr)) odd |= 1u << j;
#pragma unroll 1
                    for (; odd; odd &= odd - 1u) {
                        const int j = __ffs((int)odd) - 1;
                        const float y = pick(x, j);
                        put(kk, j, (uint32_t)AF8_MAGIC_I + al_encode(y, al_log2_fast(y, s_log2), r.min_log, r.scale, QM1, QMAX));
                    }
                }
                *reinterpret_cast<uint32_t *>(vp + ow + mb * FAST_MBLOCK) = pack4(kk[0], kk[1], kk[2], kk[3]);       // (not reached after a failed wait: the CTA left at E)
                *reinterpret_cast<uint32_t *>(vp + ow + mb * FAST_MBLOCK + 128) = pack4(kk[4], kk[5], kk[6], kk[7]);
            }
        } else if (r.thr < 0.0f) {
#pragma unroll 1
            for (int q = 0; q < FAST_EPT; ++q) {
                const float x = *stash_at<PB, P_OFF, G_OFF>(st, ow + (q >> 2) * 128 + (q & 3));
                static_cast<uint16_t *>(sT.v_q)[base + ow + (q >> 2) * 128 + (q & 3)] = (uint16_t)al_encode(x, al_log2_fast(x, s_log2), r.min_log, r.scale, QM1, QMAX);
            }
        } else {
            uint16_t *const vp = static_cast<uint16_t *>(sT.v_q) + base;
            const float2 nml2 = bc2(-r.min_log), rc2 = bc2(r.k), nd2 = bc2(-r.scale);
#pragma unroll
            for (int q = 0; q < FAST_EPT / 4; ++q) {
                uint32_t kk[4];
                const float4 v4 = stash_get<PB, P_OFF, G_OFF>(st, ow + q * 128);
                const float x[4] = {v4.x, v4.y, v4.z, v4.w};
                float lv[4];
                uint32_t odd = 0u;                               // subnormal second moments above the floor of 1e-38
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float l = log2_lane(x[j], LT);         // (shuffles: every lane takes part)
                    lv[j] = x[j] > AF8_TINY ? l : AF8_LOG2_TINY;
                    if (x[j] > AF8_TINY && x[j] < 1.17549435e-38f) odd |= 1u << j;
                }
#pragma unroll 1
                for (; odd; odd &= odd - 1u) {
                    const int j = __ffs((int)odd) - 1;
                    put(lv, j, log2_cr_fast(pick(x, j), s_log2));
                }
#pragma unroll
                for (int j = 0; j < 4; j += 2) {
                    // al_encode on a pair: (l - min_log) / scale * 65534, rounded, plus one (optimizer.py:320-321)
                    const float2 d = __fadd2_rn(make_float2(lv[j], lv[j + 1]), nml2);
                    const float2 q2 = div2_by(d, rc2, nd2);
                    // (below min_log: code 1, which the rounding constant would not give for a quotient of -2^6 and less)
                    const float2 t = make_float2(fmaxf(q2.x, 0.0f), fmaxf(q2.y, 0.0f));
                    // (scalar: the compiler fuses a packed product into a packed sum, which loses the rounding in between)
                    const int k0 = __float_as_int(__fadd_rn(__fmul_rn(t.x, QM1), AF8_MAGIC_F)) - (AF8_MAGIC_I - 1);
                    const int k1 = __float_as_int(__fadd_rn(__fmul_rn(t.y, QM1), AF8_MAGIC_F)) - (AF8_MAGIC_I - 1);
                    kk[j] = x[j] == 0.0f ? 0u : (uint32_t)min(k0, QMAX);
                    kk[j + 1] = x[j + 1] == 0.0f ? 0u : (uint32_t)min(k1, QMAX);
                }
                *reinterpret_cast<uint2 *>(vp + ow + q * 128) = make_uint2(kk[0] | (kk[1] << 16), kk[2] | (kk[3] << 16));
            }
        }
        if (STASH) {
            // the last warp to leave the slot has it refilled, for the block after the next one
            __syncwarp();
            if (lane == 0 && b + 2 * G < nfull) {
                __threadfence_block();
                if ((atomicAdd(&s_left, 1) & (FAST_WARPS - 1)) == FAST_WARPS - 1) {
                    __threadfence_block();
                    fast_issue<Ring, MF>(sT, s_ring, s_full, b, G, n, 2, 3);
                }
            }
        }
        staged = next_staged;
        csc = nsc; cml = nml;
        cms[0] = nms[0]; cms[1] = nms[1];
    }
}

}  // namespace af8
