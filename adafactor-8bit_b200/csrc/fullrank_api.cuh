// Host side of the full-rank step: argument validation, kernel selection and
// launch (af8_fullrank_step), and the per-tensor norm / Fira / clip finaliser
// (af8_norm_finalize).
#pragma once

#include "common.cuh"
#include "fullrank_fast.cuh"
#include "fullrank_generic.cuh"
#include "fullrank_stat.cuh"
#include "launch.cuh"

#include <atomic>

namespace af8 {

// ---------------------------------------------------------------------------
// norm finaliser: one CTA per tensor
// ---------------------------------------------------------------------------
// Reduces the tensor's per-block partial sums in a fixed order in binary64,
// then evaluates on one thread what the reference computes with 0-d tensors:
// _compute_fira_scale (optimizer.py:760-782), the clip denominators of
// _apply_fira_pytorch / _safe_rms_denom (optimizer.py:805-806, 859-863) and
// -alpha/denom (optimizer.py:874); in pre_div_mode 1 the RMS clip of the
// momentum-only rule (optimizer.py:897-899).
// 1024 threads: the largest tensor of the table decides how long the launch lasts (65.5 M elements, 32000 partial sums:
// 21 us with 256 threads, 13 with 1024 in binary64).
constexpr int FINALIZE_THREADS = 1024;
__global__ void __launch_bounds__(FINALIZE_THREADS)
norm_finalize_kernel(const af8_norm_tensor *tensors, const void *block_sumsq, af8_dyn_scalars *dyn)
{
    __shared__ double s_part[FINALIZE_THREADS / 32];
    await_launches();
    const af8_norm_tensor T = tensors[blockIdx.x];
    const double *const p64 = static_cast<const double *>(block_sumsq) + T.first_block;
    const float *const p32 = static_cast<const float *>(block_sumsq) + T.first_block;
    const double sum = T.n_blocks < 0 ? 0.0
                     : T.partials_f64 ? block_sum<FINALIZE_THREADS>(T.n_blocks, [=](int64_t i) { return p64[i]; }, s_part)
                                      : block_sum<FINALIZE_THREADS>(T.n_blocks, [=](int64_t i) { return (double)p32[i]; }, s_part);
    if (threadIdx.x != 0) return;

    const double total = T.n_blocks < 0 ? *reinterpret_cast<const double *>(static_cast<uintptr_t>(T.first_block)) : sum;
    float norm = __double2float_rn(sqrt(total));
    const float alpha = T.alpha_dev ? *T.alpha_dev : T.alpha;
    af8_dyn_scalars out = dyn[blockIdx.x];
    out.norm = norm;
    if (T.pre_div_mode == 1) {
        const float rms = __fdiv_rn(norm, T.sqrt_n);
        float cf = __fdiv_rn(rms, T.d);
        cf = (cf >= 1.0f || isnan(cf)) ? cf : 1.0f;
        out.pre_div = cf;
        out.step = -alpha;
        out.fira = 1.0f;
        out.zero = 0.0f;
        dyn[blockIdx.x] = out;
        return;
    }
    float fs = 1.0f;
    float zero = 0.0f;
    if (T.fira_prev != nullptr) {
        if (!isfinite(norm)) { zero = 1.0f; norm = 0.0f; }       // optimizer.py:798-800
        if (T.fira_has_prev) {
            const float fp = *T.fira_prev;
            const bool reset = fp < 1e-6f;                          // optimizer.py:774
            const float ratio = __fdiv_rn(norm, __fadd_rn(fp, 1e-8f));
            const float lim = __fdiv_rn(fmaxf(ratio, T.fira_margin1), T.fira_margin1);
            fs = reset ? 1.0f : __frcp_rn(lim);                     // optimizer.py:777
            *T.fira_prev = reset ? norm : __fmul_rn(norm, fs);      // optimizer.py:778
        } else {
            *T.fira_prev = norm;                                    // optimizer.py:780-781
        }
    }
    float denom = 1.0f;
    if (T.clip_div > 0.0f) {
        const float x = __fdiv_rn(norm, T.clip_div);
        denom = (x >= 1.0f || isnan(x)) ? x : 1.0f;
    }
    out.step = __fdiv_rn(-alpha, denom);
    out.fira = fs;
    out.zero = zero;
    if (T.pre_div_mode != 2) out.pre_div = 1.0f;
    dyn[blockIdx.x] = out;
}

// One CTA per tensor: the scalars of the one-step-lag variant (af8_lag_scalars).
__global__ void __launch_bounds__(FINALIZE_THREADS)
lag_scalars_kernel(const af8_lag_tensor *tensors, int phase, const void *block_sumsq, af8_dyn_scalars *dyn)
{
    __shared__ double s_part[FINALIZE_THREADS / 32];
    await_launches();
    const af8_lag_tensor T = tensors[blockIdx.x];
    const int tid = threadIdx.x;
    if (phase == 0) {
        if (tid != 0) return;
        const float alpha = T.alpha_dev ? *T.alpha_dev : T.alpha;
        const float fs = (T.lag_fira_scale != nullptr && T.has_lag_fira) ? *T.lag_fira_scale : 1.0f;
        const float alpha_eff = __fmul_rn(alpha, fs);                                      // optimizer.py:1062
        const float pn = *T.prev_update_norm;
        const float denom = T.clip_div > 0.0f ? fmaxf(1.0f, __fdiv_rn(pn, T.clip_div)) : 1.0f;   // kernels.cu:652-653
        af8_dyn_scalars out = dyn[blockIdx.x];
        out.fira = 1.0f;
        out.zero = 0.0f;
        out.step = -__fdiv_rn(alpha_eff, denom);
        out.pre_div = 1.0f;
        dyn[blockIdx.x] = out;
        return;
    }
    const double *const p64 = static_cast<const double *>(block_sumsq) + T.first_block;
    const float *const p32 = static_cast<const float *>(block_sumsq) + T.first_block;
    const double sum = T.partials_f64 ? block_sum<FINALIZE_THREADS>(T.n_blocks, [=](int64_t i) { return p64[i]; }, s_part)
                                      : block_sum<FINALIZE_THREADS>(T.n_blocks, [=](int64_t i) { return (double)p32[i]; }, s_part);
    if (tid != 0) return;
    const float raw = __double2float_rn(sqrt(sum));
    *T.prev_update_norm = raw;                                                              // optimizer.py:1066-1067
    dyn[blockIdx.x].norm = raw;
    if (T.lag_fira_scale == nullptr || T.fira_prev == nullptr) return;
    const float norm = isfinite(raw) ? raw : 0.0f;                                           // optimizer.py:767-768
    float fs = 1.0f;
    if (T.fira_has_prev) {
        const float fp = *T.fira_prev;
        const bool reset = fp < 1e-6f;
        const float ratio = __fdiv_rn(norm, __fadd_rn(fp, 1e-8f));
        const float lim = __fdiv_rn(fmaxf(ratio, T.fira_margin1), T.fira_margin1);
        fs = reset ? 1.0f : __frcp_rn(lim);
        *T.fira_prev = reset ? norm : __fmul_rn(norm, fs);
    } else {
        *T.fira_prev = norm;
    }
    *T.lag_fira_scale = fs;                                                                 // optimizer.py:1069-1070
}

// ---------------------------------------------------------------------------
// launch helpers
// ---------------------------------------------------------------------------
// Resident CTAs of a kernel launched with fixed threads and shared memory, by device: asked once (the question costs a small step's
// launch more than the launch itself).
struct ResidentCtas {
    std::atomic<int> of_device[64];
    // whether they are known for the current device (and the kernel's attributes set there)
    bool asked() const
    {
        int dev = -1;
        return cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 && of_device[dev].load(std::memory_order_relaxed) > 0;
    }
};
template <typename K>
inline int resident_ctas(K kernel, int threads, size_t smem, ResidentCtas *known, int *per_sm)
{
    int dev = -1;
    AF8_CUDA_TRY(cudaGetDevice(&dev));
    std::atomic<int> *const slot = known && dev >= 0 && dev < 64 ? &known->of_device[dev] : nullptr;
    *per_sm = slot ? slot->load(std::memory_order_relaxed) : 0;
    if (*per_sm > 0) return AF8_OK;
    AF8_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, kernel, threads, smem));
    if (*per_sm < 1) return fail(AF8_ERR_CUDA, "kernel does not fit on an SM (threads=%d smem=%zu)", threads, smem);
    if (slot) slot->store(*per_sm, std::memory_order_relaxed);
    return AF8_OK;
}
template <typename K>
inline int persistent_grid(K kernel, int threads, size_t smem, int64_t total_blocks, int *grid_out, ResidentCtas *known = nullptr)
{
    int per_sm = 0;
    const int rc = resident_ctas(kernel, threads, smem, known, &per_sm);
    if (rc) return rc;
    int64_t g = (int64_t)per_sm * sm_count();
    if (g > total_blocks) g = total_blocks;
    *grid_out = (int)g;
    return AF8_OK;
}

template <typename GradT, typename ParamT, int VB, int MF, bool SR, bool LAG, int ROOT>
inline int launch_fast(const FullrankLaunch &L, cudaStream_t st)
{
    using Ring = FastRing<GradT, ParamT, VB, MF>;
    auto kernel = fullrank_fast_kernel<GradT, ParamT, VB, MF, SR, LAG, ROOT>;
    int grid = 0;
    static ResidentCtas known;
    if (!known.asked()) {
        // the ring lives in dynamic shared memory (up to 44 KB per CTA): opt in and ask for the large
        // shared-memory carve-out
        AF8_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Ring::SMEM_BYTES));
        AF8_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                          (int)cudaSharedmemCarveoutMaxShared));
    }
    int rc = persistent_grid(kernel, FAST_THREADS, Ring::SMEM_BYTES, L.total_blocks, &grid, &known);
    if (rc) return rc;
    AF8_CUDA_TRY(launch_next(kernel, grid, FAST_THREADS, Ring::SMEM_BYTES, st, L));
    return AF8_OK;
}

template <typename GradT, int VB, int MF>
inline int launch_stat(const FullrankLaunch &L, cudaStream_t st)
{
    auto kernel = fullrank_stat_kernel<GradT, VB, MF>;
    static ResidentCtas known;
    int per_sm = 0;
    const int rc = resident_ctas(kernel, STAT_THREADS, 0, &known, &per_sm);
    if (rc) return rc;
    const int64_t warps_per_cta = STAT_THREADS / 32;
    int64_t grid = (int64_t)per_sm * sm_count();
    const int64_t need = (L.total_blocks + warps_per_cta - 1) / warps_per_cta;
    if (grid > need) grid = need;
    AF8_CUDA_TRY(launch_next(kernel, (unsigned)grid, STAT_THREADS, 0, st, L));
    return AF8_OK;
}

template <typename GradT, int MODE, int THREADS>
inline int launch_generic_threads(const FullrankLaunch &L, const GenericCfg &C, bool plain, cudaStream_t st)
{
    const size_t smem = plain ? 0 : (size_t)2 * C.block * sizeof(float);       // (only quantised states are staged)
    auto kernel = fullrank_generic_kernel<GradT, MODE, THREADS>;
    const int rs = allow_dynamic_smem(kernel, smem);
    if (rs) return rs;
    int grid = 0;
    static ResidentCtas known;                        // (of the plain form, whose shared memory is fixed)
    int rc = persistent_grid(kernel, THREADS, smem, L.total_blocks, &grid, plain ? &known : nullptr);
    if (rc) return rc;
    AF8_CUDA_TRY(launch_next(kernel, grid, THREADS, smem, st, L, C));
    return AF8_OK;
}

template <typename GradT, int MODE>
inline int launch_generic(const FullrankLaunch &L, const GenericCfg &C, cudaStream_t st)
{
    const bool plain = (C.v_fmt == AF8_V_FP32 || C.v_fmt == AF8_V_NONE) && (C.m_fmt == AF8_M_NONE || C.m_fmt == AF8_M_FP32);
    // (quantised blocks: 256 and 1024 threads, write pass over 144 blocks of 128 elements 10.4 and 16.5 us, of 256 10.3 and 12.2;
    // 192 of 512 12.3 and 16.4; 36 of 1024 16.4 and 12.3, of 4096 38 and 18)
    return L.total_blocks <= 2 * (int64_t)sm_count() && (plain || C.block >= 1024) ? launch_generic_threads<GradT, MODE, 1024>(L, C, plain, st)
                                                                                   : launch_generic_threads<GradT, MODE, GEN_THREADS>(L, C, plain, st);
}

// the general kernel in any mode
template <typename GradT>
inline int dispatch_generic(int mode, const FullrankLaunch &L, const GenericCfg &C, cudaStream_t st)
{
    switch (mode) {
    case AF8_MODE_NOCLIP: return launch_generic<GradT, AF8_MODE_NOCLIP>(L, C, st);
    case AF8_MODE_SUMSQ: return launch_generic<GradT, AF8_MODE_SUMSQ>(L, C, st);
    case AF8_MODE_APPLY: return launch_generic<GradT, AF8_MODE_APPLY>(L, C, st);
    case AF8_MODE_LAG: return launch_generic<GradT, AF8_MODE_LAG>(L, C, st);
    default: return launch_generic<GradT, AF8_MODE_SUMSQ_M>(L, C, st);
    }
}

// The specialised kernels cover the Adam denominator with AL8 or AL16 second moments in blocks of 2048 and
// UF8 / UF4 momentum in blocks of 256 or none, for fp32 parameters with fp32 or bf16 gradients and for bf16
// parameters with bf16 gradients: the formats that large tensors are trained with.  What is left to the
// general kernel are the formats with a codebook (d8, d4), fp16, other block sizes and the small
// binary32-state tensors.  The lag mode exists for UF8 / AL8.
inline bool fast_covers(const af8_fullrank_cfg &c)
{
    if (!c.use_adam_denom || c.momentum_only || c.block != FAST_VBLOCK || c.mode == AF8_MODE_SUMSQ_M) return false;
    if (c.v_fmt != AF8_V_AL8 && c.v_fmt != AF8_V_AL16) return false;
    if (c.m_fmt != AF8_M_NONE && (c.m_block != FAST_MBLOCK || (c.m_fmt != AF8_M_UF8 && c.m_fmt != AF8_M_UF4))) return false;
    if (c.mode == AF8_MODE_LAG && !(c.v_fmt == AF8_V_AL8 && c.m_fmt == AF8_M_UF8)) return false;
    return (c.param_dtype == AF8_F32 && (c.grad_dtype == AF8_F32 || c.grad_dtype == AF8_BF16)) ||
           (c.param_dtype == AF8_BF16 && c.grad_dtype == AF8_BF16);
}

template <typename GradT, typename ParamT, bool SR, int VB, int MF>
inline int dispatch_fast_mode(int mode, FullrankLaunch L, bool eps_hides, cudaStream_t st)
{
    if (mode == AF8_MODE_SUMSQ) return launch_stat<GradT, VB, MF>(L, st);
    if constexpr (VB == 8 && MF == AF8_M_UF8) {
        if (mode == AF8_MODE_LAG) return eps_hides ? launch_fast<GradT, ParamT, VB, MF, SR, true, ROOT_FTZ>(L, st) : launch_fast<GradT, ParamT, VB, MF, SR, true, ROOT_FULL>(L, st);
    }
    if (mode == AF8_MODE_NOCLIP) L.dyn = nullptr;        // the step size is the table's
    constexpr int HIDES = root_exact<VB, MF> ? ROOT_REFINED : ROOT_FTZ, SHOWS = root_exact<VB, MF> ? ROOT_EXACT : ROOT_FULL;
    return eps_hides ? launch_fast<GradT, ParamT, VB, MF, SR, false, HIDES>(L, st) : launch_fast<GradT, ParamT, VB, MF, SR, false, SHOWS>(L, st);
}

template <typename GradT, typename ParamT, bool SR>
inline int dispatch_fast_formats(const af8_fullrank_cfg &c, const FullrankLaunch &L, bool eps_hides, cudaStream_t st)
{
    if (c.v_fmt == AF8_V_AL8) {
        if (c.m_fmt == AF8_M_UF8) return dispatch_fast_mode<GradT, ParamT, SR, 8, AF8_M_UF8>(c.mode, L, eps_hides, st);
        if (c.m_fmt == AF8_M_UF4) return dispatch_fast_mode<GradT, ParamT, SR, 8, AF8_M_UF4>(c.mode, L, eps_hides, st);
        return dispatch_fast_mode<GradT, ParamT, SR, 8, AF8_M_NONE>(c.mode, L, eps_hides, st);
    }
    if (c.m_fmt == AF8_M_UF8) return dispatch_fast_mode<GradT, ParamT, SR, 16, AF8_M_UF8>(c.mode, L, eps_hides, st);
    if (c.m_fmt == AF8_M_UF4) return dispatch_fast_mode<GradT, ParamT, SR, 16, AF8_M_UF4>(c.mode, L, eps_hides, st);
    return dispatch_fast_mode<GradT, ParamT, SR, 16, AF8_M_NONE>(c.mode, L, eps_hides, st);
}

// c must satisfy fast_covers; eps_hides: every eps_denom of the table is at least EPS_HIDES (fullrank_fast.cuh)
inline int dispatch_fast(const af8_fullrank_cfg &c, const FullrankLaunch &L, bool eps_hides, cudaStream_t st)
{
    if (c.param_dtype == AF8_BF16)
        return c.stochastic_round ? dispatch_fast_formats<bf16_tag, bf16_tag, true>(c, L, eps_hides, st) : dispatch_fast_formats<bf16_tag, bf16_tag, false>(c, L, eps_hides, st);
    if (c.grad_dtype == AF8_BF16) return dispatch_fast_formats<bf16_tag, float, false>(c, L, eps_hides, st);
    return dispatch_fast_formats<float, float, false>(c, L, eps_hides, st);
}

inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

inline int validate_fullrank_table(const af8_fullrank_cfg &c, const af8_fullrank_tensor *T, int n, int64_t total_blocks)
{
    int64_t next = 0;
    const bool no_v = c.v_fmt == AF8_V_NONE;
    const bool v_quant = c.v_fmt != AF8_V_FP32 && !no_v;
    const bool has_m = c.m_fmt != AF8_M_NONE;
    const bool m_quant = has_m && c.m_fmt != AF8_M_FP32;
    for (int i = 0; i < n; ++i) {
        const af8_fullrank_tensor &t = T[i];
        if (t.numel <= 0) return fail(AF8_ERR_INVALID, "tensor %d: numel must be positive", i);
        if (t.numel >= ((int64_t)1 << 38)) return fail(AF8_ERR_UNSUPPORTED, "tensor %d: more than 2^38 elements", i);   // 32-bit block indices
        if (t.first_block != next) return fail(AF8_ERR_INVALID, "tensor %d: first_block %lld, expected %lld", i, (long long)t.first_block, (long long)next);
        next += (t.numel + c.block - 1) / c.block;
        if (!t.param || !t.grad) return fail(AF8_ERR_INVALID, "tensor %d: null param or grad", i);
        if (!aligned16(t.param) || !aligned16(t.grad)) return fail(AF8_ERR_INVALID, "tensor %d: param and grad must be 16-byte aligned", i);
        if (t.param_copy && (c.param_dtype != AF8_F32 || !aligned16(t.param_copy)))
            return fail(AF8_ERR_INVALID, "tensor %d: param_copy needs fp32 parameters and a 16-byte aligned address", i);
        if (v_quant) {
            if (!t.v_q || !t.v_scale || !t.v_min_log) return fail(AF8_ERR_INVALID, "tensor %d: null quantised V state", i);
            if (!aligned16(t.v_q)) return fail(AF8_ERR_INVALID, "tensor %d: v_q must be 16-byte aligned", i);
        } else if (!no_v && !t.v_f32) {
            return fail(AF8_ERR_INVALID, "tensor %d: null fp32 V state", i);
        }
        if (no_v && has_m && !(t.v_keep > 0.0f)) return fail(AF8_ERR_INVALID, "tensor %d: the SGD mode needs v_keep = 1 - beta1 > 0", i);
        if (m_quant) {
            if (!t.m_q || !t.m_scale) return fail(AF8_ERR_INVALID, "tensor %d: null quantised M state", i);
            if (!aligned16(t.m_q)) return fail(AF8_ERR_INVALID, "tensor %d: m_q must be 16-byte aligned", i);
        } else if (has_m && !t.m_f32) {
            return fail(AF8_ERR_INVALID, "tensor %d: null fp32 M state", i);
        }
    }
    if (next != total_blocks) return fail(AF8_ERR_INVALID, "total_blocks is %lld but the table holds %lld blocks", (long long)total_blocks, (long long)next);
    return AF8_OK;
}

}  // namespace af8

extern "C" int af8_fullrank_step(const af8_fullrank_cfg *cfg, const af8_fullrank_tensor *host_tensors,
                                 af8_fullrank_tensor *dev_tensors, int32_t n_tensors, int64_t total_blocks,
                                 const af8_dyn_scalars *dyn, float *block_sumsq, void *stream)
{
    using namespace af8;
    if (!cfg || !dev_tensors) return fail(AF8_ERR_INVALID, "af8_fullrank_step: null cfg or table");
    if (n_tensors <= 0 || total_blocks <= 0) return fail(AF8_ERR_INVALID, "af8_fullrank_step: empty launch (n_tensors=%d, total_blocks=%lld)", n_tensors, (long long)total_blocks);
    const af8_fullrank_cfg &c = *cfg;
    if (c.param_dtype != AF8_F32 && c.param_dtype != AF8_BF16 && c.param_dtype != AF8_F16) return fail(AF8_ERR_INVALID, "af8_fullrank_step: bad param_dtype %d", c.param_dtype);
    if (c.grad_dtype != AF8_F32 && c.grad_dtype != AF8_BF16 && c.grad_dtype != AF8_F16) return fail(AF8_ERR_INVALID, "af8_fullrank_step: bad grad_dtype %d", c.grad_dtype);
    if (c.stochastic_round && c.param_dtype == AF8_F32) return fail(AF8_ERR_INVALID, "af8_fullrank_step: stochastic rounding applies to bf16 / fp16 parameters only");
    if (c.v_fmt != AF8_V_FP32 && c.v_fmt != AF8_V_AL8 && c.v_fmt != AF8_V_AL16 && c.v_fmt != AF8_V_NONE) return fail(AF8_ERR_INVALID, "af8_fullrank_step: bad v_fmt %d", c.v_fmt);
    if (c.m_fmt < AF8_M_NONE || c.m_fmt > AF8_M_FP32) return fail(AF8_ERR_INVALID, "af8_fullrank_step: bad m_fmt %d", c.m_fmt);
    if (c.block < 128 || c.block % 128 != 0) return fail(AF8_ERR_INVALID, "af8_fullrank_step: block must be a multiple of 128, >= 128 (got %d)", c.block);
    if (c.block > GEN_MAX_BLOCK) return fail(AF8_ERR_UNSUPPORTED, "af8_fullrank_step: block %d exceeds the supported maximum %d", c.block, GEN_MAX_BLOCK);
    const bool m_quant = c.m_fmt != AF8_M_NONE && c.m_fmt != AF8_M_FP32;
    if (m_quant && (c.m_block < 32 || c.m_block % 4 != 0 || c.block % c.m_block != 0))
        return fail(AF8_ERR_INVALID, "af8_fullrank_step: m_block must be a multiple of 4, >= 32 and divide block (got %d, block %d)", c.m_block, c.block);
    if (c.mode < AF8_MODE_NOCLIP || c.mode > AF8_MODE_LAG) return fail(AF8_ERR_INVALID, "af8_fullrank_step: bad mode %d", c.mode);
    if ((c.mode == AF8_MODE_APPLY || c.mode == AF8_MODE_SUMSQ_M || c.mode == AF8_MODE_LAG) && !dyn) return fail(AF8_ERR_INVALID, "af8_fullrank_step: this mode needs dyn");
    if ((c.mode == AF8_MODE_SUMSQ || c.mode == AF8_MODE_SUMSQ_M || c.mode == AF8_MODE_LAG) && !block_sumsq) return fail(AF8_ERR_INVALID, "af8_fullrank_step: this mode needs block_sumsq");
    if (c.mode == AF8_MODE_LAG && c.momentum_only) return fail(AF8_ERR_UNSUPPORTED, "af8_fullrank_step: the lag mode does not cover the momentum-only rule");
    if (c.mode == AF8_MODE_SUMSQ_M && !(c.momentum_only && c.m_fmt != AF8_M_NONE)) return fail(AF8_ERR_INVALID, "af8_fullrank_step: SUMSQ_M needs the momentum-only rule");
    if (c.momentum_only && c.use_adam_denom) return fail(AF8_ERR_INVALID, "af8_fullrank_step: momentum_only excludes the Adam denominator");

    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (host_tensors) {
        int rc = validate_fullrank_table(c, host_tensors, n_tensors, total_blocks);
        if (rc) return rc;
        rc = upload_table(dev_tensors, host_tensors, sizeof(af8_fullrank_tensor) * (size_t)n_tensors, st);
        if (rc) return rc;
    }

    FullrankLaunch L;
    L.tensors = dev_tensors;
    L.dyn = dyn;
    L.block_sumsq = block_sumsq;
    L.total_blocks = total_blocks;
    L.n_tensors = n_tensors;
    L.negate_grad = c.negate_grad ? 1 : 0;
    L.v_floor = c.v_floor;
    L.param_dtype = c.param_dtype;
    L.sr = c.stochastic_round ? 1 : 0;
    GenericCfg C{c.v_fmt, c.m_fmt, c.block, c.m_block, c.use_adam_denom ? 1 : 0, c.momentum_only ? 1 : 0};

    if (fast_covers(c)) {
        bool eps_hides = c.use_adam_denom == AF8_ADAM_DENOM_EPS_HIDES;
        if (host_tensors) {
            eps_hides = true;
            for (int i = 0; i < n_tensors; ++i) eps_hides = eps_hides && host_tensors[i].eps_denom >= EPS_HIDES;
        }
        return dispatch_fast(c, L, eps_hides, st);
    }
    if (c.grad_dtype == AF8_BF16) return dispatch_generic<bf16_tag>(c.mode, L, C, st);
    if (c.grad_dtype == AF8_F16) return dispatch_generic<f16_tag>(c.mode, L, C, st);
    return dispatch_generic<float>(c.mode, L, C, st);
}

extern "C" int af8_fullrank_upload(const af8_fullrank_cfg *cfg, const af8_fullrank_tensor *host_tensors,
                                   af8_fullrank_tensor *dev_tensors, int32_t n_tensors, int64_t total_blocks,
                                   void *stream)
{
    using namespace af8;
    if (!cfg || !host_tensors || !dev_tensors) return fail(AF8_ERR_INVALID, "af8_fullrank_upload: null argument");
    if (n_tensors <= 0 || cfg->block < 128 || cfg->block % 128 != 0) return fail(AF8_ERR_INVALID, "af8_fullrank_upload: bad sizes");
    int rc = validate_fullrank_table(*cfg, host_tensors, n_tensors, total_blocks);
    if (rc) return rc;
    return upload_table(dev_tensors, host_tensors, sizeof(af8_fullrank_tensor) * (size_t)n_tensors, static_cast<cudaStream_t>(stream));
}

extern "C" int af8_device_status(int32_t *status_out, void *stream)
{
    using namespace af8;
    if (!status_out) return fail(AF8_ERR_INVALID, "af8_device_status: null output");
    int v = 0;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    AF8_CUDA_TRY(cudaMemcpyFromSymbolAsync(&v, g_device_error, sizeof(int), 0, cudaMemcpyDeviceToHost, st));
    AF8_CUDA_TRY(cudaStreamSynchronize(st));
    *status_out = v;
    return AF8_OK;
}

namespace af8 {
// Self-test of the bounded wait: one thread arms an mbarrier for 64 bytes, copies 32 (that copy
// completes; nothing stays in flight) and waits with the given limit.  The phase can never complete,
// so the wait must give up after the limit and record the time-out exactly as the step kernels do.
__global__ void bounded_wait_selftest_kernel(const unsigned char *src, uint64_t limit_ns, int *gave_up)
{
    __shared__ __align__(128) unsigned char s_dst[64];
    __shared__ __align__(8) uint64_t s_bar;
    if (threadIdx.x != 0) return;
    mbar_init(&s_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
    mbar_expect_tx(&s_bar, 64);
    bulk_g2s(s_dst, src, 32, &s_bar);
    const bool done = mbar_wait_bounded(&s_bar, 0, limit_ns);
    if (!done) atomicExch(&g_device_error, DEVERR_COPY_TIMEOUT);
    *gave_up = done ? 0 : 1;
    // the 32-byte copy has landed long before the limit ran out; give it a (bounded) moment anyway
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 20000ull) { }
}
}  // namespace af8

extern "C" int af8_selftest_bounded_wait(const void *src32, int64_t limit_ns, int32_t *gave_up_dev, void *stream)
{
    using namespace af8;
    if (!src32 || !gave_up_dev) return fail(AF8_ERR_INVALID, "af8_selftest_bounded_wait: null argument");
    if (!aligned16(src32)) return fail(AF8_ERR_INVALID, "af8_selftest_bounded_wait: the source must be 16-byte aligned");
    if (limit_ns <= 0 || limit_ns > 1000000000ll) return fail(AF8_ERR_INVALID, "af8_selftest_bounded_wait: the limit must be 1 ns .. 1 s");
    bounded_wait_selftest_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const unsigned char *>(src32), (uint64_t)limit_ns, gave_up_dev);
    AF8_CUDA_TRY(cudaGetLastError());
    return AF8_OK;
}

extern "C" int af8_device_status_clear(void *stream)
{
    using namespace af8;
    const int zero = 0;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    AF8_CUDA_TRY(cudaMemcpyToSymbolAsync(g_device_error, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, st));
    AF8_CUDA_TRY(cudaStreamSynchronize(st));
    return AF8_OK;
}

extern "C" int af8_lag_scalars(const af8_lag_tensor *tensors, int32_t n_tensors, int32_t phase, const void *block_sumsq,
                               af8_dyn_scalars *dyn, void *stream)
{
    using namespace af8;
    if (!tensors || !dyn) return fail(AF8_ERR_INVALID, "af8_lag_scalars: null argument");
    if (n_tensors <= 0) return fail(AF8_ERR_INVALID, "af8_lag_scalars: n_tensors must be positive");
    if (phase != 0 && phase != 1) return fail(AF8_ERR_INVALID, "af8_lag_scalars: phase must be 0 or 1");
    if (phase == 1 && !block_sumsq) return fail(AF8_ERR_INVALID, "af8_lag_scalars: phase 1 needs block_sumsq");
    AF8_CUDA_TRY(launch_next(lag_scalars_kernel, (unsigned)n_tensors, FINALIZE_THREADS, 0, static_cast<cudaStream_t>(stream), tensors, phase, block_sumsq, dyn));
    return AF8_OK;
}

extern "C" int af8_norm_finalize(const af8_norm_tensor *tensors, int32_t n_tensors, const void *block_sumsq,
                                 af8_dyn_scalars *dyn, void *stream)
{
    using namespace af8;
    if (!tensors || !block_sumsq || !dyn) return fail(AF8_ERR_INVALID, "af8_norm_finalize: null argument");
    if (n_tensors <= 0) return fail(AF8_ERR_INVALID, "af8_norm_finalize: n_tensors must be positive");
    AF8_CUDA_TRY(launch_next(norm_finalize_kernel, (unsigned)n_tensors, FINALIZE_THREADS, 0, static_cast<cudaStream_t>(stream), tensors, block_sumsq, dyn));
    return AF8_OK;
}
