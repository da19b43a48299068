// Factored step for 2-D tensors: Adafactor (row / column second moments) and
// CAME (confidence-guided, with momentum).
//
// Reference semantics: _update_param_8bit factored branch on the pure-PyTorch
// route (optimizer.py:2202-2253 statistics and small-state EMAs, 2394-2399 and
// 2543-2549 dispatch), _factored_inv_std (optimizer.py:818-821),
// _compute_ut_clipped (optimizer.py:824-829), _fallback_2d_update
// (optimizer.py:920-970).
//
// Three kernels, each launched once for a whole table of tensors:
//   factored_stats_kernel   row and column sums of g*g, or of CAME's residual
//                           (U - M)^2 + eps, over 512 x 256 tiles.  Every product
//                           is rounded to binary32 as torch does and then
//                           accumulated in binary64, so the binary32 means do not
//                           depend on the order of accumulation.
//   factored_small_kernel   one CTA per quantisation block of a row / column state:
//                           means, EMA into the (tiny) AL states with exact
//                           requantisation, partial means of the row state; the
//                           inverse-std vectors follow in factored_inv_kernel.
//   factored_update_kernel  flat chunks aligned to momentum blocks: the update
//                           itself, its sum of squares, the parameter write and
//                           the momentum requantisation.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "fullrank_fast.cuh"
#include "fullrank_generic.cuh"
#include "fullrank_stat.cuh"
#include "launch.cuh"
#include "tensormap.cuh"
#include "write_units.cuh"

namespace af8 {

constexpr int FSTAT_ROWS = 512;
constexpr int FSTAT_COLS = 256;
constexpr int FUPD_THREADS = 256;
constexpr int DEVERR_SRING_TIMEOUT = 4;      // a bulk copy of the statistic pass's input ring did not land

struct FactoredLaunch {
    const af8_factored_tensor *tensors;
    const af8_dyn_scalars *dyn;
    double *block_sumsq;
    int64_t total_units;
    int32_t n_tensors;
    int32_t grad_dtype, m_fmt, m_block, came, negate_grad, mode;
    float v_floor;
    int32_t param_dtype, sr;
    int32_t split;               // tile kernels: a unit is the (1 << split)-th part of a tile (see tile_split)
};

// Whether a tensor's squares are added eight at a time in binary32 before they enter the binary64 sum: a matrix of whole
// vectors is, in a table of such matrices and, so that its norm does not depend on its neighbours, in a table that it shares
// with batches; batches of matrices, and tables with rows of any length, add each square in binary64.
template <int ANY>
__device__ __forceinline__ bool sums_by_eight(const af8_factored_tensor &T) { return ANY == 0 || (ANY == 1 && T.batch_rows == 0); }

__device__ __forceinline__ int find_factored_tile(const af8_factored_tensor *t, int n, int64_t id)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (t[mid].first_tile <= id) lo = mid; else hi = mid - 1;
    }
    return lo;
}
__device__ __forceinline__ int find_factored_chunk(const af8_factored_tensor *t, int n, int64_t id)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (t[mid].first_chunk <= id) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// batches of matrices (batch_rows > 0): number of matrices, rows of one, and the stat tiles of one
__host__ __device__ __forceinline__ int64_t fact_mat_rows(const af8_factored_tensor &t) { return t.batch_rows > 0 ? t.batch_rows : t.rows; }
__host__ __device__ __forceinline__ int64_t fact_batch(const af8_factored_tensor &t) { return t.batch_rows > 0 ? t.rows / t.batch_rows : 1; }
__host__ __device__ __forceinline__ int64_t fact_tiles(const af8_factored_tensor &t)
{
    return fact_batch(t) * ((fact_mat_rows(t) + FSTAT_ROWS - 1) / FSTAT_ROWS) * ((t.cols + FSTAT_COLS - 1) / FSTAT_COLS);
}
// first entry of the column arrays for the matrix that holds row `row`
__device__ __forceinline__ int64_t fact_col_base(const af8_factored_tensor &t, int64_t row)
{
    return t.batch_rows > 0 ? (row / t.batch_rows) * t.cols : 0;
}

// Unit `id` of a launch over the tiles (L.split applied) of tensor T: its rows r0 .. r_end - 1 (of the flattened
// batch), its first column and the first entry of its matrix's part of the column arrays.
struct TilePos { int64_t r0, r_end, c0, cb; };
__device__ __forceinline__ TilePos tile_pos(const FactoredLaunch &L, const af8_factored_tensor &T, int64_t id)
{
    TilePos p;
    const int64_t ntc = (T.cols + FSTAT_COLS - 1) / FSTAT_COLS;
    int64_t local = (id >> L.split) - T.first_tile, first = 0, end = T.rows;
    p.cb = 0;
    if (T.batch_rows > 0) {                                          // a tile lies inside one matrix of a batch
        const int64_t tpm = ((T.batch_rows + FSTAT_ROWS - 1) / FSTAT_ROWS) * ntc;
        const int64_t mat = local / tpm;
        local -= mat * tpm;
        first = mat * T.batch_rows;
        end = first + T.batch_rows;
        p.cb = mat * T.cols;
    }
    const int64_t tr = local / ntc;
    const int part_rows = FSTAT_ROWS >> L.split, part = (int)(id & (((int64_t)1 << L.split) - 1));
    p.c0 = (local - tr * ntc) * FSTAT_COLS;
    p.r0 = first + tr * FSTAT_ROWS + part * part_rows;
    p.r_end = min(end, p.r0 + (int64_t)part_rows);                   // (an empty part: r_end <= r0)
    return p;
}

// Parts per tile, as a power of two: a 512-row tile is 131072 elements, so a table of fewer than about 58 M parameters
// has fewer tiles than three CTAs per SM, what most of these kernels keep resident (the residual pass over any rows, its
// fp32 statistic and the fp32 write pass over tiles keep two; the same line served them as well).  Tiles are halved, down
// to 64 rows, while the parts stay within `waves` times that many: a part costs a fixed 4 us or so (pipeline fill, the
// reduction over the warps, 256 column atomics), so that more waves of smaller parts lose.  One wave for the statistic, sum
// and write passes; CAME's residual pass spends several times as long on a row and gains up to three.  Measured, bf16
// gradients, us with whole tiles / halves / quarters / eighths (512 x 1376 layers have 26 tiles, 768 x 2048 ones 64,
// 1024 x 2752 ones 102):
//   statistic  104 tiles 26 / 23 / 22 / 25    208 tiles 33 / 28 / 32 / 43    512 tiles 48 / 47 / 60 / 71    612 tiles 53 / 58 / 66 / 82
//   residual    44 tiles 56 / 52 / 38 / 24    104 tiles 97 / 61 / 42 / 44    208 tiles 130 / 77 / 77 / 81
//              512 tiles 97 / 97 / 138 / 179  612 tiles 208 / 159 / 175 / 177
inline int tile_split(int64_t tiles, int waves = 1)
{
    int sh = 0;
    while (sh < 3 && (tiles << (sh + 1)) <= 3 * waves * (int64_t)sm_count()) ++sh;
    return sh;
}

__device__ __forceinline__ float load_grad_any(const void *g, int dtype, int64_t i)
{
    if (dtype == AF8_F32) return static_cast<const float *>(g)[i];
    const uint32_t h = static_cast<const uint16_t *>(g)[i];
    return dtype == AF8_BF16 ? bf16_bits_to_f32(h) : f16_bits_to_f32(h);
}

// momentum before the EMA (optimizer.py:694-697): dequantised codes or the fp32 state
__device__ __forceinline__ float m_old_at(const af8_factored_tensor &T, int m_fmt, int m_block, int64_t flat)
{
    if (m_fmt == AF8_M_FP32) return T.m_f32[flat];
    return m_decode(T.m_q, load_state(T.m_scale + flat / m_block), flat, m_fmt);
}

// Tensor.lerp_ with a weight that is the same for many elements: the choice between ATen's two
// forms is made once (LerpW), an element costs a subtraction, a select and one fma.
struct LerpW { float ww; bool small; };
__device__ __forceinline__ LerpW make_lerp(float w)
{
    LerpW l;
    l.small = fabsf(w) < 0.5f;
    l.ww = l.small ? w : __fsub_rn(w, 1.0f);
    return l;
}
__device__ __forceinline__ float lerp_w(float s, float e, const LerpW &l)
{
    return __fmaf_rn(l.ww, __fsub_rn(e, s), l.small ? s : e);
}

// U = g * inv_row * inv_col, then the RMS clip divisor (optimizer.py:825-828)
__device__ __forceinline__ float u_clipped(float g, float ir, float ic, float pre_div)
{
    float u = __fmul_rn(__fmul_rn(g, ir), ic);
    if (pre_div != 1.0f) u = __fdiv_rn(u, pre_div);
    return u;
}

// x / d for one divisor and many dividends: the correctly rounded reciprocal and one
// residual step give the IEEE quotient (checked against the division on 2e9 random
// normal operands; the unrefined product stands when it is infinite or NaN).
struct DivBy {
    float rcp, nd;
    bool one;
};
__device__ __forceinline__ DivBy make_div(float d)
{
    DivBy D;
    D.one = d == 1.0f;
    D.rcp = __frcp_rn(d);
    D.nd = -d;
    return D;
}
__device__ __forceinline__ float div_by(float x, const DivBy &D)
{
    if (D.one) return x;
    const float q = __fmul_rn(x, D.rcp);
    const float q2 = __fmaf_rn(__fmaf_rn(q, D.nd, x), D.rcp, q);
    return fabsf(q) <= 3.402823466e38f ? q2 : q;
}
__device__ __forceinline__ float u_clipped_fast(float g, float ir, float ic, const DivBy &D)
{
    return div_by(__fmul_rn(__fmul_rn(g, ir), ic), D);
}

// The same helpers on pairs of elements with Blackwell's packed binary32 instructions (one
// instruction per pair; each component rounds exactly like the scalar operation).
__device__ __forceinline__ float2 div_by2(float2 x, const DivBy &D)
{
    if (D.one) return x;
    const float2 r2 = bc2(D.rcp);
    const float2 q = __fmul2_rn(x, r2);
    const float2 q2 = __ffma2_rn(__ffma2_rn(q, bc2(D.nd), x), r2, q);
    return make_float2(fabsf(q.x) <= 3.402823466e38f ? q2.x : q.x, fabsf(q.y) <= 3.402823466e38f ? q2.y : q.y);
}
__device__ __forceinline__ float2 lerp_w2(float2 s, float2 e, const LerpW &l)
{
    return __ffma2_rn(bc2(l.ww), sub2(e, s), l.small ? s : e);
}
// Largest magnitude of a momentum block of 256, 8 elements a lane: at least 1e-12, NaNs left out.  odd: the block holds an
// infinity or a NaN.  (The bit patterns of non-negative floats are ordered: one REDUX instead of a shuffle tree.)
__device__ __forceinline__ float m_absmax256(const float (&m)[8], bool &odd)
{
    float top = max3_nan(fabsf(m[0]), fabsf(m[1]), fabsf(m[2]));
    top = max3_nan(top, fabsf(m[3]), fabsf(m[4]));
    top = max3_nan(top, fabsf(m[5]), fabsf(m[6]));
    top = max3_nan(top, fabsf(m[7]), fabsf(m[7]));
    const uint32_t bits = __reduce_max_sync(0xffffffffu, __float_as_uint(top));
    odd = bits >= 0x7f800000u;
    float am = __uint_as_float(bits);
    if (odd) {
        am = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; ++j) am = fmaxf(am, fabsf(m[j]));
        am = warp_max(am);
    }
    return fmaxf(am, 1e-12f);
}
// its UF8 codes; with an infinity or a NaN by uf8_encode, which gives both the code of zero
__device__ __forceinline__ uint2 uf8_codes8(const float (&m)[8], float am, bool odd)
{
    if (odd) {
        uint2 o = make_uint2(0u, 0u);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            o.x |= uf8_encode(m[j], am) << (8 * j);
            o.y |= uf8_encode(m[j + 4], am) << (8 * j);
        }
        return o;
    }
    // round(m / am * 128), the quotient from the correctly rounded reciprocal and one residual step (|m / am| <= 1: always finite, the
    // product exact), half to even by the rounding constant; only + 128 needs the clamp; the low byte is k mod 256, k + 128 with
    // its top bit flipped
    const float2 ra2 = bc2(__frcp_rn(am)), nam2 = bc2(-am);
    uint32_t w[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t raw[4];
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
            const float2 kf = __ffma2_rn(div2_by(make_float2(m[4 * h + j], m[4 * h + j + 1]), ra2, nam2), bc2(128.0f), bc2(AF8_MAGIC_F));
            raw[j] = (uint32_t)min(__float_as_int(kf.x), AF8_MAGIC_I + 127);
            raw[j + 1] = (uint32_t)min(__float_as_int(kf.y), AF8_MAGIC_I + 127);
        }
        w[h] = pack4(raw[0], raw[1], raw[2], raw[3]) ^ 0x80808080u;
    }
    return make_uint2(w[0], w[1]);
}

// ---------------------------------------------------------------------------
// statistics
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
factored_stats_kernel(const FactoredLaunch L)
{
    __shared__ double s_col[FSTAT_COLS];
    __shared__ af8_factored_tensor sT;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    await_launches();

    for (int64_t id = blockIdx.x; id < L.total_units; id += gridDim.x) {
        const int t = find_factored_tile(L.tensors, L.n_tensors, id);
        __syncthreads();
        if (tid < (int)(sizeof(af8_factored_tensor) / 4))
            reinterpret_cast<uint32_t *>(&sT)[tid] = reinterpret_cast<const uint32_t *>(L.tensors + t)[tid];
        s_col[tid] = 0.0;
        __syncthreads();
        const int64_t C = sT.cols;
        const int64_t ntc = (C + FSTAT_COLS - 1) / FSTAT_COLS;
        const int64_t mr = fact_mat_rows(sT);                              // a tile lies inside one matrix of a batch
        const int64_t tpm = ((mr + FSTAT_ROWS - 1) / FSTAT_ROWS) * ntc;
        const int64_t local = id - sT.first_tile;
        const int64_t mat = local / tpm, lt = local - mat * tpm;
        const int64_t r0 = mat * mr + (lt / ntc) * FSTAT_ROWS;
        const int64_t R = (mat + 1) * mr;                                  // end of the matrix's rows
        const int64_t c0 = (lt % ntc) * FSTAT_COLS;
        const int64_t cb = sT.batch_rows > 0 ? mat * C : 0;               // the matrix's part of the column arrays
        float pre_div = 1.0f;
        if (L.mode == AF8_FSTAT_RESIDUAL) pre_div = L.dyn[t].pre_div;

        double cacc[FSTAT_COLS / 32];
        float icv[FSTAT_COLS / 32];
#pragma unroll
        for (int k = 0; k < FSTAT_COLS / 32; ++k) {
            cacc[k] = 0.0;
            const int64_t c = c0 + lane + 32 * k;
            icv[k] = (L.mode == AF8_FSTAT_RESIDUAL && c < C) ? sT.inv_col[cb + c] : 0.0f;
        }
        for (int rr = warp; rr < FSTAT_ROWS; rr += 8) {
            const int64_t r = r0 + rr;
            if (r >= R) break;
            const float ir = (L.mode == AF8_FSTAT_RESIDUAL) ? sT.inv_row[r] : 0.0f;
            double racc = 0.0;
#pragma unroll
            for (int k = 0; k < FSTAT_COLS / 32; ++k) {
                const int64_t c = c0 + lane + 32 * k;
                if (c < C) {
                    const int64_t flat = r * C + c;
                    float g = load_grad_any(sT.grad, L.grad_dtype, flat);
                    if (L.negate_grad) g = -g;
                    float x;
                    if (L.mode == AF8_FSTAT_GRADSQ) {
                        x = __fmul_rn(g, g);                                         // optimizer.py:2221
                    } else {
                        const float u = u_clipped(g, ir, icv[k], pre_div);           // optimizer.py:929
                        const float m = lerp_t(m_old_at(sT, L.m_fmt, L.m_block, flat), u, sT.m_w);   // optimizer.py:930
                        const float df = __fsub_rn(u, m);
                        x = __fadd_rn(__fmul_rn(df, df), sT.eps_came);               // optimizer.py:932
                    }
                    const double xd = (double)x;
                    racc += xd;
                    cacc[k] += xd;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) racc += __shfl_xor_sync(0xffffffffu, racc, o);
            if (lane == 0) atomicAdd(sT.row_sum + r, racc);
        }
#pragma unroll
        for (int k = 0; k < FSTAT_COLS / 32; ++k) atomicAdd(&s_col[lane + 32 * k], cacc[k]);
        __syncthreads();
        if (c0 + tid < C) atomicAdd(sT.col_sum + cb + c0 + tid, s_col[tid]);
    }
}

// grid (n_tensors, slices): zero the row and column sums of every tensor
__global__ void __launch_bounds__(256)
factored_clear_kernel(const af8_factored_tensor *tensors)
{
    await_launches();
    const af8_factored_tensor &T = tensors[blockIdx.x];
    const int64_t stride = (int64_t)blockDim.x * gridDim.y, first = (int64_t)blockIdx.y * blockDim.x + threadIdx.x;
    const int64_t nr = T.rows, nc = fact_batch(T) * T.cols;
    double *const rs = T.row_sum, *const cs = T.col_sum;
    for (int64_t i = first; i < nr; i += stride) rs[i] = 0.0;
    for (int64_t i = first; i < nc; i += stride) cs[i] = 0.0;
}

// ---------------------------------------------------------------------------
// small states
// ---------------------------------------------------------------------------
constexpr int SMALL_MAX_THREADS = 1024;
constexpr int SMALL_KEPT = 2048;        // logarithms of a block that wait for its range in shared memory; those of longer blocks are taken again
// EMA + requantisation of block b of one small state of n elements (optimizer.py:2232-2238,
// 937-946, 2248-2251).  `out` receives the un-requantised values.  Returns this thread's partial
// sum of the block's values (binary64) for the mean of the row state.
__device__ __forceinline__ double small_state_block(const af8_small_state &S, const double *sums, double count, int64_t n, int64_t b,
                                    float eps_add, float w, float floor_log, float *out, const CodecTables &tab, float *s_l, float (*s_red)[SMALL_MAX_THREADS / 32])
{
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int block = S.block;
    double acc = 0.0;
    if (S.fmt == AF8_V_FP32) {
        const int64_t end = min(n, (b + 1) * (int64_t)block);
        for (int64_t i = b * block + tid; i < end; i += blockDim.x) {
            const float nv = __fadd_rn(__double2float_rn(sums[i] / count), eps_add);
            const float v = lerp_t(S.f32[i], nv, w);
            S.f32[i] = v;
            out[i] = v;
            acc += (double)v;
        }
        return acc;
    }
    const int bits = S.fmt;
    const float qm1 = bits == 16 ? 65534.0f : 254.0f;
    const int qmax = bits == 16 ? 65535 : 255;
    const float sc = S.scale[b], ml = S.min_log[b];
    float mn = INFINITY, mx = -INFINITY;
    // (rolled: the few CTAs of this launch fetch the code for the first time, which unrolled copies made the longest part)
#pragma unroll 1
    for (int i = tid; i < block; i += blockDim.x) {
        const int64_t e = b * block + i;
        float v = 0.0f;                                       // padding re-enters as zeros (optimizer.py:303-305)
        if (e < n) {
            const uint32_t code = bits == 16 ? static_cast<const uint16_t *>(S.q)[e] : static_cast<const uint8_t *>(S.q)[e];
            const float nv = __fadd_rn(__double2float_rn(sums[e] / count), eps_add);
            v = lerp_t(al_decode_tab(code, sc, ml, qm1, tab), nv, w);
            out[e] = v;
            acc += (double)v;
        }
        float l = al_log2_tab(v, tab);
        mx = fmaxf(mx, l);
        if (v != 0.0f) mn = fminf(mn, l);
        else l = -INFINITY;
        if (i < SMALL_KEPT) s_l[i] = l;
    }
    mn = warp_min(mn);
    mx = warp_max(mx);
    if (lane == 0) { s_red[0][warp] = mn; s_red[1][warp] = mx; }
    __syncthreads();
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) { mn = fminf(mn, s_red[0][k]); mx = fmaxf(mx, s_red[1][k]); }
    float min_log, scale;
    al_range(mn, mx, floor_log, min_log, scale);
#pragma unroll 1
    for (int i = tid; i < block; i += blockDim.x) {
        const int64_t e = b * block + i;
        float l;
        if (i < SMALL_KEPT) l = s_l[i];
        else {                                                // (this thread's own value again)
            const float v = e < n ? out[e] : 0.0f;
            l = v != 0.0f ? al_log2_tab(v, tab) : -INFINITY;
        }
        const uint32_t code = (l == -INFINITY) ? 0u : al_encode(1.0f, l, min_log, scale, qm1, qmax);
        if (bits == 16) static_cast<uint16_t *>(S.q)[e] = (uint16_t)code;
        else static_cast<uint8_t *>(S.q)[e] = (uint8_t)code;
    }
    if (tid == 0) { S.scale[b] = scale; S.min_log[b] = min_log; }
    return acc;
}

__device__ __forceinline__ int find_factored_small(const af8_factored_tensor *t, int n, int id)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (t[mid].first_small <= id) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// One CTA per quantisation block of a row or column state: every block of every tensor in
// parallel (a 32000-row state has 125 blocks of 256; one CTA per tensor walked them in turn).
// A thread walks block / THREADS elements with binary64 exponentials and logarithms: the short sequences with their tables in
// shared memory (the 3346 units of the TinyLlama set: 39 us with the library's functions and 32 KB of shared memory per CTA, 32).
template <int THREADS>
__global__ void __launch_bounds__(THREADS)
factored_small_kernel(const af8_factored_tensor *tensors, int n_tensors, int conf, float floor_log)
{
    __shared__ CodecTables s_codec;
    __shared__ float s_l[SMALL_KEPT];
    __shared__ float s_red[2][SMALL_MAX_THREADS / 32];
    __shared__ double s_acc[SMALL_MAX_THREADS / 32];
    load_codec_tables(s_codec);
    await_launches();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int t = find_factored_small(tensors, n_tensors, (int)blockIdx.x);
    const af8_factored_tensor &T = tensors[t];
    const int block = (conf ? T.conf_row : T.row_var).block;
    const int64_t rows = T.rows, nbr = (rows + block - 1) / block;
    const int64_t local = (int64_t)blockIdx.x - T.first_small;
    const bool is_row = local < nbr;
    const int64_t b = is_row ? local : local - nbr;
    // a batch of matrices: the states are flat over the batch (their blocks run across the matrices); a
    // column value is the mean over the rows of its own matrix
    const af8_small_state &S = is_row ? (conf ? T.conf_row : T.row_var) : (conf ? T.conf_col : T.col_var);
    float *const out = is_row ? (conf ? T.inv_row_conf : T.inv_row) : (conf ? T.inv_col_conf : T.inv_col);
    const double *const sums = is_row ? T.row_sum : T.col_sum;
    const double count = is_row ? (double)T.cols : (double)fact_mat_rows(T);
    const float eps_add = conf ? 0.0f : T.eps1;                 // optimizer.py:2222-2223 vs 933-934
    __syncthreads();
    double part = small_state_block(S, sums, count, is_row ? rows : fact_batch(T) * T.cols, b, eps_add, conf ? T.c_w : T.v_w, floor_log,
                                    out, s_codec, s_l, s_red);
    if (!is_row) return;
    // the block's share of the mean of the row state goes where its first row sum was
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if (lane == 0) s_acc[warp] = part;
    __syncthreads();                                            // (also: every thread has read its row sums)
    if (tid == 0) {
        double s = 0.0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) s += s_acc[k];
        T.row_sum[b * block] = s;
    }
}

// grid (n_tensors, slices): mean of the row state, clamped (optimizer.py:2236, 948), then the
// inverse-std vectors (optimizer.py:818-821); the CTAs of a tensor share its elements
__global__ void __launch_bounds__(256)
factored_inv_kernel(const af8_factored_tensor *tensors, int conf)
{
    __shared__ float s_rm;
    await_launches();
    const af8_factored_tensor T = tensors[blockIdx.x];
    const int tid = threadIdx.x;
    float *inv_r = conf ? T.inv_row_conf : T.inv_row;
    float *inv_c = conf ? T.inv_col_conf : T.inv_col;
    const int block = (conf ? T.conf_row : T.row_var).block;
    const int64_t stride = (int64_t)blockDim.x * gridDim.y;
    const int64_t first = (int64_t)blockIdx.y * blockDim.x + tid;
    if (T.batch_rows > 0) {
        // a batch: the mean of each matrix's own row values (row_var.mean(dim=-2)), matrices dealt out to the
        // slices; the values are read before any of them is overwritten by this CTA's own threads
        __shared__ double s_red[8];
        const int64_t mr = T.batch_rows, nb = T.rows / mr;
        for (int64_t m = blockIdx.y; m < nb; m += gridDim.y) {
            double part = 0.0;
            for (int64_t i = tid; i < mr; i += blockDim.x) part += (double)inv_r[m * mr + i];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
            __syncthreads();
            if ((tid & 31) == 0) s_red[tid >> 5] = part;
            __syncthreads();
            double s = 0.0;
            for (int k = 0; k < 8; ++k) s += s_red[k];
            float rm = __double2float_rn(s / (double)mr);
            if (rm < T.eps1) rm = T.eps1;
            for (int64_t i = tid; i < mr; i += blockDim.x) inv_r[m * mr + i] = rsqrt_t(__fdiv_rn(inv_r[m * mr + i], rm));
        }
        for (int64_t j = first; j < nb * T.cols; j += stride) inv_c[j] = rsqrt_t(inv_c[j]);
        return;
    }
    if (tid < 32) {                                                         // (fixed order; one thread took 30 us for the 125 blocks of 32000 rows)
        double s = 0.0;
        for (int64_t e = (int64_t)tid * block; e < T.rows; e += 32 * (int64_t)block) s += T.row_sum[e];
        s = warp_sum(s);
        float rm = __double2float_rn(s / (double)T.rows);
        if (rm < T.eps1) rm = T.eps1;
        if (tid == 0) s_rm = rm;
    }
    __syncthreads();
    const float rm = s_rm;
#pragma unroll 4
    for (int64_t i = first; i < T.rows; i += stride) inv_r[i] = rsqrt_t(__fdiv_rn(inv_r[i], rm));
#pragma unroll 4
    for (int64_t j = first; j < T.cols; j += stride) inv_c[j] = rsqrt_t(inv_c[j]);
}

// ---------------------------------------------------------------------------
// update
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(FUPD_THREADS)
factored_update_kernel(const FactoredLaunch L, int chunk)
{
    extern __shared__ float s_m[];                 // new momentum of the chunk (quantised formats)
    __shared__ af8_factored_tensor sT;
    __shared__ double s_acc[FUPD_THREADS / 32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    await_launches();
    const bool has_m = L.m_fmt != AF8_M_NONE;
    const bool m_quant = has_m && L.m_fmt != AF8_M_FP32;
    const bool writes = L.mode == AF8_FUPD_APPLY || L.mode == AF8_FUPD_LAG;
    const bool sums = !writes || L.mode == AF8_FUPD_LAG;

    for (int64_t id = blockIdx.x; id < L.total_units; id += gridDim.x) {
        const int t = find_factored_chunk(L.tensors, L.n_tensors, id);
        __syncthreads();
        if (tid < (int)(sizeof(af8_factored_tensor) / 4))
            reinterpret_cast<uint32_t *>(&sT)[tid] = reinterpret_cast<const uint32_t *>(L.tensors + t)[tid];
        __syncthreads();
        const int64_t C = sT.cols, numel = sT.rows * sT.cols;
        const int64_t base = (id - sT.first_chunk) * chunk;
        const int valid = (int)min((int64_t)chunk, numel - base);
        float pre_div = 1.0f, step_mul = -sT.alpha, fira = 1.0f;
        bool zero_upd = false;
        if (L.dyn != nullptr) {
            const af8_dyn_scalars ds = L.dyn[t];
            if (L.came) pre_div = ds.pre_div;
            if (writes) { step_mul = ds.step; fira = ds.fira; zero_upd = ds.zero != 0.0f; }
        }
        if (L.mode == AF8_FUPD_SUMSQ_U) pre_div = 1.0f;           // the clip divisor is what this pass measures

        int64_t row = (base + tid) / C;
        int64_t col = (base + tid) - row * C;
        double acc = 0.0;
        for (int i = tid; i < chunk; i += FUPD_THREADS) {
            float mj = 0.0f;
            if (i < valid) {
                const int64_t flat = base + i;
                float g = load_grad_any(sT.grad, L.grad_dtype, flat);
                if (L.negate_grad) g = -g;
                const int64_t cb = fact_col_base(sT, row);                         // (a batch of matrices: that matrix's columns)
                const float ir = sT.inv_row[row], ic = sT.inv_col[cb + col];
                float u;
                if (L.came) {
                    const float uc = u_clipped(g, ir, ic, pre_div);                  // optimizer.py:929
                    if (L.mode == AF8_FUPD_SUMSQ_U) {
                        u = uc;
                    } else {
                        mj = lerp_t(m_old_at(sT, L.m_fmt, L.m_block, flat), uc, sT.m_w);   // optimizer.py:930
                        u = __fmul_rn(__fmul_rn(mj, sT.inv_row_conf[row]), sT.inv_col_conf[cb + col]);   // optimizer.py:952
                    }
                } else if (has_m) {
                    mj = lerp_t(m_old_at(sT, L.m_fmt, L.m_block, flat), g, sT.m_w);        // optimizer.py:959
                    u = __fmul_rn(__fmul_rn(mj, ir), ic);                                  // optimizer.py:961
                } else {
                    u = __fmul_rn(__fmul_rn(g, ir), ic);                                   // optimizer.py:968-969
                }
                if (sums) acc += (double)__fmul_rn(u, u);
                if (writes) {
                    if (!m_quant && has_m) sT.m_f32[flat] = mj;
                    // optimizer.py:2039, 803, 874 (a zero update still applies the decay and the rounding)
                    const float uu = zero_upd ? 0.0f : __fmul_rn(u, fira);
                    const float pv = param_load(sT.param, flat, L.param_dtype);
                    const uint32_t pbits = param_step_bits(pv, sT.decay, step_mul, uu, L.param_dtype, L.sr, sT.sr_base, flat);
                    param_store_bits(sT.param, flat, pbits, L.param_dtype);
                    if (sT.param_copy != nullptr && L.param_dtype == AF8_F32)       // bf16 compute copy
                        static_cast<uint16_t *>(sT.param_copy)[flat] = (uint16_t)f32_to_bf16_rn_bits(__uint_as_float(pbits));
                }
            }
            if (writes && m_quant) s_m[i] = mj;
            col += FUPD_THREADS;
            while (col >= C) { col -= C; ++row; }
        }
        if (sums) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (lane == 0) s_acc[warp] = acc;
            __syncthreads();
            if (tid == 0) {
                double s = 0.0;
                for (int w = 0; w < FUPD_THREADS / 32; ++w) s += s_acc[w];
                L.block_sumsq[id] = s;
            }
            if (!writes) continue;
        }
        if (m_quant) {
            __syncthreads();
            const bool four_bit = (L.m_fmt == AF8_M_UF4 || L.m_fmt == AF8_M_D4);
            const int subs = chunk / L.m_block;
            for (int sb = warp; sb < subs; sb += FUPD_THREADS / 32) {
                const int s0 = sb * L.m_block;
                if (s0 >= valid) break;
                float am = 0.0f;
                for (int i = lane; i < L.m_block; i += 32) am = fmaxf(am, fabsf(s_m[s0 + i]));
                am = fmaxf(warp_max(am), 1e-12f);
                if (four_bit) {
                    for (int i = lane * 2; i < L.m_block; i += 64)
                        sT.m_q[(base + s0 + i) >> 1] = (uint8_t)((m_encode(s_m[s0 + i], am, L.m_fmt) << 4) | m_encode(s_m[s0 + i + 1], am, L.m_fmt));
                } else {
                    for (int i = lane; i < L.m_block; i += 32)
                        sT.m_q[base + s0 + i] = (uint8_t)m_encode(s_m[s0 + i], am, L.m_fmt);
                }
                if (lane == 0) sT.m_scale[(base + s0) / L.m_block] = am;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// vectorised variants: every tensor has cols % 8 == 0 and 16-byte aligned arrays, the
// momentum block (if quantised) is 256.  A thread owns 8 consecutive elements of one row:
// 128-bit loads of the gradient, the parameter and the column vectors; a warp owns one
// momentum block, so its absmax is a warp reduction.  Same arithmetic as the kernels above.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
#ifndef AF8_FUPD_PREFETCH_AHEAD
#define AF8_FUPD_PREFETCH_AHEAD 3      /* chunks ahead that the write passes named below request from L2; 0: off */
#endif
template <typename GradT> __host__ __device__ constexpr int sizeof_grad() { return std::is_same<GradT, float>::value ? 4 : 2; }

template <typename GradT>
__device__ __forceinline__ void load_g8(const void *grad, int64_t off, int negate, float (&g)[8])
{
    stat_load_g<GradT>(grad, off, g);
    if (negate) {
#pragma unroll
        for (int j = 0; j < 8; ++j) g[j] = -g[j];
    }
}

// 8 consecutive gradient elements as loaded, so that the load of the next chunk can be
// issued before the current one is processed
template <typename GradT> struct GradRaw8;
template <> struct GradRaw8<float> {
    float4 a, b;
    __device__ __forceinline__ void zero() { a = b = make_float4(0.f, 0.f, 0.f, 0.f); }
    __device__ __forceinline__ void load(const void *grad, int64_t off)
    {
        const float4 *p = reinterpret_cast<const float4 *>(static_cast<const float *>(grad) + off);
        a = __ldcs(p); b = __ldcs(p + 1);
    }
    __device__ __forceinline__ void load_part(const void *grad, int64_t off, int n)       // the first n (< 8), zeros after them
    {
        const float *p = static_cast<const float *>(grad) + off;
        float x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = j < n ? p[j] : 0.0f;
        a = make_float4(x[0], x[1], x[2], x[3]); b = make_float4(x[4], x[5], x[6], x[7]);
    }
    __device__ __forceinline__ void from_shared(const unsigned char *p)
    {
        a = *reinterpret_cast<const float4 *>(p); b = *reinterpret_cast<const float4 *>(p + 16);
    }
    __device__ __forceinline__ void unpack(int negate, float (&g)[8]) const
    {
        g[0] = a.x; g[1] = a.y; g[2] = a.z; g[3] = a.w; g[4] = b.x; g[5] = b.y; g[6] = b.z; g[7] = b.w;
        if (negate) {
#pragma unroll
            for (int j = 0; j < 8; ++j) g[j] = -g[j];
        }
    }
};
template <> struct GradRaw8<bf16_tag> {
    uint4 a;
    __device__ __forceinline__ void zero() { a = make_uint4(0u, 0u, 0u, 0u); }
    __device__ __forceinline__ void load(const void *grad, int64_t off)
    {
        a = __ldcs(reinterpret_cast<const uint4 *>(static_cast<const uint16_t *>(grad) + off));
    }
    __device__ __forceinline__ void load_part(const void *grad, int64_t off, int n)       // the first n (< 8), zeros after them
    {
        const uint16_t *p = static_cast<const uint16_t *>(grad) + off;
        uint32_t x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = j < n ? p[j] : 0u;
        a = make_uint4(x[0] | (x[1] << 16), x[2] | (x[3] << 16), x[4] | (x[5] << 16), x[6] | (x[7] << 16));
    }
    __device__ __forceinline__ void from_shared(const unsigned char *p) { a = *reinterpret_cast<const uint4 *>(p); }
    __device__ __forceinline__ void unpack(int negate, float (&g)[8]) const
    {
        const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            g[2 * k] = __uint_as_float(w[k] << 16);
            g[2 * k + 1] = __uint_as_float(w[k] & 0xffff0000u);
        }
        if (negate) {
#pragma unroll
            for (int j = 0; j < 8; ++j) g[j] = -g[j];
        }
    }
};

__device__ __forceinline__ void load_f8(const float *p, float (&x)[8])
{
    const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(p + 4);
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
}

__device__ __forceinline__ void load_f8_ro(const float *p, float (&x)[8])
{
    const float4 a = load_state(reinterpret_cast<const float4 *>(p)), b = load_state(reinterpret_cast<const float4 *>(p + 4));
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
}

// old momentum of 8 consecutive elements (one momentum block)
// `pre`: the 8 UF8 codes if the caller has loaded them already (have_pre)
__device__ __forceinline__ void m_old8(const af8_factored_tensor &T, int m_fmt, int m_block, int64_t flat, float (&m)[8],
                                       bool have_pre = false, uint2 pre = make_uint2(0u, 0u))
{
    if (m_fmt == AF8_M_FP32) { load_f8(T.m_f32 + flat, m); return; }
    const float sc = load_state(T.m_scale + (m_block == 256 ? flat >> 8 : flat / m_block));
    if (m_fmt == AF8_M_UF8) {
        const uint2 w = have_pre ? pre : *reinterpret_cast<const uint2 *>(T.m_q + flat);
        const float mc = __fmul_rn(sc, 0.0078125f);      // fl(scale / 128): a power-of-two divisor, scale >= 1e-12
#pragma unroll
        for (int j = 0; j < 8; ++j) m[j] = __fmul_rn(byte_minus_128(j < 4 ? w.x : w.y, j & 3), mc);   // no integer conversion
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) m[j] = m_decode(T.m_q, sc, flat + j, m_fmt);
    }
}

// 8 consecutive gradient elements from an offset of any alignment, for rows whose length is no multiple of 8.  A lane's
// columns stay the same from row to row, so the offset moves by the row length; bf16: the two aligned 16-byte vectors
// around the elements are loaded (the lanes' vectors overlap: the second comes from L1) and shifted when they are
// used, so that the loads of several rows are in flight together.  Nothing at or beyond element `numel` is read.
template <typename GradT> struct GradAny8;
template <> struct GradAny8<bf16_tag> {
    uint4 a, b;
    int s;
    __device__ __forceinline__ static uint4 vec(const uint16_t *p, int64_t off, int64_t numel)
    {
        if (off + 8 <= numel) return load_state(reinterpret_cast<const uint4 *>(p + off));
        GradRaw8<bf16_tag> t;
        t.load_part(p, off, (int)(numel - off));                 // (none for a negative count)
        return t.a;
    }
    __device__ __forceinline__ void zero() { a = b = make_uint4(0u, 0u, 0u, 0u); s = 0; }
    __device__ __forceinline__ void load(const void *grad, int64_t off, int64_t numel)
    {
        const uint16_t *p = static_cast<const uint16_t *>(grad);
        s = (int)(off & 7);
        a = vec(p, off - s, numel);
        b = s ? vec(p, off - s + 8, numel) : make_uint4(0u, 0u, 0u, 0u);
    }
    __device__ __forceinline__ void unpack(int negate, float (&g)[8]) const
    {
        uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        if (s & 4) {
#pragma unroll
            for (int i = 0; i < 6; ++i) w[i] = w[i + 2];
        }
        if (s & 2) {
#pragma unroll
            for (int i = 0; i < 5; ++i) w[i] = w[i + 1];
        }
        GradRaw8<bf16_tag> t;
        const uint32_t sh = (s & 1) * 16;
        t.a = make_uint4(__funnelshift_r(w[0], w[1], sh), __funnelshift_r(w[1], w[2], sh), __funnelshift_r(w[2], w[3], sh), __funnelshift_r(w[3], w[4], sh));
        t.unpack(negate, g);
    }
};
template <> struct GradAny8<float> {
    float v[8];
    __device__ __forceinline__ void zero()
    {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = 0.0f;
    }
    __device__ __forceinline__ void load(const void *grad, int64_t off, int64_t numel)
    {
        const float *p = static_cast<const float *>(grad) + off;
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = off + j < numel ? load_state(p + j) : 0.0f;
    }
    __device__ __forceinline__ void unpack(int negate, float (&g)[8]) const
    {
#pragma unroll
        for (int j = 0; j < 8; ++j) g[j] = negate ? -v[j] : v[j];
    }
};

// old momentum of 8 consecutive elements at any offset: the run may end one momentum block and begin the next
__device__ __forceinline__ void m_old8_any(const af8_factored_tensor &T, int m_fmt, int m_block, int64_t flat, int64_t numel, float (&m)[8])
{
    if (m_fmt == AF8_M_UF8 && m_block == 256) {
        const int64_t b = flat >> 8, last = (numel - 1) >> 8;
        const int left = 256 - (int)(flat & 255);                // elements of the first block
        const float s0 = __fmul_rn(load_state(T.m_scale + b), 0.0078125f), s1 = __fmul_rn(load_state(T.m_scale + min(b + 1, last)), 0.0078125f);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t code = flat + j < numel ? (uint32_t)T.m_q[flat + j] : 128u;
            m[j] = __fmul_rn(byte_minus_128(code, 0), j < left ? s0 : s1);
        }
        return;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) m[j] = flat + j < numel ? m_old_at(T, m_fmt, m_block, flat + j) : 0.0f;
}

// values col .. col + 7 of a column vector, 0 from column C on
__device__ __forceinline__ void load_cols_any(const float *p, int64_t col, int64_t C, float (&x)[8])
{
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = col + j < C ? load_state(p + col + j) : 0.0f;
}

// values i .. i + 7 of a 16-byte aligned array, i of any alignment: the two or three aligned vectors around them, shifted
// (24 cache-line accesses a warp instead of 64 for eight scalar loads).  The last vector holds value i + 7; arrays are
// allocated in multiples of 4 values.
__device__ __forceinline__ void load_cols8_shifted(const float *v, int64_t i, float (&x)[8])
{
    const int s = (int)(i & 3);
    const float4 *p = reinterpret_cast<const float4 *>(v + (i - s));
    const float4 a = load_state(p), b = load_state(p + 1);
    float4 c = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (s) c = load_state(p + 2);
    float w[11] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y, c.z};
#pragma unroll
    for (int j = 0; j < 9; ++j) w[j] = (s & 2) ? w[j + 2] : w[j];
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = (s & 1) ? w[j + 1] : w[j];
}

// The residual pass of residual_rows for rows of any length with a momentum that has no slices (not UF8 in blocks of 256, weights of
// 1/2 and more): elements beyond the row's end count as zeros, all loads through GradAny8.
template <typename GradT, int NB>
__device__ __forceinline__ void stats_rows_any(const FactoredLaunch &L, const af8_factored_tensor &sT, int64_t r0, int64_t r_end, int64_t c,
                                               float pre_div, const float (&ic)[8], double (&cacc)[8])
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t C = sT.cols, numel = sT.rows * C;
    const int nc = (int)max((int64_t)0, min((int64_t)8, C - c));     // this lane's columns
    for (int k0 = 0; r0 + warp + 8 * k0 < r_end; k0 += NB) {         // (uniform over the warp)
        GradAny8<GradT> cur[NB];
#pragma unroll
        for (int k = 0; k < NB; ++k) {
            const int64_t r = r0 + warp + 8 * (k0 + k);
            if (nc > 0 && r < r_end) cur[k].load(sT.grad, r * C + c, numel);
            else cur[k].zero();
        }
#pragma unroll
        for (int k = 0; k < NB; ++k) {
            const int64_t r = r0 + warp + 8 * (k0 + k);
            float g[8], x[8];
            cur[k].unpack(L.negate_grad, g);
            if (nc > 0 && r < r_end) {
                const float ir = sT.inv_row[r];
                const DivBy D = make_div(pre_div);
                const LerpW LW = make_lerp(sT.m_w);
                float mo[8];
                m_old8_any(sT, L.m_fmt, L.m_block, r * C + c, numel, mo);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float u = u_clipped_fast(g[j], ir, ic[j], D);
                    const float df = __fsub_rn(u, lerp_w(mo[j], u, LW));
                    x[j] = __fadd_rn(__fmul_rn(df, df), sT.eps_came);
                }
            }
            double racc = 0.0;
            const bool live = r < r_end;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const double xd = (live && j < nc) ? (double)x[j] : 0.0;
                racc += xd;
                cacc[j] += xd;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) racc += __shfl_xor_sync(0xffffffffu, racc, o);
            if (lane == 0 && live) atomicAdd(sT.row_sum + r, racc);
        }
    }
}

// Sums over the lanes of a warp of NB values each lane holds, through `buf` (32 * NB doubles of shared memory, this warp's alone): lane l
// gets the sum of value l / (32 / NB), complete in the first lane of each such group.  Value v of lane l lies at v * 32 + (l ^ (v * G)),
// so that neither the writes nor the reads of a column of lanes meet in a bank.  (30 instructions for 8 values; exchanging halves of
// them by shuffles takes 55.)
template <int NB>
__device__ __forceinline__ double transpose_sum(const double (&x)[NB], double *buf)
{
    constexpr int G = 32 / NB;
    const int lane = threadIdx.x & 31, v = lane / G;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < NB; ++k) buf[k * 32 + (lane ^ (k * G))] = x[k];
    __syncwarp();
    double t[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) t[i] = buf[v * 32 + (lane & (G - 1)) + G * (i ^ v)];
#pragma unroll
    for (int w = NB / 2; w > 0; w >>= 1)
#pragma unroll
        for (int i = 0; i < w; ++i) t[i] += t[i + w];
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) t[0] += __shfl_xor_sync(0xffffffffu, t[0], o);
    return t[0];
}

// Row and column sums of g^2 over the rows r0 + warp + 8 k of a tile, NB rows at a time, the next NB requested before they are used.
// buf: 32 * NB doubles of this warp's.
template <typename GradT, int NB>
__device__ __forceinline__ void gradsq_rows(const af8_factored_tensor &sT, int64_t r0, int64_t r_end, int64_t c, bool col_ok, double (&cacc)[8], double *buf)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t step = 8 * sT.cols;
    int64_t off = (r0 + warp) * sT.cols + c;
    int left = r0 + warp < r_end ? (int)((r_end - (r0 + warp) + 7) / 8) : 0;         // rows from the next group on
    double *to = sT.row_sum + r0 + warp + 8 * (lane / (32 / NB));
    const auto load = [&](GradRaw8<GradT> (&raw)[NB], int rows) {
#pragma unroll
        for (int k = 0; k < NB; ++k, off += step) {
            raw[k].zero();
            if (col_ok && k < rows) raw[k].load(sT.grad, off);
        }
    };
    const auto add = [&](const GradRaw8<GradT> (&raw)[NB]) {
        double rsum[NB];
#pragma unroll
        for (int k = 0; k < NB; ++k) {
            float g[8];
            raw[k].unpack(0, g);
            double t[4];
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                const float2 gj = make_float2(g[j], g[j + 1]), xx = __fmul2_rn(gj, gj);
                const double xa = (double)xx.x, xb = (double)xx.y;
                cacc[j] += xa;
                cacc[j + 1] += xb;
                t[j >> 1] = xa + xb;
            }
            rsum[k] = (t[0] + t[1]) + (t[2] + t[3]);
        }
        const double v = transpose_sum(rsum, buf);
        if ((lane & (32 / NB - 1)) == 0 && lane / (32 / NB) < left) atomicAdd(to, v);
        to += 8 * NB;
        left -= NB;
    };
    GradRaw8<GradT> a[NB], b[NB];
    load(a, left);
    while (left > 0) {                                               // (uniform over the warp)
        load(b, left - NB);
        add(a);
        if (left <= 0) break;
        load(a, left - NB);
        add(b);
    }
    __syncwarp();
}

// The residual pass over whole vectors of 8 without a ring (a momentum that is not UF8 in blocks of 256, a clip divisor below 1, momentum
// weights of 1/2 and more in tables with batches or rows of any length): rows r0 + warp + 8 k of the tile, two at a time, the loads of the next
// two issued before these are used.
template <typename GradT>
__device__ __forceinline__ void residual_rows(const FactoredLaunch &L, const af8_factored_tensor &sT, int64_t r0, int64_t r_end, int64_t c,
                                              bool col_ok, float pre_div, const float (&ic)[8], double (&cacc)[8])
{
    constexpr int NB = 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t R = r_end, C = sT.cols;            // r_end: end of the unit's rows
    GradRaw8<GradT> cur[NB], nxt[NB];
    auto fetch = [&](GradRaw8<GradT> (&dst)[NB], int k0) {
#pragma unroll
        for (int k = 0; k < NB; ++k) {
            const int64_t r = r0 + warp + 8 * (k0 + k);
            if (col_ok && r < R) dst[k].load(sT.grad, r * C + c);
            else dst[k].zero();
        }
    };
    fetch(cur, 0);
    for (int k0 = 0; r0 + warp + 8 * k0 < R; k0 += NB) {          // (uniform over the warp)
        fetch(nxt, k0 + NB);
        float g[NB][8];
        double rsum[NB];
#pragma unroll
        for (int k = 0; k < NB; ++k) {
            cur[k].unpack(L.negate_grad, g[k]);
            cur[k] = nxt[k];
        }
#pragma unroll
        for (int k = 0; k < NB; ++k) {
            const int64_t r = r0 + warp + 8 * (k0 + k);
            const bool live = col_ok && r < R;
            float x[8];
            if (live) {
                const int64_t flat = r * C + c;
                const float2 ir2 = bc2(sT.inv_row[r]);
                const DivBy D = make_div(pre_div);
                const LerpW LW = make_lerp(sT.m_w);
                const float2 eps2 = bc2(sT.eps_came);
                float mo[8];
                m_old8(sT, L.m_fmt, L.m_block, flat, mo);
#pragma unroll
                for (int j = 0; j < 8; j += 2) {       // pairs in packed binary32 arithmetic (bit-identical to element-wise)
                    const float2 u = div_by2(__fmul2_rn(__fmul2_rn(make_float2(g[k][j], g[k][j + 1]), ir2), make_float2(ic[j], ic[j + 1])), D);
                    const float2 m = lerp_w2(make_float2(mo[j], mo[j + 1]), u, LW);
                    const float2 df = sub2(u, m);
                    const float2 xx = __fadd2_rn(__fmul2_rn(df, df), eps2);
                    x[j] = xx.x; x[j + 1] = xx.y;
                }
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) x[j] = 0.0f;
            }
            double racc = 0.0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const double xd = (double)x[j];
                racc += xd;
                cacc[j] += xd;
            }
            rsum[k] = racc;
        }
        // the two row sums of the warp are reduced together: the first exchange leaves one value a lane; row k0 + i ends in lane 16 i
        const bool hi = lane & 16;
        double v = (hi ? rsum[1] : rsum[0]) + __shfl_xor_sync(0xffffffffu, hi ? rsum[0] : rsum[1], 16);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((lane & 15) == 0) {
            const int64_t r = r0 + warp + 8 * (k0 + (lane >> 4));
            if (r < R) atomicAdd(sT.row_sum + r, v);
        }
    }
}

// 8 UF8 codes of one momentum block as floats: (code - 128) * mc, two elements per instruction; each
// component rounds like the scalar form in m_old8
__device__ __forceinline__ void uf8_decode8(uint2 w, float mc, float2 (&m)[4])
{
    const float2 off = bc2(-8388736.0f), mc2 = bc2(mc);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t word = j < 2 ? w.x : w.y;
        const float2 b = make_float2(__uint_as_float(__byte_perm(word, 0x4b000000u, 0x7540u | (uint32_t)((2 * j) & 3))),
                                     __uint_as_float(__byte_perm(word, 0x4b000000u, 0x7540u | (uint32_t)((2 * j + 1) & 3))));
        m[j] = __fmul2_rn(__fadd2_rn(b, off), mc2);
    }
}

// CAME's residual (U - M)^2 + eps of 8 elements, M the momentum after this step's EMA.
// ONE: the clip divisor is 1; SMALL: |momentum weight| < 0.5 (the form of lerp).  The quotient is taken
// without div_by's test for an infinite product.  The caller guarantees a divisor d >= 1 (or NaN), as the
// RMS clip produces: then a finite t = g * r * c has a finite product t * fl(1 / d), and an infinite or NaN t
// ends as x = NaN with the true quotient as well (U and M are both infinite, U - M is NaN).
template <bool ONE, bool SMALL>
__device__ __forceinline__ void residual_m8(const float (&g)[8], const float2 (&mo)[4], float ir, const float (&ic)[8],
                                            const DivBy &D, float ww, float eps, float (&x)[8])
{
    const float2 ir2 = bc2(ir), r2 = bc2(D.rcp), nd2 = bc2(D.nd), ww2 = bc2(ww), eps2 = bc2(eps);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 t = __fmul2_rn(__fmul2_rn(make_float2(g[2 * j], g[2 * j + 1]), ir2), make_float2(ic[2 * j], ic[2 * j + 1]));
        float2 u = t;
        if (!ONE) {
            const float2 q = __fmul2_rn(t, r2);
            u = __ffma2_rn(__ffma2_rn(q, nd2, t), r2, q);
        }
        const float2 m = __ffma2_rn(ww2, sub2(u, mo[j]), SMALL ? mo[j] : u);
        const float2 df = sub2(u, m);
        const float2 xx = __fadd2_rn(__fmul2_rn(df, df), eps2);
        x[2 * j] = xx.x; x[2 * j + 1] = xx.y;
    }
}

template <bool ONE, bool SMALL>
__device__ __forceinline__ void residual_x8(const float (&g)[8], uint2 codes, float mc, float ir, const float (&ic)[8],
                                            const DivBy &D, float ww, float eps, float (&x)[8])
{
    float2 mo[4];
    uf8_decode8(codes, mc, mo);
    residual_m8<ONE, SMALL>(g, mo, ir, ic, D, ww, eps, x);
}

// Passes over the rows r0 + warp + 8 k of a tile whose row slices (up to 256 columns of gradient and, with a momentum, its UF8
// codes) come through the warp's ring, for matrices with rows of any length.  A slice may begin and end anywhere: what is copied
// are the 16-byte units around it, and the lanes read from its place inside them.  With whole vectors of 8 (VEC) a lane owns 8
// consecutive columns, as elsewhere; else the columns lane + 32 j, one 2-byte and one 1-byte access each without bank conflicts,
// which is cheaper than shifting vectors (rows of 1001 and 2731 elements, 59 M parameters: g^2 sums 113 -> 67 us).
// Requests go out for four rows at a time, by eight lanes with the same instructions (lane 2 i: the gradient of row i, lane
// 2 i + 1: its codes): a request of one lane for one row costs about 57 issue slots.  Rows are consumed in pairs whose row sums
// are reduced jointly; the per-row scalars (inverse row factor, block absmax) are loaded a pair ahead.
//   SLICE_GRADSQ    row and column sums of g^2
//   SLICE_RESIDUAL  of CAME's residual; the sign of a negated gradient rides on the row factor ((-g) * r == g * (-r) bit for bit)
//   SLICE_SUM_U     sum of squares of u = g * inv_row * inv_col
//   SLICE_SUM_M     the same with the momentum after its EMA in place of g
// The residual wants a clip divisor of at least 1, or NaN.
enum { SLICE_GRADSQ = 0, SLICE_RESIDUAL = 1, SLICE_SUM_U = 2, SLICE_SUM_M = 3 };
template <typename GradT> __host__ __device__ constexpr int slice_g_bytes() { return 256 * sizeof_grad<GradT>() + 16; }
template <typename GradT> __host__ __device__ constexpr int slice_row_bytes() { return slice_g_bytes<GradT>() + 256 + 16; }
constexpr int SLICE_ROWS = 4, SLICE_STAGES = 2;
template <typename GradT> __host__ __device__ constexpr size_t slice_warp_bytes() { return (size_t)SLICE_STAGES * SLICE_ROWS * slice_row_bytes<GradT>(); }
template <typename GradT> __host__ __device__ constexpr size_t slice_smem_bytes() { return 8 * slice_warp_bytes<GradT>(); }

// false after a time-out.  cacc: the lane's column sums; total: the sum of squares (by_eight: eight squares are added in binary32
// before they enter binary64).  FORM: SLICE_RESIDUAL: the clip divisor is 1; SLICE_SUM_M: the momentum's weight is below 1/2.
// SMALL: SLICE_RESIDUAL: the momentum's weight is below 1/2 (the form of lerp).
template <typename GradT, int MODE, bool VEC, bool FORM, bool SMALL = true>
__device__ __forceinline__ bool slice_rows(const FactoredLaunch &L, const af8_factored_tensor &sT, int64_t r0, int64_t r_end, int64_t c0,
                                           float pre_div, bool by_eight, const float (&ic)[8], double (&cacc)[8], double &total,
                                           unsigned char *ring, uint64_t *full, uint32_t &cons)
{
    constexpr int GB = sizeof_grad<GradT>(), ROWB = slice_row_bytes<GradT>(), STAGE = SLICE_ROWS * ROWB, M_OFF = slice_g_bytes<GradT>();
    constexpr bool MOM = MODE == SLICE_RESIDUAL || MODE == SLICE_SUM_M, SUM = MODE == SLICE_SUM_U || MODE == SLICE_SUM_M;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t C = sT.cols, numel = sT.rows * C, step = 8 * C;
    const int w = (int)min((int64_t)256, C - c0);
    const int64_t row0 = r0 + warp;
    const int nrows = row0 < r_end ? (int)((r_end - row0 + 7) / 8) : 0, ngroups = (nrows + SLICE_ROWS - 1) / SLICE_ROWS;
    // the gradient's last 16-byte unit, if it is not whole, is not copied: the last row's elements there are fetched one by one
    const int64_t g_end = (numel * GB) & ~(int64_t)15;
    const int k_last = nrows - 1;
    const bool tail = k_last >= 0 && row0 + 8 * (int64_t)k_last == sT.rows - 1 && ((sT.rows - 1) * C + c0 + w) * GB > g_end;
    int64_t from_off = (row0 + 8 * (int64_t)((lane >> 1) & 3)) * C + c0;      // lanes 0-7: first element of their row's slice in the next group
    auto issue = [&](int g) {                                        // lanes 0-7: group g into its stage
        const int sl = (int)((cons + (uint32_t)g) & (SLICE_STAGES - 1));
        const int i = lane >> 1, k = SLICE_ROWS * g + i;
        const bool code = lane & 1;
        int bytes = 0;
        const int64_t first = code ? from_off : from_off * GB, from = first & ~(int64_t)15;
        if (k < nrows && (MOM || !code)) {
            bytes = ((int)(first - from) + (code ? w : w * GB) + 15) & ~15;
            if (!code && tail && k == k_last) bytes = max((int)min((int64_t)bytes, g_end - from), 0);
        }
        from_off += SLICE_ROWS * step;
        const int both = bytes + (MOM ? __shfl_xor_sync(0xffu, bytes, 1) : 0);
        if (!code) mbar_expect_tx(&full[sl], (uint32_t)both);        // (four arrivals a phase)
        if (bytes > 0)
            bulk_g2s(ring + sl * STAGE + i * ROWB + (code ? M_OFF : 0),
                     (code ? sT.m_q : static_cast<const unsigned char *>(sT.grad)) + from, (uint32_t)bytes, &full[sl]);
    };
    if (lane < 8 && ngroups > 0) {
        fence_proxy_async();
        for (int g = 0; g < min(SLICE_STAGES, ngroups); ++g) issue(g);
    }
    const DivBy D = make_div(pre_div);
    const LerpW LW = make_lerp(sT.m_w);
    const float eps = sT.eps_came, sgn = (MODE == SLICE_RESIDUAL && L.negate_grad) ? -1.0f : 1.0f;
    const bool col_ok = VEC ? lane * 8 < w : true;                   // this lane's columns (VEC: all or none)
    // the scalars of the next pair of rows
    const int last_block = (int)((numel - 1) >> 8);
    const float *pr = sT.inv_row + row0;
    int64_t soff = row0 * C + c0 + (VEC && col_ok ? lane * 8 : 0);
    float nir[2], ns0[2], ns1[2];
    auto scalars = [&](int q, int k) {
        nir[q] = ns0[q] = ns1[q] = 0.0f;
        if (k < nrows) {
            if (MODE != SLICE_GRADSQ) nir[q] = load_state(pr);
            if (MOM) {
                const int block = (int)(soff >> 8);                  // (fewer than 2^31 blocks, as rows)
                ns0[q] = load_state(sT.m_scale + block);
                if (!VEC) ns1[q] = load_state(sT.m_scale + min(block + 1, last_block));
            }
        }
        pr += 8;
        soff += step;
    };
    scalars(0, 0);
    scalars(1, 1);
    uint32_t lo = (uint32_t)(row0 * C + c0);                         // low word of the offset of the row at hand
    for (int g = 0; g < ngroups; ++g) {
        const uint32_t n = cons + (uint32_t)g;
        const int sl = (int)(n & (SLICE_STAGES - 1));
        const bool landed = mbar_wait_bounded(&full[sl], (n / SLICE_STAGES) & 1u);
        if (!__all_sync(0xffffffffu, landed)) return false;
        unsigned char *st = ring + sl * STAGE;
        if (tail && k_last - SLICE_ROWS * g < SLICE_ROWS) {          // the tensor's last elements
            const int64_t off = (sT.rows - 1) * C + c0;
            const int idx = (int)max((int64_t)0, g_end / GB - off) + lane;
            unsigned char *const to = st + (k_last - SLICE_ROWS * g) * ROWB + ((int)(off * GB) & 15) + idx * GB;
            if (idx < w) {
                if (GB == 4) *reinterpret_cast<float *>(to) = static_cast<const float *>(sT.grad)[off + idx];
                else *reinterpret_cast<uint16_t *>(to) = static_cast<const uint16_t *>(sT.grad)[off + idx];
            }
            __syncwarp();
        }
#pragma unroll
        for (int h = 0; h < SLICE_ROWS / 2; ++h) {
            float gv[2][8];
            float2 mo[2][4];
            float irv[2];
#pragma unroll
            for (int q = 0; q < 2; ++q, st += ROWB, lo += (uint32_t)step) {
                irv[q] = MODE == SLICE_RESIDUAL ? __fmul_rn(nir[q], sgn) : nir[q];
                const float m0 = __fmul_rn(ns0[q], 0.0078125f), m1 = __fmul_rn(ns1[q], 0.0078125f);      // fl(scale / 128), scale >= 1e-12
                if (VEC) {
                    GradRaw8<GradT> raw;
                    raw.from_shared(st + lane * (8 * GB));
                    raw.unpack(MODE == SLICE_SUM_M ? L.negate_grad : 0, gv[q]);
                    if (MOM) uf8_decode8(*reinterpret_cast<const uint2 *>(st + M_OFF + (lo & 8u) + lane * 8), m0, mo[q]);
                } else {
                    const unsigned char *const gp = st + ((lo * GB) & 15u) + lane * GB, *const mp = st + M_OFF + (lo & 15u) + lane;
                    const int bound = 256 - (int)(lo & 255u) - lane;         // 32 j from here on: the next momentum block
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        float x;
                        if (GB == 4) x = *reinterpret_cast<const float *>(gp + 32 * j * GB);
                        else x = __uint_as_float((uint32_t)*reinterpret_cast<const uint16_t *>(gp + 32 * j * GB) << 16);
                        gv[q][j] = (MODE == SLICE_SUM_M && L.negate_grad) ? -x : x;
                        if (MOM) {
                            const float y = __fmul_rn(__uint_as_float(0x4b000000u | mp[32 * j]) - 8388736.0f, 32 * j < bound ? m0 : m1);
                            if (j & 1) mo[q][j >> 1].y = y; else mo[q][j >> 1].x = y;
                        }
                    }
                }
            }
            if (h == SLICE_ROWS / 2 - 1) {                           // the stage was read: it may be refilled
                __syncwarp();
                if (lane < 8 && g + SLICE_STAGES < ngroups) { fence_proxy_async(); issue(g + SLICE_STAGES); }
            }
            const int k0 = SLICE_ROWS * g + 2 * h;
            scalars(0, k0 + 2);
            scalars(1, k0 + 3);
            double rsum[2] = {0.0, 0.0};
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                if (k0 + q >= nrows) continue;                       // (uniform over the warp)
                float x[8];
                if (MODE == SLICE_GRADSQ) {
#pragma unroll
                    for (int j = 0; j < 8; j += 2) {
                        const float2 gj = make_float2(gv[q][j], gv[q][j + 1]), xx = __fmul2_rn(gj, gj);
                        x[j] = xx.x; x[j + 1] = xx.y;
                    }
                } else if (MODE == SLICE_RESIDUAL) {
                    residual_m8<FORM, SMALL>(gv[q], mo[q], irv[q], ic, D, LW.ww, eps, x);
                } else {
                    const float2 ir2 = bc2(irv[q]), ww2 = bc2(LW.ww);
#pragma unroll
                    for (int j = 0; j < 8; j += 2) {
                        float2 t = make_float2(gv[q][j], gv[q][j + 1]);
                        if (MOM) t = __ffma2_rn(ww2, sub2(t, mo[q][j >> 1]), FORM ? mo[q][j >> 1] : t);
                        const float2 u = __fmul2_rn(__fmul2_rn(t, ir2), make_float2(ic[j], ic[j + 1]));
                        x[j] = u.x; x[j + 1] = u.y;
                    }
                }
                if (VEC) {                                           // (beyond the slice the stage holds what it held)
                    if (!col_ok) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) x[j] = 0.0f;
                    }
                } else if (w < 256) {                                // (uniform over the warp)
#pragma unroll
                    for (int j = 0; j < 8; ++j) x[j] = lane + 32 * j < w ? x[j] : 0.0f;
                }
                if (SUM && by_eight) {
                    float2 a2 = __fmul2_rn(make_float2(x[0], x[1]), make_float2(x[0], x[1]));
#pragma unroll
                    for (int j = 2; j < 8; j += 2) a2 = __ffma2_rn(make_float2(x[j], x[j + 1]), make_float2(x[j], x[j + 1]), a2);
                    rsum[q] = (double)__fadd_rn(a2.x, a2.y);
                } else {
                    double pr2[4];                                   // (pairwise: a short dependency chain)
#pragma unroll
                    for (int j = 0; j < 8; j += 2) {
                        const double xa = (double)(SUM ? __fmul_rn(x[j], x[j]) : x[j]), xb = (double)(SUM ? __fmul_rn(x[j + 1], x[j + 1]) : x[j + 1]);
                        if (!SUM) { cacc[j] += xa; cacc[j + 1] += xb; }
                        pr2[j >> 1] = xa + xb;
                    }
                    rsum[q] = (pr2[0] + pr2[1]) + (pr2[2] + pr2[3]);
                }
            }
            if (SUM) {
                total += rsum[0] + rsum[1];
            } else {
                const bool hi = lane & 16;
                double v = (hi ? rsum[1] : rsum[0]) + __shfl_xor_sync(0xffffffffu, hi ? rsum[0] : rsum[1], 16);
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                const int k = k0 + (lane >> 4);
                if ((lane & 15) == 0 && k < nrows) atomicAdd(sT.row_sum + row0 + 8 * (int64_t)k, v);
            }
        }
    }
    cons += (uint32_t)ngroups;
    return true;
}

// a lane's eight column factors for slice_rows
template <bool VEC>
__device__ __forceinline__ void slice_cols(const float *inv_col, int64_t c0, int64_t C, float (&ic)[8])
{
    const int lane = threadIdx.x & 31;
    if constexpr (VEC) {
        if (c0 + lane * 8 < C) load_f8_ro(inv_col + c0 + lane * 8, ic);
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (c0 + lane + 32 * j < C) ic[j] = load_state(inv_col + c0 + lane + 32 * j);
    }
}

// The same pass with the input of FBOX_ROWS consecutive rows per copy: one tiled bulk tensor copy brings their
// 256-column slices of the gradient (tensor map maps[0]: bf16 [rows][cols], box 256 x FBOX_ROWS), one their UF8 codes
// (maps[1]: bytes, same box) into a stage of the warp's two-stage ring, so that the instructions of a request -
// about 57 issue slots with one lane active - are spent once per FBOX_ROWS rows instead of once per row.  Warp w
// takes the row groups r0 + FBOX_ROWS (w + 8 k); rows past the end of the unit are skipped (past the end of the tensor they arrive as zeros).
// bf16 gradients only (a stage is 3 KB).
constexpr int FBOX_ROWS = 4, FBOX_STAGES = 2;
constexpr int FBOX_G_BYTES = FBOX_ROWS * 512, FBOX_STAGE_BYTES = FBOX_G_BYTES + FBOX_ROWS * 256;
static_assert(FBOX_STAGES * FBOX_STAGE_BYTES <= (int)slice_warp_bytes<bf16_tag>() && slice_warp_bytes<bf16_tag>() % 128 == 0, "the boxes use the slices' memory");
static_assert(FBOX_STAGES == SLICE_STAGES, "and their barriers");
static_assert(FSTAT_ROWS % (8 * FBOX_ROWS) == 0, "whole row groups per warp and tile");

template <bool ONE, bool SMALL>
__device__ __forceinline__ bool residual_rows_box(const FactoredLaunch &L, const af8_factored_tensor &sT, const CUtensorMap *maps,
                                                  int64_t r0, int64_t row_end, int64_t c0, float pre_div, const float (&ic)[8], double (&cacc)[8],
                                                  unsigned char *ring, uint64_t *full, uint32_t &cons)
{
    constexpr int BR = FBOX_ROWS, NS = FBOX_STAGES;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t C = sT.cols;
    const int r_end = (int)row_end;
    const int row0 = (int)r0 + BR * warp;                        // first row of this warp's group 0; group g: + 8 * BR * g
    const int ngroups = row0 < r_end ? (r_end - row0 + 8 * BR - 1) / (8 * BR) : 0;
    auto issue = [&](int g) {                                    // lane 0: group g into its stage
        const int sl = (int)((cons + (uint32_t)g) & (uint32_t)(NS - 1));
        unsigned char *dst = ring + sl * FBOX_STAGE_BYTES;
        mbar_expect_tx(&full[sl], (uint32_t)FBOX_STAGE_BYTES);
        tma_load_2d(dst, maps, (int)c0, row0 + 8 * BR * g, &full[sl]);
        tma_load_2d(dst + FBOX_G_BYTES, maps + 1, (int)c0, row0 + 8 * BR * g, &full[sl]);
    };
    if (lane == 0 && ngroups > 0) {
        fence_proxy_async();
        for (int g = 0; g < min(NS, ngroups); ++g) issue(g);
    }
    const DivBy D = make_div(pre_div);
    const LerpW LW = make_lerp(sT.m_w);
    const float eps = sT.eps_came, sgn = L.negate_grad ? -1.0f : 1.0f;
    // row r: inverse row factor at index r, block absmax at r * (C / 256) + c0 / 256 (both fit 32 bits)
    const int scrow = (int)(C >> 8), scoff = (int)(c0 >> 8);
    float nir[2], nsc[2];                                        // the scalars of the next pair of rows
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        nir[k] = 0.0f; nsc[k] = 0.0f;
        if (row0 + k < r_end) { nir[k] = load_state(sT.inv_row + row0 + k); nsc[k] = load_state(sT.m_scale + (row0 + k) * scrow + scoff); }
    }
    for (int g = 0; g < ngroups; ++g) {
        const uint32_t n = cons + (uint32_t)g;
        const int sl = (int)(n & (uint32_t)(NS - 1));
        const bool landed = mbar_wait_bounded(&full[sl], (n / NS) & 1u);
        if (!__all_sync(0xffffffffu, landed)) return false;
        const unsigned char *st = ring + sl * FBOX_STAGE_BYTES;
        const int grow = row0 + 8 * BR * g;                      // first row of the group
#pragma unroll
        for (int h = 0; h < BR / 2; ++h) {                       // pairs of rows: their row sums are reduced jointly
            GradRaw8<bf16_tag> cur[2];
            uint2 cm[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                cur[k].from_shared(st + (2 * h + k) * 512 + lane * 16);
                cm[k] = *reinterpret_cast<const uint2 *>(st + FBOX_G_BYTES + (2 * h + k) * 256 + lane * 8);
            }
            if (h == BR / 2 - 1) {                               // the stage was read: it may be refilled
                __syncwarp();
                if (lane == 0 && g + NS < ngroups) { fence_proxy_async(); issue(g + NS); }
            }
            double rsum[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int r = grow + 2 * h + k;
                double racc = 0.0;
                const float ir = __fmul_rn(nir[k], sgn), mc = __fmul_rn(nsc[k], 0.0078125f);   // fl(scale / 128), scale >= 1e-12
                {   // this row's successor: the same place of the next pair
                    const int rn = (h == BR / 2 - 1) ? r + 8 * BR - (BR - 2) : r + 2;
                    if (rn < r_end) { nir[k] = load_state(sT.inv_row + rn); nsc[k] = load_state(sT.m_scale + rn * scrow + scoff); }
                }
                if (r < r_end) {
                    float gg[8], x[8];
                    cur[k].unpack(0, gg);
                    residual_x8<ONE, SMALL>(gg, cm[k], mc, ir, ic, D, LW.ww, eps, x);
                    double pr[4];                               // (pairwise: a short dependency chain)
#pragma unroll
                    for (int j = 0; j < 8; j += 2) {
                        const double xa = (double)x[j], xb = (double)x[j + 1];
                        cacc[j] += xa;
                        cacc[j + 1] += xb;
                        pr[j >> 1] = xa + xb;
                    }
                    racc = (pr[0] + pr[1]) + (pr[2] + pr[3]);
                }
                rsum[k] = racc;
            }
            const bool hi = lane & 16;
            double v = (hi ? rsum[1] : rsum[0]) + __shfl_xor_sync(0xffffffffu, hi ? rsum[0] : rsum[1], 16);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            const int rr = grow + 2 * h + (lane >> 4);
            if ((lane & 15) == 0 && rr < r_end) atomicAdd(sT.row_sum + rr, v);
        }
    }
    cons += (uint32_t)ngroups;
    return true;
}

// RESIDUAL: CAME's (U - M)^2 + eps statistic; otherwise g^2 (separate instantiations, so that
// the lighter one keeps its lower register count)
// resident CTAs asked of the compiler (measured on B200: 3 for both passes; the g*g pass went
// from 1.02 to 0.76 ms on the TinyLlama set with it)
#ifndef AF8_FSTAT_MIN_CTAS
#define AF8_FSTAT_MIN_CTAS 3
#endif
#ifndef AF8_FSTAT_MIN_CTAS_RES
#define AF8_FSTAT_MIN_CTAS_RES 3
#endif
// ANY: the table has batches of matrices or rows whose length is no multiple of 8 (tensor by tensor)
// IN: how the rows come.  0: direct loads, 1: slices (per tensor, where its form allows), 2: boxes through tensor maps (bf16
// gradients, cols % 256 == 0; residual pass)
template <typename GradT, bool RESIDUAL, bool ANY, int IN>
__global__ void __launch_bounds__(256, (ANY && RESIDUAL) || (std::is_same<GradT, float>::value && (ANY || IN)) ? 2 : RESIDUAL ? AF8_FSTAT_MIN_CTAS_RES : AF8_FSTAT_MIN_CTAS)
factored_stats_vec_kernel(const FactoredLaunch L, const CUtensorMap *__restrict__ maps)
{
    __shared__ double s_col[8][FSTAT_COLS];      // [warp][j * 32 + lane]
    __shared__ af8_factored_tensor sT;
    extern __shared__ __align__(128) unsigned char sr_smem[];            // the warps' input rings (IN)
    __shared__ __align__(8) uint64_t s_full[8][SLICE_STAGES];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int cur_t = -1;
    uint32_t cons = 0;                           // row slices this warp has taken from its ring
    [[maybe_unused]] int mapped = -1;            // tensor whose maps this warp's lane 0 has acquired
    if (IN) {
        if (lane == 0) {
            for (int k = 0; k < SLICE_STAGES; ++k) mbar_init(&s_full[warp][k], IN == 2 ? 1 : SLICE_ROWS);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncthreads();
    }
    await_launches();

    for (int64_t id = blockIdx.x; id < L.total_units; id += gridDim.x) {
        int t = cur_t;
        const int64_t tile = id >> L.split;
        if (t < 0) t = find_factored_tile(L.tensors, L.n_tensors, tile);
        else while (t + 1 < L.n_tensors && L.tensors[t + 1].first_tile <= tile) ++t;
        __syncthreads();                                           // s_col of the previous tile was read
        if (t != cur_t) {
            if (tid < (int)(sizeof(af8_factored_tensor) / 4))
                reinterpret_cast<uint32_t *>(&sT)[tid] = reinterpret_cast<const uint32_t *>(L.tensors + t)[tid];
            cur_t = t;
            __syncthreads();
        }
        const int64_t C = sT.cols;
        const TilePos P = tile_pos(L, sT, id);
        const int64_t r0 = P.r0, row_end = P.r_end, c0 = P.c0;
        if (r0 >= row_end) continue;                               // an empty part of a split tile
        const int64_t c = c0 + lane * 8;                           // this lane's 8 columns
        const bool col_ok = c < C;                                 // C % 8 == 0: all 8 or none
        float pre_div = 1.0f;
        float ic[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) ic[j] = 0.0f;
        // Whole rows of vectors or not; which of the row loops.  Rows of any length take the slices in both passes, whole vectors
        // in the residual pass (339 M parameters in rows of 2000: direct loads 875 us, slices 472; of 1999: 1189 and 579); the g*g
        // pass over whole vectors was slower through a ring (3.0 -> 4.3 ms on Llama-2-7B) and loads directly.
        const bool vec = !ANY || (C & 7) == 0;
        // A momentum weight of 1/2 or more takes the other form of lerp.  (Direct loads and slices: 202 M parameters with binary32
        // gradients in rows of 256 n 528 and 277 us, 235 M bf16 ones in rows of which some are such 638 and 341.)
        bool slices = IN == 1 && (RESIDUAL || !vec);
        const bool small = !RESIDUAL || fabsf(sT.m_w) < 0.5f;                    // (uniform over the tensor)
        if (RESIDUAL) {
            pre_div = L.dyn[t].pre_div;
            slices = slices && L.m_fmt == AF8_M_UF8 && L.m_block == 256 && !(pre_div < 1.0f) && (!ANY || small);
            if (slices && !vec) slice_cols<false>(sT.inv_col + P.cb, c0, C, ic);
            else if (!vec) load_cols_any(sT.inv_col + P.cb, c, C, ic);
            else if (col_ok) load_f8_ro(sT.inv_col + P.cb + c, ic);
        }
        double cacc[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) cacc[j] = 0.0;
        bool ok = true, boxes = false;
        if constexpr (IN == 2) {
            if (!(pre_div < 1.0f)) {                                             // boxes of rows through tensor maps
                boxes = true;
                const bool one = pre_div == 1.0f;
                unsigned char *ring = sr_smem + (size_t)warp * slice_warp_bytes<GradT>();
                const CUtensorMap *mp = maps + 2 * t;
                if (lane == 0 && t != mapped) { tensormap_acquire(mp); tensormap_acquire(mp + 1); mapped = t; }
                if (one) ok = small ? residual_rows_box<true, true>(L, sT, mp, r0, row_end, c0, pre_div, ic, cacc, ring, s_full[warp], cons)
                                    : residual_rows_box<true, false>(L, sT, mp, r0, row_end, c0, pre_div, ic, cacc, ring, s_full[warp], cons);
                else ok = small ? residual_rows_box<false, true>(L, sT, mp, r0, row_end, c0, pre_div, ic, cacc, ring, s_full[warp], cons)
                                : residual_rows_box<false, false>(L, sT, mp, r0, row_end, c0, pre_div, ic, cacc, ring, s_full[warp], cons);
            }
        }
        if (boxes) { }
        else if (slices) {
            if constexpr (IN == 1) {
            unsigned char *ring = sr_smem + (size_t)warp * slice_warp_bytes<GradT>();
            [[maybe_unused]] double none = 0.0;
            if constexpr (RESIDUAL) {
                const bool one = pre_div == 1.0f;
                if (!ANY && !small) ok = slice_rows<GradT, SLICE_RESIDUAL, true, false, false>(L, sT, r0, row_end, c0, pre_div, false, ic, cacc, none, ring, s_full[warp], cons);
                else if (vec) ok = one ? slice_rows<GradT, SLICE_RESIDUAL, true, true>(L, sT, r0, row_end, c0, pre_div, false, ic, cacc, none, ring, s_full[warp], cons)
                                  : slice_rows<GradT, SLICE_RESIDUAL, true, false>(L, sT, r0, row_end, c0, pre_div, false, ic, cacc, none, ring, s_full[warp], cons);
                else if constexpr (ANY)
                    ok = one ? slice_rows<GradT, SLICE_RESIDUAL, false, true>(L, sT, r0, row_end, c0, pre_div, false, ic, cacc, none, ring, s_full[warp], cons)
                             : slice_rows<GradT, SLICE_RESIDUAL, false, false>(L, sT, r0, row_end, c0, pre_div, false, ic, cacc, none, ring, s_full[warp], cons);
            } else if constexpr (ANY) {
                ok = slice_rows<GradT, SLICE_GRADSQ, false, true>(L, sT, r0, row_end, c0, 1.0f, false, ic, cacc, none, ring, s_full[warp], cons);
            }
            }
        } else if (!vec) {
            if constexpr (ANY && RESIDUAL) stats_rows_any<GradT, 4>(L, sT, r0, row_end, c, pre_div, ic, cacc);
        } else if (!RESIDUAL) gradsq_rows<GradT, sizeof_grad<GradT>() == 2 ? 4 : 2>(sT, r0, row_end, c, col_ok, cacc, s_col[warp]);
        else residual_rows<GradT>(L, sT, r0, row_end, c, col_ok, pre_div, ic, cacc);
        if (!ok) {
            atomicExch(&g_device_error, DEVERR_SRING_TIMEOUT);
            return;                      // (the whole warp; the others finish their rows and leave at the next barrier)
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) s_col[warp][j * 32 + lane] = cacc[j];
        __syncthreads();
        // thread tid owns column c0 + tid = c0 + 8 * (tid >> 3) + (tid & 7) (slices of rows of any length: lane + 32 j as they lie)
        const int place = slices && !vec ? tid : (tid & 7) * 32 + (tid >> 3);
        if (c0 + tid < C) {
            double sum = 0.0;
#pragma unroll
            for (int w = 0; w < 8; ++w) sum += s_col[w][place];
            atomicAdd(sT.col_sum + P.cb + c0 + tid, sum);
        }
    }
}

// chunk = 2048 elements = 8 warps x 256; requires m_block == 256 when the momentum is quantised
// PASS 0: a sum-of-squares pass (fewer values live, more resident CTAs); 1: the APPLY pass;
// 2: the LAG pass (APPLY plus the sums of this step's raw update)
// PT: the parameters.  0: binary32; 1, 2: bf16, rounded to nearest or stochastically, eight at a time in packed arithmetic (with
// the element-wise function, whose 64-bit generator is 60 instructions, the momentum-free write pass over the TinyLlama set took
// 4.25 ms stochastically against 2.32, and 3.75 against 2.54 to nearest with a momentum); 3: any 16-bit format, element by element.
// CTAS: resident CTAs per SM asked of the compiler.  Measured on B200: 4 for the sum passes; for the
// writing passes 3 with momentum (CAME, 0.78 ms per Llama-2-7B layer) and 2 without (which the write kernel below has
// taken over wherever it can: see factored_write_kernel).
// ANY = 1: batches of matrices, rows of a multiple of 8.  ANY = 2: rows of any length >= 8 as well.  The flat vectors of
// 8 stay aligned; a vector crosses at most one row end, so its elements take one of two row factors, and column factors
// from three aligned vectors that are shifted (one by one in a lane with a row end).  Only a tensor's last vector may be
// partial.  The squares of the sum
// passes enter binary64 one by one, as in factored_update_kernel, which such tensors took before (but see sums_by_eight).  Write pass with bf16
// gradients: 59 M parameters of odd sizes with a UF8 momentum 1 ms -> 252 us (issue and latency bound, 500 instructions
// per 256 elements), 138 M in batches without momentum 1.55 ms -> 245 us (325 us with the tests of ANY = 2).
template <typename GradT, int PASS, int CTAS, int ANY, int PT>
__global__ void __launch_bounds__(FUPD_THREADS, CTAS)
factored_update_vec_kernel(const FactoredLaunch L)
{
    constexpr bool WRITES = PASS != 0;
    constexpr bool SUMS = PASS != 1;
    __shared__ af8_factored_tensor sT;
    __shared__ double s_acc2[1][FUPD_THREADS / 32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    await_launches();
    const bool has_m = L.m_fmt != AF8_M_NONE;
    const bool m_quant = has_m && L.m_fmt != AF8_M_FP32;
    constexpr bool writes = WRITES;
    int cur_t = -1;
    GradRaw8<GradT> ng;
    float4 np0 = make_float4(0.f, 0.f, 0.f, 0.f), np1 = np0;
    uint2 nm = make_uint2(0u, 0u);
    bool have = false;
    ng.zero();

    // Every CTA takes a contiguous run of chunks, so a thread's position (flat index, row,
    // column) and the tensor's scalars advance incrementally: the division by the column
    // count and the table lookups happen once per tensor, not once per chunk.
    const int64_t per_cta = (L.total_units + gridDim.x - 1) / gridDim.x;
    const int64_t id_begin = (int64_t)blockIdx.x * per_cta;
    const int64_t id_end = min(id_begin + per_cta, L.total_units);
    int64_t next_first = 0, flat = 0, row = 0, col = 0;
    float pre_div = 1.0f, step_mul = 0.0f, fira = 1.0f;
    bool zero_upd = false;
    DivBy D = make_div(1.0f);

    // Sum-of-squares passes: a thread keeps one binary64 partial over all the chunks of a tensor
    // that its CTA processes; at the end of that run the CTA reduces it once and stores the total in
    // the slot of the run's first chunk and zero in the others (the finaliser adds a tensor's slots).
    double run_acc = 0.0;
    int64_t run_first = -1;
    auto flush_sums = [&](int64_t end) {
        double acc = run_acc;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) s_acc2[0][warp] = acc;
        __syncthreads();
        if (tid == 0) {
            double sum = 0.0;
            for (int w = 0; w < FUPD_THREADS / 32; ++w) sum += s_acc2[0][w];
            L.block_sumsq[run_first] = sum;
        }
        for (int64_t i = run_first + 1 + tid; i < end; i += FUPD_THREADS) L.block_sumsq[i] = 0.0;
        __syncthreads();
        run_acc = 0.0;
    };

    for (int64_t id = id_begin; id < id_end; ++id) {
        const int t = cur_t;
        if (cur_t < 0 || id >= next_first) {
            if (SUMS && run_first >= 0) flush_sums(id);
            run_first = id;
            int tn = cur_t;
            if (tn < 0) tn = find_factored_chunk(L.tensors, L.n_tensors, id);
            else while (tn + 1 < L.n_tensors && L.tensors[tn + 1].first_chunk <= id) ++tn;
            __syncthreads();
            if (tid < (int)(sizeof(af8_factored_tensor) / 4))
                reinterpret_cast<uint32_t *>(&sT)[tid] = reinterpret_cast<const uint32_t *>(L.tensors + tn)[tid];
            cur_t = tn;
            __syncthreads();
            next_first = tn + 1 < L.n_tensors ? L.tensors[tn + 1].first_chunk : L.total_units;
            flat = (id - sT.first_chunk) * 2048 + tid * 8;
            row = flat / sT.cols;
            col = flat - row * sT.cols;
            have = false;
            pre_div = 1.0f; step_mul = -sT.alpha; fira = 1.0f; zero_upd = false;
            if (L.dyn != nullptr) {
                const af8_dyn_scalars ds = L.dyn[tn];
                if (L.came && L.mode != AF8_FUPD_SUMSQ_U) pre_div = ds.pre_div;
                if (writes) { step_mul = ds.step; fira = ds.fira; zero_upd = ds.zero != 0.0f; }
            }
            D = make_div(pre_div);
        } else {
            flat += 2048;
            col += 2048;
            if (sT.cols >= 2048) {
                if (col >= sT.cols) { col -= sT.cols; ++row; }
            } else {
                const uint32_t q = (uint32_t)col / (uint32_t)sT.cols;
                row += q;
                col -= (int64_t)q * sT.cols;
            }
        }
        (void)t;
        const int64_t numel = sT.rows * sT.cols;
        const bool ok = flat < numel;                                // numel % 8 == 0: all 8 or none
        const bool partial = ANY == 2 && ok && flat + 8 > numel;          // (the tensor's last elements)
        const int nval = partial ? (int)(numel - flat) : 8;
        // this chunk's streams, loaded one iteration ahead when the chunk is in the same tensor
        GradRaw8<GradT> cg;
        float4 cp0 = make_float4(0.f, 0.f, 0.f, 0.f), cp1 = cp0;
        uint2 cm = make_uint2(0u, 0u);
        const bool pre_m = has_m && L.m_fmt == AF8_M_UF8 && L.mode != AF8_FUPD_SUMSQ_U;
        float *const pbase = static_cast<float *>(sT.param);
        constexpr bool lowp = PT != 0;                               // 16-bit parameters: 8 of them in cp0
        const uint16_t *const hbase = static_cast<const uint16_t *>(sT.param);
        if (have) { cg = ng; cp0 = np0; cp1 = np1; cm = nm; }
        else if (partial) {
            cg.load_part(sT.grad, flat, nval);
            if (writes && lowp) {
                uint32_t x[4] = {0u, 0u, 0u, 0u};
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (j < nval) x[j >> 1] |= (uint32_t)hbase[flat + j] << (16 * (j & 1));
                cp0 = make_float4(__uint_as_float(x[0]), __uint_as_float(x[1]), __uint_as_float(x[2]), __uint_as_float(x[3]));
            } else if (writes) {
                float x[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) x[j] = j < nval ? pbase[flat + j] : 0.0f;
                cp0 = make_float4(x[0], x[1], x[2], x[3]); cp1 = make_float4(x[4], x[5], x[6], x[7]);
            }
            if (pre_m) cm = *reinterpret_cast<const uint2 *>(sT.m_q + flat);     // (codes are stored in whole blocks)
        } else if (ok) {
            cg.load(sT.grad, flat);
            if (writes) {
                if (lowp) cp0 = *reinterpret_cast<const float4 *>(hbase + flat);
                else { cp0 = *reinterpret_cast<const float4 *>(pbase + flat); cp1 = *reinterpret_cast<const float4 *>(pbase + flat + 4); }
            }
            if (pre_m) cm = *reinterpret_cast<const uint2 *>(sT.m_q + flat);
        } else cg.zero();
#if AF8_FUPD_PREFETCH_AHEAD > 0
        if (writes && (!has_m || ANY == 2)) {
            // What is left of the momentum-free write passes beside factored_write_kernel (with the previous step's norm, 16-bit
            // parameters element by element, rows of any length) asks L2 for the chunk a few iterations ahead (same tensor), one request
            // per 128-byte line.  Passes with momentum and the sum passes were measured slower with it (CAME apply 24.9 -> 25.6 ms, sums
            // 0.87 -> 0.94 ms), so they go without; rows of any length, whose loads wait longer, gain with one too (252 -> 238 us,
            // 59 M parameters).
            const int64_t pf = flat + (int64_t)AF8_FUPD_PREFETCH_AHEAD * 2048;
            if (id + AF8_FUPD_PREFETCH_AHEAD < id_end && pf < numel) {
                constexpr int GB = sizeof_grad<GradT>();
                if ((tid & (GB == 2 ? 7 : 3)) == 0) prefetch_l2(static_cast<const char *>(sT.grad) + pf * GB);
                if (writes && (tid & (lowp ? 7 : 3)) == 0) prefetch_l2(static_cast<const char *>(sT.param) + pf * (lowp ? 2 : 4));
                if (pre_m && (tid & 15) == 0) prefetch_l2(sT.m_q + pf);
            }
        }
#endif
        {
            const int64_t nf = flat + 2048;                          // the next chunk of this CTA, if it is in this tensor
            have = id + 1 < id_end && (ANY == 2 ? nf + 8 <= numel : nf < numel);
            if (have) {
                ng.load(sT.grad, nf);
                if (writes) {
                    if (lowp) np0 = *reinterpret_cast<const float4 *>(hbase + nf);
                    else { np0 = *reinterpret_cast<const float4 *>(pbase + nf); np1 = *reinterpret_cast<const float4 *>(pbase + nf + 4); }
                }
                if (pre_m) nm = *reinterpret_cast<const uint2 *>(sT.m_q + nf);
            }
        }
        float mj[8];
        double part = 0.0;
        if (ok) {
            float g[8], ic[8], u[8];
            const LerpW LW = make_lerp(sT.m_w);
            cg.unpack(L.negate_grad, g);
            // ANY: elements j >= wrap belong to the next row; cb0 / cb1: first entries of the two rows' matrices in the
            // column arrays, irow1: index of the next row (clamped: nothing valid follows the last)
            int wrap = 8;
            int64_t cb0 = 0, cb1 = 0, irow1 = row;
            bool whole = true;                                       // the columns come as vectors
            if constexpr (ANY == 2) {
                whole = (sT.cols & 7) == 0;
                if (!whole) {
                    wrap = (int)min((int64_t)8, sT.cols - col);
                    irow1 = min(row + 1, sT.rows - 1);
                }
            }
            if constexpr (ANY != 0) {
                if (sT.batch_rows > 0) {                             // (rows < 2^31)
                    cb0 = (int64_t)((uint32_t)row / (uint32_t)sT.batch_rows) * sT.cols;
                    if (ANY == 2) cb1 = (int64_t)((uint32_t)irow1 / (uint32_t)sT.batch_rows) * sT.cols;
                }
            }
            auto cols8 = [&](const float *v, float (&x)[8]) {
                if (ANY != 2 || whole) { load_f8_ro(v + cb0 + col, x); return; }
                if (wrap == 8) { load_cols8_shifted(v, cb0 + col, x); return; }
                const float *va = v + cb0 + col, *vb = v + cb1 - wrap;
#pragma unroll
                for (int j = 0; j < 8; ++j) x[j] = load_state((j < wrap ? va : vb) + j);
            };
            auto row2 = [&](float a, float b, int j) {               // the row factors of elements j, j + 1
                return ANY == 2 ? make_float2(j < wrap ? a : b, j + 1 < wrap ? a : b) : bc2(a);
            };
            cols8(sT.inv_col, ic);
            const float ir = load_state(sT.inv_row + row), irb = ANY == 2 ? load_state(sT.inv_row + irow1) : 0.0f;
            // pairs of elements in packed binary32 arithmetic (bit-identical to the element-wise form)
            if (L.came) {
                if (L.mode == AF8_FUPD_SUMSQ_U) {
#pragma unroll
                    for (int j = 0; j < 8; j += 2) {
                        const float2 uj = __fmul2_rn(__fmul2_rn(make_float2(g[j], g[j + 1]), row2(ir, irb, j)), make_float2(ic[j], ic[j + 1]));
                        u[j] = uj.x; u[j + 1] = uj.y;
                    }
                } else {
                    float mo[8], icc[8];
                    if (partial && !m_quant) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) mo[j] = j < nval ? sT.m_f32[flat + j] : 0.0f;
                    } else m_old8(sT, L.m_fmt, 256, flat, mo, pre_m, cm);
                    cols8(sT.inv_col_conf, icc);
                    const float irc = load_state(sT.inv_row_conf + row), ircb = ANY == 2 ? load_state(sT.inv_row_conf + irow1) : 0.0f;
#pragma unroll
                    for (int j = 0; j < 8; j += 2) {
                        const float2 ut = div_by2(__fmul2_rn(__fmul2_rn(make_float2(g[j], g[j + 1]), row2(ir, irb, j)), make_float2(ic[j], ic[j + 1])), D);
                        const float2 mm = lerp_w2(make_float2(mo[j], mo[j + 1]), ut, LW);
                        const float2 uj = __fmul2_rn(__fmul2_rn(mm, row2(irc, ircb, j)), make_float2(icc[j], icc[j + 1]));
                        mj[j] = mm.x; mj[j + 1] = mm.y; u[j] = uj.x; u[j + 1] = uj.y;
                    }
                }
            } else if (has_m) {
                float mo[8];
                if (partial && !m_quant) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) mo[j] = j < nval ? sT.m_f32[flat + j] : 0.0f;
                    } else m_old8(sT, L.m_fmt, 256, flat, mo, pre_m, cm);
#pragma unroll
                for (int j = 0; j < 8; j += 2) {
                    const float2 mm = lerp_w2(make_float2(mo[j], mo[j + 1]), make_float2(g[j], g[j + 1]), LW);
                    const float2 uj = __fmul2_rn(__fmul2_rn(mm, row2(ir, irb, j)), make_float2(ic[j], ic[j + 1]));
                    mj[j] = mm.x; mj[j + 1] = mm.y; u[j] = uj.x; u[j + 1] = uj.y;
                }
            } else {
#pragma unroll
                for (int j = 0; j < 8; j += 2) {
                    const float2 uj = __fmul2_rn(__fmul2_rn(make_float2(g[j], g[j + 1]), row2(ir, irb, j)), make_float2(ic[j], ic[j + 1]));
                    u[j] = uj.x; u[j + 1] = uj.y;
                }
            }
            if (partial) {
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (j >= nval) { u[j] = 0.0f; mj[j] = 0.0f; }
            }
            if (SUMS && !sums_by_eight<ANY>(sT)) {
#pragma unroll
                for (int j = 0; j < 8; ++j) part += (double)__fmul_rn(u[j], u[j]);
            } else if (SUMS) {
                // The thread's eight squares are added in binary32 (two packed chains) and enter the binary64
                // partial as one number: the sum only feeds a norm (clip divisor, limiter), where a relative
                // 1e-7 is far below what the parameters can show, and it saves seven conversions and seven
                // binary64 additions per chunk.
                float2 a2 = __fmul2_rn(make_float2(u[0], u[1]), make_float2(u[0], u[1]));
#pragma unroll
                for (int j = 2; j < 8; j += 2) a2 = __ffma2_rn(make_float2(u[j], u[j + 1]), make_float2(u[j], u[j + 1]), a2);
                part += (double)__fadd_rn(a2.x, a2.y);
            }
            if (writes) {
                if (lowp) {
                    // bf16 / fp16 parameters: rounded after the decay and after the update, or once,
                    // stochastically (optimizer.py:873-881, 2033-2039)
                    const uint32_t w[4] = {__float_as_uint(cp0.x), __float_as_uint(cp0.y), __float_as_uint(cp0.z), __float_as_uint(cp0.w)};
                    uint32_t o[4];
                    if constexpr (PT == 1 || PT == 2) {
                        const float2 decay2 = bc2(sT.decay), step2 = bc2(step_mul), fira2 = bc2(fira);
                        float2 x[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            x[j] = __fmul2_rn(make_float2(__uint_as_float(w[j] << 16), __uint_as_float(w[j] & 0xffff0000u)), decay2);
                            if (PT == 1) {
                                const uint32_t pk = bf16x2_rn(x[j].x, x[j].y);
                                x[j] = make_float2(__uint_as_float(pk << 16), __uint_as_float(pk & 0xffff0000u));
                            }
                            float2 uu = __fmul2_rn(make_float2(u[2 * j], u[2 * j + 1]), fira2);
                            if (zero_upd) uu = make_float2(0.0f, 0.0f);
                            x[j] = __ffma2_rn(step2, uu, x[j]);
                        }
                        fast_round8<PT == 2, 0>(x, sT.sr_base, flat, 0, PT == 2 ? sr_counter(sT.sr_base, flat, 8) : SrCounter{}, o);
                    } else
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const uint32_t h = (j & 1) ? (w[j >> 1] >> 16) : (w[j >> 1] & 0xffffu);
                        const float pv = L.param_dtype == AF8_BF16 ? bf16_bits_to_f32(h) : f16_bits_to_f32(h);
                        const float uu = zero_upd ? 0.0f : __fmul_rn(u[j], fira);
                        const uint32_t r = param_step_bits(pv, sT.decay, step_mul, uu, L.param_dtype, L.sr, sT.sr_base, flat + j);
                        if (j & 1) o[j >> 1] |= r << 16; else o[j >> 1] = r;
                    }
                    if (partial) {
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            if (j < nval) const_cast<uint16_t *>(hbase)[flat + j] = (uint16_t)(o[j >> 1] >> (16 * (j & 1)));
                    } else
                    *reinterpret_cast<uint4 *>(const_cast<uint16_t *>(hbase) + flat) = make_uint4(o[0], o[1], o[2], o[3]);
                } else {
                    float *pp = pbase + flat;
                    float p[8] = {cp0.x, cp0.y, cp0.z, cp0.w, cp1.x, cp1.y, cp1.z, cp1.w};
                    const float2 decay2 = bc2(sT.decay), step2 = bc2(step_mul), fira2 = bc2(fira);
#pragma unroll
                    for (int j = 0; j < 8; j += 2) {
                        float2 pj = __fmul2_rn(make_float2(p[j], p[j + 1]), decay2);
                        if (!zero_upd) pj = __ffma2_rn(step2, __fmul2_rn(make_float2(u[j], u[j + 1]), fira2), pj);
                        p[j] = pj.x; p[j + 1] = pj.y;
                    }
                    if (partial) {
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            if (j < nval) {
                                pp[j] = p[j];
                                if (sT.param_copy != nullptr) static_cast<uint16_t *>(sT.param_copy)[flat + j] = (uint16_t)f32_to_bf16_rn_bits(p[j]);
                            }
                    } else {
                    *reinterpret_cast<float4 *>(pp) = make_float4(p[0], p[1], p[2], p[3]);
                    *reinterpret_cast<float4 *>(pp + 4) = make_float4(p[4], p[5], p[6], p[7]);
                    if (sT.param_copy != nullptr)                                    // bf16 compute copy
                        *reinterpret_cast<uint4 *>(static_cast<uint16_t *>(sT.param_copy) + flat) =
                            make_uint4(bf16x2_rn(p[0], p[1]), bf16x2_rn(p[2], p[3]), bf16x2_rn(p[4], p[5]), bf16x2_rn(p[6], p[7]));
                    }
                }
                if (partial && has_m && !m_quant) {
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (j < nval) sT.m_f32[flat + j] = mj[j];
                } else if (has_m && !m_quant) {
                    *reinterpret_cast<float4 *>(sT.m_f32 + flat) = make_float4(mj[0], mj[1], mj[2], mj[3]);
                    *reinterpret_cast<float4 *>(sT.m_f32 + flat + 4) = make_float4(mj[4], mj[5], mj[6], mj[7]);
                }
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) mj[j] = 0.0f;
        }
        if (SUMS) {
            run_acc += part;                 // reduced over the CTA once per tensor (flush_sums)
            if (!writes) continue;
        }
        if (m_quant) {
            // one warp = one momentum block of 256 (the block exists iff its first element does)
            const int64_t w0 = (id - sT.first_chunk) * 2048 + warp * 256;
            bool odd;
            const float am = m_absmax256(mj, odd);
            if (w0 < numel) {
                if (L.m_fmt == AF8_M_UF8) {
                    const uint2 codes = uf8_codes8(mj, am, odd);
                    if (ANY != 0 || ok) *reinterpret_cast<uint2 *>(sT.m_q + flat) = codes;
                } else if (L.m_fmt == AF8_M_D8) {
                    uint32_t o0 = 0, o1 = 0;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        o0 |= m_encode(mj[j], am, L.m_fmt) << (8 * j);
                        o1 |= m_encode(mj[j + 4], am, L.m_fmt) << (8 * j);
                    }
                    if (ANY != 0 || ok) *reinterpret_cast<uint2 *>(sT.m_q + flat) = make_uint2(o0, o1);
                } else {
                    uint32_t o = 0;
#pragma unroll
                    for (int j = 0; j < 8; j += 2)
                        o |= ((m_encode(mj[j], am, L.m_fmt) << 4) | m_encode(mj[j + 1], am, L.m_fmt)) << (4 * j);
                    if (ANY != 0 || ok) *reinterpret_cast<uint32_t *>(sT.m_q + (flat >> 1)) = o;
                }
                if (lane == 0) sT.m_scale[w0 / 256] = am;
            }
        }
    }
    if (SUMS && run_first >= 0) flush_sums(id_end);
}

// ---------------------------------------------------------------------------
// The APPLY pass without a momentum over rows of whole vectors of 8, and batches of such matrices (ANY): u = g * inv_row * inv_col,
// fp32 or bf16 parameters (PT as above).
//
// It moves 10 bytes per parameter (bf16 gradients, fp32 parameters) and computes next to nothing, so the order of its memory
// accesses decides: write_units.cuh.  Six CTAs per SM, 216 KB requested; two stages, or seven and eight CTAs with fewer registers, are
// within 3 %.  Against contiguous runs of units per CTA, loads into registers one unit ahead and requests to L2 three ahead: 134 M
// parameters in one matrix 218 -> 204 us (6.6 TB/s; a copy of the same streams reaches 6.85), 176 M in 28 matrices of 2048 columns
// 295 -> 276.
// ---------------------------------------------------------------------------
struct FactoredUnit : WriteUnit {
    void *copy;
    const float *inv_row, *inv_col;
    int64_t batch_rows;
    uint64_t sr_base;
    float decay, step, fira, zero;
};
struct FactoredUnits {
    const FactoredLaunch &L;
    __device__ __forceinline__ int count() const { return L.n_tensors; }
    __device__ __forceinline__ int64_t first(int t) const { return L.tensors[t].first_chunk; }
    __device__ __forceinline__ int64_t load(int t, FactoredUnit &U) const
    {
        const af8_factored_tensor T = L.tensors[t];
        U.cols = T.cols; U.param = T.param; U.grad = T.grad; U.copy = T.param_copy; U.inv_row = T.inv_row; U.inv_col = T.inv_col;
        U.batch_rows = T.batch_rows; U.sr_base = T.sr_base; U.decay = T.decay; U.step = -T.alpha; U.fira = 1.0f; U.zero = 0.0f;
        if (L.dyn != nullptr) {
            const af8_dyn_scalars ds = L.dyn[t];
            U.step = ds.step; U.fira = ds.fira; U.zero = ds.zero;
        }
        return T.rows * T.cols;
    }
};

template <typename GradT, int PT, bool ANY>
__global__ void __launch_bounds__(WRITE_THREADS + 32, sizeof_grad<GradT>() == 2 ? 6 : 4)
factored_write_kernel(const FactoredLaunch L)
{
    constexpr int GB = sizeof_grad<GradT>(), PB = PT == 0 ? 4 : 2, P_OFF = WRITE_UNIT * GB;
    extern __shared__ __align__(128) unsigned char fw_smem[];
    __shared__ __align__(16) WriteShared<FactoredUnit> sh;
    const int tid = threadIdx.x;
    const float sgn = L.negate_grad ? -1.0f : 1.0f;                  // ((-g) * r == g * (-r) bit for bit)
    write_units<GB, PB>(FactoredUnits{L}, sh, fw_smem, [&](const FactoredUnit &U, const unsigned char *st, auto release) {
        const int64_t base = U.base;
        const int count = warp_uniform(U.count);
        float2 x[2][4], u[2][4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int o = q * 512 + tid * 4;
            float2 &xa = x[q >> 1][2 * (q & 1)], &xb = x[q >> 1][2 * (q & 1) + 1], &ua = u[q >> 1][2 * (q & 1)], &ub = u[q >> 1][2 * (q & 1) + 1];
            xa = xb = ua = ub = make_float2(0.0f, 0.0f);
            if (o >= count) continue;
            int64_t row, col, cb = 0;
            write_position(U, o, row, col);
            if (ANY && U.batch_rows > 0) cb = (int64_t)((uint32_t)row / (uint32_t)U.batch_rows) * U.cols;        // (rows < 2^31)
            const float2 ir2 = bc2(__fmul_rn(load_state(U.inv_row + row), sgn));
            const float4 ic = load_state(reinterpret_cast<const float4 *>(U.inv_col + cb + col));
            float2 ga, gb;
            if (GB == 4) {
                const float4 g = *reinterpret_cast<const float4 *>(st + o * 4);
                ga = make_float2(g.x, g.y); gb = make_float2(g.z, g.w);
            } else unpack_bf16x4(*reinterpret_cast<const uint2 *>(st + o * 2), ga, gb);
            if (PB == 4) {
                const float4 p = *reinterpret_cast<const float4 *>(st + P_OFF + o * 4);
                xa = make_float2(p.x, p.y); xb = make_float2(p.z, p.w);
            } else unpack_bf16x4(*reinterpret_cast<const uint2 *>(st + P_OFF + o * 2), xa, xb);
            ua = __fmul2_rn(__fmul2_rn(ga, ir2), make_float2(ic.x, ic.y));
            ub = __fmul2_rn(__fmul2_rn(gb, ir2), make_float2(ic.z, ic.w));
        }
        const float2 decay2 = bc2(U.decay), step2 = bc2(U.step), fira2 = bc2(U.fira);
        const bool zero_upd = U.zero != 0.0f;
        void *const param = U.param;
        void *const copy = PT == 0 ? U.copy : nullptr;
        const uint64_t sr_base = PT == 2 ? U.sr_base : 0;
        release();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float2 (&y)[4] = x[h];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                y[j] = __fmul2_rn(y[j], decay2);
                if (PT == 1) {
                    const uint32_t pk = bf16x2_rn(y[j].x, y[j].y);
                    y[j] = make_float2(__uint_as_float(pk << 16), __uint_as_float(pk & 0xffff0000u));
                }
                if (PT == 0) {
                    if (!zero_upd) y[j] = __ffma2_rn(step2, __fmul2_rn(u[h][j], fira2), y[j]);
                } else {
                    const float2 uu = zero_upd ? make_float2(0.0f, 0.0f) : __fmul2_rn(u[h][j], fira2);
                    y[j] = __ffma2_rn(step2, uu, y[j]);
                }
            }
            const int oa = h * 1024 + tid * 4;
            uint32_t w[4];
            if (PT != 0) fast_round8<PT == 2, 508>(y, sr_base, base, oa, PT == 2 ? sr_counter(sr_base, base, WRITE_UNIT) : SrCounter{}, w);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int o = oa + 512 * k;
                if (o >= count) continue;
                if (PT == 0) {
                    *reinterpret_cast<float4 *>(static_cast<float *>(param) + base + o) = make_float4(y[2 * k].x, y[2 * k].y, y[2 * k + 1].x, y[2 * k + 1].y);
                    if (copy != nullptr)                    // bf16 compute copy
                        *reinterpret_cast<uint2 *>(static_cast<uint16_t *>(copy) + base + o) = make_uint2(bf16x2_rn(y[2 * k].x, y[2 * k].y), bf16x2_rn(y[2 * k + 1].x, y[2 * k + 1].y));
                } else {
                    *reinterpret_cast<uint2 *>(static_cast<uint16_t *>(param) + base + o) = make_uint2(w[2 * k], w[2 * k + 1]);
                }
            }
        }
    });
}

// ---------------------------------------------------------------------------
// The APPLY pass with a UF8 momentum (CAME, Adafactor with beta1) in flat order, inputs through per-warp rings of bulk
// asynchronous copies, for rows of any length >= 8, batches of matrices, and binary32 or bf16 parameters.
//
// A warp owns one momentum block per chunk (256 consecutive elements: gradient, parameter and momentum codes are three
// contiguous runs); lanes 0 to 2 request one run each, FRING_STAGES - 1 chunks ahead, into the warp's own ring; completion is an
// mbarrier per stage.  Warps do not synchronise with one another except when the CTA moves to its next tensor.  Copies never
// cross a tensor, and the (at most one) partial chunk at a tensor's end is loaded directly.
//
// What bounds it is instruction issue: the column factors of 8 elements come from memory (L1), at any alignment where rows are no
// multiple of 8 (ANY), and the row may end among them.  A warp without a row end among its 256 elements takes the form with one row
// factor.  Two resident CTAs without spills for ANY, three with 90 bytes of them otherwise: 181 and 215 us below.
// Write pass before (the kernel above for ANY and bf16, one lane's requests else) -> now: 59 M parameters in rows of 1001 and 2731
// elements 229 -> 180 us, 397 M in rows of 1999 with CAME 1640 -> 1446, 339 M in rows of 2000 with CAME 856 -> 826, 1.1 G bf16
// parameters 2.54 -> 2.35 ms.
// PT: the parameters, as above (0: binary32; 1, 2: bf16 to nearest, stochastically).
// ---------------------------------------------------------------------------
#ifndef AF8_FRING_STAGES
#define AF8_FRING_STAGES 4
#endif
constexpr int FRING_STAGES = AF8_FRING_STAGES;
constexpr int DEVERR_FRING_TIMEOUT = 3;
template <typename GradT, int PT = 0> __host__ __device__ constexpr int fring_stage_bytes() { return 256 * sizeof_grad<GradT>() + (PT == 0 ? 1024 : 512) + 256; }
template <typename GradT, int PT = 0> constexpr size_t fring_smem_bytes() { return (size_t)(FUPD_THREADS / 32) * FRING_STAGES * fring_stage_bytes<GradT, PT>(); }

// column factors of elements col .. col + 7 of a row, the elements from `left` (1 .. 7) on being the first of the next row
__device__ __forceinline__ void flat_cols_wrap(const float *v, int64_t cb0, int64_t cb1, int64_t col, int left, float (&x)[8])
{
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = load_state(j < left ? v + cb0 + col + j : v + cb1 + j - left);
}

// New momentum and update of 8 elements.  ir, irc: row factors of the elements before `left`, irb, ircb of the others (COMMON: no
// others, and a momentum weight below 1/2).
template <bool CAME, bool COMMON>
__device__ __forceinline__ void flat_update8(const float (&g)[8], const float2 (&mo)[4], const float (&ic)[8], const float (&icc)[8], float ir, float irb,
                                             float irc, float ircb, int left, const DivBy &D, const LerpW &LW, float (&mj)[8], float (&u)[8])
{
    const auto row2 = [&](float a, float b, int j) { return COMMON ? bc2(a) : make_float2(j < left ? a : b, j + 1 < left ? a : b); };
    const float2 ww2 = bc2(LW.ww);
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
        const float2 gj = make_float2(g[j], g[j + 1]), c2 = make_float2(ic[j], ic[j + 1]), m = mo[j >> 1];
        float2 e = gj;
        if (CAME) e = div_by2(__fmul2_rn(__fmul2_rn(gj, row2(ir, irb, j)), c2), D);
        const float2 mm = __ffma2_rn(ww2, sub2(e, m), (COMMON || LW.small) ? m : e);
        const float2 uj = CAME ? __fmul2_rn(__fmul2_rn(mm, row2(irc, ircb, j)), make_float2(icc[j], icc[j + 1]))
                               : __fmul2_rn(__fmul2_rn(mm, row2(ir, irb, j)), c2);
        mj[j] = mm.x; mj[j + 1] = mm.y; u[j] = uj.x; u[j + 1] = uj.y;
    }
}

// what a CTA keeps of its current tensor (in shared memory: in registers it costs spills)
struct FlatTensor {
    int64_t numel, next_first, full_end, adv_rows, adv_cols;     // chunk ids: the next tensor's first, the first that is not whole; 2048 elements in rows and columns
    DivBy D;
    LerpW LW;
    float step_mul, fira;
    int32_t zero_upd, whole;                                     // whole: rows are whole vectors
};

#ifndef FLAT_ANY_CTAS
#define FLAT_ANY_CTAS 2
#endif
template <typename GradT, int PT, bool ANY>
__global__ void __launch_bounds__(FUPD_THREADS, sizeof_grad<GradT>() == 2 ? (ANY ? FLAT_ANY_CTAS : 3) : 2)
factored_apply_flat_kernel(const FactoredLaunch L)
{
    constexpr int GB = sizeof_grad<GradT>(), PB = PT == 0 ? 4 : 2, NS = FRING_STAGES;
    constexpr int P_OFF = 256 * GB, M_OFF = P_OFF + 256 * PB, STAGE = fring_stage_bytes<GradT, PT>();
    extern __shared__ __align__(128) unsigned char fr_smem[];
    __shared__ af8_factored_tensor sT;
    __shared__ FlatTensor sF;
    __shared__ __align__(8) uint64_t s_full[FUPD_THREADS / 32][NS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    unsigned char *const ring = fr_smem + (size_t)warp * NS * STAGE;
    if (lane == 0) {
        for (int k = 0; k < NS; ++k) mbar_init(&s_full[warp][k], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    await_launches();

    const int64_t per_cta = (L.total_units + gridDim.x - 1) / gridDim.x;
    const int64_t id_begin = (int64_t)blockIdx.x * per_cta;
    const int64_t id_end = min(id_begin + per_cta, L.total_units);
    int cur_t = -1;
    int64_t flat = 0, row = 0, col = 0;
    uint32_t cons = 0;            // chunks this warp has taken from its ring
    int inflight = 0;             // chunks from the current one on whose copies are issued
    float nsc = 0.0f;             // absmax of this warp's block of the next chunk
    bool have_sc = false;

    for (int64_t id = id_begin; id < id_end; ++id) {
        if (cur_t < 0 || id >= sF.next_first) {
            int tn = cur_t;
            if (tn < 0) tn = find_factored_chunk(L.tensors, L.n_tensors, id);
            else while (tn + 1 < L.n_tensors && L.tensors[tn + 1].first_chunk <= id) ++tn;
            __syncthreads();
            if (tid < (int)(sizeof(af8_factored_tensor) / 4))
                reinterpret_cast<uint32_t *>(&sT)[tid] = reinterpret_cast<const uint32_t *>(L.tensors + tn)[tid];
            cur_t = tn;
            __syncthreads();
            const int64_t C = sT.cols;
            flat = (id - sT.first_chunk) * 2048 + tid * 8;
            row = flat / C;
            col = flat - row * C;
            if (tid == 0) {
                FlatTensor F;
                F.numel = sT.rows * C;
                F.next_first = tn + 1 < L.n_tensors ? L.tensors[tn + 1].first_chunk : L.total_units;
                F.full_end = min(id_end, sT.first_chunk + F.numel / 2048);
                F.adv_rows = 2048 / C;
                F.adv_cols = 2048 - F.adv_rows * C;
                F.whole = !ANY || (C & 7) == 0;
                float pre_div = 1.0f;
                F.step_mul = -sT.alpha; F.fira = 1.0f; F.zero_upd = 0;
                if (L.dyn != nullptr) {
                    const af8_dyn_scalars ds = L.dyn[tn];
                    if (L.came) pre_div = ds.pre_div;
                    F.step_mul = ds.step; F.fira = ds.fira; F.zero_upd = ds.zero != 0.0f;
                }
                F.D = make_div(pre_div);
                F.LW = make_lerp(sT.m_w);
                sF = F;
            }
            __syncthreads();
            inflight = 0;                                            // (copies never cross a tensor)
            have_sc = false;
        } else {
            flat += 2048;
            row += sF.adv_rows;
            col += sF.adv_cols;
            if (col >= sT.cols) { col -= sT.cols; ++row; }
        }
        const int64_t numel = sF.numel;
        const bool full = id < sF.full_end;
        const bool ok = flat < numel;
        const int nval = ANY ? (int)min((int64_t)8, numel - flat) : 8;       // (fewer only in a tensor's last vector)
        const int64_t block = (id - sT.first_chunk) * 8 + warp;              // this warp's momentum block

        // ---- request the chunks id .. id + NS - 1 that are whole chunks of this tensor ----
        int want = (int)min((int64_t)NS, sF.full_end - id);
        if (want < 0) want = 0;
        if (lane < 3 && inflight < want) {
            fence_proxy_async();                                     // this warp's reads of the slots came first
            const unsigned char *const src = lane == 0 ? static_cast<const unsigned char *>(sT.param) : lane == 1 ? static_cast<const unsigned char *>(sT.grad) : sT.m_q;
            const int size = lane == 0 ? 256 * PB : lane == 1 ? 256 * GB : 256, to = lane == 0 ? P_OFF : lane == 1 ? 0 : M_OFF;
            for (int k = inflight; k < want; ++k) {
                const int sl = (int)((cons + (uint32_t)k) % NS);
                if (lane == 0) mbar_expect_tx(&s_full[warp][sl], (uint32_t)STAGE);
                bulk_g2s(ring + sl * STAGE + to, src + (block + 8 * k) * size, (uint32_t)size, &s_full[warp][sl]);
            }
        }
        inflight = want > 0 ? want - 1 : 0;                          // as seen from the next chunk

        const int64_t w0 = block * 256;                              // (the block exists iff its first element does)
        float sc = nsc;
        if (!have_sc) sc = w0 < numel ? load_state(sT.m_scale + block) : 0.0f;
        have_sc = id + 1 < id_end && w0 + 2048 < numel;
        if (have_sc) nsc = load_state(sT.m_scale + block + 8);

        GradRaw8<GradT> cg;
        uint4 pa = make_uint4(0u, 0u, 0u, 0u), pb = pa;              // 8 parameters (bf16: in pa)
        uint2 cm = make_uint2(0x80808080u, 0x80808080u);
        float *const pbase = static_cast<float *>(sT.param);
        uint16_t *const hbase = static_cast<uint16_t *>(sT.param);
        if (full) {
            const int sl = (int)(cons % NS);
            const bool landed = mbar_wait_bounded(&s_full[warp][sl], (cons / NS) & 1u);
            if (!__all_sync(0xffffffffu, landed)) {                  // (uniform over the warp)
                atomicExch(&g_device_error, DEVERR_FRING_TIMEOUT);
                return;                                              // the other warps go on: nothing waits for this one
            }
            const unsigned char *st = ring + sl * STAGE;
            cg.from_shared(st + lane * (8 * GB));
            pa = *reinterpret_cast<const uint4 *>(st + P_OFF + lane * (8 * PB));
            if (PT == 0) pb = *reinterpret_cast<const uint4 *>(st + P_OFF + lane * 32 + 16);
            cm = *reinterpret_cast<const uint2 *>(st + M_OFF + lane * 8);
            ++cons;
            __syncwarp();                                            // the slot may be refilled from the next iteration on
        } else if (ok && nval == 8) {
            cg.load(sT.grad, flat);
            if (PT == 0) {
                pa = *reinterpret_cast<const uint4 *>(pbase + flat);
                pb = *reinterpret_cast<const uint4 *>(pbase + flat + 4);
            } else pa = *reinterpret_cast<const uint4 *>(hbase + flat);
            cm = *reinterpret_cast<const uint2 *>(sT.m_q + flat);
        } else if (ok) {                                             // (codes are stored in whole blocks)
            cg.load_part(sT.grad, flat, nval);
            uint32_t x[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) x[j] = j < nval ? (PT == 0 ? __float_as_uint(pbase[flat + j]) : (uint32_t)hbase[flat + j]) : 0u;
            if (PT == 0) { pa = make_uint4(x[0], x[1], x[2], x[3]); pb = make_uint4(x[4], x[5], x[6], x[7]); }
            else pa = make_uint4(x[0] | (x[1] << 16), x[2] | (x[3] << 16), x[4] | (x[5] << 16), x[6] | (x[7] << 16));
            cm = *reinterpret_cast<const uint2 *>(sT.m_q + flat);
        } else cg.zero();

        float mj[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) mj[j] = 0.0f;
        const bool whole = !ANY || sF.whole;
        const int left = whole ? 8 : (int)min((int64_t)8, sT.cols - col);     // elements before the row's end
        const bool common = sF.LW.small && !(ANY && __any_sync(0xffffffffu, left < 8));
        if (ok) {
            float g[8], ic[8], icc[8], u[8];
            float2 mo[4];
            cg.unpack(L.negate_grad, g);
            uf8_decode8(cm, __fmul_rn(sc, 0.0078125f), mo);          // fl(scale / 128), scale >= 1e-12
            int64_t cb0 = 0, cb1 = 0, next = row;
            if (ANY) {
                next = min(row + 1, sT.rows - 1);                    // (nothing valid follows the last row)
                if (sT.batch_rows > 0) {                             // (rows < 2^31)
                    cb0 = (int64_t)((uint32_t)row / (uint32_t)sT.batch_rows) * sT.cols;
                    if (left < 8) cb1 = (int64_t)((uint32_t)next / (uint32_t)sT.batch_rows) * sT.cols;
                }
            }
            const auto cols8 = [&](const float *v, float (&x)[8]) {
                if (whole) load_f8_ro(v + cb0 + col, x);
                else if (left == 8) load_cols8_shifted(v, cb0 + col, x);
                else flat_cols_wrap(v, cb0, cb1, col, left, x);
            };
            cols8(sT.inv_col, ic);
            const float ir = load_state(sT.inv_row + row);
            if (L.came) {
                cols8(sT.inv_col_conf, icc);
                const float irc = load_state(sT.inv_row_conf + row);
                if (common) flat_update8<true, true>(g, mo, ic, icc, ir, ir, irc, irc, 8, sF.D, sF.LW, mj, u);
                else flat_update8<true, false>(g, mo, ic, icc, ir, load_state(sT.inv_row + next), irc, load_state(sT.inv_row_conf + next), left, sF.D, sF.LW, mj, u);
            } else {
                if (common) flat_update8<false, true>(g, mo, ic, ic, ir, ir, ir, ir, 8, sF.D, sF.LW, mj, u);
                else flat_update8<false, false>(g, mo, ic, ic, ir, load_state(sT.inv_row + next), ir, ir, left, sF.D, sF.LW, mj, u);
            }
            if (ANY && nval < 8) {
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (j >= nval) { u[j] = 0.0f; mj[j] = 0.0f; }
            }
            const float2 decay2 = bc2(sT.decay), step2 = bc2(sF.step_mul), fira2 = bc2(sF.fira);
            const bool zero_upd = sF.zero_upd;
            if (PT == 0) {
                float p[8] = {__uint_as_float(pa.x), __uint_as_float(pa.y), __uint_as_float(pa.z), __uint_as_float(pa.w),
                              __uint_as_float(pb.x), __uint_as_float(pb.y), __uint_as_float(pb.z), __uint_as_float(pb.w)};
#pragma unroll
                for (int j = 0; j < 8; j += 2) {
                    float2 pj = __fmul2_rn(make_float2(p[j], p[j + 1]), decay2);
                    if (!zero_upd) pj = __ffma2_rn(step2, __fmul2_rn(make_float2(u[j], u[j + 1]), fira2), pj);
                    p[j] = pj.x; p[j + 1] = pj.y;
                }
                uint16_t *const copy = static_cast<uint16_t *>(sT.param_copy);        // bf16 compute copy
                if (!ANY || nval == 8) {
                    float *pp = pbase + flat;
                    *reinterpret_cast<float4 *>(pp) = make_float4(p[0], p[1], p[2], p[3]);
                    *reinterpret_cast<float4 *>(pp + 4) = make_float4(p[4], p[5], p[6], p[7]);
                    if (copy != nullptr)
                        *reinterpret_cast<uint4 *>(copy + flat) =
                            make_uint4(bf16x2_rn(p[0], p[1]), bf16x2_rn(p[2], p[3]), bf16x2_rn(p[4], p[5]), bf16x2_rn(p[6], p[7]));
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (j < nval) {
                            pbase[flat + j] = p[j];
                            if (copy != nullptr) copy[flat + j] = (uint16_t)f32_to_bf16_rn_bits(p[j]);
                        }
                }
            } else {
                // rounded to bf16 after the decay and after the update, or once, stochastically (optimizer.py:873-881, 2033-2039)
                const uint32_t w[4] = {pa.x, pa.y, pa.z, pa.w};
                uint32_t o[4];
                float2 x[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    x[j] = __fmul2_rn(make_float2(__uint_as_float(w[j] << 16), __uint_as_float(w[j] & 0xffff0000u)), decay2);
                    if (PT == 1) {
                        const uint32_t pk = bf16x2_rn(x[j].x, x[j].y);
                        x[j] = make_float2(__uint_as_float(pk << 16), __uint_as_float(pk & 0xffff0000u));
                    }
                    float2 uu = __fmul2_rn(make_float2(u[2 * j], u[2 * j + 1]), fira2);
                    if (zero_upd) uu = make_float2(0.0f, 0.0f);
                    x[j] = __ffma2_rn(step2, uu, x[j]);
                }
                fast_round8<PT == 2, 0>(x, sT.sr_base, flat, 0, PT == 2 ? sr_counter(sT.sr_base, flat, 8) : SrCounter{}, o);
                if (!ANY || nval == 8) *reinterpret_cast<uint4 *>(hbase + flat) = make_uint4(o[0], o[1], o[2], o[3]);
                else {
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (j < nval) hbase[flat + j] = (uint16_t)(o[j >> 1] >> (16 * (j & 1)));
                }
            }
        }
        bool odd;
        const float am = m_absmax256(mj, odd);
        if (w0 < numel) {
            const uint2 codes = uf8_codes8(mj, am, odd);
            if (ANY || ok) *reinterpret_cast<uint2 *>(sT.m_q + flat) = codes;        // (ANY: what lies beyond the end is coded as zero)
            if (lane == 0) sT.m_scale[block] = am;
        }
    }
}

// ---------------------------------------------------------------------------
// The same pass over fp32 parameters in tile order, for tables whose tensors all have cols % 256 == 0: a CTA takes a
// 512 x 256 statistic tile, warp w its rows r0 + w, r0 + w + 8, ...; a row slice of 256 columns is 256
// consecutive elements that start on a multiple of 256, i.e. exactly one momentum block, so the warp still owns
// its block's absmax.  What changes is that a lane works on the same 8 columns for the whole tile and keeps
// their inverse column factors (and CAME's confidence factors) in registers instead of loading 32 or 64 bytes
// of them for every 8 elements.  Ring, arithmetic and stores as above; the copies of
// a warp run FRING_STAGES - 1 rows ahead inside a tile.
// ---------------------------------------------------------------------------
template <typename GradT, int CTAS>
__global__ void __launch_bounds__(FUPD_THREADS, CTAS)
factored_apply_tile_kernel(const FactoredLaunch L)
{
    constexpr int GB = sizeof_grad<GradT>();
    constexpr int P_OFF = 256 * GB, M_OFF = P_OFF + 1024, STAGE = fring_stage_bytes<GradT>(), NS = FRING_STAGES;
    extern __shared__ __align__(128) unsigned char fr_smem[];
    __shared__ af8_factored_tensor sT;
    __shared__ __align__(8) uint64_t s_full[FUPD_THREADS / 32][NS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    unsigned char *const ring = fr_smem + (size_t)warp * NS * STAGE;
    if (lane == 0) {
        for (int k = 0; k < NS; ++k) mbar_init(&s_full[warp][k], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    await_launches();

    int cur_t = -1;
    float pre_div = 1.0f, step_mul = 0.0f, fira = 1.0f;
    bool zero_upd = false;
    DivBy D = make_div(1.0f);
    uint32_t cons = 0;            // row slices this warp has taken from its ring

    for (int64_t id = blockIdx.x; id < L.total_units; id += gridDim.x) {
        int t = cur_t;
        const int64_t tile = id >> L.split;
        if (t < 0) t = find_factored_tile(L.tensors, L.n_tensors, tile);
        else while (t + 1 < L.n_tensors && L.tensors[t + 1].first_tile <= tile) ++t;
        if (t != cur_t) {
            __syncthreads();                                         // every warp has left the previous tensor
            if (tid < (int)(sizeof(af8_factored_tensor) / 4))
                reinterpret_cast<uint32_t *>(&sT)[tid] = reinterpret_cast<const uint32_t *>(L.tensors + t)[tid];
            cur_t = t;
            __syncthreads();
            pre_div = 1.0f; step_mul = -sT.alpha; fira = 1.0f; zero_upd = false;
            if (L.dyn != nullptr) {
                const af8_dyn_scalars ds = L.dyn[t];
                if (L.came) pre_div = ds.pre_div;
                step_mul = ds.step; fira = ds.fira; zero_upd = ds.zero != 0.0f;
            }
            D = make_div(pre_div);
        }
        const int64_t C = sT.cols;                                   // (a multiple of 256)
        const TilePos P = tile_pos(L, sT, id);
        const int64_t r0 = P.r0, r_end = P.r_end, c0 = P.c0;
        const int64_t c = c0 + lane * 8;                             // this lane's 8 columns
        const int nrows = r0 + warp < r_end ? (int)((r_end - (r0 + warp) + 7) / 8) : 0;
        float ic[8], icc[8];
        load_f8_ro(sT.inv_col + P.cb + c, ic);
        if (L.came) load_f8_ro(sT.inv_col_conf + P.cb + c, icc);
        float *const pbase = static_cast<float *>(sT.param);
        const unsigned char *gp = static_cast<const unsigned char *>(sT.grad);
        const LerpW LW = make_lerp(sT.m_w);
        const float2 decay2 = bc2(sT.decay), step2 = bc2(step_mul), fira2 = bc2(fira);

        auto issue = [&](int k) {                                    // lane 0: row slice k of this warp into its stage
            const int64_t off = (r0 + warp + 8 * (int64_t)k) * C + c0;
            const int sl = (int)((cons + (uint32_t)k) % NS);
            unsigned char *dst = ring + sl * STAGE;
            mbar_expect_tx(&s_full[warp][sl], (uint32_t)STAGE);
            bulk_g2s(dst + P_OFF, reinterpret_cast<const unsigned char *>(pbase) + off * 4, 1024, &s_full[warp][sl]);
            bulk_g2s(dst, gp + off * GB, 256 * GB, &s_full[warp][sl]);
            bulk_g2s(dst + M_OFF, sT.m_q + off, 256, &s_full[warp][sl]);
        };
        if (lane == 0 && nrows > 0) {
            fence_proxy_async();                                     // this warp's reads of the slots came first
            for (int k = 0; k < min(NS, nrows); ++k) issue(k);
        }
        // the per-row scalars (inverse row factors, block absmax) are loaded one row ahead; the sign of a
        // negated gradient rides on the row factor ((-g) * r == g * (-r) bit for bit; without CAME the
        // gradient itself enters the momentum and is negated when unpacked)
        const int64_t row0 = r0 + warp;
        const int64_t scstep = 8 * (C >> 8);
        float *const scp = sT.m_scale + row0 * (C >> 8) + (c0 >> 8);             // + scstep per row of this warp
        const float sgn = (L.came && L.negate_grad) ? -1.0f : 1.0f;
        float n_ir = 0.0f, n_irc = 0.0f, n_sc = 0.0f;
        if (nrows > 0) {
            n_ir = load_state(sT.inv_row + row0); n_sc = load_state(scp);
            if (L.came) n_irc = load_state(sT.inv_row_conf + row0);
        }
        for (int k = 0; k < nrows; ++k) {
            const uint32_t n = cons + (uint32_t)k;
            const int sl = (int)(n % NS);
            const bool landed = mbar_wait_bounded(&s_full[warp][sl], (n / NS) & 1u);
            if (!__all_sync(0xffffffffu, landed)) {                  // (uniform over the warp)
                atomicExch(&g_device_error, DEVERR_FRING_TIMEOUT);
                return;
            }
            const unsigned char *st = ring + sl * STAGE;
            GradRaw8<GradT> cg;
            cg.from_shared(st + lane * (8 * GB));
            const float4 cp0 = *reinterpret_cast<const float4 *>(st + P_OFF + lane * 32);
            const float4 cp1 = *reinterpret_cast<const float4 *>(st + P_OFF + lane * 32 + 16);
            const uint2 cm = *reinterpret_cast<const uint2 *>(st + M_OFF + lane * 8);
            __syncwarp();                                            // the slot may be refilled
            if (lane == 0 && k + NS < nrows) { fence_proxy_async(); issue(k + NS); }

            const int64_t row = row0 + 8 * (int64_t)k;
            const int64_t flat = row * C + c;
            float g[8], u[8], mj[8];
            float2 mo[4];
            cg.unpack(L.came ? 0 : L.negate_grad, g);
            const float2 ir2 = bc2(__fmul_rn(n_ir, sgn)), irc2 = bc2(n_irc);
            uf8_decode8(cm, __fmul_rn(n_sc, 0.0078125f), mo);                    // fl(scale / 128), scale >= 1e-12
            if (k + 1 < nrows) {
                n_ir = load_state(sT.inv_row + row + 8); n_sc = load_state(scp + (k + 1) * scstep);
                if (L.came) n_irc = load_state(sT.inv_row_conf + row + 8);
            }
            if (L.came) {
#pragma unroll
                for (int j = 0; j < 8; j += 2) {
                    const float2 ut = div_by2(__fmul2_rn(__fmul2_rn(make_float2(g[j], g[j + 1]), ir2), make_float2(ic[j], ic[j + 1])), D);
                    const float2 mm = lerp_w2(mo[j >> 1], ut, LW);
                    const float2 uj = __fmul2_rn(__fmul2_rn(mm, irc2), make_float2(icc[j], icc[j + 1]));
                    mj[j] = mm.x; mj[j + 1] = mm.y; u[j] = uj.x; u[j + 1] = uj.y;
                }
            } else {
#pragma unroll
                for (int j = 0; j < 8; j += 2) {
                    const float2 mm = lerp_w2(mo[j >> 1], make_float2(g[j], g[j + 1]), LW);
                    const float2 uj = __fmul2_rn(__fmul2_rn(mm, ir2), make_float2(ic[j], ic[j + 1]));
                    mj[j] = mm.x; mj[j + 1] = mm.y; u[j] = uj.x; u[j + 1] = uj.y;
                }
            }
            float p[8] = {cp0.x, cp0.y, cp0.z, cp0.w, cp1.x, cp1.y, cp1.z, cp1.w};
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                float2 pj = __fmul2_rn(make_float2(p[j], p[j + 1]), decay2);
                if (!zero_upd) pj = __ffma2_rn(step2, __fmul2_rn(make_float2(u[j], u[j + 1]), fira2), pj);
                p[j] = pj.x; p[j + 1] = pj.y;
            }
            float *pp = pbase + flat;
            *reinterpret_cast<float4 *>(pp) = make_float4(p[0], p[1], p[2], p[3]);
            *reinterpret_cast<float4 *>(pp + 4) = make_float4(p[4], p[5], p[6], p[7]);
            if (sT.param_copy != nullptr)                                    // bf16 compute copy
                *reinterpret_cast<uint4 *>(static_cast<uint16_t *>(sT.param_copy) + flat) =
                    make_uint4(bf16x2_rn(p[0], p[1]), bf16x2_rn(p[2], p[3]), bf16x2_rn(p[4], p[5]), bf16x2_rn(p[6], p[7]));
            // the row slice is one momentum block of 256
            bool odd;
            const float am = m_absmax256(mj, odd);
            const uint2 codes = uf8_codes8(mj, am, odd);
            *reinterpret_cast<uint2 *>(sT.m_q + flat) = codes;
            if (lane == 0) scp[k * scstep] = am;
        }
        cons += (uint32_t)nrows;
    }
}

// ---------------------------------------------------------------------------
// The sum-of-squares pass over u = g * inv_row * inv_col (CAME's first sum, Adafactor without
// momentum): it only reads the gradient, 2 bytes per parameter, and with one 128-bit load per
// thread in flight (the kernel above) it was bound by memory latency.  Here a thread takes NE = 16
// consecutive elements per step of 4096 (8 where the columns are no multiple of 16) and the loads
// of its next step are issued before the current values are used: four times the bytes in flight.
// Partial sums as in factored_update_vec_kernel: one binary64 partial per thread over the chunks of
// a tensor that the CTA processes, reduced once per tensor into the slot of the run's first chunk.
// ---------------------------------------------------------------------------
template <typename GradT, int NE>
__device__ __forceinline__ double sumsq_span(const FactoredLaunch &L, const af8_factored_tensor &sT, int64_t e0, int64_t e1)
{
    constexpr int NV = NE / 8;                                   // 8-element vectors per thread and step
    constexpr int64_t STEP = (int64_t)FUPD_THREADS * NE;
    const int64_t C = sT.cols;
    double acc = 0.0;
    int64_t e = e0 + (int64_t)threadIdx.x * NE;
    if (e >= e1) return acc;
    int64_t row = e / C, col = e - row * C;
    GradRaw8<GradT> cur[NV], nxt[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) cur[v].load(sT.grad, e + 8 * v);
    for (; e < e1; e += STEP) {
        const bool more = e + STEP < e1;
        if (more) {
#pragma unroll
            for (int v = 0; v < NV; ++v) nxt[v].load(sT.grad, e + STEP + 8 * v);
        }
        const float2 ir2 = bc2(load_state(sT.inv_row + row));
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            float g[8], ic[8];
            cur[v].unpack(0, g);                                 // (the sign does not matter for the square)
            load_f8_ro(sT.inv_col + col + 8 * v, ic);
            float2 a2 = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                const float2 uj = __fmul2_rn(__fmul2_rn(make_float2(g[j], g[j + 1]), ir2), make_float2(ic[j], ic[j + 1]));
                a2 = j == 0 ? __fmul2_rn(uj, uj) : __ffma2_rn(uj, uj, a2);
            }
            acc += (double)__fadd_rn(a2.x, a2.y);
            if (more) cur[v] = nxt[v];
        }
        col += STEP;
        if (col >= C) {
            if (C >= STEP) { col -= C; ++row; }
            else { const int64_t q = col / C; row += q; col -= q * C; }
        }
    }
    return acc;
}

template <typename GradT>
__global__ void __launch_bounds__(FUPD_THREADS, 4)
factored_sumsq_wide_kernel(const FactoredLaunch L)
{
    await_launches();
    __shared__ af8_factored_tensor sT;
    __shared__ double s_acc2[FUPD_THREADS / 32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t per_cta = (L.total_units + gridDim.x - 1) / gridDim.x;
    const int64_t id_begin = (int64_t)blockIdx.x * per_cta;
    const int64_t id_end = min(id_begin + per_cta, L.total_units);
    int tn = -1;
    for (int64_t id = id_begin; id < id_end;) {
        if (tn < 0) tn = find_factored_chunk(L.tensors, L.n_tensors, id);
        else while (tn + 1 < L.n_tensors && L.tensors[tn + 1].first_chunk <= id) ++tn;
        __syncthreads();
        if (tid < (int)(sizeof(af8_factored_tensor) / 4))
            reinterpret_cast<uint32_t *>(&sT)[tid] = reinterpret_cast<const uint32_t *>(L.tensors + tn)[tid];
        __syncthreads();
        const int64_t next_first = tn + 1 < L.n_tensors ? L.tensors[tn + 1].first_chunk : L.total_units;
        const int64_t run_end = min(id_end, next_first);         // this CTA's chunks of this tensor: id .. run_end - 1
        const int64_t e0 = (id - sT.first_chunk) * 2048;
        const int64_t e1 = min((run_end - sT.first_chunk) * 2048, sT.rows * sT.cols);
        double acc = (sT.cols % 16 == 0) ? sumsq_span<GradT, 16>(L, sT, e0, e1) : sumsq_span<GradT, 8>(L, sT, e0, e1);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) s_acc2[warp] = acc;
        __syncthreads();
        if (tid == 0) {
            double sum = 0.0;
            for (int w = 0; w < FUPD_THREADS / 32; ++w) sum += s_acc2[w];
            L.block_sumsq[id] = sum;
        }
        for (int64_t i = id + 1 + tid; i < run_end; i += FUPD_THREADS) L.block_sumsq[i] = 0.0;
        id = run_end;
    }
}

// The sum of squares of u over the tiles with their rows in slices: with a UF8 momentum (MOM; Adafactor with beta1), or rows of any
// length.  (With a momentum the flat kernel above re-read the column factors for every element: 1.22 ms for the TinyLlama set's
// 3.3 GB, 0.79 here; 59 M parameters in rows of 1001 and 2731 elements 132 us, 92.)  Sums as in factored_sumsq_tile_kernel.
// whole: whether tensors of whole vectors add their squares by eight: 0 none, 1 matrices that are not a batch, 2 all.
template <typename GradT, bool MOM>
__global__ void __launch_bounds__(256, sizeof_grad<GradT>() == 2 ? 3 : 2)
factored_sumsq_slice_kernel(const FactoredLaunch L, const int whole)
{
    __shared__ af8_factored_tensor sT;
    __shared__ double s_acc2[8];
    extern __shared__ __align__(128) unsigned char sr_smem[];
    __shared__ __align__(8) uint64_t s_full[8][SLICE_STAGES];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (lane == 0) {
        for (int k = 0; k < SLICE_STAGES; ++k) mbar_init(&s_full[warp][k], SLICE_ROWS);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    await_launches();
    unsigned char *const ring = sr_smem + (size_t)warp * slice_warp_bytes<GradT>();
    uint32_t cons = 0;
    int cur_t = -1;
    for (int64_t id = blockIdx.x; id < L.total_units; id += gridDim.x) {
        int t = cur_t;
        const int64_t tile = id >> L.split;
        if (t < 0) t = find_factored_tile(L.tensors, L.n_tensors, tile);
        else while (t + 1 < L.n_tensors && L.tensors[t + 1].first_tile <= tile) ++t;
        __syncthreads();                                           // s_acc2 of the previous tile was read
        if (t != cur_t) {
            if (tid < (int)(sizeof(af8_factored_tensor) / 4))
                reinterpret_cast<uint32_t *>(&sT)[tid] = reinterpret_cast<const uint32_t *>(L.tensors + t)[tid];
            cur_t = t;
            __syncthreads();
        }
        const int64_t C = sT.cols;
        const TilePos P = tile_pos(L, sT, id);
        if (P.r0 >= P.r_end) continue;                             // an empty part of a split tile
        constexpr int MODE = MOM ? SLICE_SUM_M : SLICE_SUM_U;
        const bool vec = (C & 7) == 0, by_eight = vec && (whole == 2 || (whole == 1 && sT.batch_rows == 0));
        const bool small = !MOM || fabsf(sT.m_w) < 0.5f;
        float ic[8];
        double none[8], acc = 0.0;
#pragma unroll
        for (int j = 0; j < 8; ++j) { ic[j] = 0.0f; none[j] = 0.0; }
        bool ok;
        if (vec) {
            slice_cols<true>(sT.inv_col + P.cb, P.c0, C, ic);
            ok = small ? slice_rows<GradT, MODE, true, true>(L, sT, P.r0, P.r_end, P.c0, 1.0f, by_eight, ic, none, acc, ring, s_full[warp], cons)
                       : slice_rows<GradT, MODE, true, false>(L, sT, P.r0, P.r_end, P.c0, 1.0f, by_eight, ic, none, acc, ring, s_full[warp], cons);
        } else {
            slice_cols<false>(sT.inv_col + P.cb, P.c0, C, ic);
            ok = small ? slice_rows<GradT, MODE, false, true>(L, sT, P.r0, P.r_end, P.c0, 1.0f, by_eight, ic, none, acc, ring, s_full[warp], cons)
                       : slice_rows<GradT, MODE, false, false>(L, sT, P.r0, P.r_end, P.c0, 1.0f, by_eight, ic, none, acc, ring, s_full[warp], cons);
        }
        if (!ok) {
            atomicExch(&g_device_error, DEVERR_SRING_TIMEOUT);
            return;
        }
        acc = warp_sum(acc);
        if (lane == 0) s_acc2[warp] = acc;
        __syncthreads();
        if (tid == 0) {
            double sum = 0.0;
            for (int w = 0; w < 8; ++w) sum += s_acc2[w];
            atomicAdd(L.block_sumsq + sT.first_chunk, sum);
        }
    }
}

// The same sum over the 512 x 256 tiles of the statistic pass: a lane keeps the inverse column factors of
// its 8 columns in registers while its warp walks the tile's rows (the flat kernel above re-reads them for
// every element, twice the bytes of the gradient itself through L1), four rows' loads in flight.  A CTA adds
// its tile's sum to the slot of the tensor's first chunk; the caller clears the slots first.
// ANY = 1: batches of matrices (see sums_by_eight).  Whole vectors; rows of any length go through factored_sumsq_slice_kernel.
template <typename GradT, int ANY>
__global__ void __launch_bounds__(256, ANY ? 3 : 4)
factored_sumsq_tile_kernel(const FactoredLaunch L)
{
    constexpr int NB = 4;
    __shared__ af8_factored_tensor sT;
    __shared__ double s_acc2[8];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    await_launches();
    int cur_t = -1;
    for (int64_t id = blockIdx.x; id < L.total_units; id += gridDim.x) {
        int t = cur_t;
        const int64_t tile = id >> L.split;
        if (t < 0) t = find_factored_tile(L.tensors, L.n_tensors, tile);
        else while (t + 1 < L.n_tensors && L.tensors[t + 1].first_tile <= tile) ++t;
        __syncthreads();                                           // s_acc2 of the previous tile was read
        if (t != cur_t) {
            if (tid < (int)(sizeof(af8_factored_tensor) / 4))
                reinterpret_cast<uint32_t *>(&sT)[tid] = reinterpret_cast<const uint32_t *>(L.tensors + t)[tid];
            cur_t = t;
            __syncthreads();
        }
        const int64_t C = sT.cols;
        const TilePos P = tile_pos(L, sT, id);
        const int64_t r0 = P.r0, R = P.r_end;
        if (r0 >= R) continue;                                     // an empty part of a split tile
        const int64_t c = P.c0 + lane * 8;                         // this lane's 8 columns
        const bool col_ok = c < C;                                 // C % 8 == 0: all 8 or none
        float ic[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) ic[j] = 0.0f;
        double acc = 0.0;
        if (col_ok) load_f8_ro(sT.inv_col + P.cb + c, ic);
        const auto sum_rows = [&](auto by_eight) {                 // (a copy of the loop for each: the choice inside cost a third)
            GradRaw8<GradT> cur[NB], nxt[NB];
            auto fetch = [&](GradRaw8<GradT> (&dst)[NB], int k0) {
#pragma unroll
                for (int k = 0; k < NB; ++k) {
                    const int64_t r = r0 + warp + 8 * (k0 + k);
                    if (col_ok && r < R) dst[k].load(sT.grad, r * C + c);
                    else dst[k].zero();
                }
            };
            fetch(cur, 0);
            for (int k0 = 0; r0 + warp + 8 * k0 < R; k0 += NB) {   // (uniform over the warp)
                fetch(nxt, k0 + NB);
#pragma unroll
                for (int k = 0; k < NB; ++k) {
                    const int64_t r = min(r0 + warp + 8 * (int64_t)(k0 + k), R - 1);     // (a row beyond the end carries zeros)
                    const float2 ir2 = bc2(load_state(sT.inv_row + r));
                    float g[8];
                    cur[k].unpack(0, g);                           // (the sign does not matter for the square)
                    float2 a2 = make_float2(0.0f, 0.0f);
#pragma unroll
                    for (int j = 0; j < 8; j += 2) {
                        const float2 uj = __fmul2_rn(__fmul2_rn(make_float2(g[j], g[j + 1]), ir2), make_float2(ic[j], ic[j + 1]));
                        if (!decltype(by_eight)::value) { const float2 q = __fmul2_rn(uj, uj); acc += (double)q.x; acc += (double)q.y; }
                        else a2 = j == 0 ? __fmul2_rn(uj, uj) : __ffma2_rn(uj, uj, a2);
                    }
                    if (decltype(by_eight)::value) acc += (double)__fadd_rn(a2.x, a2.y);
                    cur[k] = nxt[k];
                }
            }
        };
        if (sums_by_eight<ANY>(sT)) sum_rows(std::true_type());
        else if constexpr (ANY != 0) sum_rows(std::false_type());
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) s_acc2[warp] = acc;
        __syncthreads();
        if (tid == 0) {
            double sum = 0.0;
            for (int w = 0; w < 8; ++w) sum += s_acc2[w];
            atomicAdd(L.block_sumsq + sT.first_chunk, sum);
        }
    }
}

inline int factored_chunk_for(int m_block)
{
    if (m_block <= 0) return 2048;
    int k = 2048 / m_block;
    if (k < 1) k = 1;
    return k * m_block;
}

inline int validate_factored(const af8_factored_cfg &c, const af8_factored_tensor *T, int n)
{
    const bool has_m = c.m_fmt != AF8_M_NONE;
    const bool m_quant = has_m && c.m_fmt != AF8_M_FP32;
    const int chunk = factored_chunk_for(m_quant ? c.m_block : 0);
    int64_t next_chunk = 0, next_tile = 0, next_small = 0;
    for (int i = 0; i < n; ++i) {
        const af8_factored_tensor &t = T[i];
        if (t.rows <= 0 || t.cols <= 0) return fail(AF8_ERR_INVALID, "factored tensor %d: empty shape", i);
        if (c.aligned8) {
            if (c.aligned8 != 2 && t.cols % 8 != 0) return fail(AF8_ERR_INVALID, "factored tensor %d: aligned8 needs cols %% 8 == 0", i);
            if (c.aligned8 == 2 && c.cols_mult8 && t.cols % 8) return fail(AF8_ERR_INVALID, "factored tensor %d: cols_mult8 needs cols %% 8 == 0", i);
            if (c.aligned8 == 2 && t.cols < 8) return fail(AF8_ERR_INVALID, "factored tensor %d: aligned8 = 2 needs cols >= 8", i);
            const void *ptrs[] = {t.param, t.grad, t.m_q, t.m_f32, t.inv_col, t.inv_col_conf, t.param_copy};
            for (const void *q : ptrs)
                if (q && (reinterpret_cast<uintptr_t>(q) & 15u)) return fail(AF8_ERR_INVALID, "factored tensor %d: aligned8 needs 16-byte aligned arrays", i);
        }
        if (t.rows * t.cols >= ((int64_t)1 << 40)) return fail(AF8_ERR_UNSUPPORTED, "factored tensor %d: too large", i);
        if (t.param_copy && c.param_dtype != AF8_F32) return fail(AF8_ERR_INVALID, "factored tensor %d: a bf16 copy exists only of fp32 parameters", i);
        if (!t.param || !t.grad || !t.row_sum || !t.col_sum || !t.inv_row || !t.inv_col)
            return fail(AF8_ERR_INVALID, "factored tensor %d: null pointer", i);
        if (c.came && (!t.inv_row_conf || !t.inv_col_conf)) return fail(AF8_ERR_INVALID, "factored tensor %d: CAME needs the confidence vectors", i);
        if (m_quant && (!t.m_q || !t.m_scale)) return fail(AF8_ERR_INVALID, "factored tensor %d: null quantised momentum", i);
        if (c.m_fmt == AF8_M_FP32 && !t.m_f32) return fail(AF8_ERR_INVALID, "factored tensor %d: null fp32 momentum", i);
        if (t.first_chunk != next_chunk) return fail(AF8_ERR_INVALID, "factored tensor %d: first_chunk %lld, expected %lld", i, (long long)t.first_chunk, (long long)next_chunk);
        if (t.first_tile != next_tile) return fail(AF8_ERR_INVALID, "factored tensor %d: first_tile %lld, expected %lld", i, (long long)t.first_tile, (long long)next_tile);
        next_chunk += (t.rows * t.cols + chunk - 1) / chunk;
        if (t.batch_rows < 0 || (t.batch_rows > 0 && t.rows % t.batch_rows != 0))
            return fail(AF8_ERR_INVALID, "factored tensor %d: batch_rows %lld does not divide rows %lld", i, (long long)t.batch_rows, (long long)t.rows);
        if (t.batch_rows > 0 && c.aligned8 && c.aligned8 != 2)
            return fail(AF8_ERR_INVALID, "factored tensor %d: a batch of matrices needs cfg.aligned8 = 0 or 2", i);
        if (c.aligned8 == 2 && t.rows >= ((int64_t)1 << 31)) return fail(AF8_ERR_UNSUPPORTED, "factored tensor %d: too many rows for aligned8 = 2", i);
        next_tile += fact_tiles(t);
        const af8_small_state *ss[4] = {&t.row_var, &t.col_var, &t.conf_row, &t.conf_col};
        const int sb = t.row_var.block;
        if (sb <= 0) return fail(AF8_ERR_INVALID, "factored tensor %d: small-state block must be positive", i);
        if (t.first_small != next_small) return fail(AF8_ERR_INVALID, "factored tensor %d: first_small %d, expected %lld", i, t.first_small, (long long)next_small);
        next_small += (t.rows + sb - 1) / sb + (fact_batch(t) * t.cols + sb - 1) / sb;
        if (next_small > 0x7fffffff) return fail(AF8_ERR_UNSUPPORTED, "factored table: too many small-state blocks");
        for (int k = 0; k < (c.came ? 4 : 2); ++k) {
            const af8_small_state &s = *ss[k];
            if (s.block != sb) return fail(AF8_ERR_INVALID, "factored tensor %d: the small states of a tensor must share one block size", i);
            if (s.fmt == AF8_V_FP32) {
                if (!s.f32) return fail(AF8_ERR_INVALID, "factored tensor %d: null fp32 small state %d", i, k);
            } else if (s.fmt == AF8_V_AL8 || s.fmt == AF8_V_AL16) {
                if (!s.q || !s.scale || !s.min_log) return fail(AF8_ERR_INVALID, "factored tensor %d: null quantised small state %d", i, k);
                if (s.block < 128 || s.block % 128 != 0 || s.block > GEN_MAX_BLOCK) return fail(AF8_ERR_INVALID, "factored tensor %d: bad block %d of small state %d", i, s.block, k);
            } else {
                return fail(AF8_ERR_INVALID, "factored tensor %d: bad format %d of small state %d", i, s.fmt, k);
            }
        }
    }
    return AF8_OK;
}

inline int check_factored_cfg(const af8_factored_cfg *cfg, const char *who)
{
    if (!cfg) return fail(AF8_ERR_INVALID, "%s: null cfg", who);
    if (cfg->param_dtype != AF8_F32 && cfg->param_dtype != AF8_BF16 && cfg->param_dtype != AF8_F16) return fail(AF8_ERR_INVALID, "%s: bad param_dtype %d", who, cfg->param_dtype);
    if (cfg->grad_dtype != AF8_F32 && cfg->grad_dtype != AF8_BF16 && cfg->grad_dtype != AF8_F16) return fail(AF8_ERR_INVALID, "%s: bad grad_dtype %d", who, cfg->grad_dtype);
    if (cfg->stochastic_round && cfg->param_dtype == AF8_F32) return fail(AF8_ERR_INVALID, "%s: stochastic rounding applies to bf16 / fp16 parameters only", who);
    if (cfg->m_fmt < AF8_M_NONE || cfg->m_fmt > AF8_M_FP32) return fail(AF8_ERR_INVALID, "%s: bad m_fmt %d", who, cfg->m_fmt);
    const bool m_quant = cfg->m_fmt != AF8_M_NONE && cfg->m_fmt != AF8_M_FP32;
    if (m_quant && (cfg->m_block < 32 || cfg->m_block % 4 != 0 || cfg->m_block > 2048)) return fail(AF8_ERR_INVALID, "%s: bad m_block %d", who, cfg->m_block);
    if (cfg->came && cfg->m_fmt == AF8_M_NONE) return fail(AF8_ERR_INVALID, "%s: CAME needs momentum", who);
    return AF8_OK;
}

inline FactoredLaunch make_factored_launch(const af8_factored_cfg &c, const af8_factored_tensor *dev, int n,
                                           int64_t units, const af8_dyn_scalars *dyn, double *sumsq)
{
    FactoredLaunch L;
    L.tensors = dev; L.dyn = dyn; L.block_sumsq = sumsq; L.total_units = units; L.n_tensors = n;
    L.grad_dtype = c.grad_dtype; L.m_fmt = c.m_fmt; L.m_block = c.m_block > 0 ? c.m_block : 256;
    L.came = c.came ? 1 : 0; L.negate_grad = c.negate_grad ? 1 : 0; L.mode = c.mode; L.v_floor = c.v_floor;
    L.param_dtype = c.param_dtype; L.sr = c.stochastic_round ? 1 : 0; L.split = 0;
    return L;
}

}  // namespace af8

extern "C" int32_t af8_factored_chunk(int32_t m_block) { return af8::factored_chunk_for(m_block); }
extern "C" int32_t af8_factored_tile_rows(void) { return af8::FSTAT_ROWS; }
extern "C" int32_t af8_factored_tile_cols(void) { return af8::FSTAT_COLS; }

extern "C" int af8_factored_upload(const af8_factored_cfg *cfg, const af8_factored_tensor *host_tensors,
                                   af8_factored_tensor *dev_tensors, int32_t n_tensors, void *stream)
{
    using namespace af8;
    int rc = check_factored_cfg(cfg, "af8_factored_upload");
    if (rc) return rc;
    if (!host_tensors || !dev_tensors || n_tensors <= 0) return fail(AF8_ERR_INVALID, "af8_factored_upload: null or empty table");
    rc = validate_factored(*cfg, host_tensors, n_tensors);
    if (rc) return rc;
    return upload_table(dev_tensors, host_tensors, sizeof(af8_factored_tensor) * (size_t)n_tensors, static_cast<cudaStream_t>(stream));
}

namespace af8 {
// the two tensor maps of a tensor for residual_rows_box: gradient (bf16) and UF8 codes as [rows][cols], boxes of
// 256 columns x FBOX_ROWS rows, no swizzle, zeros outside
inline int factored_box_maps(const af8_factored_tensor &t, CUtensorMap *out)
{
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return fail(AF8_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
    const cuuint64_t dim[2] = {(cuuint64_t)t.cols, (cuuint64_t)t.rows};
    const cuuint32_t box[2] = {256, FBOX_ROWS}, es[2] = {1, 1};
    const cuuint64_t gstride[1] = {(cuuint64_t)t.cols * 2}, mstride[1] = {(cuuint64_t)t.cols};
    CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(t.grad), dim, gstride, box, es,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(AF8_ERR_CUDA, "cuTensorMapEncodeTiled (gradient rows) failed with %d", (int)r);
    r = enc(out + 1, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, t.m_q, dim, mstride, box, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(AF8_ERR_CUDA, "cuTensorMapEncodeTiled (momentum codes) failed with %d", (int)r);
    return AF8_OK;
}
}  // namespace af8

static int af8_factored_stats_impl(const af8_factored_cfg *cfg, const af8_factored_tensor *dev_tensors,
                                   const af8_factored_tensor *host_tensors, int32_t n_tensors,
                                   const af8_dyn_scalars *dyn, void *host_maps, void *dev_maps, void *stream)
{
    using namespace af8;
    int rc = check_factored_cfg(cfg, "af8_factored_stats");
    if (rc) return rc;
    if (!dev_tensors || !host_tensors || n_tensors <= 0) return fail(AF8_ERR_INVALID, "af8_factored_stats: null or empty table");
    if (cfg->mode != AF8_FSTAT_GRADSQ && cfg->mode != AF8_FSTAT_RESIDUAL) return fail(AF8_ERR_INVALID, "af8_factored_stats: bad mode %d", cfg->mode);
    if (cfg->mode == AF8_FSTAT_RESIDUAL && (!cfg->came || !dyn)) return fail(AF8_ERR_INVALID, "af8_factored_stats: the residual needs CAME and dyn");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int64_t tiles = 0;
    // clear the accumulators: ranges that follow one another in memory form a run; one or two runs are cleared as such, more of them by a
    // launch over the table
    struct { char *begin, *end; } run[2] = {};
    int runs = 0;
    for (int i = 0; i < n_tensors; ++i) {
        const af8_factored_tensor &t = host_tensors[i];
        char *const ptr[2] = {reinterpret_cast<char *>(t.row_sum), reinterpret_cast<char *>(t.col_sum)};
        const size_t len[2] = {sizeof(double) * (size_t)t.rows, sizeof(double) * (size_t)(fact_batch(t) * t.cols)};
        for (int k = 0; k < 2; ++k) {
            if (runs > 0 && runs <= 2 && ptr[k] == run[runs - 1].end) { run[runs - 1].end += len[k]; continue; }
            if (runs < 2) { run[runs].begin = ptr[k]; run[runs].end = ptr[k] + len[k]; }
            if (runs < 3) ++runs;
        }
        tiles += fact_tiles(t);
    }
    if (runs <= 2) {
        const int rz = clear_doubles(reinterpret_cast<double *>(run[0].begin), (run[0].end - run[0].begin) / 8,
                                     reinterpret_cast<double *>(run[1].begin), (run[1].end - run[1].begin) / 8, st);
        if (rz) return rz;
    } else {
        launch_next(factored_clear_kernel, dim3((unsigned)n_tensors, 4), 256, 0, st, dev_tensors);
        AF8_CUDA_TRY(cudaGetLastError());
    }
    const bool bf = cfg->grad_dtype == AF8_BF16, res = cfg->mode == AF8_FSTAT_RESIDUAL;
    const bool vec = cfg->aligned8 && cfg->grad_dtype != AF8_F16;      // fp16 gradients take the general kernels
    FactoredLaunch L = make_factored_launch(*cfg, dev_tensors, n_tensors, tiles, dyn, nullptr);
    L.split = vec ? tile_split(tiles, res ? 3 : 1) : 0;
    L.total_units = tiles << L.split;
    int64_t grid = (int64_t)sm_count() * 6;
    if (grid > L.total_units) grid = L.total_units;
    static const bool box_off = getenv("AF8_NO_FACTORED_BOXES") != nullptr;
    const bool any = cfg->aligned8 == 2;
    // The warps' rings take 51 KB of shared memory a CTA (84 KB with binary32 gradients) from the L1 of the direct loads: only for
    // tables that have rows to take through them (g^2 pass over stacks of experts, 157 M parameters with binary32 gradients: 144 us
    // with the rings reserved, 117 without).
    int ring = (res ? cfg->m_fmt == AF8_M_UF8 && cfg->m_block == 256 : any && !cfg->cols_mult8) ? 1 : 0;
    // residual pass over bf16 gradients and UF8 codes of tensors with cols % 256 == 0: boxes of rows through
    // tensor maps, when the caller has given room for the maps
    const CUtensorMap *maps = nullptr;
    if (ring && res && !any && !box_off && vec && bf && host_maps && dev_maps && cfg->m_fmt == AF8_M_UF8 && cfg->m_block == 256 && cfg->cols_mult256) {
        bool ok = (reinterpret_cast<uintptr_t>(dev_maps) & 63) == 0;
        for (int i = 0; i < n_tensors && ok; ++i) {
            const af8_factored_tensor &t = host_tensors[i];
            ok = fact_batch(t) == 1 && t.rows < ((int64_t)1 << 31) && t.cols < ((int64_t)1 << 31) && (t.cols % 256) == 0 &&
                 t.rows * (t.cols >> 8) < ((int64_t)1 << 31);
        }
        if (ok) {
            CUtensorMap *hm = static_cast<CUtensorMap *>(host_maps);
            for (int i = 0; i < n_tensors; ++i) {
                rc = factored_box_maps(host_tensors[i], hm + 2 * i);
                if (rc) return rc;
            }
            rc = upload_table<true>(dev_maps, host_maps, sizeof(CUtensorMap) * 2 * (size_t)n_tensors, st);
            if (rc) return rc;
            maps = static_cast<const CUtensorMap *>(dev_maps);
            ring = 2;
        }
    }
#define AF8_LAUNCH_FSTAT_IN(G, RES, A, I) do { \
        const size_t sm = (I) ? slice_smem_bytes<G>() : 0; \
        if (sm > 0) AF8_CUDA_TRY(cudaFuncSetAttribute(factored_stats_vec_kernel<G, RES, A, I>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm)); \
        launch_next(factored_stats_vec_kernel<G, RES, A, I>, (int)grid, 256, sm, st, L, maps); } while (0)
#define AF8_LAUNCH_FSTAT(G, RES) do { \
        if (any && ring) AF8_LAUNCH_FSTAT_IN(G, RES, true, 1); else if (any) AF8_LAUNCH_FSTAT_IN(G, RES, true, 0); \
        else if (RES && ring == 1) AF8_LAUNCH_FSTAT_IN(G, RES, false, 1); else AF8_LAUNCH_FSTAT_IN(G, RES, false, 0); } while (0)
    if (vec && bf && res && ring == 2) AF8_LAUNCH_FSTAT_IN(bf16_tag, true, false, 2);
    else if (vec && bf && res) AF8_LAUNCH_FSTAT(bf16_tag, true);
    else if (vec && bf) AF8_LAUNCH_FSTAT(bf16_tag, false);
    else if (vec && res) AF8_LAUNCH_FSTAT(float, true);
    else if (vec) AF8_LAUNCH_FSTAT(float, false);
#undef AF8_LAUNCH_FSTAT
#undef AF8_LAUNCH_FSTAT_IN
    else launch_next(factored_stats_kernel, (int)grid, 256, 0, st, L);
    AF8_CUDA_TRY(cudaGetLastError());
    return AF8_OK;
}

extern "C" int af8_factored_stats(const af8_factored_cfg *cfg, const af8_factored_tensor *dev_tensors,
                                  const af8_factored_tensor *host_tensors, int32_t n_tensors,
                                  const af8_dyn_scalars *dyn, void *stream)
{
    return af8_factored_stats_impl(cfg, dev_tensors, host_tensors, n_tensors, dyn, nullptr, nullptr, stream);
}

extern "C" int af8_factored_stats_boxes(const af8_factored_cfg *cfg, const af8_factored_tensor *dev_tensors,
                                        const af8_factored_tensor *host_tensors, int32_t n_tensors,
                                        const af8_dyn_scalars *dyn, void *host_maps, void *dev_maps, void *stream)
{
    return af8_factored_stats_impl(cfg, dev_tensors, host_tensors, n_tensors, dyn, host_maps, dev_maps, stream);
}

extern "C" int af8_factored_small(const af8_factored_cfg *cfg, const af8_factored_tensor *dev_tensors,
                                  int32_t n_tensors, int32_t conf, int32_t total_units, void *stream)
{
    using namespace af8;
    int rc = check_factored_cfg(cfg, "af8_factored_small");
    if (rc) return rc;
    if (!dev_tensors || n_tensors <= 0 || total_units <= 0) return fail(AF8_ERR_INVALID, "af8_factored_small: null or empty table");
    if (conf && !cfg->came) return fail(AF8_ERR_INVALID, "af8_factored_small: confidence states exist only with CAME");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // At most one unit per SM (long blocks, few tensors): the launch lasts as long as one CTA, so more threads.  Device time of the
    // launch and factored_inv_kernel with 256, 512 and 1024 threads, few units: blocks of 256 13.3, 13.3, 14.1 us; of 512 14.0, 13.3,
    // 14.6; of 1024 15.4, 14.6, 14.4; of 2048 18.4, 15.4, 15.4 (CAME's confidence states 25.0, 20.9, 19.9); of 4096 21.5, 17.4, 17.2.
    // Many units: 480 of 256 elements 6.2 us with 256 threads, 14 with 512.
    if (total_units <= sm_count()) launch_next(factored_small_kernel<SMALL_MAX_THREADS>, total_units, SMALL_MAX_THREADS, 0, st, dev_tensors, n_tensors, conf, cfg->v_floor);
    else launch_next(factored_small_kernel<256>, total_units, 256, 0, st, dev_tensors, n_tensors, conf, cfg->v_floor);
    AF8_CUDA_TRY(cudaGetLastError());
    launch_next(factored_inv_kernel, dim3((unsigned)n_tensors, 8), 256, 0, st, dev_tensors, conf);
    AF8_CUDA_TRY(cudaGetLastError());
    return AF8_OK;
}

extern "C" int af8_factored_update(const af8_factored_cfg *cfg, const af8_factored_tensor *dev_tensors,
                                   int32_t n_tensors, int64_t total_chunks, const af8_dyn_scalars *dyn,
                                   double *block_sumsq, void *stream)
{
    using namespace af8;
    int rc = check_factored_cfg(cfg, "af8_factored_update");
    if (rc) return rc;
    if (!dev_tensors || n_tensors <= 0 || total_chunks <= 0) return fail(AF8_ERR_INVALID, "af8_factored_update: null or empty table");
    if (cfg->mode < AF8_FUPD_SUMSQ_U || cfg->mode > AF8_FUPD_LAG) return fail(AF8_ERR_INVALID, "af8_factored_update: bad mode %d", cfg->mode);
    if (cfg->mode == AF8_FUPD_LAG && (cfg->came || !dyn)) return fail(AF8_ERR_INVALID, "af8_factored_update: the lag pass needs dyn and excludes CAME");
    if (cfg->mode != AF8_FUPD_APPLY && !block_sumsq) return fail(AF8_ERR_INVALID, "af8_factored_update: this mode needs block_sumsq");
    if (cfg->mode == AF8_FUPD_SUMSQ_U && !cfg->came) return fail(AF8_ERR_INVALID, "af8_factored_update: SUMSQ_U is a CAME pass");
    if (cfg->came && cfg->mode != AF8_FUPD_SUMSQ_U && !dyn) return fail(AF8_ERR_INVALID, "af8_factored_update: CAME passes need dyn");
    const bool m_quant = cfg->m_fmt != AF8_M_NONE && cfg->m_fmt != AF8_M_FP32;
    const int chunk = factored_chunk_for(m_quant ? cfg->m_block : 0);
    FactoredLaunch L = make_factored_launch(*cfg, dev_tensors, n_tensors, total_chunks, dyn, block_sumsq);
    const size_t smem = sizeof(float) * (size_t)chunk;
    int64_t grid = (int64_t)sm_count() * 6;
    if (grid > total_chunks) grid = total_chunks;
    const bool vec = cfg->aligned8 && chunk == 2048 && (!m_quant || cfg->m_block == 256) && cfg->grad_dtype != AF8_F16;
    const bool apply = cfg->mode == AF8_FUPD_APPLY || cfg->mode == AF8_FUPD_LAG;
    const bool lag = cfg->mode == AF8_FUPD_LAG;
    if (vec) {                                   // persistent: the CTAs that are resident together
        grid = (int64_t)sm_count() * (apply ? (cfg->m_fmt == AF8_M_NONE ? 2 : 3) : 4);
        if (grid > total_chunks) grid = total_chunks;
    }
    cudaStream_t cst = static_cast<cudaStream_t>(stream);
    const bool bf = cfg->grad_dtype == AF8_BF16;
    const bool no_m = cfg->m_fmt == AF8_M_NONE;
    static const bool wide_off = getenv("AF8_NO_WIDE_SUMS") != nullptr;
    static const bool tile_off = getenv("AF8_NO_TILE_SUMS") != nullptr;
    const int64_t total_tiles = cfg->total_tiles;
    const bool any = cfg->aligned8 == 2;         // batches of matrices, rows of any length >= 8
    const bool only_g = (cfg->came && cfg->mode == AF8_FUPD_SUMSQ_U) || no_m;
    // With a UF8 momentum (not CAME's): in slices over the tiles where the table is large and fills its tiles, else in flat order.
    // Size: the sums that the tiles add to are cleared first, a launch of 2 us (3 of host time).  Slices and flat, bf16 and binary32
    // gradients: whole vectors 1 M parameters 12.7, 8.6 us; 16.8 M 27.0, 27.0 and 30.4, 29.1; 77 M 81, 107 and 108, 111; 352 M 263,
    // 404 and 334, 464; ragged rows or batches, whose flat kernel is the slower one, 1 M 14.1, 10.7; 9.4 M 24.1, 25.0 and 26.6,
    // 27.0; 132 M 184, 271 and 205, 282.
    // Filling: a warp takes up to 256 columns of a row at a time, and the CTA that gets one tile more decides.  Rows of 16 elements,
    // 16 M parameters, 189, 29; 30 M bf16 in rows of 192 52, 46, of 224 42, 46, of 117 90, 78, of 165 74, 76, of 205 56, 76; in
    // matrices of 560 x 560 84, 48.
    const int64_t slice_from = any ? 4096 : bf ? 8192 : 32768;                                           // chunks of 2048 elements
    const bool filled = total_chunks * 2048 * 10 >= total_tiles * (FSTAT_ROWS * FSTAT_COLS) * (any ? 5 : 8);
    const bool mom = !cfg->came && cfg->m_fmt == AF8_M_UF8 && cfg->m_block == 256 && filled && total_chunks >= slice_from;
    if (vec && !apply && !tile_off && total_tiles > 0 && cfg->grad_dtype != AF8_F16 && (only_g || mom)) {
        // over the statistic tiles, column factors in registers; with a momentum, or rows of any length, in slices
        const int rz = clear_doubles(block_sumsq, total_chunks, nullptr, 0, cst);
        if (rz) return rz;
        FactoredLaunch LT = L;
        LT.split = tile_split(total_tiles);
        LT.total_units = total_tiles << LT.split;
        const int kind = !any ? 0 : cfg->cols_mult8 ? 1 : 2;
        if (mom || kind == 2) {
            const int64_t sg = std::min<int64_t>((int64_t)sm_count() * (bf ? 3 : 2), LT.total_units);
#define AF8_LAUNCH_FSLICE(G, M) do { \
            AF8_CUDA_TRY(cudaFuncSetAttribute(factored_sumsq_slice_kernel<G, M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)slice_smem_bytes<G>())); \
            launch_next(factored_sumsq_slice_kernel<G, M>, (int)sg, 256, slice_smem_bytes<G>(), cst, LT, 2 - kind); } while (0)
            if (bf) { if (mom) AF8_LAUNCH_FSLICE(bf16_tag, true); else AF8_LAUNCH_FSLICE(bf16_tag, false); }
            else { if (mom) AF8_LAUNCH_FSLICE(float, true); else AF8_LAUNCH_FSLICE(float, false); }
#undef AF8_LAUNCH_FSLICE
            AF8_CUDA_TRY(cudaGetLastError());
            return AF8_OK;
        }
        const int64_t tg = std::min<int64_t>((int64_t)sm_count() * 8, LT.total_units);
#define AF8_LAUNCH_FSUM(G) do { if (kind == 0) launch_next(factored_sumsq_tile_kernel<G, 0>, (int)tg, 256, 0, cst, LT); \
        else launch_next(factored_sumsq_tile_kernel<G, 1>, (int)tg, 256, 0, cst, LT); } while (0)
        if (bf) AF8_LAUNCH_FSUM(bf16_tag);
        else AF8_LAUNCH_FSUM(float);
#undef AF8_LAUNCH_FSUM
        AF8_CUDA_TRY(cudaGetLastError());
        return AF8_OK;
    }
    if (vec && !any && !apply && !wide_off && cfg->grad_dtype != AF8_F16 && ((cfg->came && cfg->mode == AF8_FUPD_SUMSQ_U) || no_m)) {
        // the sum only needs the gradient: 16 elements per thread, next step's loads in flight
        if (bf) launch_next(factored_sumsq_wide_kernel<bf16_tag>, (int)grid, FUPD_THREADS, 0, cst, L);
        else launch_next(factored_sumsq_wide_kernel<float>, (int)grid, FUPD_THREADS, 0, cst, L);
        AF8_CUDA_TRY(cudaGetLastError());
        return AF8_OK;
    }
    static const bool tile_apply_off = getenv("AF8_NO_TILE_APPLY") != nullptr;
    if (vec && cfg->mode == AF8_FUPD_APPLY && cfg->m_fmt == AF8_M_UF8 && cfg->param_dtype == AF8_F32 && !tile_apply_off &&
        cfg->total_tiles > 0 && cfg->cols_mult256) {
        // every row slice of 256 columns is one momentum block: tile order, column factors in registers
        FactoredLaunch LT = L;
        LT.split = tile_split(cfg->total_tiles);
        LT.total_units = cfg->total_tiles << LT.split;
        if (bf) {
            int64_t tg = std::min<int64_t>((int64_t)sm_count() * 3, LT.total_units);
            AF8_CUDA_TRY(cudaFuncSetAttribute(factored_apply_tile_kernel<bf16_tag, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fring_smem_bytes<bf16_tag>()));
            launch_next(factored_apply_tile_kernel<bf16_tag, 3>, (int)tg, FUPD_THREADS, fring_smem_bytes<bf16_tag>(), cst, LT);
        } else {
            int64_t tg = std::min<int64_t>((int64_t)sm_count() * 2, LT.total_units);
            AF8_CUDA_TRY(cudaFuncSetAttribute(factored_apply_tile_kernel<float, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fring_smem_bytes<float>()));
            launch_next(factored_apply_tile_kernel<float, 2>, (int)tg, FUPD_THREADS, fring_smem_bytes<float>(), cst, LT);
        }
        AF8_CUDA_TRY(cudaGetLastError());
        return AF8_OK;
    }
    // (see PT: bf16 gradients with bf16 parameters have kernels of their own)
    const int pt = cfg->param_dtype == AF8_F32 ? 0 : (bf && cfg->param_dtype == AF8_BF16 && !lag) ? (cfg->stochastic_round ? 2 : 1) : 3;
    if (vec && cfg->mode == AF8_FUPD_APPLY && no_m && pt != 3 && (!any || cfg->cols_mult8)) {
        // no momentum, rows of whole vectors: one CTA per unit
        if (total_chunks > INT32_MAX) return fail(AF8_ERR_UNSUPPORTED, "af8_factored_update: %lld chunks in one launch", (long long)total_chunks);
#define AF8_LAUNCH_FWRITE(G, T, A) do { \
        AF8_CUDA_TRY(cudaFuncSetAttribute(factored_write_kernel<G, T, A>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)write_smem_bytes<sizeof_grad<G>(), T == 0 ? 4 : 2>())); \
        launch_next(factored_write_kernel<G, T, A>, (int)total_chunks, WRITE_THREADS + 32, write_smem_bytes<sizeof_grad<G>(), T == 0 ? 4 : 2>(), cst, L); } while (0)
#define AF8_LAUNCH_FWRITE_ANY(G, T) do { if (any) AF8_LAUNCH_FWRITE(G, T, true); else AF8_LAUNCH_FWRITE(G, T, false); } while (0)
        if (!bf) AF8_LAUNCH_FWRITE_ANY(float, 0);
        else if (pt == 0) AF8_LAUNCH_FWRITE_ANY(bf16_tag, 0);
        else if (pt == 1) AF8_LAUNCH_FWRITE_ANY(bf16_tag, 1);
        else AF8_LAUNCH_FWRITE_ANY(bf16_tag, 2);
#undef AF8_LAUNCH_FWRITE_ANY
#undef AF8_LAUNCH_FWRITE
        AF8_CUDA_TRY(cudaGetLastError());
        return AF8_OK;
    }
    if (vec && cfg->mode == AF8_FUPD_APPLY && cfg->m_fmt == AF8_M_UF8 && pt != 3) {
        // UF8 momentum: inputs through per-warp rings of bulk copies
        grid = std::min<int64_t>((int64_t)sm_count() * (bf ? (any ? FLAT_ANY_CTAS : 3) : 2), total_chunks);
#define AF8_LAUNCH_FLAT(G, T, A) do { \
        AF8_CUDA_TRY(cudaFuncSetAttribute(factored_apply_flat_kernel<G, T, A>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fring_smem_bytes<G, T>())); \
        launch_next(factored_apply_flat_kernel<G, T, A>, (int)grid, FUPD_THREADS, fring_smem_bytes<G, T>(), cst, L); } while (0)
#define AF8_LAUNCH_FLAT_ANY(G, T) do { if (any) AF8_LAUNCH_FLAT(G, T, true); else AF8_LAUNCH_FLAT(G, T, false); } while (0)
        if (!bf) AF8_LAUNCH_FLAT_ANY(float, 0);
        else if (pt == 0) AF8_LAUNCH_FLAT_ANY(bf16_tag, 0);
        else if (pt == 1) AF8_LAUNCH_FLAT_ANY(bf16_tag, 1);
        else AF8_LAUNCH_FLAT_ANY(bf16_tag, 2);
#undef AF8_LAUNCH_FLAT_ANY
#undef AF8_LAUNCH_FLAT
        AF8_CUDA_TRY(cudaGetLastError());
        return AF8_OK;
    }
#define AF8_LAUNCH_FUPD(G, P, C, A, T) launch_next(factored_update_vec_kernel<G, P, C, A, T>, (int)grid, FUPD_THREADS, 0, cst, L)
#define AF8_LAUNCH_FUPD_PT(P, C, A) do { \
        if (bf && pt == 0) AF8_LAUNCH_FUPD(bf16_tag, P, C, A, 0); else if (bf && pt == 3) AF8_LAUNCH_FUPD(bf16_tag, P, C, A, 3); \
        else if (pt == 0) AF8_LAUNCH_FUPD(float, P, C, A, 0); else if (pt == 3) AF8_LAUNCH_FUPD(float, P, C, A, 3); \
        else if (P == 1 && pt == 1) AF8_LAUNCH_FUPD(bf16_tag, 1, C, A, 1); else AF8_LAUNCH_FUPD(bf16_tag, 1, C, A, 2); } while (0)
#define AF8_LAUNCH_FUPD_SUM(C, A) do { if (bf) AF8_LAUNCH_FUPD(bf16_tag, 0, C, A, 0); else AF8_LAUNCH_FUPD(float, 0, C, A, 0); } while (0)
    if (vec && any) {                            // (writing: 2 resident CTAs; the sum pass: 3)
        grid = std::min<int64_t>((int64_t)sm_count() * (apply ? 2 : 3), total_chunks);
        if (lag) { if (cfg->cols_mult8) AF8_LAUNCH_FUPD_PT(2, 2, 1); else AF8_LAUNCH_FUPD_PT(2, 2, 2); }
        else if (apply) { if (cfg->cols_mult8) AF8_LAUNCH_FUPD_PT(1, 2, 1); else AF8_LAUNCH_FUPD_PT(1, 2, 2); }
        else if (cfg->cols_mult8) AF8_LAUNCH_FUPD_SUM(3, 1);
        else AF8_LAUNCH_FUPD_SUM(3, 2);
    }
    else if (vec && lag) { if (no_m) AF8_LAUNCH_FUPD_PT(2, 2, 0); else AF8_LAUNCH_FUPD_PT(2, 3, 0); }
    else if (vec && apply && no_m) { if (bf) AF8_LAUNCH_FUPD(bf16_tag, 1, 2, 0, 3); else AF8_LAUNCH_FUPD(float, 1, 2, 0, 3); }     // (pt 3)
    else if (vec && apply) AF8_LAUNCH_FUPD_PT(1, 3, 0);
    else if (vec) AF8_LAUNCH_FUPD_SUM(4, 0);
#undef AF8_LAUNCH_FUPD_SUM
#undef AF8_LAUNCH_FUPD_PT
#undef AF8_LAUNCH_FUPD
    else launch_next(factored_update_kernel, (int)grid, FUPD_THREADS, smem, static_cast<cudaStream_t>(stream), L, chunk);
    AF8_CUDA_TRY(cudaGetLastError());
    return AF8_OK;
}
