// Group quantizer: fp16/fp32 -> b-bit codes packed in int32 words + per-group scale and min.
//
// Arithmetic (must be bit-identical to upstream quant_cuda/csrc/quantization_cuda.cu:553-596 with
// IEEE division; this file is compiled without fast-math):
//   mn, mx   fp32 min / max of the group
//   scale32  (mx - mn) / (2^b - 1)
//   code     clamp(roundf((x - mn) / scale32), 0, 2^b - 1), roundf = half away from zero;
//            3-bit: the 11th element of each group clamps to 3; 0/0 (constant group) -> 0
//   stored scale = scale32 narrowed to the input dtype, stored mn = mn
//
// Four kernels, one result:
//   quant_contig_kernel   groups run along the contiguous axis (values: [.., T, D], groups over D;
//                         or keys already transposed to [.., D, T]).  A thread owns one to four output
//                         words at a time; the threads of a group combine min/max with shuffles.
//   quant_strided_kernel  groups run along a strided axis while the *other* axis is contiguous
//                         (keys left as [.., T, D], groups over T).  A thread owns two adjacent
//                         channels, keeps a whole group in registers (all loads in flight at
//                         once), and the CTA transposes words through shared memory so global
//                         writes are contiguous runs per channel.
//   quant_rope_kernel     the same for keys that still have to be rotated (a prompt that prefill.cu does not take in one launch).
//   quant_generic_kernel  any strides / any group-to-word relation; one thread per word.
#include "quant_tiles.cuh"

namespace kvq {

// ---------------------------------------------------------------------------------------------
// Contiguous groups: blockIdx.y = (b, h); inside a (b, h) slab units of WPT words are numbered linearly.  A thread takes `upt` of them
// where there are CTAs enough: what it does once (addresses, constants in register pairs) is as much as 13 elements' work.
template <int BITS, typename T, int WPT>
__global__ void __launch_bounds__(256) quant_contig_kernel(const T *__restrict__ x, int32_t *__restrict__ code,
                                                           T *__restrict__ scale, T *__restrict__ mn, QuantDims d,
                                                           int tpg, bool vec_ok, bool linear, int upt) {
    const int b = blockIdx.y / (int)d.H, h = blockIdx.y - b * (int)d.H, total = (int)(d.A * (d.S / (fields_per_word(BITS) * WPT)));
    int idx = blockIdx.x * (256 * upt) + threadIdx.x;
#pragma unroll 1
    for (int k = 0; k < upt && idx - (int)threadIdx.x < total; ++k, idx += 256)
        quant_contig_unit<BITS, T, WPT>(x, code, scale, mn, d, tpg, vec_ok, linear, b, h, idx);
}

// ---------------------------------------------------------------------------------------------
// Strided groups over s, contiguous channel axis a (x_sA == 1), fp16, A % 128 == 0.
// CTA: 256 threads = 64 channel pairs x 4 group slots; covers 128 channels x GPC groups.
template <int BITS, int G>
struct StridedCfg {
    static constexpr int FPI = fields_per_word(BITS);
    static constexpr int WPG = G / FPI;                       // words per group (1 for 3-bit)
    static constexpr int GPC = (G == 11) ? 24 : (256 / G < 4 ? 4 : 256 / G);  // groups per CTA
    static constexpr int WPC = GPC * WPG;                     // words per channel per CTA
    static constexpr int WPAD = WPC + 1;
};

// ROWS128: tokens lie 128 elements apart (keys as [.., T, 128], back to back), so that the loads of a group differ by immediates: the
// addresses were an eighth of the kernel's instructions.
template <int BITS, int G, bool ROWS128>
__global__ void __launch_bounds__(256, 3) quant_strided_kernel(const __half *__restrict__ x, int32_t *__restrict__ code,
                                                            __half *__restrict__ scale, __half *__restrict__ mn,
                                                            QuantDims d) {
    using C = StridedCfg<BITS, G>;
    __shared__ int32_t s_code[128 * C::WPAD];
    __shared__ __half s_scale[128 * (C::GPC + 2)];
    __shared__ __half s_mn[128 * (C::GPC + 2)];

    const int pair = threadIdx.x & 63, slot = threadIdx.x >> 6;
    const int64_t bh = blockIdx.z, b = bh / d.H, h = bh % d.H;
    const int64_t a0 = (int64_t)blockIdx.y * 128;
    const int64_t g0 = (int64_t)blockIdx.x * C::GPC;          // first group of this CTA
    const int64_t n_groups = d.S / G;
    const int groups_here = (int)min((int64_t)C::GPC, n_groups - g0);
    const __half *px = x + b * d.x_sB + h * d.x_sH + (a0 + 2 * pair);
    constexpr int QMAX = (1 << BITS) - 1;
    // element pair (2 pair, 2 pair + 1) of token s of this (b, h) slab
    const int64_t row = ROWS128 ? 128 : d.x_sS;
    auto load = [&](const __half *pg, int i) -> __half2 {
        if constexpr (ROWS128) return __ldg(reinterpret_cast<const __half2 *>(pg) + i * 64);
        else return __ldg(reinterpret_cast<const __half2 *>(pg + i * row));
    };

    // tokens held in registers at a time: a whole group up to 32 tokens; longer groups are walked twice anyway (min/max,
    // then codes from L1/L2), and for them 16 at a time measured 5-10 % faster for 2- and 4-bit codes (fewer live
    // registers under the 80-register cap); a 1-bit word needs 32 tokens
    constexpr int CH = G > 32 ? (BITS == 1 ? 32 : 16) : G;
    constexpr int NCH = G / CH;
    constexpr int WPCH = CH / C::FPI;                         // words per chunk (1 for the 11-token group)
    for (int g = slot; g < groups_here; g += 4) {
        const __half *pg = px + (g0 + g) * G * row;           // the group's first token
        __half2 raw[CH];
        // min / max of the two channels in fp16x2 (exact: the data are fp16; NaN operands are skipped as by fminf)
        __half2 lo2 = __floats2half2_rn(65504.f, 65504.f), hi2 = __floats2half2_rn(-65504.f, -65504.f);
        bool first = true;
#pragma unroll 1
        for (int c = 0; c < NCH; ++c) {
#pragma unroll
            for (int i = 0; i < CH; ++i) raw[i] = load(pg + c * CH * row, i);
            if (first) { lo2 = raw[0]; hi2 = raw[0]; first = false; }
#pragma unroll
            for (int i = 0; i < CH; ++i) { lo2 = __hmin2(lo2, raw[i]); hi2 = __hmax2(hi2, raw[i]); }
        }
        const float lo0 = __low2float(lo2), lo1 = __high2float(lo2), hi0 = __low2float(hi2), hi1 = __high2float(hi2);
        const float sc0 = (hi0 - lo0) / (float)QMAX, sc1 = (hi1 - lo1) / (float)QMAX;
        const float ri0 = __frcp_rn(sc0), ri1 = __frcp_rn(sc1);     // correctly rounded reciprocals
#pragma unroll 1
        for (int c = 0; c < NCH; ++c) {
            if (NCH > 1) {                                    // long groups: second pass over the chunk (cache hit)
#pragma unroll
                for (int i = 0; i < CH; ++i) raw[i] = load(pg + c * CH * row, i);
            }
#pragma unroll
            for (int w = 0; w < WPCH; ++w) {
                const uint32_t w0 = quant_word<BITS>([&](int i) { return __low2float(raw[w * C::FPI + i]); }, lo0, sc0, ri0);
                const uint32_t w1 = quant_word<BITS>([&](int i) { return __high2float(raw[w * C::FPI + i]); }, lo1, sc1, ri1);
                s_code[(2 * pair) * C::WPAD + g * C::WPG + c * WPCH + w] = (int32_t)w0;
                s_code[(2 * pair + 1) * C::WPAD + g * C::WPG + c * WPCH + w] = (int32_t)w1;
            }
        }
        s_scale[(2 * pair) * (C::GPC + 2) + g] = __float2half_rn(stored_scale<QMAX>(hi0 - lo0, sc0, d.by_div));
        s_scale[(2 * pair + 1) * (C::GPC + 2) + g] = __float2half_rn(stored_scale<QMAX>(hi1 - lo1, sc1, d.by_div));
        s_mn[(2 * pair) * (C::GPC + 2) + g] = __float2half_rn(lo0);
        s_mn[(2 * pair + 1) * (C::GPC + 2) + g] = __float2half_rn(lo1);
    }
    __syncthreads();
    const int words_here = groups_here * C::WPG;
    int32_t *pc = code + b * d.c_sB + h * d.c_sH + a0 * d.c_sA + g0 * C::WPG;
    const int64_t zo = b * d.z_sB + h * d.z_sH + a0 * d.z_sA + g0;
    if (groups_here == C::GPC) {                              // full CTA: row lengths are compile-time constants
        for (int i = threadIdx.x; i < 128 * C::WPC; i += 256) {
            const int ch = i / C::WPC, w = i % C::WPC;
            pc[ch * d.c_sA + w] = s_code[ch * C::WPAD + w];
        }
        for (int i = threadIdx.x; i < 128 * C::GPC; i += 256) {
            const int ch = i / C::GPC, g = i % C::GPC;
            scale[zo + ch * d.z_sA + g] = s_scale[ch * (C::GPC + 2) + g];
            mn[zo + ch * d.z_sA + g] = s_mn[ch * (C::GPC + 2) + g];
        }
    } else {
        for (int i = threadIdx.x; i < 128 * words_here; i += 256) {
            const int ch = i / words_here, w = i % words_here;
            pc[ch * d.c_sA + w] = s_code[ch * C::WPAD + w];
        }
        for (int i = threadIdx.x; i < 128 * groups_here; i += 256) {
            const int ch = i / groups_here, g = i % groups_here;
            scale[zo + ch * d.z_sA + g] = s_scale[ch * (C::GPC + 2) + g];
            mn[zo + ch * d.z_sA + g] = s_mn[ch * (C::GPC + 2) + g];
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Keys rotated on the way in, as a launch of their own.
template <int BITS, int G>
__global__ void __launch_bounds__(256, 4) quant_rope_kernel(const __half *__restrict__ x, int32_t *__restrict__ code,
                                                         __half *__restrict__ scale, __half *__restrict__ mn, QuantDims d, RopeTables rope) {
    quant_rope_tile<BITS, G>(x, code, scale, mn, d, rope, blockIdx.x, blockIdx.z);
}

// ---------------------------------------------------------------------------------------------
// Any layout: one thread per output word, group statistics recomputed as needed.
template <int BITS, typename T>
__global__ void __launch_bounds__(128) quant_generic_kernel(const T *__restrict__ x, int32_t *__restrict__ code,
                                                            T *__restrict__ scale, T *__restrict__ mn, QuantDims d) {
    constexpr int E = fields_per_word(BITS);
    constexpr int QMAX = (1 << BITS) - 1;
    const int64_t words_per_row = d.S / E;
    const int64_t total = d.B * d.H * d.A * words_per_row;
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const int64_t row = idx / words_per_row, w = idx % words_per_row;
    const int64_t a = row % d.A, h = (row / d.A) % d.H, b = row / (d.A * d.H);
    const T *px = x + b * d.x_sB + h * d.x_sH + a * d.x_sA;
    const int64_t zo = b * d.z_sB + h * d.z_sH + a * d.z_sA;
    const int G = d.group;
    int64_t cur = -1;
    float lo = 0.f, sc = 0.f, range = 0.f;
    uint32_t word = 0;
    for (int i = 0; i < E; ++i) {
        const int64_t s = w * E + i, g = s / G;
        if (g != cur) {
            cur = g;
            float hi = -3.402823466e+38f;
            lo = 3.402823466e+38f;
            for (int j = 0; j < G; ++j) {
                const float f = to_f32<T>(px[(g * G + j) * d.x_sS]);
                lo = fminf(lo, f); hi = fmaxf(hi, f);
            }
            range = hi - lo;
            sc = range / (float)QMAX;
        }
        if (s % G == 0) {
            scale[zo + g] = from_f32<T>(stored_scale<QMAX>(range, sc, d.by_div));
            mn[zo + g] = from_f32<T>(lo);
        }
        const float n = (to_f32<T>(px[s * d.x_sS]) - lo) / sc;
        if constexpr (BITS == 3) {
            const int pos = (int)(s % G);   // position inside the 11-group (G == 11 enforced by the host)
            word |= (uint32_t)round_code(n, pos < 10 ? 7 : 3) << (i < 10 ? 3 * i : 30);
        } else {
            word |= (uint32_t)round_code(n, QMAX) << (BITS * i);
        }
    }
    code[b * d.c_sB + h * d.c_sH + a * d.c_sA + w] = (int32_t)word;
}

// ---------------------------------------------------------------------------------------------
// 3-bit groups of 11 with a short last group: one thread per word.
template <typename T>
__global__ void __launch_bounds__(128) quant_ragged3_kernel(const T *__restrict__ x, int32_t *__restrict__ code,
                                                            T *__restrict__ scale, T *__restrict__ mn, QuantDims d) {
    quant_ragged3_word<T>(x, code, scale, mn, d, (int64_t)blockIdx.x * blockDim.x + threadIdx.x);
}

template <typename T>
static int launch_ragged3(const kvq_quant_args *a, const QuantDims &d, cudaStream_t st) {
    const int64_t total = d.B * d.H * d.A * ((d.S + 10) / 11);
    quant_ragged3_kernel<T><<<(unsigned)((total + 127) / 128), 128, 0, st>>>(
        static_cast<const T *>(a->x), a->code, static_cast<T *>(a->scale), static_cast<T *>(a->mn), d);
    return check_launch();
}

// ---------------------------------------------------------------------------------------------
template <int BITS, typename T>
static int launch_bits(const kvq_quant_args *a, const QuantDims &d, cudaStream_t st, const RopeTables *rope = nullptr) {
    constexpr int E = fields_per_word(BITS);
    const T *x = static_cast<const T *>(a->x);
    T *sc = static_cast<T *>(a->scale), *mn = static_cast<T *>(a->mn);
    const int G = a->group;
    const int64_t total_words = d.B * d.H * d.A * (d.S / E);
    if (total_words == 0) return KVQ_OK;

    // groups along the contiguous axis
    if (!rope && a->x_sS == 1 && G % E == 0) {
        bool vec_ok = sizeof(T) == 2 && (reinterpret_cast<uintptr_t>(x) % 16 == 0) && d.x_sB % 8 == 0 &&
                      d.x_sH % 8 == 0 && d.x_sA % 8 == 0;
        // 32 elements (64 B of fp16 in flight) per thread where the group and the row allow it: 4 / 2 words for 4 / 2 bits
        constexpr int WMAX = (sizeof(T) == 2 && E < 32 && 32 % E == 0) ? 32 / E : 1;
        const bool wide = WMAX > 1 && vec_ok && G % (WMAX * E) == 0 && (d.S / E) % WMAX == 0;
        const int wpt = wide ? WMAX : 1;
        const int tpg = G / (E * wpt);
        const int64_t per_slab = d.A * (d.S / (E * wpt));
        if (tpg <= 32 && (tpg & (tpg - 1)) == 0 && per_slab < (1LL << 31) && d.B * d.H <= 65535) {
            const int64_t wpr = d.S / E;
            const bool linear = d.x_sA == d.S && d.c_sA == wpr && d.z_sA == d.S / G;
            // four units a thread from eight waves of CTAs on (eight to an SM)
            const int upt = (per_slab + 255) / 256 * d.B * d.H >= 8 * 8 * 148 && per_slab >= 4096 && per_slab < (1LL << 30) ? 4 : 1;
            dim3 grid((unsigned)((per_slab + 256 * upt - 1) / (256 * upt)), (unsigned)(d.B * d.H));
            if (wide) quant_contig_kernel<BITS, T, WMAX><<<grid, 256, 0, st>>>(x, a->code, sc, mn, d, tpg, vec_ok, linear, upt);
            else quant_contig_kernel<BITS, T, 1><<<grid, 256, 0, st>>>(x, a->code, sc, mn, d, tpg, vec_ok, linear, upt);
            return check_launch();
        }
    }
    // groups along a strided axis, channels contiguous (keys in [T, D] order)
    if constexpr (sizeof(T) == 2) {
        const bool ok = a->x_sA == 1 && d.A % 128 == 0 && (reinterpret_cast<uintptr_t>(x) % 4 == 0) &&
                        d.x_sB % 2 == 0 && d.x_sH % 2 == 0 && d.x_sS % 2 == 0 && d.B * d.H <= 65535 &&
                        d.A / 128 <= 65535;
        if (ok) {
            const __half *xh = reinterpret_cast<const __half *>(x);
            __half *sh = reinterpret_cast<__half *>(sc), *mh = reinterpret_cast<__half *>(mn);
            const int64_t ng = d.S / G;
#define KVQ_LAUNCH_STRIDED(GG)                                                                     \
    {                                                                                              \
        using C = StridedCfg<BITS, GG>;                                                            \
        dim3 grid((unsigned)((ng + C::GPC - 1) / C::GPC), (unsigned)(d.A / 128), (unsigned)(d.B * d.H)); \
        if (rope) {                                                                                \
            grid.x = (unsigned)((ng + RopeCfg<BITS, GG>::GPC - 1) / RopeCfg<BITS, GG>::GPC);       \
            quant_rope_kernel<BITS, GG><<<grid, 256, 0, st>>>(xh, a->code, sh, mh, d, *rope);      \
        } else {                                                                                   \
            if (d.x_sS == 128) quant_strided_kernel<BITS, GG, true><<<grid, 256, 0, st>>>(xh, a->code, sh, mh, d); \
            else quant_strided_kernel<BITS, GG, false><<<grid, 256, 0, st>>>(xh, a->code, sh, mh, d); \
        }                                                                                          \
        return check_launch();                                                                     \
    }
            if constexpr (BITS == 3) {
                if (G == 11) KVQ_LAUNCH_STRIDED(11)
            } else {
                if (G == 32) KVQ_LAUNCH_STRIDED(32)
                if (G == 64) KVQ_LAUNCH_STRIDED(64)
                if (G == 128) KVQ_LAUNCH_STRIDED(128)
            }
#undef KVQ_LAUNCH_STRIDED
        }
    }
    if (rope) return KVQ_ERR_UNSUPPORTED;                      // rotation on the way in needs the strided-key layout
    const int64_t blocks = (total_words + 127) / 128;
    quant_generic_kernel<BITS, T><<<(unsigned)blocks, 128, 0, st>>>(x, a->code, sc, mn, d);
    return check_launch();
}

int quant_lastdim_impl(const kvq_quant_args *a, kvq_stream_t stream, const RopeTables *rope);

}  // namespace kvq

extern "C" int kvq_quant_lastdim(const kvq_quant_args *a, kvq_stream_t stream) {
    return kvq::quant_lastdim_impl(a, stream, nullptr);
}

int kvq::quant_lastdim_impl(const kvq_quant_args *a, kvq_stream_t stream, const RopeTables *rope) {
    using namespace kvq;
    if (!a) return KVQ_ERR_NULL;
    if (a->bits < 1 || a->bits > 4) return KVQ_ERR_BITS;
    if (a->B < 0 || a->H < 0 || a->A < 0 || a->S < 0) return KVQ_ERR_SHAPE;
    if (a->bits == 3) {
        if (a->group != 11) return KVQ_ERR_GROUP3;
        if (a->S % 11 != 0 && !a->ragged_tail) return KVQ_ERR_DIV11;
    } else {
        if (a->group <= 0 || a->S % a->group != 0) return KVQ_ERR_DIVGROUP;
        if (a->S % (32 / a->bits) != 0) return KVQ_ERR_DIVWORD;
    }
    if (a->B * a->H * a->A * a->S == 0) return KVQ_OK;
    if (!a->x || !a->code || !a->scale || !a->mn) return KVQ_ERR_NULL;
    if (a->bits == 3 && a->S % 11 != 0) {                      // the short-last-group extension
        if (rope) return KVQ_ERR_UNSUPPORTED;
        QuantDims r{a->B, a->H, a->A, a->S, a->x_sB, a->x_sH, a->x_sA, a->x_sS, a->c_sB, a->c_sH, a->c_sA,
                    a->z_sB, a->z_sH, a->z_sA, 11, a->scale_by_division ? 1 : 0};
        cudaStream_t rs = reinterpret_cast<cudaStream_t>(stream);
        return a->x_is_f32 ? launch_ragged3<float>(a, r, rs) : launch_ragged3<__half>(a, r, rs);
    }
    QuantDims d{a->B, a->H, a->A, a->S, a->x_sB, a->x_sH, a->x_sA, a->x_sS, a->c_sB, a->c_sH, a->c_sA,
                a->z_sB, a->z_sH, a->z_sA, a->group, a->scale_by_division ? 1 : 0};
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
#define KVQ_DISPATCH(BITS)                                                             \
    case BITS:                                                                         \
        return a->x_is_f32 ? launch_bits<BITS, float>(a, d, st, rope) : launch_bits<BITS, __half>(a, d, st, rope);
    switch (a->bits) {
        KVQ_DISPATCH(1)
        KVQ_DISPATCH(2)
        KVQ_DISPATCH(3)
        KVQ_DISPATCH(4)
    }
#undef KVQ_DISPATCH
    return KVQ_ERR_BITS;
}

// ---------------------------------------------------------------------------------------------
// Functional append forms: copy the previous tensors into the front of the outputs (strided device-to-device
// copies on the same stream), then quantize the new tokens in place behind them.
namespace kvq {
static int copy_rows(void *dst, size_t dst_pitch, const void *src, size_t src_pitch, size_t width, size_t rows,
                     cudaStream_t st) {
    if (width == 0 || rows == 0) return KVQ_OK;
    if (!src || !dst) return KVQ_ERR_NULL;
    return record_cuda_error(cudaMemcpy2DAsync(dst, dst_pitch, src, src_pitch, width, rows, cudaMemcpyDeviceToDevice, st));
}
}  // namespace kvq

extern "C" int kvq_append_k(const kvq_append_form_args *a, kvq_stream_t stream) {
    using namespace kvq;
    if (!a) return KVQ_ERR_NULL;
    if (a->bits < 1 || a->bits > 4) return KVQ_ERR_BITS;
    if (a->B < 0 || a->H < 0 || a->A < 0 || a->S < 0 || a->old_words < 0 || a->old_groups < 0) return KVQ_ERR_SHAPE;
    if (a->bits == 3 && a->group != 11) return KVQ_ERR_GROUP3;
    if (a->group <= 0) return KVQ_ERR_DIVGROUP;
    if (a->bits == 3) {
        if (a->S % 11 != 0) return KVQ_ERR_DIV11;
    } else {
        if (a->S % a->group != 0) return KVQ_ERR_DIVGROUP;
        if (a->S % (32 / a->bits) != 0) return KVQ_ERR_DIVWORD;
    }
    const int fpi = fields_per_word(a->bits);
    const int64_t new_words = a->S / fpi, new_groups = a->S / a->group;
    const int64_t rows = a->B * a->H * a->A, W = a->old_words + new_words, Gn = a->old_groups + new_groups;
    const size_t es = a->x_is_f32 ? 4 : 2;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    int rc = copy_rows(a->code, (size_t)W * 4, a->prev_code, (size_t)a->old_words * 4, (size_t)a->old_words * 4, (size_t)rows, st);
    if (rc) return rc;
    rc = copy_rows(a->scale, (size_t)Gn * es, a->prev_scale, (size_t)a->old_groups * es, (size_t)a->old_groups * es, (size_t)rows, st);
    if (rc) return rc;
    rc = copy_rows(a->mn, (size_t)Gn * es, a->prev_mn, (size_t)a->old_groups * es, (size_t)a->old_groups * es, (size_t)rows, st);
    if (rc) return rc;
    kvq_quant_args q{a->x, a->x_is_f32, a->B, a->H, a->A, a->S, a->x_sB, a->x_sH, a->x_sA, a->x_sS, a->group, a->bits, 1,
                     a->code ? a->code + a->old_words : nullptr, a->H * a->A * W, a->A * W, W,
                     a->scale ? static_cast<char *>(a->scale) + (size_t)a->old_groups * es : nullptr,
                     a->mn ? static_cast<char *>(a->mn) + (size_t)a->old_groups * es : nullptr,
                     a->H * a->A * Gn, a->A * Gn, Gn};
    return kvq_quant_lastdim(&q, stream);
}

extern "C" int kvq_append_v(const kvq_append_form_args *a, kvq_stream_t stream) {
    using namespace kvq;
    if (!a) return KVQ_ERR_NULL;
    if (a->bits < 1 || a->bits > 4) return KVQ_ERR_BITS;
    if (a->B < 0 || a->H < 0 || a->A < 0 || a->S < 0 || a->old_tokens < 0) return KVQ_ERR_SHAPE;
    if (a->bits == 3 && a->group != 11) return KVQ_ERR_GROUP3;
    if (a->group <= 0) return KVQ_ERR_DIVGROUP;
    if (a->bits == 3) {
        if (a->S % 11 != 0) return KVQ_ERR_DIV11;
    } else {
        if (a->S % a->group != 0) return KVQ_ERR_DIVGROUP;
        if (a->S % (32 / a->bits) != 0) return KVQ_ERR_DIVWORD;
    }
    const int fpi = fields_per_word(a->bits);
    const int64_t wpt = a->S / fpi, gpt = a->S / a->group;           // words / groups per token row
    const int64_t rows = a->B * a->H, Tt = a->old_tokens + a->A;
    const size_t es = a->x_is_f32 ? 4 : 2;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    int rc = copy_rows(a->code, (size_t)(Tt * wpt) * 4, a->prev_code, (size_t)(a->old_tokens * wpt) * 4,
                       (size_t)(a->old_tokens * wpt) * 4, (size_t)rows, st);
    if (rc) return rc;
    rc = copy_rows(a->scale, (size_t)(Tt * gpt) * es, a->prev_scale, (size_t)(a->old_tokens * gpt) * es,
                   (size_t)(a->old_tokens * gpt) * es, (size_t)rows, st);
    if (rc) return rc;
    rc = copy_rows(a->mn, (size_t)(Tt * gpt) * es, a->prev_mn, (size_t)(a->old_tokens * gpt) * es,
                   (size_t)(a->old_tokens * gpt) * es, (size_t)rows, st);
    if (rc) return rc;
    kvq_quant_args q{a->x, a->x_is_f32, a->B, a->H, a->A, a->S, a->x_sB, a->x_sH, a->x_sA, a->x_sS, a->group, a->bits, 1,
                     a->code ? a->code + a->old_tokens * wpt : nullptr, a->H * Tt * wpt, Tt * wpt, wpt,
                     a->scale ? static_cast<char *>(a->scale) + (size_t)(a->old_tokens * gpt) * es : nullptr,
                     a->mn ? static_cast<char *>(a->mn) + (size_t)(a->old_tokens * gpt) * es : nullptr,
                     a->H * Tt * gpt, Tt * gpt, gpt};
    return kvq_quant_lastdim(&q, stream);
}
