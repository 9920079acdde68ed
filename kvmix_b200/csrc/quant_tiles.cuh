// Pieces of the quantizer kernels that more than one kernel is made of: a run of contiguous groups, a tile of keys that are
// rotated on the way in, a word of the short-last-group extension, a chunk of a prompt's fp16 tails.  Their loads are plain ones and
// their pointers not __restrict__: see grid_wait().
#pragma once
#include "quant_core.cuh"

namespace kvq {

template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }

struct QuantDims {
    int64_t B, H, A, S;
    int64_t x_sB, x_sH, x_sA, x_sS;
    int64_t c_sB, c_sH, c_sA;
    int64_t z_sB, z_sH, z_sA;
    int group;
    int by_div;   // stored scale: 1 = (mx-mn)/qmax, 0 = (mx-mn) * fl32(1/qmax)
};

// ---------------------------------------------------------------------------------------------
// Contiguous groups.  A thread owns WPT consecutive words (E * WPT elements, 32 where the shapes allow: 64 bytes
// of loads in flight per thread, and the per-thread index arithmetic, division and shuffles spread over enough
// elements); tpg = group / (E * WPT) threads share a group.
template <int BITS, typename T, int WPT>
__device__ __forceinline__ void quant_contig_unit(const T *x, int32_t *code, T *scale, T *mn,
                                                  const QuantDims &d, int tpg, bool vec_ok, bool linear, int b, int h, int idx) {
    constexpr int E = fields_per_word(BITS);
    constexpr int EW = E * WPT;
    const int units_per_row = (int)(d.S / EW);
    const int total = (int)d.A * units_per_row;
    const bool active = idx < total;
    if (!active) idx = total - 1;  // keep the lane alive for the shuffles
    int a, u;
    if (linear) { a = 0; u = idx; }                      // rows of the slab are back to back in x, code and scale
    else { a = idx / units_per_row; u = idx - a * units_per_row; }
    const T *px = x + b * d.x_sB + h * d.x_sH + a * d.x_sA + (int64_t)u * EW;

    float v[EW];
    float lo, hi;
    bool have_range = false;
    if constexpr (sizeof(T) == 2 && (EW % 8 == 0)) {
        if (vec_ok) {
            // min / max in fp16x2 on the raw loads (exact: the data are fp16; NaN operands are skipped as by fminf):
            // one instruction per two elements instead of one per element
            __half2 lo2, hi2;
#pragma unroll
            for (int j = 0; j < EW / 8; ++j) {
                uint4 q = reinterpret_cast<const uint4 *>(px)[j];
                const __half2 *hp = reinterpret_cast<const __half2 *>(&q);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (j == 0 && k == 0) { lo2 = hp[0]; hi2 = hp[0]; }
                    else { lo2 = __hmin2(lo2, hp[k]); hi2 = __hmax2(hi2, hp[k]); }
                    float2 f = __half22float2(hp[k]);
                    v[j * 8 + 2 * k] = f.x;
                    v[j * 8 + 2 * k + 1] = f.y;
                }
            }
            lo = fminf(__low2float(lo2), __high2float(lo2));
            hi = fmaxf(__low2float(hi2), __high2float(hi2));
            have_range = true;
        } else {
#pragma unroll
            for (int i = 0; i < EW; ++i) v[i] = to_f32<T>(px[i]);
        }
    } else {
#pragma unroll
        for (int i = 0; i < EW; ++i) v[i] = to_f32<T>(px[i]);
    }
    if (!have_range) {
        lo = v[0];
        hi = v[0];
#pragma unroll
        for (int i = 1; i < EW; ++i) { lo = fminf(lo, v[i]); hi = fmaxf(hi, v[i]); }
    }
    for (int o = 1; o < tpg; o <<= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    constexpr int QMAX = (1 << BITS) - 1;
    const float sc = (hi - lo) / (float)QMAX;
    const float rinv = __frcp_rn(sc);                          // correctly rounded 1 / sc
    uint32_t word[WPT];
#pragma unroll
    for (int k = 0; k < (BITS == 3 ? WPT : 0); ++k) word[k] = quant_word<BITS>([&](int i) { return v[k * E + i]; }, lo, sc, rinv);
    if constexpr (BITS != 3) quant_words<BITS, WPT>([&](int k, int i) { return v[k * E + i]; }, lo, sc, rinv, word);
    if (active) {
        int32_t *pc = code + b * d.c_sB + h * d.c_sH + a * d.c_sA + u * WPT;
#pragma unroll
        for (int k = 0; k < WPT; ++k) pc[k] = (int32_t)word[k];
        if ((u & (tpg - 1)) == 0) {                           // tpg is a power of two
            const int64_t zo = b * d.z_sB + h * d.z_sH + a * d.z_sA + (u >> (__ffs(tpg) - 1));
            scale[zo] = from_f32<T>(stored_scale<QMAX>(hi - lo, sc, d.by_div));
            mn[zo] = from_f32<T>(lo);
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Rotary embedding applied while loading (prefill of keys straight from the k_proj output): element (b, s, c) of the
// cos / sin tables at b * r_sB + s * r_sS + c, fp16.  HF's rotate_half form (the one upstream's model files import):
// out[c] = k[c] * cos[c] + rot[c] * sin[c] with rot = (-k[c + 64], k[c - 64]) for c < 64 / c >= 64, every product and
// the sum rounded to fp16 as the framework's fp16 tensor arithmetic rounds them.
struct RopeTables {
    const __half *cos, *sin;
    int64_t r_sB, r_sS;
};


// Keys straight from the projection.  A CTA rotates 128 tokens (132 for groups of 11) x 128 channels into shared memory -- a
// lane takes four channels of a row, the rotation partner (64 channels away) is a shuffle, so rows and table rows are
// read once -- and then works parts of 32 (11) tokens of a channel pair from there; groups of 64 and 128 tokens meet over
// shared memory.  Loops stay rolled: with a warp's 32 tokens in registers and every word unrolled, tie path included, the same
// work took 46 .. 71 us, waiting for instructions; read from global memory twice and rotated twice (a thread per
// pair and group, four loads an element pair) 38 us.  2 x 8 kv heads x 8191 tokens, group 64, 4 bits: 22 us (with values
// and tails 37.1 us in three launches, 26.7 in one).
template <int BITS, int G>
struct RopeCfg {
    static constexpr int FPI = fields_per_word(BITS);
    static constexpr int PT = G == 11 ? 11 : 32;              // tokens of a part
    static constexpr int NP = G == 11 ? 12 : 4;               // parts of a tile
    static constexpr int TOK = NP * PT;                       // tokens of a tile: 132 / 128
    static constexpr int PPG = G > 32 ? G / 32 : 1;           // parts of a group
    static constexpr int GPC = NP / PPG;                      // groups of a tile
    static constexpr int WPP = PT / FPI;                      // words of a part: 4 / 2 / 1 / 1
    static constexpr int WPC = NP * WPP, WPAD = WPC + 1;
};

template <int BITS, int G>
__device__ __forceinline__ void quant_rope_tile(const __half *x, int32_t *code, __half *scale, __half *mn,
                                                const QuantDims &d, const RopeTables &rope, int tile, int bh) {
    using C = RopeCfg<BITS, G>;
    constexpr int QMAX = (1 << BITS) - 1;
    __shared__ __align__(16) __half2 s_tile[C::TOK * 64];
    __shared__ int32_t s_code[128 * C::WPAD];
    __shared__ __half s_scale[128 * (C::GPC + 2)], s_mn[128 * (C::GPC + 2)];
    __shared__ __half2 s_lo[C::PPG > 1 ? C::NP * 64 : 1], s_hi[C::PPG > 1 ? C::NP * 64 : 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t b = bh / (int)d.H, h = bh - (int)b * (int)d.H;
    const int64_t g0 = (int64_t)tile * C::GPC, n_groups = d.S / G;
    const int groups_here = (int)min((int64_t)C::GPC, n_groups - g0), tokens = groups_here * G;
    {
        const __half *px = x + b * d.x_sB + h * d.x_sH + g0 * G * d.x_sS + 4 * lane;
        const __half *pc = rope.cos + b * rope.r_sB + g0 * G * rope.r_sS + 4 * lane;
        const __half *ps = rope.sin + b * rope.r_sB + g0 * G * rope.r_sS + 4 * lane;
        const uint32_t turn = lane < 16 ? 0x80008000u : 0u;   // rot = (-k[c + 64], k[c - 64])
        auto h2 = [](const uint32_t &u) { return *reinterpret_cast<const __half2 *>(&u); };
        constexpr int NB = 4;                                 // rows in flight per warp (x 3 loads)
#pragma unroll 1
        for (int t0 = warp; t0 < tokens; t0 += 8 * NB) {
            uint2 k[NB], cs[NB], sn[NB];
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                const int64_t t = min(t0 + 8 * i, tokens - 1);
                k[i] = *reinterpret_cast<const uint2 *>(px + t * d.x_sS);
                cs[i] = *reinterpret_cast<const uint2 *>(pc + t * rope.r_sS);
                sn[i] = *reinterpret_cast<const uint2 *>(ps + t * rope.r_sS);
            }
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                const uint32_t r0 = __shfl_xor_sync(0xffffffffu, k[i].x, 16) ^ turn, r1 = __shfl_xor_sync(0xffffffffu, k[i].y, 16) ^ turn;
                const __half2 o0 = __hadd2_rn(__hmul2_rn(h2(k[i].x), h2(cs[i].x)), __hmul2_rn(h2(r0), h2(sn[i].x)));
                const __half2 o1 = __hadd2_rn(__hmul2_rn(h2(k[i].y), h2(cs[i].y)), __hmul2_rn(h2(r1), h2(sn[i].y)));
                if (t0 + 8 * i < tokens) {
                    uint2 o;
                    o.x = *reinterpret_cast<const uint32_t *>(&o0);
                    o.y = *reinterpret_cast<const uint32_t *>(&o1);
                    *reinterpret_cast<uint2 *>(&s_tile[(t0 + 8 * i) * 64 + 2 * lane]) = o;
                }
            }
        }
    }
    __syncthreads();
    const int pair = threadIdx.x & 63, parts = groups_here * C::PPG;
    // min / max of a part in fp16x2 (exact: the data are fp16; NaN operands are skipped as by fminf)
    auto range = [&](int part, __half2 &lo2, __half2 &hi2) {
        const __half2 *t = s_tile + part * C::PT * 64 + pair;
        lo2 = hi2 = t[0];
#pragma unroll
        for (int i = 1; i < C::PT; ++i) { const __half2 v = t[i * 64]; lo2 = __hmin2(lo2, v); hi2 = __hmax2(hi2, v); }
    };
    if constexpr (C::PPG > 1) {                               // four parts: one per thread
        const int part = threadIdx.x >> 6;
        if (part < parts) {
            __half2 lo2, hi2;
            range(part, lo2, hi2);
            s_lo[part * 64 + pair] = lo2;
            s_hi[part * 64 + pair] = hi2;
        }
        __syncthreads();
    }
#pragma unroll 1
    for (int part = threadIdx.x >> 6; part < parts; part += 4) {
        __half2 lo2, hi2;
        if constexpr (C::PPG > 1) {
            const int p0 = part / C::PPG * C::PPG;
            lo2 = s_lo[p0 * 64 + pair];
            hi2 = s_hi[p0 * 64 + pair];
#pragma unroll
            for (int p = 1; p < C::PPG; ++p) { lo2 = __hmin2(lo2, s_lo[(p0 + p) * 64 + pair]); hi2 = __hmax2(hi2, s_hi[(p0 + p) * 64 + pair]); }
        } else {
            range(part, lo2, hi2);
        }
        const float lo0 = __low2float(lo2), lo1 = __high2float(lo2), hi0 = __low2float(hi2), hi1 = __high2float(hi2);
        const float sc0 = (hi0 - lo0) / (float)QMAX, sc1 = (hi1 - lo1) / (float)QMAX;
        const float ri0 = __frcp_rn(sc0), ri1 = __frcp_rn(sc1);     // correctly rounded reciprocals
#pragma unroll 1
        for (int w = 0; w < C::WPP; ++w) {
            const __half2 *t = s_tile + (part * C::PT + w * C::FPI) * 64 + pair;
            __half2 raw[C::FPI];
#pragma unroll
            for (int i = 0; i < C::FPI; ++i) raw[i] = t[i * 64];
            s_code[(2 * pair) * C::WPAD + part * C::WPP + w] = (int32_t)quant_word<BITS>([&](int i) { return __low2float(raw[i]); }, lo0, sc0, ri0);
            s_code[(2 * pair + 1) * C::WPAD + part * C::WPP + w] = (int32_t)quant_word<BITS>([&](int i) { return __high2float(raw[i]); }, lo1, sc1, ri1);
        }
        if (part % C::PPG == 0) {
            const int g = part / C::PPG, o = (2 * pair) * (C::GPC + 2) + g;
            s_scale[o] = __float2half_rn(stored_scale<QMAX>(hi0 - lo0, sc0, d.by_div));
            s_scale[o + C::GPC + 2] = __float2half_rn(stored_scale<QMAX>(hi1 - lo1, sc1, d.by_div));
            s_mn[o] = __float2half_rn(lo0);
            s_mn[o + C::GPC + 2] = __float2half_rn(lo1);
        }
    }
    __syncthreads();
    const int words_here = groups_here * (G / C::FPI);
    int32_t *dc = code + b * d.c_sB + h * d.c_sH + g0 * (G / C::FPI);
    const int64_t zo = b * d.z_sB + h * d.z_sH + g0;
    for (int i = threadIdx.x; i < 128 * C::WPC; i += 256) {
        const int ch = i / C::WPC, w = i % C::WPC;
        if (w < words_here) dc[ch * d.c_sA + w] = s_code[ch * C::WPAD + w];
    }
    for (int i = threadIdx.x; i < 128 * C::GPC; i += 256) {
        const int ch = i / C::GPC, g = i % C::GPC;
        if (g < groups_here) {
            scale[zo + ch * d.z_sA + g] = s_scale[ch * (C::GPC + 2) + g];
            mn[zo + ch * d.z_sA + g] = s_mn[ch * (C::GPC + 2) + g];
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Extension without an upstream counterpart: 3-bit groups of 11 along an axis whose length is not a multiple of 11
// (3-bit values at head_dim 128).  Every group is one word; the last group holds S % 11 elements, its unused fields
// stay 0.  Upstream's 3-bit group rule otherwise (quantization_cuda.cu:553-596, :612-626).  One thread per word.
template <typename T>
__device__ __forceinline__ void quant_ragged3_word(const T *x, int32_t *code, T *scale, T *mn,
                                                   const QuantDims &d, int64_t idx) {
    const int64_t words_per_row = (d.S + 10) / 11;
    const int64_t total = d.B * d.H * d.A * words_per_row;
    if (idx >= total) return;
    const int64_t row = idx / words_per_row, w = idx % words_per_row;
    const int64_t a = row % d.A, h = (row / d.A) % d.H, b = row / (d.A * d.H);
    const T *px = x + b * d.x_sB + h * d.x_sH + a * d.x_sA + w * 11 * d.x_sS;
    const int n = (int)min((int64_t)11, d.S - w * 11);
    float v[11], lo = 3.402823466e+38f, hi = -3.402823466e+38f;
#pragma unroll
    for (int i = 0; i < 11; ++i) {
        v[i] = i < n ? to_f32<T>(px[i * d.x_sS]) : 0.f;
        if (i < n) { lo = fminf(lo, v[i]); hi = fmaxf(hi, v[i]); }
    }
    const float range = hi - lo, sc = range / 7.0f;
    uint32_t word = 0;
#pragma unroll
    for (int i = 0; i < 11; ++i)
        if (i < n) word |= (uint32_t)round_code((v[i] - lo) / sc, i < 10 ? 7 : 3) << (i < 10 ? 3 * i : 30);
    code[b * d.c_sB + h * d.c_sH + a * d.c_sA + w] = (int32_t)word;
    const int64_t zo = b * d.z_sB + h * d.z_sH + a * d.z_sA + w;
    scale[zo] = from_f32<T>(stored_scale<7>(range, sc, d.by_div));
    mn[zo] = from_f32<T>(lo);
}

// ---------------------------------------------------------------------------------------------
// Prompt tails: tokens [nk, L) of the keys (rotated on the way when tables are given) and [nv, L) of the values go to
// rows 0.. of the fp16 rings.  One thread per (b, h, token, 8-channel chunk j < 8) handles chunk j and chunk j + 8,
// the rotation partners.
__device__ __forceinline__ void prefill_tail_chunk(const kvq_prefill_args &a, int64_t i) {
    const int nkt = a.L - a.nk, nvt = a.L - a.nv;
    const int64_t per_k = (int64_t)a.B * a.Hkv * nkt * 8, per_v = (int64_t)a.B * a.Hkv * nvt * 8;
    if (i >= per_k + per_v) return;
    const bool is_v = i >= per_k;
    if (is_v) i -= per_k;
    const int j = (int)(i & 7);
    const int n = is_v ? nvt : nkt;
    const int64_t r = (i >> 3) % n, bh = (i >> 3) / n;
    const int b = (int)(bh / a.Hkv), h = (int)(bh % a.Hkv);
    if (is_v) {
        const __half *src = static_cast<const __half *>(a.v) + b * a.v_sB + (a.nv + r) * a.v_sT + h * a.v_sH;
        __half *dst = static_cast<__half *>(a.vfull) + b * a.vf_sB + h * a.vf_sH + r * a.vf_sT;
        const uint4 lo = reinterpret_cast<const uint4 *>(src)[j], hi = reinterpret_cast<const uint4 *>(src)[j + 8];
        reinterpret_cast<uint4 *>(dst)[j] = lo;
        reinterpret_cast<uint4 *>(dst)[j + 8] = hi;
        return;
    }
    const int64_t t = a.nk + r;
    const __half *src = static_cast<const __half *>(a.k) + b * a.k_sB + t * a.k_sT + h * a.k_sH;
    __half *dst = static_cast<__half *>(a.kfull) + b * a.kf_sB + h * a.kf_sH + r * a.kf_sT;
    uint4 lo = reinterpret_cast<const uint4 *>(src)[j], hi = reinterpret_cast<const uint4 *>(src)[j + 8];
    if (a.cos) {
        const __half *pc = static_cast<const __half *>(a.cos) + b * a.r_sB + t * a.r_sT;
        const __half *ps = static_cast<const __half *>(a.sin) + b * a.r_sB + t * a.r_sT;
        const uint4 cl = reinterpret_cast<const uint4 *>(pc)[j], ch = reinterpret_cast<const uint4 *>(pc)[j + 8];
        const uint4 sl = reinterpret_cast<const uint4 *>(ps)[j], sh = reinterpret_cast<const uint4 *>(ps)[j + 8];
        uint4 ol, oh;
        const __half2 *kl = reinterpret_cast<const __half2 *>(&lo), *kh = reinterpret_cast<const __half2 *>(&hi);
        const __half2 *c0 = reinterpret_cast<const __half2 *>(&cl), *c1 = reinterpret_cast<const __half2 *>(&ch);
        const __half2 *s0 = reinterpret_cast<const __half2 *>(&sl), *s1 = reinterpret_cast<const __half2 *>(&sh);
        __half2 *pl = reinterpret_cast<__half2 *>(&ol), *ph = reinterpret_cast<__half2 *>(&oh);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            pl[q] = __hadd2_rn(__hmul2_rn(kl[q], c0[q]), __hmul2_rn(__hneg2(kh[q]), s0[q]));
            ph[q] = __hadd2_rn(__hmul2_rn(kh[q], c1[q]), __hmul2_rn(kl[q], s1[q]));
        }
        lo = ol;
        hi = oh;
    }
    reinterpret_cast<uint4 *>(dst)[j] = lo;
    reinterpret_cast<uint4 *>(dst)[j + 8] = hi;
}

}  // namespace kvq
