// The arithmetic core of the group quantizer, shared by the stand-alone quantizer kernels (quant.cu) and by the
// attention kernels' fused cache update (attn_update.cuh): bit-identical to upstream
// quant_cuda/csrc/quantization_cuda.cu:553-596 with IEEE division.
#pragma once
#include "common.cuh"

namespace kvq {

// q = clamp(roundf(n), 0, emax) for n >= 0 or NaN.  n - trunc(n) is exact for these magnitudes,
// so comparing the fraction with 0.5 is roundf's half-away-from-zero rule.
__device__ __forceinline__ int round_code(float n, int emax) {
    int k = (n == n) ? __float2int_rz(n) : 0;
    float frac = n - (float)k;
    k += (frac >= 0.5f) ? 1 : 0;
    return max(0, min(k, emax));
}

// Two fp32 operations in one instruction (each rounded by itself, as the scalar forms are).
__device__ __forceinline__ unsigned long long f32x2(float x, float y) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 f32x2_split(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ unsigned long long add_f32x2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long mul_f32x2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long fma_f32x2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// max(t, |x|, |y|), NaN if any is
__device__ __forceinline__ float max_abs(float t, float x, float y) {
    float r;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(t), "f"(fabsf(x)), "f"(fabsf(y)));
    return r;
}

// One packed word of E = fields_per_word(BITS) consecutive elements get(0..E-1) of a group with minimum lo, scale
// sc and rinv = fl(1/sc), bit-identical to OR_i clamp(roundf((v_i - lo) / sc), 0, emax_i) << shift_i with IEEE
// division -- without a division, an int conversion or a clamp per element:
//   m  = fma(a, rinv, 1.5 * 2^23), a = v - lo     the addition rounds a*rinv to the nearest integer (low mantissa bits)
//   ny = 1.5 * 2^23 - m                          minus that integer as a float (exact)
//   e  = fma(a, rinv, ny)                        signed distance of a*rinv from it, in [-0.5, 0.5]
// a*rinv and the IEEE quotient differ by < 1.3e-7 relative (< 2e-6 for codes up to 15), so unless |e| is within
// 1e-5 of 0.5 both round to the same integer, whatever the tie rule; 0 <= a*rinv <= qmax (1 + 2e-7) keeps it in
// range.  The word is summed in two fp32 chunks of <= 17 bits (exact) and converted once.  If any element is near
// a tie or not finite (constant group: 0 * inf), the word is put together element by element and only the elements in
// question are divided: fp16 data tie often enough that some lane of every eighth warp gets here, and dividing for all
// elements of the word was a fifth of the quantizers' instructions (1, 2 and 4 bits).
// Elements go in pairs (f32x2), the tie test is one three-input maximum a pair.  16 x 32 x 8192 x 128 fp16:
// keys (2 bits, groups of 32 tokens) 348 -> 310 us, values (4 bits, groups of 32) 309 -> 296 us; words put together by a byte permute
// keys 304 -> 282 us (which look for ties once a word and channel); that, one look for ties a thread and several units a thread
// values 291 -> 252 us.
// 3-bit words are worked one element at a time and divided whole: eleven fields in two chunks split badly into pairs, and
// their lone word a group leaves too little between two tie tests (keys 457 us in pairs with single divisions, 426 us so;
// contiguous groups 464 and 436 us).
constexpr float kQuantMagic = 12582912.0f;                 // 1.5 * 2^23
constexpr float kQuantTie = 0.49999f;                      // |e| up to here: no tie

// 1, 2 and 4 bits: the word without its ties; `worst` is the largest |e| (NaN where an element is not finite).  The two chunks are
// summed on top of 2^23, so that their 16 bits are the low halves of two fp32 words: one byte permute puts them together (two
// conversions, a shift and an or before).
template <int BITS, typename Get>
__device__ __forceinline__ uint32_t quant_word_fast(Get get, float lo, float rinv, float &worst) {
    constexpr int E = fields_per_word(BITS), NLO = E / 2;      // fields in the low chunk: 16 bits
    const unsigned long long nlo2 = f32x2(-lo, -lo), rinv2 = f32x2(rinv, rinv), magic2 = f32x2(kQuantMagic, kQuantMagic), minus2 = f32x2(-1.f, -1.f);
    unsigned long long wl2 = f32x2(8388608.f, 0.f), wh2 = wl2;
    worst = 0.f;
    auto weight = [](int i) -> float { return (float)(1 << (BITS * (i < NLO ? i : i - NLO))); };   // of field i in its chunk
#pragma unroll
    for (int i = 0; i < E; i += 2) {
        const unsigned long long a = add_f32x2(f32x2(get(i), get(i + 1)), nlo2);
        const unsigned long long m = fma_f32x2(a, rinv2, magic2);
        const unsigned long long ny = fma_f32x2(m, minus2, magic2);
        const float2 e = f32x2_split(fma_f32x2(a, rinv2, ny));
        worst = max_abs(worst, e.x, e.y);
        if (i < NLO) wl2 = fma_f32x2(ny, f32x2(-weight(i), -weight(i + 1)), wl2);
        else wh2 = fma_f32x2(ny, f32x2(-weight(i), -weight(i + 1)), wh2);
    }
    const float2 l2 = f32x2_split(wl2), h2 = f32x2_split(wh2);
    return __byte_perm(__float_as_uint(l2.x + l2.y), __float_as_uint(h2.x + h2.y), 0x5410);
}

// The word element by element, those near a tie or not finite divided.
template <int BITS, typename Get>
__device__ __forceinline__ uint32_t quant_word_ties(Get get, float lo, float sc, float rinv) {
    constexpr int E = fields_per_word(BITS), QMAX = (1 << BITS) - 1;
    uint32_t word = 0;
#pragma unroll
    for (int i = 0; i < E; ++i) {
        const float a = get(i) - lo, m = fmaf(a, rinv, kQuantMagic), e = fmaf(a, rinv, kQuantMagic - m);
        int q = min((int)(__float_as_uint(m) & 31u), QMAX);        // the integer sits in the low mantissa bits
        if (!(fabsf(e) <= kQuantTie)) q = round_code(a / sc, QMAX);
        word |= (uint32_t)q << (BITS * i);
    }
    return word;
}

template <int BITS, typename Get>
__device__ __forceinline__ uint32_t quant_word(Get get, float lo, float sc, float rinv) {
    if constexpr (BITS == 3) {
        constexpr int E = fields_per_word(BITS);
        float wl = 0.f, wh = 0.f, worst = 0.f;
#pragma unroll
        for (int i = 0; i < E; ++i) {
            const float a = get(i) - lo, m = fmaf(a, rinv, kQuantMagic);
            float yr = m - kQuantMagic;
            const float e = fmaf(a, rinv, -yr);
            worst = max_abs(worst, e, e);
            if (i == 10) yr = fminf(yr, 3.f);                  // the 11th code of a 3-bit group has two bits
            if (i < 5) wl = fmaf(yr, (float)(1 << (3 * i)), wl);
            else wh = fmaf(yr, (float)(1 << (i < 10 ? 3 * (i - 5) : 15)), wh);
        }
        if (worst <= kQuantTie) return __float2uint_rz(wl) | (__float2uint_rz(wh) << 15);
        uint32_t word = 0;
#pragma unroll
        for (int i = 0; i < E; ++i) word |= (uint32_t)round_code((get(i) - lo) / sc, i < 10 ? 7 : 3) << (i < 10 ? 3 * i : 30);
        return word;
    } else {
        float worst;
        const uint32_t word = quant_word_fast<BITS>(get, lo, rinv, worst);
        if (worst <= kQuantTie) return word;
        return quant_word_ties<BITS>(get, lo, sc, rinv);
    }
}

// N words of one group (1, 2 or 4 bits), get(k, i) element i of word k: one look for ties at all of them.
template <int BITS, int N, typename Get>
__device__ __forceinline__ void quant_words(Get get, float lo, float sc, float rinv, uint32_t (&word)[N]) {
    float worst[N], all = 0.f;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        word[k] = quant_word_fast<BITS>([&](int i) { return get(k, i); }, lo, rinv, worst[k]);
        all = max_abs(all, worst[k], worst[k]);
    }
    if (all <= kQuantTie) return;
#pragma unroll
    for (int k = 0; k < N; ++k)
        if (!(worst[k] <= kQuantTie)) word[k] = quant_word_ties<BITS>([&](int i) { return get(k, i); }, lo, sc, rinv);
}

template <int QMAX>
__device__ __forceinline__ float stored_scale(float range, float quotient, int by_div) {
    return by_div ? quotient : __fmul_rn(range, 1.0f / (float)QMAX);
}

}  // namespace kvq
