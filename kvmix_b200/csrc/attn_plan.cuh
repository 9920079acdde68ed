// Work plan of the tensor-core attention kernels: which tokens of which head a CTA scores.
//
// The token axis of every head (a query head, or the group of query heads that share a kv head) is cut into
// units of `unit` tokens (a warp's key tile: 256, or four of them for 3-bit keys: 352 = 4 x 88, whichever tile the loops load); a head has
// uph = ceil(T / unit) units, the last one possibly short.  One CTA works one segment = a run of units of one head:
//   * the first n_whole CTAs take one whole head each (only when a head fits the score buffer); n_whole is a multiple
//     of the number of SMs, so these CTAs load all SMs alike;
//   * every remaining head (n_cut of them) is cut into k segments of seg_units units (the last one shorter), launched
//     after the whole heads, first segments of all heads first.  k is chosen so that these smaller CTAs, which the
//     hardware hands to whichever slot frees up, finish as early as possible: the last wave of a grid is then made of
//     short CTAs and fills all slots, whatever the number of heads.
// A head cut into several segments is merged by the CTA that finishes last (per-head counter), in segment order, so
// results do not depend on timing.
#pragma once
#include <stdint.h>

namespace kvq {

// Division by an invariant integer (Granlund and Montgomery, 1994), 1 .. 2^31, of numbers below 2^31: a high product, an addition and a shift where the compiler's
// division takes some twenty-five instructions, several of them in a row at the start of every CTA.
struct FastDiv {
    uint32_t mul, shr, d;
#ifdef __CUDACC__
    __device__ __forceinline__ uint32_t operator()(uint32_t n) const { return (__umulhi(n, mul) + n) >> shr; }
#endif
};
inline FastDiv fast_div(uint32_t d) {
    uint32_t s = 0;
    while (s < 31 && (1u << s) < d) ++s;
    return {(uint32_t)((((uint64_t)1 << 32) * (((uint64_t)1 << s) - d)) / d + 1), s, d};
}

struct AttnPlan {
    int unit;            // tokens per unit
    int uph;             // units per head
    int n_whole;         // CTAs (= heads) that take a whole head
    int n_cut;           // heads that are cut
    int k;               // segments per cut head (1: a whole head per CTA here too)
    int seg_units;       // units per segment of a cut head
    int n_scores;        // most tokens in a segment, rounded up to 32
    int warps;           // warps of a CTA: 8 (two CTAs to an SM) or 4 (three or four)
    int ks_log2;         // the channels of a key tile are shared by 1 << ks_log2 warps (partial scores, summed by the softmax)
    // how a CTA finds its place (plan_place): heads (or groups of them) per sequence, and those of a kv head
    FastDiv by_cut, by_seq, by_kv;
    int rep;             // query heads per kv head
};

constexpr int kSmCount = 148;
constexpr int kPlanSlots = 2 * kSmCount;       // resident CTAs: two of eight warps per SM
constexpr int kPlanWarps = 8;
constexpr int kWholeWave = 6 * kSmCount;       // grouped kernel: whole head groups in multiples of three waves
// One partial result of a cut head: 128 accumulators, the segment's maximum and sum, padded so that rows stay 16-byte
// aligned (the merge reads them with 128-bit loads).
constexpr int kPartStride = 128 + 4;
constexpr int kMaxCtaRounds = 8;       // cut heads are never spread over more CTAs than this many waves (bounds the workspace)

inline int plan_round32(int n) { return (n + 31) / 32 * 32; }

// Channel split of a segment's key tiles.  A warp walks a tile's 128 channels in four steps of 32; where a segment has fewer
// tiles than the CTA has warps, 2 or 4 warps share a tile's channels and each leaves partial scores.  Steps a warp takes
// (x 2), with about half a step's time of per-tile overhead; `max_scores` bounds the score buffer (tokens x splits).
inline int plan_key_steps(int n, int tile, int ks_log2, int warps = kPlanWarps) {
    const int tiles = (n + tile - 1) / tile;
    const int passes = ((tiles << ks_log2) + warps - 1) / warps;
    return passes * ((8 >> ks_log2) + 1);
}
inline int plan_key_split(int n, int tile, int max_scores, int warps = kPlanWarps) {
    int best = 0;
    for (int l = 1; l <= 2; ++l)
        if ((plan_round32(n) << l) <= max_scores && plan_key_steps(n, tile, l, warps) < plan_key_steps(n, tile, best, warps)) best = l;
    return best;
}

// SM cycles a segment of n tokens takes (one of two CTAs on its SM; measured with clock stamps inside the kernels on
// B200): 850 per two half-steps of keys, 850 per 32 tokens of values a warp works, the softmax, and 5500 for
// the launch, the ring fill, the fp16 tails and the final sum.
inline long long plan_segment_cycles(int n, int tile, int max_scores) {
    const int key = plan_key_steps(n, tile, plan_key_split(n, tile, max_scores)) * 850;
    const int val = (n + 32 * kPlanWarps - 1) / (32 * kPlanWarps) * 850;
    return key + val + 1500 + n / 2 + 5500;
}
// What cutting a head adds to its last CTA: publishing the partials and the merge of k of them.
inline long long plan_merge_cycles(int k) { return k > 1 ? 2500 + 40LL * k : 0; }

// Whole heads for more than half of the SMs and no more than there are: a CTA that has its SM to itself takes this percentage of the time the
// model gives it, and halves of all heads would only put two on it and a merge behind.  Up to 98 heads three pieces of each also fit one
// round, the last ones short, which is the better form from some 1200 tokens on (80); 3-bit keys are counted dearer than they are next to
// what a CTA does once (70).  Every form timed at 75 .. 148 heads x 350 .. 7000 tokens x 2, 4 and 3-bit keys, one head and four a CTA
// (770 points): 0.942 of the time of the plan without this rule, no point more than 1 % slower, 0.7 % from the best form of each point on
// average (us, whole and halves, whole taken: 128 heads of 1023 tokens, 2 bits 10.7 and 13.1, 3-bit keys 12.9 and 14.6, of 2000 18.4 and
// 20.7; 128 groups of 4 heads x 1023, 4 bits 14.2 and 18.1; whole and thirds, thirds taken: 96 groups x 1700, 4 bits 17.0 and 15.3).
// From some 2500 tokens on halves are taken although whole heads would be up to 4 % faster (128 heads of 4096, 2 bits 22.7 and 23.1, 3-bit
// keys 28.7 and 30.0): with a long fp16 tail they are the slower form (128 heads on 32 kv heads of 3001 tokens, 600 of them fp16, three
// layers 79.8 us whole, 76.8 halved).
inline int plan_lone_percent(long long heads, int unit) { return unit % 11 == 0 ? 70 : 3 * heads <= kPlanSlots ? 80 : 77; }
inline bool plan_lone(long long ctas, int k) { return k == 1 && ctas <= kSmCount && 2 * ctas > kSmCount; }
// Whole heads for all SMs but a few are not launched early: CTAs that are placed while those of the launch before still hold some SMs come to
// lie two to an SM, and no SM is left over to make up for it (148 heads whole, launched early / ordinarily: 1.11 of the time on average
// over 350 .. 6000 tokens, 148 groups of four heads 1.17; 144: 1.02; 128: 0.99).
inline bool plan_early(const AttnPlan &p) {
    const long long ctas = p.n_whole + (long long)p.n_cut * p.k;
    return !(p.k == 1 && ctas > kSmCount * 7 / 8 && ctas <= kSmCount);
}

// Pieces a head is cut into where `heads` of them (fewer than SMs) are left behind whole ones: the SM that gets most of the pieces
// finishes last; a piece costs its tokens and some 600 more, one whole head by itself on its SM `lone` percent of that.
inline int plan_left_pieces(int T, int unit, int heads, int lone) {
    if (heads == 0) return 1;
    const int uph = (T + unit - 1) / unit;
    int best_k = 1;
    long long best = (T + 600) * (long long)lone / 100;
    for (int k = 2; k <= 8 && k <= uph; ++k) {
        const int su = (uph + k - 1) / k;
        const long long cost = (long long)((heads * k + kSmCount - 1) / kSmCount) * (su * unit + 600) + 200;
        if ((uph + su - 1) / su == k && cost < best) { best = cost; best_k = k; }
    }
    return best_k;
}

inline void plan_finish(AttnPlan &p, int T, int tile, int max_scores) {
    long long ns = (long long)(p.n_whole ? p.uph : p.seg_units) * p.unit;
    if (ns > T) ns = T;
    p.n_scores = plan_round32((int)ns);
    p.ks_log2 = plan_key_split((int)ns, tile, max_scores, p.warps);
}

// heads: number of heads (or head groups); tile: tokens of a warp's key tile; max_scores: tokens the score buffer holds.
inline AttnPlan make_attn_plan(int T, int unit, int tile, int max_scores, long long heads) {
    AttnPlan p;
    p.unit = unit;
    p.warps = kPlanWarps;
    p.uph = (T + unit - 1) / unit;
    const int max_units = max_scores / unit;
    const bool whole_ok = T <= max_units * unit;
    p.n_whole = (int)(whole_ok ? (heads / kWholeWave) * kWholeWave : 0);
    p.n_cut = (int)(heads - p.n_whole);
    p.k = 1;
    p.seg_units = p.uph;
    if (p.n_cut > 0) {
        // candidates: segments of su units; estimated finish = rounds of CTAs x cycles of one + merge
        long long best = -1;
        for (int su = whole_ok ? p.uph : max_units; su >= 1; --su) {
            const int k = (p.uph + su - 1) / su;
            const long long ctas = (long long)p.n_cut * k;
            if (ctas > (long long)kMaxCtaRounds * kPlanSlots && best >= 0) break;
            const long long rounds = (ctas + kPlanSlots - 1) / kPlanSlots;
            const int n = su * unit < T ? su * unit : T;
            long long cost = rounds * plan_segment_cycles(n, tile, max_scores) + plan_merge_cycles(k);
            if (plan_lone(ctas, k)) cost = cost * plan_lone_percent(ctas, unit) / 100;
            if (best < 0 || cost < best) {
                best = cost;
                p.k = k;
                p.seg_units = su;
            }
        }
        p.seg_units = (p.uph + p.k - 1) / p.k;                                   // even the segments out
        p.k = (p.uph + p.seg_units - 1) / p.seg_units;
    }
    plan_finish(p, T, tile, max_scores);
    return p;
}

// The kernel with one query head per CTA, which also comes with four warps per CTA.  narrow_max: most tokens of a segment of those (a
// multiple of the unit); narrow_split: scores that leave room for four of them on an SM; wide_from: tokens from which eight warps
// a CTA pay up to six and a half heads an SM.
//
// More heads than eight-warp slots: the multiple of the SM count whole, the others cut (us on B200, whole heads in multiples of 888
// and eight warps for all that is cut -> this; 4096 tokens: 448 heads 2 bits 78 -> 70, 640 heads 99 -> 91, 1280 heads 173 ->
// 150, 3-bit keys 1536 heads 260 -> 233; 7000 tokens, 4 bits: 896 heads 235 -> 208, 2048 heads 488 -> 444).  What a CTA does once
// (addresses, ring fill, tails, sums: 20k of the 72k warp instructions of a head of 4096 tokens) is done by half as many warps
// in the four-warp form, so it is the better one where there are many CTAs or short ones: 300 tokens 0.76 .. 0.9 of the eight-warp
// form's time, 2000 tokens 0.9 .. 1.0; at 4096 tokens 320 and 448 heads take 1.10 .. 1.16 of it, 1024 heads 0.95 .. 0.98, 1280 heads 0.92.
inline AttnPlan make_attn_plan_mma(int T, int unit, int tile, int max_scores, long long heads, int narrow_max, int narrow_split, int wide_from) {
    const int wide_max = max_scores / unit * unit;
    const bool many = heads > kPlanSlots;
    // between one and two heads an SM, too long for the eight-warp form whole: four-warp quarters (256 heads of 8000 tokens, 3-bit keys:
    // 106 -> 96 us against two eight-warp halves)
    const bool quarters = !many && heads > kSmCount && T > wide_max;
    if (T > narrow_max || !(many || quarters)) return make_attn_plan(T, unit, tile, max_scores, heads);
    AttnPlan p;
    p.unit = unit;
    p.uph = (T + unit - 1) / unit;
    p.warps = many && T >= wide_from && T <= wide_max && 2 * heads <= 13 * kSmCount ? 8 : 4;
    // long heads are three to an SM: two or four an SM whole would leave it with one or two for most of the time (592 heads of 8000
    // tokens, 2 bits: 166 us whole, 143 us as 444 and 148 cut; 320 heads 107 and 86 us all cut in five)
    const bool three = T > wide_max;
    int per_sm = quarters ? 0 : (int)(heads / kSmCount);
    if (three && per_sm == 4) per_sm = 3;
    if (three && per_sm == 2) per_sm = 0;
    p.n_whole = per_sm * kSmCount;
    p.k = quarters ? 4 : per_sm == 0 ? 5 : per_sm == 3 && heads >= 4 * kSmCount ? 3 : plan_left_pieces(T, unit, (int)(heads % kSmCount), three ? 125 : 100);
    if (p.k == 1) p.n_whole = (int)(heads / kWholeWave * kWholeWave);             // all whole: the same launch wherever the line is drawn
    p.n_cut = (int)(heads - p.n_whole);
    p.seg_units = (p.uph + p.k - 1) / p.k;
    p.k = (p.uph + p.seg_units - 1) / p.seg_units;
    plan_finish(p, T, tile, p.warps == 4 ? narrow_split : max_scores);
    return p;
}

// CTA index -> (head, segment): whole heads first, then the cut heads segment-major (all first segments, then all
// second segments, ...), so the shortest segments -- the last of each head -- come last.
#ifdef __CUDACC__
__device__ __forceinline__ void plan_head(const AttnPlan &p, int c, int &head, int &seg) {
    head = c;
    seg = 0;
    if (c >= p.n_whole) {
        const int cc = c - p.n_whole;
        seg = (int)p.by_cut((uint32_t)cc);
        head = p.n_whole + cc - seg * p.n_cut;
    }
}
// The tokens of segment `seg` of that head (of T), and how many segments the head has.
__device__ __forceinline__ void plan_tokens(const AttnPlan &p, int T, int c, int seg, int &t0, int &t1, int &cnt) {
    t0 = 0;
    t1 = T;
    cnt = 1;
    if (c >= p.n_whole) {
        cnt = p.k;
        t0 = seg * p.seg_units * p.unit;
        t1 = min(t0 + p.seg_units * p.unit, T);
    }
}
// Head s -> sequence, kv head, number within the kv head.
__device__ __forceinline__ void plan_place(const AttnPlan &p, int s, int &b, int &hk, int &within) {
    b = (int)p.by_seq((uint32_t)s);
    const uint32_t r = (uint32_t)s - b * p.by_seq.d;
    hk = (int)p.by_kv(r);
    within = (int)(r - hk * p.by_kv.d);
}
#endif
// `per_kv` heads (or groups of them) of one kv head are neighbours.
inline void plan_set_place(AttnPlan &p, int nh, int nh_kv, int per_kv) {
    p.rep = nh / nh_kv;
    p.by_cut = fast_div((uint32_t)(p.n_cut > 0 ? p.n_cut : 1));
    p.by_kv = fast_div((uint32_t)per_kv);
    p.by_seq = fast_div((uint32_t)per_kv * (uint32_t)nh_kv);
}

}  // namespace kvq
