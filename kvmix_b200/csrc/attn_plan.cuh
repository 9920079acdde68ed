// Work plan of the tensor-core attention kernels: which tokens of which head a CTA scores.
//
// The token axis of every head (a query head, or the group of query heads that share a kv head) is cut into
// units of `unit` tokens (a warp's key tile: 256, or four of them for 3-bit keys: 352 = 4 x 88); a head has
// uph = ceil(T / unit) units, the last one possibly short.  One CTA works one segment = a run of units of one head:
//   * the first n_whole CTAs take one whole head each (only when a head fits the score buffer); n_whole is a multiple
//     of kWholeWave, so these CTAs fill whole waves;
//   * every remaining head (n_cut of them) is cut into k segments of seg_units units (the last one shorter), launched
//     after the whole heads, first segments of all heads first.  k is chosen so that these smaller CTAs, which the
//     hardware hands to whichever slot frees up, finish as early as possible: the last wave of a grid is then made of
//     short CTAs and fills all slots, whatever the number of heads.
// A head cut into several segments is merged by the CTA that finishes last (per-head counter), in segment order, so
// results do not depend on timing.
#pragma once
#include <stdint.h>

namespace kvq {

struct AttnPlan {
    int unit;            // tokens per unit
    int uph;             // units per head
    int n_whole;         // CTAs (= heads) that take a whole head
    int n_cut;           // heads that are cut
    int k;               // segments per cut head (1: a whole head per CTA here too)
    int seg_units;       // units per segment of a cut head
    int n_scores;        // most tokens in a segment, rounded up to 32
    int ks_log2;         // the channels of a key tile are shared by 1 << ks_log2 warps (partial scores, summed by the softmax)
};

constexpr int kSmCount = 148;
constexpr int kPlanSlots = 2 * kSmCount;       // resident CTAs: two of eight warps per SM
constexpr int kPlanWarps = 8;
// Whole heads: multiples of two and of three CTAs per SM
constexpr int kWholeWave = 6 * kSmCount;
// One partial result of a cut head: 128 accumulators, the segment's maximum and sum, padded so that rows stay 16-byte
// aligned (the merge reads them with 128-bit loads).
constexpr int kPartStride = 128 + 4;
constexpr int kMaxCtaRounds = 8;       // cut heads are never spread over more CTAs than this many waves (bounds the workspace)

inline int plan_round32(int n) { return (n + 31) / 32 * 32; }

// Channel split of a segment's key tiles.  A warp walks a tile's 128 channels in four steps of 32; where a segment has fewer
// tiles than the CTA has warps, 2 or 4 warps share a tile's channels and each leaves partial scores.  Steps a warp takes
// (x 2), with about half a step's time of per-tile overhead; `max_scores` bounds the score buffer (tokens x splits).
inline int plan_key_steps(int n, int tile, int ks_log2) {
    const int tiles = (n + tile - 1) / tile;
    const int passes = ((tiles << ks_log2) + kPlanWarps - 1) / kPlanWarps;
    return passes * ((8 >> ks_log2) + 1);
}
inline int plan_key_split(int n, int tile, int max_scores) {
    int best = 0;
    for (int l = 1; l <= 2; ++l)
        if ((plan_round32(n) << l) <= max_scores && plan_key_steps(n, tile, l) < plan_key_steps(n, tile, best)) best = l;
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

// heads: number of heads (or head groups); tile: tokens of a warp's key tile; max_scores: tokens the score buffer holds.
// narrow_scores: tokens up to which a kernel also has four-warp CTAs, four to an SM (0: it has none).  Heads that fill the eight-warp
// slots more than once and the four-warp ones at most once are then left whole: 320 heads of 4096 tokens at 2 bits
// take 57 us that way, 68 us cut for the eight-warp CTAs.
inline AttnPlan make_attn_plan(int T, int unit, int tile, int max_scores, long long heads, int narrow_scores = 0) {
    AttnPlan p;
    p.unit = unit;
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
        const bool one_wave = T <= narrow_scores && heads > kPlanSlots && heads <= 2 * kPlanSlots;
        for (int su = whole_ok ? p.uph : max_units; su >= 1; --su) {
            const int k = (p.uph + su - 1) / su;
            const long long ctas = (long long)p.n_cut * k;
            if (ctas > (long long)kMaxCtaRounds * kPlanSlots && best >= 0) break;
            const long long rounds = (ctas + kPlanSlots - 1) / kPlanSlots;
            const int n = su * unit < T ? su * unit : T;
            const long long cost = rounds * plan_segment_cycles(n, tile, max_scores) + plan_merge_cycles(k);
            if (best < 0 || cost < best) {
                best = cost;
                p.k = k;
                p.seg_units = su;
            }
        }
        if (one_wave) p.k = 1;
        p.seg_units = (p.uph + p.k - 1) / p.k;                                   // even the segments out
        p.k = (p.uph + p.seg_units - 1) / p.seg_units;
    }
    long long ns = (long long)(p.n_whole ? p.uph : p.seg_units) * unit;
    if (ns > T) ns = T;
    p.n_scores = plan_round32((int)ns);
    p.ks_log2 = plan_key_split((int)ns, tile, max_scores);
    return p;
}

// CTA index -> (head, segment): whole heads first, then the cut heads segment-major (all first segments, then all
// second segments, ...), so the shortest segments -- the last of each head -- come last.
__host__ __device__ inline void plan_cta(const AttnPlan &p, int T, int c, int &head, int &t0, int &t1, int &seg, int &cnt) {
    if (c < p.n_whole) {
        head = c; t0 = 0; t1 = T; seg = 0; cnt = 1;
        return;
    }
    const int cc = c - p.n_whole;
    seg = cc / p.n_cut;
    head = p.n_whole + cc - seg * p.n_cut;
    cnt = p.k;
    t0 = seg * p.seg_units * p.unit;
    const int e = t0 + p.seg_units * p.unit;
    t1 = e < T ? e : T;
}

}  // namespace kvq
