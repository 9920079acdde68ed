// Fused decode attention for grouped-query models, tensor-core path: one CTA (8 warps) serves up to FOUR query heads
// that share a kv head, so every packed code is fetched, unpacked and fed to the tensor core once for all of them.
//
// Same formulation as decode_attn_mma.cu (codes reach mma.sync as fp16 subnormals, q*scale carried as an exact
// fp16 pair hi + lo, per-warp cp.async rings); what changes is the meaning of the eight B columns:
//   keys    column 2h / 2h+1 = hi / lo of q_h[d] * scale[d, group] for query head h of the quad.  An MMA's 16 token
//           rows therefore have to lie in ONE scale group: 1-, 2- and 4-bit keys are all fetched with transposing
//           ldmatrix loads (a 16-byte block of a channel row = 128 / 64 / 32 tokens; needs k_group >= that), and
//           3-bit keys (group 11 = one word) put the 11 tokens of a word in the rows of an MMA, extracting field g with a
//           per-lane byte permute and mask.  The zero terms sum_d q_h[d] * zero[d, group] of all groups of a tile come
//           from one MMA per 16 channels: the zero tile in shared memory ([channel][group]) read transposed is the A
//           operand (row = group), q the B operand.
//   values  column 2h / 2h+1 = p_h[t] * scale[t, group] / p_h[t] * midpoint[t, group]; an MMA's 16 channel rows lie
//           in one channel group (a 16-byte block of a token row = 128 / 64 / 32 channels; needs v_group >= that --
//           except 1-bit values at group 64, where a block spans two groups and every code tile is multiplied by both
//           groups' operands, each lane keeping the product of the group its rows belong to).
// Scores of the four heads sit side by side in shared memory ([4][n]); two warps run the softmax of a head.
//
// Bound by the instruction stream around the codes (issue about half busy, the half-rate logic pipe as much), so the loops know their
// group sizes: conditions on them cost a compare, a branch or a select per group and k-step.  Warp instructions per 32 codes, 2-bit
// keys and values, group 64: 2.98 with the group sizes looked up, 2.34 so (0.63 of it the isolation of the fields, 0.14 MMAs);
// 8 x 8 kv heads of 32768 tokens, group 64: 88.7 -> 78.2 us, 4-bit 101.5 -> 87.8, 3-bit keys with 4-bit values 156.3 -> 129.7.
#include "attn_mma_common.cuh"
#include "attn_plan.cuh"
#include "attn_update.cuh"

namespace kvq {

constexpr int kQH = 4;                  // query-head slots per CTA
constexpr int kGqaMaxScores = 2048, kGqaMaxScores3 = 2112;   // tokens the score buffer holds (x 4 heads): two CTAs per SM

struct GqaSmem {
    float *scores;          // [1 << ks_log2][kQH][n_scores]
    unsigned char *ring;    // this warp's region
    __half *q;              // [kQH][kHeadDim]
    float *misc;            // [64]
    int n_scores, ks_log2;
};

// A stage carries the scale and zero rows of its channels behind the codes.  3-bit keys: 8 groups per tile, 16-byte scale
// rows followed by the zero rows; other widths (<= 4 groups per tile): 16-byte rows that hold 4 scales then 4 zeros.
template <int KB> constexpr int gqa_zero_off() { return KB == 3 ? KGeom<KB>::ROWS * 16 : 8; }
template <int KB> using GqaKRing = KRing<KB, KGeom<KB>::ROWS * (KB == 3 ? 32 : 16), KB == 1 ? 4 : 3>;
template <int VB> using GqaVGeom = VGeom<VB, VB == 4 ? 3 : VB == 2 ? 5 : 7>;
// operand tiles of the values: 512 bytes per channel group (4 / 2 / 2 groups at most)
template <int VB> constexpr int gqa_op_bytes() { return VB == 4 ? 2048 : 1024; }

// 3-bit values (the short-last-group extension: 12 words and 12 groups a token): 48 + 2 x 24 bytes a token, two slots, operand
// tiles of four groups, the tile of the probabilities and the groups' powers of two
constexpr int kV3Words = (kHeadDim + 10) / 11;
constexpr int kV3Stage = 32 * (kV3Words * 4 + 2 * kV3Words * 2), kV3Slots = 2, kV3SzOff = 32 * kV3Words * 4;
constexpr int kV3Region = kV3Slots * kV3Stage + 4 * 512 + 512 + 32;
template <int VB> constexpr int gqa_v_region() { return GqaVGeom<VB>::NS * GqaVGeom<VB>::STAGE_BYTES + gqa_op_bytes<VB>(); }
template <> constexpr int gqa_v_region<3>() { return kV3Region; }
template <int KB, int VB> constexpr int gqa_region_bytes() {
    return GqaKRing<KB>::BYTES > gqa_v_region<VB>() ? GqaKRing<KB>::BYTES : gqa_v_region<VB>();
}

__device__ __forceinline__ uint2 lds64(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}

// ---------------------------------------------------------------------------------------------
// fp16 key tail for tokens [lo, t1): 16-token tiles straight from global memory; B column n = query head n.  EARLY: the first
// tile is asked for before the CTA barrier behind which q is in shared memory, and every warp passes that barrier in here.  For keys
// and values that together have six bits and more, in calls the host drives (16 .. 160 head groups x 350 .. 8000 tokens: 3-bit keys with 4-bit
// values 0.964 of the time, 4 and 4 bits 0.989, 4 and 2 bits 0.984; 3 and 2 bits 1.022, 2 and 2 bits 1.014; the device-driven kernels spill
// for it, 32k tokens 531 -> 535 us).
template <bool EARLY>
__device__ __forceinline__ void gqa_qk_tail(const kvq_attn_args &a, const __half *kf, int b, int hk, const GqaSmem &sm,
                                            int t0, int lo, int t1) {
    const int warp = uniform_warp(), lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    const int n_tiles = (t1 - lo + 15) / 16;                   // <= 0: no tail in this segment
    uint4 ra[4], rb[4];
    auto load = [&](int tile) {
        const int ta = lo + 16 * tile + g;
        const __half *pa = k_tail_row(a, kf, b, hk, min(ta, t1 - 1)) + 8 * tig;
        const __half *pb = k_tail_row(a, kf, b, hk, min(ta + 8, t1 - 1)) + 8 * tig;
#pragma unroll
        for (int S = 0; S < 4; ++S) {
            ra[S] = __ldcg(reinterpret_cast<const uint4 *>(pa + 32 * S));
            rb[S] = __ldcg(reinterpret_cast<const uint4 *>(pb + 32 * S));
        }
    };
    if constexpr (EARLY) {
        if (warp < n_tiles) load(warp);
        __syncthreads();
        if (warp >= n_tiles) return;
    }
    uint4 qf[4];
#pragma unroll
    for (int S = 0; S < 4; ++S)
        qf[S] = g < kQH ? *reinterpret_cast<const uint4 *>(sm.q + g * kHeadDim + 32 * S + 8 * tig) : make_uint4(0u, 0u, 0u, 0u);
    for (int tile = warp; tile < n_tiles; tile += kMmaWarps) {
        const int ta = lo + 16 * tile + g, tb = ta + 8;
        if (!EARLY || tile != warp) load(tile);
        float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int S = 0; S < 4; ++S) {
            mma16816(c, ra[S].x, rb[S].x, ra[S].y, rb[S].y, qf[S].x, qf[S].y);
            mma16816(c, ra[S].z, rb[S].z, ra[S].w, rb[S].w, qf[S].z, qf[S].w);
        }
        if (tig < 2) {                                         // columns 2 tig, 2 tig + 1 = heads 2 tig, 2 tig + 1
            for (int p = 0; p < (1 << sm.ks_log2); ++p) {      // the whole score in the first partial, zero in the others
                float *d0 = sm.scores + (p * kQH + 2 * tig) * sm.n_scores - t0, *d1 = d0 + sm.n_scores;
                if (ta < t1) { d0[ta] = p ? 0.f : c[0]; d1[ta] = p ? 0.f : c[1]; }
                if (tb < t1) { d0[tb] = p ? 0.f : c[2]; d1[tb] = p ? 0.f : c[3]; }
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// q . K^T over packed keys, tokens [t0, hi), for the four heads of the quad.  Stage geometry, tile order and channel
// splits of the single-head kernel, which for 3-bit keys also has tiles of 176 tokens (here always 88); scores[split][h][t - t0] receive the raw scores.
template <int KB, bool WIDE, bool EARLY>
__device__ __forceinline__ void gqa_qk_packed(const kvq_attn_args &a, const int32_t *kc, const __half *ks,
                                              const __half *kz, const GqaSmem &sm, int t0, int hi, const __half *kf,
                                              int tail_lo, int t1, int b, int hk) {
    using G = KGeom<KB>;
    using R = GqaKRing<KB>;
    const int warp = uniform_warp(), lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    constexpr int LGK = WIDE ? 7 : 6, NGW = KB == 3 ? 8 : G::WT >> LGK;         // groups of a tile: 8 (3 bits) / 2 / 4
    const int n_words = a.Tkq / G::FPI;
    const int n_tiles = (hi - t0 + G::WT - 1) / G::WT;                         // <= 0: no packed keys in this segment
    const int split = warp & ((1 << sm.ks_log2) - 1), wt = warp >> sm.ks_log2, tile_lanes = kMmaWarps >> sm.ks_log2;
    const int my_tiles = (n_tiles - wt + tile_lanes - 1) / tile_lanes;
    const int ch0 = split * (kHeadDim >> sm.ks_log2), steps = (kHeadDim / 32) >> sm.ks_log2;   // channels of this warp
    const int tile_stages = G::NSTAGE >> sm.ks_log2;
    const int kc_sD = (int)a.kc_sD, ks_sD = (int)a.ks_sD;
    const uint32_t ring_s = smem_u32(sm.ring);
    constexpr int ZOFF = gqa_zero_off<KB>();
    const int gr = lane % G::GPR, row0 = lane / G::GPR;
    const uint32_t cp_dst = ring_s + row0 * G::RS + gr * 16;
    constexpr int FH = (KB == 3) ? 2 : 16 / KB;                                // fields per half-word: 4 / 8 / 16
    constexpr int NBK = G::RB / 16;                                            // 16-byte blocks per channel row: 8 / 4 / 2
    constexpr int MPB = FH / 2;                                                // MMAs per block and k-step: 2 / 4 / 8
    constexpr int NACC = (KB == 3) ? 8 : NBK * MPB;                            // accumulators per tile: 8 words / 16 token pairs
    const uint32_t ldk_s = ring_s + ((lane & 7) + 8 * ((lane >> 3) & 1)) * G::RS + (lane >> 4) * 16;
    const uint32_t w3_s = ring_s + (2 * tig) * G::RS;                          // 3-bit: word rows 2 tig, +1, +8, +9
    const uint32_t szrow_s = ring_s + G::CODE_BYTES + (2 * tig) * 16;         // + slot + 256 k [+16 | +128 | +144] [+ZOFF zero]
    const uint32_t szm_s = ring_s + G::CODE_BYTES + (KB == 3 ? ZOFF : 0) + (lane & 15) * 16;   // zero tile as an A operand
    const uint32_t q_s = smem_u32(sm.q) + (g >> 1) * (kHeadDim * 2) + (ch0 + 2 * tig) * 2;     // this column's head; + 32 per k-step [+16]
    const uint32_t neg_mask = (g & 1) ? 0xffffffffu : 0u;
    const int tile_words = tile_lanes * G::WT / G::FPI;
    const int tile_groups = tile_lanes * NGW;
    // 3-bit keys: field g of a word sits at bits 3g..3g+2; one byte permute brings the two bytes that hold it (of both
    // channel words) into the 16-bit halves, a mask isolates it in place at bit p0 = 3g mod 8 (<= 7: linear fp16 range).
    // Fields 8..10 (rows g + 8, g < 3) sit in byte 3 at bits 0, 3, 6 (the last one 2 bits wide).
    const int byte0 = (3 * g) >> 3, p0 = 3 * g - 8 * byte0;
    const uint32_t sel0 = (uint32_t)(byte0 | ((byte0 + 1) << 4) | ((4 + byte0) << 8) | ((5 + byte0) << 12));
    const uint32_t msk0 = 0x00070007u << p0;
    const uint32_t sel1 = 0x7733u;
    const uint32_t msk1 = g == 0 ? 0x00070007u : g == 1 ? 0x00380038u : g == 2 ? 0x00c000c0u : 0u;
    const int p1 = 3 * (g < 3 ? g : 0);
    const float sc0 = __int_as_float((151 - p0) << 23), sc1 = __int_as_float((151 - p1) << 23);   // 2^(24 - position)

    // the next stage to issue: its addresses, its word column, its position in its tile and the tiles left.  A stage of 16
    // channels takes one scale / zero copy per lane (zeros: lanes 16-31), one of 32 channels two.
    uint32_t iss = 4u * ((uint32_t)(ch0 + row0) * kc_sD + (t0 + wt * G::WT) / G::FPI + 4 * gr);   // bytes from the head's first word
    constexpr bool kOneSz = G::ROWS == 16;
    const int sz_row = kOneSz ? (lane & 15) : lane;
    const bool sz_zero = kOneSz && lane >= 16;
    uint32_t iss_s = 2u * ((uint32_t)(ch0 + sz_row) * ks_sD + (KB == 3 ? (t0 + wt * G::WT) / 11 : (t0 + wt * G::WT) >> LGK));
    const char *sz_b = reinterpret_cast<const char *>(sz_zero ? kz : ks);
    const uint32_t szcp_dst = ring_s + G::CODE_BYTES + sz_row * 16 + (sz_zero ? ZOFF : 0);
    int iss_col = (t0 + wt * G::WT) / G::FPI + 4 * gr, iss_st = 0, iss_tiles = my_tiles;
    uint32_t iss_slot = 0, slot = 0;
    bool iss_ok = iss_col < n_words;

    const char *kc_b = reinterpret_cast<const char *>(kc), *kz_b = reinterpret_cast<const char *>(kz);
    const uint32_t row_step = (uint32_t)(G::RPI * 4) * kc_sD, stage_step = (uint32_t)(G::ROWS * 4) * kc_sD, sz_step = (uint32_t)(G::ROWS * 2) * ks_sD;
    const uint32_t tile_step = 4 * tile_words - tile_stages * stage_step, tile_sz_step = 2 * tile_groups - tile_stages * sz_step;

    auto issue_stage = [&]() {
        if (iss_tiles > 0) {
            if (iss_ok) {
#pragma unroll
                for (int i = 0; i < G::GPL; ++i)
                    cp_async<16>(cp_dst + iss_slot + i * G::RPI * G::RS, kc_b + (iss + i * row_step));
            }
            const uint32_t d = szcp_dst + iss_slot;
            if (KB == 3) { cp_async<16>(d, sz_b + iss_s); cp_async<16>(d + ZOFF, kz_b + iss_s); }
            else if (NGW == 4) { cp_async<8>(d, sz_b + iss_s); if (!kOneSz) cp_async<8>(d + ZOFF, kz_b + iss_s); }
            else { cp_async<4>(d, sz_b + iss_s); if (!kOneSz) cp_async<4>(d + ZOFF, kz_b + iss_s); }
        }
        cp_async_commit();
        iss_slot = iss_slot == (R::NS - 1) * R::STAGE_BYTES ? 0u : iss_slot + R::STAGE_BYTES;
        iss += stage_step;
        iss_s += sz_step;
        if (++iss_st == tile_stages) {
            iss_st = 0;
            iss += tile_step;
            iss_s += tile_sz_step;
            iss_col += tile_words;
            iss_ok = iss_col < n_words;
            --iss_tiles;
        }
    };

#pragma unroll 1
    for (int q = 0; q < R::P; ++q) issue_stage();
    if constexpr (!EARLY) {
        __syncthreads();                                       // q is in shared memory (stored by the caller without a barrier)
        if (tail_lo < t1) gqa_qk_tail<false>(a, kf, b, hk, sm, t0, tail_lo, t1);
    } else {
        gqa_qk_tail<true>(a, kf, b, hk, sm, t0, tail_lo, t1);
    }

    for (int j = 0; j < my_tiles; ++j) {
        const int tile0 = t0 + (j * tile_lanes + wt) * G::WT;
        uint32_t q_cur = q_s;
        // A group behind the packed prefix (its scale and zero words may hold anything) spoils the accumulators of its own
        // tokens and its own row of the zero terms, which nothing reads: all groups are formed, without a condition.
        float acc[NACC][4], zsum = 0.f;
#pragma unroll
        for (int m = 0; m < NACC; ++m) acc[m][0] = acc[m][1] = acc[m][2] = acc[m][3] = 0.f;

        // two k-steps a turn: unrolled over all eight the loop missed the instruction cache (2.7 of 7.3 cycles per issued
        // instruction at 2 bits were fetch stalls)
#pragma unroll 1
        for (int it = 0; it < steps; ++it) {
          float accz[4] = {0.f, 0.f, 0.f, 0.f};               // zero terms of two k-steps
#pragma unroll
          for (int s2 = 0; s2 < 2 / G::KSPS; ++s2) {
            issue_stage();
            cp_async_wait<R::P>();
            __syncwarp();
            const uint32_t stage_s = slot;
#pragma unroll
            for (int k = 0; k < G::KSPS; ++k) {
                const uint32_t q01u = lds32(q_cur), q89u = lds32(q_cur + 16);
                q_cur += 32;
                const __half2 q01 = as_h2(q01u), q89 = as_h2(q89u);
                const uint32_t zrow = szrow_s + slot + 256 * k;      // scale rows 16 k + 2 tig (+1, +8, +9); zeros + ZOFF
                if constexpr (KB == 3) {
                    // every word is its own group: per word j one B operand and one code MMA (rows = its 11 tokens); words
                    // are taken in pairs so that scales arrive as 32-bit loads.  The zero terms sum_d q[d] * zero[d, j] of
                    // all eight words come from ONE MMA per k-step: the zero tile ([channel][word], 16 bytes per channel)
                    // read transposed is an A operand with row = word and k = channel, B = q in the even columns
                    // (fp16 x fp16 products are exact in the tensor core, so no hi / lo split is needed here); a word
                    // beyond the packed prefix only spoils its own row, which nothing reads
                    {
                        uint32_t za0, za2;
                        asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];\n"
                                     : "=r"(za0), "=r"(za2) : "r"(szm_s + slot + 256 * k));
                        mma16816(accz, za0, 0u, za2, 0u, q01u & ~neg_mask, q89u & ~neg_mask);
                    }
#pragma unroll
                    for (int jp = 0; jp < 4; ++jp) {
                        uint32_t sA = lds32(zrow + 4 * jp), sB = lds32(zrow + 16 + 4 * jp);
                        uint32_t sC = lds32(zrow + 128 + 4 * jp), sD = lds32(zrow + 144 + 4 * jp);
                        const uint32_t src = w3_s + stage_s + (k * 16) * G::RS + 8 * jp;
                        const uint2 wA = lds64(src), wB = lds64(src + G::RS), wC = lds64(src + 8 * G::RS), wD = lds64(src + 9 * G::RS);
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int jw = 2 * jp + u;
                            const uint32_t psel = u ? 0x7632u : 0x5410u;
                            const __half2 s01 = as_h2(prmt(sA, sB, psel)), s89 = as_h2(prmt(sC, sD, psel));
                            const uint32_t a_lo = u ? wA.y : wA.x, b_lo = u ? wB.y : wB.x, a_hi = u ? wC.y : wC.x, b_hi = u ? wD.y : wD.x;
                            mma16816(acc[jw], prmt(a_lo, b_lo, sel0) & msk0, prmt(a_lo, b_lo, sel1) & msk1,
                                     prmt(a_hi, b_hi, sel0) & msk0, prmt(a_hi, b_hi, sel1) & msk1,
                                     hilo(q01, s01, neg_mask), hilo(q89, s89, neg_mask));
                        }
                    }
                } else {
                    // The zero terms sum_d q[d] * zero[d, j] of the tile's groups: one MMA per k-step whose A operand is the
                    // scale/zero tile read transposed (a channel's 16-byte row holds 4 scales then 4 zeros, so rows 4..7
                    // of the product are the zero terms of groups 0..3; rows 0..3 are not used) and whose B operand is
                    // q in the even columns (fp16 x fp16 is exact in the tensor core).  A group beyond the packed prefix
                    // only spoils its own row, which nothing reads.
                    {
                        uint32_t za0, za2;
                        asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];\n"
                                     : "=r"(za0), "=r"(za2) : "r"(szm_s + slot + 256 * k));
                        mma16816(accz, za0, 0u, za2, 0u, q01u & ~neg_mask, q89u & ~neg_mask);
                    }
                    // B operands of the tile's groups: two of 128 tokens or four of 64
                    constexpr int NB = KB == 3 ? 1 : NGW;
                    uint2 sA, sB, sC, sD;
                    if constexpr (WIDE) {
                        sA.x = lds32(zrow); sB.x = lds32(zrow + 16); sC.x = lds32(zrow + 128); sD.x = lds32(zrow + 144);
                        sA.y = sB.y = sC.y = sD.y = 0u;
                    } else {
                        sA = lds64(zrow); sB = lds64(zrow + 16); sC = lds64(zrow + 128); sD = lds64(zrow + 144);
                    }
                    uint32_t b[NB][2];
#pragma unroll
                    for (int jk = 0; jk < NB; ++jk) {
                        const uint32_t psel = (jk & 1) ? 0x7632u : 0x5410u;
                        const uint32_t a0 = (jk & 2) ? sA.y : sA.x, a1 = (jk & 2) ? sB.y : sB.x, a2 = (jk & 2) ? sC.y : sC.x, a3 = (jk & 2) ? sD.y : sD.x;
                        b[jk][0] = hilo(q01, as_h2(prmt(a0, a1, psel)), neg_mask);
                        b[jk][1] = hilo(q89, as_h2(prmt(a2, a3, psel)), neg_mask);
                    }
                    using H = KHalf<KB>;
                    const uint32_t lsrc = ldk_s + stage_s + (k * 16) * G::RS;
#pragma unroll
                    for (int pb2 = 0; pb2 < NBK / 2; ++pb2) {
                        uint32_t x[2][2];
                        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                                     : "=r"(x[0][0]), "=r"(x[0][1]), "=r"(x[1][0]), "=r"(x[1][1]) : "r"(lsrc + pb2 * 32));
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int bb = 2 * pb2 + u;
                            uint32_t rlo[H::N], rhi[H::N];
                            H::unpack(x[u][0], rlo);
                            H::unpack(x[u][1], rhi);
                            const uint32_t bx = b[(bb * 8 * FH) >> LGK][0], by = b[(bb * 8 * FH) >> LGK][1];   // the block's group in the tile
#pragma unroll
                            for (int i = 0; i < H::N; i += 2)
                                mma16816(acc[bb * MPB + i / 2], rlo[i], rlo[i + 1], rhi[i], rhi[i + 1], bx, by);
                        }
                    }
                }
            }
            __syncwarp();                                      // the slot may be refilled
            slot = slot == (R::NS - 1) * R::STAGE_BYTES ? 0u : slot + R::STAGE_BYTES;
          }
          zsum += accz[0] + accz[1];
        }

        // ---- epilogue: lane (g, tig) holds, per accumulator, row g / g + 8 of head tig as (hi, lo) ------------
        // row g = group g of the tile: its zero term for head tig (hi + lo columns)
        float *dst_h = sm.scores + (split * kQH + tig) * sm.n_scores - t0;
        if constexpr (KB == 3) {
#pragma unroll
            for (int jw = 0; jw < 8; ++jw) {
                const float corr = __shfl_sync(0xffffffffu, zsum, 4 * jw + tig);
                const int ta = tile0 + 11 * jw + g, tb = ta + 8;
                float s0 = fmaf(acc[jw][0] + acc[jw][1], sc0, corr);
                float s1 = fmaf(acc[jw][2] + acc[jw][3], sc1, corr);
                if (11 * jw + tile0 < hi) {                    // words are whole or absent (hi is a group multiple)
                    dst_h[ta] = s0;
                    if (g < 3) dst_h[tb] = s1;
                }
            }
        } else {
            float zj[NGW];
#pragma unroll
            for (int jk = 0; jk < NGW; ++jk) zj[jk] = __shfl_sync(0xffffffffu, zsum, 4 * (4 + jk) + tig);   // rows 4..7
#pragma unroll
            for (int bb = 0; bb < NBK; ++bb) {
                const float corr = zj[(bb * 8 * FH) >> LGK];
                const int tok0 = tile0 + bb * 8 * FH + g * FH;
                if (tok0 < hi) {                               // FH-token chunks are whole or absent (hi is a group multiple)
                    float *dst = dst_h + tok0;
#pragma unroll
                    for (int ip = 0; ip < MPB; ++ip) {
                        const int m = bb * MPB + ip;
                        float s0 = fmaf(acc[m][0] + acc[m][1], (float)(1 << (24 - KHalf<KB>::pos(2 * ip))), corr);
                        float s1 = fmaf(acc[m][2] + acc[m][3], (float)(1 << (24 - KHalf<KB>::pos(2 * ip + 1))), corr);
                        *reinterpret_cast<float2 *>(dst + 2 * ip) = make_float2(s0, s1);
                    }
                }
            }
        }
    }
    cp_async_wait<0>();
}

// ---------------------------------------------------------------------------------------------
// p . V over packed values for tokens [t0, hi), (hi - t0) % 32 == 0, for the four heads.  scores[h] hold p_h.  Leaves
// this warp's partial sums float[kQH][128] at the base of its region.  MODE as in the single-head kernel.
template <int VB, int MODE, int NGV>
__device__ __forceinline__ void gqa_pv_packed(const kvq_attn_args &a, const int32_t *vc, const __half *vs,
                                              const __half *vz, const GqaSmem &sm, int t0, int hi) {
    using G = GqaVGeom<VB>;
    using F = VHalf<VB>;
    constexpr int NB = G::GPT;                                // 16-byte blocks per token row: 1 / 2 / 4
    constexpr int CPB = kHeadDim / NB;                        // channels per block: 128 / 64 / 32
    constexpr int MPB = F::N / 2;                             // MMAs per block: 8 / 4 / 2
    const int warp = uniform_warp(), lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    constexpr int ngv = NGV, Gv = kHeadDim / NGV;             // channel groups: 4 / 2 / 1
    const int n_blocks = (hi - t0 + G::TPS - 1) / G::TPS;
    const int my_blocks = (n_blocks - warp + kMmaWarps - 1) / kMmaWarps;
    float *my_red = reinterpret_cast<float *>(sm.ring);
    if (my_blocks <= 0) {
        if (MODE != 1)
            for (int i = lane; i < kQH * kHeadDim; i += 32) my_red[i] = 0.f;
        return;
    }
    const uint32_t ring_s = smem_u32(sm.ring);
    const uint32_t pb_s = ring_s + G::NS * G::STAGE_BYTES;                               // operand tiles [ngv][16 pairs][8 cols]
    const int cp_tl0 = lane / G::GPT, cp_gr = lane % G::GPT;
    auto swz = [](int tl) { return (VB == 4) ? ((tl >> 1) & 3) : (VB == 2) ? ((tl >> 2) & 1) : 0; };
    const int cp_grs = cp_gr ^ swz(cp_tl0);
    const uint32_t cp_dst = ring_s + cp_tl0 * G::RBV + cp_grs * 16;
    const int ldm_tl = 8 * ((lane >> 3) & 1) + (lane & 7);
    const int ldm_b = (lane >> 4) & (NB - 1);
    const uint32_t ldm_s0 = ring_s + ldm_tl * G::RBV + ((ldm_b ^ swz(ldm_tl)) * 16);
    const uint32_t ldm_s1 = ring_s + ldm_tl * G::RBV + (((ldm_b + 2) & (NB - 1)) ^ swz(ldm_tl)) * 16;
    const uint32_t pb_rd = pb_s + (tig * 8 + g) * 4;                                     // + jv * 512 + (8 h2 + 4 b) * 32
    // operand build: lane -> token pair pi = lane & 15 and head pair hh = lane >> 4 (heads 2 hh, 2 hh + 1)
    const int pi = lane & 15, hh = lane >> 4;
    const int bt0 = 16 * (pi >> 3) + 8 * ((pi >> 2) & 1) + 2 * (pi & 3);                 // the pair's first token in the stage
    const uint32_t sz_rd = ring_s + G::SZ_OFF + (bt0 * ngv) * 2;                         // scale row of token bt0; + ngv * 2 next token
    const uint32_t pb_wr = pb_s + (pi * 8 + 4 * hh) * 4;
    const float *pa = sm.scores + (2 * hh) * sm.n_scores + warp * G::TPS + bt0, *pb = pa + sm.n_scores;

    const int block_stride = kMmaWarps * G::TPS;
    const char *vc_b = reinterpret_cast<const char *>(vc);                               // 32-bit byte offsets from the head's first row
    uint32_t src_codes = (uint32_t)(t0 + warp * G::TPS) * G::RBV + lane * 16;
    const int ngran = 4 * ngv;
    const int sz_arr = lane >= ngran ? 1 : 0;
    const int sz_off = (lane - sz_arr * ngran) * 16;
    const bool sz_on = lane < 2 * ngran;
    const char *sz_b = reinterpret_cast<const char *>(sz_arr ? vz : vs);
    uint32_t src_sz = (uint32_t)(t0 + warp * G::TPS) * (ngv * 2) + sz_off;
    const uint32_t sz_dst = ring_s + G::SZ_OFF + sz_arr * (G::TPS * 4 * 2) + sz_off;
    const uint32_t codes_step = block_stride * G::RBV, sz_step = block_stride * ngv * 2;

    int to_issue = my_blocks;
    auto issue_stage = [&](uint32_t slot_off) {
        if (to_issue > 0) {
#pragma unroll
            for (int i = 0; i < G::GPL; ++i)
                if (G::TPS * G::GPT % 32 == 0 || lane + 32 * i < G::TPS * G::GPT)
                    cp_async<16>(cp_dst + slot_off + i * (32 / G::GPT) * G::RBV, vc_b + (src_codes + i * 512));
            if (sz_on) cp_async<16>(sz_dst + slot_off, sz_b + src_sz);
        }
        --to_issue;
        src_codes += codes_step;
        src_sz += sz_step;
    };

    float acc[8][4], accz[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};    // ones-MMAs alternate between two accumulators
#pragma unroll
    for (int m = 0; m < 8; ++m) acc[m][0] = acc[m][1] = acc[m][2] = acc[m][3] = 0.f;
    // 1-bit values in groups of 64 channels: a 16-byte block (128 channels) then spans two groups, and the rows of an
    // MMA (lane octet g = channels 16 g .. 16 g + 15) lie in group g / 4.  Every code tile is multiplied twice, the rows of
    // group 1 cleared by the operands of group 0 and the other way round, into the same accumulators.
    constexpr bool split = VB == 1 && Gv == 64;
    const uint32_t rows0 = !split || g < 4 ? 0xffffffffu : 0u, rows1 = g >= 4 ? 0xffffffffu : 0u;
    const uint32_t ones = 0x3c003c00u;
    // accumulation chains stay short by themselves (see the single-head kernel): 2112 tokens are at most nine blocks a warp
    if (MODE != 2) {
#pragma unroll
        for (int q = 0; q < G::P; ++q) { issue_stage(q * G::STAGE_BYTES); cp_async_commit(); }
        if (MODE == 1) return;
    } else {
        to_issue -= G::P;
        src_codes += G::P * codes_step;
        src_sz += G::P * sz_step;
    }

    uint32_t st = 0, issue_st = G::P * G::STAGE_BYTES;
    for (int q = 0; q < my_blocks; ++q) {
        issue_stage(issue_st);
        cp_async_commit();
        cp_async_wait<G::P>();
        __syncwarp();
        // ---- B operands for the stage: per channel group 16 token pairs x 8 columns (head x {p*scale, p*midpoint}) ----
        {
            // a lane's two tokens (rows back to back) in pairs: {scale, scale} and {zero, zero} of a group
            const unsigned long long k256 = f32x2(256.f, 256.f), mid = f32x2(G::MID, G::MID);                    // p carries 2^8
            const unsigned long long pa2 = mul_f32x2(*reinterpret_cast<const unsigned long long *>(pa), k256);
            const unsigned long long pb2 = mul_f32x2(*reinterpret_cast<const unsigned long long *>(pb), k256);
            uint32_t sw[2][2], zw[2][2];                       // [token][pair of groups]
            if constexpr (NGV == 4) {
                const uint2 x = lds64(sz_rd + st), y = lds64(sz_rd + st + 8), z = lds64(sz_rd + st + 256), w = lds64(sz_rd + st + 264);
                sw[0][0] = x.x; sw[0][1] = x.y; sw[1][0] = y.x; sw[1][1] = y.y;
                zw[0][0] = z.x; zw[0][1] = z.y; zw[1][0] = w.x; zw[1][1] = w.y;
            } else if constexpr (NGV == 2) {
                const uint2 x = lds64(sz_rd + st), z = lds64(sz_rd + st + 256);
                sw[0][0] = x.x; sw[1][0] = x.y; zw[0][0] = z.x; zw[1][0] = z.y;
            } else {                                           // one group: the two tokens share a word
                const uint32_t x = lds32(sz_rd + st), z = lds32(sz_rd + st + 256);
                sw[0][0] = x; sw[1][0] = x >> 16; zw[0][0] = z; zw[1][0] = z >> 16;
            }
#pragma unroll
            for (int jv = 0; jv < NGV; ++jv) {
                auto half_of = [&](uint32_t w) { return (jv & 1) ? __high2float(as_h2(w)) : __low2float(as_h2(w)); };
                const unsigned long long s2 = f32x2(half_of(sw[0][jv >> 1]), half_of(sw[1][jv >> 1]));
                const unsigned long long m2 = fma_f32x2(mid, s2, f32x2(half_of(zw[0][jv >> 1]), half_of(zw[1][jv >> 1])));
                auto pack = [](unsigned long long v) { const float2 f = f32x2_split(v); return pack_h2_sat(f.x, f.y); };
                const uint32_t c0 = pack(mul_f32x2(pa2, s2)), c1 = pack(mul_f32x2(pa2, m2)), c2 = pack(mul_f32x2(pb2, s2)), c3 = pack(mul_f32x2(pb2, m2));
                asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(pb_wr + jv * 512), "r"(c0), "r"(c1), "r"(c2), "r"(c3));
            }
        }
        __syncwarp();
#pragma unroll
        for (int h2 = 0; h2 < 2; ++h2) {
            uint32_t b[NGV][2];
#pragma unroll
            for (int jv = 0; jv < NGV; ++jv) {
                {
                    b[jv][0] = lds32(pb_rd + jv * 512 + (8 * h2) * 32);
                    b[jv][1] = lds32(pb_rd + jv * 512 + (8 * h2 + 4) * 32);
                    const uint32_t row1 = (g == jv) ? ones : 0u;    // sums of group jv land in row jv
                    mma16816(accz[jv & 1], row1, 0u, row1, 0u, b[jv][0], b[jv][1]);
                }
            }
            uint32_t x[NB][2];
            const uint32_t ad = st + (16 * h2) * G::RBV;
            if constexpr (VB == 1) {
                asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];\n"
                             : "=r"(x[0][0]), "=r"(x[0][1]) : "r"(ldm_s0 + ad));
            } else {
                asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                             : "=r"(x[0][0]), "=r"(x[0][1]), "=r"(x[1][0]), "=r"(x[1][1]) : "r"(ldm_s0 + ad));
                if constexpr (VB == 4)
                    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                                 : "=r"(x[NB - 2][0]), "=r"(x[NB - 2][1]), "=r"(x[NB - 1][0]), "=r"(x[NB - 1][1])
                                 : "r"(ldm_s1 + ad));
            }
#pragma unroll
            for (int bb = 0; bb < NB; ++bb) {
                uint32_t rlo[F::N], rhi[F::N];
                F::unpack(VB == 1 ? x[bb][0] & rows0 : x[bb][0], rlo);
                F::unpack(VB == 1 ? x[bb][1] & rows0 : x[bb][1], rhi);
                const uint32_t bx = b[split ? 0 : bb * CPB / Gv][0], by = b[split ? 0 : bb * CPB / Gv][1];        // the block's channel group
#pragma unroll
                for (int i = 0; i < F::N; i += 2)
                    mma16816(acc[bb * MPB + i / 2], rlo[i], rlo[i + 1], rhi[i], rhi[i + 1], bx, by);
                if constexpr (VB == 1) {
                    if constexpr (split) {
                        F::unpack(x[bb][0] & rows1, rlo);
                        F::unpack(x[bb][1] & rows1, rhi);
#pragma unroll
                        for (int i = 0; i < F::N; i += 2)
                            mma16816(acc[i / 2], rlo[i], rlo[i + 1], rhi[i], rhi[i + 1], b[NGV - 1][0], b[NGV - 1][1]);
                    }
                }
            }
        }
        __syncwarp();
        st = (st + G::STAGE_BYTES == G::NS * G::STAGE_BYTES) ? 0u : st + G::STAGE_BYTES;
        issue_st = (issue_st + G::STAGE_BYTES == G::NS * G::STAGE_BYTES) ? 0u : issue_st + G::STAGE_BYTES;
        pa += block_stride;
        pb += block_stride;
    }
    cp_async_wait<0>();
    __syncwarp();
    // epilogue: lane (g, tig) holds channels of rows g / g + 8 for head tig (column 2 tig); row jv of the ones-MMAs holds
    // (sum p*scale, sum p*mid) of channel group jv for head tig
    const float corr_mine = ((accz[0][1] + accz[1][1]) - G::MID * (accz[0][0] + accz[1][0])) * (1.f / 256.f);
    float cj[NGV];
#pragma unroll
    for (int jv = 0; jv < NGV; ++jv) cj[jv] = __shfl_sync(0xffffffffu, corr_mine, 4 * jv + tig);
#pragma unroll
    for (int bb = 0; bb < NB; ++bb) {
        const int c0 = bb * CPB + g * F::N;
        const float corr = split ? (g >= 4 ? cj[NGV - 1] : cj[0]) : cj[bb * CPB / Gv];
#pragma unroll
        for (int ip = 0; ip < MPB; ++ip) {
            my_red[tig * kHeadDim + c0 + 2 * ip] = fmaf(acc[bb * MPB + ip][0], (float)(1 << (16 - F::pos(2 * ip))), corr);
            my_red[tig * kHeadDim + c0 + 2 * ip + 1] = fmaf(acc[bb * MPB + ip][2], (float)(1 << (16 - F::pos(2 * ip + 1))), corr);
        }
    }
}

// The loops for the call's number of channel groups: 4 (4-bit values only, gqa_heads_per_cta), 2 or 1.
template <int VB, int MODE>
__device__ __forceinline__ void gqa_pv(const kvq_attn_args &a, const int32_t *vc, const __half *vs, const __half *vz, const GqaSmem &sm, int t0, int hi) {
    if (VB == 4 && a.v_group == 32) gqa_pv_packed<VB, MODE, VB == 4 ? 4 : 2>(a, vc, vs, vz, sm, t0, hi);
    else if (a.v_group == 64) gqa_pv_packed<VB, MODE, 2>(a, vc, vs, vz, sm, t0, hi);
    else gqa_pv_packed<VB, MODE, 1>(a, vc, vs, vz, sm, t0, hi);
}

// ---------------------------------------------------------------------------------------------
// p . V over 3-bit values: twelve words a token, each its own group of 11 channels (the last of 7).  As for 3-bit keys the
// channels of a word are the rows of an MMA (11 of 16 used); p * scale is carried as an fp16 pair hi + lo of the fp32
// product, columns 2h / 2h + 1 of head h, the zero terms come from one MMA per 16 tokens (rows = groups, B = p hi / lo).
// lo ends at 2^-24 whatever the product, so p (<= 1) is carried as 2^13 p and the scales of a group times a power of two that
// brings the largest of this warp's tokens to 2 .. 4 (exactly, but for those 2^-15 of it): what a pair loses is 2^-38 of the
// largest p and scale.  The largest scales are found by reading the warp's scale rows once ahead (a quarter of a token's bytes,
// asked for before the softmax and in L2 by then).  Infinite and NaN scales come out as fp32 products give them: a warp whose
// tokens hold one works without the complement below, whose halves would meet as inf - inf.
// Every other 16 tokens use the complemented codes and the operands' sign turned, so that what the tensor core cuts off
// the products (codes are subnormal) cancels instead of adding up; the sums of p * scale this needs are one more such MMA.
// Bound by the operand tiles (12 groups x 4 heads of p * scale for 352 bytes of a token pair).  8 x 8 kv heads, 32768
// tokens, 3-bit keys and values: 219 us a layer (215 with 4 p and the scales as they are), 735 us with the CUDA-core kernel.
// 0.99 of the weight on one token of next to nothing, values of sigma 0.03: 2.3e-4 from 64 bits (fp32 products 2.3e-4; 9e-4 so).
template <int MODE>
__device__ __forceinline__ void gqa_pv_packed3(const kvq_attn_args &a, const int32_t *vc, const __half *vs, const __half *vz,
                                               const GqaSmem &sm, int t0, int hi) {
    constexpr int W = kV3Words;
    const int warp = uniform_warp(), lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    const int n_blocks = (hi - t0 + 31) / 32;
    const int my_blocks = (n_blocks - warp + kMmaWarps - 1) / kMmaWarps;
    float *my_red = reinterpret_cast<float *>(sm.ring);
    if (my_blocks <= 0) {
        if (MODE != 1)
            for (int i = lane; i < kQH * kHeadDim; i += 32) my_red[i] = 0.f;
        return;
    }
    const uint32_t ring_s = smem_u32(sm.ring);
    const uint32_t op_s = ring_s + kV3Slots * kV3Stage, pp_s = op_s + 4 * 512;
    const char *vc_b = reinterpret_cast<const char *>(vc);
    uint32_t src_codes = (uint32_t)(t0 + warp * 32) * (W * 4) + lane * 16;
    // granules lane, lane + 32, lane + 64 of the 48 + 48 of a stage's scale and zero rows
    uint32_t src_sz = (uint32_t)(t0 + warp * 32) * (W * 2);
    constexpr uint32_t codes_step = kMmaWarps * 32 * W * 4, sz_step = kMmaWarps * 32 * W * 2;
    int to_issue = my_blocks;
    auto issue_stage = [&](uint32_t slot) {
        if (to_issue > 0) {
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                cp_async<16>(ring_s + slot + lane * 16 + i * 512, vc_b + (src_codes + i * 512));
                const int x = lane + 32 * i, z = x >= 48;
                cp_async<16>(ring_s + slot + kV3SzOff + x * 16, reinterpret_cast<const char *>(z ? vz : vs) + (src_sz + (x - 48 * z) * 16));
            }
        }
        cp_async_commit();
        --to_issue;
        src_codes += codes_step;
        src_sz += sz_step;
    };
    const char *sz_row = reinterpret_cast<const char *>(vs) + src_sz;                 // scale rows of the warp's first block
    if (MODE == 1) {
        issue_stage(0);
        // the scale rows of the blocks to come, 768 bytes (seven lines at most) each
        for (int x = lane; x < 7 * my_blocks; x += 32)
            asm volatile("prefetch.global.L2 [%0];\n" ::"l"(sz_row + (x / 7) * sz_step + min(128 * (x % 7), 764)));
        return;
    }
    --to_issue;
    src_codes += codes_step;
    src_sz += sz_step;

    const uint32_t up_s = ring_s + kV3Slots * kV3Stage + 4 * 512 + 512;               // [12] fp16 powers of two
    bool finite;
    {
        // granule x of a block's 48 holds halves 8 x .. 8 x + 7, groups 8 (x mod 3) + i (mod 12): lanes 0 .. 23 take granules
        // lane and lane + 24; magnitudes as integers, 2^-14 at least
        uint32_t mx[4] = {0x04000400u, 0x04000400u, 0x04000400u, 0x04000400u};
        if (lane < 24) {
#pragma unroll 3
            for (int q = 0; q < my_blocks; ++q) {
                const uint4 u = reinterpret_cast<const uint4 *>(sz_row + q * sz_step)[lane];
                const uint4 v = reinterpret_cast<const uint4 *>(sz_row + q * sz_step)[lane + 24];
                mx[0] = __vmaxu2(mx[0], __vmaxu2(u.x & 0x7fff7fffu, v.x & 0x7fff7fffu));
                mx[1] = __vmaxu2(mx[1], __vmaxu2(u.y & 0x7fff7fffu, v.y & 0x7fff7fffu));
                mx[2] = __vmaxu2(mx[2], __vmaxu2(u.z & 0x7fff7fffu, v.z & 0x7fff7fffu));
                mx[3] = __vmaxu2(mx[3], __vmaxu2(u.w & 0x7fff7fffu, v.w & 0x7fff7fffu));
            }
        }
#pragma unroll
        for (int o = 12; o >= 3; o >>= 1)
#pragma unroll
            for (int i = 0; i < 4; ++i) mx[i] = __vmaxu2(mx[i], __shfl_down_sync(0xffffffffu, mx[i], o));
        // lane 0 holds groups 0 .. 7, lane 1 groups 8 .. 11, 0 .. 3, lane 2 groups 4 .. 11
        uint32_t up[6];
        finite = true;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const uint32_t x = i < 2 ? __vmaxu2(__shfl_sync(0xffffffffu, mx[i], 0), __shfl_sync(0xffffffffu, mx[i + 2], 1))
                             : i < 4 ? __vmaxu2(__shfl_sync(0xffffffffu, mx[i], 0), __shfl_sync(0xffffffffu, mx[i - 2], 2))
                                     : __vmaxu2(__shfl_sync(0xffffffffu, mx[i - 4], 1), __shfl_sync(0xffffffffu, mx[i - 2], 2));
            up[i] = 0x7c007c00u - (x & 0x7c007c00u);           // exponent e of the largest: 2^(16 - e); 0 for infinity and NaN
            if (!(up[i] & 0xffffu)) { up[i] |= 0x0400u; finite = false; }      // 2^-14: the group's finite scales stay so
            if (!(up[i] >> 16)) { up[i] |= 0x04000000u; finite = false; }
        }
        if (lane == 0) {
            asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(up_s), "r"(up[0]), "r"(up[1]), "r"(up[2]), "r"(up[3]));
            asm volatile("st.shared.v2.b32 [%0], {%1,%2};\n" ::"r"(up_s + 16), "r"(up[4]), "r"(up[5]));
        }
        __syncwarp();
    }

    // field g / g + 8 of a word (see gqa_qk_packed)
    const int byte0 = (3 * g) >> 3, p0 = 3 * g - 8 * byte0;
    const uint32_t sel0 = (uint32_t)(byte0 | ((byte0 + 1) << 4) | ((4 + byte0) << 8) | ((5 + byte0) << 12));
    const uint32_t msk0 = 0x00070007u << p0, sel1 = 0x7733u;
    const uint32_t msk1 = g == 0 ? 0x00070007u : g == 1 ? 0x00380038u : g == 2 ? 0x00c000c0u : 0u;
    const int p1 = 3 * (g < 3 ? g : 0);
    // operand build: lane -> token pair pi = lane & 15, head pair hh = lane >> 4
    const int pi = lane & 15, hh = lane >> 4;
    const int bt0 = 16 * (pi >> 3) + 8 * ((pi >> 2) & 1) + 2 * (pi & 3);
    const uint32_t sz_rd = ring_s + kV3SzOff + bt0 * (W * 2);
    const uint32_t op_wr = op_s + (pi * 8 + 4 * hh) * 4, op_rd = op_s + (tig * 8 + g) * 4;
    const float *pa = sm.scores + (2 * hh) * sm.n_scores + warp * 32 + bt0, *pb = pa + sm.n_scores;
    const uint32_t w_rd = ring_s + (2 * tig) * (W * 4);
    const uint32_t g_rd = ring_s + kV3SzOff + (2 * tig) * (W * 2) + 2 * g;            // scale of (token 2 tig, group g); zeros + 768

    float acc[W][4], accz[4] = {0.f, 0.f, 0.f, 0.f}, accs[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < W; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    auto put = [&](uint32_t addr, float x0, float x1, float y0, float y1) {           // hi, lo of (x0, x1), then of (y0, y1)
        const uint32_t hx = as_u32(__floats2half2_rn(x0, x1)), hy = as_u32(__floats2half2_rn(y0, y1));
        const float2 fx = __half22float2(as_h2(hx)), fy = __half22float2(as_h2(hy));
        __half2 lx = __floats2half2_rn(x0 - fx.x, x1 - fx.y), ly = __floats2half2_rn(y0 - fy.x, y1 - fy.y);
        if (!finite) {                                         // behind an infinite hi the minimum keeps a number, and the sum infinite
            const __half2 big = __floats2half2_rn(65504.f, 65504.f);
            lx = __hmin2(lx, big);
            ly = __hmin2(ly, big);
        }
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(addr), "r"(hx), "r"(as_u32(lx)), "r"(hy), "r"(as_u32(ly)));
    };
    // A fragment of a [token][group] tile read transposed: rows g, g + 8 = groups (12 of 16), k = 16 tokens
    auto group_rows = [&](uint32_t addr, uint32_t (&r)[4]) {
        const uint32_t n = W * 2;
        r[0] = lds16(addr) | (lds16(addr + n) << 16);
        r[2] = lds16(addr + 8 * n) | (lds16(addr + 9 * n) << 16);
        r[1] = r[3] = 0u;
        if (g < W - 8) {
            r[1] = lds16(addr + 16) | (lds16(addr + n + 16) << 16);
            r[3] = lds16(addr + 8 * n + 16) | (lds16(addr + 9 * n + 16) << 16);
        }
    };

    uint32_t st = 0;
#pragma unroll 1
    for (int q = 0; q < my_blocks; ++q) {
        issue_stage(kV3Stage - st);
        cp_async_wait<1>();
        __syncwarp();
        const float2 fa = *reinterpret_cast<const float2 *>(pa), fb = *reinterpret_cast<const float2 *>(pb);
        const float a0 = 8192.f * fa.x, a1 = 8192.f * fa.y, b0 = 8192.f * fb.x, b1 = 8192.f * fb.y;
        put(pp_s + (pi * 8 + 4 * hh) * 4, a0, a1, b0, b1);
#pragma unroll
        for (int r = 0; r < W / 4; ++r) {
            const uint2 c = lds64(up_s + 8 * r), e0 = lds64(sz_rd + st + 8 * r), e1 = lds64(sz_rd + st + 8 * r + W * 2);
#pragma unroll
            for (int half = 0; half < 2; ++half) {             // groups 4 r, 4 r + 1, then 4 r + 2, 4 r + 3
                const __half2 f = as_h2(half ? c.y : c.x);
                const float2 s0 = __half22float2(__hmul2(as_h2(half ? e0.y : e0.x), f)), s1 = __half22float2(__hmul2(as_h2(half ? e1.y : e1.x), f));
                put(op_wr + (2 * half) * 512, a0 * s0.x, a1 * s1.x, b0 * s0.x, b1 * s1.x);
                put(op_wr + (2 * half + 1) * 512, a0 * s0.y, a1 * s1.y, b0 * s0.y, b1 * s1.y);
            }
            __syncwarp();
#pragma unroll
            for (int h2 = 0; h2 < 2; ++h2) {
                const uint32_t flip = h2 && finite ? 0xffffffffu : 0u, sign = flip & 0x80008000u;
                if (r == 0) {
                    const uint32_t pp_rd = pp_s + (tig * 8 + g + 64 * h2) * 4, x0 = lds32(pp_rd), x1 = lds32(pp_rd + 128);
                    uint32_t z[4];
                    group_rows(g_rd + st + h2 * 16 * (W * 2) + 32 * (W * 2), z);
                    mma16816(accz, z[0], z[1], z[2], z[3], x0, x1);
                    if (h2) {
                        group_rows(g_rd + st + h2 * 16 * (W * 2), z);
                        mma16816(accs, z[0], z[1], z[2], z[3], x0, x1);
                    }
                }
                uint32_t w[4][4];                              // tokens 2 tig, 2 tig + 1, + 8, + 9 of the k-step, words 4 r ..
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];\n" : "=r"(w[i][0]), "=r"(w[i][1]), "=r"(w[i][2]), "=r"(w[i][3])
                                 : "r"(w_rd + st + (16 * h2 + (i & 1) + 8 * (i >> 1)) * (W * 4) + 16 * r));
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const uint32_t b_lo = lds32(op_rd + u * 512 + 256 * h2) ^ sign, b_hi = lds32(op_rd + u * 512 + 256 * h2 + 128) ^ sign;
                    mma16816(acc[4 * r + u], (prmt(w[0][u], w[1][u], sel0) ^ flip) & msk0, (prmt(w[0][u], w[1][u], sel1) ^ flip) & msk1,
                             (prmt(w[2][u], w[3][u], sel0) ^ flip) & msk0, (prmt(w[2][u], w[3][u], sel1) ^ flip) & msk1, b_lo, b_hi);
                }
            }
            __syncwarp();                                      // the operand tiles (and at the end the slot) may be overwritten
        }
        st = kV3Stage - st;
        pa += kMmaWarps * 32;
        pb += kMmaWarps * 32;
    }
    cp_async_wait<0>();
    __syncwarp();
    // lane (g, tig): channels of rows g, g + 8 for head tig; the group's zero term and complement sum sit in the lanes of row j
    const float sc0 = __int_as_float((151 - 13 - p0) << 23), sc1 = __int_as_float((151 - 13 - p1) << 23);   // 2^(24 - position - 13)
    const float z0 = accz[0] + accz[1], z1 = accz[2] + accz[3], s0 = finite ? accs[0] + accs[1] : 0.f, s1 = finite ? accs[2] + accs[3] : 0.f;
    const float max1 = g == 2 ? 3.f : 7.f;                     // the 11th field has two bits
#pragma unroll
    for (int j = 0; j < W; ++j) {
        const int from = 4 * (j & 7) + tig;
        constexpr float k = 1.f / 8192.f;
        const float z = k * __shfl_sync(0xffffffffu, j < 8 ? z0 : z1, from), sv = k * __shfl_sync(0xffffffffu, j < 8 ? s0 : s1, from);
        const float undo = __int_as_float((127 + 15 - (int)(lds16(up_s + 2 * j) >> 10)) << 23);             // 1 / the group's power of two
        if (11 * j + g < kHeadDim) my_red[tig * kHeadDim + 11 * j + g] = fmaf(acc[j][0] + acc[j][1], sc0 * undo, fmaf(7.f, sv, z));
        if (g < 3 && 11 * j + 8 + g < kHeadDim) my_red[tig * kHeadDim + 11 * j + 8 + g] = fmaf(acc[j][2] + acc[j][3], sc1 * undo, fmaf(max1, sv, z));
    }
}

// ---------------------------------------------------------------------------------------------
// One segment: tokens [t0, t1) of head group s (sequence b, kv head hk, quad of query heads); segment `seg` of `cnt`.
template <int KB, int VB, bool DEV>
__device__ __forceinline__ void gqa_segment(const kvq_attn_args &a, const kvq_attn_args &ac, unsigned int before, __half2 q_mine, const AttnPlan &plan, int qhv, int s, int b, int hk, int h_first, int t0, int t1,
                                            int seg, int cnt, float *__restrict__ parts,
                                            unsigned int *__restrict__ counters) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    constexpr int kRegion = gqa_region_bytes<KB, VB>();
    const int n_scores = plan.n_scores, ks_log2 = plan.ks_log2, n_whole = plan.n_whole;
    GqaSmem sm;
    sm.n_scores = n_scores;
    sm.ks_log2 = ks_log2;
    sm.scores = reinterpret_cast<float *>(smem_raw);
    unsigned char *after_scores = smem_raw + ((size_t)kQH * n_scores << ks_log2) * 4;
    sm.ring = after_scores + warp * kRegion;
    sm.q = reinterpret_cast<__half *>(after_scores + kMmaWarps * kRegion);
    sm.misc = reinterpret_cast<float *>(sm.q + kQH * kHeadDim);

    const int v_hi = min(t1, a.Tvq), v_lo = max(t0, a.Tvq);
    const __half *vf = static_cast<const __half *>(a.vfull) + (int64_t)b * a.vf_sB + (int64_t)hk * a.vf_sH;
    const __half *kf = static_cast<const __half *>(a.kfull) + (int64_t)b * a.kf_sB + (int64_t)hk * a.kf_sH;
    prefetch_tails(a, kf, vf, b, hk, t0, t1, tid, kMmaThreads);
    fused_cache_update<KB, VB, kMmaThreads>(a, b, hk, t0, t1, tid);        // the step's own cache update, when the caller fused it in
    *reinterpret_cast<__half2 *>(sm.q + (tid >> 6) * kHeadDim + 2 * (tid & 63)) = q_mine;                  // two warps store a head slot

    // ---- 1. scores ------------------------------------------------------------------------------
    {
        const int32_t *kc = a.kcode + (int64_t)b * a.kc_sB + (int64_t)hk * a.kc_sH;
        const __half *ks = static_cast<const __half *>(a.kscale) + (int64_t)b * a.ks_sB + (int64_t)hk * a.ks_sH;
        const __half *kz = static_cast<const __half *>(a.kmn) + (int64_t)b * a.ks_sB + (int64_t)hk * a.ks_sH;
        constexpr bool kEarly = !DEV && KB + VB >= 6;          // see gqa_qk_tail
        if (KB != 1 && (KB == 3 || a.k_group == 64)) gqa_qk_packed<KB, false, kEarly>(a, kc, ks, kz, sm, t0, min(t1, a.Tkq), kf, max(t0, a.Tkq), t1, b, hk);
        else gqa_qk_packed<KB, KB != 3, kEarly>(a, kc, ks, kz, sm, t0, min(t1, a.Tkq), kf, max(t0, a.Tkq), t1, b, hk);
    }
    const int32_t *vc = a.vcode + (int64_t)b * a.vc_sB + (int64_t)hk * a.vc_sH;
    const __half *vs = static_cast<const __half *>(a.vscale) + (int64_t)b * a.vs_sB + (int64_t)hk * a.vs_sH;
    const __half *vz = static_cast<const __half *>(a.vmn) + (int64_t)b * a.vs_sB + (int64_t)hk * a.vs_sH;
    if constexpr (VB == 3) gqa_pv_packed3<1>(a, vc, vs, vz, sm, t0, v_hi);
    else gqa_pv<VB, 1>(a, vc, vs, vz, sm, t0, v_hi);         // start filling this warp's value ring now
    __syncthreads();

    // ---- 2. softmax numerators: two warps per head slot --------------------------------------------
    const int n = t1 - t0, n4 = (n + 3) >> 2, hs_mine = warp >> 1;
    const int h_mine = h_first + min(hs_mine, qhv - 1);
    float m = kMaskFloor;
    float4 *sc4 = reinterpret_cast<float4 *>(sm.scores + hs_mine * n_scores);
#pragma unroll 4
    for (int i = tid & 63; i < n4; i += 64) {
        float4 v = score_quad(a, sc4 + i, kQH * (n_scores >> 2), ks_log2);
        if (a.mask) mask_quad(a, b, h_mine, t0 + 4 * i, v);
        if (4 * i + 3 >= n) pad_quad(v, n - 4 * i);
        sc4[i] = v;
        m = fmaxf(fmaxf(m, fmaxf(v.x, v.y)), fmaxf(v.z, v.w));
    }
    m = warp_max(m);
    if (lane == 0) sm.misc[warp] = m;
    __syncthreads();
    m = fmaxf(sm.misc[2 * hs_mine], sm.misc[2 * hs_mine + 1]);
    float l = 0.f;
#pragma unroll 4
    for (int i = tid & 63; i < n4; i += 64) {
        float4 v = sc4[i];
        v.x = __expf(v.x - m);
        v.y = __expf(v.y - m);
        v.z = __expf(v.z - m);
        v.w = __expf(v.w - m);
        sc4[i] = v;
        l += (v.x + v.y) + (v.z + v.w);
    }
    l = warp_sum(l);
    if (lane == 0) sm.misc[8 + warp] = l;
    __syncthreads();

    // ---- 3. p . V -----------------------------------------------------------------------------------
    if constexpr (VB == 3) gqa_pv_packed3<2>(a, vc, vs, vz, sm, t0, v_hi);
    else gqa_pv<VB, 2>(a, vc, vs, vz, sm, t0, v_hi);
    __syncwarp();
    if (v_lo < t1) pv_tail<kQH>(a, vf, b, hk, sm.scores, n_scores, t0, v_lo, t1, reinterpret_cast<float *>(sm.ring), warp, kMmaWarps, lane);
    __syncthreads();

    if (ac.state) dev_state_publish(ac, a, before);

    launch_next();                                             // what is left is short: the next launch may come

    // ---- 4. finish / merge: a thread owns channel ch of head slots 2 hp, 2 hp + 1 -------------------------
    constexpr int kPart = kPartStride;
    const int ch = tid & (kHeadDim - 1), hp = tid >> 7, n_mine = max(0, min(2, qhv - 2 * hp));
    float o[2];
    __half res[2] = {};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < kMmaWarps; ++w) v += reinterpret_cast<const float *>(after_scores + w * kRegion)[(2 * hp + i) * kHeadDim + ch];
        o[i] = v;
    }
    __half *out = static_cast<__half *>(a.out) + (int64_t)b * a.o_sB + (int64_t)(h_first + 2 * hp) * a.o_sH + ch;
    if (cnt == 1) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (i < n_mine) {
                const int hs = 2 * hp + i;
                res[i] = __float2half_rn(o[i] / (sm.misc[8 + 2 * hs] + sm.misc[9 + 2 * hs]));
                out[(int64_t)i * a.o_sH] = res[i];
            }
        }
        peer_publish(ac, b, h_first + 2 * hp, n_mine, res, ch, tid, qhv);
        return;
    }
    float *part = parts + ((int64_t)(s - n_whole) * cnt + seg) * qhv * kPart;    // partials of the cut head groups only
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        if (i < n_mine) {
            const int hs = 2 * hp + i;
            part[hs * kPart + ch] = o[i];
            if (ch == 0) {
                part[hs * kPart + kHeadDim] = fmaxf(sm.misc[2 * hs], sm.misc[2 * hs + 1]);
                part[hs * kPart + kHeadDim + 1] = sm.misc[8 + 2 * hs] + sm.misc[9 + 2 * hs];
            }
        }
    }
    __syncthreads();
    if (tid == 0) {
        sm.misc[16] = count_in(&counters[s]) == (unsigned)(cnt - 1) ? 1.f : 0.f;
    }
    __syncthreads();
    if (sm.misc[16] == 0.f) return;
    // The last CTA merges the cnt segments of its head group.  A long context over few heads means a hundred or more
    // segments, and a merge that walks them one dependent round trip at a time becomes the kernel, so many 128-bit loads
    // are kept in flight: warp w merges head slot w, lane l owning channels 4l .. 4l + 3; the maximum over the segments
    // first (lanes over segments), then the weighted sums, sixteen segments' loads issued before the first is used.  The
    // order is fixed, so results are run-to-run identical.
    __half *stage = reinterpret_cast<__half *>(after_scores);             // [kQH][128] results, regions are idle by now
    if (warp < qhv) {
        const float *bh = parts + (int64_t)(s - n_whole) * cnt * qhv * kPart + warp * kPart;
        const int stride = qhv * kPart;
        float M = kMaskFloor;
        for (int i = lane; i < cnt; i += 32) M = fmaxf(M, __ldcg(bh + (int64_t)i * stride + kHeadDim));
        M = warp_max(M);
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        float L = 0.f;
        constexpr int U = 16;                                  // loads in flight; behind the last segment it is read again, as zeros
        for (int i0 = 0; i0 < cnt; i0 += U) {
            float2 ml[U];
            float4 p[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const float *pi = bh + (int64_t)min(i0 + u, cnt - 1) * stride;
                ml[u] = __ldcg(reinterpret_cast<const float2 *>(pi + kHeadDim));
                p[u] = __ldcg(reinterpret_cast<const float4 *>(pi) + lane);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const bool in = i0 + u < cnt;
                const float w = __expf(ml[u].x - M);
                L = fmaf(in ? ml[u].y : 0.f, w, L);
                acc.x = fmaf(in ? p[u].x : 0.f, w, acc.x); acc.y = fmaf(in ? p[u].y : 0.f, w, acc.y);
                acc.z = fmaf(in ? p[u].z : 0.f, w, acc.z); acc.w = fmaf(in ? p[u].w : 0.f, w, acc.w);
            }
        }
        const float inv = 1.f / L;
        __half2 *dst = reinterpret_cast<__half2 *>(stage + warp * kHeadDim + 4 * lane);
        dst[0] = __floats2half2_rn(acc.x * inv, acc.y * inv);
        dst[1] = __floats2half2_rn(acc.z * inv, acc.w * inv);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        if (i < n_mine) {
            res[i] = stage[(2 * hp + i) * kHeadDim + ch];
            out[(int64_t)i * a.o_sH] = res[i];
        }
    }
    if (tid == 0) counters[s] = 0u;
    peer_publish(ac, b, h_first + 2 * hp, n_mine, res, ch, tid, qhv);
}

template <int KB, int VB, bool DEV>
__global__ void __launch_bounds__(kMmaThreads, 2) decode_attn_gqa_kernel(const __grid_constant__ kvq_attn_args a,
                                                                     const __grid_constant__ AttnPlan plan, int qhv,
                                                                     float *__restrict__ parts,
                                                                     unsigned int *__restrict__ counters) {
    grid_wait();
    DevState state;
    if constexpr (DEV) state = dev_state_load(a);
    int group, seg, b, hk, within, t0, t1, cnt;
    plan_head(plan, blockIdx.x, group, seg);
    plan_place(plan, group, b, hk, within);
    const int h_first = hk * plan.rep + within * qhv;
    // this thread's two channels of q (head slots beyond qhv repeat the last head: their columns are computed and dropped): the key
    // phase waits for them, and nothing of them depends on the cache's state
    const __half *q = static_cast<const __half *>(a.q) + (int64_t)b * a.q_sB + (int64_t)(h_first + min((int)threadIdx.x >> 6, qhv - 1)) * a.q_sH + 2 * (threadIdx.x & 63);
    const __half2 q_mine = __halves2half2(q[0], q[1]);         // q rows start at any fp16
    if constexpr (DEV) {                                       // device-resident cache state: see decode_attn_mma_kernel
        kvq_attn_args d = a;
        const unsigned int before = dev_state_step(a, state, d);
        plan_tokens(plan, d.T, blockIdx.x, seg, t0, t1, cnt);
        if (cnt > 1) cnt = min(cnt, (d.T + plan.seg_units * plan.unit - 1) / (plan.seg_units * plan.unit));
        if (t0 < d.T) gqa_segment<KB, VB, true>(d, a, before, q_mine, plan, qhv, group, b, hk, h_first, t0, t1, seg, cnt, parts, counters);
        else dev_state_publish(a, d, before);
    } else {
        plan_tokens(plan, a.T, blockIdx.x, seg, t0, t1, cnt);
        gqa_segment<KB, VB, false>(a, a, 0u, q_mine, plan, qhv, group, b, hk, h_first, t0, t1, seg, cnt, parts, counters);
    }
}

// ---------------------------------------------------------------------------------------------
// Query heads per CTA for this call (0: the grouped kernel does not take it and the single-head kernel runs): the
// heads of a kv head in quads (or the pair, for two heads per kv head), and group sizes that keep an MMA's rows in
// one group.
int gqa_heads_per_cta(const kvq_attn_args &a) {
    if (a.nh_kv <= 0 || a.nh % a.nh_kv != 0) return 0;
    const int n_rep = a.nh / a.nh_kv;
    if (n_rep != 2 && n_rep % 4 != 0) return 0;
    const int kmin = a.k_bits == 1 ? 128 : a.k_bits == 2 ? 64 : a.k_bits == 4 ? 64 : 11;
    const int vmin = a.v_bits == 1 ? 64 : a.v_bits == 2 ? 64 : a.v_bits == 3 ? 11 : 32;     // 1-bit values at group 64: two MMAs per code tile
    if (a.k_bits != 3 && a.k_group < kmin) return 0;
    if (a.v_group < vmin) return 0;
    return n_rep == 2 ? 2 : 4;
}

AttnPlan plan_attn_gqa(int T, int k_bits, long long head_groups) {
    return k_bits == 3 ? make_attn_plan(T, 352, KGeom<3>::WT, kGqaMaxScores3, head_groups)
                       : make_attn_plan(T, 256, KGeom<4>::WT, kGqaMaxScores, head_groups);
}

template <int KB, int VB> constexpr int gqa_smem_bytes(int scores) {
    return kQH * scores * 4 + kMmaWarps * gqa_region_bytes<KB, VB>() + kQH * kHeadDim * 2 + 64 * 4;
}

template <int KB, int VB>
static int launch_gqa(const kvq_attn_args &a, AttnPlan plan, int qhv, float *parts, unsigned int *counters,
                      cudaStream_t st) {
    plan_set_place(plan, a.nh, a.nh_kv, a.nh / a.nh_kv / qhv);
    static_assert(gqa_smem_bytes<KB, VB>(KB == 3 ? kGqaMaxScores3 : kGqaMaxScores) <= kMmaSmemMax, "two CTAs to an SM");
    const size_t smem = gqa_smem_bytes<KB, VB>(plan.n_scores << plan.ks_log2);
    static bool attr_set[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return record_cuda_error(e);
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        e = cudaFuncSetAttribute(decode_attn_gqa_kernel<KB, VB, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMmaSmemMax);
        if (VB != 3 && e == cudaSuccess)
            e = cudaFuncSetAttribute(decode_attn_gqa_kernel<KB, VB == 3 ? 4 : VB, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMmaSmemMax);
        if (e != cudaSuccess) return record_cuda_error(e);
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    const unsigned grid = (unsigned)(plan.n_whole + plan.n_cut * plan.k);
    // launched early (grid_wait): four small layers of 4 x 8 kv heads x 1537 tokens from a host loop 69.5 -> 60.2 us, 131k tokens from a graph
    // 407 -> 403; let in at the start of the kernel instead of behind p . V the next launch's CTAs cost more than they gain (66.7)
    if (VB != 3 && a.state) return launch_early(plan_early(plan), decode_attn_gqa_kernel<KB, VB == 3 ? 4 : VB, true>, grid, kMmaThreads, smem, st, a, plan, qhv, parts, counters);
    return launch_early(plan_early(plan), decode_attn_gqa_kernel<KB, VB, false>, grid, kMmaThreads, smem, st, a, plan, qhv, parts, counters);
}

int launch_decode_attn_gqa(const kvq_attn_args &a, const AttnPlan &plan, int qhv, float *parts, unsigned int *counters,
                           cudaStream_t st) {
#define KVQ_GQA_CASE(KB, VB) \
    if (a.k_bits == KB && a.v_bits == VB) return launch_gqa<KB, VB>(a, plan, qhv, parts, counters, st);
    KVQ_GQA_CASE(4, 4) KVQ_GQA_CASE(4, 2) KVQ_GQA_CASE(4, 1)
    KVQ_GQA_CASE(3, 4) KVQ_GQA_CASE(3, 2) KVQ_GQA_CASE(3, 1)
    KVQ_GQA_CASE(2, 4) KVQ_GQA_CASE(2, 2) KVQ_GQA_CASE(2, 1)
    KVQ_GQA_CASE(1, 4) KVQ_GQA_CASE(1, 2) KVQ_GQA_CASE(1, 1)
    KVQ_GQA_CASE(4, 3) KVQ_GQA_CASE(3, 3) KVQ_GQA_CASE(2, 3) KVQ_GQA_CASE(1, 3)
#undef KVQ_GQA_CASE
    return KVQ_ERR_UNSUPPORTED;
}

}  // namespace kvq
