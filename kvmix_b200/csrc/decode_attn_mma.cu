// Fused decode attention, tensor-core path: one CTA (8 warps, or 4) per query head and token split; the query heads of a
// kv head are neighbouring CTAs and share its cache through L2.
//
// Why tensor cores for a mat-vec: at the HBM rate a B200 has only ~1-3 issue slots per packed code (2.8 per 2-bit
// code at 5.6 TB/s and 1.9 GHz).  Shift-mask-convert-FMA per code does not fit; one logic op per *pair* of codes
// plus one mma.sync per 256 codes does.
//
// Codes go to the tensor core without ever being converted: a b-bit field left in place inside a 16-bit lane, with
// all other bits masked off, *is* an fp16 number with value field * 2^(pos-24) (subnormals and the first normal
// binade are linear in the bit pattern).  mma.sync multiplies such inputs exactly and accumulates in fp32, so the
// product with the fp16 operand is exact and the power of two is undone per output row in the epilogue.  Pairs
// along the contraction axis arrive ready-made from transposing ldmatrix loads (values; 1- and 2-bit keys) or are
// formed with one byte-permute of two words (3- and 4-bit keys).
//
// Keys (codes [D, T/fpi], one word = fpi tokens of one channel; scale/zero [D, T/G]):
//   A (16x16) = codes, rows = tokens, cols = 16 channels.  q[d]*scale[d,g] is carried as an exact fp16 pair hi + lo.
//   A 256-token warp tile is worked as two halves whose MMA rows touch at most four groups, so B (16x8) holds
//   {hi, lo} x 4 groups side by side and one MMA per code tile yields both parts.  3-bit keys (tiles of 88 or 176 tokens,
//   every word its own group of 11) multiply each code tile by the hi and by the lo operand instead.  The zero terms
//   sum_d q[d]*zero[d,g] of all groups of a tile come from one MMA per 16 channels whose A operand is the zero tile
//   read transposed (row = group) and whose B operand is q.
// Values (codes [T, D/fpi], one word = fpi channels of one token; scale/zero [T, D/G]):
//   A (16x16) = codes, rows = channels, cols = 16 tokens;  B (16x8): column 2j = p[t]*scale[t,j], column 2j+1 =
//   p[t]*midpoint[t,j] (codes are used centred on the group midpoint); one extra MMA with A = ones sums both columns.
// Code words and scale/zero rows stream through per-warp multi-stage cp.async rings in shared memory (128-bit
// copies, several KB in flight per warp).  The fp16 key tail is scored on the tensor cores straight from global
// memory; the softmax, the optional additive mask and the fp16 value tail run on the CUDA cores.
#include "attn_mma_common.cuh"
#include "attn_plan.cuh"
#include "attn_update.cuh"

namespace kvq {

// Score buffers: of an eight-warp CTA, two to an SM; of a four-warp CTA, three to an SM, and four to an SM.
constexpr int kWideScores = 6144, kWideScores3 = 7040, kNarrowMax = 8192, kNarrowMax3 = 8096, kNarrowScores = 5216;

// Key geometry of this kernel.  3 bits come in two forms with the same sums in the same order.  H = 1: one word (group) an octet, tiles
// of 88 tokens, 32 channels a stage.  H = 2: two words an octet, tiles of 176 tokens, 16 channels a stage -- what a k-step does once
// (q, addresses, copies, loop) is a third of the instructions of H = 1, and a channel row is fetched 64 bytes at a time.  But a warp whose
// last pass is half empty works 88 tokens for nothing.  us, all in tiles of 88 / all in tiles of 176 (laid out as one tile's work) / this
// choice, 2-bit values: 2048 heads of 4096 tokens 278 / 273 / 272, 1024 of 2000 85.3 / 82.1 / 82.3, 256 of 9000 101 / 102 / 101,
// 230 of 9000 91 / 100 / 91, 160 of 3001 36.0 / 38.7 / 35.2, 64 of 6000 27.5 / 26.4 / 25.9, 64 of 704 11.2 / 12.2 / 11.4.
template <int KB, int H> struct MmaKGeom : KGeom<KB> { static constexpr int SZ = 2 * KGeom<KB>::ROWS * 16; };
template <> struct MmaKGeom<3, 2> {
    static constexpr int FPI = 11, WPL = 2, TPO = 11, WT = 176, KSPS = 1, NSTAGE = 8, NMMA = 12;
    static constexpr int RB = 64, RS = RB + 16, ROWS = 16, CODE_BYTES = ROWS * RS, GPR = RB / 16, GPL = ROWS * GPR / 32, RPI = 32 / GPR;
    static constexpr int SZ = 2 * ROWS * 32;                           // [half of the tile][scales, zeros][channel][8 groups]
};
// The form for a segment of n packed tokens: the larger tile where the slowest warp works no more tokens than in tiles of 88, or one tile of
// 88 more out of sixteen -- out of five where two or four warps share a tile's channels, and what a tile costs once counts double.
__device__ __forceinline__ bool wide_key_tiles(int n, int warps, int ks_log2) {
    auto passes = [&](int tile) { return (((n + tile - 1) / tile << ks_log2) + warps - 1) / warps; };
    const int p = passes(MmaKGeom<3, 1>::WT);
    return n > 0 && 2 * passes(MmaKGeom<3, 2>::WT) <= p + (p >= (ks_log2 ? 5 : 16));
}

struct MmaSmem {
    float *scores;          // [1 << ks_log2][n_scores]
    unsigned char *ring;    // this warp's region
    __half *q;              // [kHeadDim]
    float *misc;            // [32]
    int n_scores, ks_log2;
};
// Rings of a CTA of NW warps: the scale rows, then the zero rows of a stage, 16 B each, follow its codes.  Four warps: sized so
// that four CTAs fit an SM next to 5000 scores each.
template <int KB, int NW, int H> struct MmaKRing {
    static constexpr int NS = (KB == 2 ? 3 : 4) - (NW == 4), P = NS - 1;
    static constexpr int STAGE_BYTES = MmaKGeom<KB, H>::CODE_BYTES + MmaKGeom<KB, H>::SZ;
    static constexpr int BYTES = NS * STAGE_BYTES;
};
template <int VB, int NW> using MmaVGeom = VGeom<VB, (VB == 4 ? 4 : VB == 2 ? 6 : 8) - (NW == 4 && VB != 1)>;
template <int KB, int VB, int NW> constexpr int warp_region_bytes() {
    static_assert(KB != 3 || MmaKRing<3, NW, 2>::BYTES <= MmaKRing<3, NW, 1>::BYTES, "one ring for both forms");
    return MmaKRing<KB, NW, 1>::BYTES > MmaVGeom<VB, NW>::WARP_BYTES ? MmaKRing<KB, NW, 1>::BYTES : MmaVGeom<VB, NW>::WARP_BYTES;
}

// ---------------------------------------------------------------------------------------------
// q . K^T over packed keys for tokens [t0, hi) (t0 is a multiple of 256, or 352 for 3-bit keys).
// Raw fp32 scores go to sm.scores[split][t - t0].  Warps work independently: with `ns` = 1 << ks_log2 channel splits, warp w
// takes channels [128 / ns * (w % ns), ..) of the warp tiles w / ns, w / ns + 8 / ns, ... and streams their code words
// through its own ring.
template <int NW>
__device__ __forceinline__ void qk_tail_mma(const kvq_attn_args &a, const __half *kf, int b, int hk, const MmaSmem &sm,
                                            int t0, int lo, int t1);

// If the split also holds fp16 tail keys (tail_lo < t1) they are scored right after the first code stages
// have been issued, so the tail's global-load latency overlaps the ring fill.
// LGK: log2 of the group size; H: words an octet owns of 3-bit keys (MmaKGeom).
template <int KB, int NW, int LGK, int H>
__device__ __forceinline__ void qk_packed_mma(const kvq_attn_args &a, const int32_t *kc, const __half *ks,
                                              const __half *kz, const MmaSmem &sm, int t0, int hi,
                                              const __half *kf, int tail_lo, int t1, int b, int hk) {
    using G = MmaKGeom<KB, H>;
    using R = MmaKRing<KB, NW, H>;
    using F = Fields<KB>;
    const int warp = uniform_warp(), lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    const int n_words = a.Tkq / G::FPI;                       // valid code words per channel row
    const int n_tiles = (hi - t0 + G::WT - 1) / G::WT;
    const int split = warp & ((1 << sm.ks_log2) - 1), wt = warp >> sm.ks_log2, tile_lanes = NW >> sm.ks_log2;
    const int my_tiles = (n_tiles - wt + tile_lanes - 1) / tile_lanes;   // <= 0: none
    const int ch0 = split * (kHeadDim >> sm.ks_log2), steps = (kHeadDim / 32) >> sm.ks_log2;   // channels of this warp
    const int tile_stages = G::NSTAGE >> sm.ks_log2;

    const int kc_sD = (int)a.kc_sD, ks_sD = (int)a.ks_sD;
    // ---- per-lane constants --------------------------------------------------------------------
    const uint32_t ring_s = smem_u32(sm.ring);
    const int gr = lane % G::GPR, row0 = lane / G::GPR;
    const uint32_t cp_dst = ring_s + row0 * G::RS + gr * 16;                   // + slot*STAGE + i*RPI*RS
    // 3-bit: octet g owns the word of group g (11 tokens) of each half (H) of the tile, fetched with plain 32-bit loads.
    // Other widths: code fragments come from transposing ldmatrix loads.  A channel row of the tile is NBK blocks of
    // 16 bytes; one x4 load covers channel rows 16 ksx + (0..7 | 8..15) x two neighbouring blocks and hands lane
    // (g, tig) the half-word g of each block for the channel pair (2 tig, 2 tig + 1) [+8]: an A-fragment register pair
    // along k without a byte permute.  Octet g of block bb therefore owns tokens bb * 8 FH + g * FH .. + FH - 1
    // (FH = 16 / bits fields per half-word).  The first NBK / 2 blocks are the first 128 tokens: their MMA rows touch
    // at most four groups, so the eight B columns carry {hi, lo} of q*scale for those four side by side (b0); the
    // other blocks use b1.
    constexpr int FH = (KB == 3) ? 2 : 16 / KB;                                // fields per half-word: 4 / 8 / 16
    constexpr int NBK = G::RB / 16;                                            // 16-byte blocks per channel row: 8 / 4 / 2
    constexpr int MPB = FH / 2;                                                // MMAs per block and k-step: 2 / 4 / 8
    constexpr int HW = 2;                                                      // 4-bit: code words per octet per half
    const uint32_t frag_s = ring_s + (2 * tig) * G::RS + ((KB == 4) ? 8 * g : 4 * g);   // 3-bit and 4-bit (plain loads)
    const uint32_t ldk_s = ring_s + ((lane & 7) + 8 * ((lane >> 3) & 1)) * G::RS + (lane >> 4) * 16;   // + k*16*RS + 32*pair
    // ldmatrix.x4 row addresses: lanes 0-7 scale rows 0..7 of a k-step, 8-15 scale rows 8..15, 16-31 the same of the zero rows
    const uint32_t ldm_s = ring_s + G::CODE_BYTES + (((lane >> 3) & 1) * 8 + (lane & 7)) * 16 + (lane >> 4) * (G::ROWS * 16);
    const uint32_t q_s = smem_u32(sm.q) + (ch0 + 2 * tig) * 2;                 // + 32 per k-step [+16]
    constexpr int ngw = KB == 3 ? 8 * H : G::WT >> LGK;                        // groups per warp tile: 16 / 8 / 4 / 2
    const uint32_t szcp_dst = ring_s + G::CODE_BYTES + lane * 16;                  // one granule per lane (16 channels a stage) or two
    const int tile_words = tile_lanes * G::WT / G::FPI;                        // word-column distance between my tiles
    const int tile_groups = tile_lanes * ngw;

    // the next stage to issue: its addresses, its word column, its position in its tile and the tiles left.  Stages
    // carry the scale and zero rows of their own channels, so the operands are formed k-step by k-step and the loop over
    // a tile's stages stays rolled (two k-steps a turn; unrolled over all
    // eight it missed the instruction cache: 1.6 of 7.9 cycles per issued instruction were fetch stalls, 0.4 now).
    uint32_t iss = 4u * ((uint32_t)(ch0 + row0) * kc_sD + (t0 + wt * G::WT) / G::FPI + 4 * gr);   // bytes from the head's first word
    constexpr bool kOneSz = 2 * G::ROWS == 32;                                 // 16 channels: lanes 16-31 fetch the zero rows
    const int sz_row = kOneSz ? (lane & 15) : lane;
    uint32_t iss_s = 2u * ((uint32_t)(ch0 + sz_row) * ks_sD + (KB == 3 ? (t0 + wt * G::WT) / 11 : (t0 + wt * G::WT) >> LGK));
    const char *sz_b = reinterpret_cast<const char *>(kOneSz && lane >= 16 ? kz : ks);
    int iss_col = (t0 + wt * G::WT) / G::FPI + 4 * gr, iss_st = 0, iss_tiles = my_tiles;
    uint32_t iss_slot = 0, slot = 0;                                            // byte offsets of the slot being filled / read
    bool iss_ok = iss_col < n_words;
    int iss_second = n_words - ((t0 + wt * G::WT) / G::FPI + 8);                // H = 2: > 0: the second half of the tile's groups exists

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
            if (KB == 3 && H == 2) {
                cp_async<16>(d, sz_b + iss_s);
                if (iss_second > 0) cp_async<16>(d + G::SZ / 2, sz_b + (iss_s + 16));
            } else if (ngw == 8) { cp_async<16>(d, sz_b + iss_s); if (!kOneSz) cp_async<16>(d + G::ROWS * 16, kz_b + iss_s); }
            else if (ngw == 4) { cp_async<8>(d, sz_b + iss_s); if (!kOneSz) cp_async<8>(d + G::ROWS * 16, kz_b + iss_s); }
            else { cp_async<4>(d, sz_b + iss_s); if (!kOneSz) cp_async<4>(d + G::ROWS * 16, kz_b + iss_s); }
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
            iss_second -= tile_words;
            --iss_tiles;
        }
    };

#pragma unroll 1
    for (int q = 0; q < R::P; ++q) issue_stage();
    // The caller stored q to shared memory just before this call without a barrier, so that the first code stages
    // are in flight while q arrives; every warp passes exactly one barrier here before anything reads q.
    __syncthreads();
    if (tail_lo < t1) qk_tail_mma<NW>(a, kf, b, hk, sm, t0, tail_lo, t1);

    for (int j = 0; j < my_tiles; ++j) {
        const int tile0 = t0 + (j * tile_lanes + wt) * G::WT;
        uint32_t q_cur = q_s;

        // ---- B fragments q*scale and the zero term sum_d q[d]*zero[d,g] ----------------------------------
        // q*scale needs 22 bits; it is carried as an fp16 pair hi + lo (lo = fma(q, s, -hi) is exact), so the key
        // side adds no rounding beyond the fp32 accumulation.
        // 3-bit keys: hi and lo of the eight groups of a half of the tile, every code tile is multiplied by both.
        // Other widths: b0 / b1 serve the first / second half of the tile; column n carries group (n / 2) of that
        // half, hi in even and lo in odd columns, so one MMA per code tile yields both parts.
        float zsum = 0.f, zsum3 = 0.f;                         // (H = 2: of the halves of the tile)
        constexpr int gph = ngw / 2;                           // groups per half tile: 4 / 2 / 1
        const int src0 = 4 * ((g >> 1) % gph) + tig;           // lane holding group (n / 2) of the first half
        const int src1 = src0 + 4 * (ngw / 2);
        const uint32_t neg_mask = (g & 1) ? 0xffffffffu : 0u;  // odd columns: the lo part

        float acc[G::NMMA][4];
#pragma unroll
        for (int m = 0; m < G::NMMA; ++m) acc[m][0] = acc[m][1] = acc[m][2] = acc[m][3] = 0.f;

#pragma unroll 1
        for (int it = 0; it < steps; ++it) {
          float accz[4] = {0.f, 0.f, 0.f, 0.f}, accz3[4] = {0.f, 0.f, 0.f, 0.f};      // zero terms of two k-steps
#pragma unroll
          for (int s2 = 0; s2 < 2 / G::KSPS; ++s2) {
            issue_stage();
            cp_async_wait<R::P>();
            __syncwarp();
            const uint32_t src = frag_s + slot;
#pragma unroll
            for (int k = 0; k < G::KSPS; ++k) {
                const uint32_t q01u = lds32(q_cur), q89u = lds32(q_cur + 16);
                q_cur += 32;
                const __half2 q01 = as_h2(q01u), q89 = as_h2(q89u);
                if constexpr (KB == 3) {
#pragma unroll
                    for (int hf = 0; hf < H; ++hf) {
                        uint32_t r0, r1, r2, r3;               // scales and zeros of this half's eight groups, see below
                        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                                     : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(ldm_s + slot + k * 256 + hf * (G::SZ / 2)));
                        if (hf) mma16816(accz3, r2, 0u, r3, 0u, q01u, q89u);
                        else mma16816(accz, r2, 0u, r3, 0u, q01u, q89u);
                        const __half2 s01 = as_h2(r0), s89 = as_h2(r1);
                        const __half2 p01 = __hmul2(q01, s01), p89 = __hmul2(q89, s89);
                        const uint32_t hi0 = as_u32(p01), hi1 = as_u32(p89);
                        const uint32_t lo0 = as_u32(__hfma2(q01, s01, __hneg2(p01))), lo1 = as_u32(__hfma2(q89, s89, __hneg2(p89)));
                        uint32_t w[4];
#pragma unroll
                        for (int r = 0; r < 4; ++r) w[r] = lds32(src + 32 * hf + (k * 16 + (r & 1) + (r >> 1) * 8) * G::RS);
                        uint32_t rlo[F::N], rhi[F::N];
                        F::unpack(w[0], w[1], rlo);
                        F::unpack(w[2], w[3], rhi);
#pragma unroll
                        for (int i = 0; i < F::N; i += 2) {
                            const uint32_t a1 = (i + 1 < F::N) ? rlo[i + 1] : 0u, a3 = (i + 1 < F::N) ? rhi[i + 1] : 0u;
                            mma16816(acc[6 * hf + i / 2], rlo[i], a1, rhi[i], a3, hi0, hi1);
                        }
#pragma unroll
                        for (int i = 0; i < F::N; i += 2) {
                            const uint32_t a1 = (i + 1 < F::N) ? rlo[i + 1] : 0u, a3 = (i + 1 < F::N) ? rhi[i + 1] : 0u;
                            mma16816(acc[6 * hf + i / 2], rlo[i], a1, rhi[i], a3, lo0, lo1);
                        }
                    }
                } else {
                // the tile rows are 8 groups x fp16 = one 8x8 matrix per 8 channels: a transposing ldmatrix hands
                // lane (g, tig) exactly {row 2tig, row 2tig+1} x column g, i.e. its B-fragment pairs of group g, in one go
                // (with fewer than 8 groups per tile the columns past the last group are stale and feed unused columns)
                uint32_t r0, r1, r2, r3;
                asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                             : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(ldm_s + slot + k * 256));
                // The zero terms: the same two registers are also the A fragment of the transposed zero tile (row = group g,
                // k = channels 2tig, 2tig+1 / +8), so ONE MMA with B = q (in every column) leaves sum_d q[d] * zero[d, g] in
                // row g; fp16 x fp16 products are exact in the tensor core, no hi / lo split is needed.  Chains of
                // two MMAs (the tensor core truncates as it accumulates).  A stale group only spoils its own row.
                mma16816(accz, r2, 0u, r3, 0u, q01u, q89u);
                uint32_t b0[2], b1[2];
                {
                    b0[0] = hilo(q01, as_h2(__shfl_sync(0xffffffffu, r0, src0)), neg_mask);
                    b0[1] = hilo(q89, as_h2(__shfl_sync(0xffffffffu, r1, src0)), neg_mask);
                    b1[0] = hilo(q01, as_h2(__shfl_sync(0xffffffffu, r0, src1)), neg_mask);
                    b1[1] = hilo(q89, as_h2(__shfl_sync(0xffffffffu, r1, src1)), neg_mask);
                }
                if constexpr (KB == 4) {
                    // 4-bit keys: two words (16 tokens) per octet and half, plain 64-bit loads + byte permutes (measured 1.5 %
                    // faster than the ldmatrix form below for this width: 4 loads of 2 blocks each per k-step)
                    constexpr int NF = F::N;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        uint32_t w[4][HW];
#pragma unroll
                        for (int r = 0; r < 4; ++r) {
                            const uint32_t ad = src + (k * 16 + (r & 1) + (r >> 1) * 8) * G::RS + h * (G::RB / 2);
                            asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];\n" : "=r"(w[r][0]), "=r"(w[r][1]) : "r"(ad));
                        }
#pragma unroll
                        for (int x = 0; x < HW; ++x) {
                            uint32_t rlo[F::N], rhi[F::N];
                            F::unpack(w[0][x], w[1][x], rlo);
                            F::unpack(w[2][x], w[3][x], rhi);
#pragma unroll
                            for (int i = 0; i < NF; i += 2) {
                                const int m = h * 8 + (x * NF + i) / 2;
                                if (h == 0) mma16816(acc[m], rlo[i], rlo[i + 1], rhi[i], rhi[i + 1], b0[0], b0[1]);
                                else mma16816(acc[m], rlo[i], rlo[i + 1], rhi[i], rhi[i + 1], b1[0], b1[1]);
                            }
                        }
                    }
                } else {
                    using H = KHalf<KB>;
                    const uint32_t lsrc = ldk_s + slot + (k * 16) * G::RS;
#pragma unroll
                    for (int pb2 = 0; pb2 < NBK / 2; ++pb2) {              // two blocks per load
                        uint32_t x[2][2];
                        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                                     : "=r"(x[0][0]), "=r"(x[0][1]), "=r"(x[1][0]), "=r"(x[1][1]) : "r"(lsrc + pb2 * 32));
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int bb = 2 * pb2 + u;
                            uint32_t rlo[H::N], rhi[H::N];
                            H::unpack(x[u][0], rlo);                        // channels 2tig, 2tig+1  -> k cols 2tig, 2tig+1
                            H::unpack(x[u][1], rhi);                        // channels 2tig+8, +9    -> k cols 2tig+8, 2tig+9
                            const uint32_t bx = (bb >= NBK / 2) ? b1[0] : b0[0];
                            const uint32_t by = (bb >= NBK / 2) ? b1[1] : b0[1];
#pragma unroll
                            for (int i = 0; i < H::N; i += 2)
                                mma16816(acc[bb * MPB + i / 2], rlo[i], rlo[i + 1], rhi[i], rhi[i + 1], bx, by);
                        }
                    }
                }
                }
            }
            __syncwarp();                                      // the slot may be refilled
            slot = slot == (R::NS - 1) * R::STAGE_BYTES ? 0u : slot + R::STAGE_BYTES;
          }
          zsum += accz[0];
          zsum3 += accz3[0];
        }

        float *dst0 = sm.scores + split * sm.n_scores - t0;
        // ---- epilogue ----------------------------------------------------------------------------------
        if constexpr (KB == 3) {
            // the octet's column is n = g, held by the lane with tig == g/2
#pragma unroll
            for (int hf = 0; hf < H; ++hf) {
                const int tok0 = tile0 + 88 * hf + g * G::TPO;     // first token of this octet's word of the half
                if (tok0 < hi && tig == (g >> 1)) {            // words are whole or absent (hi is a group multiple)
                    const bool sel = g & 1;
                    const float corr = hf ? zsum3 : zsum;      // row g of the zero-term product = group g = this octet's word
                    float *dst = dst0 + tok0;
#pragma unroll
                    for (int m = 0; m < 6; ++m) {
                        const int i0 = 2 * m, i1 = 2 * m + 1;
                        const float *c = acc[6 * hf + m];
                        dst[i0] = fmaf(sel ? c[1] : c[0], (float)(1 << (24 - F::pos(i0))), corr);
                        if (i1 < G::TPO) dst[i1] = fmaf(sel ? c[3] : c[2], (float)(1 << (24 - F::pos(i1 % F::N))), corr);
                    }
                }
            }
        } else if constexpr (KB == 4) {
            // octet g of half h is in group h*gph + cp of the tile, cp = 16 g / Gk; its hi and lo sums are the column
            // pair cp, held by the lane with tig == cp; the group's zero term sits in the lanes of octet grp
            constexpr int NF = F::N;
            const int cp = (16 * g) >> LGK;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int grp = h * gph + cp;
                const float corr = __shfl_sync(0xffffffffu, zsum, 4 * grp);    // row grp of the zero-term product
                const int tok0 = tile0 + 128 * h + 16 * g;
                if (tok0 < hi && tig == cp) {                  // 16-token chunks are whole or absent (hi is a group multiple)
                    float *dst = dst0 + tok0;
#pragma unroll
                    for (int m = 0; m < 8; ++m) {
                        const int i0 = (2 * m) % NF, i1 = (2 * m + 1) % NF;
                        float s0 = fmaf(acc[h * 8 + m][0] + acc[h * 8 + m][1], (float)(1 << (24 - F::pos(i0))), corr);
                        float s1 = fmaf(acc[h * 8 + m][2] + acc[h * 8 + m][3], (float)(1 << (24 - F::pos(i1))), corr);
                        *reinterpret_cast<float2 *>(dst + 2 * m) = make_float2(s0, s1);
                    }
                }
            }
        } else {
            // octet g of block bb owns tokens bb*8FH + g*FH ..; in its half of the tile they are in group cp, whose hi and
            // lo sums are the column pair cp, held by the lane with tig == cp; the group's zero term sits in the lanes
            // of octet grp
#pragma unroll
            for (int bb = 0; bb < NBK; ++bb) {
                constexpr int kHalfBlocks = NBK / 2;
                const int h = bb / kHalfBlocks;
                const int cp = (((bb % kHalfBlocks) * 8 * FH) + g * FH) >> LGK;
                const int grp = h * gph + cp;
                const float corr = __shfl_sync(0xffffffffu, zsum, 4 * grp);    // row grp of the zero-term product
                const int tok0 = tile0 + bb * 8 * FH + g * FH;
                if (tok0 < hi && tig == cp) {                  // FH-token chunks are whole or absent (hi is a group multiple)
                    float *dst = dst0 + tok0;
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
// p . V over packed values for tokens [t0, hi), (hi - t0) % 32 == 0.  sm.scores holds p.  Warp w
// takes 32-token blocks w, w+4, ... through its own ring (codes + scale + zero rows per stage).  Per
// stage the warp first forms the B operands once for all its lanes (p*scale and p*midpoint for 16
// token pairs x 8 columns, half2 per pair) in a small tile, then every lane reads its two B registers
// per k-step with one 32-bit load each.  Returns this warp's 128 partial channel sums in its own
// ring region (float [128] at the region base).
// MODE 1 only issues the first stages (called before the softmax, whose latency then hides the ring fill);
// MODE 2 continues after such a call; MODE 0 does both.
template <int VB, int MODE, int NW, int NGV>
__device__ __forceinline__ void pv_packed_mma(const kvq_attn_args &a, const int32_t *vc, const __half *vs,
                                              const __half *vz, const MmaSmem &sm, int t0, int hi) {
    using G = MmaVGeom<VB, NW>;
    using F = VHalf<VB>;
    constexpr int NB = G::GPT;                                // 16-byte blocks per token row: 1 / 2 / 4
    constexpr int CPB = kHeadDim / NB;                        // channels per block: 128 / 64 / 32
    constexpr int MPB = F::N / 2;                             // MMAs (channel pairs per octet) per block: 8 / 4 / 2
    const int warp = uniform_warp(), lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    constexpr int ngv = NGV, Gv = kHeadDim / NGV;             // channel groups: 4 / 2 / 1
    const int n_blocks = (hi - t0 + G::TPS - 1) / G::TPS;      // <= 0: no packed values in this segment
    const int my_blocks = (n_blocks - warp + NW - 1) / NW;
    float *my_red = reinterpret_cast<float *>(sm.ring);
    if (my_blocks <= 0) {
        if (MODE != 1)
            for (int i = lane; i < kHeadDim; i += 32) my_red[i] = 0.f;
        return;
    }

    // ---- per-lane constants ----------------------------------------------------------------------
    const uint32_t ring_s = smem_u32(sm.ring);
    const uint32_t pb_s = ring_s + G::PB_OFF;
    // cp.async: granule x = lane + 32 i -> token row tl = x / GPT, granule gr = x % GPT (source is contiguous)
    const int cp_tl0 = lane / G::GPT, cp_gr = lane % G::GPT;
    // rows are XOR-swizzled by token so that the 8 rows x 16 bytes of every ldmatrix tile hit all 32 banks once
    auto swz = [](int tl) { return (VB == 4) ? ((tl >> 1) & 3) : (VB == 2) ? ((tl >> 2) & 1) : 0; };
    const int cp_grs = cp_gr ^ swz(cp_tl0);                                              // (tl + 8 k, 16 k keep the swizzle)
    const uint32_t cp_dst = ring_s + cp_tl0 * G::RBV + cp_grs * 16;                      // + slot*STAGE + i*(32/GPT)*RBV
    // fragment loads: one transposing ldmatrix hands lane (g, tig) the half-word g of a 16-byte block for the
    // token pair (2 tig, 2 tig + 1) in one register, i.e. an A-fragment register pair along k without a byte permute.
    // Tile j of an x4 load (lanes 8j .. 8j+7 give its row addresses): tokens 8 (j & 1) .. +7 of the k-step, block
    // b0 + (j >> 1); the x2 load of 1-bit values has tiles j = 0, 1 only.
    const int ldm_tl = 8 * ((lane >> 3) & 1) + (lane & 7);                               // + 16 h2
    const int ldm_b = (lane >> 4) & (NB - 1);                                            // + b0 (4-bit: 0 or 2)
    const uint32_t ldm_s0 = ring_s + ldm_tl * G::RBV + ((ldm_b ^ swz(ldm_tl)) * 16);
    const uint32_t ldm_s1 = ring_s + ldm_tl * G::RBV + (((ldm_b + 2) & (NB - 1)) ^ swz(ldm_tl)) * 16;   // 4-bit: blocks 2, 3
    // operand tile: pair pi = 8 h2 + 4 b + tig holds tokens (16 h2 + 8 b + 2 tig, +1); reader column g
    const uint32_t pb_rd = pb_s + (tig * 8 + g) * 4;                                     // + (8 h2 + 4 b) * 32
    // operand build: lane -> pair pi = lane & 15, column half ch = lane >> 4 (groups 2ch, 2ch+1)
    const int pi = lane & 15, ch = lane >> 4;
    const int bt0 = 16 * (pi >> 3) + 8 * ((pi >> 2) & 1) + 2 * (pi & 3);                 // the pair's first token in the stage
    // (columns beyond the last channel group repeat others: C columns nobody reads)
    const uint32_t sz_rd = ring_s + G::SZ_OFF + bt0 * (ngv * 2) + (ngv == 4 ? 4 * ch : 0);         // this half's groups of token bt0; zeros + 256
    const uint32_t pb_wr = pb_s + (pi * 8 + 4 * ch) * 4;

    const int block_stride = NW * G::TPS;
    const char *vc_b = reinterpret_cast<const char *>(vc);                               // 32-bit byte offsets from the head's first row
    uint32_t src_codes = (uint32_t)(t0 + warp * G::TPS) * G::RBV + lane * 16;
    const int ngran = 4 * ngv;                                                           // 16-byte granules per array per stage
    const int sz_arr = lane >= ngran ? 1 : 0;                                            // 0: scale rows, 1: zero rows
    const int sz_off = (lane - sz_arr * ngran) * 16;
    const bool sz_on = lane < 2 * ngran;
    const char *sz_b = reinterpret_cast<const char *>(sz_arr ? vz : vs);
    uint32_t src_sz = (uint32_t)(t0 + warp * G::TPS) * (ngv * 2) + sz_off;
    const uint32_t sz_dst = ring_s + G::SZ_OFF + sz_arr * (G::TPS * 4 * 2) + sz_off;
    const uint32_t codes_step = block_stride * G::RBV, sz_step = block_stride * ngv * 2;

    int to_issue = my_blocks;                                                            // blocks not yet issued
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

    float acc[8][4], accz[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int m = 0; m < 8; ++m) acc[m][0] = acc[m][1] = acc[m][2] = acc[m][3] = 0.f;
    const uint32_t ones = 0x3c003c00u;
    // The MMA accumulators hold sums of non-negative terms (codes and p are >= 0) whose centred difference is
    // the result, and the tensor core adds into its fp32 accumulator with truncation: measured on a chain of
    // 128 MMAs the sum comes out 1.7e-6 low (1e-7 after 32, exact to 2e-8 when restarted every 16), which the
    // cancellation multiplies by a few hundred at 131k diffuse tokens.  Chains are therefore kept short: every
    // kFlush stages the columns this lane owns are added to fp32 sums (round to nearest) and restart from zero.
    constexpr int kFlush = 16;
    float sum[8][2], sumz[2] = {0.f, 0.f};
#pragma unroll
    for (int m = 0; m < 8; ++m) sum[m][0] = sum[m][1] = 0.f;
    auto flush = [&]() {
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            sum[m][0] += acc[m][0];
            sum[m][1] += acc[m][2];
            acc[m][0] = acc[m][1] = acc[m][2] = acc[m][3] = 0.f;
        }
        sumz[0] += accz[0];
        sumz[1] += accz[1];
        accz[0] = accz[1] = accz[2] = accz[3] = 0.f;
    };

    if (MODE != 2) {
#pragma unroll
        for (int q = 0; q < G::P; ++q) { issue_stage(q * G::STAGE_BYTES); cp_async_commit(); }
        if (MODE == 1) return;
    } else {                                                   // those stages are already in flight
        to_issue -= G::P;
        src_codes += G::P * codes_step;
        src_sz += G::P * sz_step;
    }

    uint32_t st = 0, issue_st = G::P * G::STAGE_BYTES;         // byte offsets of the slot being read / filled
    const float *pp = sm.scores + warp * G::TPS;               // p of this warp's current block
    for (int q = 0; q < my_blocks; ++q) {
        issue_stage(issue_st);
        cp_async_commit();
        cp_async_wait<G::P>();
        __syncwarp();
        // ---- B operands for the stage: 16 token pairs x 8 columns -----------------------------------
        {
            // p is scaled by 2^8 before the fp16 rounding so that the many small probabilities of a long, diffuse
            // context stay in the normal fp16 range (p <= 1, so this saturates only if a scale exceeds 255)
            const unsigned long long p01 = mul_f32x2(*reinterpret_cast<const unsigned long long *>(pp + bt0), f32x2(256.f, 256.f)), mid = f32x2(G::MID, G::MID);
            uint32_t sx, sy, zx, zy;                           // the two groups of tokens bt0 and bt0 + 1
            if constexpr (NGV == 4) {
                sx = lds32(sz_rd + st); sy = lds32(sz_rd + st + 8); zx = lds32(sz_rd + st + 256); zy = lds32(sz_rd + st + 264);
            } else if constexpr (NGV == 2) {
                asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];\n" : "=r"(sx), "=r"(sy) : "r"(sz_rd + st));
                asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];\n" : "=r"(zx), "=r"(zy) : "r"(sz_rd + st + 256));
            } else {                                           // one group, the two tokens in a word
                const uint32_t x = lds32(sz_rd + st), z = lds32(sz_rd + st + 256);
                sx = prmt(x, x, 0x1010); sy = prmt(x, x, 0x3232); zx = prmt(z, z, 0x1010); zy = prmt(z, z, 0x3232);
            }
            // columns 4ch .. 4ch+3 = (p*scale_g0, p*mid_g0, p*scale_g1, p*mid_g1), each a half2 over the token pair;
            // mid = zero + MID*scale is the midpoint of the group: codes are used as (code - MID)
            const unsigned long long s0 = f32x2(__low2float(as_h2(sx)), __low2float(as_h2(sy))), s1 = f32x2(__high2float(as_h2(sx)), __high2float(as_h2(sy)));
            const unsigned long long m0 = fma_f32x2(mid, s0, f32x2(__low2float(as_h2(zx)), __low2float(as_h2(zy))));
            const unsigned long long m1 = fma_f32x2(mid, s1, f32x2(__high2float(as_h2(zx)), __high2float(as_h2(zy))));
            auto pack = [](unsigned long long v) { const float2 f = f32x2_split(v); return pack_h2_sat(f.x, f.y); };
            const uint32_t c0 = pack(mul_f32x2(p01, s0)), c1 = pack(mul_f32x2(p01, m0)), c2 = pack(mul_f32x2(p01, s1)), c3 = pack(mul_f32x2(p01, m1));
            asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(pb_wr), "r"(c0), "r"(c1), "r"(c2), "r"(c3));
        }
        __syncwarp();
#pragma unroll
        for (int h2 = 0; h2 < 2; ++h2) {
            const uint32_t b0 = lds32(pb_rd + (8 * h2) * 32), b1 = lds32(pb_rd + (8 * h2 + 4) * 32);
            // x[b][0] / x[b][1]: block b, tokens (2 tig, 2 tig + 1) / (2 tig + 8, 2 tig + 9) of the k-step
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
            mma16816(accz, ones, ones, ones, ones, b0, b1);
#pragma unroll
            for (int bb = 0; bb < NB; ++bb) {
                uint32_t rlo[F::N], rhi[F::N];
                F::unpack(x[bb][0], rlo);
                F::unpack(x[bb][1], rhi);
#pragma unroll
                for (int i = 0; i < F::N; i += 2)              // rows g / g+8: channels bb*CPB + g*F::N + i / + i + 1
                    mma16816(acc[bb * MPB + i / 2], rlo[i], rlo[i + 1], rhi[i], rhi[i + 1], b0, b1);
            }
        }
        __syncwarp();
        st = (st + G::STAGE_BYTES == G::NS * G::STAGE_BYTES) ? 0u : st + G::STAGE_BYTES;
        issue_st = (issue_st + G::STAGE_BYTES == G::NS * G::STAGE_BYTES) ? 0u : issue_st + G::STAGE_BYTES;
        pp += block_stride;
        if ((q % kFlush) == kFlush - 1) flush();
    }
    flush();
    cp_async_wait<0>();
    __syncwarp();
    // epilogue: accumulator m = bb * MPB + ip holds channels c = bb*CPB + g*F::N + 2 ip (+1) in rows g (g+8); the column
    // of its group grp = c / Gv (sum p*scale) and the group's correction (sum p*mid, sum p*scale) sit in the lane with
    // tig == grp
    const float corr = (sumz[1] - G::MID * sumz[0]) * (1.f / 256.f);              // undo the 2^8 carried by the B operands
#pragma unroll
    for (int bb = 0; bb < NB; ++bb) {
        const int c0 = bb * CPB + g * F::N;
        if (tig == c0 / Gv) {                                                       // F::N <= 16 <= Gv: one group per octet block
#pragma unroll
            for (int ip = 0; ip < MPB; ++ip) {
                my_red[c0 + 2 * ip] = fmaf(sum[bb * MPB + ip][0], (float)(1 << (16 - F::pos(2 * ip))), corr);
                my_red[c0 + 2 * ip + 1] = fmaf(sum[bb * MPB + ip][1], (float)(1 << (16 - F::pos(2 * ip + 1))), corr);
            }
        }
    }
}

// The loops for the call's number of channel groups (see the keys: 4096 tokens, 64 x 32 heads, 4 bits 257.8 -> 250.4 us, 2 bits
// 213.3 -> 208.5 with both group sizes known).
template <int VB, int MODE, int NW>
__device__ __forceinline__ void pv_mma(const kvq_attn_args &a, const int32_t *vc, const __half *vs, const __half *vz, const MmaSmem &sm, int t0, int hi) {
    if (a.v_group == 32) pv_packed_mma<VB, MODE, NW, 4>(a, vc, vs, vz, sm, t0, hi);
    else if (a.v_group == 64) pv_packed_mma<VB, MODE, NW, 2>(a, vc, vs, vz, sm, t0, hi);
    else pv_packed_mma<VB, MODE, NW, 1>(a, vc, vs, vz, sm, t0, hi);
}

// ---------------------------------------------------------------------------------------------
// q . K^T over the fp16 tail for tokens [lo, t1): 16-token tiles on the tensor core, straight from
// global memory (row g and g+8 of a tile per lane-octet, 16-byte loads of 8 channels; the k axis is
// permuted identically in the q fragments).  Every B column carries q, so each lane sees its rows' sums.
template <int NW>
__device__ __forceinline__ void qk_tail_mma(const kvq_attn_args &a, const __half *kf, int b, int hk, const MmaSmem &sm,
                                            int t0, int lo, int t1) {
    const int warp = uniform_warp(), lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    uint4 qf[4];
#pragma unroll
    for (int S = 0; S < 4; ++S) qf[S] = *reinterpret_cast<const uint4 *>(sm.q + 32 * S + 8 * tig);
    const int n_tiles = (t1 - lo + 15) / 16;
    for (int tile = warp; tile < n_tiles; tile += NW) {
        const int ta = lo + 16 * tile + g, tb = ta + 8;
        const __half *pa = k_tail_row(a, kf, b, hk, min(ta, t1 - 1)) + 8 * tig;
        const __half *pb = k_tail_row(a, kf, b, hk, min(tb, t1 - 1)) + 8 * tig;
        uint4 ra[4], rb[4];
#pragma unroll
        for (int S = 0; S < 4; ++S) {
            ra[S] = __ldcg(reinterpret_cast<const uint4 *>(pa + 32 * S));
            rb[S] = __ldcg(reinterpret_cast<const uint4 *>(pb + 32 * S));
        }
        float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int S = 0; S < 4; ++S) {
            mma16816(c, ra[S].x, rb[S].x, ra[S].y, rb[S].y, qf[S].x, qf[S].y);
            mma16816(c, ra[S].z, rb[S].z, ra[S].w, rb[S].w, qf[S].z, qf[S].w);
        }
        if (tig == 0) {
            for (int p = 0; p < (1 << sm.ks_log2); ++p) {      // the whole score in the first partial, zero in the others
                float *dst = sm.scores + p * sm.n_scores - t0;
                if (ta < t1) dst[ta] = p ? 0.f : c[0];
                if (tb < t1) dst[tb] = p ? 0.f : c[2];
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// One segment: tokens [t0, t1) of query head (b, h); segment `seg` of the `cnt` the head is cut into.
template <int KB, int VB, int NW>
__device__ __forceinline__ void attn_segment(const kvq_attn_args &a, const kvq_attn_args &ac, unsigned int before, __half q_mine, const AttnPlan &plan, int s, int b, int h, int hk, int t0, int t1,
                                             int seg, int cnt, float *__restrict__ parts, unsigned int *__restrict__ counters) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
    const int n_scores = plan.n_scores, ks_log2 = plan.ks_log2, n_whole = plan.n_whole;
    MmaSmem sm;
    sm.n_scores = n_scores;
    sm.ks_log2 = ks_log2;
    sm.scores = reinterpret_cast<float *>(smem_raw);
    unsigned char *after_scores = smem_raw + ((size_t)n_scores << ks_log2) * 4;
    sm.ring = after_scores + warp * warp_region_bytes<KB, VB, NW>();
    sm.q = reinterpret_cast<__half *>(after_scores + NW * warp_region_bytes<KB, VB, NW>());
    sm.misc = reinterpret_cast<float *>(sm.q + kHeadDim);

    const int v_hi = min(t1, a.Tvq), v_lo = max(t0, a.Tvq);
    const __half *vf = static_cast<const __half *>(a.vfull) + (int64_t)b * a.vf_sB + (int64_t)hk * a.vf_sH;
    const __half *kf = static_cast<const __half *>(a.kfull) + (int64_t)b * a.kf_sB + (int64_t)hk * a.kf_sH;
    prefetch_tails(a, kf, vf, b, hk, t0, t1, tid, (32 * NW));
    fused_cache_update<KB, VB, 32 * NW>(a, b, hk, t0, t1, tid);        // the step's own cache update, when the caller fused it in
    if (tid < kHeadDim) sm.q[tid] = q_mine;

    if (ac.state) dev_state_publish(ac, a, before);

    // ---- 1. scores ------------------------------------------------------------------------------
    {
        const int32_t *kc = a.kcode + (int64_t)b * a.kc_sB + (int64_t)hk * a.kc_sH;
        const __half *ks = static_cast<const __half *>(a.kscale) + (int64_t)b * a.ks_sB + (int64_t)hk * a.ks_sH;
        const __half *kz = static_cast<const __half *>(a.kmn) + (int64_t)b * a.ks_sB + (int64_t)hk * a.ks_sH;
        const int k_hi = min(t1, a.Tkq), k_tail = max(t0, a.Tkq);
        // the loops for the call's group size: looked up, it cost a compare, a branch or a select per group and k-step
        if constexpr (KB == 3) {
            if (wide_key_tiles(k_hi - t0, NW, ks_log2)) qk_packed_mma<3, NW, 5, 2>(a, kc, ks, kz, sm, t0, k_hi, kf, k_tail, t1, b, hk);
            else qk_packed_mma<3, NW, 5, 1>(a, kc, ks, kz, sm, t0, k_hi, kf, k_tail, t1, b, hk);
        } else {
            if (a.k_group == 32) qk_packed_mma<KB, NW, 5, 1>(a, kc, ks, kz, sm, t0, k_hi, kf, k_tail, t1, b, hk);
            else if (a.k_group == 64) qk_packed_mma<KB, NW, 6, 1>(a, kc, ks, kz, sm, t0, k_hi, kf, k_tail, t1, b, hk);
            else qk_packed_mma<KB, NW, 7, 1>(a, kc, ks, kz, sm, t0, k_hi, kf, k_tail, t1, b, hk);
        }
    }
    const int32_t *vc = a.vcode + (int64_t)b * a.vc_sB + (int64_t)hk * a.vc_sH;
    const __half *vs = static_cast<const __half *>(a.vscale) + (int64_t)b * a.vs_sB + (int64_t)hk * a.vs_sH;
    const __half *vz = static_cast<const __half *>(a.vmn) + (int64_t)b * a.vs_sB + (int64_t)hk * a.vs_sH;
    pv_mma<VB, 1, NW>(a, vc, vs, vz, sm, t0, v_hi);         // start filling this warp's value ring now
    __syncthreads();

    // ---- 2. softmax numerators ------------------------------------------------------------------
    // upstream rounds the raw score to fp16 before scaling it (round_scores)
    const int n = t1 - t0, n4 = (n + 3) >> 2;
    float m = kMaskFloor;                                      // a fully masked range then weighs uniformly, as upstream's does
    float4 *sc4 = reinterpret_cast<float4 *>(sm.scores);
    // a thread's scores stay in registers between the maximum and the exponentials
    constexpr int QN = ((NW == 8 ? kWideScores3 : kNarrowMax) + 128 * NW - 1) / (128 * NW);
    float4 sv[QN];
#pragma unroll
    for (int j = 0; j < QN; ++j) {
        if (32 * NW * j >= n4) break;
        const int i = tid + 32 * NW * j;
        float4 v = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
        if (i < n4) {
            v = score_quad(a, sc4 + i, n_scores >> 2, ks_log2);
            if (a.mask) mask_quad(a, b, h, t0 + 4 * i, v);
            if (4 * i + 3 >= n) pad_quad(v, n - 4 * i);
        }
        sv[j] = v;
        m = fmaxf(fmaxf(m, fmaxf(v.x, v.y)), fmaxf(v.z, v.w));
    }
    m = warp_max(m);
    if (lane == 0) sm.misc[warp] = m;
    __syncthreads();
    m = sm.misc[lane & (NW - 1)];
    m = warp_max(m);
    float l = 0.f;
#pragma unroll
    for (int j = 0; j < QN; ++j) {
        if (32 * NW * j >= n4) break;
        const int i = tid + 32 * NW * j;
        float4 v = sv[j];
        v.x = __expf(v.x - m);
        v.y = __expf(v.y - m);
        v.z = __expf(v.z - m);
        v.w = __expf(v.w - m);
        if (i < n4) sc4[i] = v;
        l += (v.x + v.y) + (v.z + v.w);
    }
    l = warp_sum(l);
    if (lane == 0) sm.misc[8 + warp] = l;
    __syncthreads();

    // ---- 3. p.V -----------------------------------------------------------------------------------
    pv_mma<VB, 2, NW>(a, vc, vs, vz, sm, t0, v_hi);
    __syncwarp();
    if (v_lo < t1) pv_tail<1>(a, vf, b, hk, sm.scores, 0, t0, v_lo, t1, reinterpret_cast<float *>(sm.ring), warp, NW, lane);
    __syncthreads();

    launch_next();                                             // what is left is short: the next launch may come

    // ---- 4. finish / merge --------------------------------------------------------------------------
    const bool own = NW == 4 || tid < kHeadDim;                         // thread tid owns channel tid
    float o = 0.f, l_all = 0.f;
    if (own) {
#pragma unroll
        for (int w = 0; w < NW; ++w) o += reinterpret_cast<const float *>(after_scores + w * warp_region_bytes<KB, VB, NW>())[tid];
    }
#pragma unroll
    for (int w = 0; w < NW; ++w) l_all += sm.misc[8 + w];
    __half *out = static_cast<__half *>(a.out) + (int64_t)b * a.o_sB + (int64_t)h * a.o_sH;
    if (cnt == 1) {
        const __half r[1] = {__float2half_rn(o / l_all)};
        if (own) out[tid] = r[0];
        peer_publish(ac, b, h, own ? 1 : 0, r, tid & (kHeadDim - 1), tid, 1);
        return;
    }
    constexpr int kPart = kPartStride;
    float *part = parts + ((int64_t)(s - n_whole) * cnt + seg) * kPart;          // partials of the cut heads only
    if (own) part[tid] = o;
    if (tid == 0) { part[kHeadDim] = m; part[kHeadDim + 1] = l_all; }
    __syncthreads();
    if (tid == 0) {
        // the CTA barrier and the count's release publish every thread's partial; its acquire orders the merging CTA's reads
        // (ld.cg, from L2) behind the other CTAs' counts
        sm.misc[16] = count_in(&counters[s]) == (unsigned)(cnt - 1) ? 1.f : 0.f;
    }
    __syncthreads();
    if (sm.misc[16] == 0.f) return;
    const float *base = parts + (int64_t)(s - n_whole) * cnt * kPart;
    float M = kMaskFloor;
    for (int i = lane; i < cnt; i += 32) M = fmaxf(M, __ldcg(base + i * kPart + kHeadDim));
    M = warp_max(M);
    float L = 0.f, acc = 0.f;
    const int ch = tid & (kHeadDim - 1);
    constexpr int U = 8;                                     // loads in flight; behind the last segment it is read again, as zeros
    for (int i0 = 0; i0 < cnt; i0 += U) {
        float2 ml[U];
        float p[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const float *pi = base + min(i0 + u, cnt - 1) * kPart;
            ml[u] = __ldcg(reinterpret_cast<const float2 *>(pi + kHeadDim));
            p[u] = __ldcg(pi + ch);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool in = i0 + u < cnt;
            const float w = __expf(ml[u].x - M);
            L = fmaf(in ? ml[u].y : 0.f, w, L);
            acc = fmaf(in ? p[u] : 0.f, w, acc);
        }
    }
    const __half r[1] = {__float2half_rn(acc / L)};
    if (own) out[tid] = r[0];
    if (tid == 0) counters[s] = 0u;                          // the head is done: its counter is ready for the next launch
    peer_publish(ac, b, h, own ? 1 : 0, r, ch, tid, 1);
}

// CTA = one segment (see attn_plan.cuh): a whole head, or one of the k pieces of a head that is cut.
// DEV: lengths and ring starts come from the device-resident state (attn_update.cuh); the plan was laid out for an
// upper bound of the length, so segments beyond the real length are empty and a head counts fewer of them.
template <int KB, int VB, bool DEV, int NW>
__global__ void __launch_bounds__(32 * NW, 16 / NW) decode_attn_mma_kernel(const __grid_constant__ kvq_attn_args a,
                                                                     const __grid_constant__ AttnPlan plan,
                                                                     float *__restrict__ parts,
                                                                     unsigned int *__restrict__ counters) {
    grid_wait();
    DevState state;
    if constexpr (DEV) state = dev_state_load(a);
    // grouped queries: each query head is its own segment and reads kv head hk; the heads of one kv head are
    // neighbouring units of work, so the cache is fetched from HBM once and re-read from L2
    int head, seg, b, hk, within, t0, t1, cnt;
    plan_head(plan, blockIdx.x, head, seg);
    plan_place(plan, head, b, hk, within);
    const int h = hk * plan.rep + within;
    // this thread's channel of q: the key phase waits for it, and nothing of it depends on the cache's state
    const __half q_mine = static_cast<const __half *>(a.q)[(int64_t)b * a.q_sB + (int64_t)h * a.q_sH + (threadIdx.x & (kHeadDim - 1))];
    if constexpr (DEV) {
        kvq_attn_args d = a;
        const unsigned int before = dev_state_step(a, state, d);
        plan_tokens(plan, d.T, blockIdx.x, seg, t0, t1, cnt);
        if (cnt > 1) cnt = min(cnt, (d.T + plan.seg_units * plan.unit - 1) / (plan.seg_units * plan.unit));
        if (t0 < d.T) attn_segment<KB, VB, NW>(d, a, before, q_mine, plan, head, b, h, hk, t0, t1, seg, cnt, parts, counters);
        else dev_state_publish(a, d, before);
    } else {
        plan_tokens(plan, a.T, blockIdx.x, seg, t0, t1, cnt);
        attn_segment<KB, VB, NW>(a, a, 0u, q_mine, plan, head, b, h, hk, t0, t1, seg, cnt, parts, counters);
    }
}

// ---------------------------------------------------------------------------------------------
// The tensor-core path needs a whole number of query heads per kv head, supported group sizes, 16-byte aligned
// and row-contiguous packed tensors (cp.async granules), and a packed-value length that is a multiple of 32.
int gqa_heads_per_cta(const kvq_attn_args &a);               // decode_attn_gqa.cu

bool mma_path_eligible(const kvq_attn_args &a) {
    if (a.nh_kv <= 0 || a.nh % a.nh_kv != 0 || a.D != kHeadDim) return false;
    if (a.k_bits == 3) {
        if (a.k_group != 11) return false;
    } else if (a.k_group != 32 && a.k_group != 64 && a.k_group != 128) {
        return false;
    }
    if (a.v_bits == 3) {                                       // only the grouped kernel has 3-bit values
        if (a.v_group != 11 || gqa_heads_per_cta(a) == 0) return false;
    } else if (a.v_group != 32 && a.v_group != 64 && a.v_group != 128) {
        return false;
    }
    if (a.Tvq % 32 != 0) return false;
    auto al16 = [](const void *p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
    if (a.T > a.Tkq && (!al16(a.kfull) || a.kf_sB % 8 || a.kf_sH % 8 || a.kf_sT % 8)) return false;
    if (a.T > a.Tvq && (!al16(a.vfull) || a.vf_sB % 8 || a.vf_sH % 8 || a.vf_sT % 8)) return false;
    if (a.Tkq > 0) {
        if (!al16(a.kcode) || a.kc_sB % 4 || a.kc_sH % 4 || a.kc_sD % 4) return false;
        if (!al16(a.kscale) || !al16(a.kmn) || a.ks_sB % 8 || a.ks_sH % 8 || a.ks_sD % 8) return false;
        // a head's keys are addressed by 32-bit byte offsets, unsigned (128 rows of 4-byte words, of 2-byte scales)
        if (a.kc_sD < 0 || a.kc_sD >= (1 << 23) || a.ks_sD < 0 || a.ks_sD >= (1 << 24)) return false;
    }
    if (a.Tvq > 0) {
        const int fv = fields_per_word(a.v_bits);              // rows back to back (3 bits: 12 words and groups a token)
        if (!al16(a.vcode) || a.vc_sB % 4 || a.vc_sH % 4 || a.vc_sT != (kHeadDim + fv - 1) / fv) return false;
        if (!al16(a.vscale) || !al16(a.vmn) || a.vs_sB % 8 || a.vs_sH % 8 || a.vs_sT != (kHeadDim + a.v_group - 1) / a.v_group) return false;
    }
    return true;
}


template <int KB, int VB, int NW> constexpr int mma_smem_bytes(int scores) {
    return scores * 4 + NW * warp_region_bytes<KB, VB, NW>() + kHeadDim * 2 + 32 * 4;
}

template <int KB, int VB, int NW>
static int launch_mma(const kvq_attn_args &a, AttnPlan plan, float *parts, unsigned int *counters,
                      cudaStream_t st) {
    plan_set_place(plan, a.nh, a.nh_kv, a.nh / a.nh_kv);
    constexpr int kSmSmem = 227 * 1024;                      // of an SM, 1 KB of it taken by every CTA
    static_assert(NW == 4 || mma_smem_bytes<KB, VB, 8>(KB == 3 ? kWideScores3 : kWideScores) <= kMmaSmemMax, "two eight-warp CTAs");
    static_assert(NW == 8 || 3 * (mma_smem_bytes<KB, VB, 4>(KB == 3 ? kNarrowMax3 : kNarrowMax) + 1024) <= kSmSmem, "three four-warp CTAs");
    static_assert(NW == 8 || 4 * (mma_smem_bytes<KB, VB, 4>(kNarrowScores) + 1024) <= kSmSmem, "four four-warp CTAs");
    const size_t smem = mma_smem_bytes<KB, VB, NW>(plan.n_scores << plan.ks_log2);
    static bool attr_set[64] = {};                           // per device: the opt-in is sticky for the process
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return record_cuda_error(e);
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        e = cudaFuncSetAttribute(decode_attn_mma_kernel<KB, VB, false, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMmaSmemMax);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(decode_attn_mma_kernel<KB, VB, true, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMmaSmemMax);
        if (e != cudaSuccess) return record_cuda_error(e);
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    const unsigned grid = (unsigned)(plan.n_whole + plan.n_cut * plan.k);
    // device-driven steps are replayed from graphs, whose launches follow each other closely anyway: early CTAs of the next layer then
    // only crowd the SMs that are done first (8 x 32 heads of 4096 tokens, five layers: 236.7 us so, 238.8 launched early)
    if (a.state) {
        decode_attn_mma_kernel<KB, VB, true, NW><<<grid, 32 * NW, smem, st>>>(a, plan, parts, counters);
        return check_launch();
    }
    return launch_early(plan_early(plan), decode_attn_mma_kernel<KB, VB, false, NW>, grid, 32 * NW, smem, st, a, plan, parts, counters);
}

int launch_decode_attn_mma(const kvq_attn_args &a, const AttnPlan &plan, float *parts, unsigned int *counters,
                           cudaStream_t st) {
#define KVQ_MMA_CASE(KB, VB) \
    if (a.k_bits == KB && a.v_bits == VB)                                                            \
        return plan.warps == 4 ? launch_mma<KB, VB, 4>(a, plan, parts, counters, st) : launch_mma<KB, VB, 8>(a, plan, parts, counters, st);
    KVQ_MMA_CASE(4, 4) KVQ_MMA_CASE(4, 2) KVQ_MMA_CASE(4, 1)
    KVQ_MMA_CASE(3, 4) KVQ_MMA_CASE(3, 2) KVQ_MMA_CASE(3, 1)
    KVQ_MMA_CASE(2, 4) KVQ_MMA_CASE(2, 2) KVQ_MMA_CASE(2, 1)
    KVQ_MMA_CASE(1, 4) KVQ_MMA_CASE(1, 2) KVQ_MMA_CASE(1, 1)
#undef KVQ_MMA_CASE
    return KVQ_ERR_UNSUPPORTED;
}

// Plan of the tensor-core kernel for B * nh query heads (one head per segment).
AttnPlan plan_attn_mma(int T, int k_bits, long long heads) {
    return k_bits == 3 ? make_attn_plan_mma(T, 352, MmaKGeom<3, 1>::WT, kWideScores3, heads, kNarrowMax3, kNarrowScores, 1760)
                       : make_attn_plan_mma(T, 256, KGeom<4>::WT, kWideScores, heads, kNarrowMax, kNarrowScores, 3072);
}

}  // namespace kvq
