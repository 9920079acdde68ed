// Stand-alone dequantising mat-vec (M = 1) over the upstream cache layout, read in place.
//
//   out[n] = fp16( sum_k in[k] * (scale[k, n/G] * code[k, n] + zero[k, n/G]) ),  fp32 accumulation
//
// Two kernels:
//   gemv_mma_kernel   1, 2 and 4 bits, groups of 32 / 64 / 128: the codes go to mma.sync as fp16 subnormals, as in the
//                     attention kernels; rows (k) are the contraction, so q . K^T (K = head_dim rows, thousands of columns)
//                     and p . V (thousands of rows, 128 columns) are the same loop, split differently over the warps.
//   gemv_kernel       everything else (3-bit words, other groups): one thread per word column.
#include <cooperative_groups.h>

#include "attn_mma_common.cuh"

namespace kvq {

// ---------------------------------------------------------------------------------------------
// The zero term is hoisted: sum_k in[k]*zero[k,g] is accumulated once per packed word instead of
// once per field, and in[k]*scale[k,g] is formed once per word.  A CTA is WX word columns x KY
// k-lanes; lanes along the word axis read consecutive words (coalesced) for both uses of the
// routine: q.K^T (K = head_dim rows, thousands of word columns) and p.V (thousands of rows,
// head_dim/fpi word columns).
template <int BITS>
__global__ void __launch_bounds__(256) gemv_kernel(kvq_gemv_args a, int wx_log2, int nblk) {
    constexpr int FPI = fields_per_word(BITS);
    __shared__ float red[256];
    const int WX = 1 << wx_log2, KY = 256 >> wx_log2;
    const int wx = threadIdx.x & (WX - 1), ky = threadIdx.x >> wx_log2;
    const int64_t w = (int64_t)(blockIdx.x % nblk) * WX + wx;
    const int64_t s = blockIdx.x / nblk, b = s / a.nh, h = s % a.nh, hk = h / (a.nh / a.nh_kv);
    const int64_t n_pack = (a.n_groups * a.group) / FPI;
    const bool live = w < n_pack;
    const __half *in = static_cast<const __half *>(a.fA) + b * a.a_sB + h * a.a_sH;
    const int32_t *qb = a.qB + b * a.q_sB + hk * a.q_sH + w;
    const int64_t grp = (w * FPI) / a.group;
    const __half *sp = static_cast<const __half *>(a.scale) + b * a.s_sB + hk * a.s_sH + grp;
    const __half *zp = static_cast<const __half *>(a.zero) + b * a.s_sB + hk * a.s_sH + grp;

    float acc[FPI];
#pragma unroll
    for (int i = 0; i < FPI; ++i) acc[i] = 0.f;
    float zacc = 0.f;
    if (live) {
        for (int64_t k = ky; k < a.K; k += KY) {
            const uint32_t word = (uint32_t)__ldg(qb + k * a.q_sK);
            const float x = __half2float(__ldg(in + k));
            const float xs = x * __half2float(__ldg(sp + k * a.s_sK));
            zacc = fmaf(x, __half2float(__ldg(zp + k * a.s_sK)), zacc);
#pragma unroll
            for (int i = 0; i < FPI; ++i) acc[i] = fmaf(xs, (float)field<BITS>(word, i), acc[i]);
        }
    }
    __half *out = static_cast<__half *>(a.out) + b * a.o_sB + h * a.o_sH;
#pragma unroll 1
    for (int i = 0; i < FPI; ++i) {
        red[ky * WX + wx] = acc[i] + zacc;
        __syncthreads();
        if (ky == 0 && live) {
            float v = 0.f;
            for (int j = 0; j < KY; ++j) v += red[j * WX + wx];
            out[w * FPI + i] = __float2half_rn(v);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------------------
// Tensor-core form.  A warp works tiles of 128 columns (16 * BITS bytes of a row) x 32 rows a stage:
//   A (16x16)  codes, rows = columns n of the result, k = 16 rows of the matrix (transposing ldmatrix, fields left in place);
//   B (16x8)   column 2j / 2j + 1 = hi / lo of in[k] * scale[k, group j], j < 4 groups: the product of two fp16 numbers needs
//              22 bits and is carried as an fp16 pair.  lo ends at 2^-24 whatever the product, so both factors are first
//              brought to the upper half of the fp16 range by powers of two: `in` by one per chunk of rows (only upwards, hence
//              exactly: its largest magnitude to 2^7 .. 2^8), the scales of a group by one per window of stages (the largest
//              of the first stage to 2^4 .. 2^5, the others below 2^8).  What the pair loses is then at most 2^-36 of the largest
//              input times the largest scale, 2^-24 of a product 2^12 times smaller; what is left is the fp32 accumulation.
//              Softmax weights of 0.9 on one row of next to nothing and 0.1 on 2047 others with scales of 0.03: 2e-4 from 64
//              bits (the fp16 result), 6e-4 (2 bits) and 4e-3 (4 bits) with `in` brought below 1 and the scales as they are.
//   Every other 16 rows use the complement of the codes with the operand's sign turned, c = MAX - (MAX - c): the tensor core cuts
//   products off downwards (codes are subnormal: 2^-20 of a product), which over thousands of rows of non-negative
//   probabilities adds up to 3e-6 of the magnitude summed; with opposite signs the two halves cancel.
//   zeros      one MMA per 16 rows with the [4 scales | 4 zeros] rows read transposed as A and `in` as B: row 4 + j of the
//              product is the zero term of group j (and row j the sum of in * scale that the complemented rows need).
//   Infinities and NaN come out as fp32 products and sums give them: a window that holds an infinity works without the complement,
//              whose two halves would meet as inf - inf.
// Bound by the instruction stream: 0.6 logic operations a code, and whatever surrounds them.  A stage of whole rows is copied by
// 32-bit offsets from the head's first word (64-bit row arithmetic per granule was a quarter of all instructions), the group size is
// known to the loops, heads and columns are numbered in 32 bits, and where the rows are few (q . K^T) a warp takes up to four
// column tiles one after the other, the copies running on from tile to tile.  16 sequences x 32 heads x 4096 tokens, group 32, us:
// q . K^T 2 bits 64 -> 50, 4 bits 68 -> 54, 1 bit (group 128) 60 -> 44; p . V 50 -> 46, 54 -> 52, 48 -> 43 (229 for the 2-bit
// pair with one thread per word column); warp instructions per 32 codes of q . K^T 4.1 -> 3.6, of p . V 2.8.
template <int BITS> struct GemvGeom {
    static constexpr int RB = 16 * BITS;                       // code bytes of a tile row
    static constexpr int RS = BITS == 1 ? RB : RB + 16;        // padded: conflict-free ldmatrix
    static constexpr int CODE_BYTES = 32 * RS;
    static constexpr int STAGE_BYTES = CODE_BYTES + 32 * 16;
    static constexpr int NS = BITS == 4 ? 3 : 4;
    static constexpr int WARP_BYTES = NS * STAGE_BYTES;
};
constexpr int kGemvWarps = 8, kGemvThreads = 32 * kGemvWarps;
constexpr int kGemvChunk = 2048;                               // rows whose `in` is held (and normalised) at a time
// A warp takes several column tiles where a tile is short (rows) and the CTAs still fill the GPU: with 128 rows a tile is four stages, and a
// warp that works only one spends as long on its first copies.
constexpr int kGemvTileRows = 512, kGemvTiles = 4, kGemvMinCtas = 2 * 296;
constexpr int kGemvFlush = 8;                                  // stages between flushes of the MMA accumulators (short chains): a window

__device__ __forceinline__ float pow2f(int e) { return __uint_as_float((uint32_t)(127 + e) << 23); }

struct GemvPlan {
    int wk_log2;         // warps that share a column tile (the other factor of 8: column tiles of a CTA)
    int col_ctas;        // CTAs per head along the columns
    int tpw;             // column tiles a warp takes one after the other
    int kc;              // CTAs of a cluster, each with rows_per_cta rows
    int rows_per_cta;
    int code_align;      // 16, 8 or 4: what every row of a tile is aligned to
    int sz_vec;          // scale / zero rows of a whole tile can be copied as one vector
    int fast;            // 16-byte granules and vectors, all rows of a head within 32-bit byte offsets
    int rep;             // query heads per kv head
    int out_vec;         // output rows are 8-byte aligned
    int early;           // launched early, and lets the next launch in early
};

template <int CG, int BITS>
__device__ __forceinline__ void gemv_copy_codes(uint32_t dst, const int32_t *src, int64_t q_sK, int rows, int words, int lane) {
    using G = GemvGeom<BITS>;
    constexpr int GPR = G::RB / CG;                            // granules per row
#pragma unroll
    for (int i = 0; i < GPR; ++i) {
        const int x = lane + 32 * i, row = x / GPR, col = x % GPR;
        if (row < rows && col * (CG / 4) < words) cp_async<CG>(dst + row * G::RS + col * CG, src + row * q_sK + col * (CG / 4));
    }
}

// GS_LOG2: log2 of the group size
template <int BITS, int GS_LOG2>
__global__ void __launch_bounds__(kGemvThreads, 2) gemv_mma_kernel(const __grid_constant__ kvq_gemv_args a,
                                                                   const __grid_constant__ GemvPlan plan) {
    using G = GemvGeom<BITS>;
    using F = VHalf<BITS>;
    constexpr int FPI = fields_per_word(BITS), FH = 16 / BITS, MPB = FH / 2, NBLK = BITS, ngw = 128 >> GS_LOG2, kSzBytes = ngw == 4 ? 8 : 4;
    extern __shared__ __align__(128) unsigned char smem[];
    float *red = reinterpret_cast<float *>(smem);                               // [kGemvWarps][128] tile sums
    __half *xs = reinterpret_cast<__half *>(red + kGemvWarps * 128);            // [kGemvChunk] normalised `in`
    float *misc = reinterpret_cast<float *>(xs + kGemvChunk);                   // [8]
    unsigned char *ring = reinterpret_cast<unsigned char *>(misc + 8) + 96;     // 128-byte aligned
    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31, g = lane >> 2, tig = lane & 3;
    const int WK = 1 << plan.wk_log2, wk = warp & (WK - 1), wc = warp >> plan.wk_log2, WC = kGemvWarps >> plan.wk_log2;
    // everything that numbers CTAs, heads and columns fits 32 bits (gemv_mma_plan); 64-bit divisions cost 100 instructions each
    const uint32_t rank = blockIdx.x % (uint32_t)plan.kc, job = blockIdx.x / (uint32_t)plan.kc;
    const uint32_t s = job / (uint32_t)plan.col_ctas, col_cta = job - s * (uint32_t)plan.col_ctas;
    const uint32_t b = s / (uint32_t)a.nh, h = s - b * (uint32_t)a.nh, hk = h / (uint32_t)plan.rep;
    const int N = (int)(a.n_groups << GS_LOG2), n_pack = N / FPI;
    const int col0 = (int)col_cta * plan.tpw * WC * 128;                        // the CTA's first column
    const int k_beg = (int)rank * plan.rows_per_cta, k_end = min((int)a.K, k_beg + plan.rows_per_cta);
    const __half *in = static_cast<const __half *>(a.fA) + b * a.a_sB + h * a.a_sH;
    const int32_t *qh = a.qB + b * a.q_sB + hk * a.q_sH;
    const __half *sh = static_cast<const __half *>(a.scale) + b * a.s_sB + hk * a.s_sH;
    const __half *zh = static_cast<const __half *>(a.zero) + b * a.s_sB + hk * a.s_sH;
    __half *out = static_cast<__half *>(a.out) + b * a.o_sB + h * a.o_sH;

    const uint32_t ring_s = smem_u32(ring) + warp * G::WARP_BYTES;
    const uint32_t sz_dst = ring_s + G::CODE_BYTES + lane * 16;
    const uint32_t szm_s = ring_s + G::CODE_BYTES + (lane & 15) * 16;
    const uint32_t ldk_s = ring_s + (lane & 15) * G::RS + (BITS == 1 ? 0 : (lane >> 4) * 16);
    const uint32_t x_s = smem_u32(xs) + (2 * tig) * 2;
    const int src = 4 * (g >> 1) + tig;                                         // lane holding group (column / 2)
    const uint32_t neg_mask = (g & 1) ? 0xffffffffu : 0u;

    // a stage of the fast path: granule x = lane + 32 i -> row x / GPR, granule x % GPR; bytes from the head's first word / scale
    constexpr int GPR = G::RB / 16;
    const uint32_t q_row = (uint32_t)a.q_sK * 4u, s_row = (uint32_t)a.s_sK * 2u;
    const uint32_t lane_q = (uint32_t)(lane / GPR) * q_row + (lane % GPR) * 16u, lane_s = (uint32_t)lane * s_row;
    const uint32_t lane_dst = ring_s + (lane / GPR) * G::RS + (lane % GPR) * 16;
    const char *qh_b = reinterpret_cast<const char *>(qh), *sh_b = reinterpret_cast<const char *>(sh), *zh_b = reinterpret_cast<const char *>(zh);

    grid_wait();
    if (plan.early) launch_next();
    float acc[8][4], sum[8][2], accz[2][4] = {}, zsum = 0.f;
    auto clear = [&]() {
#pragma unroll
        for (int m = 0; m < 8; ++m) sum[m][0] = sum[m][1] = 0.f;
        zsum = 0.f;
    };
    clear();
#pragma unroll
    for (int m = 0; m < 8; ++m) acc[m][0] = acc[m][1] = acc[m][2] = acc[m][3] = 0.f;

    // tile sums: octet g of block bb owns columns bb * 8 FH + g * FH .. + FH - 1, their group's pair of B columns is held by
    // the lane with tig == group, its zero term by row 4 + group
    auto tile_sums = [&]() {
#pragma unroll
        for (int bb = 0; bb < NBLK; ++bb) {
            const int c = bb * 8 * FH + g * FH, cp = c >> GS_LOG2;
            constexpr float kMax = (float)((1 << BITS) - 1);
            const float corr = fmaf(kMax, __shfl_sync(0xffffffffu, zsum, 4 * cp), __shfl_sync(0xffffffffu, zsum, 4 * (4 + cp)));
            if (tig == cp) {
#pragma unroll
                for (int ip = 0; ip < MPB; ++ip) {
                    red[warp * 128 + c + 2 * ip] = fmaf(sum[bb * MPB + ip][0], (float)(1 << (24 - F::pos(2 * ip))), corr);
                    red[warp * 128 + c + 2 * ip + 1] = fmaf(sum[bb * MPB + ip][1], (float)(1 << (24 - F::pos(2 * ip + 1))), corr);
                }
            }
        }
    };

    for (int c0 = k_beg; c0 < k_end; c0 += kGemvChunk) {
        const int rows = min(kGemvChunk, k_end - c0), n_st = (rows + 31) / 32, my_st = (n_st - wk + WK - 1) / WK;
        // Stages of this warp's tiles in one sequence: the ring runs on from one tile to the next.  (More than one tile only where
        // all rows are one chunk.)
        const int n0_first = col0 + wc * 128;
        int iss_n0 = n0_first, iss_st = wk, iss_left = my_st * plan.tpw;
        uint32_t iss_q = (uint32_t)(c0 + 32 * wk) * q_row + (uint32_t)(n0_first / FPI) * 4u, iss_s = (uint32_t)(c0 + 32 * wk) * s_row + (uint32_t)(n0_first >> GS_LOG2) * 2u;
        bool iss_whole = plan.fast && n0_first + 128 <= N;                      // a whole tile, and aligned
        auto issue_any = [&](uint32_t slot) {                                   // ragged, unaligned or far apart
            const int words = min(128 / FPI, n_pack - iss_n0 / FPI);            // <= 0: no such tile
            if (words > 0) {
                const int left = rows - 32 * iss_st;                            // rows of the stage that exist
                const int grp0 = iss_n0 >> GS_LOG2, groups = min(ngw, (int)a.n_groups - grp0);
                const int64_t r0 = c0 + 32 * iss_st;
                const int32_t *p = qh + iss_n0 / FPI + r0 * a.q_sK;
                if (plan.code_align == 16) gemv_copy_codes<16, BITS>(ring_s + slot, p, a.q_sK, left, words, lane);
                else if (plan.code_align == 8) gemv_copy_codes<8, BITS>(ring_s + slot, p, a.q_sK, left, words, lane);
                else gemv_copy_codes<4, BITS>(ring_s + slot, p, a.q_sK, left, words, lane);
                const __half *ps = sh + grp0 + (r0 + lane) * a.s_sK, *pz = zh + grp0 + (r0 + lane) * a.s_sK;
                const uint32_t d = sz_dst + slot;
                if (ngw > 1 && lane < left && plan.sz_vec && groups == ngw) {
                    cp_async<kSzBytes>(d, ps);
                    cp_async<kSzBytes>(d + 8, pz);
                } else {                                                        // odd group counts, one group a tile, missing rows: zeros
                    uint32_t v[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int jj = j & 1;
                        const __half *q = j < 2 ? ps : pz;
                        const bool ok0 = lane < left && 2 * jj < groups, ok1 = lane < left && 2 * jj + 1 < groups;
                        const uint32_t lo = ok0 ? __half_as_ushort(q[2 * jj]) : 0u, hi = ok1 ? __half_as_ushort(q[2 * jj + 1]) : 0u;
                        v[j] = lo | (hi << 16);
                    }
                    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(d), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]));
                }
            }
        };
        auto issue = [&](uint32_t slot) {
            if (iss_left > 0) {
                if (iss_whole && 32 * iss_st + 32 <= rows) {
#pragma unroll
                    for (int i = 0; i < GPR; ++i)
                        cp_async<16>(lane_dst + slot + i * (32 / GPR) * G::RS, qh_b + (iss_q + lane_q + i * (32 / GPR) * q_row));
                    const uint32_t d = sz_dst + slot, o = iss_s + lane_s;
                    if constexpr (ngw > 1) {
                        cp_async<kSzBytes>(d, sh_b + o);
                        cp_async<kSzBytes>(d + 8, zh_b + o);
                    } else {
                        const uint32_t v = __half_as_ushort(*reinterpret_cast<const __half *>(sh_b + o)), z = __half_as_ushort(*reinterpret_cast<const __half *>(zh_b + o));
                        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%2};\n" ::"r"(d), "r"(v), "r"(0u), "r"(z));
                    }
                } else {
                    issue_any(slot);
                }
            }
            cp_async_commit();
            --iss_left;
            iss_st += WK;
            iss_q += 32u * q_row << plan.wk_log2;
            iss_s += 32u * s_row << plan.wk_log2;
            if (iss_st >= n_st) {                                               // the next tile
                iss_n0 += WC * 128;
                iss_st = wk;
                iss_q = (uint32_t)(c0 + 32 * wk) * q_row + (uint32_t)(iss_n0 / FPI) * 4u;
                iss_s = (uint32_t)(c0 + 32 * wk) * s_row + (uint32_t)(iss_n0 >> GS_LOG2) * 2u;
                iss_whole = plan.fast && iss_n0 + 128 <= N;
            }
        };
        uint32_t iss_slot = 0, slot = 0;
#pragma unroll 1
        for (int q = 0; q < G::NS - 1; ++q) { issue(iss_slot); iss_slot += G::STAGE_BYTES; }

        // ---- in * 2^up_e: the largest magnitude to 2^7 .. 2^8, larger ones (and a chunk with an infinity) as they are ----
        if (c0 > k_beg) __syncthreads();                                        // the previous chunk has been read
        float mx = 0.f;
        constexpr int NX = kGemvChunk / kGemvThreads;
        __half xr[NX];                                                          // asked for in one go, read once
#pragma unroll
        for (int j = 0; j < NX; ++j) {
            const int i = tid + kGemvThreads * j;
            xr[j] = i < rows ? in[c0 + i] : __float2half_rn(0.f);
            mx = fmaxf(mx, fabsf(__half2float(xr[j])));
        }
        mx = warp_max(mx);
        if (lane == 0) misc[warp] = mx;
        __syncthreads();
        mx = warp_max(misc[lane & 7]);
        const bool in_finite = mx <= 65504.f;
        const int in_e = in_finite ? max((int)((__float_as_uint(mx) >> 23) & 255u) - 126, -24) : 16;   // mx < 2^in_e
        const int up_e = max(8 - in_e, 0);
        const float up = pow2f(up_e), down = pow2f(-up_e);
        const int room = 16 - max(in_e, 8);                                     // scales below 2^room: products below 2^16
#pragma unroll
        for (int j = 0; j < NX; ++j) {
            const int i = tid + kGemvThreads * j;
            if (i < n_st * 32) xs[i] = __float2half_rn(__half2float(xr[j]) * up);
        }
        __syncthreads();

        // the window's powers of two: of the group of this lane's B column, undone for the group of its C columns; lanes g < 4 watch
        // that the scales of group g stay below `lim`
        __half2 s_up = __floats2half2_rn(1.f, 1.f), lim = s_up;
        float undo = 1.f;
        uint32_t top = 0u;                                                      // exponent bits of the window's largest scale of the group
        bool turn = false;                                                      // every other 16 rows complemented
        int since = 0;
        auto flush = [&]() {
#pragma unroll
            for (int m = 0; m < 8; ++m) {
                sum[m][0] = fmaf(acc[m][0] + acc[m][1], undo, sum[m][0]);
                sum[m][1] = fmaf(acc[m][2] + acc[m][3], undo, sum[m][1]);
                acc[m][0] = acc[m][1] = acc[m][2] = acc[m][3] = 0.f;
            }
            // lanes of rows 4 .. 7: zero terms of all rows; of rows 0 .. 3: sums of in * scale of the complemented rows
            const float z = g < 4 ? (turn ? accz[1][0] : 0.f) : accz[0][0] + accz[1][0];
            zsum = fmaf(z, down, zsum);
#pragma unroll
            for (int i = 0; i < 4; ++i) accz[0][i] = accz[1][i] = 0.f;
            since = 0;
        };
        // A window opens with the largest scales of its first stage (`m`: a lane's largest, four lanes hold a group); a stage with a
        // scale of more than eight times that closes it early.
        auto open_window = [&](__half2 m) {
            if (since) flush();
            else top = 0u;
            m = __hmax2(m, as_h2(__shfl_xor_sync(0xffffffffu, as_u32(m), 1)));
            m = __hmax2(m, as_h2(__shfl_xor_sync(0xffffffffu, as_u32(m), 2)));
            top = max(top, (uint32_t)__half_as_ushort(__hmax(__low2half(m), __high2half(m))) & 0x7c00u);
            const uint32_t l = g < ngw && top < 0x7c00u ? min(top + 0x0fffu, 0x7bffu) : 0x7c00u;      // scales up to here are below 2^(exponent - 11)
            lim = as_h2(l | (l << 16));
            const float f = pow2f(min(room - ((int)(top >> 10) - 11), 15));
            const float fb = __shfl_sync(0xffffffffu, f, 4 * (g >> 1)), fc = __shfl_sync(0xffffffffu, f, 4 * tig);
            s_up = __floats2half2_rn(fb, fb);
            undo = down * __uint_as_float((254u << 23) - __float_as_uint(fc));
            turn = in_finite && !__any_sync(0xffffffffu, g < ngw && top == 0x7c00u);
        };

        for (int t = 0; t < plan.tpw; ++t) {
        const int n0 = n0_first + t * WC * 128;
        if (n0 >= N) break;
#pragma unroll 1
        for (int st = wk; st < n_st; st += WK) {
            issue(iss_slot);
            iss_slot = iss_slot == (G::NS - 1) * G::STAGE_BYTES ? 0u : iss_slot + G::STAGE_BYTES;
            cp_async_wait<G::NS - 1>();
            __syncwarp();
            uint32_t r[2][2];                                                   // scales (lanes g < 4) and zeros of 16 rows, transposed
#pragma unroll
            for (int k = 0; k < 2; ++k)
                asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];\n"
                             : "=r"(r[k][0]), "=r"(r[k][1]) : "r"(szm_s + slot + k * 256));
            const __half2 m = __hmax2(__hmax2(__habs2(as_h2(r[0][0])), __habs2(as_h2(r[0][1]))), __hmax2(__habs2(as_h2(r[1][0])), __habs2(as_h2(r[1][1]))));
            if (__any_sync(0xffffffffu, since == 0 || __hgt2_mask(m, lim) != 0u)) open_window(m);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const uint32_t xa = x_s + (32 * st + 16 * k) * 2;
                const uint32_t x01u = lds32(xa), x89u = lds32(xa + 16);
                const uint32_t r0 = r[k][0], r1 = r[k][1];
                mma16816(accz[k], r0, 0u, r1, 0u, x01u, x89u);
                const uint32_t flip = k && turn ? 0xffffffffu : 0u, sign = flip & 0x80008000u;
                uint32_t b0 = hilo(as_h2(x01u ^ sign), __hmul2(as_h2(__shfl_sync(0xffffffffu, r0, src)), s_up), neg_mask);
                uint32_t b1 = hilo(as_h2(x89u ^ sign), __hmul2(as_h2(__shfl_sync(0xffffffffu, r1, src)), s_up), neg_mask);
                if (!turn) {                                                    // behind an infinite hi the minimum keeps a number, and the sum infinite
                    const __half2 big = __floats2half2_rn(65504.f, 65504.f);
                    b0 = (as_u32(__hmin2(as_h2(b0), big)) & neg_mask) | (b0 & ~neg_mask);
                    b1 = (as_u32(__hmin2(as_h2(b1), big)) & neg_mask) | (b1 & ~neg_mask);
                }
                uint32_t x[NBLK][2];
                const uint32_t ad = ldk_s + slot + (16 * k) * G::RS;
                if constexpr (BITS == 1) {
                    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];\n" : "=r"(x[0][0]), "=r"(x[0][1]) : "r"(ad));
                } else {
#pragma unroll
                    for (int p = 0; p < NBLK / 2; ++p)
                        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                                     : "=r"(x[2 * p][0]), "=r"(x[2 * p][1]), "=r"(x[2 * p + 1][0]), "=r"(x[2 * p + 1][1]) : "r"(ad + 32 * p));
                }
#pragma unroll
                for (int bb = 0; bb < NBLK; ++bb) {
                    uint32_t rlo[F::N], rhi[F::N];
                    F::unpack(x[bb][0] ^ flip, rlo);
                    F::unpack(x[bb][1] ^ flip, rhi);
#pragma unroll
                    for (int i = 0; i < F::N; i += 2)
                        mma16816(acc[bb * MPB + i / 2], rlo[i], rlo[i + 1], rhi[i], rhi[i + 1], b0, b1);
                }
            }
            __syncwarp();
            slot = slot == (G::NS - 1) * G::STAGE_BYTES ? 0u : slot + G::STAGE_BYTES;
            if (++since == kGemvFlush) flush();
        }
        if (since) flush();
        if (WK > 1 || plan.kc > 1 || k_end - k_beg > kGemvChunk) continue;
        // ---- a tile of one warp: its sums are the result
        tile_sums();
        __syncwarp();
        const float4 v = *reinterpret_cast<const float4 *>(red + warp * 128 + 4 * lane);
        __syncwarp();
        if (n0 + 128 <= N && plan.out_vec) {
            const __half2 lo = __floats2half2_rn(v.x, v.y), hi = __floats2half2_rn(v.z, v.w);
            *reinterpret_cast<uint2 *>(out + n0 + 4 * lane) = make_uint2(as_u32(lo), as_u32(hi));
        } else {
            const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (n0 + 4 * lane + i < N) out[n0 + 4 * lane + i] = __float2half_rn(e[i]);
        }
        clear();
        }
        cp_async_wait<0>();
        __syncwarp();
    }
    if (WK == 1 && plan.kc == 1 && k_end - k_beg <= kGemvChunk) return;

    if (col0 + wc * 128 < N) tile_sums();
    __syncthreads();
    namespace cg = cooperative_groups;
    if (plan.kc > 1) {                                                          // every rank: the sums over its warps; rank 0 adds the ranks
        for (int i = tid; i < WC * 128; i += kGemvThreads) {
            float v = 0.f;
            for (int j = 0; j < WK; ++j) v += red[((i >> 7) * WK + j) * 128 + (i & 127)];
            red[((i >> 7) * WK) * 128 + (i & 127)] = v;                         // only this thread reads or writes these entries
        }
        cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();
        if (rank == 0) {
            for (int i = tid; i < WC * 128; i += kGemvThreads) {
                float v = 0.f;
                for (int r = 0; r < plan.kc; ++r) v += cluster.map_shared_rank(red, r)[((i >> 7) * WK) * 128 + (i & 127)];
                if (col0 + i < N) out[col0 + i] = __float2half_rn(v);
            }
        }
        cluster.sync();                                                         // nobody leaves while its sums are read
    } else {
        for (int i = tid; i < WC * 128; i += kGemvThreads) {
            float v = 0.f;
            for (int j = 0; j < WK; ++j) v += red[((i >> 7) * WK + j) * 128 + (i & 127)];
            if (col0 + i < N) out[col0 + i] = __float2half_rn(v);
        }
    }
}

template <int BITS, int GS_LOG2>
static int launch_gemv_mma(const kvq_gemv_args &a, const GemvPlan &p, unsigned grid, cudaStream_t st) {
    const size_t smem = kGemvWarps * 128 * 4 + kGemvChunk * 2 + 8 * 4 + 96 + (size_t)kGemvWarps * GemvGeom<BITS>::WARP_BYTES;
    static bool attr_set[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return record_cuda_error(e);
    if (dev < 0 || dev >= 64 || !attr_set[dev]) {
        e = cudaFuncSetAttribute(gemv_mma_kernel<BITS, GS_LOG2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return record_cuda_error(e);
        if (dev >= 0 && dev < 64) attr_set[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kGemvThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;            // see grid_wait()
    attr[0].val.programmaticStreamSerializationAllowed = p.early;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)p.kc;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = p.kc > 1 ? 2 : 1;
    e = cudaLaunchKernelEx(&cfg, gemv_mma_kernel<BITS, GS_LOG2>, a, p);
    if (e != cudaSuccess) return record_cuda_error(e);
    return check_launch();
}

// The split of the work: a CTA's eight warps take as many column tiles as there are (p . V has one) and share each tile's rows
// with the rest; where heads x column CTAs leave half of the resident CTAs (296) idle, clusters of up to eight CTAs cut
// the rows further, at least 512 a CTA.
static bool gemv_mma_plan(const kvq_gemv_args &a, int64_t n_pack, GemvPlan &p, int64_t &grid) {
    if (a.bits == 3 || (a.group != 32 && a.group != 64 && a.group != 128)) return false;
    if (a.K <= 0 || a.K > (1 << 30) || a.n_groups * a.group > (1 << 30)) return false;
    const int64_t tiles = (a.n_groups * a.group + 127) / 128;
    p.wk_log2 = tiles > 4 ? 0 : tiles > 2 ? 1 : tiles > 1 ? 2 : 3;
    const int wc = kGemvWarps >> p.wk_log2;
    // a warp's tiles one after the other where they are short (all rows in one chunk) and there are CTAs enough
    p.tpw = 1;
    while (p.wk_log2 == 0 && a.K <= kGemvTileRows && p.tpw < kGemvTiles && a.B * a.nh * ((tiles + 2 * wc * p.tpw - 1) / (2 * wc * p.tpw)) >= kGemvMinCtas) p.tpw *= 2;
    p.col_ctas = (int)((tiles + (int64_t)wc * p.tpw - 1) / ((int64_t)wc * p.tpw));
    const int64_t jobs = a.B * a.nh * p.col_ctas;
    p.kc = 1;
    while (p.kc < 8 && jobs * p.kc * 2 <= 2 * 148 && a.K >= 512LL * p.kc * 2) p.kc *= 2;
    p.rows_per_cta = (int)((a.K + 32LL * p.kc - 1) / (32LL * p.kc) * 32);
    const uint64_t bits = reinterpret_cast<uintptr_t>(a.qB) | (uint64_t)(4 * (a.q_sB | a.q_sH | a.q_sK | n_pack));
    p.code_align = bits % 16 == 0 ? 16 : bits % 8 == 0 ? 8 : 4;
    const int ngw = 128 / a.group;
    p.sz_vec = (reinterpret_cast<uintptr_t>(a.scale) | reinterpret_cast<uintptr_t>(a.zero)) % (2 * ngw) == 0 &&
               a.s_sB % ngw == 0 && a.s_sH % ngw == 0 && a.s_sK % ngw == 0;
    p.fast = p.code_align == 16 && p.sz_vec && a.q_sK >= 0 && a.s_sK >= 0 && a.K * a.q_sK < (1LL << 30) && a.K * a.s_sK < (1LL << 31) &&
             a.q_sK < (1 << 24) && a.s_sK < (1 << 25);
    p.rep = (int)(a.nh / a.nh_kv);
    // Clusters of CTAs, where there are many of them, neither come early nor let anybody in early: CTAs that are placed while others still hold
    // their SMs come to lie two to an SM with SMs left over.  q . K^T and p . V in turn, us, early / ordinary: 32 heads of 4096 tokens 15.7 /
    // 13.2, of 2048 14.4 / 11.8, 128 heads of 1024 15.4 / 13.4 (15.1, 13.6 and 15.2 before early launches); without clusters: 128 heads of 256
    // 9.3 / 10.4, 512 of 128 14.4 / 15.0.
    p.early = p.kc == 1 || jobs * p.kc < 64;
    p.out_vec = (reinterpret_cast<uintptr_t>(a.out) | (uint64_t)(2 * (a.o_sB | a.o_sH))) % 8 == 0;
    grid = jobs * p.kc;
    return grid <= 2147483647LL && a.B * a.nh <= 2147483647LL;
}

}  // namespace kvq

extern "C" int kvq_gemv(const kvq_gemv_args *a, kvq_stream_t stream) {
    using namespace kvq;
    if (!a) return KVQ_ERR_NULL;
    if (a->bits < 1 || a->bits > 4) return KVQ_ERR_BITS;
    if (a->nh_kv <= 0 || a->nh % a->nh_kv != 0) return KVQ_ERR_HEADS;
    if (a->bits == 3 && a->group != 11) return KVQ_ERR_GROUP3;
    const int fpi = fields_per_word(a->bits);
    if (a->group <= 0 || a->group % fpi != 0) return KVQ_ERR_GROUPWORD;
    if (a->B < 0 || a->K < 0 || a->n_groups < 0) return KVQ_ERR_SHAPE;
    const int64_t n_pack = (a->n_groups * a->group) / fpi;
    if (n_pack > a->n_words) return KVQ_ERR_SHAPE;
    if (a->B * a->nh == 0 || n_pack == 0) return KVQ_OK;
    if (!a->fA || !a->out) return KVQ_ERR_NULL;
    if (a->K > 0 && (!a->qB || !a->scale || !a->zero)) return KVQ_ERR_NULL;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    GemvPlan p;
    int64_t mma_grid = 0;
    if (gemv_mma_plan(*a, n_pack, p, mma_grid)) {
#define KVQ_GEMV_CASE(BITS, GS_LOG2) \
        if (a->bits == BITS && a->group == 1 << GS_LOG2) return launch_gemv_mma<BITS, GS_LOG2>(*a, p, (unsigned)mma_grid, st);
        KVQ_GEMV_CASE(1, 5) KVQ_GEMV_CASE(1, 6) KVQ_GEMV_CASE(1, 7)
        KVQ_GEMV_CASE(2, 5) KVQ_GEMV_CASE(2, 6) KVQ_GEMV_CASE(2, 7)
        KVQ_GEMV_CASE(4, 5) KVQ_GEMV_CASE(4, 6) KVQ_GEMV_CASE(4, 7)
#undef KVQ_GEMV_CASE
    }
    int wx_log2 = 5;
    while (wx_log2 > 2 && (1 << (wx_log2 - 1)) >= n_pack) --wx_log2;
    const int WX = 1 << wx_log2;
    const int64_t nblk = (n_pack + WX - 1) / WX;
    if (nblk * a->B * a->nh > 2147483647LL) return KVQ_ERR_UNSUPPORTED;
    dim3 grid((unsigned)(nblk * a->B * a->nh));
    switch (a->bits) {
        case 1: gemv_kernel<1><<<grid, 256, 0, st>>>(*a, wx_log2, (int)nblk); break;
        case 2: gemv_kernel<2><<<grid, 256, 0, st>>>(*a, wx_log2, (int)nblk); break;
        case 3: gemv_kernel<3><<<grid, 256, 0, st>>>(*a, wx_log2, (int)nblk); break;
        case 4: gemv_kernel<4><<<grid, 256, 0, st>>>(*a, wx_log2, (int)nblk); break;
    }
    return check_launch();
}
