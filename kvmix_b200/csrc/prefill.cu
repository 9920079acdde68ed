// A prompt into the cache: keys (rotated on the way when tables are given) and values quantized, the fp16 tails into their rings.
#include "quant_tiles.cuh"

namespace kvq {

int quant_lastdim_impl(const kvq_quant_args *a, kvq_stream_t stream, const RopeTables *rope);   // quant.cu

__global__ void __launch_bounds__(256) prefill_tails_kernel(kvq_prefill_args a) {
    prefill_tail_chunk(a, (int64_t)blockIdx.x * 256 + threadIdx.x);
}

// Everything at once: CTAs [0, k_ctas) take a tile of keys each, the next v_ctas 256 units of 32 values (3 bits: 256 words), the
// others 256 chunks of the tails.  One launch instead of three: the keys alone are 1.7 waves of long CTAs at 2 x 8 kv heads x 8191
// tokens, and the short ones behind them fill what the last of them leaves idle: three such layers (4, 3 and 2 bits, groups of 64)
// 131 -> 103 us, 95 where a layer's launch overlaps the end of the one before.  Bound by the instructions of rotation and of bit-exact
// codes.
struct PrefillGrid { int k_tiles, k_ctas, v_per_slab, v_ctas; };

template <int KB, int KG, int VB>
__global__ void __launch_bounds__(256, 4) prefill_kernel(const __grid_constant__ kvq_prefill_args a, const __grid_constant__ QuantDims kd,
                                                         const __grid_constant__ QuantDims vd, const __grid_constant__ RopeTables rope,
                                                         const __grid_constant__ PrefillGrid p) {
    int c = blockIdx.x;
    grid_wait();
    launch_next();
    if (c < p.k_ctas) {
        const int bh = c / p.k_tiles;
        quant_rope_tile<KB, KG>(static_cast<const __half *>(a.k), a.kcode, static_cast<__half *>(a.kscale), static_cast<__half *>(a.kmn), kd, rope, c - bh * p.k_tiles, bh);
        return;
    }
    c -= p.k_ctas;
    if (c < p.v_ctas) {
        const __half *x = static_cast<const __half *>(a.v);
        __half *sc = static_cast<__half *>(a.vscale), *mn = static_cast<__half *>(a.vmn);
        if constexpr (VB == 3) {
            quant_ragged3_word<__half>(x, a.vcode, sc, mn, vd, (int64_t)c * 256 + threadIdx.x);
        } else {
            const int bh = c / p.v_per_slab, b = bh / (int)vd.H;
            quant_contig_unit<VB, __half, VB>(x, a.vcode, sc, mn, vd, vd.group / 32, true, false, b, bh - b * (int)vd.H, (c - bh * p.v_per_slab) * 256 + threadIdx.x);
        }
        return;
    }
    prefill_tail_chunk(a, (int64_t)(c - p.v_ctas) * 256 + threadIdx.x);
}

template <int KB, int KG, int VB>
static int launch_prefill(const kvq_prefill_args &a, const QuantDims &kd, const QuantDims &vd, const RopeTables &rope, cudaStream_t st) {
    PrefillGrid p;
    const int64_t slabs = (int64_t)a.B * a.Hkv;
    p.k_tiles = (a.nk / KG + RopeCfg<KB, KG>::GPC - 1) / RopeCfg<KB, KG>::GPC;
    p.v_per_slab = (int)(((int64_t)a.nv * (kHeadDim / 32) + 255) / 256);
    const int64_t k_ctas = slabs * p.k_tiles, v_ctas = VB == 3 ? (slabs * a.nv * 12 + 255) / 256 : slabs * p.v_per_slab;
    const int64_t t_ctas = (slabs * ((int64_t)(a.L - a.nk) + (a.L - a.nv)) * 8 + 255) / 256;
    if (k_ctas + v_ctas + t_ctas > 2147483647LL) return KVQ_ERR_UNSUPPORTED;
    p.k_ctas = (int)k_ctas;
    p.v_ctas = (int)v_ctas;
    return launch_early(true, prefill_kernel<KB, KG, VB>, (unsigned)(k_ctas + v_ctas + t_ctas), 256, 0, st, a, kd, vd, rope, p);
}

// KVQ_ERR_UNSUPPORTED: not for this kernel.
static int prefill_at_once(const kvq_prefill_args &a, const QuantDims &kd, const QuantDims &vd, const RopeTables &rope, cudaStream_t st) {
    if (a.k_bits == 3 ? a.k_group != 11 : a.k_group != 32 && a.k_group != 64 && a.k_group != 128) return KVQ_ERR_UNSUPPORTED;
    if (a.v_bits == 3 ? a.v_group != 11 : a.v_group != 32 && a.v_group != 64 && a.v_group != 128) return KVQ_ERR_UNSUPPORTED;
    if (a.nk % a.k_group != 0 || (int64_t)a.B * a.Hkv > 65535) return KVQ_ERR_UNSUPPORTED;
#define KVQ_V(KB, KG)                                                                  \
    switch (a.v_bits) {                                                                \
        case 1: return launch_prefill<KB, KG, 1>(a, kd, vd, rope, st);                 \
        case 2: return launch_prefill<KB, KG, 2>(a, kd, vd, rope, st);                 \
        case 3: return launch_prefill<KB, KG, 3>(a, kd, vd, rope, st);                 \
        default: return launch_prefill<KB, KG, 4>(a, kd, vd, rope, st);                \
    }
#define KVQ_K(KB)                                                                      \
    if (a.k_bits == KB) {                                                              \
        if (a.k_group == 32) KVQ_V(KB, 32)                                             \
        if (a.k_group == 64) KVQ_V(KB, 64)                                             \
        KVQ_V(KB, 128)                                                                 \
    }
    KVQ_K(1) KVQ_K(2) KVQ_K(4)
    KVQ_V(3, 11)
#undef KVQ_K
#undef KVQ_V
}

}  // namespace kvq

extern "C" int kvq_prefill(const kvq_prefill_args *a, kvq_stream_t stream) {
    using namespace kvq;
    if (!a) return KVQ_ERR_NULL;
    if (a->D != kHeadDim) return KVQ_ERR_UNSUPPORTED;
    if (a->B <= 0 || a->Hkv <= 0 || a->L <= 0) return KVQ_OK;
    if (a->nk < 0 || a->nv < 0 || a->nk > a->L || a->nv > a->L) return KVQ_ERR_TOKENS;
    if (!a->k || !a->v) return KVQ_ERR_NULL;
    if ((a->cos == nullptr) != (a->sin == nullptr)) return KVQ_ERR_NULL;
    if (a->k_bits < 1 || a->k_bits > 4 || a->v_bits < 1 || a->v_bits > 4) return KVQ_ERR_BITS;
    auto al16 = [](const void *p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
    if (!al16(a->k) || !al16(a->v) || a->k_sB % 8 || a->k_sT % 8 || a->k_sH % 8 || a->v_sB % 8 || a->v_sT % 8 || a->v_sH % 8)
        return KVQ_ERR_ALIGN;
    if (a->cos && (!al16(a->cos) || !al16(a->sin) || a->r_sB % 8 || a->r_sT % 8)) return KVQ_ERR_ALIGN;
    if (a->nk < a->L && (!a->kfull || !al16(a->kfull) || a->kf_sB % 8 || a->kf_sH % 8 || a->kf_sT % 8)) return KVQ_ERR_ALIGN;
    if (a->nv < a->L && (!a->vfull || !al16(a->vfull) || a->vf_sB % 8 || a->vf_sH % 8 || a->vf_sT % 8)) return KVQ_ERR_ALIGN;
    kvq_quant_args kq{a->k, 0, a->B, a->Hkv, a->D, a->nk, a->k_sB, a->k_sH, 1, a->k_sT, a->k_group, a->k_bits, 0,
                      a->kcode, a->kc_sB, a->kc_sH, a->kc_sD, a->kscale, a->kmn, a->ks_sB, a->ks_sH, a->ks_sD};
    kvq_quant_args vq{a->v, 0, a->B, a->Hkv, a->nv, a->D, a->v_sB, a->v_sH, a->v_sT, 1, a->v_group, a->v_bits, 0,
                      a->vcode, a->vc_sB, a->vc_sH, a->vc_sT, a->vscale, a->vmn, a->vs_sB, a->vs_sH, a->vs_sT,
                      a->v_bits == 3 ? 1 : 0};                 // 3-bit values: the short-last-group extension
    const RopeTables rope{static_cast<const __half *>(a->cos), static_cast<const __half *>(a->sin), a->r_sB, a->r_sT};
    if (a->cos && a->nk > 0 && a->nv > 0 && a->kcode && a->kscale && a->kmn && a->vcode && a->vscale && a->vmn) {
        auto dims = [](const kvq_quant_args &q) {
            return QuantDims{q.B, q.H, q.A, q.S, q.x_sB, q.x_sH, q.x_sA, q.x_sS, q.c_sB, q.c_sH, q.c_sA, q.z_sB, q.z_sH, q.z_sA, q.group, 0};
        };
        const int rc = prefill_at_once(*a, dims(kq), dims(vq), rope, reinterpret_cast<cudaStream_t>(stream));
        if (rc != KVQ_ERR_UNSUPPORTED) return rc;
    }
    if (a->nk > 0) {                                           // keys: groups over tokens, channels contiguous, read in place
        const int rc = quant_lastdim_impl(&kq, stream, a->cos ? &rope : nullptr);
        if (rc) return rc;
    }
    if (a->nv > 0) {                                           // values: groups over channels
        const int rc = kvq_quant_lastdim(&vq, stream);
        if (rc) return rc;
    }
    const int64_t n = (int64_t)a->B * a->Hkv * ((int64_t)(a->L - a->nk) + (a->L - a->nv)) * 8;
    if (n > 0) {
        prefill_tails_kernel<<<(unsigned)((n + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(*a);
        return check_launch();
    }
    return KVQ_OK;
}
