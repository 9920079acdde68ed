// Shared device/host helpers for the kvmix_b200 kernels (sm_100a only).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/kvmix_b200.h"

#if defined(__CUDA_ARCH__) && (__CUDA_ARCH__ < 1000)
#error "kvmix_b200 kernels are written for sm_100a only"
#endif

namespace kvq {

constexpr int kHeadDim = 128;

__host__ __device__ constexpr int fields_per_word(int bits) { return bits == 3 ? 11 : 32 / bits; }

// Field i of a packed word.  3-bit words hold ten 3-bit fields and a 2-bit field at bit 30.
template <int BITS>
__device__ __forceinline__ uint32_t field(uint32_t w, int i) {
    if constexpr (BITS == 3) {
        return i < 10 ? ((w >> (3 * i)) & 7u) : (w >> 30);
    } else {
        return (w >> (BITS * i)) & ((1u << BITS) - 1u);
    }
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Records the text of the last failing CUDA call for kvq_last_cuda_error().
// Additive attention mask value for (sequence b, query head h, key position t); the caller checked a.mask != NULL.
__device__ __forceinline__ float attn_mask_at(const kvq_attn_args &a, int b, int h, int t) {
    const int64_t off = (int64_t)b * a.mask_sB + (int64_t)h * a.mask_sH + t;
    return a.mask_is_f32 ? __ldca(static_cast<const float *>(a.mask) + off)
                         : __half2float(__ldca(static_cast<const __half *>(a.mask) + off));
}
// upstream clamps masked weights from below at torch.finfo(float32).min (models/modeling_llama_KVmix.py:192)
constexpr float kMaskFloor = -3.4028234663852886e38f;

// Programmatic launches: a kernel launched by launch_early() may be put on the GPU while the kernel before it in the stream is still
// running its last CTAs, as soon as each of those has called launch_next(); grid_wait() then holds it until that kernel
// is complete and its writes are visible.  Nothing before grid_wait() touches global memory.  Behind a kernel that does not call
// launch_next() it is an ordinary launch.  Data are read by plain loads, __ldca, __ldcg or cp.async: __ldg(), and whatever the compiler turns into it
// (const __restrict__), wants memory that nobody writes while the kernel is resident, which here the kernel before may.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void launch_next() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// Counts a CTA in, device-wide: what its threads wrote before the CTA barrier in front of it is visible to whoever reads the last count
// and synchronises behind it.  One acquire-release atomic; between two __threadfence() (sequentially consistent ones) it took 2700
// cycles at the end of every CTA, with its SM half idle.
__device__ __forceinline__ unsigned int count_in(unsigned int *counter) {
    unsigned int old;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;\n" : "=r"(old) : "l"(counter) : "memory");
    return old;
}

int record_cuda_error(cudaError_t e);
inline int check_launch() { return record_cuda_error(cudaGetLastError()); }
template <typename... P, typename... A>
inline int launch_early(bool early, void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = early;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
    return e == cudaSuccess ? check_launch() : record_cuda_error(e);
}

}  // namespace kvq
