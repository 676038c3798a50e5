// What the two decode attention kernels share (attn_decode.cu on tensor cores, attn_decode_f32.cu on f32 multiply-adds): block shape, page copies
// with bounded waits, the forms of the result.
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace forge {
namespace decode {

constexpr int kThreads = 128;     // consumer threads (four warps); warp 4 is the producer
constexpr int kBlock = kThreads + 32;
constexpr int kStages = 4;        // most pages (K and V) in flight per CTA
constexpr int kMaxGroup = 16;     // query heads per KV head
constexpr int kMaxSplits = 32;    // context splits per KV head
constexpr uint32_t kSpin = 1u << 22;

struct DecParams {
    AttnDecodeArgs a;
    float scale;  // of the scores
    int stages;   // ring depth of this launch (<= kStages)
    float scale_lo;   // what `scale` leaves of its exact value
};

#ifdef __CUDACC__
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    const uint32_t addr = smem_u32(bar);
    for (uint32_t i = 0; i < kSpin; ++i) {
        uint32_t done;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
                     : "=r"(done) : "r"(addr), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}
// one page of one KV head from dimension `dim` on, as wide as the map's box
__device__ __forceinline__ void tma_page(void* dst, const CUtensorMap* map, int dim, int kvh, int row, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(dim), "r"(kvh), "r"(row), "r"(smem_u32(bar)) : "memory");
}
// the result in the form the caller asked for: f32, or fp16 hi (+ lo)
__device__ __forceinline__ void store_out(const AttnDecodeArgs& a, size_t i, float x) {
    if (a.out16) {
        const __half h = __float2half_rn(x);
        a.out16[i] = h;
        if (a.out16_lo) a.out16_lo[i] = __float2half_rn(x - __half2float(h));
    } else {
        a.out[i] = x;
    }
}
__device__ __forceinline__ void store_out2(const AttnDecodeArgs& a, size_t i, float2 x) {
    if (a.out16) {
        const __half2 h = __floats2half2_rn(x.x, x.y);
        *reinterpret_cast<__half2*>(a.out16 + i) = h;
        if (a.out16_lo) {
            const float2 hf = __half22float2(h);
            *reinterpret_cast<__half2*>(a.out16_lo + i) = __floats2half2_rn(x.x - hf.x, x.y - hf.y);
        }
    } else {
        *reinterpret_cast<float2*>(a.out + i) = x;
    }
}
__device__ __forceinline__ void csync() { asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory"); }
#endif

}  // namespace decode
}  // namespace forge
