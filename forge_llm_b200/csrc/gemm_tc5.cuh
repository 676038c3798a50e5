// What the two tcgen05 products of quantised weights with many rows share (gemm_tc5.cu: one CTA per tile; gemm_pair.cu: pairs of CTAs that stay):
// parameters and the split of a weight into two fp16 values.
#pragma once

#include "common.cuh"

namespace forge {
namespace tc5w {

struct Tc5Params {
    float* out; const float* resid;
    const uint8_t* qs; const __half* d; const float4* sf;
    int m, N, K;
    int* err;
    int ksplit;            // K slices (grid.z); slice z leaves its partial product at out + z * part_stride
    size_t part_stride;
    // gate/up product (weight rows 2j = gate_j, 2j + 1 = up_j): when act_hi is set the epilogue stores
    // SiLU(gate_j) * up_j as fp16 hi (+ lo) into act[token][N / 2] instead of the f32 rows
    __half* act_hi; __half* act_lo;
};

#ifdef __CUDACC__
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}
__device__ __forceinline__ __half2 as_h2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
__device__ __forceinline__ uint32_t as_u32(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }

// two integer weights (exact in fp16) times the block scale: hi = rn16(q*d), lo = rn16(q*d - hi).  The fp16 multiply
// rounds the exact product once and the fused multiply-add forms q*d - hi exactly before its one rounding, so
// hi + lo carries the 19-bit product q*d to the last bit (|lo| <= ulp(hi)/2 is itself exact in fp16).
__device__ __forceinline__ void scale_split(__half2 q, __half2 d, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __hmul2(q, d);
    hi = as_u32(h);
    lo = as_u32(__hfma2(q, d, __hneg2(h)));
}

// 32 consecutive weights of one row (one quantisation block) -> 16 + 16 packed fp16 pairs (hi, lo)
template <int QUANT, bool SPLIT>
__device__ __forceinline__ void dequant_block(const uint32_t* cur, __half2 d2, uint32_t (&hi)[16], uint32_t (&lo)[16]) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {      // 8 values per group
#pragma unroll
        for (int i = 0; i < 4; ++i) {  // 2 values per register
            __half2 q;
            const uint32_t sel = (i & 1) ? 0x4342u : 0x4140u;
            if (QUANT == FORGE_Q8_0) {
                const uint32_t word = cur[2 * c + (i >> 1)];
                q = __hsub2(as_h2(prmt(word ^ 0x80808080u, 0x64646464u, sel)), __float2half2_rn(1152.f));
            } else {
                const uint32_t word = cur[2 * (c & 1) + (i >> 1)];
                const uint32_t two = prmt(word, 0u, sel) >> ((c >> 1) * 4);
                q = __hsub2(as_h2((two & 0x000F000Fu) | 0x64006400u), __float2half2_rn(1032.f));
            }
            if (SPLIT) scale_split(q, d2, hi[4 * c + i], lo[4 * c + i]);
            else hi[4 * c + i] = as_u32(__hmul2(q, d2));
        }
    }
}

// K-quant rows in the expanded row-major layout (FORGE_KQ_SOA): 32 int8 values and {s_lo, s_hi, mn}; the value
// s * q - mn is formed in f32 (one fused rounding) and split into hi = rn16(w), lo = rn16(w - hi): 22 bits of w.
template <bool SPLIT>
__device__ __forceinline__ void dequant_block_kq(const uint32_t* cur, float4 sc, uint32_t (&hi)[16], uint32_t (&lo)[16]) {
#pragma unroll
    for (int j = 0; j < 16; ++j) {  // register j = elements 2j, 2j + 1
        const uint32_t word = cur[j >> 1];
        const int q0 = int(int8_t(word >> (16 * (j & 1)))), q1 = int(int8_t(word >> (16 * (j & 1) + 8)));
        const float s = j < 8 ? sc.x : sc.y;
        const float w0 = fmaf(s, float(q0), -sc.z), w1 = fmaf(s, float(q1), -sc.z);
        const __half2 h = __floats2half2_rn(w0, w1);
        hi[j] = as_u32(h);
        if (SPLIT) {
            const float2 hf = __half22float2(h);
            lo[j] = as_u32(__floats2half2_rn(w0 - hf.x, w1 - hf.y));
        }
    }
}
#endif

}  // namespace tc5w
}  // namespace forge
