// The prompt product of gemm_tc5.cu on CTA pairs that stay: out[m][N] = A[m][K] x W[N][K]^T, W as Q8_0 / Q4_0 blocks, split precision.
//
// A pair of CTAs (a cluster of two, tcgen05 cta_group::2) forms tiles of 256 weight rows x NT tokens (NT <= 192, a multiple of 32, chosen per launch), 128 rows
// in each CTA's tensor memory.  Every CTA copies half of a tile's tokens; a product reads both halves, so each activation byte reaches shared memory once per
// 256 weight rows.  There are at most as many pairs as the chip holds, and they walk over the tiles:
//   warp 0       activation tiles (hi and lo fp16 parts of this CTA's half of the tokens) by tensor copies into a ring of five stages; both CTAs' copies
//                complete on the first CTA's barrier;
//   warp 1       of the first CTA: issues per K step of 64 twelve products (w_hi x_hi + w_hi x_lo + w_lo x_hi) and one commit that gives the step's activation
//                and weight stages back to both CTAs;
//   warp 2       quantised bytes by tensor copies, 128 rows x 128 bytes per stage;
//   warp 3       tensor memory;
//   warps 4..11  weights: one 32-value block of one row per thread and K step, split into hi = rn16(q d) and lo = rn16(q d - hi), into tensor memory (two stages);
//   warps 12..19 epilogue, under the products of the next tile (two accumulators): two groups of four warps take 32 tokens in turn through shared memory, from
//                where a tensor copy stores them.
// A tensor-memory accumulator rounds toward zero at every step, so long K runs as slices (gemm_tc5_ksplit): a pair takes the slices of a tile one after another, each
// in its own accumulator, and adds them up in f32 in slice order in the output, or spreads them over `parts` partial outputs where tiles alone would leave
// pairs idle.
// (Added by the copy engine: one sum per element at a time, rounded to nearest; it may flush sums below 2^-126.)
// Every wait is bounded; a wait that gives up sets an error word, and the pair still meets and frees its tensor memory.
//
// What bounds it: the tensor pipe (12 products of 96 clocks per K step at 192 tokens = 0.61 us, measured 0.66) and from about 1500 TFLOP/s on the board's power.
// The one-CTA kernel of gemm_tc5.cu runs a K step as fast but begins and ends every tile with 11-12 us in which the tensor pipe stands still; here they lie
// under other tiles' products.  us per product, before -> now: Q4_0 2501 tokens 2048 -> 16384 with SiLU 373 -> 323, 8192 -> 2048 206 -> 168, 2048 -> 2048
// 80 -> 49; 2048 tokens 4096 -> 12288 556 -> 404; Q8_0 1282 tokens 896 -> 9728 with SiLU 88 -> 53, 64 tokens 896 -> 151936 171 -> 70, 896 -> 1152 20.5 -> 12.3.
// Tried: threads that store the output themselves (17 us a tile of 192 tokens, longer than its products at K = 896); four epilogue warps (14 us with the SiLU);
// barriers with cluster-wide ordering (each wait and arrival about 500 clocks: a K step of 1.15 us).
#include <cuda.h>

#include <algorithm>

#include "common.cuh"
#include "gemm_tc5.cuh"
#include "tc5.cuh"

namespace forge {

namespace {

using namespace tc5;
using namespace tc5w;

constexpr int kStep = 64;          // columns per K step: one 128-byte swizzle row of fp16
constexpr int kMaxTokens = 192;    // two accumulators and two weight stages fill the 512 columns of tensor memory
constexpr int kPairThreads = 640;
constexpr int kXStages = 5, kQStages = 4;
constexpr int kXStage = 2 * (kMaxTokens / 2) * kStep * 2, kQStage = 128 * 128;
constexpr int kOut = 32 * 128 * 4;   // 32 tokens x 128 rows on their way out, one buffer per epilogue group
constexpr int kPairSmem = kXStages * kXStage + kQStages * kQStage + 2 * kOut + 1024;
constexpr uint32_t kWCol = 2 * kMaxTokens;   // first column of the weight stages

struct PairParams {
    Tc5Params t;
    int nt;                 // tokens per tile
    int n_tiles, m_tiles;   // tiles along the weight rows (256) and the tokens
    int parts, slices;      // partial outputs, and K slices per partial output
    int bulk;               // the output's address and row length allow tensor copies
};
// one K slice of a tile
struct Slice { int n0, m0, part, first, k0, nk; };
__device__ __forceinline__ bool locate(const PairParams& p, int i, Slice& s) {
    const int item = int(blockIdx.x >> 1) + (i / p.slices) * int(gridDim.x >> 1), j = i % p.slices;
    if (item >= p.n_tiles * p.m_tiles * p.parts) return false;
    const int rest = item / p.n_tiles;
    s.n0 = (item - rest * p.n_tiles) * 256 + int(blockIdx.x & 1) * 128;
    s.part = rest / p.m_tiles;
    s.m0 = (rest - s.part * p.m_tiles) * p.nt;
    s.first = j == 0;
    const int steps = p.t.K / kStep, all = p.parts * p.slices, z = s.part * p.slices + j;
    s.k0 = steps * z / all;
    s.nk = steps * (z + 1) / all - s.k0;
    return true;
}

// Waits for barriers that the other CTA arrives at too (b may be null); bounded by time, since a query of a barrier can take any time up to the hardware's own limit
constexpr long long kWaitClocks = 1ll << 31;   // about a second
__device__ __forceinline__ bool pair_wait(uint64_t* a, uint32_t pa, uint64_t* b, uint32_t pb, const volatile int* cta_err) {
    const uint32_t aa = smem_u32(a), ab = b ? smem_u32(b) : 0;
    long long start = 0;
    for (uint32_t i = 1;; ++i) {
        uint32_t da, db = 1;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(da) : "r"(aa), "r"(pa) : "memory");
        if (b) asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(db) : "r"(ab), "r"(pb) : "memory");
        if (da && db) return true;
        if (!(i & 63u)) {
            const long long now = clock64();
            if (!start) start = now;
            if (*cta_err || now - start > kWaitClocks) return false;
        }
    }
}
// arrival at the first CTA's barrier
__device__ __forceinline__ void arrive_first(uint32_t addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
// tensor copy into this CTA's shared memory that completes on a barrier of either CTA of the pair
__device__ __forceinline__ void pair_load(void* dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void pair_mma(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t id, uint32_t accumulate) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n}"
                 ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(id), "r"(accumulate) : "memory");
}
// 32 tokens x 128 rows from shared memory to the output, or added to it there
__device__ __forceinline__ void bulk_store(const CUtensorMap* map, int x, int y, int z, const void* src) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(src)) : "memory");
}
__device__ __forceinline__ void bulk_add(const CUtensorMap* map, int x, int y, int z, const void* src) {
    asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(src)) : "memory");
}
__device__ __forceinline__ void epilogue_sync(int group) {
    if (group) asm volatile("bar.sync 2, 128;" ::: "memory");
    else asm volatile("bar.sync 1, 128;" ::: "memory");
}
// arrives at the barrier of both CTAs when all products issued before are complete
__device__ __forceinline__ void pair_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"(uint16_t(3)) : "memory");
}

// A chunk of the accumulator (v: 32 tokens of the weight row of thread e) as the output takes it: f32 [token][128 rows], or SiLU(gate) * up as fp16 hi [token][64]
// and lo behind it
__device__ __forceinline__ void stage_chunk(const uint32_t (&v)[32], unsigned char* stage, bool silu, int e) {
    if (silu) {
        // neighbouring lanes hold gate_j and up_j of the same tokens: the even lane takes the first sixteen tokens, the odd lane the others
        const bool even = !(e & 1);
        __half* hi = reinterpret_cast<__half*>(stage) + (even ? 0 : 16 * 64) + (e >> 1);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const uint32_t got = __shfl_xor_sync(0xffffffffu, even ? v[16 + j] : v[j], 1);
            const float g = __uint_as_float(even ? v[j] : got), u = __uint_as_float(even ? got : v[16 + j]);
            const float x = (g / (1.0f + expf(-g))) * u;
            const __half h = __float2half_rn(x);
            hi[j * 64] = h;
            hi[32 * 64 + j * 64] = __float2half_rn(x - __half2float(h));
        }
    } else {
        float* f = reinterpret_cast<float*>(stage) + e;
#pragma unroll
        for (int j = 0; j < 32; ++j) f[j * 128] = __uint_as_float(v[j]);
    }
}
// the staged chunk to global memory by the group's threads: outputs that tensor copies cannot store, and those that something is added to
__device__ __forceinline__ void copy_chunk(const Tc5Params& p, const unsigned char* stage, float* out, const float* add, int row0, int n0, int e) {
    const int rows = min(32, p.m - row0);
    if (n0 + e >= p.N) return;
    const float* f = reinterpret_cast<const float*>(stage) + e;
    const size_t at = size_t(row0) * p.N + n0 + e;
#pragma unroll 1
    for (int j = 0; j < rows; j += 8) {   // what is added may lie in the output: eight loads in front of their stores
        float x[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = add && j + k < rows ? add[at + size_t(j + k) * p.N] : 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (j + k < rows) out[at + size_t(j + k) * p.N] = x[k] + f[(j + k) * 128];
    }
}

template <int QUANT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1) gemm_pair_kernel(const __grid_constant__ CUtensorMap map_hi,
                                                                                            const __grid_constant__ CUtensorMap map_lo,
                                                                                            const __grid_constant__ CUtensorMap map_w,
                                                                                            const __grid_constant__ CUtensorMap map_out,
                                                                                            const __grid_constant__ CUtensorMap map_out_lo, PairParams p) {
    constexpr int kSuper = QUANT == FORGE_Q4_0 ? 4 : 2;    // K steps per stage of quantised bytes
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* sX = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char* sQ = sX + kXStages * kXStage;
    unsigned char* sO = sQ + kQStages * kQStage;
    // full_x, full_w and acc_free are the first CTA's: both arrive there.  done and acc_full are arrived at by commits, in both CTAs.
    __shared__ uint64_t full_x[kXStages], done[kXStages], full_w[2], full_q[kQStages], empty_q[kQStages], acc_full[2], acc_free[2];
    __shared__ uint32_t s_tmem;
    __shared__ int s_err;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, rank = int(blockIdx.x & 1);
    if (tid == 0) {
        for (int s = 0; s < kXStages; ++s) { mbar_init(&full_x[s], 1); mbar_init(&done[s], 1); }
        for (int s = 0; s < kQStages; ++s) { mbar_init(&full_q[s], 1); mbar_init(&empty_q[s], 8); }
        for (int s = 0; s < 2; ++s) { mbar_init(&full_w[s], 16); mbar_init(&acc_full[s], 1); mbar_init(&acc_free[s], 16); }
        s_err = 0;
        mbar_fence_init();
    }
    if (warp == 3) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&s_tmem)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    cluster_sync();   // the other CTA's barriers are set up
    fence_after();
    const uint32_t tmem = s_tmem;
    const int half = p.nt / 2, x_tile = half * kStep * 2;   // this CTA's tokens of a tile, bytes of one part
    Slice s;

    if (warp == 0) {
        // ---------------- activations
        if (lane == 0) {
            pdl_wait();
            pdl_trigger();
            bool ok = true;
            int st = 0;
            uint32_t use = 0;
            for (int i = 0; ok && locate(p, i, s); ++i) {
                for (int kt = 0; kt < s.nk; ++kt) {
                    if (use > 0 && !pair_wait(&done[st], (use - 1) & 1, nullptr, 0, &s_err)) { atomicExch(&s_err, 1); ok = false; break; }
                    if (rank == 0) mbar_expect_tx(&full_x[st], uint32_t(4 * x_tile));
                    const uint32_t bar = cluster_addr(&full_x[st], 0);
                    unsigned char* dst = sX + st * kXStage;
                    pair_load(dst, &map_hi, (s.k0 + kt) * kStep, s.m0 + rank * half, bar);
                    pair_load(dst + x_tile, &map_lo, (s.k0 + kt) * kStep, s.m0 + rank * half, bar);
                    if (++st == kXStages) { st = 0; ++use; }
                }
            }
            // every commit has arrived here before this CTA can leave: one that came later would arrive at a barrier of whatever runs here next
            for (int j = 0; ok && j < kXStages; ++j) {
                if (use > 0 && !pair_wait(&done[st], (use - 1) & 1, nullptr, 0, &s_err)) { atomicExch(&s_err, 1); ok = false; }
                if (++st == kXStages) { st = 0; ++use; }
            }
        }
    } else if (warp == 1) {
        // ---------------- products: the whole warp runs the loop of the first CTA, one elected lane issues
        if (rank == 0) {
            const uint32_t id = (1u << 4) | (uint32_t(p.nt >> 3) << 17) | (uint32_t(256 >> 4) << 24);   // D f32, A and B f16, M = 256
            bool ok = true;
            int st = 0, it = 0;
            uint32_t use = 0;
            for (int i = 0; ok && locate(p, i, s); ++i) {
                const int buf = i & 1;
                if (i >= 2 && !all_lanes(pair_wait(&acc_free[buf], ((i >> 1) - 1) & 1, nullptr, 0, &s_err))) { atomicExch(&s_err, 1); ok = false; }
                const uint32_t d = tmem + uint32_t(buf * kMaxTokens);
                for (int kt = 0; ok && kt < s.nk; ++kt, ++it) {
                    const int sw = it & 1;
                    if (!all_lanes(pair_wait(&full_x[st], use & 1, &full_w[sw], (it >> 1) & 1, &s_err))) { atomicExch(&s_err, 1); ok = false; break; }
                    fence_after();
                    const uint64_t x_hi = desc_kmajor(smem_u32(sX + st * kXStage)), x_lo = x_hi + uint64_t(x_tile >> 4);
                    const uint32_t w = tmem + kWCol + uint32_t(sw * 64);
                    if (elected()) {
#pragma unroll
                        for (int b = 0; b < 2; ++b) {           // 32-column block: hi parts in columns 0..15 of its stage, lo parts behind them
#pragma unroll
                            for (int pass = 0; pass < 3; ++pass)   // w_hi x_hi, w_hi x_lo, w_lo x_hi
#pragma unroll
                                for (int k16 = 0; k16 < 2; ++k16)
                                    pair_mma(d, w + uint32_t(b * 32 + (pass == 2 ? 16 : 0) + k16 * 8), (pass == 1 ? x_lo : x_hi) + uint64_t(b * 4 + k16 * 2), id,
                                             (kt > 0 || b > 0 || pass > 0 || k16 > 0) ? 1u : 0u);
                        }
                        pair_commit(&done[st]);
                        if (kt == s.nk - 1) pair_commit(&acc_full[buf]);
                    }
                    __syncwarp();
                    if (++st == kXStages) { st = 0; ++use; }
                }
                if (!ok) {   // what was issued ends before the pair parts
                    if (elected()) pair_commit(&acc_full[buf]);
                    __syncwarp();
                }
            }
        }
    } else if (warp == 2) {
        // ---------------- quantised bytes: constant, so their copies start before the kernel in front has ended
        if (lane == 0) {
            bool ok = true;
            int st = 0;
            uint32_t use = 0;
            for (int i = 0; ok && locate(p, i, s); ++i) {
                for (int kt = 0; kt < s.nk; kt += kSuper) {
                    if (use > 0 && !pair_wait(&empty_q[st], (use - 1) & 1, nullptr, 0, &s_err)) { atomicExch(&s_err, 1); ok = false; break; }
                    mbar_expect_tx(&full_q[st], uint32_t(kQStage));
                    tma_2d(sQ + st * kQStage, &map_w, (s.k0 + kt) * (128 / kSuper), s.n0, &full_q[st]);
                    if (++st == kQStages) { st = 0; ++use; }
                }
            }
        }
    } else if (warp >= 4 && warp < 12) {
        // ---------------- weights: lane = row of the warp's quadrant, the warp's half of the eight = 32-column block of the K step
        const int quad = warp & 3, blk = (warp - 4) >> 2, r = quad * 32 + lane;
        constexpr int QV = QUANT == FORGE_Q4_0 ? 1 : 2;   // 16-byte pieces per block
        const uint32_t col = tmem + (uint32_t(quad * 32) << 16) + kWCol + uint32_t(blk * 32);
        const uint32_t row7 = uint32_t(r & 7), bar_w = cluster_addr(&full_w[0], 0);
        const size_t d_row = size_t(p.t.K / 32);
        // the scales of a stage's K steps, both blocks of a step in a word; those of the next stage are requested a stage ahead, across slices and tiles
        uint32_t dcur[kSuper], dnext[kSuper];
        auto dload = [&](const Slice& a, int kt) {
            const int n = a.n0 + r;
            const uint32_t* src = reinterpret_cast<const uint32_t*>(p.t.d + size_t(n < p.t.N ? n : 0) * d_row) + a.k0 + kt;
#pragma unroll
            for (int j = 0; j < kSuper; ++j) dnext[j] = n < p.t.N && kt + j < a.nk ? __ldg(src + j) : 0u;
        };
        bool ok = true, more = locate(p, 0, s);
        int sq = 0, it = 0, sd = 0;
        uint32_t use_q = 0, use_d = 0;
        if (more) dload(s, 0);
        for (int i = 0; more; ++i) {
            Slice nxt;
            const bool have = locate(p, i + 1, nxt);
            for (int kt0 = 0; kt0 < s.nk; kt0 += kSuper) {
#pragma unroll
                for (int j = 0; j < kSuper; ++j) dcur[j] = dnext[j];
                if (kt0 + kSuper < s.nk) dload(s, kt0 + kSuper);
                else if (have) dload(nxt, 0);
                if (ok && !pair_wait(&full_q[sq], use_q & 1, nullptr, 0, &s_err)) { atomicExch(&s_err, 1); ok = false; }
                const unsigned char* stage = sQ + sq * kQStage + r * 128;
#pragma unroll
                for (int j = 0; j < kSuper; ++j) {
                    if (kt0 + j >= s.nk) break;
                    uint32_t cur[4 * QV], hi[16], lo[16];
#pragma unroll
                    for (int v = 0; v < QV; ++v) {
                        const uint4 u = *reinterpret_cast<const uint4*>(stage + ((uint32_t((j * 2 + blk) * QV + v) ^ row7) << 4));
                        cur[4 * v] = u.x; cur[4 * v + 1] = u.y; cur[4 * v + 2] = u.z; cur[4 * v + 3] = u.w;
                    }
                    dequant_block<QUANT, true>(cur, as_h2(prmt(dcur[j], 0u, blk ? 0x3232u : 0x1010u)), hi, lo);
                    // this stage was read by the products of the step before last
                    if (it >= 2) {
                        if (ok && !pair_wait(&done[sd], use_d & 1, nullptr, 0, &s_err)) { atomicExch(&s_err, 1); ok = false; }
                        if (++sd == kXStages) { sd = 0; ++use_d; }
                    }
                    fence_after();
                    const int sw = it & 1;
                    tmem_st16(col + uint32_t(sw * 64), hi);
                    tmem_st16(col + uint32_t(sw * 64 + 16), lo);
                    if (j == kSuper - 1 || kt0 + j == s.nk - 1) {   // what the stage of bytes held has been used
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&empty_q[sq]);
                    }
                    wait_st();
                    fence_before();
                    __syncwarp();
                    if (lane == 0) arrive_first(bar_w + uint32_t(sw * 8));
                    ++it;
                }
                if (++sq == kQStages) { sq = 0; ++use_q; }
            }
            more = have;
            s = nxt;
        }
    } else if (warp >= 12) {
        // ---------------- epilogue: lane = weight row, columns = tokens
        const int quad = warp & 3, e = tid & 127, group = (warp - 12) >> 2;
        unsigned char* const stage = sO + group * kOut;
        pdl_wait();
        bool ok = true;
        for (int i = 0; ok && locate(p, i, s); ++i) {
            const int buf = i & 1;
            float* const out = p.t.out + size_t(s.part) * p.t.part_stride;
            const float* const add = s.first ? p.t.resid : out;
            if (!all_lanes(pair_wait(&acc_full[buf], (i >> 1) & 1, nullptr, 0, &s_err))) { atomicExch(&s_err, 1); ok = false; }
            fence_after();
            // the slice in front of this one is in memory before this one is added to it
            if (!s.first && p.bulk && e == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
#pragma unroll 1
            for (int c0 = group * 32; c0 < p.nt && s.m0 + c0 < p.t.m; c0 += 64) {
                uint32_t v[32];
                tmem_ld32(tmem + (uint32_t(quad * 32) << 16) + uint32_t(buf * kMaxTokens + c0), v);
                wait_ld();
                if (e == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // what this buffer held has been read
                epilogue_sync(group);
                stage_chunk(v, stage, p.t.act_hi != nullptr, e);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                epilogue_sync(group);
                if (!p.bulk) copy_chunk(p.t, stage, out, add, s.m0 + c0, s.n0, e);
                else if (e == 0) {
                    if (s.n0 < p.t.N) {
                        if (p.t.act_hi) {
                            bulk_store(&map_out, s.n0 / 2, s.m0 + c0, 0, stage);
                            bulk_store(&map_out_lo, s.n0 / 2, s.m0 + c0, 0, stage + kOut / 4);
                        } else if (s.first) bulk_store(&map_out, s.n0, s.m0 + c0, s.part, stage);
                        else bulk_add(&map_out, s.n0, s.m0 + c0, s.part, stage);
                    }
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            }
            fence_before();
            __syncwarp();
            if (lane == 0) arrive_first(cluster_addr(&acc_free[buf], 0));
        }
        if (e == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    cluster_sync();   // neither CTA leaves while the other's products read its memory or arrive at its barriers
    if (warp == 3) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
    if (tid == 0 && s_err && p.t.err) atomicExch(p.t.err, 1);
}

int32_t encode(CUtensorMap* map, CUtensorMapDataType type, CUtensorMapSwizzle swizzle, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides,
               const cuuint32_t* box) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) { set_error("cuTensorMapEncodeTiled is not available from this driver"); return FORGE_ERR_UNSUPPORTED; }
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = fn(map, type, cuuint32_t(rank), const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled failed (%d)", int(r)); return FORGE_ERR_CUDA; }
    return FORGE_OK;
}
int32_t rows_map(CUtensorMap* map, CUtensorMapDataType type, const void* base, uint64_t cols, uint64_t rows, uint64_t row_bytes, uint32_t box_cols, uint32_t box_rows) {
    const cuuint64_t dims[2] = {cols, rows}, strides[1] = {row_bytes};
    const cuuint32_t box[2] = {box_cols, box_rows};
    return encode(map, type, CU_TENSOR_MAP_SWIZZLE_128B, base, 2, dims, strides, box);
}
int32_t out_map(CUtensorMap* map, CUtensorMapDataType type, const void* base, uint64_t cols, uint64_t rows, uint64_t parts, uint64_t row_bytes, uint64_t part_bytes, uint32_t box_cols) {
    const cuuint64_t dims[3] = {cols, rows, parts}, strides[2] = {row_bytes, part_bytes};
    const cuuint32_t box[3] = {box_cols, 32, 1};
    return encode(map, type, CU_TENSOR_MAP_SWIZZLE_NONE, base, 3, dims, strides, box);
}

template <int QUANT>
int32_t launch_pair(const __half* A, const __half* Alo, PairParams p, int pairs, cudaStream_t st) {
    CUtensorMap mh, ml, mw, mo{}, mol{};
    const Tc5Params& t = p.t;
    FORGE_TRY(rows_map(&mh, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, A, t.K, t.m, uint64_t(t.K) * 2, kStep, uint32_t(p.nt / 2)));
    FORGE_TRY(rows_map(&ml, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, Alo, t.K, t.m, uint64_t(t.K) * 2, kStep, uint32_t(p.nt / 2)));
    const uint64_t row_bytes = QUANT == FORGE_Q4_0 ? uint64_t(t.K) / 2 : uint64_t(t.K);
    FORGE_TRY(rows_map(&mw, CU_TENSOR_MAP_DATA_TYPE_UINT8, t.qs, row_bytes, t.N, row_bytes, 128, 128));
    // tensor copies store rows of multiples of 16 bytes at 16-byte addresses; other outputs are stored by the epilogue's threads
    auto fits = [](const void* a, size_t row, size_t part) { return !((reinterpret_cast<uintptr_t>(a) | row | part) & 15); };
    if (t.act_hi) {
        // (an intermediate size is whole blocks of 32, the rows are the library's own)
        if (!t.act_lo || !fits(t.act_hi, size_t(t.N), 0) || !fits(t.act_lo, size_t(t.N), 0)) { set_error("tcgen05 gemm: the SiLU epilogue needs 16-byte rows"); return FORGE_ERR_SHAPE; }
        p.bulk = 1;
        FORGE_TRY(out_map(&mo, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, t.act_hi, t.N / 2, t.m, 1, size_t(t.N), size_t(t.N) * t.m, 64));
        FORGE_TRY(out_map(&mol, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, t.act_lo, t.N / 2, t.m, 1, size_t(t.N), size_t(t.N) * t.m, 64));
    } else {
        const size_t part = p.parts > 1 ? t.part_stride * 4 : size_t(t.N) * t.m * 4;
        p.bulk = !t.resid && fits(t.out, size_t(t.N) * 4, part);
        if (p.bulk) FORGE_TRY(out_map(&mo, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, t.out, t.N, t.m, p.parts, size_t(t.N) * 4, part, 128));
    }
    FORGE_CUDA(cudaFuncSetAttribute(gemm_pair_kernel<QUANT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem));
    FORGE_CUDA(launch_pdl(gemm_pair_kernel<QUANT>, dim3(2 * pairs), dim3(kPairThreads), kPairSmem, st, mh, ml, mw, mo, mol, p));
    FORGE_LAUNCH_CHECK();
    return FORGE_OK;
}

}  // namespace

// Tokens per tile and partial outputs of the least cost.  Measured over 28 shapes (K 896 to 11008, 64 to 2501 tokens, tiles of 64 to 192): a launch takes about
// 6 us, and in each round of tiles over the pairs a K step max(0.44, 0.12 + 0.0029 NT) us (0.44 is what the weights' two stages allow, 0.61 would be
// the tensor pipe's time at 192) and a slice 1.2 us, to within a tenth.  A further partial output costs its reader the bytes, here at 5 TB/s.
PairPlan gemm_pair_plan(const QWeight& w, int m, int ksplit, int parts_only, int sms) {
    PairPlan best;
    const int pairs = std::max(1, sms / 2), n_tiles = (w.N + 255) / 256;
    double least = 1e30;
    for (int parts = 1; parts <= ksplit; ++parts) {
        if (ksplit % parts || (parts_only && parts != parts_only)) continue;
        for (int nt = 32; nt <= kMaxTokens && (nt == 32 || nt - 32 < m); nt += 32) {
            const long items = long(n_tiles) * ((m + nt - 1) / nt) * parts, rounds = (items + pairs - 1) / pairs;
            const double step = std::max(0.44, 0.12 + 0.0029 * nt), slices = double(rounds) * (ksplit / parts);
            const double cost = 6.0 + slices * (double(w.K / kStep) / ksplit * step + 1.2) + (parts - 1) * 4e-6 * w.N * m / 5.0;
            if (cost < least) { least = cost; best.nt = nt; best.parts = parts; best.pairs = int(std::min<long>(items, pairs)); best.cost = cost; }
        }
    }
    return best;
}

int32_t gemm_pair(float* out, const __half* A, const __half* Alo, const QWeight& w, int m, const float* resid, int* err, cudaStream_t st, const PairPlan& plan, int ksplit,
                  size_t part_stride, __half* act_hi, __half* act_lo) {
    PairParams p{};
    p.t = Tc5Params{out, resid, w.qs, w.d, nullptr, m, w.N, w.K, err, ksplit, part_stride, act_hi, act_lo};
    p.nt = plan.nt; p.n_tiles = (w.N + 255) / 256; p.m_tiles = (m + plan.nt - 1) / plan.nt; p.parts = plan.parts; p.slices = ksplit / plan.parts;
    return w.quant == FORGE_Q8_0 ? launch_pair<FORGE_Q8_0>(A, Alo, p, plan.pairs, st) : launch_pair<FORGE_Q4_0>(A, Alo, p, plan.pairs, st);
}

}  // namespace forge
