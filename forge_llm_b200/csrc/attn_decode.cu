// Single-query decode attention over the paged fp16 KV cache (replaces attention_flash,
// crates/forgellm-codegen-cpu/src/emit.rs:657-715; GQA mapping kv_head = h / (nq/nkv), :660-666).
//
// What bounds it: for one sequence the chain launch -> query -> page -> merge, for many sequences the bytes of K and V.  The context is split
// over CTAs; a producer lane pulls the CTA's pages - 64 rows of one KV head, K and V - into a ring of shared-memory stages with 3-D tiled TMA copies
// (SWIZZLE_128B, boxes of 64 dimensions; the tensor map spans this GPU's own pool), before the dependency wait: every cached row but the
// newest was written by earlier steps.
//
// Four consumer warps take sixteen keys of a page each, as mma.sync products: up to eight query heads of the group are rows 0..7 of the A tile as fp16 hi
// parts and rows 8..15 as lo parts, so that one product serves both halves of the query and a thread adds them from its own registers; the weights
// enter their product with the values the same way.  A power of two in front of either split keeps all bits of it in fp16's range, no
// product is carried further than its neighbour, and f32 sums take over: against 64 bits the result is nearer than f32 multiply-adds bring it (0.9 of their
// error for scores around 1, 0.65 around 10; 8000 keys of one weight 1.6e-7, 3.8e-7 with sums carried through the tensor core).
// A page costs a warp about forty tensor instructions at head_dim 64 whatever the group; with scores and sums
// formed by fused multiply-adds (four heads per pass over the page) one page took 1.7 us.
// The splits of a (sequence, KV head) are a cluster and merge through distributed shared memory; more than eight (few KV heads over many
// pages) leave partials in global memory, which the last CTA to finish merges (atomic ticket).  Every wait is bounded.
#include <algorithm>
#include <cmath>
#include <mutex>

#include "attn_decode.cuh"
#include "mma.cuh"
#include "tc5.cuh"

namespace forge {

namespace {

using namespace decode;
using tc5::cluster_addr;
using tc5::cluster_sync;

constexpr int kHeads = 8;         // query heads of a KV head in one pass over the keys
constexpr int kClusterSplits = 8; // context splits in a cluster
constexpr float kUp = 32768.f;    // of a weight in front of its product: the lo part of 2^-14 of the largest one is still a normal fp16 number

__device__ __forceinline__ float exp2_rel(float x, float m) { return x == -INFINITY ? 0.f : exp2f(x - m); }   // 0 for an empty part, never NaN

__device__ __forceinline__ void mma16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// two values as packed fp16 hi parts and lo parts
__device__ __forceinline__ void split_h2(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(x, y);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(x - f.x, y - f.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}
__device__ __forceinline__ float remote_f32(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}

// barrier of the consumers that also tells whether any of them says so
__device__ __forceinline__ bool csync_or(bool x) {
    uint32_t any;
    asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbar.red.or.pred q, 1, %2, p;\nselp.u32 %0, 1, 0, q;\n}" : "=r"(any) : "r"(uint32_t(x)), "n"(kThreads) : "memory");
    return any != 0;
}

// One head's sums over the CTA's pages by f32 multiply-adds, a warp per head, from global memory.  Taken where a sum came out as NaN: the two parts of a
// query or a weight meet an infinite key or value with a zero or with the other sign, where their sum would have given an infinity; or a page did not
// come within the wait's limit.
template <int HD, bool SW>
__device__ __noinline__ void plain_head(const AttnDecodeArgs& a, float scale, int b, int kvh, int head, int split, int n_ctx, int t_first, size_t row0, float* sums, float* ml) {
    constexpr int D = HD / 32;
    const int lane = threadIdx.x & 31, kvd = a.nkv * HD;
    const int32_t* pt = a.page_table ? a.page_table + size_t(b) * a.pages_per_seq : nullptr;
    float q[D], acc[D], m = -INFINITY, l = 0.f;
#pragma unroll
    for (int i = 0; i < D; ++i) { q[i] = a.q[(size_t(b) * a.nq + head) * HD + i * 32 + lane] * scale; acc[i] = 0.f; }
    for (int lp = split; lp * FORGE_KV_PAGE < n_ctx; lp += a.splits) {
        const size_t page = row0 + size_t(pt ? pt[lp] : lp) * FORGE_KV_PAGE;
        for (int r = SW ? max(0, t_first - lp * FORGE_KV_PAGE) : 0; r < min(FORGE_KV_PAGE, n_ctx - lp * FORGE_KV_PAGE); ++r) {
            const size_t at = (page + r) * kvd + size_t(kvh) * HD + lane;
            float s = 0.f;
#pragma unroll
            for (int i = 0; i < D; ++i) s = fmaf(q[i], __half2float(a.k_pool[at + i * 32]), s);
#pragma unroll
            for (int x = 16; x > 0; x >>= 1) s += __shfl_xor_sync(0xffffffffu, s, x);
            const float mn = fmaxf(m, s);
            if (mn == -INFINITY) continue;
            const float es = exp2_rel(m, mn), w = exp2_rel(s, mn);
            m = mn;
            l = l * es + w;
#pragma unroll
            for (int i = 0; i < D; ++i) acc[i] = acc[i] * es + w * __half2float(a.v_pool[at + i * 32]);
        }
    }
#pragma unroll
    for (int i = 0; i < D; ++i) sums[i * 32 + lane] = acc[i];
    if (lane == 0) { ml[0] = m; ml[1] = l; }
}

// SW: sliding-window instantiation (the full-attention one carries no window tests); CL: the splits are a cluster
template <int HD, bool SW, bool CL>
__global__ void __launch_bounds__(kBlock, HD == 64 ? 3 : 2) attn_decode_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const __grid_constant__ DecParams p) {
    constexpr int BOXES = (HD + 63) / 64;                 // boxes of 64 dimensions (the second one of 96-wide heads is half zeros)
    constexpr int BOX_BYTES = FORGE_KV_PAGE * 128;
    constexpr int PAGE_BYTES = BOXES * BOX_BYTES;
    constexpr int KS = HD / 16, NV = HD / 8;
    extern __shared__ __align__(1024) unsigned char ring_raw[];   // [stages][K page | V page], then [warp][head][HD] sums
    unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(ring_raw) + 1023) & ~uintptr_t(1023));
    float* s_acc = reinterpret_cast<float*>(ring + size_t(p.stages) * 2 * PAGE_BYTES);
    __shared__ uint64_t full_bar[kStages], empty_bar[kStages];
    __shared__ float s_ml[4][kHeads][2], s_cml[kMaxGroup][2];
    __shared__ int s_last;
    const AttnDecodeArgs& a = p.a;
    pdl_trigger();
    const int split = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lr = lane >> 2, lc = (lane & 3) * 2;
    const int G = a.nq / a.nkv, kvd = a.nkv * HD;
    float* s_sum = G > kHeads ? s_acc + 4 * kHeads * HD : s_acc;   // [head][HD] sums of the CTA (of one pass: over warp 0's own values)
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], kThreads / 32); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // Split s owns the logical pages s, s + splits, ...: which pages a CTA reads does not depend on the context
    // length.  The length, the page table and every cached row but the newest were written before the kernel in front
    // of this one started, so they are read without waiting for it.
    const int32_t* pt = a.page_table ? a.page_table + size_t(b) * a.pages_per_seq : nullptr;
    const int n_ctx = a.seq_len ? a.seq_len[b] + 1 : a.seq_len_host;
    const int n_pages = (n_ctx + FORGE_KV_PAGE - 1) / FORGE_KV_PAGE;
    // without a cluster, CTAs beyond the context's pages have no part in it: a launch's splits are those of the longest context that it may meet
    const int splits = CL ? a.splits : min(a.splits, n_pages);
    if (!CL && split >= splits) return;
    const int t_first = (SW && n_ctx > a.window) ? n_ctx - a.window : 0;  // sliding window: first position seen
    const size_t seq_base = a.page_table ? 0 : size_t(b) * a.max_ctx;  // contiguous: [batch][max_ctx][kvd]

    if (warp == kThreads / 32) {
        // ---- producer: the CTA's pages, once per pass over the query heads, as ring space frees up
        if (lane == 0) {
            int i = 0;
            for (int g0 = 0; g0 < G; g0 += kHeads)
                for (int lp = split; lp < n_pages; lp += a.splits) {
                    if (SW && (lp + 1) * FORGE_KV_PAGE <= t_first) continue;
                    const int st = i % p.stages, use = i / p.stages;
                    if (use > 0 && !mbar_wait(&empty_bar[st], (use - 1) & 1)) { if (a.err) atomicExch(a.err, 1); return; }
                    const int row = a.row_base + int(seq_base) + (pt ? pt[lp] : lp) * FORGE_KV_PAGE;
                    unsigned char* dst = ring + size_t(st) * 2 * PAGE_BYTES;
                    mbar_expect_tx(&full_bar[st], 2 * PAGE_BYTES);
#pragma unroll
                    for (int x = 0; x < BOXES; ++x) {
                        tma_page(dst + x * BOX_BYTES, &map_k, x * 64, kvh, row, &full_bar[st]);
                        tma_page(dst + PAGE_BYTES + x * BOX_BYTES, &map_v, x * 64, kvh, row, &full_bar[st]);
                    }
                    ++i;
                }
        }
        return;
    }
    pdl_wait();  // q and the newest cache row come from the kernel before this one
    int pi = 0;  // pages consumed so far (ring position)
    const uint32_t sw = uint32_t(lane & 7);   // swizzle of the row this lane addresses (rows are taken eight at a time)

    for (int g0 = 0; g0 < G; g0 += kHeads) {
        const int gc = min(kHeads, G - g0);
        // A fragments of the queries: row lr = hi part of head lr, row lr + 8 = lo part.  A power of two takes the head's largest value to [2^14, 2^15), so that
        // the parts hold what they can of any size of query and none overflows; `unit` takes a score back, and to powers of two
        uint32_t qf[KS][4];
        float unit, unit_lo;
        {
            float q[KS][4], big = 0.f;
#pragma unroll
            for (int k = 0; k < KS; ++k) {
                float2 x = make_float2(0.f, 0.f), y = x;
                if (lr < gc) {
                    const float* qp = a.q + (size_t(b) * a.nq + kvh * G + g0 + lr) * HD + k * 16 + lc;
                    x = *reinterpret_cast<const float2*>(qp);
                    y = *reinterpret_cast<const float2*>(qp + 8);
                }
                q[k][0] = x.x; q[k][1] = x.y; q[k][2] = y.x; q[k][3] = y.y;
                big = fmaxf(fmaxf(big, fmaxf(fabsf(x.x), fabsf(x.y))), fmaxf(fabsf(y.x), fabsf(y.y)));
            }
            big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, 1));
            big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, 2));
            const int up = min(268 - (__float_as_int(big) >> 23), 253);   // exponent fields: 2^(up - 127) is the factor, 2^(127 - up) takes it back
            const float f = __int_as_float(up << 23);
            unit = __int_as_float((254 - up) << 23) * p.scale;
            unit_lo = __int_as_float((254 - up) << 23) * p.scale_lo;
#pragma unroll
            for (int k = 0; k < KS; ++k) {
                split_h2(q[k][0] * f, q[k][1] * f, qf[k][0], qf[k][1]);
                split_h2(q[k][2] * f, q[k][3] * f, qf[k][2], qf[k][3]);
            }
        }
        // sums relative to 2^m: of the values (times kUp), of the weights
        float o[NV][2], m = -INFINITY, l = 0.f;
#pragma unroll
        for (int v = 0; v < NV; ++v) o[v][0] = o[v][1] = 0.f;
        for (int lp = split; lp < n_pages; lp += a.splits) {
            if (SW && (lp + 1) * FORGE_KV_PAGE <= t_first) continue;  // the whole page lies before the window
            const int t0 = lp * FORGE_KV_PAGE + warp * 16;            // the warp's sixteen keys
            const int st = pi % p.stages;
            if (!mbar_wait(&full_bar[st], (pi / p.stages) & 1)) {   // a session's call fails; an operator call has no such word, and its sums are formed again
                if (a.err) atomicExch(a.err, 1);
                l = NAN;
            }
            unsigned char* const ks = ring + size_t(st) * 2 * PAGE_BYTES + warp * 16 * 128;
            if (t0 < n_ctx && (!SW || t0 + 16 > t_first)) {
                if (n_ctx - 1 - t0 < 16) {
                    // the newest row was being written by the kernel in front while the page was copied: it is taken from global memory
                    const int r = n_ctx - 1 - t0;
                    if (lane < HD / 4) {
                        const int c = lane % (HD / 8), which = lane / (HD / 8);
                        const __half* src = (which ? a.v_pool : a.k_pool) + (seq_base + size_t(pt ? pt[lp] : lp) * FORGE_KV_PAGE + warp * 16 + r) * kvd + size_t(kvh) * HD + c * 8;
                        *reinterpret_cast<uint4*>(ks + which * PAGE_BYTES + (c >> 3) * BOX_BYTES + r * 128 + (((c & 7) ^ (r & 7)) << 4)) = __ldcg(reinterpret_cast<const uint4*>(src));
                    }
                    __syncwarp();
                }
                if (n_ctx - t0 < 16 || (SW && t0 < t_first)) {
                    // a weight of zero must not meet what lies in rows that are not seen (another sequence's, or nothing yet)
                    for (int i = lane; i < 16 * BOXES * 8; i += 32) {
                        const int r = i & 15, c = i >> 4;
                        if (t0 + r >= n_ctx || (SW && t0 + r < t_first)) *reinterpret_cast<uint4*>(ks + PAGE_BYTES + (c >> 3) * BOX_BYTES + r * 128 + ((c & 7) << 4)) = make_uint4(0, 0, 0, 0);
                    }
                    __syncwarp();
                }
                const uint32_t kb = smem_u32(ks), vb = kb + PAGE_BYTES;
                const uint32_t krow = kb + uint32_t((lane & 7) + ((lane >> 4) << 3)) * 128, vrow = vb + uint32_t(lane & 15) * 128;
                // Two products in a row, then sums in f32 that keep what they round away (in front of which it stands with the lo parts): the additions of eight
                // score terms in f32 alone were half of the result's error, and a longer chain of products rounds toward zero once per step
                float s[2][2][2] = {};   // [key tile][key][hi part, rest]
#pragma unroll
                for (int k0 = 0; k0 < KS; k0 += 2) {
                    float d[2][4] = {};
#pragma unroll
                    for (int k = k0; k < k0 + 2; ++k) {
                        uint32_t f[4];
                        const uint32_t c = uint32_t(2 * k + ((lane >> 3) & 1));   // 16-byte piece of the row
                        ldsm4(f, krow + (c >> 3) * BOX_BYTES + (((c & 7) ^ sw) << 4));
                        mma16(d[0], qf[k], f[0], f[1]);
                        mma16(d[1], qf[k], f[2], f[3]);
                    }
#pragma unroll
                    for (int t = 0; t < 2; ++t)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            if (k0 == 0) { s[t][e][0] = d[t][e]; s[t][e][1] = d[t][e + 2]; continue; }
                            const float x = s[t][e][0], y = d[t][e], sum = x + y, z = sum - x;
                            s[t][e][0] = sum;
                            s[t][e][1] += ((x - (sum - z)) + (y - z)) + d[t][e + 2];
                        }
                }
                float sc[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int key = t0 + (j >> 1) * 8 + lc + (j & 1);
                    sc[j] = key < n_ctx && (!SW || key >= t_first) ? s[j >> 1][j & 1][0] : -INFINITY;
                }
                float mn = fmaxf(fmaxf(sc[0], sc[1]), fmaxf(sc[2], sc[3]));
                mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 1));
                mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 2));
                mn = fmaxf(mn * unit, m);
                const float at = mn == -INFINITY ? 0.f : mn, es = exp2f(m - at);   // a tile holds a visible key, but its score may be -inf
                float pr[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float hi = s[j >> 1][j & 1][0], rest = s[j >> 1][j & 1][1];
                    const float x = fmaf(rest, unit, fmaf(hi, unit_lo, fmaf(hi, unit, -at)));
                    pr[j] = sc[j] == -INFINITY ? 0.f : exp2f(x);
                }
                m = mn;
                l = l * es + ((pr[0] + pr[1]) + (pr[2] + pr[3]));
                uint32_t pf[4];
                split_h2(pr[0] * kUp, pr[1] * kUp, pf[0], pf[1]);
                split_h2(pr[2] * kUp, pr[3] * kUp, pf[2], pf[3]);
#pragma unroll
                for (int v = 0; v < NV; v += 2) {
                    uint32_t f[4];
                    const uint32_t c = uint32_t(v + (lane >> 4));
                    ldsm4t(f, vrow + (c >> 3) * BOX_BYTES + (((c & 7) ^ sw) << 4));
                    float d0[4] = {0.f, 0.f, 0.f, 0.f}, d1[4] = {0.f, 0.f, 0.f, 0.f};
                    mma16(d0, pf, f[0], f[1]);
                    mma16(d1, pf, f[2], f[3]);
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        o[v][e] = fmaf(o[v][e], es, d0[e] + d0[e + 2]);
                        o[v + 1][e] = fmaf(o[v + 1][e], es, d1[e] + d1[e + 2]);
                    }
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // this warp may have written a row of the page
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty_bar[st]);
            ++pi;
        }
        // ---- the warps' parts become the CTA's
        l += __shfl_xor_sync(0xffffffffu, l, 1);
        l += __shfl_xor_sync(0xffffffffu, l, 2);
        if (lc == 0) { s_ml[warp][lr][0] = m; s_ml[warp][lr][1] = l; }
#pragma unroll
        for (int v = 0; v < NV; ++v)
            *reinterpret_cast<float2*>(s_acc + (warp * kHeads + lr) * HD + v * 8 + lc) = make_float2(o[v][0] * (1.f / kUp), o[v][1] * (1.f / kUp));
        csync();
        auto put = [&](int idx, float M, float A, float L) {
            const int g = idx / HD;
            if (splits == 1) {
                store_out(a, (size_t(b) * a.nq + kvh * G + g0) * HD + idx, A * (1.0f / L));
            } else if (CL) {
                s_sum[g0 * HD + idx] = A;
                if (idx % HD == 0) { s_cml[g0 + g][0] = M; s_cml[g0 + g][1] = L; }
            } else {
                float* w = a.ws + ((size_t(b) * a.nq + kvh * G + g0 + g) * a.splits + split) * (HD + 2);
                w[2 + idx % HD] = A;
                if (idx % HD == 0) { w[0] = M; w[1] = L; }
            }
        };
        bool nan = false;
        for (int idx = threadIdx.x; idx < gc * HD; idx += kThreads) {
            const int g = idx / HD;
            float M = -INFINITY, A = 0.f, L = 0.f;
#pragma unroll
            for (int w = 0; w < 4; ++w) M = fmaxf(M, s_ml[w][g][0]);
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                const float f = exp2_rel(s_ml[w][g][0], M);
                A += s_acc[w * kHeads * HD + idx] * f;
                L += s_ml[w][g][1] * f;
            }
            nan |= A != A || L != L;
            put(idx, M, A, L);
        }
        if (csync_or(nan)) {
            for (int g = warp; g < gc; g += kThreads / 32)
                plain_head<HD, SW>(a, p.scale, b, kvh, kvh * G + g0 + g, split, n_ctx, t_first, seq_base, s_acc + g * HD, s_ml[0][g]);
            csync();
            for (int idx = threadIdx.x; idx < gc * HD; idx += kThreads) put(idx, s_ml[0][idx / HD][0], s_acc[idx], s_ml[0][idx / HD][1]);
            csync();
        }
    }
    if (CL && splits > 1) {
        // ---- the CTAs' parts become the result, each CTA finishing a share of it.  Only here, behind the last pass: until then the producer lane may be
        // waiting for ring space, and a cluster waits for every thread that has not left
        cluster_sync();
        const int items = G * HD, share = (items + splits - 1) / splits;
        for (int idx = split * share + threadIdx.x; idx < min(items, (split + 1) * share); idx += kThreads) {
            const int g = idx / HD;
            float pm[kClusterSplits], pl[kClusterSplits], px[kClusterSplits], M = -INFINITY, A = 0.f, L = 0.f;
#pragma unroll
            for (int s = 0; s < kClusterSplits; ++s) {
                const bool on = s < splits;
                pm[s] = on ? remote_f32(cluster_addr(&s_cml[g][0], s)) : -INFINITY;
                pl[s] = on ? remote_f32(cluster_addr(&s_cml[g][1], s)) : 0.f;
                px[s] = on ? remote_f32(cluster_addr(s_sum + idx, s)) : 0.f;
            }
#pragma unroll
            for (int s = 0; s < kClusterSplits; ++s) M = fmaxf(M, pm[s]);
#pragma unroll
            for (int s = 0; s < kClusterSplits; ++s) {
                const float f = exp2_rel(pm[s], M);
                A += px[s] * f;
                L += pl[s] * f;
            }
            store_out(a, (size_t(b) * a.nq + size_t(kvh) * G) * HD + idx, A * (1.0f / L));
        }
        cluster_sync();   // nobody leaves while its sums are read
    }
    if (CL || splits == 1) return;

    // ---- last CTA of this (batch, kv head) merges the splits
    __threadfence();
    csync();
    if (threadIdx.x == 0) {
        int old = atomicAdd(a.counters + b * a.nkv + kvh, 1);
        s_last = (old == splits - 1);
        if (s_last) a.counters[b * a.nkv + kvh] = 0;  // ready for the next launch
    }
    csync();
    if (!s_last) return;
    __threadfence();
    // One round trip: a thread asks for its two columns of all splits, then the warps turn the splits' (max, sum) pairs into weights (lane = split)
    float (*s_fw)[kMaxGroup] = reinterpret_cast<float (*)[kMaxGroup]>(s_acc);   // [split][head]: over the warps' sums, which are no longer needed
    const float* ws_kvh = a.ws + (size_t(b) * a.nq + size_t(kvh) * G) * a.splits * (HD + 2);
    for (int i0 = 0; i0 < G * HD / 2; i0 += kThreads) {
        const int idx = i0 + threadIdx.x;
        const bool on = idx < G * HD / 2;
        const int g = on ? idx / (HD / 2) : 0, d2 = on ? idx % (HD / 2) : 0;
        const float* w0 = ws_kvh + size_t(g) * a.splits * (HD + 2) + 2 + 2 * d2;
        float2 pa[kMaxSplits];
#pragma unroll
        for (int s = 0; s < kMaxSplits; ++s)
            pa[s] = (on && s < splits) ? __ldcg(reinterpret_cast<const float2*>(w0 + size_t(s) * (HD + 2))) : make_float2(0.f, 0.f);
        if (i0 == 0) {
            for (int g2 = warp; g2 < G; g2 += kThreads / 32) {
                const float* w = ws_kvh + (size_t(g2) * a.splits + lane) * (HD + 2);
                const float m = lane < splits ? __ldcg(w) : -INFINITY;
                const float l = lane < splits ? __ldcg(w + 1) : 0.f;
                float M = m;
#pragma unroll
                for (int x = 16; x > 0; x >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, x));
                const float wt = exp2_rel(m, M);
                float L = l * wt;
#pragma unroll
                for (int x = 16; x > 0; x >>= 1) L += __shfl_xor_sync(0xffffffffu, L, x);
                s_fw[lane][g2] = wt * (1.0f / L);
            }
            csync();
        }
        float2 A = make_float2(0.f, 0.f);
#pragma unroll
        for (int s = 0; s < kMaxSplits; ++s) {
            const float wt = s < splits ? s_fw[s][g] : 0.f;
            A.x += pa[s].x * wt;
            A.y += pa[s].y * wt;
        }
        if (on) store_out2(a, (size_t(b) * a.nq + size_t(kvh) * G + g) * HD + 2 * d2, A);
    }
}

}  // namespace

// Context splits for `groups` = batch * kv_heads independent (sequence, KV head) pairs over `pages` pages, by what a launch took (cold caches, us): a CTA
// 2.4 + 0.62 a page at 64 dimensions, 3.2 + 0.78 at 96 and 128, its pages longer where an SM's CTAs share it, in rounds over the resident CTAs; the meeting of
// a cluster 1.8 (2.2), that through global memory 2.2 + 0.063 a split (3.3 + 0.094).  Beyond a cluster's eight only sixteen and 32: in between, CTAs of
// unequal lengths were slower than the better of the two.  So 32 heads over 8 KV heads of 64 take 7.0 us over 25 pages with eight splits (sixteen
// 6.6), 9.3 over 64 pages (sixteen 8.0, 32 7.8), 14.2 over 128 (10.3, 9.7); sixteen sequences of 32 KV heads take one.
int attn_decode_splits(int pages, int groups, int sms, int hd, int window) {
    if (window > 0) pages = std::min(pages, (window + FORGE_KV_PAGE - 2) / FORGE_KV_PAGE + 1);   // those that a window can touch
    const bool wide = hd > 64;
    const long slots = long(sms) * (wide ? 2 : 3);
    const double fixed = wide ? 3.2 : 2.4, page = wide ? 0.78 : 0.62;
    int best = 1;
    double best_cost = 1e30;
    for (int s = 1; s <= std::min(pages, kMaxSplits); s = s < kClusterSplits ? s + 1 : 2 * s) {
        const long ctas = long(groups) * s, rounds = (ctas + slots - 1) / slots;
        const double load = std::max(1.0, 0.85 * double(std::min(ctas, slots)) / sms);
        const double meeting = s == 1 ? 0.0 : s <= kClusterSplits ? (wide ? 2.2 : 1.8) : wide ? 3.3 + 0.094 * s : 2.2 + 0.063 * s;
        const double cost = double(rounds) * (fixed + page * load * ((pages + s - 1) / s)) + meeting;
        if (cost < best_cost + 1e-9) { best_cost = cost; best = s; }   // of equals the larger: more of its CTAs have a page less
    }
    return best;
}

// workspace of the splits that are merged through global memory (0: none is needed)
size_t attn_decode_ws_floats(int batch, int nq, int hd, int splits) { return splits > kClusterSplits ? size_t(batch) * nq * splits * (hd + 2) : 0; }

template <int HD, bool SW>
int32_t launch_decode(const CUtensorMap& mk, const CUtensorMap& mv, const DecParams& p, dim3 grid, cudaStream_t st) {
    constexpr int kPage = (HD + 63) / 64 * FORGE_KV_PAGE * 128, kSums = (4 * kHeads + kMaxGroup) * HD * 4;
    const size_t smem = size_t(p.stages) * 2 * kPage + (p.a.nq > kHeads * p.a.nkv ? kSums : 4 * kHeads * HD * 4) + 1024;
    auto kern = p.a.splits <= kClusterSplits ? attn_decode_kernel<HD, SW, true> : attn_decode_kernel<HD, SW, false>;
    FORGE_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kStages * 2 * kPage + kSums + 1024));
    FORGE_CUDA(launch_pdl_cluster(kern, grid, dim3(kBlock), p.a.splits <= kClusterSplits ? p.a.splits : 1, smem, st, mk, mv, p));
    FORGE_LAUNCH_CHECK();
    return FORGE_OK;
}

int32_t attn_decode(const AttnDecodeArgs& a, cudaStream_t st) {
    if (a.f32) return attn_decode_f32(a, st);
    if (a.nq % a.nkv) { set_error("attention: num_heads %d not a multiple of num_kv_heads %d", a.nq, a.nkv); return FORGE_ERR_SHAPE; }
    if (a.splits < 1 || (a.splits > kClusterSplits && (!a.ws || !a.counters))) { set_error("attention: split workspace missing"); return FORGE_ERR_INVALID_ARG; }
    if (a.nq / a.nkv > kMaxGroup) { set_error("attention: at most %d query heads per KV head", kMaxGroup); return FORGE_ERR_SHAPE; }
    if (a.splits > kMaxSplits) { set_error("attention: at most %d context splits", kMaxSplits); return FORGE_ERR_INVALID_ARG; }
    if (a.hd != 64 && a.hd != 96 && a.hd != 128) { set_error("attention: head_dim %d unsupported (64, 96, 128)", a.hd); return FORGE_ERR_SHAPE; }
    // tensor maps of the two pools: the caller's (a paged cache keeps them), or made here for a contiguous cache
    CUtensorMap mk, mv;
    if (a.map_k && a.map_v) {
        mk = *static_cast<const CUtensorMap*>(a.map_k);
        mv = *static_cast<const CUtensorMap*>(a.map_v);
    } else {
        const size_t rows = a.page_table ? 0 : size_t(a.batch) * a.max_ctx;
        if (!rows) { set_error("attention: a paged cache needs its tensor maps"); return FORGE_ERR_INVALID_ARG; }
        FORGE_TRY(make_kv_map(&mk, a.k_pool, a.hd, a.nkv, rows));
        FORGE_TRY(make_kv_map(&mv, a.v_pool, a.hd, a.nkv, rows));
    }
    // ring depth: the pages a CTA will see, at most what lets three CTAs (two with wider heads) share an SM: 64-wide heads four stages of 16 KB and 8 KB of
    // sums (with the second pass's 4 KB more two CTAs)
    const int ctx = a.seq_len ? a.max_ctx : a.seq_len_host;
    const int pages_per_cta = ((ctx + FORGE_KV_PAGE - 1) / FORGE_KV_PAGE + a.splits - 1) / a.splits;
    const double scale = 1.4426950408889634 / std::sqrt(double(a.hd));   // log2 e / sqrt(head_dim)
    DecParams p{a, float(scale), std::max(1, std::min(pages_per_cta, a.hd == 64 ? 4 : 2)), float(scale - double(float(scale)))};
    dim3 grid(a.splits, a.nkv, a.batch);
    const bool sw = a.window > 0;
    if (a.hd == 64) return sw ? launch_decode<64, true>(mk, mv, p, grid, st) : launch_decode<64, false>(mk, mv, p, grid, st);
    if (a.hd == 96) return sw ? launch_decode<96, true>(mk, mv, p, grid, st) : launch_decode<96, false>(mk, mv, p, grid, st);
    return sw ? launch_decode<128, true>(mk, mv, p, grid, st) : launch_decode<128, false>(mk, mv, p, grid, st);
}

}  // namespace forge

// ------------------------------------------------------------------------------------------------
// forge_attention_flash_static: the same single-query attention for callers that must not allocate.
//
// Some hosts cannot let a library call cudaMalloc: a serving process whose own pool has already claimed
// the whole device (an allocation here would fail or fragment it), or a loop with a latency budget that
// cannot absorb the device-wide synchronisation an allocation or a free may imply.  forge_attention_flash
// gets its split-KV workspace from the stream-ordered allocator on every call; this variant keeps that
// workspace in a fixed array inside the library image instead (about 1.1 MB on every GPU that loads the
// library, until the process exits) and therefore accepts only shapes that fit it.
namespace {

constexpr int kStaticMaxHeads = 64;    // query heads (and KV heads)
constexpr int kStaticMaxSplits = 32;   // context splits, the same rule as forge_attention_flash
constexpr int kStaticMaxHeadDim = 128;
constexpr int kStaticMaxSeq = 1 << 20;

struct StaticScratch {
    float ws[size_t(kStaticMaxHeads) * kStaticMaxSplits * (kStaticMaxHeadDim + 2)];  // partial (m, l, acc) per head and split
    int counters[kStaticMaxHeads];                                                  // arrival tickets per KV head
};

// In host code this name is only a handle for the runtime; the device address comes from
// cudaGetSymbolAddress below and is what the kernel receives.
static __device__ __align__(256) unsigned char g_static_scratch[sizeof(StaticScratch)];

constexpr int kMaxDevices = 64;
std::mutex g_static_mutex;
StaticScratch* g_static_ptr[kMaxDevices] = {};

// Device address of the scratch on the current device; resolved once per device.
int32_t static_scratch(StaticScratch** out) {
    int dev = -1;
    FORGE_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) { forge::set_error("device index %d beyond %d", dev, kMaxDevices); return FORGE_ERR_UNSUPPORTED; }
    std::lock_guard<std::mutex> lock(g_static_mutex);
    if (!g_static_ptr[dev]) {
        void* p = nullptr;
        FORGE_CUDA(cudaGetSymbolAddress(&p, g_static_scratch));
        g_static_ptr[dev] = static_cast<StaticScratch*>(p);
    }
    *out = g_static_ptr[dev];
    return FORGE_OK;
}

}  // namespace

extern "C" int32_t forge_attention_flash_static(float* out, const float* q, const uint16_t* k_cache, const uint16_t* v_cache,
                                                int32_t seq_len, int32_t num_heads, int32_t num_kv_heads, int32_t head_dim,
                                                void* stream) {
    using namespace forge;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        set_error("no CUDA device: this backend has no CPU fallback");
        return FORGE_ERR_CUDA;
    }
    if (!out || !q || !k_cache || !v_cache || seq_len <= 0 || num_heads <= 0 || num_kv_heads <= 0) {
        set_error("bad argument to forge_attention_flash_static");
        return FORGE_ERR_INVALID_ARG;
    }
    if (num_heads > kStaticMaxHeads || num_kv_heads > kStaticMaxHeads || head_dim > kStaticMaxHeadDim || seq_len > kStaticMaxSeq) {
        set_error("forge_attention_flash_static: shape (%d heads, %d kv heads, head_dim %d, %d positions) exceeds the built-in scratch "
                  "(%d heads, head_dim %d, %d positions); use forge_attention_flash",
                  num_heads, num_kv_heads, head_dim, seq_len, kStaticMaxHeads, kStaticMaxHeadDim, kStaticMaxSeq);
        return FORGE_ERR_SHAPE;
    }
    StaticScratch* sc = nullptr;
    FORGE_TRY(static_scratch(&sc));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int splits = std::min(kStaticMaxSplits, attn_decode_splits((seq_len + FORGE_KV_PAGE - 1) / FORGE_KV_PAGE, num_kv_heads, 148, head_dim));
    // the tickets must start at zero; the partials are fully rewritten by every call that reads them
    FORGE_CUDA(cudaMemsetAsync(sc->counters, 0, sizeof(int) * num_kv_heads, st));
    AttnDecodeArgs a{out, q, reinterpret_cast<const __half*>(k_cache), reinterpret_cast<const __half*>(v_cache), nullptr, 0, nullptr,
                     seq_len, 1, num_heads, num_kv_heads, head_dim, seq_len, sc->ws, sc->counters, splits};
    return attn_decode(a, st);
}
