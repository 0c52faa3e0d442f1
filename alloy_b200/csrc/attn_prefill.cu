// Causal attention of a long prompt chunk over an fp16 cache on the 5th-generation tensor cores (head_dim 128, fp16
// queries): the same numbers as attn_chunk.cu, which keeps short chunks, q8_0 caches and the other head sizes.
//
// What bounds it: per 128 rows x 128 keys three products of 128 x 128 x 128 (P enters P V as fp16 hi + lo halves, as
// there) take 1536 clocks of the tensor pipe, and the softmax of 128 x 128 scores about as many issue slots of a scheduler;
// on mma.sync, a quarter of the rate, the products alone are three times that.  So a CTA works on two groups of 128
// (token, head) rows in turns: while one group's scores are in the softmax warps, the tensor pipe has the other's.
//
// * Q (two groups), K and V tiles of 128 tokens in shared memory, 128-byte swizzle; K and V in two stages by cp.async (rows
//   past the last key are zero-filled: what a cache holds there is nobody's business).  K is a K-major operand, V an
//   MN-major one, so neither is transposed.
// * Scores and output accumulators live in tensor memory, 2 x (128 + 128) columns: all of it.  A thread owns a row: maximum
//   and sum need no shuffles, and its 128 scores are loaded once and stay in registers (loaded in pieces of 32, once for the
//   maximum and once for the exponentials, every piece waited for on its own, the 2048-token prompt took 208 us instead of
//   103).  P overwrites the scores in place (32 scores -> 16 columns of hi + 16 of lo) and is read from
//   there as the A operand.
// * The output is rescaled only when a row's maximum grows by more than 2^8 (P then stays below 2^14 with its bias of 2^6);
//   the stale maximum cancels in the normalisation.
// Measured (32/8 heads, with the KV write): 2048 tokens 103 us (attn_chunk.cu 215), 800 behind 1500 68 (142), 8192 tokens
// 784 us = 702 TFLOP/s of useful products; the tensor pipe is busy 45 % of the time, the rest is a group's scores on their
// way through one warp per scheduler.
// Every wait is bounded: on a time-out the sticky error word is set, tensor memory is freed and the CTA returns.
#include "kv.cuh"

namespace alloyb {
namespace ap {

constexpr int D = 128, ROWS = 256, GROUP = 128, KT = 128, STAGES = 2;
constexpr int THREADS = 12 * 32;             // warp 1 MMA, warps 0, 2, 3 copies, warps 4-7 and 8-11 the groups' softmax
constexpr int HALF = 128 * 128;              // bytes of 128 rows x 64 halves
constexpr int TILE = 2 * HALF;
constexpr int SMEM = 1024 + 2 * TILE + 2 * STAGES * TILE + 256;
constexpr uint32_t SPIN = 1u << 22;
constexpr float NEG_BIG = -1.0e30f, NEG_LIVE = 0.5f * NEG_BIG, P_BIAS_LOG2 = 6.0f, RESCALE_LOG2 = 8.0f;

__device__ int g_ap_error = 0;               // sticky: a bounded wait of this file's kernel ran out

struct Params {
    const __half* q;
    int64_t q_bs, q_hs, q_ts;
    KVPtrs kv;
    const int32_t* start;
    int start_count;
    __half* out;                             // (B, S, H, D) dense
    int H, KV_H, S, G, gp_shift, HG;         // heads per KV head; log2 of the heads per CTA (padded); CTAs per KV head
    float scale_log2;
    int* status;
};
struct Bars {
    uint64_t k_full[STAGES], v_full[STAGES], k_empty[STAGES], v_empty[STAGES];
    uint64_t s_full[2], p_full[2], o_full;
    uint32_t tmem_base;
};

__device__ __forceinline__ uint32_t s32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void bar_init(uint64_t* b, uint32_t n) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s32(b)), "r"(n));
}
__device__ __forceinline__ void bar_arrive(uint64_t* b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(s32(b)) : "memory");
}
__device__ __forceinline__ bool bar_try(uint64_t* b, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(s32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __noinline__ bool bar_wait_slow(uint64_t* b, uint32_t parity) {
    for (uint32_t i = 0; i < SPIN; ++i) {
        if (bar_try(b, parity)) return true;
        if (i > 32) __nanosleep(64);
    }
    atomicExch(&g_ap_error, 1);
    return false;
}
__device__ __forceinline__ void bar_wait(bool& ok, uint64_t* b, uint32_t parity) {
    if (ok && !bar_try(b, parity)) ok = bar_wait_slow(b, parity);
}
// Shared-memory operand in the 128-byte swizzle, rows of 128 bytes, groups of eight rows 1024 bytes apart.  K-major: the
// leading offset is unused; MN-major: it leads to the next 64 elements.
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, uint32_t leading) {
    return static_cast<uint64_t>((addr >> 4) & 0x3fffu) | static_cast<uint64_t>((leading >> 4) & 0x3fffu) << 16 |
           static_cast<uint64_t>(1024 >> 4) << 32 | static_cast<uint64_t>(1) << 46 | static_cast<uint64_t>(2) << 61;
}
// kind::f16, fp16 operands, fp32 accumulators, 128 x 128; b_mn: B is MN-major
__device__ __forceinline__ constexpr uint32_t umma_idesc(bool b_mn) {
    return 1u << 4 | (b_mn ? 1u << 16 : 0u) | (128u >> 3) << 17 | (128u >> 4) << 24;
}
__device__ __forceinline__ void umma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b),
        "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a), "l"(b),
        "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* b) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s32(b)) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t addr, float (&v)[32]) {
    uint32_t* u = reinterpret_cast<uint32_t*>(v);
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]), "=r"(u[9]),
          "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15]), "=r"(u[16]), "=r"(u[17]), "=r"(u[18]),
          "=r"(u[19]), "=r"(u[20]), "=r"(u[21]), "=r"(u[22]), "=r"(u[23]), "=r"(u[24]), "=r"(u[25]), "=r"(u[26]), "=r"(u[27]),
          "=r"(u[28]), "=r"(u[29]), "=r"(u[30]), "=r"(u[31])
        : "r"(addr));
}
__device__ __forceinline__ void tmem_ld16(uint32_t addr, float (&v)[16]) {
    uint32_t* u = reinterpret_cast<uint32_t*>(v);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]), "=r"(u[9]),
                   "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
                 : "r"(addr));
}
// Two fp32 values in one 64-bit register and the two-wide instructions on them.
__device__ __forceinline__ uint64_t f2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unf2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(addr), "r"(v[0]),
        "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
        "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
__device__ __forceinline__ void wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// Byte offset of 16-byte piece c (0..15) of a row in a tile: two halves of 64 elements, each in the 128-byte swizzle.
__device__ __forceinline__ uint32_t piece_at(int row, int c) { return (c >> 3) * HALF + row * 128 + (((c & 7) ^ (row & 7)) << 4); }

__global__ void __launch_bounds__(THREADS, 1) attn_prefill_kernel(const Params P) {
    pdl_launch_dependents();
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t q_s = s32(smem), k_s = q_s + 2 * TILE, v_s = k_s + STAGES * TILE;
    Bars* bars = reinterpret_cast<Bars*>(smem + 2 * TILE + 2 * STAGES * TILE);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kvh = blockIdx.y / P.HG, hgrp = blockIdx.y - kvh * P.HG, b = blockIdx.z;
    const int TQ = ROWS >> P.gp_shift;                          // query tokens per CTA
    const int tok0 = (gridDim.x - 1 - blockIdx.x) * TQ;         // the last rows, which see the most keys, go first
    const int heads_here = min(8, P.G - hgrp * 8);

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            bar_init(&bars->k_full[s], 3);
            bar_init(&bars->v_full[s], 3);
            bar_init(&bars->k_empty[s], 1);
            bar_init(&bars->v_empty[s], 1);
        }
        for (int g = 0; g < 2; ++g) {
            bar_init(&bars->s_full[g], 1);
            bar_init(&bars->p_full[g], 4);
        }
        bar_init(&bars->o_full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(&bars->tmem_base)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    pdl_wait();
    int start = P.start[P.start_count == 1 ? 0 : b];
    if (start < 0 || start + P.S > P.kv.S_max) {
        if (threadIdx.x == 0 && P.status) atomicOr(P.status, KV_STATUS_POS_RANGE);
        start = max(0, min(start, P.kv.S_max - P.S));
    }
    const int n_kv = start + min(P.S, tok0 + TQ), n_tiles = (n_kv + KT - 1) / KT;
    // ---- Q rows (token, head); dead rows are zero
    for (int i = threadIdx.x; i < ROWS * 16; i += THREADS) {
        const int r = i >> 4, c = i & 15, tl = r >> P.gp_shift, hg = r & ((1 << P.gp_shift) - 1);
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (tok0 + tl < P.S && hg < heads_here)
            v = ld_after_wait(P.q + b * P.q_bs + static_cast<int64_t>(kvh * P.G + hgrp * 8 + hg) * P.q_hs + static_cast<int64_t>(tok0 + tl) * P.q_ts + c * 8);
        *reinterpret_cast<uint4*>(smem + (r >> 7) * TILE + piece_at(r & 127, c)) = v;
    }
    fence_async();
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = bars->tmem_base;
    bool ok = true;

    if (warp < 4) {
        if (warp == 1) {
            // ------------------------------------------------ MMA issue (one lane)
            if (lane == 0) {
                auto scores = [&](int g, int s) {
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk) {
                        const uint32_t off = (kk >> 2) * HALF + (kk & 3) * 32;
                        umma_ss(tmem + g * 256, umma_desc(q_s + g * TILE + off, 16), umma_desc(k_s + s * TILE + off, 16), umma_idesc(false), kk > 0);
                    }
                    umma_commit(&bars->s_full[g]);
                };
                bar_wait(ok, &bars->k_full[0], 0);
                fence_after();
                if (ok) {
                    scores(0, 0);
                    scores(1, 0);
                    umma_commit(&bars->k_empty[0]);
                }
                for (int j = 0; j < n_tiles && ok; ++j) {
                    const int s = j % STAGES, s1 = (j + 1) % STAGES;
                    for (int g = 0; g < 2 && ok; ++g) {
                        bar_wait(ok, &bars->p_full[g], j & 1);
                        if (g == 0) bar_wait(ok, &bars->v_full[s], (j / STAGES) & 1);
                        fence_after();
                        if (!ok) break;
                        // P V: sixteen keys per instruction, the hi and the lo halves of P
#pragma unroll
                        for (int kk = 0; kk < 8; ++kk) {
                            const uint32_t p = tmem + g * 256 + (kk >> 1) * 32 + (kk & 1) * 8;
                            const uint64_t v = umma_desc(v_s + s * TILE + kk * 2048, HALF);
                            umma_ts(tmem + g * 256 + 128, p, v, umma_idesc(true), j > 0 || kk > 0);
                            umma_ts(tmem + g * 256 + 128, p + 16, v, umma_idesc(true), 1);
                        }
                        if (g == 1) umma_commit(&bars->v_empty[s]);
                        if (j + 1 < n_tiles) {
                            if (g == 0) {
                                bar_wait(ok, &bars->k_full[s1], ((j + 1) / STAGES) & 1);
                                fence_after();
                            }
                            if (ok) scores(g, s1);
                            if (ok && g == 1) umma_commit(&bars->k_empty[s1]);
                        }
                    }
                }
                if (ok) umma_commit(&bars->o_full);
            }
            __syncwarp();
        } else {
            // ------------------------------------------------ K and V tiles: 96 threads, cp.async
            const int ct = (warp == 0 ? 0 : warp - 1) * 32 + lane;
            const int64_t head = (static_cast<int64_t>(b) * P.KV_H + kvh) * P.kv.S_max;
            // copy n: K of tile n / 2 (even), V (odd)
            auto request = [&](int n) {
                const int j = n >> 1, s = j % STAGES;
                const bool is_v = n & 1;
                if (j >= STAGES) bar_wait(ok, is_v ? &bars->v_empty[s] : &bars->k_empty[s], ((j / STAGES) - 1) & 1);
                const uint8_t* src = static_cast<const uint8_t*>(is_v ? P.kv.v0 : P.kv.k0) + head * (D * 2);
                const uint32_t dst = (is_v ? v_s : k_s) + s * TILE;
                if (ok)
                    for (int i = ct; i < KT * 16; i += 96) {
                        const int r = i >> 4, c = i & 15, tok = j * KT + r;
                        const bool live = tok < n_kv;
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + piece_at(r, c)),
                                     "l"(src + static_cast<int64_t>(live ? tok : 0) * (D * 2) + c * 16), "r"(live ? 16 : 0)
                                     : "memory");
                    }
                asm volatile("cp.async.commit_group;" ::: "memory");
            };
            auto publish = [&](int n) {                               // copy n has landed: hand it to the tensor pipe's proxy
                fence_async();
                __syncwarp();
                if (lane == 0) bar_arrive(n & 1 ? &bars->v_full[(n >> 1) % STAGES] : &bars->k_full[(n >> 1) % STAGES]);
            };
            const int n_copies = 2 * n_tiles;
            for (int n = 0; n < n_copies; ++n) {
                request(n);
                if (n >= 2) {
                    asm volatile("cp.async.wait_group 2;" ::: "memory");
                    publish(n - 2);
                }
            }
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            for (int n = n_copies >= 2 ? n_copies - 2 : 0; n < n_copies; ++n) publish(n);
        }
    } else {
        // ------------------------------------------------ softmax: a thread per row
        const int g = (warp - 4) >> 2, r = g * GROUP + (warp & 3) * 32 + lane;
        const uint32_t lanes = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + g * 256;
        const int tl = r >> P.gp_shift, hg = r & ((1 << P.gp_shift) - 1);
        const int pos = start + tok0 + tl;                        // last position this row may see
        const int first_pos = start + tok0 + ((r - lane) >> P.gp_shift);
        float m_run = NEG_BIG, l_run = 0.f;                       // (l times 64, like the accumulators)
        for (int j = 0; j < n_tiles; ++j) {
            const int j0 = j * KT;
            bar_wait(ok, &bars->s_full[g], j & 1);
            fence_after();
            // the row's 128 scores stay in registers between the maximum and the exponentials
            float s[KT];
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_ld32(lanes + c * 32, *reinterpret_cast<float(*)[32]>(s + c * 32));
            wait_ld();
            if (j0 + KT - 1 > first_pos) {                        // (uniform in the warp)
#pragma unroll
                for (int e = 0; e < KT; ++e)
                    if (j0 + e > pos) s[e] = NEG_BIG;
            }
            float mx4[4] = {NEG_BIG, NEG_BIG, NEG_BIG, NEG_BIG};
#pragma unroll
            for (int e = 0; e < KT; e += 8)
#pragma unroll
                for (int k = 0; k < 4; ++k) mx4[k] = fmaxf(mx4[k], fmaxf(s[e + k], s[e + 4 + k]));
            const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
            const float m_new = fmaxf(m_run, mx > NEG_LIVE ? mx * P.scale_log2 : NEG_BIG);
            // the accumulators follow the maximum only in steps; with the first real score they are still empty
            const bool grow = m_new > m_run + RESCALE_LOG2;
            if (__any_sync(0xffffffffu, grow)) {
                const float alpha = grow ? ex2(m_run - m_new) : 1.0f;
                if (grow) m_run = m_new;
                l_run *= alpha;
                if (j > 0) {                                      // (these scores came behind the last P V: it is complete)
#pragma unroll 1
                    for (int c = 0; c < 8; ++c) {
                        float o[16];
                        uint32_t w[16];
                        tmem_ld16(lanes + 128 + c * 16, o);
                        wait_ld();
#pragma unroll
                        for (int e = 0; e < 16; ++e) w[e] = __float_as_uint(o[e] * alpha);
                        tmem_st16(lanes + 128 + c * 16, w);
                    }
                    wait_st();
                }
            }
            // a NaN score counts as absent (the maximum with NEG_BIG drops it), as does a row without a real score
            const float sub = m_run > NEG_LIVE ? P_BIAS_LOG2 - m_run : 0.f;
            const uint64_t scale2 = f2(P.scale_log2, P.scale_log2), sub2 = f2(sub, sub);
            uint64_t sum[2] = {f2(0.f, 0.f), f2(0.f, 0.f)};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const int at = c * 32 + 2 * e;
                    float x0, x1;
                    unf2(f2_fma(f2(fmaxf(s[at], NEG_BIG), fmaxf(s[at + 1], NEG_BIG)), scale2, sub2), x0, x1);
                    const float p0 = ex2(x0), p1 = ex2(x1);
                    sum[e & 1] = f2_add(sum[e & 1], f2(p0, p1));
                    hi[e] = pack_h2(p0, p1);
                    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hi[e]));
                    float r0, r1;
                    unf2(f2_add(f2(p0, p1), f2(-f.x, -f.y)), r0, r1);
                    lo[e] = pack_h2(r0, r1);
                }
                tmem_st16(lanes + c * 32, hi);
                tmem_st16(lanes + c * 32 + 16, lo);
            }
            float a0, a1, b0, b1;
            unf2(sum[0], a0, a1);
            unf2(sum[1], b0, b1);
            l_run += (a0 + a1) + (b0 + b1);
            wait_st();
            fence_before();
            __syncwarp();
            if (lane == 0) bar_arrive(&bars->p_full[g]);
        }
        // ---- normalise and store
        bar_wait(ok, &bars->o_full, 0);
        fence_after();
        const float inv = l_run > 0.f ? 1.0f / l_run : 0.f;
        const bool row_live = ok && tok0 + tl < P.S && hg < heads_here;
        __half* out = P.out + ((static_cast<int64_t>(b) * P.S + tok0 + tl) * P.H + kvh * P.G + hgrp * 8 + hg) * D;
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
            float o[32];
            tmem_ld32(lanes + 128 + c * 32, o);
            wait_ld();
            if (row_live) {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    *reinterpret_cast<uint4*>(out + c * 32 + q * 8) =
                        make_uint4(pack_h2(o[8 * q] * inv, o[8 * q + 1] * inv), pack_h2(o[8 * q + 2] * inv, o[8 * q + 3] * inv),
                                   pack_h2(o[8 * q + 4] * inv, o[8 * q + 5] * inv), pack_h2(o[8 * q + 6] * inv, o[8 * q + 7] * inv));
            }
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

}  // namespace ap

// NOT_TAKEN unless: fp16 queries in 16-byte-aligned rows, head_dim 128, an fp16 cache, and enough live (token, head) rows in
// tiles of 256.
int try_attn_prefill(const void* q, int64_t q_bs, int64_t q_hs, int64_t q_ts, int q_dtype, const KVPtrs& kv, const int32_t* start,
                     int start_count, void* out, int B, int H, int KV_H, int dim, int n_tokens, float scale_log2, int* status, cudaStream_t st) {
    using namespace ap;
    if (q_dtype != ALLOYB_F16 || dim != D) return ALLOYB_NOT_TAKEN;
    if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(out) | (q_bs * 2) | (q_hs * 2) | (q_ts * 2)) & 15) return ALLOYB_NOT_TAKEN;
    Params P;
    P.q = static_cast<const __half*>(q);
    P.q_bs = q_bs; P.q_hs = q_hs; P.q_ts = q_ts;
    P.kv = kv;
    P.start = start; P.start_count = start_count;
    P.out = static_cast<__half*>(out);
    P.H = H; P.KV_H = KV_H; P.S = n_tokens; P.G = H / KV_H;
    P.HG = (P.G + 7) / 8;
    const int per = P.G < 8 ? P.G : 8;
    P.gp_shift = per <= 1 ? 0 : (per <= 2 ? 1 : (per <= 4 ? 2 : 3));
    P.scale_log2 = scale_log2;
    P.status = status;
    const int TQ = ROWS >> P.gp_shift, tiles = (n_tokens + TQ - 1) / TQ;
    static bool configured[64] = {};
    static int sm_count[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
    if (!configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(attn_prefill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sm_count[dev], cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) { set_cuda_error(e); return ALLOYB_E_CUDA; }
        configured[dev] = true;
    }
    // Worth it from a third of the SMs on (32/8 heads: 448 tokens, 56 CTAs, 25.5 us against 28.0 of attn_chunk.cu, behind 1000
    // more 51 / 80; 256 tokens, 32 CTAs, 18.2 / 18.5 and 42 / 48), unless most rows are dead.  Two of attn_chunk.cu's tiles of
    // 64 rows cost an SM about as much as one tile here, so a chunk that it covers with fewer than two per tile stays there
    // (batch 32, 16 tokens behind 300: 25 us, here 38; 32 tokens: 47 / 43) -- but for a single round that fills most of the
    // SMs, where that kernel has to split its keys for it (16 tokens: batch 16 behind 3000 91 us, here 85; batch 12 behind 300
    // 22 / 21, behind 3000 80 / 81).
    const int64_t ctas = static_cast<int64_t>(tiles) * KV_H * P.HG * B, sms = sm_count[dev];
    const int small_tiles = (n_tokens + TQ / 4 - 1) / (TQ / 4);
    if (small_tiles < 2 * tiles ? 8 * ctas < 5 * sms || ctas > sms : 3 * ctas < sms) return ALLOYB_NOT_TAKEN;
    const cudaError_t e = launch_pdl(attn_prefill_kernel, dim3(tiles, KV_H * P.HG, B), dim3(THREADS), SMEM, st, P);
    if (e != cudaSuccess) { set_cuda_error(e); return ALLOYB_E_CUDA; }
    return check_launch();
}

int attn_prefill_device_error(int clear) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, ap::g_ap_error, sizeof(int)) != cudaSuccess) return 0;
    if (clear && v) {
        const int z = 0;
        cudaMemcpyToSymbol(ap::g_ap_error, &z, sizeof(int));
    }
    return v;
}

}  // namespace alloyb
