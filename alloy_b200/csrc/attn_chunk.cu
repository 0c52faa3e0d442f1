// Causal attention of a CHUNK of query tokens (prefill, or the 2..16 tokens of a speculative
// verify step) over a KV cache that already holds the chunk's own rows: fp16, split q8_0 or the
// paged q8_0 pool.  Query token i of the chunk sits at position start + i and attends to cache
// positions [0, start + i].
//
// The reference runs this case as "dequantise history + chunk to an fp16 scratch in cache layout,
// then fp16 prefill attention" (torch/ops/kv_quant.py:121-162 with metal/std/kv_quant.py:73-108);
// here the q8_0 codes are read directly: a CTA dequantises each 64-token K/V tile ONCE into shared
// memory as fp16(code * scale) -- the same values the reference's scratch would hold -- and no
// global scratch exists.
//
// Work split.  A CTA owns one KV head, up to eight of its query heads and 64 / Gp query tokens
// (Gp = heads per CTA rounded up to a power of two), i.e. 64 (token, head) rows, 16 per warp; the
// K/V tile in shared memory is shared by every row.  S = Q K^T and O += P V run on
// mma.sync.m16n8k16 (fp16 operands, fp32 accumulation) with ldmatrix fragment loads; the softmax
// is the usual online one in the exp2 frame; P enters the second product as fp16 hi + lo halves.
//
// (fp16 queries over an fp16 cache at head_dim 128 with many rows: attn_prefill.cu.)
//
// What bounds it: a long prompt, the mma.sync pipe (three products of 64 x 64 x D per tile); a short chunk behind a long
// history, the length of the chain of tiles.  So the next tile's K and V are copied (cp.async) while this one is computed
// -- q8_0 caches: their raw bytes, which are expanded to the fp16 tile from shared memory --, and when the rows alone
// give too few CTAs, the key range is split over a cluster of up to eight CTAs, which merge their partial results through
// distributed shared memory (no scratch in global memory, one launch).
#include "kv.cuh"

namespace alloyb {
namespace ac {

constexpr int ROWS = 64;          // (token, head) rows per CTA
constexpr int WARPS = 4;
constexpr float NEG_BIG = -1.0e30f;
constexpr float NEG_LIVE = 0.5f * NEG_BIG;    // scores above it are real
constexpr float P_BIAS_LOG2 = 6.0f;           // P * 64 keeps small probabilities out of fp16's subnormal range in the P * V product

struct Params {
    const void* q;
    int64_t q_bs, q_hs, q_ts;     // strides in elements: batch, head, token
    int q_dtype;
    KVPtrs kv;
    const int32_t* start;
    int start_count;
    void* out;                    // (B, S, H, D) dense, q's dtype
    int B, H, KV_H, S;
    int G, Gp, HG;                // query heads per KV head; heads per CTA padded; CTAs per KV head
    float scale_log2;
    int* status;
    int pool_aligned;             // paged: the pool starts on a 16-byte boundary
    int splits;                   // CTAs (a cluster) that share the key range of the same rows
};

__device__ __forceinline__ uint32_t s32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// A value of the same place in a cluster peer's shared memory.
__device__ __forceinline__ uint32_t peer_addr(const void* p, int rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(s32(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ float peer_f32(const float* p, int rank) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(peer_addr(p, rank)) : "memory");
    return v;
}
__device__ __forceinline__ float4 peer_f32x4(const float* p, int rank) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(peer_addr(p, rank)) : "memory");
    return v;
}
__device__ __forceinline__ float q_as_f16(const void* q, int dtype, int64_t i) {
    // the attention runs on fp16 queries, like the reference (torch/ops/kv_quant.py:175-180)
    if (dtype == ALLOYB_F16) return __half2float(static_cast<const __half*>(q)[i]);
    if (dtype == ALLOYB_BF16)
        return __half2float(__float2half_rn(__bfloat162float(static_cast<const __nv_bfloat16*>(q)[i])));
    return __half2float(__float2half_rn(static_cast<const float*>(q)[i]));
}
__device__ __forceinline__ void store_out(void* out, int dtype, int64_t i, float a, float b) {
    if (dtype == ALLOYB_F16) *reinterpret_cast<__half2*>(static_cast<__half*>(out) + i) = __floats2half2_rn(a, b);
    else if (dtype == ALLOYB_BF16)
        *reinterpret_cast<__nv_bfloat162*>(static_cast<__nv_bfloat16*>(out) + i) = __floats2bfloat162_rn(a, b);
    else *reinterpret_cast<float2*>(static_cast<float*>(out) + i) = make_float2(a, b);
}

// fp16(code * scale) of eight codes held in two 32-bit words -> four packed half2.  code + 128 becomes a half by one byte
// permute (1024 + u), the subtraction is exact and the product of two halves is rounded once.
__device__ __forceinline__ uint4 dequant8(uint32_t w0, uint32_t w1, __half2 scale) {
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t u = (i < 2 ? w0 : w1) ^ 0x80808080u;
        const uint32_t m = __byte_perm(u, 0x64646464u, (i & 1) ? 0x4342 : 0x4140);
        const __half2 c = __hsub2(*reinterpret_cast<const __half2*>(&m), __float2half2_rn(1152.0f));
        const __half2 v = __hmul2(c, scale);
        o[i] = *reinterpret_cast<const uint32_t*>(&v);
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// 16 bytes of global memory to shared memory, asynchronously; zeros when !live.
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}

// KT: KV tokens per tile.  64; at head_dim 256 also 32, with which two CTAs (of ~100 KB) fit an SM.
template <int LAYOUT, int D, int KT>
struct Smem {
    static constexpr int PARTS = WARPS * 32 / KT;                           // q8_0: threads that expand a token's row
    static constexpr int PITCH = D + 8;                                     // halves
    static constexpr int TILE = KT * PITCH * 2;                             // an fp16 tile of K or V
    static constexpr bool RAW = LAYOUT != ALLOYB_KV_F16;
    static constexpr int RAW_ROW = LAYOUT == ALLOYB_KV_Q8_PAGED ? D / 32 * KV_BLOCK_BYTES : D;
    static constexpr int RAW_TILE = KT * RAW_ROW;
    static constexpr int Q = ROWS * PITCH * 2;
    static constexpr int TILES = RAW ? 2 * TILE + 4 * RAW_TILE : 4 * TILE;  // fp16: two stages; q8: one tile, two raw stages
    static constexpr int BYTES = Q + (TILES > ROWS * D * 4 ? TILES : ROWS * D * 4) + 2 * ROWS * 4;
};

// Request tile j0 (KT tokens) of K (which = 0) or V (1): fp16 rows into the tile itself, q8 bytes into the raw buffer.
template <int LAYOUT, int D, int KT>
__device__ __forceinline__ void request_tile(uint32_t dst, const Params& P, int which, int b, int kvh, int j0, int n_kv) {
    using M = Smem<LAYOUT, D, KT>;
    const int tid = threadIdx.x;
    if (LAYOUT == ALLOYB_KV_Q8_PAGED) {
        // whole pages: a head's slab of 16 rows is contiguous
        constexpr int SLAB16 = PAGE_TOKENS * M::RAW_ROW / 16;
        const int32_t* table = static_cast<const int32_t*>(P.kv.k1) + static_cast<int64_t>(b) * P.kv.max_pages;
        const uint8_t* pool = static_cast<const uint8_t*>(P.kv.k0);
#pragma unroll
        for (int pg = 0; pg < KT / PAGE_TOKENS; ++pg) {
            const int j = j0 + pg * PAGE_TOKENS;
            const int64_t page = j < n_kv ? table[j / PAGE_TOKENS] : -1;
            const bool live = page >= 0 && page < P.kv.num_pages;
            if (j < n_kv && !live && tid == 0 && P.status) atomicOr(P.status, KV_STATUS_PAGE_RANGE);
            const uint8_t* src = pool + (live ? paged_row_offset(page, which, kvh, 0, P.KV_H, D) : 0);
            for (int i = tid; i < SLAB16; i += WARPS * 32) {
                if (P.pool_aligned) {
                    copy16(dst + (pg * SLAB16 + i) * 16, src + i * 16, live);
                } else {                                 // a pool that starts off a 16-byte boundary (it is 2-byte aligned)
                    const uint16_t* h = reinterpret_cast<const uint16_t*>(src + i * 16);
#pragma unroll 1
                    for (int e = 0; e < 8; ++e)
                        asm volatile("st.shared.u16 [%0], %1;" ::"r"(dst + (pg * SLAB16 + i) * 16 + 2 * e), "h"(live ? __ldg(h + e) : uint16_t(0)) : "memory");
                }
            }
        }
    } else {
        constexpr int PER = (LAYOUT == ALLOYB_KV_F16 ? D * 2 : D) / 16, PITCH_B = LAYOUT == ALLOYB_KV_F16 ? M::PITCH * 2 : D;
        const uint8_t* base = static_cast<const uint8_t*>(which ? P.kv.v0 : P.kv.k0) + (static_cast<int64_t>(b) * P.KV_H + kvh) * P.kv.S_max * (PER * 16);
#pragma unroll
        for (int i = tid; i < KT * PER; i += WARPS * 32) {
            const int tok = i / PER, c = i - tok * PER;
            const bool live = j0 + tok < n_kv;
            copy16(dst + tok * PITCH_B + c * 16, base + static_cast<int64_t>(live ? j0 + tok : 0) * (PER * 16) + c * 16, live);
        }
    }
}

// The split layout's scales of this thread's blocks (see expand_tile), loaded a tile ahead.
template <int LAYOUT, int D, int KT>
struct Scales {
    static constexpr int N = D / 32 / Smem<LAYOUT, D, KT>::PARTS;
    __half s[N];
};
template <int LAYOUT, int D, int KT>
__device__ __forceinline__ void load_scales(Scales<LAYOUT, D, KT>& o, const Params& P, int which, int b, int kvh, int j0, int n_kv) {
    if (LAYOUT != ALLOYB_KV_Q8_SPLIT) return;
    using M = Smem<LAYOUT, D, KT>;
    constexpr int NB = D / 32, N = Scales<LAYOUT, D, KT>::N;
    const int tok = threadIdx.x / M::PARTS, j = min(j0 + tok, n_kv - 1);
    const __half* src = static_cast<const __half*>(which ? P.kv.v1 : P.kv.k1) +
                        ((static_cast<int64_t>(b) * P.KV_H + kvh) * P.kv.S_max + j) * NB + (threadIdx.x % M::PARTS) * N;
#pragma unroll
    for (int i = 0; i < N; ++i) o.s[i] = __ldg(src + i);
}

// Raw q8_0 bytes of a tile -> fp16(code * scale): PARTS threads per token, their shares of its 32-code blocks; tokens at or past
// n_kv become zero rows (whatever their page holds).
template <int LAYOUT, int D, int KT>
__device__ __forceinline__ void expand_tile(__half* dst, uint32_t raw, const Scales<LAYOUT, D, KT>& sc, int j0, int n_kv) {
    using M = Smem<LAYOUT, D, KT>;
    constexpr int N = Scales<LAYOUT, D, KT>::N;
    const int tok = threadIdx.x / M::PARTS, b0 = (threadIdx.x % M::PARTS) * N;
    const bool live = j0 + tok < n_kv;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        uint32_t w[8];
        __half s;
        if (LAYOUT == ALLOYB_KV_Q8_PAGED) {
            const uint32_t at = raw + tok * M::RAW_ROW + (b0 + i) * KV_BLOCK_BYTES, base = at & ~3u, sh = (at & 2u) * 8u;
            // scale, then 32 codes: nine words from the word that holds the scale, shifted into place
            uint32_t x[9];
#pragma unroll
            for (int k = 0; k < 9; ++k) x[k] = lds32(base + 4 * k);
            s = __ushort_as_half(static_cast<unsigned short>(sh ? x[0] >> 16 : x[0] & 0xffffu));
#pragma unroll
            for (int k = 0; k < 8; ++k) w[k] = sh ? x[k + 1] : __funnelshift_r(x[k], x[k + 1], 16);
        } else {
            const uint32_t at = raw + tok * M::RAW_ROW + (b0 + i) * 32;
#pragma unroll
            for (int k = 0; k < 8; ++k) w[k] = lds32(at + 4 * k);
            s = sc.s[i];
        }
        const __half2 s2 = __half2half2(s);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            uint4 o = dequant8(w[2 * u], w[2 * u + 1], s2);
            if (!live) o = make_uint4(0u, 0u, 0u, 0u);
            *reinterpret_cast<uint4*>(dst + tok * M::PITCH + (b0 + i) * 32 + u * 8) = o;
        }
    }
}

template <int LAYOUT, int D, int KT>
__global__ void __launch_bounds__(WARPS * 32) attn_chunk_kernel(const Params P) {
    using M = Smem<LAYOUT, D, KT>;
    pdl_launch_dependents();
    constexpr int PITCH = M::PITCH;
    extern __shared__ __align__(16) uint8_t smem[];
    __half* Qs = reinterpret_cast<__half*>(smem);
    uint8_t* tiles = smem + M::Q;
    float* Ms = reinterpret_cast<float*>(smem + M::BYTES - 2 * ROWS * 4);   // merge: row maxima, row sums
    float* Ls = Ms + ROWS;

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int split = blockIdx.x % P.splits;                // rank in the cluster
    const int kvh = blockIdx.y / P.HG, hgrp = blockIdx.y - kvh * P.HG, b = blockIdx.z;
    const int TQ = ROWS / P.Gp;                         // query tokens per CTA
    // the last rows, which see the most keys, go first
    const int tok0 = (gridDim.x / P.splits - 1 - blockIdx.x / P.splits) * TQ;
    const int gp_shift = P.Gp == 1 ? 0 : (P.Gp == 2 ? 1 : (P.Gp == 4 ? 2 : 3));
    const int heads_here = min(8, P.G - hgrp * 8);      // live heads of this CTA
    pdl_wait();
    int start = P.start[P.start_count == 1 ? 0 : b];
    if (start < 0 || start + P.S > P.kv.S_max) {
        if (threadIdx.x == 0 && P.status) atomicOr(P.status, KV_STATUS_POS_RANGE);
        start = max(0, min(start, P.kv.S_max - P.S));
    }
    const int tok_last = min(P.S, tok0 + TQ) - 1;
    const int n_kv = start + tok_last + 1;              // positions this CTA may read
    const int n_tiles = (n_kv + KT - 1) / KT, per = (n_tiles + P.splits - 1) / P.splits;
    const int tile0 = split * per, tile1 = min(n_tiles, tile0 + per);

    auto request = [&](int tile, int buf) {
        const uint32_t at = s32(tiles) + (M::RAW ? 2 * M::TILE + buf * 2 * M::RAW_TILE : buf * 2 * M::TILE);
        request_tile<LAYOUT, D, KT>(at, P, 0, b, kvh, tile * KT, n_kv);
        request_tile<LAYOUT, D, KT>(at + (M::RAW ? M::RAW_TILE : M::TILE), P, 1, b, kvh, tile * KT, n_kv);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    Scales<LAYOUT, D, KT> sk, sv;
    if (tile0 < tile1) {
        request(tile0, 0);
        load_scales<LAYOUT, D, KT>(sk, P, 0, b, kvh, tile0 * KT, n_kv);
        load_scales<LAYOUT, D, KT>(sv, P, 1, b, kvh, tile0 * KT, n_kv);
    }

    // ---- Q rows -> shared memory (fp16); dead rows are zero
    const bool q_vec = P.q_dtype == ALLOYB_F16 &&
                       ((reinterpret_cast<uintptr_t>(P.q) | (P.q_bs * 2) | (P.q_hs * 2) | (P.q_ts * 2)) & 15) == 0;
    for (int i = threadIdx.x; i < ROWS * (D / 8); i += WARPS * 32) {
        const int r = i / (D / 8), d = (i - r * (D / 8)) * 8;
        const int tl = r >> gp_shift, hg = r & (P.Gp - 1);
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (tok0 + tl < P.S && hg < heads_here) {
            const int64_t base = b * P.q_bs + static_cast<int64_t>(kvh * P.G + hgrp * 8 + hg) * P.q_hs +
                                 static_cast<int64_t>(tok0 + tl) * P.q_ts + d;
            if (q_vec) {
                v = ld_after_wait(static_cast<const __half*>(P.q) + base);
            } else {
                uint32_t* e = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    e[k] = pack_h2(q_as_f16(P.q, P.q_dtype, base + 2 * k), q_as_f16(P.q, P.q_dtype, base + 2 * k + 1));
            }
        }
        *reinterpret_cast<uint4*>(Qs + r * PITCH + d) = v;
    }

    // this thread's two rows: warp*16 + g and + 8
    int row_pos[2];                                     // last position each row may see
    bool row_live[2];
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
        const int r = warp * 16 + g + 8 * rr;
        const int tl = r >> gp_shift, hg = r & (P.Gp - 1);
        row_live[rr] = tok0 + tl < P.S && hg < heads_here;
        row_pos[rr] = start + tok0 + tl;
    }
    const int first_pos = start + tok0 + ((warp * 16) >> gp_shift);      // the warp's earliest row

    float o[D / 8][4];
#pragma unroll
    for (int i = 0; i < D / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
    float m_run[2] = {NEG_BIG, NEG_BIG}, l_run[2] = {0.f, 0.f};          // (l times 64, like o)

    const uint32_t q_addr = s32(Qs + (warp * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * PITCH + ((lane >> 4) & 1) * 8);
    const uint32_t k_off = (((lane & 7) + ((lane >> 4) & 1) * 8) * PITCH + ((lane >> 3) & 1) * 8) * 2;
    const uint32_t v_off = (((lane & 7) + ((lane >> 3) & 1) * 8) * PITCH + ((lane >> 4) & 1) * 8) * 2;

    for (int tile = tile0; tile < tile1; ++tile) {
        const int buf = (tile - tile0) & 1, j0 = tile * KT;
        const bool more = tile + 1 < tile1;
        if (more) {
            request(tile + 1, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();                                // this tile has arrived for every thread (and Q is stored)
        uint32_t k_tile = s32(tiles) + buf * 2 * M::TILE;
        if (M::RAW) {
            const uint32_t raw = s32(tiles) + 2 * M::TILE + buf * 2 * M::RAW_TILE;
            expand_tile<LAYOUT, D, KT>(reinterpret_cast<__half*>(tiles), raw, sk, j0, n_kv);
            expand_tile<LAYOUT, D, KT>(reinterpret_cast<__half*>(tiles + M::TILE), raw + M::RAW_TILE, sv, j0, n_kv);
            if (more) {
                load_scales<LAYOUT, D, KT>(sk, P, 0, b, kvh, j0 + KT, n_kv);
                load_scales<LAYOUT, D, KT>(sv, P, 1, b, kvh, j0 + KT, n_kv);
            }
            k_tile = s32(tiles);
            __syncthreads();
        }
        const uint32_t k_addr = k_tile + k_off, v_addr = k_tile + M::TILE + v_off;

        // ---- S = Q K^T : 16 rows x 64 tokens per warp
        float s[KT / 8][4];
#pragma unroll
        for (int n = 0; n < KT / 8; ++n) s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
            uint32_t a[4];
            ldsm_x4(q_addr + kk * 32, a);
#pragma unroll
            for (int n2 = 0; n2 < KT / 16; ++n2) {
                uint32_t bq[4];
                ldsm_x4(k_addr + (n2 * 16 * PITCH) * 2 + kk * 32, bq);
                mma16816(s[2 * n2], a, bq[0], bq[1]);
                mma16816(s[2 * n2 + 1], a, bq[2], bq[3]);
            }
        }
        // ---- mask (tiles that reach past the warp's earliest row only) + online softmax (rows g and g + 8; columns
        // 8n + 2t, + 1)
        if (j0 + KT - 1 > first_pos) {
#pragma unroll
            for (int n = 0; n < KT / 8; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (j0 + 8 * n + 2 * t + (e & 1) > row_pos[e >> 1]) s[n][e] = NEG_BIG;
        }
        float mx[2] = {NEG_BIG, NEG_BIG};
#pragma unroll
        for (int n = 0; n < KT / 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                // (a score of -inf or below the masked value counts as masked, NaN as absent, as it is below)
                mx[e >> 1] = fmaxf(mx[e >> 1], s[n][e]);
            }
        float alpha[2], m_sub[2];
#pragma unroll
        for (int rr = 0; rr < 2; ++rr) {
            mx[rr] = fmaxf(mx[rr], __shfl_xor_sync(0xffffffffu, mx[rr], 1));
            mx[rr] = fmaxf(mx[rr], __shfl_xor_sync(0xffffffffu, mx[rr], 2));
            const float m_new = fmaxf(m_run[rr], mx[rr] > NEG_LIVE ? mx[rr] * P.scale_log2 : NEG_BIG);
            alpha[rr] = ex2(m_run[rr] - m_new);
            m_run[rr] = m_new;
            m_sub[rr] = P_BIAS_LOG2 - m_new;            // probabilities come out times 64
        }
        if (__any_sync(0xffffffffu, alpha[0] != 1.0f || alpha[1] != 1.0f)) {
#pragma unroll
            for (int i = 0; i < D / 8; ++i) {
                o[i][0] *= alpha[0];
                o[i][1] *= alpha[0];
                o[i][2] *= alpha[1];
                o[i][3] *= alpha[1];
            }
        }
        // ---- O += P V, sixteen tokens at a time.  P enters the tensor core as fp16 hi + lo halves (two
        // products), which keeps ~22 bits of it: a single fp16 rounding of P alone would cost ~1e-3 of
        // the output's rms, more than the parity tolerance allows on outputs that cancel to near zero.
        float ls[2] = {0.f, 0.f};
#pragma unroll
        for (int k2 = 0; k2 < KT / 16; ++k2) {
            uint32_t ph[4], pl[4];
#pragma unroll
            for (int nn = 0; nn < 2; ++nn) {
                const int n = 2 * k2 + nn;
                float pv[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int rr = e >> 1;
                    pv[e] = s[n][e] > NEG_LIVE ? ex2(fmaf(s[n][e], P.scale_log2, m_sub[rr])) : 0.f;
                }
                ls[0] += pv[0] + pv[1];
                ls[1] += pv[2] + pv[3];
                const uint32_t h01 = pack_h2(pv[0], pv[1]), h23 = pack_h2(pv[2], pv[3]);
                const float2 f01 = __half22float2(*reinterpret_cast<const __half2*>(&h01));
                const float2 f23 = __half22float2(*reinterpret_cast<const __half2*>(&h23));
                ph[nn * 2] = h01;
                ph[nn * 2 + 1] = h23;
                pl[nn * 2] = pack_h2(pv[0] - f01.x, pv[1] - f01.y);
                pl[nn * 2 + 1] = pack_h2(pv[2] - f23.x, pv[3] - f23.y);
            }
#pragma unroll
            for (int n2 = 0; n2 < D / 16; ++n2) {
                uint32_t bv[4];
                ldsm_x4_t(v_addr + (k2 * 16 * PITCH) * 2 + n2 * 32, bv);
                mma16816(o[2 * n2], ph, bv[0], bv[1]);
                mma16816(o[2 * n2 + 1], ph, bv[2], bv[3]);
                mma16816(o[2 * n2], pl, bv[0], bv[1]);
                mma16816(o[2 * n2 + 1], pl, bv[2], bv[3]);
            }
        }
#pragma unroll
        for (int rr = 0; rr < 2; ++rr) {
            ls[rr] += __shfl_xor_sync(0xffffffffu, ls[rr], 1);
            ls[rr] += __shfl_xor_sync(0xffffffffu, ls[rr], 2);
            l_run[rr] = l_run[rr] * alpha[rr] + ls[rr];
        }
        __syncthreads();                                // the tile has been read: its buffer may be refilled
    }

    if (P.splits == 1) {
        // ---- normalise and store: out (B, S, H, D)
#pragma unroll
        for (int rr = 0; rr < 2; ++rr) {
            if (!row_live[rr]) continue;
            const int r = warp * 16 + g + 8 * rr;
            const int tl = r >> gp_shift, hg = r & (P.Gp - 1);
            const float inv = l_run[rr] > 0.f ? 1.0f / l_run[rr] : 0.f;
            const int64_t base = ((static_cast<int64_t>(b) * P.S + tok0 + tl) * P.H + kvh * P.G + hgrp * 8 + hg) * D;
#pragma unroll
            for (int i = 0; i < D / 8; ++i)
                store_out(P.out, P.q_dtype, base + 8 * i + 2 * t, o[i][2 * rr] * inv, o[i][2 * rr + 1] * inv);
        }
        return;
    }
    // ---- merge the cluster's partial results: every CTA leaves its own in its shared memory and finishes ROWS / splits rows
    float* Os = reinterpret_cast<float*>(tiles);        // [row][D]
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
        const int r = warp * 16 + g + 8 * rr;
#pragma unroll
        for (int i = 0; i < D / 8; ++i) *reinterpret_cast<float2*>(Os + r * D + 8 * i + 2 * t) = make_float2(o[i][2 * rr], o[i][2 * rr + 1]);
        if (t == 0) {
            Ms[r] = m_run[rr];
            Ls[r] = l_run[rr];
        }
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    const int rows_here = ROWS / P.splits, r0 = split * rows_here;
    for (int i = threadIdx.x; i < rows_here * (D / 4); i += WARPS * 32) {
        const int r = r0 + i / (D / 4), c = (i % (D / 4)) * 4;
        const int tl = r >> gp_shift, hg = r & (P.Gp - 1);
        if (tok0 + tl >= P.S || hg >= heads_here) continue;
        float top = NEG_BIG;
        for (int k = 0; k < P.splits; ++k) top = fmaxf(top, peer_f32(Ms + r, k));
        float l = 0.f;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int k = 0; k < P.splits; ++k) {
            const float w = ex2(peer_f32(Ms + r, k) - top);
            const float4 v = peer_f32x4(Os + r * D + c, k);
            l = fmaf(w, peer_f32(Ls + r, k), l);
            acc.x = fmaf(w, v.x, acc.x);
            acc.y = fmaf(w, v.y, acc.y);
            acc.z = fmaf(w, v.z, acc.z);
            acc.w = fmaf(w, v.w, acc.w);
        }
        const float inv = l > 0.f ? 1.0f / l : 0.f;
        const int64_t base = ((static_cast<int64_t>(b) * P.S + tok0 + tl) * P.H + kvh * P.G + hgrp * 8 + hg) * D + c;
        store_out(P.out, P.q_dtype, base, acc.x * inv, acc.y * inv);
        store_out(P.out, P.q_dtype, base + 2, acc.z * inv, acc.w * inv);
    }
    // nobody's shared memory goes away while a peer still reads it
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int LAYOUT, int D, int KT>
static int launch_one(Params& P, cudaStream_t st) {
    static bool configured[64] = {};
    auto kern = attn_chunk_kernel<LAYOUT, D, KT>;
    constexpr int SMEM = Smem<LAYOUT, D, KT>::BYTES;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
    if (!configured[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (e != cudaSuccess) { set_cuda_error(e); return ALLOYB_E_CUDA; }
        configured[dev] = true;
    }
    const int TQ = ROWS / P.Gp;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((P.S + TQ - 1) / TQ * P.splits, P.KV_H * P.HG, P.B);
    cfg.blockDim = dim3(WARPS * 32);
    cfg.dynamicSmemBytes = SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = P.splits;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = P.splits > 1 ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, P);
    if (e != cudaSuccess) { set_cuda_error(e); return ALLOYB_E_CUDA; }
    return check_launch();
}

// The key range is split over a cluster while there are fewer CTAs than two per SM and the cache (the history's length is
// known on the device only) has four tiles for each: a short chunk's few CTAs otherwise walk the whole history one tile
// after the other (77 tokens behind 1500, 32/8 heads: 40 CTAs of 25 tiles, 162 us of which one CTA's chain was all).
template <int LAYOUT>
static int launch_d(Params& P, int D, cudaStream_t st) {
    static int sm_count[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
    if (!sm_count[dev]) {
        int sms = 0;
        const cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) { set_cuda_error(e); return ALLOYB_E_CUDA; }
        sm_count[dev] = sms;
    }
    const int TQ = ROWS / P.Gp, sms = sm_count[dev];
    const int64_t ctas = static_cast<int64_t>((P.S + TQ - 1) / TQ) * P.KV_H * P.HG * P.B;
    P.splits = 1;
    while (P.splits < 8 && ctas * P.splits < 2 * sms && P.kv.S_max >= 2 * P.splits * 4 * 64) P.splits *= 2;
    switch (D) {
        case 64: return launch_one<LAYOUT, 64, 64>(P, st);
        case 128: return launch_one<LAYOUT, 128, 64>(P, st);
        case 256:
            // one CTA per SM is enough: the longer tiles (300 tokens, fp16: 27 us, with the shorter ones 38); more CTAs: two
            // per SM (512 tokens, fp16 / q8_0 / paged: 102 / 131 / 141 us with the longer tiles, 74 / 102 / 111)
            if (20 * ctas * P.splits <= 21 * sms) return launch_one<LAYOUT, 256, 64>(P, st);
            return launch_one<LAYOUT, 256, 32>(P, st);
        default: return ALLOYB_E_SHAPE;
    }
}

}  // namespace ac

// defined in attn_prefill.cu
int try_attn_prefill(const void* q, int64_t q_bs, int64_t q_hs, int64_t q_ts, int q_dtype, const KVPtrs& kv, const int32_t* start,
                     int start_count, void* out, int B, int H, int KV_H, int dim, int n_tokens, float scale_log2, int* status, cudaStream_t st);

// defined in kv.cu (shares the block quantiser with the one-token append)
int launch_kv_write_range(int layout, const void* new_k, const void* new_v, int64_t sb, int64_t sh, int64_t stok,
                          const KVPtrs& kv, const int32_t* start, int start_count, int B, int KV_H, int D,
                          int n_tokens, int* status, cudaStream_t st);

}  // namespace alloyb

using namespace alloyb;

static int fill_kv(int layout, void* k0, void* k1, void* v0, void* v1, int S_max, int64_t num_pages, KVPtrs& kv) {
    kv.k0 = k0; kv.k1 = k1; kv.v0 = v0; kv.v1 = v1;
    kv.S_max = S_max;
    kv.max_pages = S_max / PAGE_TOKENS;
    kv.num_pages = num_pages;
    if (!k0) return ALLOYB_E_NULL;
    if (layout == ALLOYB_KV_F16) { if (!v0) return ALLOYB_E_NULL; }
    else if (layout == ALLOYB_KV_Q8_SPLIT) { if (!k1 || !v0 || !v1) return ALLOYB_E_NULL; }
    else if (layout == ALLOYB_KV_Q8_PAGED) {
        if (!k1) return ALLOYB_E_NULL;
        if (S_max % PAGE_TOKENS || num_pages <= 0) return ALLOYB_E_SHAPE;
    } else return ALLOYB_E_SHAPE;
    return ALLOYB_OK;
}

extern "C" int alloyb_kv_write(int layout, const void* new_k, const void* new_v, int64_t batch_stride,
                               int64_t head_stride, int64_t tok_stride, void* k0, void* k1, void* v0, void* v1,
                               const int32_t* start, int start_count, int B, int KV_H, int D, int S_max,
                               int64_t num_pages, int n_tokens, int32_t* status, void* stream) {
    if (!new_k || !new_v || !start) return ALLOYB_E_NULL;
    if (B <= 0 || KV_H <= 0 || D <= 0 || D % 32 || S_max <= 0 || n_tokens < 0 || n_tokens > S_max)
        return ALLOYB_E_SHAPE;
    if (start_count != 1 && start_count != B) return ALLOYB_E_SHAPE;
    KVPtrs kv;
    const int rc = fill_kv(layout, k0, k1, v0, v1, S_max, num_pages, kv);
    if (rc != ALLOYB_OK) return rc;
    if (n_tokens == 0) return ALLOYB_OK;
    return launch_kv_write_range(layout, new_k, new_v, batch_stride, head_stride, tok_stride, kv, start, start_count,
                                 B, KV_H, D, n_tokens, reinterpret_cast<int*>(status), as_stream(stream));
}

extern "C" int alloyb_attn_chunk(int layout, const void* q, int64_t q_batch_stride, int64_t q_head_stride,
                                 int64_t q_tok_stride, int q_dtype, void* k0, void* k1, void* v0, void* v1,
                                 const int32_t* start, int start_count, void* out, int B, int H, int KV_H, int D,
                                 int n_tokens, int S_max, int64_t num_pages, float scale, int32_t* status,
                                 void* stream) {
    if (!q || !start || !out) return ALLOYB_E_NULL;
    if (B <= 0 || H <= 0 || KV_H <= 0 || H % KV_H || D <= 0 || S_max <= 0 || n_tokens < 0 || n_tokens > S_max)
        return ALLOYB_E_SHAPE;
    if (D != 64 && D != 128 && D != 256) return ALLOYB_E_SHAPE;
    if (start_count != 1 && start_count != B) return ALLOYB_E_SHAPE;
    if (q_dtype != ALLOYB_F16 && q_dtype != ALLOYB_BF16 && q_dtype != ALLOYB_F32) return ALLOYB_E_DTYPE;
    ac::Params P;
    const int rc = fill_kv(layout, k0, k1, v0, v1, S_max, num_pages, P.kv);
    if (rc != ALLOYB_OK) return rc;
    if (layout != ALLOYB_KV_Q8_PAGED &&
        (reinterpret_cast<uintptr_t>(k0) % 16 || reinterpret_cast<uintptr_t>(v0) % 16))
        return ALLOYB_E_ALIGN;
    if (n_tokens == 0) return ALLOYB_OK;
    P.q = q; P.q_bs = q_batch_stride; P.q_hs = q_head_stride; P.q_ts = q_tok_stride; P.q_dtype = q_dtype;
    P.start = start; P.start_count = start_count; P.out = out;
    P.B = B; P.H = H; P.KV_H = KV_H; P.S = n_tokens;
    P.G = H / KV_H;
    P.HG = (P.G + 7) / 8;
    const int per = P.G < 8 ? P.G : 8;
    P.Gp = per <= 1 ? 1 : (per <= 2 ? 2 : (per <= 4 ? 4 : 8));
    const float sc = scale > 0.f ? scale : 1.0f / sqrtf(static_cast<float>(D));
    P.scale_log2 = sc * 1.4426950408889634f;
    P.status = reinterpret_cast<int*>(status);
    P.pool_aligned = reinterpret_cast<uintptr_t>(k0) % 16 == 0;
    cudaStream_t st = as_stream(stream);
    if (layout == ALLOYB_KV_F16) {
        const int taken = try_attn_prefill(q, q_batch_stride, q_head_stride, q_tok_stride, q_dtype, P.kv, start, start_count, out, B, H, KV_H,
                                           D, n_tokens, P.scale_log2, P.status, st);
        if (taken != ALLOYB_NOT_TAKEN) return taken;
    }
    switch (layout) {
        case ALLOYB_KV_F16: return ac::launch_d<ALLOYB_KV_F16>(P, D, st);
        case ALLOYB_KV_Q8_SPLIT: return ac::launch_d<ALLOYB_KV_Q8_SPLIT>(P, D, st);
        default: return ac::launch_d<ALLOYB_KV_Q8_PAGED>(P, D, st);
    }
}
