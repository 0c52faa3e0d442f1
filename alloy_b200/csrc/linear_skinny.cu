// Dequant-GEMM for a handful of fp16 tokens (2..27) against Q4_K / Q6_K matrices: the linears of batched decode
// and of verification chunks.
//
// What bounds it: with so few tokens a weight is used a few times only, so the cost is the instructions that turn
// packed codes into MMA operands (a B200 streams ~11e12 Q4_K weights per second from HBM and issues ~1.1e12 warp
// instructions), then the mma.sync rate, then the traffic of the tokens out of L2.  The layout follows from that:
//
// * Weights as the MMA's A operand (16 rows), tokens as its columns.  A Q4_K weight enters as the INTEGER
//   nibble * scale (at most 945, exact in fp16; the nibble comes out of one AND as an fp16 subnormal and one
//   multiplication per two weights applies the six-bit scale), so a whole super-block of 256 accumulates in the
//   tensor core and fp32 work per token is left for the super-block's d only, not for every 32 weights.
// * Lane (g, t) holds rows g and g + 8 and the 64 weights of the two sub-blocks 2t, 2t + 1.  The k slots of an MMA
//   may be any weights as long as both operands agree, so the four lanes of a row take different sub-blocks, each lane
//   needs the scales of its own two only, and reads its weights with 128-bit loads.
// * The minima (dmin * m * sum of x) are one MMA per super-block: A = the integers m, B = the sums of x per sub-block in two
//   pieces (22 bits, scaled to fit any activations).  On tokens whose products cancel, where the output's rounding hides
//   nothing, the error of the whole sum is 0.07 .. 0.2 x 2^-24 of sum |w x| rms (K = 2048 .. 14336); linear_mma.cu, which
//   keeps the sums in fp32 and adds up after every 32 weights, leaves 0.4 .. 2.3.  The sums come from MMAs against ones with the TOKENS as rows, whose
//   accumulator layout is the layout the B operand wants.
// * Q6_K: codes minus 32 as fp16, one MMA per 16-weight sub-block, the sub-block's d * scale applied in fp32 to the
//   sums (a product of code and scale would need 12 bits).
//
// Work split: the stacked output rows are cut into tiles of 16 (a gate/up pair: 8 gate rows and the same 8 up rows), a
// contiguous range of tiles per CTA.  Its eight warps are RS row groups x KS slices of K (super-blocks k, k + KS, ...): a
// warp walks up to RT tiles together, so that a super-block's token fragments, held in registers, serve all of them, and
// the RS warps of a slice share the token buffers.  Few tiles per CTA: KS = 8, which keeps all warps busy; many: KS = 2,
// which leaves long K walks and little to add up at the end (with KS = 8 throughout, K = 4096 is two super-blocks per warp
// and pass, and the barriers around the sums took as long as the arithmetic).  Every warp has its own ring of weight stages;
// weights are requested before griddepcontrol.wait.  The KS partial tiles of a row group are added up in shared memory.
#include <cuda.h>

#include "linear.cuh"
#include "linear_rows.cuh"

namespace alloyb {
namespace sk {

constexpr int WARPS = 8;
constexpr int MAX_STAGES = 4, MAX_XD = 2;
constexpr int Q4_PITCH = 144, Q6_PITCH = 240;       // Q6_K: the 16-byte-aligned window around the 210-byte block
constexpr int TBL_PITCH = 20;                       // floats: 16-byte reads of eight rows fall on distinct banks
constexpr int RED_PITCH = 20;                       // floats per token of a partial tile
constexpr int RED_GROUPS = 2;                       // token groups added up at a time
constexpr uint32_t SPIN = 1u << 22;

__device__ int g_sk_error = 0;                      // sticky: a bounded wait of this file's kernel ran out

struct Seg {
    void* y;
    int64_t ldy;
    int n_rows;
    int tile0;                                      // first tile of this matrix in the launch
    int q6;
    int n, box;                                     // most tiles of a warp; tiles of a large copy
};
struct Params {
    Seg seg[MAX_SEGS];
    const __half* x;
    const __half* residual;
    int n_seg, n_tiles;
    int M, K, nsb;
    int gated, act;
    int ks, rs, pass_tiles;                         // K slices x row groups = warps; tiles of a CTA's pass
    int xd;                                         // token buffers of a K slice
    int stages, stage_bytes;                        // ring of every warp: a stage is one super-block of a pass's tiles
};
struct Maps {
    CUtensorMap x;                                  // tokens: 32 elements x 8 NT rows, 64-byte swizzle
    CUtensorMap all[MAX_SEGS];                      // packed rows as 32-bit words: the rows of a full pass,
    CUtensorMap one[MAX_SEGS];                      // and of one tile
};

// Token buffers of a K slice: the sub-blocks of one nibble plane, four boxes of 32 elements in the 64-byte swizzle.  Box t
// starts t * PHASE bytes late, which turns the swizzle's phase by t: the 128-bit reads of the lanes (g, t), which take the
// same piece of row g of four different boxes, then fall on distinct banks.
template <int NT>
struct Cfg {
    static constexpr int ROW = 64, PHASE = 128, BOX = 8 * NT * ROW;
    static constexpr int X_BYTES = (4 * BOX + 3 * PHASE + 8 * ROW - 1) / (8 * ROW) * (8 * ROW);
    static constexpr int RG = RED_GROUPS;
    // per warp: the scale table of a Q6_K tile while it walks K, 16 tokens of a partial tile afterwards
    static constexpr int SCRATCH = 16 * TBL_PITCH;
    static constexpr int BAR_BYTES = (WARPS * MAX_STAGES + 2 * WARPS * MAX_XD) * 8;
    static constexpr int FIXED = 1024 + WARPS * SCRATCH * 4 + (BAR_BYTES + 127) / 128 * 128;    // without token buffers and rings
};

__device__ __forceinline__ uint32_t s32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t n) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(n));
}
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __noinline__ bool bar_wait_slow(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < SPIN; ++i) {
        if (bar_try(bar, parity)) return true;
        if (i > 32) __nanosleep(32);
    }
    atomicExch(&g_sk_error, 1);
    return false;
}
// After a wait has run out (sticky error word set, results void) the warp no longer waits and issues no more copies.
__device__ __forceinline__ void bar_wait(bool& ok, uint32_t bar, uint32_t parity) {
    if (ok && !bar_try(bar, parity)) ok = bar_wait_slow(bar, parity);
}
__device__ __forceinline__ void tma_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
        "l"(map), "r"(bar), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t addr) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
    return v;
}
// 32 bits at a shared address that is 4-byte aligned (AL) or 2 bytes past a 4-byte boundary.
template <bool AL> __device__ __forceinline__ uint32_t lds32_u(uint32_t addr) {
    if (AL) return lds32(addr);
    return __funnelshift_r(lds32(addr - 2u), lds32(addr + 2u), 16);
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}
__device__ __forceinline__ uint32_t hmul2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t hadd2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t hfma2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_zero(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("{\n\t.reg .f32 z;\n\tmov.f32 z, 0f00000000;\n\t"
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {z,z,z,z};\n\t}"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// The sums of x over a lane's two sub-blocks as a B operand: S / 32 (in range whatever the activations) as a half and
// 2^11 times what that half leaves out (the matching A entries are m and m / 2^11), 22 bits in all.
__device__ __forceinline__ uint2 split_sums(float s0, float s1) {
    s0 *= 0.03125f;
    s1 *= 0.03125f;
    const __half2 h = __floats2half2_rn(s0, s1);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn((s0 - f.x) * 2048.0f, (s1 - f.y) * 2048.0f);
    return make_uint2(*reinterpret_cast<const uint32_t*>(&h), *reinterpret_cast<const uint32_t*>(&l));
}

// One super-block (NP = 2) or one nibble plane of it (NP = 1, plane `half`) of a 16-row Q4_K tile.
//   b[p][s][nt]: the lane's eight activations (64t + 32 plane + 8s ..) of token 8 nt + g
//   sx: split_sums of sub-blocks 2t, 2t + 1 of token 8 nt + g (used with the last plane)
//   rg, rh: shared addresses of the lane's two rows
template <int NT, int NP>
__device__ __forceinline__ void tile_q4(uint32_t rg, uint32_t rh, int half, const uint4 (&b)[NP][4][NT], const uint2 (&sx)[NT], int t,
                                        float (&acc)[NT][4]) {
    const uint4 hg = lds128(rg), hh = lds128(rh);
    uint4 wg[2], wh[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        wg[i] = lds128(rg + 16 + 32 * t + 16 * i);
        wh[i] = lds128(rh + 16 + 32 * t + 16 * i);
    }
    // six-bit scales and minima of sub-blocks 2t, 2t+1 of both rows: bytes {g: 2t, 2t+1; g+8: 2t, 2t+1}
    const bool high = t >= 2;
    const uint32_t b2 = 2u * (t & 1), sel = b2 | ((b2 + 1u) << 4) | ((b2 + 4u) << 8) | ((b2 + 5u) << 12);
    const uint32_t m_a = high ? 0x0f0f0f0fu : 0x3f3f3f3fu, m_b = high ? 0x30303030u : 0u;
    const uint32_t Y = prmt(hg.y, hh.y, sel), Z = prmt(hg.z, hh.z, sel), W = prmt(hg.w, hh.w, sel);
    const uint32_t sc4 = ((high ? W : Y) & m_a) | ((Y >> 2) & m_b);
    float c[NT][4];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const int plane = NP == 2 ? p : half;
        // the scale in both halves of a register: 1024 + sc, then sc (low plane) or sc / 16 (high plane, whose nibbles
        // sit four bits up); both exact
        const uint32_t mul = plane ? 0x2C002C00u : 0x3C003C00u, add = plane ? 0xD400D400u : 0xE400E400u;
        const uint32_t mask = plane ? 0x00f000f0u : 0x000f000fu;
        const uint32_t sg = hfma2(prmt(sc4, 0x64646464u, 0x4040u + 0x0101u * plane), mul, add);
        const uint32_t sh = hfma2(prmt(sc4, 0x64646464u, 0x4242u + 0x0101u * plane), mul, add);
#pragma unroll
        for (int s = 0; s < 4; ++s) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const uint4 vg = wg[s >> 1], vh = wh[s >> 1];
                const uint32_t qg = (s & 1) ? (i ? vg.w : vg.z) : (i ? vg.y : vg.x);
                const uint32_t qh = (s & 1) ? (i ? vh.w : vh.z) : (i ? vh.y : vh.x);
                const uint32_t a0 = hmul2(prmt(qg, 0u, 0x4140u) & mask, sg), a2 = hmul2(prmt(qg, 0u, 0x4342u) & mask, sg);
                const uint32_t a1 = hmul2(prmt(qh, 0u, 0x4140u) & mask, sh), a3 = hmul2(prmt(qh, 0u, 0x4342u) & mask, sh);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    const uint32_t b0 = i ? b[p][s][nt].z : b[p][s][nt].x, b1 = i ? b[p][s][nt].w : b[p][s][nt].y;
                    if (p == 0 && s == 0 && i == 0) mma_zero(c[nt], a0, a1, a2, a3, b0, b1);
                    else mma(c[nt], a0, a1, a2, a3, b0, b1);
                }
            }
        }
    }
    const float2 dg = __half22float2(*reinterpret_cast<const __half2*>(&hg.x));
    const float2 dh = __half22float2(*reinterpret_cast<const __half2*>(&hh.x));
    const float d0 = dg.x * 16777216.0f, d1 = dh.x * 16777216.0f;      // the nibbles entered as n * 2^-24
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        acc[nt][0] = fmaf(d0, c[nt][0], acc[nt][0]);
        acc[nt][1] = fmaf(d0, c[nt][1], acc[nt][1]);
        acc[nt][2] = fmaf(d1, c[nt][2], acc[nt][2]);
        acc[nt][3] = fmaf(d1, c[nt][3], acc[nt][3]);
    }
    if (NP == 2 || half == 1) {
        const uint32_t mn4 = ((high ? (W >> 4) : Z) & m_a) | ((Z >> 2) & m_b);
        const uint32_t a0 = hadd2(prmt(mn4, 0x64646464u, 0x4140u), 0xE400E400u), a1 = hadd2(prmt(mn4, 0x64646464u, 0x4342u), 0xE400E400u);
        const uint32_t a2 = hmul2(a0, 0x10001000u), a3 = hmul2(a1, 0x10001000u);       // 2^-11
        const float m0 = -32.0f * dg.y, m1 = -32.0f * dh.y;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            float m[4];
            mma_zero(m, a0, a1, a2, a3, sx[nt].x, sx[nt].y);
            acc[nt][0] = fmaf(m0, m[0], acc[nt][0]);
            acc[nt][1] = fmaf(m0, m[1], acc[nt][1]);
            acc[nt][2] = fmaf(m1, m[2], acc[nt][2]);
            acc[nt][3] = fmaf(m1, m[3], acc[nt][3]);
        }
    }
}

// The d * scale of a 16-row Q6_K super-block as floats, [row][h][qa | qb][low i0, low i1, high i0, high i1] (see tile_q6).
__device__ __forceinline__ void table_q6(uint32_t blk, float* tbl, int lane) {
    const int r = lane >> 1, h = lane & 1;
    const uint32_t row = blk + r * Q6_PITCH;
    const float d = half_bits_to_f32(lds16(row + 208));
    float s[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t two = lds16(row + 192 + 8 * h + 2 * i) ^ 0x8080u;         // code + 128
        s[2 * i] = d * (__uint_as_float(prmt(two, 0x4B000000u, 0x7540u)) - 8388736.0f);
        s[2 * i + 1] = d * (__uint_as_float(prmt(two, 0x4B000000u, 0x7541u)) - 8388736.0f);
    }
    float4* o = reinterpret_cast<float4*>(tbl + r * TBL_PITCH + h * 8);
    o[0] = make_float4(s[0], s[1], s[4], s[5]);
    o[1] = make_float4(s[2], s[3], s[6], s[7]);
}

// The sub-blocks of one half of the codes: half 0 = the bytes "qa" of both 128-weight halves h (planes 0 and 2),
// half 1 = the bytes "qb" (planes 1 and 3).
template <int NT, bool AL>
__device__ __forceinline__ void tile_q6(uint32_t blk, int half, const uint2 (&b)[2][2][2][NT], const float* tbl, int g, int t,
                                        float (&acc)[NT][4]) {
    const uint32_t rg = blk + g * Q6_PITCH + 4 * t;
    const uint32_t sh_lo = half ? 2u : 4u;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const float4 sg = *reinterpret_cast<const float4*>(tbl + g * TBL_PITCH + h * 8 + half * 4);
        const float4 sh = *reinterpret_cast<const float4*>(tbl + (g + 8) * TBL_PITCH + h * 8 + half * 4);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            uint32_t lo[4], hi[4];
#pragma unroll
            for (int rr = 0; rr < 2; ++rr) {
                const uint32_t r = rg + rr * 8 * Q6_PITCH + 16 * i;
                const uint32_t q = lds32_u<AL>(r + 64 * h + 32 * half), qh = lds32_u<AL>(r + 128 + 32 * h);
                // bit pairs: plane 0 / 1 at bits 0 / 2, plane 2 / 3 at bits 4 / 6
                const uint32_t cl = (q & 0x0f0f0f0fu) | ((qh << sh_lo) & 0x30303030u);
                const uint32_t ch = ((q >> 4) & 0x0f0f0f0fu) | ((qh >> (4u - sh_lo)) & 0x30303030u);
                lo[rr] = hadd2(prmt(cl, 0x64646464u, 0x4140u), 0xE420E420u);            // 1024 + code - 1056
                lo[rr + 2] = hadd2(prmt(cl, 0x64646464u, 0x4342u), 0xE420E420u);
                hi[rr] = hadd2(prmt(ch, 0x64646464u, 0x4140u), 0xE420E420u);
                hi[rr + 2] = hadd2(prmt(ch, 0x64646464u, 0x4342u), 0xE420E420u);
            }
            const float g0 = i ? sg.y : sg.x, g1 = i ? sg.w : sg.z, h0 = i ? sh.y : sh.x, h1 = i ? sh.w : sh.z;
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                float c[4], e[4];
                mma_zero(c, lo[0], lo[1], lo[2], lo[3], b[h][0][i][nt].x, b[h][0][i][nt].y);
                mma_zero(e, hi[0], hi[1], hi[2], hi[3], b[h][1][i][nt].x, b[h][1][i][nt].y);
                acc[nt][0] = fmaf(g0, c[0], acc[nt][0]);
                acc[nt][1] = fmaf(g0, c[1], acc[nt][1]);
                acc[nt][2] = fmaf(h0, c[2], acc[nt][2]);
                acc[nt][3] = fmaf(h0, c[3], acc[nt][3]);
                acc[nt][0] = fmaf(g1, e[0], acc[nt][0]);
                acc[nt][1] = fmaf(g1, e[1], acc[nt][1]);
                acc[nt][2] = fmaf(h1, e[2], acc[nt][2]);
                acc[nt][3] = fmaf(h1, e[3], acc[nt][3]);
            }
        }
    }
}

// A pass: consecutive tiles of one matrix, shared out over the row groups.
struct Pass {
    int tile, n, seg;
};
__device__ __forceinline__ void enter_pass(Pass& p, const Params& P, int hi) {
    while (p.seg + 1 < P.n_seg && p.tile >= P.seg[p.seg + 1].tile0) ++p.seg;
    const int end = p.seg + 1 < P.n_seg ? min(hi, P.seg[p.seg + 1].tile0) : hi;
    p.n = min(min(P.pass_tiles, P.rs * P.seg[p.seg].n), end - p.tile);
}
// Row group r's tiles of a pass: how many, and from which on.
__device__ __forceinline__ int share_n(const Pass& p, int rs, int r) { return (p.n + rs - 1 - r) / rs; }
__device__ __forceinline__ int share_at(const Pass& p, int rs, int r) { return r * (p.n / rs) + min(r, p.n % rs); }

template <int NT, int RT>
__global__ void __launch_bounds__(WARPS * 32, 1) linear_skinny_kernel(const __grid_constant__ Maps maps, const Params P) {
    using C = Cfg<NT>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int kg = warp & (P.ks - 1), rg = warp / P.ks;          // (ks is a power of two)
    const uint32_t x_bytes = P.ks * P.xd * C::X_BYTES, x_buf = s32(smem) + kg * P.xd * C::X_BYTES;
    float* red = reinterpret_cast<float*>(smem + x_bytes);
    float* tbl = red + warp * C::SCRATCH;
    const uint32_t bar0 = s32(red) + WARPS * C::SCRATCH * 4;
    const uint32_t bars = bar0 + warp * MAX_STAGES * 8;
    const uint32_t x_full = bar0 + WARPS * MAX_STAGES * 8 + kg * 2 * MAX_XD * 8, x_empty = x_full + MAX_XD * 8;
    const uint32_t ring = s32(smem) + x_bytes + C::FIXED - 1024 + warp * P.stages * P.stage_bytes;

    const int lo = static_cast<int>(static_cast<int64_t>(P.n_tiles) * blockIdx.x / gridDim.x);
    const int hi = static_cast<int>(static_cast<int64_t>(P.n_tiles) * (blockIdx.x + 1) / gridDim.x);
    if (lane == 0) {
        for (int s = 0; s < P.stages; ++s) bar_init(bars + 8 * s, 1);
        if (rg == 0)
            for (int s = 0; s < P.xd; ++s) {
                bar_init(x_full + 8 * s, 1);
                bar_init(x_empty + 8 * s, P.rs);
            }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_launch_dependents();

    bool ok = true;
    // ---- weight copies, one super-block of the warp's tiles after the other, in the order they are consumed.  Rows of a
    // stage: the tiles' rows one behind the other; a gate/up pair: all gate rows, then all up rows.
    const int tile_rows = P.gated ? 8 : 16, up_off = P.gated ? 8 * P.seg[0].n * Q4_PITCH : 0;
    Pass lp = {lo, 0, 0};
    int l_sb = kg, l_stage = 0;
    enter_pass(lp, P, hi);
    auto load_stage = [&]() {
        if (lp.tile >= hi || kg >= P.nsb) return;
        if (lane == 0 && ok) {
            const Seg& sg = P.seg[lp.seg];
            const uint32_t bar = bars + 8 * l_stage, dst = ring + l_stage * P.stage_bytes;
            const int n = share_n(lp, P.rs, rg), row = (lp.tile + share_at(lp, P.rs, rg) - sg.tile0) * tile_rows;
            const int pitch = sg.q6 ? Q6_PITCH : Q4_PITCH, col = sg.q6 ? ((l_sb * Q6K_BYTES) & ~15) >> 2 : l_sb * (Q4K_BYTES / 4);
            bar_expect(bar, n * 16 * pitch);             // (no tiles: the stage is complete at once)
            int i = 0;
            for (; i + sg.box <= n; i += sg.box) {
                tma_2d(dst + i * tile_rows * pitch, &maps.all[lp.seg], col, row + i * tile_rows, bar);
                if (P.gated) tma_2d(dst + up_off + i * tile_rows * pitch, &maps.all[1], col, row + i * tile_rows, bar);
            }
            for (; i < n; ++i) {
                tma_2d(dst + i * tile_rows * pitch, &maps.one[lp.seg], col, row + i * tile_rows, bar);
                if (P.gated) tma_2d(dst + up_off + i * tile_rows * pitch, &maps.one[1], col, row + i * tile_rows, bar);
            }
        }
        if (++l_stage == P.stages) l_stage = 0;
        l_sb += P.ks;
        if (l_sb >= P.nsb) {
            l_sb = kg;
            lp.tile += lp.n;
            if (lp.tile < hi) enter_pass(lp, P, hi);
        }
    };
    for (int s = 0; s < P.stages; ++s) load_stage();
    // ---- token copies of the slice, by the first row group's lane 0: plane after plane, super-block after super-block
    Pass xp = {lo, 0, 0};
    int x_sb = kg, x_half = 0;
    enter_pass(xp, P, hi);
    auto load_x = [&](int buf) {
        if (xp.tile >= hi || kg >= P.nsb) return;
        if (ok) {
            bar_expect(x_full + 8 * buf, 4 * C::BOX);
#pragma unroll
            for (int q = 0; q < 4; ++q)
                tma_2d(x_buf + buf * C::X_BYTES + q * (C::BOX + C::PHASE), &maps.x, x_sb * QK_K + 64 * q + 32 * x_half, 0, x_full + 8 * buf);
        }
        x_half ^= 1;
        if (x_half == 0) {
            x_sb += P.ks;
            if (x_sb >= P.nsb) {
                x_sb = kg;
                xp.tile += xp.n;
                if (xp.tile < hi) enter_pass(xp, P, hi);
            }
        }
    };
    pdl_wait();      // activations (and the output buffer) belong to the previous kernel until here
    if (rg == 0 && lane == 0)
        for (int s = 0; s < P.xd; ++s) load_x(s);

    uint32_t par = 0, stage = 0;                     // next parity of the ring, next stage
    uint32_t xb = 0, x_par = 0;                      // the same of the token buffers
    // the fragments are in registers: the buffer can be filled again once all row groups have got this far
    auto free_x = [&]() {
        __syncwarp();
        if (lane == 0) {
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(x_empty + 8 * xb) : "memory");
            if (rg == 0) {
                bar_wait(ok, x_empty + 8 * xb, x_par);
                load_x(xb);
            }
        }
        __syncwarp();
        if (++xb == static_cast<uint32_t>(P.xd)) {
            xb = 0;
            x_par ^= 1;
        }
    };
    Pass ps = {lo, 0, 0};
    while (ps.tile < hi) {
        enter_pass(ps, P, hi);
        const Seg& sg = P.seg[ps.seg];
        const int n = share_n(ps, P.rs, rg);
        float acc[RT][NT][4];
#pragma unroll
        for (int rt = 0; rt < RT; ++rt)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[rt][nt][i] = 0.f;
        for (int sb = kg; sb < P.nsb; sb += P.ks) {
            const uint32_t st = ring + stage * P.stage_bytes, bar = bars + 8 * stage;
            if (!sg.q6) {
                const uint32_t row_g = st + g * Q4_PITCH, off_h = P.gated ? up_off : 8 * Q4_PITCH, step = tile_rows * Q4_PITCH;
                float sum[(NT + 1) / 2][4];
                uint2 sx[NT];
#pragma unroll
                for (int i = 0; i < (NT + 1) / 2; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) sum[i][j] = 0.f;
#pragma unroll 1
                for (int half = 0; half < 2; ++half) {
                    uint4 b[1][4][NT];
                    bar_wait(ok, x_full + 8 * xb, x_par);
                    const uint32_t x_row = x_buf + xb * C::X_BYTES + g * C::ROW + t * (C::BOX + C::PHASE);
#pragma unroll
                    for (int s = 0; s < 4; ++s) {
                        const uint32_t piece = s ^ (((g >> 1) + t) & 3);
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt) b[0][s][nt] = lds128(x_row + (piece << 4) + nt * 8 * C::ROW);
                    }
                    // sums of x per sub-block: tokens as the rows, column n = sub-block n
                    const uint32_t one = g == 2 * t + half ? 0x3C003C00u : 0u;
#pragma unroll
                    for (int s = 0; s < 4; ++s)
#pragma unroll
                        for (int n2 = 0; n2 < (NT + 1) / 2; ++n2) {
                            const uint4 u = b[0][s][2 * n2];
                            const uint4 v = 2 * n2 + 1 < NT ? b[0][s][2 * n2 + 1 < NT ? 2 * n2 + 1 : 0] : make_uint4(0u, 0u, 0u, 0u);
                            mma(sum[n2], u.x, v.x, u.y, v.y, one, one);
                            mma(sum[n2], u.z, v.z, u.w, v.w, one, one);
                        }
                    free_x();
                    if (half == 1) {
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt) sx[nt] = split_sums(sum[nt >> 1][2 * (nt & 1)], sum[nt >> 1][2 * (nt & 1) + 1]);
                    }
                    if (half == 0) bar_wait(ok, bar, par);
#pragma unroll
                    for (int rt = 0; rt < RT; ++rt)
                        if (rt < n) tile_q4<NT, 1>(row_g + rt * step, row_g + rt * step + off_h, half, b, sx, t, acc[rt]);
                }
            } else {
                const uint32_t off = (sb * Q6K_BYTES) & 15;
#pragma unroll 1
                for (int half = 0; half < 2; ++half) {
                    // [h][low | high plane][i][token group]: weights 128h + 32 (half + 2 hi) + 16i + 4t = box 2h + hi, element
                    // 32 half + 16i + 4t
                    uint2 b[2][2][2][NT];
                    bar_wait(ok, x_full + 8 * xb, x_par);
                    const uint32_t x_row = x_buf + xb * C::X_BYTES + g * C::ROW + 8 * (t & 1);
#pragma unroll
                    for (int q = 0; q < 4; ++q)
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const uint32_t c = 2 * i + (t >> 1);
                            const uint32_t piece = c ^ (((g >> 1) + q) & 3);
#pragma unroll
                            for (int nt = 0; nt < NT; ++nt)
                                b[q >> 1][q & 1][i][nt] = lds64(x_row + q * (C::BOX + C::PHASE) + (piece << 4) + nt * 8 * C::ROW);
                        }
                    if (half == 0) bar_wait(ok, bar, par);
#pragma unroll
                    for (int rt = 0; rt < RT; ++rt) {
                        if (rt < n) {
                            const uint32_t blk = st + rt * 16 * Q6_PITCH + off;
                            __syncwarp();
                            table_q6(blk, tbl, lane);
                            __syncwarp();
                            if (off & 2) tile_q6<NT, false>(blk, half, b, tbl, g, t, acc[rt]);
                            else tile_q6<NT, true>(blk, half, b, tbl, g, t, acc[rt]);
                        }
                    }
                    free_x();                       // (the fragments have been used)
                }
            }
            __syncwarp();                           // all lanes have read the stage
            load_stage();
            if (++stage == static_cast<uint32_t>(P.stages)) {
                stage = 0;
                par ^= 1;
            }
        }
        // ---- add the row group's partial tiles up, [warp][token][row], RG token groups at a time
        const int row_base = (ps.tile + share_at(ps, P.rs, rg) - sg.tile0) * tile_rows;
        auto group_sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + rg), "r"(32 * P.ks) : "memory"); };
        group_sync();                               // (the scale tables share this memory)
#pragma unroll
        for (int rt = 0; rt < RT; ++rt) {
            if (rt < n) {
#pragma unroll
                for (int n0 = 0; n0 < NT; n0 += C::RG) {
#pragma unroll
                    for (int j = 0; j < C::RG; ++j)
                        if (n0 + j < NT) {
                            float* at = tbl + (8 * j + 2 * t) * RED_PITCH + g;
                            at[0] = acc[rt][n0 + j < NT ? n0 + j : 0][0];
                            at[RED_PITCH] = acc[rt][n0 + j < NT ? n0 + j : 0][1];
                            at[8] = acc[rt][n0 + j < NT ? n0 + j : 0][2];
                            at[RED_PITCH + 8] = acc[rt][n0 + j < NT ? n0 + j : 0][3];
                        }
                    group_sync();
                    for (int idx = kg * 32 + lane; idx < 8 * C::RG * tile_rows; idx += 32 * P.ks) {
                        const int r = idx & (tile_rows - 1), tl = P.gated ? idx >> 3 : idx >> 4;
                        const int tok = 8 * n0 + tl, row = row_base + rt * tile_rows + r;
                        if (tok < P.M && row < sg.n_rows) {
                            const float* at = red + rg * P.ks * C::SCRATCH + tl * RED_PITCH + r;
                            const int64_t to = static_cast<int64_t>(tok) * sg.ldy + row;
                            float v = 0.f, u = 0.f;
#pragma unroll
                            for (int w = 0; w < WARPS; ++w)
                                if (w < P.ks) {
                                    v += at[w * C::SCRATCH];
                                    if (P.gated) u += at[w * C::SCRATCH + 8];
                                }
                            __half y;
                            if (P.gated) {
                                y = __float2half_rn((P.act == ALLOYB_ACT_SILU ? act_silu(v) : act_gelu_tanh(v)) * u);
                            } else {
                                y = __float2half_rn(v);
                                if (P.residual) y = __float2half_rn(__half2float(P.residual[to]) + __half2float(y));
                            }
                            static_cast<__half*>(sg.y)[to] = y;
                        }
                    }
                    group_sync();
                }
            }
        }
        ps.tile += ps.n;
    }
    // a wait ran out: give copies that are still in flight time to land before the shared memory is released
    if (!ok)
        for (int i = 0; i < 2048; ++i) __nanosleep(512);
}

// ---- up to sixteen tokens, rows of up to 32 super-blocks (9..16 tokens: 16): every one of a CTA's W warps keeps the token
// fragments of its own NSB super-blocks in registers for the whole launch.
//
// In the kernel above the token path -- copies, waits, sums, once per super-block and warp -- took as long as the weights'
// arithmetic at these sizes (gate/up 14336 x 4096, 8 tokens: 28 us, 14 of them without any weight arithmetic).  With the
// fragments and sums in registers a tile costs one wait, NSB tiles' arithmetic and its share of a barrier: the W warps'
// partial results of two tiles meet in shared memory, double-buffered, one barrier per two tiles.
template <int NSB> struct FixedGeom {
    // two super-blocks per row: 16 spare bytes make the pitch 16 modulo 128 (conflict-free 128-bit reads of eight rows)
    static constexpr int PITCH = NSB == 2 ? 2 * Q4_PITCH + 16 : Q4_PITCH, SLOT = 16 * PITCH;
};
template <int NT, int W> struct FixedRed {
    static constexpr int WARP = 2 * 8 * NT * RED_PITCH, BYTES = 2 * W * WARP * 4;       // two tiles of a warp (floats); both buffers
    static constexpr int BARS = (W * MAX_STAGES * 8 + 127) / 128 * 128;                 // (the rings behind it start on 128 bytes)
};

template <int NT, int W, int NSB, int MINB>
__global__ void __launch_bounds__(W * 32, MINB) linear_skinny_fixed_kernel(const __grid_constant__ Maps maps, const Params P) {
    using G = FixedGeom<NSB>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    float* red = reinterpret_cast<float*>(smem);
    const uint32_t bars = s32(smem) + FixedRed<NT, W>::BYTES + warp * MAX_STAGES * 8;
    const uint32_t ring = s32(smem) + FixedRed<NT, W>::BYTES + FixedRed<NT, W>::BARS + warp * P.stages * G::SLOT;
    const int lo = static_cast<int>(static_cast<int64_t>(P.n_tiles) * blockIdx.x / gridDim.x);
    const int hi = static_cast<int>(static_cast<int64_t>(P.n_tiles) * (blockIdx.x + 1) / gridDim.x);
    if (lane == 0) {
        for (int s = 0; s < P.stages; ++s) bar_init(bars + 8 * s, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    pdl_launch_dependents();
    bool ok = true;
    const int tile_rows = P.gated ? 8 : 16;
    auto seg_of = [&](int tile) {
        int s = 0;
        while (s + 1 < P.n_seg && tile >= P.seg[s + 1].tile0) ++s;
        return s;
    };
    int next = lo, l_stage = 0;
    auto load_tile = [&]() {
        if (next >= hi) return;
        if (lane == 0 && ok) {
            const int s = seg_of(next), row = (next - P.seg[s].tile0) * tile_rows, col = warp * NSB * (Q4K_BYTES / 4);
            const uint32_t bar = bars + 8 * l_stage, dst = ring + l_stage * G::SLOT;
            bar_expect(bar, G::SLOT);
            tma_2d(dst, &maps.one[s], col, row, bar);
            if (P.gated) tma_2d(dst + 8 * G::PITCH, &maps.one[1], col, row, bar);
        }
        ++next;
        if (++l_stage == P.stages) l_stage = 0;
    };
    for (int s = 0; s < P.stages; ++s) load_tile();
    pdl_wait();      // activations (and the output buffer) belong to the previous kernel until here

    // ---- the tokens of this warp's super-blocks: fragments and split sums.  A column past the last token repeats the
    // last one: columns do not mix, and it is never stored.  A super-block past the row's end (an odd number of them, two per
    // warp) is zero here and in the ring, whose tensor copies fill with zeros there.
    uint4 b[NSB][2][4][NT];
    uint2 sx[NSB][NT];
#pragma unroll
    for (int j = 0; j < NSB; ++j) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            const __half* xp = P.x + static_cast<int64_t>(min(8 * nt + g, P.M - 1)) * P.K + (warp * NSB + j) * QK_K + 64 * t;
#pragma unroll
            for (int p = 0; p < 2; ++p)
#pragma unroll
                for (int s = 0; s < 4; ++s)
                    b[j][p][s][nt] = NSB == 1 || warp * NSB + j < P.nsb ? ld_after_wait(xp + 32 * p + 8 * s)
                                                                        : make_uint4(0u, 0u, 0u, 0u);
        }
        float sum[(NT + 1) / 2][4];
#pragma unroll
        for (int i = 0; i < (NT + 1) / 2; ++i) sum[i][0] = sum[i][1] = sum[i][2] = sum[i][3] = 0.f;
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const uint32_t one = g == 2 * t + p ? 0x3C003C00u : 0u;
#pragma unroll
            for (int s = 0; s < 4; ++s)
#pragma unroll
                for (int n2 = 0; n2 < (NT + 1) / 2; ++n2) {
                    const uint4 u = b[j][p][s][2 * n2];
                    const uint4 v = 2 * n2 + 1 < NT ? b[j][p][s][2 * n2 + 1 < NT ? 2 * n2 + 1 : 0] : make_uint4(0u, 0u, 0u, 0u);
                    mma(sum[n2], u.x, v.x, u.y, v.y, one, one);
                    mma(sum[n2], u.z, v.z, u.w, v.w, one, one);
                }
        }
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) sx[j][nt] = split_sums(sum[nt >> 1][2 * (nt & 1)], sum[nt >> 1][2 * (nt & 1) + 1]);
    }

    uint32_t stage = 0, par = 0, buf = 0;
    for (int base = lo; base < hi; base += 2) {
        float* out = red + buf * (W * FixedRed<NT, W>::WARP) + warp * FixedRed<NT, W>::WARP;
#pragma unroll 1
        for (int q = 0; q < 2 && base + q < hi; ++q) {
            float acc[NT][4];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
            bar_wait(ok, bars + 8 * stage, par);
            const uint32_t rg = ring + stage * G::SLOT + g * G::PITCH, rh = rg + 8 * G::PITCH;
#pragma unroll
            for (int j = 0; j < NSB; ++j) tile_q4<NT, 2>(rg + j * Q4_PITCH, rh + j * Q4_PITCH, 0, b[j], sx[j], t, acc);
            __syncwarp();                           // all lanes have read the slot
            load_tile();
            if (++stage == static_cast<uint32_t>(P.stages)) {
                stage = 0;
                par ^= 1;
            }
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                float* at = out + (q * 8 * NT + 8 * nt + 2 * t) * RED_PITCH + g;
                at[0] = acc[nt][0];
                at[RED_PITCH] = acc[nt][1];
                at[8] = acc[nt][2];
                at[RED_PITCH + 8] = acc[nt][3];
            }
        }
        __syncthreads();
        for (int idx = threadIdx.x; idx < 2 * 16 * 8 * NT; idx += W * 32) {
            const int r = idx & 15, tok = (idx >> 4) % (8 * NT), q = idx / (16 * 8 * NT), tile = base + q;
            const float* at = red + buf * (W * FixedRed<NT, W>::WARP) + (q * 8 * NT + tok) * RED_PITCH + r;
            float v = 0.f;
#pragma unroll
            for (int w = 0; w < W; ++w) v += at[w * FixedRed<NT, W>::WARP];
            const float u = __shfl_down_sync(0xffffffffu, v, 8);             // gate/up: row r + 8 is the up row of row r
            if (tile >= hi || tok >= P.M || (P.gated && r >= 8)) continue;
            const Seg& sg = P.seg[seg_of(tile)];
            const int row = (tile - sg.tile0) * tile_rows + r;
            if (row >= sg.n_rows) continue;
            const int64_t to = static_cast<int64_t>(tok) * sg.ldy + row;
            __half y;
            if (P.gated) {
                y = __float2half_rn((P.act == ALLOYB_ACT_SILU ? act_silu(v) : act_gelu_tanh(v)) * u);
            } else {
                y = __float2half_rn(v);
                if (P.residual) y = __float2half_rn(__half2float(P.residual[to]) + __half2float(y));
            }
            static_cast<__half*>(sg.y)[to] = y;
        }
        buf ^= 1;
    }
    // a wait ran out: give copies that are still in flight time to land before the shared memory is released
    if (!ok)
        for (int i = 0; i < 2048; ++i) __nanosleep(512);
}

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                              const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeFn encoder() {
    static EncodeFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) != cudaSuccess ||
            qr != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<EncodeFn>(p);
    }();
    return fn;
}
static bool map2d(CUtensorMap* m, CUtensorMapDataType type, const void* base, uint64_t inner, uint64_t rows, uint64_t pitch,
                  uint32_t box_inner, uint32_t box_rows, CUtensorMapSwizzle swizzle) {
    const cuuint64_t gdim[2] = {inner, rows};
    const cuuint64_t gstr[1] = {pitch};
    const cuuint32_t box[2] = {box_inner, box_rows}, estr[2] = {1, 1};
    return encoder()(m, type, 2, const_cast<void*>(base), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int NT, int RT>
static int launch(const WeightSeg* seg, int n_mats, Params& P, cudaStream_t st) {
    using C = Cfg<NT>;
    static bool configured[64] = {};
    static int sm_count[64] = {};
    auto kern = linear_skinny_kernel<NT, RT>;
    constexpr int SMEM_MAX = 227 * 1024;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
    if (!configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sm_count[dev], cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) { set_cuda_error(e); return ALLOYB_E_CUDA; }
        configured[dev] = true;
    }
    // Row groups: as few (that is: as many K slices) as hold a CTA's tiles in one pass.  Token buffers: as many as leave two
    // stages of at least a tile in every ring.
    const int most = sm_count[dev], grid = P.n_tiles < most ? P.n_tiles : most, per_cta = (P.n_tiles + grid - 1) / grid;
    Maps maps = {};
    for (P.rs = 1;; P.rs *= 2) {
        P.ks = WARPS / P.rs;
        P.xd = P.rs == 1 ? 1 : 2;
        const int room = (SMEM_MAX - C::FIXED - P.ks * P.xd * C::X_BYTES) / WARPS;
        int least = RT;
        P.stage_bytes = 0;
        for (int i = 0; i < P.n_seg; ++i) {
            const int slot = 16 * (P.seg[i].q6 ? Q6_PITCH : Q4_PITCH), fit = room / (2 * slot);
            P.seg[i].n = fit < RT ? fit : RT;
            if (P.seg[i].n < least) least = P.seg[i].n;
            if (P.seg[i].n * slot > P.stage_bytes) P.stage_bytes = P.seg[i].n * slot;
        }
        if (least < 1) return ALLOYB_E_LIMIT;
        P.stages = room / P.stage_bytes < MAX_STAGES ? room / P.stage_bytes : MAX_STAGES;
        if (per_cta <= P.rs * least || P.rs == 4) {
            const int passes = (per_cta + P.rs * least - 1) / (P.rs * least);
            P.pass_tiles = (per_cta + passes - 1) / passes;
            for (int i = 0; i < P.n_seg; ++i) {          // a warp's usual share is one box
                const int share = P.pass_tiles / P.rs > 0 ? P.pass_tiles / P.rs : 1;
                P.seg[i].box = share < P.seg[i].n ? share : P.seg[i].n;
            }
            break;
        }
    }
    bool ok = map2d(&maps.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, P.x, P.K, P.M, static_cast<uint64_t>(P.K) * 2, C::ROW / 2, 8 * NT,
                    CU_TENSOR_MAP_SWIZZLE_64B);
    for (int i = 0; i < n_mats && ok; ++i) {
        const Seg& sg = P.seg[P.gated ? 0 : i];
        const int words = (sg.q6 ? Q6_PITCH : Q4_PITCH) / 4, rows = P.gated ? 8 : 16;
        for (int full = 0; full < 2 && ok; ++full)
            ok = map2d(full ? &maps.all[i] : &maps.one[i], CU_TENSOR_MAP_DATA_TYPE_UINT32, seg[i].data, seg[i].row_bytes / 4, seg[i].N,
                       seg[i].row_bytes, words, full ? rows * sg.box : rows, CU_TENSOR_MAP_SWIZZLE_NONE);
    }
    if (!ok) {
        set_cuda_error(cudaErrorInvalidValue);
        return ALLOYB_E_CUDA;
    }
    const cudaError_t e = launch_pdl(kern, dim3(grid), dim3(WARPS * 32), C::FIXED + P.ks * P.xd * C::X_BYTES + WARPS * P.stages * P.stage_bytes, st, maps, P);
    if (e != cudaSuccess) { set_cuda_error(e); return ALLOYB_E_CUDA; }
    return ALLOYB_OK;
}

template <int NT, int W, int NSB>
static int launch_fixed(const WeightSeg* seg, int n_mats, Params& P, cudaStream_t st) {
    using G = FixedGeom<NSB>;
    static bool configured[64] = {};
    static int sm_count[64] = {};
    // CTAs per SM: as many as leave a thread the 128 registers (two token groups of two super-blocks: 255) that its fragments
    // need.  28 KB are left to the first-level cache, through which the tokens come (K = 2048, 16 tokens, 4800 rows: 12.4 us
    // without, 9.1 with), unless that leaves no ring.
    constexpr int MINB = NT * NSB == 4 || W > 8 ? 1 : 16 / W;
    constexpr int FIXED = 128 + FixedRed<NT, W>::BYTES + FixedRed<NT, W>::BARS, SLOTS = W * G::SLOT;
    constexpr int FIT_CACHED = (200 * 1024 / MINB - 1024 - FIXED) / SLOTS, FIT_ALL = (228 * 1024 / MINB - 1024 - FIXED) / SLOTS;
    constexpr int FIT = FIT_CACHED >= 2 ? FIT_CACHED : FIT_ALL, STAGES = FIT < MAX_STAGES ? FIT : MAX_STAGES, SMEM = FIXED + STAGES * SLOTS;
    static_assert(FIT >= 2 && FixedRed<NT, W>::BYTES % 128 == 0 && G::SLOT % 256 == 0, "ring, and its 128-byte boundaries");
    auto kern = linear_skinny_fixed_kernel<NT, W, NSB, MINB>;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
    if (!configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sm_count[dev], cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) { set_cuda_error(e); return ALLOYB_E_CUDA; }
        configured[dev] = true;
    }
    // The tokens' way into the registers costs about three tiles' time, so whether it pays depends on the rounds of CTAs that the
    // tokens-as-columns kernel of linear_mma.cu needs (16 rows each, a gate/up pair 16 of both; two per SM at once).  One
    // round: that kernel (K = 4096, 8 tokens: 4096 rows 5.6 us, here 8.4; pair of 4000 7.9 / 11.3).  Two: this one (4800
    // rows, 8 tokens 9.5 / 9.4, 16 tokens 15.4 / 11.8), except from five to eight tokens in middling rows where the second
    // round is more than half full (8192 rows, 8 tokens: K = 2048 7.5 / 6.6, 4096 11.1 / 11.3, 6144 14.9 / 15.9, 8192 18.9 /
    // 17.5).  More: this one (14336 rows, K = 3072: 8 tokens 18.4 / 15.2, 16 tokens 29.9 / 16.9).
    const int sms = sm_count[dev], others = P.gated ? (P.seg[0].n_rows + 15) / 16 : P.n_tiles;
    if (others <= 2 * sms) return ALLOYB_NOT_TAKEN;
    if (P.M > 4 && P.M <= 8 && P.nsb > 8 && P.nsb < 28 && others > 3 * sms && others <= 4 * sms) return ALLOYB_NOT_TAKEN;
    // (seven warps with two token groups each spill: 8192 rows, K = 1792, 16 tokens 10.6 / 11.9, 14336 rows 33.6 / 21.2)
    if (NT == 2 && P.nsb == 7 && others <= 4 * sms) return ALLOYB_NOT_TAKEN;
    P.stages = STAGES;
    Maps maps = {};
    for (int i = 0; i < n_mats; ++i)             // (the row's words only: what pads its pitch reads as zero)
        if (!map2d(&maps.one[i], CU_TENSOR_MAP_DATA_TYPE_UINT32, seg[i].data, static_cast<uint64_t>(P.nsb) * (Q4K_BYTES / 4), seg[i].N,
                   seg[i].row_bytes, G::PITCH / 4, P.gated ? 8 : 16, CU_TENSOR_MAP_SWIZZLE_NONE)) {
            set_cuda_error(cudaErrorInvalidValue);
            return ALLOYB_E_CUDA;
        }
    const int most = MINB * sms, grid = P.n_tiles < most ? P.n_tiles : most;
    const cudaError_t e = launch_pdl(kern, dim3(grid), dim3(W * 32), SMEM, st, maps, P);
    if (e != cudaSuccess) { set_cuda_error(e); return ALLOYB_E_CUDA; }
    return ALLOYB_OK;
}
// One super-block per warp up to eight of them, two from there on.
template <int NT>
static int launch_fixed_rows(const WeightSeg* seg, int n_mats, Params& P, cudaStream_t st) {
    switch (P.nsb <= 8 ? P.nsb : 100 + (P.nsb + 1) / 2) {
        case 1: return launch_fixed<NT, 1, 1>(seg, n_mats, P, st);
        case 2: return launch_fixed<NT, 2, 1>(seg, n_mats, P, st);
        case 3: return launch_fixed<NT, 3, 1>(seg, n_mats, P, st);
        case 4: return launch_fixed<NT, 4, 1>(seg, n_mats, P, st);
        case 5: return launch_fixed<NT, 5, 1>(seg, n_mats, P, st);
        case 6: return launch_fixed<NT, 6, 1>(seg, n_mats, P, st);
        case 7: return launch_fixed<NT, 7, 1>(seg, n_mats, P, st);
        case 8: return launch_fixed<NT, 8, 1>(seg, n_mats, P, st);
        case 105: return launch_fixed<NT, 5, 2>(seg, n_mats, P, st);
        case 106: return launch_fixed<NT, 6, 2>(seg, n_mats, P, st);
        case 107: return launch_fixed<NT, 7, 2>(seg, n_mats, P, st);
        case 108: return launch_fixed<NT, 8, 2>(seg, n_mats, P, st);
    }
    if constexpr (NT == 1) {                     // (two token groups: the registers hold no more than that)
        switch ((P.nsb + 1) / 2) {
            case 9: return launch_fixed<1, 9, 2>(seg, n_mats, P, st);
            case 10: return launch_fixed<1, 10, 2>(seg, n_mats, P, st);
            case 11: return launch_fixed<1, 11, 2>(seg, n_mats, P, st);
            case 12: return launch_fixed<1, 12, 2>(seg, n_mats, P, st);
            case 13: return launch_fixed<1, 13, 2>(seg, n_mats, P, st);
            case 14: return launch_fixed<1, 14, 2>(seg, n_mats, P, st);
            case 15: return launch_fixed<1, 15, 2>(seg, n_mats, P, st);
            case 16: return launch_fixed<1, 16, 2>(seg, n_mats, P, st);
        }
    }
    return ALLOYB_NOT_TAKEN;
}

}  // namespace sk

// 2..SKINNY_MAX_M fp16 tokens against Q4_K / Q6_K matrices: up to MAX_SEGS row-stacked outputs, or a Q4_K gate/up pair with the
// activation fused.  NOT_TAKEN for anything else.
int try_linear_skinny(const void* x, int M, int K, int dtype, const WeightSeg* seg, int n_seg, bool gated, int act,
                      const void* residual, cudaStream_t st) {
    using namespace sk;
    if (M < 2 || M > SKINNY_MAX_M || dtype != ALLOYB_F16 || K % QK_K || n_seg < 1 || n_seg > MAX_SEGS) return ALLOYB_NOT_TAKEN;
    if (gated && (n_seg != 2 || seg[0].N != seg[1].N || seg[0].format != ALLOYB_Q4_K || seg[1].format != ALLOYB_Q4_K)) return ALLOYB_NOT_TAKEN;
    if (reinterpret_cast<uintptr_t>(x) % 16 || (residual && n_seg != 1)) return ALLOYB_NOT_TAKEN;
    const int nsb = K / QK_K, rows = gated ? 8 : 16;
    int64_t tiles = 0;
    bool any_q6 = false;
    Params P = {};
    for (int i = 0; i < n_seg; ++i) {
        const bool q6 = seg[i].format == ALLOYB_Q6_K;
        if ((!q6 && seg[i].format != ALLOYB_Q4_K) || seg[i].N <= 0) return ALLOYB_NOT_TAKEN;
        if (reinterpret_cast<uintptr_t>(seg[i].data) % 16 || seg[i].row_bytes % 16 ||
            seg[i].row_bytes < static_cast<int64_t>(nsb) * (q6 ? Q6K_BYTES : Q4K_BYTES))
            return ALLOYB_NOT_TAKEN;
        any_q6 |= q6;
        P.seg[i] = {seg[i].y, seg[i].ldy, seg[i].N, static_cast<int>(tiles), q6 ? 1 : 0, 1, 1};
        if (!gated || i == 0) tiles += (seg[i].N + rows - 1) / rows;
    }
    if (tiles > (1 << 26)) return ALLOYB_NOT_TAKEN;
    if (!encoder()) { set_cuda_error(cudaErrorNotSupported); return ALLOYB_E_CUDA; }
    P.x = static_cast<const __half*>(x);
    P.residual = static_cast<const __half*>(residual);
    P.n_seg = gated ? 1 : n_seg;
    P.n_tiles = static_cast<int>(tiles);
    P.M = M;
    P.K = K;
    P.nsb = nsb;
    P.gated = gated ? 1 : 0;
    P.act = act;
    if (M <= 16) {
        if (any_q6) return ALLOYB_NOT_TAKEN;
        return M <= 8 ? launch_fixed_rows<1>(seg, n_seg, P, st) : launch_fixed_rows<2>(seg, n_seg, P, st);
    }
    if (M <= 24) return launch<3, 4>(seg, n_seg, P, st);
    return launch<4, 4>(seg, n_seg, P, st);
}

int linear_skinny_device_error(int clear) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, sk::g_sk_error, sizeof(int)) != cudaSuccess) return 0;
    if (clear && v) {
        const int z = 0;
        cudaMemcpyToSymbol(sk::g_sk_error, &z, sizeof(int));
    }
    return v;
}

}  // namespace alloyb
