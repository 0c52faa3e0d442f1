// Q8_0 dequant-GEMV for 1..4 tokens per pass (more tokens: more passes), plain and gate/up fused.  (One token and K from
// 4096 to 16384: q8_gemv_one_kernel, further down.)
//
// Weights arrive in the reference's normalised pair (server/gguf/quant.py:497-521): int8 codes
// (N, K) and fp16 scales (N, K/32), w = scale * code; 1.0625 bytes per weight, so the kernel is a
// pure streaming problem like the Q4_K / Q6_K GEMVs, and follows the reference kernel's plan
// (metal/std/quant.py:61-273: split K over the lanes, several rows per SIMD group):
//
//   * a CTA stages the tokens in shared memory once; a warp owns four consecutive weight rows (two
//     of each matrix for a gate/up pair) and the 32 lanes split K: per step a lane takes 16 codes of
//     every row (one 128-bit load per row, all inside one 32-element block, so one scale per row)
//     against 16 activations it converts to fp32 once and reuses for the rows; the loads of the
//     next step are issued before the current one is computed, which keeps ~64 KB in flight per SM;
//   * int8 -> fp32 without the conversion pipe: the byte goes into the mantissa of 2^23 (one PRMT),
//     minus 2^23 + 128 (one FADD, exact); products accumulate in fp32 per block and the block's
//     scale multiplies the partial sum -- the factored form the reference uses;
//   * rows are reduced with warp shuffles; the gate/up variant keeps both sums and applies the
//     activation in the epilogue (metal/std/quant.py:358-695).
#include "linear.cuh"
#include "linear_rows.cuh"

namespace alloyb {
namespace q8 {

constexpr int WARPS = 8;
constexpr int ROWS = 4;              // row loads per warp and step: 4 rows, or 2 rows of gate + 2 of up
constexpr int MT = 4;                // tokens per pass

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}
// the four int8 codes of a word as floats
__device__ __forceinline__ void codes4(uint32_t w, float (&c)[4]) {
    const uint32_t u = w ^ 0x80808080u;                           // code + 128, unsigned
    constexpr uint32_t MAGIC = 0x4B000000u;                       // 2^23: the byte lands in the mantissa
    c[0] = __uint_as_float(prmt(u, MAGIC, 0x7650u)) - 8388736.0f;
    c[1] = __uint_as_float(prmt(u, MAGIC, 0x7651u)) - 8388736.0f;
    c[2] = __uint_as_float(prmt(u, MAGIC, 0x7652u)) - 8388736.0f;
    c[3] = __uint_as_float(prmt(u, MAGIC, 0x7653u)) - 8388736.0f;
}

struct Params {
    const void* x;                   // (M, K) activations
    int M, K, N;
    const int8_t* w[2];              // [gate | up] or [w | -]
    const __half* s[2];
    void* y;                         // (M, N)
    int64_t ldy;
    const void* residual;            // plain only
    int act;
    int constant;                    // codes and scales do not depend on earlier launches
};

// MTOK: tokens per pass (1: the decode case, light enough on registers for two CTAs per SM; 4)
template <typename XT, bool GATED, int MTOK>
__global__ void __launch_bounds__(WARPS * 32, MTOK == 1 ? 2 : 1) q8_gemv_kernel(const Params P) {
    constexpr int MT = MTOK;
    pdl_launch_dependents();
    extern __shared__ __align__(16) uint8_t smem_raw[];
    XT* xs = reinterpret_cast<XT*>(smem_raw);                     // [M][K]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int NM = GATED ? 2 : 1, R = ROWS / NM;
    const int row0 = (blockIdx.x * WARPS + warp) * R;
    const int K = P.K, M = P.M, nblk = K / Q8_BLOCK;
    pdl_wait();
    for (int i = threadIdx.x * 8; i < M * K; i += WARPS * 32 * 8)
        *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(xs) + static_cast<size_t>(i) * sizeof(XT)) =
            *reinterpret_cast<const uint4*>(static_cast<const uint8_t*>(P.x) + static_cast<size_t>(i) * sizeof(XT));
    if (sizeof(XT) == 4)                                          // fp32: the second half of each 8-element group
        for (int i = threadIdx.x * 8 + 4; i < M * K; i += WARPS * 32 * 8)
            *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(xs) + static_cast<size_t>(i) * 4) =
                *reinterpret_cast<const uint4*>(static_cast<const uint8_t*>(P.x) + static_cast<size_t>(i) * 4);
    __syncthreads();
    if (row0 >= P.N) return;
    float acc[NM][R][MT];
#pragma unroll
    for (int a = 0; a < NM; ++a)
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int m = 0; m < MT; ++m) acc[a][r][m] = 0.f;
    const int8_t* wrow[NM][R];
    const __half* srow[NM][R];
#pragma unroll
    for (int a = 0; a < NM; ++a)
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int row = min(row0 + r, P.N - 1);               // tail rows re-read the last row
            wrow[a][r] = P.w[a] + static_cast<int64_t>(row) * K;
            srow[a][r] = P.s[a] + static_cast<int64_t>(row) * nblk;
        }
    uint4 cw[NM][R], nw[NM][R];
    float sc[NM][R], ns[NM][R];
    auto load = [&](int k0, uint4 (&c)[NM][R], float (&s)[NM][R]) {
#pragma unroll
        for (int a = 0; a < NM; ++a)
#pragma unroll
            for (int r = 0; r < R; ++r) {
                c[a][r] = __ldg(reinterpret_cast<const uint4*>(wrow[a][r] + k0));
                s[a][r] = __half2float(__ldg(srow[a][r] + k0 / Q8_BLOCK));
            }
    };
    load(lane * 16, cw, sc);
    for (int k0 = lane * 16; k0 < K; k0 += 32 * 16) {
        const bool more = k0 + 32 * 16 < K;
        if (more) load(k0 + 32 * 16, nw, ns);                     // in flight while this step is computed
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            if (m >= M) break;
            float xf[16];
            const XT* xr = xs + static_cast<size_t>(m) * K + k0;
#pragma unroll
            for (int e = 0; e < 16; ++e) xf[e] = to_f32<XT>(xr[e]);
#pragma unroll
            for (int a = 0; a < NM; ++a)
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const uint32_t wv[4] = {cw[a][r].x, cw[a][r].y, cw[a][r].z, cw[a][r].w};
                    float part = 0.f;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        float c[4];
                        codes4(wv[q], c);
#pragma unroll
                        for (int e = 0; e < 4; ++e) part = fmaf(xf[4 * q + e], c[e], part);
                    }
                    acc[a][r][m] = fmaf(sc[a][r], part, acc[a][r][m]);
                }
        }
        if (more) {
#pragma unroll
            for (int a = 0; a < NM; ++a)
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    cw[a][r] = nw[a][r];
                    sc[a][r] = ns[a][r];
                }
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            if (m >= M) break;
            const float v = warp_sum(acc[0][r][m]);
            const float u = GATED ? warp_sum(acc[NM - 1][r][m]) : 0.f;
            if (lane == 0 && row0 + r < P.N) {
                const int64_t o = static_cast<int64_t>(m) * P.ldy + row0 + r;
                XT* y = static_cast<XT*>(P.y);
                if (GATED) {
                    const float a = (P.act == ALLOYB_ACT_SILU) ? act_silu(v) : act_gelu_tanh(v);
                    y[o] = from_f32<XT>(a * u);
                } else {
                    XT out = from_f32<XT>(v);
                    if (P.residual) out = from_f32<XT>(to_f32<XT>(static_cast<const XT*>(P.residual)[o]) + to_f32<XT>(out));
                    y[o] = out;
                }
            }
        }
}

// ---- one token, K up to 16384: the token stays in registers.
//
// The kernel above spends its time on instructions (4.4 per code: activations converted again for every four rows) and on
// its waves (14336 gate/up rows: 896 CTAs, 3.03 waves of 296).  Here the eight warps of a CTA split K -- a lane keeps its 16
// activations of up to NS 512-wide slices as fp32 pairs for the whole launch -- and walk the CTA's share of the rows
// together, RB rows (or gate and up rows) at a time with the next step's loads in flight.  Codes become fp32 pairs by two
// byte permutes and the two-wide add, products run on the two-wide FMA: 9 instructions per four codes.  The lanes' sums of
// RB rows are folded together (9 shuffles for 8 rows); the warps' sums meet in shared memory once, at the end.
__device__ __forceinline__ uint64_t pair(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
constexpr int SLICE = 512;           // 32 lanes x 16 codes
constexpr int MAX_SLICES = 4;        // per warp

template <typename XT, bool GATED, int NS, int RB>
__global__ void __launch_bounds__(WARPS * 32, 2) q8_gemv_one_kernel(const Params P) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) float part[];                 // [row of the CTA][matrix][warp]
    constexpr int NM = GATED ? 2 : 1, R = RB / NM;                // rows of each matrix per step
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int K = P.K, nblk = K / Q8_BLOCK, slices = K / SLICE;
    const int units = (P.N + R - 1) / R;
    const int u0 = static_cast<int>(static_cast<int64_t>(units) * blockIdx.x / gridDim.x);
    const int u1 = static_cast<int>(static_cast<int64_t>(units) * (blockIdx.x + 1) / gridDim.x);
    const int mine = (slices - warp + WARPS - 1) / WARPS;         // this warp's slices: warp, warp + 8, ...

    struct Step {
        uint4 c[RB];
        __half s[RB];
    };
    // step i: rows u0 * R + (i / NS) * R .., slice i % NS (of `mine`; the others are skipped)
    auto load = [&](int unit, int sl, Step& o) {
        const int k = (warp + sl * WARPS) * SLICE + lane * 16;
#pragma unroll
        for (int a = 0; a < NM; ++a)
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int64_t row = min(unit * R + r, P.N - 1);   // tail rows re-read the last row
                o.c[a * R + r] = __ldg(reinterpret_cast<const uint4*>(P.w[a] + row * K + k));
                o.s[a * R + r] = __ldg(P.s[a] + row * nblk + k / Q8_BLOCK);
            }
    };
    if (!P.constant) pdl_wait();                                  // a launch before this one may have written codes or scales
    Step even, odd;
    if (u0 < u1 && mine > 0) load(u0, 0, even);
    pdl_wait();
    uint64_t x[NS][8];
#pragma unroll
    for (int sl = 0; sl < NS; ++sl) {
        const XT* xp = static_cast<const XT*>(P.x) + (warp + (sl < mine ? sl : 0) * WARPS) * SLICE + lane * 16;
        alignas(16) XT v[16];
#pragma unroll
        for (int q = 0; q < 16 * static_cast<int>(sizeof(XT)) / 16; ++q)
            reinterpret_cast<uint4*>(v)[q] = mine > 0 ? ld_after_wait(reinterpret_cast<const uint4*>(xp) + q) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int e = 0; e < 8; ++e) x[sl][e] = pair(to_f32<XT>(v[2 * e]), to_f32<XT>(v[2 * e + 1]));
    }
    const uint64_t unbias = pair(-8388736.0f, -8388736.0f);      // -(2^23 + 128)
    float acc[RB];
    auto compute = [&](const Step& o, const uint64_t (&xs)[8], bool first) {
#pragma unroll
        for (int j = 0; j < RB; ++j) {
            const uint32_t wv[4] = {o.c[j].x, o.c[j].y, o.c[j].z, o.c[j].w};
            uint64_t sum = pair(0.f, 0.f);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t u = wv[q] ^ 0x80808080u;
                constexpr uint32_t MAGIC = 0x4B000000u;
                sum = fma2(add2(pair(__uint_as_float(prmt(u, MAGIC, 0x7650u)), __uint_as_float(prmt(u, MAGIC, 0x7651u))), unbias), xs[2 * q], sum);
                sum = fma2(add2(pair(__uint_as_float(prmt(u, MAGIC, 0x7652u)), __uint_as_float(prmt(u, MAGIC, 0x7653u))), unbias), xs[2 * q + 1], sum);
            }
            float a, b;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(sum));
            acc[j] = fmaf(__half2float(o.s[j]), a + b, first ? 0.f : acc[j]);
        }
    };
    auto finish = [&](int unit) {
        // fold: after the steps with lane distance 16, 8, (4) a lane holds one row's sum over its lane group
        float v[RB];
#pragma unroll
        for (int j = 0; j < RB; ++j) v[j] = acc[j];
        int idx = 0;
#pragma unroll
        for (int h = RB / 2, d = 16; h >= 1; h /= 2, d /= 2) {
            const bool up = (lane & d) != 0;
            idx = idx * 2 + (up ? 1 : 0);
#pragma unroll
            for (int j = 0; j < h; ++j) {
                const float give = up ? v[j] : v[j + h], keep = up ? v[j + h] : v[j];
                v[j] = keep + __shfl_xor_sync(0xffffffffu, give, d);
            }
        }
        constexpr int LEFT = 32 / RB;                             // lanes that share a row
#pragma unroll
        for (int d = LEFT / 2; d >= 1; d /= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], d);
        if ((lane & (LEFT - 1)) == 0) part[((unit - u0) * RB + idx) * WARPS + warp] = v[0];
    };
    // (every warp has work: slices >= WARPS, see the caller)
    const int steps = (u1 - u0) * mine;
    int unit = u0, sl = 0, l_unit = u0, l_sl = 0;
    auto advance = [&](int& un, int& s) {
        if (++s == mine) {
            s = 0;
            ++un;
        }
    };
    auto run = [&](Step& cur, Step& next, bool more) {
        advance(l_unit, l_sl);
        if (more) load(l_unit, l_sl, next);                       // in flight while this step is computed
        if (NS == 1) {
            compute(cur, x[0], true);
        } else {
#pragma unroll
            for (int s = 0; s < NS; ++s)
                if (s == sl) compute(cur, x[s], s == 0);
        }
        if (sl == mine - 1) finish(unit);
        advance(unit, sl);
    };
    for (int i = 0; i < steps; i += 2) {
        run(even, odd, i + 1 < steps);
        if (i + 1 < steps) run(odd, even, i + 2 < steps);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < (u1 - u0) * R; i += WARPS * 32) {
        const int un = i / R, r = i - un * R, row = (u0 + un) * R + r;
        if (row >= P.N) continue;
        float v = 0.f, u = 0.f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            v += part[(un * RB + r) * WARPS + w];
            if (GATED) u += part[(un * RB + R + r) * WARPS + w];
        }
        XT* y = static_cast<XT*>(P.y);
        if (GATED) {
            const float a = (P.act == ALLOYB_ACT_SILU) ? act_silu(v) : act_gelu_tanh(v);
            y[row] = from_f32<XT>(a * u);
        } else {
            XT out = from_f32<XT>(v);
            if (P.residual) out = from_f32<XT>(to_f32<XT>(static_cast<const XT*>(P.residual)[row]) + to_f32<XT>(out));
            y[row] = out;
        }
    }
}

template <typename XT, bool GATED, int NS, int RB>
static int launch_one_ns(const Params& P, cudaStream_t st) {
    static bool configured[64] = {};
    static int sm_count[64] = {};
    auto kern = q8_gemv_one_kernel<XT, GATED, NS, RB>;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
    if (!configured[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sm_count[dev], cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) { set_cuda_error(e); return ALLOYB_E_CUDA; }
        configured[dev] = true;
    }
    const int units = (P.N + RB / (GATED ? 2 : 1) - 1) / (RB / (GATED ? 2 : 1));
    const int grid = units < 2 * sm_count[dev] ? units : 2 * sm_count[dev];
    const size_t smem = static_cast<size_t>((units + grid - 1) / grid) * RB * WARPS * 4;
    if (smem > 100 * 1024) return ALLOYB_NOT_TAKEN;
    const cudaError_t e = launch_pdl(kern, dim3(grid), dim3(WARPS * 32), smem, st, P);
    if (e != cudaSuccess) { set_cuda_error(e); return ALLOYB_E_CUDA; }
    return check_launch();
}
// Every warp has at least one slice from K = 4096 on; one slice each leaves the registers for eight rows at a time.
template <typename XT, bool GATED>
static int launch_one(const Params& P, cudaStream_t st) {
    const int slices = P.K / SLICE, ns = (slices + WARPS - 1) / WARPS;
    if (slices < WARPS || ns > MAX_SLICES) return ALLOYB_NOT_TAKEN;
    switch (ns) {
        case 1: return launch_one_ns<XT, GATED, 1, 8>(P, st);
        case 2: return launch_one_ns<XT, GATED, 2, 4>(P, st);
        default: return launch_one_ns<XT, GATED, 4, 4>(P, st);
    }
}

template <typename XT, bool GATED, int MTOK>
static int launch_m(const Params& P, cudaStream_t st) {
    static bool configured[64] = {};
    auto kern = q8_gemv_kernel<XT, GATED, MTOK>;
    const size_t smem = static_cast<size_t>(P.M) * P.K * sizeof(XT);
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
    if (!configured[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        if (e != cudaSuccess) { set_cuda_error(e); return ALLOYB_E_CUDA; }
        configured[dev] = true;
    }
    constexpr int rows_per_cta = WARPS * ROWS / (GATED ? 2 : 1);
    const int blocks = (P.N + rows_per_cta - 1) / rows_per_cta;
    const cudaError_t e = launch_pdl(kern, dim3(blocks), dim3(WARPS * 32), smem, st, P);
    if (e != cudaSuccess) { set_cuda_error(e); return ALLOYB_E_CUDA; }
    return check_launch();
}

template <typename XT, bool GATED>
static int launch(const Params& P, cudaStream_t st) {
    if (P.M == 1) {
        const int rc = launch_one<XT, GATED>(P, st);
        return rc == ALLOYB_NOT_TAKEN ? launch_m<XT, GATED, 1>(P, st) : rc;
    }
    return launch_m<XT, GATED, MT>(P, st);
}

}  // namespace q8

// M tokens against one or two (gate/up) Q8_0 matrices; NOT_TAKEN when the shape or alignment is
// outside the kernel (the row kernels then serve it).  More than four tokens run as passes of four.
int try_q8_gemv(const void* x, int M, int K, int dtype, const void* w0, const void* s0, const void* w1, const void* s1,
                void* y, int N, int64_t ldy, const void* residual, bool gated, int act, bool constant, cudaStream_t st) {
    if (M < 1 || M >= 64 || K % 512 || N < 1) return ALLOYB_NOT_TAKEN;
    const size_t esz = dtype == ALLOYB_F32 ? 4 : 2;
    if (static_cast<size_t>(q8::MT) * K * esz > 190 * 1024) return ALLOYB_NOT_TAKEN;
    if (reinterpret_cast<uintptr_t>(x) % 16 || reinterpret_cast<uintptr_t>(w0) % 16 || (gated && reinterpret_cast<uintptr_t>(w1) % 16))
        return ALLOYB_NOT_TAKEN;
    for (int m0 = 0; m0 < M; m0 += q8::MT) {
        q8::Params P;
        P.x = static_cast<const uint8_t*>(x) + static_cast<size_t>(m0) * K * esz;
        P.M = M - m0 < q8::MT ? M - m0 : q8::MT;
        P.K = K;
        P.N = N;
        P.w[0] = static_cast<const int8_t*>(w0);
        P.s[0] = static_cast<const __half*>(s0);
        P.w[1] = static_cast<const int8_t*>(gated ? w1 : w0);
        P.s[1] = static_cast<const __half*>(gated ? s1 : s0);
        P.y = static_cast<uint8_t*>(y) + static_cast<size_t>(m0) * ldy * esz;
        P.ldy = ldy;
        P.residual = residual ? static_cast<const uint8_t*>(residual) + static_cast<size_t>(m0) * ldy * esz : nullptr;
        P.act = act;
        P.constant = constant ? 1 : 0;
        int rc;
        if (dtype == ALLOYB_F16) rc = gated ? q8::launch<__half, true>(P, st) : q8::launch<__half, false>(P, st);
        else if (dtype == ALLOYB_BF16) rc = gated ? q8::launch<__nv_bfloat16, true>(P, st) : q8::launch<__nv_bfloat16, false>(P, st);
        else if (dtype == ALLOYB_F32) rc = gated ? q8::launch<float, true>(P, st) : q8::launch<float, false>(P, st);
        else return ALLOYB_E_DTYPE;
        if (rc != ALLOYB_OK) return rc;
    }
    return ALLOYB_OK;
}

}  // namespace alloyb
