// The prompt of the plain decoder in one pass over the weights: the tokens of a chunk go through a layer together, with
// the float order of the one-token step (wd_dense_decoder.cuh) kept per token, so that caches, logits and tokens are
// bit-identical to feeding the prompt token by token.
//
// What the step spends per prompt token is one read of every matrix and 82 dependent launches (300 us on the
// 16-layer benchmark model, 400 with 500 positions in the cache). Here a chunk of up to 512 tokens shares both.
#pragma once

#include "wd_dense_decoder.cuh"

namespace wd {

constexpr int kPrefillChunk = 512;      // tokens per pass at most (workspace: about 100 KB per token at ffn 8192)

// The quantised activations [token][n] of a chunk, in one of two orders. tile = 0: rows of PairedQuant, scales [token][n / 32]
// (prefill_gemm_kernel). tile > 0: the B operand of prompt_tc_gemm_kernel: per `tile` tokens and block (in entry order: block 32 t + l at
// bitrev(l) * n_t + t) a record of 8-token x 16-byte matrices, the first half of the block and then the second, and the tokens' scales.
struct PromptAct {
    uint8_t *q;
    float *d;
    int n, tile;
    __device__ __forceinline__ uint8_t *record(int m, int b) const {
        const int n_t = (n + 1023) >> 10, e = static_cast<int>(__brev(static_cast<unsigned>(b) & 31u) >> 27) * n_t + (b >> 5);
        return q + (static_cast<size_t>(m / tile) * 32 * n_t + e) * (tile * 36);
    }
    // where value e (a multiple of four) of token m goes, with the three behind it: in rows, in tiles
    __device__ __forceinline__ uint8_t *row_quad(int m, int e) const { return q + m * n + (e & ~31) + paired_place(e & 31); }       // fewer than 2^31 bytes
    __device__ __forceinline__ uint8_t *tile_quad(int m, int e) const {
        const int c = m % tile;
        return record(m, e >> 5) + (e >> 4 & 1) * (tile * 16) + (c >> 3) * 128 + (c & 7) * 16 + (e & 15);
    }
    __device__ __forceinline__ float *row_scale(int m, int b) const { return d + m * (n >> 5) + b; }
    __device__ __forceinline__ float *tile_scale(int m, int b) const { return reinterpret_cast<float *>(record(m, b) + tile * 32) + m % tile; }
};

// RMSNorm + Q8_0 of every token of the chunk, one CTA per token; the body is the one-token kernel's.
__global__ void __launch_bounds__(1024) prefill_norm_quant_kernel(float *hidden, const float *proj, const float *w, int n, float eps,
                                                                 PromptAct x, const uint8_t *embd, const int *tokens, int vocab,
                                                                 int embd_q8) {
    grid_dep_launch();
    const size_t m = blockIdx.x;
    float *h = hidden + m * n;
    const NormInput in = {h, proj != nullptr ? proj + m * n : nullptr, w, embd != nullptr || proj != nullptr ? h : nullptr, embd, tokens + m, eps,
                          n, vocab, embd_q8};
    dense_norm_quant_body<1>(in, [] { grid_dep_wait(); }, [&](int e, uint32_t packed, float d) {
        *reinterpret_cast<uint32_t *>(x.tile == 0 ? x.row_quad(blockIdx.x, e) : x.tile_quad(blockIdx.x, e)) = packed;
        if ((e & 31) == 0) *(x.tile == 0 ? x.row_scale(blockIdx.x, e >> 5) : x.tile_scale(blockIdx.x, e >> 5)) = d;
    });
}

// ---- Y[m][row] = W[row] . X[m] for the tokens of a chunk: short prompts, short rows (the others: wd_dense_prompt_tc.cuh) ----
// The one-token order is: lane l of 32 runs one fmaf(d_w * d_x, (float)int_dot, acc) per block b = l, l + 32, ... ascending,
// then the butterfly ^16 ^8 ^4 ^2 ^1. The integer dot of one block is a contraction of depth 32, i.e. exactly one
// mma.m16n8k32 (s8) for 16 rows x 8 tokens; it cannot be accumulated over blocks, because every block is scaled by its own
// d_w * d_x in float. That float side (packed subtract, multiply and fmaf, two of each per lane and tile), the expansion
// of the nibbles and the staging are what the kernel issues. The form on halves (two m16n8k16 per block, the sums exact as
// well, no conversion afterwards) measured 10 % slower: its operands take twice the shared memory and more instructions.
//
// A warp owns 16 rows, 8 * NT tokens and one residue c = l mod 4 of the lanes: ^16, ^8 and ^4 pair lanes of one residue,
// so it walks the lanes l = 4 x + c with x in bit-reversed order and folds the finished lane sums with a three-deep stack;
// the four residues meet in shared memory at the end ((c0 + c2) + (c1 + c3)). A stage of the copy pipeline holds, for
// every row and token, the four neighbouring blocks 32 t + 4 x + {0..3} of two values of t.
__device__ __forceinline__ void cp_async8(void *dst, const void *src, int bytes) {     // the rest of the eight bytes is zeroed
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async4(void *dst, const void *src, bool live) {
    const int bytes = live ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}
// The integer accumulator starts at the bit pattern of 12582912.0f = 1.5 * 2^23: for |sum| < 2^22 the result read as a float
// is 12582912 + sum, and one exact subtraction gives (float)sum. Sums here stay below 2^20.
constexpr int kMagicBits = 0x4b400000;
constexpr float kMagic = 12582912.0f;
__device__ __forceinline__ void mma_s8(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    int i[4];
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=r"(i[0]), "=r"(i[1]), "=r"(i[2]), "=r"(i[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(kMagicBits));
#pragma unroll
    for (int k = 0; k < 4; ++k) d[k] = __int_as_float(i[k]);
}

// Shared-memory plan of one stage (TC = 2 values of t, four blocks each). The pads put the rows (or tokens) of a
// fragment into different banks.
template <bool Q8, int RG, int NT>
struct PrefillGemm {
    static constexpr int kTc = 2, kRows = 16 * RG, kTok = 8 * NT, kThreads = 128 * RG;
    static constexpr int kBlk = Q8 ? 32 : 16;
    static constexpr int kWStride = kTc * 4 * kBlk + 16, kXStride = kTc * 4 * 32 + 32;
    static constexpr int kDwStride = kTc * 4 * 2 + 8, kDxStride = kTok * 4;     // d_x: [block][token]
    static constexpr int kOffX = kRows * kWStride, kOffDw = kOffX + kTok * kXStride, kOffDx = kOffDw + kRows * kDwStride;
    static constexpr int kStage = (kOffDx + kTc * 4 * kDxStride + 127) / 128 * 128;
    static constexpr int kRed = 4 * kTok * (kRows + 4) * 4;              // the residues' sums, after the last stage
    // few tokens: the weights are all there is to stream, so more of them travel
    static constexpr int kDeep = NT == 4 ? 4 : NT == 2 ? 8 : 12, kFit = 200 * 1024 / kStage;
    static constexpr int kStages = kDeep < kFit ? kDeep : kFit;
    static constexpr int kSmem = kStages * kStage > kRed ? kStages * kStage : kRed;
};

template <bool Q8, int RG, int NT>
__global__ void __launch_bounds__(128 * RG) prefill_gemm_kernel(const uint8_t *wp, int rows, int nb, const PairedQuant *xq, const float *xd, int m_tokens,
                                                               float *y) {
    using G = PrefillGemm<Q8, RG, NT>;
    extern __shared__ __align__(128) uint8_t gsm[];
    grid_dep_launch();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int res = warp & 3, rg = warp >> 2, g = lane >> 2, q = lane & 3;
    const int row0 = blockIdx.x * G::kRows, tok0 = blockIdx.y * G::kTok;
    const uint8_t *q_all = wp;
    const int nbp = dense_row_stride(nb);
    const uint16_t *d_all = reinterpret_cast<const uint16_t *>(wp + static_cast<size_t>(rows) * nbp * G::kBlk);
    const int n_t = (nb + 31) >> 5, n_tc = (n_t + G::kTc - 1) / G::kTc, n_stage = 8 * n_tc;
    auto bitrev3 = [](int j) { return ((j & 1) << 2) | (j & 2) | ((j >> 2) & 1); };
    // position of a producer in the sequence of stages: slot in the ring, first block of the stage
    struct Cursor {
        int slot = 0, j = 0, tc = 0;
    };
    auto base_of = [&](const Cursor &c) { return 32 * G::kTc * c.tc + 4 * bitrev3(c.j); };
    auto advance = [&](Cursor &c) {
        if (++c.slot == G::kStages) c.slot = 0;
        if (++c.tc == n_tc) {
            c.tc = 0;
            ++c.j;
        }
    };
    auto issue_w = [&](const Cursor &c) {
        uint8_t *st = gsm + c.slot * G::kStage;
        const int b0 = base_of(c);
        constexpr int kPer = G::kTc * 4 * (G::kBlk / 16);       // 16-byte pieces of a row
#pragma unroll
        for (int i = 0; i < G::kRows * kPer / G::kThreads; ++i) {
            const int e = tid + i * G::kThreads, r = e / kPer, p = e % kPer, k = p / (G::kBlk / 16), h = p % (G::kBlk / 16);
            const int b = b0 + 32 * (k >> 2) + (k & 3);
            const bool live = row0 + r < rows && b < nb;
            cp_async16(st + r * G::kWStride + p * 16, live ? q_all + static_cast<size_t>((row0 + r) * nbp + b) * G::kBlk + h * 16 : q_all, live);
        }
        if (tid < G::kRows * G::kTc) {      // four scales of a row (zero past its end, so a missing block adds nothing)
            const int r = tid / G::kTc, k = tid % G::kTc, b = b0 + 32 * k;
            const bool live = row0 + r < rows && b < nb;
            cp_async8(st + G::kOffDw + r * G::kDwStride + k * 8, live ? d_all + static_cast<size_t>(row0 + r) * nbp + b : d_all,
                      live ? 2 * min(4, nb - b) : 0);
        }
    };
    auto issue_x = [&](const Cursor &c) {
        uint8_t *st = gsm + c.slot * G::kStage;
        const int b0 = base_of(c);
        constexpr int kPer = G::kTc * 4 * 2;
#pragma unroll
        for (int i = 0; i < (G::kTok * kPer + G::kThreads - 1) / G::kThreads; ++i) {
            const int e = tid + i * G::kThreads, r = e / kPer, p = e % kPer, b = b0 + 32 * (p >> 3) + ((p >> 1) & 3);
            const bool live = tok0 + r < m_tokens && b < nb;
            if (G::kTok * kPer >= G::kThreads || e < G::kTok * kPer)
                cp_async16(st + G::kOffX + r * G::kXStride + p * 16,
                           live ? xq + static_cast<size_t>((tok0 + r) * nb + b) * 32 + (p & 1) * 16 : xq, live);
        }
#pragma unroll
        for (int e = tid; e < G::kTok * G::kTc * 4; e += G::kThreads) {
            const int r = e / (G::kTc * 4), k = e % (G::kTc * 4), b = b0 + 32 * (k >> 2) + (k & 3);
            const bool live = tok0 + r < m_tokens && b < nb;
            cp_async4(st + G::kOffDx + k * G::kDxStride + r * 4, live ? xd + static_cast<size_t>(tok0 + r) * nb + b : xd, live);
        }
    };
    static_assert(G::kRows * G::kTc <= G::kThreads, "one piece of the scales per thread and stage");

    // the weights do not depend on the kernel before this one: the first stages' rows leave before the wait for it
    Cursor cw, cx;
    for (int s = 0; s < G::kStages - 1; ++s)
        if (s < n_stage) {
            issue_w(cw);
            advance(cw);
        }
    grid_dep_wait();
    for (int s = 0; s < G::kStages - 1; ++s) {
        if (s < n_stage) {
            issue_x(cx);
            advance(cx);
        }
        cp_async_commit();
    }
    f32x2 acc[NT][2], s0[NT][2], s1[NT][2], s2[NT][2];      // (token 2 q, token 2 q + 1) of row g, then of row g + 8
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 2; ++i) acc[n][i] = s0[n][i] = s1[n][i] = s2[n][i] = 0ull;
    const f32x2 unmagic = pack2(-kMagic, -kMagic);
    int slot = 0, left = n_stage - (G::kStages - 1);        // stages still to be requested
    const uint8_t *wbase = gsm + (rg * 16 + g) * G::kWStride, *xbase = gsm + G::kOffX + g * G::kXStride + q * 8;
    const uint8_t *dwbase = gsm + G::kOffDw + (rg * 16 + g) * G::kDwStride, *dxbase = gsm + G::kOffDx + 8 * q;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
#pragma unroll 1
        for (int tc = 0; tc < n_tc; ++tc) {
        cp_async_wait<G::kStages - 2>();
        __syncthreads();            // this stage has landed for everyone; the slot of the one before is free
        if (left > 0) {
            --left;
            issue_w(cw);
            issue_x(cw);
            advance(cw);
        }
        cp_async_commit();
        const int so = slot * G::kStage;
        if (++slot == G::kStages) slot = 0;
        const uint8_t *wrow = wbase + so, *xrow = xbase + so, *dwr = dwbase + so, *dxr = dxbase + so;
#pragma unroll
        for (int t = 0; t < G::kTc; ++t) {
            const int k = t * 4 + res;
            uint32_t a[4];
            if constexpr (Q8) {
                a[0] = *reinterpret_cast<const uint32_t *>(wrow + k * 32 + q * 4);
                a[1] = *reinterpret_cast<const uint32_t *>(wrow + 8 * G::kWStride + k * 32 + q * 4);
                a[2] = *reinterpret_cast<const uint32_t *>(wrow + k * 32 + 16 + q * 4);
                a[3] = *reinterpret_cast<const uint32_t *>(wrow + 8 * G::kWStride + k * 32 + 16 + q * 4);
            } else {        // a nibble at the top of its byte with the top bit flipped is 16 * (q - 8)
                const uint32_t w0 = *reinterpret_cast<const uint32_t *>(wrow + k * 16 + q * 4);
                const uint32_t w1 = *reinterpret_cast<const uint32_t *>(wrow + 8 * G::kWStride + k * 16 + q * 4);
                a[0] = ((w0 << 4) & 0xf0f0f0f0u) ^ 0x80808080u;
                a[1] = ((w1 << 4) & 0xf0f0f0f0u) ^ 0x80808080u;
                a[2] = (w0 & 0xf0f0f0f0u) ^ 0x80808080u;
                a[3] = (w1 & 0xf0f0f0f0u) ^ 0x80808080u;
            }
            // d_w carries the 1/16 of a Q4_0 sum (a power of two: exact)
            const float f = Q8 ? 1.0f : 0.0625f;
            const float dw0 = half_bits_to_float(*reinterpret_cast<const uint16_t *>(dwr + k * 2)) * f;
            const float dw1 = half_bits_to_float(*reinterpret_cast<const uint16_t *>(dwr + 8 * G::kDwStride + k * 2)) * f;
            const f32x2 dwp0 = pack2(dw0, dw0), dwp1 = pack2(dw1, dw1);
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const uint2 x = *reinterpret_cast<const uint2 *>(xrow + n * 8 * G::kXStride + k * 32);
                float d[4];
                mma_s8(d, a, x.x, x.y);
                const f32x2 dx = *reinterpret_cast<const f32x2 *>(dxr + k * G::kDxStride + n * 32);
                acc[n][0] = fma2(mul2(dwp0, dx), add2(pack2(d[0], d[1]), unmagic), acc[n][0]);
                acc[n][1] = fma2(mul2(dwp1, dx), add2(pack2(d[2], d[3]), unmagic), acc[n][1]);
            }
        }
        }
        // lane 4 x + c is complete: fold it into the tree
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                f32x2 v = acc[n][i];
                if (j & 1) v = add2(s0[n][i], v);
                else s0[n][i] = v;
                if ((j & 3) == 3) v = add2(s1[n][i], v);
                else if (j & 1) s1[n][i] = v;
                if (j == 7) v = add2(s2[n][i], v);
                else if (j == 3) s2[n][i] = v;
                acc[n][i] = j == 7 ? v : 0ull;
            }
    }
    cp_async_wait<0>();
    __syncthreads();
    // the four residues meet: [residue][token][row]
    float *red = reinterpret_cast<float *>(gsm);
    constexpr int kRs = G::kRows + 4;
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float lo, hi;
            unpack2(acc[n][i], lo, hi);
            float *dst = red + (res * G::kTok + n * 8 + 2 * q) * kRs + rg * 16 + g + i * 8;
            dst[0] = lo;
            dst[kRs] = hi;
        }
    __syncthreads();
    for (int e = tid; e < G::kTok * G::kRows; e += G::kThreads) {
        const int t = e / G::kRows, r = e % G::kRows;
        if (tok0 + t < m_tokens && row0 + r < rows) {
            const float c0 = red[t * kRs + r], c1 = red[(G::kTok + t) * kRs + r], c2 = red[(2 * G::kTok + t) * kRs + r],
                        c3 = red[(3 * G::kTok + t) * kRs + r];
            y[static_cast<size_t>(tok0 + t) * rows + row0 + r] = __fadd_rn(__fadd_rn(c0, c2), __fadd_rn(c1, c3));
        }
    }
}

// ---- rotary embedding and cache store of the chunk ----------------------------------------------------------------------
// One CTA of eight warps per token, one warp per head: the q heads go to `qrot` [token][heads * head_dim], the k heads (with
// their v head) into the caches. Biases, head norms and the rotation are the one-token kernel's, in the same order: the sum
// of squares is the binary tree in double over the head's elements, zero-padded to 128 leaves (lane l holds leaves l + 32 i).
constexpr int kRopeWarps = 8;
__global__ void __launch_bounds__(32 * kRopeWarps) prefill_rope_kernel(const float *qkv, const float *table, float *kcache, float *vcache,
                                                                     int pos0, int heads, int kv_heads, int head_dim, float *qrot,
                                                                     const float *bqkv, const float *q_norm, const float *k_norm, float eps) {
    __shared__ float rows[kRopeWarps][128];
    grid_dep_launch();
    grid_dep_wait();
    const int m = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = head_dim / 2, nd = head_dim / 32;
    const int step = kRopeWarps * gridDim.y;            // short prompts: several CTAs share a token's heads
    const int kv_dim = kv_heads * head_dim, pos = pos0 + m;
    const float *src = qkv + static_cast<size_t>(m) * (heads + 2 * kv_heads) * head_dim;
    float *row = rows[warp];
    for (int h = blockIdx.y * kRopeWarps + warp; h < heads + kv_heads; h += step) {
        const bool is_q = h < heads;
        const float *norm = is_q ? q_norm : k_norm;
        float x[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = h * head_dim + i * 32 + lane;         // q heads, then k heads
            x[i] = i < nd ? src[e] : 0.0f;
            if (i < nd && bqkv != nullptr) x[i] = __fadd_rn(x[i], bqkv[e]);
        }
        if (norm != nullptr) {
            double s2[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                s2[i] = __dmul_rn(static_cast<double>(x[i]), static_cast<double>(x[i]));
#pragma unroll
                for (int s = 1; s < 32; s <<= 1) s2[i] = __dadd_rn(s2[i], __shfl_xor_sync(0xffffffffu, s2[i], s));
            }
            const double t = __dadd_rn(__dadd_rn(s2[0], s2[1]), __dadd_rn(s2[2], s2[3]));
            const float sc = __double2float_rn(
                __ddiv_rn(1.0, __dsqrt_rn(__dadd_rn(__ddiv_rn(t, static_cast<double>(head_dim)), static_cast<double>(eps)))));
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (i < nd) x[i] = __fmul_rn(__fmul_rn(x[i], sc), norm[i * 32 + lane]);
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (i < nd) row[i * 32 + lane] = x[i];
        __syncwarp();
        float *dst = is_q ? qrot + (static_cast<size_t>(m) * heads + h) * head_dim
                          : kcache + static_cast<size_t>(pos) * kv_dim + static_cast<size_t>(h - heads) * head_dim;
        for (int p = lane; p < half; p += 32) {
            const float2 c = reinterpret_cast<const float2 *>(table)[static_cast<size_t>(pos) * half + p];
            const float a = row[p], b = row[p + half];
            dst[p] = __fadd_rn(__fmul_rn(a, c.x), -__fmul_rn(b, c.y));
            dst[p + half] = __fadd_rn(__fmul_rn(a, c.y), __fmul_rn(b, c.x));
        }
        if (!is_q) {
            for (int i = lane; i < head_dim; i += 32) {
                const int e = (h + kv_heads) * head_dim + i;
                float v = src[e];
                if (bqkv != nullptr) v = __fadd_rn(v, bqkv[e]);
                vcache[static_cast<size_t>(pos) * kv_dim + static_cast<size_t>(h - heads) * head_dim + i] = v;
            }
        }
    }
}

// ---- attention of the chunk ----------------------------------------------------------------------------------------------
constexpr int kPrefillAttnThreads = 288;    // eight warps on scores and values, one on the sums of the weights

// One CTA per (head, QT consecutive tokens). Scores, weights and the sums over positions keep the one-token order: maximum,
// p = exp(score - max), the sum of p and every output element ascending in the position. What is serial per (token,
// element) runs side by side for QT tokens; a thread holds one element of several tokens, so a value is loaded once for
// all of them. Shared memory: [positions][QT] scores, then the QT query heads.
template <int HD, int QT>
__global__ void __launch_bounds__(kPrefillAttnThreads, HD <= 64 ? 2 : 1) prefill_attention_kernel(const float *qrot, const float *kcache, const float *vcache,
                                                                              int pos0, int m_tokens, int heads, int kv_heads,
                                                                              float inv_sqrt, PromptAct o) {
    extern __shared__ __align__(16) float asm_[];
    __shared__ float mx[QT], lsum[QT], part[QT * 16];
    grid_dep_launch();
    grid_dep_wait();
    const int h = blockIdx.x, tok0 = blockIdx.y * QT, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n_tok = min(QT, m_tokens - tok0), kv_dim = kv_heads * HD, kvh = (h * kv_heads) / heads;
    const int first = pos0 + tok0, last = first + n_tok - 1;    // token r attends to positions 0 .. first + r
    const float *kc = kcache + static_cast<size_t>(kvh) * HD, *vc = vcache + static_cast<size_t>(kvh) * HD;
    float *qs = asm_, *sc = asm_ + QT * HD;
    for (int i = tid; i < QT * HD; i += kPrefillAttnThreads) {
        const int r = i / HD, d = i - r * HD;
        qs[i] = r < n_tok ? qrot[(static_cast<size_t>(tok0 + r) * heads + h) * HD + d] : 0.0f;
    }
    __syncthreads();
    // scores: a thread takes one position and, while there are fewer positions than threads, a share of the tokens
    int groups = 1;
    while (groups < QT / 2 && 2 * groups * (last + 1) <= 256) groups *= 2;
    const int rows = QT / groups;
    for (int i = tid; i < (last + 1) * groups; i += kPrefillAttnThreads) {
        const int gidx = i / (last + 1), t = i - gidx * (last + 1);
        ulonglong2 k[HD / 4];
#pragma unroll
        for (int e = 0; e < HD / 4; ++e) k[e] = *reinterpret_cast<const ulonglong2 *>(kc + static_cast<size_t>(t) * kv_dim + e * 4);
#pragma unroll 1
        for (int r = gidx * rows; r < (gidx + 1) * rows; r += 2) {
            const float a = __fmul_rn(lane_order_dot<HD>(qs + r * HD, [&](int e) { return k[e]; }), inv_sqrt);
            const float b = __fmul_rn(lane_order_dot<HD>(qs + (r + 1) * HD, [&](int e) { return k[e]; }), inv_sqrt);
            *reinterpret_cast<float2 *>(sc + static_cast<size_t>(t) * QT + r) = make_float2(a, b);
        }
    }
    __syncthreads();
    {       // maxima: thread (token, part); the comparison skips NaN as the one-token loop does
        const int r = tid % QT, p = tid / QT;
        constexpr int kParts = 16;
        float m = -INFINITY;
        if (p < kParts)
            for (int t = p; t <= min(first + r, last); t += kParts) {
                const float v = sc[static_cast<size_t>(t) * QT + r];
                m = v > m ? v : m;
            }
        if (p < kParts) part[p * QT + r] = m;
        __syncthreads();
        if (tid < QT) {
            m = part[tid];
            for (int i = 1; i < kParts; ++i) m = part[i * QT + tid] > m ? part[i * QT + tid] : m;
            mx[tid] = m;
        }
        __syncthreads();
    }
    for (int i = tid; i < (last + 1) * QT; i += kPrefillAttnThreads) sc[i] = exp_ggml(__fadd_rn(sc[i], -mx[i % QT]));
    __syncthreads();
    constexpr int kGroups = 256 / HD < QT ? 256 / HD : QT, kPer = QT / kGroups;   // tokens of one thread
    constexpr int kPairs = (kPer + 1) / 2;
    f32x2 acc[kPairs];
    const int grp = tid / HD, d = tid - grp * HD;
#pragma unroll
    for (int i = 0; i < kPairs; ++i) acc[i] = 0ull;
    if (warp == 8) {
        if (lane < QT) {
            float l = 0.0f;
#pragma unroll 8
            for (int t = 0; t <= min(first + lane, last); ++t) l = __fadd_rn(l, sc[static_cast<size_t>(t) * QT + lane]);
            lsum[lane] = l;
        }
    } else if (grp < kGroups) {
        const float *pr = sc + grp * kPer, *v = vc + d;
        auto weights = [&](int t, f32x2 (&p)[kPairs]) {
            const float *s = pr + static_cast<size_t>(t) * QT;
            if constexpr (kPer >= 4) {
#pragma unroll
                for (int i = 0; i < kPer / 4; ++i) {
                    const ulonglong2 w = *reinterpret_cast<const ulonglong2 *>(s + 4 * i);
                    p[2 * i] = w.x;
                    p[2 * i + 1] = w.y;
                }
            } else if constexpr (kPer == 2) {
                p[0] = *reinterpret_cast<const f32x2 *>(s);
            } else {
                p[0] = pack2(s[0], 0.0f);
            }
        };
#pragma unroll 8
        for (int t = 0; t <= first; ++t) {          // positions every token of the CTA attends to
            const float x = v[static_cast<size_t>(t) * kv_dim];
            const f32x2 xx = pack2(x, x);
            f32x2 p[kPairs];
            weights(t, p);
#pragma unroll
            for (int i = 0; i < kPairs; ++i) acc[i] = fma2(p[i], xx, acc[i]);
        }
        for (int t = first + 1; t <= last; ++t) {   // the causal edge: token i stops at position first + i
            const float x = v[static_cast<size_t>(t) * kv_dim];
#pragma unroll
            for (int i = 0; i < kPairs; ++i) {
                float lo, hi;
                unpack2(acc[i], lo, hi);
                const int r = grp * kPer + 2 * i;
                if (t <= first + r) lo = __fmaf_rn(sc[static_cast<size_t>(t) * QT + r], x, lo);
                if (2 * i + 1 < kPer && t <= first + r + 1) hi = __fmaf_rn(sc[static_cast<size_t>(t) * QT + r + 1], x, hi);
                acc[i] = pack2(lo, hi);
            }
        }
    }
    __syncthreads();
    if (warp < 8 && grp < kGroups) {
#pragma unroll
        for (int i = 0; i < kPairs; ++i) {
            const int r = grp * kPer + 2 * i;
            float lo, hi;
            unpack2(acc[i], lo, hi);
            qs[r * HD + d] = __fdiv_rn(lo, lsum[r]);
            if (2 * i + 1 < kPer) qs[(r + 1) * HD + d] = __fdiv_rn(hi, lsum[r + 1]);
        }
    }
    __syncthreads();
    for (int b = warp; b < n_tok * (HD / 32); b += kPrefillAttnThreads / 32) {
        const int r = b / (HD / 32), k = b - r * (HD / 32), blk = h * (HD / 32) + k;
        const float v = qs[r * HD + k * 32 + lane];
        if (o.tile == 0) q8_0_block_warp(v, lane, QuantAt{o.row_quad(tok0 + r, blk * 32 + (lane & ~3))}, o.row_scale(tok0 + r, blk));
        else q8_0_block_warp(v, lane, QuantAt{o.tile_quad(tok0 + r, blk * 32 + (lane & ~3))}, o.tile_scale(tok0 + r, blk));
    }
    if (o.tile > 0 && h == heads - 1) {         // as in prefill_swiglu_quant_kernel
        const int nb = o.n >> 5, gap = ((nb + 31) & ~31) - nb;
        for (int i = tid; i < n_tok * gap; i += kPrefillAttnThreads) *o.tile_scale(tok0 + i / gap, nb + i % gap) = 0.0f;
    }
}

// act = SiLU(g) * u of every token, -> Q8_0; a thread takes four values, eight neighbouring lanes a block of 32.
__global__ void __launch_bounds__(256) prefill_swiglu_quant_kernel(const float *gate_up, int n, PromptAct x) {
    grid_dep_launch();
    grid_dep_wait();
    const size_t m = blockIdx.y;
    const int ch = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = 4 * ch < n;       // n is a multiple of 32: the lanes of a block leave together
    gate_up += m * 2 * n;
    float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (live) {
        const float4 g = reinterpret_cast<const float4 *>(gate_up)[ch], u = reinterpret_cast<const float4 *>(gate_up + n)[ch];
        v[0] = __fmul_rn(silu_ggml(g.x), u.x);
        v[1] = __fmul_rn(silu_ggml(g.y), u.y);
        v[2] = __fmul_rn(silu_ggml(g.z), u.z);
        v[3] = __fmul_rn(silu_ggml(g.w), u.w);
    }
    float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
    if (!live) {        // blocks behind the end of a row: prompt_tc_gemm_kernel multiplies them by a scale of zero
        if (x.tile > 0 && (ch & 7) == 0) *x.tile_scale(blockIdx.y, ch >> 3) = 0.0f;
        return;
    }
    int q[4] = {0, 0, 0, 0};
    if (amax != 0.0f) {
        const float inv = __fdiv_rn(127.0f, amax);
#pragma unroll
        for (int j = 0; j < 4; ++j) q[j] = max(-128, min(127, __float2int_rn(__fmul_rn(v[j], inv))));
    }
    const uint32_t packed = (q[0] & 0xff) | ((q[1] & 0xff) << 8) | ((q[2] & 0xff) << 16) | (static_cast<uint32_t>(q[3]) << 24);
    *reinterpret_cast<uint32_t *>(x.tile == 0 ? x.row_quad(blockIdx.y, 4 * ch) : x.tile_quad(blockIdx.y, 4 * ch)) = packed;
    if ((ch & 7) == 0)
        *(x.tile == 0 ? x.row_scale(blockIdx.y, ch >> 3) : x.tile_scale(blockIdx.y, ch >> 3)) = __half2float(__float2half_rn(__fdiv_rn(amax, 127.0f)));
}

}  // namespace wd
