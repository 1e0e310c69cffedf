// The prompt of the plain decoder in one pass over the weights: the tokens of a chunk go through a layer together, with
// the float order of the one-token step (wd_dense_decoder.cuh) kept per token, so that caches, logits and tokens are
// bit-identical to feeding the prompt token by token.
//
// What the step spends per prompt token is one read of every matrix and about 130 dependent launches (540 us on the
// 16-layer benchmark model, 1.2 ms with 500 positions in the cache). Here a chunk of up to 512 tokens shares both.
#pragma once

#include "wd_dense_decoder.cuh"

namespace wd {

constexpr int kPrefillChunk = 512;      // tokens per pass at most (workspace: about 100 KB per token at ffn 8192)

// RMSNorm + Q8_0 of every token of the chunk, one CTA per token; the body is the one-token kernel's.
__global__ void __launch_bounds__(kDecThreads) prefill_norm_quant_kernel(float *hidden, const float *proj, const float *w, int n, float eps,
                                                                       int8_t *xq, float *xd, const uint8_t *embd, const int *tokens,
                                                                       int vocab, int embd_q8) {
    grid_dep_launch();
    grid_dep_wait();
    const size_t m = blockIdx.x;
    hidden += m * n;
    if (proj != nullptr) proj += m * n;
    xq += m * n;
    xd += m * (n >> 5);
    const uint8_t *row = nullptr;
    if (embd != nullptr) row = embd + static_cast<size_t>(max(0, min(vocab - 1, tokens[m]))) * (n >> 5) * (embd_q8 ? 34 : 18);
    const bool q8 = embd_q8 != 0;
    switch (n / kDecThreads) {
        case 1: dense_norm_quant_body<1>(hidden, proj, w, n, eps, xq, xd, row, q8); break;
        case 2: dense_norm_quant_body<2>(hidden, proj, w, n, eps, xq, xd, row, q8); break;
        case 4: dense_norm_quant_body<4>(hidden, proj, w, n, eps, xq, xd, row, q8); break;
        case 8: dense_norm_quant_body<8>(hidden, proj, w, n, eps, xq, xd, row, q8); break;
        default: dense_norm_quant_body<16>(hidden, proj, w, n, eps, xq, xd, row, q8); break;
    }
}

// ---- Y[m][row] = W[row] . X[m] for the tokens of a chunk ---------------------------------------------------------------
// The one-token order is: lane l of 32 runs one fmaf(d_w * d_x, (float)int_dot, acc) per block b = l, l + 32, ... ascending,
// then the butterfly ^16 ^8 ^4 ^2 ^1. The integer dot of one block is a contraction of depth 32, i.e. exactly one
// mma.m16n8k32 (s8) for 16 rows x 8 tokens; its result cannot be accumulated over blocks, because every block is scaled
// by its own d_w * d_x in float. That float side (convert, scale, fmaf: 12 instructions per lane and MMA) is what bounds
// the kernel, so the fragments are taken from mma.sync, whose result is already in registers; tcgen05 would add a TMEM
// read-back per block to the same float work.
//
// A warp owns 16 rows, 8 * NT tokens and one residue c = l mod 4 of the lanes: ^16, ^8 and ^4 pair lanes of one residue,
// so it walks the lanes l = 4 x + c with x in bit-reversed order and folds the finished lane sums with a three-deep stack;
// the four residues meet in shared memory at the end ((c0 + c2) + (c1 + c3)). A stage of the copy pipeline holds, for
// every row and token, the four neighbouring blocks 32 t + 4 x + {0..3} of two values of t.
__device__ __forceinline__ void cp_async4(void *dst, const void *src, bool live) {
    const int bytes = live ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mma_s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}

// Shared-memory plan of one stage (TC = 2 values of t, four blocks each). The 16-byte pads put the eight rows (or tokens)
// of a fragment into different banks.
template <bool Q8, int RG, int NT>
struct PrefillGemm {
    static constexpr int kTc = 2, kRows = 16 * RG, kTok = 8 * NT, kThreads = 128 * RG;
    static constexpr int kBlk = Q8 ? 32 : 16;
    static constexpr int kWStride = kTc * 4 * kBlk + 16, kXStride = kTc * 4 * 32 + 16;
    static constexpr int kDwStride = kTc * 4 * 2 + 8, kDxStride = kTc * 4 * 4 + 16;
    static constexpr int kOffX = kRows * kWStride, kOffDw = kOffX + kTok * kXStride, kOffDx = kOffDw + kRows * kDwStride;
    static constexpr int kStage = (kOffDx + kTok * kDxStride + 127) / 128 * 128;
    static constexpr int kRed = 4 * kTok * (kRows + 4) * 4;              // the residues' sums, after the last stage
    static constexpr int kStages = NT == 4 ? 4 : 6;
    static constexpr int kSmem = kStages * kStage > kRed ? kStages * kStage : kRed;
    static constexpr int kDwPer = kRows * kTc * 4 / kThreads;            // scales one thread moves per stage
};

template <bool Q8, int RG, int NT>
__global__ void __launch_bounds__(128 * RG) prefill_gemm_kernel(const uint8_t *wp, int rows, int nb, const int8_t *xq, const float *xd, int m_tokens,
                                                               float *y) {
    using G = PrefillGemm<Q8, RG, NT>;
    extern __shared__ __align__(128) uint8_t gsm[];
    grid_dep_launch();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int res = warp & 3, rg = warp >> 2, g = lane >> 2, q = lane & 3;
    const int row0 = blockIdx.x * G::kRows, tok0 = blockIdx.y * G::kTok;
    const uint8_t *q_all = wp;
    const uint16_t *d_all = reinterpret_cast<const uint16_t *>(wp + static_cast<size_t>(rows) * nb * G::kBlk);
    const int n_t = (nb + 31) >> 5, n_tc = (n_t + G::kTc - 1) / G::kTc, n_stage = 8 * n_tc;
    auto bitrev3 = [](int j) { return ((j & 1) << 2) | (j & 2) | ((j >> 2) & 1); };

    uint16_t dw_next[G::kDwPer];
    auto load_dw = [&](int s) {
        const int x4 = 4 * bitrev3(s / n_tc), t0 = (s % n_tc) * G::kTc;
#pragma unroll
        for (int i = 0; i < G::kDwPer; ++i) {
            const int e = tid + i * G::kThreads, r = e / (G::kTc * 4), k = e % (G::kTc * 4);
            const int b = 32 * (t0 + (k >> 2)) + x4 + (k & 3);
            dw_next[i] = (row0 + r < rows && b < nb) ? __ldg(d_all + static_cast<size_t>(row0 + r) * nb + b) : static_cast<uint16_t>(0);
        }
    };
    auto store_dw = [&](int s) {
        uint8_t *st = gsm + (s % G::kStages) * G::kStage + G::kOffDw;
#pragma unroll
        for (int i = 0; i < G::kDwPer; ++i) {
            const int e = tid + i * G::kThreads, r = e / (G::kTc * 4), k = e % (G::kTc * 4);
            *reinterpret_cast<uint16_t *>(st + r * G::kDwStride + k * 2) = dw_next[i];
        }
    };
    auto issue_w = [&](int s) {
        uint8_t *st = gsm + (s % G::kStages) * G::kStage;
        const int x4 = 4 * bitrev3(s / n_tc), t0 = (s % n_tc) * G::kTc;
        constexpr int kPer = G::kTc * 4 * (G::kBlk / 16);       // 16-byte pieces of a row
#pragma unroll
        for (int e = tid; e < G::kRows * kPer; e += G::kThreads) {
            const int r = e / kPer, p = e % kPer, k = p / (G::kBlk / 16), h = p % (G::kBlk / 16);
            const int b = 32 * (t0 + (k >> 2)) + x4 + (k & 3);
            const bool live = row0 + r < rows && b < nb;
            cp_async16(st + r * G::kWStride + p * 16, live ? q_all + (static_cast<size_t>(row0 + r) * nb + b) * G::kBlk + h * 16 : q_all, live);
        }
    };
    auto issue_x = [&](int s) {
        uint8_t *st = gsm + (s % G::kStages) * G::kStage;
        const int x4 = 4 * bitrev3(s / n_tc), t0 = (s % n_tc) * G::kTc;
        constexpr int kPer = G::kTc * 4 * 2;
#pragma unroll
        for (int e = tid; e < G::kTok * kPer; e += G::kThreads) {
            const int r = e / kPer, p = e % kPer, b = 32 * (t0 + (p >> 3)) + x4 + ((p >> 1) & 3);
            const bool live = tok0 + r < m_tokens && b < nb;
            cp_async16(st + G::kOffX + r * G::kXStride + p * 16,
                       live ? xq + (static_cast<size_t>(tok0 + r) * nb + b) * 32 + (p & 1) * 16 : xq, live);
        }
        for (int e = tid; e < G::kTok * G::kTc * 4; e += G::kThreads) {
            const int r = e / (G::kTc * 4), k = e % (G::kTc * 4), b = 32 * (t0 + (k >> 2)) + x4 + (k & 3);
            const bool live = tok0 + r < m_tokens && b < nb;
            cp_async4(st + G::kOffDx + r * G::kDxStride + k * 4, live ? xd + static_cast<size_t>(tok0 + r) * nb + b : xd, live);
        }
    };

    // the weights do not depend on the kernel before this one: the first stages' rows leave before the wait for it
    for (int s = 0; s < G::kStages - 1; ++s)
        if (s < n_stage) {
            issue_w(s);
            load_dw(s);
            store_dw(s);
        }
    grid_dep_wait();
    for (int s = 0; s < G::kStages - 1; ++s) {
        if (s < n_stage) issue_x(s);
        cp_async_commit();
    }
    float acc[NT][4], s0[NT][4], s1[NT][4], s2[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[n][i] = s0[n][i] = s1[n][i] = s2[n][i] = 0.0f;
    int j = 0, tc = 0;
#pragma unroll 1
    for (int s = 0; s < n_stage; ++s) {
        cp_async_wait<G::kStages - 2>();
        __syncthreads();            // stage s has landed for everyone; the slot of stage s - 1 is free
        const int nx = s + G::kStages - 1;
        if (nx < n_stage) {
            issue_w(nx);
            issue_x(nx);
            load_dw(nx);
        }
        cp_async_commit();
        const uint8_t *st = gsm + (s % G::kStages) * G::kStage;
        const uint8_t *wrow = st + (rg * 16 + g) * G::kWStride, *xrow = st + G::kOffX + g * G::kXStride;
        const uint8_t *dwr = st + G::kOffDw + (rg * 16 + g) * G::kDwStride, *dxr = st + G::kOffDx + 2 * q * G::kDxStride;
#pragma unroll
        for (int t = 0; t < G::kTc; ++t) {
            const int k = t * 4 + res;
            uint32_t a0, a1, a2, a3;
            if constexpr (Q8) {
                a0 = *reinterpret_cast<const uint32_t *>(wrow + k * 32 + q * 4);
                a1 = *reinterpret_cast<const uint32_t *>(wrow + 8 * G::kWStride + k * 32 + q * 4);
                a2 = *reinterpret_cast<const uint32_t *>(wrow + k * 32 + 16 + q * 4);
                a3 = *reinterpret_cast<const uint32_t *>(wrow + 8 * G::kWStride + k * 32 + 16 + q * 4);
            } else {        // a nibble at the top of its byte with the top bit flipped is 16 * (q - 8)
                const uint32_t w0 = *reinterpret_cast<const uint32_t *>(wrow + k * 16 + q * 4);
                const uint32_t w1 = *reinterpret_cast<const uint32_t *>(wrow + 8 * G::kWStride + k * 16 + q * 4);
                a0 = ((w0 << 4) & 0xf0f0f0f0u) ^ 0x80808080u;
                a1 = ((w1 << 4) & 0xf0f0f0f0u) ^ 0x80808080u;
                a2 = (w0 & 0xf0f0f0f0u) ^ 0x80808080u;
                a3 = (w1 & 0xf0f0f0f0u) ^ 0x80808080u;
            }
            // d_w carries the 1/16 of a Q4_0 sum (a power of two: exact)
            const float f = Q8 ? 1.0f : 0.0625f;
            const float dw0 = half_bits_to_float(*reinterpret_cast<const uint16_t *>(dwr + k * 2)) * f;
            const float dw1 = half_bits_to_float(*reinterpret_cast<const uint16_t *>(dwr + 8 * G::kDwStride + k * 2)) * f;
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const uint8_t *xb = xrow + n * 8 * G::kXStride + k * 32 + q * 4;
                int d[4];
                mma_s8(d, a0, a1, a2, a3, *reinterpret_cast<const uint32_t *>(xb), *reinterpret_cast<const uint32_t *>(xb + 16));
                const float dx0 = *reinterpret_cast<const float *>(dxr + n * 8 * G::kDxStride + k * 4);
                const float dx1 = *reinterpret_cast<const float *>(dxr + (n * 8 + 1) * G::kDxStride + k * 4);
                acc[n][0] = __fmaf_rn(__fmul_rn(dw0, dx0), static_cast<float>(d[0]), acc[n][0]);
                acc[n][1] = __fmaf_rn(__fmul_rn(dw0, dx1), static_cast<float>(d[1]), acc[n][1]);
                acc[n][2] = __fmaf_rn(__fmul_rn(dw1, dx0), static_cast<float>(d[2]), acc[n][2]);
                acc[n][3] = __fmaf_rn(__fmul_rn(dw1, dx1), static_cast<float>(d[3]), acc[n][3]);
            }
        }
        if (nx < n_stage) store_dw(nx);
        if (++tc == n_tc) {         // lane 4 x + c is complete: fold it into the tree
            tc = 0;
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float v = acc[n][i];
                    if (j & 1) {
                        v = __fadd_rn(s0[n][i], v);
                        if (j & 2) {
                            v = __fadd_rn(s1[n][i], v);
                            if (j & 4) acc[n][i] = __fadd_rn(s2[n][i], v);
                            else s2[n][i] = v;
                        } else {
                            s1[n][i] = v;
                        }
                    } else {
                        s0[n][i] = v;
                    }
                    if (j != 7) acc[n][i] = 0.0f;
                }
            ++j;
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
        for (int i = 0; i < 4; ++i)
            red[(res * G::kTok + n * 8 + 2 * q + (i & 1)) * kRs + rg * 16 + g + (i >> 1) * 8] = acc[n][i];
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
// One CTA of 128 threads per (token, head): the q heads go to `qrot` [token][heads * head_dim], the k heads (with their v
// head) into the caches. Biases, head norms and the rotation are the one-token kernel's, in the same order.
__global__ void __launch_bounds__(128) prefill_rope_kernel(const float *qkv, const float *table, float *kcache, float *vcache, int pos0,
                                                           int heads, int kv_heads, int head_dim, float *qrot, const float *bqkv,
                                                           const float *q_norm, const float *k_norm, float eps) {
    __shared__ float row[128];
    __shared__ double red[4];
    grid_dep_launch();
    grid_dep_wait();
    const int m = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, half = head_dim / 2;
    const int kv_dim = kv_heads * head_dim, pos = pos0 + m;
    const float *src = qkv + static_cast<size_t>(m) * (heads + 2 * kv_heads) * head_dim;
    const bool is_q = h < heads;
    const float *norm = is_q ? q_norm : k_norm;
    float x = 0.0f;
    if (tid < head_dim) {
        const size_t e = static_cast<size_t>(h) * head_dim + tid;       // q heads, then k heads
        x = src[e];
        if (bqkv != nullptr) x = __fadd_rn(x, bqkv[e]);
    }
    if (norm != nullptr) {      // the binary tree in double over the head's elements, zero-padded to 128 leaves
        double s2 = __dmul_rn(static_cast<double>(x), static_cast<double>(x));
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) s2 = __dadd_rn(s2, __shfl_xor_sync(0xffffffffu, s2, s));
        if (lane == 0) red[warp] = s2;
        __syncthreads();
        const double t = __dadd_rn(__dadd_rn(red[0], red[1]), __dadd_rn(red[2], red[3]));
        const float sc = __double2float_rn(
            __ddiv_rn(1.0, __dsqrt_rn(__dadd_rn(__ddiv_rn(t, static_cast<double>(head_dim)), static_cast<double>(eps)))));
        if (tid < head_dim) x = __fmul_rn(__fmul_rn(x, sc), norm[tid]);
    }
    row[tid] = x;
    __syncthreads();
    float *dst = is_q ? qrot + (static_cast<size_t>(m) * heads + h) * head_dim
                      : kcache + static_cast<size_t>(pos) * kv_dim + static_cast<size_t>(h - heads) * head_dim;
    if (tid < half) {
        const float cs = table[(static_cast<size_t>(pos) * half + tid) * 2], sn = table[(static_cast<size_t>(pos) * half + tid) * 2 + 1];
        const float a = row[tid], b = row[tid + half];
        dst[tid] = __fadd_rn(__fmul_rn(a, cs), -__fmul_rn(b, sn));
        dst[tid + half] = __fadd_rn(__fmul_rn(a, sn), __fmul_rn(b, cs));
    }
    if (!is_q && tid < head_dim) {
        const size_t e = static_cast<size_t>(h + kv_heads) * head_dim + tid;
        float v = src[e];
        if (bqkv != nullptr) v = __fadd_rn(v, bqkv[e]);
        vcache[static_cast<size_t>(pos) * kv_dim + static_cast<size_t>(h - heads) * head_dim + tid] = v;
    }
}

// ---- attention of the chunk ----------------------------------------------------------------------------------------------
constexpr int kPrefillAttnThreads = 288;    // eight warps on scores and values, one on the sums of the weights

// One CTA per (head, QT consecutive tokens). Scores, weights and the sums over positions keep the one-token order: maximum,
// p = exp(score - max), the sum of p and every output element ascending in the position. What is serial per (token,
// element) runs side by side for QT tokens; a thread holds one element of several tokens, so a value is loaded once for
// all of them. Shared memory: [positions][QT] scores, then the QT query heads.
template <int HD, int QT>
__global__ void __launch_bounds__(kPrefillAttnThreads) prefill_attention_kernel(const float *qrot, const float *kcache, const float *vcache,
                                                                              int pos0, int m_tokens, int heads, int kv_heads,
                                                                              float inv_sqrt, int8_t *oq, float *od) {
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
    for (int t = tid; t <= last; t += kPrefillAttnThreads) {
        float4 k[HD / 4];
#pragma unroll
        for (int i = 0; i < HD / 4; ++i) k[i] = *reinterpret_cast<const float4 *>(kc + static_cast<size_t>(t) * kv_dim + i * 4);
#pragma unroll 1
        for (int r = 0; r < QT; r += 2) {
            const float a = __fmul_rn(lane_order_dot<HD>(qs + r * HD, k), inv_sqrt);
            const float b = __fmul_rn(lane_order_dot<HD>(qs + (r + 1) * HD, k), inv_sqrt);
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
    float acc[kPer];
    const int grp = tid / HD, d = tid - grp * HD;
#pragma unroll
    for (int i = 0; i < kPer; ++i) acc[i] = 0.0f;
    if (warp == 8) {
        if (lane < QT) {
            float l = 0.0f;
#pragma unroll 8
            for (int t = 0; t <= min(first + lane, last); ++t) l = __fadd_rn(l, sc[static_cast<size_t>(t) * QT + lane]);
            lsum[lane] = l;
        }
    } else if (grp < kGroups) {
        const float *pr = sc + grp * kPer, *v = vc + d;
#pragma unroll 8
        for (int t = 0; t <= first; ++t) {          // positions every token of the CTA attends to
            const float x = v[static_cast<size_t>(t) * kv_dim];
#pragma unroll
            for (int i = 0; i < kPer; ++i) acc[i] = __fmaf_rn(pr[static_cast<size_t>(t) * QT + i], x, acc[i]);
        }
        for (int t = first + 1; t <= last; ++t) {
            const float x = v[static_cast<size_t>(t) * kv_dim];
#pragma unroll
            for (int i = 0; i < kPer; ++i)
                if (t <= first + grp * kPer + i) acc[i] = __fmaf_rn(pr[static_cast<size_t>(t) * QT + i], x, acc[i]);
        }
    }
    __syncthreads();
    if (warp < 8 && grp < kGroups) {
#pragma unroll
        for (int i = 0; i < kPer; ++i) qs[(grp * kPer + i) * HD + d] = __fdiv_rn(acc[i], lsum[grp * kPer + i]);
    }
    __syncthreads();
    for (int b = warp; b < n_tok * (HD / 32); b += kPrefillAttnThreads / 32) {
        const int r = b / (HD / 32), k = b - r * (HD / 32);
        const size_t blk = (static_cast<size_t>(tok0 + r) * heads + h) * (HD / 32) + k;
        q8_0_block_warp(qs[r * HD + k * 32 + lane], lane, oq + blk * 32, od + blk);
    }
}

// act = SiLU(g) * u of every token, -> Q8_0; one warp per block of 32.
__global__ void prefill_swiglu_quant_kernel(const float *gate_up, int n, int8_t *xq, float *xd) {
    grid_dep_launch();
    grid_dep_wait();
    const size_t m = blockIdx.y;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    gate_up += m * 2 * n;
    const float v = __fmul_rn(silu_ggml(gate_up[i]), gate_up[n + i]);
    q8_0_block_warp(v, threadIdx.x & 31, xq + m * n + (i & ~31), xd + m * (n >> 5) + (i >> 5));
}

}  // namespace wd
