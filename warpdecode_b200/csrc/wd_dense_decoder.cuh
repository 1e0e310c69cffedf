// Kernels of the plain (dense) Q4_0 decoder step: the per-token path of the reference's Runtime::emit_step
// (src/warodecode.cu:2053-2104) for Llama-style models: embedding row, [residual add + RMSNorm + Q8_0 activation,
// fused QKV product, rotary embedding + cache store, decode attention, output product, residual add + RMSNorm + Q8_0,
// gate/up product, SiLU(g) * u + Q8_0, down product] per layer, output norm, output head with the arg-max.
//
// The reference's kernels carry no float order (src/warodecode.cu:1490-1491) and keep activations in F16. Here every
// step has ONE defined order, activations stay F32, and the results are bit-identical to the CPU restatement in
// oracle/wd_oracle_dense.c. The orders are chosen so that every product keeps the whole GPU busy:
//   row dot     a warp splits a row's blocks over its lanes (lane l: blocks l, l + 32, ... ascending, one
//               fmaf(d_w * d_x, (float)int_dot, acc) per block), then a butterfly ^16 ^8 ^4 ^2 ^1
//   RMSNorm     sum of squares as a binary tree in double (the MoE stack's definition)
//   attention   score dots in the same lane order, p = exp(score - max), sums ascending in the position
// Weights: Q4_0 repacked row by row into [rows][blocks][16 B] quants followed by [rows][blocks] f16 scales, so that a
// warp reads 512 consecutive bytes per step (18 B per 32 weights as in ggml).
#pragma once

#include "wd_dense.cuh"

namespace wd {

constexpr int kDecThreads = 256;
constexpr int kDenseMaxCtx = 8192;      // longest context a decoder may be created for

// Blocks per row in the packed layouts: rounded up, so that a row's scales start on 8 bytes (the prompt pass copies four).
// The blocks behind a row's end are never read.
__host__ __device__ inline int dense_row_stride(int nb) { return (nb + 3) & ~3; }

// ggml Q4_0 blocks [rows][nb][18 B] -> [rows][stride][16 B] quants, then [rows][stride] f16 scales.
__global__ void repack_q4_0_rows_kernel(const uint8_t *src, uint8_t *dst, long long nblocks, int nb) {
    const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (i >= nblocks) return;
    const long long row = i / nb, stride = dense_row_stride(nb), o = row * stride + (i - row * nb);
    const uint8_t *s = src + i * 18;
    uint8_t *q = dst + o * 16;
    uint16_t *d = reinterpret_cast<uint16_t *>(dst + nblocks / nb * stride * 16) + o;
    *d = static_cast<uint16_t>(s[0] | (s[1] << 8));
    for (int j = 0; j < 16; ++j) q[j] = s[2 + j];
}

// ggml Q4_0 blocks [rows][nb][18 B] -> per row [nb][16 B] quants followed by [nb] f16 scales (18 * nb bytes per row).
__global__ void repack_q4_0_rowpack_kernel(const uint8_t *src, uint8_t *dst, long long nblocks, int nb) {
    const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (i >= nblocks) return;
    const long long row = i / nb;
    const int b = static_cast<int>(i - row * nb);
    const uint8_t *s = src + i * 18;
    uint8_t *r = dst + row * nb * 18;
    for (int j = 0; j < 16; ++j) r[b * 16 + j] = s[2 + j];
    r[nb * 16 + b * 2] = s[0];
    r[nb * 16 + b * 2 + 1] = s[1];
}

// N(0, sigma) values quantised to ggml Q4_0 blocks by ggml's published rule (quantize_row_q4_0_ref): d = (the value of
// largest magnitude, sign kept) / -8; q = min(15, (int)(v / d + 8.5)); byte j = q[j] | q[j + 16] << 4.
__global__ void synth_q4_0_kernel(uint8_t *dst, long long nblocks, float sigma, uint64_t seed, uint64_t stream_id) {
    const long long b = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (b >= nblocks) return;
    float v[32], amax = 0.0f, vmax = 0.0f;
    for (int i = 0; i < 32; ++i) {
        v[i] = sigma * synth_normal(seed, stream_id, static_cast<uint64_t>(b) * 32 + i);
        if (fabsf(v[i]) > amax) {
            amax = fabsf(v[i]);
            vmax = v[i];
        }
    }
    const float d = vmax / -8.0f;
    const float id = d != 0.0f ? 1.0f / d : 0.0f;
    uint8_t *o = dst + b * 18;
    const uint16_t bits = __half_as_ushort(__float2half_rn(d));
    o[0] = bits & 0xff;
    o[1] = bits >> 8;
    for (int j = 0; j < 16; ++j) {
        const int q0 = min(15, static_cast<int>(v[j] * id + 8.5f));
        const int q1 = min(15, static_cast<int>(v[j + 16] * id + 8.5f));
        o[2 + j] = static_cast<uint8_t>(q0 | (q1 << 4));
    }
}

// A quant in the order the prompt pass multiplies with: lane q of an MMA reads values 4 q .. 4 q + 3 and 16 + 4 q .. of a
// block as one 8-byte word (wd_dense_prefill.cuh).
struct PairedQuant {
    int8_t v;
};
__device__ __forceinline__ int paired_place(int v) { return ((v >> 2) & 3) * 8 + (v >> 4) * 4 + (v & 3); }
__device__ __forceinline__ void store_quant(int8_t *out, int e, int q) { out[e] = static_cast<int8_t>(q); }
struct QuantAt {        // four neighbouring quants
    uint8_t *quad;
};
__device__ __forceinline__ void store_quant(const QuantAt &out, int e, int q) { out.quad[e & 3] = static_cast<uint8_t>(q); }

// Q8_0 of 32 floats held one per lane: quant byte and the f16-rounded scale (ggml's rule, as quantize_q8_0_cta).
template <class Quant>
__device__ __forceinline__ void q8_0_block_warp(float v, int lane, Quant q_out, float *d_out) {
    float amax = fabsf(v);
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, s));
    int q = 0;
    if (amax != 0.0f) {
        q = __float2int_rn(__fmul_rn(v, __fdiv_rn(127.0f, amax)));
        q = max(-128, min(127, q));
    }
    store_quant(q_out, lane, q);
    if (lane == 0) *d_out = __half2float(__float2half_rn(__fdiv_rn(amax, 127.0f)));
}

// hidden_out = hidden + proj (proj: when given; hidden_out: when given); y = RMSNorm(that) * w -> Q8_0 (int8 [n], float scale per
// block), by one CTA, n = 256 * 2^k up to 4096: with blockDim.x threads, thread t owns elements 4 t .. 4 t + 3 (of every
// 4 * blockDim.x), a Q8_0 block eight neighbouring lanes (residual_rmsnorm_kernel, src/warodecode.cu:1408). The sum of squares
// is the binary tree in double of the MoE stack's RMSNorm. `embd` (optional): the step starts here, and the token's embedding
// row takes the place of hidden (embedding_q4_kernel). `wait`: what the norm weights, which no kernel writes, are fetched in
// front of. PASSES: ceil(n / (4 * blockDim.x)). store(e, packed, d): four quants from element e on, and their block's scale.
// Bound: latency (a chain of one load, two reductions and two divisions). One warp finishes the sum: done by all 16, the
// double-precision pipe is busy for longer than the second barrier takes.
struct NormInput {
    const float *hidden, *proj, *w;     // proj, w: nullable
    float *hidden_out;                  // nullable
    const uint8_t *embd;                // nullable: embedding table in ggml layout, Q4_0 blocks of 18 bytes or Q8_0 blocks of 34
    const int *token;
    float eps;
    int n, vocab, embd_q8;
};
template <int PASSES, class Wait, class Store>
__device__ __forceinline__ void dense_norm_quant_body(const NormInput &in, Wait wait, Store store) {
    __shared__ double red[32];
    __shared__ float scale_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n = in.n;
    float v[PASSES][4];
    float4 nw[PASSES];
#pragma unroll
    for (int p = 0; p < PASSES; ++p) {
        const int e0 = (p * blockDim.x + tid) * 4;
        nw[p] = in.w != nullptr && e0 < n ? *reinterpret_cast<const float4 *>(in.w + e0) : make_float4(1.0f, 1.0f, 1.0f, 1.0f);
    }
    wait();
#pragma unroll
    for (int p = 0; p < PASSES; ++p) {
        const int e0 = (p * blockDim.x + tid) * 4;
        if (e0 >= n) {                      // whole warps: n is a multiple of 256
            v[p][0] = v[p][1] = v[p][2] = v[p][3] = 0.0f;
        } else if (in.embd != nullptr) {
            const int bytes = in.embd_q8 ? 34 : 18, j = e0 & 31;
            const uint8_t *wb = in.embd + (static_cast<size_t>(max(0, min(in.vocab - 1, *in.token))) * (n >> 5) + (e0 >> 5)) * bytes;
            const float d = half_bits_to_float(static_cast<uint16_t>(wb[0] | (wb[1] << 8)));
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int q = in.embd_q8 ? static_cast<int>(static_cast<int8_t>(wb[2 + j + i]))
                                         : (j < 16 ? (wb[2 + j + i] & 0x0f) : (wb[2 + j + i - 16] >> 4)) - 8;
                v[p][i] = __fmul_rn(d, static_cast<float>(q));
            }
        } else {
            const float4 h = *reinterpret_cast<const float4 *>(in.hidden + e0);
            v[p][0] = h.x; v[p][1] = h.y; v[p][2] = h.z; v[p][3] = h.w;
            if (in.proj != nullptr) {
                const float4 q = *reinterpret_cast<const float4 *>(in.proj + e0);
                v[p][0] = __fadd_rn(v[p][0], q.x);
                v[p][1] = __fadd_rn(v[p][1], q.y);
                v[p][2] = __fadd_rn(v[p][2], q.z);
                v[p][3] = __fadd_rn(v[p][3], q.w);
            }
        }
        if (in.hidden_out != nullptr && e0 < n) *reinterpret_cast<float4 *>(in.hidden_out + e0) = make_float4(v[p][0], v[p][1], v[p][2], v[p][3]);
        double sq[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) sq[i] = __dmul_rn(static_cast<double>(v[p][i]), static_cast<double>(v[p][i]));
        double ss = __dadd_rn(__dadd_rn(sq[0], sq[1]), __dadd_rn(sq[2], sq[3]));
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) ss = __dadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, s));
        if (lane == 0 && e0 < n) red[p * (blockDim.x >> 5) + warp] = ss;
    }
    __syncthreads();
    if (warp == 0) {
        double ss = lane < (n >> 7) ? red[lane] : 0.0;      // a power of two of warps; adding +0.0 beyond them changes nothing
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) ss = __dadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, s));
        // n is a power of two: the division by it is an exact multiplication
        const double inv_n = __longlong_as_double(static_cast<long long>(1023 - (31 - __clz(n))) << 52);
        if (lane == 0) scale_s = __double2float_rn(__ddiv_rn(1.0, __dsqrt_rn(__dadd_rn(__dmul_rn(ss, inv_n), static_cast<double>(in.eps)))));
    }
    __syncthreads();
    const float scale = scale_s;
#pragma unroll
    for (int p = 0; p < PASSES; ++p) {
        const int e0 = (p * blockDim.x + tid) * 4;
        if (e0 >= n) break;
        const float g[4] = {nw[p].x, nw[p].y, nw[p].z, nw[p].w};
        float amax = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[p][i] = __fmul_rn(v[p][i], scale);
            if (in.w != nullptr) v[p][i] = __fmul_rn(v[p][i], g[i]);
            amax = fmaxf(amax, fabsf(v[p][i]));
        }
#pragma unroll
        for (int s = 1; s < 8; s <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, s));
        const float inv = amax != 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
        uint32_t packed = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            int q = amax != 0.0f ? __float2int_rn(__fmul_rn(v[p][i], inv)) : 0;
            q = max(-128, min(127, q));
            packed |= static_cast<uint32_t>(q & 0xff) << (8 * i);
        }
        store(e0, packed, __half2float(__float2half_rn(__fdiv_rn(amax, 127.0f))));
    }
}

__device__ __forceinline__ int dp4a_u8s8(uint32_t a, int b, int c) {
    int d;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// The activation in shared memory as the products read it, nb blocks: their first halves, their second halves (neighbouring
// lanes read neighbouring 16 bytes), then (scale, -8 * sum) per block.
struct BlockInput {
    uint4 *lo, *hi;
    int2 *x;
    __device__ __forceinline__ BlockInput(uint8_t *sm, int nb)
        : lo(reinterpret_cast<uint4 *>(sm)), hi(lo + nb), x(reinterpret_cast<int2 *>(hi + nb)) {}
    static constexpr int kBlockBytes = 40;
};

// A block of 32 weights of a packed matrix, and its term of a row's chain: fmaf(d_w * d_x, (float)int_dot, acc).
template <bool Q8>
struct RowBlock {
    uint4 q[Q8 ? 2 : 1];
    uint16_t d;
    __device__ __forceinline__ void load(const uint4 *quants, const uint16_t *scales, size_t blk) {
#pragma unroll
        for (int i = 0; i < (Q8 ? 2 : 1); ++i) q[i] = __ldg(quants + (Q8 ? 2 : 1) * blk + i);
        d = __ldg(scales + blk);
    }
    // The same in front of grid_dep_wait(), by ordinary loads that the wait's memory clobber holds in place: read-only (nc) loads, volatile
    // or not, end up behind it, where their values are first used, and the weights then set out only when the kernel in front has ended.
    // us per token, nc / ordinary / ordinary past L1 (this): 342 / 304 / 303 with 16 layers of 2048 / 8192 and a 128256-row head, 180 / 165 /
    // 163 with 12 of 1024 / 2816, 215 / 197 / 199 with 8 Q8_0 layers of 2048 / 8192.
    __device__ __forceinline__ void load_early(const uint4 *quants, const uint16_t *scales, size_t blk) {
#pragma unroll
        for (int i = 0; i < (Q8 ? 2 : 1); ++i)
            asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(q[i].x), "=r"(q[i].y), "=r"(q[i].z), "=r"(q[i].w)
                         : "l"(quants + (Q8 ? 2 : 1) * blk + i)
                         : "memory");
        asm volatile("ld.global.L1::no_allocate.u16 %0, [%1];" : "=h"(d) : "l"(scales + blk) : "memory");
    }
    // lo, hi: quants 0 .. 15 and 16 .. 31 of the activation's block; x: its scale (as bits) and -8 times the sum of its quants
    __device__ __forceinline__ float term(const uint4 &lo, const uint4 &hi, const int2 &x, float acc) const {
        const int al[4] = {static_cast<int>(lo.x), static_cast<int>(lo.y), static_cast<int>(lo.z), static_cast<int>(lo.w)};
        const int ah[4] = {static_cast<int>(hi.x), static_cast<int>(hi.y), static_cast<int>(hi.z), static_cast<int>(hi.w)};
        const uint32_t w0[4] = {q[0].x, q[0].y, q[0].z, q[0].w};
        int s = 0;
        if constexpr (Q8) {
            const uint32_t w1[4] = {q[1].x, q[1].y, q[1].z, q[1].w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                s = dp4a_s8(static_cast<int>(w0[k]), al[k], s);
                s = dp4a_s8(static_cast<int>(w1[k]), ah[k], s);
            }
        } else {        // sum (q - 8) a = sum q a - 8 sum a, unsigned nibbles; the high ones where they are, worth 16 times as much
            int s_hi = 0;
            s = x.y;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                s = dp4a_u8s8(w0[k] & 0x0f0f0f0fu, al[k], s);
                s_hi = dp4a_u8s8(w0[k] & 0xf0f0f0f0u, ah[k], s_hi);
            }
            s += s_hi >> 4;
        }
        return __fmaf_rn(__fmul_rn(half_bits_to_float(d), __int_as_float(x.x)), static_cast<float>(s), acc);
    }
};

// y = W x: W in the row layout, x already Q8_0 (plain layout, copied into shared memory once per CTA), one warp per row; see
// the header for the order. A Q8_0 block (what every 2-D tensor of a model file that is not Q4_0 becomes: planarize_q4,
// src/warodecode.cu:1027-1075) is two 16-byte loads, a Q4_0 block one. Dynamic shared memory: nb * 40
// bytes. U blocks per lane in flight: with one warp per row every byte of the matrix is requested at once.
template <bool Q8, int U>
__global__ void __launch_bounds__(kDecThreads, 4) dense_product_kernel(const uint8_t *wp, int rows, int nb, const int8_t *xq, const float *xd,
                                                                      float *y) {
    extern __shared__ __align__(16) uint8_t dsm[];
    grid_dep_launch();
    const BlockInput in(dsm, nb);
    const int lane = threadIdx.x & 31, row = blockIdx.x * (kDecThreads / 32) + (threadIdx.x >> 5), stride = dense_row_stride(nb);
    const uint4 *q_all = reinterpret_cast<const uint4 *>(wp);
    const uint16_t *d_all = reinterpret_cast<const uint16_t *>(wp + static_cast<size_t>(rows) * stride * (Q8 ? 32 : 16));
    RowBlock<Q8> w[U];
    // The weights do not depend on the kernel before this one: the first loads leave before the wait for it, and the
    // activation (its output) is fetched after.
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (lane + 32 * u < nb && row < rows) w[u].load_early(q_all, d_all, static_cast<size_t>(row) * stride + lane + 32 * u);
    grid_dep_wait();
#pragma unroll 2
    for (int i = threadIdx.x; i < ((nb * 2 + 31) & ~31); i += kDecThreads) {        // half a block per thread; whole warps
        const int b = i >> 1;
        const uint4 v = b < nb ? reinterpret_cast<const uint4 *>(xq)[i] : make_uint4(0, 0, 0, 0);
        const float d = b < nb ? xd[b] : 0.0f;
        int sum = dp4a_s8(static_cast<int>(v.x), 0x01010101, dp4a_s8(static_cast<int>(v.y), 0x01010101, 0));
        sum = dp4a_s8(static_cast<int>(v.z), 0x01010101, dp4a_s8(static_cast<int>(v.w), 0x01010101, sum));
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        if (b < nb) {
            ((i & 1) ? in.hi : in.lo)[b] = v;
            if ((i & 1) == 0) in.x[b] = make_int2(__float_as_int(d), -8 * sum);
        }
    }
    __syncthreads();
    if (row >= rows) return;
    float acc = 0.0f;
#pragma unroll 1
    for (int b0 = lane; b0 < nb; b0 += 32 * U) {
        if (b0 != lane) {
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (b0 + 32 * u < nb) w[u].load(q_all, d_all, static_cast<size_t>(row) * stride + b0 + 32 * u);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int b = b0 + 32 * u;
            if (b < nb) acc = w[u].term(in.lo[b], in.hi[b], in.x[b], acc);
        }
    }
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1) acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, s));
    if (lane == 0) y[row] = acc;
}

// ggml Q8_0 [rows][nb] blocks of 34 bytes -> the row layout of dense_product_kernel: [rows][stride][32 B] quants, then
// [rows][stride] f16 scales. One thread per block.
__global__ void repack_q8_0_dense_kernel(const uint8_t *src, uint8_t *dst, long long nblocks, int nb) {
    const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (i >= nblocks) return;
    const long long row = i / nb, stride = dense_row_stride(nb), o = row * stride + (i - row * nb);
    const uint8_t *s = src + i * 34;
    uint8_t *q = dst + o * 32;
    uint16_t *d = reinterpret_cast<uint16_t *>(dst + nblocks / nb * stride * 32) + o;
    *d = static_cast<uint16_t>(s[0] | (s[1] << 8));
    for (int j = 0; j < 32; ++j) q[j] = s[2 + j];
}

// The attention of one query head over cache positions 0..pos by one CTA of `nthreads` threads. qs: the rotated q head,
// kn / vn: the new (rotated) k and the new v of position pos (shared memory); kc / vc: the head's KV group in the
// caches, row stride kv_dim; sc: [max_ctx] scores; vbuf: [32][head_dim] staging for the values. Returns the head's
// output element `tid` to threads tid < head_dim. Order (the oracle's): score_t = lane-strided fmaf dot + butterfly,
// times inv_sqrt; m = max; p_t = exp(score_t - m); l and out ascending in t. The loads are arranged so that a warp's
// keys are in flight together and the values come through shared memory in chunks of 32 positions.
__device__ __forceinline__ float dense_attention_core(const float *qs, const float *kn, const float *vn, const float *kc, const float *vc,
                                                      int pos, int kv_dim, int head_dim, float inv_sqrt, float *sc, float *vbuf,
                                                      int nthreads) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = nthreads >> 5;
    const float q0 = qs[lane], q1 = lane + 32 < head_dim ? qs[lane + 32] : 0.0f, q2 = lane + 64 < head_dim ? qs[lane + 64] : 0.0f,
                q3 = lane + 96 < head_dim ? qs[lane + 96] : 0.0f;
#pragma unroll 1
    for (int t0 = warp; t0 <= pos; t0 += 8 * nw) {
        float k0[8], k1[8], k2[8], k3[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {               // every position's loads leave before the first dot
            const int t = t0 + i * nw;
            k0[i] = k1[i] = k2[i] = k3[i] = 0.0f;
            if (t <= pos) {
                const float *k = t == pos ? kn : kc + static_cast<size_t>(t) * kv_dim;
                k0[i] = k[lane];
                if (lane + 32 < head_dim) k1[i] = k[lane + 32];
                if (lane + 64 < head_dim) k2[i] = k[lane + 64];
                if (lane + 96 < head_dim) k3[i] = k[lane + 96];
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int t = t0 + i * nw;
            if (t <= pos) {
                float acc = __fmaf_rn(q0, k0[i], 0.0f);
                if (head_dim > 32) acc = __fmaf_rn(q1, k1[i], acc);
                if (head_dim > 64) acc = __fmaf_rn(q2, k2[i], acc);
                if (head_dim > 96) acc = __fmaf_rn(q3, k3[i], acc);
#pragma unroll
                for (int s = 16; s >= 1; s >>= 1) acc = __fadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, s));
                if (lane == 0) sc[t] = __fmul_rn(acc, inv_sqrt);
            }
        }
    }
    __syncthreads();
    float m = -INFINITY;
    for (int t = 0; t <= pos; ++t) m = sc[t] > m ? sc[t] : m;
    __syncthreads();
    for (int t = tid; t <= pos; t += nthreads) sc[t] = exp_ggml(__fadd_rn(sc[t], -m));
    float l = 0.0f, acc = 0.0f;
#pragma unroll 1
    for (int c0 = 0; c0 < pos; c0 += 32) {
        const int n = min(32, pos - c0);
        __syncthreads();                            // the scores are final; the previous chunk has been consumed
        for (int i = tid; i < n * head_dim; i += nthreads) {
            const int r = i / head_dim, d = i - r * head_dim;
            vbuf[i] = vc[static_cast<size_t>(c0 + r) * kv_dim + d];
        }
        __syncthreads();
        if (tid < head_dim) {
            for (int r = 0; r < n; ++r) {
                const float p = sc[c0 + r];
                l = __fadd_rn(l, p);
                acc = __fmaf_rn(p, vbuf[r * head_dim + tid], acc);
            }
        }
    }
    __syncthreads();
    if (tid < head_dim) {
        l = __fadd_rn(l, sc[pos]);
        acc = __fmaf_rn(sc[pos], vn[tid], acc);
        return __fdiv_rn(acc, l);
    }
    return 0.0f;
}

// Two floats per instruction (each half rounded like the scalar operation).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// The dot q . k of the one-token order - lane l runs fmaf over d = l, l + 32, ..., then the butterfly - by ONE thread, two
// lanes per instruction: quads of lanes meet in the butterfly's own pairs (16 apart, 8 apart, 4, 2, 1), so nothing is shuffled.
// key(e): elements 4 e .. 4 e + 3 of the key.
template <int HD, class Key>
__device__ __forceinline__ float lane_order_dot(const float *q, Key key) {
    auto quad = [&](int b, f32x2 (&a)[2]) {         // lanes 4 b .. 4 b + 3
        a[0] = a[1] = 0ull;
#pragma unroll
        for (int r = 0; r < HD / 32; ++r) {
            const ulonglong2 qv = *reinterpret_cast<const ulonglong2 *>(q + r * 32 + b * 4), kv = key(r * 8 + b);
            a[0] = fma2(qv.x, kv.x, a[0]);
            a[1] = fma2(qv.y, kv.y, a[1]);
        }
    };
    f32x2 s8[2][2];
#pragma unroll
    for (int p = 0; p < 2; ++p) {                   // lanes 4 p .. 4 p + 3 with those 16, 8 and 24 above
        f32x2 a[2], b[2], c[2], d[2];
        quad(p, a);
        quad(p + 4, b);
        quad(p + 2, c);
        quad(p + 6, d);
#pragma unroll
        for (int i = 0; i < 2; ++i) s8[p][i] = add2(add2(a[i], b[i]), add2(c[i], d[i]));
    }
    float e0, e1;
    unpack2(add2(add2(s8[0][0], s8[1][0]), add2(s8[0][1], s8[1][1])), e0, e1);      // lanes (0, 1) + (2, 3)
    return __fadd_rn(e0, e1);
}
// Maximum over the lanes of a warp (no NaN among them).
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// Loads from shared memory, at a window address plus a constant, that keep their place among others of their kind.
template <int OFF>
__device__ __forceinline__ float lds_here(uint32_t a) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1 + %2];" : "=f"(v) : "r"(a), "n"(OFF));
    return v;
}
template <int OFF>
__device__ __forceinline__ float4 lds4_here(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4 + %5];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a), "n"(OFF));
    return v;
}
// The attention's sums over positions, one element per thread: l += p[t], acc = fmaf(p[t], v[t], acc), t ascending. p at p_at, v every ROW
// bytes from v_at on. A step is two dependent instructions of 4.7 cycles, but a shared-memory load takes a warp's issue for about five, and the
// compiler does not keep loads ahead of the chain by itself: eight steps run between the loads of the next eight (7 cycles a step, before 12).
struct WeightedEight {
    float4 w[2];
    float x[8];
};
template <int ROW, int I>
__device__ __forceinline__ void weighted_load(WeightedEight &b, uint32_t p_at, uint32_t v_at) {
    if constexpr (I % 4 == 0) b.w[I / 4] = lds4_here<I * 4>(p_at);
    b.x[I] = lds_here<I * ROW>(v_at);
}
template <int ROW, int I = 0>
__device__ __forceinline__ void weighted_load_all(WeightedEight &b, uint32_t p_at, uint32_t v_at) {
    weighted_load<ROW, I>(b, p_at, v_at);
    if constexpr (I < 7) weighted_load_all<ROW, I + 1>(b, p_at, v_at);
}
__device__ __forceinline__ void weighted_step(float &l, float &acc, float w, float x) {       // in place among the loads
    asm volatile("add.rn.f32 %0, %0, %1;" : "+f"(l) : "f"(w));
    asm volatile("fma.rn.f32 %0, %1, %2, %0;" : "+f"(acc) : "f"(w), "f"(x));
}
template <int ROW, int I = 0>
__device__ __forceinline__ void weighted_eight(float &l, float &acc, const WeightedEight &now, WeightedEight &next, uint32_t p_at, uint32_t v_at) {
    weighted_load<ROW, I>(next, p_at, v_at);
    const float4 &w = now.w[I / 4];
    weighted_step(l, acc, I % 4 == 0 ? w.x : I % 4 == 1 ? w.y : I % 4 == 2 ? w.z : w.w, now.x[I]);
    if constexpr (I < 7) weighted_eight<ROW, I + 1>(l, acc, now, next, p_at, v_at);
}
template <int ROW>
__device__ __forceinline__ void weighted_sum(float &l, float &acc, const float *p, const float *v, int n) {
    const uint32_t p0 = smem_u32(p), v0 = smem_u32(v);
    const int eights = n >> 3;
    if (eights > 0) {
        WeightedEight a, b;
        weighted_load_all<ROW>(a, p0, v0);
        int k = 0;
        auto at = [&](int i) { return i < eights ? i : 0; };      // past the end: loads that nobody uses, of what is there
#pragma unroll 1
        for (; k + 2 <= eights; k += 2) {
            weighted_eight<ROW>(l, acc, a, b, p0 + (k + 1) * 32, v0 + (k + 1) * (8 * ROW));
            weighted_eight<ROW>(l, acc, b, a, p0 + at(k + 2) * 32, v0 + at(k + 2) * (8 * ROW));
        }
        if (k < eights) weighted_eight<ROW>(l, acc, a, b, p0, v0);
    }
    const int r = eights * 8;
    if (r < n) {            // fewer than eight are left: requested together
        float w[7], x[7];
#pragma unroll
        for (int i = 0; i < 7; ++i) {
            w[i] = lds_here<0>(p0 + min(r + i, n - 1) * 4);
            x[i] = lds_here<0>(v0 + min(r + i, n - 1) * ROW);
        }
#pragma unroll
        for (int i = 0; i < 7; ++i)
            if (r + i < n) weighted_step(l, acc, w[i], x[i]);
    }
}

// The same sums, 32 positions' loads at a time in front of their chains; ROW in floats.
template <int ROW>
__device__ __forceinline__ void weighted_sum_batches(float &l, float &acc, const float *p, const float *v, int n) {
    int r = 0;
    for (; r + 32 <= n; r += 32) {
        float4 w[8];
        float x[32];
#pragma unroll
        for (int i = 0; i < 8; ++i) w[i] = *reinterpret_cast<const float4 *>(p + r + 4 * i);
#pragma unroll
        for (int i = 0; i < 32; ++i) x[i] = v[(r + i) * ROW];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            l = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(l, w[i].x), w[i].y), w[i].z), w[i].w);
            acc = __fmaf_rn(w[i].x, x[4 * i], acc);
            acc = __fmaf_rn(w[i].y, x[4 * i + 1], acc);
            acc = __fmaf_rn(w[i].z, x[4 * i + 2], acc);
            acc = __fmaf_rn(w[i].w, x[4 * i + 3], acc);
        }
    }
    for (; r < n; ++r) {
        l = __fadd_rn(l, p[r]);
        acc = __fmaf_rn(p[r], v[r * ROW], acc);
    }
}

// Asynchronous 16-byte copy global -> shared; !live fills the destination with zeros.
__device__ __forceinline__ void cp_async16(void *dst, const void *src, bool live) {
    const int bytes = live ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Cluster of CTAs that share one head: a barrier in two halves, and a store into a peer's shared memory.
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void store_peer(float *p, uint32_t rank, float v) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}

// Geometry of the decode attention for a head dimension and C CTAs per head: chunks of 64 key rows, and of 64 C value rows of
// HD / C elements, in padded rows, so that neighbouring positions start in different banks.
template <int HD, int C>
struct DecodeAttn {
    static constexpr int kThreads = 512, kChunk = 64, kRow = HD + 4, kSlice = HD / C, kChunkV = kChunk * C, kRowV = kSlice + 4;
    static constexpr int kSlot = kChunk * kRow > kChunkV * kRowV ? kChunk * kRow : kChunkV * kRowV;      // floats
    static constexpr int kSlotBytes = kSlot * 4;
    static constexpr int kRoom = 190 * 1024;                    // slots and scores together; the rest of an SM is for the product before it
    // Values longer than the ring are refilled: after chunk c is consumed, chunk c + slots is requested, and chunk c + 1 is read once
    // all but the kInFlight youngest requests have landed. It was requested `slots` - 1 requests before the youngest.
    static constexpr int kInFlight = 3;
    static_assert((kRoom - kDenseMaxCtx * 4) / kSlotBytes > kInFlight, "a refilled chunk would be read before it has landed");
    static int want(int max_ctx) { return ((max_ctx + kChunk - 1) / kChunk + C - 1) / C + (max_ctx + kChunkV - 1) / kChunkV; }
    // slots of the ring: both caches of the longest context, or what fits beside its scores
    static int slots(int max_ctx) {
        const int fit = (kRoom - max_ctx * 4) / kSlotBytes, w = want(max_ctx);
        return w < fit ? w : fit;
    }
};

// Rotary embedding + cache store + decode attention + Q8_0 of the head's output, one CTA per query head (rope_store_kernel
// :1855 and attention_decode_kernel :1902 of src/warodecode.cu, the latter as two passes; orders in the header and in the
// oracle). The rotary embedding pairs element p with p + head_dim / 2 (GPT-NeoX) and takes cos/sin from the table row of
// *pos. Every CTA rotates its own q head and, for itself, the new k head of its KV group; the first CTA of a group also
// stores the rotated k and the v into the caches [max_ctx][kv_dim]. Cache position pos itself is taken from the CTA's own
// copy, so no CTA waits for another's store.
//
// Bound: latency. The sums over positions run ascending (one fmaf per position and element, four cycles each), so the
// keys and values must be there when they are needed: the cache below pos was written by earlier tokens, and the first
// chunks of it (all of it up to 320 positions of 64) are copied to shared memory in a ring, keys before values,
// requested BEFORE the wait for the QKV product; a score is one thread's work, without shuffles.
// Measured per layer inside the step of the 16-layer model (32 heads of 64), from the end of the kernel in front: 2.2 us at 77 positions (2.8
// before the sums' loads ran ahead of their chains), 4.6 us at 485 (5.2), of which the sums 2.3; by one CTA per head 0.9 us more there.
//
// C: CTAs per head, a cluster. One CTA takes in 512 bytes per position through its SM, and once a context is longer than its
// ring holds, the last values only follow when the first keys have been scored. With C = HD / 32 each CTA scores every C-th
// chunk of keys, stores the scores into its peers' shared memory too, and sums 32 elements of the values (one Q8_0 block) over
// all positions: the orders stay, an SM takes in 1 / C of the bytes. For decoders whose longest context does not fit one ring.
//
// EXTRAS: the layer has q/k/v biases (Qwen2-style files: added to the QKV product's rows) and / or RMSNorm weights for
// the q and k heads (Qwen3-style: qk_norm_kernel, src/warodecode.cu:1836), applied in that order before the rotary
// embedding (emit_step :2069-2075). Layers without them run the instantiation that has none of that code.
// LONG (heads of 64 elements in clusters, contexts that may outgrow the ring): the sums chunk by chunk, 32 positions' loads at a time, because chunks of
// 128 positions leave loads that run ahead of the chains too little to hide behind at either end. Four layers of 32 heads, per token: 2,000
// positions 141.5 us in this form, 149 in the other; 8,000 positions 411 and 439; 500 positions 75.0 and 73.3. At most 64 registers, so that the
// kernel can start beside the product in front (68: 20 positions 58.4 -> 62.3 us). The other head sizes gain from the loads ahead at every length.
// Dynamic shared memory: `slots` chunks, then max_ctx scores.
template <int HD, bool EXTRAS, int C, bool LONG>
__global__ void __launch_bounds__(DecodeAttn<HD, C>::kThreads, LONG ? 2 : 0) dense_attention_kernel(const float *qkv, const float *table, float *kcache,
                                                                                 float *vcache, const int *pos_ptr, int heads,
                                                                                 int kv_heads, int slots, float inv_sqrt, int8_t *oq,
                                                                                 float *od, const float *bqkv, const float *q_norm,
                                                                                 const float *k_norm, float eps) {
    using A = DecodeAttn<HD, C>;
    constexpr int kNt = A::kThreads, kChunk = A::kChunk, kRow = A::kRow, kHalf = HD / 2, kRow16 = HD / 4;
    constexpr int kSlice = A::kSlice, kChunkV = A::kChunkV, kRowV = A::kRowV, kSlice16 = kSlice / 4;
    extern __shared__ __align__(16) float vring[];
    __shared__ __align__(16) float qs[HD], kn[HD];
    __shared__ float vn[HD], outv[kSlice], wmax[kNt / 32];
    float *sc = vring + static_cast<size_t>(slots) * A::kSlot;
    grid_dep_launch();
    if constexpr (C > 1) cluster_arrive();          // answered before the first store into a peer
    const int rank = C > 1 ? static_cast<int>(cluster_rank()) : 0;
    const int h = blockIdx.x / C, tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    // The position comes from the finish kernel of the token before. That kernel has ended (it releases nothing early), but this is in
    // front of the wait, so its store is ordered by the fence behind it and read past L1.
    int pos;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(pos) : "l"(pos_ptr) : "memory");
    pos = __shfl_sync(0xffffffffu, pos, 0);         // the same in every lane, and known to be
    const int kv_dim = kv_heads * HD, kvh = (h * kv_heads) / heads;
    float *kc = kcache + static_cast<size_t>(kvh) * HD, *vc = vcache + static_cast<size_t>(kvh) * HD;
    // positions 0 .. pos - 1: this CTA's key chunks (every C-th), then all value chunks of its slice
    const int n_chunks = ((pos + kChunk - 1) / kChunk - rank + C - 1) / C, n_vchunks = (pos + kChunkV - 1) / kChunkV, n_items = n_chunks + n_vchunks;
    auto slot_of = [&](int item) { return vring + static_cast<size_t>(item % slots) * A::kSlot; };
    auto request = [&](int item) {
        if (item >= n_items) return;
        float *dst = slot_of(item);
        if (item < n_chunks) {
            const int t0 = (item * C + rank) * kChunk;
            for (int i = tid; i < kChunk * kRow16; i += kNt) {
                const int r = i / kRow16, e = i - r * kRow16;
                if (t0 + r < pos) cp_async16(dst + r * kRow + e * 4, kc + static_cast<size_t>(t0 + r) * kv_dim + e * 4, true);
            }
        } else {
            const int t0 = (item - n_chunks) * kChunkV;
            for (int i = tid; i < kChunkV * kSlice16; i += kNt) {
                const int r = i / kSlice16, e = i - r * kSlice16;
                if (t0 + r < pos) cp_async16(dst + r * kRowV + e * 4, vc + static_cast<size_t>(t0 + r) * kv_dim + rank * kSlice + e * 4, true);
            }
        }
    };
    for (int i = 0; i < min(slots, n_chunks); ++i) request(i);
    cp_async_commit();
    for (int i = n_chunks; i < min(slots, n_items); ++i) request(i);
    cp_async_commit();
    float cs = 0.0f, sn = 0.0f;
    if (tid < kHalf) {
        cs = table[(static_cast<size_t>(pos) * kHalf + tid) * 2];
        sn = table[(static_cast<size_t>(pos) * kHalf + tid) * 2 + 1];
    }
    grid_dep_wait();
    const float *q_raw = qkv + static_cast<size_t>(h) * HD;
    const float *k_raw = qkv + static_cast<size_t>(heads + kvh) * HD;
    const float *v_raw = qkv + static_cast<size_t>(heads + kv_heads + kvh) * HD;
    if constexpr (EXTRAS) {
        __shared__ float qn[HD], kn_in[HD], vn_in[HD];
        __shared__ double nred[2][4];
        float xq_ = 0.0f, xk_ = 0.0f, xv_ = 0.0f;
        if (tid < HD) {
            xq_ = q_raw[tid];
            xk_ = k_raw[tid];
            xv_ = v_raw[tid];
            if (bqkv != nullptr) {
                xq_ = __fadd_rn(xq_, bqkv[static_cast<size_t>(h) * HD + tid]);
                xk_ = __fadd_rn(xk_, bqkv[static_cast<size_t>(heads + kvh) * HD + tid]);
                xv_ = __fadd_rn(xv_, bqkv[static_cast<size_t>(heads + kv_heads + kvh) * HD + tid]);
            }
        }
        if (q_norm != nullptr || k_norm != nullptr) {
            // the sum of squares is the binary tree in double over the head's elements, zero-padded to 128 leaves (adding
            // +0.0 changes nothing), thread t owns leaf t
            double sq_ = __dmul_rn(static_cast<double>(xq_), static_cast<double>(xq_));
            double sk_ = __dmul_rn(static_cast<double>(xk_), static_cast<double>(xk_));
#pragma unroll
            for (int s = 1; s < 32; s <<= 1) {
                sq_ = __dadd_rn(sq_, __shfl_xor_sync(0xffffffffu, sq_, s));
                sk_ = __dadd_rn(sk_, __shfl_xor_sync(0xffffffffu, sk_, s));
            }
            if (lane == 0 && warp < 4) {
                nred[0][warp] = sq_;
                nred[1][warp] = sk_;
            }
            __syncthreads();
            const double tq = __dadd_rn(__dadd_rn(nred[0][0], nred[0][1]), __dadd_rn(nred[0][2], nred[0][3]));
            const double tk = __dadd_rn(__dadd_rn(nred[1][0], nred[1][1]), __dadd_rn(nred[1][2], nred[1][3]));
            const double hd = static_cast<double>(HD), ep = static_cast<double>(eps);
            const float scq = __double2float_rn(__ddiv_rn(1.0, __dsqrt_rn(__dadd_rn(__ddiv_rn(tq, hd), ep))));
            const float sck = __double2float_rn(__ddiv_rn(1.0, __dsqrt_rn(__dadd_rn(__ddiv_rn(tk, hd), ep))));
            if (tid < HD) {
                if (q_norm != nullptr) xq_ = __fmul_rn(__fmul_rn(xq_, scq), q_norm[tid]);
                if (k_norm != nullptr) xk_ = __fmul_rn(__fmul_rn(xk_, sck), k_norm[tid]);
            }
        }
        if (tid < HD) {
            qn[tid] = xq_;
            kn_in[tid] = xk_;
            vn_in[tid] = xv_;
        }
        __syncthreads();
        q_raw = qn;
        k_raw = kn_in;
        v_raw = vn_in;
    }
    const bool writer = h % (heads / kv_heads) == 0 && rank == 0;       // the first head of its KV group
    if (tid < kHalf) {
        const float a = q_raw[tid], b = q_raw[tid + kHalf], c = k_raw[tid], d = k_raw[tid + kHalf];
        const float v0 = v_raw[tid], v1 = v_raw[tid + kHalf];
        qs[tid] = __fadd_rn(__fmul_rn(a, cs), -__fmul_rn(b, sn));
        qs[tid + kHalf] = __fadd_rn(__fmul_rn(a, sn), __fmul_rn(b, cs));
        const float k0 = __fadd_rn(__fmul_rn(c, cs), -__fmul_rn(d, sn)), k1 = __fadd_rn(__fmul_rn(c, sn), __fmul_rn(d, cs));
        kn[tid] = k0;
        kn[tid + kHalf] = k1;
        vn[tid] = v0;
        vn[tid + kHalf] = v1;
        if (writer) {
            const size_t off = static_cast<size_t>(pos) * kv_dim;
            kc[off + tid] = k0;
            kc[off + tid + kHalf] = k1;
            vc[off + tid] = v0;
            vc[off + tid + kHalf] = v1;
        }
    }
    __syncthreads();
    if constexpr (C > 1) cluster_wait();        // the peers run
    auto key_row = [](const float *k) { return [k](int e) { return *reinterpret_cast<const ulonglong2 *>(k + 4 * e); }; };
    float m = -INFINITY;
    const int batch = min(kNt / kChunk, slots);         // key chunks scored side by side, one position per thread
#pragma unroll 1
    for (int c0 = 0; c0 < max(n_chunks, 1); c0 += batch) {
        if (c0 == 0) cp_async_wait<1>();
        else cp_async_wait<0>();
        __syncthreads();
        const int c = c0 + tid / kChunk, t = (c * C + rank) * kChunk + (tid & (kChunk - 1));
        const bool newest = c0 == 0 && tid == kNt - 1;
        if ((tid < batch * kChunk && c < n_chunks && t < pos) || newest) {
            // the last thread scores the new position, and an old one too when it has one
            if (!newest || (tid < batch * kChunk && t < pos)) {
                const float v = __fmul_rn(lane_order_dot<HD>(qs, key_row(slot_of(c) + (tid & (kChunk - 1)) * kRow)), inv_sqrt);
                sc[t] = v;
                if constexpr (C > 1) {
#pragma unroll
                    for (int r = 1; r < C; ++r) store_peer(sc + t, rank + r < C ? rank + r : rank + r - C, v);
                }
                m = v > m ? v : m;          // a NaN score never becomes the maximum
            }
            if (newest) {
                const float v = __fmul_rn(lane_order_dot<HD>(qs, key_row(kn)), inv_sqrt);
                sc[pos] = v;
                m = v > m ? v : m;
            }
        }
        if (n_items > slots) {
            __syncthreads();
            for (int k = c0; k < min(c0 + batch, n_chunks); ++k) request(k + slots);
            cp_async_commit();
        }
    }
    if constexpr (C > 1) {          // all scores are here; nothing is stored into a peer after this
        cluster_arrive();
        cluster_wait();
        for (int t = tid; t <= pos; t += kNt) m = sc[t] > m ? sc[t] : m;
    }
    m = warp_max(m);
    if (lane == 0) wmax[warp] = m;
    __syncthreads();
    m = warp_max(wmax[lane & (kNt / 32 - 1)]);
    for (int t = tid; t <= pos; t += kNt) sc[t] = exp_ggml(__fadd_rn(sc[t], -m));
    cp_async_wait<0>();
    __syncthreads();
    float l = 0.0f, acc = 0.0f;
    const bool whole = !LONG && n_items <= slots;       // everything is in the ring, and the value rows lie in a row: a slot is exactly its rows
    static_assert(A::kSlot == kChunkV * kRowV, "a slot of values ends where the next begins");
#pragma unroll 1
    for (int c = 0; c < (whole ? 1 : n_vchunks); ++c) {
        if (warp < kSlice / 32) {
            const int n = whole ? pos : min(kChunkV, pos - c * kChunkV);
            const float *p = sc + c * kChunkV, *v = slot_of(n_chunks + c) + tid;
            if constexpr (LONG) weighted_sum_batches<kRowV>(l, acc, p, v, n);
            else weighted_sum<kRowV * 4>(l, acc, p, v, n);
        }
        if (n_vchunks > slots) {     // longer than the ring: refill the slot
            __syncthreads();
            request(n_chunks + c + slots);
            cp_async_commit();
            cp_async_wait<A::kInFlight>();
            __syncthreads();
        }
    }
    if (tid < kSlice) {
        l = __fadd_rn(l, sc[pos]);
        acc = __fmaf_rn(sc[pos], vn[rank * kSlice + tid], acc);
        outv[tid] = __fdiv_rn(acc, l);
    }
    __syncthreads();
    if (warp < kSlice / 32) {
        const int b = (h * HD + rank * kSlice) / 32 + warp;
        q8_0_block_warp(outv[warp * 32 + lane], lane, oq + static_cast<size_t>(b) * 32, od + b);
    }
}

// y = W RMSNorm(hidden + proj) in one kernel: every CTA forms the norm and its Q8_0 form for itself (in shared memory), the
// first one also stores the sum. The norm is a chain of a load, two reductions and two divisions that one CTA of a kernel of
// its own took 3.2 us for, launch and hand-over included, while the other SMs waited; here it runs next to the weights that are
// already on their way (2.2 us from the end of the kernel in front to the first product). CTAs of 512 threads, two per SM, so
// that an SM reads hidden and proj twice and not four times.
// Measured, 16 layers of 2048 / 8192 and a 128256-row head, 72 positions: 376 us per token with separate norm, product and
// SwiGLU kernels, 303 with this kernel and its first weight loads in front of the wait (RowBlock::load_early; 342 behind it). Matrices of
// later kernels asked into L2 ahead of them gain nothing beside that: 305 us here, and where a layer's matrices approach the size of L2
// they cost 6 to 25 % (4096 / 16384: 220 -> 245 us with 5 Q4_0 layers, 188 -> 235 with 3 Q8_0 layers).
// MODE 0: y[row]; 1: rows are [ffn gate rows | ffn up rows], and a CTA takes 32 of both at once: SiLU(g) * u is quantised to
// Q8_0 where it is formed (swiglu_kernel, :1956), without a kernel and a pass over memory of its own; 2: y[row] and the
// arg-max of the finite results: key = order_key(value) << 32 | ~row, so the largest value wins and
// ties go to the lowest row (dense_argmax_reduce_kernel, :1603-1632). Rows: R per warp, U blocks per lane and row in flight. Dynamic shared memory:
// nb * 40 bytes.
constexpr int kNormProductThreads = 512;
template <bool Q8, int R, int U, int MODE, int PASSES, bool AHEAD>
__global__ void __launch_bounds__(kNormProductThreads, 2) dense_norm_product_kernel(NormInput in, const uint8_t *wp, int rows, float *y,
                                                                                   unsigned long long *key, int8_t *oq, float *od) {
    static_assert(MODE != 1 || R == 4, "two gate rows and two up rows per warp");
    constexpr int kWarpsHere = kNormProductThreads / 32;
    extern __shared__ __align__(16) uint8_t dsm[];
    __shared__ float outs[64];
    grid_dep_launch();
    if (blockIdx.x != 0) in.hidden_out = nullptr;
    const int nb = in.n >> 5, stride = dense_row_stride(nb), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const BlockInput x(dsm, nb);
    const uint4 *q_all = reinterpret_cast<const uint4 *>(wp);
    const uint16_t *d_all = reinterpret_cast<const uint16_t *>(wp + static_cast<size_t>(rows) * stride * (Q8 ? 32 : 16));
    auto row_of = [&](int unit, int r) {
        if constexpr (MODE == 1) return (r >> 1) * (rows >> 1) + unit * 32 + warp * 2 + (r & 1);
        return (unit * kWarpsHere + warp) * R + r;
    };
    const int units = MODE == 1 ? rows >> 6 : (rows + kWarpsHere * R - 1) / (kWarpsHere * R);
    // AHEAD: a long walk over rows asks for the next blocks before it multiplies the ones in hand (see dense_launch_norm_product)
    static_assert(!AHEAD || U == 1, "one block per lane and row ahead");
    RowBlock<Q8> w[R][U], next[AHEAD ? R : 1][U];
    auto load = [&](RowBlock<Q8> (*to)[U], int unit, int b0, bool early) {
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int b = b0 + 32 * u, row = row_of(unit, r);
                if (b < nb && (MODE == 1 || row < rows)) {
                    const size_t blk = static_cast<size_t>(row) * stride + b;
                    if (early) to[r][u].load_early(q_all, d_all, blk);
                    else to[r][u].load(q_all, d_all, blk);
                }
            }
    };
    int unit = blockIdx.x;
    load(w, unit, lane, true);           // weights do not depend on the kernel before this one
    dense_norm_quant_body<PASSES>(in, [] { grid_dep_wait(); }, [&](int e, uint32_t packed, float d) {
        const int b = e >> 5, j = e & 31;
        *reinterpret_cast<uint32_t *>(reinterpret_cast<uint8_t *>((j & 16) ? x.hi + b : x.lo + b) + (j & 15)) = packed;
        int sum = dp4a_s8(static_cast<int>(packed), 0x01010101, 0);
#pragma unroll
        for (int s = 1; s < 8; s <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, s);
        if (j == 0) x.x[b] = make_int2(__float_as_int(d), -8 * sum);
    });
    __syncthreads();
    unsigned long long best = 0ull;
    for (; unit < units; unit += gridDim.x) {
        float acc[R];
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r] = 0.0f;
#pragma unroll 1
        for (int b0 = lane; b0 < nb; b0 += 32 * U) {
            if constexpr (AHEAD) {
                const bool wrap = b0 + 32 >= nb;
                const int unit2 = wrap ? unit + static_cast<int>(gridDim.x) : unit;
                if (unit2 < units) load(next, unit2, wrap ? lane : b0 + 32, true);
            } else if (unit != static_cast<int>(blockIdx.x) || b0 != lane) {
                load(w, unit, b0, false);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int b = b0 + 32 * u;
                if (b < nb) {
                    const uint4 lo = x.lo[b], hi = x.hi[b];
                    const int2 d = x.x[b];
#pragma unroll
                    for (int r = 0; r < R; ++r)
                        if (MODE == 1 || row_of(unit, r) < rows) acc[r] = w[r][u].term(lo, hi, d, acc[r]);
                }
            }
            if constexpr (AHEAD) {
#pragma unroll
                for (int r = 0; r < R; ++r) w[r][0] = next[r][0];
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
#pragma unroll
            for (int s = 16; s >= 1; s >>= 1) acc[r] = __fadd_rn(acc[r], __shfl_xor_sync(0xffffffffu, acc[r], s));
        }
        float v = acc[0];
#pragma unroll
        for (int r = 1; r < R; ++r) v = lane == r ? acc[r] : v;
        if constexpr (MODE == 1) {
            if (lane < R) outs[(lane >> 1) * 32 + warp * 2 + (lane & 1)] = v;
            __syncthreads();
            if (warp == 0) q8_0_block_warp(__fmul_rn(silu_ggml(outs[lane]), outs[32 + lane]), lane, oq + unit * 32, od + unit);
            __syncthreads();
        } else {
            const int row = row_of(unit, lane);
            if (lane < R && row < rows) {
                y[row] = v;
                if (MODE == 2 && v == v && fabsf(v) != INFINITY) {
                    const unsigned long long k = (static_cast<unsigned long long>(order_key(v)) << 32) | (0xffffffffu - static_cast<unsigned>(row));
                    best = k > best ? k : best;
                }
            }
        }
    }
    if constexpr (MODE == 2) {      // one atomic per CTA
        __shared__ unsigned long long bests[kWarpsHere];
#pragma unroll
        for (int s = 1; s < R; s <<= 1) {
            const unsigned long long o = __shfl_xor_sync(0xffffffffu, best, s);
            best = o > best ? o : best;
        }
        if (lane == 0) bests[warp] = best;
        __syncthreads();
        if (warp == 0) {
            best = bests[lane & (kWarpsHere - 1)];
#pragma unroll
            for (int s = 1; s < kWarpsHere; s <<= 1) {
                const unsigned long long o = __shfl_xor_sync(0xffffffffu, best, s);
                best = o > best ? o : best;
            }
            if (lane == 0 && best != 0ull) atomicMax(key, best);
        }
    }
}

// End of a step: the arg-max key becomes the next token (0 when no logit was finite), is recorded at out[pos + 1],
// the position advances, the key is cleared for the next step (dense_argmax_finish_kernel + increment_pos_kernel).
// `forced` (nullable): forced[pos + 1] >= 0 replaces the generated token (prompt tokens).
// The next token's attention reads the position in front of its wait, so its store is followed by a fence; a second warp does that beside the
// token's own chain (in the same thread it costs 0.6 us per token, 1.2 % of a four-layer model's).
constexpr int kFinishThreads = 64;
__global__ void __launch_bounds__(kFinishThreads) dense_finish_kernel(unsigned long long *key, int *token, int *pos, int *out, const int *forced) {
    grid_dep_wait();
    const int p = *pos + 1;
    __syncthreads();            // both warps have the old position
    if (threadIdx.x == 32) {
        *pos = p;
        __threadfence();
    }
    if (threadIdx.x == 0) {
        const unsigned long long k = *key;
        int t = k == 0ull ? 0 : static_cast<int>(0xffffffffu - static_cast<unsigned>(k & 0xffffffffull));
        if (forced != nullptr && forced[p] >= 0) t = forced[p];
        out[p] = t;
        *token = t;
        *key = 0ull;
    }
}

}  // namespace wd
