// The plain-layout MoE block on WIDE expert tensors (wd_formats.cuh: one 4-bit code per weight), for engines whose experts
// fit the GPU in that form; wd_plain_moe.cuh has the same two kernels on tensors as the file holds them.
//
// Layout: 144 bytes per 256 weights for every type, rows and experts contiguous as in the file.
//   IQ3_S, IQ2_S  per superblock: 128 bytes of codes ([sub-block][word k = chunks k and k + 4], as in a wide tile), 8 bytes of
//                 scale nibbles (four used by IQ3_S), f16 block scale, 6 bytes unused. The 144-byte stride puts the
//                 superblocks that neighbouring lanes read into different banks.
//   IQ4_NL        per row: [block][16 bytes: word l = codes of chunk l in its low 16 bits, of chunk l + 4 in its high 16],
//                 then the f16 scales: 18 bytes per 32 weights as in the file, only the nibbles reordered so that prmt can
//                 take a chunk's four codes as one selector.
// What bounded the kernels on the file's bytes was instruction issue (codebook lookups from shared memory, sign masks,
// byte tables: about 5 instructions per weight and lane); here a lane needs about one.
#pragma once

#include "wd_plain_moe.cuh"

namespace wd {

constexpr int kPlainSb = 144;

__host__ __device__ inline size_t plain_wide_row_bytes(int cols) { return static_cast<size_t>(cols / 64) * (kPlainSb / 4); }

// ggml blocks -> wide rows. One thread per superblock (IQ types) or per block of 32 (IQ4_NL); `rows` rows of `cols`.
__global__ void plain_repack_wide_kernel(int type, const uint8_t *__restrict__ src, uint8_t *__restrict__ dst, long long rows, int cols,
                                         const uint16_t *__restrict__ grid3, const uint16_t *__restrict__ grid2) {
    const int per_row = type == kTypeIq4nl ? cols / 32 : cols / 256;
    const long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (i >= rows * per_row) return;
    const long long row = i / per_row;
    const int b = static_cast<int>(i - row * per_row);
    if (type == kTypeIq4nl) {
        const uint8_t *s = src + i * 18;
        uint8_t *r = dst + row * plain_wide_row_bytes(cols);
        for (int l = 0; l < 4; ++l) {
            uint32_t w = 0;
            for (int j = 0; j < 4; ++j) {
                const uint32_t v = s[2 + 4 * l + j];
                w |= (v & 15u) << (4 * j) | (v >> 4) << (16 + 4 * j);
            }
            uint8_t *o = r + b * 16 + l * 4;            // a row starts on 36 bytes times cols / 64: four-byte aligned
            *reinterpret_cast<uint32_t *>(o) = w;
        }
        *reinterpret_cast<uint16_t *>(r + static_cast<size_t>(per_row) * 16 + b * 2) = static_cast<uint16_t>(s[0] | (s[1] << 8));
        return;
    }
    uint8_t *o = dst + i * kPlainSb;
    if (type == kTypeIq2s) {
        const uint8_t *s = src + i * 82, *qs = s + 2, *sg = s + 34, *qh = s + 66, *sc = s + 74;
        for (int k = 0; k < 8; ++k) {
            uint32_t w[4] = {0, 0, 0, 0};
            for (int c = 0; c < 8; ++c) {
                const uint32_t m = grid2[qs[k * 4 + (c >> 1)] | (((qh[k] >> (2 * (c >> 1))) & 3) << 8)] >> (8 * (c & 1));
                const uint32_t sign = sg[k * 4 + (c >> 1)] >> (4 * (c & 1));
                for (int j = 0; j < 4; ++j) w[c & 3] |= (((m >> (2 * j)) & 3u) | (((sign >> j) & 1u) << 2)) << (4 * j + 16 * (c >> 2));
            }
            *reinterpret_cast<uint4 *>(o + k * 16) = make_uint4(w[0], w[1], w[2], w[3]);
            o[128 + k] = sc[k];
        }
        *reinterpret_cast<uint16_t *>(o + 136) = static_cast<uint16_t>(s[0] | (s[1] << 8));
    } else {
        const uint8_t *s = src + i * 110, *qs = s + 2, *qh = s + 66, *sg = s + 74;
        for (int k = 0; k < 8; ++k) {
            uint32_t w[4] = {0, 0, 0, 0};
            for (int c = 0; c < 8; ++c) {
                const uint32_t m = grid3[qs[k * 8 + c] | (((qh[k] >> c) & 1) << 8)], sign = sg[k * 4 + (c >> 1)] >> (4 * (c & 1));
                for (int j = 0; j < 4; ++j)
                    w[c & 3] |= (((m >> (3 * j)) & 7u) ^ (((sign >> j) & 1u) ? 15u : 0u)) << (8 * j + 4 * (c >> 2));
            }
            *reinterpret_cast<uint4 *>(o + k * 16) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        for (int k = 0; k < 4; ++k) o[128 + k] = s[106 + k];
        *reinterpret_cast<uint16_t *>(o + 136) = static_cast<uint16_t>(s[0] | (s[1] << 8));
    }
}

// The eight integer sums of one superblock (one lane, all of it) against the Q8_K quants at `a` (16-byte aligned).
__device__ __forceinline__ void plain_wide_unit(int type, const uint8_t *blk, const int8_t *a, int p[8]) {
    const uint4 *qv = reinterpret_cast<const uint4 *>(blk), *av = reinterpret_cast<const uint4 *>(a);
    const uint2 sc = *reinterpret_cast<const uint2 *>(blk + 128);
#pragma unroll
    for (int c = 0; c < 8; ++c) p[c] = 0;
    if (type == kTypeIq2s) {
        const uint32_t pos = 0x3b2b1908u, neg = 0xc5d5e7f8u;
#pragma unroll 4
        for (int i = 0; i < 8; ++i) {
            const uint4 q = qv[i], lo = av[2 * i], hi = av[2 * i + 1];
            const uint32_t scb = ((i & 4) ? sc.y : sc.x) >> (8 * (i & 3));
            const int ls_lo = 1 + 2 * static_cast<int>(scb & 15u), ls_hi = 1 + 2 * static_cast<int>((scb >> 4) & 15u);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t w = word_of(q, k);
                p[k] += dp4a_s8(static_cast<int>(prmt(pos, neg, w)), static_cast<int>(word_of(lo, k)), 0) * ls_lo;
                p[k + 4] += dp4a_s8(static_cast<int>(prmt(pos, neg, w >> 16)), static_cast<int>(word_of(hi, k)), 0) * ls_hi;
            }
        }
    } else {
#pragma unroll 4
        for (int i = 0; i < 8; ++i) {
            const uint4 q = qv[i], lo = av[2 * i], hi = av[2 * i + 1];
            const int ls = 1 + 2 * static_cast<int>((sc.x >> (4 * i)) & 15u);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t w = word_of(q, k);
                p[k] += dp4a_s8(static_cast<int>(((w << 4) & 0xf0f0f0f0u) | 0x08080808u), static_cast<int>(word_of(lo, k)), 0) * ls;
                p[k + 4] += dp4a_s8(static_cast<int>((w & 0xf0f0f0f0u) | 0x08080808u), static_cast<int>(word_of(hi, k)), 0) * ls;
            }
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) p[c] >>= 3;
    }
}

// A row's superblocks in shared memory for the float side: [sb][8] sums, a stride that keeps four rows in different banks,
// and the scales d_w * d_x.
__host__ __device__ inline int plain_part_stride(int nsb) { return 8 * nsb + 8; }
__device__ __forceinline__ void plain_store_part(float *part, const int p[8]) {
    *reinterpret_cast<float4 *>(part) = make_float4(static_cast<float>(p[0]), static_cast<float>(p[1]), static_cast<float>(p[2]), static_cast<float>(p[3]));
    *reinterpret_cast<float4 *>(part + 4) = make_float4(static_cast<float>(p[4]), static_cast<float>(p[5]), static_cast<float>(p[6]), static_cast<float>(p[7]));
}
// chain of one (row, chunk-lane): one fmaf per superblock in order
__device__ __forceinline__ float plain_chain(const float *part, const float *d, int nsb, int c) {
    float acc = 0.0f;
#pragma unroll 5
    for (int s = 0; s < nsb; ++s) acc = __fmaf_rn(d[s], part[s * 8 + c], acc);
    return acc;
}

__host__ __device__ inline size_t plain_gate_up_wide_chunks_off(int H) { return (256 + static_cast<size_t>(H / 256) * kPlainActStride + 127) / 128 * 128; }
__host__ __device__ inline size_t plain_gate_up_wide_smem(int H) {
    const int nsb = H / 256;
    return plain_gate_up_wide_chunks_off(H) + static_cast<size_t>(32) * nsb * kPlainSb + 32 * static_cast<size_t>(plain_part_stride(nsb)) * 4 +
           32 * static_cast<size_t>(nsb) * 4;
}
inline int plain_gate_up_wide_threads(int H) { const int n = 32 * (H / 256); return n < 128 ? 128 : n > 512 ? 512 : n; }

// Gate and up rows: CTA = (slot j, sixteen consecutive rows of both matrices) of token blockIdx.y. A thread takes one
// superblock of one row (the model's 32 rows of ten superblocks are exactly 320 threads); the chains of a gate row and its
// up row then run side by side in one thread per chunk-lane.
__global__ void __launch_bounds__(512) plain_gate_up_wide_kernel(const PlainParams P) {
    extern __shared__ __align__(128) uint8_t psm[];
    const int t = blockIdx.y, tid = threadIdx.x;
    const int chunks = P.F / 16, j = blockIdx.x / chunks, r0 = (blockIdx.x - j * chunks) * 16, nsb = P.H / 256;
    uint64_t *bar = reinterpret_cast<uint64_t *>(psm);
    float *da = reinterpret_cast<float *>(psm + 128);
    int8_t *a = reinterpret_cast<int8_t *>(psm + 256);
    uint8_t *ws = psm + plain_gate_up_wide_chunks_off(P.H);
    const size_t half = static_cast<size_t>(16) * nsb * kPlainSb;
    float *part = reinterpret_cast<float *>(ws + 2 * half), *dsc = part + 32 * plain_part_stride(nsb);
    if (tid == 0) {
        mbar_init(bar, 1);
        mbar_fence_init();
    }
    WD_PSTAMP(0, 0)
    grid_dep_wait();
    grid_dep_launch();
    WD_PSTAMP(0, 2)
    if (tid == 0) {
        const size_t e = static_cast<size_t>(P.ids[t * P.K + j]), off = (e * P.F + r0) * nsb * kPlainSb;
        mbar_expect_tx(bar, static_cast<uint32_t>(2 * half));
        bulk_load(ws, P.gate + off, static_cast<uint32_t>(half), bar);
        bulk_load(ws + half, P.up + off, static_cast<uint32_t>(half), bar);
    }
    for (int i = tid; i < P.H / 16; i += blockDim.x)       // sixteen bytes at a time, superblock i / 16
        *reinterpret_cast<uint4 *>(a + (i >> 4) * kPlainActStride + (i & 15) * 16) =
            reinterpret_cast<const uint4 *>(P.xk + static_cast<size_t>(t) * P.H)[i];
    if (tid < nsb) da[tid] = P.xdk[static_cast<size_t>(t) * nsb + tid];
    __syncthreads();
    WD_PSTAMP(0, 3)
    mbar_wait(bar, 0, P.status);
    WD_PSTAMP(0, 4)
    for (int u = tid; u < 32 * nsb; u += blockDim.x) {
        const int rm = u / nsb, sb = u - rm * nsb;
        const uint8_t *blk = ws + static_cast<size_t>(u) * kPlainSb;
        int p[8];
        plain_wide_unit(rm < 16 ? P.gate_type : P.up_type, blk, a + sb * kPlainActStride, p);
        plain_store_part(part + rm * plain_part_stride(nsb) + sb * 8, p);
        dsc[u] = __fmul_rn(half_bits_to_float(*reinterpret_cast<const uint16_t *>(blk + 136)), da[sb]);
    }
    __syncthreads();
    if (tid < 128) {
        const int r = tid >> 3, c = tid & 7;
        const float *pg = part + r * plain_part_stride(nsb), *pu = pg + 16 * plain_part_stride(nsb);
        const float *dg = dsc + r * nsb, *du = dg + 16 * nsb;
        float g = 0.0f, u = 0.0f;
#pragma unroll 5
        for (int s = 0; s < nsb; ++s) {
            g = __fmaf_rn(dg[s], pg[s * 8 + c], g);
            u = __fmaf_rn(du[s], pu[s * 8 + c], u);
        }
        g = __fmul_rn(iq_row_post(P.gate_type), hsum8_lanes(g));
        u = __fmul_rn(iq_row_post(P.up_type), hsum8_lanes(u));
        if (c == 0) P.act[(static_cast<size_t>(t) * P.K + j) * P.F + r0 + r] = __fmul_rn(silu_ggml(g), u);
    }
    WD_PSTAMP(0, 5)
}

// Four consecutive IQ4_NL rows against a Q8_0 activation, lanes and orders as plain_rows4_iq4nl. A code's value comes from
// two 8-entry halves of the table (its low three bits as selector) and its top bit.
__device__ __forceinline__ float plain_rows4_iq4nl_wide(const uint8_t *rows, size_t row_bytes, int nb, const int8_t *aq, const float *ad, int lane) {
    const uint8_t *row = rows + (lane >> 3) * row_bytes;
    const int par = (lane >> 2) & 1, l = lane & 3;
    const uint32_t t0 = 0xbfad9881u, t1 = 0xf6eaddcfu, t2 = 0x26190d01u, t3 = 0x71594535u;     // -127 .. -65, -49 .. -10, 1 .. 38, 53 .. 113
    const uint16_t *dw = reinterpret_cast<const uint16_t *>(row + static_cast<size_t>(nb) * 16);
    float lo = 0.0f, hi = 0.0f;
#pragma unroll 5
    for (int b = par; b < nb; b += 2) {
        const uint32_t w = *reinterpret_cast<const uint32_t *>(row + b * 16 + l * 4);
        const uint32_t s = w & 0x77777777u, top = ((w >> 1) & 0x44444444u) | 0x32103210u;
        const uint32_t v0 = prmt(prmt(t0, t1, s), prmt(t2, t3, s), top);
        const uint32_t v1 = prmt(prmt(t0, t1, s >> 16), prmt(t2, t3, s >> 16), top >> 16);
        const int a0 = *reinterpret_cast<const int *>(aq + b * 32 + 4 * l), a1 = *reinterpret_cast<const int *>(aq + b * 32 + 16 + 4 * l);
        const float d = __fmul_rn(half_bits_to_float(dw[b]), ad[b]);
        lo = __fmaf_rn(d, static_cast<float>(dp4a_s8(a0, static_cast<int>(v0), 0)), lo);
        hi = __fmaf_rn(d, static_cast<float>(dp4a_s8(a1, static_cast<int>(v1), 0)), hi);
    }
    lo = __fadd_rn(lo, __shfl_xor_sync(0xffffffffu, lo, 4));        // even + odd blocks, chunk-lane l
    hi = __fadd_rn(hi, __shfl_xor_sync(0xffffffffu, hi, 4));        // chunk-lane l + 4
    float r = __fadd_rn(lo, hi);                                    // v[l] + v[l + 4]
    r = __fadd_rn(r, __shfl_xor_sync(0xffffffffu, r, 2));           // r0 + r2, r1 + r3
    return __fadd_rn(r, __shfl_xor_sync(0xffffffffu, r, 1));
}

// plain_quantize_q8_0_cta with four groups of a thread in flight: its chain of shuffles and divisions is 0.6 us, and the
// activations of ten slots (6400 values) take three rounds of it.
__device__ __forceinline__ void plain_quantize_q8_0_cta4(const float *xf, int n, int8_t *q_out, float *d_out) {
    const int nchunks = n >> 2;         // a multiple of eight: the lanes of a block are live together
    for (int base = threadIdx.x; base < ((nchunks + 31) & ~31); base += 4 * blockDim.x) {
        float4 v[4];
        float amax[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int ch = base + k * blockDim.x;
            v[k] = ch < nchunks ? *reinterpret_cast<const float4 *>(xf + 4 * ch) : make_float4(0, 0, 0, 0);
            amax[k] = fmaxf(fmaxf(fabsf(v[k].x), fabsf(v[k].y)), fmaxf(fabsf(v[k].z), fabsf(v[k].w)));
        }
#pragma unroll
        for (int s = 1; s < 8; s <<= 1)
#pragma unroll
            for (int k = 0; k < 4; ++k) amax[k] = fmaxf(amax[k], __shfl_xor_sync(0xffffffffu, amax[k], s));
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int ch = base + k * blockDim.x;
            if (ch >= nchunks) continue;
            uint32_t packed = 0;
            if (amax[k] != 0.0f) {
                const float inv = __fdiv_rn(127.0f, amax[k]);
                const float f[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    int q = __float2int_rn(__fmul_rn(f[j], inv));
                    q = max(-128, min(127, q));
                    packed |= static_cast<uint32_t>(q & 0xff) << (8 * j);
                }
            }
            *reinterpret_cast<uint32_t *>(q_out + 4 * ch) = packed;
            if ((ch & 7) == 0) d_out[ch >> 3] = __half2float(__float2half_rn(__fdiv_rn(amax[k], 127.0f)));
        }
    }
}

// Q8_K superblocks of the activations of an IQ down tensor sit kPlainActStride apart; IQ4_NL's Q8_0 quants are plain.
__host__ __device__ inline size_t plain_down_wide_act_bytes(int F, int K, bool nl) {
    return nl ? static_cast<size_t>(K) * F : static_cast<size_t>(K) * (F / 256) * kPlainActStride;
}
__host__ __device__ inline size_t plain_down_wide_chunks_off(int F, int K, bool nl) {
    return (256 + 16 * 64 + plain_down_wide_act_bytes(F, K, nl) + static_cast<size_t>(K) * (F / 32) * 4 + 127) / 128 * 128;
}
// after the chunks: the shared expert's tasks and activation, then one region that is the activations as floats first and
// the parts of the IQ rows later
__host__ __device__ inline size_t plain_down_wide_smem(int F, int SF, int K, bool nl) {
    size_t tail = static_cast<size_t>(K) * F > static_cast<size_t>(SF) ? static_cast<size_t>(K) * F : static_cast<size_t>(SF);
    if (!nl) {
        const size_t parts = static_cast<size_t>(K) * 16 * (plain_part_stride(F / 256) + F / 256);
        tail = parts > tail ? parts : tail;
    }
    return plain_down_wide_chunks_off(F, K, nl) + static_cast<size_t>(K) * 16 * plain_wide_row_bytes(F) + static_cast<size_t>(4) * (SF / 32) * 136 + SF +
           (SF / 32 + 3) / 4 * 16 + tail * 4;
}

// Down rows and combine: the structure of plain_down_kernel, the rows from wide tensors.
__global__ void __launch_bounds__(kThreads) plain_down_wide_kernel(const PlainParams P) {
    extern __shared__ __align__(128) uint8_t psm[];
    const int t = blockIdx.y, h0 = blockIdx.x * 16, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool nl = P.down_type == kTypeIq4nl;
    const int K = P.K, F = P.F, SF = P.SF, nbs = SF / 32, nsb = F / 256;
    uint64_t *bar = reinterpret_cast<uint64_t *>(psm);
    float *shd_s = reinterpret_cast<float *>(psm + 128);                    // [16] shared expert rows
    float *eo_s = reinterpret_cast<float *>(psm + 256);                     // [K][16] expert rows
    int8_t *actq = reinterpret_cast<int8_t *>(psm + 256 + kMaxK * 64);
    float *actd = reinterpret_cast<float *>(reinterpret_cast<uint8_t *>(actq) + plain_down_wide_act_bytes(F, K, nl));
    const size_t drb = plain_wide_row_bytes(F);
    uint8_t *chunks = psm + plain_down_wide_chunks_off(F, K, nl);
    uint8_t *shs = chunks + static_cast<size_t>(K) * 16 * drb;             // the shared expert's four tasks
    uint8_t *shq = shs + 4 * static_cast<size_t>(nbs) * 136;               // its activation, Q8_0 in task layout
    float *shd = reinterpret_cast<float *>(shq + SF);
    float *actf = reinterpret_cast<float *>(shq + SF + (nbs + 3) / 4 * 16); // F32 staging of the activations
    WD_PSTAMP(1, 0)
    // The ids come from the selection, two kernels back: the weight copies leave before the wait for the gate/up rows.
    if (warp == 0) {        // lane j fetches slot j's expert id and issues its copy; the loads of the ids overlap
        const uint32_t shb = SF > 0 ? 4u * static_cast<uint32_t>(nbs) * 136u : 0u;
        const size_t e = lane < K ? static_cast<size_t>(P.ids[t * K + lane]) : 0;
        if (lane == 0) {
            mbar_init(bar, 1);
            mbar_fence_init();
            mbar_expect_tx(bar, static_cast<uint32_t>(K * 16 * drb) + shb);
        }
        __syncwarp();
        if (lane < K) bulk_load(chunks + static_cast<size_t>(lane) * 16 * drb, P.down + (e * P.H + h0) * drb, static_cast<uint32_t>(16 * drb), bar);
        if (lane == K && shb) bulk_load(shs, P.sh_down + static_cast<size_t>(h0 / 4) * nbs * 136, shb, bar);
    }
    // the shared expert's activation, its gate and the weights are older than the kernel before this one
    float *w_s = reinterpret_cast<float *>(psm + 64), *gate_s = reinterpret_cast<float *>(psm + 16);
    if (warp == kWarps - 1 && lane < K) w_s[lane] = P.weights[t * K + lane];
    if (warp == kWarps - 2 && lane == 0 && SF > 0) *gate_s = P.sgate[t];
    for (int i = threadIdx.x; i < SF / 4; i += kThreads)
        reinterpret_cast<float4 *>(actf)[i] = reinterpret_cast<const float4 *>(P.shact + static_cast<size_t>(t) * SF)[i];
    __syncthreads();
    if (SF > 0) quantize_q8_0_cta(actf, SF, shq, shd);
    __syncthreads();
    WD_PSTAMP(1, 1)
    grid_dep_wait();
    grid_dep_launch();
    WD_PSTAMP(1, 2)
    // the activations of all slots arrive in one round of loads
    const float *act = P.act + static_cast<size_t>(t) * K * F;
#pragma unroll 4
    for (int i = threadIdx.x; i < K * F / 4; i += kThreads) reinterpret_cast<float4 *>(actf)[i] = reinterpret_cast<const float4 *>(act)[i];
    __syncthreads();
    WD_PSTAMP(1, 3)
    if (nl) {
        plain_quantize_q8_0_cta4(actf, K * F, actq, actd);
    } else {
        for (int s = warp; s < K * nsb; s += kWarps)
            quantize_q8_K_warp(actf + s * 256, lane, reinterpret_cast<uint8_t *>(actq) + s * kPlainActStride, actd + s);
    }
    __syncthreads();
    WD_PSTAMP(1, 4)
    mbar_wait(bar, 0, P.status);
    WD_PSTAMP(1, 5)
    const int n_exp = nl ? K * 4 : 0, n_tasks = n_exp + (SF > 0 ? 4 : 0);
    for (int task = warp; task < n_tasks; task += kWarps) {
        if (task >= n_exp) {
            const int i = task - n_exp;
            const float v = q8_task_row(shs + static_cast<size_t>(i) * nbs * 136, nbs, shq, shd, lane);
            if ((lane & 7) == 0) shd_s[i * 4 + (lane >> 3)] = v;
        } else {
            const int j = task >> 2, rg = task & 3;
            const float v = plain_rows4_iq4nl_wide(chunks + (static_cast<size_t>(j) * 16 + rg * 4) * drb, drb, F / 32, actq + j * F, actd + j * (F / 32), lane);
            if ((lane & 7) == 0) eo_s[j * 16 + rg * 4 + (lane >> 3)] = v;
        }
    }
    if (!nl) {              // one superblock of one row per thread, then one chunk-lane of one row
        float *part = actf, *dsc = part + static_cast<size_t>(K) * 16 * plain_part_stride(nsb);
        for (int u = threadIdx.x; u < K * 16 * nsb; u += kThreads) {
            const int r = u / nsb, sb = u - r * nsb, as = (r >> 4) * nsb + sb;
            const uint8_t *blk = chunks + static_cast<size_t>(u) * kPlainSb;
            int p[8];
            plain_wide_unit(P.down_type, blk, actq + as * kPlainActStride, p);
            plain_store_part(part + r * plain_part_stride(nsb) + sb * 8, p);
            dsc[u] = __fmul_rn(half_bits_to_float(*reinterpret_cast<const uint16_t *>(blk + 136)), actd[as]);
        }
        __syncthreads();
        for (int ch = threadIdx.x; ch < K * 128; ch += kThreads) {
            const int r = ch >> 3, c = ch & 7;
            const float v = hsum8_lanes(plain_chain(part + r * plain_part_stride(nsb), dsc + r * nsb, nsb, c));
            if (c == 0) eo_s[r] = __fmul_rn(iq_row_post(P.down_type), v);
        }
    }
    __syncthreads();
    WD_PSTAMP(1, 6)
    if (threadIdx.x < 16) {
        const size_t o = static_cast<size_t>(t) * P.H + h0 + threadIdx.x;
        float r = 0.0f;
        for (int j = 0; j < K; ++j) r = __fadd_rn(r, __fmul_rn(eo_s[j * 16 + threadIdx.x], w_s[j]));
        P.out[o] = SF > 0 ? __fadd_rn(r, __fmul_rn(shd_s[threadIdx.x], *gate_s)) : r;
        P.routed[o] = r;
        if (SF > 0) P.shdown[o] = shd_s[threadIdx.x];
    }
    for (int i = threadIdx.x; i < K * 16; i += kThreads)
        P.eo[(static_cast<size_t>(t) * K + (i >> 4)) * P.H + h0 + (i & 15)] = eo_s[i];
    WD_PSTAMP(1, 7)
}

}  // namespace wd
