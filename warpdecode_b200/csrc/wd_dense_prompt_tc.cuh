// The prompt pass's matrix products on the fifth-generation tensor cores: Y[m][row] = W[row] . X[m] for the tokens of a chunk, in
// the float order of the one-token step (wd_dense_decoder.cuh), for prompts that fill tiles of tokens.
//
// The float chain of a row's dot needs the exact integer sum of EVERY block of 32 by itself, so the tensor core's accumulator holds
// one block: one tcgen05.mma.kind::i8 of depth 32 makes the sums of 128 rows x TN tokens (TN = 32, 48 or 64), and eight warps read them
// back (tcgen05.ld), scale them and run the chains. Roles, in warpgroups of four warps:
//
//   warps 0 .. 7    quadrant w & 3 of the rows (a warp reads its own 32 lanes of tensor memory), half w >> 2 of the tokens. A thread holds one row
//                   and TN / 2 tokens; half of a block's sums travel from tensor memory while the other half is scaled
//   warps 8 .. 11   nibbles -> bytes -> tensor memory, where the MMA reads its A operand: once per 64 tokens, and no shared memory for it
//   warp 12         waits for both operands and a free accumulator, issues the MMAs
//   warp 13         asks for the stages: bulk copies of PER blocks of 128 rows and TN tokens, quants and scales
//
// Lane order: the step's lane l runs over the blocks l, l + 32, ..., and the lanes meet in the butterfly ^16 ^8 ^4 ^2 ^1. The lanes are
// walked in bit-reversed order, so that finished ones fold with a five-deep stack: two levels in registers, three in tensor memory. Both operands
// are laid out in that order ("entry" e = bitrev(l) * n_t + t for block 32 t + l): the activations by the kernels that write them (PromptAct), the
// weights by a pass over the layer's four matrices (prompt_lay_out_kernel) that costs what reading and writing them costs (10 us for 19 MB).
// PER = 2 blocks a stage while a lane's chain has an even number of them, else 1.
//
// Bound: issue, 2.4 of 4 instructions per cycle: per 32 x 32 sums of a warp 32 conversions, 40 two-wide float operations and about as many
// moves, waits and addresses. 480 tokens, the mma.sync kernel (wd_dense_prefill.cuh) -> this one, us without / with the laying out:
// 16384 x 2048 247 -> 139 / 150, 2048 x 8192 136 -> 74 / 80 (Q8_0 149 -> 74 / 84), 3072 x 2048 53 -> 41 / 44. On the way: sums read and scaled by
// 16 warps that also expand weights 317 us (247 instructions per 16 x 32 sums, most of them moves around a dynamic fold), folds unrolled and
// waits by stage 190, eight warps 176, reads in halves 166, roles apart 145, one wait per stage 139.
#pragma once

#include <type_traits>

#include "wd_dense_prefill.cuh"

namespace wd {

constexpr int kTcRows = 128;
// bytes of a block of a row tile: quants as planes of [128][16 B], then the scales as floats (a Q4_0 scale carries the 1/16 of
// its nibbles' place)
__host__ __device__ constexpr int tc_w_record(bool q8) { return kTcRows * (q8 ? 32 : 16) + kTcRows * 4; }

// The matrices of a layer -> row tiles in entry order. A CTA takes 128 rows by 8 neighbouring blocks.
struct LayOutMatrix {
    const uint8_t *src;         // the packed row layout
    uint8_t *dst;
    int rows, nb, q8, first_cta;
};
struct LayOutParams {
    LayOutMatrix m[4];
};
__host__ __device__ inline int lay_out_ctas(int rows, int nb) { return (rows + kTcRows - 1) / kTcRows * ((nb + 31) / 32) * 4; }
__global__ void __launch_bounds__(256) prompt_lay_out_kernel(const __grid_constant__ LayOutParams P) {
    __shared__ uint4 buf[2][8][kTcRows + 1];
    __shared__ float sc[8][kTcRows + 1];
    grid_dep_launch();
    int w = 3;
    while (w > 0 && static_cast<int>(blockIdx.x) < P.m[w].first_cta) --w;
    const LayOutMatrix M = P.m[w];
    const int at = static_cast<int>(blockIdx.x) - M.first_cta, n_t = (M.nb + 31) >> 5, x = at & 3, t = (at >> 2) % n_t, tile = (at >> 2) / n_t;
    const int b0 = 32 * t + 8 * x, stride = dense_row_stride(M.nb), planes = M.q8 ? 2 : 1, tid = threadIdx.x;
    const uint4 *q = reinterpret_cast<const uint4 *>(M.src);
    const uint16_t *d = reinterpret_cast<const uint16_t *>(M.src + static_cast<size_t>(M.rows) * stride * 16 * planes);
#pragma unroll 4
    for (int i = tid; i < kTcRows * 8 * planes; i += 256) {
        const int r = i / (8 * planes), p = i % (8 * planes), k = p / planes, row = tile * kTcRows + r, b = b0 + k;
        buf[p % planes][k][r] = row < M.rows && b < M.nb ? __ldg(q + (static_cast<size_t>(row) * stride + b) * planes + p % planes) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll 4
    for (int i = tid; i < kTcRows * 8; i += 256) {
        const int r = i / 8, k = i % 8, row = tile * kTcRows + r, b = b0 + k;
        sc[k][r] = row < M.rows && b < M.nb ? half_bits_to_float(__ldg(d + static_cast<size_t>(row) * stride + b)) * (M.q8 ? 1.0f : 0.0625f) : 0.0f;
    }
    grid_dep_wait();            // the products of the layer before have read the buffer
    __syncthreads();
    const int record = tc_w_record(M.q8 != 0);
#pragma unroll 1
    for (int k = 0; k < 8; ++k) {
        const int e = static_cast<int>(__brev(8 * x + k) >> 27) * n_t + t;
        uint8_t *o = M.dst + (static_cast<size_t>(tile) * 32 * n_t + e) * record;
        const int r = tid & (kTcRows - 1), half = tid / kTcRows;
        if (half < planes) reinterpret_cast<uint4 *>(o)[half * kTcRows + r] = buf[half][k][r];
        if (half == 1) reinterpret_cast<float *>(o + planes * kTcRows * 16)[r] = sc[k][r];
    }
}

// ---- tensor memory and the tensor core -----------------------------------------------------------------------------------
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// a warp's 32 lanes x N columns, N a multiple of 4; the values are there after tc_wait_ld
__device__ __forceinline__ void tc_ld4(uint32_t a, uint32_t *v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void tc_ld8(uint32_t a, uint32_t *v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(a)
                 : "memory");
}
__device__ __forceinline__ void tc_ld16(uint32_t a, uint32_t *v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
                   "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(a)
                 : "memory");
}
// The wait for a read into v, and nothing that uses v is moved in front of it (there is no form without v: the read's own output does not
// tie its uses to the wait).
template <int N>
__device__ __forceinline__ void tc_wait_ld(uint32_t (&v)[N]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < N; ++i) asm volatile("" : "+r"(v[i])::"memory");
}
template <int N>
__device__ __forceinline__ void tc_ld(uint32_t a, uint32_t (&v)[N]) {
    static_assert(N % 4 == 0 && N <= 32, "columns of one read");
#pragma unroll
    for (int i = 0; i + 16 <= N; i += 16) tc_ld16(a + i, v + i);
    if constexpr (N % 16 >= 8) tc_ld8(a + N / 16 * 16, v + N / 16 * 16);
    if constexpr (N % 8 == 4) tc_ld4(a + N - 4, v + N - 4);
}
__device__ __forceinline__ void tc_st4(uint32_t a, const uint32_t *v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
__device__ __forceinline__ void tc_st8(uint32_t a, const uint32_t *v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(a), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
                 "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
template <int N>
__device__ __forceinline__ void tc_st(uint32_t a, const uint32_t (&v)[N]) {
#pragma unroll
    for (int i = 0; i + 8 <= N; i += 8) tc_st8(a + i, v + i);
    if constexpr (N % 8 == 4) tc_st4(a + N - 4, v + N - 4);
}
// Descriptor of a K-major operand without swizzle: 16-byte rows of 8 x 16 B matrices, `k_step` bytes from one to the next in K and 128 in N.
__device__ __forceinline__ uint64_t tc_smem_desc(uint32_t addr, uint32_t k_step) {
    return static_cast<uint64_t>((addr >> 4) & 0x3fffu) | static_cast<uint64_t>((k_step >> 4) & 0x3fffu) << 16 | static_cast<uint64_t>(128u >> 4) << 32 |
           1ull << 46;
}
// D[128][N] (s32, tensor memory) = A[128][32] (s8, tensor memory) * B[N][32] (s8, shared memory); by one thread
__device__ __forceinline__ void tc_mma_s8(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n}" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(0u)
                 : "memory");
}
__device__ __forceinline__ void tc_commit(uint64_t *bar) {      // the barrier takes an arrival when the MMAs issued so far are done
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Bounded wait of this kernel's pipeline: by a count of polls, inline; a poll suspends the thread for 1.3 us, so that the limit is 1.4 s, or 0.3 ms
// when another wait of the pass has run out. (These waits stand between the stages of the warps that compute: a limit by the timer takes 2 to 3 %
// of the kernel, a flag in shared memory or a fence behind the loop 5 to 15.)
__device__ __forceinline__ bool tc_wait(uint64_t *bar, uint32_t parity, unsigned *status) {
#pragma unroll 1
    for (unsigned i = 0; i < kSpinLimit; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 255u) == 255u && *reinterpret_cast<volatile unsigned *>(status) != 0u) break;
    }
    atomicOr(status, kErrCopyTimeout);
    return false;
}
// What is under way ends before the CTA's memory is given back, whether a wait has run out or not.
__device__ __forceinline__ void tc_drain(uint64_t *bar, uint32_t parity) {
#pragma unroll 1
    for (unsigned i = 0; i < kSpinLimit && !mbar_try_wait(bar, parity); ++i) {
    }
}

// warps 0 .. 7 compute, 8 .. 11 expand weights, 12 issues the MMAs, 13 asks for the copies (14 and 15 complete its warpgroup)
constexpr int kTcWarps = 8, kTcThreads = 512;
// Registers a thread: two warpgroups that compute take what the two others give back, and no more than the launch's 128 a thread.
constexpr int kTcRegsMore = 192, kTcRegsLess = 64;
static_assert(2 * (kTcRegsMore + kTcRegsLess) <= 4 * 128, "more than the block was launched with: the increase would wait for ever");
template <bool Q8, int TN, int PER>
struct PromptTc {
    static constexpr int kSub = TN / (kTcWarps / 4), kPairs = kSub / 2;                 // tokens of a warp
    static constexpr int kW = tc_w_record(Q8), kX = TN * 36;
    static constexpr int kStage = PER * (kW + kX), kFit = 200 * 1024 / kStage, kStages = kFit < 16 ? kFit / 4 * 4 : 16;
    static constexpr int kSmem = kStages * kStage + 1024;
    // columns of tensor memory: two accumulators of two blocks, four stages of A (2 x 8 columns), three levels of the stack
    static constexpr int kColD = 0, kColA = 4 * TN, kColStack = kColA + 64;
    static_assert(kColStack + 3 * TN <= 512 && kStages >= 4, "plan of the tensor memory and the ring");
    static constexpr uint32_t kIdesc = 2u << 4 | 1u << 7 | 1u << 10 | (TN >> 3) << 17 | (kTcRows >> 4) << 24;
};

// status[0]: what the bounded waits raise (y is then undefined); host_status: page-locked, written when it is not zero. When a wait has run out the
// warps that ask for copies and issue MMAs stop at once, those that expand weights within 32 stages and those that compute at the end of the tile;
// copies and MMAs under way end before the CTA does. stop_at: the tile of a CTA at which its copies stop as if their wait had run out (tests).
template <bool Q8, int TN, int PER>
__global__ void __launch_bounds__(kTcThreads, 1) prompt_tc_gemm_kernel(const uint8_t *w, int rows, int nb, const uint8_t *x, int m_tokens, float *y,
                                                                      unsigned *status, unsigned *host_status, int stop_at) {
    using G = PromptTc<Q8, TN, PER>;
    extern __shared__ __align__(1024) uint8_t tsm[];
    __shared__ __align__(8) uint64_t full[G::kStages], empty[G::kStages], a_full[4], a_free[4], d_full[2], d_free[2];
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);     // the same in every lane, and known to be
    grid_dep_launch();
    if (warp == 0) {
        if (lane < G::kStages) {
            mbar_init(&full[lane], 1);
            mbar_init(&empty[lane], kTcWarps);
        }
        if (lane < 4) {
            mbar_init(&a_full[lane], 4);
            mbar_init(&a_free[lane], 1);
        }
        if (lane < 2) {
            mbar_init(&d_full[lane], 2);        // the MMAs' completion, and the thread that issued them
            mbar_init(&d_free[lane], kTcWarps);
        }
        mbar_fence_init();
    }
    if (warp == 12) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_base)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_dep_wait();            // activations and the weights in their order are the kernels' in front
    const uint32_t tm = tmem_base;
    const int n_t = (nb + 31) >> 5, entries = 32 * n_t, per_tile = entries / PER;
    const int row_tiles = (rows + kTcRows - 1) / kTcRows, tok_tiles = (m_tokens + TN - 1) / TN, n_tiles = row_tiles * tok_tiles;
    const int mine = static_cast<int>(blockIdx.x) < n_tiles ? (n_tiles - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x) : 0;
    const int total = mine * per_tile;          // stages of this CTA, over all of its tiles
    if (warp >= 12) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kTcRegsLess));
    if (warp >= 14) {
    } else if (warp == 13) {
        if (lane == 0) {
            int g = 0, slot = 0;
            uint32_t par = 1;
            bool ok = true;
            for (int k = 0; k < mine && ok; ++k) {
                if (k == stop_at) {
                    atomicOr(status, kErrCopyTimeout);
                    break;
                }
                const int tile = static_cast<int>(blockIdx.x) + k * static_cast<int>(gridDim.x);
                const uint8_t *ws = w + static_cast<size_t>(tile % row_tiles) * entries * G::kW, *xs = x + static_cast<size_t>(tile / row_tiles) * entries * G::kX;
                for (int s = 0; s < per_tile; ++s, ++g) {
                    if (!(ok = tc_wait(&empty[slot], par, status))) break;
                    uint8_t *dst = tsm + slot * G::kStage;
                    mbar_expect_tx(&full[slot], G::kStage);
                    bulk_load(dst, ws, PER * G::kW, &full[slot]);
                    bulk_load(dst + PER * G::kW, xs, PER * G::kX, &full[slot]);
                    ws += PER * G::kW;
                    xs += PER * G::kX;
                    if (++slot == G::kStages) {
                        slot = 0;
                        par ^= 1;
                    }
                }
            }
            for (int i = max(0, g - G::kStages); i < g; ++i) tc_drain(&full[i % G::kStages], static_cast<uint32_t>(i / G::kStages & 1));
        }
    } else if (warp == 12) {
        if (lane == 0) {
            int slot = 0;
            uint32_t par = 0;
            const uint64_t desc0 = tc_smem_desc(smem_u32(tsm + PER * G::kW), TN * 16);
            uint64_t desc = desc0;
            int g = 0;
            for (; g < total; ++g) {
                if (!(tc_wait(&full[slot], par, status) && tc_wait(&a_full[g & 3], static_cast<uint32_t>(g >> 2) & 1u, status) &&
                      tc_wait(&d_free[g & 1], (static_cast<uint32_t>(g >> 1) & 1u) ^ 1u, status)))
                    break;
                tc_fence_after();
#pragma unroll
                for (int b = 0; b < PER; ++b)
                    tc_mma_s8(tm + G::kColD + (g & 1) * (2 * TN) + b * TN, tm + G::kColA + (g & 3) * 16 + b * 8, desc + b * (G::kX >> 4), G::kIdesc);
                tc_commit(&d_full[g & 1]);
                mbar_arrive(&d_full[g & 1]);        // what this thread saw land, for those who read the stage's scales
                tc_commit(&a_free[g & 3]);
                desc += G::kStage >> 4;
                if (++slot == G::kStages) {
                    slot = 0;
                    par ^= 1;
                    desc = desc0;
                }
            }
            for (int i = max(0, g - 2); i < g; ++i) tc_drain(&d_full[i & 1], static_cast<uint32_t>(i >> 1) & 1u);
            for (int i = max(0, g - 4); i < g; ++i) tc_drain(&a_free[i & 3], static_cast<uint32_t>(i >> 2) & 1u);
        }
    } else if (warp >= kTcWarps) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kTcRegsLess));
        const int quad = warp & 3;
        const uint32_t lanes = tm + (static_cast<uint32_t>(quad * 32) << 16);
        int slot = 0;
        uint32_t par = 0;
#pragma unroll 1
        for (int g = 0; g < total; ++g) {
            if ((g & 31) == 31 && __any_sync(0xffffffffu, *reinterpret_cast<volatile unsigned *>(status) != 0u)) break;
            tc_wait(&full[slot], par, status);
            const uint8_t *src = tsm + slot * G::kStage + (quad * 32 + lane) * 16;
            uint32_t a[PER][8];
#pragma unroll
            for (int b = 0; b < PER; ++b) {
                const uint4 q = *reinterpret_cast<const uint4 *>(src + b * G::kW);
                if constexpr (Q8) {
                    const uint4 q1 = *reinterpret_cast<const uint4 *>(src + b * G::kW + kTcRows * 16);
                    a[b][0] = q.x; a[b][1] = q.y; a[b][2] = q.z; a[b][3] = q.w;
                    a[b][4] = q1.x; a[b][5] = q1.y; a[b][6] = q1.z; a[b][7] = q1.w;
                } else {        // a nibble at the top of its byte with the top bit flipped is 16 * (q - 8)
                    const uint32_t n[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        a[b][i] = ((n[i] << 4) & 0xf0f0f0f0u) ^ 0x80808080u;
                        a[b][4 + i] = (n[i] & 0xf0f0f0f0u) ^ 0x80808080u;
                    }
                }
            }
            tc_wait(&a_free[g & 3], (static_cast<uint32_t>(g >> 2) & 1u) ^ 1u, status);
            tc_fence_after();
#pragma unroll
            for (int b = 0; b < PER; ++b) tc_st8(lanes + G::kColA + ((g & 3) * 2 + b) * 8, a[b]);
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&a_full[g & 3]);
            if (++slot == G::kStages) {
                slot = 0;
                par ^= 1;
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kTcRegsMore));
        const int quad = warp & 3, sub = warp >> 2, r = quad * 32 + lane;
        const uint32_t lanes = tm + (static_cast<uint32_t>(quad * 32) << 16);
        int g = 0, slot = 0;
        // One stage: PER blocks of a lane's chain. A block's sums are read in two halves, one of them on its way from tensor memory while the
        // other is scaled and added to the chains in A. A read's registers hold nothing before its wait, and a compiler may copy registers
        // where paths meet: between a read and its wait there is no branch, and no read is under way when a stage ends.
        constexpr int kHalf = G::kSub / 2;
        uint32_t v[2][kHalf];
        // The first half of stage g; behind the last stage, what nobody uses. The stage's scales are read from what its copies wrote: the
        // barrier has an arrival of the thread that waited for them (the MMAs' completion answers for tensor memory only). A wait for the copies'
        // own barrier here costs 5 % of the time of tiles of 64 tokens.
        auto begin = [&]() {
            if (g < total) tc_wait(&d_full[g & 1], static_cast<uint32_t>(g >> 1) & 1u, status);
            tc_fence_after();
            tc_ld(lanes + G::kColD + (g & 1) * (2 * TN) + sub * G::kSub, v[0]);
        };
        begin();
        tc_wait_ld(v[0]);
        auto stage = [&](auto first, f32x2 (&A)[G::kPairs]) {
            const uint8_t *st = tsm + slot * G::kStage;
            const uint8_t *dwa = st + (G::kW - kTcRows * 4) + r * 4, *dxa = st + PER * G::kW + TN * 32 + sub * G::kSub * 4;
            const uint32_t col = lanes + G::kColD + (g & 1) * (2 * TN) + sub * G::kSub;
            uint64_t *done = &empty[slot];
#pragma unroll
            for (int c = 0; c < 2 * PER; ++c) {
                const int h = c >> 1, o = (c & 1) * (kHalf / 2);
                uint32_t (&u)[kHalf] = v[c & 1];
                if (c > 0) tc_wait_ld(u);
                if (c + 1 < 2 * PER) {
                    tc_ld(col + ((c + 1) >> 1) * TN + ((c + 1) & 1) * kHalf, v[(c + 1) & 1]);
                } else {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&d_free[g & 1]);
                    if (++slot == G::kStages) slot = 0;
                    ++g;
                    begin();
                }
                const float dw = *reinterpret_cast<const float *>(dwa + h * G::kW);
                const ulonglong2 *dx = reinterpret_cast<const ulonglong2 *>(dxa + h * G::kX + o * 8);
                const f32x2 dwp = pack2(dw, dw);
#pragma unroll
                for (int i = 0; i < kHalf / 4; ++i) {
                    const ulonglong2 s = dx[i];
                    const f32x2 f0 = pack2(__int2float_rn(static_cast<int>(u[4 * i])), __int2float_rn(static_cast<int>(u[4 * i + 1])));
                    const f32x2 f1 = pack2(__int2float_rn(static_cast<int>(u[4 * i + 2])), __int2float_rn(static_cast<int>(u[4 * i + 3])));
                    const f32x2 s0 = mul2(dwp, s.x), s1 = mul2(dwp, s.y);
                    if constexpr (decltype(first)::value) {         // fmaf(s, f, 0) but for the sign of a zero, which the end sets right
                        A[o + 2 * i] = h == 0 ? mul2(s0, f0) : fma2(s0, f0, A[o + 2 * i]);
                        A[o + 2 * i + 1] = h == 0 ? mul2(s1, f1) : fma2(s1, f1, A[o + 2 * i + 1]);
                    } else {
                        A[o + 2 * i] = fma2(s0, f0, A[o + 2 * i]);
                        A[o + 2 * i + 1] = fma2(s1, f1, A[o + 2 * i + 1]);
                    }
                }
            }
            tc_wait_ld(v[0]);
            __syncwarp();
            if (lane == 0) mbar_arrive(done);
        };
        auto chain = [&](f32x2 (&A)[G::kPairs]) {        // one lane of the step
            stage(std::true_type{}, A);
#pragma unroll 1
            for (int t = PER; t < n_t; t += PER) stage(std::false_type{}, A);
        };
        auto fold = [&](f32x2 (&A)[G::kPairs], const f32x2 (&B)[G::kPairs]) {
#pragma unroll
            for (int i = 0; i < G::kPairs; ++i) A[i] = add2(A[i], B[i]);
        };
#pragma unroll 1
        for (int k = 0; k < mine; ++k) {
            const int tile = static_cast<int>(blockIdx.x) + k * static_cast<int>(gridDim.x);
            const unsigned before = *reinterpret_cast<volatile unsigned *>(status);        // looked at behind the tile
#pragma unroll 1
            for (int j = 0; j < 8; ++j) {
                f32x2 A[G::kPairs], B[G::kPairs], C[G::kPairs];
                chain(A);
                chain(B);
                fold(A, B);
                chain(B);
                chain(C);
                fold(B, C);
                fold(A, B);
                uint32_t u[G::kSub];
                int level = 0;
#pragma unroll 1
                for (; j >> level & 1; ++level) {       // ^4, ^2, ^1
                    tc_wait_st();
                    tc_ld<G::kSub>(lanes + G::kColStack + level * TN + sub * G::kSub, u);
                    tc_wait_ld(u);
#pragma unroll
                    for (int i = 0; i < G::kPairs; ++i) A[i] = add2(pack2(__uint_as_float(u[2 * i]), __uint_as_float(u[2 * i + 1])), A[i]);
                }
                if (level < 3) {
#pragma unroll
                    for (int i = 0; i < G::kPairs; ++i) {
                        float lo, hi;
                        unpack2(A[i], lo, hi);
                        u[2 * i] = __float_as_uint(lo);
                        u[2 * i + 1] = __float_as_uint(hi);
                    }
                    tc_st<G::kSub>(lanes + G::kColStack + level * TN + sub * G::kSub, u);
                } else {
                    const int row = tile % row_tiles * kTcRows + r, tok = tile / row_tiles * TN + sub * G::kSub;
                    float *o = y + static_cast<size_t>(tok) * rows + row;
#pragma unroll
                    for (int i = 0; i < G::kPairs; ++i) {
                        float lo, hi;
                        unpack2(A[i], lo, hi);
                        if (row < rows && tok + 2 * i < m_tokens) o[static_cast<size_t>(2 * i) * rows] = __fadd_rn(lo, 0.0f);
                        if (row < rows && tok + 2 * i + 1 < m_tokens) o[static_cast<size_t>(2 * i + 1) * rows] = __fadd_rn(hi, 0.0f);
                    }
                }
            }
            if (__any_sync(0xffffffffu, before != 0u)) break;
        }
        tc_wait_st();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 12) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tm) : "memory");
    if (tid == 0) {
        const unsigned st = *reinterpret_cast<volatile unsigned *>(status);
        if (st != 0u) *host_status = st;
    }
}

}  // namespace wd
