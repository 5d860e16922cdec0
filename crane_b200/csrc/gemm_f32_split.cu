// C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]) of 32-bit numbers on the 5th-generation tensor cores, with the precision of
// 32-bit multiply-adds: the matrix product of the true 32-bit path.
//
// A number is the sum of two of 11 bits each, x = x1 + x2 (kind::tf32 takes 11 bits and cuts the rest off), up to 2^-23 of x,
// half a unit in the last place of a 32-bit number.  Products of such pieces are exact in 32 bits, and of the four
//     w x = w1 x1 + (w1 x2 + w2 x1) + w2 x2
// the last, below 2^-22 of w x and, since w1 is w rounded, of either sign, is left out.  The tensor cores add into their
// accumulator by cutting off, not by rounding (measured: a loss of 1.1e-8 of the sum per instruction, always towards zero: 2e-6
// over K = 2048).  So w1 x1 is added there over 32 products only; then threads take the sum out and add it, rounded, to a
// 32-bit sum in registers, while the products go on into a second accumulator.  The small products have an accumulator of their
// own, whose cuts are 2^-11 of that.
// Error against 64 bits, 2-norm, 97 rows, before (two chains of 32-bit multiply-adds a result) / now, in 1e-7: standard normal
// operands N 3072, K 2048: 2.6 / 1.5; 12288, 2048: 2.9 / 1.6; 2048, 6144: 3.6 / 1.7; 4096, 14336: 7.6 / 2.4; short K are the other
// way round (512, 64: 1.1 / 1.3), and so are operands that are all positive (2048, 2048: 0.6 / 1.3).  A whole prompt of 97
// tokens at hidden 2048, 32 layers: 7.8 / 5.
//
// A sum that is not finite (operands with infinities or NaN, or so large that w1 is one) is computed again by 32-bit
// multiply-adds, which treat these as they should be: the pieces of an infinity do not.
//
// The order in which an output element's products are added depends on N and K alone, whatever M is and wherever the
// element lies in its tile, so a row's result does not depend on what else is in the batch.
//
// Weights fill the 128-wide side of the MMA.  They come by TMA as they are, are cut by warps and put into tensor memory, from where
// the MMA reads them; rows of A come by TMA too and are cut in shared memory.  (Both operands
// through shared memory would need more of its bandwidth than there is.)  What bounds it: per 32 k about 1,300 clocks at 97 rows, 1,050
// at 16, of which the twelve products take 770 and 550 by themselves; the rest is the way from the end of a stage's products over
// the warps that wait for it to the next products with the same accumulator or place, two stages of which tensor memory holds
// beside 128 rows' sums.  One thread for all products, or operands cut by the threads that also fetch them through registers: 1,700
// to 1,900.  The slices of the inner dimension as clusters that add up through distributed shared memory: 5 to 8 us more per product,
// and a cluster size that suits many rows, of which one CTA fits an SM, does not suit few.  97 rows, us, before / now: 12288 x 2048
// 177 / 53, 3072 x 2048 49 / 18, 2048 x 2048 63 / 16, 2048 x 6144 170 / 29 (the weights from DRAM: 15, 4, 3, 8); 16 rows: 40 / 22,
// 29 / 12, 17 / 11, 43 / 22; one row: 22 / 21, 13 / 11, 12 / 9, 22 / 21.
//
// y = x W^T + b with W stored [out, in]:
// crane-core/src/models/hunyuan_dense/modeling.rs:273-330.
#include <cuda.h>

#include "common.cuh"
#include "gemm_f32_split.h"

namespace {

constexpr int FK = 32;                 // floats of the inner dimension per stage (a row of 128 bytes)
constexpr int FN = 128;                // weight rows per tile = MMA M
constexpr uint32_t RAW_BYTES = FN * FK * 4;
constexpr uint32_t PIECE_COLS = FK;                    // tensor-memory columns of a piece of a stage's weights
constexpr uint32_t WAIT_LIMIT = 1u << 22;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait.  Returns false (and raises the CTA's abort flag) when it gives up.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    for (uint32_t i = 0; i < WAIT_LIMIT; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
    }
    *abort_flag = 1;
    return false;
}
// The same by a whole warp, whose lanes go on or give up together.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1)
        : "memory");
}
// K-major operand with rows of 128 bytes, 128-byte swizzle: groups of 8 rows are 1024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}
// kind::tf32, A in tensor memory (an element a column)
__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t id, uint32_t acc) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n"
        "}\n" ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(id), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const float* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "f"(r[0]), "f"(r[1]), "f"(r[2]), "f"(r[3]), "f"(r[4]), "f"(r[5]), "f"(r[6]), "f"(r[7]), "f"(r[8]),
          "f"(r[9]), "f"(r[10]), "f"(r[11]), "f"(r[12]), "f"(r[13]), "f"(r[14]), "f"(r[15])
        : "memory");
}
__device__ __forceinline__ void cut(float x, float& hi, float& lo) {
    hi = __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u);
    lo = x - hi;
}
__device__ __forceinline__ float4 lds4(uint32_t at) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ void sts4(uint32_t at, float4 v) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(at), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
// two sums at once
__device__ __forceinline__ void add2(unsigned long long& c, uint32_t lo, uint32_t hi) {
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(c) : "l"((unsigned long long)lo | (unsigned long long)hi << 32));
}

struct SplitParams {
    const float* a;
    const float* w;
    const float* bias;           // over N, or null
    float* c;
    int m, n, k;
    long long lda, ldw, ldc;
    int slices;                  // of the inner dimension: they are added in order
    long long part_stride;       // > 0: elements between their sums in c, a tensor each; 0: c is the result
    int* err;                    // or null
};

// What a slice of the inner dimension adds to one result, by multiply-adds.
__device__ __noinline__ float slice_dot(const float* a, const float* w, int k0, int k1) {
    float sum = 0.f;
    for (int k = k0; k < k1; ++k) sum = fmaf(a[k], w[k], sum);
    return sum;
}

// NT: rows of A per tile (the narrow side of the MMA), a multiple of 16.  RAW: stages of weights on their way from memory;
// AST: stages of pieces (weights in tensor memory, rows of A in shared memory).
template <int NT> struct Shape {
    static constexpr int CTAS = NT <= 16 ? 2 : 1;              // per SM
    // Warps, by fours: one copies, one issues the products w1 x1, one the small products; then those that take the
    // accumulators out (one or two per 32 lanes of tensor memory), that cut weights (one or two groups, which take the stages in
    // turn) and that cut rows of A.
    static constexpr int SUM_WARPS = NT <= 32 ? 4 : NT <= 80 ? 8 : 16, W_GROUPS = NT <= 16 ? 1 : 2;
    static constexpr int FIRST_W = 4 + SUM_WARPS, LAST = FIRST_W + 4 * W_GROUPS, THREADS = 32 * (LAST + 4);
    static constexpr int AST = NT <= 80 ? 3 : 2;
    static constexpr int BST = NT <= 96 ? 4 : 3;
    static constexpr int RAW = NT <= 16 ? 4 : NT <= 64 ? 8 : 6;
    // Few rows: w1 [x1 | x2] is one instruction of twice the rows, into two accumulators side by side (8 instructions of 46 clocks
    // a stage instead of 12; one row, us: 12288 x 2048 22.7 -> 20.6, 2048 x 6144 21.9 -> 20.6, a head of 120818 x 2048 207 -> 190).
    static constexpr bool STACK = NT <= 32;
    static constexpr uint32_t B_PIECE = NT * FK * 4, B_BYTES = (STACK ? 3 : 2) * B_PIECE;
    static constexpr uint32_t COLS_USED = 3 * NT + AST * 2 * PIECE_COLS;
    static constexpr uint32_t TMEM_COLS = COLS_USED <= 256 ? 256 : 512;
    static constexpr size_t BARS = 2 * RAW + 3 * BST + AST;
    static constexpr size_t SMEM = RAW * RAW_BYTES + BST * B_BYTES + BARS * 8 + 16 + 1024;
    static_assert(BST >= AST, "the products' barriers, one per stage of A, are asked AST stages later too");
    static_assert(NT % 16 == 0 && NT >= 16 && NT <= 128 && COLS_USED <= 512 && TMEM_COLS * CTAS <= 512, "columns of tensor memory");
    static_assert(CTAS * (SMEM + 1024) <= 233472, "shared memory");
};

template <int NT>
__global__ void __launch_bounds__(Shape<NT>::THREADS, Shape<NT>::CTAS)
gemm_f32_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a,
                      const SplitParams p) {
    using S = Shape<NT>;
    constexpr int AST = S::AST, BST = S::BST, RAW = S::RAW;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sm_w = smem;                                        // [RAW][128 rows][128 bytes], 128-byte swizzle
    uint8_t* sm_b = smem + RAW * RAW_BYTES;                      // [BST][x1, x2 (, x1)][NT rows][128 bytes], 128-byte swizzle
    uint64_t* raw_full = (uint64_t*)(sm_b + BST * S::B_BYTES);   // [RAW] weights have landed
    uint64_t* raw_empty = raw_full + RAW;        // [RAW] they have been read
    uint64_t* a_full = raw_empty + RAW;          // [BST] a stage's rows of A have landed
    uint64_t* b_full = a_full + BST;             // [BST] they are there in pieces
    uint64_t* done = b_full + BST;               // [BST] the stage's products are done
    uint64_t* ready = done + BST;                // [AST] its weights and its rows of A are there in pieces, and the accumulator for
                                                 // its w1 x1 has been taken out
    uint32_t* tmem_slot = (uint32_t*)(ready + AST);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = blockIdx.y * FN, m0 = blockIdx.z * NT, rows = min(NT, p.m - m0);
    const int blocks = (p.k + FK - 1) / FK;
    auto begin = [&](int slice) { return (int)((long long)blocks * slice / p.slices); };
    // this CTA's slices: one, whose sums are a tensor of their own, or all, added up in C
    const int slice0 = p.part_stride > 0 ? blockIdx.x : 0, slice1 = p.part_stride > 0 ? slice0 + 1 : p.slices;
    const int first = begin(slice0), mine = begin(slice1) - first;

    if (threadIdx.x == 0) {
        for (int s = 0; s < RAW; ++s) {
            mbar_init(smem_u32(&raw_full[s]), 1);
            mbar_init(smem_u32(&raw_empty[s]), 4);
        }
        for (int s = 0; s < BST; ++s) {
            mbar_init(smem_u32(&a_full[s]), 1);
            mbar_init(smem_u32(&b_full[s]), 4);
            mbar_init(smem_u32(&done[s]), S::STACK ? 1 : 2);
        }
        for (int s = 0; s < AST; ++s) mbar_init(smem_u32(&ready[s]), 4 + S::SUM_WARPS);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        // the first weights, which are no kernel's result, before tensor memory is asked for: a kernel that still has it all keeps
        // this one waiting there
        for (int i = 0; i < min(mine, RAW); ++i) {
            mbar_expect_tx(smem_u32(&raw_full[i]), RAW_BYTES);
            tma_load_2d(smem_u32(sm_w + i * RAW_BYTES), &map_w, smem_u32(&raw_full[i]), (first + i) * FK, n0);
        }
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(S::TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    // the two sums of w1 x1 and that of the small products; STACK: the latter between the former, so that it lies beside both
    const uint32_t tm_small = tmem + (S::STACK ? 1 : 2) * NT, tm_pieces = tmem + 3 * NT;
    auto tm_main = [&](int i) { return tmem + (uint32_t)((i & 1) * (S::STACK ? 2 : 1) * NT); };
    pdl_launch_dependents();

    if (warp == 0) {
        // ---------------- copies of the weights ----------------
        if (lane == 0) {
            for (int i = RAW; i < mine; ++i) {
                const int s = i % RAW;
                if (!mbar_wait(smem_u32(&raw_empty[s]), ((i / RAW) & 1) ^ 1, abort_flag)) break;
                mbar_expect_tx(smem_u32(&raw_full[s]), RAW_BYTES);
                tma_load_2d(smem_u32(sm_w + s * RAW_BYTES), &map_w, smem_u32(&raw_full[s]), (first + i) * FK, n0);
            }
        }
    } else if (warp == 3) {
        // ---------------- copies of the rows of A, which come from the kernel before ----------------
        pdl_wait();
        if (lane == 0) {
            for (int i = 0; i < mine; ++i) {
                const int s = i % BST;
                if (i >= BST && !mbar_wait(smem_u32(&done[s]), ((i / BST) & 1) ^ 1, abort_flag)) break;
                mbar_expect_tx(smem_u32(&a_full[s]), S::B_PIECE);
                tma_load_2d(smem_u32(sm_b + s * S::B_BYTES), &map_a, smem_u32(&a_full[s]), (first + i) * FK, m0);
            }
        }
    } else if (warp < 3) {
        // ---------------- products: an accumulator is written by one thread alone ----------------
        if (S::STACK && warp == 1 && lane == 0) {
            // Stages take turns with [x1 | x2] -> [sum 0 | small] and [x2 | x1] -> [small | sum 1].  The same additions in the same
            // order as below: the accumulators begin as zeros, which those who take them out write.
            const uint32_t two = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(2 * NT >> 3) << 17) | ((uint32_t)(FN >> 4) << 24);
            const uint32_t one = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(FN >> 4) << 24);
            for (int i = 0; i < mine; ++i) {
                const int s = i % AST, bs = i % BST;
                if (!mbar_wait(smem_u32(&ready[s]), (i / AST) & 1, abort_flag)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a1 = tm_pieces + (uint32_t)(s * 2 * PIECE_COLS), a2 = a1 + PIECE_COLS, to = tmem + (uint32_t)((i & 1) * NT);
                const uint64_t b1 = smem_desc_sw128(smem_u32(sm_b + bs * S::B_BYTES)), b12 = b1 + (i & 1) * (S::B_PIECE >> 4);
#pragma unroll
                for (int kk = 0; kk < FK / 8; ++kk) {
                    umma_ts(to, a1 + 8 * kk, b12 + 2 * kk, two, 1u);
                    umma_ts(tm_small, a2 + 8 * kk, b1 + 2 * kk, one, 1u);
                }
                umma_commit(smem_u32(&done[bs]));
            }
        }
        if (!S::STACK && lane == 0) {
            const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(NT >> 3) << 17) |
                                   ((uint32_t)(FN >> 4) << 24);
            int slice = slice0, next = 0;                        // the stage that a slice begins with
            for (int i = 0; i < mine; ++i) {
                const int s = i % AST, bs = i % BST;
                const bool fresh = i == next;
                if (fresh) next = begin(++slice) - first;
                if (!mbar_wait(smem_u32(&ready[s]), (i / AST) & 1, abort_flag)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a1 = tm_pieces + (uint32_t)(s * 2 * PIECE_COLS), a2 = a1 + PIECE_COLS;
                const uint64_t b1 = smem_desc_sw128(smem_u32(sm_b + bs * S::B_BYTES)), b2 = b1 + (S::B_PIECE >> 4);
                if (warp == 1) {
#pragma unroll
                    for (int kk = 0; kk < FK / 8; ++kk)          // 8 elements: 8 columns, 32 bytes
                        umma_ts(tm_main(i), a1 + 8 * kk, b1 + 2 * kk, idesc, kk > 0 ? 1u : 0u);
                } else {
#pragma unroll
                    for (int kk = 0; kk < FK / 8; ++kk) {
                        umma_ts(tm_small, a1 + 8 * kk, b2 + 2 * kk, idesc, (!fresh || kk > 0) ? 1u : 0u);
                        umma_ts(tm_small, a2 + 8 * kk, b1 + 2 * kk, idesc, 1u);
                    }
                }
                umma_commit(smem_u32(&done[bs]));
            }
        }
    } else if (warp >= S::LAST) {
        // ---------------- rows of A in pieces: the first in their place, the second beside them ----------------
        const int t = threadIdx.x - 32 * S::LAST, b_row = t >> 3, b_chunk = t & 7;      // 4 floats of every 16th row
        const uint32_t at = b_row * 128 + ((b_chunk ^ (b_row & 7)) << 4);
        for (int i = 0; i < mine; ++i) {
            const int s = i % BST;
            if (!mbar_wait_warp(smem_u32(&a_full[s]), (i / BST) & 1, abort_flag)) break;
            const uint32_t base = smem_u32(sm_b + s * S::B_BYTES) + at;
            float4 v[NT / 16];
#pragma unroll
            for (int j = 0; j < NT / 16; ++j) v[j] = lds4(base + j * 2048);
#pragma unroll
            for (int j = 0; j < NT / 16; ++j) {
                float4 hi, lo;
                cut(v[j].x, hi.x, lo.x);
                cut(v[j].y, hi.y, lo.y);
                cut(v[j].z, hi.z, lo.z);
                cut(v[j].w, hi.w, lo.w);
                sts4(base + j * 2048, hi);
                sts4(base + S::B_PIECE + j * 2048, lo);
                if (S::STACK) sts4(base + 2 * S::B_PIECE + j * 2048, hi);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&b_full[s]));
        }
    } else if (warp >= S::FIRST_W && warp < S::LAST) {
        // ---------------- weights in pieces ----------------
        const int group = (warp - S::FIRST_W) >> 2, quarter = warp & 3, row = (quarter << 5) | lane, swz = row & 7;
        for (int i = group; i < mine; i += S::W_GROUPS) {
            const int s = i % AST, ws = i % RAW, bs = i % BST, before = i - AST;
            if (!mbar_wait_warp(smem_u32(&raw_full[ws]), (i / RAW) & 1, abort_flag)) break;
            if (before >= 0 && !mbar_wait_warp(smem_u32(&done[before % BST]), (before / BST) & 1, abort_flag)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t from = smem_u32(sm_w + ws * RAW_BYTES) + row * 128;
            const uint32_t ta = tm_pieces + (uint32_t)(s * 2 * PIECE_COLS) + ((uint32_t)(quarter * 32) << 16);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                float w1[16], w2[16];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float4 v = lds4(from + (((half * 4 + c) ^ swz) << 4));
                    cut(v.x, w1[4 * c], w2[4 * c]);
                    cut(v.y, w1[4 * c + 1], w2[4 * c + 1]);
                    cut(v.z, w1[4 * c + 2], w2[4 * c + 2]);
                    cut(v.w, w1[4 * c + 3], w2[4 * c + 3]);
                }
                tmem_st16(ta + half * 16, w1);
                tmem_st16(ta + PIECE_COLS + half * 16, w2);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&raw_empty[ws]));
            // (the rows of A last: the first stages' weights are cut before the kernel before has written them)
            if (!mbar_wait_warp(smem_u32(&b_full[bs]), (i / BST) & 1, abort_flag)) break;
            if (lane == 0) mbar_arrive(smem_u32(&ready[s]));
        }
    } else if (warp < S::FIRST_W) {
        // ---------------- sums ----------------
        constexpr int COLS = NT * 4 / S::SUM_WARPS;
        const int half = (warp - 4) >> 2, quarter = warp & 3;
        const uint32_t from_lanes = ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * COLS);
        unsigned long long acc[COLS / 2];
#pragma unroll
        for (int j = 0; j < COLS / 2; ++j) acc[j] = 0ull;
        auto take = [&](uint32_t from) {                         // acc += these columns, as many at a time as registers hold
            constexpr int BATCH = COLS <= 32 ? COLS : 8;
#pragma unroll
            for (int c0 = 0; c0 < COLS; c0 += BATCH) {
                uint32_t r[BATCH];
#pragma unroll
                for (int c = 0; c < BATCH; c += 8) tmem_ld8(from + from_lanes + (uint32_t)(c0 + c), r + c);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int j = 0; j < BATCH; j += 2) add2(acc[(c0 + j) / 2], r[j], r[j + 1]);
            }
        };
        auto clear = [&](uint32_t at) {                          // these columns = 0
            const float zeros[16] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < COLS; c += 16) tmem_st16(at + from_lanes + (uint32_t)c, zeros);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        };
        if (S::STACK) {
            clear(tm_main(0));
            clear(tm_main(1));
            clear(tm_small);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
        }
        if (lane == 0) {                                         // both accumulators are free
            mbar_arrive(smem_u32(&ready[0]));
            mbar_arrive(smem_u32(&ready[1]));
        }
        pdl_wait();
        const int col = n0 + quarter * 32 + lane;                // this thread's row of the weights
        const bool there = col < p.n;
        int slice = slice0, begun = 0, last = begin(slice0 + 1) - first - 1;
        for (int i = 0; i < mine; ++i) {
            const bool ok = mbar_wait_warp(smem_u32(&done[i % BST]), (i / BST) & 1, abort_flag);
            if (ok) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                take(tm_main(i));
                if (S::STACK) clear(tm_main(i));
                if (i == last) {
                    take(tm_small);
                    if (S::STACK) clear(tm_small);
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                // (the first products of a slice go into both accumulators: they wait for the end of the slice before)
                if (lane == 0 && i == last) mbar_arrive(smem_u32(&ready[(i + 1) % AST]));
                if (lane == 0 && i + 1 != last) mbar_arrive(smem_u32(&ready[(i + 2) % AST]));
            }
            if (i != last && ok) continue;
            const int k0 = (first + begun) * FK, k1 = min(p.k, (first + i + 1) * FK);
            float* c = p.c + (p.part_stride > 0 ? (long long)slice * p.part_stride : 0) + (long long)m0 * p.ldc + col;
            const bool add = slice > 0 && p.part_stride == 0;
            const float bias = slice == 0 && p.bias != nullptr && there ? p.bias[col] : 0.f;
#pragma unroll
            for (int j = 0; j < COLS; ++j) {
                const int r = half * COLS + j;
                if (r >= rows || !there) continue;
                float v = __uint_as_float((uint32_t)(acc[j / 2] >> (j & 1) * 32));
                if (!ok) v = __uint_as_float(0x7fffffffu);       // (gave up: the result must not pass for one)
                else if (!isfinite(v)) v = slice_dot(p.a + (long long)(m0 + r) * p.lda, p.w + (long long)col * p.ldw, k0, k1);
                v += bias;
                float* at = c + (long long)r * p.ldc;
                *at = add ? *at + v : v;
            }
            if (!ok) break;
#pragma unroll
            for (int j = 0; j < COLS / 2; ++j) acc[j] = 0ull;
            begun = i + 1;
            last = begin(++slice + 1) - first - 1;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*abort_flag) {
        if (threadIdx.x == 0 && p.err != nullptr) atomicOr(p.err, CRANE_ERR_WAIT_TIMEOUT);
        // copies that were issued may still be landing: give them time before the CTA ends
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
        __syncthreads();
    }
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::TMEM_COLS) : "memory");
    }
}

// ------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// [rows, k] float, `ld` elements between rows; box of 32 x box_rows.  The last descriptors are kept per thread and found again
// by their arguments, which are all that they depend on.
struct MapSlot {
    const void* ptr;
    long long ld;
    int rows, k, box_rows;
    bool used;
    CUtensorMap map;
};
constexpr int MAP_SLOTS = 512;                       // a power of two

bool make_map(CUtensorMap* map, const float* ptr, int rows, int k, long long ld, int box_rows) {
    static thread_local MapSlot* slots = nullptr;
    if (!slots) slots = new MapSlot[MAP_SLOTS]();
    uint64_t h = ((uint64_t)(uintptr_t)ptr >> 4) ^ ((uint64_t)(uint32_t)rows << 20) ^ ((uint64_t)(uint32_t)k << 8) ^
                 ((uint64_t)(uint32_t)box_rows << 44);
    h *= 0x9E3779B97F4A7C15ull;
    MapSlot& sl = slots[(h >> 40) & (MAP_SLOTS - 1)];
    if (sl.used && sl.ptr == ptr && sl.rows == rows && sl.k == k && sl.ld == ld && sl.box_rows == box_rows) {
        *map = sl.map;
        return true;
    }
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return false;
        fn = (EncodeTiledFn)sym;
    }
    cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
    cuuint32_t box[2] = {FK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    if (fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(ptr), dims, strides, box, estr,
           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    sl.ptr = ptr; sl.ld = ld; sl.rows = rows; sl.k = k; sl.box_rows = box_rows; sl.map = *map; sl.used = true;
    return true;
}

template <int NT>
int launch_split(const SplitParams& p, cudaStream_t st) {
    CUtensorMap map_w, map_a;
    if (!make_map(&map_w, p.w, p.n, p.k, p.ldw, FN) || !make_map(&map_a, p.a, p.m, p.k, p.lda, NT)) return (int)cudaErrorInvalidValue;
    auto kern = gemm_f32_split_kernel<NT>;
    static bool configured = false;
    if (!configured) {
        const cudaError_t rc = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Shape<NT>::SMEM);
        if (rc != cudaSuccess) { cudaGetLastError(); return (int)rc; }
        configured = true;
    }
    return crane_launch(kern, dim3(p.part_stride > 0 ? p.slices : 1, (p.n + FN - 1) / FN, (p.m + NT - 1) / NT),
                        dim3(Shape<NT>::THREADS), Shape<NT>::SMEM, st, map_w, map_a, p);
}
}  // namespace

bool crane_f32_split_takes(const float* A, const float* W, int M, int N, int K, long long lda, long long ldw) {
    // (the grid's second and third extent count tiles of weight rows and of rows)
    return K > 0 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && lda >= K && ldw >= K && ((uintptr_t)A | (uintptr_t)W) % 16 == 0 &&
           (M + 127) / 128 <= 65535 && (N + FN - 1) / FN <= 65535;
}

// Slices of the inner dimension: the number for which the rounds over the SMs take the least time, a CTA an SM, where a CTA
// costs about 6 blocks beside its own (fewer slices where more gain little); at most 8, which the readers of partial sums fetch
// at a time, of at least 4 blocks.  Of N and K alone, so that neither M nor the device at hand changes a sum: 148 SMs are
// those of the device the times were taken on.
CRANE_API int crane_f32_slices(int N, int K) {
    const int tiles = (N + FN - 1) / FN, blocks = (K + FK - 1) / FK;
    int best = 1;
    double best_time = 1e30;
    for (int s = 1; s <= 8 && (s == 1 || blocks / s >= 4); ++s) {
        const double time = (double)((tiles * s + 147) / 148) * ((double)blocks / s + 6.0);
        if (time < best_time * 0.97) { best = s; best_time = time; }
    }
    return best;
}

int crane_f32_split(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, long long lda,
                    long long ldw, long long ldc, long long part_stride, int* err, cudaStream_t st) {
    const SplitParams p{A, W, bias, C, M, N, K, lda, ldw, ldc, crane_f32_slices(N, K), part_stride, err};
    // tiles of at most 128 rows, all about as high
    const int tiles = (M + 127) / 128, nt = ((M + tiles - 1) / tiles + 15) / 16;
    switch (nt) {
        case 1: return launch_split<16>(p, st);
        case 2: return launch_split<32>(p, st);
        case 3: return launch_split<48>(p, st);
        case 4: return launch_split<64>(p, st);
        case 5: return launch_split<80>(p, st);
        case 6: return launch_split<96>(p, st);
        default: return launch_split<128>(p, st);
    }
}
