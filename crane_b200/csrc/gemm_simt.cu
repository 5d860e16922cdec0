// C[M,N] = A[M,K] * W[N,K]^T (+ bias[N]) on the FP32 cores: the matrix product
// of the true 32-bit path (no tensor cores, hence no reduced-precision matrix
// mode), and a fallback of the bf16 path for sizes the tensor-core kernel
// refuses.  The order in which an output element's products are added depends on
// N and K alone, whatever M is and wherever the element lies in its tile, so a
// row's result does not depend on what else is in the batch.
//
// Two kernels.  `gemm_f32_kernel` takes float operands whose rows are whole 16-byte pieces (what the
// 32-bit path has): see there.  `gemm_nt_kernel` takes everything else: bf16 operands, odd widths.
//
// y = x W^T + b with W stored [out, in]:
// crane-core/src/models/hunyuan_dense/modeling.rs:273-330.
#include "common.cuh"

namespace {
constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

template <typename TA, typename TO>
__global__ void __launch_bounds__(256)
gemm_nt_kernel(const TA* __restrict__ A, const TA* __restrict__ W, const float* __restrict__ bias,
               TO* __restrict__ C, int M, int N, int K, long long lda, long long ldw,
               long long ldc) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int tx = tid % 16, ty = tid / 16;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    // each thread loads 4 elements of A and 4 of W per k-slab: row = tid / 4, 4 k's
    const int lr = tid / 4, lk = (tid % 4) * 4;
    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = k0 + lk + i;
            const int m = m0 + lr, n = n0 + lr;
            As[lk + i][lr] = (m < M && k < K) ? to_f32(A[(long long)m * lda + k]) : 0.f;
            Ws[lk + i][lr] = (n < N && k < K) ? to_f32(W[(long long)n * ldw + k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = As[k][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = Ws[k][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty * TM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx * TN + j;
            if (n >= N) continue;
            float v = acc[i][j];
            if (bias) v += bias[n];
            C[(long long)m * ldc + n] = from_f32<TO>(v);
        }
    }
}

// ---- float operands, rows of whole 16-byte pieces --------------------------------------------------
// What bounds it: with few rows the weights' way from DRAM; with many the latency of the operands' way from shared memory
// into registers (16 bytes a lane take four clocks of an SM, whether or not the lanes read the same ones) and of a barrier
// every 32 k, which two warps a scheduler do not cover: 97 x 12288 x 2048 takes 187 us with the multiply-add pipe 48 %, issue
// slots 42 % and shared memory 40 % of the SMs' active cycles.  Whole prompts at hidden 2048, inner 6144, 32 layers, 32-bit: 97 tokens 39.3 -> 22.2 ms
// (17.0 with the slices below and wider loads in the attention), 24 tokens 34.5 -> 6.1 ms; `gemm_nt_kernel`, which
// reads every operand 4 bytes at a time and has no slices, took nearly all of it before.
//
// A CTA computes BM x BN results over a slice of the inner dimension, which a cluster of up to 8 CTAs
// shares (the products of a step of 97 tokens have 16 to 96 tiles for 148 SMs); the slices' sums are
// added in order through distributed shared memory.  How many slices there are depends on N and K.
// Operands lie in shared memory as they come (rows along k, copied asynchronously, three stages; a row's
// pitch of 36 floats puts the rows that a quarter of a warp reads side by side on different banks).  The
// sums of even and of odd k are kept apart: then both operands of the paired multiply-add (two
// products an instruction) are neighbours in memory and nothing has to be rearranged or copied.
// Many rows: each of 8 warps takes TM rows and all 128 columns, 4 a lane; few rows (at most 16): each of
// 4 warps takes all of them and 32 columns, so that a weight is read once.
constexpr int FK = 32, FPITCH = FK + 4, FN = 128, FSTAGES = 3;

typedef unsigned long long f32x2;
__device__ __forceinline__ void fma2(f32x2& c, f32x2 a, f32x2 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ void copy16(float* dst, const float* src, bool there) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(there ? 16 : 0) : "memory");
}

template <int WM, int WN, int TM, int TN>
__global__ void __launch_bounds__(WM * WN * 32)
gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ C,
                int M, int N, int K, long long lda, long long ldw, long long ldc) {
    constexpr int THREADS = WM * WN * 32, BM = WM * TM;
    static_assert(WN * 32 * TN == FN, "128 columns a tile");
    extern __shared__ __align__(16) float tiles[];               // [FSTAGES][BM + FN][FPITCH]; later [BM][FN] sums
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int slice = blockIdx.x, slices = gridDim.x, n0 = blockIdx.y * FN, m0 = blockIdx.z * BM;
    const int blocks = (K + FK - 1) / FK;
    const int first = (int)((long long)blocks * slice / slices), mine = (int)((long long)blocks * (slice + 1) / slices) - first;

    auto load = [&](int i, bool weights) {                       // block i of this slice
        float* to = tiles + (i % FSTAGES) * (BM + FN) * FPITCH + (weights ? BM * FPITCH : 0);
        const int k0 = (first + i) * FK;
        for (int c = tid; c < (weights ? FN : BM) * (FK / 4); c += THREADS) {
            const int r = c / (FK / 4), k = k0 + c % (FK / 4) * 4, at = (weights ? n0 : m0) + r;
            const bool there = at < (weights ? N : M) && k < K;
            const float* src = weights ? W : A;
            copy16(to + r * FPITCH + c % (FK / 4) * 4, there ? src + (long long)at * (weights ? ldw : lda) + k : src, there);
        }
    };
    auto commit = []() { asm volatile("cp.async.commit_group;" ::: "memory"); };
    pdl_launch_dependents();
#pragma unroll
    for (int i = 0; i < FSTAGES - 1; ++i)
        if (i < mine) load(i, true);
    pdl_wait();                                                  // (the weights are no kernel's result)
#pragma unroll
    for (int i = 0; i < FSTAGES - 1; ++i) {
        if (i < mine) load(i, false);
        commit();
    }

    f32x2 acc[TM][TN];
#pragma unroll
    for (int m = 0; m < TM; ++m)
#pragma unroll
        for (int n = 0; n < TN; ++n) acc[m][n] = 0ull;
    const int wm = WM > 1 ? warp : 0, wn = WN > 1 ? warp : 0;
    const bool rows = m0 + wm * TM < M;
    for (int i = 0; i < mine; ++i) {
        asm volatile("cp.async.wait_group %0;" ::"n"(FSTAGES - 2) : "memory");
        __syncthreads();
        if (i + FSTAGES - 1 < mine) { load(i + FSTAGES - 1, true); load(i + FSTAGES - 1, false); }
        commit();
        const float* a_s = tiles + (i % FSTAGES) * (BM + FN) * FPITCH + wm * TM * FPITCH;
        const float* w_s = tiles + (i % FSTAGES) * (BM + FN) * FPITCH + (BM + wn * 32 * TN + lane) * FPITCH;
        if (rows) {
#pragma unroll 2
            for (int k = 0; k < FK; k += 4) {
                ulonglong2 b[TN];
#pragma unroll
                for (int n = 0; n < TN; ++n) b[n] = *(const ulonglong2*)(w_s + n * 32 * FPITCH + k);
#pragma unroll
                for (int m = 0; m < TM; ++m) {
                    const ulonglong2 a = *(const ulonglong2*)(a_s + m * FPITCH + k);
#pragma unroll
                    for (int n = 0; n < TN; ++n) fma2(acc[m][n], a.x, b[n].x);
#pragma unroll
                    for (int n = 0; n < TN; ++n) fma2(acc[m][n], a.y, b[n].y);
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    auto value = [&](int m, int n) {
        return __uint_as_float((unsigned)acc[m][n]) + __uint_as_float((unsigned)(acc[m][n] >> 32));
    };
    if (slices == 1) {
#pragma unroll
        for (int m = 0; m < TM; ++m)
#pragma unroll
            for (int n = 0; n < TN; ++n) {
                const int row = m0 + wm * TM + m, col = n0 + wn * 32 * TN + n * 32 + lane;
                if (row < M && col < N) C[(long long)row * ldc + col] = value(m, n) + (bias ? bias[col] : 0.f);
            }
        return;
    }
    __syncthreads();                                             // the last block has been read: the sums take its place
#pragma unroll
    for (int m = 0; m < TM; ++m)
#pragma unroll
        for (int n = 0; n < TN; ++n) tiles[(wm * TM + m) * FN + wn * 32 * TN + n * 32 + lane] = value(m, n);
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    const int total = min(BM, M - m0) * FN;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(tiles);
    for (int i = slice * THREADS + tid; i < total; i += slices * THREADS) {
        float v[8], sum = 0.f;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            v[q] = 0.f;
            if (q < slices) {
                uint32_t at;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(base + i * 4), "r"(q));
                asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[q]) : "r"(at) : "memory");
            }
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) sum += v[q];
        const int row = m0 + i / FN, col = n0 + i % FN;
        if (col < N) C[(long long)row * ldc + col] = sum + (bias ? bias[col] : 0.f);
    }
    // (nobody leaves while others read its shared memory)
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Slices of the inner dimension: the number for which the rounds over the SMs take the least time, a CTA an SM
// (fewer slices where more gain little); a slice has at least 8 blocks.  Of N and K alone, so that neither M nor
// the device at hand changes a sum: 148 SMs and their GPCs are those of the device the times were taken on.  A cluster
// lies in one GPC (at least 16 SMs there), so clusters of 3, 5, 6 and 7 leave SMs idle.  (97 tokens, 12288 x 2048: 3 slices are 288
// CTAs, but only 135 of them run at once; the SMs were busy for 64 % of the kernel's 245 us.)
int f32_slices(int N, int K) {
    const int tiles = (N + FN - 1) / FN, blocks = (K + FK - 1) / FK;
    int best = 1;
    double best_time = 1e30;
    for (int s = 1; s <= 8 && blocks / s >= 8; ++s) {
        const int at_once = s <= 2 ? 148 : 8 * (16 / s * s) + (16 % s == 0 ? 8 : 0);     // (20 SMs more lie in some GPCs)
        const double time = (double)((tiles * s + at_once - 1) / at_once) / s;
        if (time < best_time * 0.95) { best = s; best_time = time; }
    }
    return best;
}

template <int WM, int WN, int TM, int TN>
int launch_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, long long lda, long long ldw,
               long long ldc, cudaStream_t st) {
    constexpr int BM = WM * TM;
    auto kern = gemm_f32_kernel<WM, WN, TM, TN>;
    const size_t smem = (size_t)FSTAGES * (BM + FN) * FPITCH * sizeof(float);        // (more than the sums take)
    const cudaError_t rc = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (rc != cudaSuccess) { cudaGetLastError(); return (int)rc; }
    const int slices = f32_slices(N, K);
    return crane_launch_cluster(kern, dim3(slices, (N + FN - 1) / FN, (M + BM - 1) / BM), dim3(WM * WN * 32), smem,
                                dim3(slices, 1, 1), st, A, W, bias, C, M, N, K, lda, ldw, ldc);
}

int run_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, long long lda, long long ldw,
            long long ldc, cudaStream_t st) {
#define CRANE_F32(WM, WN, TM, TN) return launch_f32<WM, WN, TM, TN>(A, W, bias, C, M, N, K, lda, ldw, ldc, st)
    if (M <= 1) CRANE_F32(1, 4, 1, 1);
    if (M <= 2) CRANE_F32(1, 4, 2, 1);
    if (M <= 4) CRANE_F32(1, 4, 4, 1);
    if (M <= 8) CRANE_F32(1, 4, 8, 1);
    if (M <= 16) CRANE_F32(1, 4, 16, 1);
    // tiles of at most 128 rows, all about as high
    const int tiles = (M + 127) / 128, tm = ((M + tiles - 1) / tiles + 7) / 8;
    if (tm <= 4) CRANE_F32(8, 1, 4, 4);
    if (tm <= 6) CRANE_F32(8, 1, 6, 4);
    if (tm <= 8) CRANE_F32(8, 1, 8, 4);
    if (tm <= 10) CRANE_F32(8, 1, 10, 4);
    if (tm <= 12) CRANE_F32(8, 1, 12, 4);
    if (tm <= 14) CRANE_F32(8, 1, 14, 4);
    CRANE_F32(8, 1, 16, 4);
#undef CRANE_F32
}
}  // namespace

// in_dtype / out_dtype: 0 = float, 1 = bf16 (out may be float with bf16 inputs).
CRANE_API int crane_gemm_simt(int in_dtype, int out_dtype, const void* A, const void* W,
                              const float* bias, void* C, int M, int N, int K, long long lda,
                              long long ldw, long long ldc, cudaStream_t st) {
    if (M <= 0 || N <= 0) return 0;
    // (the grid's third extent counts tiles of rows)
    if (in_dtype == 0 && out_dtype == 0 && K > 0 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 &&
        ((uintptr_t)A | (uintptr_t)W) % 16 == 0 && (M + 127) / 128 <= 65535 && (N + FN - 1) / FN <= 65535)
        return run_f32((const float*)A, (const float*)W, bias, (float*)C, M, N, K, lda, ldw, ldc, st);
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (in_dtype == 0 && out_dtype == 0)
        gemm_nt_kernel<float, float><<<grid, 256, 0, st>>>((const float*)A, (const float*)W, bias,
                                                           (float*)C, M, N, K, lda, ldw, ldc);
    else if (in_dtype == 1 && out_dtype == 1)
        gemm_nt_kernel<__nv_bfloat16, __nv_bfloat16><<<grid, 256, 0, st>>>(
            (const __nv_bfloat16*)A, (const __nv_bfloat16*)W, bias, (__nv_bfloat16*)C, M, N, K,
            lda, ldw, ldc);
    else if (in_dtype == 1 && out_dtype == 0)
        gemm_nt_kernel<__nv_bfloat16, float><<<grid, 256, 0, st>>>(
            (const __nv_bfloat16*)A, (const __nv_bfloat16*)W, bias, (float*)C, M, N, K, lda, ldw,
            ldc);
    else
        return (int)cudaErrorInvalidValue;
    return crane_launch_status();
}
