// Shared device helpers for the sm_100a kernels of this engine.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

#define CRANE_API extern "C" __attribute__((visibility("default")))

// Bits of the device-side error word.  Kernels never trap: they record what
// went wrong, skip the access and return; the host reads the word after a step.
enum CraneErr : int {
    CRANE_ERR_TOKEN_RANGE = 1,      // token id outside the vocabulary
    CRANE_ERR_PAGE_RANGE = 2,       // block-table entry outside the page pool
    CRANE_ERR_POSITION_RANGE = 4,   // position outside the rotary table
    CRANE_ERR_WAIT_TIMEOUT = 8,     // a bounded mbarrier wait ran out
    CRANE_ERR_SLOT_RANGE = 16,
};

__device__ __forceinline__ float to_f32(float v) { return v; }
__device__ __forceinline__ float to_f32(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) {
    return __float2bfloat16_rn(v);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Sum over a whole block of up to 1024 threads; every thread gets the result.
__device__ __forceinline__ float block_sum(float v, float* scratch32) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nwarps = (blockDim.x + 31) >> 5;
    v = warp_sum(v);
    __syncthreads();                 // scratch may still be read from an earlier call
    if (lane == 0) scratch32[warp] = v;
    __syncthreads();
    float t = (lane < nwarps) ? scratch32[lane] : 0.f;
    return warp_sum(t);
}

// How a mixer's heads are rotated and normalised.  The defaults are Hunyuan Dense's: the whole head
// rotated in the contiguous-halves pairing, RMSNorm after the rotation, plain weights.
struct RopeParams {
    int rotary_dim;      // the leading elements of a head that are rotated (even, <= head size)
    int interleaved;     // 0: element i pairs with i + rotary_dim / 2;  1: 2i with 2i + 1
    int norm_first;      // 0: per-head RMSNorm after the rotation;  1: before it
    float norm_offset;   // the norm multiplies by (norm_offset + w): 0 plain, 1 for weights stored as w - 1
};
static inline bool rope_is_default(const RopeParams& p, int d) {
    return p.rotary_dim == d && !p.interleaved && !p.norm_first && p.norm_offset == 0.f;
}
// A head of d elements seen as d / 2 slots of two elements: slot i < rotary_dim / 2 holds a rotated
// pair (its angle is column i of the tables), the other slots hold the neighbours behind the rotated part.
__device__ __forceinline__ void rope_slot(const RopeParams& p, int i, int& ea, int& eb, bool& rot) {
    const int hr = p.rotary_dim >> 1;
    rot = i < hr;
    if (rot) {
        ea = p.interleaved ? 2 * i : i;
        eb = p.interleaved ? 2 * i + 1 : i + hr;
    } else {
        ea = p.rotary_dim + 2 * (i - hr);
        eb = ea + 1;
    }
}
// One head row by one warp for any RopeParams: `load(e)` gives element e as float, `store(e, v)`
// takes the result.  cos/sin tables are [positions][rotary_dim / 2].  nw: the norm's weight or null.
template <int MAXS, typename Load, typename Store>
__device__ __forceinline__ void rope_norm_general(const RopeParams& rp, int d, int pos, bool rotate,
                                                  const float* __restrict__ cos_tab,
                                                  const float* __restrict__ sin_tab,
                                                  const float* __restrict__ nw, float eps, int lane,
                                                  Load load, Store store) {
    const int hr = rp.rotary_dim >> 1, slots = d >> 1;
    float a[MAXS], b[MAXS];
    float ss = 0.f;
#pragma unroll
    for (int s = 0; s < MAXS; ++s) {
        const int i = lane + 32 * s;
        a[s] = b[s] = 0.f;
        if (i < slots) {
            int ea, eb; bool rot;
            rope_slot(rp, i, ea, eb, rot);
            a[s] = load(ea);
            b[s] = load(eb);
            ss += a[s] * a[s] + b[s] * b[s];
        }
    }
    if (nw != nullptr && rp.norm_first) {
        unsigned m = 0xffffffffu;
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(m, ss, o);
        const float rstd = rsqrtf(ss / (float)d + eps);
#pragma unroll
        for (int s = 0; s < MAXS; ++s) {
            const int i = lane + 32 * s;
            if (i < slots) {
                int ea, eb; bool rot;
                rope_slot(rp, i, ea, eb, rot);
                a[s] = a[s] * rstd * (rp.norm_offset + nw[ea]);
                b[s] = b[s] * rstd * (rp.norm_offset + nw[eb]);
            }
        }
    }
    ss = 0.f;
#pragma unroll
    for (int s = 0; s < MAXS; ++s) {
        const int i = lane + 32 * s;
        if (i < slots) {
            if (rotate && i < hr) {
                const float c = cos_tab[(long long)pos * hr + i], sn = sin_tab[(long long)pos * hr + i];
                const float x1 = a[s], x2 = b[s];
                a[s] = x1 * c - x2 * sn;
                b[s] = x2 * c + x1 * sn;
            }
            ss += a[s] * a[s] + b[s] * b[s];
        }
    }
    float rstd = 1.f;
    const bool after = nw != nullptr && !rp.norm_first;
    if (after) {
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        rstd = rsqrtf(ss / (float)d + eps);
    }
#pragma unroll
    for (int s = 0; s < MAXS; ++s) {
        const int i = lane + 32 * s;
        if (i < slots) {
            int ea, eb; bool rot;
            rope_slot(rp, i, ea, eb, rot);
            store(ea, after ? a[s] * rstd * (rp.norm_offset + nw[ea]) : a[s]);
            store(eb, after ? b[s] * rstd * (rp.norm_offset + nw[eb]) : b[s]);
        }
    }
}

__device__ __forceinline__ float2 ld2(const float* p) { return *(const float2*)p; }
__device__ __forceinline__ float2 ld2(const __nv_bfloat16* p) {
    return __bfloat1622float2(*(const __nv_bfloat162*)p);
}
__device__ __forceinline__ void st2(float* p, float a, float b) { *(float2*)p = make_float2(a, b); }
__device__ __forceinline__ void st2(__nv_bfloat16* p, float a, float b) {
    *(__nv_bfloat162*)p = __floats2bfloat162_rn(a, b);
}

// 32 neighbouring bytes of a row (at least 16-byte aligned) in one store.  Where every lane of a warp writes a row of its own, as
// behind the accumulators of the tensor cores, a store takes the load/store unit a cycle per row whatever its width: 16-byte
// stores kept it busy for most of the 3.6 us that the epilogue of a 128 x 256 tile of bf16 took an SM, and what they wrote were
// half sectors; with these it takes 1.9.
__device__ __forceinline__ void store32(void* dst, const uint32_t (&w)[8]) {
    if (((uintptr_t)dst & 31) == 0) {
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]),
                     "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                     : "memory");
    } else {
        ((uint4*)dst)[0] = make_uint4(w[0], w[1], w[2], w[3]);
        ((uint4*)dst)[1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
}
__device__ __forceinline__ uint32_t bf16x2_bits(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *(const uint32_t*)&h;
}

// A GEMM result is either one tensor of T or `n_parts` float partial sums
// (split-K), laid out [part][row][col]; readers add the partials in a fixed
// order and round once to T, so that both forms give the same value.
template <typename T>
struct GemmOut {
    const T* whole;
    const float* parts;
    int n_parts;
    long long part_stride;
    // The partial sums are fetched eight at a time (all loads in flight together) and added in
    // slice order, so the sum is the same as a one-by-one loop's.
    __device__ __forceinline__ float load(long long idx) const {
        if (parts == nullptr) return to_f32(whole[idx]);
        float s = 0.f;
        for (int i = 0; i < n_parts; i += 8) {
            float p[8];
#pragma unroll
            for (int j = 0; j < 8; ++j)
                p[j] = (i + j < n_parts) ? parts[(long long)(i + j) * part_stride + idx] : 0.f;
#pragma unroll
            for (int j = 0; j < 8; ++j) s += p[j];
        }
        return to_f32(from_f32<T>(s));
    }
    // two neighbours at once; idx even and the tensors' rows evenly long
    __device__ __forceinline__ float2 load2(long long idx) const {
        if (parts == nullptr) return ld2(whole + idx);
        float2 s = make_float2(0.f, 0.f);
        for (int i = 0; i < n_parts; i += 8) {
            float2 p[8];
#pragma unroll
            for (int j = 0; j < 8; ++j)
                p[j] = (i + j < n_parts) ? *(const float2*)(parts + (long long)(i + j) * part_stride + idx)
                                         : make_float2(0.f, 0.f);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                s.x += p[j].x;
                s.y += p[j].y;
            }
        }
        return make_float2(to_f32(from_f32<T>(s.x)), to_f32(from_f32<T>(s.y)));
    }
};

// Runs the statement with T = float (dtype 0) or bf16 (dtype 1).
#define DISPATCH_T(dtype, ...)                                   \
    if ((dtype) == 0) { using T = float; __VA_ARGS__; }          \
    else { using T = __nv_bfloat16; __VA_ARGS__; }

// Programmatic dependent launch: a kernel launched with the attribute may start
// while the kernel before it in the stream is still running.  It must not touch
// anything that kernel (or one before it) writes or reads-then-overwrites until
// it has called pdl_wait(), which returns once all earlier kernels are complete
// and their writes visible.  pdl_launch_dependents() lets the NEXT kernel start
// early in the same way.  Without the attribute both are no-ops.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

static inline int crane_launch_status() { return (int)cudaGetLastError(); }

// 1: kernels of a decoder step are launched with programmatic dependent launch.
extern int g_crane_pdl;

template <typename... KArgs, typename... Args>
static inline int crane_launch(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem,
                               cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_crane_pdl ? 1 : 0;
    const cudaError_t rc = cudaLaunchKernelEx(&cfg, kern, KArgs(args)...);
    const cudaError_t last = cudaGetLastError();        // read, and with that cleared, in either case:
    return rc != cudaSuccess ? (int)rc : (int)last;     // a refused launch must not fail the next one too
}

// The same for a kernel whose CTAs form thread-block clusters of `cluster` CTAs.
template <typename... KArgs, typename... Args>
static inline int crane_launch_cluster(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem,
                                       dim3 cluster, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster.x;
    attr[0].val.clusterDim.y = cluster.y;
    attr[0].val.clusterDim.z = cluster.z;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_crane_pdl ? 2 : 1;
    const cudaError_t rc = cudaLaunchKernelEx(&cfg, kern, KArgs(args)...);
    const cudaError_t last = cudaGetLastError();        // read, and with that cleared, in either case:
    return rc != cudaSuccess ? (int)rc : (int)last;     // a refused launch must not fail the next one too
}
