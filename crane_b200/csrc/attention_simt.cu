// Attention over the paged cache on the FP32 cores, for any batch of prompt
// portions and single decoded tokens, any key width up to 1024 and any value
// width up to 512.  Values are rows of `dv` elements, `v_stride` elements apart,
// in `v_pool`: a pool of their own, or (v_pool == k_pool, v_stride == d) the
// leading dv columns of the key rows, which is how latent attention keeps them.
// One warp per (token, query head): the token at position p of
// request e attends the keys of positions max(0, p - window + 1) .. p of the
// same request, found through the request's block table.  Scores, softmax
// statistics and the weighted sum are float whatever the storage type.  `sink`: the
// softmax has one more candidate of score 0 and no value (p_j = exp(s_j) / (1 + sum exp(s))); `sinks`: of a
// score of its own per query head.
// `ScoreMod` says what happens to a score before it becomes a weight: squashed to cap * tanh(s / cap);
// keys seen only within the query's own block of `chunk` positions (blocks counted from position 0);
// weights sigmoid(s + bias of the head) that are not normalised over the keys instead of a softmax; a
// head of `maps` maps of d elements side by side in its query and key rows (rows of `d_row` elements, map
// i at i * d_map), each map an attention of its own over the same values; results in float
// [token][head][map][dv].
//
// scores = q k^T / sqrt(d), causal j <= p, softmax over the last dimension,
// query head h reads kv head h / (nq / nkv):
// crane-core/src/models/hunyuan_dense/modeling.rs:572-636, 1012-1033.
#include <type_traits>

#include "common.cuh"

namespace {
constexpr int WARPS = 4;
constexpr int MAXD = 1024;     // widest key row
constexpr int MAXDV = 512;     // widest value row

struct ScoreMod {
    float softcap;              // 0: none
    int chunk;                  // 0: none
    int sigmoid;                // weights sigmoid(s + head_bias[h]), not normalised
    const float* head_bias;     // [nq] or null
    int maps;                   // maps per head (1: a plain head)
    int d_row;                  // elements of a query / key row of a head (>= maps * d_map)
    int d_map;                  // elements from one map's start to the next
    float* out_f32;             // float [token][head][map][dv] instead of `out`, or null
    const float* sinks;         // [nq]: one more candidate of this score and no value per head, or null
};

// What bounds it: a lane reads a key row of its own, so every load of a warp touches 32 rows and takes that many
// look-ups in L1.  WIDE (float rows of whole 16-byte pieces) makes a quarter as many loads, added in the same order;
// NACC is for values of at most 32 * NACC columns (4: 128).  97 tokens, 16 / 4 heads of 128,
// 32-bit: 123 us a layer before; with it and the products' slices chosen by rounds the whole prompt 22.2 -> 17.0 ms.
template <typename T, int NACC, bool WIDE>
__global__ void __launch_bounds__(WARPS * 32)
paged_attention_simt_kernel(const T* __restrict__ q, T* __restrict__ out,
                            const T* __restrict__ k_pool, const T* __restrict__ v_pool,
                            const int* __restrict__ positions, const int* __restrict__ tok_entry,
                            const int* __restrict__ block_table, int max_blocks, int num_pages,
                            int page_size, int n_tokens, int nq, int nkv, int d, int dv,
                            int v_stride, int window, float scale, int sink, float* __restrict__ out_cross,
                            const ScoreMod sm, int* err) {
    extern __shared__ __align__(16) float q_all[];              // [WARPS][d]
    float* q_s = q_all + (threadIdx.x >> 5) * d;
    const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long warp = (long long)blockIdx.x * WARPS + wib;
    // `out_cross`: every query head is paired with every key/value head's values (its keys stay its own
    // group's): nq * nkv warps a token, results float [token][query head][value head][dv]
    const int pairs = out_cross != nullptr ? nq * nkv : nq * sm.maps;
    if (warp >= (long long)n_tokens * pairs) return;
    const int t = (int)(warp / pairs), hv = (int)(warp % pairs);
    const int h = out_cross != nullptr ? hv / nkv : hv / sm.maps;
    const int map_off = out_cross != nullptr ? 0 : (hv % sm.maps) * sm.d_map;
    const int g = h / (nq / nkv);
    const int gv = out_cross != nullptr ? hv % nkv : g;
    const int pos = positions[t];
    if (tok_entry[t] < 0) return;                 // a row that pads the step: it attends to nothing
    const int* table = block_table + (long long)tok_entry[t] * max_blocks;
    const T* qp = q + ((long long)t * nq + h) * sm.d_row + map_off;
    for (int c = lane; c < d; c += 32) q_s[c] = to_f32(qp[c]);
    __syncwarp();

    int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
    if (sm.chunk > 0) lo = max(lo, pos / sm.chunk * sm.chunk);
    const float bias = sm.head_bias != nullptr ? sm.head_bias[h] : 0.f;
    float acc[NACC];
#pragma unroll
    for (int i = 0; i < NACC; ++i) acc[i] = 0.f;
    float m = -INFINITY, l = 0.f;
    bool bad = false;
    const long long v_shift = (long long)(gv - g) * page_size;      // from a key row to the value row read with it

    for (int base = lo; base <= pos; base += 32) {
        const int j = base + lane;
        float s = -INFINITY;
        long long row = -1;                       // this lane's key/value row in the pools
        if (j <= pos) {
            const int page = table[j / page_size];
            if (page < 0 || page >= num_pages) {
                bad = true;
            } else {
                row = ((long long)page * nkv + g) * page_size + j % page_size;
                const T* kp = k_pool + row * sm.d_row + map_off;
                float dot = 0.f;
                if (WIDE) {
#pragma unroll 8
                    for (int c = 0; c < d; c += 4) {
                        const float4 kv = *(const float4*)((const float*)kp + c), qv = *(const float4*)(q_s + c);
                        dot = fmaf(qv.x, kv.x, dot);
                        dot = fmaf(qv.y, kv.y, dot);
                        dot = fmaf(qv.z, kv.z, dot);
                        dot = fmaf(qv.w, kv.w, dot);
                    }
                } else {
                    for (int c = 0; c < d; ++c) dot = fmaf(q_s[c], to_f32(kp[c]), dot);
                }
                s = dot * scale;
                if (sm.softcap > 0.f) s = sm.softcap * tanhf(s / sm.softcap);
            }
        }
        float p;
        if (sm.sigmoid) {
            p = (s == -INFINITY) ? 0.f : 1.f / (1.f + expf(-(s + bias)));
        } else {
            const float m_new = fmaxf(m, warp_max(s));
            if (m_new == -INFINITY) continue;         // every key of this chunk was unreadable
            p = (s == -INFINITY) ? 0.f : expf(s - m_new);
            const float corr = (m == -INFINITY) ? 0.f : expf(m - m_new);
            l = l * corr + warp_sum(p);
            m = m_new;
#pragma unroll
            for (int i = 0; i < NACC; ++i) acc[i] *= corr;
        }
        const int cnt = min(32, pos - base + 1);
        for (int jj = 0; jj < cnt; ++jj) {
            const float pj = __shfl_sync(0xffffffffu, p, jj);
            const long long rj = __shfl_sync(0xffffffffu, row, jj);
            if (rj < 0) continue;
            const T* vp = v_pool + (rj + v_shift) * v_stride;
#pragma unroll
            for (int i = 0; i < NACC; ++i) {
                const int c = lane + 32 * i;
                if (c < dv) acc[i] = fmaf(pj, to_f32(vp[c]), acc[i]);
            }
        }
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(err, CRANE_ERR_PAGE_RANGE);
    // a sink: one more candidate of score 0 that has no value, so it only adds exp(0 - m) to the sum
    if (sink) l += expf(-m);
    float inv = sm.sigmoid ? 1.f : l > 0.f ? 1.f / l : 0.f;
    if (sm.sinks != nullptr) {
        const float s = sm.sinks[h], top = fmaxf(m, s), mine = expf(m - top);
        inv = mine / fmaf(l, mine, expf(s - top));
    }
    if (sm.out_f32 != nullptr) {
        float* op = sm.out_f32 + ((long long)t * pairs + hv) * dv;
#pragma unroll
        for (int i = 0; i < NACC; ++i) {
            const int c = lane + 32 * i;
            if (c < dv) op[c] = acc[i] * inv;
        }
        return;
    }
    if (out_cross != nullptr) {
        float* op = out_cross + ((long long)t * pairs + hv) * dv;
#pragma unroll
        for (int i = 0; i < NACC; ++i) {
            const int c = lane + 32 * i;
            if (c < dv) op[c] = acc[i] * inv;
        }
        return;
    }
    T* op = out + ((long long)t * nq + h) * dv;
#pragma unroll
    for (int i = 0; i < NACC; ++i) {
        const int c = lane + 32 * i;
        if (c < dv) op[c] = from_f32<T>(acc[i] * inv);
    }
}

// ---- plain softmax attention over float rows, several query rows of a key/value head per CTA ------------------------
// What bounds it: shared-memory reads (about 1,400 wavefronts a tile of 32 keys), the barriers between a
// tile's steps and the way of the first tiles from memory.  16
// query rows (the heads of a group times as many neighbouring tokens as fit) share every key and value that comes in, 32
// keys at a time by asynchronous copies, one tile ahead; a thread has 2 x 2 scores, then 4 x 4 results.  97 tokens, 16 / 4 heads
// of 128: 66 us with a warp per (token, head), whose lanes each read a key row of their own, 17 us
// here (25 when a lane looked up 8 keys one after the other); 2,048 tokens 5,370 / 910, one token behind 8,192 keys 3,070 / 740.
// Tiles of keys start at multiples of 32 and a row leaves out what is not its own, so that its result does not
// depend on the rows beside it.  Tokens of several requests in one CTA are taken request by request.
constexpr int TROWS = 16, TKEYS = 32, TDIM = 128, TPITCH = TDIM + 4;

struct TileParams {
    const float* q;
    float* out;
    const float* k_pool;
    const float* v_pool;
    const int* positions;
    const int* tok_entry;
    const int* block_table;
    int max_blocks, num_pages, page_size, n_tokens, nq, nkv, d, dv, v_stride, window;
    float scale;
    int sink;
    const float* sinks;
    int* err;
};

__device__ __forceinline__ float half_max(float v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float half_sum(float v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__global__ void __launch_bounds__(128)
paged_attention_tile_kernel(const TileParams p) {
    extern __shared__ __align__(16) float tile_smem[];
    float* q_s = tile_smem;                                      // [TROWS][TPITCH]
    float* k_s = q_s + TROWS * TPITCH;                           // [2][TKEYS][TPITCH]
    float* v_s = k_s + 2 * TKEYS * TPITCH;                       // [2][TKEYS][TDIM]
    float* p_s = v_s + 2 * TKEYS * TDIM;                         // [TROWS][TKEYS]
    float* corr_s = p_s + TROWS * TKEYS;                         // [TROWS]
    int* there_s = (int*)(corr_s + TROWS);                       // [2][TKEYS]: the key's page is one of the pool
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int group = p.nq / p.nkv, tokens = TROWS / group, g = blockIdx.x;
    const int t0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * tokens;              // (later tokens have more keys: they begin)
    const int d4 = p.d >> 2, dv4 = p.dv >> 2;
    pdl_launch_dependents();
    pdl_wait();
    for (int i = tid; i < TROWS * d4; i += 128) {
        const int r = i / d4, c = i - r * d4, t = t0 + r / group;
        const float4 v = r / group < tokens && t < p.n_tokens
                             ? *(const float4*)(p.q + ((long long)t * p.nq + g * group + r % group) * p.d + 4 * c)
                             : make_float4(0.f, 0.f, 0.f, 0.f);
        *(float4*)(q_s + r * TPITCH + 4 * c) = v;
    }
    // scores: rows 2 ry and 2 ry + 1, keys kx and kx + 16 of a tile; results: rows 4 warp .. + 3, columns 4 lane .. + 3
    const int ry = tid >> 4, kx = tid & 15;
    int pos[2], lo[2], entry[2];
    float m[2], l[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int r = 2 * ry + i, t = t0 + r / group;
        const bool mine = r / group < tokens && t < p.n_tokens;
        entry[i] = mine ? p.tok_entry[t] : -1;
        pos[i] = mine ? p.positions[t] : -1;
        lo[i] = p.window > 0 ? max(0, pos[i] - p.window + 1) : 0;
        m[i] = -INFINITY;
        l[i] = 0.f;
    }
    float4 acc[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    bool bad = false;

    const int t_end = min(t0 + tokens, p.n_tokens);
    for (int t = t0; t < t_end;) {
        // a run of tokens of one request: which keys they see
        const int e = p.tok_entry[t];
        int from = 0x7fffffff, to = -1, all_from = 0, all_to = 0x7fffffff;       // keys of some token, of every token
        const bool alone = t == t0;
        for (; t < t_end && p.tok_entry[t] == e; ++t) {
            const int at = p.positions[t], begin = p.window > 0 ? max(0, at - p.window + 1) : 0;
            from = min(from, begin);
            to = max(to, at);
            all_from = max(all_from, begin);
            all_to = min(all_to, at);
        }
        const bool one_run = alone && t == t_end;
        if (e < 0) continue;                                     // rows that pad the step attend to nothing
        const int* table = p.block_table + (long long)e * p.max_blocks;
        const int first = from / TKEYS, count = to / TKEYS + 1 - first;
        auto load = [&](int i) {                                 // tile i of the run
            float* kt = k_s + (i & 1) * TKEYS * TPITCH;
            float* vt = v_s + (i & 1) * TKEYS * TDIM;
            // every lane looks up a key of the tile, so that the look-ups take the time of one
            const int j = (first + i) * TKEYS + lane, slot = j / p.page_size;
            const int page = j <= to ? table[slot] : -1;
            const bool there = page >= 0 && page < p.num_pages;
            if (!there && j >= from && j <= to) bad = true;
            const long long row = there ? ((long long)page * p.nkv + g) * p.page_size + (j - slot * p.page_size) : -1;
            if (warp == 0) there_s[(i & 1) * TKEYS + lane] = there;
#pragma unroll
            for (int r = 0; r < TKEYS / 4; ++r) {
                const long long mine = __shfl_sync(0xffffffffu, row, 4 * r + warp);
                const uint32_t bytes = mine >= 0 ? 16 : 0;                       // (0: zeros)
                const long long from_row = mine >= 0 ? mine : 0;
                if (lane < d4)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::
                                 "r"((uint32_t)__cvta_generic_to_shared(kt + (4 * r + warp) * TPITCH + 4 * lane)),
                                 "l"(p.k_pool + from_row * p.d + 4 * lane), "r"(bytes) : "memory");
                if (lane < dv4)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::
                                 "r"((uint32_t)__cvta_generic_to_shared(vt + (4 * r + warp) * TDIM + 4 * lane)),
                                 "l"(p.v_pool + from_row * p.v_stride + 4 * lane), "r"(bytes) : "memory");
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        __syncthreads();                                         // (nobody reads the run before any more; q_s is there)
        load(0);
        for (int i = 0; i < count; ++i) {
            if (i + 1 < count) load(i + 1);
            if (i + 1 < count) asm volatile("cp.async.wait_group 1;" ::: "memory");
            else asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            const float* kt = k_s + (i & 1) * TKEYS * TPITCH;
            const float* vt = v_s + (i & 1) * TKEYS * TDIM;
            float s[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
            const float* qa = q_s + 2 * ry * TPITCH;
            const float* ka = kt + kx * TPITCH;
#pragma unroll 8
            for (int c = 0; c < p.d; c += 4) {
                const float4 q0 = *(const float4*)(qa + c), q1 = *(const float4*)(qa + TPITCH + c);
                const float4 k0 = *(const float4*)(ka + c), k1 = *(const float4*)(ka + 16 * TPITCH + c);
                s[0][0] = fmaf(q0.w, k0.w, fmaf(q0.z, k0.z, fmaf(q0.y, k0.y, fmaf(q0.x, k0.x, s[0][0]))));
                s[0][1] = fmaf(q0.w, k1.w, fmaf(q0.z, k1.z, fmaf(q0.y, k1.y, fmaf(q0.x, k1.x, s[0][1]))));
                s[1][0] = fmaf(q1.w, k0.w, fmaf(q1.z, k0.z, fmaf(q1.y, k0.y, fmaf(q1.x, k0.x, s[1][0]))));
                s[1][1] = fmaf(q1.w, k1.w, fmaf(q1.z, k1.z, fmaf(q1.y, k1.y, fmaf(q1.x, k1.x, s[1][1]))));
            }
            const int j0 = (first + i) * TKEYS + kx;
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                float w[2];
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const int j = j0 + 16 * b;
                    const bool sees = entry[a] == e && j >= lo[a] && j <= pos[a] && there_s[(i & 1) * TKEYS + kx + 16 * b];
                    w[b] = sees ? s[a][b] * p.scale : -INFINITY;
                }
                const float m_new = fmaxf(m[a], half_max(fmaxf(w[0], w[1])));
#pragma unroll
                for (int b = 0; b < 2; ++b) w[b] = w[b] == -INFINITY ? 0.f : expf(w[b] - m_new);
                const float corr = m_new == -INFINITY ? 1.f : m[a] == -INFINITY ? 0.f : expf(m[a] - m_new);
                l[a] = l[a] * corr + half_sum(w[0] + w[1]);
                m[a] = m_new;
                p_s[(2 * ry + a) * TKEYS + kx] = w[0];
                p_s[(2 * ry + a) * TKEYS + kx + 16] = w[1];
                if (kx == 0) corr_s[2 * ry + a] = corr;
            }
            __syncthreads();
            if (lane < dv4) {
                const float* pr = p_s + 4 * warp * TKEYS;
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    const float corr = corr_s[4 * warp + a];
                    acc[a].x *= corr; acc[a].y *= corr; acc[a].z *= corr; acc[a].w *= corr;
                }
                // (a weight of 0 leaves a key's values out, whatever they are, in tiles that not every row sees all of)
                auto values = [&](auto some) {
#pragma unroll 2
                    for (int j = 0; j < TKEYS; j += 4) {
                        float4 w[4];
#pragma unroll
                        for (int a = 0; a < 4; ++a) w[a] = *(const float4*)(pr + a * TKEYS + j);
#pragma unroll
                        for (int b = 0; b < 4; ++b) {
                            const float4 v = *(const float4*)(vt + (j + b) * TDIM + 4 * lane);
#pragma unroll
                            for (int a = 0; a < 4; ++a) {
                                const float x = b == 0 ? w[a].x : b == 1 ? w[a].y : b == 2 ? w[a].z : w[a].w;
                                if (decltype(some)::value && x == 0.f) continue;
                                acc[a].x = fmaf(x, v.x, acc[a].x);
                                acc[a].y = fmaf(x, v.y, acc[a].y);
                                acc[a].z = fmaf(x, v.z, acc[a].z);
                                acc[a].w = fmaf(x, v.w, acc[a].w);
                            }
                        }
                    }
                };
                const int j0 = (first + i) * TKEYS;
                if (one_run && j0 >= all_from && j0 + TKEYS - 1 <= all_to) values(std::false_type{});
                else values(std::true_type{});
            }
            __syncthreads();                                     // before the tile after next and its weights come here
        }
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(p.err, CRANE_ERR_PAGE_RANGE);
    // what a row's sum is divided by, with the candidates that have no value
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        float sum = l[a];
        if (p.sink) sum += expf(-m[a]);
        float inv = sum > 0.f ? 1.f / sum : 0.f;
        if (p.sinks != nullptr) {
            const float s = p.sinks[g * group + (2 * ry + a) % group], top = fmaxf(m[a], s), mine = expf(m[a] - top);
            inv = mine / fmaf(sum, mine, expf(s - top));
        }
        __syncwarp();
        if (kx == 0) corr_s[2 * ry + a] = inv;
    }
    __syncthreads();
    if (lane < dv4) {
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int r = 4 * warp + a, t = t0 + r / group;
            if (r / group >= tokens || t >= p.n_tokens || p.tok_entry[t] < 0) continue;
            const float inv = corr_s[r];
            *(float4*)(p.out + ((long long)t * p.nq + g * group + r % group) * p.dv + 4 * lane) =
                make_float4(acc[a].x * inv, acc[a].y * inv, acc[a].z * inv, acc[a].w * inv);
        }
    }
}
}  // namespace

static int launch_simt(int dtype, const void* q, void* out, const void* k_pool, const void* v_pool,
                       const int* positions, const int* tok_entry, const int* block_table, int max_blocks,
                       int num_pages, int page_size, int n_tokens, int nq, int nkv, int d, int dv, int v_stride,
                       int window, float scale, int sink, float* out_cross, ScoreMod sm, int* err,
                       cudaStream_t st) {
    if (n_tokens <= 0) return 0;
    if (d > MAXD || d <= 0 || dv > MAXDV || dv <= 0 || v_stride < dv || nkv <= 0 || nq % nkv != 0 ||
        sm.maps < 1 || sm.d_row < (sm.maps - 1) * sm.d_map + d || (out_cross != nullptr && sm.maps != 1))
        return (int)cudaErrorInvalidValue;
    // Plain softmax over heads of at most 128 elements in whole 16-byte pieces, whose groups fit 16 rows: many rows share what they
    // read.  (By what the attention is, never by the step: a row's result must not depend on the rows beside it.)
    const bool plain = dtype == 0 && out_cross == nullptr && sm.maps == 1 && sm.softcap == 0.f && sm.chunk == 0 && !sm.sigmoid &&
                       sm.out_f32 == nullptr && sm.d_row == d;
    if (plain && d <= TDIM && dv <= TDIM && (d | dv | v_stride) % 4 == 0 && nq / nkv <= TROWS &&
        ((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_pool | (uintptr_t)v_pool) % 16 == 0) {
        const int tokens = TROWS / (nq / nkv);
        const size_t need = (size_t)(TROWS * TPITCH + 2 * TKEYS * (TPITCH + TDIM) + TROWS * (TKEYS + 1) + 2 * TKEYS) * sizeof(float);
        static bool configured = false;
        if (!configured) {
            const cudaError_t rc = cudaFuncSetAttribute(paged_attention_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)need);
            if (rc != cudaSuccess) { cudaGetLastError(); return (int)rc; }
            configured = true;
        }
        const int tiles = (n_tokens + tokens - 1) / tokens;
        if (tiles <= 65535) {
            const TileParams tp{(const float*)q, (float*)out, (const float*)k_pool, (const float*)v_pool, positions, tok_entry, block_table,
                                max_blocks, num_pages, page_size, n_tokens, nq, nkv, d, dv, v_stride, window, scale, sink, sm.sinks, err};
            return crane_launch(paged_attention_tile_kernel, dim3(nkv, tiles), dim3(128), need, st, tp);
        }
    }
    const size_t smem = (size_t)WARPS * d * sizeof(float);
    const long long warps = (long long)n_tokens * nq * (out_cross != nullptr ? nkv : sm.maps);
    const int blocks = (int)((warps + WARPS - 1) / WARPS);
    const bool wide = dtype == 0 && (d | sm.d_row | sm.d_map) % 4 == 0 && (uintptr_t)k_pool % 16 == 0;
    auto run = [&](auto kern, auto* type) {
        using T = std::remove_pointer_t<decltype(type)>;
        kern<<<blocks, WARPS * 32, smem, st>>>((const T*)q, (T*)out, (const T*)k_pool, (const T*)v_pool, positions, tok_entry,
                                               block_table, max_blocks, num_pages, page_size, n_tokens, nq, nkv, d, dv, v_stride,
                                               window, scale, sink, out_cross, sm, err);
    };
    constexpr int FEW = 4, MOST = MAXDV / 32;
    if (dtype != 0) {
        if (dv <= FEW * 32) run(paged_attention_simt_kernel<__nv_bfloat16, FEW, false>, (__nv_bfloat16*)nullptr);
        else run(paged_attention_simt_kernel<__nv_bfloat16, MOST, false>, (__nv_bfloat16*)nullptr);
    } else if (wide) {
        if (dv <= FEW * 32) run(paged_attention_simt_kernel<float, FEW, true>, (float*)nullptr);
        else run(paged_attention_simt_kernel<float, MOST, true>, (float*)nullptr);
    } else {
        if (dv <= FEW * 32) run(paged_attention_simt_kernel<float, FEW, false>, (float*)nullptr);
        else run(paged_attention_simt_kernel<float, MOST, false>, (float*)nullptr);
    }
    return crane_launch_status();
}

CRANE_API int crane_paged_attention_simt(int dtype, const void* q, void* out, const void* k_pool,
                                         const void* v_pool, const int* positions,
                                         const int* tok_entry, const int* block_table,
                                         int max_blocks, int num_pages, int page_size,
                                         int n_tokens, int nq, int nkv, int d, int dv,
                                         int v_stride, int window, float scale, int sink, const float* sinks,
                                         float* out_cross, int* err, cudaStream_t st) {
    const ScoreMod plain{0.f, 0, 0, nullptr, 1, d, d, nullptr, sinks};
    return launch_simt(dtype, q, out, k_pool, v_pool, positions, tok_entry, block_table, max_blocks, num_pages,
                       page_size, n_tokens, nq, nkv, d, dv, v_stride, window, scale, sink, out_cross, plain, err, st);
}

// The same with the scores worked on (see ScoreMod): d is the width of one map.
CRANE_API int crane_scored_attention_simt(int dtype, const void* q, void* out, const void* k_pool,
                                          const void* v_pool, const int* positions, const int* tok_entry,
                                          const int* block_table, int max_blocks, int num_pages, int page_size,
                                          int n_tokens, int nq, int nkv, int d, int dv, int v_stride, int window,
                                          float scale, float softcap, int chunk, int sigmoid,
                                          const float* head_bias, int maps, int d_row, int d_map, float* out_f32,
                                          int* err, cudaStream_t st) {
    const ScoreMod sm{softcap, chunk, sigmoid, head_bias, maps, d_row, d_map, out_f32, nullptr};
    return launch_simt(dtype, q, out, k_pool, v_pool, positions, tok_entry, block_table, max_blocks, num_pages,
                       page_size, n_tokens, nq, nkv, d, dv, v_stride, window, scale, 0, nullptr, sm, err, st);
}
