// Paged GQA attention in fp32 arithmetic throughout: the 32-bit path's attention and the fallback for sizes
// the tensor-core kernels refuse.
//
// Query at absolute position p of request row r sees keys j with
// max(0, p + 1 - window) <= j <= p (kairyu/engine/core/attention/torch_backend.py:57-71;
// the window is this engine's addition for cache groups that keep only recent keys).
// Query head h reads KV head h / (Hq / Hkv).  S = q.k * scale, softmax, P.V.
//
// The order of every sum depends only on (p, window, D), so a token's output does not
// depend on what else is in the batch or how the prompt was cut.  Two kernels, chosen by type, widths and alignment alone:
//
//   tiled    fp32 rows of whole 16 bytes, D up to 256 (below)
//   generic  any type and size: one block per (query token, query head); warp w of the block
//            takes keys start+w, start+w+4, ... with an online softmax of its own, and the
//            four partial results are merged in warp order
//
// sinks (optional, one fp32 logit a query head): the softmax's denominator also holds exp(sink_h).
// A sink is a term exp(sink) of the denominator alone, taken as stored; it is added once, after all merges.
//
// v_dim (<= D): how many columns of a value row are used and written (out rows are Hq * v_dim wide).
// Keys and values may be the same rows (a cache whose rows serve as both) with the values their
// first v_dim columns.  Head h's output starts at column h * out_head_stride of its token's row.
#include "common.cuh"

#define ATT_WARPS 4
#define ATT_MAX_D 1024
#define ATT_MAX_K (ATT_MAX_D / 32)

template <typename T>
__global__ void __launch_bounds__(ATT_WARPS * 32)
paged_attention_generic_kernel(const T* __restrict__ q, int q_stride, T* __restrict__ out,
                               int out_stride, const T* __restrict__ k_cache,
                               const T* __restrict__ v_cache, const int* __restrict__ positions,
                               const int* __restrict__ row_ids,
                               const int* __restrict__ block_table, int max_pages, int Hq, int Hkv,
                               int D, int page_size, int num_pages, float scale, int window,
                               const float* __restrict__ sinks, int v_dim, int out_head_stride, int* flag) {
    pdl_wait();
    __shared__ float sm_acc[ATT_WARPS][ATT_MAX_D];
    __shared__ float sm_m[ATT_WARPS];
    __shared__ float sm_l[ATT_WARPS];

    const int t = blockIdx.x;
    const int h = blockIdx.y;
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int pos = positions[t];
    const int row = row_ids[t];
    const int kvh = h / (Hq / Hkv);
    const int* table = block_table + (size_t)row * max_pages;
    const int start = (window > 0 && pos + 1 > window) ? pos + 1 - window : 0;

    float qv[ATT_MAX_K];
    const T* qp = q + (size_t)t * q_stride + (size_t)h * D;
#pragma unroll
    for (int k = 0; k < ATT_MAX_K; ++k) {
        const int e = lane + 32 * k;
        qv[k] = e < D ? to_float(qp[e]) : 0.0f;
    }

    float m = -INFINITY, l = 0.0f;
    float acc[ATT_MAX_K];
#pragma unroll
    for (int k = 0; k < ATT_MAX_K; ++k) acc[k] = 0.0f;

    for (int j = start + warp; j <= pos; j += ATT_WARPS) {
        const int page_index = j / page_size;
        int page = page_index < max_pages ? table[page_index] : -1;
        if (page < 0 || page >= num_pages) {
            if (lane == 0 && flag) atomicOr(flag, KB_FLAG_BAD_PAGE);
            continue;
        }
        const size_t base = (((size_t)page * page_size + (j % page_size)) * Hkv + kvh) * D;
        const T* kp = k_cache + base;
        const T* vp = v_cache + base;
        float dot = 0.0f;
#pragma unroll
        for (int k = 0; k < ATT_MAX_K; ++k) {
            const int e = lane + 32 * k;
            if (e < D) dot += qv[k] * to_float(kp[e]);
        }
        dot = warp_sum(dot) * scale;
        const float m_new = fmaxf(m, dot);
        const float alpha = expf(m - m_new);
        const float p = expf(dot - m_new);
        l = l * alpha + p;
#pragma unroll
        for (int k = 0; k < ATT_MAX_K; ++k) {
            const int e = lane + 32 * k;
            if (e < v_dim) acc[k] = acc[k] * alpha + p * to_float(vp[e]);
        }
        m = m_new;
    }

#pragma unroll
    for (int k = 0; k < ATT_MAX_K; ++k) {
        const int e = lane + 32 * k;
        if (e < v_dim) sm_acc[warp][e] = acc[k];
    }
    if (lane == 0) {
        sm_m[warp] = m;
        sm_l[warp] = l;
    }
    __syncthreads();

    float big = -INFINITY;
#pragma unroll
    for (int w = 0; w < ATT_WARPS; ++w) big = fmaxf(big, sm_m[w]);
    const float sink = sinks ? sinks[h] : -INFINITY;
    big = fmaxf(big, sink);
    float weights[ATT_WARPS];
    float denom = 0.0f;
#pragma unroll
    for (int w = 0; w < ATT_WARPS; ++w) {
        weights[w] = sm_m[w] == -INFINITY ? 0.0f : expf(sm_m[w] - big);
        denom += sm_l[w] * weights[w];
    }
    if (sinks) denom += expf(sink - big);
    T* op = out + (size_t)t * out_stride + (size_t)h * out_head_stride;
    for (int e = threadIdx.x; e < v_dim; e += blockDim.x) {
        float v = 0.0f;
#pragma unroll
        for (int w = 0; w < ATT_WARPS; ++w) v += sm_acc[w][e] * weights[w];
        op[e] = from_float<T>(denom > 0.0f ? v / denom : 0.0f);
    }
}

// ------------------------------------------------------------------ tiled
//
// A block has up to 16 * TM query rows: neighbouring tokens of one request, each with all query heads of one key/value head, so that a tile of
// 64 keys and values in shared memory serves them all.  Keys are cut at multiples of 64 of their position into tiles and at multiples of 256 into segments.  Within a
// segment an online softmax goes from tile to tile; a segment begins anew, and segments are merged in order.  A row's scores of a tile lie with sixteen
// lanes, four each, and are summed in lane order, so that a row's arithmetic is the same whichever rows share its block, and the same when
// the segments of a step of single tokens are spread over blocks and merged by a kernel of their own.
//
// What bounds it: reads of shared memory, (4 + TM) 16-byte reads for 16 TM multiply-adds a thread in both products.  What it
// replaces read every key once a query head and token: 826 us of a layer of 700 tokens in three prompts, 16 heads of 128 over 4.
#define TILE_KEYS 64
#define SEGMENT_KEYS 256
#define TILED_THREADS 256

namespace {

__device__ __forceinline__ void copy16(float* dst, const float* src, bool live) {
    const int bytes = live ? 16 : 0;  // the rest is filled with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}

// two multiply-adds in one instruction, each rounded as fmaf rounds
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(d) : "l"(*reinterpret_cast<uint64_t*>(&a)), "l"(*reinterpret_cast<uint64_t*>(&b)), "l"(*reinterpret_cast<uint64_t*>(&c)));
    return *reinterpret_cast<float2*>(&d);
}

// (m, l, acc) of the segments so far with one more: the same few operations wherever segments are merged
struct Merge {
    float before, after;  // factors of the sums so far and of the segment's
    __device__ __forceinline__ Merge(float& m, float& l, float m_seg, float l_seg) {
        const float big = fmaxf(m, m_seg);
        before = m == -INFINITY ? 0.0f : expf(m - big);
        after = m_seg == -INFINITY ? 0.0f : expf(m_seg - big);
        l = fmaf(l, before, l_seg * after);
        m = big;
    }
    __device__ __forceinline__ float operator()(float acc, float seg) const { return fmaf(acc, before, seg * after); }
};
// a row's sums over its denominator, with the sink in it
struct Final {
    float keep = 1.0f, denom;
    __device__ __forceinline__ Final(float m, float l, const float* sinks, int h) : denom(l) {
        if (sinks) {
            const float big = fmaxf(m, sinks[h]);
            keep = m == -INFINITY ? 0.0f : expf(m - big);
            denom = fmaf(l, keep, expf(sinks[h] - big));
        }
    }
    __device__ __forceinline__ float operator()(float acc) const { return denom > 0.0f ? acc * keep / denom : 0.0f; }
};

struct Tiled {
    const float *q, *k_cache, *v_cache, *sinks;
    float *out, *parts;  // parts: [token][head][segment][v_dim + 2], null: the block merges its segments itself
    const int *positions, *row_ids, *block_table;
    int* flag;
    int q_stride, out_stride, max_pages, T, Hq, Hkv, D, page_size, num_pages, window, v_dim, out_head_stride, tokens_a_tile, segments;
    float scale;
};

// DP: D padded to 64, 128 or 256; TM: query rows a thread row
template <int DP, int TM>
__global__ void __launch_bounds__(TILED_THREADS)
paged_attention_tiled_kernel(const Tiled p) {
    constexpr int LD = DP + 4, LS = TILE_KEYS + 4, ROWS = 16 * TM, CG = DP / 64;  // CG: groups of 4 columns of a thread
    extern __shared__ __align__(16) float sm[];
    float* qs = sm;
    float* ks = qs + ROWS * LD;
    float* vs = ks + TILE_KEYS * LD;
    float* ps = vs + TILE_KEYS * LD;
    __shared__ int key_page[2][TILE_KEYS];
    const int t = blockIdx.x, kvh = blockIdx.y, group = p.Hq / p.Hkv;
    const int pos = p.positions[t], row = p.row_ids[t];
    // A tile of tokens begins where a request's begin in this step and at multiples of its size of the position; the other blocks have nothing to do.
    int count = 1;
    if (p.tokens_a_tile > 1) {
        if (t > 0 && pos % p.tokens_a_tile != 0 && p.row_ids[t - 1] == row) return;
        while (t + count < p.T && count < p.tokens_a_tile - pos % p.tokens_a_tile && p.row_ids[t + count] == row) ++count;
    }
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int first = p.window > 0 && pos + 1 > p.window ? pos + 1 - p.window : 0, last = pos + count - 1;
    const int* table = p.block_table + (size_t)row * p.max_pages;
    const int seg_first = first / SEGMENT_KEYS, seg_last = last / SEGMENT_KEYS;
    int tile = first / TILE_KEYS, tile_end = last / TILE_KEYS + 1;
    if (p.parts) {  // one segment of a single token
        const int seg = seg_first + blockIdx.z;
        if (seg > seg_last) return;
        tile = max(tile, seg * (SEGMENT_KEYS / TILE_KEYS));
        tile_end = min(tile_end, (seg + 1) * (SEGMENT_KEYS / TILE_KEYS));
    }
    // where each of a tile's keys lies, -1: none of these rows sees it
    auto look_up = [&](int tile_at) {
        if (tid < TILE_KEYS) {
            const int j = tile_at * TILE_KEYS + tid;
            int page = -1;
            if (j >= first && j <= last) {
                const int index = j / p.page_size;
                page = index < p.max_pages ? table[index] : -1;
                if (page < 0 || page >= p.num_pages) {
                    if (p.flag) atomicOr(p.flag, KB_FLAG_BAD_PAGE);
                    page = -1;
                }
            }
            key_page[tile_at & 1][tid] = page;
        }
    };
    auto fetch = [&](float* dst, const float* cache, int tile_at, int width) {
        for (int i = tid; i < TILE_KEYS * (DP / 4); i += TILED_THREADS) {
            const int key = i / (DP / 4), c = i % (DP / 4) * 4;
            const int page = key_page[tile_at & 1][key];
            const bool live = page >= 0 && c < width;
            const size_t at = live ? (((size_t)page * p.page_size + (tile_at * TILE_KEYS + key) % p.page_size) * p.Hkv + kvh) * p.D + c : 0;
            copy16(dst + key * LD + c, cache + at, live);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    pdl_wait();
    for (int i = tid; i < ROWS * (DP / 4); i += TILED_THREADS) {
        const int r = i / (DP / 4), c = i % (DP / 4) * 4;
        const int token = r / group, h = kvh * group + r % group;
        const bool live = token < count && c < p.D;
        copy16(qs + r * LD + c, live ? p.q + (size_t)(t + token) * p.q_stride + (size_t)h * p.D + c : p.q, live);
    }
    look_up(tile);
    __syncthreads();
    fetch(ks, p.k_cache, tile, p.D);  // the queries' copies are in the same group
    fetch(vs, p.v_cache, tile, p.v_dim);
    float m[TM], l[TM], m_all[TM], l_all[TM];
    float acc[TM][4 * CG], all[TM][4 * CG];
    int low[TM], high[TM];  // the keys a row sees
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        m[i] = m_all[i] = -INFINITY;
        l[i] = l_all[i] = 0.0f;
#pragma unroll
        for (int c = 0; c < 4 * CG; ++c) acc[i][c] = all[i][c] = 0.0f;
        const int token = (ty * TM + i) / group;
        high[i] = token < count ? pos + token : -1;
        low[i] = p.window > 0 && high[i] + 1 > p.window ? high[i] + 1 - p.window : 0;
    }
    for (; tile < tile_end; ++tile) {
        const bool more = tile + 1 < tile_end;
        if (more) look_up(tile + 1);
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();
        // scores: a thread's keys are tx, tx + 16, tx + 32, tx + 48; 32 channels at a time, the even and the odd ones
        // into a sum each, those sums into another
        float s[TM][4];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = 0.0f;
        for (int d0 = 0; d0 < DP; d0 += 32) {
            float2 part[TM][4];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) part[i][j] = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int d = 0; d < 32; d += 4) {
                float4 kv[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) kv[j] = *reinterpret_cast<const float4*>(ks + (tx + 16 * j) * LD + d0 + d);
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const float4 qv = *reinterpret_cast<const float4*>(qs + (ty * TM + i) * LD + d0 + d);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        part[i][j] = fma2(make_float2(qv.x, qv.y), make_float2(kv[j].x, kv[j].y), part[i][j]);
                        part[i][j] = fma2(make_float2(qv.z, qv.w), make_float2(kv[j].z, kv[j].w), part[i][j]);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) s[i][j] += part[i][j].x + part[i][j].y;
        }
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            float big = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = tile * TILE_KEYS + tx + 16 * j;
                const bool seen = key >= low[i] && key <= high[i] && key_page[tile & 1][tx + 16 * j] >= 0;
                s[i][j] = seen ? s[i][j] * p.scale : -INFINITY;
                big = fmaxf(big, s[i][j]);
            }
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, o));
            big = fmaxf(big, m[i]);
            float sum = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float e = s[i][j] == -INFINITY ? 0.0f : expf(s[i][j] - big);
                ps[(ty * TM + i) * LS + tx + 16 * j] = e;
                sum += e;
            }
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            const float alpha = m[i] == -INFINITY ? 0.0f : expf(m[i] - big);
            l[i] = fmaf(l[i], alpha, sum);
            m[i] = big;
#pragma unroll
            for (int c = 0; c < 4 * CG; ++c) acc[i][c] *= alpha;
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();
        if (more) fetch(ks, p.k_cache, tile + 1, p.D);
        // values: a thread's columns are 4 tx .. 4 tx + 3 of every 64
        for (int j0 = 0; j0 < TILE_KEYS; j0 += 4) {
            float4 e[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) e[i] = *reinterpret_cast<const float4*>(ps + (ty * TM + i) * LS + j0);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
#pragma unroll
                for (int c = 0; c < CG; ++c) {
                    const float4 v = *reinterpret_cast<const float4*>(vs + (j0 + j) * LD + c * 64 + tx * 4);
#pragma unroll
                    for (int i = 0; i < TM; ++i) {
                        const float w = j == 0 ? e[i].x : j == 1 ? e[i].y : j == 2 ? e[i].z : e[i].w;
                        const float2 ww = make_float2(w, w);
                        const float2 lo = fma2(ww, make_float2(v.x, v.y), make_float2(acc[i][4 * c], acc[i][4 * c + 1]));
                        const float2 hi = fma2(ww, make_float2(v.z, v.w), make_float2(acc[i][4 * c + 2], acc[i][4 * c + 3]));
                        acc[i][4 * c] = lo.x, acc[i][4 * c + 1] = lo.y, acc[i][4 * c + 2] = hi.x, acc[i][4 * c + 3] = hi.y;
                    }
                }
            }
        }
        if (!p.parts && (tile + 1) % (SEGMENT_KEYS / TILE_KEYS) == 0) {
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const Merge merge(m_all[i], l_all[i], m[i], l[i]);
#pragma unroll
                for (int c = 0; c < 4 * CG; ++c) {
                    all[i][c] = merge(all[i][c], acc[i][c]);
                    acc[i][c] = 0.0f;
                }
                m[i] = -INFINITY;
                l[i] = 0.0f;
            }
        }
        __syncthreads();
        if (more) fetch(vs, p.v_cache, tile + 1, p.v_dim);
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int r = ty * TM + i, token = r / group, h = kvh * group + r % group;
        if (token >= count) continue;
        if (p.parts) {
            float* part = p.parts + (((size_t)t * p.Hq + h) * p.segments + blockIdx.z) * (p.v_dim + 2);
#pragma unroll
            for (int c = 0; c < 4 * CG; ++c) {
                const int e = c / 4 * 64 + tx * 4 + c % 4;
                if (e < p.v_dim) part[e] = acc[i][c];
            }
            if (tx == 0) {
                part[p.v_dim] = m[i];
                part[p.v_dim + 1] = l[i];
            }
            continue;
        }
        const Merge merge(m_all[i], l_all[i], m[i], l[i]);  // what is left of the last segment (nothing, if it was whole)
        const Final final(m_all[i], l_all[i], p.sinks, h);
        float* o = p.out + (size_t)(t + token) * p.out_stride + (size_t)h * p.out_head_stride;
#pragma unroll
        for (int c = 0; c < 4 * CG; ++c) {
            const int e = c / 4 * 64 + tx * 4 + c % 4;
            if (e < p.v_dim) o[e] = final(merge(all[i][c], acc[i][c]));
        }
    }
}

// The segments of single tokens in order: a block a (token, head)
__global__ void __launch_bounds__(128)
paged_attention_tiled_merge_kernel(const Tiled p) {
    const int t = blockIdx.x, h = blockIdx.y;
    const int pos = p.positions[t];
    const int first = p.window > 0 && pos + 1 > p.window ? pos + 1 - p.window : 0;
    const int segments = pos / SEGMENT_KEYS - first / SEGMENT_KEYS + 1;
    pdl_wait();
    const float* part = p.parts + ((size_t)t * p.Hq + h) * p.segments * (p.v_dim + 2);
    for (int e = threadIdx.x; e < p.v_dim; e += blockDim.x) {
        float m = -INFINITY, l = 0.0f, acc = 0.0f;
        for (int s = 0; s < segments; ++s, part += p.v_dim + 2) {
            const Merge merge(m, l, part[p.v_dim], part[p.v_dim + 1]);
            acc = merge(acc, part[e]);
        }
        part -= (size_t)segments * (p.v_dim + 2);
        // a segment that ends at its last key is merged once more with nothing where one block does all
        p.out[(size_t)t * p.out_stride + (size_t)h * p.out_head_stride + e] = Final(m, l, p.sinks, h)(acc);
    }
}

template <int DP, int TM>
int launch_tiled(const Tiled& p, int blocks_z, cudaStream_t stream) {
    constexpr size_t bytes = (size_t)((16 * TM + 2 * TILE_KEYS) * (DP + 4) + 16 * TM * (TILE_KEYS + 4)) * sizeof(float);
    if (cudaError_t e = cudaFuncSetAttribute(paged_attention_tiled_kernel<DP, TM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes)) return (int)e;
    kb_launch(paged_attention_tiled_kernel<DP, TM>, dim3(p.T, p.Hkv, blocks_z), dim3(TILED_THREADS), bytes, stream, p);
    return kb_launch_result();
}

bool tiled_takes(const float* q, int q_stride, const float* k, const float* v, int D, int v_dim, int group) {
    return D % 4 == 0 && v_dim % 4 == 0 && D <= 256 && group <= 64 && q_stride % 4 == 0 && (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v) & 15) == 0;
}

}  // namespace

// Floats of scratch with which a step of `T` single tokens spreads its segments of keys over blocks (0: there is one segment at most, or the sizes go to the
// other kernel); without it a block takes them one behind the other, with the same results.
KB_EXPORT long long kb_paged_attention_generic_scratch(int T, int Hq, int Hkv, int D, int v_dim, int max_positions) {
    const long long segments = (max_positions + SEGMENT_KEYS - 1) / SEGMENT_KEYS;
    if (segments <= 1 || D % 4 || v_dim % 4 || D > 256 || Hkv < 1 || Hq / Hkv > 64) return 0;
    return (long long)T * Hq * segments * (v_dim + 2);
}

KB_EXPORT int kb_paged_attention_generic(const void* q, int q_stride, void* out, int out_stride,
                                         const void* k_cache, const void* v_cache, int is_bf16,
                                         const int* positions, const int* row_ids,
                                         const int* block_table, int max_pages, int T, int Hq,
                                         int Hkv, int D, int page_size, int num_pages, float scale,
                                         int window, const float* sinks, int v_dim, int out_head_stride, int rows, float* scratch,
                                         long long scratch_floats, int* flag, cudaStream_t stream) {
    if (T == 0) return 0;
    if (!q || !out || !k_cache || !v_cache || !positions || !row_ids || !block_table) return KB_ERR_NULL;
    if (D < 1 || D > ATT_MAX_D) return KB_ERR_UNSUPPORTED_SIZE;
    if (v_dim < 1 || v_dim > D || out_head_stride < v_dim) return KB_ERR_BAD_ARG;
    if (Hkv < 1 || Hq % Hkv != 0 || Hq > 65535) return KB_ERR_BAD_ARG;
    const int group = Hq / Hkv;
    if (!is_bf16 && tiled_takes((const float*)q, q_stride, (const float*)k_cache, (const float*)v_cache, D, v_dim, group)) {
        // As many neighbouring tokens a block as make 64 rows with the heads of a key/value head; a step of single tokens (as many tokens as rows of the block
        // table) has none, and where its rows leave SMs idle its segments go to blocks of their own.
        Tiled p{(const float*)q, (const float*)k_cache, (const float*)v_cache, sinks, (float*)out, nullptr, positions, row_ids, block_table, flag, q_stride, out_stride,
                max_pages, T, Hq, Hkv, D, page_size, num_pages, window, v_dim, out_head_stride, 1, (max_pages * page_size + SEGMENT_KEYS - 1) / SEGMENT_KEYS, scale};
        const bool singles = T == rows;
        if (!singles)
            while (2 * p.tokens_a_tile * group <= 64) p.tokens_a_tile *= 2;
        int z = 1;
        if (singles && scratch && p.segments > 1 && (long long)T * Hq * p.segments * (v_dim + 2) <= scratch_floats) {
            p.parts = scratch;
            z = p.segments;
        }
        const bool few = p.tokens_a_tile * group <= 16;
        int code;
        if (D <= 64) code = few ? launch_tiled<64, 1>(p, z, stream) : launch_tiled<64, 4>(p, z, stream);
        else if (D <= 128) code = few ? launch_tiled<128, 1>(p, z, stream) : launch_tiled<128, 4>(p, z, stream);
        else code = few ? launch_tiled<256, 1>(p, z, stream) : launch_tiled<256, 4>(p, z, stream);
        if (code || !p.parts) return code;
        kb_launch(paged_attention_tiled_merge_kernel, dim3(T, Hq), dim3(128), 0, stream, p);
        return kb_launch_result();
    }
    dim3 grid(T, Hq);
    if (is_bf16)
        kb_launch(paged_attention_generic_kernel<__nv_bfloat16>, dim3(grid), dim3(ATT_WARPS * 32), 0, stream, 
            (const __nv_bfloat16*)q, q_stride, (__nv_bfloat16*)out, out_stride,
            (const __nv_bfloat16*)k_cache, (const __nv_bfloat16*)v_cache, positions, row_ids,
            block_table, max_pages, Hq, Hkv, D, page_size, num_pages, scale, window, sinks, v_dim, out_head_stride, flag);
    else
        kb_launch(paged_attention_generic_kernel<float>, dim3(grid), dim3(ATT_WARPS * 32), 0, stream, 
            (const float*)q, q_stride, (float*)out, out_stride, (const float*)k_cache,
            (const float*)v_cache, positions, row_ids, block_table, max_pages, Hq, Hkv, D,
            page_size, num_pages, scale, window, sinks, v_dim, out_head_stride, flag);
    return kb_launch_result();
}
