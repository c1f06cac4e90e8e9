// The matrix-valued recurrences of linear_recurrence.cuh over prompt portions, a chunk of 64 tokens at a time as
// matrix products instead of token by token:
//
//     S_i = g_i S_{i-1} + k_i u_i^T,    o_i = S_i^T q_i
//     DELTA: u_i = beta_i (v_i - (g_i S_{i-1})^T k_i)      !DELTA: u_i = beta_i v_i
//
// With G_ij = g_{j+1} ... g_i (a number, or with CHANNEL a number a key channel; one for i = j) and S the memory before
// the chunk, unrolling gives, for tokens i, j of a chunk,
//
//     u_i = beta_i v_i - beta_i (G_i0 k_i)^T S - sum_{j<i} L_ij u_j,   L_ij = beta_i k_i^T G_ij k_j
//     o_i = (G_i0 q_i)^T S + sum_{j<=i} P_ij u_j,                      P_ij = q_i^T G_ij k_j
//     S'  = G_C0 S + sum_j (G_Cj k_j) u_j^T
//
// so that with (1 + L)^-1 applied once to both right-hand sides, U = U0 - W S, and the chain from chunk to chunk is two
// products.  Two kernels:
//
//   prepare  a block per (chunk, head), all chunks at once: L and P, then W and U0 by forward substitution, a thread two columns
//   walk     a block per (request, head, 16 or 32 columns of S): per chunk Z = [W; q] S, u = U0 - Z, S' and o
//
// All decays enter as running products of the g themselves, never as exponentials of differences of sums, so a decay of
// zero and decays that underflow over a chunk need no care: products that underflow are of terms that are zero.  With CHANNEL
// the pairs of two different 16-token blocks go through the border between them (what is left of k_j at the border, what a
// query keeps since then, both at most one), and pairs within a block are formed one by one.
//
// Precision.  Everything is held in 32-bit.  The products run on mma.sync m16n8k8 (TF32), each factor cut into its leading 11 bits and the next
// 11, three products of the four.  Against 64-bit arithmetic on the same inputs the read-outs are off by 2.0e-7 to 2.5e-7 (relative, 2-norm) with the decays of
// trained layers, where the walk token by token is off by 2.1e-7, and by up to 3.8e-7 where it is off by 1e-7 to 1.6e-7 (decays near zero, keys that repeat);
// the layers' own results, whose packed inputs are 16-bit, are off by the same 3.4e-3 to 4.1e-3 either way.  The 32-bit mode does not come here.
//
// What bounds it.  One request of 16 heads and 128 columns is 128 blocks of the walk kernel, which take their chunks one behind the other: a chunk is
// 458k multiply-adds a block, thrice, on tensor cores that take 490 a cycle and SM (measured), 2,800 cycles, and takes 7,500: the first product 2,850, u and its barrier 500,
// the memory and the read-outs 3,000.  2,048 tokens: 58 us to prepare and 133 to walk, where token by token takes 685 (one decay a head); 245 against
// 648 with a decay a key channel; 231 against 738 without the delta, 64 heads of 64 columns.
#include "umma.cuh"

namespace {

constexpr int C = 64;        // tokens a chunk
constexpr int LP = C + 4;    // row stride of a C x C tile in shared memory: fragment loads touch every bank once
constexpr int TILE = 128;    // floats of a fragment tile: 16 x 8 of a first factor, four a lane

// x = hi + lo and less than 2^-23 of x: hi has 11 significant bits (rounded, ties away from zero), lo at most 12, of which the tensor cores, which
// pass over the last 13 bits of a TF32 factor, take the first 11.  By integer operations: the conversion instruction runs at a
// sixteenth of their rate.  A NaN stays one in lo.
__device__ __forceinline__ void split(float x, uint32_t& hi, uint32_t& lo) {
    hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
    lo = __float_as_uint(x - __uint_as_float(hi));
}

__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_fresh(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
}

// A 16 x 8 sum of products.  The tensor cores cut an accumulator's last bits off instead of rounding it, eight terms at a time; so the
// large terms' eight start from zero and are added by a rounding 32-bit sum, and the small ones have accumulators of their own.
struct Sum {
    float main[4] = {0.0f, 0.0f, 0.0f, 0.0f}, first[4] = {0.0f, 0.0f, 0.0f, 0.0f}, second[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    __device__ __forceinline__ void add(const uint32_t (&ah)[4], const uint32_t (&al)[4], uint32_t bh0, uint32_t bh1, uint32_t bl0, uint32_t bl1) {
        float eight[4];
        mma_fresh(eight, ah, bh0, bh1);
        mma(first, al, bh0, bh1);
        mma(second, ah, bl0, bl1);
#pragma unroll
        for (int e = 0; e < 4; ++e) main[e] += eight[e];
    }
    __device__ __forceinline__ float at(int e) const { return main[e] + (first[e] + second[e]); }
};

// The fragment of a 16 x 8 tile of a first factor: rows g and g + 8, columns t and t + 4 of a lane (g = lane / 4, t = lane % 4).
__device__ __forceinline__ void load_a(const float* src, int stride, uint32_t (&hi)[4], uint32_t (&lo)[4]) {
    const int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
    split(src[g * stride + t], hi[0], lo[0]);
    split(src[(g + 8) * stride + t], hi[1], lo[1]);
    split(src[g * stride + t + 4], hi[2], lo[2]);
    split(src[(g + 8) * stride + t + 4], hi[3], lo[3]);
}
// ... from a tile that stands as it is loaded, four floats a lane, columns t and t + 4 times a factor each
__device__ __forceinline__ void load_tile(const float* tile, uint32_t (&hi)[4], uint32_t (&lo)[4], float f0 = 1.0f, float f1 = 1.0f) {
    const float4 a = *reinterpret_cast<const float4*>(tile + (threadIdx.x & 31) * 4);
    split(a.x * f0, hi[0], lo[0]);
    split(a.y * f0, hi[1], lo[1]);
    split(a.z * f1, hi[2], lo[2]);
    split(a.w * f1, hi[3], lo[3]);
}

// A second factor's 8 x 8 tile in shared memory: a lane's two elements (k = t and t + 4 of column g), leading and further bits of each.
__device__ __forceinline__ void put_b(float* tiles, int ksteps, int k, int n, float x) {
    uint32_t hi, lo;
    split(x, hi, lo);
    float* at = tiles + ((n >> 3) * ksteps + (k >> 3)) * TILE + ((n & 7) * 4 + (k & 3)) * 4 + ((k >> 2) & 1) * 2;
    *reinterpret_cast<float2*>(at) = make_float2(__uint_as_float(hi), __uint_as_float(lo));
}
__device__ __forceinline__ void add_b(Sum& sum, const uint32_t (&ah)[4], const uint32_t (&al)[4], const float* tile) {
    const uint4 b = *reinterpret_cast<const uint4*>(tile + (threadIdx.x & 31) * 4);
    sum.add(ah, al, b.x, b.z, b.y, b.w);
}

__device__ __forceinline__ void copy16(float* dst, const float* src, bool live) {
    const int bytes = live ? 16 : 0;  // the rest is filled with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_addr(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// `all` rows of W floats (a multiple of 4, at most LD), `src_stride` apart, into rows of LD floats; what lies behind `rows` or `width` is zero
template <int THREADS>
__device__ __forceinline__ void copy_rows(float* dst, int ld, const float* src, size_t src_stride, int rows, int all, int width, int W) {
    const int per = W / 4;
    for (int i = threadIdx.x; i < all * per; i += THREADS) {
        const int r = i / per, c = (i % per) * 4;
        const bool live = r < rows && c < width;
        copy16(dst + r * ld + c, live ? src + (size_t)r * src_stride + c : src, live);
    }
}
// a run of `floats` (a multiple of 4) as it stands, by the copy engine, its bytes counted on `bar`; one thread's work
__device__ __forceinline__ void copy_run(float* dst, const float* src, int floats, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(smem_addr(dst)), "l"(src), "r"(floats * 4),
                 "r"(smem_addr(bar))
                 : "memory");
}

__host__ __device__ inline int chunks_of(int tokens) { return (tokens + C - 1) / C; }

// What the prepare kernel leaves in the scratch, in floats.  Factors stand tile by tile as the walk's fragments take them.  Keys and queries are the
// same for the H / KH heads that share them unless each head has decays a key channel, which are then multiplied in.
struct Layout {
    int p, w, u, from_start, total, head;  // a (chunk, head): P, W, U0, [G_i0 | beta | G_Cj] a token, G_C0, its size
    int q, k, shared;                      // a (chunk, key head) (CHANNEL: head): queries, keys, their size
    __host__ __device__ Layout(bool delta, bool channel, int DP, int V) {
        const int VP = (V + 7) / 8 * 8;
        int at = 0;
        p = at, at += C * C;
        w = at, at += delta ? C * DP : 0;
        u = at, at += delta ? C * VP : 0;
        from_start = at, at += 3 * C;
        total = at, at += channel ? DP : 4;
        head = at;
        q = 0, k = C * DP, shared = 2 * C * DP;
    }
};
struct Scratch {
    float* heads;   // [chunk][head of the group][Layout::head]
    float* shared;  // [chunk][key head of the group (CHANNEL: head)][Layout::shared]
};
__device__ __forceinline__ const float* tile_at(const float* tiles, int ksteps, int rt, int ks) { return tiles + (rt * ksteps + ks) * TILE; }

// The row that chunk `chunk` of the step belongs to (rows' chunks side by side, in order): by warp 0, told to the block.
struct Where {
    int row, first, n;  // its first token and how many it has; row < 0: there is no such chunk
};
__device__ __forceinline__ void find_chunk(const int* __restrict__ qo_indptr, int rows, int chunk, Where* where) {
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        if (lane == 0) where->row = -1;
        __syncwarp();
        int base = 0;
        for (int r0 = 0; r0 < rows; r0 += 32) {
            const int r = r0 + lane;
            const int begin = r < rows ? qo_indptr[r] : 0, end = r < rows ? qo_indptr[r + 1] : 0;
            const int count = chunks_of(end - begin);
            int upto = count;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int other = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += other;
            }
            const int place = chunk - (base + upto - count);  // which of the row's chunks it is
            if (place >= 0 && place < count) {
                where->row = r;
                where->first = begin + place * C;
                where->n = min(C, end - where->first);
            }
            base += __shfl_sync(0xffffffffu, upto, 31);
            if (chunk < base) break;
        }
    }
    __syncthreads();
}

// x_i = rhs_i - sum_{j<i} L_ij x_j for two neighbouring columns of a tile (rows of LD), in place; L by columns (lt[j * LP + i]).  Two columns, because
// what bounds it is handing every thread the L it shares with all others.  Sixteen rows at a time, so that the code stays small: with all
// 64 rows in registers it is 2,500 instructions that every block fetches, and the kernel took 1.7 times as long.
__device__ __forceinline__ void substitute(float* columns, int LD, const float* __restrict__ lt) {
    auto take = [](float2& x, float l, float2 known) {
        x.x = fmaf(-l, known.x, x.x);
        x.y = fmaf(-l, known.y, x.y);
    };
#pragma unroll 1
    for (int i0 = 0; i0 < C; i0 += 16) {
        float2 x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = *reinterpret_cast<const float2*>(columns + (i0 + i) * LD);
#pragma unroll 1
        for (int j0 = 0; j0 < i0; j0 += 8) {
            float2 known[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) known[j] = *reinterpret_cast<const float2*>(columns + (j0 + j) * LD);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
#pragma unroll
                for (int i = 0; i < 16; i += 4) {
                    const float4 l = *reinterpret_cast<const float4*>(lt + (j0 + j) * LP + i0 + i);
                    take(x[i], l.x, known[j]);
                    take(x[i + 1], l.y, known[j]);
                    take(x[i + 2], l.z, known[j]);
                    take(x[i + 3], l.w, known[j]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 15; ++j) {
#pragma unroll
            for (int i4 = (j + 1) / 4 * 4; i4 < 16; i4 += 4) {
                const float4 l = *reinterpret_cast<const float4*>(lt + (i0 + j) * LP + i0 + i4);
                if (i4 + 0 > j) take(x[i4 + 0], l.x, x[j]);
                if (i4 + 1 > j) take(x[i4 + 1], l.y, x[j]);
                if (i4 + 2 > j) take(x[i4 + 2], l.z, x[j]);
                if (i4 + 3 > j) take(x[i4 + 3], l.w, x[j]);
            }
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) *reinterpret_cast<float2*>(columns + (i0 + i) * LD) = x[i];
    }
}

// A matrix in shared memory (rows of LD; TRANSPOSED: its columns are the rows here) written tile by tile as first-factor fragments
template <int THREADS, bool TRANSPOSED>
__device__ __forceinline__ void put_tiles(float* __restrict__ dst, const float* src, int LD, int row_tiles, int ksteps) {
    for (int i = threadIdx.x; i < row_tiles * ksteps * 32; i += THREADS) {
        const int lane = i & 31, tile = i >> 5;
        const int r = tile / ksteps * 16 + (lane >> 2), c = tile % ksteps * 8 + (lane & 3);
        auto get = [&](int rr, int cc) { return TRANSPOSED ? src[cc * LD + rr] : src[rr * LD + cc]; };
        *reinterpret_cast<float4*>(dst + i * 4) = make_float4(get(r, c), get(r + 8, c), get(r, c + 4), get(r + 8, c + 4));
    }
}

// Both right-hand sides through (1 + L)^-1, a thread two columns, and out to the scratch: W in place of the keys `ks` (which hold its right-hand side
// but for beta, and with `ga` for G_i0 a token), U0 in `us` (DP columns at a time).
template <int THREADS, int DP>
__device__ __forceinline__ void solve(const float* lt, float* ks, float* us, int LD, const float* bs, const float* ga, const float* __restrict__ vv, size_t v_stride,
                                      int n, int V, float* __restrict__ w, float* __restrict__ u) {
    const int VP = (V + 7) / 8 * 8;
    for (int c0 = 0; c0 < VP; c0 += DP) {
        const int width = min(DP, V - c0), padded = min(DP, VP - c0);
        for (int i = threadIdx.x; i < C * DP / 4; i += THREADS) {  // V is a multiple of 4
            const int r = i / (DP / 4), c = i % (DP / 4) * 4;
            float4 v4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (r < n && c < width) v4 = *reinterpret_cast<const float4*>(vv + (size_t)r * v_stride + c0 + c);
            const float b = bs[r];
            *reinterpret_cast<float4*>(us + r * LD + c) = make_float4(b * v4.x, b * v4.y, b * v4.z, b * v4.w);
        }
        if (c0 == 0)
            for (int i = threadIdx.x; i < C * DP; i += THREADS) ks[i / DP * LD + i % DP] *= bs[i / DP] * (ga ? ga[i / DP] : 1.0f);
        __syncthreads();
        for (int col = 2 * threadIdx.x + (c0 == 0 ? 0 : DP); col < DP + padded; col += 2 * THREADS) substitute(col < DP ? ks + col : us + (col - DP), LD, lt);
        __syncthreads();
        if (c0 == 0) put_tiles<THREADS, false>(w, ks, LD, C / 16, DP / 8);
        // U0 as the walk's sums stand: tiles of 16 x 8, column tile by column tile, a lane's (g, 2t), (g, 2t + 1), (g + 8, 2t), (g + 8, 2t + 1)
        for (int i = threadIdx.x; i < padded / 8 * (C / 16) * 32; i += THREADS) {
            const int lane = i & 31, tile = i >> 5;
            const float* at = us + (tile % (C / 16) * 16 + (lane >> 2)) * LD + tile / (C / 16) * 8 + 2 * (lane & 3);
            *reinterpret_cast<float4*>(u + (size_t)c0 / 8 * (C / 16) * TILE + i * 4) = make_float4(at[0], at[1], at[8 * LD], at[8 * LD + 1]);
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------ prepare, one decay a head

constexpr int PREPARE = 256;

// blockIdx.x: chunk, blockIdx.y: HB heads that share their keys and queries (DELTA: one head; else L and P differ by their decays alone)
template <int DP, bool DELTA>
__global__ void __launch_bounds__(PREPARE, 2)
prepare_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ vv, const float* __restrict__ beta,
               const float* __restrict__ decay, const int* __restrict__ qo_indptr, int rows, int KH, int D, int H, int V, int head0, int heads, int HB,
               Scratch scratch) {
    constexpr int LD = DP + 4;
    extern __shared__ __align__(128) float sm[];
    float* ks = sm;                  // [C][LD]
    float* qs = ks + C * LD;         // queries, later U0
    float* qk = qs + C * LD;         // [i][j] of q_i.k_j
    float* kk = qk + C * LP;         // DELTA: [j][i] of k_i.k_j, then L by columns
    float* gs = kk + (DELTA ? C * LP : 0);
    float* bs = gs + C;
    float* ga = bs + C;              // G_i0
    float* gb = ga + C;              // G_Cj
    float* suffix = gb + C;          // what is left of a key at the end of its block of 16
    float* pb = suffix + C;          // a block's whole product
    __shared__ Where where;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    find_chunk(qo_indptr, rows, blockIdx.x, &where);
    pdl_wait();
    if (where.row < 0) return;
    const int t0 = where.first, n = where.n;
    const int first_head = head0 + blockIdx.y * HB;
    const int sharing = H / KH, kh = first_head / sharing;
    const size_t stride = (size_t)KH * D;
    copy_rows<PREPARE>(ks, LD, kn + (size_t)t0 * stride + (size_t)kh * D, stride, n, C, D, DP);
    copy_rows<PREPARE>(qs, LD, qn + (size_t)t0 * stride + (size_t)kh * D, stride, n, C, D, DP);
    copies_commit();
    copies_wait();
    __syncthreads();
    {   // Sixteen rows of queries (DELTA: or of keys) against the keys up to their own diagonal, up to four column tiles at a time: units (rows, first tile,
        // tiles) = (0,0,2) (1,0,4) (2,0,4) (2,4,2) (3,0,4) (3,4,4).  DELTA: four warps a matrix, the first two with two units each.
        const int g = lane >> 2, t = lane & 3;
        const bool queries = !DELTA || warp >= 4;
        int unit = DELTA ? (warp & 3) == 0 ? 1 : (warp & 3) == 1 ? 2 : (warp & 3) + 2 : warp;
        int next = DELTA ? (warp & 3) == 0 ? 0 : (warp & 3) == 1 ? 3 : 6 : 6;
        while (unit < 6) {
            const int mt = unit < 2 ? unit : unit / 2 + 1, first = unit == 3 || unit == 5 ? 4 : 0;
            const int tiles = unit == 0 || unit == 3 ? 2 : 4;
            const float* a = (queries ? qs : ks) + mt * 16 * LD;
            Sum sum[4];
#pragma unroll 2
            for (int k0 = 0; k0 < DP; k0 += 8) {
                uint32_t ah[4], al[4];
                load_a(a + k0, LD, ah, al);
#pragma unroll
                for (int nt = 0; nt < 4; ++nt) {
                    if (nt < tiles) {
                        const float* b = ks + ((first + nt) * 8 + g) * LD + k0 + t;
                        uint32_t bh0, bl0, bh1, bl1;
                        split(b[0], bh0, bl0);
                        split(b[4], bh1, bl1);
                        sum[nt].add(ah, al, bh0, bh1, bl0, bl1);
                    }
                }
            }
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                if (nt < tiles) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int i = mt * 16 + g + (e >> 1) * 8, j = (first + nt) * 8 + 2 * t + (e & 1);
                        if (queries) qk[i * LP + j] = sum[nt].at(e);
                        else kk[j * LP + i] = sum[nt].at(e);
                    }
                }
            }
            unit = next;
            next = 6;
        }
    }
    const Layout at(DELTA, false, DP, V);
    if (first_head % sharing == 0) {
        float* shared = scratch.shared + ((size_t)blockIdx.x * (heads / sharing) + (first_head - head0) / sharing) * at.shared;
        put_tiles<PREPARE, false>(shared + at.q, qs, LD, C / 16, DP / 8);
        put_tiles<PREPARE, true>(shared + at.k, ks, LD, DP / 16, C / 8);
    }
    for (int hb = 0; hb < HB; ++hb) {
        const int h = first_head + hb;
        float* mine = scratch.heads + ((size_t)blockIdx.x * heads + (h - head0)) * at.head;
        __syncthreads();
        if (threadIdx.x < C) {
            const bool live = threadIdx.x < n;
            gs[threadIdx.x] = live ? decay[(size_t)(t0 + threadIdx.x) * H + h] : 1.0f;
            bs[threadIdx.x] = live ? beta[(size_t)(t0 + threadIdx.x) * H + h] : 0.0f;
        }
        __syncthreads();
        if (warp < 2) {
            // products from the chunk's start through each token, and from behind each token to the chunk's end: scans of 64 numbers, a warp each
            const bool forward = warp == 0;
            const float a = forward ? gs[2 * lane] : gs[C - 1 - 2 * lane], b = forward ? gs[2 * lane + 1] : gs[C - 2 - 2 * lane];
            float upto = a * b;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float other = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto *= other;
            }
            float before = __shfl_up_sync(0xffffffffu, upto, 1);
            if (lane == 0) before = 1.0f;
            if (forward) {
                ga[2 * lane] = before * a;
                ga[2 * lane + 1] = upto;
                if (lane == 31) mine[at.total] = upto;
            } else {
                gb[C - 1 - 2 * lane] = before;
                gb[C - 2 - 2 * lane] = before * a;
            }
        } else if (warp < 4) {
            const int j = threadIdx.x - 64;
            float run = 1.0f;
            for (int i = j + 1; i < (j | 15) + 1; ++i) run *= gs[i];
            suffix[j] = run;
            if ((j & 15) == 0) pb[j >> 4] = run * gs[j];
        }
        __syncthreads();
        // G_ij a pair, by a running product: thread (j, quarter) goes down its sixteen i.  P goes out tile by tile as fragments; L stays, by columns.
        {
            const int j = threadIdx.x & (C - 1), quarter = threadIdx.x >> 6;
            float run = j >> 4 < quarter ? suffix[j] : 1.0f;
            for (int block = (j >> 4) + 1; block < quarter; ++block) run *= pb[block];
            float* tile = mine + at.p + (quarter * (C / 8) + (j >> 3)) * TILE + (j & 3) * 4 + ((j >> 2) & 1) * 2;
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                const int i = quarter * 16 + r;
                if (i > j) run *= gs[i];
                tile[(r & 7) * 16 + (r >> 3)] = i >= j ? run * qk[i * LP + j] : 0.0f;
                if (DELTA) kk[j * LP + i] = i > j ? bs[i] * run * kk[j * LP + i] : 0.0f;
            }
        }
        if (threadIdx.x < C) {
            mine[at.from_start + threadIdx.x] = ga[threadIdx.x];
            mine[at.from_start + C + threadIdx.x] = bs[threadIdx.x];
            mine[at.from_start + 2 * C + threadIdx.x] = gb[threadIdx.x];
        }
        if constexpr (DELTA)  // begins behind a barrier of its own
            solve<PREPARE, DP>(kk, ks, qs, LD, bs, ga, vv + ((size_t)t0 * H + h) * V, (size_t)H * V, n, V, mine + at.w, mine + at.u);
    }
}

// ------------------------------------------------------------------ prepare, one decay a head and key channel (with the delta)

constexpr int PREPARE_CHANNEL = 512;

template <int DP>
__global__ void __launch_bounds__(PREPARE_CHANNEL)
prepare_channel_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ vv, const float* __restrict__ beta,
                       const float* __restrict__ decay, const int* __restrict__ qo_indptr, int rows, int KH, int D, int H, int V, int head0, int heads,
                       Scratch scratch) {
    constexpr int T = PREPARE_CHANNEL;
    constexpr int LD = DP + 4;
    constexpr int B = 16, NB = C / B;  // the chunk's blocks
    constexpr int SLABS = T / C;       // threads that share a key
    extern __shared__ __align__(128) float sm[];
    float* ks = sm;               // keys, then times what is kept from their block's start through their token, in the end W's right-hand side
    float* qs = ks + C * LD;      // queries, the same way
    float* gs = qs + C * LD;      // decays, in the end U0
    float* kb = gs + C * LD;      // keys times what is left of them at the border in front of the block at hand
    float* qk = kb + C * LD;      // [i][j]
    float* lt = qk + C * LP;      // [j][i]
    float* pb = lt + C * LP;      // [NB][DP] a block's whole product
    float* bs = pb + NB * DP;
    __shared__ Where where;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    find_chunk(qo_indptr, rows, blockIdx.x, &where);
    pdl_wait();
    if (where.row < 0) return;
    const int t0 = where.first, n = where.n;
    const int h = head0 + blockIdx.y;
    const int kh = h / (H / KH);
    const size_t stride = (size_t)KH * D;
    copy_rows<T>(ks, LD, kn + (size_t)t0 * stride + (size_t)kh * D, stride, n, C, D, DP);
    copy_rows<T>(qs, LD, qn + (size_t)t0 * stride + (size_t)kh * D, stride, n, C, D, DP);
    copy_rows<T>(gs, LD, decay + ((size_t)t0 * H + h) * D, (size_t)H * D, n, C, D, DP);
    copies_commit();
    if (threadIdx.x < C) bs[threadIdx.x] = threadIdx.x < n ? beta[(size_t)(t0 + threadIdx.x) * H + h] : 0.0f;
    for (int i = threadIdx.x; i < C * LP; i += T) qk[i] = lt[i] = 0.0f;
    copies_wait();
    __syncthreads();
    for (int i = n * DP + threadIdx.x; i < C * DP; i += T) gs[(i / DP) * LD + i % DP] = 1.0f;  // no token: nothing decays
    __syncthreads();
    {   // pairs within a block: SLABS threads a key, each with every SLABS-th group of four channels, down the block's tokens
        const int j = threadIdx.x / SLABS, slab = threadIdx.x % SLABS;
        const int i0 = j / B * B;
        constexpr int GROUPS = DP / 4 / SLABS;
        float x[4 * GROUPS];
#pragma unroll
        for (int m = 0; m < 4 * GROUPS; ++m) x[m] = 0.0f;
#pragma unroll 2
        for (int i = i0; i < i0 + B; ++i) {
            float sk = 0.0f, sq = 0.0f;
#pragma unroll
            for (int m = 0; m < GROUPS; ++m) {
                const int d = 4 * (slab + SLABS * m);
                const float4 k4 = *reinterpret_cast<const float4*>(ks + i * LD + d);
                const float4 q4 = *reinterpret_cast<const float4*>(qs + i * LD + d);
                const float4 g4 = *reinterpret_cast<const float4*>(gs + i * LD + d);
                const float kv[4] = {k4.x, k4.y, k4.z, k4.w}, qv[4] = {q4.x, q4.y, q4.z, q4.w}, gv[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float& at = x[4 * m + e];
                    at = i == j ? kv[e] : at * gv[e];  // zero until the key's own token
                    sk = fmaf(kv[e], at, sk);
                    sq = fmaf(qv[e], at, sq);
                }
            }
#pragma unroll
            for (int o = 1; o < SLABS; o <<= 1) {
                sk += __shfl_xor_sync(0xffffffffu, sk, o);
                sq += __shfl_xor_sync(0xffffffffu, sq, o);
            }
            if (slab == 0) {
                qk[i * LP + j] = sq;
                lt[j * LP + i] = i > j ? sk : 0.0f;
            }
        }
    }
    __syncthreads();
    for (int task = threadIdx.x; task < NB * DP; task += T) {
        const int d = task % DP, i0 = task / DP * B;
        float run = 1.0f;
#pragma unroll
        for (int i = i0 + B - 1; i >= i0; --i) {
            kb[i * LD + d] = ks[i * LD + d] * run;
            run *= gs[i * LD + d];
        }
        run = 1.0f;
#pragma unroll
        for (int i = i0; i < i0 + B; ++i) {
            run *= gs[i * LD + d];
            ks[i * LD + d] *= run;
            qs[i * LD + d] *= run;
        }
        pb[task] = run;
    }
    __syncthreads();
    for (int block = 1; block < NB; ++block) {
        // 16 tokens of this block, as keys and as queries, against every key before it; a warp a tile of 16 x 8
        const int g = lane >> 2, t = lane & 3;
        for (int tile = warp; tile < 4 * block; tile += T / 32) {
            const bool queries = tile & 1;
            const int nt = tile >> 1;
            Sum sum;
            const float* a = (queries ? qs : ks) + block * B * LD;
            const float* b = kb + (nt * 8 + g) * LD + t;
#pragma unroll 4
            for (int k0 = 0; k0 < DP; k0 += 8) {
                uint32_t ah[4], al[4], bh0, bl0, bh1, bl1;
                load_a(a + k0, LD, ah, al);
                split(b[k0], bh0, bl0);
                split(b[k0 + 4], bh1, bl1);
                sum.add(ah, al, bh0, bh1, bl0, bl1);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = block * B + g + (e >> 1) * 8, j = nt * 8 + 2 * t + (e & 1);
                if (queries) qk[i * LP + j] = sum.at(e);
                else lt[j * LP + i] = sum.at(e);
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < block * B * DP; i += T) kb[(i / DP) * LD + i % DP] *= pb[block * DP + i % DP];
        __syncthreads();
    }
    const Layout at(true, true, DP, V);
    float* mine = scratch.heads + ((size_t)blockIdx.x * heads + blockIdx.y) * at.head;
    float* shared = scratch.shared + ((size_t)blockIdx.x * heads + blockIdx.y) * at.shared;
    for (int i = threadIdx.x; i < C * DP; i += T) {
        const int r = i / DP, d = i % DP;
        float before = 1.0f;  // what the blocks in front of the token's keep
        for (int block = 0; block < r / B; ++block) before *= pb[block * DP + d];
        ks[r * LD + d] *= before;
        qs[r * LD + d] *= before;
        if (r == 0) {
            float all = 1.0f;
            for (int block = 0; block < NB; ++block) all *= pb[block * DP + d];
            mine[at.total + d] = all;
        }
    }
    for (int i = threadIdx.x; i < C * C; i += T) lt[i / C * LP + i % C] *= bs[i % C];
    __syncthreads();
    put_tiles<T, false>(mine + at.p, qk, LP, C / 16, C / 8);
    put_tiles<T, false>(shared + at.q, qs, LD, C / 16, DP / 8);
    put_tiles<T, true>(shared + at.k, kb, LD, DP / 16, C / 8);
    solve<T, DP>(lt, ks, gs, LD, bs, nullptr, vv + ((size_t)t0 * H + h) * V, (size_t)H * V, n, V, mine + at.w, mine + at.u);
}

// ------------------------------------------------------------------ the walk over chunks

constexpr int WALK = 256;

template <int DP, int NT, bool DELTA, bool CHANNEL>
struct WalkShared {
    static constexpr int N = 8 * NT;
    static constexpr int wq = 0;                           // tiles of W (DELTA), tiles of q
    static constexpr int k = wq + (DELTA ? 2 : 1) * C * DP;
    static constexpr int p = k + C * DP;
    static constexpr int v = p + C * C;                    // tiles of U0; !DELTA: values, rows of N
    static constexpr int s = v + C * N;
    static constexpr int u = s + 2 * N * DP;
    static constexpr int ga = u + 2 * N * C;
    static constexpr int gb = ga + 2 * C;                  // G_i0, beta; then G_Cj, G_C0
    static constexpr int gt = gb + C;
    static constexpr int floats = gt + (CHANNEL ? DP : 4);
};

// grid: (request, head of the group, columns / N).  Eight warps: a warp has sixteen tokens and half of the column tiles in the first product, both for W and for
// q, and in the read-outs; and sixteen key channels of the memory.  The factors come in by bulk copies that one thread asks for (as 16-byte
// copies by all threads, asking took two fifths of a chunk's time): what the first product reads while the second runs, and the other way round.
template <int DP, int NT, bool DELTA, bool CHANNEL>
__global__ void __launch_bounds__(WALK, NT == 2 && !DELTA ? 2 : 1)
walk_kernel(const float* __restrict__ vv, Scratch scratch, float* __restrict__ states, const int* __restrict__ qo_indptr, const int* __restrict__ state_slots, int KH,
            int D, int H, int V, int head0, int heads, float* __restrict__ out, int* flag) {
    using Sh = WalkShared<DP, NT, DELTA, CHANNEL>;
    constexpr int N = Sh::N, KS = DP / 8, CS = C / 8;
    extern __shared__ __align__(128) float sm[];
    __shared__ int before_shared, abort_word;
    __shared__ __align__(8) uint64_t first_full, second_full;
    const int row = blockIdx.x, h = head0 + blockIdx.y, col0 = blockIdx.z * N;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int begin = qo_indptr[row], end = qo_indptr[row + 1];
    if (warp == 0) {  // how many chunks the rows before this one have
        int count = 0;
        for (int r = lane; r < row; r += 32) count += chunks_of(qo_indptr[r + 1] - qo_indptr[r]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) count += __shfl_xor_sync(0xffffffffu, count, o);
        if (lane == 0) {
            before_shared = count;
            abort_word = 0;
            mbar_init(&first_full, 1);
            mbar_init(&second_full, 1);
            fence_proxy_async_smem();
        }
    }
    float* Sg = states + ((size_t)state_slots[row] * H + h) * V * D;
    __syncthreads();
    const Layout at(DELTA, CHANNEL, DP, V);
    const int sharing = CHANNEL ? 1 : H / KH;
    const int VT = (V + 7) / 8;  // column tiles there are
    const int chunks = chunks_of(end - begin);
    const size_t first_chunk = before_shared;
    pdl_wait();

    auto mine_of = [&](int chunk) { return scratch.heads + ((first_chunk + chunk) * heads + blockIdx.y) * at.head; };
    auto shared_of = [&](int chunk) { return scratch.shared + ((first_chunk + chunk) * (heads / sharing) + blockIdx.y / sharing) * at.shared; };
    // By warp 0: W, q, U0 or the values, the decays and betas.
    auto fetch_first = [&](int chunk) {
        const float* mine = mine_of(chunk);
        const int t0 = begin + chunk * C, n = min(C, end - t0), width = min(N, V - col0);
        const int u_floats = DELTA ? min(NT, VT - col0 / 8) * (C / 16) * TILE : 0;
        if (lane == 0) {
            mbar_arrive_expect_tx(&first_full, 4 * ((DELTA ? 2 : 1) * C * DP + (DELTA ? u_floats : n * width) + (CHANNEL ? 0 : 2 * C)));
            if (DELTA) copy_run(sm + Sh::wq, mine + at.w, C * DP, &first_full);
            copy_run(sm + Sh::wq + (DELTA ? C * DP : 0), shared_of(chunk) + at.q, C * DP, &first_full);
            if (DELTA) copy_run(sm + Sh::v, mine + at.u + (size_t)col0 / 8 * (C / 16) * TILE, u_floats, &first_full);
            if (!CHANNEL) copy_run(sm + Sh::ga, mine + at.from_start, 2 * C, &first_full);
        }
        if (!DELTA) {
            __syncwarp();
            for (int i = lane; i < n; i += 32) copy_run(sm + Sh::v + i * N, vv + ((size_t)(t0 + i) * H + h) * V + col0, width, &first_full);
        }
    };
    // k, P, what is left of a key and what the memory keeps at the chunk's end
    auto fetch_second = [&](int chunk) {
        const float* mine = mine_of(chunk);
        if (lane == 0) {
            mbar_arrive_expect_tx(&second_full, 4 * (C * DP + C * C + (CHANNEL ? DP : C + 4)));
            copy_run(sm + Sh::k, shared_of(chunk) + at.k, C * DP, &second_full);
            copy_run(sm + Sh::p, mine + at.p, C * C, &second_full);
            if (CHANNEL) copy_run(sm + Sh::gt, mine + at.total, DP, &second_full);
            else copy_run(sm + Sh::gb, mine + at.from_start + 2 * C, C + 4, &second_full);
        }
    };
    if (warp == 0 && chunks > 0) {
        fetch_first(0);
        fetch_second(0);
    }
    constexpr int NW = NT / 2;                       // column tiles of a warp in the first product and the read-outs
    const int rt = warp & 3, nt0 = (warp >> 2) * NW;  // which sixteen tokens, and its first column tile
    // The memory: a warp holds sixteen key channels of all column tiles as sums stand, and its leading and further bits are in shared memory
    // as the second factor of the next chunk's first product.
    const bool owner = warp < DP / 16;
    float S[NT][4];
    auto publish = [&]() {
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) put_b(sm + Sh::s, KS, warp * 16 + g + (e >> 1) * 8, j * 8 + 2 * t + (e & 1), S[j][e]);
    };
    if (owner) {
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int d = warp * 16 + g + (e >> 1) * 8, c = col0 + j * 8 + 2 * t + (e & 1);
                S[j][e] = d < D && c < V ? Sg[(size_t)c * D + d] : 0.0f;
            }
        publish();
    }
    bool lost = false;  // a copy did not come within the wait's limit
    int chunk = 0;
    for (; chunk < chunks; ++chunk) {
        const int t0 = begin + chunk * C, n = min(C, end - t0);
        lost = __syncthreads_or(!mbar_wait(&first_full, chunk & 1, &abort_word));
        if (lost) break;
        Sum zw[NW], zq[NW];
#pragma unroll 4
        for (int ks = 0; ks < KS; ++ks) {
            uint32_t ah[4], al[4];
            if (DELTA) {
                load_tile(tile_at(sm + Sh::wq, KS, rt, ks), ah, al);
#pragma unroll
                for (int j = 0; j < NW; ++j) add_b(zw[j], ah, al, tile_at(sm + Sh::s, KS, nt0 + j, ks));
            }
            load_tile(tile_at(sm + Sh::wq + (DELTA ? C * DP : 0), KS, rt, ks), ah, al);
#pragma unroll
            for (int j = 0; j < NW; ++j) add_b(zq[j], ah, al, tile_at(sm + Sh::s, KS, nt0 + j, ks));
        }
        const int i0 = rt * 16 + g;
        const float keep[2] = {CHANNEL ? 1.0f : sm[Sh::ga + i0], CHANNEL ? 1.0f : sm[Sh::ga + i0 + 8]};
#pragma unroll
        for (int j = 0; j < NW; ++j) {
            float u[4];
            if (DELTA) {
                const float4 u0 = *reinterpret_cast<const float4*>(sm + Sh::v + ((nt0 + j) * (C / 16) + rt) * TILE + lane * 4);
                u[0] = u0.x - zw[j].at(0), u[1] = u0.y - zw[j].at(1), u[2] = u0.z - zw[j].at(2), u[3] = u0.w - zw[j].at(3);
            } else {
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const float2 v2 = *reinterpret_cast<const float2*>(sm + Sh::v + (i0 + 8 * half) * N + (nt0 + j) * 8 + 2 * t);
                    const float b = sm[Sh::ga + C + i0 + 8 * half];
                    const bool live = i0 + 8 * half < n;  // a row behind the last token holds what was there before
                    u[2 * half] = live ? b * v2.x : 0.0f;
                    u[2 * half + 1] = live ? b * v2.y : 0.0f;
                }
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = i0 + (e >> 1) * 8, c = (nt0 + j) * 8 + 2 * t + (e & 1);
                put_b(sm + Sh::u, CS, i, c, u[e]);
            }
        }
        lost = __syncthreads_or(!mbar_wait(&second_full, chunk & 1, &abort_word));
        if (lost) break;
        if (warp == 0 && chunk + 1 < chunks) fetch_first(chunk + 1);
        if (owner) {
            Sum add[NT];
#pragma unroll 4
            for (int ks = 0; ks < CS; ++ks) {
                uint32_t ah[4], al[4];
                const float left0 = CHANNEL ? 1.0f : sm[Sh::gb + ks * 8 + t], left1 = CHANNEL ? 1.0f : sm[Sh::gb + ks * 8 + t + 4];
                load_tile(tile_at(sm + Sh::k, CS, warp, ks), ah, al, left0, left1);
#pragma unroll
                for (int j = 0; j < NT; ++j) add_b(add[j], ah, al, tile_at(sm + Sh::u, CS, j, ks));
            }
            const float k0 = CHANNEL ? sm[Sh::gt + warp * 16 + g] : sm[Sh::gt], k1 = CHANNEL ? sm[Sh::gt + warp * 16 + g + 8] : k0;
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) S[j][e] = fmaf(e < 2 ? k0 : k1, S[j][e], add[j].at(e));
            publish();  // the first product of this chunk has read what stood there
        }
        Sum o[NW];
#pragma unroll 2
        for (int ks = 0; ks < 2 * (rt + 1); ++ks) {
            uint32_t ah[4], al[4];
            load_tile(tile_at(sm + Sh::p, CS, rt, ks), ah, al);
#pragma unroll
            for (int j = 0; j < NW; ++j) add_b(o[j], ah, al, tile_at(sm + Sh::u, CS, nt0 + j, ks));
        }
#pragma unroll
        for (int j = 0; j < NW; ++j)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int i = i0 + half * 8, c = col0 + (nt0 + j) * 8 + 2 * t;
                if (i < n && c < V)  // V is even
                    *reinterpret_cast<float2*>(out + ((size_t)(t0 + i) * H + h) * V + c) =
                        make_float2(fmaf(keep[half], zq[j].at(2 * half), o[j].at(2 * half)), fmaf(keep[half], zq[j].at(2 * half + 1), o[j].at(2 * half + 1)));
            }
        __syncthreads();
        if (warp == 0 && chunk + 1 < chunks) fetch_second(chunk + 1);
    }
    if (lost) {  // the call's results are void; let the copies asked for land before the block's memory is given back
        if (threadIdx.x == 0) {
            if (flag) atomicOr(flag, KB_FLAG_TIMEOUT);
            mbar_wait(&first_full, chunk & 1, &abort_word, 1u << 20);
            mbar_wait(&second_full, chunk & 1, &abort_word, 1u << 20);
        }
        __syncthreads();
        return;
    }
    if (owner) {
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int d = warp * 16 + g + (e >> 1) * 8, c = col0 + j * 8 + 2 * t + (e & 1);
                if (d < D && c < V) Sg[(size_t)c * D + d] = S[j][e];
            }
    }
}

struct Call {
    const float *q, *k, *v, *beta, *decay;
    float *states, *out, *scratch;
    const int *qo_indptr, *state_slots;
    int KH, D, H, V, rows, chunks;
    int* flag;
    cudaStream_t stream;
};

template <typename K>
int allow(K kernel, size_t bytes) {
    if (bytes <= 48 * 1024) return 0;
    return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

template <int DP, int NT, bool DELTA, bool CHANNEL>
int launch_walk(const Call& c, Scratch scratch, int head0, int heads) {
    constexpr size_t bytes = WalkShared<DP, NT, DELTA, CHANNEL>::floats * sizeof(float);
    if (int code = allow(walk_kernel<DP, NT, DELTA, CHANNEL>, bytes)) return code;
    kb_launch(walk_kernel<DP, NT, DELTA, CHANNEL>, dim3(c.rows, heads, (c.V + 8 * NT - 1) / (8 * NT)), dim3(WALK), bytes, c.stream, c.v, scratch, c.states,
              c.qo_indptr, c.state_slots, c.KH, c.D, c.H, c.V, head0, heads, c.out, c.flag);
    return kb_launch_result();
}

template <int DP, bool DELTA, bool CHANNEL>
int launch(const Call& c, int head0, int heads, int sms) {
    const Layout at(DELTA, CHANNEL, DP, c.V);
    const Scratch scratch{c.scratch, c.scratch + (size_t)c.chunks * heads * at.head};
    int code;
    if constexpr (CHANNEL) {
        constexpr size_t bytes = (size_t)(4 * C * (DP + 4) + 2 * C * LP + 4 * DP + C) * sizeof(float);
        if ((code = allow(prepare_channel_kernel<DP>, bytes))) return code;
        kb_launch(prepare_channel_kernel<DP>, dim3(c.chunks, heads), dim3(PREPARE_CHANNEL), bytes, c.stream, c.q, c.k, c.v, c.beta, c.decay, c.qo_indptr, c.rows, c.KH,
                  c.D, c.H, c.V, head0, heads, scratch);
    } else {
        constexpr size_t bytes = (size_t)(2 * C * (DP + 4) + (DELTA ? 2 : 1) * C * LP + 5 * C + 4) * sizeof(float);
        if ((code = allow(prepare_kernel<DP, DELTA>, bytes))) return code;
        const int HB = DELTA ? 1 : c.H / c.KH;
        kb_launch(prepare_kernel<DP, DELTA>, dim3(c.chunks, heads / HB), dim3(PREPARE), bytes, c.stream, c.q, c.k, c.v, c.beta, c.decay, c.qo_indptr, c.rows, c.KH,
                  c.D, c.H, c.V, head0, heads, HB, scratch);
    }
    if ((code = kb_launch_result())) return code;
    // 32 columns a block fetch and cut W, q, k and P half as often; 16 where 32 would leave SMs without a block
    if ((long long)c.rows * heads * ((c.V + 31) / 32) < 2 * sms) return launch_walk<DP, 2, DELTA, CHANNEL>(c, scratch, head0, heads);
    return launch_walk<DP, 4, DELTA, CHANNEL>(c, scratch, head0, heads);
}

long long floats_a_chunk(int D, int V, bool delta, bool channel, int heads, int sharing) {
    const Layout at(delta, channel, D <= 64 ? 64 : 128, V);
    return (long long)heads * at.head + (long long)(channel ? heads : heads / sharing) * at.shared;
}

}  // namespace

// Floats of scratch that `heads` heads of a chunk take (`sharing`: heads that share their keys; they go together).
KB_EXPORT int kb_chunked_recurrence_scratch(int D, int V, int delta, int channel, int heads, int sharing) {
    return (int)floats_a_chunk(D, V, delta != 0, channel != 0, heads, sharing);
}

// q, k: [tokens, KH, D]; v, out: [tokens, H, V]; beta: [tokens, H]; decay: [tokens, H], with `channel` [tokens, H, D]; states: [slots, H, V, D].
// `chunks`: at least the step's chunks of 64 tokens, rows cut one by one.  The heads go `group` at a time (a multiple of H / KH), for which `scratch` holds
// `scratch_floats`.
KB_EXPORT int kb_chunked_recurrence(const float* q, const float* k, const float* v, const float* beta, const float* decay, float* states,
                                    const int* qo_indptr, const int* state_slots, int KH, int D, int H, int V, float* out, int rows, int chunks, int delta,
                                    int channel, int group, float* scratch, long long scratch_floats, int* flag, cudaStream_t stream) {
    if (rows == 0 || chunks == 0) return 0;
    if (!q || !k || !v || !beta || !decay || !states || !qo_indptr || !state_slots || !out || !scratch) return KB_ERR_NULL;
    if (D < 4 || D > 128 || D % 4 || V < 4 || V % 4 || KH < 1 || H % KH || (channel && !delta) || H > 65535) return KB_ERR_UNSUPPORTED_SIZE;
    if ((((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)decay | (uintptr_t)scratch | (uintptr_t)out) & 15) != 0) return KB_ERR_BAD_ARG;
    const int sharing = H / KH;
    if (group < 1 || group % sharing || chunks * floats_a_chunk(D, V, delta, channel, group, sharing) > scratch_floats) return KB_ERR_BAD_ARG;
    int device = 0, sms = 0;
    if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) sms = 148;
    const Call call{q, k, v, beta, decay, states, out, scratch, qo_indptr, state_slots, KH, D, H, V, rows, chunks, flag, stream};
    for (int head0 = 0; head0 < H; head0 += group) {
        const int heads = H - head0 < group ? H - head0 : group;
        int code;
        if (D <= 64)
            code = channel ? launch<64, true, true>(call, head0, heads, sms) : delta ? launch<64, true, false>(call, head0, heads, sms) : launch<64, false, false>(call, head0, heads, sms);
        else
            code = channel ? launch<128, true, true>(call, head0, heads, sms) : delta ? launch<128, true, false>(call, head0, heads, sms) : launch<128, false, false>(call, head0, heads, sms);
        if (code) return code;
    }
    return 0;
}
