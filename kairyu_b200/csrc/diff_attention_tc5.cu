// Differential attention over prompt portions on the 5th-generation tensor cores: what diff_attention_mma.cu computes, for heads of
// two maps of 64 or 128 columns and values of 64 or 128.
//
//     s_m = cap * tanh(q_m . k_m * scale / cap),  a_m = softmax(s_m) V,  o = a_1 - lambda a_2,  head norm
//
// A block has a tile of 128 queries of one head and walks the keys in tiles of 64.  A query row and a key row hold both maps side by side, so
// a copy of a run of positions brings both maps' keys, and the value tile serves both.  Roles (320 threads, one block an SM):
//   warp 0      producer: TMA copies of the queries and of the key and value tiles, two stages ahead
//   warp 1      one thread issues the products: S_m = Q_m K_m^T into two buffers of 64 columns of tensor memory a map, two key tiles ahead, and
//               O_m += P_m V; two maps' scores and outputs fill the 512 columns
//   warps 2-5   softmax of the first map, 6-9 of the second: thread r owns row r, as in attention_prefill_tc5.cu (P over S, O rescaled
//               only when the row's maximum grows by 2^8); in the end the first map's threads read both outputs of their row
// The cap costs two special functions a score where x = score * scale / cap is large; where every score of a warp's tile has |x| <= 0.45,
// which is nearly always, x p(x^2) with the polynomial of softcap.cuh does, and the special-function unit is left to the exponentials.
//
// What bounds it: the copies, 12 a key tile with pages of 16 positions (an SM issues one every 50 to 75 ns), then the products, 900 cycles a key
// tile.  The mma.sync kernel's products run at a quarter of the rate and its cap always takes the special functions: 2,048 tokens, 16 heads over 4,
// window 1,024: 227 -> 66 us.
#include "softcap.cuh"
#include "umma.cuh"

namespace {

constexpr int THREADS = 320, BM = 128, BN = 64, STAGES = 2;
constexpr float LOG2E = 1.4426950408889634f, RESCALE_STEP = 8.0f;
constexpr int FLAG_MISALIGNED = 32, FLAG_PREFILL = 128;

__device__ __forceinline__ float ex2_ftz(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(d) : "l"(*reinterpret_cast<uint64_t*>(&a)), "l"(*reinterpret_cast<uint64_t*>(&b)), "l"(*reinterpret_cast<uint64_t*>(&c)));
    return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(d) : "l"(*reinterpret_cast<uint64_t*>(&a)), "l"(*reinterpret_cast<uint64_t*>(&b)));
    return *reinterpret_cast<float2*>(&d);
}

template <int D, int DV>
struct Cfg {
    static constexpr int MAP_BANDS = D / 64, K_BANDS = 2 * MAP_BANDS, V_BANDS = DV / 64;
    static constexpr int Q_BAND = BM * 128, KV_BAND = BN * 128;
    static constexpr int Q_BYTES = K_BANDS * Q_BAND, K_BYTES = K_BANDS * KV_BAND, V_BYTES = V_BANDS * KV_BAND;
    static constexpr int OFF_K = Q_BYTES, OFF_V = OFF_K + STAGES * K_BYTES, OFF_L = OFF_V + STAGES * V_BYTES, OFF_BAR = OFF_L + BM * 4;
    static constexpr int NUM_BARS = 1 + 4 * STAGES + 3 * 4 + 1;
    static constexpr size_t SMEM = OFF_BAR + NUM_BARS * 8 + 16;
    static constexpr int O_COL = 4 * BN;  // S of map m, buffer b at (2 m + b) * 64; O of map m at O_COL + m * DV
};

template <int D, int DV>
__global__ void __launch_bounds__(THREADS, 1)
diff_attention_tc5_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                          __nv_bfloat16* __restrict__ out, int out_stride, const int* __restrict__ qo_indptr, const int* __restrict__ seq_lens,
                          const int* __restrict__ block_table, int max_pages, const int* __restrict__ tile_rows, const int* __restrict__ tile_starts, int num_tiles, int Hq,
                          int Hkv, int page_size, int page_shift, int num_pages, float scale, int window, int merged, float lambda, int head_norm, float eps, float out_scale,
                          const KbSoftcap cap, float near_limit, int* flag) {
    using C = Cfg<D, DV>;
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char *sQ = smem, *sK = smem + C::OFF_K, *sV = smem + C::OFF_V;
    float* second_inv = reinterpret_cast<float*>(smem + C::OFF_L);  // the second map's 1 / sum a row
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
    uint64_t *q_full = bars, *k_full = bars + 1, *v_full = k_full + STAGES, *k_empty = v_full + STAGES, *v_empty = k_empty + STAGES;
    // one a map and S buffer, used in turn by the key tiles: a softmax may be a tile ahead of the thread that issues the products, and a parity cannot tell a
    // phase from the one two before it
    uint64_t *s_full = v_empty + STAGES, *p_full = s_full + 4, *pv_done = p_full + 4, *second_done = pv_done + 4;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + C::NUM_BARS);
    volatile int* abort_word = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        prefetch_tensormap(&map_q);
        prefetch_tensormap(&map_k);
        prefetch_tensormap(&map_v);
        for (int i = 0; i < 1 + 4 * STAGES + 4; ++i) mbar_init(bars + i, 1);
        for (int i = 0; i < 4; ++i) {
            mbar_init(p_full + i, 4);
            mbar_init(pv_done + i, 1);
        }
        mbar_init(second_done, 4);
        *abort_word = 0;
        if ((smem_addr(smem) & 1023u) != 0) {  // the swizzled layouts below assume it
            if (flag) atomicOr(flag, FLAG_MISALIGNED);
            *abort_word = 1;
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        fence_proxy_async_smem();
    }
    if (warp == 1) tmem_alloc(tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();

    const int h = blockIdx.x, kvh = h / (Hq / Hkv);
    const int tile = num_tiles - 1 - (int)blockIdx.y;  // later tiles of a portion see more keys: they go first
    const int row = tile_rows[tile], q0 = tile_starts[tile], tok0 = qo_indptr[row];
    const int portion = qo_indptr[row + 1] - tok0;
    const int rows_here = min(BM, portion - q0);
    const int first_pos = seq_lens[row] - portion + q0, last_pos = first_pos + rows_here - 1, key_end = last_pos + 1;
    const int key_lo = window > 0 && first_pos + 1 > window ? first_pos + 1 - window : 0;
    const int first_kt = key_lo / BN, num_kt = (key_end - 1) / BN - first_kt + 1;
    // a value tile: rows of a band lie run_rows x 128 bytes from the next band's, a run of positions V_BANDS x run_rows x 128 bytes from the next run
    const int box_rows = page_size < BN ? page_size : BN, run_rows = merged ? box_rows : BN;
    const int band_bytes = run_rows * 128, run_bytes = C::V_BANDS * band_bytes;
    auto timed_out = [&]() {
        if (!*abort_word && flag) atomicOr(flag, KB_FLAG_TIMEOUT | FLAG_PREFILL);
        *abort_word = 1;
    };

    if (*abort_word) {
        // fall through to the common exit
    } else if (warp == 0) {
        // ---------------- producer
        const int runs = BN / box_rows, per_k = C::K_BANDS * runs, per_v = merged ? runs : C::V_BANDS * runs;
        if (lane == 0) {
            mbar_arrive_expect_tx(q_full, C::Q_BYTES);
#pragma unroll
            for (int band = 0; band < C::K_BANDS; ++band) tma_load_2d_plain(sQ + band * C::Q_BAND, &map_q, h * 2 * D + band * 64, tok0 + q0, q_full);
        }
        const int* table = block_table + (size_t)row * max_pages;
        bool ok = true;
        for (int g = 0; g < num_kt && ok; ++g) {
            const int st = g % STAGES, use = g / STAGES;
#pragma unroll
            for (int is_v = 0; is_v < 2; ++is_v) {
                if (use > 0 && !mbar_wait((is_v ? v_empty : k_empty) + st, (use - 1) & 1, abort_word)) {
                    if (lane == 0) timed_out();
                    ok = false;
                    break;
                }
                uint64_t* bar = (is_v ? v_full : k_full) + st;
                if (lane == 0) mbar_arrive_expect_tx(bar, is_v ? C::V_BYTES : C::K_BYTES);
                __syncwarp();
                for (int op = lane; op < (is_v ? per_v : per_k); op += 32) {
                    const int band = op / runs, run = op % runs;  // band 0 where a copy takes every band
                    const int key = (first_kt + g) * BN + run * box_rows;
                    const int index = key >> page_shift;
                    int page = 0, within = 0;  // the reserved page stands in for rows nobody may see
                    if (key < key_end && key + box_rows > key_lo && index < max_pages) {
                        const int p = table[index];
                        if (p >= 0 && p < num_pages) {
                            page = p;
                            within = key - (index << page_shift);
                        }
                    }
                    if (!is_v) tma_load_4d_plain(sK + st * C::K_BYTES + band * C::KV_BAND + run * box_rows * 128, &map_k, band * 64, kvh, within, page, bar);
                    else if (merged) tma_load_5d_plain(sV + st * C::V_BYTES + run * run_bytes, &map_v, 0, kvh, within, 0, page, bar);
                    else tma_load_4d_plain(sV + st * C::V_BYTES + band * C::KV_BAND + run * box_rows * 128, &map_v, band * 64, kvh, within, page, bar);
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- one thread issues the products
        if (lane == 0) {
            constexpr uint32_t idesc_qk = umma_idesc(BN), idesc_pv = umma_idesc_b_mn(DV);
            const uint64_t q_desc = umma_desc_sw128(smem_addr(sQ)), k_desc = umma_desc_sw128(smem_addr(sK));
            const uint64_t v_desc = umma_desc_mn_sw128(smem_addr(sV), (uint32_t)band_bytes, 1024);
            uint64_t v_step[BN / 16];  // where the 16 keys of a P V step lie in a value tile
#pragma unroll
            for (int ks = 0; ks < BN / 16; ++ks) v_step[ks] = (uint64_t)(((ks * 16 / run_rows) * run_bytes + (ks * 16 % run_rows) * 128) >> 4);
            bool ok = true;
            auto wait = [&](uint64_t* bar, uint32_t parity) {
                if (ok && !mbar_wait(bar, parity, abort_word)) {
                    timed_out();
                    ok = false;
                }
                return ok;
            };
            auto issue_qk = [&](int g) {
                const int st = g % STAGES;
                const uint64_t k_tile = k_desc + (uint64_t)((st * C::K_BYTES) >> 4);
#pragma unroll
                for (int m = 0; m < 2; ++m) {
#pragma unroll
                    for (int band = 0; band < C::MAP_BANDS; ++band)
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            umma_bf16(tmem_base + (2 * m + (g & 1)) * BN, q_desc + (uint64_t)(((m * C::MAP_BANDS + band) * C::Q_BAND + k * 32) >> 4),
                                      k_tile + (uint64_t)(((m * C::MAP_BANDS + band) * C::KV_BAND + k * 32) >> 4), idesc_qk, band > 0 || k > 0 ? 1u : 0u);
                    if (m == 1) umma_commit(k_empty + st);
                    umma_commit(s_full + 2 * m + (g & 1));
                }
            };
            wait(q_full, 0);
            for (int g = 0; g < 2 && g < num_kt && ok; ++g)
                if (wait(k_full + g, 0)) {
                    tc_fence_after();
                    issue_qk(g);
                }
            for (int g = 0; g < num_kt && ok; ++g) {
                const int st = g % STAGES;
                const uint64_t v_tile = v_desc + (uint64_t)((st * C::V_BYTES) >> 4);
                if (!wait(v_full + st, (g / STAGES) & 1)) break;
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    if (!wait(p_full + 2 * m + (g & 1), (g >> 1) & 1)) break;
                    tc_fence_after();
#pragma unroll
                    for (int ks = 0; ks < BN / 16; ++ks)
                        umma_bf16_a_tmem(tmem_base + C::O_COL + m * DV, tmem_base + (2 * m + (g & 1)) * BN + ks * 8, v_tile + v_step[ks], idesc_pv, g > 0 || ks > 0 ? 1u : 0u);
                    umma_commit(pv_done + 2 * m + (g & 1));
                }
                if (!ok) break;
                umma_commit(v_empty + st);
                if (g + 2 < num_kt) {
                    // both softmaxes hold S_g in registers (they have written P_g): its buffers take tile g + 2
                    if (!wait(k_full + st, ((g + 2) / STAGES) & 1)) break;
                    tc_fence_after();
                    issue_qk(g + 2);
                }
            }
        }
    } else {
        // ---------------- softmax and epilogue: a thread a row and map
        const int m = warp >= 6 ? 1 : 0;
        const int quarter = warp & 3;  // the tensor-memory lanes this warp may touch
        const int r = quarter * 32 + lane, soft_tid = (threadIdx.x - 64) & 127;
        const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16);
        const uint32_t o_base = lane_base + C::O_COL + m * DV;
        const bool valid = r < rows_here;
        const int pos = valid ? first_pos + r : last_pos;
        const int lo = window > 0 && pos + 1 > window ? pos + 1 - window : 0;
        const int lo_last = window > 0 && last_pos + 1 > window ? last_pos + 1 - window : 0;
        const bool capped = cap.mode != KB_SOFTCAP_NONE;
        const float sl2 = capped ? 1.0f : scale * LOG2E;  // capped scores come with the scale in them
        float m_ref = -INFINITY, l = 0.0f;                // the maximum the row's P and O are scaled by
        bool ok = true;
        for (int g = 0; g < num_kt; ++g) {
            const int key0 = (first_kt + g) * BN;
            const uint32_t s_at = lane_base + (2 * m + (g & 1)) * BN;
            if (!mbar_wait(s_full + 2 * m + (g & 1), (g >> 1) & 1, abort_word)) { ok = false; break; }
            tc_fence_after();
            uint32_t raw[2][32];
            tmem_load32_nowait(s_at, raw[0]);
            tmem_load32_nowait(s_at + 32, raw[1]);
            tmem_wait_ld();
            float tt[BN];
#pragma unroll
            for (int c = 0; c < BN; ++c) tt[c] = __uint_as_float(raw[c >> 5][c & 31]);
            if (capped) {
                float big = 0.0f;
#pragma unroll
                for (int c = 0; c < BN; ++c) big = fmaxf(big, fabsf(tt[c]));
                if (!__any_sync(0xffffffffu, big > near_limit)) {
#pragma unroll
                    for (int c = 0; c < BN; c += 2) {
                        const float2 x = make_float2(tt[c], tt[c + 1]), z = mul2(x, x);
                        float2 p = fma2(z, make_float2(cap.c[3], cap.c[3]), make_float2(cap.c[2], cap.c[2]));
                        p = fma2(z, p, make_float2(cap.c[1], cap.c[1]));
                        p = mul2(x, fma2(z, p, make_float2(cap.c[0], cap.c[0])));
                        tt[c] = p.x;
                        tt[c + 1] = p.y;
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < BN; ++c) tt[c] = fmaf(-2.0f * cap.b, __fdividef(1.0f, 1.0f + ex2_ftz(cap.a * tt[c])), cap.b);
                }
            }
            if (key0 + BN - 1 > first_pos || key0 < lo_last) {  // the diagonal or the window's edge crosses this tile
#pragma unroll
                for (int c = 0; c < BN; ++c) tt[c] = key0 + c <= pos && key0 + c >= lo ? tt[c] : -INFINITY;
            }
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int c = 0; c < BN; ++c) mx4[c & 3] = fmaxf(mx4[c & 3], tt[c]);
            const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * sl2;  // -inf stays -inf
            float alpha = 1.0f;
            if (m_ref == -INFINITY) {
                m_ref = mx;  // nothing accumulated for this row yet
            } else if (mx > m_ref + RESCALE_STEP) {
                alpha = exp2f(m_ref - mx);
                m_ref = mx;
            }
            // every phase of the two pv_done barriers is observed in order, two tiles late; only a rescale of O needs the product before complete
            if (g > 1 && !mbar_wait(pv_done + 2 * m + (g & 1), ((g - 2) >> 1) & 1, abort_word)) { ok = false; break; }
            if (__any_sync(0xffffffffu, alpha != 1.0f)) {
                if (g > 0 && !mbar_wait(pv_done + 2 * m + ((g - 1) & 1), ((g - 1) >> 1) & 1, abort_word)) { ok = false; break; }
                tc_fence_after();
#pragma unroll
                for (int c = 0; c < DV / 32; ++c) {
                    uint32_t o[32];
                    tmem_load32_nowait(o_base + c * 32, o);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                    tmem_store32(o_base + c * 32, o);
                }
                tmem_wait_st();
                l *= alpha;
            }
            const float neg_base = m_ref == -INFINITY ? 0.0f : -m_ref;
            float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            uint32_t packed[BN / 2];
#pragma unroll
            for (int c = 0; c < BN; c += 2) {
                const float2 arg = fma2(make_float2(tt[c], tt[c + 1]), make_float2(sl2, sl2), make_float2(neg_base, neg_base));  // (-inf) * scale + base = -inf
                const float2 p = make_float2(ex2_ftz(arg.x), ex2_ftz(arg.y));
                sum[c & 2] += p.x;
                sum[(c & 2) + 1] += p.y;
                __nv_bfloat162 pair = __floats2bfloat162_rn(p.x, p.y);
                packed[c >> 1] = *reinterpret_cast<uint32_t*>(&pair);
            }
            l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
            tmem_store32(s_at, packed);
            tmem_wait_st();
            if (key0 + BN > key_end) {
                // keys beyond the last query have probability 0, but what lies there may be anything and 0 * NaN is NaN: clear those rows of V (both maps'
                // threads do, with the same zeros, so that neither product waits for the other map)
                const int st = g % STAGES;
                if (!mbar_wait(v_full + st, (g / STAGES) & 1, abort_word)) { ok = false; break; }
                unsigned char* v_tile = sV + st * C::V_BYTES;
                for (int idx = soft_tid; idx < BN * C::V_BANDS * 8; idx += 128) {
                    const int vr = idx / (C::V_BANDS * 8), c = idx % (C::V_BANDS * 8);
                    if (key0 + vr >= key_end)
                        *reinterpret_cast<uint4*>(v_tile + (vr / run_rows) * run_bytes + (c >> 3) * band_bytes + (vr % run_rows) * 128 + (c & 7) * 16) = make_uint4(0, 0, 0, 0);
                }
                fence_proxy_async_smem();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full + 2 * m + (g & 1));
        }
        if (ok && num_kt > 1 && !mbar_wait(pv_done + 2 * m + ((num_kt - 2) & 1), ((num_kt - 2) >> 1) & 1, abort_word)) ok = false;
        if (ok && !mbar_wait(pv_done + 2 * m + ((num_kt - 1) & 1), ((num_kt - 1) >> 1) & 1, abort_word)) ok = false;
        const float inv = l > 0.0f ? 1.0f / l : 0.0f;
        if (ok && m == 1) {
            second_inv[r] = inv;
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(second_done);
        }
        if (ok && m == 0 && !mbar_wait(second_done, 0, abort_word)) ok = false;
        if (ok && m == 0) {
            tc_fence_after();
            const float other = second_inv[r] * lambda;
            float factor = 1.0f;
            // twice over the row where the head norm wants its sum of squares first
            for (int pass = head_norm ? 0 : 1; pass < 2; ++pass) {
                float squares = 0.0f;
                __nv_bfloat16* dst = out + (size_t)(tok0 + q0 + r) * out_stride + (size_t)h * DV;
#pragma unroll
                for (int c = 0; c < DV / 32; ++c) {
                    uint32_t a[32], b[32];
                    tmem_load32_nowait(lane_base + C::O_COL + c * 32, a);
                    tmem_load32_nowait(lane_base + C::O_COL + DV + c * 32, b);
                    tmem_wait_ld();
                    float o[32];
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        o[i] = __uint_as_float(a[i]) * inv - other * __uint_as_float(b[i]);
                        squares += o[i] * o[i];
                    }
                    if (pass == 1 && valid) {
#pragma unroll
                        for (int i = 0; i < 32; i += 8) {
                            uint32_t w[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                __nv_bfloat162 pair = __floats2bfloat162_rn(o[i + 2 * e] * factor, o[i + 2 * e + 1] * factor);
                                w[e] = *reinterpret_cast<uint32_t*>(&pair);
                            }
                            *reinterpret_cast<uint4*>(dst + c * 32 + i) = make_uint4(w[0], w[1], w[2], w[3]);
                        }
                    }
                }
                if (pass == 0) factor = rsqrtf(squares / (float)DV + eps) * out_scale;
            }
        }
        if (!ok && lane == 0) timed_out();
    }
    tc_fence_before();
    __syncthreads();
    if (*abort_word && threadIdx.x == 0) {
        // copies still in flight target this block's shared memory: one more short wait on the barriers they complete, whichever phase they are in
        volatile int ignore = 0;
        for (int s = 0; s < 1 + 2 * STAGES; ++s) {
            mbar_wait(bars + s, 0, &ignore, 1024);
            mbar_wait(bars + s, 1, &ignore, 1024);
        }
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

}  // namespace

// 1 where maps of D columns, values of DV and pages of page_size positions go to this kernel.
KB_EXPORT int kb_diff_attention_tc5_supported(int D, int DV, int page_size) {
    return (D == 64 || D == 128) && (DV == 64 || DV == 128) && page_size >= 8 && (page_size & (page_size - 1)) == 0;
}
// 1 where the map of the values has every 64-column band in a box (kb_attention_encode_cache_map with bands = 1)
KB_EXPORT int kb_diff_attention_tc5_merged(int DV, int page_size) { return DV > 64 && page_size >= 16; }

template <int KD, int KV>
struct Sizes {
    static constexpr int D = KD, DV = KV;
};

// map_q: 2-D map over the packed query rows [tokens, q_stride] with boxes of [128 rows, 64 columns]; map_k, map_v: maps over the caches as
// kb_attention_prefill_tc5 takes them (a key row: both maps, 2 D columns).  The list holds 128 queries a tile.  softcap (optional): a host KbSoftcap with the
// coefficients of both forms; near_limit: the largest |raw score| that its near form covers.
KB_EXPORT int kb_diff_attention_tc5(const void* map_q, const void* map_k, const void* map_v, void* out, int out_stride, const int* qo_indptr, const int* seq_lens,
                                    const int* block_table, int max_pages, const int* tile_rows, const int* tile_starts, int num_tiles, int Hq, int Hkv, int D, int DV,
                                    int page_size, int num_pages, float scale, int window, float lambda, int head_norm, float eps, float out_scale, const void* softcap,
                                    float near_limit, int* flag, cudaStream_t stream) {
    if (num_tiles == 0) return 0;
    if (!map_q || !map_k || !map_v || !out || !qo_indptr || !seq_lens || !block_table || !tile_rows || !tile_starts) return KB_ERR_NULL;
    if (Hkv < 1 || Hq % Hkv != 0 || num_tiles > 65535 || out_stride % 8 != 0 || ((uintptr_t)out % 16) != 0) return KB_ERR_BAD_ARG;
    if (!kb_diff_attention_tc5_supported(D, DV, page_size)) return KB_ERR_UNSUPPORTED_SIZE;
    int shift = 0;
    while ((1 << shift) < page_size) ++shift;
    const KbSoftcap cap = kb_softcap_of(softcap);
    auto launch = [&](auto sizes) {
        constexpr int KD = decltype(sizes)::D, KV = decltype(sizes)::DV;
        static bool configured = false;  // of this pair of sizes
        if (!configured) {
            if (cudaError_t e = cudaFuncSetAttribute(diff_attention_tc5_kernel<KD, KV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg<KD, KV>::SMEM)) return (int)e;
            configured = true;
        }
        kb_launch(diff_attention_tc5_kernel<KD, KV>, dim3(Hq, num_tiles), dim3(THREADS), Cfg<KD, KV>::SMEM, stream, *(const CUtensorMap*)map_q, *(const CUtensorMap*)map_k,
                  *(const CUtensorMap*)map_v, (__nv_bfloat16*)out, out_stride, qo_indptr, seq_lens, block_table, max_pages, tile_rows, tile_starts, num_tiles, Hq, Hkv,
                  page_size, shift, num_pages, scale, window, kb_diff_attention_tc5_merged(DV, page_size), lambda, head_norm, eps, out_scale, cap, near_limit, flag);
        return kb_launch_result();
    };
    if (D == 64) return DV == 64 ? launch(Sizes<64, 64>{}) : launch(Sizes<64, 128>{});
    return DV == 64 ? launch(Sizes<128, 64>{}) : launch(Sizes<128, 128>{});
}
