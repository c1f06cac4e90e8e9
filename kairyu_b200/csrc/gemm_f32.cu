// y[M,N] = x[M,K] . W[N,K]^T (+ bias[N]) in true fp32: plain FMA on CUDA cores,
// no tensor cores and no reduced-precision mode.  Each output element adds its terms
// in order of k, 256 at a time into one accumulator whose sums are then added in
// order into a second (a sum of 8,192 terms carries the rounding of 256 + 32
// additions, not of 8,192), so a row's result does not depend on M, on the tile's shape or on which tile
// it falls in: the 32-bit path is bit-stable however a prompt is cut into steps.
//
// What bounds it: shared memory hands out 128 bytes a cycle and SM, one float for every four of the 128 multiply-adds, so a thread's block of
// TM x TN outputs takes (TM + TN) floats a k where TM * TN / 4 are free: 8 x 8 outputs are level, 16 x 8 are ahead.  Two multiply-adds go in one
// instruction, which leaves issue slots for those reads (700 x 3,072 x 2,048: 485 -> 217 us, 41 TFLOP/s; with 4 x 4 outputs a thread and
// loads that waited for the products 466; 2,048 x 8,192 x 2,048: 1,278 us, 54 TFLOP/s, and 3,090).
// 16 x 8 outputs leave no registers for the second accumulators, which are needed
// once in 256 terms and stand in shared memory (SPILL).  The next BK columns of both factors are
// fetched into registers while this BK is multiplied and go into the other half of shared memory.
#include "common.cuh"

#define F32_SUM_BLOCK 256  // terms a first-level accumulator takes before it is added to the second

// Two multiply-adds in one instruction (each rounded as fmaf rounds), with one factor for both
__device__ __forceinline__ void fma_pair(float& x0, float& x1, float a0, float a1, float b) {
    asm("{\n .reg .b64 x, a, b;\n mov.b64 x, {%0, %1};\n mov.b64 a, {%2, %3};\n mov.b64 b, {%4, %4};\n fma.rn.f32x2 x, a, b, x;\n mov.b64 {%0, %1}, x;\n}\n"
        : "+f"(x0), "+f"(x1)
        : "f"(a0), "f"(a1), "f"(b));
}

// Four consecutive floats of row r at column k, zeros outside the matrix; `wide`: rows are whole aligned 16-byte groups
__device__ __forceinline__ float4 f32_fetch(const float* __restrict__ a, int ld, int r, int rows, int k, int K, bool wide) {
    if (r >= rows || k >= K) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float* at = a + (size_t)r * ld + k;
    if (wide) return *reinterpret_cast<const float4*>(at);
    return make_float4(at[0], k + 1 < K ? at[1] : 0.0f, k + 2 < K ? at[2] : 0.0f, k + 3 < K ? at[3] : 0.0f);
}

// A thread's TM rows are groups of G that lie BM / (TM / G) apart (so that a warp's 16-byte reads of one group are side by side), its TN columns likewise.
template <int BM, int BN, int TM, int TN, int BK, bool SPILL>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_f32_kernel(const float* __restrict__ x, int ldx, const float* __restrict__ w, int ldw,
                const float* __restrict__ bias, float* __restrict__ y, int ldy, int M, int N, int K, int x_wide, int w_wide) {
    constexpr int THREADS = (BM / TM) * (BN / TN), COLS = BN / TN;
    constexpr int GM = TM < 4 ? TM : 4, GN = TN < 4 ? TN : 4;
    constexpr int LA = BM + 4, LB = BN + 4;
    constexpr int NA = BM * BK / 4 / THREADS, NB = BN * BK / 4 / THREADS;
    static_assert(NA * 4 * THREADS == BM * BK && NB * 4 * THREADS == BN * BK && F32_SUM_BLOCK % BK == 0, "whole loads");
    extern __shared__ __align__(16) float sm[];
    float(*As)[BK][LA] = reinterpret_cast<float(*)[BK][LA]>(sm);
    float(*Bs)[BK][LB] = reinterpret_cast<float(*)[BK][LB]>(sm + 2 * BK * LA);
    float* totals = sm + 2 * BK * (LA + LB) + threadIdx.x;  // SPILL: TM * TN of them, THREADS apart
    const int tid = threadIdx.x, tx = tid % COLS, ty = tid / COLS;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    pdl_wait();

    float acc[TN][TM], total[SPILL ? 1 : TM][SPILL ? 1 : TN];
    auto second = [&](int i, int j) -> float& {
        if constexpr (SPILL) return totals[(i * TN + j) * THREADS];
        else return total[i][j];
    };
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[j][i] = second(i, j) = 0.0f;
    float4 na[NA], nb[NB];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < NA; ++i) {
            const int idx = tid + i * THREADS;
            na[i] = f32_fetch(x, ldx, m0 + idx / (BK / 4), M, k0 + idx % (BK / 4) * 4, K, x_wide);
        }
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            const int idx = tid + i * THREADS;
            nb[i] = f32_fetch(w, ldw, n0 + idx / (BK / 4), N, k0 + idx % (BK / 4) * 4, K, w_wide);
        }
    };
    auto place = [&](int buf) {
#pragma unroll
        for (int i = 0; i < NA; ++i) {
            const int idx = tid + i * THREADS, r = idx / (BK / 4), c = idx % (BK / 4) * 4;
            As[buf][c][r] = na[i].x, As[buf][c + 1][r] = na[i].y, As[buf][c + 2][r] = na[i].z, As[buf][c + 3][r] = na[i].w;
        }
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            const int idx = tid + i * THREADS, r = idx / (BK / 4), c = idx % (BK / 4) * 4;
            Bs[buf][c][r] = nb[i].x, Bs[buf][c + 1][r] = nb[i].y, Bs[buf][c + 2][r] = nb[i].z, Bs[buf][c + 3][r] = nb[i].w;
        }
    };
    // rows (columns) of a thread's group `i`
    auto row_at = [&](int i) { return i / GM * (BM / (TM / GM)) + ty * GM + i % GM; };
    auto col_at = [&](int j) { return j / GN * (BN / (TN / GN)) + tx * GN + j % GN; };
    fetch(0);
    place(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += BK, buf ^= 1) {
        if (k0 > 0 && k0 % F32_SUM_BLOCK == 0) {  // a block of 256 terms is complete
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    second(i, j) += acc[j][i];
                    acc[j][i] = 0.0f;
                }
        }
        const bool more = k0 + BK < K;
        if (more) fetch(k0 + BK);
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; i += GM) {
                const float* at = &As[buf][kk][row_at(i)];
                if constexpr (GM == 4) {
                    const float4 v = *reinterpret_cast<const float4*>(at);
                    a[i] = v.x, a[i + 1] = v.y, a[i + 2] = v.z, a[i + 3] = v.w;
                } else {
#pragma unroll
                    for (int e = 0; e < GM; ++e) a[i + e] = at[e];
                }
            }
#pragma unroll
            for (int j = 0; j < TN; j += GN) {
                const float* at = &Bs[buf][kk][col_at(j)];
                if constexpr (GN == 4) {
                    const float4 v = *reinterpret_cast<const float4*>(at);
                    b[j] = v.x, b[j + 1] = v.y, b[j + 2] = v.z, b[j + 3] = v.w;
                } else {
#pragma unroll
                    for (int e = 0; e < GN; ++e) b[j + e] = at[e];
                }
            }
#pragma unroll
            for (int j = 0; j < TN; ++j)
#pragma unroll
                for (int i = 0; i < TM; i += 2) fma_pair(acc[j][i], acc[j][i + 1], a[i], a[i + 1], b[j]);
        }
        if (more) place(buf ^ 1);  // the other half was read before the last barrier
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + row_at(i);
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + col_at(j);
            if (n >= N) continue;
            float v = second(i, j) + acc[j][i];
            if (bias) v += bias[n];
            y[(size_t)m * ldy + n] = v;
        }
    }
}

template <int BM, int BN, int TM, int TN, int BK, bool SPILL>
static int launch_gemm_f32(const float* x, int ldx, const float* w, int ldw, const float* bias, float* y, int ldy, int M, int N, int K, cudaStream_t stream) {
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) return KB_ERR_UNSUPPORTED_SIZE;
    const int x_wide = K % 4 == 0 && ldx % 4 == 0 && ((uintptr_t)x & 15) == 0, w_wide = K % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)w & 15) == 0;
    constexpr size_t bytes = (2 * BK * (BM + BN + 8) + (SPILL ? BM * BN : 0)) * sizeof(float);
    if (bytes > 48 * 1024)
        if (cudaError_t e = cudaFuncSetAttribute(gemm_f32_kernel<BM, BN, TM, TN, BK, SPILL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes)) return (int)e;
    kb_launch(gemm_f32_kernel<BM, BN, TM, TN, BK, SPILL>, grid, dim3((BM / TM) * (BN / TN)), bytes, stream, x, ldx, w, ldw, bias, y, ldy, M, N, K, x_wide, w_wide);
    return kb_launch_result();
}

KB_EXPORT int kb_gemm_f32(const float* x, int ldx, const float* w, int ldw, const float* bias,
                          float* y, int ldy, int M, int N, int K, cudaStream_t stream) {
    if (M == 0 || N == 0) return 0;
    if (!x || !w || !y) return KB_ERR_NULL;
    if (K < 1) return KB_ERR_BAD_ARG;
    if (M > 65535 * 64) return KB_ERR_UNSUPPORTED_SIZE;
#define F32_ARGS x, ldx, w, ldw, bias, y, ldy, M, N, K, stream
    // A few rows: what counts is that many blocks stream the weight (N = 3,072, K = 2,048: 37 us at 16 rows, where tiles of 64 x 64 take 91).
    if (M <= 96) return launch_gemm_f32<16, 32, 2, 2, 64, false>(F32_ARGS);
    int device = 0, sms = 0;
    if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) sms = 148;
    // The larger a tile, the fewer reads a multiply-add; the smaller, the more evenly the outputs lie on the SMs (tiles on one SM share its pipes).  Time in
    // outputs of the fullest SM, over a tile's rate relative to the largest.
    auto time = [&](int bm, int bn, double rate) {
        const long long blocks = (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn);
        return (double)((blocks + sms - 1) / sms) * bm * bn / rate;
    };
    const double huge = time(128, 128, 1.0), large = time(96, 128, 0.95), middle = time(64, 128, 0.8), small = time(64, 64, 0.5);
    if (huge <= large && huge <= middle && huge <= small) return launch_gemm_f32<128, 128, 16, 8, 16, true>(F32_ARGS);
    if (large <= middle && large <= small) return launch_gemm_f32<96, 128, 12, 8, 16, true>(F32_ARGS);
    if (middle <= small) return launch_gemm_f32<64, 128, 8, 8, 16, true>(F32_ARGS);
    return launch_gemm_f32<64, 64, 4, 4, 16, false>(F32_ARGS);
#undef F32_ARGS
}
