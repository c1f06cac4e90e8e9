// y[M,N] = x[M,K] . W[N,K]^T (+ bias[N]) in true fp32: plain FMA on CUDA cores,
// no tensor cores and no reduced-precision mode.  Each output element adds its terms
// in order of k, 256 at a time into one accumulator whose sums are then added in
// order into a second (a sum of 8,192 terms carries the rounding of 256 + 32
// additions, not of 8,192), so a row's result does not depend on M, on the tile's shape or on which tile
// it falls in: the 32-bit path is bit-stable however a prompt is cut into steps.
//
// What bounds it: the FMA pipes, 128 a cycle and SM, for which every thread keeps a TM x TN block of outputs in registers, so that
// the factors' reads from shared memory (TM + TN floats a k) stay below the multiply-adds (TM * TN); the next BK columns of both factors are
// fetched into registers while this BK is multiplied and go into the other half of shared memory.
#include "common.cuh"

#define F32_SUM_BLOCK 256  // terms a first-level accumulator takes before it is added to the second

// Four consecutive floats of row r at column k, zeros outside the matrix; `wide`: rows are whole aligned 16-byte groups
__device__ __forceinline__ float4 f32_fetch(const float* __restrict__ a, int ld, int r, int rows, int k, int K, bool wide) {
    if (r >= rows || k >= K) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float* at = a + (size_t)r * ld + k;
    if (wide) return *reinterpret_cast<const float4*>(at);
    return make_float4(at[0], k + 1 < K ? at[1] : 0.0f, k + 2 < K ? at[2] : 0.0f, k + 3 < K ? at[3] : 0.0f);
}

// A thread's TM rows are groups of G that lie BM / (TM / G) apart (so that a warp's 16-byte reads of one group are side by side), its TN columns likewise.
template <int BM, int BN, int TM, int TN, int BK>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_f32_kernel(const float* __restrict__ x, int ldx, const float* __restrict__ w, int ldw,
                const float* __restrict__ bias, float* __restrict__ y, int ldy, int M, int N, int K, int x_wide, int w_wide) {
    constexpr int THREADS = (BM / TM) * (BN / TN), COLS = BN / TN;
    constexpr int GM = TM < 4 ? TM : 4, GN = TN < 4 ? TN : 4;
    constexpr int LA = BM + 4, LB = BN + 4;
    constexpr int NA = BM * BK / 4 / THREADS, NB = BN * BK / 4 / THREADS;
    static_assert(NA * 4 * THREADS == BM * BK && NB * 4 * THREADS == BN * BK && F32_SUM_BLOCK % BK == 0, "whole loads");
    __shared__ __align__(16) float As[2][BK][LA];
    __shared__ __align__(16) float Bs[2][BK][LB];
    const int tid = threadIdx.x, tx = tid % COLS, ty = tid / COLS;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    pdl_wait();

    float acc[TM][TN], total[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = total[i][j] = 0.0f;
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
                    total[i][j] += acc[i][j];
                    acc[i][j] = 0.0f;
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
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
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
            float v = total[i][j] + acc[i][j];
            if (bias) v += bias[n];
            y[(size_t)m * ldy + n] = v;
        }
    }
}

template <int BM, int BN, int TM, int TN, int BK>
static int launch_gemm_f32(const float* x, int ldx, const float* w, int ldw, const float* bias, float* y, int ldy, int M, int N, int K, cudaStream_t stream) {
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) return KB_ERR_UNSUPPORTED_SIZE;
    const int x_wide = K % 4 == 0 && ldx % 4 == 0 && ((uintptr_t)x & 15) == 0, w_wide = K % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)w & 15) == 0;
    kb_launch(gemm_f32_kernel<BM, BN, TM, TN, BK>, grid, dim3((BM / TM) * (BN / TN)), 0, stream, x, ldx, w, ldw, bias, y, ldy, M, N, K, x_wide, w_wide);
    return kb_launch_result();
}

KB_EXPORT int kb_gemm_f32(const float* x, int ldx, const float* w, int ldw, const float* bias,
                          float* y, int ldy, int M, int N, int K, cudaStream_t stream) {
    if (M == 0 || N == 0) return 0;
    if (!x || !w || !y) return KB_ERR_NULL;
    if (K < 1) return KB_ERR_BAD_ARG;
    if (M > 65535 * 64) return KB_ERR_UNSUPPORTED_SIZE;
#define F32_ARGS x, ldx, w, ldw, bias, y, ldy, M, N, K, stream
    // A few rows: what counts is that many blocks stream the weight.
    if (M <= 16) return launch_gemm_f32<16, 32, 2, 2, 64>(F32_ARGS);
    int device = 0, sms = 0;
    if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) sms = 148;
    // The larger a tile, the fewer reads a multiply-add; the smaller, the less of the last wave is empty.  Time in units of outputs an SM
    // multiplies one behind the other, a tile's rate as measured relative to the largest.
    auto waves = [&](int bm, int bn, int resident, double rate) {
        const long long blocks = (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn);
        return (double)((blocks + (long long)sms * resident - 1) / ((long long)sms * resident)) * resident * bm * bn / rate;
    };
    const double large = waves(128, 128, 1, 1.0), middle = waves(64, 128, 2, 0.9), small = waves(64, 64, 3, 0.7);
    if (large <= middle && large <= small) return launch_gemm_f32<128, 128, 8, 8, 16>(F32_ARGS);
    if (middle <= small) return launch_gemm_f32<64, 128, 8, 4, 16>(F32_ARGS);
    return launch_gemm_f32<64, 64, 4, 4, 16>(F32_ARGS);
#undef F32_ARGS
}
