// Y[M, N] = X[M, K] * W[N, K]^T on the CUDA cores with fused multiply-adds in true 32-bit
// (no tensor-core tf32 mode): the matrix product of the 32-bit path, and of sizes that the
// tensor-core kernels refuse.  `y = x @ W.T`, weight stored (out, in):
// src/scratch_llm/model.py:125-133 of the reference.
//
// Every output element is one chain of fmaf over k = 0..K-1 in ascending order, whatever M
// and N are, so a token's result does not depend on what else is in the batch.
//
// Three kernels.  32-bit operands whose rows allow 16-byte requests, by size:
//   gemm_f32_wide_kernel   tiles of 64 x 64, 64 x 48 or 64 x 32, where `wide_columns` finds them faster
//   gemm_f32_kernel        smaller tiles behind a ring of cp.async stages: few tokens are bound by the chain
//                          of steps over k, whose loads the ring keeps ahead of.  Tiles of 32 x 32, and of
//                          16 x 16 up to 16 tokens.
// gemm_simt_kernel: every other type and layout (one step of loads, then its arithmetic).
// us (all on gemm_simt_kernel / with a row a lane in the wide kernel / now), K = 2,048:
//   1 token    N 3,072: 116 / 25 / 25         16,384: 213 / 70 / 71          128,256: 1,161 / 419 / 419
//   64         134 / 62 / 62                  236 / 184 / 173                1,369 / 973 / 827
//   256        214 / 137 / 124                701 / 560 / 469                5,258 / 3,751 / 2,996
//   777        497 / 366 / 258                2,194 / 1,594 / 1,258          - / 11,730 / 9,383
//   2,048      1,067 / 811 / 600              5,337 / 3,767 / 3,020          - / 28,897 / 22,874 (47 TF/s)
// What bounds the wide kernel now is shared memory: a read of 16 bytes a lane takes four cycles of it
// whether or not lanes ask for the same, 16 per 64 multiply-adds a lane, as many as the four schedulers have.
#include "common.cuh"

namespace sllm {

constexpr int BM = 64, BN = 64, BK = 16, PAD = 4;

template <typename TIn, typename TOut>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const TIn* __restrict__ X, const TIn* __restrict__ W, TOut* __restrict__ Y,
                 int M, int N, int K, int64_t ldx, int64_t ldw, int64_t ldy) {
    __shared__ float As[BK][BM + PAD];
    __shared__ float Bs[BK][BN + PAD];
    const int tid = threadIdx.x;
    const int bm = blockIdx.y * BM, bn = blockIdx.x * BN;
    const int lr = tid >> 2, lc = (tid & 3) * 4;  // load: row 0..63, 4 consecutive k
    const int ty = tid >> 4, tx = tid & 15;       // compute: 4x4 outputs
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = k0 + lc + i;
            const int m = bm + lr, n = bn + lr;
            As[lc + i][lr] = (m < M && k < K) ? to_float(X[(int64_t)m * ldx + k]) : 0.f;
            Bs[lc + i][lr] = (n < N && k < K) ? to_float(W[(int64_t)n * ldw + k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = bm + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = bn + tx * 4 + j;
            if (n < N) Y[(int64_t)m * ldy + n] = from_float<TOut>(acc[i][j]);
        }
    }
}

__device__ __forceinline__ unsigned long long pack2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float part(const float4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// Thread (ty, tx) has rows ty + i * (BM / TM) and columns tx + j * (BN / TN).  K % 4 == 0.
template <int BM, int BN, int TM, int TN, int BK, int STAGES>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_f32_kernel(const float* __restrict__ X, const float* __restrict__ W, float* __restrict__ Y, int M, int N,
                int K, int64_t ldx, int64_t ldw, int64_t ldy) {
    constexpr int THREADS = (BM / TM) * (BN / TN), LD = BK + 4, QUADS = BK / 4;
    constexpr int STAGE = (BM + BN) * LD;
    extern __shared__ __align__(16) float sm[];
    const int tid = threadIdx.x, tx = tid % (BN / TN), ty = tid / (BN / TN);
    const int bm = blockIdx.y * BM, bn = blockIdx.x * BN;
    auto request = [&](int stage, int k0) {      // rows and columns beyond the matrices: zeros
        float* dst = sm + stage * STAGE;
#pragma unroll
        for (int n = 0; n < ((BM + BN) * QUADS + THREADS - 1) / THREADS; ++n) {
            const int i = tid + n * THREADS, r = i / QUADS, k = k0 + i % QUADS * 4;
            if (((BM + BN) * QUADS) % THREADS && i >= (BM + BN) * QUADS) break;
            const bool left = r < BM;
            const int row = left ? bm + r : bn + r - BM;
            const bool there = row < (left ? M : N) && k < K;
            const float* src = !there ? X : left ? X + row * ldx + k : W + row * ldw + k;
            const int bytes = there ? 16 : 0;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::
                         "r"((uint32_t)__cvta_generic_to_shared(dst + r * LD + i % QUADS * 4)), "l"(src), "r"(bytes)
                         : "memory");
        }
    };
    const int steps = (K + BK - 1) / BK;
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < steps) request(s, s * BK);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    unsigned long long acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;
    for (int s = 0; s < steps; ++s) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
        __syncthreads();       // the stage is there for all, and the one before it is done with
        const int next = s + STAGES - 1;
        if (next < steps) request(next % STAGES, next * BK);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        const float* xs = sm + s % STAGES * STAGE + ty * LD;
        const float* ws = sm + s % STAGES * STAGE + (BM + tx) * LD;
#pragma unroll
        for (int q = 0; q < QUADS; ++q) {
            float4 a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(xs + i * (BM / TM) * LD + 4 * q);
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const float4*>(ws + j * (BN / TN) * LD + 4 * q);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                unsigned long long w[TN / 2];
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) w[j] = pack2(part(b[2 * j], k), part(b[2 * j + 1], k));
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const unsigned long long x = pack2(part(a[i], k), part(a[i], k));
#pragma unroll
                    for (int j = 0; j < TN / 2; ++j)
                        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(x), "l"(w[j]));
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = bm + ty + i * (BM / TM);
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = bn + tx + j * (BN / TN);
            const unsigned long long v = acc[i][j / 2];
            if (n < N) Y[(int64_t)m * ldy + n] = __uint_as_float((unsigned)(j & 1 ? v >> 32 : v));
        }
    }
}

// The widest tiles: 64 x (8 TN) by 64 threads of 8 x TN outputs, TN = 4, 6 or 8.  Four neighbouring lanes
// request a row's next 16 elements (64 bytes) while a step is worked on, so that a warp's request touches 8
// rows (a row a lane: 365 us for 777 tokens by 3,072 in tiles of 64 x 64, 320 so).  They are
// stored [k][row], so that per k four reads of 16 bytes feed 64 multiply-adds without a move between
// registers; quad k / 4 of the row's elements stands 8 k / 4 places further (modulo the tile), so that the
// four lanes of a row store to different banks.
constexpr int WIDE = 64, WK = 16;
template <int TN>
__global__ void __launch_bounds__(WIDE, 6)
gemm_f32_wide_kernel(const float* __restrict__ X, const float* __restrict__ W, float* __restrict__ Y, int M, int N,
                     int K, int64_t ldx, int64_t ldw, int64_t ldy) {
    constexpr int COLS = 8 * TN, XN = WIDE / 16, WN = COLS / 16;     // pieces of 16 rows
    __shared__ __align__(16) float xs[2][WK][WIDE];
    __shared__ __align__(16) float ws[2][WK][WIDE];     // (rows of 64 places whatever the tile)
    const int tid = threadIdx.x, tx = tid % 8 * 4, ty = tid / 8 * 4;
    const int bm = blockIdx.y * WIDE, bn = blockIdx.x * COLS;
    const int q = tid % 4, lr = tid / 4;                // this thread's quad of a step, and rows lr + 16 i
    // (rows beyond the matrices read the last one again; their outputs are not stored)
    const float* x[XN];
    const float* w[WN];
#pragma unroll
    for (int i = 0; i < XN; ++i) x[i] = X + (int64_t)min(bm + lr + 16 * i, M - 1) * ldx + 4 * q;
#pragma unroll
    for (int i = 0; i < WN; ++i) w[i] = W + (int64_t)min(bn + lr + 16 * i, N - 1) * ldw + 4 * q;
    float4 xr[XN], wr[WN];
    auto request = [&](int k0) {
        const bool there = k0 + 4 * q < K;
#pragma unroll
        for (int i = 0; i < XN; ++i)
            xr[i] = there ? *reinterpret_cast<const float4*>(x[i] + k0) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < WN; ++i)
            wr[i] = there ? *reinterpret_cast<const float4*>(w[i] + k0) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    auto store = [&](int buf) {
#pragma unroll
        for (int i = 0; i < XN; ++i)
#pragma unroll
            for (int k = 0; k < 4; ++k) xs[buf][4 * q + k][(lr + 16 * i + 8 * q) % WIDE] = part(xr[i], k);
#pragma unroll
        for (int i = 0; i < WN; ++i)
#pragma unroll
            for (int k = 0; k < 4; ++k) ws[buf][4 * q + k][(lr + 16 * i + 8 * q) % WIDE] = part(wr[i], k);
    };
    // rows ty .. + 3 and 32 + ty .., columns tx .. and 32 + (TN - 4) / 4 tx ..
    float acc[8][TN];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
    request(0);
    store(0);
    __syncthreads();
    for (int k0 = 0, buf = 0; k0 < K; k0 += WK, buf ^= 1) {
        if (k0 + WK < K) request(k0 + WK);
#pragma unroll
        for (int k = 0; k < WK; ++k) {
            const int shift = 8 * (k / 4);
            const int a0 = (ty + shift) % WIDE, b0 = (tx + shift) % WIDE;
            float a[8], b[TN];
            *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(&xs[buf][k][a0]);
            *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(&xs[buf][k][a0 ^ 32]);
            *reinterpret_cast<float4*>(b) = *reinterpret_cast<const float4*>(&ws[buf][k][b0]);
            if constexpr (TN == 8)
                *reinterpret_cast<float4*>(b + 4) = *reinterpret_cast<const float4*>(&ws[buf][k][b0 ^ 32]);
            if constexpr (TN == 6)
                *reinterpret_cast<float2*>(b + 4) =
                    *reinterpret_cast<const float2*>(&ws[buf][k][(32 + tx / 2 + shift) % WIDE]);
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        if (k0 + WK < K) store(buf ^ 1);
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = bm + ty + i % 4 + i / 4 * 32;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = bn + (j < 4 ? tx + j : 32 + tx * (TN - 4) / 4 + j - 4);
            if (n < N) Y[(int64_t)m * ldy + n] = acc[i][j];
        }
    }
}

template <int TN>
static int launch_wide(const float* X, const float* W, float* Y, int M, int N, int K, int64_t ldx, int64_t ldw,
                       int64_t ldy, cudaStream_t stream) {
    const dim3 tiles((N + 8 * TN - 1) / (8 * TN), (M + WIDE - 1) / WIDE);
    if (tiles.y > 65535) return (int)cudaErrorInvalidValue;
    gemm_f32_wide_kernel<TN><<<tiles, WIDE, 0, stream>>>(X, W, Y, M, N, K, ldx, ldw, ldy);
    SLLM_LAUNCH_CHECK();
    return 0;
}

template <int BM, int BN, int TM, int TN, int BK, int STAGES>
static int launch_f32(const float* X, const float* W, float* Y, int M, int N, int K, int64_t ldx, int64_t ldw,
                      int64_t ldy, cudaStream_t stream) {
    constexpr int smem = STAGES * (BM + BN) * (BK + 4) * 4;
    auto kernel = gemm_f32_kernel<BM, BN, TM, TN, BK, STAGES>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) return (int)cudaErrorInvalidValue;
    kernel<<<grid, (BM / TM) * (BN / TN), smem, stream>>>(X, W, Y, M, N, K, ldx, ldw, ldy);
    SLLM_LAUNCH_CHECK();
    return 0;
}

// Columns of the wide kernel's tiles for M > 16 rows of X by N of W, or 0 where the ring's tiles of 32 x 32 take less, by
// what the SM with the most tiles takes (in units of 0.138 us at K = 2,048).  The ring: rounds of two tiles an SM (65
// tokens by 6,144, 576 tiles: 95 us, 122 in wide tiles 48 columns across; by 8,192, 768: 135 and, 32 across, 151; 256 by
// 3,072, 768: 136 and, 48 across, 123).  Wide tiles: rounds of six (twelve warps, three a scheduler); one or two
// tiles take half a full round, three or four 0.73 of it, latencies being hidden less.  A narrow tile reads more of shared
// memory per multiply-add (777 tokens by 3,072: 320 us 64 across, 257 so).  Where no other row of tiles reads the
// weights again, weights beyond what the L2 is sure to hold come late, which the ring's loads stay further ahead of (33
// tokens by 12,288: 135 us, 158 in wide tiles; K = 256: 20.4 and 18.2).  Measured over 17 to 2,048 tokens by 512 to 65,536.
static int wide_columns(int M, int N, int K, int n_sm) {
    static const int tail[6] = {0, 15, 15, 22, 22, 30};
    const auto per_sm = [&](int rows, int cols) {
        return ((int64_t)((M + rows - 1) / rows) * ((N + cols - 1) / cols) + n_sm - 1) / n_sm;
    };
    int best = 0;
    int64_t least = (per_sm(32, 32) + 1) / 2 * (K < 512 ? 345 : 327);      // (its ring fills and empties)
    for (int tn = 8; tn >= 4; tn -= 2) {
        const int64_t tiles = per_sm(WIDE, 8 * tn);
        int64_t cost = (tiles / 6 * 30 + tail[tiles % 6]) * (tn == 8 ? 80 : tn == 6 ? 62 : 48);
        if (M <= WIDE && (int64_t)N * K >= 1 << 24) cost += cost / 5;
        if (cost < least) { best = 8 * tn; least = cost; }
    }
    return best;
}

}  // namespace sllm

using namespace sllm;

// The columns of the wide kernel's tiles, 0: another kernel.
SLLM_EXPORT int sllm_gemm_simt_columns(int M, int N, int K, int n_sm) { return M > 16 ? wide_columns(M, N, K, n_sm) : 0; }

// in_dtype / out_dtype: 0 = float32, 1 = bfloat16.  Supported: (0,0), (1,1), (1,0).
SLLM_EXPORT int sllm_gemm_simt(const void* X, const void* W, void* Y, int M, int N, int K,
                               int64_t ldx, int64_t ldw, int64_t ldy, int in_dtype,
                               int out_dtype, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return (int)cudaErrorInvalidValue;
    if (in_dtype == 0 && out_dtype == 0 && K % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 &&
        !(((uintptr_t)X | (uintptr_t)W) & 15)) {
        const auto x = (const float*)X, w = (const float*)W;
        const auto y = (float*)Y;
        if (M <= 16) return launch_f32<16, 16, 2, 2, 64, 4>(x, w, y, M, N, K, ldx, ldw, ldy, stream);
        int dev = 0, n_sm = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            return (int)cudaErrorInvalidDevice;
        switch (wide_columns(M, N, K, n_sm)) {
        case 64: return launch_wide<8>(x, w, y, M, N, K, ldx, ldw, ldy, stream);
        case 48: return launch_wide<6>(x, w, y, M, N, K, ldx, ldw, ldy, stream);
        case 32: return launch_wide<4>(x, w, y, M, N, K, ldx, ldw, ldy, stream);
        }
        return launch_f32<32, 32, 4, 4, 32, 4>(x, w, y, M, N, K, ldx, ldw, ldy, stream);
    }
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) return (int)cudaErrorInvalidValue;
    if (in_dtype == 0 && out_dtype == 0)
        gemm_simt_kernel<float, float><<<grid, 256, 0, stream>>>(
            (const float*)X, (const float*)W, (float*)Y, M, N, K, ldx, ldw, ldy);
    else if (in_dtype == 1 && out_dtype == 1)
        gemm_simt_kernel<__nv_bfloat16, __nv_bfloat16><<<grid, 256, 0, stream>>>(
            (const __nv_bfloat16*)X, (const __nv_bfloat16*)W, (__nv_bfloat16*)Y, M, N, K, ldx,
            ldw, ldy);
    else if (in_dtype == 1 && out_dtype == 0)
        gemm_simt_kernel<__nv_bfloat16, float><<<grid, 256, 0, stream>>>(
            (const __nv_bfloat16*)X, (const __nv_bfloat16*)W, (float*)Y, M, N, K, ldx, ldw, ldy);
    else
        return (int)cudaErrorInvalidValue;
    SLLM_LAUNCH_CHECK();
    return 0;
}
