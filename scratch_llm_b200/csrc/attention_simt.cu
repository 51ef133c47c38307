// Causal attention of a packed batch over the paged cache, on the CUDA cores in 32-bit
// arithmetic.  One kernel serves portions of prompts and single decoded tokens: the token at
// absolute position p of row r attends to keys 0..p of row r (or to the last `window` of
// them) through r's block table.  This is the attention of the 32-bit path for every head
// size, and of the bfloat16 path where no tensor-core kernel takes the shape.
//
// Restates src/scratch_llm/model.py:172-182 (scores = q k^T scaled, disallowed keys -inf,
// max-subtracted softmax in 32-bit, times v) and :330-345 (query head h reads kv head
// h / (H/G); key j is visible to the query at position p iff j <= p) of the reference, with
// the online softmax of its paged kernel (src/scratch_llm/kernels/attention/decode/paged.py:49-83).
//
// Keys are consumed in tiles of 32 that are aligned to absolute positions, in ascending
// order, so a query's result does not depend on how its prompt was cut or on its neighbours.
// Compiled once per head size: -DSLLM_HEAD_DIM=<1 to 640>.
#include "common.cuh"

#ifndef SLLM_HEAD_DIM
#error "compile with -DSLLM_HEAD_DIM=<head size>"
#endif

namespace sllm {

constexpr int HD = SLLM_HEAD_DIM;
static_assert(HD >= 1 && HD <= 640, "head size: 1 to 640");
constexpr int BKV = 32, THREADS = 128, WARPS = THREADS / 32;
constexpr int DPL = (HD + 31) / 32;  // head dims per lane
constexpr bool QUADS = HD % 4 == 0;  // rows of whole 16-byte words
constexpr int KS_LD = QUADS ? HD + 4 : HD + 1;     // (neighbouring keys start on other banks)
constexpr bool PAIRS = HD % 64 == 0; // a lane's dims are pairs of neighbours
// Queries of a warp: a read of a key or a value in shared memory serves all of them, and a tile of keys
// that a CTA fetches serves WARPS times as many.  Eight for long portions, where registers and shared
// memory hold them; one for steps of a few tokens, whose other queries would be worked on for nothing.
// 777 tokens, 32 heads of 64: 317 us with four queries a warp and a read per operand, 220 with eight.
constexpr int LONG_QUERIES = HD <= 128 ? 8 : 4;

constexpr size_t smem_floats(int rpw) {
    return (size_t)WARPS * rpw * HD + (size_t)BKV * KS_LD + (size_t)BKV * HD + (size_t)WARPS * rpw * BKV;
}

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
    const uint2 r = *reinterpret_cast<const uint2*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&r);
    return make_float4(__low2float(h[0]), __high2float(h[0]), __low2float(h[1]), __high2float(h[1]));
}

// RPW queries a warp.  vec: pages allow reads of four elements.  Every query is one chain over the dims per
// score and over the keys per output, whatever RPW is.
template <typename T, int RPW>
__global__ void __launch_bounds__(THREADS)
attn_simt_kernel(const T* __restrict__ q, int64_t q_stride, const T* __restrict__ pages,
                 const int* __restrict__ block_table, int table_stride, int page_size,
                 const int* __restrict__ row_start, const int* __restrict__ row_pos0,
                 T* __restrict__ out, int64_t out_stride, int H, int G, float scale, int window,
                 const float* __restrict__ slopes, const float* __restrict__ sinks, int planes,
                 float softcap, int chunk, int vec) {
    constexpr int BQ = WARPS * RPW;
    extern __shared__ __align__(16) float smem[];
    __shared__ long long key_base[BKV];  // element offset of each key's K row, -1 if absent
    float* Qs = smem;                    // [BQ][HD]
    float* Ks = Qs + BQ * HD;            // [BKV][KS_LD]
    float* Vs = Ks + BKV * KS_LD;        // [BKV][HD]
    float* Ss = Vs + BKV * HD;           // [WARPS][BKV][RPW]: probabilities

    const int r = blockIdx.y, h = blockIdx.z;
    const int g = h / (H / G);
    const int t0 = row_start[r];
    const int n_new = row_start[r + 1] - t0;
    const int q0 = (gridDim.x - 1 - blockIdx.x) * BQ;    // the queries with the most keys first
    if (q0 >= n_new) return;
    const int nq = min(BQ, n_new - q0);
    const int first_pos = row_pos0[r] + q0;
    const int last_pos = first_pos + nq - 1;
    int k_lo = 0;
    if (window > 0) k_lo = max(0, first_pos - window + 1) / BKV * BKV;
    if (chunk > 0) k_lo = max(k_lo, first_pos / chunk * chunk / BKV * BKV);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const float slope = slopes ? slopes[h] : 0.f;

    for (int idx = tid; idx < BQ * HD; idx += THREADS) {
        const int i = idx / HD, d = idx - i * HD;
        Qs[idx] = i < nq ? to_float(q[(int64_t)(t0 + q0 + i) * q_stride + (int64_t)h * HD + d])
                         : 0.f;
    }

    float m[RPW], l[RPW], acc[RPW][DPL];
#pragma unroll
    for (int a = 0; a < RPW; ++a) {
        m[a] = -INFINITY;
        l[a] = 0.f;
#pragma unroll
        for (int c = 0; c < DPL; ++c) acc[a][c] = 0.f;
    }
    // (one plane: the values are the leading entries of the keys themselves)
    const int64_t v_offset = (int64_t)(planes - 1) * G * page_size * HD;
    const float* qs = Qs + warp * HD;              // query a of this warp: row warp + WARPS * a
    const float* kj = Ks + lane * KS_LD;
    float* ps = Ss + warp * BKV * RPW;

    for (int kt = k_lo; kt <= last_pos; kt += BKV) {
        __syncthreads();  // the previous tile's Ks / Vs / key_base are no longer read
        if (tid < BKV) {
            const int kpos = kt + tid;
            long long base = -1;
            if (kpos <= last_pos) {
                const int page = block_table[(int64_t)r * table_stride + kpos / page_size];
                if (page >= 0)
                    base = (((long long)page * planes * G + g) * page_size + kpos % page_size) * HD;
            }
            key_base[tid] = base;
        }
        __syncthreads();
        if (QUADS && vec) {
#pragma unroll 4
            for (int idx = tid; idx < BKV * HD / 4; idx += THREADS) {
                const int j = idx / (HD / 4), d = (idx - j * (HD / 4)) * 4;
                const long long base = key_base[j];
                float4 kv = make_float4(0.f, 0.f, 0.f, 0.f), vv = kv;
                if (base >= 0) {
                    kv = load4(pages + base + d);
                    vv = load4(pages + base + v_offset + d);
                }
                *reinterpret_cast<float4*>(Ks + j * KS_LD + d) = kv;
                *reinterpret_cast<float4*>(Vs + j * HD + d) = vv;
            }
        } else {
            for (int idx = tid; idx < BKV * HD; idx += THREADS) {
                const int j = idx / HD, d = idx - j * HD;
                const long long base = key_base[j];
                float kv = 0.f, vv = 0.f;
                if (base >= 0) {
                    kv = to_float(pages[base + d]);
                    vv = to_float(pages[base + v_offset + d]);
                }
                Ks[j * KS_LD + d] = kv;
                Vs[j * HD + d] = vv;
            }
        }
        __syncthreads();

        const int kpos = kt + lane;
        float dot[RPW];
#pragma unroll
        for (int a = 0; a < RPW; ++a) dot[a] = 0.f;
        if (QUADS) {
#pragma unroll 4
            for (int d = 0; d < HD; d += 4) {
                const float4 k = load4(kj + d);
#pragma unroll
                for (int a = 0; a < RPW; ++a) {
                    const float4 x = load4(qs + a * WARPS * HD + d);
                    dot[a] = fmaf(x.w, k.w, fmaf(x.z, k.z, fmaf(x.y, k.y, fmaf(x.x, k.x, dot[a]))));
                }
            }
        } else {
#pragma unroll 4
            for (int d = 0; d < HD; ++d) {
                const float k = kj[d];
#pragma unroll
                for (int a = 0; a < RPW; ++a) dot[a] = fmaf(qs[a * WARPS * HD + d], k, dot[a]);
            }
        }
        const bool there = key_base[lane] >= 0;
#pragma unroll
        for (int a = 0; a < RPW; ++a) {
            const int i = warp + WARPS * a, qpos = first_pos + i;
            const bool valid = i < nq && kpos <= qpos && (window <= 0 || kpos > qpos - window) &&
                               (chunk <= 0 || kpos >= qpos / chunk * chunk) && there;
            float sc = dot[a] * scale;
            if (softcap > 0.f) sc = softcap * tanhf(sc / softcap);
            const float s = valid ? sc - slope * (float)(qpos - kpos) : -INFINITY;
            const float m_new = fmaxf(m[a], warp_max(s));
            float p = 0.f, corr = 1.f;
            if (m_new != -INFINITY) {
                p = expf(s - m_new);        // s = -inf gives 0
                corr = expf(m[a] - m_new);  // m = -inf gives 0
            }
            l[a] = l[a] * corr + warp_sum(p);
            m[a] = m_new;
#pragma unroll
            for (int c = 0; c < DPL; ++c) acc[a][c] *= corr;
            ps[lane * RPW + a] = p;
        }
        __syncwarp();  // each warp reads back only what it wrote
#pragma unroll 4
        for (int j = 0; j < BKV; ++j) {
            float p[RPW];
            if (RPW % 4 == 0) {
#pragma unroll
                for (int a = 0; a < RPW; a += 4) {
                    const float4 x = load4(ps + j * RPW + a);
                    p[a] = x.x; p[a + 1] = x.y; p[a + 2] = x.z; p[a + 3] = x.w;
                }
            } else {
#pragma unroll
                for (int a = 0; a < RPW; ++a) p[a] = ps[j * RPW + a];
            }
#pragma unroll
            for (int c = 0; c < DPL; ++c) {
                if (PAIRS) {          // dims 32 c + 2 lane and the next, in the entries c and c + 1
                    if (c % 2) continue;
                    const float2 v = *reinterpret_cast<const float2*>(Vs + j * HD + 32 * c + 2 * lane);
#pragma unroll
                    for (int a = 0; a < RPW; ++a) {
                        acc[a][c] = fmaf(p[a], v.x, acc[a][c]);
                        acc[a][c + 1] = fmaf(p[a], v.y, acc[a][c + 1]);
                    }
                } else {
                    const int d = lane + 32 * c;
                    if (d < HD) {
                        const float v = Vs[j * HD + d];
#pragma unroll
                        for (int a = 0; a < RPW; ++a) acc[a][c] = fmaf(p[a], v, acc[a][c]);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int a = 0; a < RPW; ++a) {
        const int i = warp + WARPS * a;
        if (i >= nq) continue;
        float total = l[a], keep = 1.f;
        if (sinks && m[a] != -INFINITY) {
            // the sink: one more term of the denominator, without a key or a value
            const float sink = sinks[h], top = fmaxf(m[a], sink);
            keep = expf(m[a] - top);
            total = total * keep + expf(sink - top);
        }
        const float inv = total > 0.f ? keep / total : 0.f;
        T* o = out + (int64_t)(t0 + q0 + i) * out_stride + (int64_t)h * HD;
#pragma unroll
        for (int c = 0; c < DPL; ++c) {
            const int d = PAIRS ? 32 * (c & ~1) + 2 * lane + (c & 1) : lane + 32 * c;
            if (d < HD) o[d] = from_float<T>(acc[a][c] * inv);
        }
    }
}

template <typename T, int RPW>
static int launch(const void* q, int64_t q_stride, const void* pages, const int* block_table, int table_stride,
                  int page_size, const int* row_start, const int* row_pos0, void* out, int64_t out_stride,
                  int n_rows, int max_new, int H, int G, float scale, int window, const float* slopes,
                  const float* sinks, int planes, float softcap, int chunk, cudaStream_t stream) {
    const size_t smem = smem_floats(RPW) * sizeof(float);
    const cudaError_t e = cudaFuncSetAttribute(attn_simt_kernel<T, RPW>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    constexpr int BQ = WARPS * RPW;
    const int vec = ((uintptr_t)pages & 15) == 0;
    attn_simt_kernel<T, RPW><<<dim3((max_new + BQ - 1) / BQ, n_rows, H), THREADS, smem, stream>>>(
        (const T*)q, q_stride, (const T*)pages, block_table, table_stride, page_size, row_start, row_pos0,
        (T*)out, out_stride, H, G, scale, window, slopes, sinks, planes, softcap, chunk, vec);
    SLLM_LAUNCH_CHECK();
    return 0;
}

template <typename T, typename... Args>
static int launch_for(int max_new, Args... args) {
    if (max_new <= WARPS) return launch<T, 1>(args...);
    if (max_new <= 4 * WARPS) return launch<T, 4>(args...);
    return launch<T, LONG_QUERIES>(args...);
}

}  // namespace sllm

using namespace sllm;

SLLM_EXPORT int sllm_attn_simt_head_dim() { return HD; }

// q: [n_tokens, q_stride] with head h at columns [h*HD, (h+1)*HD); out likewise.
// pages: [n_pages, planes, G, page_size, HD]; planes = 2: keys, then values; planes = 1: one
// vector per token that is its key and, by its leading entries, its value.  block_table: [n_rows, table_stride], -1 = no page.
// row_start: [n_rows + 1] token offsets; row_pos0: [n_rows] position of each row's first token.
// max_new: the largest number of new tokens of any row.  window: 0 = all keys.
// slopes (may be null): float [H]; slopes[h] * (query position - key position) is taken off the
// scaled score of head h.  sinks (may be null): float [H]; exp(sinks[h]) is added to the softmax's
// denominator of head h, once, with no value behind it.  softcap > 0: the scaled score s becomes
// softcap * tanh(s / softcap) (before the slopes).  chunk > 0: the query at position p sees only
// keys from floor(p / chunk) * chunk on (positions count from the sequence's start).
SLLM_EXPORT int sllm_attn_simt(const void* q, int64_t q_stride, const void* pages,
                               const int* block_table, int table_stride, int page_size,
                               const int* row_start, const int* row_pos0, void* out,
                               int64_t out_stride, int n_rows, int max_new, int H, int G,
                               float scale, int window, const float* slopes, const float* sinks,
                               int planes, float softcap, int chunk, int dtype,
                               cudaStream_t stream) {
    if (n_rows <= 0 || max_new <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G != 0 || page_size <= 0 || window < 0 || chunk < 0 || planes < 1 || planes > 2)
        return (int)cudaErrorInvalidValue;
    if (n_rows > 65535 || H > 65535) return (int)cudaErrorInvalidValue;
    if (dtype == 0)
        return launch_for<float>(max_new, q, q_stride, pages, block_table, table_stride, page_size, row_start,
                                 row_pos0, out, out_stride, n_rows, max_new, H, G, scale, window, slopes, sinks,
                                 planes, softcap, chunk, stream);
    if (dtype == 1)
        return launch_for<__nv_bfloat16>(max_new, q, q_stride, pages, block_table, table_stride, page_size,
                                         row_start, row_pos0, out, out_stride, n_rows, max_new, H, G, scale,
                                         window, slopes, sinks, planes, softcap, chunk, stream);
    return (int)cudaErrorInvalidValue;
}
