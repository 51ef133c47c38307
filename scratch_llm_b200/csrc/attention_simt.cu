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
// Quads of keys and of values that a thread requests before it stores them: left to the compiler, a request
// waited for the stores before it (777 tokens, 32 heads of 128: 347 us, 316 so; a decoded token 418, 226).
constexpr int TRIPS = (HD + 15) / 16 <= 5 ? (HD + 15) / 16 : 4;
constexpr bool PAIRS = HD % 64 == 0; // a lane's dims are pairs of neighbours
// Queries of a warp: a read of a key or a value in shared memory serves all of them, and a tile of keys
// that a CTA fetches serves WARPS times as many.  Eight for long portions, where registers and shared
// memory hold them; one for rows of a few tokens, whose other queries would be worked on for nothing.
// 777 tokens, 32 heads of 64: 317 us with four queries a warp and a read per operand, 213 with eight, 178 with the
// blocks of the most keys first over all heads (heads of 128: 313 and 249).
constexpr int LONG_QUERIES = HD <= 128 ? 8 : 4;

constexpr size_t smem_floats(int rpw) {
    return (size_t)WARPS * rpw * HD + (size_t)BKV * KS_LD + (size_t)BKV * HD + (size_t)WARPS * rpw * BKV;
}

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
// of the cache: read-only loads, which leave together however many stores lie between them
__device__ __forceinline__ float4 fetch4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 fetch4(const __nv_bfloat16* p) {
    const uint2 r = __ldg(reinterpret_cast<const uint2*>(p));
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&r);
    return make_float4(__low2float(h[0]), __high2float(h[0]), __low2float(h[1]), __high2float(h[1]));
}

struct Args {
    int64_t q_stride, out_stride;
    int table_stride, page_size;
    int H, G;
    float scale, softcap;
    int window, chunk, planes;
    int vec;                             // pages allow reads of four elements
};

// Queries q0 .. q0 + nq - 1 of row r, RPW a warp.  Every query is one chain over the dims per score and over
// the keys per output, whatever RPW is.
template <typename T, int RPW>
__device__ __forceinline__ void
attend(const T* __restrict__ q, const T* __restrict__ pages, const int* __restrict__ table, int pos0,
       T* __restrict__ out, float slope, const float* __restrict__ sinks, const Args& args, float* smem,
       long long* key_base, int h, int t0, int q0, int nq) {
    constexpr int BQ = WARPS * RPW;
    const int page_size = args.page_size, planes = args.planes, G = args.G, window = args.window, chunk = args.chunk;
    const float scale = args.scale, softcap = args.softcap;
    float* Qs = smem;                    // [BQ][HD]
    float* Ks = Qs + BQ * HD;            // [BKV][KS_LD]
    float* Vs = Ks + BKV * KS_LD;        // [BKV][HD]
    float* Ss = Vs + BKV * HD;           // [WARPS][BKV][RPW]: probabilities
    const int g = h / (args.H / G);
    const int first_pos = pos0 + q0;
    const int last_pos = first_pos + nq - 1;
    int k_lo = 0;
    if (window > 0) k_lo = max(0, first_pos - window + 1) / BKV * BKV;
    if (chunk > 0) k_lo = max(k_lo, first_pos / chunk * chunk / BKV * BKV);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    for (int idx = tid; idx < BQ * HD; idx += THREADS) {
        const int i = idx / HD, d = idx - i * HD;
        Qs[idx] = i < nq ? to_float(__ldg(q + (int64_t)(t0 + q0 + i) * args.q_stride + (int64_t)h * HD + d))
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

    auto sees = [&](int a, int kpos) {             // query a of this warp, the key at that position
        const int i = warp + WARPS * a, qpos = first_pos + i;
        return i < nq && kpos <= qpos && (window <= 0 || kpos > qpos - window) &&
               (chunk <= 0 || kpos >= qpos / chunk * chunk);
    };
    auto dim = [&](int c) { return PAIRS ? 32 * (c & ~1) + 2 * lane + (c & 1) : lane + 32 * c; };   // of entry c
    for (int kt = k_lo; kt <= last_pos; kt += BKV) {
        __syncthreads();  // the previous tile's Ks / Vs / key_base are no longer read
        if (tid < BKV) {
            const int kpos = kt + tid;
            long long base = -1;
            if (kpos <= last_pos) {
                const int page = table[kpos / page_size];
                if (page >= 0)
                    base = (((long long)page * planes * G + g) * page_size + kpos % page_size) * HD;
            }
            key_base[tid] = base;
        }
        __syncthreads();
        float odd = 0.f;                 // NaN if a value of the tile is an infinity or a NaN
        if (QUADS && args.vec) {
            for (int at = tid; at < BKV * HD / 4; at += TRIPS * THREADS) {      // all requests, then all stores
                float4 kv[TRIPS], vv[TRIPS];
#pragma unroll
                for (int u = 0; u < TRIPS; ++u) {
                    const int idx = at + u * THREADS, j = idx / (HD / 4), d = (idx - j * (HD / 4)) * 4;
                    kv[u] = vv[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                    const long long base = idx < BKV * HD / 4 ? key_base[j] : -1;
                    if (base >= 0) {
                        kv[u] = fetch4(pages + base + d);
                        vv[u] = fetch4(pages + base + v_offset + d);
                    }
                }
#pragma unroll
                for (int u = 0; u < TRIPS; ++u) {
                    const int idx = at + u * THREADS, j = idx / (HD / 4), d = (idx - j * (HD / 4)) * 4;
                    if (idx < BKV * HD / 4) {
                        *reinterpret_cast<float4*>(Ks + j * KS_LD + d) = kv[u];
                        *reinterpret_cast<float4*>(Vs + j * HD + d) = vv[u];
                        odd = fmaf(vv[u].x, 0.f, fmaf(vv[u].y, 0.f, fmaf(vv[u].z, 0.f, fmaf(vv[u].w, 0.f, odd))));
                    }
                }
            }
        } else {
            for (int idx = tid; idx < BKV * HD; idx += THREADS) {
                const int j = idx / HD, d = idx - j * HD;
                const long long base = key_base[j];
                float kv = 0.f, vv = 0.f;
                if (base >= 0) {
                    kv = to_float(__ldg(pages + base + d));
                    vv = to_float(__ldg(pages + base + v_offset + d));
                }
                Ks[j * KS_LD + d] = kv;
                Vs[j * HD + d] = vv;
                odd = fmaf(vv, 0.f, odd);
            }
        }
        const bool guard = __syncthreads_or(odd != 0.f);

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
            const int qpos = first_pos + warp + WARPS * a;
            const bool valid = sees(a, kpos) && there;
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
        if (guard) {   // zero times such a value is not zero: a query leaves out the keys that it does not see
#pragma unroll 1
            for (int j = 0; j < BKV; ++j) {
#pragma unroll
                for (int a = 0; a < RPW; ++a) {
                    const float p = ps[j * RPW + a];
                    if (!sees(a, kt + j)) continue;
#pragma unroll
                    for (int c = 0; c < DPL; ++c) {
                        const int d = dim(c);
                        if (d < HD) acc[a][c] = fmaf(p, Vs[j * HD + d], acc[a][c]);
                    }
                }
            }
            continue;
        }
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
        T* o = out + (int64_t)(t0 + q0 + i) * args.out_stride + (int64_t)h * HD;
#pragma unroll
        for (int c = 0; c < DPL; ++c) {
            const int d = dim(c);
            if (d < HD) o[d] = from_float<T>(acc[a][c] * inv);
        }
    }
}

// Blocks of WARPS * MOST queries; a block with fewer (a row's last, a decoded token beside a prompt or in a
// padded step) takes as few a warp as they need.  Registers for the CTAs that an SM's shared memory holds.
// 64 rows of one token and 2,000 keys, 32 heads of 64 / 128, in a launch for 64 new tokens: 1,714 / 4,463 us with
// 16 queries a block, 1,934 / 3,142 with 32 that all blocks worked on, 663 / 1,208 so.
template <typename T, int MOST>
__global__ void __launch_bounds__(THREADS, HD <= 64 ? 5 : HD <= 128 ? 4 : 1)
attn_simt_kernel(const T* __restrict__ q, const T* __restrict__ pages, const int* __restrict__ block_table,
                 const int* __restrict__ row_start, const int* __restrict__ row_pos0, T* __restrict__ out,
                 const float* __restrict__ slopes, const float* __restrict__ sinks, const Args args) {
    extern __shared__ __align__(16) float smem[];
    __shared__ long long key_base[BKV];  // element offset of each key's K row, -1 if absent
    constexpr int BQ = WARPS * MOST;
    const int r = blockIdx.y, h = blockIdx.x % args.H;
    const int t0 = row_start[r], n_new = row_start[r + 1] - t0;
    // the queries with the most keys first, of all heads
    const int q0 = (gridDim.x - 1 - blockIdx.x) / args.H * BQ;
    if (q0 >= n_new) return;
    const int nq = min(BQ, n_new - q0);
    const int* table = block_table + (int64_t)r * args.table_stride;
    const float slope = slopes ? slopes[h] : 0.f;
    const int pos0 = row_pos0[r];
    if (MOST > 1 && nq <= WARPS)
        attend<T, 1>(q, pages, table, pos0, out, slope, sinks, args, smem, key_base, h, t0, q0, nq);
    else if (MOST > 4 && nq <= 4 * WARPS)
        attend<T, 4>(q, pages, table, pos0, out, slope, sinks, args, smem, key_base, h, t0, q0, nq);
    else
        attend<T, MOST>(q, pages, table, pos0, out, slope, sinks, args, smem, key_base, h, t0, q0, nq);
}

template <typename T, int MOST>
static int launch(const void* q, const void* pages, const int* block_table, const int* row_start,
                  const int* row_pos0, void* out, const float* slopes, const float* sinks, const Args& args,
                  int n_rows, int max_new, cudaStream_t stream) {
    const size_t smem = smem_floats(MOST) * sizeof(float);
    const cudaError_t e = cudaFuncSetAttribute(attn_simt_kernel<T, MOST>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    constexpr int BQ = WARPS * MOST;
    attn_simt_kernel<T, MOST><<<dim3(args.H * ((max_new + BQ - 1) / BQ), n_rows), THREADS, smem, stream>>>(
        (const T*)q, (const T*)pages, block_table, row_start, row_pos0, (T*)out, slopes, sinks, args);
    SLLM_LAUNCH_CHECK();
    return 0;
}

// max_new decides the shared memory and the number of blocks; what a block computes with goes by its own queries.
template <typename T, typename... Rest>
static int launch_for(int max_new, Rest... rest) {
    if (max_new <= WARPS) return launch<T, 1>(rest...);
    if (max_new <= 4 * WARPS) return launch<T, 4>(rest...);
    return launch<T, LONG_QUERIES>(rest...);
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
    const Args args = {q_stride, out_stride, table_stride, page_size, H, G, scale, softcap, window, chunk, planes,
                       ((uintptr_t)pages & 15) == 0};
    if (dtype == 0)
        return launch_for<float>(max_new, q, pages, block_table, row_start, row_pos0, out, slopes, sinks, args,
                                 n_rows, max_new, stream);
    if (dtype == 1)
        return launch_for<__nv_bfloat16>(max_new, q, pages, block_table, row_start, row_pos0, out, slopes, sinks,
                                         args, n_rows, max_new, stream);
    return (int)cudaErrorInvalidValue;
}
