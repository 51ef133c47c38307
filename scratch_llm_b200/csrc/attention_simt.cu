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

__device__ __forceinline__ float capped(float score, float cap) { return cap * tanhf(score / cap); }
__device__ __forceinline__ bool visible(int qpos, int kpos, int window, int chunk) {
    return kpos <= qpos && (window <= 0 || kpos > qpos - window) && (chunk <= 0 || kpos >= qpos / chunk * chunk);
}
// What a query's sums are multiplied with at the end, from its maximum and its denominator.
__device__ __forceinline__ float last_factor(float m, float l, const float* sinks, int h) {
    float total = l, keep = 1.f;
    if (sinks && m != -INFINITY) {
        // the sink: one more term of the denominator, without a key or a value
        const float sink = sinks[h], top = fmaxf(m, sink);
        keep = expf(m - top);
        total = total * keep + expf(sink - top);
    }
    return total > 0.f ? keep / total : 0.f;
}

// Queries q0 .. q0 + nq - 1 of row r, RPW a warp.  Every query is one chain over the dims per score and over
// the keys per output, whatever RPW is.
template <typename T, int RPW>
__device__ __forceinline__ void
attend(const T* __restrict__ q, const T* __restrict__ pages, const int* __restrict__ table, int pos0,
       T* __restrict__ out, float slope, const float* __restrict__ sinks, const Args& args, float* smem,
       long long* key_base, int h, int t0, int q0, int nq) {
    constexpr int BQ = WARPS * RPW;
    const int page_size = args.page_size, planes = args.planes, G = args.G, window = args.window, chunk = args.chunk;
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
        return i < nq && visible(qpos, kpos, window, chunk);
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
            float sc = dot[a] * args.scale;
            if (args.softcap > 0.f) sc = capped(sc, args.softcap);
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
        const float inv = last_factor(m[a], l[a], sinks, h);
        T* o = out + (int64_t)(t0 + q0 + i) * args.out_stride + (int64_t)h * HD;
#pragma unroll
        for (int c = 0; c < DPL; ++c) {
            const int d = dim(c);
            if (d < HD) o[d] = from_float<T>(acc[a][c] * inv);
        }
    }
}

// Long portions of 32-bit rows: a warp has TROWS consecutive tokens of one head, a thread TQ of them with 8
// of a tile's 32 keys (lane = 4 qg + kl: tokens qg + 8 i, keys kl + 4 m), then with a quarter of the
// dims: per four dims TQ + 8 reads of 16 bytes feed 32 TQ multiply-adds, where a key a lane took nine for
// 32, and the softmax's sums meet across four lanes instead of 32.  The four warps are the heads of one
// kv head where it has four, and share its tiles, which come a tile ahead (cp.async).  Every sum is the
// one that `attend` forms, in its order (the denominator's tree over a tile's keys: j + 16, 8, 4 within a
// thread, 2, 1 across lanes), so a token has the same bits on either way.  32 heads of 64, us with
// attn_simt_kernel and so: 100 tokens 22 / 21, 777 178 / 165, 2,048 914 / 658, 64 after 3,000 468 / 396; heads of
// 80, 777 tokens 275 / 195.  Heads of 128, of which half as many blocks fit an SM: 249 / 258, so not those.  Bound by
// shared memory (0.8 of its cycles on the fullest SM).  Four tokens a thread: 175 us at 777 tokens, 560 at 2,048, 587
// for 64 after 3,000.
#if SLLM_HEAD_DIM % 16 == 0 && SLLM_HEAD_DIM < 128
#define SLLM_TILED
constexpr int TQ = 2, TROWS = 8 * TQ;
constexpr int TLD = HD + 4;                        // row stride of queries and keys
constexpr int PLD = 24;                            // of a key's probabilities: token qg + 8 i stands at TQ qg + i
constexpr int TDQ = HD / 16;                       // quads of dims a thread: kl + 4 c
constexpr size_t tile_smem() {
    return sizeof(float) * ((size_t)WARPS * TROWS * TLD + 2 * BKV * TLD + 2 * BKV * HD + (size_t)WARPS * BKV * PLD);
}

// Rows of fewer than min_new tokens are left to attn_simt_kernel.  grid (H / heads x token blocks, rows),
// heads: of a kv head's query heads, 4, 2 or 1 to a CTA, with 1, 2 or 4 blocks of TROWS tokens.
__global__ void __launch_bounds__(THREADS, 2)
attn_simt_tile_kernel(const float* __restrict__ q, const float* __restrict__ pages, const int* __restrict__ block_table,
                      const int* __restrict__ row_start, const int* __restrict__ row_pos0, float* __restrict__ out,
                      const float* __restrict__ slopes, const float* __restrict__ sinks, const Args args,
                      int heads, int min_new) {
    extern __shared__ __align__(16) float smem[];
    __shared__ int there[2][BKV];
    const int r = blockIdx.y;
    const int t0 = row_start[r], n_new = row_start[r + 1] - t0;
    const int cta_rows = WARPS / heads * TROWS;
    const int groups = args.H / heads;
    // the tokens with the most keys first, of all heads
    const int q0 = (gridDim.x - 1 - blockIdx.x) / groups * cta_rows;
    if (n_new < min_new || q0 >= n_new) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, qg = lane >> 2, kl = lane & 3;
    const int h = blockIdx.x % groups * heads + warp % heads, w0 = q0 + warp / heads * TROWS;
    const int nq = max(0, min(TROWS, n_new - w0));
    const int pos0 = row_pos0[r], first_pos = pos0 + q0, last_pos = pos0 + min(q0 + cta_rows, n_new) - 1;
    const int window = args.window, chunk = args.chunk, page_size = args.page_size, planes = args.planes;
    const int G = args.G, g = h / (args.H / G);
    const float slope = slopes ? slopes[h] : 0.f;
    const int* table = block_table + (int64_t)r * args.table_stride;
    float* Qs = smem + warp * TROWS * TLD;             // [TROWS][TLD] of this warp
    float* Ks = smem + WARPS * TROWS * TLD;            // [2][BKV][TLD]
    float* Vs = Ks + 2 * BKV * TLD;                    // [2][BKV][HD]
    float* Ps = Vs + 2 * BKV * HD + warp * BKV * PLD;  // [BKV][PLD] of this warp
    int k_lo = 0;
    if (window > 0) k_lo = max(0, first_pos - window + 1) / BKV * BKV;
    if (chunk > 0) k_lo = max(k_lo, first_pos / chunk * chunk / BKV * BKV);

    // four neighbouring threads fetch a key and its value; the page of the tile after next is asked for early
    const int row = tid / 4, quad = tid % 4 * 4;
    const int64_t v_offset = (int64_t)(planes - 1) * G * page_size * HD;
    auto page_of = [&](int kt) { return kt + row <= last_pos ? table[(kt + row) / page_size] : -1; };
    auto request = [&](int kt, int page, int buf) {
        const int64_t base = (((int64_t)max(page, 0) * planes * G + g) * page_size + (kt + row) % page_size) * HD;
        const int bytes = page >= 0 ? 16 : 0;          // (no such key: zeros)
        const float* src = pages + (page >= 0 ? base : 0) + quad;
        const uint32_t k_dst = (uint32_t)__cvta_generic_to_shared(Ks + (buf * BKV + row) * TLD + quad);
        const uint32_t v_dst = (uint32_t)__cvta_generic_to_shared(Vs + (buf * BKV + row) * HD + quad);
#pragma unroll
        for (int c = 0; c < HD; c += 16) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(k_dst + 4 * c), "l"(src + c), "r"(bytes) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(v_dst + 4 * c),
                         "l"(src + (page >= 0 ? v_offset : 0) + c), "r"(bytes) : "memory");
        }
        if (quad == 0) there[buf][row] = page >= 0;
    };
    request(k_lo, page_of(k_lo), 0);
    int next_page = page_of(k_lo + BKV);
    for (int i = lane; i < TROWS * HD; i += 32) {
        const int t = i / HD, d = i - t * HD;
        Qs[t * TLD + d] = t < nq ? __ldg(q + (int64_t)(t0 + w0 + t) * args.q_stride + (int64_t)h * HD + d) : 0.f;
    }
    float m[TQ], l[TQ];
    float4 acc[TQ][TDQ];
#pragma unroll
    for (int i = 0; i < TQ; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < TDQ; ++c) acc[i][c] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const int w_pos = pos0 + w0, w_last = w_pos + nq - 1;
    int from[TQ], upto[TQ];              // the keys that a token sees; none for one that is not there
#pragma unroll
    for (int i = 0; i < TQ; ++i) {
        const int qpos = w_pos + qg + 8 * i;
        from[i] = max(window > 0 ? qpos - window + 1 : 0, chunk > 0 ? qpos / chunk * chunk : 0);
        upto[i] = qg + 8 * i < nq ? qpos : -1;
    }
    for (int kt = k_lo, buf = 0; kt <= last_pos; kt += BKV, buf ^= 1) {
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
        float odd = 0.f;                 // NaN if a value that this thread fetched is an infinity or a NaN
        const float* v_own = Vs + (buf * BKV + row) * HD + quad;
#pragma unroll
        for (int c = 0; c < HD; c += 16) {
            const float4 v = load4(v_own + c);
            odd = fmaf(v.x, 0.f, fmaf(v.y, 0.f, fmaf(v.z, 0.f, fmaf(v.w, 0.f, odd))));
        }
        // (the tile is there for all, and all are done with the one before it)
        const bool guard = __syncthreads_or(odd != 0.f);
        if (kt + BKV <= last_pos) {
            request(kt + BKV, next_page, buf ^ 1);
            next_page = page_of(kt + 2 * BKV);
        }
        if (nq == 0 || kt > w_last) continue;
        const float* kp = Ks + (buf * BKV + kl) * TLD;
        const float* qp = Qs + qg * TLD;
        float p[8][TQ];
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int i = 0; i < TQ; ++i) p[j][i] = 0.f;
#pragma unroll 4
        for (int d = 0; d < HD; d += 4) {
            float4 x[TQ];
#pragma unroll
            for (int i = 0; i < TQ; ++i) x[i] = load4(qp + 8 * i * TLD + d);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float4 k = load4(kp + 4 * j * TLD + d);
#pragma unroll
                for (int i = 0; i < TQ; ++i)
                    p[j][i] = fmaf(x[i].w, k.w, fmaf(x[i].z, k.z, fmaf(x[i].y, k.y, fmaf(x[i].x, k.x, p[j][i]))));
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int i = 0; i < TQ; ++i) p[j][i] = p[j][i] * args.scale;
        if (args.softcap > 0.f) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
#pragma unroll
                for (int i = 0; i < TQ; ++i) p[j][i] = capped(p[j][i], args.softcap);
        }
#pragma unroll
        for (int i = 0; i < TQ; ++i) {
            float top = -INFINITY;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int kpos = kt + kl + 4 * j;
                const bool valid = kpos >= from[i] && kpos <= upto[i] && there[buf][kl + 4 * j];
                p[j][i] = valid ? p[j][i] - slope * (float)(w_pos + qg + 8 * i - kpos) : -INFINITY;
                top = fmaxf(top, p[j][i]);
            }
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
            const float m_new = fmaxf(m[i], top);
            float corr = 1.f;
            if (m_new != -INFINITY) {
                corr = expf(m[i] - m_new);       // m = -inf gives 0
#pragma unroll
                for (int j = 0; j < 8; ++j) p[j][i] = expf(p[j][i] - m_new);     // -inf gives 0
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) p[j][i] = 0.f;
            }
            float a = (((p[0][i] + p[4][i]) + (p[2][i] + p[6][i])) + ((p[1][i] + p[5][i]) + (p[3][i] + p[7][i])));
            a += __shfl_xor_sync(0xffffffffu, a, 2);
            a += __shfl_xor_sync(0xffffffffu, a, 1);
            l[i] = l[i] * corr + a;
            m[i] = m_new;
#pragma unroll
            for (int c = 0; c < TDQ; ++c) {
                acc[i][c].x *= corr; acc[i][c].y *= corr; acc[i][c].z *= corr; acc[i][c].w *= corr;
            }
        }
        __syncwarp();  // (the tile before it is read)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float* to = Ps + (kl + 4 * j) * PLD + TQ * qg;
            *reinterpret_cast<float2*>(to) = make_float2(p[j][0], p[j][1]);
        }
        __syncwarp();
        const float* vp = Vs + buf * BKV * HD + 4 * kl;
        if (guard) {   // zero times such a value is not zero: a query leaves out the keys that it does not see
#pragma unroll 1
            for (int j = 0; j < BKV; ++j)
#pragma unroll
                for (int i = 0; i < TQ; ++i) {
                    if (kt + j < from[i] || kt + j > upto[i]) continue;
                    const float w = Ps[j * PLD + TQ * qg + i];
#pragma unroll
                    for (int c = 0; c < TDQ; ++c) {
                        const float4 v = load4(vp + j * HD + 16 * c);
                        float4& o = acc[i][c];
                        o.x = fmaf(w, v.x, o.x); o.y = fmaf(w, v.y, o.y); o.z = fmaf(w, v.z, o.z); o.w = fmaf(w, v.w, o.w);
                    }
                }
            continue;
        }
#pragma unroll 4
        for (int j = 0; j < BKV; ++j) {
            float w[TQ];
            *reinterpret_cast<float2*>(w) = *reinterpret_cast<const float2*>(Ps + j * PLD + TQ * qg);
#pragma unroll
            for (int c = 0; c < TDQ; ++c) {
                const float4 v = load4(vp + j * HD + 16 * c);
#pragma unroll
                for (int i = 0; i < TQ; ++i) {
                    float4& o = acc[i][c];
                    o.x = fmaf(w[i], v.x, o.x); o.y = fmaf(w[i], v.y, o.y); o.z = fmaf(w[i], v.z, o.z); o.w = fmaf(w[i], v.w, o.w);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < TQ; ++i) {
        if (qg + 8 * i >= nq) continue;
        const float inv = last_factor(m[i], l[i], sinks, h);
        float* o = out + (int64_t)(t0 + w0 + qg + 8 * i) * args.out_stride + (int64_t)h * HD + 4 * kl;
#pragma unroll
        for (int c = 0; c < TDQ; ++c) {
            o[16 * c] = acc[i][c].x * inv;
            o[16 * c + 1] = acc[i][c].y * inv;
            o[16 * c + 2] = acc[i][c].z * inv;
            o[16 * c + 3] = acc[i][c].w * inv;
        }
    }
}
#endif

// Blocks of WARPS * MOST queries; a block with fewer (a row's last, a decoded token beside a prompt or in a
// padded step) takes as few a warp as they need.  Registers for the CTAs that an SM's shared memory holds.
// 64 rows of one token and 2,000 keys, 32 heads of 64 / 128, in a launch for 64 new tokens: 1,714 / 4,463 us with
// 16 queries a block, 1,934 / 3,142 with 32 that all blocks worked on, 663 / 1,208 so.
template <typename T, int MOST>
__global__ void __launch_bounds__(THREADS, HD <= 64 ? 5 : HD <= 128 ? 4 : 1)
attn_simt_kernel(const T* __restrict__ q, const T* __restrict__ pages, const int* __restrict__ block_table,
                 const int* __restrict__ row_start, const int* __restrict__ row_pos0, T* __restrict__ out,
                 const float* __restrict__ slopes, const float* __restrict__ sinks, const Args args, int max_new,
                 int first_block) {
    extern __shared__ __align__(16) float smem[];
    __shared__ long long key_base[BKV];  // element offset of each key's K row, -1 if absent
    constexpr int BQ = WARPS * MOST;
    // (the head as it comes from the grid: as a remainder it took a register, and eight queries a warp spilled: 3-5 %)
    const int r = blockIdx.z, h = blockIdx.x;
    const int t0 = row_start[r], n_new = row_start[r + 1] - t0;
    // the queries with the most keys first, of all heads
    const int q0 = (first_block + gridDim.y - 1 - blockIdx.y) * BQ;
    if (q0 >= n_new || n_new > max_new) return;          // (longer rows: attn_simt_tile_kernel)
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
    constexpr int BQ = WARPS * MOST, AT_ONCE = 65535;
    for (int end = (max_new + BQ - 1) / BQ; end > 0; end -= AT_ONCE) {
        const int blocks = end < AT_ONCE ? end : AT_ONCE;
        attn_simt_kernel<T, MOST><<<dim3(args.H, blocks, n_rows), THREADS, smem, stream>>>(
            (const T*)q, (const T*)pages, block_table, row_start, row_pos0, (T*)out, slopes, sinks, args, max_new,
            end - blocks);
        SLLM_LAUNCH_CHECK();
    }
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
// n_tokens: of all rows; max_new: the largest number of new tokens of any row.  window: 0 = all keys.
// slopes (may be null): float [H]; slopes[h] * (query position - key position) is taken off the
// scaled score of head h.  sinks (may be null): float [H]; exp(sinks[h]) is added to the softmax's
// denominator of head h, once, with no value behind it.  softcap > 0: the scaled score s becomes
// softcap * tanh(s / softcap) (before the slopes).  chunk > 0: the query at position p sees only
// keys from floor(p / chunk) * chunk on (positions count from the sequence's start).
SLLM_EXPORT int sllm_attn_simt(const void* q, int64_t q_stride, const void* pages,
                               const int* block_table, int table_stride, int page_size,
                               const int* row_start, const int* row_pos0, void* out,
                               int64_t out_stride, int n_rows, int n_tokens, int max_new, int H, int G,
                               float scale, int window, const float* slopes, const float* sinks,
                               int planes, float softcap, int chunk, int dtype,
                               cudaStream_t stream) {
    if (n_rows <= 0 || max_new <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G != 0 || page_size <= 0 || window < 0 || chunk < 0 || planes < 1 || planes > 2)
        return (int)cudaErrorInvalidValue;
    if (n_rows > 65535 || H > 65535) return (int)cudaErrorInvalidValue;
    const Args args = {q_stride, out_stride, table_stride, page_size, H, G, scale, softcap, window, chunk, planes,
                       ((uintptr_t)pages & 15) == 0};
#ifdef SLLM_TILED
    // 32-bit rows whose pages and heads are whole 16-byte words.  us with attn_simt_kernel and so: a row of 48 tokens
    // without keys before them, 32 heads of 64 on 8 kv heads 11.8 / 14.7, of 112 13.8 / 19.9; of 64 16.3 / 15.1 and 19.8 / 20.4; of
    // 48 after 200 44 / 39 and 61 / 56; of 33, 2 heads of 80 on a kv head 13.7 / 11.3.  Several rows take two launches (rows
    // of up to 16 tokens are the other kernel's), which short ones do not earn; nor do rows of just more than 16 where
    // every head has a kv head of its own and a block thus 64 tokens (one of 512 and 63 of 17, 8 heads of 64: 185 / 214;
    // 20 of 30: 289 / 219; 64 of one: 113 / 103).
    const int gs = H / G, heads = gs % 4 == 0 ? 4 : gs % 2 == 0 ? 2 : 1;
    const bool alone = n_rows == 1, far = (int64_t)table_stride * page_size >= 256;
    const int least = far || HD <= 32 || (HD % 64 && HD < 96 && heads < 4) ? 8 * WARPS : HD < 96 ? 12 * WARPS : 16 * WARPS;
    const bool short_rows = n_tokens > 16 * (int64_t)n_rows && n_tokens < 40 * (int64_t)n_rows;    // on average
    const bool tiles = alone ? max_new > least : max_new >= 512 && !(heads == 1 && short_rows);
    if (dtype == 0 && args.vec && tiles) {
        if (!alone) {
            const int e = launch<float, 4>(q, pages, block_table, row_start, row_pos0, out, slopes, sinks, args,
                                           n_rows, 4 * WARPS, stream);
            if (e) return e;
        }
        const cudaError_t e = cudaFuncSetAttribute(attn_simt_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)tile_smem());
        if (e != cudaSuccess) return (int)e;
        const int cta_rows = WARPS / heads * TROWS;
        attn_simt_tile_kernel<<<dim3(H / heads * ((max_new + cta_rows - 1) / cta_rows), n_rows), THREADS, tile_smem(),
                                stream>>>((const float*)q, (const float*)pages, block_table, row_start, row_pos0,
                                          (float*)out, slopes, sinks, args, heads, alone ? 1 : 4 * WARPS + 1);
        SLLM_LAUNCH_CHECK();
        return 0;
    }
#endif
    if (dtype == 0)
        return launch_for<float>(max_new, q, pages, block_table, row_start, row_pos0, out, slopes, sinks, args,
                                 n_rows, max_new, stream);
    if (dtype == 1)
        return launch_for<__nv_bfloat16>(max_new, q, pages, block_table, row_start, row_pos0, out, slopes, sinks,
                                         args, n_rows, max_new, stream);
    return (int)cudaErrorInvalidValue;
}
