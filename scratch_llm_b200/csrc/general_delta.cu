// The generalized delta rule: a recurrent mixer whose state per request and head is a matrix
// S [key channel, value channel] in 32-bit,
//
//     S_t = diag(w_t) S_{t-1} - (a_t * u_t) (u_t^T S_{t-1}) + k_t v_t^T,     o_t = S_t^T r_t,
//
// with a decay w_t and a removal rate a_t per key channel, and u_t = k_t / sqrt(|k_t|^2 + eps)
// the unit key.  Both terms read the old state.  A column of S (one value channel) never meets
// another column: s <- w * s - (a * u) (u . s) + k v_c, o_c = s . r.
//
// Layout: a column is spread over LANES neighbouring lanes of a warp, each with EPL = 4 of its
// elements in registers as pairs (the key size D is padded to DP = 16 * 2^i; the padding stays
// zero; keys of more than 128 elements have more of them a lane), and a thread holds such slices of CPT
// neighbouring columns, four, or two in small launches, which the vectors that it reads from shared memory
// per token serve together.  A CTA has four COMPUTE warps, one per scheduler, which own
// 128 / LANES * CPT columns of one (row, head), and four LOADER warps (fewer of both where many heads of few
// columns share an SM: `launch`); a head's columns are spread over several CTAs.  The row's tokens come in chunks through two
// buffers: while the compute warps run chunk c, the loader warps, which have requested chunk
// c + 1 (r, k, w, a of the head, v of the CTA's columns) a chunk earlier, form -a * k, 1 / (|k|^2 +
// eps) and the products of neighbouring tokens; all warps meet once per chunk.
//
// What bounds a long row is the chain from token to token, so the chain is cut: with
// g_t = w_t s_{t-1} + k_t v_t (the new state before the removal), i_t = 1 / (|k_t|^2 + eps) and
// d_t = i_t k_t . s_{t-1}, so that s_t = g_t - (a_t k_t) d_t,
//     d_{t+1} = i_{t+1} k_{t+1} . s_t = i_{t+1} (k_{t+1} . g_t) - i_{t+1} (k_{t+1} . (a_t k_t)) d_t.
// The dot product with g_t and its shuffles need d_{t-1}, not d_t: two tokens are in flight, and
// what joins them is one multiply-add with a number that the loaders have formed.  Shuffles are
// issued in the order in which they are written, so a token's step is written as the two tokens
// run: the second half of one sum beside the first half of the next (`Pipe`).
// Multiply-adds come in pairs (fma.rn.f32x2: the same rate, half the instructions).
//
// A token's dot product is thus formed in another order when it is the first of a step: the same bits whatever else
// is in the step, not however a row is cut into steps.
//
// us before (a column a thread, sixteen elements a lane, five vectors) and now (columns a thread), bfloat16, 64 x 64:
//   32 heads, a row of 2,048 tokens   590 / 233 (2)   64 heads, a row of 2,400       908 / 340 (4)
//   32 heads, a row of 100             34 / 15 (2)    64 heads, eight rows of 300    547 / 238 (4)
//   32 heads, four rows of 1,024      481 / 232 (4)   128 x 128, 16 heads, 2,048     758 / 328 (4)
//   32 heads, 64 single tokens         41 / 29 (4)
// Latencies: 138 instructions per token and scheduler in 300 cycles with four columns a thread, 92 in 250 with two
// (twice the CTAs).  With the other number the first takes 300, four rows of 1,024 348 and 64 single tokens 48.
//
// state: float32 [slots, H, V, DP] with DP = the padded key size; a fresh slot holds zeros.
// Compiled once per key size (-DSLLM_HEAD_DIM=D).
#include "common.cuh"

#ifndef SLLM_HEAD_DIM
#define SLLM_HEAD_DIM 64
#endif

namespace sllm {

constexpr int D = SLLM_HEAD_DIM;
constexpr int padded(int d) {
    int p = 16;
    while (p < d) p *= 2;
    return p;
}
constexpr int DP = padded(D);                 // padded key size
static_assert(DP <= 512, "key sizes up to 512");
constexpr int EPL = DP <= 128 ? 4 : DP / 32;  // elements of a column per lane
constexpr int LANES = DP / EPL;
constexpr int UNITS = EPL / 4;                // float4 units per lane
// tokens per chunk: two buffers of four vectors of DP floats per token, within 64 KB
constexpr int CHUNK = DP <= 128 ? 16 : 2048 / DP;
static_assert(CHUNK >= 2, "chunk too small");

// two 32-bit numbers in one register pair
typedef unsigned long long f2;
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 pair(float x) {
    f2 d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(x));
    return d;
}
__device__ __forceinline__ float pair_sum(f2 a) {
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
    return x + y;
}

__device__ __forceinline__ float4 load4(const float* p) {
    return *reinterpret_cast<const float4*>(p);
}
// Dot products are formed with the key itself and not with the unit key, so a large key would overflow them where
// the rule does not.  A chunk with a key of LARGE or more is therefore changed once it is staged (`shrink`).  The
// question costs decode steps 0 to 2 % (heads of 16: 64 single tokens 18.0 / 18.5 us) and long rows nothing.
constexpr float LARGE = 1024.f;
__device__ __forceinline__ bool large(float x) { return fabsf(x) >= LARGE; }
__device__ __forceinline__ bool large(const float4& x) {
    return large(fmaxf(fmaxf(fabsf(x.x), fabsf(x.y)), fmaxf(fabsf(x.z), fabsf(x.w))));
}
// Four elements as they lie in memory, and as numbers.
template <typename T> struct Four;
template <> struct Four<float> { typedef float4 Raw; };
template <> struct Four<__nv_bfloat16> { typedef uint2 Raw; };
__device__ __forceinline__ float4 numbers(const float4& r) { return r; }
__device__ __forceinline__ float4 numbers(const uint2& r) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&r);
    return make_float4(__low2float(h[0]), __high2float(h[0]), __low2float(h[1]), __high2float(h[1]));
}

// The rule for threads with slices of CPT columns: 4, or 2 where that still leaves the launch within one CTA an
// SM (half of each token's work a warp, twice the CTAs); WARPS compute warps: 4, or one where many CTAs with heads
// of few columns have to share an SM.
template <int CPT, int WARPS> struct Rule {
static constexpr int COMPUTE = 32 * WARPS;
static constexpr int QUADS = CHUNK * DP / 4;         // units of 4 elements in a chunk
// (64 loaders for rows that are fetched element by element: 48 single tokens and one row of 64, 32 heads of 9 x 9, 24.6 us,
// with 32 of them 34.0)
static constexpr int LOADERS = WARPS > 1 ? 128 : D % 4 || QUADS / 4 > 32 ? 64 : 32;
static constexpr int THREADS = COMPUTE + LOADERS;
static constexpr int COLS = COMPUTE / LANES * CPT;   // columns of S per CTA
static __device__ __forceinline__ void loaders_sync() {
    asm volatile("bar.sync 1, %0;\n" ::"n"(LOADERS) : "memory");
}
struct alignas(16) Staged {
    float k[CHUNK + 1][DP];     // (the last: the first key of the chunk that follows)
    float r[CHUNK][DP], w[CHUNK][DP], nak[CHUNK][DP];   // nak: -a * k
    float v[CHUNK][COLS];
    float2 ic[CHUNK];           // i_t = 1 / (|k_t|^2 + eps), and i_t (k_t . nak_{t-1})
    float by[CHUNK];            // (of `shrink` alone)
};
static constexpr int SMEM = 2 * (int)sizeof(Staged);

static constexpr int QPT = (QUADS + LOADERS - 1) / LOADERS;        // of which a loader thread takes
static constexpr int VPT = (CHUNK * COLS + LOADERS - 1) / LOADERS; // values that a loader thread takes
static constexpr int APT = (DP / 4 + LOADERS - 1) / LOADERS;       // units of the key after the chunk
// a token's units fit the lanes of one warp (and LOADERS is a multiple of them): its sums are
// formed from registers
static constexpr bool FUSED = DP / 4 <= 32;

template <typename T> struct Operands {
    const T* __restrict__ rkv;
    const float* __restrict__ wa;
    int64_t ld, ldwa;
    int r0, k0, v0, HD, head, V, col0;
    float unit_eps;
};

// What a loader thread has requested of a chunk, as it lies in memory: nothing waits for a request
// before the chunk is staged.  VEC: every row of every operand starts on a multiple of 4 elements,
// so four elements come per load.
template <typename T, bool VEC> struct Request {
    typename Four<T>::Raw r[VEC ? QPT : 1], k[VEC ? QPT : 1], k_after[VEC ? APT : 1];
    float4 w[VEC ? QPT : 1], a[VEC ? QPT : 1];
    T v[VPT];
};

template <typename T, bool VEC>
static __device__ __forceinline__ void request_chunk(Request<T, VEC>& q, int lt, const Operands<T>& x,
                                              int64_t tok0, int n, bool more) {
    typedef typename Four<T>::Raw Raw;
    if (VEC) {
#pragma unroll
        for (int j = 0; j < APT; ++j) {
            const int e = (lt + j * LOADERS) * 4;
            q.k_after[j] = Raw();
            if (more && e < D)
                q.k_after[j] = *reinterpret_cast<const Raw*>(x.rkv + (tok0 + n) * x.ld + x.k0 + x.head * D + e);
        }
#pragma unroll
        for (int j = 0; j < QPT; ++j) {
            const int i = lt + j * LOADERS;
            const int t = i / (DP / 4), e = (i - t * (DP / 4)) * 4;
            q.r[j] = q.k[j] = Raw();
            q.w[j] = q.a[j] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (i < QUADS && t < n && e < D) {
                const T* row = x.rkv + (tok0 + t) * x.ld + x.head * D + e;
                const float* wa = x.wa + (tok0 + t) * x.ldwa + x.head * D + e;
                q.r[j] = *reinterpret_cast<const Raw*>(row + x.r0);
                q.k[j] = *reinterpret_cast<const Raw*>(row + x.k0);
                q.w[j] = load4(wa);
                q.a[j] = load4(wa + x.HD);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
        const int i = lt + j * LOADERS, t = i / COLS, c = i - t * COLS;
        q.v[j] = T(0.f);
        if (t < n && x.col0 + c < x.V)
            q.v[j] = x.rkv[(tok0 + t) * x.ld + x.v0 + x.head * x.V + x.col0 + c];
    }
}

// 1 / (|k_t|^2 + eps) and the product with the neighbour's row p of nak (or null), by a warp.
static __device__ __forceinline__ void token_sums(Staged& st, int lane, int t, const float* p, float eps) {
    float ss = 0.f, c = 0.f;
    for (int e = lane; e < DP; e += 32) {
        const float k = st.k[t][e];
        ss = fmaf(k, k, ss);
        if (p) c = fmaf(k, p[e], c);
    }
    ss = warp_sum(ss);
    c = warp_sum(c);
    const float inv = 1.0f / (ss + eps);
    if (lane == 0) st.ic[t] = make_float2(inv, inv * c);
}

// The large keys of a staged chunk of n tokens, by the loader warps: each is divided by a power of two that brings its
// largest element below 4, and its token's values multiplied by it.  k v, a k d and k . s / (|k|^2 + eps) stay what
// they were, eps being divided by the square.  (A token's key is the same wherever it is staged: large or not by itself.)
static __device__ __noinline__ void shrink(Staged& st, int lt, const float* before, int n, bool more, float unit_eps) {
    const int lane = lt & 31;
    for (int t = lt >> 5; t < n + more; t += LOADERS / 32) {       // a warp per key; the last: st.k[CHUNK]
        unsigned most = 0u;
        for (int e = lane; e < DP; e += 32) most = max(most, __float_as_uint(fabsf(st.k[t][e])));
        most = __reduce_max_sync(0xffffffffu, most);
        if (lane == 0 && t < n) st.by[t] = 1.f;
        if (most < __float_as_uint(LARGE)) continue;
        const unsigned x = min(most >> 23, 254u);                  // (exponents from 2^2 on: 129)
        const float by = __uint_as_float((255u - x) << 23), grow = __uint_as_float((x - 1u) << 23);
        for (int e = lane; e < DP; e += 32) {
            st.k[t][e] *= by;
            if (t < n) st.nak[t][e] *= by;
        }
        if (t < n) {
            for (int c = lane; c < COLS; c += 32) st.v[t][c] *= grow;
            if (lane == 0) st.by[t] = by;
        }
    }
    loaders_sync();
    for (int t = lt >> 5; t < n; t += LOADERS / 32) {
        const float by = st.by[t];
        if (by != 1.f || (t > 0 && st.by[t - 1] != 1.f))
            token_sums(st, lane, t, t == 0 ? before : st.nak[t - 1], unit_eps * by * by);
    }
}

// The loader warps bring the chunk [tok0, tok0 + n), which they have requested, into `st` (`left` tokens come after
// it).  `before`: the row of nak of the token before tok0, or null.  Returns whether this thread has met a large key.
template <typename T, bool VEC>
static __device__ __forceinline__ bool stage_chunk(Staged& st, Request<T, VEC>& q, int lt,
                                            const Operands<T>& x, const float* before,
                                            int64_t tok0, int n, int left) {
    bool met = false;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
        const int i = lt + j * LOADERS, t = i / COLS, c = i - t * COLS;
        if (i < CHUNK * COLS) st.v[t][c] = to_float(q.v[j]);
    }
    if (VEC) {
#pragma unroll
        for (int j = 0; j < APT; ++j)
            if ((lt + j * LOADERS) * 4 < DP) {
                const float4 k = numbers(q.k_after[j]);
                met = met || large(k);
                *reinterpret_cast<float4*>(&st.k[CHUNK][(lt + j * LOADERS) * 4]) = k;
            }
#pragma unroll
        for (int j = 0; j < QPT; ++j) {
            const int i = lt + j * LOADERS;
            const int t = i / (DP / 4), e = (i - t * (DP / 4)) * 4;
            if (i < QUADS && t < n) {
                const float4 k = numbers(q.k[j]), a = q.a[j];
                met = met || large(k);
                *reinterpret_cast<float4*>(&st.r[t][e]) = numbers(q.r[j]);
                *reinterpret_cast<float4*>(&st.k[t][e]) = k;
                *reinterpret_cast<float4*>(&st.w[t][e]) = q.w[j];
                *reinterpret_cast<float4*>(&st.nak[t][e]) =
                    make_float4(-a.x * k.x, -a.y * k.y, -a.z * k.z, -a.w * k.w);
            }
        }
    } else {
        for (int i = lt; i < n * DP; i += LOADERS) {
            const int t = i / DP, e = i - t * DP;
            const int64_t tok = tok0 + t;
            float r = 0.f, k = 0.f, w = 0.f, a = 0.f;
            if (e < D) {
                r = to_float(x.rkv[tok * x.ld + x.r0 + x.head * D + e]);
                k = to_float(x.rkv[tok * x.ld + x.k0 + x.head * D + e]);
                w = x.wa[tok * x.ldwa + x.head * D + e];
                a = x.wa[tok * x.ldwa + x.HD + x.head * D + e];
            }
            st.r[t][e] = r; st.k[t][e] = k; st.w[t][e] = w; st.nak[t][e] = -a * k;
            met = met || large(k);
        }
        for (int e = lt; e < DP; e += LOADERS) {
            const float k = left > 0 && e < D ? to_float(x.rkv[(tok0 + n) * x.ld + x.k0 + x.head * D + e]) : 0.f;
            st.k[CHUNK][e] = k;
            met = met || large(k);
        }
    }
    loaders_sync();
    if (VEC && FUSED) {
        // a token's DP / 4 units lie in neighbouring lanes of one warp
        float ss[QPT], c[QPT];
#pragma unroll
        for (int j = 0; j < QPT; ++j) {
            const int i = lt + j * LOADERS;
            const int t = i / (DP / 4), e = (i - t * (DP / 4)) * 4;
            const float* p = t == 0 ? before : st.nak[t < CHUNK ? t - 1 : 0];
            const float4 k = numbers(q.k[j]);
            ss[j] = fmaf(k.x, k.x, fmaf(k.y, k.y, fmaf(k.z, k.z, k.w * k.w)));
            c[j] = 0.f;
            if (i < QUADS && t < n && p) {
                const float4 y = load4(p + e);
                c[j] = fmaf(k.x, y.x, fmaf(k.y, y.y, fmaf(k.z, y.z, k.w * y.w)));
            }
        }
#pragma unroll
        for (int o = (DP / 4) >> 1; o > 0; o >>= 1)
#pragma unroll
            for (int j = 0; j < QPT; ++j) {
                ss[j] += __shfl_xor_sync(0xffffffffu, ss[j], o);
                c[j] += __shfl_xor_sync(0xffffffffu, c[j], o);
            }
#pragma unroll
        for (int j = 0; j < QPT; ++j) {
            const int i = lt + j * LOADERS;
            const int t = i / (DP / 4), e = (i - t * (DP / 4)) * 4;
            const float inv = 1.0f / (ss[j] + x.unit_eps);
            if (i < QUADS && t < n && e == 0) st.ic[t] = make_float2(inv, inv * c[j]);
        }
    } else {
        for (int t = lt >> 5; t < n; t += LOADERS / 32)     // a warp per token
            token_sums(st, lt & 31, t, t == 0 ? before : st.nak[t - 1], x.unit_eps);
    }
    if (!VEC && left > 0) request_chunk<T, VEC>(q, lt, x, tok0 + n, min(CHUNK, left), left > CHUNK);
    return met;
}

static constexpr int SHARE = LANES / CPT;          // lanes that go on with the same column
static_assert(SHARE >= 1 && CPT <= 4, "no more columns a thread than lanes a column");

// Sums across a column's lanes begin with CPT values per lane (one per column) that become one: each
// exchange halves the columns that a lane goes on with.  A lane goes on with column
// lane_in_col / SHARE.  One exchange of x's `have` pairs:
template <int HAVE>
static __device__ __forceinline__ void share(float (&x)[CPT], int lane_in_col) {
    constexpr int SH = LANES / CPT * HAVE;
    const bool upper = lane_in_col & SH;
#pragma unroll
    for (int i = 0; i < HAVE; ++i) {
        const float send = upper ? x[i] : x[i + HAVE], keep = upper ? x[i + HAVE] : x[i];
        x[i] = keep + __shfl_xor_sync(0xffffffffu, send, SH);
    }
}
// ... of two sums at a time, until one value of each is left.
static __device__ __forceinline__ void share_both(float (&x)[CPT], float (&y)[CPT], int lane_in_col) {
    if constexpr (CPT >= 4) {
        share<2>(x, lane_in_col);
        share<2>(y, lane_in_col);
    }
    if constexpr (CPT >= 2) {
        share<1>(x, lane_in_col);
        share<1>(y, lane_in_col);
    }
}

template <int N> static __device__ __forceinline__ void fetch(f2 (&x)[2 * UNITS], const float* row) {
#pragma unroll
    for (int i = 0; i < UNITS; ++i) {
        const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(row + N * i);
        x[2 * i] = y.x;
        x[2 * i + 1] = y.y;
    }
}
static __device__ __forceinline__ float dot(const f2 (&x)[2 * UNITS], const f2 (&y)[2 * UNITS]) {
    f2 acc = mul2(x[0], y[0]);
#pragma unroll
    for (int i = 1; i < 2 * UNITS; ++i) acc = fma2(x[i], y[i], acc);
    return pair_sum(acc);
}

// What a thread carries from token t - 1 to token t: g_{t-1}, d_{t-1}, its slices of a_{t-1} k_{t-1}
// (negated), r_{t-1} and k_t, and k_t . g_{t-1} summed as far as `share` goes.
struct Pipe {
    f2 g[CPT][2 * UNITS], nak[2 * UNITS], r[2 * UNITS], k[2 * UNITS];
    float d[CPT], x;
    int lane_in_col, col_local;

    // The state after token t - 1.
    __device__ __forceinline__ void state(f2 (&s)[CPT][2 * UNITS]) const {
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
            const f2 dd = pair(d[c]);
#pragma unroll
            for (int i = 0; i < 2 * UNITS; ++i) s[c][i] = fma2(nak[i], dd, g[c][i]);
        }
    }
    // k_t . g_{t-1} and the read-out of token t - 1, as far as `share` goes.
    __device__ __forceinline__ float begin(const f2 (&s)[CPT][2 * UNITS]) {
        float xp[CPT], op[CPT];
#pragma unroll
        for (int c = 0; c < CPT; ++c) xp[c] = dot(k, g[c]);
#pragma unroll
        for (int c = 0; c < CPT; ++c) op[c] = dot(r, s[c]);
        share_both(xp, op, lane_in_col);
        x = xp[0];
        return op[0];
    }
    // Token t of the chunk; returns the read-out of the token before it (see begin).
    __device__ __forceinline__ float step(const Staged& st, int t) {
        const int e0 = 4 * lane_in_col;
        f2 w[2 * UNITS], kn[2 * UNITS], s[CPT][2 * UNITS], rn[2 * UNITS], an[2 * UNITS];
        fetch<4 * LANES>(w, &st.w[t][e0]);
        fetch<4 * LANES>(kn, &st.k[t + 1][e0]);
        const float2 ic = st.ic[t];
        float v[CPT];
#pragma unroll
        for (int c = 0; c < CPT; ++c) v[c] = st.v[t][col_local + c];
        fetch<4 * LANES>(an, &st.nak[t][e0]);
        fetch<4 * LANES>(rn, &st.r[t][e0]);
        float y;
        if (SHARE >= 2) y = __shfl_xor_sync(0xffffffffu, x, SHARE / 2);
        state(s);
        if (SHARE >= 2) x += y;
        if (SHARE >= 4) y = __shfl_xor_sync(0xffffffffu, x, SHARE / 4);
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
            const f2 vv = pair(v[c]);
#pragma unroll
            for (int i = 0; i < 2 * UNITS; ++i) g[c][i] = fma2(w[i], s[c][i], mul2(k[i], vv));
        }
        if (SHARE >= 4) x += y;
#pragma unroll
        for (int o = SHARE / 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        float sum[CPT];      // every lane gets its columns' sums from the lanes that have them
#pragma unroll
        for (int c = 0; c < CPT; ++c)
            sum[c] = CPT == 1 ? x : __shfl_sync(0xffffffffu, x, c * SHARE, LANES);
        float xp[CPT], op[CPT];
#pragma unroll
        for (int c = 0; c < CPT; ++c) xp[c] = dot(kn, g[c]);
#pragma unroll
        for (int c = 0; c < CPT; ++c) op[c] = dot(r, s[c]);
#pragma unroll
        for (int c = 0; c < CPT; ++c) d[c] = fmaf(ic.y, d[c], ic.x * sum[c]);
        share_both(xp, op, lane_in_col);
        x = xp[0];
#pragma unroll
        for (int i = 0; i < 2 * UNITS; ++i) {
            k[i] = kn[i];
            nak[i] = an[i];
            r[i] = rn[i];
        }
        return op[0];
    }
};

// Sums of GROUP tokens' read-outs across the lanes of a column: each exchange halves the tokens
// that a lane goes on with; a lane ends with the tokens first .. of its column.
static constexpr int GROUP = CHUNK < 4 ? CHUNK : 4;
static constexpr int KEPT = GROUP >= SHARE ? GROUP / SHARE : 1;
static __device__ __forceinline__ int share_tokens(float (&o)[GROUP], int lane_in_col) {
    int first = 0, have = GROUP;
#pragma unroll
    for (int sh = SHARE >> 1; sh > 0; sh >>= 1) {
        if (have > 1) {
            have >>= 1;
            const bool upper = lane_in_col & sh;
#pragma unroll
            for (int i = 0; i < GROUP / 2; ++i) {
                if (i >= have) break;
                const float send = upper ? o[i] : o[i + have], keep = upper ? o[i + have] : o[i];
                o[i] = keep + __shfl_xor_sync(0xffffffffu, send, sh);
            }
            first += upper ? have : 0;
        } else {
            o[0] += __shfl_xor_sync(0xffffffffu, o[0], sh);
        }
    }
    return first;
}
};

// rkv: [N, ld] with the heads' r at column r0, k at k0, v at v0 (each heads x D or heads x V);
// wa: float32 [N, ldwa] with the decays at column 0 and the removal rates at column H * D.
// (two CTAs an SM at every key size: 4 heads of 300 x 300, 64 single tokens 311 us with one, 159 so)
template <typename T, bool VEC, int CPT, int WARPS>
__global__ void __launch_bounds__(Rule<CPT, WARPS>::THREADS, WARPS > 1 ? 2 : 512 / Rule<CPT, WARPS>::THREADS)
general_delta_kernel(const T* __restrict__ rkv, int64_t ld, int r0, int k0, int v0,
                     const float* __restrict__ wa, int64_t ldwa, float* __restrict__ state,
                     const int* __restrict__ row_start, const int* __restrict__ row_slot,
                     float* __restrict__ out, int H, int V, float unit_eps) {
    pdl_wait();
    pdl_trigger();
    extern __shared__ __align__(16) uint8_t smem[];
    typedef Rule<CPT, WARPS> R;
    typedef typename R::Staged Staged;
    constexpr int SHARE = R::SHARE, GROUP = R::GROUP;
    Staged* stage = reinterpret_cast<Staged*>(smem);
    const int row = blockIdx.z, head = blockIdx.y;
    const int t0 = row_start[row], n_new = row_start[row + 1] - t0;
    if (n_new <= 0) return;
    const int tid = threadIdx.x;
    const bool loader = tid >= R::COMPUTE;
    const int col0 = blockIdx.x * R::COLS;
    if (loader) {
        const int lt = tid - R::COMPUTE;
        const typename R::template Operands<T> x{rkv, wa, ld, ldwa, r0, k0, v0, H * D, head, V, col0, unit_eps};
        typename R::template Request<T, VEC> q;
        R::template request_chunk<T, VEC>(q, lt, x, t0, min(CHUNK, n_new), n_new > CHUNK);
        for (int c0 = 0, buf = 0; c0 < n_new; c0 += CHUNK, buf ^= 1) {
            const float* before = c0 ? stage[buf ^ 1].nak[CHUNK - 1] : nullptr;
            const int n = min(CHUNK, n_new - c0), left = n_new - c0 - CHUNK;
            const bool met = R::template stage_chunk<T, VEC>(stage[buf], q, lt, x, before, (int64_t)t0 + c0, n, left);
            // chunk c is staged, chunk c - 1 is done with (the compute warps wait again while large keys are changed)
            if (__syncthreads_or(met)) {
                R::shrink(stage[buf], lt, before, n, left > 0, unit_eps);
                __syncthreads();
            }
            // (after the call: held across it, the requests were waited for; in a layer of 32 heads of 64 x 64 and 2,048
            // tokens 382 us, 370 so)
            if (VEC && left > 0)
                R::template request_chunk<T, VEC>(q, lt, x, (int64_t)t0 + c0 + n, min(CHUNK, left), left > CHUNK);
        }
        return;
    }
    typename R::Pipe p;
    p.lane_in_col = tid % LANES;
    p.col_local = tid / LANES * CPT;
    const int e0 = 4 * p.lane_in_col, col = col0 + p.col_local;
    float* sp = state + (((int64_t)row_slot[row] * H + head) * V + col) * DP + e0;
#pragma unroll
    for (int c = 0; c < CPT; ++c) {
        p.d[c] = 0.f;
        if (col + c < V) {
            R::template fetch<4 * LANES>(p.g[c], sp + c * DP);
        } else {
#pragma unroll
            for (int i = 0; i < 2 * UNITS; ++i) p.g[c][i] = 0;
        }
    }
#pragma unroll
    for (int i = 0; i < 2 * UNITS; ++i) p.nak[i] = p.r[i] = 0;
    const int64_t ld_out = (int64_t)H * V;
    const int o_col = col0 + p.col_local + p.lane_in_col / SHARE;
    const bool stores = o_col < V;
    float* o_row = out + t0 * ld_out + (int64_t)head * V + o_col;    // of token 0
    f2 s[CPT][2 * UNITS];
    if (__syncthreads_or(false)) __syncthreads();       // the first chunk is staged
    R::template fetch<4 * LANES>(p.k, &stage[0].k[0][e0]);
    p.state(s);
    p.begin(s);
    // (a step gives the read-out of the token before it: the first one's belongs to no token)
    for (int c0 = 0, buf = 0; c0 < n_new; c0 += CHUNK, buf ^= 1) {
        const int n = min(CHUNK, n_new - c0);
        int t = 0;
#pragma unroll 1
        for (; t + GROUP <= n; t += GROUP) {
            float o[GROUP];
#pragma unroll
            for (int i = 0; i < GROUP; ++i) o[i] = p.step(stage[buf], t + i);
            const int first = c0 + t - 1 + R::share_tokens(o, p.lane_in_col);
            // (with fewer tokens than lanes, the lanes that hold the same token store the same sum)
#pragma unroll
            for (int i = 0; i < R::KEPT; ++i)
                if (stores && first + i >= 0) o_row[(first + i) * ld_out] = o[i];
        }
#pragma unroll 1
        for (; t < n; ++t) {
            float o = p.step(stage[buf], t);
#pragma unroll
            for (int sh = SHARE >> 1; sh > 0; sh >>= 1) o += __shfl_xor_sync(0xffffffffu, o, sh);
            if (stores && c0 + t > 0) o_row[(c0 + t - 1) * ld_out] = o;
        }
        if (c0 + CHUNK < n_new && __syncthreads_or(false)) __syncthreads();
    }
    p.state(s);
    float o = p.begin(s);
#pragma unroll
    for (int sh = SHARE >> 1; sh > 0; sh >>= 1) o += __shfl_xor_sync(0xffffffffu, o, sh);
    if (stores) o_row[(n_new - 1) * ld_out] = o;
#pragma unroll
    for (int c = 0; c < CPT; ++c)
        if (col + c < V)
#pragma unroll
            for (int i = 0; i < UNITS; ++i)
                *reinterpret_cast<ulonglong2*>(sp + c * DP + 4 * LANES * i) =
                    make_ulonglong2(s[c][2 * i], s[c][2 * i + 1]);
}

template <typename T, bool VEC, int CPT, int WARPS, typename... Args>
static int launch_rule(int n_rows, int H, int V, bool beside, cudaStream_t stream, Args... args) {
    constexpr int SMEM = Rule<CPT, WARPS>::SMEM, COLS = Rule<CPT, WARPS>::COLS, THREADS = Rule<CPT, WARPS>::THREADS;
    const auto kernel = general_delta_kernel<T, VEC, CPT, WARPS>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return (int)e;
    const dim3 grid((V + COLS - 1) / COLS, H, n_rows);
    if (beside) return (int)sllm_launch_pdl(kernel, grid, dim3(THREADS), SMEM, stream, args...);
    kernel<<<grid, THREADS, SMEM, stream>>>(args...);
    SLLM_LAUNCH_CHECK();
    return 0;
}

// Two columns a thread while the launch has at most one CTA an SM even so: 32 heads of 64 x 64, a row of 2,048
// tokens 300 us with four, 231 with two; 100 tokens 18 and 15; beyond, the SMs' throughput counts (64 heads, a
// row of 2,400: 353 and 404).
// One compute warp and few loaders (64 threads at key size 16) where an SM gets more than the two CTAs of 256
// threads that it holds, and the head's columns leave most of such a CTA idle.  us with 256 threads and so: 256 single
// tokens, 32 heads of 16 x 16 67.6 / 21.2, of 9 x 9 69.7 / 22.8, 16 of 32 x 32 27.8 / 18.9, 16 of 64 x 5 28.6 / 14.1; 48 rows
// of 8 tokens, 32 heads of 16 x 16 21.8 / 10.2.  (8 heads of 16 x 100, which take four such CTAs: 19.2 / 21.2.)  With 16
// elements a key from more CTAs than SMs on (8 single tokens, 32 heads of 16 x 16 3.9 / 3.7, 8 rows of 64 18.9 / 13.5; of
// 24 x 24 3.3 / 3.8 and 17.6 / 17.7, of 9 x 9 8 rows of 300 77 / 83).
// `beside`: begun beside the kernel before it, a launch's CTAs take the places that come free first, two on some SMs,
// and long rows of a launch that does not fill the SMs go by the slowest.  us of decays, rule and read-out in
// turn, ordinary / beside: 32 heads of 64 x 64, 2,048 tokens 299 / 391, 300 52 / 67, 64 20.9 / 23.6, 8 13.0 / 12.7, 2
// 10.0 / 9.8; 48 single tokens and one of 64 44.4 / 43.8; 48 rows of 8 50.2 / 49.9; more CTAs than the SMs hold:
// 16 heads of 128 x 128, four rows of 1,024 660 / 635, eight of 300 396 / 392.  So: launches that fill the SMs, and those
// of a chunk a row at most on average.
template <typename T, bool VEC>
static int launch(const T* rkv, int64_t ld, int r0, int k0, int v0, const float* wa, int64_t ldwa, float* state,
                  const int* row_start, const int* row_slot, float* out, int n_rows, int H, int V, float unit_eps,
                  int n_sm, int n_tokens, cudaStream_t stream) {
    constexpr int MOST = EPL == 4 ? 4 : 16 / EPL, FEW = EPL == 4 ? 2 : MOST;
    const auto ctas = [&](int cols) { return (int64_t)((V + cols - 1) / cols) * H * n_rows; };
    const bool many = ctas(Rule<MOST, 4>::COLS) > 2 * n_sm, beside = many || n_tokens <= CHUNK * (int64_t)n_rows;
#define SLLM_GD_RULE(CPT, WARPS)                                                                                \
    return launch_rule<T, VEC, CPT, WARPS>(n_rows, H, V, beside, stream, rkv, ld, r0, k0, v0, wa, ldwa, state,  \
                                           row_start, row_slot, out, H, V, unit_eps)
    if (FEW != MOST && ctas(Rule<FEW, 4>::COLS) <= n_sm) SLLM_GD_RULE(FEW, 4);
    if constexpr (DP <= 64) {
        const bool crowded = DP == 16 && D % 4 == 0 ? ctas(Rule<MOST, 4>::COLS) > n_sm : many;
        if (crowded && V <= 2 * Rule<MOST, 1>::COLS) SLLM_GD_RULE(MOST, 1);
    }
    SLLM_GD_RULE(MOST, 4);
#undef SLLM_GD_RULE
}

}  // namespace sllm

using namespace sllm;

SLLM_EXPORT int sllm_general_delta_padded_dim() { return DP; }

// dtype of rkv: 0 = float32, 1 = bfloat16.  n_tokens: of all rows.
SLLM_EXPORT int sllm_general_delta(const void* rkv, int64_t ld, int r0, int k0, int v0,
                                   const float* wa, int64_t ldwa, float* state,
                                   const int* row_start, const int* row_slot, float* out,
                                   int n_rows, int n_tokens, int H, int V, float unit_eps, int dtype,
                                   cudaStream_t stream) {
    if (n_rows <= 0) return 0;
    if (H <= 0 || V <= 0 || H > 65535 || n_rows > 65535) return (int)cudaErrorInvalidValue;
    // four elements per load where every operand's rows start on multiples of four elements
    const bool vec = D % 4 == 0 && ld % 4 == 0 && r0 % 4 == 0 && k0 % 4 == 0 && ldwa % 4 == 0 &&
                     !(((uintptr_t)rkv | (uintptr_t)wa) & 15);
    typedef __nv_bfloat16 bf16;
    int dev = 0, n_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return (int)cudaErrorInvalidDevice;
#define SLLM_GD_LAUNCH(T, VEC)                                                                  \
    return launch<T, VEC>((const T*)rkv, ld, r0, k0, v0, wa, ldwa, state, row_start, row_slot,  \
                          out, n_rows, H, V, unit_eps, n_sm, n_tokens, stream)
    if (dtype == 0) {
        if (vec) SLLM_GD_LAUNCH(float, true);
        SLLM_GD_LAUNCH(float, false);
    }
    if (dtype == 1) {
        if (vec) SLLM_GD_LAUNCH(bf16, true);
        SLLM_GD_LAUNCH(bf16, false);
    }
#undef SLLM_GD_LAUNCH
    return (int)cudaErrorInvalidValue;
}
