// Long portions of the gated delta rule in chunks of TC = 64 tokens: what a chunk's tokens do to each other
// is formed for all chunks at once, and only a short pass over the chunks is sequential.
//
// Per head, with the state S [D, V], a decay e^{l_t} per key channel (or one for all channels), L_t the
// sums of l up to token t of the chunk, S0 the state at the chunk's start and the rule as delta_rule.cu
// states it, the tokens' writes u_t (rows of X) are
//
//     (I + A) X  =  beta (v - k~ S0)           A_ts = beta_t <k_t e^{L_t}, k_s e^{-L_s}>      s < t
//     o_t  =  q~_t S0 + sum_{s<=t} M_ts X_s    M_ts = <q_t e^{L_t}, k_s e^{-L_s}>
//     S    =  e^{L_last} S0 + y~^T X
//
// with k~ = k e^{L}, q~ = q e^{L}, y~ = k e^{L_last - L}.  Three kernels:
//   prep (a CTA per chunk and head): A by blocks of BT = 16 tokens, then W = (I + A)^{-1} beta k~ and
//        X0 = (I + A)^{-1} beta v by forward substitution, a thread per column: 2,016 multiply-adds in
//        registers, A broadcast from shared memory, no inverse is formed.  Writes W, X0, q~, y~, M.
//   pass (a CTA per row, head and 16 columns, the chunks in order): X = X0 - W S0,
//        S <- e^{L_last} S0 + y~^T X.  This is the sequential part.  Writes X in X0's place and S0.
//   out  (a CTA per chunk, head and 64 columns): o.
//
// Exponents: none is above 0, and none is a difference of sums over more than a block.  Inside a block
// e^{L_t - L_s} comes from sums that start at the block's border; between blocks it is the product of
// e^{(border before t) .. t}, the blocks between, and e^{s .. (border after s)}; decays per channel are
// multiplied up token by token inside blocks.
//
// Why: a row's tokens in order are a chain of 128 pieces of 16 tokens for 2,048 tokens, 5.9 us each
// whatever the GPU's width.  In chunks the chain has 32 links of two small products.  2,048 tokens, 16
// heads of 128 x 128, bfloat16: one decay per head 733 -> 186 us, per channel 666 -> 260 us.  One by one, per
// head: 56, 89 and 46 us.
#pragma once

#include <algorithm>

#include "scan_chunks.cuh"

namespace sllm {
namespace chunks {

constexpr int BT = 16, NB = TC / BT;
constexpr int LDT = TC + 4;              // row stride of A in shared memory
constexpr int PREP_THREADS = 256, OUT_THREADS = 256, OUT_COLS = 64;
constexpr int NC = 16;                   // columns of the state per CTA of the pass

struct Scratch {                         // per (slot, head), 32-bit
    float *W, *Y;                        // [TC][D] in the order in which the pass's threads take them
    float* Q;                            // [TC][D]
    float* X;                            // [V][TC]: X0, after the pass X
    float* M;                            // [TC][TC]
    float* S;                            // [V][D]: S0
    float* decay;                        // [D]: e^{L_last}
};

__host__ __device__ constexpr int64_t scratch_floats(int D, int64_t V) {
    return 3 * TC * D + TC * V + TC * TC + V * D + D;
}
// `at`: scratch_floats x n floats on a 16-byte boundary (every piece is whole quads).
static inline Scratch scratch_at(float* at, int64_t n, int D, int64_t V) {
    Scratch s;
    s.W = at; at += n * TC * D;
    s.Y = at; at += n * TC * D;
    s.Q = at; at += n * TC * D;
    s.M = at; at += n * TC * TC;
    s.S = at; at += n * V * D;
    s.decay = at; at += n * D;
    s.X = at;
    return s;
}

// The chunks of a step are numbered over the rows that have any (at least min_chunked tokens), row after
// row.  They are worked on in groups of as many as the scratch has slots: chunk `first` + i has slot i.
struct Group { int first, count; bool beside; };     // beside: see launch()
struct RowAt { int row, t0, n_new, first; };     // first: the number of the row's first chunk
// BY_CHUNK: the row of the group's chunk number `which`; else the row number `which` of those that have chunks
// in the group or after it.
template <bool BY_CHUNK>
__device__ __forceinline__ bool find_row(const int* row_start, int n_rows, int min_chunked, const Group& group,
                                         int which, RowAt& at) {
    const int lane = threadIdx.x & 31;
    int chunks_before = 0, rows_before = 0;
    for (int r0 = 0; r0 < n_rows; r0 += 32) {
        const int r = r0 + lane;
        int start = 0, count = 0;
        if (r < n_rows) {
            start = row_start[r];
            count = row_start[r + 1] - start;
        }
        const bool has = r < n_rows && count >= min_chunked;
        if (!__any_sync(0xffffffffu, has)) continue;
        const int chunks = has ? (count + TC - 1) / TC : 0;
        int end = chunks;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int more = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= o) end += more;
        }
        end += chunks_before;
        const int first = end - chunks;
        const unsigned open = __ballot_sync(0xffffffffu, has && end > group.first);
        const bool mine = BY_CHUNK ? group.first + which >= first && group.first + which < end
                                   : (open >> lane & 1) && rows_before + __popc(open & ((1u << lane) - 1)) == which;
        const unsigned hit = __ballot_sync(0xffffffffu, mine);
        if (hit) {
            const int who = __ffs(hit) - 1;
            at.row = r0 + who;
            at.t0 = __shfl_sync(0xffffffffu, start, who);
            at.n_new = __shfl_sync(0xffffffffu, count, who);
            at.first = __shfl_sync(0xffffffffu, first, who);
            return true;
        }
        chunks_before = __shfl_sync(0xffffffffu, end, 31);
        rows_before += __popc(open);
    }
    return false;
}

// Two multiply-adds in one instruction, each rounded as fmaf rounds.
struct Two { unsigned long long v; };
__device__ __forceinline__ Two two(float a, float b) {
    Two r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float first(Two a) { return __uint_as_float((unsigned)a.v); }
__device__ __forceinline__ float second(Two a) { return __uint_as_float((unsigned)(a.v >> 32)); }
__device__ __forceinline__ Two fma2(Two a, Two b, Two c) {
    Two r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
struct Four { Two a, b; };
__device__ __forceinline__ Four load22(const float* p) {        // 16 bytes of shared memory
    const ulonglong2 r = *reinterpret_cast<const ulonglong2*>(p);
    return {{r.x}, {r.y}};
}

__device__ __forceinline__ void cp16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_wait_all() {
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

// -------------------------------------------------------------------------------------- prep

// Forward substitution of one column: acc <- (I + A)^{-1} acc, At[s][t] = -A_ts.
__device__ __forceinline__ void substitute(Two (&acc)[TC / 2], const float* At) {
#pragma unroll
    for (int s = 0; s < TC - 1; ++s) {
        // (a column's entries are requested one column at a time: more do not fit the registers, and
        // the compiler does not move loads over this)
        __syncwarp();
        const float us = s & 1 ? second(acc[s / 2]) : first(acc[s / 2]);
        const Two u = two(us, us);
        // the pair that holds s itself: only its second entry may come after s
        if (!(s & 1))
            acc[s / 2] = two(us, fmaf(At[s * LDT + s + 1], us, second(acc[s / 2])));
        const int p0 = s / 2 + 1;        // pairs from here on lie after s
        if ((p0 & 1) && p0 < TC / 2) {
            const Two a = {*reinterpret_cast<const unsigned long long*>(At + s * LDT + 2 * p0)};
            acc[p0] = fma2(a, u, acc[p0]);
        }
#pragma unroll
        for (int t4 = (p0 + 1) / 2; t4 < TC / 4; ++t4) {
            const Four a = load22(At + s * LDT + 4 * t4);
            acc[2 * t4] = fma2(a.a, u, acc[2 * t4]);
            acc[2 * t4 + 1] = fma2(a.b, u, acc[2 * t4 + 1]);
        }
    }
}

// Forward substitution of one column of (I + A)^{-1} b, At[s][t] = -A_ts, a block of BT tokens at a time: what
// the blocks before it do to a block, then the block itself.  Per entry one chain over s in ascending order.
// The loops over blocks and over the tokens before one stay loops: as straight code over all 64 tokens (1,600
// instructions, and twice 1,700 for the pairs of tokens inside the blocks) instruction fetches were what the kernel
// of decays per channel waited for most (2.45 of 6 cycles an instruction, 0.32 now; 247 -> 227 us at 3,001 tokens,
// four rows, 16 heads).  The kernel with one decay per head, two CTAs an SM and no other long code, keeps
// `substitute`: 186 us for 2,048 tokens, 188 so.  The same bits.
// X: this thread's place for solved entries, rows PREP_THREADS apart.  fetch(t): b_t as it lies in memory; it is asked
// for a block ahead.  right(t, raw): b_t.  store(t0, acc): the solved entries t0 .. t0 + BT - 1.
template <typename Fetch, typename Right, typename Store>
__device__ __forceinline__ void solve_column(const float* At, float* X, const Fetch& fetch, const Right& right,
                                             const Store& store) {
    float raw[BT];
#pragma unroll
    for (int t = 0; t < BT; ++t) raw[t] = fetch(t);
#pragma unroll 1
    for (int t0 = 0; t0 < TC; t0 += BT) {
        Two acc[BT / 2];
#pragma unroll
        for (int t = 0; t < BT; t += 2) acc[t / 2] = two(right(t0 + t, raw[t]), right(t0 + t + 1, raw[t + 1]));
        if (t0 + BT < TC) {
#pragma unroll
            for (int t = 0; t < BT; ++t) raw[t] = fetch(t0 + BT + t);
        }
        const float* a = At + t0;
#pragma unroll 4
        for (int s = 0; s < t0; ++s) {
            const float us = X[s * PREP_THREADS];
            const Two u = two(us, us);
#pragma unroll
            for (int t4 = 0; t4 < BT / 4; ++t4) {
                const Four v = load22(a + s * LDT + 4 * t4);
                acc[2 * t4] = fma2(v.a, u, acc[2 * t4]);
                acc[2 * t4 + 1] = fma2(v.b, u, acc[2 * t4 + 1]);
            }
        }
        a += t0 * LDT;
#pragma unroll
        for (int s = 0; s < BT - 1; ++s) {
            const float us = s & 1 ? second(acc[s / 2]) : first(acc[s / 2]);
            const Two u = two(us, us);
            // the pair that holds s itself: only its second entry may come after s
            if (!(s & 1)) acc[s / 2] = two(us, fmaf(a[s * LDT + s + 1], us, second(acc[s / 2])));
            const int p0 = s / 2 + 1;        // pairs from here on lie after s
            if ((p0 & 1) && p0 < BT / 2) {
                const Two v = {*reinterpret_cast<const unsigned long long*>(a + s * LDT + 2 * p0)};
                acc[p0] = fma2(v, u, acc[p0]);
            }
#pragma unroll
            for (int t4 = (p0 + 1) / 2; t4 < BT / 4; ++t4) {
                const Four v = load22(a + s * LDT + 4 * t4);
                acc[2 * t4] = fma2(v.a, u, acc[2 * t4]);
                acc[2 * t4 + 1] = fma2(v.b, u, acc[2 * t4 + 1]);
            }
        }
        if (t0 + BT < TC) {
#pragma unroll
            for (int t = 0; t < BT; t += 2) {
                X[(t0 + t) * PREP_THREADS] = first(acc[t / 2]);
                X[(t0 + t + 1) * PREP_THREADS] = second(acc[t / 2]);
            }
        }
        store(t0, acc);
    }
}
constexpr int SOLVED = (TC - BT) * PREP_THREADS;     // floats of shared memory for the solved entries

// Where the pass finds W_td and y~_td (its threads' operands of mma.m16n8k16, four elements each):
// W as [d / 16][t / 8][lane][4], y~ as [d / 16][t / 16][d % 16 / 8][lane][4].
__device__ __forceinline__ int w_place(int t, int d) {
    return ((d / 16 * 8 + t / 8) * 32 + t % 8 * 4 + d % 8 / 2) * 4 + d % 16 / 8 * 2 + d % 2;
}
__device__ __forceinline__ void y_source(int i, int& t, int& d) {      // of piece i: tokens t, t + 1, t + 8, t + 9
    t = i / 64 % 4 * 16 + i % 4 * 2;
    d = i / 256 * 16 + i / 32 % 2 * 8 + i % 32 / 4;
}
// A solved column of W (d >= 0), or of X0.
__device__ __forceinline__ void store_column(const Two (&acc)[TC / 2], float* W, int d, float* X0) {
    if (d >= 0) {
#pragma unroll
        for (int t = 0; t < TC; t += 2) {
            W[w_place(t, d)] = first(acc[t / 2]);
            W[w_place(t + 1, d)] = second(acc[t / 2]);
        }
    } else {
#pragma unroll
        for (int t = 0; t < TC; t += 4)
            *reinterpret_cast<float4*>(X0 + t) = make_float4(first(acc[t / 2]), second(acc[t / 2]),
                                                             first(acc[t / 2 + 1]), second(acc[t / 2 + 1]));
    }
}

// Solved entries t0 .. t0 + BT - 1 of a column of W (d >= 0), or of X0.
__device__ __forceinline__ void store_column(const Two (&acc)[BT / 2], int t0, float* W, int d, float* X0) {
    if (d >= 0) {
#pragma unroll
        for (int t = 0; t < BT; t += 2) {
            W[w_place(t0 + t, d)] = first(acc[t / 2]);
            W[w_place(t0 + t + 1, d)] = second(acc[t / 2]);
        }
    } else {
#pragma unroll
        for (int t = 0; t < BT; t += 4)
            *reinterpret_cast<float4*>(X0 + t0 + t) = make_float4(first(acc[t / 2]), second(acc[t / 2]),
                                                                  first(acc[t / 2 + 1]), second(acc[t / 2 + 1]));
    }
}

// A warp's product of 16 rows of x with 16 rows of y, [row][LD] in shared memory: lane (tg, sg) gets
// rows tg + 4 a and columns sg + 8 b.  `mid` (or null): a factor per channel.
template <int D, int LD>
__device__ __forceinline__ void tile16(const float* x, const float* y, const float* mid, int lane,
                                       float (&r)[4][2]) {
    const int tg = lane >> 3, sg = lane & 7;
    Two acc[4][2];
#pragma unroll
    for (int a = 0; a < 4; ++a) acc[a][0] = acc[a][1] = two(0.f, 0.f);
    for (int d0 = 0; d0 < D; d0 += 32) {
        Two part[4][2];              // (sums of 32 channels each: chains over all of them round more)
#pragma unroll
        for (int a = 0; a < 4; ++a) part[a][0] = part[a][1] = two(0.f, 0.f);
#pragma unroll 4
        for (int d = d0; d < d0 + 32; d += 4) {
            Four yv[2];
#pragma unroll
            for (int b = 0; b < 2; ++b) yv[b] = load22(y + (sg + 8 * b) * LD + d);
            if (mid) {
                const Four m = load22(mid + d);
                const Two zero = two(0.f, 0.f);
#pragma unroll
                for (int b = 0; b < 2; ++b) yv[b] = {fma2(yv[b].a, m.a, zero), fma2(yv[b].b, m.b, zero)};
            }
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const Four xv = load22(x + (tg + 4 * a) * LD + d);
#pragma unroll
                for (int b = 0; b < 2; ++b)
                    part[a][b] = fma2(xv.b, yv[b].b, fma2(xv.a, yv[b].a, part[a][b]));
            }
        }
        const Two one = two(1.f, 1.f);
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b) acc[a][b] = fma2(part[a][b], one, acc[a][b]);
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) r[a][b] = first(acc[a][b]) + second(acc[a][b]);
}

// Block pair number p of the lower triangle: (0,0), (1,0), (1,1), (2,0) ..
__device__ __forceinline__ void block_pair(int p, int& i, int& j) {
    i = p >= 6 ? 3 : p >= 3 ? 2 : p >= 1 ? 1 : 0;
    j = p - i * (i + 1) / 2;
}

// The entries of M above the diagonal blocks are zero in memory (out reads whole blocks).
__device__ __forceinline__ void clear_above(float* M) {
#pragma unroll
    for (int n = 0; n < TC * TC / 4 / PREP_THREADS; ++n) {
        const int i = threadIdx.x + n * PREP_THREADS, t = i / (TC / 4), s = i % (TC / 4) * 4;
        if (s / BT > t / BT) *reinterpret_cast<float4*>(M + t * TC + s) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

struct PrepArgs {
    const void* x; int64_t ld;           // the tokens' rows: query heads, key heads, value heads
    int k0, v0, per;                     // keys and values start at these columns; heads per key head
    const float* log_decay; int64_t ldl; // a decay per channel: [tokens, >= H * D]
    const float* ab; int64_t ldab;       // decay inputs (one per head) and step inputs
    int b_col;
    const float* A_log; const float* dt_bias;
    const int* row_start;
    int n_rows, min_chunked, H, V;
    int vec4;                            // the tokens' rows allow reads of four elements
};

// Four elements of a row of one operand per thread and item, D / 4 neighbouring lanes to a row; zeros after
// the chunk's tokens.  All requests leave before the first is waited for: rows beyond the chunk's read
// its last token again.
template <int D> constexpr int ITEMS = TC * D / 4 / PREP_THREADS;
template <int D> __device__ __forceinline__ int item_token(int n) { return (threadIdx.x + n * PREP_THREADS) / (D / 4); }
template <int D> __device__ __forceinline__ int item_channel() { return threadIdx.x % (D / 4) * 4; }
template <int D, typename T>
__device__ __forceinline__ void fetch(float4 (&r)[ITEMS<D>], const T* src, int64_t ld, int nt, bool vec4) {
    const T* p = src + item_channel<D>();
    if (vec4) {
#pragma unroll
        for (int n = 0; n < ITEMS<D>; ++n) r[n] = load4(p + min(item_token<D>(n), nt - 1) * ld);
    } else {
#pragma unroll
        for (int n = 0; n < ITEMS<D>; ++n) {
            const T* e = p + min(item_token<D>(n), nt - 1) * ld;
            r[n] = make_float4(to_float(e[0]), to_float(e[1]), to_float(e[2]), to_float(e[3]));
        }
    }
#pragma unroll
    for (int n = 0; n < ITEMS<D>; ++n)
        if (item_token<D>(n) >= nt) r[n] = make_float4(0.f, 0.f, 0.f, 0.f);
}
__device__ __forceinline__ void store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void store4(bf16* p, float4 v) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&a),
                                              *reinterpret_cast<const uint32_t*>(&b));
}
__device__ __forceinline__ float4 scaled(float4 v, float f) {
    return make_float4(v.x * f, v.y * f, v.z * f, v.w * f);
}
// The sum of the squares of an item's row.
template <int D>
__device__ __forceinline__ float row_square(float4 v) {
    float s = fmaf(v.w, v.w, fmaf(v.z, v.z, fmaf(v.y, v.y, v.x * v.x)));
#pragma unroll
    for (int o = D / 8; o >= 1; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}
// A column of the values times a factor per token: tokens beyond the chunk's give zeros.
template <typename T>
__device__ __forceinline__ void load_column(Two (&acc)[TC / 2], const T* v, int64_t ld, int nt, const float* factor) {
    float r[TC];
#pragma unroll
    for (int t = 0; t < TC; ++t) r[t] = to_float(v[min(t, nt - 1) * ld]);
#pragma unroll
    for (int t = 0; t < TC; t += 2)
        acc[t / 2] = two(t < nt ? factor[t] * r[t] : 0.f, t + 1 < nt ? factor[t + 1] * r[t + 1] : 0.f);
}

template <int D, typename T> constexpr int HEAD_LD = D + (sizeof(T) == 2 ? 8 : 4);
template <int D, typename T> constexpr size_t prep_head_smem() {
    return (size_t)2 * TC * HEAD_LD<D, T> * sizeof(T) + TC * LDT * 4;
}

// One decay per head.  The tables are products of keys and queries as they stand (bfloat16: on the tensor
// cores, exact products summed in 32-bit); the norms and decays are factors per token and per pair of
// tokens.  56 us at 2,048 tokens and 16 heads of 128 x 128; bound by the substitution's shared-memory reads
// (544 of 16 bytes a warp) and, with two CTAs of eight warps an SM, by latencies.
template <int D, typename T>
__device__ __forceinline__ void prep_head(const PrepArgs& a, const Scratch& z, const Group& group) {
    constexpr int LD = HEAD_LD<D, T>;
    extern __shared__ __align__(16) float sm[];
    float* At = sm;
    T* ks = reinterpret_cast<T*>(At + TC * LDT);
    T* qs = ks + TC * LD;
    __shared__ float log_g[TC], beta[TC], loc[TC], grow[TC], bgrow[TC], rest[TC], tot[NB], unit_k[TC], unit_q[TC];
    const int slot = blockIdx.x, head = blockIdx.y;
    RowAt row;
    if (!find_row<true>(a.row_start, a.n_rows, a.min_chunked, group, slot, row)) return;
    const int c0 = (group.first + slot - row.first) * TC, nt = min(TC, row.n_new - c0);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t tok = row.t0 + c0, at = (int64_t)slot * a.H + head;
    const T* x = reinterpret_cast<const T*>(a.x) + tok * a.ld;
    const int g = head / a.per;
    {
        float4 k[ITEMS<D>], q[ITEMS<D>];
        fetch<D, T>(k, x + a.k0 + g * D, a.ld, nt, a.vec4);
        fetch<D, T>(q, x + g * D, a.ld, nt, a.vec4);
        if (tid < TC) {
            const float* ab = a.ab + (tok + min(tid, nt - 1)) * a.ldab;
            const float v = ab[head] + a.dt_bias[head], b = ab[a.b_col + head];
            log_g[tid] = tid < nt ? -expf(a.A_log[head]) * (v > 20.f ? v : log1pf(expf(v))) : 0.f;
            beta[tid] = tid < nt ? 1.0f / (1.0f + expf(-b)) : 0.f;
        }
#pragma unroll
        for (int n = 0; n < ITEMS<D>; ++n) {
            const int t = item_token<D>(n), e = item_channel<D>();
            const float sk = row_square<D>(k[n]), sq = row_square<D>(q[n]);
            if (e == 0) {
                unit_k[t] = 1.0f / sqrtf(sk + 1e-6f);
                unit_q[t] = rsqrtf((float)D) / sqrtf(sq + 1e-6f);
            }
            store4(ks + t * LD + e, k[n]);
            store4(qs + t * LD + e, q[n]);
        }
    }
    float* M = z.M + at * TC * TC;
    clear_above(M);
    __syncthreads();
    if (tid < TC) {
        float c = 0.f, all = 0.f;
#pragma unroll
        for (int i = 0; i < BT; ++i) {
            all += log_g[tid / BT * BT + i];
            if (i == tid % BT) c = all;
        }
        loc[tid] = c;
        if (tid % BT == 0) tot[tid / BT] = all;
    }
    __syncthreads();
    if (tid < TC) {
        float pre = 0.f, post = 0.f;
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            if (i < tid / BT) pre += tot[i];
            if (i > tid / BT) post += tot[i];
        }
        grow[tid] = expf(pre + loc[tid]);
        bgrow[tid] = beta[tid] * grow[tid] * unit_k[tid];
        rest[tid] = expf(tot[tid / BT] - loc[tid] + post) * unit_k[tid];
    }
    for (int e = tid; e < D; e += PREP_THREADS)
        z.decay[at * D + e] = expf((tot[0] + tot[1]) + (tot[2] + tot[3]));
    auto entry = [&](bool with_q, int t, int s, float dot) {     // a table's entry from its product
        const int i = t / BT, j = s / BT;
        float mid = 0.f;
#pragma unroll
        for (int b = 1; b < NB - 1; ++b)
            if (b > j && b < i) mid += tot[b];
        const float e = i == j ? loc[t] - loc[s] : loc[t] + mid + (tot[j] - loc[s]);
        const float w = dot * unit_k[s] * expf(e);
        if (with_q) M[t * TC + s] = s <= t ? unit_q[t] * w : 0.f;
        else At[s * LDT + t] = s < t ? -beta[t] * unit_k[t] * w : 0.f;
    };
    if constexpr (sizeof(T) == 2) {
        // a warp has 16 rows of one table, up to the diagonal block
        const int i = warp >> 1;
        const bool with_q = warp & 1;
        float acc[NB][2][4];
#pragma unroll
        for (int j = 0; j < NB; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int w = 0; w < 4; ++w) acc[j][h][w] = 0.f;
        const uint32_t left = smem_addr((with_q ? qs : ks) + (BT * i + (lane & 15)) * LD + (lane >> 4) * 8);
        const uint32_t right = smem_addr(ks + ((lane >> 4) * 8 + (lane & 7)) * LD + ((lane >> 3) & 1) * 8);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
            uint32_t f[4];
            ldsm4(f, left + 32 * kk);
#pragma unroll
            for (int j = 0; j < NB; ++j)
                if (j <= i) {
                    uint32_t b[4];
                    ldsm4(b, right + (BT * j * LD + 16 * kk) * 2);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        float part[4] = {0.f, 0.f, 0.f, 0.f};
                        mma_bf16(part, f, b + 2 * h);
#pragma unroll
                        for (int w = 0; w < 4; ++w) acc[j][h][w] += part[w];
                    }
                }
        }
#pragma unroll
        for (int j = 0; j < NB; ++j)
            if (j <= i)
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int w = 0; w < 4; ++w)
                        entry(with_q, BT * i + (lane >> 2) + (w >> 1) * 8, BT * j + 8 * h + (lane & 3) * 2 + (w & 1),
                              acc[j][h][w]);
    } else {
        for (int it = warp; it < 20; it += PREP_THREADS / 32) {
            int i, j;
            block_pair(it >> 1, i, j);
            const bool with_q = it & 1;
            float r[4][2];
            tile16<D, LD>((const float*)(with_q ? qs : ks) + BT * i * LD, (const float*)ks + BT * j * LD, nullptr, lane, r);
#pragma unroll
            for (int ra = 0; ra < 4; ++ra)
#pragma unroll
                for (int rb = 0; rb < 2; ++rb)
                    entry(with_q, BT * i + (lane >> 3) + 4 * ra, BT * j + (lane & 7) + 8 * rb, r[ra][rb]);
        }
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < ITEMS<D>; ++n) {
        const int t = item_token<D>(n), e = item_channel<D>();
        store4(z.Q + (at * TC + t) * D + e, scaled(load4(qs + t * LD + e), grow[t] * unit_q[t]));
        int ty, d;
        y_source(tid + n * PREP_THREADS, ty, d);
        const T* k = ks + ty * LD + d;
        store4(z.Y + at * TC * D + 4 * (tid + n * PREP_THREADS),
               make_float4(to_float(k[0]) * rest[ty], to_float(k[LD]) * rest[ty + 1],
                           to_float(k[8 * LD]) * rest[ty + 8], to_float(k[9 * LD]) * rest[ty + 9]));
    }
    for (int at_col = tid; at_col < (D + a.V + 31) / 32 * 32; at_col += PREP_THREADS) {    // whole warps
        const int col = min(at_col, D + a.V - 1);
        Two acc[TC / 2];
        if (col < D) {
#pragma unroll
            for (int t = 0; t < TC; t += 2)
                acc[t / 2] = two(bgrow[t] * to_float(ks[t * LD + col]), bgrow[t + 1] * to_float(ks[(t + 1) * LD + col]));
        } else {
            load_column(acc, x + a.v0 + (int64_t)head * a.V + (col - D), a.ld, nt, beta);
        }
        substitute(acc, At);
        if (at_col < D + a.V)
            store_column(acc, z.W + at * TC * D, col < D ? col : -1, z.X + (at * a.V + (col - D)) * TC);
    }
}

template <int D> constexpr size_t prep_channels_smem() {
    return (size_t)(3 * TC * (D + 4) + TC * LDT + 15 * D + SOLVED) * 4;
}

// The pairs of tokens inside a block: x_t with every y_s, s < t (own: s <= t), decayed from s to t.  D / 4 lanes
// share the channels; a lane keeps its channels of the y's in registers and fades them token by token, so
// that no exponential is needed, and the lanes' sums are exchanged per t.  `fade`: the tokens' decays.
// The result, times -factor[t] if there are factors, goes to to[t * to_t + s * to_s]; zero for other s.  (One body for
// both tables: it is 1,700 instructions long.)
template <int D>
__device__ __forceinline__ void block_pairs(const float* x, const float* y, const float* fade, bool own_too,
                                            const float* factor, float* to, int to_t, int to_s) {
    constexpr int LD = D + 4, LANES = D / 4;
    const int e = threadIdx.x % LANES * 4, lane = threadIdx.x & 31;
    const Two zero = two(0.f, 0.f);
    Two ys[BT][2];
#pragma unroll
    for (int t = 0; t < BT; ++t) {
        const Four xv = load22(x + t * LD + e), gv = load22(fade + t * LD + e), own = load22(y + t * LD + e);
#pragma unroll
        for (int s = 0; s < t; ++s) {
            ys[s][0] = fma2(ys[s][0], gv.a, zero);
            ys[s][1] = fma2(ys[s][1], gv.b, zero);
        }
        ys[t][0] = own.a;
        ys[t][1] = own.b;
        float v[BT];
#pragma unroll
        for (int s = 0; s < BT; ++s) {
            v[s] = 0.f;
            if (s <= t) {
                const Two d = fma2(xv.b, ys[s][1], fma2(xv.a, ys[s][0], zero));
                v[s] = first(d) + second(d);
                if (s == t && !own_too) v[s] = 0.f;
            }
        }
        int n = BT;
#pragma unroll
        for (int o = LANES / 2; o >= 1; o >>= 1) {
            if (n > 1) {        // a lane keeps the half of its values that its own number says
                n >>= 1;
                const bool up = lane & o;
#pragma unroll
                for (int i = 0; i < BT / 2; ++i)
                    if (i < n) {
                        const float give = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
                        v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                    }
            } else {
                v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
            }
        }
        const float by = factor ? -factor[t] : 1.f;
        if (LANES == 8) {
            to[t * to_t + (lane & 7) * 2 * to_s] = by * v[0];
            to[t * to_t + ((lane & 7) * 2 + 1) * to_s] = by * v[1];
        } else if (LANES == 16) {
            to[t * to_t + (lane & 15) * to_s] = by * v[0];
        } else if (!(lane & 1)) {
            to[t * to_t + (lane >> 1) * to_s] = by * v[0];
        }
    }
}

// A decay per key channel.  Arrays in shared memory change what they hold: R = q, then q e^{l}; U = k, then
// k e^{l}; L = the decays, then k e^{border - l} (l: sums of logarithms from the block's border on).  One
// CTA an SM: its shared memory allows no second.  227 us at 3,001 tokens in four rows and 16 heads of 128 x 128
// (960 CTAs, 6.5 rounds): latencies of eight warps (0.34 instructions a cycle and scheduler).
template <int D, typename T>
__device__ __forceinline__ void prep_channels(const PrepArgs& a, const Scratch& z, const Group& group) {
    constexpr int LD = D + 4;
    extern __shared__ __align__(16) float sm[];
    float* R = sm;
    float* U = R + TC * LD;
    float* L = U + TC * LD;
    float* At = L + TC * LD;                      // [s][t]: -A_ts
    float* tot = At + TC * LDT;                   // [NB][D]: a block's sum
    float* pre = tot + NB * D;                    // [NB][D]: e^{blocks before}
    float* post = pre + NB * D;                   // [NB][D]: e^{blocks after}
    float* mids = post + NB * D;                  // [3][D]: e^{blocks between} of (2,0), (3,1), (3,0)
    __shared__ float beta[TC];
    const int slot = blockIdx.x, head = blockIdx.y;
    RowAt row;
    if (!find_row<true>(a.row_start, a.n_rows, a.min_chunked, group, slot, row)) return;
    const int c0 = (group.first + slot - row.first) * TC, nt = min(TC, row.n_new - c0);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t tok = row.t0 + c0, at = (int64_t)slot * a.H + head;
    const T* x = reinterpret_cast<const T*>(a.x) + tok * a.ld;
    const float* lg = a.log_decay + tok * a.ldl + (int64_t)head * D;
    const int g = head / a.per;
    {
        float4 k[ITEMS<D>], q[ITEMS<D>], l[ITEMS<D>];
        fetch<D, T>(k, x + a.k0 + g * D, a.ld, nt, a.vec4);
        fetch<D, T>(q, x + g * D, a.ld, nt, a.vec4);
        fetch<D, float>(l, lg, a.ldl, nt, a.vec4);
        if (tid < TC) {
            const float b = a.ab[(tok + min(tid, nt - 1)) * a.ldab + a.b_col + head];
            beta[tid] = tid < nt ? 1.0f / (1.0f + expf(-b)) : 0.f;
        }
#pragma unroll
        for (int n = 0; n < ITEMS<D>; ++n) {
            const int o = item_token<D>(n) * LD + item_channel<D>();
            store4(U + o, scaled(k[n], 1.0f / sqrtf(row_square<D>(k[n]) + 1e-6f)));
            store4(R + o, scaled(q[n], rsqrtf((float)D) / sqrtf(row_square<D>(q[n]) + 1e-6f)));
            store4(L + o, make_float4(expf(l[n].x), expf(l[n].y), expf(l[n].z), expf(l[n].w)));
        }
    }
    float* M = z.M + at * TC * TC;
    clear_above(M);
    __syncthreads();
    // pairs inside the blocks: D / 4 lanes have a block of one table
    for (int unit = tid / (D / 4); unit < 2 * NB; unit += PREP_THREADS / (D / 4)) {
        const int r0 = BT * (unit % NB);
        const float *u = U + r0 * LD, *fade = L + r0 * LD;
        const bool with_q = unit >= NB;
        block_pairs<D>(with_q ? R + r0 * LD : u, u, fade, with_q, with_q ? nullptr : beta + r0,
                       with_q ? M + r0 * TC + r0 : At + r0 * LDT + r0, with_q ? TC : 1, with_q ? 1 : LDT);
    }
    __syncthreads();
    for (int i = tid; i < NB * D; i += PREP_THREADS) {       // decays into the operands
        const int b = i / D, e = i - b * D;
        float l[BT], all = 0.f;
        // (the logarithms as they were given: a decay that underflows still has its own)
#pragma unroll
        for (int t = 0; t < BT; ++t) l[t] = lg[min(BT * b + t, nt - 1) * a.ldl + e];
#pragma unroll
        for (int t = 0; t < BT; ++t) {
            all += BT * b + t < nt ? l[t] : 0.f;
            l[t] = all;
        }
        tot[i] = all;
#pragma unroll
        for (int t = 0; t < BT; ++t) {
            const int o = (BT * b + t) * LD + e;
            const float own = expf(l[t]), u = U[o];
            L[o] = u * expf(all - l[t]);
            U[o] = u * own;
            R[o] *= own;
        }
    }
    __syncthreads();
    for (int e = tid; e < D; e += PREP_THREADS) {
        const float a0 = tot[e], a1 = tot[D + e], a2 = tot[2 * D + e], a3 = tot[3 * D + e];
        pre[e] = 1.f; pre[D + e] = expf(a0); pre[2 * D + e] = expf(a0 + a1); pre[3 * D + e] = expf(a0 + a1 + a2);
        post[3 * D + e] = 1.f; post[2 * D + e] = expf(a3); post[D + e] = expf(a2 + a3); post[e] = expf(a1 + a2 + a3);
        mids[e] = expf(a1); mids[D + e] = expf(a2); mids[2 * D + e] = expf(a1 + a2);
        z.decay[at * D + e] = expf((a0 + a1) + (a2 + a3));
    }
    __syncthreads();
    for (int it = warp; it < 12; it += PREP_THREADS / 32) {    // pairs between blocks
        const int p = it % 6, i = p >= 3 ? 3 : p >= 1 ? 2 : 1, j = p - (i * (i - 1)) / 2;
        const bool with_q = it >= 6;
        const float* mid = i - j == 1 ? nullptr : mids + (i - j == 3 ? 2 : j) * D;
        float r[4][2];
        tile16<D, LD>((with_q ? R : U) + BT * i * LD, L + BT * j * LD, mid, lane, r);
#pragma unroll
        for (int ra = 0; ra < 4; ++ra)
#pragma unroll
            for (int rb = 0; rb < 2; ++rb) {
                const int t = BT * i + (lane >> 3) + 4 * ra, s = BT * j + (lane & 7) + 8 * rb;
                if (with_q) M[t * TC + s] = r[ra][rb];
                else At[s * LDT + t] = -beta[t] * r[ra][rb];
            }
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < ITEMS<D>; ++n) {
        const int i = tid + n * PREP_THREADS, t = item_token<D>(n), e = item_channel<D>();
        const float4 q = load4(R + t * LD + e), gq = load4(pre + t / BT * D + e);
        store4(z.Q + (at * TC + t) * D + e, make_float4(q.x * gq.x, q.y * gq.y, q.z * gq.z, q.w * gq.w));
        int ty, d;
        y_source(i, ty, d);
        const float* y = L + ty * LD + d;
        const float gy = post[ty / BT * D + d];
        store4(z.Y + at * TC * D + 4 * i, make_float4(y[0] * gy, y[LD] * gy, y[8 * LD] * gy, y[9 * LD] * gy));
    }
    float* solved = mids + 3 * D;
    for (int at_col = tid; at_col < (D + a.V + 31) / 32 * 32; at_col += PREP_THREADS) {    // whole warps
        const int col = min(at_col, D + a.V - 1);
        const bool is_w = col < D;
        const T* v = x + a.v0 + (int64_t)head * a.V + max(col - D, 0);
        float* X0 = z.X + (at * a.V + (col - D)) * TC;
        solve_column(At, solved + tid,
                     [&](int t) { return is_w ? U[t * LD + col] : to_float(v[min(t, nt - 1) * a.ld]); },
                     [&](int t, float raw) {
                         return is_w ? beta[t] * pre[t / BT * D + col] * raw : t < nt ? beta[t] * raw : 0.f;
                     },
                     [&](int t0, const Two (&acc)[BT / 2]) {
                         if (at_col < D + a.V) store_column(acc, t0, z.W + at * TC * D, is_w ? col : -1, X0);
                     });
    }
}

// `beside`: the kernel runs beside its predecessor, whose results it does not use, and ends after it.
template <int D, typename T, bool CHANNEL>
__global__ void __launch_bounds__(PREP_THREADS, CHANNEL ? 1 : 2)
prep_kernel(const PrepArgs a, const Scratch z, const Group group) {
    if (!group.beside) pdl_wait();
    pdl_trigger();
    if constexpr (CHANNEL) prep_channels<D, T>(a, z, group);
    else prep_head<D, T>(a, z, group);
    if (group.beside) pdl_wait();
}

// ------------------------------------------------------------------------------------- pass

// c += a b of 32-bit operands as bfloat16 parts (PARTS each, which hold all of their 24 bits): the six
// products of parts that reach above 2^-24, small ones first.  mma.sync cuts its sums off instead of
// rounding them: longer sums are therefore added up outside, from a fresh accumulator per 16 products.
// (600 tokens, weak decays, 128 x 128, error of the read-outs against 64 bits: 1.3e-6 with one accumulator
// over all 192 products, 2.2e-7 now, 3.2e-7 token by token in fmaf; 2,048 tokens, 16 heads: 245 -> 252 us.)
__device__ __forceinline__ void mma_parts(float* c, const uint32_t (*a)[4], const uint32_t (*b)[2]) {
    mma_bf16(c, a[1], b[1]);
    mma_bf16(c, a[0], b[2]);
    mma_bf16(c, a[2], b[0]);
    mma_bf16(c, a[0], b[1]);
    mma_bf16(c, a[1], b[0]);
    mma_bf16(c, a[0], b[0]);
}
__device__ __forceinline__ void add_parts(float* c, const uint32_t (*a)[4], const uint32_t (*b)[2]) {
    float sum[4] = {0.f, 0.f, 0.f, 0.f};
    mma_parts(sum, a, b);
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] += sum[i];
}
__device__ __forceinline__ void split_b(float4 v, uint32_t (*b)[2]) {
    uint32_t p[PARTS];
    split2(v.x, v.y, p);
#pragma unroll
    for (int i = 0; i < PARTS; ++i) b[i][0] = p[i];
    split2(v.z, v.w, p);
#pragma unroll
    for (int i = 0; i < PARTS; ++i) b[i][1] = p[i];
}

constexpr int LDP = TC + 8;              // row stride of what the pass's warps exchange

// A warp has 16 channels of 16 columns, S^T as mma.m16n8k16 leaves it, which is how the next product
// takes it as its left operand: the state never leaves the registers.  X^T = X0^T - S0^T W^T: each warp
// multiplies its own channels and the warps' sums meet in shared memory; S^T <- e^{L_last} S0^T + X^T y~:
// each warp for its own channels, X split into parts once by whom adds it up.  W and y~ are used once per
// CTA and come straight from memory into the registers of the thread that needs them, a chunk ahead.
//
// What bounds it, for one row: the chain of chunks, each two barriers and two products of K = 16 and 64, of
// which the 192 mma.sync a scheduler issues take the most: 89 us for 32 chunks of 128 x 128 with 16 heads (128
// CTAs), 2.8 us a chunk.  With more CTAs than SMs, the mma.sync and the reads of W and y~, which every 16 columns
// repeat: four rows of 401 to 1,201 tokens 138 us, where the longest alone is 19 chunks.  As fused
// multiply-adds from shared memory the layer of one row took 348 us where this took 333.
template <int D>
__global__ void __launch_bounds__(2 * D)
pass_kernel(const Scratch z, const Group group, float* __restrict__ state, const int* __restrict__ row_start,
            const int* __restrict__ row_slot, int n_rows, int min_chunked, int H, int V) {
    constexpr int WARPS = D / 16, THREADS = 32 * WARPS, QUADS = NC * TC / 4 / THREADS;
    __shared__ __align__(16) float sums[WARPS][NC][LDP];
    __shared__ __align__(16) bf16 parts[PARTS][NC][LDP];
    pdl_wait();
    pdl_trigger();
    const int head = blockIdx.y, col0 = blockIdx.x * NC;
    RowAt row;
    if (!find_row<false>(row_start, n_rows, min_chunked, group, blockIdx.z, row)) return;
    // the row's chunks of this group: the state goes through memory between groups
    const int slot0 = max(row.first - group.first, 0);
    const int n_chunks = min(row.first + (row.n_new + TC - 1) / TC - group.first, group.count) - slot0;
    if (n_chunks <= 0) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t chunk0 = (int64_t)slot0 * H + head;
    // S[n][i]: column lane / 4 + 8 (i / 2), channel 16 warp + 8 n + 2 (lane % 4) + i % 2
    const int column = lane >> 2, channel = 16 * warp + (lane & 3) * 2;
    const bool live[2] = {col0 + column < V, col0 + column + 8 < V};
    float S[2][4];
    float* st = state + (((int64_t)row_slot[row.row] * H + head) * V + col0 + column) * D + channel;
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float2 v = make_float2(0.f, 0.f);
            if (live[h]) v = *reinterpret_cast<const float2*>(st + 8 * h * D + 8 * n);
            S[n][2 * h] = v.x;
            S[n][2 * h + 1] = v.y;
        }
    float4 w[8], y[8];
    auto fetch_pieces = [&](float4 (&v)[8], const float* src) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = load4(src + ((warp * 8 + i) * 32 + lane) * 4);
    };
    fetch_pieces(w, z.W + chunk0 * TC * D);
    for (int j = 0; j < n_chunks; ++j) {
        const int64_t at = chunk0 + (int64_t)j * H;
        fetch_pieces(y, z.Y + at * TC * D);
        float* Xg = z.X + (at * V + col0) * TC;
        float4 x0[QUADS];
#pragma unroll
        for (int i = 0; i < QUADS; ++i) {
            const int q = tid + i * THREADS, c = q / (TC / 4);
            x0[i] = col0 + c < V ? load4(Xg + q * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        // ---- S0^T W^T of this warp's channels
        uint32_t left[PARTS][4];
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t p[PARTS];
                split2(S[n][2 * h], S[n][2 * h + 1], p);
#pragma unroll
                for (int i = 0; i < PARTS; ++i) left[i][2 * n + h] = p[i];
            }
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
            uint32_t right[PARTS][2];
            split_b(w[n], right);
            mma_parts(acc, left, right);
            float* p = &sums[warp][column][8 * n + (lane & 3) * 2];
            *reinterpret_cast<float2*>(p) = make_float2(acc[0], acc[1]);
            *reinterpret_cast<float2*>(p + 8 * LDP) = make_float2(acc[2], acc[3]);
        }
        if (j + 1 < n_chunks) fetch_pieces(w, z.W + (at + H) * TC * D);
        // ---- the state that the out kernel reads
        float* Sg = z.S + (at * V + col0 + column) * D + channel;
        float2 dec[2];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            dec[n] = *reinterpret_cast<const float2*>(z.decay + at * D + channel + 8 * n);
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (live[h])
                    *reinterpret_cast<float2*>(Sg + 8 * h * D + 8 * n) = make_float2(S[n][2 * h], S[n][2 * h + 1]);
        }
        __syncthreads();
        // ---- X, and its parts
#pragma unroll
        for (int i = 0; i < QUADS; ++i) {
            const int q = tid + i * THREADS, c = q / (TC / 4), t = q % (TC / 4) * 4;
            float4 x = x0[i];
            float4 sum = load4(&sums[0][c][t]);
#pragma unroll
            for (int k = 1; k < WARPS; ++k) {
                const float4 more = load4(&sums[k][c][t]);
                sum.x += more.x; sum.y += more.y; sum.z += more.z; sum.w += more.w;
            }
            x.x -= sum.x; x.y -= sum.y; x.z -= sum.z; x.w -= sum.w;
            if (col0 + c < V) *reinterpret_cast<float4*>(Xg + q * 4) = x;
            uint32_t a[PARTS], b[PARTS];
            split2(x.x, x.y, a);
            split2(x.z, x.w, b);
#pragma unroll
            for (int k = 0; k < PARTS; ++k)
                *reinterpret_cast<uint2*>(&parts[k][c][t]) = make_uint2(a[k], b[k]);
        }
        __syncthreads();
        // ---- S^T <- e^{L_last} S0^T + X^T y~
        float acc[2][4];
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[n][i] = 0.f;
#pragma unroll
        for (int k = 0; k < TC / 16; ++k) {
#pragma unroll
            for (int i = 0; i < PARTS; ++i)
                ldsm4(left[i], smem_addr(&parts[i][lane & 15][16 * k + (lane >> 4) * 8]));
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                uint32_t right[PARTS][2];
                split_b(y[2 * k + n], right);
                add_parts(acc[n], left, right);
            }
        }
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                S[n][2 * h] = fmaf(dec[n].x, S[n][2 * h], acc[n][2 * h]);
                S[n][2 * h + 1] = fmaf(dec[n].y, S[n][2 * h + 1], acc[n][2 * h + 1]);
            }
    }
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (live[h])
                *reinterpret_cast<float2*>(st + 8 * h * D + 8 * n) = make_float2(S[n][2 * h], S[n][2 * h + 1]);
}

// -------------------------------------------------------------------------------------- out

constexpr int LDO = TC + 8;
template <int D> constexpr size_t out_smem() { return (size_t)(TC + OUT_COLS) * (D + 8 + LDO) * 4; }

// o of a chunk, head and 64 columns: a warp has 16 tokens and 32 columns, both operands of both products
// lie in shared memory with the summed index last and are split into parts as they are read.  Row strides
// are 8 banks apart: a half-warp's reads of two elements meet every bank once.  46 us at
// 2,048 tokens and 16 heads of 128 x 128, 78 us at 3,001 (1,056 and 1,920 CTAs, two an SM): mma.sync, the split's
// arithmetic, and 106 KB of loads a CTA that only the other CTA of the SM covers.  (As fused multiply-adds it
// was bound by shared-memory reads.)
template <int D>
__global__ void __launch_bounds__(OUT_THREADS, 2)
out_kernel(const Scratch z, const Group group, const int* __restrict__ row_start, float* __restrict__ out,
           int n_rows, int min_chunked, int H, int V) {
    constexpr int LD = D + 8;
    extern __shared__ __align__(16) float sm[];
    float* Qs = sm;                       // [TC][LD]
    float* Ss = Qs + TC * LD;             // [OUT_COLS][LD]
    float* Ms = Ss + OUT_COLS * LD;       // [TC][LDO]
    float* Xs = Ms + TC * LDO;            // [OUT_COLS][LDO]
    pdl_wait();
    pdl_trigger();
    const int slot = blockIdx.z, head = blockIdx.y, col0 = blockIdx.x * OUT_COLS;
    RowAt row;
    if (!find_row<true>(row_start, n_rows, min_chunked, group, slot, row)) return;
    const int c0 = (group.first + slot - row.first) * TC, nt = min(TC, row.n_new - c0);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t at = (int64_t)slot * H + head;
    const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int i = tid; i < TC * D / 4; i += OUT_THREADS) {
        const int t = i / (D / 4), e = (i - t * (D / 4)) * 4;
        cp16(Qs + t * LD + e, z.Q + at * TC * D + t * D + e);
        if (col0 + t < V) cp16(Ss + t * LD + e, z.S + (at * V + col0 + t) * D + e);
        else *reinterpret_cast<float4*>(Ss + t * LD + e) = none;
    }
    for (int i = tid; i < TC * TC / 4; i += OUT_THREADS) {
        const int t = i / (TC / 4), e = (i - t * (TC / 4)) * 4;
        cp16(Ms + t * LDO + e, z.M + at * TC * TC + t * TC + e);
        if (col0 + t < V) cp16(Xs + t * LDO + e, z.X + (at * V + col0 + t) * TC + e);
        else *reinterpret_cast<float4*>(Xs + t * LDO + e) = none;
    }
    cp_wait_all();
    __syncthreads();
    const int r0 = (warp & 3) * 16, n0 = (warp >> 2) * 32;
    const int place = lane >> 2, pair = (lane & 3) * 2;
    float acc[4][4];
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[n][i] = 0.f;
    auto add = [&](const float* left, const float* right, int ld, int K) {
        const float* l = left + (r0 + place) * ld + pair;
        const float* q = right + (n0 + place) * ld + pair;
#pragma unroll 2
        for (int k = 0; k < K; k += 16) {
            uint32_t a[PARTS][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {       // rows place, place + 8 and again eight columns on
                const float2 x = *reinterpret_cast<const float2*>(l + (i & 1) * 8 * ld + k + (i >> 1) * 8);
                uint32_t p[PARTS];
                split2(x.x, x.y, p);
#pragma unroll
                for (int w = 0; w < PARTS; ++w) a[w][i] = p[w];
            }
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                const float2 x = *reinterpret_cast<const float2*>(q + 8 * n * ld + k);
                const float2 y = *reinterpret_cast<const float2*>(q + 8 * n * ld + k + 8);
                uint32_t b[PARTS][2];
                split_b(make_float4(x.x, x.y, y.x, y.y), b);
                add_parts(acc[n], a, b);
            }
        }
    };
    add(Qs, Ss, LD, D);
    add(Ms, Xs, LDO, r0 + 16);            // (the table is zero beyond the warp's last token)
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int t = r0 + place + (i >> 1) * 8, c = col0 + n0 + 8 * n + pair + (i & 1);
            if (t < nt && c < V) out[((int64_t)(row.t0 + c0 + t) * H + head) * V + c] = acc[n][i];
        }
}

// --------------------------------------------------------------------------------- launches

// beside: the kernel before this launch in the stream belongs to the same step (the rows without chunks), was
// launched as an ordinary kernel, so that all before it is done once it runs, and lets its successor start.  It
// shares only inputs with the first prep, which then runs at its side; as prep ends after it, every later kernel
// waits for both.  Rows of 127 and 128 tokens, 4 heads of 128 x 128, one decay per head / per channel: 81 / 93 us
// one after the other, 64 / 64 so (47 / 49 if the tokens of both were taken in order); 16 heads: 95 / 103,
// 95 / 97 (92 / 92); 32 heads: 143 / 148, 142 / 148 (181 / 176).
// `slots`: room of the scratch.  Launches for every chunk that a step of n_tokens tokens can have: a row with
// chunks ends at most one short of a whole one more than its tokens fill.
template <int D, typename T, bool CHANNEL>
static inline int launch(const PrepArgs& a, const Scratch& z, float* state, const int* row_slot, float* out,
                         int n_tokens, int slots, bool beside, cudaStream_t stream) {
    const auto prep = prep_kernel<D, T, CHANNEL>;
    constexpr size_t smem = CHANNEL ? prep_channels_smem<D>() : prep_head_smem<D, T>();
    cudaError_t e = cudaFuncSetAttribute(prep, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    e = cudaFuncSetAttribute(out_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)out_smem<D>());
    if (e != cudaSuccess) return (int)e;
    const int rows = std::min(a.n_rows, n_tokens / a.min_chunked), chunks = n_tokens / TC + rows;
    const int per_row = (a.min_chunked + TC - 1) / TC;
    if (rows == 0) return 0;
    for (Group g = {0, 0, beside}; g.first < chunks; g.first += slots, g.beside = false) {
        g.count = std::min(slots, chunks - g.first);
        e = sllm_launch_pdl(prep, dim3(g.count, a.H), dim3(PREP_THREADS), smem, stream, a, z, g);
        if (e != cudaSuccess) return (int)e;
        // (rows of at least per_row chunks: this many can have some in the group)
        const int group_rows = std::min(rows, g.count / per_row + 2);
        // (an ordinary launch: begun beside prep, its CTAs take the places that prep leaves first, two on some
        // SMs and none on others, and one row's chain of chunks goes by the slowest: the three kernels took
        // 256 us so, 186 now, 350 and 277 per channel; four rows of 601 to 1,201 tokens 314 and 303)
        pass_kernel<D><<<dim3((a.V + NC - 1) / NC, a.H, group_rows), 2 * D, 0, stream>>>(
            z, g, state, a.row_start, row_slot, a.n_rows, a.min_chunked, a.H, a.V);
        e = cudaGetLastError();
        if (e != cudaSuccess) return (int)e;
        e = sllm_launch_pdl(out_kernel<D>, dim3((a.V + OUT_COLS - 1) / OUT_COLS, a.H, g.count), dim3(OUT_THREADS),
                            out_smem<D>(), stream, z, g, a.row_start, out, a.n_rows, a.min_chunked, a.H, a.V);
        if (e != cudaSuccess) return (int)e;
    }
    return 0;
}

}  // namespace chunks
}  // namespace sllm
