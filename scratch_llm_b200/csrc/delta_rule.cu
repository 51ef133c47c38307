// The gated delta rule: a linear recurrence whose state is one matrix S [D, V] per head and
// request, carried in 32-bit from token to token.  Per token, with a unit key k and a scaled
// unit query q of size D, a value v of size V, a decay g in (0, 1) and a step size beta:
//
//     S  <-  g S
//     u   =  beta (v - S^T k)
//     S  <-  S + k u^T
//     o   =  S^T q                       (the read-out sees the token's own write)
//
// with, computed here in 32-bit from what the projections and the short convolution left:
//     k = k_raw / sqrt(sum(k_raw^2) + 1e-6),   q = q_raw / sqrt(sum(q_raw^2) + 1e-6) * D^(-1/2)
//     beta = sigmoid(b),   g = exp(-exp(A_log) * softplus(a + dt_bias))
// Head h of H reads key/query head h / (H / G).
//
// Columns of S are independent of each other: u_j and o_j need column j of S only.  A warp
// owns one column (its 32 lanes hold D / 32 elements each, in quads), a CTA of 16 warps takes
// 16 columns of one (row, head).  Tokens are taken in chunks of CT = 16, and inside a chunk the
// recurrence is unrolled so that only a small triangular system is sequential.  With S0 the
// state at the chunk's start, L_t the sum of log g up to token t of the chunk, per column:
//
//     p_t = S0^T k_t,  r_t = S0^T q_t                          (independent dot products)
//     u_t = beta_t ( v_t - e^{L_t} p_t - sum_{s<t} e^{L_t - L_s} (k_s . k_t) u_s )
//     o_t = e^{L_t} r_t + sum_{s<=t} e^{L_t - L_s} (k_s . q_t) u_s
//     S   = e^{L_last} S0 + sum_s e^{L_last - L_s} k_s u_s^T
//
// which is the rule above written out (S'_t = e^{L_t} S0 + sum_{s<t} e^{L_t - L_s} k_s u_s^T).
// The CTA norms the chunk's keys and queries, evaluates its gates and the table of weighted dot
// products once (all of this is shared by its 16 columns).  A warp then forms its 32 partial
// dot products with S0, sums them across its lanes so that lane t holds p_t and lane 16 + t
// holds r_t (31 shuffles), and solves the triangular system column by column: lane s
// announces u_s, every lane adds its row's weight times u_s to its own sum, so that the lanes
// 16 + t end with the read-outs o_t.  Last comes the rank-16 update of its elements of S.
// All of it is 32-bit.  A chunk's inputs are requested one chunk ahead and wait in registers.
// A row reads its state from its slot and writes it back; rows without tokens touch nothing.  Rows of one
// token (decoding) have a kernel of their own, delta_rule_step_kernel.
//
// A decay per key CHANNEL (log_decay != null: float [tokens, H * D], the logarithm of each
// channel's factor, at most 0): S <- diag(g) S in the rule's first line.  With L_t now the vector
// of the channels' sums of log g up to token t of the chunk, the same unrolling holds with
//     p_t = S0^T (e^{L_t} * k_t),   r_t = S0^T (e^{L_t} * q_t),
//     weights  sum_d k_s[d] x_t[d] e^{L_t[d] - L_s[d]}   (x = k for s < t, x = q for s <= t),
//     S = diag(e^{L_last}) S0 + sum_s (e^{L_last - L_s} * k_s) u_s^T.
// Every exponent that is formed is at most 0 (a later token's sum minus an earlier one's), so
// nothing overflows however strong the decay; the weights cost one exponential per channel and
// pair of tokens, shared by the CTA's 16 columns.  The step size then comes from column b_col +
// head of `ab`, and A_log / dt_bias are the caller's business (they are inside log_decay).
//
// Rows of at least min_chunked tokens go to the kernels of delta_chunks.cuh where the key size fits them.  A row
// takes one path whatever else is in its step, and the paths of a step run side by side as far as the stream's
// order lets them (sllm_delta_rule).
//
// The weights depend on keys, queries and decays alone: delta_weights_kernel forms the tables of
// ALL chunks of a step in parallel before the scan starts, which then reads its chunk's table.
//
// Compiled once per key size: -DSLLM_HEAD_DIM=<D>.
#include "delta_chunks.cuh"

#ifndef SLLM_HEAD_DIM
#error "compile with -DSLLM_HEAD_DIM=<key size>"
#endif

namespace sllm {

constexpr int D = SLLM_HEAD_DIM;
static_assert(D >= 1 && D <= 256, "key size: 1 to 256 (a chunk of keys and queries is staged in shared memory)");
constexpr int QUADS = (D + 3) / 4;                  // groups of 4 elements of a column
constexpr int QPL = (QUADS + 31) / 32;              // quads per lane
constexpr int LDK = 4 * QUADS + 4;                  // row stride of the staged keys / queries
constexpr int CT = 16;                              // tokens per chunk
constexpr int COLS = 16;                            // columns (warps) per CTA
constexpr int THREADS = 32 * COLS;

struct DeltaArgs {
    const void* act; int64_t ld_act;     // [tokens, >= 2 G D + H V]: q heads, k heads, v heads
    const float* ab; int64_t ld_ab;      // [tokens, >= 2 H]: a (decay input) then b (step input)
    const float* A_log; const float* dt_bias;   // [H]
    float* state;                        // [slots, H, V, D]
    const int* row_start; const int* row_slot;
    float* out;                          // [tokens, H * V]
    int H; int G; int V;
    // a decay per key channel: [tokens, >= H * D] logarithms (null: one decay per head from a)
    const float* log_decay; int64_t ld_decay;
    int b_col;                           // the step input of head h is ab[b_col + h]
    // with a decay per channel: the chunks' tables of weights, made by delta_weights_kernel before
    // this launch (null: every CTA forms its chunk's table itself).  The chunk that starts at
    // token t of row r has slot t / CT + r; a slot holds [H][2 CT][CT] floats.
    const float* tables;
    int min_chunked;                     // rows of at least so many tokens are the chunk kernels'
};
// the kernel for a decay per channel stages a third [CT][D] table in (static) shared memory
constexpr bool CHANNEL_FITS = D <= 192;

// Rows of one token (decoding).  A warp has CPW columns, all of them requested at once: unit vectors, gates
// and decays are formed once for the CPW, and the lanes' partial products of all columns are summed together,
// each round halving what a lane still carries (16 shuffles for 8 columns' two sums instead of 80).  48 rows x
// 32 heads of 128 x 128 (200 MB of states read and written): 89 us with a column a warp, bound by its
// instructions; 27 us now, states partly in L2 (memory alone: 31).
// `beside`: the kernel before it in the stream (other rows of the same step) shares only inputs with it; it
// runs at that kernel's side and ends after it (see launch() in delta_chunks.cuh).  64 such rows beside one of
// 130 tokens, 16 heads, one decay per head / per channel: 175 / 191 us when the kernel for several tokens
// took them a warp per column, 71 / 87 so (149 / 152 before rows of 130 tokens ran in chunks).
constexpr int CPW = QPL == 1 ? 8 : 4;
constexpr int STEP_WARPS = 4, STEP_COLS = STEP_WARPS * CPW;
template <typename T, bool CHANNEL, bool WORDS>
__device__ __forceinline__ void step(const DeltaArgs& a) {
    constexpr int LANES = 32 / CPW;       // lanes that end with a column's sums
    const int r = blockIdx.z, head = blockIdx.y;
    const int t0 = a.row_start[r];
    if (a.row_start[r + 1] - t0 != 1) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int col0 = blockIdx.x * STEP_COLS + warp * CPW;
    if (col0 >= a.V) return;
    const int n_cols = min(CPW, a.V - col0);
    float* st = a.state + (((int64_t)a.row_slot[r] * a.H + head) * a.V + col0) * D;
    float S[CPW][4 * QPL];
#pragma unroll
    for (int c = 0; c < CPW; ++c)
#pragma unroll
        for (int i = 0; i < QPL; ++i) {
            const int e = (i * 32 + lane) * 4;
            if (WORDS) {
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (c < n_cols && e < D) v = *reinterpret_cast<const float4*>(st + c * D + e);
                S[c][4 * i] = v.x; S[c][4 * i + 1] = v.y; S[c][4 * i + 2] = v.z; S[c][4 * i + 3] = v.w;
            } else {
#pragma unroll
                for (int w = 0; w < 4; ++w) S[c][4 * i + w] = (c < n_cols && e + w < D) ? st[c * D + e + w] : 0.f;
            }
        }
    const int g = head / (a.H / a.G);
    const T* act = reinterpret_cast<const T*>(a.act) + (int64_t)t0 * a.ld_act;
    const float* ab = a.ab + (int64_t)t0 * a.ld_ab;
    const int mine = lane / LANES;        // the column whose sums this lane ends with
    const float value = mine < n_cols
        ? to_float(act[2 * (int64_t)a.G * D + (int64_t)head * a.V + col0 + mine]) : 0.f;
    float kq[4 * QPL], qq[4 * QPL], fade[4 * QPL];
    float sk = 0.f, sq = 0.f, decay = 1.f;
#pragma unroll
    for (int i = 0; i < QPL; ++i)
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const int e = (i * 32 + lane) * 4 + w;
            kq[4 * i + w] = e < D ? to_float(act[(int64_t)(a.G + g) * D + e]) : 0.f;
            qq[4 * i + w] = e < D ? to_float(act[(int64_t)g * D + e]) : 0.f;
            if (CHANNEL)
                fade[4 * i + w] = e < D ? expf(a.log_decay[(int64_t)t0 * a.ld_decay + (int64_t)head * D + e]) : 1.f;
        }
    if (!CHANNEL) {
        const float x = ab[head] + a.dt_bias[head];
        decay = expf(-expf(a.A_log[head]) * (x > 20.f ? x : log1pf(expf(x))));
    }
    const float beta = 1.0f / (1.0f + expf(-ab[a.b_col + head]));
#pragma unroll
    for (int i = 0; i < 4 * QPL; ++i) {
        sk = fmaf(kq[i], kq[i], sk);
        sq = fmaf(qq[i], qq[i], sq);
    }
    sk = warp_sum(sk);
    sq = warp_sum(sq);
    const float ik = 1.0f / sqrtf(sk + 1e-6f), iq = rsqrtf((float)D) / sqrtf(sq + 1e-6f);
    float kdq = 0.f;
#pragma unroll
    for (int i = 0; i < 4 * QPL; ++i) {
        kq[i] *= ik;
        qq[i] *= iq;
        kdq = fmaf(kq[i], qq[i], kdq);
    }
    kdq = warp_sum(kdq);
    float sums[2 * CPW];                  // per column: S^T k, S^T q with the faded state
#pragma unroll
    for (int c = 0; c < CPW; ++c) {
        float p = 0.f, o = 0.f;
#pragma unroll
        for (int i = 0; i < 4 * QPL; ++i) {
            S[c][i] *= CHANNEL ? fade[i] : decay;
            p = fmaf(S[c][i], kq[i], p);
            o = fmaf(S[c][i], qq[i], o);
        }
        sums[2 * c] = p;
        sums[2 * c + 1] = o;
    }
    int n = 2 * CPW;
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        if (n > 1) {                      // a lane keeps the half of its sums that its own number says
            n >>= 1;
            const bool up = lane & o;
#pragma unroll
            for (int i = 0; i < CPW; ++i)
                if (i < n) {
                    const float give = up ? sums[i] : sums[i + n], keep = up ? sums[i + n] : sums[i];
                    sums[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                }
        } else {
            sums[0] += __shfl_xor_sync(0xffffffffu, sums[0], o);
        }
    }
    // the first half of a column's lanes holds S^T k, the second S^T q
    const float other = __shfl_xor_sync(0xffffffffu, sums[0], LANES / 2);
    const bool has_k = !(lane & (LANES / 2));
    const float u = beta * (value - (has_k ? sums[0] : other));
    if (lane % LANES == 0 && mine < n_cols)
        a.out[((int64_t)t0 * a.H + head) * a.V + col0 + mine] = fmaf(u, kdq, other);
#pragma unroll
    for (int c = 0; c < CPW; ++c) {
        const float uc = __shfl_sync(0xffffffffu, u, c * LANES);
        if (c < n_cols) {
#pragma unroll
            for (int i = 0; i < QPL; ++i) {
                const int e = (i * 32 + lane) * 4;
                float v[4];
#pragma unroll
                for (int w = 0; w < 4; ++w) v[w] = fmaf(kq[4 * i + w], uc, S[c][4 * i + w]);
                if (WORDS) {
                    if (e < D) *reinterpret_cast<float4*>(st + c * D + e) = make_float4(v[0], v[1], v[2], v[3]);
                } else {
#pragma unroll
                    for (int w = 0; w < 4; ++w)
                        if (e + w < D) st[c * D + e + w] = v[w];
                }
            }
        }
    }
}

// WORDS: columns are whole 16-byte words on 16-byte boundaries; else the state goes element by element.
template <typename T, bool CHANNEL, bool WORDS>
__global__ void __launch_bounds__(32 * STEP_WARPS) delta_rule_step_kernel(const DeltaArgs a, bool beside) {
    if (!beside) pdl_wait();
    pdl_trigger();
    step<T, CHANNEL, WORDS>(a);
    if (beside) pdl_wait();
}

// VECTOR: keys and queries are fetched in 16-byte pieces (D a multiple of 16 / sizeof(T), rows
// and base 16-byte aligned); else element by element.
template <typename T, bool VECTOR, bool CHANNEL>
__global__ void __launch_bounds__(THREADS) delta_rule_kernel(const DeltaArgs a) {
    constexpr int VEC = VECTOR ? 16 / (int)sizeof(T) : 1;
    constexpr int PER_ROW = D / VEC;                               // pieces of a key or query
    constexpr int QK_PIECES = 2 * CT * PER_ROW;                    // of a chunk
    constexpr int QK_ITEMS = (QK_PIECES + THREADS - 1) / THREADS;  // per thread
    struct alignas(16) Piece { T e[VEC]; };
    // keys and queries of the chunk as unit vectors (the query scaled), padded with zeros to
    // whole quads; lane l of a warp owns the quads l, l + 32, ... of its column
    __shared__ __align__(16) float ks[CT][LDK];
    __shared__ __align__(16) float qs[CT][LDK];
    __shared__ float vs[CT][COLS];
    // row t < 16: -e^{L_t - L_s} (k_s . k_t) for s < t; row 16 + t: e^{L_t - L_s} (k_s . q_t) for
    // s <= t; zero elsewhere
    __shared__ float weight[2 * CT][CT + 1];
    __shared__ float log_g[CT], cum_s[CT], beta_s[CT], grow_s[CT], rest_s[CT];
    // a decay per channel: the channels' log decays of the chunk's tokens, then their running
    // sums L_t, and at last e^{L_t} * k_t (the keys that meet S0); last_s: L of the chunk's last token
    __shared__ __align__(16) float lam[CHANNEL ? CT : 1][CHANNEL ? LDK : 4];
    __shared__ float last_s[CHANNEL ? LDK : 4];

    pdl_wait();
    pdl_trigger();
    const int r = blockIdx.z, head = blockIdx.y;
    const int t0 = a.row_start[r], n_new = a.row_start[r + 1] - t0;
    if (n_new <= 1 || n_new >= a.min_chunked) return;     // (one token: the step kernel)
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = head / (a.H / a.G);
    const int col0 = blockIdx.x * COLS;
    const int col = col0 + warp;
    const bool live = col < a.V;
    const T* act = reinterpret_cast<const T*>(a.act);
    const int64_t k_col0 = (int64_t)a.G * D, v_col0 = 2 * (int64_t)a.G * D;

    float S[4 * QPL];
    float* st = a.state + (((int64_t)a.row_slot[r] * a.H + head) * a.V + (live ? col : 0)) * D;
#pragma unroll
    for (int i = 0; i < QPL; ++i)
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const int e = (i * 32 + lane) * 4 + w;
            S[4 * i + w] = (live && e < D) ? st[e] : 0.f;
        }
    const float decay_rate = CHANNEL ? 0.f : expf(a.A_log[head]);
    const float dt_bias = CHANNEL ? 0.f : a.dt_bias[head];
    const float q_scale = rsqrtf((float)D);

    // columns beyond D (where D is no multiple of 4) stay zero for good
    for (int idx = tid; idx < CT * LDK; idx += THREADS) {
        (&ks[0][0])[idx] = 0.f;
        (&qs[0][0])[idx] = 0.f;
        if (CHANNEL) (&lam[0][0])[idx] = 0.f;
    }
    if (CHANNEL && tid < LDK) last_s[tid] = 0.f;
    Piece raw[QK_ITEMS];
    T raw_v = from_float<T>(0.f);
    float raw_a = 0.f, raw_b = 0.f;
    // a decay per channel: the chunk's log decays and this thread's entry of its table of weights
    // travel with the same request
    constexpr int L_ITEMS = CHANNEL ? (CT * D + THREADS - 1) / THREADS : 1;
    float raw_l[L_ITEMS], raw_w = 0.f;
    auto fetch = [&](int c0) {     // requests the chunk at c0 (tokens beyond the row: nothing)
        const int nt = min(CT, n_new - c0);
        if (CHANNEL) {
            const float* lg = a.log_decay + (int64_t)(t0 + c0) * a.ld_decay + (int64_t)head * D;
#pragma unroll
            for (int i = 0; i < L_ITEMS; ++i) {
                const int idx = tid + i * THREADS, t = idx / D, e = idx - t * D;
                raw_l[i] = (idx < CT * D && t < nt) ? lg[(int64_t)t * a.ld_decay + e] : 0.f;
            }
            if (a.tables != nullptr)
                raw_w = a.tables[(((int64_t)(t0 + c0) / CT + r) * a.H + head) * 2 * CT * CT + tid];
        }
#pragma unroll
        for (int i = 0; i < QK_ITEMS; ++i) {
            const int item = tid + i * THREADS;
            const int which = item / (CT * PER_ROW), rem = item - which * (CT * PER_ROW);
            const int t = rem / PER_ROW, c = rem - t * PER_ROW;
            if (item < QK_PIECES && t < nt) {
                const T* src = act + (int64_t)(t0 + c0 + t) * a.ld_act + (int64_t)g * D +
                               (which ? k_col0 : 0) + c * VEC;
                if (VECTOR) raw[i] = *reinterpret_cast<const Piece*>(src);
                else raw[i].e[0] = src[0];
            }
        }
        if (tid < CT * COLS) {
            const int t = tid / COLS, j = tid - t * COLS;
            if (t < nt && col0 + j < a.V)
                raw_v = act[(int64_t)(t0 + c0 + t) * a.ld_act + v_col0 + (int64_t)head * a.V +
                            col0 + j];
        }
        if (tid < nt) {
            const float* ab = a.ab + (int64_t)(t0 + c0 + tid) * a.ld_ab;
            raw_a = CHANNEL ? 0.f : ab[head];
            raw_b = ab[a.b_col + head];
        }
    };
    auto commit = [&](int nt) {    // what fetch() requested, into shared memory as 32-bit
#pragma unroll
        for (int i = 0; i < QK_ITEMS; ++i) {
            const int item = tid + i * THREADS;
            const int which = item / (CT * PER_ROW), rem = item - which * (CT * PER_ROW);
            const int t = rem / PER_ROW, c = rem - t * PER_ROW;
            if (item < QK_PIECES) {
                float* dst = (which ? &ks[t][0] : &qs[t][0]) + c * VEC;
#pragma unroll
                for (int w = 0; w < VEC; ++w) dst[w] = t < nt ? to_float(raw[i].e[w]) : 0.f;
            }
        }
        if (tid < CT * COLS) {
            const int t = tid / COLS, j = tid - t * COLS;
            vs[t][j] = (t < nt && col0 + j < a.V) ? to_float(raw_v) : 0.f;
        }
        if (tid < CT) {
            float lg = 0.f, beta = 0.f;
            if (tid < nt) {
                const float x = raw_a + dt_bias;
                const float softplus = x > 20.f ? x : log1pf(expf(x));
                lg = -decay_rate * softplus;                 // log of the decay
                beta = 1.0f / (1.0f + expf(-raw_b));
            }
            log_g[tid] = lg;
            beta_s[tid] = beta;
        }
    };
    __syncthreads();
    fetch(0);

    for (int c0 = 0; c0 < n_new; c0 += CT) {
        const int nt = min(CT, n_new - c0);
        __syncthreads();   // the previous chunk's staging is no longer read
        commit(nt);
        float table_entry = 0.f;
        if (CHANNEL) {     // the chunk's log decays per channel (zeros beyond its tokens)
#pragma unroll
            for (int i = 0; i < L_ITEMS; ++i) {
                const int idx = tid + i * THREADS, t = idx / D, e = idx - t * D;
                if (idx < CT * D) lam[t][e] = raw_l[i];
            }
            table_entry = raw_w;
        }
        if (c0 + CT < n_new) fetch(c0 + CT);   // in flight while this chunk is worked on
        __syncthreads();
        // unit vectors and the query's scale: one warp per token
        if (warp < nt) {
            const int t = warp;
            float sk = 0.f, sq = 0.f;
            for (int e = lane; e < D; e += 32) {
                sk += ks[t][e] * ks[t][e];
                sq += qs[t][e] * qs[t][e];
            }
            sk = warp_sum(sk);
            sq = warp_sum(sq);
            const float ik = 1.0f / sqrtf(sk + 1e-6f), iq = q_scale / sqrtf(sq + 1e-6f);
            for (int e = lane; e < D; e += 32) {
                ks[t][e] *= ik;
                qs[t][e] *= iq;
            }
        }
        if (CHANNEL) {               // running sums of the log decays, channel by channel
            // (warps nt .. 15 have no token to norm; with a full chunk everyone shares the work)
            for (int e = tid; e < D; e += THREADS) {
                float c = 0.f;
#pragma unroll
                for (int t = 0; t < CT; ++t) {
                    c += lam[t][e];
                    lam[t][e] = c;
                }
                last_s[e] = lam[nt - 1][e];
            }
        } else if (tid >= THREADS - CT) {   // (the last warp: it has no token to norm unless nt is 16)
            const int t = tid - (THREADS - CT);
            float c = 0.f, last = 0.f;
            for (int i = 0; i < CT; ++i) {
                if (i <= t) c += log_g[i];
                if (i < nt) last += log_g[i];
            }
            cum_s[t] = c;
            grow_s[t] = expf(c);            // e^{L_t}
            rest_s[t] = expf(last - c);     // e^{L_last - L_t}
        }
        __syncthreads();
        // the table of weights: thread -> (row, s); rows 0..15 pair keys with keys, 16..31 keys
        // with queries
        {
            const int row = tid >> 4, s = tid & 15, t = row & 15;
            const bool with_q = row >= CT;
            float dot = 0.f;
            const bool used = t < nt && s < nt && (with_q ? s <= t : s < t);
            if (CHANNEL && a.tables != nullptr) {
                dot = table_entry;       // (entry [row][s] = [tid / CT][tid % CT], as requested)
            } else if (used && CHANNEL) {
                const float* x = with_q ? &qs[t][0] : &ks[t][0];
                for (int e = 0; e < D; ++e)
                    dot = fmaf(x[e] * ks[s][e], expf(lam[t][e] - lam[s][e]), dot);
            } else if (used) {
                const float* x = with_q ? &qs[t][0] : &ks[t][0];
#pragma unroll 4
                for (int c = 0; c < QUADS; ++c) {
                    const float4 xa = *reinterpret_cast<const float4*>(x + 4 * c);
                    const float4 kb = *reinterpret_cast<const float4*>(&ks[s][4 * c]);
                    dot += xa.x * kb.x + xa.y * kb.y + xa.z * kb.z + xa.w * kb.w;
                }
                dot *= expf(cum_s[t] - cum_s[s]);
            }
            weight[row][s] = with_q ? dot : -dot;
        }
        __syncthreads();
        if (CHANNEL) {
            // what the rest of the chunk needs: e^{L_t} * k_t (in lam's place) and e^{L_t} * q_t for
            // the products with S0, and e^{L_last - L_t} * k_t for the state's update
            for (int idx = tid; idx < CT * D; idx += THREADS) {
                const int t = idx / D, e = idx - t * D;
                const float L = lam[t][e], grow = expf(L), k = ks[t][e];
                lam[t][e] = grow * k;
                qs[t][e] *= grow;
                ks[t][e] = t < nt ? k * expf(last_s[e] - L) : 0.f;
            }
            __syncthreads();
        }

        // ---- this lane's share of S0^T k_t (v[t]) and S0^T q_t (v[16 + t])
        float v[2 * CT];
#pragma unroll
        for (int t = 0; t < CT; ++t) {
            float pk = 0.f, pq = 0.f;
#pragma unroll
            for (int i = 0; i < QPL; ++i) {
                const int c = i * 32 + lane;
                if (c < QUADS) {
                    const float4 kt = *reinterpret_cast<const float4*>(
                        CHANNEL ? &lam[t][4 * c] : &ks[t][4 * c]);
                    const float4 qt = *reinterpret_cast<const float4*>(&qs[t][4 * c]);
                    pk += S[4 * i] * kt.x + S[4 * i + 1] * kt.y + S[4 * i + 2] * kt.z +
                          S[4 * i + 3] * kt.w;
                    pq += S[4 * i] * qt.x + S[4 * i + 1] * qt.y + S[4 * i + 2] * qt.z +
                          S[4 * i + 3] * qt.w;
                }
            }
            v[t] = pk;
            v[CT + t] = pq;
        }
        // ---- sum over the lanes, so that lane i ends with the total of v[i]: in the round
        // with offset o a lane keeps the half of its values whose index has bit o as its own
        // lane number has, and hands the other half to its partner
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) {
            const bool upper = (lane & o) != 0;
#pragma unroll
            for (int i = 0; i < o; ++i) {
                const float give = upper ? v[i] : v[i + o];
                const float keep = upper ? v[i + o] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
        }
        // lane t < 16: the sum that becomes u_t; lane 16 + t: the sum that becomes o_t
        const int t_mine = lane & 15;
        const float grow_mine = CHANNEL ? 1.f : grow_s[t_mine];   // (per channel: inside v[0])
        float acc = lane < CT ? vs[t_mine][warp] - grow_mine * v[0] : grow_mine * v[0];
        const float beta_mine = lane < CT ? beta_s[t_mine] : 0.f;
        float u[CT];
#pragma unroll
        for (int s = 0; s < CT; ++s) {
            u[s] = __shfl_sync(0xffffffffu, beta_mine * acc, s);   // lane s has all of its sum
            acc = fmaf(weight[lane][s], u[s], acc);                 // (weight[s][s] is 0)
        }
        if (lane >= CT && t_mine < nt && live)
            a.out[(int64_t)(t0 + c0 + t_mine) * a.H * a.V + (int64_t)head * a.V + col] = acc;
        // ---- the state after the chunk
        if (CHANNEL) {
#pragma unroll
            for (int i = 0; i < QPL; ++i)
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    const int e = (i * 32 + lane) * 4 + w;
                    if (e < D) S[4 * i + w] *= expf(last_s[e]);
                }
        } else {
            const float keep_all = grow_s[nt - 1];
#pragma unroll
            for (int i = 0; i < 4 * QPL; ++i) S[i] *= keep_all;
        }
#pragma unroll
        for (int t = 0; t < CT; ++t) {
            // (u is zero beyond the chunk's tokens; per channel the keys carry their factors)
            const float f = CHANNEL ? u[t] : rest_s[t] * u[t];
#pragma unroll
            for (int i = 0; i < QPL; ++i) {
                const int c = i * 32 + lane;
                if (c < QUADS) {
                    const float4 kt = *reinterpret_cast<const float4*>(&ks[t][4 * c]);
                    S[4 * i] = fmaf(kt.x, f, S[4 * i]);
                    S[4 * i + 1] = fmaf(kt.y, f, S[4 * i + 1]);
                    S[4 * i + 2] = fmaf(kt.z, f, S[4 * i + 2]);
                    S[4 * i + 3] = fmaf(kt.w, f, S[4 * i + 3]);
                }
            }
        }
    }
    if (live) {
#pragma unroll
        for (int i = 0; i < QPL; ++i)
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                const int e = (i * 32 + lane) * 4 + w;
                if (e < D) st[e] = S[4 * i + w];
            }
    }
}

// The tables of weights of all chunks of a step at once, for a decay per channel (the comment at
// the top): they depend on the keys, queries and decays alone, not on the state, so the chunks of
// a row need not wait for each other.  grid (chunks of the longest row, H, rows), 256 threads: a
// thread per pair of tokens that the table uses (120 pairs of keys with earlier keys, 136 of
// queries with keys up to their own).  tables: [slots][H][2 CT][CT] as DeltaArgs says; entries
// that no pair uses are zero.
constexpr int TABLE_THREADS = 256;
template <typename T>
__global__ void __launch_bounds__(TABLE_THREADS) delta_weights_kernel(const DeltaArgs a, float* tables) {
    __shared__ __align__(16) float ks[CT][LDK];
    __shared__ __align__(16) float qs[CT][LDK];
    __shared__ __align__(16) float lam[CT][LDK];
    pdl_wait();
    pdl_trigger();
    const int r = blockIdx.z, head = blockIdx.y, c0 = blockIdx.x * CT;
    const int t0 = a.row_start[r], n_new = a.row_start[r + 1] - t0;
    if (c0 >= n_new || n_new <= 1 || n_new >= a.min_chunked) return;     // (rows of one token need no table)
    const int nt = min(CT, n_new - c0);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = head / (a.H / a.G);
    const T* act = reinterpret_cast<const T*>(a.act);
    const int64_t k_col0 = (int64_t)a.G * D;
    for (int idx = tid; idx < CT * D; idx += TABLE_THREADS) {
        const int t = idx / D, e = idx - t * D;
        float k = 0.f, q = 0.f, l = 0.f;
        if (t < nt) {
            const T* row = act + (int64_t)(t0 + c0 + t) * a.ld_act + (int64_t)g * D;
            q = to_float(row[e]);
            k = to_float(row[k_col0 + e]);
            l = a.log_decay[(int64_t)(t0 + c0 + t) * a.ld_decay + (int64_t)head * D + e];
        }
        ks[t][e] = k; qs[t][e] = q; lam[t][e] = l;
    }
    __syncthreads();
    const float q_scale = rsqrtf((float)D);
    for (int t = warp; t < nt; t += TABLE_THREADS / 32) {
        float sk = 0.f, sq = 0.f;
        for (int e = lane; e < D; e += 32) {
            sk += ks[t][e] * ks[t][e];
            sq += qs[t][e] * qs[t][e];
        }
        sk = warp_sum(sk);
        sq = warp_sum(sq);
        const float ik = 1.0f / sqrtf(sk + 1e-6f), iq = q_scale / sqrtf(sq + 1e-6f);
        for (int e = lane; e < D; e += 32) {
            ks[t][e] *= ik;
            qs[t][e] *= iq;
        }
    }
    for (int e = tid; e < D; e += TABLE_THREADS) {
        float c = 0.f;
#pragma unroll
        for (int t = 0; t < CT; ++t) {
            c += lam[t][e];
            lam[t][e] = c;
        }
    }
    __syncthreads();
    float* table = tables + (((int64_t)(t0 + c0) / CT + r) * a.H + head) * 2 * CT * CT;
    // thread -> pair: the first 120 threads take (t, s < t) of keys with keys, the other 136 take
    // (t, s <= t) of queries with keys; both triangles are walked row by row
    const bool with_q = tid >= CT * (CT - 1) / 2;
    int p = with_q ? tid - CT * (CT - 1) / 2 : tid, t = 0;
    if (with_q) { while (p > t) { p -= t + 1; ++t; } }        // row t has t + 1 pairs
    else { t = 1; while (p >= t) { p -= t; ++t; } }           // row t has t pairs
    const int sidx = p;
    float dot = 0.f;
    if (t < nt) {
        const float* x = with_q ? &qs[t][0] : &ks[t][0];
#pragma unroll 4
        for (int e = 0; e < D; ++e)
            dot = fmaf(x[e] * ks[sidx][e], __expf(lam[t][e] - lam[sidx][e]), dot);
    }
    table[((with_q ? CT : 0) + t) * CT + sidx] = dot;
    // the entries that no pair uses
    for (int idx = tid; idx < 2 * CT * CT; idx += TABLE_THREADS) {
        const int row = idx / CT, s2 = idx - row * CT, t2 = row & (CT - 1);
        if (row >= CT ? s2 > t2 : s2 >= t2) table[idx] = 0.f;
    }
}

}  // namespace sllm

using namespace sllm;

SLLM_EXPORT int sllm_delta_rule_head_dim() { return D; }

// The chunk kernels' lanes share out channels in sixteenths and quads that have to fill warps evenly, and a
// chunk's keys, queries and sums of decays fit shared memory together: these key sizes.
constexpr bool CHUNKS = D == 32 || D == 64 || D == 128;

// Floats of scratch the chunk kernels take per chunk and head; 0: this key size has none.
SLLM_EXPORT int64_t sllm_delta_rule_chunk_floats(int V) {
    return CHUNKS ? chunks::scratch_floats(D, V) : 0;
}

template <typename T, bool CHANNEL>
static int launch_chunks(const DeltaArgs& a, float* scratch, int slots, int n_tokens, int n_rows, bool beside,
                         cudaStream_t stream) {
    if constexpr (CHUNKS) {
        const chunks::Scratch z = chunks::scratch_at(scratch, (int64_t)slots * a.H, D, a.V);
        chunks::PrepArgs p = {};
        p.x = a.act; p.ld = a.ld_act; p.k0 = a.G * D; p.v0 = 2 * a.G * D; p.per = a.H / a.G;
        p.log_decay = a.log_decay; p.ldl = a.ld_decay; p.ab = a.ab; p.ldab = a.ld_ab; p.b_col = a.b_col;
        p.A_log = a.A_log; p.dt_bias = a.dt_bias; p.row_start = a.row_start; p.n_rows = n_rows;
        p.min_chunked = a.min_chunked; p.H = a.H; p.V = a.V;
        p.vec4 = a.ld_act % 4 == 0 && ((uintptr_t)a.act & 15) == 0 &&
                 (!CHANNEL || (a.ld_decay % 4 == 0 && ((uintptr_t)a.log_decay & 15) == 0));
        return chunks::launch<D, T, CHANNEL>(p, z, a.state, a.row_slot, a.out, n_tokens, slots, beside, stream);
    }
    return (int)cudaErrorInvalidValue;
}

// The rows without chunks.  tables (or null): room for the weights of (tokens / CT + n_rows + 1) slots of
// H * 2 CT * CT floats; longest: the most tokens any row of the step brings.
template <typename T, bool CHANNEL>
static int launch_in_order(DeltaArgs& a, float* tables, int longest, int n_rows, bool vector, cudaStream_t stream) {
    if constexpr (CHANNEL_FITS || !CHANNEL) {
        if (CHANNEL && tables != nullptr && longest > 1) {       // all chunks' tables at once
            const dim3 tgrid((std::min(longest, a.min_chunked - 1) + CT - 1) / CT, a.H, n_rows);
            if (tgrid.x > 65535u * 32u) return (int)cudaErrorInvalidValue;
            delta_weights_kernel<T><<<tgrid, TABLE_THREADS, 0, stream>>>(a, tables);
            SLLM_LAUNCH_CHECK();
            a.tables = tables;
        }
        const dim3 grid((a.V + COLS - 1) / COLS, a.H, n_rows);
        if (vector) delta_rule_kernel<T, D % (16 / sizeof(T)) == 0, CHANNEL><<<grid, THREADS, 0, stream>>>(a);
        else delta_rule_kernel<T, false, CHANNEL><<<grid, THREADS, 0, stream>>>(a);
        SLLM_LAUNCH_CHECK();
        return 0;
    }
    return (int)cudaErrorInvalidValue;
}

template <typename T, bool CHANNEL>
static int launch_step(const DeltaArgs& a, int n_rows, bool beside, cudaStream_t stream) {
    if constexpr (CHANNEL_FITS || !CHANNEL) {
        const dim3 grid((a.V + STEP_COLS - 1) / STEP_COLS, a.H, n_rows);
        const bool words = D % 4 == 0 && ((uintptr_t)a.state & 15) == 0;
        const auto kernel = words ? delta_rule_step_kernel<T, CHANNEL, D % 4 == 0> : delta_rule_step_kernel<T, CHANNEL, false>;
        if (beside) return (int)sllm_launch_pdl(kernel, grid, dim3(32 * STEP_WARPS), 0, stream, a, true);
        kernel<<<grid, 32 * STEP_WARPS, 0, stream>>>(a, false);
        SLLM_LAUNCH_CHECK();
        return 0;
    }
    return (int)cudaErrorInvalidValue;
}

// dtype: 0 = float32, 1 = bfloat16 (of act).  n_rows rows of the packed batch (row_start has
// n_rows + 1 entries); state slots are indexed by row_slot.  max_new: the most tokens any row
// brings (1 selects the kernel for decode steps).  chunk_scratch (or null): room for chunk_slots x H x
// sllm_delta_rule_chunk_floats floats on a 16-byte boundary; rows of at least min_chunked tokens then run in
// chunks, so many at a time.  shortest: no row brings fewer tokens (rows without tokens apart);
// shortest_multi: no row of several tokens brings fewer.
SLLM_EXPORT int sllm_delta_rule(const void* act, int64_t ld_act, const float* ab, int64_t ld_ab,
                                const float* A_log, const float* dt_bias, float* state,
                                const int* row_start, const int* row_slot, float* out, int n_rows,
                                int max_new, int H, int G, int V, const float* log_decay,
                                int64_t ld_decay, int b_col, float* tables, int longest,
                                float* chunk_scratch, int chunk_slots, int n_tokens, int min_chunked,
                                int shortest, int shortest_multi, int dtype, cudaStream_t stream) {
    if (n_rows <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G != 0 || V <= 0 || n_rows > 65535 || H > 65535 ||
        ld_act < 2 * (int64_t)G * D + (int64_t)H * V || b_col < 0 || ld_ab < b_col + H ||
        (!log_decay && (ld_ab < H || !A_log || !dt_bias)) ||
        (log_decay && (ld_decay < (int64_t)H * D || !CHANNEL_FITS)) || (dtype != 0 && dtype != 1))
        return (int)cudaErrorInvalidValue;
    DeltaArgs a;
    a.log_decay = log_decay; a.ld_decay = ld_decay; a.b_col = b_col;
    a.tables = nullptr;
    a.min_chunked = chunk_scratch ? min_chunked : 0x7fffffff;
    a.act = act; a.ld_act = ld_act; a.ab = ab; a.ld_ab = ld_ab; a.A_log = A_log;
    a.dt_bias = dt_bias; a.state = state; a.row_start = row_start; a.row_slot = row_slot;
    a.out = out; a.H = H; a.G = G; a.V = V;
    const size_t esize = dtype == 0 ? 4 : 2;
    const int vec = (int)(16 / esize);
    // 16-byte pieces need every key, query and row of `act` to start on a 16-byte boundary
    const bool vector = D % vec == 0 && ld_act % vec == 0 && ((uintptr_t)act & 15) == 0 &&
                        ((int64_t)G * D) % vec == 0;
    if (chunk_scratch && (min_chunked < 2 || n_tokens < 0 || chunk_slots < 1 || chunk_slots > 65535 ||
                          ((uintptr_t)chunk_scratch & 15) || ((uintptr_t)state & 15)))
        return (int)cudaErrorInvalidValue;
    // The rows by their tokens: several, fewer than min_chunked: in order; one: the step kernel; the others in
    // chunks.  Each launch runs beside the one before it (the weights' tables apart).
    const bool in_order = max_new != 1 && (!chunk_scratch || shortest_multi < min_chunked);
    const bool single = max_new == 1 || shortest <= 1;
    int code = 0;
    if (in_order)
        code = log_decay
            ? (dtype == 0 ? launch_in_order<float, true>(a, tables, longest, n_rows, vector, stream)
                          : launch_in_order<__nv_bfloat16, true>(a, tables, longest, n_rows, vector, stream))
            : (dtype == 0 ? launch_in_order<float, false>(a, tables, longest, n_rows, vector, stream)
                          : launch_in_order<__nv_bfloat16, false>(a, tables, longest, n_rows, vector, stream));
    if (!code && single)
        code = log_decay
            ? (dtype == 0 ? launch_step<float, true>(a, n_rows, in_order, stream)
                          : launch_step<__nv_bfloat16, true>(a, n_rows, in_order, stream))
            : (dtype == 0 ? launch_step<float, false>(a, n_rows, in_order, stream)
                          : launch_step<__nv_bfloat16, false>(a, n_rows, in_order, stream));
    if (code || !chunk_scratch || max_new == 1) return code;
    const bool beside = in_order || single;
    return log_decay
        ? (dtype == 0 ? launch_chunks<float, true>(a, chunk_scratch, chunk_slots, n_tokens, n_rows, beside, stream)
                      : launch_chunks<__nv_bfloat16, true>(a, chunk_scratch, chunk_slots, n_tokens, n_rows, beside, stream))
        : (dtype == 0 ? launch_chunks<float, false>(a, chunk_scratch, chunk_slots, n_tokens, n_rows, beside, stream)
                      : launch_chunks<__nv_bfloat16, false>(a, chunk_scratch, chunk_slots, n_tokens, n_rows, beside, stream));
}
