// A matrix state per head that decays by ONE factor per token and head:
//
//     S_t = a_t S_(t-1) + b_t k_t v_t^T          (S: dk x dv; a_t, b_t scalars of the token and head)
//     o_t = S_t^T q_t  (+ skip_h v_t)
//
// which is the recurrence of a selective state space layer (a_t = e^(A dt_t), b_t = dt_t, k = B, q = C,
// v = x, skip = D) and of a matrix memory with exponential gates (a_t = e^(f_t + m_(t-1) - m_t),
// b_t = e^(i_t - m_t), m the running maximum of the log gates).  The matrix memory also keeps a
// normalizer n_t = a_t n_(t-1) + b_t k_t, stored as one more value column of the state, and divides:
// o_t <- o_t / (max(|n_t . q_t|, e^(-m_t)) + 1e-6).
//
// The state lives in 32-bit floats per sequence slot, [slot][head][dv (+1)][dk]; log a_t and b_t come as
// 32-bit numbers per token and head; q, k, v are 32-bit rows (any row stride, any column offset); several
// heads may share one q and k (a group).  Everything is computed in 32-bit.
//
// Work of the token-by-token kernel: a block is (16 value columns, head, sequence) and walks the
// sequence's tokens in order; a value column is owned by 8 lanes, lane p holding rows p, p+8, ... of that
// column in registers.  With a normalizer every block carries that column too (as a 17th group of lanes),
// so that it can divide without waiting for another block; the block of the first tile stores it.  The
// order of every sum depends on nothing but dk, so a prompt gives the same numbers however it is cut.
#include "chunked_state.cuh"

#define SS_COLS 16
#define SS_PART 8
#define SS_CHUNK 8

template <int R>
__global__ void __launch_bounds__(SS_COLS * SS_PART + 32)
scalar_scan_kernel(const float* __restrict__ q, int ldq, const float* __restrict__ k, int ldk,
                   const float* __restrict__ v, int ldv, const float* __restrict__ log_a, int ld_a,
                   const float* __restrict__ b_in, int ld_b, const float* __restrict__ skip,
                   const float* __restrict__ m_tok, float q_scale, float* __restrict__ state,
                   const int* __restrict__ slots, const int* __restrict__ cu, float* __restrict__ o, int n_heads,
                   int heads_per_group, int dk, int dv, int normalizer) {
    mv_pdl_begin();
    extern __shared__ float smem[];
    float* qs = smem;                           // [SS_CHUNK][dk]
    float* ks = qs + SS_CHUNK * dk;             // [SS_CHUNK][dk], already times b_t
    float* vs = ks + SS_CHUNK * dk;             // [SS_CHUNK][SS_COLS]
    float* as = vs + SS_CHUNK * SS_COLS;        // [SS_CHUNK] decay factors
    float* ms = as + SS_CHUNK;                  // [SS_CHUNK] e^(-m_t)
    float* acc_s = ms + SS_CHUNK;               // [SS_CHUNK][SS_COLS + 1]
    const int tile = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
    const int tid = threadIdx.x, p = tid & (SS_PART - 1), jl = tid >> 3;
    const int n_threads = blockDim.x;
    const bool is_n = jl == SS_COLS;                          // the normalizer's lanes
    const int cols = dv + (normalizer ? 1 : 0);
    const int j = jl >= SS_COLS ? dv : tile * SS_COLS + jl;
    const bool live = is_n ? normalizer != 0 : (jl < SS_COLS && j < dv);    // a whole last warp: its other lanes idle
    const int row0 = cu[b], len = cu[b + 1] - row0;
    if (len <= 0) return;
    const int slot = mv_read_slot(slots[b]);
    const size_t qk_off = (size_t)(h / heads_per_group) * dk;
    float* srow = state + (((size_t)slot * n_heads + h) * cols + (live ? j : 0)) * dk;
    float S[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = p + SS_PART * r;
        S[r] = (live && i < dk) ? srow[i] : 0.f;
    }
    const float sk = skip ? skip[h] : 0.f;
    for (int c0 = 0; c0 < len; c0 += SS_CHUNK) {
        const int nt = min(SS_CHUNK, len - c0);
        __syncthreads();
        if (tid < nt) {
            const size_t row = (size_t)(row0 + c0 + tid);
            as[tid] = expf(log_a[row * ld_a + h]);
            ms[tid] = m_tok ? expf(-m_tok[row * n_heads + h]) : 0.f;
        }
        for (int idx = tid; idx < nt * dk; idx += n_threads) {
            const int t = idx / dk, i = idx - t * dk;
            const size_t row = (size_t)(row0 + c0 + t);
            qs[idx] = q[row * ldq + qk_off + i] * q_scale;
            ks[idx] = k[row * ldk + qk_off + i] * b_in[row * ld_b + h];
        }
        for (int idx = tid; idx < nt * SS_COLS; idx += n_threads) {
            const int t = idx / SS_COLS, c = idx - t * SS_COLS, col = tile * SS_COLS + c;
            vs[idx] = col < dv ? v[(size_t)(row0 + c0 + t) * ldv + (size_t)h * dv + col] : 0.f;
        }
        __syncthreads();
        for (int t = 0; t < nt; ++t) {
            const float vj = is_n ? 1.f : vs[t * SS_COLS + (jl < SS_COLS ? jl : 0)];
            const float a = as[t];
            const float* qt = qs + t * dk;
            const float* kt = ks + t * dk;
            float acc = 0.f;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int i = p + SS_PART * r;
                if (i < dk) {
                    S[r] = fmaf(a, S[r], kt[i] * vj);
                    acc = fmaf(S[r], qt[i], acc);
                }
            }
            acc += __shfl_xor_sync(0xffffffffu, acc, 1);
            acc += __shfl_xor_sync(0xffffffffu, acc, 2);
            acc += __shfl_xor_sync(0xffffffffu, acc, 4);
            if (p == 0 && jl <= SS_COLS) acc_s[t * (SS_COLS + 1) + jl] = acc + (is_n ? 0.f : sk * vj);
        }
        __syncthreads();
        for (int idx = tid; idx < nt * SS_COLS; idx += n_threads) {
            const int t = idx / SS_COLS, c = idx - t * SS_COLS, col = tile * SS_COLS + c;
            if (col >= dv) continue;
            float val = acc_s[t * (SS_COLS + 1) + c];
            if (normalizer) val = val / (fmaxf(fabsf(acc_s[t * (SS_COLS + 1) + SS_COLS]), ms[t]) + 1e-6f);
            o[(size_t)(row0 + c0 + t) * n_heads * dv + (size_t)h * dv + col] = val;
        }
    }
    if (live && (!is_n || tile == 0) && mv_slot_ok(slots[b])) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int i = p + SS_PART * r;
            if (i < dk) srow[i] = S[r];
        }
    }
}

MV_GUARD_SETTER(scalar_scan)

// q, k [N, >= (n_heads / heads_per_group) * dk], v [N, >= n_heads * dv] with row strides (elements);
// log_a, b [N, >= n_heads] with row strides; skip [n_heads] or null; m_tok [N, n_heads] dense or null
// (needed with a normalizer); state [slots][n_heads][dv + normalizer][dk]; o [N, n_heads * dv] dense.
MV_API int mv_scalar_scan(const float* q, int ldq, const float* k, int ldk, const float* v, int ldv,
                          const float* log_a, int ld_a, const float* b, int ld_b, const float* skip,
                          const float* m_tok, float q_scale, float* state, const int* slots, const int* cu, float* o,
                          int n_seqs, int n_heads, int heads_per_group, int dk, int dv, int normalizer,
                          cudaStream_t stream) {
    if (n_seqs <= 0) return 0;
    if (dk < 1 || dk > 256 || dv < 1 || heads_per_group < 1 || n_heads % heads_per_group || (normalizer && !m_tok))
        return (int)cudaErrorInvalidValue;
    const dim3 grid((dv + SS_COLS - 1) / SS_COLS, n_heads, n_seqs);
    const int threads = SS_COLS * SS_PART + (normalizer ? 32 : 0);
    const size_t smem = sizeof(float) * ((size_t)SS_CHUNK * (2 * dk + SS_COLS + 2 + SS_COLS + 1));
#define SS_LAUNCH(R)                                                                                              \
    mv_launch(scalar_scan_kernel<R>, grid, threads, smem, stream, q, ldq, k, ldk, v, ldv, log_a, ld_a, b, ld_b,  \
              skip, m_tok, q_scale, state, slots, cu, o, n_heads, heads_per_group, dk, dv, normalizer)
    if (dk <= 64) SS_LAUNCH(8);
    else if (dk <= 128) SS_LAUNCH(16);
    else SS_LAUNCH(32);
#undef SS_LAUNCH
    return mv_launch_status();
}

// ------------------------------------------------------------------------------------------------
// The log gates of a matrix memory and their running maximum, per sequence and head:
//     i_t = cap tanh((zi_t + bi) / cap),  f_t = log sigmoid(cap tanh((zf_t + bf) / cap)),
//     m_t = max(f_t + m_(t-1), i_t)   (m before a sequence's first token is 0: a zeroed state),
//     log a_t = f_t + m_(t-1) - m_t,  b_t = e^(i_t - m_t).
// The step m -> max(m + f, i) composes: first (f1, i1), then (f2, i2) is m -> max(m + f1 + f2, max(i1 + f2, i2)).
// A warp is one (sequence, head): it takes 32 tokens at a time, a lane a token, scans the pairs with that rule
// (five shuffles) and hands the last maximum on to the next 32.  A step of one token a sequence is the rule itself.
// m is kept per slot and head.
__device__ __forceinline__ float ss_log_sigmoid(float z) { return fminf(z, 0.f) - log1pf(expf(-fabsf(z))); }

__global__ void __launch_bounds__(128)
memory_gates_kernel(const float* __restrict__ zi, int ld_i, const float* __restrict__ zf, int ld_f,
                    const float* __restrict__ bi, const float* __restrict__ bf, float cap, float* __restrict__ m_state,
                    const int* __restrict__ slots, const int* __restrict__ cu, float* __restrict__ log_a,
                    float* __restrict__ b_out, float* __restrict__ m_tok, int n_seqs, int n_heads) {
    mv_pdl_begin();
    const int warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (warp >= n_seqs * n_heads) return;
    const int b = warp / n_heads, h = warp - b * n_heads;
    const int row0 = cu[b], len = cu[b + 1] - row0;
    if (len <= 0) return;
    const float inv_cap = 1.0f / cap;
    const int slot = mv_read_slot(slots[b]);
    float m = m_state[(size_t)slot * n_heads + h];
    const float bih = bi[h], bfh = bf[h];
    for (int t0 = 0; t0 < len; t0 += 32) {
        const int t = t0 + lane;
        const bool in = t < len;
        const size_t row = (size_t)(row0 + (in ? t : 0));
        const float il = in ? cap * tanhf((zi[row * ld_i + h] + bih) * inv_cap) : -INFINITY;
        const float fl = in ? ss_log_sigmoid(cap * tanhf((zf[row * ld_f + h] + bfh) * inv_cap)) : 0.f;
        float A = fl, B = il;                         // the tokens up to this lane's as one step m -> max(m + A, B)
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const float a_up = __shfl_up_sync(0xffffffffu, A, d), b_up = __shfl_up_sync(0xffffffffu, B, d);
            if (lane >= d) {
                B = fmaxf(b_up + A, B);
                A = a_up + A;
            }
        }
        const float m_t = fmaxf(m + A, B);
        float m_before = __shfl_up_sync(0xffffffffu, m_t, 1);
        if (lane == 0) m_before = m;
        if (in) {
            const size_t at = row * n_heads + h;
            log_a[at] = fl + m_before - m_t;
            b_out[at] = expf(il - m_t);
            m_tok[at] = m_t;
        }
        m = __shfl_sync(0xffffffffu, m_t, min(31, len - t0 - 1));
    }
    if (lane == 0 && mv_slot_ok(slots[b])) m_state[(size_t)slot * n_heads + h] = m;
}

// The same for sequences of many tokens, a block a sequence and head: a warp works out the gates of 32 tokens and adds them up as one step, the
// steps of the warps before it carry the maximum to it, and no warp waits for another's gates.  One warp for a sequence is one chain of a thousand
// cycles every 32 tokens (two sequences of 611 and 1,437 tokens, 8 heads: 36 -> 8.5 us; one of 65 tokens 2.3 -> 2.1).  The maxima are the same numbers: a warp's step is added up
// as above, and the carried maximum passes the same steps in the same order.
#define MG_WARPS 16
__global__ void __launch_bounds__(32 * MG_WARPS)
memory_gates_block_kernel(const float* __restrict__ zi, int ld_i, const float* __restrict__ zf, int ld_f,
                          const float* __restrict__ bi, const float* __restrict__ bf, float cap, float* __restrict__ m_state,
                          const int* __restrict__ slots, const int* __restrict__ cu, float* __restrict__ log_a,
                          float* __restrict__ b_out, float* __restrict__ m_tok, int n_heads) {
    mv_pdl_begin();
    __shared__ float step_a[2][MG_WARPS], step_b[2][MG_WARPS];
    const int b = blockIdx.x / n_heads, h = blockIdx.x - b * n_heads;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row0 = cu[b], len = cu[b + 1] - row0;
    if (len <= 0) return;
    const float inv_cap = 1.0f / cap;
    const int slot = mv_read_slot(slots[b]);
    float m = m_state[(size_t)slot * n_heads + h];           // the maximum before the block's tokens
    const float bih = bi[h], bfh = bf[h];
    int buf = 0;
    for (int first = 0; first < len; first += 32 * MG_WARPS, buf ^= 1) {
        const int t = first + 32 * warp + lane;
        const bool in = t < len;
        const size_t row = (size_t)(row0 + (in ? t : 0));
        const float il = in ? cap * tanhf((zi[row * ld_i + h] + bih) * inv_cap) : -INFINITY;
        const float fl = in ? ss_log_sigmoid(cap * tanhf((zf[row * ld_f + h] + bfh) * inv_cap)) : 0.f;
        float A = fl, B = il;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const float a_up = __shfl_up_sync(0xffffffffu, A, d), b_up = __shfl_up_sync(0xffffffffu, B, d);
            if (lane >= d) {
                B = fmaxf(b_up + A, B);
                A = a_up + A;
            }
        }
        if (lane == min(31, len - 1 - first - 32 * warp)) { step_a[buf][warp] = A; step_b[buf][warp] = B; }
        __syncthreads();                                     // the buffers alternate: the next round's writes meet no reader of this one's
        const int steps = min(MG_WARPS, (len - first + 31) / 32);
        float at_warp = m;
        for (int i = 0; i < steps; ++i) {
            if (i == warp) at_warp = m;
            m = fmaxf(m + step_a[buf][i], step_b[buf][i]);
        }
        const float m_t = fmaxf(at_warp + A, B);
        float m_before = __shfl_up_sync(0xffffffffu, m_t, 1);
        if (lane == 0) m_before = at_warp;
        if (in) {
            const size_t at = row * n_heads + h;
            log_a[at] = fl + m_before - m_t;
            b_out[at] = expf(il - m_t);
            m_tok[at] = m_t;
        }
    }
    if (threadIdx.x == 0 && mv_slot_ok(slots[b])) m_state[(size_t)slot * n_heads + h] = m;
}

// zi, zf: the gates' projections [N, >= n_heads] with row strides; bi, bf [n_heads]; m_state [slots][n_heads];
// log_a, b_out, m_tok [N, n_heads] dense.
MV_API int mv_memory_gates(const float* zi, int ld_i, const float* zf, int ld_f, const float* bi, const float* bf,
                           float cap, float* m_state, const int* slots, const int* cu, float* log_a, float* b_out,
                           float* m_tok, int N, int n_seqs, int n_heads, cudaStream_t stream) {
    if (n_seqs <= 0) return 0;
    if (!(cap > 0.f) || n_heads < 1) return (int)cudaErrorInvalidValue;
    if (N > 64 * n_seqs) {                                   // from three chunks a sequence on the chain is the longer one
        mv_launch(memory_gates_block_kernel, n_seqs * n_heads, 32 * MG_WARPS, 0, stream, zi, ld_i, zf, ld_f, bi, bf, cap, m_state, slots, cu,
                  log_a, b_out, m_tok, n_heads);
        return mv_launch_status();
    }
    const int warps = n_seqs * n_heads;
    mv_launch(memory_gates_kernel, (warps + 3) / 4, 128, 0, stream, zi, ld_i, zf, ld_f, bi, bf, cap, m_state, slots, cu, log_a,
              b_out, m_tok, n_seqs, n_heads);
    return mv_launch_status();
}

// ------------------------------------------------------------------------------------------------
// The same recurrence for steps that bring many tokens a sequence, in chunks of SC_CHUNK tokens.  With c_t the
// sum of log a over the chunk's tokens up to t (all of it <= 0) and S0 the state before the chunk,
//
//     o_t   = e^(c_t) q_t^T S0 + sum_{s <= t} (q_t . k_s) e^(c_t - c_s) b_s v_s  (+ skip v_t),
//     S_end = e^(c_last) S0 + sum_s e^(c_last - c_s) b_s k_s v_s^T.
//
// Every exponent is a difference of cumulative logarithms taken the right way round, so every factor lies in
// (0, 1] (times b): nothing overflows however small a decay is.  Because the decay is one number a head, q and k
// need no decayed copies: the products q_t . k_s are worked out once per GROUP of heads that share q and k
// (ss_products_kernel), and each head puts its own factors on them (ss_factors_kernel).  ss_walk_kernel walks a sequence's chunks
// with nothing but the state, a tile of which lies in a block's registers, and leaves the state before every chunk;
// ss_output_kernel then has a block for every chunk, head and 64 value columns.  With a normalizer the state's last column is fed
// ones instead of values and comes out as n . q, by which the outputs are divided.  All of it is float32 on the CUDA cores.
//
// Every sum is added up in a fixed order: a state's element token by token; an output as the sums over 4 key channels (8 from
// dk 129 on), these one after the other, times the decay, then the chunk's tokens in order.  A layer behind a matrix memory
// divides by sums that may nearly cancel and routers compare what comes out, so another order moves whole outputs by percents.
// Two sequences of 611 and 1,437 tokens, 64 heads of 128 x 64 in one group: 125 us the walk, 105 the outputs, 10 the products and
// factors, where a kernel that walked 16 columns and worked the outputs out on the way took 430 (half of it in adding up 32
// half-warps' shares from shared memory).  The walk and the outputs are bound by the multiply-adds and the reads that feed them.
//
// Chunks are numbered floor(cu[b] / SC_CHUNK) + b + c for chunk c of the step's sequence b: distinct numbers
// below N / SC_CHUNK + n_seqs + 1 that need nothing from the host.
#define SC_CHUNK 32
#define SC_WALK_THREADS 256

struct ScArgs {
    const float *q, *k, *v;             // rows of the step's tokens; head h reads the columns (h / heads_per_group) dk, the same, h dv
    int ldq, ldk, ldv;
    const float *log_a, *b, *skip, *m_tok;
    int ld_a, ld_b;
    float q_scale;
    float *state, *before;              // [slot][head][cols][dk]; [chunk - w0][head][cols][lds]: the state before every chunk
    float *G;                           // q_t . k_s [chunk][group][SC_CHUNK][SC_CHUNK]
    float *run, *e1, *e2, *el;          // [chunk][head][SC_CHUNK]: running log decay, e^(c_t) q_scale, e^(c_last - c_t) b_t; [chunk][head]: e^(c_last)
    const int *slots, *cu;
    float* o;
    int n_heads, heads_per_group, dk, dv, lds, wide, normalizer;
    int w0, w1, room;                   // as in CsArgs
};

namespace {

// a warp a chunk and head
__global__ void __launch_bounds__(128)
ss_factors_kernel(const ScArgs a) {
    mv_pdl_begin();
    const int c = blockIdx.x, h = blockIdx.y * 4 + (threadIdx.x >> 5), b = blockIdx.z, t = threadIdx.x & 31;
    const int row0 = a.cu[b], len = a.cu[b + 1] - row0;
    if (c * SC_CHUNK >= len || h >= a.n_heads) return;
    const int nt = min(SC_CHUNK, len - c * SC_CHUNK);
    const size_t row = (size_t)row0 + c * SC_CHUNK + t, at = (size_t)(row0 / SC_CHUNK + b + c) * a.n_heads + h;
    float run = t < nt ? a.log_a[row * a.ld_a + h] : 0.f;
    const float bt = t < nt ? a.b[row * a.ld_b + h] : 0.f;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, run, d);
        if (t >= d) run += up;
    }
    const float last = __shfl_sync(0xffffffffu, run, nt - 1);
    a.run[at * SC_CHUNK + t] = run;
    a.e1[at * SC_CHUNK + t] = expf(run) * a.q_scale;
    a.e2[at * SC_CHUNK + t] = t < nt ? expf(last - run) * bt : 0.f;
    if (t == 0) a.el[at] = expf(last);
}

constexpr int SP_LD = 36;

// 64 threads, 4 x 4 products each; channels in order
__global__ void __launch_bounds__(64)
ss_products_kernel(const ScArgs a) {
    __shared__ __align__(16) float qs[2][SC_CHUNK * SP_LD], ks[2][SC_CHUNK * SP_LD];
    mv_pdl_begin();
    const int c = blockIdx.x, g = blockIdx.y, b = blockIdx.z, ts = threadIdx.x & 7, tt = threadIdx.x >> 3;
    const int row0 = a.cu[b], len = a.cu[b + 1] - row0;
    if (c * SC_CHUNK >= len) return;
    const int nt = min(SC_CHUNK, len - c * SC_CHUNK), slices = (a.dk + 31) / 32;
    const size_t first = (size_t)row0 + c * SC_CHUNK;
    auto load = [&](int s) {
        cs_load<SC_CHUNK, 32, SP_LD, false, 64>(qs[s & 1], a.q + first * a.ldq + (size_t)g * a.dk + s * 32, a.ldq, nt, a.dk - s * 32, a.wide);
        cs_load<SC_CHUNK, 32, SP_LD, false, 64>(ks[s & 1], a.k + first * a.ldk + (size_t)g * a.dk + s * 32, a.ldk, nt, a.dk - s * 32, a.wide);
        cs_commit();
    };
    float acc[4][4];
#pragma unroll
    for (int y = 0; y < 4; ++y)
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[y][x] = 0.f;
    load(0);
    for (int s = 0; s < slices; ++s) {
        if (s + 1 < slices) { load(s + 1); cs_wait<1>(); }
        else cs_wait<0>();
        __syncthreads();
#pragma unroll 4
        for (int kk = 0; kk < 32; kk += 4) {
            float4 w[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) w[x] = *reinterpret_cast<const float4*>(ks[s & 1] + (ts + 8 * x) * SP_LD + kk);
#pragma unroll
            for (int y = 0; y < 4; ++y) {
                const float4 u = *reinterpret_cast<const float4*>(qs[s & 1] + (tt + 8 * y) * SP_LD + kk);
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    acc[y][x] = fmaf(u.x, w[x].x, acc[y][x]); acc[y][x] = fmaf(u.y, w[x].y, acc[y][x]);
                    acc[y][x] = fmaf(u.z, w[x].z, acc[y][x]); acc[y][x] = fmaf(u.w, w[x].w, acc[y][x]);
                }
            }
        }
        __syncthreads();
    }
    float* to = a.G + ((size_t)(row0 / SC_CHUNK + b + c) * (a.n_heads / a.heads_per_group) + g) * SC_CHUNK * SC_CHUNK;
#pragma unroll
    for (int y = 0; y < 4; ++y)
#pragma unroll
        for (int x = 0; x < 4; ++x) to[(tt + 8 * y) * SC_CHUNK + ts + 8 * x] = acc[y][x];
}

// A block has 64 value columns x 64 key channels of a head's state, a thread 4 x 4; two chunks' rows are on their way
// while one is worked on, whose values are first multiplied by their factors in place.
constexpr int SW_STAGES = 3;
constexpr size_t SW_SMEM = sizeof(float) * SW_STAGES * (2 * SC_CHUNK * 64 + SC_CHUNK);

__global__ void __launch_bounds__(SC_WALK_THREADS)
ss_walk_kernel(const ScArgs a) {
    extern __shared__ __align__(16) float sw_smem[];
    float* ks = sw_smem;                                // [STAGES][SC_CHUNK][64]
    float* vs = ks + SW_STAGES * SC_CHUNK * 64;         // [STAGES][SC_CHUNK][64]
    float* ws = vs + SW_STAGES * SC_CHUNK * 64;         // [STAGES][SC_CHUNK]
    mv_pdl_begin();
    const int tiles_i = (a.dk + 63) / 64, i0 = (blockIdx.x % tiles_i) * 64, j0 = (blockIdx.x / tiles_i) * 64;
    const int h = blockIdx.y, b = blockIdx.z, tid = threadIdx.x, ti = tid & 15, tj = tid >> 4;
    const int row0 = a.cu[b], len = a.cu[b + 1] - row0;
    const int n_chunks = (len + SC_CHUNK - 1) / SC_CHUNK, chunk0 = row0 / SC_CHUNK + b;
    const int2 win = cs_window(chunk0, n_chunks, a.w0, a.w1);       // (as in chunked_state.cuh)
    if (win.x >= win.y) return;
    const int cols = a.dv + a.normalizer, slot = mv_read_slot(a.slots[b]);
    const bool with_n = a.normalizer && j0 == 0;
    const int i = i0 + ti * 4, j = j0 + tj * 4;
    float* st = a.state + ((size_t)slot * a.n_heads + h) * cols * a.dk;
    const bool vec = a.dk % 4 == 0;                     // the state's rows start on 16 bytes
    const float* carried = a.before + ((size_t)cs_carry(a.w0, a.room) * a.n_heads + h) * cols * a.lds;
    float S[4][4], n[4];
    auto read4 = [&](const float* p, float* out) {
        float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
        if (vec && i < a.dk) r = *reinterpret_cast<const float4*>(p + i);
        else {
            if (i < a.dk) r.x = p[i];
            if (i + 1 < a.dk) r.y = p[i + 1];
            if (i + 2 < a.dk) r.z = p[i + 2];
            if (i + 3 < a.dk) r.w = p[i + 3];
        }
        out[0] = r.x; out[1] = r.y; out[2] = r.z; out[3] = r.w;
    };
#pragma unroll
    for (int y = 0; y < 4; ++y) {
        if (j + y < a.dv) read4(win.x ? carried + (size_t)(j + y) * a.lds : st + (size_t)(j + y) * a.dk, S[y]);
        else S[y][0] = S[y][1] = S[y][2] = S[y][3] = 0.f;
    }
    n[0] = n[1] = n[2] = n[3] = 0.f;
    if (with_n) read4(win.x ? carried + (size_t)a.dv * a.lds : st + (size_t)a.dv * a.dk, n);
    const float* kp = a.k + (size_t)row0 * a.ldk + (size_t)(h / a.heads_per_group) * a.dk + i0;
    const float* vp = a.v + (size_t)row0 * a.ldv + (size_t)h * a.dv + j0;
    auto load = [&](int c) {
        if (c < win.y) {
            const int st_ = c % SW_STAGES;
            const size_t t = (size_t)c * SC_CHUNK;
            cs_load<SC_CHUNK, 64, 64, false, SC_WALK_THREADS>(ks + st_ * SC_CHUNK * 64, kp + t * a.ldk, a.ldk, len - (int)t, a.dk - i0, a.wide);
            cs_load<SC_CHUNK, 64, 64, false, SC_WALK_THREADS>(vs + st_ * SC_CHUNK * 64, vp + t * a.ldv, a.ldv, len - (int)t, a.dv - j0, a.wide);
            if (tid < SC_CHUNK / 4)
                cs_copy(ws + st_ * SC_CHUNK + tid * 4, a.e2 + ((size_t)(chunk0 + c) * a.n_heads + h) * SC_CHUNK + tid * 4, true, true);
        }
        cs_commit();
    };
#pragma unroll
    for (int c = 0; c < SW_STAGES - 1; ++c) load(win.x + c);
    float d_next = a.el[(size_t)(chunk0 + win.x) * a.n_heads + h];        // the chunk's decay, requested a chunk ahead
    auto leave = [&](int place) {
        float* to = a.before + ((size_t)place * a.n_heads + h) * cols * a.lds;
        if (i < a.lds) {
#pragma unroll
            for (int y = 0; y < 4; ++y)
                if (j + y < a.dv)
                    *reinterpret_cast<float4*>(to + (size_t)(j + y) * a.lds + i) = make_float4(S[y][0], S[y][1], S[y][2], S[y][3]);
            if (with_n && tj == 0) *reinterpret_cast<float4*>(to + (size_t)a.dv * a.lds + i) = make_float4(n[0], n[1], n[2], n[3]);
        }
    };
    for (int c = win.x; c < win.y; ++c) {
        leave(chunk0 + c - a.w0);                       // the state as it is before this chunk
#pragma unroll
        for (int x = 0; x < 4; ++x) {
#pragma unroll
            for (int y = 0; y < 4; ++y) S[y][x] *= d_next;
            n[x] *= d_next;
        }
        if (c + 1 < win.y) d_next = a.el[(size_t)(chunk0 + c + 1) * a.n_heads + h];
        cs_wait<SW_STAGES - 2>();
        __syncthreads();                                // this chunk's rows are there, the ones before are done with
        load(c + SW_STAGES - 1);
        const float* kt = ks + c % SW_STAGES * SC_CHUNK * 64 + ti * 4;
        float* vt = vs + c % SW_STAGES * SC_CHUNK * 64;
        const float* wt = ws + c % SW_STAGES * SC_CHUNK;
#pragma unroll
        for (int e = 0; e < SC_CHUNK * 16 / SC_WALK_THREADS; ++e) {
            const int at = tid + e * SC_WALK_THREADS;
            const float w = wt[at >> 4];
            float4 x = reinterpret_cast<float4*>(vt)[at];
            x.x *= w; x.y *= w; x.z *= w; x.w *= w;
            reinterpret_cast<float4*>(vt)[at] = x;
        }
        __syncthreads();
#pragma unroll 2
        for (int s0 = 0; s0 < SC_CHUNK; s0 += 4) {
            float4 k[4], v[4];
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                k[s] = *reinterpret_cast<const float4*>(kt + (s0 + s) * 64);
                v[s] = *reinterpret_cast<const float4*>(vt + (s0 + s) * 64 + tj * 4);
            }
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const float vy[4] = {v[s].x, v[s].y, v[s].z, v[s].w};
#pragma unroll
                for (int y = 0; y < 4; ++y) {
                    S[y][0] = fmaf(k[s].x, vy[y], S[y][0]); S[y][1] = fmaf(k[s].y, vy[y], S[y][1]);
                    S[y][2] = fmaf(k[s].z, vy[y], S[y][2]); S[y][3] = fmaf(k[s].w, vy[y], S[y][3]);
                }
            }
            if (with_n) {
                const float4 w = *reinterpret_cast<const float4*>(wt + s0);
                const float wy[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    n[0] = fmaf(k[s].x, wy[s], n[0]); n[1] = fmaf(k[s].y, wy[s], n[1]);
                    n[2] = fmaf(k[s].z, wy[s], n[2]); n[3] = fmaf(k[s].w, wy[s], n[3]);
                }
            }
        }
    }
    if (win.y < n_chunks) leave(cs_carry(a.w1, a.room));
    else if (mv_slot_ok(a.slots[b])) {
        auto write4 = [&](float* p, const float* from) {
            if (vec && i < a.dk) *reinterpret_cast<float4*>(p + i) = make_float4(from[0], from[1], from[2], from[3]);
            else
#pragma unroll
                for (int x = 0; x < 4; ++x)
                    if (i + x < a.dk) p[i + x] = from[x];
        };
#pragma unroll
        for (int y = 0; y < 4; ++y)
            if (j + y < a.dv) write4(st + (size_t)(j + y) * a.dk, S[y]);
        if (with_n && tj == 0) write4(st + (size_t)a.dv * a.dk, n);
    }
}

// A block has one chunk's outputs in 64 value columns of one head, a thread 4 x 4 of them.  q and the state come in slices of
// 32 key channels, the next slice on its way (the state's row of the normalizer behind its 64 rows).  RH: key channels a group.
constexpr int SO_LD = 36, SO_THREADS = 128, SO_STAGE = (SC_CHUNK + 64 + 1) * SO_LD;
constexpr size_t SO_SMEM = sizeof(float) * (2 * SO_STAGE + SC_CHUNK * SO_LD + SC_CHUNK * 64 + 2 * SC_CHUNK);

template <int RH>
__global__ void __launch_bounds__(SO_THREADS)
ss_output_kernel(const ScArgs a) {
    extern __shared__ __align__(16) float so_smem[];    // 2 x [q: 32 rows | state: 64 rows | n: 1 row][SO_LD]
    float* ps = so_smem + 2 * SO_STAGE;                 // [32][SO_LD]
    float* vs = ps + SC_CHUNK * SO_LD;                  // [32][64]
    float* e1 = vs + SC_CHUNK * 64;                     // [32]
    float* dn = e1 + SC_CHUNK;                          // [32] denominators
    mv_pdl_begin();
    const int tiles_j = (a.dv + 63) / 64, j0 = (blockIdx.x % tiles_j) * 64;
    const int h = blockIdx.y, b = blockIdx.z, tid = threadIdx.x, tj = tid & 15, tt = tid >> 4;
    const int row0 = a.cu[b], len = a.cu[b + 1] - row0, chunk0 = row0 / SC_CHUNK + b;
    const int2 win = cs_window(chunk0, (len + SC_CHUNK - 1) / SC_CHUNK, a.w0, a.w1);
    const int c = win.x + blockIdx.x / tiles_j, chunk = chunk0 + c;
    if (c >= win.y) return;
    const int nt = min(SC_CHUNK, len - c * SC_CHUNK);
    const size_t first = (size_t)row0 + c * SC_CHUNK, at = (size_t)chunk * a.n_heads + h;
    const int cols = a.dv + a.normalizer, g = h / a.heads_per_group, n_groups = a.n_heads / a.heads_per_group;
    const float* S0 = a.before + ((size_t)(chunk - a.w0) * a.n_heads + h) * cols * a.lds;
    const float* qp = a.q + first * a.ldq + (size_t)g * a.dk;
    const int slices = (a.dk + 31) / 32;
    auto load = [&](int s) {
        float* to = so_smem + (s & 1) * SO_STAGE;
        cs_load<SC_CHUNK, 32, SO_LD, false, SO_THREADS>(to, qp + s * 32, a.ldq, nt, a.dk - s * 32, a.wide);
        cs_load<64, 32, SO_LD, true, SO_THREADS>(to + SC_CHUNK * SO_LD, S0 + (size_t)j0 * a.lds + s * 32, a.lds, a.dv - j0, a.lds - s * 32, 1);
        if (a.normalizer && tid < 8) {
            const bool in = s * 32 + tid * 4 < a.lds;
            cs_copy(to + (SC_CHUNK + 64) * SO_LD + tid * 4, S0 + (size_t)a.dv * a.lds + (in ? s * 32 + tid * 4 : 0), in, true);
        }
        cs_commit();
    };
    load(0);
    cs_load<SC_CHUNK, 64, 64, false, SO_THREADS>(vs, a.v + first * a.ldv + (size_t)h * a.dv + j0, a.ldv, nt, a.dv - j0, a.wide);
    cs_commit();
    {
        // this head's factors on the group's products
        const float* Gc = a.G + ((size_t)chunk * n_groups + g) * SC_CHUNK * SC_CHUNK;
        const float *run = a.run + at * SC_CHUNK, *bp = a.b + first * a.ld_b + h;
        if (tid < SC_CHUNK) e1[tid] = a.e1[at * SC_CHUNK + tid];
        const int s = tid & 31;
        const float cs = run[s], bs = s < nt ? bp[(size_t)s * a.ld_b] : 0.f;
#pragma unroll
        for (int e = 0; e < SC_CHUNK * SC_CHUNK / SO_THREADS; ++e) {
            const int t = (tid >> 5) + e * (SO_THREADS / 32);
            ps[t * SO_LD + s] = (s <= t && t < nt) ? Gc[t * SC_CHUNK + s] * expf(run[t] - cs) * bs * a.q_scale : 0.f;
        }
    }
    float acc[4][4];
#pragma unroll
    for (int y = 0; y < 4; ++y)
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[y][x] = 0.f;
    float dot = 0.f;                                    // with a normalizer, warp 0: token tid's q . n
    for (int s = 0; s < slices; ++s) {
        if (s + 1 < slices) { load(s + 1); cs_wait<1>(); }
        else cs_wait<0>();
        __syncthreads();
        const float* stage = so_smem + (s & 1) * SO_STAGE;
        const float *q = stage + tt * SO_LD, *st = stage + (SC_CHUNK + tj) * SO_LD;
#pragma unroll 2
        for (int kk = 0; kk < 32; kk += RH) {
            float part[4][4];
#pragma unroll
            for (int f = 0; f < RH; f += 4) {
                float4 w[4];
#pragma unroll
                for (int x = 0; x < 4; ++x) w[x] = *reinterpret_cast<const float4*>(st + x * 16 * SO_LD + kk + f);
#pragma unroll
                for (int y = 0; y < 4; ++y) {
                    const float4 u = *reinterpret_cast<const float4*>(q + y * 8 * SO_LD + kk + f);
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        float p = f == 0 ? u.x * w[x].x : fmaf(u.x, w[x].x, part[y][x]);
                        p = fmaf(u.y, w[x].y, p); p = fmaf(u.z, w[x].z, p);
                        part[y][x] = fmaf(u.w, w[x].w, p);
                    }
                }
            }
#pragma unroll
            for (int y = 0; y < 4; ++y)
#pragma unroll
                for (int x = 0; x < 4; ++x) acc[y][x] += part[y][x];
        }
        if (a.normalizer && tid < 32) {
            const float *qt = stage + tid * SO_LD, *n0 = stage + (SC_CHUNK + 64) * SO_LD;
#pragma unroll 2
            for (int kk = 0; kk < 32; kk += RH) {
                float p = 0.f;
#pragma unroll
                for (int f = 0; f < RH; f += 4) {
                    const float4 u = *reinterpret_cast<const float4*>(qt + kk + f), w = *reinterpret_cast<const float4*>(n0 + kk + f);
                    p = fmaf(u.x, w.x, p); p = fmaf(u.y, w.y, p); p = fmaf(u.z, w.z, p); p = fmaf(u.w, w.w, p);
                }
                dot += p;
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int y = 0; y < 4; ++y) {
        const float f = e1[tt + 8 * y];
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[y][x] *= f;
    }
    if (a.normalizer) {
        if (tid < nt) {
            dot = __fmul_rn(dot, e1[tid]);              // (rounded before the sum goes on, as the outputs are)
            for (int s = 0; s <= tid; ++s) dot = __fadd_rn(dot, ps[tid * SO_LD + s]);
            dn[tid] = fmaxf(fabsf(dot), expf(-a.m_tok[(first + tid) * a.n_heads + h])) + 1e-6f;
        }
        __syncthreads();
    }
    // what the chunk's tokens read from one another, in order (tokens 8 sb .. 8 sb + 7 for the rows from 8 sb on; a later token's
    // value, which may not be finite, never meets an earlier row)
    const int n_sb = (nt + 7) / 8;
#pragma unroll 1
    for (int s = 0; s < n_sb * 8; s += 4) {
        const int sb = s >> 3, ds = s & 7;
        float4 w[4];
#pragma unroll
        for (int z = 0; z < 4; ++z) w[z] = *reinterpret_cast<const float4*>(vs + (s + z) * 64 + tj * 4);
#pragma unroll
        for (int y = 0; y < 4; ++y) {
            if (y < sb) continue;
            const float4 u = *reinterpret_cast<const float4*>(ps + (tt + 8 * y) * SO_LD + s);
            const float uz[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int z = 0; z < 4; ++z)
                if (y > sb || ds + z <= tt) {
                    acc[y][0] = fmaf(uz[z], w[z].x, acc[y][0]); acc[y][1] = fmaf(uz[z], w[z].y, acc[y][1]);
                    acc[y][2] = fmaf(uz[z], w[z].z, acc[y][2]); acc[y][3] = fmaf(uz[z], w[z].w, acc[y][3]);
                }
        }
    }
    const float sk = a.skip ? a.skip[h] : 0.f;
    const int j = j0 + tj * 4;
    const bool vec = a.dv % 4 == 0 && j + 3 < a.dv;
#pragma unroll
    for (int y = 0; y < 4; ++y) {
        const int t = tt + 8 * y;
        if (t >= nt) continue;
        float* to = a.o + (first + t) * a.n_heads * a.dv + (size_t)h * a.dv + j;
        if (a.skip)
#pragma unroll
            for (int x = 0; x < 4; ++x) acc[y][x] = fmaf(sk, vs[t * 64 + tj * 4 + x], acc[y][x]);
        if (a.normalizer) {
            const float d = dn[t];
#pragma unroll
            for (int x = 0; x < 4; ++x) acc[y][x] = acc[y][x] / d;
        }
        if (vec) *reinterpret_cast<float4*>(to) = make_float4(acc[y][0], acc[y][1], acc[y][2], acc[y][3]);
        else
#pragma unroll
            for (int x = 0; x < 4; ++x)
                if (j + x < a.dv) to[x] = acc[y][x];
    }
}

}  // namespace

// How many chunks the scratch of a step of N tokens in n_seqs sequences must hold.
MV_API int mv_scalar_chunks(int N, int n_seqs) { return N / SC_CHUNK + n_seqs + 1; }

// Arguments as mv_scalar_scan, plus the longest sequence's tokens (max_len) and scratch with chunks =
// mv_scalar_chunks(N, n_seqs): G [chunks, groups, SC_CHUNK, SC_CHUNK], before [room (+ 2 where room < chunks), n_heads, dv (+ 1), dk rounded up to 4] for windows of `room` chunks
// and factors [chunks, n_heads, 3 SC_CHUNK + 4], both 16-byte aligned.
MV_API int mv_scalar_scan_chunked(const float* q, int ldq, const float* k, int ldk, const float* v, int ldv,
                                  const float* log_a, int ld_a, const float* b, int ld_b, const float* skip,
                                  const float* m_tok, float q_scale, float* state, const int* slots, const int* cu,
                                  float* o, float* G, float* before, float* factors, int room, int chunks, int n_seqs, int max_len,
                                  int n_heads, int heads_per_group, int dk, int dv, int normalizer, cudaStream_t stream) {
    if (n_seqs <= 0 || max_len <= 0) return 0;
    if (dk < 1 || dk > 256 || dv < 1 || heads_per_group < 1 || n_heads % heads_per_group || (normalizer && !m_tok) || room < 1 ||
        ((uintptr_t)before | (uintptr_t)factors) % 16)
        return (int)cudaErrorInvalidValue;
    ScArgs a = {};
    a.q = q; a.ldq = ldq; a.k = k; a.ldk = ldk; a.v = v; a.ldv = ldv;
    a.log_a = log_a; a.ld_a = ld_a; a.b = b; a.ld_b = ld_b; a.skip = skip; a.m_tok = m_tok; a.q_scale = q_scale;
    a.state = state; a.before = before; a.G = G; a.slots = slots; a.cu = cu; a.o = o;
    const size_t rows = (size_t)chunks * n_heads;
    a.run = factors; a.e1 = a.run + rows * SC_CHUNK; a.e2 = a.e1 + rows * SC_CHUNK; a.el = a.e2 + rows * SC_CHUNK;
    a.n_heads = n_heads; a.heads_per_group = heads_per_group; a.dk = dk; a.dv = dv; a.lds = (dk + 3) & ~3;
    a.normalizer = normalizer ? 1 : 0; a.room = room;
    a.wide = cs_aligned(q, ldq, dk) && cs_aligned(k, ldk, dk) && cs_aligned(v, ldv, dv);
    cudaError_t attr = mv_allow_smem<ss_walk_kernel>(SW_SMEM);
    if (attr == cudaSuccess) attr = dk <= 128 ? mv_allow_smem<ss_output_kernel<4>>(SO_SMEM) : mv_allow_smem<ss_output_kernel<8>>(SO_SMEM);
    if (attr != cudaSuccess) return (int)attr;
    const int n_chunks = (max_len + SC_CHUNK - 1) / SC_CHUNK;
    mv_launch(ss_factors_kernel, dim3(n_chunks, (n_heads + 3) / 4, n_seqs), 128, 0, stream, a);
    int code = mv_launch_status();
    if (code) return code;
    mv_launch(ss_products_kernel, dim3(n_chunks, n_heads / heads_per_group, n_seqs), 64, 0, stream, a);
    if ((code = mv_launch_status())) return code;
    const dim3 grid(min(n_chunks, room) * ((dv + 63) / 64), n_heads, n_seqs);
    for (a.w0 = 0; a.w0 < chunks; a.w0 += room) {
        a.w1 = a.w0 + room;
        mv_launch(ss_walk_kernel, dim3((dv + 63) / 64 * ((dk + 63) / 64), n_heads, n_seqs), SC_WALK_THREADS, SW_SMEM, stream, a);
        if ((code = mv_launch_status())) return code;
        if (dk <= 128) mv_launch(ss_output_kernel<4>, grid, SO_THREADS, SO_SMEM, stream, a);
        else mv_launch(ss_output_kernel<8>, grid, SO_THREADS, SO_SMEM, stream, a);
        if ((code = mv_launch_status())) return code;
    }
    return 0;
}

// ------------------------------------------------------------------------------------------------
// Chunks for steps of few tokens (the wrapper's scan_takes_few): the same sums in the same order in two launches (three
// with a normalizer).  The second kernel walks a sequence's chunks with the state in registers and works the outputs out on the way: a block is
// 16 value columns of one head of one sequence, its 32 half-warps each hold RH key channels of every column.  Such a step is bound by its
// launches: 16 tokens of 64 heads of 128 x 64 in one group 36 us against 46 with the four kernels above, 64 tokens 46 against 51, 128 57
// against 55; 8 heads of 128 x 256 with a normalizer 36 against 46, 41 against 45, 50 against 50.
#define SF_COLS 16
#define SF_THREADS 256
#define SF_SCAN_THREADS 512
#define SF_GROUPS (SF_SCAN_THREADS / 16)
#define SF_RED_STRIDE (SC_CHUNK * SF_COLS + 16)

__global__ void __launch_bounds__(SF_THREADS)
scalar_few_products_kernel(const float* __restrict__ q, int ldq, const float* __restrict__ k, int ldk,
                             const int* __restrict__ cu, float* __restrict__ G, int n_groups, int dk) {
    mv_pdl_begin();
    extern __shared__ float smem[];
    const int lds = dk + 1;                         // odd row stride: rows of different tokens fall into different banks
    float* qa = smem;                               // [SC_CHUNK][lds]
    float* ka = qa + SC_CHUNK * lds;
    const int c = blockIdx.x, g = blockIdx.y, b = blockIdx.z;
    const int row0 = cu[b], len = cu[b + 1] - row0;
    if (c * SC_CHUNK >= len) return;
    const int nt = min(SC_CHUNK, len - c * SC_CHUNK);
    const int first = row0 + c * SC_CHUNK;
    const int chunk = row0 / SC_CHUNK + b + c;
    for (int idx = threadIdx.x; idx < nt * dk; idx += SF_THREADS) {
        const int t = idx / dk, i = idx - t * dk;
        qa[t * lds + i] = q[(size_t)(first + t) * ldq + (size_t)g * dk + i];
        ka[t * lds + i] = k[(size_t)(first + t) * ldk + (size_t)g * dk + i];
    }
    __syncthreads();
    float* Gc = G + ((size_t)chunk * n_groups + g) * SC_CHUNK * SC_CHUNK;
    for (int p = threadIdx.x; p < SC_CHUNK * SC_CHUNK; p += SF_THREADS) {
        const int t = p / SC_CHUNK, s = p - t * SC_CHUNK;
        float sum = 0.f;
        if (s <= t && t < nt) {
            const float* qt = qa + t * lds;
            const float* kt = ka + s * lds;
            for (int i = 0; i < dk; ++i) sum = fmaf(qt[i], kt[i], sum);
        }
        Gc[p] = sum;
    }
}

template <int RH>
__global__ void __launch_bounds__(SF_SCAN_THREADS)
scalar_few_scan_kernel(const float* __restrict__ q, int ldq, const float* __restrict__ k, int ldk,
                         const float* __restrict__ v, int ldv, const float* __restrict__ log_a, int ld_a,
                         const float* __restrict__ b_in, int ld_b, const float* __restrict__ skip, float q_scale,
                         const float* __restrict__ G, float* __restrict__ state, const int* __restrict__ slots,
                         const int* __restrict__ cu, float* __restrict__ o, int n_heads, int heads_per_group, int dk,
                         int dv, int ones_col) {
    mv_pdl_begin();
    constexpr int DKP = SF_GROUPS * RH;
    extern __shared__ __align__(16) float smem[];
    float* qt = smem;                               // [SC_CHUNK][DKP], zero beyond dk
    float* kt = qt + SC_CHUNK * DKP;
    float* vt = kt + SC_CHUNK * DKP;                // [SC_CHUNK][SF_COLS]
    float* pt = vt + SC_CHUNK * SF_COLS;            // [SC_CHUNK][SC_CHUNK]
    float* la = pt + SC_CHUNK * SC_CHUNK;           // [SC_CHUNK] log decays, then their running sum
    float* bs = la + SC_CHUNK;                      // [SC_CHUNK] input factors
    float* e1 = bs + SC_CHUNK;                      // [SC_CHUNK] e^(c_t) q_scale
    float* e2 = e1 + SC_CHUNK;                      // [SC_CHUNK] e^(c_last - c_t) b_t
    float* el = e2 + SC_CHUNK;                      // [1] e^(c_last) (padded to 16 floats)
    float* red = el + 16;                           // [SF_GROUPS][SF_RED_STRIDE]: [SC_CHUNK][SF_COLS] a group
    const int tile = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
    const int tid = threadIdx.x, col = tid & 15, grp = tid >> 4;
    const int cols = dv + (ones_col >= 0 ? 1 : 0);  // the state's and the output's columns
    const int j = tile * SF_COLS + col;
    const int row0 = cu[b], len = cu[b + 1] - row0;
    if (len <= 0) return;
    const int slot = mv_read_slot(slots[b]);
    const int n_groups = n_heads / heads_per_group, g = h / heads_per_group;
    const size_t goff = (size_t)g * dk;
    float* srow = state + (((size_t)slot * n_heads + h) * cols + (j < cols ? j : 0)) * dk;
    float S[RH];
#pragma unroll
    for (int r = 0; r < RH; ++r) {
        const int i = grp * RH + r;
        S[r] = (j < cols && i < dk) ? srow[i] : 0.f;
    }
    const float sk = skip ? skip[h] : 0.f;
    const int n_chunks = (len + SC_CHUNK - 1) / SC_CHUNK;
    constexpr int IT = SC_CHUNK * DKP / SF_SCAN_THREADS;
    static_assert(SC_CHUNK * SF_COLS == SF_SCAN_THREADS && SC_CHUNK * SC_CHUNK % SF_SCAN_THREADS == 0,
                  "a thread requests one value of v and whole rounds of the products");
    float rq[IT], rk[IT], rv, rp[SC_CHUNK * SC_CHUNK / SF_SCAN_THREADS], rla = 0.f, rb = 0.f;
    auto request = [&](int c) {
        const int nt = min(SC_CHUNK, len - c * SC_CHUNK);
        const int first = row0 + c * SC_CHUNK;
        const int chunk = row0 / SC_CHUNK + b + c;
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            const int idx = tid + it * SF_SCAN_THREADS, t = idx / DKP, i = idx - t * DKP;
            const bool in = t < nt && i < dk;
            rq[it] = in ? q[(size_t)(first + t) * ldq + goff + i] : 0.f;
            rk[it] = in ? k[(size_t)(first + t) * ldk + goff + i] : 0.f;
        }
        {
            const int t = tid / SF_COLS, cc = tile * SF_COLS + (tid - t * SF_COLS);
            rv = t < nt ? (cc < dv ? v[(size_t)(first + t) * ldv + (size_t)h * dv + cc] : (cc == ones_col ? 1.f : 0.f)) : 0.f;
        }
        const float* Gc = G + ((size_t)chunk * n_groups + g) * SC_CHUNK * SC_CHUNK;
#pragma unroll
        for (int it = 0; it < SC_CHUNK * SC_CHUNK / SF_SCAN_THREADS; ++it) rp[it] = Gc[tid + it * SF_SCAN_THREADS];
        if (tid < SC_CHUNK) {
            rla = tid < nt ? log_a[(size_t)(first + tid) * ld_a + h] : 0.f;
            rb = tid < nt ? b_in[(size_t)(first + tid) * ld_b + h] : 0.f;
        }
    };
    request(0);
    for (int c = 0; c < n_chunks; ++c) {
        const int nt = min(SC_CHUNK, len - c * SC_CHUNK);
        const int first = row0 + c * SC_CHUNK;
        __syncthreads();                            // the chunk before is done with shared memory
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            qt[tid + it * SF_SCAN_THREADS] = rq[it];
            kt[tid + it * SF_SCAN_THREADS] = rk[it];
        }
        vt[tid] = rv;
#pragma unroll
        for (int it = 0; it < SC_CHUNK * SC_CHUNK / SF_SCAN_THREADS; ++it) pt[tid + it * SF_SCAN_THREADS] = rp[it];
        if (tid < SC_CHUNK) {
            // the running sum of the log decays over the chunk (one warp), and the factors that follow from it
            float run = rla;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const float up = __shfl_up_sync(0xffffffffu, run, d);
                if (tid >= d) run += up;
            }
            const float last = __shfl_sync(0xffffffffu, run, nt - 1);
            la[tid] = run;
            bs[tid] = rb;
            e1[tid] = expf(run) * q_scale;
            e2[tid] = tid < nt ? expf(last - run) * rb : 0.f;
            if (tid == 0) el[0] = expf(last);
        }
        __syncthreads();
        if (c + 1 < n_chunks) request(c + 1);
        // this head's factors on the group's products: e^(c_t - c_s) b_s q_scale (own entries only: no one else reads them yet)
#pragma unroll
        for (int it = 0; it < SC_CHUNK * SC_CHUNK / SF_SCAN_THREADS; ++it) {
            const int p = tid + it * SF_SCAN_THREADS, t = p / SC_CHUNK, s = p - t * SC_CHUNK;
            pt[p] = (s <= t && t < nt) ? pt[p] * expf(la[t] - la[s]) * bs[s] * q_scale : 0.f;
        }
        // what the chunk's tokens read from the state before the chunk: this half-warp's key channels
#pragma unroll 4
        for (int t = 0; t < SC_CHUNK; ++t) {
            const float4* q4 = reinterpret_cast<const float4*>(qt + t * DKP + grp * RH);
            float acc = 0.f;
#pragma unroll
            for (int r = 0; r < RH; r += 4) {
                const float4 x = q4[r >> 2];
                acc = fmaf(x.x, S[r], acc); acc = fmaf(x.y, S[r + 1], acc);
                acc = fmaf(x.z, S[r + 2], acc); acc = fmaf(x.w, S[r + 3], acc);
            }
            red[grp * SF_RED_STRIDE + t * SF_COLS + col] = acc;
        }
        // the state after the chunk
        const float decay = el[0];
#pragma unroll
        for (int r = 0; r < RH; ++r) S[r] *= decay;
#pragma unroll 4
        for (int s = 0; s < SC_CHUNK; ++s) {
            const float vj = vt[s * SF_COLS + col] * e2[s];
            const float4* k4 = reinterpret_cast<const float4*>(kt + s * DKP + grp * RH);
#pragma unroll
            for (int r = 0; r < RH; r += 4) {
                const float4 x = k4[r >> 2];
                S[r] = fmaf(x.x, vj, S[r]); S[r + 1] = fmaf(x.y, vj, S[r + 1]);
                S[r + 2] = fmaf(x.z, vj, S[r + 2]); S[r + 3] = fmaf(x.w, vj, S[r + 3]);
            }
        }
        __syncthreads();
        // outputs: the groups' shares in a fixed order, then the chunk's own tokens
        for (int idx = tid; idx < nt * SF_COLS; idx += SF_SCAN_THREADS) {
            const int t = idx / SF_COLS, cc = idx - t * SF_COLS;
            float sum = 0.f;
#pragma unroll
            for (int gg = 0; gg < SF_GROUPS; ++gg) sum += red[gg * SF_RED_STRIDE + t * SF_COLS + cc];
            sum *= e1[t];
            for (int s = 0; s <= t; ++s) sum = fmaf(pt[t * SC_CHUNK + s], vt[s * SF_COLS + cc], sum);
            const int oc = tile * SF_COLS + cc;
            if (oc < dv) sum = fmaf(sk, vt[t * SF_COLS + cc], sum);
            if (oc < cols) o[(size_t)(first + t) * n_heads * cols + (size_t)h * cols + oc] = sum;
        }
    }
    if (j < cols && mv_slot_ok(slots[b])) {
#pragma unroll
        for (int r = 0; r < RH; ++r) {
            const int i = grp * RH + r;
            if (i < dk) srow[i] = S[r];
        }
    }
}

template <int RH>
static int scalar_few_scan_launch(dim3 grid, cudaStream_t stream, const float* q, int ldq, const float* k, int ldk,
                                    const float* v, int ldv, const float* log_a, int ld_a, const float* b, int ld_b,
                                    const float* skip, float q_scale, const float* G, float* state, const int* slots,
                                    const int* cu, float* o, int n_heads, int hpg, int dk, int dv, int ones_col) {
    const size_t smem = sizeof(float) * ((size_t)2 * SC_CHUNK * SF_GROUPS * RH + SC_CHUNK * SF_COLS + SC_CHUNK * SC_CHUNK +
                                         4 * SC_CHUNK + 16 + SF_GROUPS * SF_RED_STRIDE);
    const cudaError_t attr = mv_allow_smem<scalar_few_scan_kernel<RH>>(smem);
    if (attr != cudaSuccess) return (int)attr;
    mv_launch(scalar_few_scan_kernel<RH>, grid, SF_SCAN_THREADS, smem, stream, q, ldq, k, ldk, v, ldv, log_a, ld_a, b, ld_b,
              skip, q_scale, G, state, slots, cu, o, n_heads, hpg, dk, dv, ones_col);
    return mv_launch_status();
}

// o[n, h, :] = o_aug[n, h, :dv] / (max(|o_aug[n, h, dv]|, e^(-m[n, h])) + 1e-6)
__global__ void __launch_bounds__(256)
memory_normalize_kernel(const float* __restrict__ o_aug, const float* __restrict__ m_tok, float* __restrict__ o,
                        long long total, int dv) {
    mv_pdl_begin();
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const long long nh = idx / dv;
    const int d = (int)(idx - nh * dv);
    const float den = fmaxf(fabsf(o_aug[nh * (dv + 1) + dv]), expf(-m_tok[nh])) + 1e-6f;
    o[idx] = o_aug[nh * (dv + 1) + d] / den;
}

// Arguments as mv_scalar_scan, plus the longest sequence's tokens (max_len) and scratch: G [chunks, groups,
// SC_CHUNK, SC_CHUNK] with chunks = mv_scalar_chunks(N, n_seqs), and with a normalizer o_aug [N, n_heads * (dv + 1)].
MV_API int mv_scalar_scan_few(const float* q, int ldq, const float* k, int ldk, const float* v, int ldv,
                                  const float* log_a, int ld_a, const float* b, int ld_b, const float* skip,
                                  const float* m_tok, float q_scale, float* state, const int* slots, const int* cu,
                                  float* o, float* G, float* o_aug, int N, int n_seqs, int max_len, int n_heads,
                                  int heads_per_group, int dk, int dv, int normalizer, cudaStream_t stream) {
    if (n_seqs <= 0 || max_len <= 0) return 0;
    if (dk < 1 || dk > 256 || dv < 1 || heads_per_group < 1 || n_heads % heads_per_group ||
        (normalizer && (!m_tok || !o_aug)))
        return (int)cudaErrorInvalidValue;
    const int n_groups = n_heads / heads_per_group;
    const size_t smem_a = sizeof(float) * (size_t)2 * SC_CHUNK * (dk + 1);
    const cudaError_t attr = mv_allow_smem<scalar_few_products_kernel>(sizeof(float) * 2 * SC_CHUNK * 257);   // what the largest dk needs
    if (attr != cudaSuccess) return (int)attr;
    mv_launch(scalar_few_products_kernel, dim3((max_len + SC_CHUNK - 1) / SC_CHUNK, n_groups, n_seqs), SF_THREADS, smem_a,
              stream, q, ldq, k, ldk, cu, G, n_groups, dk);
    int code = mv_launch_status();
    if (code) return code;
    const int cols = dv + (normalizer ? 1 : 0);
    const dim3 grid((cols + SF_COLS - 1) / SF_COLS, n_heads, n_seqs);
    float* out = normalizer ? o_aug : o;
    const int ones_col = normalizer ? dv : -1;
    if (dk <= 128)
        code = scalar_few_scan_launch<4>(grid, stream, q, ldq, k, ldk, v, ldv, log_a, ld_a, b, ld_b, skip, q_scale, G, state,
                                           slots, cu, out, n_heads, heads_per_group, dk, dv, ones_col);
    else
        code = scalar_few_scan_launch<8>(grid, stream, q, ldq, k, ldk, v, ldv, log_a, ld_a, b, ld_b, skip, q_scale, G, state,
                                           slots, cu, out, n_heads, heads_per_group, dk, dv, ones_col);
    if (code || !normalizer) return code;
    const long long total = (long long)N * n_heads * dv;
    mv_launch(memory_normalize_kernel, (unsigned)((total + 255) / 256), 256, 0, stream, (const float*)o_aug, m_tok, o, total, dv);
    return mv_launch_status();
}
