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

// zi, zf: the gates' projections [N, >= n_heads] with row strides; bi, bf [n_heads]; m_state [slots][n_heads];
// log_a, b_out, m_tok [N, n_heads] dense.
MV_API int mv_memory_gates(const float* zi, int ld_i, const float* zf, int ld_f, const float* bi, const float* bf,
                           float cap, float* m_state, const int* slots, const int* cu, float* log_a, float* b_out,
                           float* m_tok, int n_seqs, int n_heads, cudaStream_t stream) {
    if (n_seqs <= 0) return 0;
    if (!(cap > 0.f) || n_heads < 1) return (int)cudaErrorInvalidValue;
    const int warps = n_seqs * n_heads;
    mv_launch(memory_gates_kernel, (warps + 3) / 4, 128, 0, stream, zi, ld_i, zf, ld_f, bi, bf, cap, m_state, slots, cu, log_a,
              b_out, m_tok, n_seqs, n_heads);
    return mv_launch_status();
}

// ------------------------------------------------------------------------------------------------
// The same recurrence for steps that bring many tokens a sequence, in chunks of CS_CHUNK tokens (chunked_state.cuh): with
// c_t the sum of log a over the chunk's tokens up to t (all of it <= 0) and S0 the state before the chunk,
//
//     o_t   = e^(c_t) q_t^T S0 + sum_{s <= t} (q_t . k_s) e^(c_t - c_s) b_s v_s  (+ skip v_t),
//     S_end = e^(c_last) S0 + sum_s e^(c_last - c_s) b_s k_s v_s^T.
//
// Every exponent is a difference of cumulative logarithms taken the right way round, so every factor lies in
// (0, 1] (times b): nothing overflows however small a decay is.  Because the decay is one number a head, the products
// q_t . k_s are worked out once per GROUP of heads that share q and k.
// Bound by the walk and the outputs, both near 0.35 to 0.4 of the multiply-adds' rate.  Two sequences of 611 and 1,437 tokens, 64
// heads of 128 x 64 in one group: 110 us the walk, 90 the outputs, 10 the products, 3 the factors, where the kernel that walked
// 32 tokens and 16 columns at a time and worked the outputs out on the way (half of its time in adding up 32 half-warps'
// shares) took 430.
// How many chunks the scratch of a step of N tokens in n_seqs sequences must hold.
MV_API int mv_scalar_chunks(int N, int n_seqs) { return N / CS_CHUNK + n_seqs + 1; }
// And how many floats a chunk its factors take.
MV_API int mv_scalar_factor_floats(int n_heads) { return cs_factor_floats(n_heads); }

// Arguments as mv_scalar_scan, plus the longest sequence's tokens (max_len) and scratch with chunks =
// mv_scalar_chunks(N, n_seqs): G [chunks, groups, CS_CHUNK, CS_CHUNK], before [chunks, n_heads, dv (+ 1), dk rounded up to 4] and factors
// [chunks, mv_scalar_factor_floats(n_heads)].
MV_API int mv_scalar_scan_chunked(const float* q, int ldq, const float* k, int ldk, const float* v, int ldv,
                                  const float* log_a, int ld_a, const float* b, int ld_b, const float* skip,
                                  const float* m_tok, float q_scale, float* state, const int* slots, const int* cu,
                                  float* o, float* G, float* before, float* factors, int chunks, int n_seqs, int max_len, int n_heads,
                                  int heads_per_group, int dk, int dv, int normalizer, cudaStream_t stream) {
    if (n_seqs <= 0 || max_len <= 0) return 0;
    if (dk < 1 || dk > 256 || dv < 1 || heads_per_group < 1 || n_heads % heads_per_group || (normalizer && !m_tok))
        return (int)cudaErrorInvalidValue;
    CsArgs a = {};
    a.q = q; a.ldq = ldq; a.k = k; a.ldk = ldk; a.v = v; a.ldv = ldv;
    a.log_a = log_a; a.ld_a = ld_a; a.b = b; a.ld_b = ld_b;
    a.skip = skip; a.m_tok = normalizer ? m_tok : nullptr; a.q_scale = q_scale;
    a.state = state; a.before = before; a.slots = slots; a.cu = cu; a.o = o;
    a.n_heads = n_heads; a.heads_per_group = heads_per_group; a.dk = dk; a.dv = dv;
    return cs_launch<false>(a, G, factors, chunks, n_seqs, max_len, stream);
}
