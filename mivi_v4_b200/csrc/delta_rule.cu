// The gated delta rule with a decay per key channel, one head at a time:
//
//     S  <- diag(g_t) S                        (S: dk x dv; g_t: a factor in (0, 1] per key channel)
//     u_t = beta_t (v_t - S^T k_t)             (what the state does not yet say about v_t)
//     S  <- S + k_t u_t^T
//     o_t = S^T q_t                            (the read-out sees the token's own write)
//
// with q and k made unit vectors per head first (x / sqrt(sum x^2 + norm_eps), q also times q_scale),
// beta_t = sigmoid(b_t) per head, and g = exp(-exp(A_log_h) softplus(a + dt_bias)) per head and key channel
// (with head_decay: a and dt_bias hold one number a head, and all key channels of a head share its decay).
// Head h reads q and k of head h / (heads / kv_heads).  The state lives in 32-bit floats per sequence slot and
// is carried from step to step; a step brings any number of next tokens for each of its sequences.  Everything
// here is 32-bit.
//
// Work: a block is (16 value columns, head, sequence) and walks the sequence's tokens in order.  A value column
// is owned by 8 lanes, lane p holding the state's rows p, p + 8, ... of that column in registers; the state is
// stored [slot][head][dv][dk], so these 8 lanes read 32 contiguous bytes.  Tokens come through shared memory
// eight at a time.  The order of every sum depends on nothing but dk, so a prompt gives the same numbers
// however it is cut into steps.
#include "common.cuh"

#define DR_COLS 16
#define DR_PART 8
#define DR_CHUNK 8

__device__ __forceinline__ float dr_softplus(float z) { return z > 20.f ? z : log1pf(expf(z)); }

template <int R>
__global__ void __launch_bounds__(DR_COLS * DR_PART)
delta_scan_kernel(const float* __restrict__ q, int ldq, const float* __restrict__ k, int ldk,
                  const float* __restrict__ v, int ldv, const float* __restrict__ b, int ldb,
                  const float* __restrict__ a, int lda, const float* __restrict__ dt_bias,
                  const float* __restrict__ a_log, float q_scale, float norm_eps, float* __restrict__ state,
                  const int* __restrict__ slots, const int* __restrict__ cu, float* __restrict__ o, int n_heads,
                  int kv_heads, int dk, int dv, int head_decay) {
    mv_pdl_begin();
    extern __shared__ float smem[];
    float* qs = smem;                           // [DR_CHUNK][dk]
    float* ks = qs + DR_CHUNK * dk;
    float* gs = ks + DR_CHUNK * dk;
    float* vs = gs + DR_CHUNK * dk;             // [DR_CHUNK][DR_COLS]
    float* bs = vs + DR_CHUNK * DR_COLS;        // [DR_CHUNK]
    float* ns = bs + DR_CHUNK;                  // [DR_CHUNK][2]: what q and k are multiplied by
    const int tile = blockIdx.x, h = blockIdx.y, sq = blockIdx.z;
    const int tid = threadIdx.x, p = tid & (DR_PART - 1), jl = tid >> 3;
    const int j = tile * DR_COLS + jl;
    const int row0 = cu[sq], len = cu[sq + 1] - row0;
    if (len <= 0) return;
    const int hk = h / (n_heads / kv_heads);
    const int slot = mv_read_slot(slots[sq]);
    float* srow = state + (((size_t)slot * n_heads + h) * dv + (j < dv ? j : 0)) * dk;
    float S[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = p + DR_PART * r;
        S[r] = (j < dv && i < dk) ? srow[i] : 0.f;
    }
    const float rate = expf(a_log[h]);
    for (int c0 = 0; c0 < len; c0 += DR_CHUNK) {
        const int nt = min(DR_CHUNK, len - c0);
        __syncthreads();
        for (int idx = tid; idx < nt * dk; idx += DR_COLS * DR_PART) {
            const int t = idx / dk, i = idx - t * dk;
            const size_t row = (size_t)(row0 + c0 + t);
            qs[idx] = q[row * ldq + (size_t)hk * dk + i];
            ks[idx] = k[row * ldk + (size_t)hk * dk + i];
            // one decay logit a head (head_decay) or one a head and key channel
            const size_t ai = head_decay ? (size_t)h : (size_t)h * dk + i;
            gs[idx] = expf(-rate * dr_softplus(a[row * lda + ai] + dt_bias[ai]));
        }
        for (int idx = tid; idx < nt * DR_COLS; idx += DR_COLS * DR_PART) {
            const int t = idx / DR_COLS, c = idx - t * DR_COLS, col = tile * DR_COLS + c;
            vs[idx] = col < dv ? v[(size_t)(row0 + c0 + t) * ldv + (size_t)h * dv + col] : 0.f;
        }
        if (tid < nt) bs[tid] = 1.0f / (1.0f + expf(-b[(size_t)(row0 + c0 + tid) * ldb + h]));
        __syncthreads();
        {
            // sixteen groups of eight lanes: group (t, which) sums the squares of token t's q or k
            const int t = jl >> 1, which = jl & 1;
            const float* src = (which ? ks : qs) + t * dk;
            float ss = 0.f;
            if (t < nt)
                for (int i = p; i < dk; i += DR_PART) ss = fmaf(src[i], src[i], ss);
            ss += __shfl_xor_sync(0xffffffffu, ss, 1);
            ss += __shfl_xor_sync(0xffffffffu, ss, 2);
            ss += __shfl_xor_sync(0xffffffffu, ss, 4);
            if (p == 0 && t < nt) ns[2 * t + which] = (which ? 1.f : q_scale) / sqrtf(ss + norm_eps);
        }
        __syncthreads();
        for (int idx = tid; idx < nt * dk; idx += DR_COLS * DR_PART) {
            const int t = idx / dk;
            qs[idx] *= ns[2 * t];
            ks[idx] *= ns[2 * t + 1];
        }
        __syncthreads();
        for (int t = 0; t < nt; ++t) {
            const float vj = vs[t * DR_COLS + jl], bt = bs[t];
            const float* qt = qs + t * dk;
            const float* kt = ks + t * dk;
            const float* gt = gs + t * dk;
            float said = 0.f;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int i = p + DR_PART * r;
                if (i < dk) {
                    S[r] *= gt[i];
                    said = fmaf(S[r], kt[i], said);
                }
            }
            said += __shfl_xor_sync(0xffffffffu, said, 1);
            said += __shfl_xor_sync(0xffffffffu, said, 2);
            said += __shfl_xor_sync(0xffffffffu, said, 4);
            const float u = bt * (vj - said);
            float acc = 0.f;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int i = p + DR_PART * r;
                if (i < dk) {
                    S[r] = fmaf(kt[i], u, S[r]);
                    acc = fmaf(S[r], qt[i], acc);
                }
            }
            acc += __shfl_xor_sync(0xffffffffu, acc, 1);
            acc += __shfl_xor_sync(0xffffffffu, acc, 2);
            acc += __shfl_xor_sync(0xffffffffu, acc, 4);
            if (p == 0 && j < dv) o[(size_t)(row0 + c0 + t) * n_heads * dv + (size_t)h * dv + j] = acc;
        }
    }
    if (j < dv && mv_slot_ok(slots[sq])) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int i = p + DR_PART * r;
            if (i < dk) srow[i] = S[r];
        }
    }
}

MV_GUARD_SETTER(delta_rule)

// q, k [N, >= kv_heads * dk], v [N, >= n_heads * dv], b [N, >= n_heads] (beta's logits), a [N, >= n_heads * dk] (the
// decay's logits) with row strides ldq, ldk, ldv, ldb, lda (elements); dt_bias [n_heads * dk]; a_log [n_heads];
// state [slots][n_heads][dv][dk]; slots [n_seqs]; cu [n_seqs + 1]; o [N, n_heads * dv] dense.
MV_API int mv_delta_scan(const float* q, int ldq, const float* k, int ldk, const float* v, int ldv, const float* b, int ldb,
                         const float* a, int lda, const float* dt_bias, const float* a_log, float q_scale, float norm_eps,
                         float* state, const int* slots, const int* cu, float* o, int n_seqs, int n_heads, int kv_heads,
                         int dk, int dv, int head_decay, cudaStream_t stream) {
    if (n_seqs <= 0) return 0;
    if (dk < 1 || dk > 256 || dv < 1 || kv_heads < 1 || n_heads % kv_heads) return (int)cudaErrorInvalidValue;
    const dim3 grid((dv + DR_COLS - 1) / DR_COLS, n_heads, n_seqs);
    const size_t smem = (size_t)DR_CHUNK * (3 * dk + DR_COLS + 3) * sizeof(float);
#define DR_LAUNCH(R)                                                                                                   \
    mv_launch(delta_scan_kernel<R>, grid, DR_COLS * DR_PART, smem, stream, q, ldq, k, ldk, v, ldv, b, ldb, a, lda, dt_bias, \
              a_log, q_scale, norm_eps, state, slots, cu, o, n_heads, kv_heads, dk, dv, head_decay)
    if (dk <= 32) DR_LAUNCH(4);
    else if (dk <= 64) DR_LAUNCH(8);
    else if (dk <= 128) DR_LAUNCH(16);
    else DR_LAUNCH(32);
#undef DR_LAUNCH
    return mv_launch_status();
}

// ------------------------------------------------------------------------------------------- steps of many tokens
// Two kernels.  delta_prepare does, once per token, what does not depend on the state: q and k as unit vectors
// (q also times q_scale), k . q of each q/k head, the decays g, and beta; one row of `prep` a token:
//     [q: kv_heads W | k: kv_heads W | g: heads W | beta: heads | k.q: kv_heads]      (row stride ldp, 32-bit)
// W is dk, or from 64 key channels on what delta_scan_wide_kernel reads: dk rounded up to 32 R = 64, 128, 192 or 256 (zeros beyond dk)
// in the order in which its lanes own them.
// delta_scan_long then walks a sequence with nothing but the recurrence in its loop.  The tokens come through
// shared memory sixteen at a time, the next sixteen on their way (cp.async) while these are worked on.  In the
// loop  S' = diag(g) S  is read twice at once, a = S'^T k and b = S'^T q, so that one round of shuffles serves
// both; u = beta (v - a); o = b + u (k . q), which is (S' + k u^T)^T q; S = S' + k u^T.
#define DL_CHUNK 16

// Where channel i of a head's 32 R lies in its W = 8 (4 R + 4) floats of prep: lane i % 8 owns the channels i, i + 8, .. and finds
// them side by side, 16 bytes of padding behind them keep the lanes' reads from shared memory in different banks.
__device__ __forceinline__ int dl_place(int i, int R) { return R ? (i & 7) * (4 * R + 4) + (i >> 3) : i; }

__global__ void __launch_bounds__(256)
delta_prepare_kernel(const float* __restrict__ q, int ldq, const float* __restrict__ k, int ldk,
                     const float* __restrict__ b, int ldb, const float* __restrict__ a, int lda,
                     const float* __restrict__ dt_bias, const float* __restrict__ a_log, float q_scale, float norm_eps,
                     float* __restrict__ prep, int ldp, int n_heads, int kv_heads, int dk, int W, int R, int head_decay) {
    mv_pdl_begin();
    const int n = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    float* row = prep + (size_t)n * ldp;
    const int qk = kv_heads * W, hk = n_heads * W;
    for (int h = warp; h < kv_heads; h += nwarps) {
        const float* qh = q + (size_t)n * ldq + (size_t)h * dk;
        const float* kh = k + (size_t)n * ldk + (size_t)h * dk;
        float sq = 0.f, sk = 0.f, dot = 0.f;
        for (int i = lane; i < dk; i += 32) {
            const float x = qh[i], y = kh[i];
            sq = fmaf(x, x, sq);
            sk = fmaf(y, y, sk);
            dot = fmaf(x, y, dot);
        }
        sq = mv_warp_sum(sq);
        sk = mv_warp_sum(sk);
        dot = mv_warp_sum(dot);
        const float fq = q_scale / sqrtf(sq + norm_eps), fk = 1.0f / sqrtf(sk + norm_eps);
        for (int i = lane; i < (R ? 32 * R : dk); i += 32) {
            const int at = h * W + dl_place(i, R);
            row[at] = i < dk ? qh[i] * fq : 0.f;
            row[qk + at] = i < dk ? kh[i] * fk : 0.f;
        }
        if (lane == 0) row[2 * qk + hk + n_heads + h] = dot * fq * fk;
    }
    const int n_ch = R ? 32 * R : dk;
    for (int e = threadIdx.x; e < n_heads * n_ch; e += blockDim.x) {
        const int h = e / n_ch, i = e - h * n_ch;
        const int ai = head_decay ? h : h * dk + i;
        row[2 * qk + h * W + dl_place(i, R)] =
            i < dk ? expf(-expf(a_log[h]) * dr_softplus(a[(size_t)n * lda + ai] + dt_bias[ai])) : 0.f;
    }
    for (int h = threadIdx.x; h < n_heads; h += blockDim.x)
        row[2 * qk + hk + h] = 1.0f / (1.0f + expf(-b[(size_t)n * ldb + h]));
}

__device__ __forceinline__ void dl_copy4(float* smem, const float* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void dl_copy16(float* smem, const float* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void dl_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void dl_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// The rows of q, k and g, DR_COLS columns of v, beta and k.q of up to DL_CHUNK tokens from token c0 of a sequence on
// their way into one buffer of shared memory.
__device__ __forceinline__ void dl_stage(float* buf, const float* __restrict__ prep, int ldp, const float* __restrict__ v,
                                         int ldv, int row0, int c0, int len, int h, int hk, int qk, int n_heads, int dk,
                                         int dv, int col0, int wide, int tid, int nthreads) {
        const int nt = min(DL_CHUNK, len - c0);
        float* qs = buf;
        float* ks = qs + DL_CHUNK * dk;
        float* gs = ks + DL_CHUNK * dk;
        float* vs = gs + DL_CHUNK * dk;
        float* bs = vs + DL_CHUNK * DR_COLS;
        float* ds = bs + DL_CHUNK;
        if (wide) {
            const int dk4 = dk >> 2;
            for (int idx = tid; idx < nt * dk4; idx += nthreads) {
                const int t = idx / dk4, i = (idx - t * dk4) << 2;
                const float* src = prep + (size_t)(row0 + c0 + t) * ldp;
                dl_copy16(qs + t * dk + i, src + (size_t)hk * dk + i);
                dl_copy16(ks + t * dk + i, src + qk + (size_t)hk * dk + i);
                dl_copy16(gs + t * dk + i, src + 2 * qk + (size_t)h * dk + i);
            }
        } else {
            for (int idx = tid; idx < nt * dk; idx += nthreads) {
                const int t = idx / dk, i = idx - t * dk;
                const float* src = prep + (size_t)(row0 + c0 + t) * ldp;
                dl_copy4(qs + idx, src + (size_t)hk * dk + i);
                dl_copy4(ks + idx, src + qk + (size_t)hk * dk + i);
                dl_copy4(gs + idx, src + 2 * qk + (size_t)h * dk + i);
            }
        }
        for (int idx = tid; idx < nt * DR_COLS; idx += nthreads) {
            const int t = idx / DR_COLS, c = idx - t * DR_COLS;
            if (col0 + c < dv) dl_copy4(vs + idx, v + (size_t)(row0 + c0 + t) * ldv + (size_t)h * dv + col0 + c);
        }
        if (tid < nt) {
            const float* src = prep + (size_t)(row0 + c0 + tid) * ldp + 2 * qk + (size_t)n_heads * dk;
            dl_copy4(bs + tid, src + h);
            dl_copy4(ds + tid, src + n_heads + hk);
        }
    }

// One buffer of shared memory: [q: CHUNK dk | k: CHUNK dk | g: CHUNK dk | v: CHUNK DR_COLS | beta: CHUNK | k.q: CHUNK]
// DR_PART lanes share a column of the state (element i of it with lane i % DR_PART).  Keys under 64 channels run here; from 64 channels on delta_scan_wide_kernel below takes over.
template <int R>
__global__ void __launch_bounds__(DR_COLS * DR_PART)
delta_scan_long_kernel(const float* __restrict__ prep, int ldp, const float* __restrict__ v, int ldv,
                       float* __restrict__ state, const int* __restrict__ slots, const int* __restrict__ cu,
                       float* __restrict__ o, int n_heads, int kv_heads, int dk, int dv, int wide) {
    mv_pdl_wait();                          // the successor is let go when the last token is done
    extern __shared__ __align__(16) float dl_smem[];
    const int per = DL_CHUNK * (3 * dk + DR_COLS + 2);
    const int tile = blockIdx.x, h = blockIdx.y, sq = blockIdx.z;
    const int tid = threadIdx.x, p = tid & (DR_PART - 1), jl = tid / DR_PART;
    const int j = tile * DR_COLS + jl;
    const int row0 = cu[sq], len = cu[sq + 1] - row0;
    if (len <= 0) return;
    const int hk = h / (n_heads / kv_heads);
    const int qk = kv_heads * dk;
    const int slot = mv_read_slot(slots[sq]);
    float* srow = state + (((size_t)slot * n_heads + h) * dv + (j < dv ? j : 0)) * dk;
    float S[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = p + DR_PART * r;
        S[r] = (j < dv && i < dk) ? srow[i] : 0.f;
    }
    const int col0 = tile * DR_COLS;

    auto stage = [&](int c0, float* buf) {
        dl_stage(buf, prep, ldp, v, ldv, row0, c0, len, h, hk, qk, n_heads, dk, dv, col0, wide, tid, DR_COLS * DR_PART);
    };

    stage(0, dl_smem);
    dl_commit();
    int which = 0;
    for (int c0 = 0; c0 < len; c0 += DL_CHUNK, which ^= 1) {
        float* buf = dl_smem + which * per;
        if (c0 + DL_CHUNK < len) {
            stage(c0 + DL_CHUNK, dl_smem + (which ^ 1) * per);
            dl_commit();
            dl_wait<1>();
        } else {
            dl_wait<0>();
        }
        __syncthreads();
        const int nt = min(DL_CHUNK, len - c0);
        const float* qs = buf;
        const float* ks = qs + DL_CHUNK * dk;
        const float* gs = ks + DL_CHUNK * dk;
        const float* vs = gs + DL_CHUNK * dk;
        const float* bs = vs + DL_CHUNK * DR_COLS;
        const float* ds = bs + DL_CHUNK;
        for (int t = 0; t < nt; ++t) {
            const float* qt = qs + t * dk;
            const float* kt = ks + t * dk;
            const float* gt = gs + t * dk;
            float a0 = 0.f, a1 = 0.f, b0 = 0.f, b1 = 0.f;
#pragma unroll
            for (int r = 0; r < R; r += 2) {
                const int i0 = p + DR_PART * r, i1 = i0 + DR_PART;
                if (i0 < dk) {
                    S[r] *= gt[i0];
                    a0 = fmaf(S[r], kt[i0], a0);
                    b0 = fmaf(S[r], qt[i0], b0);
                }
                if (r + 1 < R && i1 < dk) {
                    S[r + 1] *= gt[i1];
                    a1 = fmaf(S[r + 1], kt[i1], a1);
                    b1 = fmaf(S[r + 1], qt[i1], b1);
                }
            }
            float said = a0 + a1, read = b0 + b1;
#pragma unroll
            for (int d = 1; d < DR_PART; d <<= 1) {
                said += __shfl_xor_sync(0xffffffffu, said, d);
                read += __shfl_xor_sync(0xffffffffu, read, d);
            }
            const float u = bs[t] * ((j < dv ? vs[t * DR_COLS + jl] : 0.f) - said);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int i = p + DR_PART * r;
                if (i < dk) S[r] = fmaf(kt[i], u, S[r]);
            }
            if (p == 0 && j < dv) o[(size_t)(row0 + c0 + t) * n_heads * dv + (size_t)h * dv + j] = fmaf(u, ds[t], read);
        }
        __syncthreads();
    }
    mv_pdl_launch_dependents();
    if (j < dv && mv_slot_ok(slots[sq])) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int i = p + DR_PART * r;
            if (i < dk) srow[i] = S[r];
        }
    }
}

// From 64 key channels on: four warps carry 16 columns of the state, 8 lanes a column, lane l the channels l, l + 8, .. (4 R of
// dk <= 32 R).  What bounds it is the chain from one token to the next - decay, dot product with k, its sum over the lanes,
// u, the state's update - and what the warps issue beside it.  So a lane adds its channels in four chains (those 32 apart) and
// joins them two and two, which leaves three exchanges, after which all eight lanes have the sum; the next token's rows are
// requested between the exchanges; a fifth warp does all copying; and the lanes only leave their parts of q's read-out (and
// u) behind, which a sixth warp adds up and writes out a chunk later.  (Two columns a warp of 32 lanes: six exchanges in the chain,
// 690 us for 2,048 tokens of 16 heads of 128 x 128; without the two further warps 540.  The order in which a sum's parts are
// added is the same in all of them, and so is every bit.)  2,048 tokens of 16 heads of
// 128 x 128: 690 -> 395 us (four sequences of 130 to 1,500 tokens, 8 heads: 572 -> 345).
// `bufs`: two buffers, or one where no sequence brings more than a chunk, so that more blocks fit a multiprocessor (32 sequences of
// 16 tokens, 8 heads of 128 x 128: 63 us with two buffers, 57 with one, 55 with two columns a warp; of 160 x 128, with R 8 127, now 78
// and 70).
constexpr int DW_THREADS = DR_COLS * 8, DW_ALL = DW_THREADS + 64;
constexpr size_t dw_smem(int R, int bufs) {
    return sizeof(float) * bufs * (DL_CHUNK * (3 * 8 * (4 * R + 4) + DR_COLS + 1 + 3) + DL_CHUNK * (DW_THREADS + DR_COLS));
}

template <int R>
__global__ void __launch_bounds__(DW_ALL)
delta_scan_wide_kernel(const float* __restrict__ prep, int ldp, const float* __restrict__ v, int ldv,
                       float* __restrict__ state, const int* __restrict__ slots, const int* __restrict__ cu,
                       float* __restrict__ o, int n_heads, int kv_heads, int dk, int dv, int bufs) {
    constexpr int E = 4 * R, LANE = E + 4, ROW = 8 * LANE;
    constexpr int BUF = DL_CHUNK * (3 * ROW + DR_COLS + 4), PART = DL_CHUNK * DW_THREADS;
    mv_pdl_wait();                          // the successor is let go when the last token is done
    extern __shared__ __align__(16) float dl_smem[];    // bufs x [q | k | g: 16 x ROW; v: 16 x 16; beta: 16 (64)], as many parts and u
    float* parts = dl_smem + bufs * BUF;    // [16 tokens][16 columns][8 lanes]
    float* us = parts + bufs * PART;        // [16 tokens][16 columns]
    const int odd = bufs - 1;               // (one buffer: no sequence has a second chunk)
    const int tile = blockIdx.x, h = blockIdx.y, sq = blockIdx.z;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int col0 = tile * DR_COLS;
    const int row0 = cu[sq], len = cu[sq + 1] - row0;
    if (len <= 0) return;
    const int hk = h / (n_heads / kv_heads), qk = kv_heads * ROW, hw = n_heads * ROW;
    const int n_chunks = (len + DL_CHUNK - 1) / DL_CHUNK;

    if (warp == DW_THREADS / 32) {          // copies: the rows of q, k and g, DR_COLS columns of v, and beta of 16 tokens
        const float* qp = prep + (size_t)row0 * ldp + (size_t)hk * ROW + lane * 4;
        const size_t to_g = 2 * (size_t)qk + (size_t)(h - hk) * ROW;
        auto load = [&](int c) {
            const int nt = min(DL_CHUNK, len - c * DL_CHUNK);
            float* buf = dl_smem + (c & odd) * BUF;
            for (int t = 0; t < nt; ++t) {
                const float* src = qp + (size_t)(c * DL_CHUNK + t) * ldp;
                float* to = buf + t * ROW + lane * 4;
#pragma unroll
                for (int i = 0; i < ROW; i += 128)
                    if (i + 128 <= ROW || i + lane * 4 < ROW) {
                        dl_copy16(to + i, src + i);
                        dl_copy16(to + DL_CHUNK * ROW + i, src + qk + i);
                        dl_copy16(to + 2 * DL_CHUNK * ROW + i, src + to_g + i);
                    }
            }
            float* vs = buf + 3 * DL_CHUNK * ROW;
            for (int idx = lane; idx < nt * DR_COLS; idx += 32) {
                const int t = idx / DR_COLS, x = idx % DR_COLS;
                if (col0 + x < dv) dl_copy4(vs + idx, v + (size_t)(row0 + c * DL_CHUNK + t) * ldv + (size_t)h * dv + col0 + x);
            }
            if (lane < nt) dl_copy4(vs + DL_CHUNK * DR_COLS + lane, prep + (size_t)(row0 + c * DL_CHUNK + lane) * ldp + 2 * qk + hw + h);
            dl_commit();
        };
        load(0);
        dl_wait<0>();
        __syncthreads();
        for (int c = 0; c < n_chunks; ++c) {
            if (c + 1 < n_chunks) load(c + 1);
            dl_wait<0>();
            __syncthreads();
        }
        return;
    }
    if (warp > DW_THREADS / 32) {           // outputs of the chunk before
        auto write = [&](int c) {
            const int nt = min(DL_CHUNK, len - c * DL_CHUNK);
            const float *p = parts + (c & odd) * PART, *u = us + (c & odd) * DL_CHUNK * DR_COLS;
#pragma unroll 4
            for (int e = 0; e < DL_CHUNK * DR_COLS / 32; ++e) {
                const int idx = lane + 32 * e, t = idx / DR_COLS, x = idx % DR_COLS;
                if (t >= nt || col0 + x >= dv) continue;
                const size_t row = (size_t)(row0 + c * DL_CHUNK + t);
                const float kq = prep[row * ldp + 2 * qk + hw + n_heads + hk];
                const float4 y = *reinterpret_cast<const float4*>(p + idx * 8), z = *reinterpret_cast<const float4*>(p + idx * 8 + 4);
                const float out = ((y.x + z.x) + (y.z + z.z)) + ((y.y + z.y) + (y.w + z.w));     // as exchanges 4, 2 and 1 lanes apart
                o[row * n_heads * dv + (size_t)h * dv + col0 + x] = fmaf(u[idx], kq, out);
            }
        };
        __syncthreads();
        for (int c = 0; c < n_chunks; ++c) {
            if (c > 0) write(c - 1);
            __syncthreads();
        }
        write(n_chunks - 1);
        return;
    }

    const int l = tid & 7, jl = tid >> 3, j = col0 + jl;
    const int slot = mv_read_slot(slots[sq]);
    float* srow = state + (((size_t)slot * n_heads + h) * dv + (j < dv ? j : 0)) * dk;
    float S[R][4];                          // channel l + 8 c + 32 r
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int i = l + 8 * c + 32 * r;
            S[r][c] = (j < dv && i < dk) ? srow[i] : 0.f;
        }
    struct Token { float q[R][4], g[R][4], k[R][4], v, beta; };
    auto read = [&](const float* from, float (&x)[R][4]) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float4 y = *reinterpret_cast<const float4*>(from + 4 * r);
            x[r][0] = y.x; x[r][1] = y.y; x[r][2] = y.z; x[r][3] = y.w;
        }
    };
    __syncthreads();
    for (int chunk = 0; chunk < n_chunks; ++chunk) {
        const int nt = min(DL_CHUNK, len - chunk * DL_CHUNK);
        const float* buf = dl_smem + (chunk & odd) * BUF;
        const float* qs = buf + l * LANE;
        const float* ks = qs + DL_CHUNK * ROW;
        const float* gs = ks + DL_CHUNK * ROW;
        const float* vs = buf + 3 * DL_CHUNK * ROW + jl;
        const float* bs = buf + 3 * DL_CHUNK * ROW + DL_CHUNK * DR_COLS;
        float* p = parts + (chunk & odd) * PART + tid;
        float* up = us + (chunk & odd) * DL_CHUNK * DR_COLS + jl;
        auto token = [&](int t, const Token& x, Token& next) {
            float a[4] = {0.f, 0.f, 0.f, 0.f}, b[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    S[r][c] *= x.g[r][c];
                    a[c] = fmaf(S[r][c], x.k[r][c], a[c]);
                }
            const int n = t + 1 < nt ? t + 1 : t;           // (behind the last token: its own rows again)
            float said = (a[0] + a[2]) + (a[1] + a[3]);
            said += __shfl_xor_sync(0xffffffffu, said, 4);
            read(gs + n * ROW, next.g);
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) b[c] = fmaf(S[r][c], x.q[r][c], b[c]);
            said += __shfl_xor_sync(0xffffffffu, said, 2);
            read(ks + n * ROW, next.k);
            p[t * DW_THREADS] = (b[0] + b[2]) + (b[1] + b[3]);
            said += __shfl_xor_sync(0xffffffffu, said, 1);
            read(qs + n * ROW, next.q);
            next.v = vs[n * DR_COLS];
            next.beta = bs[n];
            const float u = x.beta * ((j < dv ? x.v : 0.f) - said);
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) S[r][c] = fmaf(x.k[r][c], u, S[r][c]);
            if (l == 0) up[t * DR_COLS] = u;
        };
        Token x0, x1;
        read(gs, x0.g);
        read(ks, x0.k);
        read(qs, x0.q);
        x0.v = vs[0];
        x0.beta = bs[0];
        int t = 0;
        for (; t + 1 < nt; t += 2) {
            token(t, x0, x1);
            token(t + 1, x1, x0);
        }
        if (t < nt) token(t, x0, x1);
        __syncthreads();
    }
    mv_pdl_launch_dependents();
    if (j < dv && mv_slot_ok(slots[sq])) {
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int i = l + 8 * c + 32 * r;
                if (i < dk) srow[i] = S[r][c];
            }
    }
}

// Row width of `prep` for these sizes (a multiple of 4 floats, so that rows start on 16 bytes).
static inline int dl_rounds(int dk) { return dk < 64 ? 0 : dk == 64 ? 2 : dk <= 128 ? 4 : dk <= 192 ? 6 : 8; }
static inline int dl_width(int dk) { return dk < 64 ? dk : 8 * (4 * dl_rounds(dk) + 4); }
MV_API int mv_delta_prep_width(int n_heads, int kv_heads, int dk) {
    const int w = (2 * kv_heads + n_heads) * dl_width(dk) + n_heads + kv_heads;
    return (w + 3) & ~3;
}

// As mv_delta_scan, for steps of many tokens a sequence; prep [N, mv_delta_prep_width()] is scratch.
MV_API int mv_delta_scan_long(const float* q, int ldq, const float* k, int ldk, const float* v, int ldv, const float* b,
                              int ldb, const float* a, int lda, const float* dt_bias, const float* a_log, float q_scale,
                              float norm_eps, float* prep, float* state, const int* slots, const int* cu, float* o, int N,
                              int n_seqs, int max_len, int n_heads, int kv_heads, int dk, int dv, int head_decay, cudaStream_t stream) {
    if (n_seqs <= 0 || N <= 0) return 0;
    if (dk < 1 || dk > 256 || dv < 1 || kv_heads < 1 || n_heads % kv_heads) return (int)cudaErrorInvalidValue;
    const int ldp = mv_delta_prep_width(n_heads, kv_heads, dk), W = dl_width(dk), R = dl_rounds(dk);
    mv_launch(delta_prepare_kernel, N, 256, 0, stream, q, ldq, k, ldk, b, ldb, a, lda, dt_bias, a_log, q_scale, norm_eps, prep,
              ldp, n_heads, kv_heads, dk, W, R, head_decay);
    // The walk is launched as an ordinary successor, not a programmatic one.  Started while the preparing kernel's blocks
    // still hold the multiprocessors, its few blocks (one sequence of 16 heads x 128 values: 128) went where room came
    // up first, several to a multiprocessor, and the walk, bound by what ONE multiprocessor issues, took 1.75 times as
    // long as when they are dealt out over an idle device (measured: 1.26 ms against 0.72 for 2,048 tokens).
    const dim3 grid((dv + DR_COLS - 1) / DR_COLS, n_heads, n_seqs);
    if (R && ((uintptr_t)prep & 15)) return (int)cudaErrorInvalidValue;
    const int bufs = max_len > DL_CHUNK ? 2 : 1;
    const size_t smem = R ? dw_smem(R, bufs) : 2 * (size_t)DL_CHUNK * (3 * dk + DR_COLS + 2) * sizeof(float);      // below 48 KB with R 0
    // 16-byte copies: every row of q, k and g of a head starts on 16 bytes (ldp is a multiple of 4 floats)
    const int wide = dk % 4 == 0 && (((uintptr_t)prep) & 15) == 0;
#define DL_LAUNCH(R)                                                                                                     \
    delta_scan_long_kernel<R><<<grid, DR_COLS * DR_PART, smem, stream>>>((const float*)prep, ldp, v, ldv, state, slots, cu, o,  \
                                                                         n_heads, kv_heads, dk, dv, wide)
#define DW_LAUNCH(R)                                                                                                     \
    do {                                                                                                                 \
        const cudaError_t e = mv_allow_smem<delta_scan_wide_kernel<R>>(dw_smem(R, 2));                                  \
        if (e != cudaSuccess) return (int)e;                                                                             \
        delta_scan_wide_kernel<R><<<grid, DW_ALL, smem, stream>>>((const float*)prep, ldp, v, ldv, state, slots, cu, o,  \
                                                                  n_heads, kv_heads, dk, dv, bufs);                      \
    } while (0)
    if (dk <= 32) DL_LAUNCH(4);
    else if (dk < 64) DL_LAUNCH(8);
    else if (R == 2) DW_LAUNCH(2);
    else if (R == 4) DW_LAUNCH(4);
    else if (R == 6) DW_LAUNCH(6);
    else DW_LAUNCH(8);
#undef DW_LAUNCH
#undef DL_LAUNCH
    return mv_launch_status();
}
