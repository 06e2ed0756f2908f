// Linear attention with a decaying matrix state, one head at a time:
//
//     S_t = diag(a_t) S_(t-1) + k_t v_t^T        (S: dk x dv, a_t: a factor per key channel)
//     o_t = S_t^T q_t
//
// The state lives in 32-bit floats per sequence slot and is carried from step to step; a step
// brings any number of next tokens for each of its sequences.  Everything here is 32-bit: the
// decay, the state, the sums.  Two ways to say the decay cover the designs in use:
//   * per token and key channel from logits z: a = sigmoid(z)^(1/tau) = exp(log_sigmoid(z) / tau)
//     (gated linear attention), or
//   * one constant per head (lightning attention).
// q, k and v come as 32-bit rows of a projection (any row stride, any column offset); an
// activation (none or silu) and a factor on q are applied as they are read.
//
// Work: a block is (16 value columns, head, sequence) and walks the sequence's tokens in order.
// A value column is owned by 8 lanes, lane p holding the state's rows p, p+8, p+16, ... of that
// column in registers; the state is stored [slot][head][dv][dk], so these 8 lanes read 32
// contiguous bytes.  Tokens come through shared memory eight at a time.  The order of every sum
// depends on nothing but dk, so a prompt gives the same numbers however it is cut into steps.
#include "chunked_state.cuh"

#define DS_COLS 16
#define DS_PART 8
#define DS_CHUNK 8

__device__ __forceinline__ float ds_silu(float x) { return x / (1.0f + expf(-x)); }
// log(sigmoid(z)) without overflow: min(z, 0) - log1p(exp(-|z|))
__device__ __forceinline__ float ds_log_sigmoid(float z) { return fminf(z, 0.f) - log1pf(expf(-fabsf(z))); }

template <int R>
__global__ void __launch_bounds__(DS_COLS * DS_PART)
decay_scan_kernel(const float* __restrict__ q, int ldq, const float* __restrict__ k, int ldk,
                  const float* __restrict__ v, int ldv, const float* __restrict__ z, int ldz,
                  const float* __restrict__ head_decay, float inv_tau, float q_scale, int act,
                  float* __restrict__ state, const int* __restrict__ slots, const int* __restrict__ cu,
                  float* __restrict__ o, int n_heads, int dk, int dv) {
    mv_pdl_begin();
    extern __shared__ float smem[];
    float* qs = smem;                           // [DS_CHUNK][dk]
    float* ks = qs + DS_CHUNK * dk;
    float* as = ks + DS_CHUNK * dk;
    float* vs = as + DS_CHUNK * dk;             // [DS_CHUNK][DS_COLS]
    const int tile = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
    const int tid = threadIdx.x, p = tid & (DS_PART - 1), jl = tid >> 3;
    const int j = tile * DS_COLS + jl;
    const int row0 = cu[b], len = cu[b + 1] - row0;
    if (len <= 0) return;
    const int slot = mv_read_slot(slots[b]);
    float* srow = state + (((size_t)slot * n_heads + h) * dv + (j < dv ? j : 0)) * dk;
    float S[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = p + DS_PART * r;
        S[r] = (j < dv && i < dk) ? srow[i] : 0.f;
    }
    const float hd = head_decay ? head_decay[h] : 1.f;
    for (int c0 = 0; c0 < len; c0 += DS_CHUNK) {
        const int nt = min(DS_CHUNK, len - c0);
        __syncthreads();
        for (int idx = tid; idx < nt * dk; idx += DS_COLS * DS_PART) {
            const int t = idx / dk, i = idx - t * dk;
            const size_t row = (size_t)(row0 + c0 + t);
            float qv = q[row * ldq + (size_t)h * dk + i], kv = k[row * ldk + (size_t)h * dk + i];
            if (act) { qv = ds_silu(qv); kv = ds_silu(kv); }
            qs[t * dk + i] = qv * q_scale;
            ks[t * dk + i] = kv;
            as[t * dk + i] = z ? expf(ds_log_sigmoid(z[row * ldz + (size_t)h * dk + i]) * inv_tau) : hd;
        }
        for (int idx = tid; idx < nt * DS_COLS; idx += DS_COLS * DS_PART) {
            const int t = idx / DS_COLS, c = idx - t * DS_COLS, col = tile * DS_COLS + c;
            float vv = col < dv ? v[(size_t)(row0 + c0 + t) * ldv + (size_t)h * dv + col] : 0.f;
            vs[idx] = act ? ds_silu(vv) : vv;
        }
        __syncthreads();
        for (int t = 0; t < nt; ++t) {
            const float vj = vs[t * DS_COLS + jl];
            const float* qt = qs + t * dk;
            const float* kt = ks + t * dk;
            const float* at = as + t * dk;
            float acc = 0.f;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int i = p + DS_PART * r;
                if (i < dk) {
                    S[r] = fmaf(at[i], S[r], kt[i] * vj);
                    acc = fmaf(S[r], qt[i], acc);
                }
            }
            acc += __shfl_xor_sync(0xffffffffu, acc, 1);
            acc += __shfl_xor_sync(0xffffffffu, acc, 2);
            acc += __shfl_xor_sync(0xffffffffu, acc, 4);
            if (p == 0 && j < dv) o[(size_t)(row0 + c0 + t) * n_heads * dv + (size_t)h * dv + j] = acc;
        }
    }
    if (j < dv && mv_slot_ok(slots[b])) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int i = p + DS_PART * r;
            if (i < dk) srow[i] = S[r];
        }
    }
}

MV_GUARD_SETTER(decay_scan)

// q, k [N, >= n_heads * dk], v [N, >= n_heads * dv] with row strides ldq, ldk, ldv (elements);
// z: decay logits [N, >= n_heads * dk] with stride ldz, or null, then head_decay [n_heads];
// state [slots][n_heads][dv][dk]; slots [n_seqs]; cu [n_seqs + 1]; o [N, n_heads * dv] dense.
MV_API int mv_decay_scan(const float* q, int ldq, const float* k, int ldk, const float* v, int ldv,
                         const float* z, int ldz, const float* head_decay, float inv_tau, float q_scale, int act,
                         float* state, const int* slots, const int* cu, float* o, int n_seqs, int n_heads, int dk,
                         int dv, cudaStream_t stream) {
    if (n_seqs <= 0) return 0;
    if (dk < 1 || dk > 256 || dv < 1 || (!z && !head_decay)) return (int)cudaErrorInvalidValue;
    const dim3 grid((dv + DS_COLS - 1) / DS_COLS, n_heads, n_seqs);
    const size_t smem = (size_t)DS_CHUNK * (3 * dk + DS_COLS) * sizeof(float);
    if (dk <= 64)
        mv_launch(decay_scan_kernel<8>, grid, DS_COLS * DS_PART, smem, stream, q, ldq, k, ldk, v, ldv, z, ldz,
                  head_decay, inv_tau, q_scale, act, state, slots, cu, o, n_heads, dk, dv);
    else if (dk <= 128)
        mv_launch(decay_scan_kernel<16>, grid, DS_COLS * DS_PART, smem, stream, q, ldq, k, ldk, v, ldv, z, ldz,
                  head_decay, inv_tau, q_scale, act, state, slots, cu, o, n_heads, dk, dv);
    else
        mv_launch(decay_scan_kernel<32>, grid, DS_COLS * DS_PART, smem, stream, q, ldq, k, ldk, v, ldv, z, ldz,
                  head_decay, inv_tau, q_scale, act, state, slots, cu, o, n_heads, dk, dv);
    return mv_launch_status();
}

// ---------------------------------------------------------------------------------------------
// The same recurrence for steps that bring many tokens a sequence, in chunks of CS_CHUNK tokens (chunked_state.cuh):
// what a token reads from the tokens of its own chunk and what it reads from the state before the
// chunk are separated, so that only the state's hand-over from chunk to chunk is sequential.  With
// c_t the sum of log a over the chunk's tokens up to t (per key channel; all of it <= 0),
//
//     o_t  = sum_i q_t,i e^(c_t,i) S0[i, :]  +  sum_{s <= t} P[t, s] v_s ,
//     P[t, s] = sum_i q_t,i k_s,i e^(c_t,i - c_s,i) ,
//     S_end[i, :] = e^(c_last,i) S0[i, :] + sum_s k_s,i e^(c_last,i - c_s,i) v_s .
//
// Every exponent is a difference of cumulative logarithms taken the right way round, so every factor
// lies in (0, 1]: nothing overflows however small a decay is.  All of it is float32 on the CUDA cores.
// With one constant decay a head the chunks take the path with one decay for all channels; with a decay a channel
// the kernel below prepares, per (sequence, head, chunk), the decayed q and k, the chunk's total decay and P.  The factors
// e^(c_t - c_s) of P are products of the tokens' own decays: a warp takes eight s and walks t, multiplying the eight
// rows k_s e^(c_t - c_s) that its lanes hold by the next token's decay; the eight sums over the lanes are folded.  A row meets up
// to 63 decays, and a decay near 1 in 32 bits is off by up to 2^-25 of what it takes away from a row that hardly decays: from 1/2
// on it is held as a - 1 to full relative precision and the row becomes fma(p, a - 1, p), rounded once a step and nowhere else
// (64 tokens with decays about 1 - 2^-13: 4.2e-7 off the 64-bit outputs with plain factors, 1.9e-7 so; with an exponential for every
// difference of sums, as in the kernels for few tokens, 2.1e-7).
// 2,048 tokens of 8 heads of 128 x 256 with a decay a channel: 52 us this kernel (43 with plain factors), 59 the walk, 48 the outputs, where preparing
// with an exponential for every t, s and channel and walking 32 tokens and 16 columns at a time took 64 and 243; of 16 heads
// of 128 x 128 with a constant decay and the activation: 20 + 3 + 23 + 65 + 55 us against 64 and 243.

#define DC_THREADS 256

// The activation before anything else: rows of q, k and v into dense copies.
__global__ void __launch_bounds__(256)
decay_activate_kernel(const float* __restrict__ q, int ldq, const float* __restrict__ k, int ldk, const float* __restrict__ v,
                      int ldv, float* __restrict__ qa, float* __restrict__ ka, float* __restrict__ va, int wk, int wv) {
    mv_pdl_begin();
    const size_t n = blockIdx.x;
    const int which = blockIdx.y, w = which < 2 ? wk : wv;
    const float* from = which == 0 ? q + n * ldq : which == 1 ? k + n * ldk : v + n * ldv;
    float* to = which == 0 ? qa + n * wk : which == 1 ? ka + n * wk : va + n * wv;
    if (((uintptr_t)from | (uintptr_t)to) % 16 == 0 && w % 4 == 0) {
#pragma unroll 2
        for (int i = threadIdx.x; i < w / 4; i += 256) {
            const float4 x = reinterpret_cast<const float4*>(from)[i];
            reinterpret_cast<float4*>(to)[i] = make_float4(ds_silu(x.x), ds_silu(x.y), ds_silu(x.z), ds_silu(x.w));
        }
    } else {
        for (int i = threadIdx.x; i < w; i += 256) to[i] = ds_silu(from[i]);
    }
}

// NC channels a lane: dk <= 32 NC.
template <int NC>
__global__ void __launch_bounds__(DC_THREADS)
decay_chunk_prepare_kernel(const float* __restrict__ q, int ldq, const float* __restrict__ k, int ldk,
                           const float* __restrict__ z, int ldz, float inv_tau, float q_scale, const int* __restrict__ cu,
                           float* __restrict__ qd, float* __restrict__ kd, float* __restrict__ ed, float* __restrict__ P,
                           int n_heads, int dk) {
    constexpr int W = 32 * NC;
    extern __shared__ __align__(16) float smem[];
    float* qs = smem;                               // [CS_CHUNK][W] scaled q, zero beyond the tokens and channels
    float* as = qs + CS_CHUNK * W;                  // the decays' logarithms, then the decays: a - 1 (its sign set) from 1/2 on, else a
    float* cs = as + CS_CHUNK * W;                  // running sums of the logarithms
    mv_pdl_begin();
    const int c = blockIdx.x, h = blockIdx.y, b = blockIdx.z, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row0 = cu[b], len = cu[b + 1] - row0;
    if (c * CS_CHUNK >= len) return;
    const int nt = min(CS_CHUNK, len - c * CS_CHUNK), chunk = row0 / CS_CHUNK + b + c;
    const size_t first = (size_t)row0 + c * CS_CHUNK;
    const int width = n_heads * dk;
    // (counted loops: eight requests are on their way at a time)
#pragma unroll 8
    for (int e = 0; e < CS_CHUNK * W / DC_THREADS; ++e) {
        const int idx = tid + e * DC_THREADS, t = idx / W, i = idx % W;
        const bool in = i < dk && t < nt;
        qs[idx] = in ? q[(first + t) * ldq + (size_t)h * dk + i] * q_scale : 0.f;
        as[idx] = in ? ds_log_sigmoid(z[(first + t) * ldz + (size_t)h * dk + i]) * inv_tau : 0.f;
    }
    __syncthreads();
    for (int i = tid; i < W; i += DC_THREADS) {
        float run = 0.f;
#pragma unroll 8
        for (int t = 0; t < nt; ++t) {
            run += as[t * W + i];
            cs[t * W + i] = run;
        }
        if (i < dk) ed[(size_t)chunk * width + (size_t)h * dk + i] = expf(run);
    }
    __syncthreads();
#pragma unroll 8
    for (int e = 0; e < CS_CHUNK * W / DC_THREADS; ++e) {
        const int idx = tid + e * DC_THREADS, t = idx / W, i = idx % W;
        if (i < dk && t < nt) qd[(first + t) * width + (size_t)h * dk + i] = qs[idx] * expf(cs[idx]);
    }
    __syncthreads();
    // the sums from the chunk's end: no difference of two large ones
    for (int i = tid; i < W; i += DC_THREADS) {
        float run = 0.f;
#pragma unroll 8
        for (int t = nt - 1; t >= 0; --t) {
            cs[t * W + i] = run;
            run += as[t * W + i];
        }
    }
    __syncthreads();
#pragma unroll 8
    for (int e = 0; e < CS_CHUNK * W / DC_THREADS; ++e) {
        const int idx = tid + e * DC_THREADS, t = idx / W, i = idx % W;
        const float l = as[idx];
        as[idx] = l >= -0.6931f ? -fabsf(expm1f(l)) : expf(l);
        if (i < dk && t < nt) kd[(first + t) * width + (size_t)h * dk + i] = k[(first + t) * ldk + (size_t)h * dk + i] * expf(cs[idx]);
    }
    __syncthreads();
    // warps w and w + 4 share a scheduler: the blocks of eight s are dealt out so that both together have 72 steps
    const int s0 = (warp < 4 ? warp : 11 - warp) * 8;
    float* Pc = P + ((size_t)chunk * n_heads + h) * CS_CHUNK * CS_CHUNK;
    float p[8][NC], own[8][NC];                     // k_s e^(c_t - c_s) of the eight s; k_s itself
#pragma unroll
    for (int s = 0; s < 8; ++s)
#pragma unroll
        for (int x = 0; x < NC; ++x) {
            const int i = x / 4 * 128 + lane * 4 + x % 4;
            p[s][x] = 0.f;
            own[s][x] = i < dk && s0 + s < nt ? k[(first + s0 + s) * ldk + (size_t)h * dk + i] : 0.f;
        }
    for (int t = s0; t < nt; ++t) {
        float qt[NC], at[NC], sum[8];
#pragma unroll
        for (int x = 0; x < NC; x += 4) {
            // channels 4 lane .. 4 lane + 3 (and 128 further on)
            const float4 q4 = *reinterpret_cast<const float4*>(qs + t * W + x * 32 + lane * 4);
            const float4 a4 = *reinterpret_cast<const float4*>(as + t * W + x * 32 + lane * 4);
            qt[x] = q4.x; qt[x + 1] = q4.y; qt[x + 2] = q4.z; qt[x + 3] = q4.w;
            at[x] = a4.x; at[x + 1] = a4.y; at[x + 2] = a4.z; at[x + 3] = a4.w;
        }
        int weak = -1;
#pragma unroll
        for (int x = 0; x < NC; ++x) weak &= __float_as_int(at[x]);
        if (__all_sync(0xffffffffu, weak < 0)) {
#pragma unroll
            for (int s = 0; s < 8; ++s)
#pragma unroll
                for (int x = 0; x < NC; ++x) p[s][x] = fmaf(p[s][x], at[x], p[s][x]);
        } else {
#pragma unroll
            for (int x = 0; x < NC; ++x) {
                const int keep = __float_as_int(at[x]) >> 31;
#pragma unroll
                for (int s = 0; s < 8; ++s) p[s][x] = fmaf(p[s][x], at[x], __int_as_float(__float_as_int(p[s][x]) & keep));
            }
        }
        if (t - s0 < 8) {                           // token t's own row begins
#pragma unroll
            for (int s = 0; s < 8; ++s)
#pragma unroll
                for (int x = 0; x < NC; ++x) p[s][x] = s == t - s0 ? own[s][x] : p[s][x];
        }
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            sum[s] = 0.f;
#pragma unroll
            for (int x = 0; x < NC; ++x) sum[s] = fmaf(qt[x], p[s][x], sum[s]);
        }
        // eight sums over 32 lanes: halves change hands until a lane has one, then its four lanes add up
        int bit = 16;
#pragma unroll
        for (int n = 4; n >= 1; n /= 2) {
            const bool high = lane & bit;
#pragma unroll
            for (int i = 0; i < n; ++i) {
                const float send = high ? sum[i] : sum[n + i], keep = high ? sum[n + i] : sum[i];
                sum[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
            }
            bit >>= 1;
        }
        sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], 2);
        sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], 1);
        if ((lane & 3) == 0) Pc[t * CS_CHUNK + s0 + (lane >> 2)] = sum[0];
    }
}

template <int NC>
static int decay_prepare_launch(const float* q, int ldq, const float* k, int ldk, const float* z, int ldz, float inv_tau,
                                float q_scale, const int* cu, float* qd, float* kd, float* ed, float* P, int n_seqs, int max_len,
                                int n_heads, int dk, cudaStream_t stream) {
    constexpr size_t smem = sizeof(float) * 3 * CS_CHUNK * 32 * NC;
    const cudaError_t attr = mv_allow_smem<decay_chunk_prepare_kernel<NC>>(smem);
    if (attr != cudaSuccess) return (int)attr;
    mv_launch(decay_chunk_prepare_kernel<NC>, dim3((max_len + CS_CHUNK - 1) / CS_CHUNK, n_heads, n_seqs), DC_THREADS, smem, stream,
              q, ldq, k, ldk, z, ldz, inv_tau, q_scale, cu, qd, kd, ed, P, n_heads, dk);
    return mv_launch_status();
}

// How many chunks the scratch of a step of N tokens in n_seqs sequences must hold.
MV_API int mv_decay_chunks(int N, int n_seqs) { return N / CS_CHUNK + n_seqs + 1; }
// And how many floats a chunk its factors take.
MV_API int mv_decay_factor_floats(int n_heads) { return cs_factor_floats(n_heads); }

// Arguments as mv_decay_scan, plus the step's tokens N, the longest sequence's (max_len) and scratch with chunks =
// mv_decay_chunks(N, n_seqs): copies [N, n_heads * (2 dk + dv)] (with act), qd, kd [N, n_heads * dk] and ed
// [chunks, n_heads * dk] (with z), P [chunks, n_heads, CS_CHUNK, CS_CHUNK], before [room (+ 2 where room < chunks), n_heads, dv, dk rounded up to 4]
// for windows of `room` chunks, factors [chunks, mv_decay_factor_floats(n_heads)] (without z).
MV_API int mv_decay_scan_chunked(const float* q, int ldq, const float* k, int ldk, const float* v, int ldv,
                                 const float* z, int ldz, const float* head_decay, float inv_tau, float q_scale, int act,
                                 float* state, const int* slots, const int* cu, float* o, float* copies, float* qd, float* kd,
                                 float* ed, float* P, float* before, float* factors, int room, int chunks, int N, int n_seqs, int max_len, int n_heads, int dk, int dv,
                                 cudaStream_t stream) {
    if (n_seqs <= 0 || max_len <= 0) return 0;
    if (dk < 1 || dk > 256 || dv < 1 || (!z && !head_decay) || (act && !copies) || (!z && !factors)) return (int)cudaErrorInvalidValue;
    const int wk = n_heads * dk, wv = n_heads * dv;
    CsArgs a = {};
    a.q = q; a.ldq = ldq; a.k = k; a.ldk = ldk; a.v = v; a.ldv = ldv;
    a.q_scale = q_scale; a.head_decay = head_decay;
    a.state = state; a.before = before; a.slots = slots; a.cu = cu; a.o = o;
    a.n_heads = n_heads; a.dk = dk; a.dv = dv; a.room = room;
    if (act) {
        float *qa = copies, *ka = qa + (size_t)N * wk, *va = ka + (size_t)N * wk;
        mv_launch(decay_activate_kernel, dim3(N, 3), 256, 0, stream, q, ldq, k, ldk, v, ldv, qa, ka, va, wk, wv);
        const int code = mv_launch_status();
        if (code) return code;
        a.q = qa; a.k = ka; a.v = va;
        a.ldq = a.ldk = wk; a.ldv = wv;
    }
    if (!z) return cs_launch<false>(a, P, factors, chunks, n_seqs, max_len, stream);
    const int code = dk <= 128 ? decay_prepare_launch<4>(a.q, a.ldq, a.k, a.ldk, z, ldz, inv_tau, q_scale, cu, qd, kd, ed, P, n_seqs,
                                                         max_len, n_heads, dk, stream)
                               : decay_prepare_launch<8>(a.q, a.ldq, a.k, a.ldk, z, ldz, inv_tau, q_scale, cu, qd, kd, ed, P, n_seqs,
                                                         max_len, n_heads, dk, stream);
    if (code) return code;
    a.q = qd; a.k = kd; a.ed = ed; a.P = P;
    a.ldq = a.ldk = wk;
    return cs_launch<true>(a, nullptr, nullptr, chunks, n_seqs, max_len, stream);
}

// ---------------------------------------------------------------------------------------------
// Chunks for steps of few tokens (the wrapper's scan_takes_few): the same sums with 32 tokens a chunk in two launches.
// The first kernel prepares, per (sequence, head, chunk), the decayed q and k, the chunk's total decay and P; the second walks a
// sequence's chunks with the state in registers and works the outputs out on the way.  Such a step is bound by its launches and by
// a handful of chunks one after the other: one sequence of 16 tokens 41 us (8 heads of 128 x 256, a decay a channel) and 35 (16 heads
// of 128 x 128, one a head, with the activation) against 57 and 58 with the three to five kernels above; 256 tokens 74 and 67 against 84 and
// 74; four sequences of 96 84 and 81 against 86 and 87, of 128 96 and 93 against 86 and 80.
//
// Chunks are numbered floor(cu[b] / DF_CHUNK) + b + c for chunk c of the step's sequence b: distinct
// numbers below N / DF_CHUNK + n_seqs + 1 that need nothing from the host.
#define DF_CHUNK 32
#define DF_COLS 16
#define DF_THREADS 256            // the preparing kernel
#define DF_SCAN_THREADS 512       // the scanning kernel: 32 half-warps
#define DF_GROUPS (DF_SCAN_THREADS / 16)
// a group's shares of a chunk's outputs, padded by half a row of banks: the two groups of a warp then store into
// different banks
#define DF_RED_STRIDE (DF_CHUNK * DF_COLS + 16)

__global__ void __launch_bounds__(DF_THREADS)
decay_few_prepare_kernel(const float* __restrict__ q, int ldq, const float* __restrict__ k, int ldk,
                           const float* __restrict__ z, int ldz, const float* __restrict__ head_decay, float inv_tau,
                           float q_scale, int act, const int* __restrict__ cu, float* __restrict__ qd,
                           float* __restrict__ kd, float* __restrict__ ed, float* __restrict__ P, int n_heads, int dk) {
    mv_pdl_begin();
    extern __shared__ float smem[];
    const int lds = dk + 1;                         // odd row stride: rows of different tokens fall into different banks
    float* cs = smem;                               // [DF_CHUNK][lds] cumulative log decay
    float* qa = cs + DF_CHUNK * lds;                // activated, scaled q
    float* ka = qa + DF_CHUNK * lds;                // activated k
    const int c = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
    const int row0 = cu[b], len = cu[b + 1] - row0;
    if (c * DF_CHUNK >= len) return;
    const int nt = min(DF_CHUNK, len - c * DF_CHUNK);
    const int first = row0 + c * DF_CHUNK;
    const int chunk = row0 / DF_CHUNK + b + c;
    const int tid = threadIdx.x;
    // a decay of exactly 0 has no logarithm; e^-80 stands in for it (what is left of the state then lies 35
    // decimal places down)
    const float log_hd = head_decay ? fmaxf(logf(head_decay[h]), -80.f) : 0.f;
    for (int idx = tid; idx < nt * dk; idx += DF_THREADS) {
        const int t = idx / dk, i = idx - t * dk;
        const size_t row = (size_t)(first + t);
        float qv = q[row * ldq + (size_t)h * dk + i], kv = k[row * ldk + (size_t)h * dk + i];
        if (act) { qv = ds_silu(qv); kv = ds_silu(kv); }
        qa[t * lds + i] = qv * q_scale;
        ka[t * lds + i] = kv;
        cs[t * lds + i] = z ? ds_log_sigmoid(z[row * ldz + (size_t)h * dk + i]) * inv_tau : log_hd;
    }
    __syncthreads();
    for (int i = tid; i < dk; i += DF_THREADS) {
        float run = 0.f;
        for (int t = 0; t < nt; ++t) {
            run += cs[t * lds + i];
            cs[t * lds + i] = run;
        }
    }
    __syncthreads();
    const int width = n_heads * dk;
    for (int idx = tid; idx < nt * dk; idx += DF_THREADS) {
        const int t = idx / dk, i = idx - t * dk;
        const size_t at = (size_t)(first + t) * width + (size_t)h * dk + i;
        qd[at] = qa[t * lds + i] * expf(cs[t * lds + i]);
        kd[at] = ka[t * lds + i] * expf(cs[(nt - 1) * lds + i] - cs[t * lds + i]);
    }
    for (int i = tid; i < dk; i += DF_THREADS) ed[(size_t)chunk * width + (size_t)h * dk + i] = expf(cs[(nt - 1) * lds + i]);
    float* Pc = P + ((size_t)chunk * n_heads + h) * DF_CHUNK * DF_CHUNK;
    for (int p = tid; p < DF_CHUNK * DF_CHUNK; p += DF_THREADS) {
        const int t = p / DF_CHUNK, s = p - t * DF_CHUNK;
        float sum = 0.f;
        if (s <= t && t < nt) {
            const float* ct = cs + t * lds;
            const float* cq = cs + s * lds;
            const float* qt = qa + t * lds;
            const float* kt = ka + s * lds;
            if (z) {
                for (int i = 0; i < dk; ++i) sum = fmaf(qt[i] * kt[i], expf(ct[i] - cq[i]), sum);
            } else {
                // one decay for all of the head's channels: its power is a factor of the whole sum
                for (int i = 0; i < dk; ++i) sum = fmaf(qt[i], kt[i], sum);
                sum *= expf(ct[0] - cq[0]);
            }
        }
        Pc[p] = sum;
    }
}

// A block is 16 value columns of one head of one sequence; its 16 warps are 32 half-warps, each holding RH key
// channels of every column in registers (dk <= 32 * RH): lane & 15 is the column, the half-warp the channel group.
template <int RH>
__global__ void __launch_bounds__(DF_SCAN_THREADS)
decay_few_scan_kernel(const float* __restrict__ qd, const float* __restrict__ kd, const float* __restrict__ ed,
                        const float* __restrict__ P, const float* __restrict__ v, int ldv, int act,
                        float* __restrict__ state, const int* __restrict__ slots, const int* __restrict__ cu,
                        float* __restrict__ o, int n_heads, int dk, int dv) {
    mv_pdl_begin();
    constexpr int DKP = DF_GROUPS * RH;
    extern __shared__ __align__(16) float smem[];
    float* qt = smem;                               // [DF_CHUNK][DKP], zero beyond dk
    float* kt = qt + DF_CHUNK * DKP;
    float* vt = kt + DF_CHUNK * DKP;                // [DF_CHUNK][DF_COLS]
    float* pt = vt + DF_CHUNK * DF_COLS;            // [DF_CHUNK][DF_CHUNK]
    float* et = pt + DF_CHUNK * DF_CHUNK;           // [DKP]
    float* red = et + DKP;                          // [DF_GROUPS][DF_RED_STRIDE]: [DF_CHUNK][DF_COLS] a group
    const int tile = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
    const int tid = threadIdx.x, col = tid & 15, grp = tid >> 4;
    const int j = tile * DF_COLS + col;
    const int row0 = cu[b], len = cu[b + 1] - row0;
    if (len <= 0) return;
    const int slot = mv_read_slot(slots[b]);
    const int width = n_heads * dk;
    float* srow = state + (((size_t)slot * n_heads + h) * dv + (j < dv ? j : 0)) * dk;
    float S[RH];
#pragma unroll
    for (int r = 0; r < RH; ++r) {
        const int i = grp * RH + r;
        S[r] = (j < dv && i < dk) ? srow[i] : 0.f;
    }
    const int n_chunks = (len + DF_CHUNK - 1) / DF_CHUNK;
    // A chunk's rows are requested into registers while the chunk before is worked on, and go to shared
    // memory when that one is done: per thread IT values of the decayed q and of the decayed k, 2 of v, 4 of P
    // and at most one of the chunk's total decay.
    constexpr int IT = DF_CHUNK * DKP / DF_SCAN_THREADS;
    static_assert(DF_CHUNK * DF_COLS == DF_SCAN_THREADS && DF_CHUNK * DF_CHUNK % DF_SCAN_THREADS == 0 && DKP <= DF_SCAN_THREADS,
                  "a thread requests one value of v, whole rounds of P and at most one of the total decay");
    float rq[IT], rk[IT], rv[DF_CHUNK * DF_COLS / DF_SCAN_THREADS], rp[DF_CHUNK * DF_CHUNK / DF_SCAN_THREADS], re = 0.f;
    auto request = [&](int c) {
        const int nt = min(DF_CHUNK, len - c * DF_CHUNK);
        const int first = row0 + c * DF_CHUNK;
        const int chunk = row0 / DF_CHUNK + b + c;
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            const int idx = tid + it * DF_SCAN_THREADS, t = idx / DKP, i = idx - t * DKP;
            const bool in = t < nt && i < dk;
            const size_t at = in ? (size_t)(first + t) * width + (size_t)h * dk + i : 0;
            rq[it] = in ? qd[at] : 0.f;
            rk[it] = in ? kd[at] : 0.f;
        }
#pragma unroll
        for (int it = 0; it < DF_CHUNK * DF_COLS / DF_SCAN_THREADS; ++it) {
            const int idx = tid + it * DF_SCAN_THREADS, t = idx / DF_COLS, cc = tile * DF_COLS + (idx - t * DF_COLS);
            const float vv = (t < nt && cc < dv) ? v[(size_t)(first + t) * ldv + (size_t)h * dv + cc] : 0.f;
            rv[it] = act ? ds_silu(vv) : vv;
        }
        const float* Pc = P + ((size_t)chunk * n_heads + h) * DF_CHUNK * DF_CHUNK;
#pragma unroll
        for (int it = 0; it < DF_CHUNK * DF_CHUNK / DF_SCAN_THREADS; ++it) rp[it] = Pc[tid + it * DF_SCAN_THREADS];
        if (tid < DKP) re = tid < dk ? ed[(size_t)chunk * width + (size_t)h * dk + tid] : 0.f;
    };
    request(0);
    for (int c = 0; c < n_chunks; ++c) {
        const int nt = min(DF_CHUNK, len - c * DF_CHUNK);
        const int first = row0 + c * DF_CHUNK;
        __syncthreads();                            // the chunk before is done with shared memory
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            qt[tid + it * DF_SCAN_THREADS] = rq[it];
            kt[tid + it * DF_SCAN_THREADS] = rk[it];
        }
#pragma unroll
        for (int it = 0; it < DF_CHUNK * DF_COLS / DF_SCAN_THREADS; ++it) vt[tid + it * DF_SCAN_THREADS] = rv[it];
#pragma unroll
        for (int it = 0; it < DF_CHUNK * DF_CHUNK / DF_SCAN_THREADS; ++it) pt[tid + it * DF_SCAN_THREADS] = rp[it];
        if (tid < DKP) et[tid] = re;
        __syncthreads();
        if (c + 1 < n_chunks) request(c + 1);
        // what the chunk's tokens read from the state before the chunk: this half-warp's key channels
#pragma unroll 4
        for (int t = 0; t < DF_CHUNK; ++t) {
            const float4* q4 = reinterpret_cast<const float4*>(qt + t * DKP + grp * RH);
            float acc = 0.f;
#pragma unroll
            for (int r = 0; r < RH; r += 4) {
                const float4 x = q4[r >> 2];
                acc = fmaf(x.x, S[r], acc); acc = fmaf(x.y, S[r + 1], acc);
                acc = fmaf(x.z, S[r + 2], acc); acc = fmaf(x.w, S[r + 3], acc);
            }
            red[grp * DF_RED_STRIDE + t * DF_COLS + col] = acc;
        }
        // the state after the chunk
#pragma unroll
        for (int r = 0; r < RH; ++r) S[r] *= et[grp * RH + r];
#pragma unroll 4
        for (int s = 0; s < DF_CHUNK; ++s) {
            const float vj = vt[s * DF_COLS + col];
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
        for (int idx = tid; idx < nt * DF_COLS; idx += DF_SCAN_THREADS) {
            const int t = idx / DF_COLS, cc = idx - t * DF_COLS;
            float sum = 0.f;
#pragma unroll
            for (int g = 0; g < DF_GROUPS; ++g) sum += red[g * DF_RED_STRIDE + t * DF_COLS + cc];
            for (int s = 0; s <= t; ++s) sum = fmaf(pt[t * DF_CHUNK + s], vt[s * DF_COLS + cc], sum);
            if (tile * DF_COLS + cc < dv) o[(size_t)(first + t) * n_heads * dv + (size_t)h * dv + tile * DF_COLS + cc] = sum;
        }
    }
    if (j < dv && mv_slot_ok(slots[b])) {
#pragma unroll
        for (int r = 0; r < RH; ++r) {
            const int i = grp * RH + r;
            if (i < dk) srow[i] = S[r];
        }
    }
}

template <int RH>
static int decay_few_scan_launch(dim3 grid, cudaStream_t stream, const float* qd, const float* kd, const float* ed,
                                   const float* P, const float* v, int ldv, int act, float* state, const int* slots,
                                   const int* cu, float* o, int n_heads, int dk, int dv) {
    const size_t smem = sizeof(float) * ((size_t)2 * DF_CHUNK * DF_GROUPS * RH + DF_CHUNK * DF_COLS + DF_CHUNK * DF_CHUNK +
                                         DF_GROUPS * RH + DF_GROUPS * DF_RED_STRIDE);
    const cudaError_t attr = mv_allow_smem<decay_few_scan_kernel<RH>>(smem);
    if (attr != cudaSuccess) return (int)attr;
    mv_launch(decay_few_scan_kernel<RH>, grid, DF_SCAN_THREADS, smem, stream, qd, kd, ed, P, v, ldv, act, state, slots, cu, o,
              n_heads, dk, dv);
    return mv_launch_status();
}

// Arguments as mv_decay_scan, plus the longest sequence's tokens (max_len) and scratch: qd, kd [N, n_heads * dk],
// ed [chunks, n_heads * dk], P [chunks, n_heads, DF_CHUNK, DF_CHUNK] with chunks = mv_decay_few_chunks(N, n_seqs).
MV_API int mv_decay_few_chunks(int N, int n_seqs) { return N / DF_CHUNK + n_seqs + 1; }

MV_API int mv_decay_scan_few(const float* q, int ldq, const float* k, int ldk, const float* v, int ldv,
                                 const float* z, int ldz, const float* head_decay, float inv_tau, float q_scale, int act,
                                 float* state, const int* slots, const int* cu, float* o, float* qd, float* kd, float* ed,
                                 float* P, int n_seqs, int max_len, int n_heads, int dk, int dv, cudaStream_t stream) {
    if (n_seqs <= 0 || max_len <= 0) return 0;
    if (dk < 1 || dk > 256 || dv < 1 || (!z && !head_decay)) return (int)cudaErrorInvalidValue;
    const size_t smem_a = sizeof(float) * (size_t)3 * DF_CHUNK * (dk + 1);
    const cudaError_t attr = mv_allow_smem<decay_few_prepare_kernel>(sizeof(float) * 3 * DF_CHUNK * 257);     // what the largest dk needs
    if (attr != cudaSuccess) return (int)attr;
    mv_launch(decay_few_prepare_kernel, dim3((max_len + DF_CHUNK - 1) / DF_CHUNK, n_heads, n_seqs), DF_THREADS, smem_a,
              stream, q, ldq, k, ldk, z, ldz, head_decay, inv_tau, q_scale, act, cu, qd, kd, ed, P, n_heads, dk);
    int code = mv_launch_status();
    if (code) return code;
    const dim3 grid((dv + DF_COLS - 1) / DF_COLS, n_heads, n_seqs);
    if (dk <= 128) return decay_few_scan_launch<4>(grid, stream, qd, kd, ed, P, v, ldv, act, state, slots, cu, o, n_heads, dk, dv);
    return decay_few_scan_launch<8>(grid, stream, qd, kd, ed, P, v, ldv, act, state, slots, cu, o, n_heads, dk, dv);
}
