// A decaying matrix state walked in chunks of CS_CHUNK tokens: the kernels of decay_scan.cu for steps of many tokens (scalar_scan.cu uses
// the copies into shared memory).  Per head, with S0 the state before a chunk,
//
//     S_end[j, i] = d_i S0[j, i] + sum_s v_s[j] (w_s k_s[i]),
//     o_t[j]      = f_t sum_i q_t[i] S0[j, i] + sum_{s <= t} P[t, s] v_s[j].
//
// "By head" (CHANNEL false): one decay a head; d_i = e^(c_last), w_s = e^(c_last - c_s), f_t = e^(c_t) q_scale
// with c the running sum of log a over the chunk, and P[t, s] = (q_t . k_s) e^(c_t - c_s) q_scale from the products
// q_t . k_s.  "By channel": q, k, d and P come prepared, w = f = 1.
// cs_walk_kernel has a tile of a head's state in registers, walks the sequence's chunks and leaves the state before every
// chunk; that is all that is sequential.  cs_output_kernel then works on all chunks at once.  Everything is float32 on the CUDA
// cores: both are bound by the multiply-adds and the shared-memory loads that feed them.
//
// Chunks are numbered floor(cu[b] / CS_CHUNK) + b + c for chunk c of the step's sequence b: distinct numbers below
// N / CS_CHUNK + n_seqs + 1, ascending, that need nothing from the host.
//
// The states before all chunks would be as large as the step is long (2 MB for every 32 tokens of 64 heads of 128 x 64), so walk and outputs go
// over the numbers in windows of as many chunks as the caller has room for.  At a window's end at most one sequence is cut: its state
// goes into one of two places behind the window's (in turn: the next window reads it while another sequence's may be left).
#pragma once
#include "common.cuh"

#define CS_CHUNK 64
#define CS_THREADS 128

struct CsArgs {
    const float *q, *k, *v;             // rows of the step's tokens; head h reads the columns h dk, h dk, h dv
    int ldq, ldk, ldv;
    const float* head_decay;            // by head: [n_heads]
    const float* ed;                    // by channel: the chunks' decays [chunk][n_heads * dk]
    const double* c;                    // by head: the running sums of log a [chunk][head][CS_CHUNK]
    const float *w, *d;                 // by head: w_s [chunk][head][CS_CHUNK] and d [chunk][head]
    const float* P;                     // by head: q . k [chunk][head][CS_CHUNK][CS_CHUNK]; by channel: P [chunk][head][..][..]
    float q_scale;
    float *state, *before;              // [slot][head][dv][dk]; [chunk - w0][head][dv][lds]: the state before every chunk
    const int *slots, *cu;
    float* o;                           // [N, n_heads * dv]
    int n_heads, dk, dv, lds, wide;
    int w0, w1, room;                   // this window's chunk numbers; the chunks that `before` holds (and, with more than one window, two states)
};

namespace {

__device__ __forceinline__ void cs_copy(float* to, const float* from, bool in, bool wide) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(to);
    if (wide) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(from), "r"(in ? 16 : 0) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(s), "l"(from), "r"(in ? 4 : 0) : "memory");
}
// The chunks of a sequence that lie in the window: from .first up to .second.
__device__ __forceinline__ int2 cs_window(int chunk0, int n_chunks, int w0, int w1) {
    return make_int2(max(0, w0 - chunk0), min(n_chunks, w1 - chunk0));
}
// Where a sequence that a window's end cuts leaves its state: behind the window's chunks.
__device__ __forceinline__ int cs_carry(int w1, int room) { return room + (w1 / room & 1); }

__device__ __forceinline__ void cs_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cs_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// ROWS x COLS floats from row `row` and column `col` of a matrix on their way into shared memory (row stride LD); what lies
// beyond n_rows or n_cols is zeroed.  `wide`: rows and columns start on 16 bytes and n_cols is a multiple of 4.  PERM: the
// smem row r is the matrix row (r % 16) * 4 + r / 16.
template <int ROWS, int COLS, int LD, bool PERM = false, int THREADS = CS_THREADS>
__device__ __forceinline__ void cs_load(float* to, const float* from, size_t ld, int n_rows, int n_cols, int wide) {
    if (wide) {
#pragma unroll
        for (int e = 0; e < (ROWS * COLS / 4 + THREADS - 1) / THREADS; ++e) {
            const int idx = threadIdx.x + e * THREADS, r = idx / (COLS / 4), c = (idx % (COLS / 4)) * 4;
            if (ROWS * COLS / 4 % THREADS && r >= ROWS) break;
            const int src = PERM ? (r & 15) * 4 + (r >> 4) : r;
            const bool in = src < n_rows && c < n_cols;
            cs_copy(to + r * LD + c, in ? from + src * ld + c : from, in, true);
        }
    } else {
#pragma unroll 4
        for (int idx = threadIdx.x; idx < ROWS * COLS; idx += THREADS) {
            const int r = idx / COLS, c = idx % COLS, src = PERM ? (r & 15) * 4 + (r >> 4) : r;
            const bool in = src < n_rows && c < n_cols;
            cs_copy(to + r * LD + c, in ? from + src * ld + c : from, in, false);
        }
    }
}

// The running sum of a chunk's log decays (lane l of a warp has tokens 2l and 2l + 1); beyond nt the sum stays.  In 64 bits: the
// factors need DIFFERENCES of these sums, which are small beside the sums where a decay is strong (in 32 bits a chunk that
// decays by e^-5000 gives neighbours' factors off by 3e-4).
__device__ __forceinline__ double2 cs_running(float l0, float l1) {
    const int lane = threadIdx.x & 31;
    double run = (double)l0 + (double)l1;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const double up = __shfl_up_sync(0xffffffffu, run, d);
        if (lane >= d) run += up;
    }
    double before = __shfl_up_sync(0xffffffffu, run, 1);
    if (lane == 0) before = 0.0;
    return make_double2(before + l0, run);
}

// What follows from the decays alone, a warp a chunk and head: the running sums, w and d.
__global__ void __launch_bounds__(CS_THREADS)
cs_factors_kernel(const CsArgs a, double* __restrict__ c_out, float* __restrict__ w_out, float* __restrict__ d_out) {
    mv_pdl_begin();
    const int c = blockIdx.x, h = blockIdx.y * (CS_THREADS / 32) + (threadIdx.x >> 5), b = blockIdx.z, lane = threadIdx.x & 31;
    const int row0 = a.cu[b], len = a.cu[b + 1] - row0;
    if (c * CS_CHUNK >= len || h >= a.n_heads) return;
    const int nt = min(CS_CHUNK, len - c * CS_CHUNK);
    const size_t at = (size_t)(row0 / CS_CHUNK + b + c) * a.n_heads + h;
    const bool in0 = 2 * lane < nt, in1 = 2 * lane + 1 < nt;
    // a decay of exactly 0 has no logarithm; e^-80 stands in for it (what is left of the state then lies 35 decimal places down)
    const float log_a = fmaxf(logf(a.head_decay[h]), -80.f);
    const double2 run = cs_running(in0 ? log_a : 0.f, in1 ? log_a : 0.f);
    const double last = __shfl_sync(0xffffffffu, run.y, 31);
    *reinterpret_cast<double2*>(c_out + at * CS_CHUNK + 2 * lane) = run;
    *reinterpret_cast<float2*>(w_out + at * CS_CHUNK + 2 * lane) =
        make_float2(in0 ? expf((float)(last - run.x)) : 0.f, in1 ? expf((float)(last - run.y)) : 0.f);
    if (lane == 0) d_out[at] = expf((float)last);
}

// ---- the walk ------------------------------------------------------------------------------------------------
// A block has a tile of 8 TJ value columns x 64 key channels, a thread TJ x 4 of it; a chunk's tokens come at once, the next
// chunk's on their way.  GROUPS groups of 128 threads have the same tile and every GROUPS-th share of the tokens, each a sum of
// its own that decays like the state; at a chunk's end the sums meet in shared memory (one group alone, one warp a scheduler,
// issued in 0.43 of the cycles; with 16 tokens at a time more than half of the instructions were copies and loop).
template <int TJ, int GROUPS, bool CHANNEL>
__global__ void __launch_bounds__(CS_THREADS * GROUPS)
cs_walk_kernel(const CsArgs a) {
    constexpr int JT = 8 * TJ, SUB = CS_CHUNK, STAGES = 2, SHARE = SUB / GROUPS, THREADS = CS_THREADS * GROUPS;
    extern __shared__ __align__(16) float cw_smem[];
    float* ks = cw_smem;                                // [STAGES][SUB][64]
    float* vs = ks + STAGES * SUB * 64;                 // [STAGES][SUB][JT]
    float* ws = vs + STAGES * SUB * JT;                 // [STAGES][SUB]
    float4* meet = reinterpret_cast<float4*>(ws + STAGES * SUB);    // [GROUPS - 1][TJ][CS_THREADS]
    mv_pdl_begin();
    const int tiles_i = (a.dk + 63) / 64, i0 = (blockIdx.x % tiles_i) * 64, j0 = (blockIdx.x / tiles_i) * JT;
    const int h = blockIdx.y, b = blockIdx.z, tid = threadIdx.x, grp = tid / CS_THREADS, lt = tid % CS_THREADS, ti = lt & 15, tj = lt >> 4;
    const int row0 = a.cu[b], len = a.cu[b + 1] - row0;
    const int n_sub = (len + SUB - 1) / SUB, chunk0 = row0 / CS_CHUNK + b;
    const int2 win = cs_window(chunk0, n_sub, a.w0, a.w1);
    if (win.x >= win.y) return;
    const int slot = mv_read_slot(a.slots[b]);
    const int i = i0 + ti * 4, j = j0 + tj * TJ;
    float* st = a.state + ((size_t)slot * a.n_heads + h) * a.dv * a.dk;
    const bool vec = a.dk % 4 == 0;                     // the state's rows start on 16 bytes
    float S[TJ][4];
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
    for (int y = 0; y < TJ; ++y) {
        if (grp == 0 && j + y < a.dv)
            read4(win.x ? a.before + (((size_t)cs_carry(a.w0, a.room) * a.n_heads + h) * a.dv + j + y) * a.lds : st + (size_t)(j + y) * a.dk, S[y]);
        else
#pragma unroll
            for (int x = 0; x < 4; ++x) S[y][x] = 0.f;
    }
    const float* kp = a.k + (size_t)row0 * a.ldk + (size_t)h * a.dk + i0;
    const float* vp = a.v + (size_t)row0 * a.ldv + (size_t)h * a.dv + j0;
    auto load = [&](int sub) {
        const size_t t = (size_t)sub * SUB;
        if (sub < win.y) {
            const int st = sub % STAGES;
            cs_load<SUB, 64, 64, false, THREADS>(ks + st * SUB * 64, kp + t * a.ldk, a.ldk, len - (int)t, a.dk - i0, a.wide);
            cs_load<SUB, JT, JT, false, THREADS>(vs + st * SUB * JT, vp + t * a.ldv, a.ldv, len - (int)t, a.dv - j0, a.wide);
            if (!CHANNEL && tid < SUB / 4)
                cs_copy(ws + st * SUB + tid * 4, a.w + ((size_t)(chunk0 + t / CS_CHUNK) * a.n_heads + h) * CS_CHUNK + t % CS_CHUNK + tid * 4, true, true);
        }
        cs_commit();
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) load(win.x + s);
    float d_next[4];                                    // the chunk's decay, requested a chunk ahead
    auto decay = [&](int c) {
#pragma unroll
        for (int x = 0; x < 4; ++x)
            d_next[x] = CHANNEL ? (i + x < a.dk ? a.ed[(size_t)(chunk0 + c) * a.n_heads * a.dk + (size_t)h * a.dk + i + x] : 0.f)
                                : a.d[(size_t)(chunk0 + c) * a.n_heads + h];
    };
    decay(win.x);
    // the other groups' sums go into the first group's
    auto join = [&]() {
        if (grp > 0) {
            float4* m = meet + (size_t)(grp - 1) * TJ * CS_THREADS + lt;
#pragma unroll
            for (int y = 0; y < TJ; ++y) {
                m[y * CS_THREADS] = make_float4(S[y][0], S[y][1], S[y][2], S[y][3]);
                S[y][0] = S[y][1] = S[y][2] = S[y][3] = 0.f;
            }
        }
        __syncthreads();
        if (grp == 0) {
#pragma unroll
            for (int q = 0; q < GROUPS - 1; ++q) {
                const float4* m = meet + (size_t)q * TJ * CS_THREADS + lt;
#pragma unroll
                for (int y = 0; y < TJ; ++y) {
                    const float4 r = m[y * CS_THREADS];
                    S[y][0] += r.x; S[y][1] += r.y; S[y][2] += r.z; S[y][3] += r.w;
                }
            }
        }
    };
    auto leave = [&](int place) {
        float* to = a.before + ((size_t)place * a.n_heads + h) * a.dv * a.lds;
        if (grp == 0 && i < a.lds) {
#pragma unroll
            for (int y = 0; y < TJ; ++y)
                if (j + y < a.dv)
                    *reinterpret_cast<float4*>(to + (size_t)(j + y) * a.lds + i) = make_float4(S[y][0], S[y][1], S[y][2], S[y][3]);
        }
    };
    for (int sub = win.x; sub < win.y; ++sub) {
        {
            const int c = sub;
            if (GROUPS > 1 && c > win.x) join();
            leave(chunk0 + c - a.w0);                   // the state as it is before this chunk
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int y = 0; y < TJ; ++y) S[y][x] *= d_next[x];
            if (c + 1 < win.y) decay(c + 1);
        }
        cs_wait<STAGES - 2>();
        __syncthreads();                                // these tokens are there, the ones before are done with
        load(sub + STAGES - 1);
        const float* kt = ks + (sub % STAGES * SUB + grp * SHARE) * 64 + ti * 4;
        const float* vt = vs + (sub % STAGES * SUB + grp * SHARE) * JT + tj * TJ;
        const float* wt = ws + sub % STAGES * SUB + grp * SHARE;
#pragma unroll 2
        for (int s0 = 0; s0 < SHARE; s0 += 4) {
            float4 k[4], v[4][TJ / 4];
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                k[s] = *reinterpret_cast<const float4*>(kt + (s0 + s) * 64);
#pragma unroll
                for (int y = 0; y < TJ / 4; ++y) v[s][y] = *reinterpret_cast<const float4*>(vt + (s0 + s) * JT + 4 * y);
            }
            if (!CHANNEL) {
                const float4 w = *reinterpret_cast<const float4*>(wt + s0);
                k[0].x *= w.x; k[0].y *= w.x; k[0].z *= w.x; k[0].w *= w.x;
                k[1].x *= w.y; k[1].y *= w.y; k[1].z *= w.y; k[1].w *= w.y;
                k[2].x *= w.z; k[2].y *= w.z; k[2].z *= w.z; k[2].w *= w.z;
                k[3].x *= w.w; k[3].y *= w.w; k[3].z *= w.w; k[3].w *= w.w;
            }
#pragma unroll
            for (int s = 0; s < 4; ++s) {
#pragma unroll
                for (int y = 0; y < TJ; ++y) {
                    const float4 v4 = v[s][y / 4];
                    const float vy = y % 4 == 0 ? v4.x : y % 4 == 1 ? v4.y : y % 4 == 2 ? v4.z : v4.w;
                    S[y][0] = fmaf(k[s].x, vy, S[y][0]); S[y][1] = fmaf(k[s].y, vy, S[y][1]);
                    S[y][2] = fmaf(k[s].z, vy, S[y][2]); S[y][3] = fmaf(k[s].w, vy, S[y][3]);
                }
            }
        }
    }
    if (GROUPS > 1) join();
    if (win.y < n_sub) leave(cs_carry(a.w1, a.room));
    else if (grp == 0 && mv_slot_ok(a.slots[b])) {
        auto write4 = [&](float* p, const float* from) {
            if (vec && i < a.dk) *reinterpret_cast<float4*>(p + i) = make_float4(from[0], from[1], from[2], from[3]);
            else
#pragma unroll
                for (int x = 0; x < 4; ++x)
                    if (i + x < a.dk) p[i + x] = from[x];
        };
#pragma unroll
        for (int y = 0; y < TJ; ++y)
            if (j + y < a.dv) write4(st + (size_t)(j + y) * a.dk, S[y]);
    }
}

// ---- the outputs ---------------------------------------------------------------------------------------------
// A block has the outputs of one chunk (64 tokens) in 64 value columns of one head, a thread 8 x 4 of them.  q and the state
// come in slices of 32 key channels, the next slice on its way; rows of 36 floats keep the 16-byte reads of neighbouring rows
// apart in the banks, and the state's rows are laid down so that a thread's four columns lie together in the result.
constexpr int CO_LD = 36, CO_PLD = CS_CHUNK + 4;
constexpr size_t CO_SMEM = sizeof(float) * (2 * 2 * 64 * CO_LD + CS_CHUNK * 64 + 2 * CS_CHUNK);
static_assert(CS_CHUNK * CO_PLD <= 2 * 64 * CO_LD, "P takes one stage's place");

template <bool CHANNEL>
__global__ void __launch_bounds__(CS_THREADS, 4)
cs_output_kernel(const CsArgs a) {
    extern __shared__ __align__(16) float co_smem[];
    constexpr int STAGE = 2 * 64 * CO_LD;               // [64][CO_LD] of q, then of the state
    float* vs = co_smem + 2 * STAGE;                    // [64][64]
    double* cs = reinterpret_cast<double*>(vs + CS_CHUNK * 64);     // [64] running sums of the log decays
    mv_pdl_begin();
    const int tiles_j = (a.dv + 63) / 64, j0 = (blockIdx.x % tiles_j) * 64;
    const int h = blockIdx.y, b = blockIdx.z, tid = threadIdx.x, tj = tid & 15, tt = tid >> 4;
    const int row0 = a.cu[b], len = a.cu[b + 1] - row0, chunk0 = row0 / CS_CHUNK + b;
    const int2 win = cs_window(chunk0, (len + CS_CHUNK - 1) / CS_CHUNK, a.w0, a.w1);
    const int c = win.x + blockIdx.x / tiles_j, chunk = chunk0 + c;
    if (c >= win.y) return;
    const int nt = min(CS_CHUNK, len - c * CS_CHUNK);
    const size_t first = (size_t)row0 + c * CS_CHUNK;
    const float* S0 = a.before + ((size_t)(chunk - a.w0) * a.n_heads + h) * a.dv * a.lds;
    const float* qp = a.q + first * a.ldq + (size_t)h * a.dk;
    const int slices = (a.dk + 31) / 32;
    auto load = [&](int s) {
        cs_load<64, 32, CO_LD>(co_smem + (s & 1) * STAGE, qp + s * 32, a.ldq, nt, a.dk - s * 32, a.wide);
        cs_load<64, 32, CO_LD, true>(co_smem + (s & 1) * STAGE + 64 * CO_LD, S0 + (size_t)j0 * a.lds + s * 32, a.lds, a.dv - j0,
                                     a.lds - s * 32, 1);
        cs_commit();
    };
    load(0);
    cs_load<CS_CHUNK, 64, 64>(vs, a.v + first * a.ldv + (size_t)h * a.dv + j0, a.ldv, nt, a.dv - j0, a.wide);
    cs_commit();
    if (!CHANNEL && tid < CS_CHUNK) cs[tid] = a.c[((size_t)chunk * a.n_heads + h) * CS_CHUNK + tid];    // read after the loop's barriers
    const float* Pc = a.P + ((size_t)chunk * a.n_heads + h) * CS_CHUNK * CS_CHUNK;
    float* ps = co_smem + (slices & 1) * STAGE;         // [64][CO_PLD]: comes behind the last slice, into the stage that is free
    float acc[8][4];
#pragma unroll
    for (int y = 0; y < 8; ++y)
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[y][x] = 0.f;
    for (int s = 0; s < slices; ++s) {
        if (s + 1 < slices) load(s + 1);
        else {
            cs_load<CS_CHUNK, CS_CHUNK, CO_PLD>(ps, Pc, CS_CHUNK, nt, CS_CHUNK, 1);
            cs_commit();
        }
        cs_wait<1>();                                   // the newest group may still be on its way
        __syncthreads();
        const float *q = co_smem + (s & 1) * STAGE + tt * CO_LD, *st = co_smem + (s & 1) * STAGE + (64 + tj) * CO_LD;
#pragma unroll 2
        for (int kk = 0; kk < 32; kk += 4) {
            float4 w[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) w[x] = *reinterpret_cast<const float4*>(st + x * 16 * CO_LD + kk);
#pragma unroll
            for (int y = 0; y < 8; ++y) {
                const float4 u = *reinterpret_cast<const float4*>(q + y * 8 * CO_LD + kk);
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    acc[y][x] = fmaf(u.x, w[x].x, acc[y][x]); acc[y][x] = fmaf(u.y, w[x].y, acc[y][x]);
                    acc[y][x] = fmaf(u.z, w[x].z, acc[y][x]); acc[y][x] = fmaf(u.w, w[x].w, acc[y][x]);
                }
            }
        }
        __syncthreads();
    }
    cs_wait<0>();                                       // P is there
    __syncthreads();
    if (!CHANNEL) {
        // the decays on the products (what lies above the diagonal is not read)
#pragma unroll 4
        for (int idx = tid; idx < CS_CHUNK * CS_CHUNK / 4; idx += CS_THREADS) {
            const int t = idx / (CS_CHUNK / 4), s = idx % (CS_CHUNK / 4) * 4;
            if (s > t || t >= nt) continue;
            float4 p = *reinterpret_cast<const float4*>(ps + t * CO_PLD + s);
            const double ct = cs[t];
            p.x *= expf((float)(ct - cs[s])) * a.q_scale;
            p.y *= s + 1 <= t ? expf((float)(ct - cs[s + 1])) * a.q_scale : 0.f;
            p.z *= s + 2 <= t ? expf((float)(ct - cs[s + 2])) * a.q_scale : 0.f;
            p.w *= s + 3 <= t ? expf((float)(ct - cs[s + 3])) * a.q_scale : 0.f;
            *reinterpret_cast<float4*>(ps + t * CO_PLD + s) = p;
        }
#pragma unroll
        for (int y = 0; y < 8; ++y) {
            const float f = expf((float)cs[tt + 8 * y]) * a.q_scale;
#pragma unroll
            for (int x = 0; x < 4; ++x) acc[y][x] *= f;
        }
    }
    if (!CHANNEL) __syncthreads();
    // what the chunk's tokens read from one another
    // (tokens 8 sb .. 8 sb + 7 for the rows from 8 sb on; a later token's value, which may not be finite, never meets an earlier row)
    // (short loops: unrolled whole, a third of the time went to fetching instructions)
    const int n_sb = (nt + 7) / 8;
#pragma unroll 1
    for (int s = 0; s < n_sb * 8; s += 4) {
        const int sb = s >> 3, ds = s & 7;
        float4 w[4];
#pragma unroll
        for (int z = 0; z < 4; ++z) w[z] = *reinterpret_cast<const float4*>(vs + (s + z) * 64 + tj * 4);
#pragma unroll
        for (int y = 0; y < 8; ++y) {
            if (y < sb) continue;
            const float4 u = *reinterpret_cast<const float4*>(ps + (tt + 8 * y) * CO_PLD + s);
            const float uz[4] = {u.x, u.y, u.z, u.w};
            if (y > sb) {
#pragma unroll
                for (int z = 0; z < 4; ++z) {
                    acc[y][0] = fmaf(uz[z], w[z].x, acc[y][0]); acc[y][1] = fmaf(uz[z], w[z].y, acc[y][1]);
                    acc[y][2] = fmaf(uz[z], w[z].z, acc[y][2]); acc[y][3] = fmaf(uz[z], w[z].w, acc[y][3]);
                }
            } else {
#pragma unroll
                for (int z = 0; z < 4; ++z)
                    if (ds + z <= tt) {
                        acc[y][0] = fmaf(uz[z], w[z].x, acc[y][0]); acc[y][1] = fmaf(uz[z], w[z].y, acc[y][1]);
                        acc[y][2] = fmaf(uz[z], w[z].z, acc[y][2]); acc[y][3] = fmaf(uz[z], w[z].w, acc[y][3]);
                    }
            }
        }
    }
    const int j = j0 + tj * 4;
    const bool vec = a.dv % 4 == 0 && j + 3 < a.dv;
#pragma unroll
    for (int y = 0; y < 8; ++y) {
        const int t = tt + 8 * y;
        if (t >= nt) continue;
        float* to = a.o + (first + t) * a.n_heads * a.dv + (size_t)h * a.dv + j;
        if (vec) *reinterpret_cast<float4*>(to) = make_float4(acc[y][0], acc[y][1], acc[y][2], acc[y][3]);
        else
#pragma unroll
            for (int x = 0; x < 4; ++x)
                if (j + x < a.dv) to[x] = acc[y][x];
    }
}

// G[chunk][head][t][s] = q_t . k_s of every chunk (all 64 x 64; what lies beyond a chunk's tokens is zero).
__global__ void __launch_bounds__(CS_THREADS)
cs_products_kernel(const CsArgs a, float* __restrict__ G) {
    __shared__ __align__(16) float qs[2][64 * CO_LD], ks[2][64 * CO_LD];
    mv_pdl_begin();
    const int c = blockIdx.x, g = blockIdx.y, b = blockIdx.z, tid = threadIdx.x, tj = tid & 15, tt = tid >> 4;
    const int row0 = a.cu[b], len = a.cu[b + 1] - row0;
    if (c * CS_CHUNK >= len) return;
    const int nt = min(CS_CHUNK, len - c * CS_CHUNK), slices = (a.dk + 31) / 32;
    const size_t first = (size_t)row0 + c * CS_CHUNK;
    auto load = [&](int s) {
        cs_load<64, 32, CO_LD>(qs[s & 1], a.q + first * a.ldq + (size_t)g * a.dk + s * 32, a.ldq, nt, a.dk - s * 32, a.wide);
        cs_load<64, 32, CO_LD, true>(ks[s & 1], a.k + first * a.ldk + (size_t)g * a.dk + s * 32, a.ldk, nt, a.dk - s * 32, a.wide);
        cs_commit();
    };
    float acc[8][4];
#pragma unroll
    for (int y = 0; y < 8; ++y)
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[y][x] = 0.f;
    load(0);
    for (int s = 0; s < slices; ++s) {
        if (s + 1 < slices) { load(s + 1); cs_wait<1>(); }
        else cs_wait<0>();
        __syncthreads();
        const float *q = qs[s & 1] + tt * CO_LD, *k = ks[s & 1] + tj * CO_LD;
#pragma unroll 2
        for (int kk = 0; kk < 32; kk += 4) {
            float4 w[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) w[x] = *reinterpret_cast<const float4*>(k + x * 16 * CO_LD + kk);
#pragma unroll
            for (int y = 0; y < 8; ++y) {
                const float4 u = *reinterpret_cast<const float4*>(q + y * 8 * CO_LD + kk);
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    acc[y][x] = fmaf(u.x, w[x].x, acc[y][x]); acc[y][x] = fmaf(u.y, w[x].y, acc[y][x]);
                    acc[y][x] = fmaf(u.z, w[x].z, acc[y][x]); acc[y][x] = fmaf(u.w, w[x].w, acc[y][x]);
                }
            }
        }
        __syncthreads();
    }
    float* to = G + ((size_t)(row0 / CS_CHUNK + b + c) * a.n_heads + g) * CS_CHUNK * CS_CHUNK + tj * 4;
#pragma unroll
    for (int y = 0; y < 8; ++y)
        *reinterpret_cast<float4*>(to + (tt + 8 * y) * CS_CHUNK) = make_float4(acc[y][0], acc[y][1], acc[y][2], acc[y][3]);
}

inline bool cs_aligned(const float* p, int ld, int cols) { return ((uintptr_t)p & 15) == 0 && ld % 4 == 0 && cols % 4 == 0; }

// Which tile and how many token groups: two groups where there are more tiles than multiprocessors (two blocks fit on one), four
// where a block is alone on its own, and half the tile where even then multiprocessors are left over (8 heads of 128 x 256: 64
// tiles; 59 us with 128 half tiles of four groups, 104 with one group).
template <int TJ, int GROUPS, bool CHANNEL>
int cs_walk_launch(const CsArgs& a, int tiles, int n_seqs, cudaStream_t stream) {
    constexpr size_t smem = sizeof(float) * (2 * CS_CHUNK * (64 + 8 * TJ + 1) + (GROUPS - 1) * TJ * CS_THREADS * 4);
    const cudaError_t attr = mv_allow_smem<cs_walk_kernel<TJ, GROUPS, CHANNEL>>(smem);
    if (attr != cudaSuccess) return (int)attr;
    mv_launch(cs_walk_kernel<TJ, GROUPS, CHANNEL>, dim3(tiles, a.n_heads, n_seqs), CS_THREADS * GROUPS, smem, stream, a);
    return mv_launch_status();
}

// All kernels; a.wide, a.lds and by head a.P, a.c, a.w and a.d are filled in here.  By head G is scratch for the products
// [chunks][heads][CS_CHUNK][CS_CHUNK] and `factors` (16-byte aligned) for cs_factor_floats(n_heads) floats a chunk.
inline int cs_factor_floats(int n_heads) { return n_heads * (3 * CS_CHUNK + 1); }

template <bool CHANNEL>
int cs_launch(CsArgs a, float* G, float* factors, int chunks, int n_seqs, int max_len, cudaStream_t stream) {
    if (a.room < 1) return (int)cudaErrorInvalidValue;
    a.lds = (a.dk + 3) & ~3;
    a.wide = cs_aligned(a.q, a.ldq, a.dk) && cs_aligned(a.k, a.ldk, a.dk) && cs_aligned(a.v, a.ldv, a.dv);
    if (!CHANNEL) {
        double* c = reinterpret_cast<double*>(factors);
        float* w = factors + (size_t)2 * chunks * a.n_heads * CS_CHUNK;
        float* d = w + (size_t)chunks * a.n_heads * CS_CHUNK;
        a.P = G; a.c = c; a.w = w; a.d = d;
        mv_launch(cs_factors_kernel, dim3((max_len + CS_CHUNK - 1) / CS_CHUNK, (a.n_heads + CS_THREADS / 32 - 1) / (CS_THREADS / 32), n_seqs),
                  CS_THREADS, 0, stream, a, c, w, d);
        int code = mv_launch_status();
        if (code) return code;
        mv_launch(cs_products_kernel, dim3((max_len + CS_CHUNK - 1) / CS_CHUNK, a.n_heads, n_seqs), CS_THREADS, 0,
                  stream, a, G);
        code = mv_launch_status();
        if (code) return code;
    }
    const int tiles_i = (a.dk + 63) / 64;
    const long tiles = (long)((a.dv + 63) / 64) * tiles_i * a.n_heads * n_seqs;
    const cudaError_t attr = mv_allow_smem<cs_output_kernel<CHANNEL>>(CO_SMEM);
    if (attr != cudaSuccess) return (int)attr;
    const int per_seq = min((max_len + CS_CHUNK - 1) / CS_CHUNK, a.room);       // the most chunks a sequence has in a window
    for (a.w0 = 0; a.w0 < chunks; a.w0 += a.room) {
        a.w1 = a.w0 + a.room;
        int code;
        if (tiles > 148) code = cs_walk_launch<8, 2, CHANNEL>(a, (a.dv + 63) / 64 * tiles_i, n_seqs, stream);
        else if (tiles > 74) code = cs_walk_launch<8, 4, CHANNEL>(a, (a.dv + 63) / 64 * tiles_i, n_seqs, stream);
        else code = cs_walk_launch<4, 4, CHANNEL>(a, (a.dv + 31) / 32 * tiles_i, n_seqs, stream);
        if (code) return code;
        mv_launch(cs_output_kernel<CHANNEL>, dim3(per_seq * ((a.dv + 63) / 64), a.n_heads, n_seqs), CS_THREADS, CO_SMEM, stream, a);
        code = mv_launch_status();
        if (code) return code;
    }
    return 0;
}

}  // namespace
