// Routing of a mixture of experts, and the gated activation of the chosen experts.
//
// Router: s_e = sigmoid(z_e) from 32-bit logits (a bias may be added to them first), or softmax over all of them, or
// the logits themselves with weights softmax(the chosen logits); a correction per expert may be added
// for the choice alone; some of the routed entries may be identity experts (no matrices: their output is their input).  The experts form `n_groups` equal groups of neighbours; a
// group's score is the sum of its two largest s (of its only one, in groups of one); only experts of the
// `keep` best groups can be chosen; the `top` largest s among those are chosen; their weights are s divided
// by the sum of the chosen s (+ 1e-20), or s itself where they are not to be renormalized.  Ties go to the lower index.  A shared expert's gate, sigmoid of one
// more logit, is written as one more column (a shared expert without a gate has none).  All of it is 32-bit.
//
// Output: a dense row of weights per token, [experts (+ 1)], zero for the experts that were not chosen, and
// the chosen experts with their weights as lists [top].
#include "common.cuh"

#define RE_MAX_EXPERTS 1024

__device__ __forceinline__ void re_argmax(float& v, int& i) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, i, o);
        if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
    }
}

// one warp a token.  z <- z + bias (or null).  mode 0: scores sigmoid(z); mode 1: scores softmax(z) over all E routed
// entries; mode 2: scores z, the weights are softmax over the chosen z alone, times out_scale.  `correction`
// (or null) is added to the scores for the CHOICE only; the weights are the chosen entries' own scores over their sum
// (+ 1e-20) (without renorm: the scores themselves), times out_scale.  The last n_identity of the E entries are identity experts: the dense row is laid out
// [E - n_identity experts | the shared gate, if any | n_identity identity weights].
__global__ void __launch_bounds__(128)
route_kernel(const float* __restrict__ z, int ld, float* __restrict__ dense, int* __restrict__ pick,
             float* __restrict__ pick_w, int N, int E, int n_groups, int keep, int top, int shared_gate, int mode,
             const float* __restrict__ correction, float out_scale, int n_identity, const float* __restrict__ bias, int renorm) {
    mv_pdl_begin();
    extern __shared__ float re_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = blockIdx.x * (blockDim.x >> 5) + warp;
    if (n >= N) return;
    const float NEG = -3.0e38f;
    float* s = re_smem + (size_t)warp * (2 * E + n_groups);   // scores
    float* ch = s + E;                                        // choice scores; NEG once taken or not allowed
    float* gs = ch + E;                                       // group scores
    const float* zr = z + (size_t)n * ld;
    const int n_real = E - n_identity, sg = shared_gate ? 1 : 0;
    const int cols = E + sg;
    float* dr = dense + (size_t)n * cols;
    for (int e = lane; e < E; e += 32) s[e] = zr[e] + (bias ? bias[e] : 0.f);       // a lane's own entries
    if (mode == 1) {
        float mx = NEG;
        for (int e = lane; e < E; e += 32) mx = fmaxf(mx, s[e]);
        mx = mv_warp_max(mx);
        float sum = 0.f;
        for (int e = lane; e < E; e += 32) {
            const float v = expf(s[e] - mx);
            s[e] = v;
            sum += v;
        }
        sum = mv_warp_sum(sum);
        const float inv = 1.0f / sum;
        for (int e = lane; e < E; e += 32) s[e] *= inv;
    } else if (mode == 0) {
        for (int e = lane; e < E; e += 32) s[e] = 1.0f / (1.0f + expf(-s[e]));
    }
    for (int e = lane; e < E; e += 32) ch[e] = s[e] + (correction ? correction[e] : 0.f);
    for (int c = lane; c < cols; c += 32) dr[c] = 0.f;
    __syncwarp();
    if (shared_gate && lane == 0) dr[n_real] = 1.0f / (1.0f + expf(-zr[E]));
    const int per = E / n_groups;
    if (keep < n_groups) {
        for (int g = lane; g < n_groups; g += 32) {
            float a = NEG, b = NEG;                            // the two largest of the group
            for (int e = g * per; e < (g + 1) * per; ++e) {
                const float v = ch[e];
                if (v > a) { b = a; a = v; } else if (v > b) b = v;
            }
            gs[g] = a + (per > 1 ? b : 0.f);
        }
        __syncwarp();
        // the best `keep` groups are marked; then the others' experts are struck out
        for (int r = 0; r < keep; ++r) {
            float v = NEG; int i = 0x7fffffff;
            for (int g = lane; g < n_groups; g += 32)
                if (gs[g] > v) { v = gs[g]; i = g; }
            re_argmax(v, i);
            if (lane == 0) gs[i] = 2.f * NEG;                  // chosen
            __syncwarp();
        }
        for (int e = lane; e < E; e += 32)
            if (gs[e / per] != 2.f * NEG) ch[e] = NEG;
        __syncwarp();
    }
    float sum = 0.f, best = NEG;
    for (int r = 0; r < top; ++r) {
        float v = NEG; int i = 0x7fffffff;
        for (int e = lane; e < E; e += 32)
            if (ch[e] > v) { v = ch[e]; i = e; }
        re_argmax(v, i);
        const float sc = s[i];
        sum += sc;
        best = fmaxf(best, sc);
        if (lane == 0) {
            pick[(size_t)n * top + r] = i;
            pick_w[(size_t)n * top + r] = sc;
            ch[i] = NEG;
        }
        __syncwarp();
    }
    // (top <= 32 is checked by the host)
    float w = lane < top ? pick_w[(size_t)n * top + lane] : 0.f;
    if (mode == 2) {
        w = lane < top ? expf(w - best) : 0.f;
        sum = mv_warp_sum(w);
    }
    w *= mode == 2 ? out_scale / sum : (renorm ? out_scale / (sum + 1e-20f) : out_scale);
    if (lane < top) {
        pick_w[(size_t)n * top + lane] = w;
        const int i = pick[(size_t)n * top + lane];
        dr[i < n_real ? i : i + sg] = w;
    }
}

// z [N, >= E (+ 1)] with row stride ld; dense [N, E (+ 1)]; pick, pick_w [N, top]; correction, bias [E] or null.
MV_API int mv_route(const float* z, int ld, float* dense, int* pick, float* pick_w, int N, int E, int n_groups,
                    int keep, int top, int shared_gate, int mode, const float* correction, float out_scale,
                    int n_identity, const float* bias, int renorm, cudaStream_t stream) {
    if (N <= 0) return 0;
    if (E < 1 || E > RE_MAX_EXPERTS || n_groups < 1 || E % n_groups || keep < 1 || keep > n_groups || top < 1 ||
        top > 32 || top > keep * (E / n_groups) || n_identity < 0 || n_identity > E || mode < 0 || mode > 2)
        return (int)cudaErrorInvalidValue;
    const int warps = 4;
    const size_t smem = sizeof(float) * warps * (size_t)(2 * E + n_groups);
    mv_launch(route_kernel, (N + warps - 1) / warps, warps * 32, smem, stream, z, ld, dense, pick, pick_w, N, E,
              n_groups, keep, top, shared_gate, mode, correction, out_scale, n_identity, bias, renorm);
    return mv_launch_status();
}

// resid[n, :] += (sum of dense[n, col0 .. col0 + n_cols)) * h[n, :]: experts whose output is their input; V columns a thread (4 where H is a
// multiple: 2,048 tokens of 2,048 28.6 -> 13.6 us).
template <typename T, int V>
__global__ void __launch_bounds__(256)
identity_experts_kernel(const T* __restrict__ h, const float* __restrict__ dense, int ld, int col0, int n_cols,
                        float* __restrict__ resid, long long total, int H, int accumulate) {
    mv_pdl_begin();
    const long long idx = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * V;
    if (idx >= total) return;
    const long long n = idx / H;
    float x[V], old[V];
    if constexpr (V == 4) {
        if constexpr (sizeof(T) == 2) {
            const uint2 r = *reinterpret_cast<const uint2*>(h + idx);
            x[0] = __uint_as_float(r.x << 16); x[1] = __uint_as_float(r.x & 0xffff0000u);
            x[2] = __uint_as_float(r.y << 16); x[3] = __uint_as_float(r.y & 0xffff0000u);
        } else {
            const float4 r = *reinterpret_cast<const float4*>(h + idx);
            x[0] = r.x; x[1] = r.y; x[2] = r.z; x[3] = r.w;
        }
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
        if (accumulate) o = *reinterpret_cast<const float4*>(resid + idx);
        old[0] = o.x; old[1] = o.y; old[2] = o.z; old[3] = o.w;
    } else {
        x[0] = mv_to_f32(h[idx]);
        old[0] = accumulate ? resid[idx] : 0.f;
    }
    float w = 0.f;
    for (int c = 0; c < n_cols; ++c) w += dense[n * ld + col0 + c];
#pragma unroll
    for (int j = 0; j < V; ++j) {
        const float v = __fmul_rn(w, x[j]);
        x[j] = accumulate ? __fadd_rn(old[j], v) : v;
    }
    if constexpr (V == 4) *reinterpret_cast<float4*>(resid + idx) = make_float4(x[0], x[1], x[2], x[3]);
    else resid[idx] = x[0];
}

MV_API int mv_identity_experts(const void* h, int dtype, const float* dense, int ld, int col0, int n_cols, float* resid,
                               int N, int H, int accumulate, cudaStream_t stream) {
    if (N <= 0 || n_cols <= 0) return 0;
    const long long total = (long long)N * H;
    const bool vec = H % 4 == 0 && (((uintptr_t)h | (uintptr_t)resid) & 15) == 0;
    const unsigned blocks = (unsigned)((total / (vec ? 4 : 1) + 255) / 256);
#define ID_LAUNCH(T, V) mv_launch(identity_experts_kernel<T, V>, blocks, 256, 0, stream, (const T*)h, dense, ld, col0, n_cols, resid, total, H, accumulate)
    if (dtype == MV_DT_BF16) { if (vec) ID_LAUNCH(__nv_bfloat16, 4); else ID_LAUNCH(__nv_bfloat16, 1); }
    else { if (vec) ID_LAUNCH(float, 4); else ID_LAUNCH(float, 1); }
#undef ID_LAUNCH
    return mv_launch_status();
}

// ------------------------------------------------------------------------------------------------
// hid[n, c] = w[n, expert(c)] * act(gate[n, c], up[n, c]) (silu(gate) * up, or with `limit` > 0 the clamped gated
// activation with that limit, `shared_limit` for the shared expert, and `alpha`) over the columns of all experts laid end to end
// (expert e owns [e * ff, (e + 1) * ff), a shared expert the `shared_ff` columns after them, with the weight of
// column E, or 1 where it has no gate).  gu [N, 2 * F] holds an expert's gates and ups together, [e * 2 ff, (e + 1) * 2 ff): alternating in
// groups of 16 columns (16 gates, their 16 ups, ...) where `group` says so, else the gates, then the ups; the
// shared expert's block follows with `shared_group`.  Where the weight is zero nothing is computed.  on_input: the weight
// multiplies the expert's INPUT, hid = act(w gate, w up) (gate and up are linear in it).
template <typename TO>
__global__ void __launch_bounds__(256)
routed_glu_kernel(const float* __restrict__ gu, const float* __restrict__ dense, TO* __restrict__ hid, long long total,
                  int F, int E, int ff, int shared_ff, int cols, int group, int shared_group, int shared_gate, int on_input,
                  float limit, float shared_limit, float alpha) {
    mv_pdl_begin();
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const long long n = idx / F;
    const int c = (int)(idx - n * F);
    const int e = c < E * ff ? c / ff : E;
    const float w = e < E || shared_gate ? dense[n * cols + e] : 1.f;
    float out = 0.f;
    if (w != 0.f) {
        const int cc = c - e * ff, width = e < E ? ff : shared_ff, grp = e < E ? group : shared_group;
        const float* blk = gu + n * 2 * F + (size_t)e * 2 * ff;
        const int gi = grp ? (cc / grp) * 2 * grp + cc % grp : cc;
        const bool first = on_input && e < E;                // (a shared expert's gate is always on its output)
        const float wi = first ? w : 1.f;
        const float g = wi * blk[gi], u = wi * blk[gi + (grp ? grp : width)];
        out = (first ? 1.f : w) * (limit > 0.f ? mv_glu_clamped(g, u, e < E ? limit : shared_limit, alpha) : mv_glu_silu(g, u));
    }
    hid[idx] = mv_from_f32<TO>(out);
}

// extra_cols: columns of a dense row after the experts' (and the shared gate's) that belong to others
MV_API int mv_routed_glu(const float* gu, const float* dense, void* hid, int hid_dtype, int N, int E, int ff,
                         int shared_ff, int group, int shared_group, int extra_cols, int shared_gate, int on_input,
                         float limit, float shared_limit, float alpha, cudaStream_t stream) {
    if (N <= 0) return 0;
    const int F = E * ff + shared_ff, cols = E + (shared_ff && shared_gate ? 1 : 0) + extra_cols;
    if ((group && ff % group) || (shared_group && shared_ff % shared_group)) return (int)cudaErrorInvalidValue;
    const long long total = (long long)N * F;
    const unsigned blocks = (unsigned)((total + 255) / 256);
    if (hid_dtype == MV_DT_BF16)
        mv_launch(routed_glu_kernel<__nv_bfloat16>, blocks, 256, 0, stream, gu, dense, (__nv_bfloat16*)hid, total, F, E,
                  ff, shared_ff, cols, group, shared_group, shared_gate, on_input, limit, shared_limit, alpha);
    else
        mv_launch(routed_glu_kernel<float>, blocks, 256, 0, stream, gu, dense, (float*)hid, total, F, E, ff, shared_ff, cols,
                  group, shared_group, shared_gate, on_input, limit, shared_limit, alpha);
    return mv_launch_status();
}

// ------------------------------------------------------------------------------------------------
// For steps of many tokens: the (token, choice) entries sorted by expert, so that every expert multiplies its own
// tokens' rows only.  The sort is a stable counting sort: a block an expert walks the entries in order and ranks
// its own; the ranks depend on the entries alone, not on which block ran first.
// 1,024 threads take 4 entries each a round, the loads of a round ahead of its barrier (24,000 entries are 6 rounds and were 94 of 256: ranks, tiles and
// rows of 6,000 tokens together 140 -> 36 us).
constexpr int RANK_THREADS = 1024;
__global__ void __launch_bounds__(RANK_THREADS)
expert_rank_kernel(const int* __restrict__ pick, int total, int* __restrict__ rank, int* __restrict__ counts) {
    mv_pdl_begin();
    __shared__ int warp_sum[2][RANK_THREADS / 32];
    const int e = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool vec = ((uintptr_t)pick & 15) == 0;
    auto load = [&](int t0) {
        const int i = t0 + 4 * tid;
        int4 v = make_int4(-1, -1, -1, -1);
        if (vec && i + 3 < total) v = *reinterpret_cast<const int4*>(pick + i);
        else {
            if (i < total) v.x = pick[i];
            if (i + 1 < total) v.y = pick[i + 1];
            if (i + 2 < total) v.z = pick[i + 2];
            if (i + 3 < total) v.w = pick[i + 3];
        }
        return v;
    };
    int base = 0, buf = 0;
    int4 v = load(0);
    for (int t0 = 0; t0 < total; t0 += 4 * RANK_THREADS, buf ^= 1) {
        const int4 next = t0 + 4 * RANK_THREADS < total ? load(t0 + 4 * RANK_THREADS) : v;
        const int m[4] = {v.x == e, v.y == e, v.z == e, v.w == e};
        const int mine = m[0] + m[1] + m[2] + m[3];
        int upto = mine;                                      // of this lane and the ones before it
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += x;
        }
        if (lane == 31) warp_sum[buf][warp] = upto;
        __syncthreads();                                      // (two buffers: the next round writes the other one)
        const int w = warp_sum[buf][lane];
        int before = lane < warp ? w : 0, all = w;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            before += __shfl_xor_sync(0xffffffffu, before, o);
            all += __shfl_xor_sync(0xffffffffu, all, o);
        }
        int at = base + before + upto - mine;
        const int i = t0 + 4 * tid;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (m[j]) rank[i + j] = at++;
        base += all;
        v = next;
    }
    if (tid == 0) counts[e] = base;
}

// place[entry] = (entries of the experts before its own) + its rank; the token's row is copied there (in_w not null: times
// the entry's weight).
template <typename T>
__global__ void __launch_bounds__(128)
expert_gather_kernel(const int* __restrict__ pick, const int* __restrict__ rank, const int* __restrict__ counts,
                     const int* __restrict__ offsets, const T* __restrict__ x, const float* __restrict__ in_w, int E, int top, int H,
                     int* __restrict__ place, T* __restrict__ xs) {
    mv_pdl_begin();
    __shared__ float scratch[33];
    const int idx = blockIdx.x;
    const int e = pick[idx];
    if (e >= E) {                                  // an identity expert has no rows
        if (threadIdx.x == 0) place[idx] = -1;
        return;
    }
    int p;
    if (offsets) {
        p = offsets[e] + rank[idx];                // where the expert's (padded) run of rows starts
    } else {
        int before = 0;
        for (int i = threadIdx.x; i < e; i += blockDim.x) before += counts[i];
        p = (int)(mv_block_sum((float)before, scratch) + 0.5f) + rank[idx];       // exact: counts are far below 2^24
    }
    if (threadIdx.x == 0) place[idx] = p;
    const T* src = x + (size_t)(idx / top) * H;
    T* dst = xs + (size_t)p * H;
    if (in_w) {
        const float w = in_w[idx];
        for (int h = threadIdx.x; h < H; h += blockDim.x) dst[h] = mv_from_f32<T>(w * mv_to_f32(src[h]));
        return;
    }
    for (int h = threadIdx.x; h < H; h += blockDim.x) dst[h] = src[h];
}

// The same for rows of whole 16-byte words and padded runs: a block is a token, its row is read once, 16 bytes a thread, and written to all its places (number
// by number, a block an entry, 72 us of those 140).
template <typename T>
__global__ void __launch_bounds__(128)
expert_gather_vec_kernel(const int* __restrict__ pick, const int* __restrict__ rank, const int* __restrict__ offsets,
                         const T* __restrict__ x, const float* __restrict__ in_w, int E, int top, int H, int* __restrict__ place, T* __restrict__ xs) {
    mv_pdl_begin();
    __shared__ int at[32];
    const int n = blockIdx.x;
    if ((int)threadIdx.x < top) {
        const int idx = n * top + threadIdx.x, e = pick[idx], p = e < E ? offsets[e] + rank[idx] : -1;    // (an identity expert has no rows)
        place[idx] = p;
        at[threadIdx.x] = p;
    }
    __syncthreads();
    constexpr int V = 16 / sizeof(T);
    const int words = H / V;
    const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)n * H);
    for (int i = threadIdx.x; i < words; i += blockDim.x) {
        const uint4 v = src[i];
        for (int k = 0; k < top; ++k) {
            if (at[k] < 0) continue;
            T* dst = xs + (size_t)at[k] * H + i * V;
            if (in_w) {
                const float w = in_w[n * top + k];
                float f[V];
                mv_unpack16(v, f, (const T*)nullptr);
#pragma unroll
                for (int j = 0; j < V; j += 4) mv_store4(dst + j, w * f[j], w * f[j + 1], w * f[j + 2], w * f[j + 3]);
            } else {
                *reinterpret_cast<uint4*>(dst) = v;
            }
        }
    }
}

// pick_w null: every chosen expert's result counts as it is.
// out[n, :] (+)= sum_k w[n, k] ys[place[n * top + k], :] + gate[n] shared[n, :], the choices in their order; V columns a thread (4: rows of whole 16-byte
// words; 6,000 tokens of 2,048, 4 choices and a shared expert 82 -> 61 us).
template <int V>
__global__ void __launch_bounds__(256)
expert_combine_kernel(const float* __restrict__ ys, const int* __restrict__ place, const float* __restrict__ pick_w,
                      const float* __restrict__ shared, const float* __restrict__ gate, int ld_gate,
                      float* __restrict__ out, int top, int H, int accumulate) {
    mv_pdl_begin();
    __shared__ int at[32];
    __shared__ float ws[32];
    const int n = blockIdx.x;
    if ((int)threadIdx.x < min(top, 32)) {
        at[threadIdx.x] = place[(size_t)n * top + threadIdx.x];
        ws[threadIdx.x] = pick_w ? pick_w[(size_t)n * top + threadIdx.x] : 1.f;
    }
    __syncthreads();
    const float g = shared ? (gate ? gate[(size_t)n * ld_gate] : 1.f) : 0.f;
    for (int h = V * threadIdx.x; h < H; h += V * blockDim.x) {
        float* o = out + (size_t)n * H + h;
        float sum[V], y[V], old[V];
        auto load = [&](const float* p, float (&d)[V]) {
            if constexpr (V == 4) {
                const float4 a = *reinterpret_cast<const float4*>(p);
                d[0] = a.x; d[1] = a.y; d[2] = a.z; d[3] = a.w;
            } else {
                d[0] = *p;
            }
        };
#pragma unroll
        for (int j = 0; j < V; ++j) { sum[j] = 0.f; old[j] = 0.f; }
        if (accumulate) load(o, old);
#pragma unroll 4
        for (int k = 0; k < top; ++k) {
            const int row = k < 32 ? at[k] : place[(size_t)n * top + k];
            const float w = k < 32 ? ws[k] : pick_w ? pick_w[(size_t)n * top + k] : 1.f;
            load(ys + (size_t)row * H + h, y);
#pragma unroll
            for (int j = 0; j < V; ++j) sum[j] = fmaf(w, y[j], sum[j]);
        }
        if (shared) {
            load(shared + (size_t)n * H + h, y);
#pragma unroll
            for (int j = 0; j < V; ++j) sum[j] = fmaf(g, y[j], sum[j]);
        }
        if (accumulate) {
#pragma unroll
            for (int j = 0; j < V; ++j) sum[j] = old[j] + sum[j];
        }
        if constexpr (V == 4) *reinterpret_cast<float4*>(o) = make_float4(sum[0], sum[1], sum[2], sum[3]);
        else *o = sum[0];
    }
}

// pick [N, top] -> rank [N * top], counts [E]
MV_API int mv_expert_rank(const int* pick, int total, int E, int* rank, int* counts, cudaStream_t stream) {
    if (total <= 0 || E <= 0) return 0;
    mv_launch(expert_rank_kernel, E, RANK_THREADS, 0, stream, pick, total, rank, counts);
    return mv_launch_status();
}

// x [N, H] in `dtype` -> xs [N * top, H] sorted by expert; place [N * top] says where each entry went
// offsets (or null): where every expert's run of rows starts (mv_expert_tiles), instead of the plain sums of counts; picks from E on
// (identity experts) have no row and place -1
MV_API int mv_expert_gather(const int* pick, const int* rank, const int* counts, const int* offsets, const void* x,
                            int dtype, const float* in_w, int E, int N, int top, int H, int* place, void* xs, cudaStream_t stream) {
    if (N <= 0) return 0;
    if (offsets && top <= 32 && (H * (dtype == MV_DT_BF16 ? 2 : 4)) % 16 == 0 && (((uintptr_t)x | (uintptr_t)xs) & 15) == 0) {
        if (dtype == MV_DT_BF16)
            mv_launch(expert_gather_vec_kernel<__nv_bfloat16>, N, 128, 0, stream, pick, rank, offsets, (const __nv_bfloat16*)x, in_w, E, top, H,
                      place, (__nv_bfloat16*)xs);
        else
            mv_launch(expert_gather_vec_kernel<float>, N, 128, 0, stream, pick, rank, offsets, (const float*)x, in_w, E, top, H, place, (float*)xs);
        return mv_launch_status();
    }
    if (dtype == MV_DT_BF16)
        mv_launch(expert_gather_kernel<__nv_bfloat16>, N * top, 128, 0, stream, pick, rank, counts, offsets,
                  (const __nv_bfloat16*)x, in_w, E, top, H, place, (__nv_bfloat16*)xs);
    else
        mv_launch(expert_gather_kernel<float>, N * top, 128, 0, stream, pick, rank, counts, offsets, (const float*)x, in_w, E, top, H,
                  place, (float*)xs);
    return mv_launch_status();
}

// Every expert's run of rows padded to whole tiles of `tile_rows`, so that a grouped product's tile never holds two
// experts: offsets[e] = where expert e's run starts, tile_group[t] = the expert of tile t, -1 for the spare tiles
// after the last run.  One block; the host needs to know nothing (n_tiles is an upper bound:
// (entries + E * (tile_rows - 1)) / tile_rows).
__global__ void __launch_bounds__(256)
expert_tiles_kernel(const int* __restrict__ counts, int E, int tile_rows, int* __restrict__ offsets,
                    int* __restrict__ tile_group, int n_tiles) {
    mv_pdl_begin();
    __shared__ int first_tile[RE_MAX_EXPERTS + 1];
    if (threadIdx.x == 0) {
        int t = 0;
        for (int e = 0; e < E; ++e) {
            first_tile[e] = t;
            offsets[e] = t * tile_rows;
            t += (counts[e] + tile_rows - 1) / tile_rows;
        }
        first_tile[E] = t;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < n_tiles; t += blockDim.x) {
        int g = -1;
        if (t < first_tile[E]) {
            int lo = 0, hi = E;                    // the last expert whose first tile is <= t and that has tiles
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (first_tile[mid] <= t) lo = mid; else hi = mid;
            }
            g = lo;
        }
        tile_group[t] = g;
    }
}

MV_API int mv_expert_tiles(const int* counts, int E, int tile_rows, int* offsets, int* tile_group, int n_tiles,
                           cudaStream_t stream) {
    if (E <= 0 || n_tiles <= 0) return 0;
    if (E > RE_MAX_EXPERTS || tile_rows < 1) return (int)cudaErrorInvalidValue;
    mv_launch(expert_tiles_kernel, 1, 256, 0, stream, counts, E, tile_rows, offsets, tile_group, n_tiles);
    return mv_launch_status();
}

MV_API int mv_expert_combine(const float* ys, const int* place, const float* pick_w, const float* shared,
                             const float* gate, int ld_gate, float* out, int N, int top, int H, int accumulate,
                             cudaStream_t stream) {
    if (N <= 0) return 0;
    const bool vec = H % 4 == 0 && (((uintptr_t)ys | (uintptr_t)shared | (uintptr_t)out) & 15) == 0;
    if (vec) mv_launch(expert_combine_kernel<4>, N, 256, 0, stream, ys, place, pick_w, shared, gate, ld_gate, out, top, H, accumulate);
    else mv_launch(expert_combine_kernel<1>, N, 256, 0, stream, ys, place, pick_w, shared, gate, ld_gate, out, top, H, accumulate);
    return mv_launch_status();
}

// h[n, e * ff + c] = w * hs[place, c] where token n chose expert e (rounded again), 0 where it did not: the experts' gated activations, worked out over
// sorted rows, laid out as one product with all down matrices side by side reads them.  A block is a token; eight numbers a thread at a time (2,048
// tokens of 16 experts of 1,024: 22.5 us, 5 TB/s).
__global__ void __launch_bounds__(256)
expert_spread_kernel(const int* __restrict__ pick, const int* __restrict__ place, const float* __restrict__ pick_w,
                     const __nv_bfloat16* __restrict__ hs, __nv_bfloat16* __restrict__ h, int E, int top, int ff) {
    mv_pdl_begin();
    __shared__ int row[RE_MAX_EXPERTS];
    __shared__ float weight[RE_MAX_EXPERTS];
    const int n = blockIdx.x;
    for (int e = threadIdx.x; e < E; e += blockDim.x) row[e] = -1;
    __syncthreads();
    if ((int)threadIdx.x < top) {
        const int idx = n * top + threadIdx.x, e = pick[idx];
        if (e < E) { row[e] = place[idx]; weight[e] = pick_w[idx]; }
    }
    __syncthreads();
    const int words = ff / 8;
    uint4* dst = reinterpret_cast<uint4*>(h + (size_t)n * E * ff);
    for (int i = threadIdx.x; i < E * words; i += blockDim.x) {
        const int e = i / words;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (row[e] >= 0) {
            float x[8];
            mv_load8(hs + (size_t)row[e] * ff + (i - e * words) * 8, x);
            const float w = weight[e];
            unsigned p[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const __nv_bfloat162 y = __floats2bfloat162_rn(x[2 * j] * w, x[2 * j + 1] * w);
                p[j] = *reinterpret_cast<const unsigned*>(&y);
            }
            v = make_uint4(p[0], p[1], p[2], p[3]);
        }
        dst[i] = v;
    }
}

// pick, place, pick_w [N, top] (place: mv_expert_gather's), hs [.., ff] bfloat16 -> h [N, E ff]; ff a multiple of 8, 16-byte aligned
MV_API int mv_expert_spread(const int* pick, const int* place, const float* pick_w, const void* hs, void* h, int N, int E, int top, int ff,
                            cudaStream_t stream) {
    if (N <= 0) return 0;
    if (E < 1 || E > RE_MAX_EXPERTS || top < 1 || top > 256 || ff < 8 || ff % 8 || (((uintptr_t)hs | (uintptr_t)h) & 15)) return (int)cudaErrorInvalidValue;
    mv_launch(expert_spread_kernel, N, 256, 0, stream, pick, place, pick_w, (const __nv_bfloat16*)hs, (__nv_bfloat16*)h, E, top, ff);
    return mv_launch_status();
}

// h[n, c] *= w[n, expert(c)] in place, for activations that a product's epilogue has already gated: eight
// columns a thread (ff and shared_ff are multiples of 8 then), or one.
template <typename T, int V>
__global__ void __launch_bounds__(256)
scale_expert_columns_kernel(T* __restrict__ h, const float* __restrict__ dense, long long total, int F, int E, int ff,
                            int cols, int shared_gate) {
    mv_pdl_begin();
    const long long idx = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * V;
    if (idx >= total) return;
    const long long n = idx / F;
    const int c = (int)(idx - n * F);
    if (c >= E * ff && !shared_gate) return;                   // a shared expert without a gate: as it is
    const float w = dense[n * cols + (c < E * ff ? c / ff : E)];
    if (V == 8) {
        float x[8];
        mv_load8(h + idx, x);
        mv_store4(h + idx, x[0] * w, x[1] * w, x[2] * w, x[3] * w);
        mv_store4(h + idx + 4, x[4] * w, x[5] * w, x[6] * w, x[7] * w);
    } else {
        h[idx] = mv_from_f32<T>(mv_to_f32(h[idx]) * w);
    }
}

MV_API int mv_scale_expert_columns(void* h, int dtype, const float* dense, int N, int E, int ff, int shared_ff,
                                   int extra_cols, int shared_gate, cudaStream_t stream) {
    if (N <= 0) return 0;
    const int F = E * ff + shared_ff, cols = E + (shared_ff && shared_gate ? 1 : 0) + extra_cols;
    const long long total = (long long)N * F;
    const bool wide = ff % 8 == 0 && shared_ff % 8 == 0 && ((uintptr_t)h % 16) == 0;
    const unsigned blocks = (unsigned)((total / (wide ? 8 : 1) + 255) / 256);
#define SE_LAUNCH(T, V) mv_launch(scale_expert_columns_kernel<T, V>, blocks, 256, 0, stream, (T*)h, dense, total, F, E, ff, cols, shared_gate)
    if (dtype == MV_DT_BF16) { if (wide) SE_LAUNCH(__nv_bfloat16, 8); else SE_LAUNCH(__nv_bfloat16, 1); }
    else { if (wide) SE_LAUNCH(float, 8); else SE_LAUNCH(float, 1); }
#undef SE_LAUNCH
    return mv_launch_status();
}
