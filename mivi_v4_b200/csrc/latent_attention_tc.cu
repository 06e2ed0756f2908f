// Attention over a compressed cache (see latent_attention_prefill.cu) for steps that bring a sequence many tokens, on the
// fifth-generation tensor cores: heads of 64 + 32 or 64 + 64 channels with values of 64, bfloat16.  Both products are tcgen05.mma with their
// results in tensor memory.
//
// Block = 256 consecutive query tokens of one sequence for one head, as two tiles of 128 that share the keys and values; these come in
// blocks of 64 rows by TMA out of the rows that one product built from the cache (kx: every head's unrotated keys and its values; r:
// the rotated part that all heads share).
//
//   warp 0      TMA: the two Q tiles once, then keys and values into rings of four stages each;
//   warp 1      S = Q K^T (128 x 64 x 96 or 128);
//   warp 3      O += P V (128 x 64 x 64, twice: P is two bfloat16 numbers), P read from tensor memory;
//   warp 2      looks through the values of the blocks that some row of the pair does not see whole (attention_tc.cuh): another sequence's rows
//               become zeros, and so do infinities and NaNs, which would pass through a weight of 0;
//   warps 4-11  softmax, four warps a tile, one query row a thread.
//
// Tensor memory: two buffers of 64 columns a tile for S, and O of 64 a tile.  A row's thread takes its 64 scores into registers and
// puts the weights in their place, the rounded numbers in the first 32 columns and what the rounding left in the others: the
// sum over the values carries the weights to 16 bits of mantissa.  The scores of a tile's next block are under way while it works on
// this one's, so no tile waits for them; O stays in tensor memory.
//
// Every sum is added in the order of latent_attention_prefill.cu, so that a row's result does not hang on which of the two kernels its step
// took (a router behind it would choose other experts): both kinds of tensor-core instruction add alike; key blocks lie at multiples of 64; a row's
// reference is its running maximum after every block; its denominator is four sums, of every eighth key and its neighbour.  Only the sink of a row whose keys are all far
// below it (e^-60 of it) is left out of the reference, and joins at the end: nothing is lost where it is all that the row shows.
//
// Bound by the softmax (a block of 64 keys of both tiles needs 1,024 clocks of the exponential unit at 16 a clock and some 1,000 instructions of each
// scheduler; over one prompt of 2,048 tokens, whose tiles are two rounds of unequal length, schedulers 41 % busy, that unit 31 %, tensor cores 19 %).  32 heads of 64 + 32 / 64 with a gate, this kernel / latent_attention_prefill.cu: one prompt of 6,000 tokens
// 372 / 1,132 us, of 2,048 73 / 190, three of 333 to 2,048 108 / 226.  What it took: an elected lane of a whole warp issues the products (see
// tc_common.cuh; a first form of the kernel with a lane by itself 495 us), one warp for
// either product (one for both: the waits of one hold up the other, 296 against 273 for a form of other sums), gates read 32 bytes at a time (a block's gates element by
// element took longer than its softmax: 344 against 317).
#include "attention_tc.cuh"

namespace {

constexpr int LT_THREADS = 384;
constexpr int BQ = 128, TILES = 2, BKV = 64, DIM = 64, DV = 64, KSTAGES = 4, SBUFS = 4;
constexpr int V_BYTES = BKV * DV * 2;
constexpr unsigned O_COL0 = SBUFS * BKV;           // tile t: O at O_COL0 + 64 t
constexpr float FAR_BELOW = 60.0f;                 // a row whose keys are that far below its sink
constexpr float LOG2E = 1.4426950408889634f;

template <int ROT> struct LtLayout {
    // queries and keys lie as two swizzled parts, the 64 unrotated channels and the rotated ones
    static constexpr int Q_PART = BQ * DIM * 2, Q_BYTES = Q_PART + BQ * ROT * 2, K_PART = BKV * DIM * 2, K_BYTES = K_PART + BKV * ROT * 2;
    static constexpr int K_AT = TILES * Q_BYTES, V_AT = K_AT + KSTAGES * K_BYTES, BAR_AT = V_AT + KSTAGES * V_BYTES;
    static constexpr int TOTAL = BAR_AT + 512 + 1024;
};

// barriers, 8 bytes each.  Scores, weights and products have two a tile, by the key block's parity: the next block's may be complete before
// whoever waits for this block's has looked, the one after that cannot.
enum { B_Q = 0, B_KFULL = 1, B_KEMPTY = B_KFULL + KSTAGES, B_VFULL = B_KEMPTY + KSTAGES, B_VEMPTY = B_VFULL + KSTAGES,
       B_SFULL = B_VEMPTY + KSTAGES, B_PFULL = B_SFULL + 2 * TILES, B_PVDONE = B_PFULL + 2 * TILES, B_VFIX = B_PVDONE + 2 * TILES,
       B_LOOKED = B_VFIX + KSTAGES, B_COUNT };
static_assert(B_COUNT * 8 + 8 <= 512, "barrier area");

// scores of the keys outside [from, upto) become -inf; the chunk's first key is key c of the block
__device__ __forceinline__ void mask_chunk(unsigned (&s)[32], int c, int from, int upto) {
#pragma unroll
    for (int i = 0; i < 32; ++i)
        if (c + i >= upto || c + i < from) s[i] = 0xff800000u;
}
__device__ __forceinline__ float chunk_max(const unsigned (&s)[32]) {
    float a[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int i = 0; i < 32; i += 8)
#pragma unroll
        for (int e = 0; e < 4; ++e) a[e] = fmaxf(a[e], fmaxf(__uint_as_float(s[i + e]), __uint_as_float(s[i + 4 + e])));
    return fmaxf(fmaxf(a[0], a[1]), fmaxf(a[2], a[3]));
}
// the weights of 32 keys of a row, as two bfloat16 numbers each, into the row's columns p and p + BKV / 2; keys 8 i + 2 t and
// 8 i + 2 t + 1 are added to sum t
__device__ __forceinline__ void chunk_weights(const unsigned (&s)[32], float scale, float ref, unsigned p, float (&sum)[4]) {
    const float2 rf = make_float2(-ref, -ref), l2e = make_float2(LOG2E, LOG2E);
    unsigned hi[16], lo[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float2 x = mul2(add2(make_float2(__fmul_rn(__uint_as_float(s[2 * i]), scale), __fmul_rn(__uint_as_float(s[2 * i + 1]), scale)), rf), l2e);
        const float2 w = make_float2(ex2(x.x), ex2(x.y));
        sum[i & 3] = __fadd_rn(sum[i & 3], __fadd_rn(w.x, w.y));
        hi[i] = bits(__floats2bfloat162_rn(w.x, w.y));
        const float2 rest = add2(w, make_float2(-__uint_as_float(hi[i] << 16), -__uint_as_float(hi[i] & 0xffff0000u)));
        lo[i] = bits(__floats2bfloat162_rn(rest.x, rest.y));
    }
    tmem_st16(p, hi);
    tmem_st16(p + BKV / 2, lo);
}

// first position a step's tokens of a sequence that starts the step at `start` can see
__device__ __forceinline__ int first_seen(int start, int window) { return window > 0 ? max(0, start - window + 1) : 0; }

template <int ROT>
__global__ void __launch_bounds__(LT_THREADS, 1)
latent_attention_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_qr,
                           const __grid_constant__ CUtensorMap map_kx, const __grid_constant__ CUtensorMap map_r,
                           const __nv_bfloat16* __restrict__ kx, int ld_kx, int v0,
                           const int* __restrict__ cu, const int* __restrict__ starts, const float* __restrict__ sinks,
                           const float* __restrict__ gate, int ld_gate, int gate_heads, __nv_bfloat16* __restrict__ o, int B,
                           int nh, float scale, int window, int* __restrict__ err) {
    using L = LtLayout<ROT>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const unsigned q_s = smem_u32(smem), k_s = q_s + L::K_AT, v_s = q_s + L::V_AT;
    unsigned long long* bars = (unsigned long long*)(smem + L::BAR_AT);
    unsigned* tmem_holder = (unsigned*)(bars + B_COUNT);
    volatile int* found = (volatile int*)(tmem_holder + 1);               // warp 2 has met a value that is not finite
    const unsigned bar0 = smem_u32(bars);
    auto bar = [&](int i) { return bar0 + 8u * (unsigned)i; };

    // heads first, then pairs of tiles, the late (long) pairs of a sequence first
    int b = 0, pair = (int)(gridDim.y - 1 - blockIdx.y), base = 0;       // base: the gathered row of this sequence's first seen position
    for (; b < B; ++b) {
        const int len = cu[b + 1] - cu[b];
        const int pairs = (len + TILES * BQ - 1) / (TILES * BQ);
        if (pair < pairs) break;
        pair -= pairs;
        base += starts[b] + len - first_seen(starts[b], window);
    }
    if (b >= B) return;
    const int h = blockIdx.x;
    const int row0 = cu[b] + pair * TILES * BQ;
    const int nq = min(TILES * BQ, cu[b + 1] - row0);
    const int pos0 = starts[b] + pair * TILES * BQ;
    const int lo = first_seen(starts[b], window);
    const int key_first = first_seen(pos0, window) / BKV * BKV;          // where the pair's first key block starts
    const int key_row = base + key_first - lo;                          // (below 0 at most for rows that nobody sees)
    // key blocks of either tile: up to the block of its last query
    int nb[TILES];
#pragma unroll
    for (int t = 0; t < TILES; ++t) nb[t] = nq > t * BQ ? (pos0 + min(nq, (t + 1) * BQ) - 1 - key_first) / BKV + 1 : 0;
    const int nb_max = max(nb[0], nb[1]);
    // rows of the first and the last block that are not this sequence's, or come after the pair's last query
    const int rows_before = max(0, lo - key_first), last_rows = min(BKV, pos0 + nq - key_first - (nb_max - 1) * BKV);
    // some row of a tile that walks block j does not see all of it: from the block on that reaches past the first query (the second tile's own are among
    // them), and before the last query's window (a block with rows of others is one of these)
    const int seen_to = max(0, pos0 + 1 - key_first) / BKV, seen_from = window > 0 ? max(0, pos0 + nq - window - key_first + BKV - 1) / BKV : 0;
    auto partly_seen = [&](int j) { return j >= seen_to || j < seen_from; };
    const int warp = warp_index(), lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int i = 0; i < B_COUNT; ++i) mbar_init(bar(i), i >= B_PFULL && i < B_PFULL + 2 * TILES ? 4 : 1);
        *found = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_holder)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem_base = *tmem_holder;

    if (warp < 4) {
        // registers move from this warpgroup to the softmax warps (168 each at launch)
        asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
        if (warp == 0) {
            if (elect_one()) {
                mbar_expect_tx(bar(B_Q), TILES * L::Q_BYTES);
                for (int t = 0; t < TILES; ++t) {
                    tma_load_2d(q_s + t * L::Q_BYTES, &map_q, h * (DIM + ROT), row0 + t * BQ, bar(B_Q));
                    tma_load_2d(q_s + t * L::Q_BYTES + L::Q_PART, &map_qr, h * (DIM + ROT) + DIM, row0 + t * BQ, bar(B_Q));
                }
            }
            for (int j = 0; j < nb_max; ++j) {
                const int s = j % KSTAGES, row = key_row + j * BKV;
                const unsigned ph = (unsigned)(j / KSTAGES) & 1u;
                if (!mbar_wait_warp(bar(B_KEMPTY + s), ph ^ 1u, err, 51)) break;
                if (elect_one()) {
                    mbar_expect_tx(bar(B_KFULL + s), L::K_BYTES);
                    tma_load_2d(k_s + s * L::K_BYTES, &map_kx, h * DIM, row, bar(B_KFULL + s));
                    tma_load_2d(k_s + s * L::K_BYTES + L::K_PART, &map_r, 0, row, bar(B_KFULL + s));
                }
                if (!mbar_wait_warp(bar(B_VEMPTY + s), ph ^ 1u, err, 52)) break;
                // blocks that are partly seen go by way of warp 2, which then says that they are there
                const unsigned full = bar((partly_seen(j) ? B_VFIX : B_VFULL) + s);
                if (elect_one()) {
                    mbar_expect_tx(full, V_BYTES);
                    tma_load_2d(v_s + s * V_BYTES, &map_kx, v0 + h * DV, row, full);
                }
            }
        } else if (warp == 1) {
            // S(t, j) = Q_t K_j^T as soon as the keys are there and the buffer's weights, those of the tile's block before the last, are used
            const unsigned idesc = instr_desc(BQ, BKV);
            bool ok = mbar_wait_warp(bar(B_Q), 0, err, 53);
            for (int j = 0; j < nb_max && ok; ++j) {
                const int s = j % KSTAGES;
                if (!(ok = mbar_wait_warp(bar(B_KFULL + s), (unsigned)(j / KSTAGES) & 1u, err, 54))) break;
#pragma unroll
                for (int t = 0; t < TILES; ++t) {
                    if (!ok || j >= nb[t]) continue;
                    if (j > 1 && !(ok = mbar_wait_warp(bar(B_PVDONE + 2 * t + (j & 1)), (unsigned)((j - 2) >> 1) & 1u, err, 55))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const unsigned d = tmem_base + (unsigned)(2 * t + (j & 1)) * BKV;
                    const unsigned qa = q_s + t * L::Q_BYTES, ka = k_s + s * L::K_BYTES;
                    const unsigned long long q0 = smem_desc(qa), k0 = smem_desc(ka);
                    const unsigned long long q1 = ROT == 64 ? smem_desc(qa + L::Q_PART) : smem_desc_64(qa + L::Q_PART);
                    const unsigned long long k1 = ROT == 64 ? smem_desc(ka + L::K_PART) : smem_desc_64(ka + L::K_PART);
                    if (elect_one()) {
                        // 16 channels are 32 bytes, two units of a descriptor's address
#pragma unroll
                        for (int k = 0; k < DIM / 16; ++k) mma_f16(d, q0 + 2 * k, k0 + 2 * k, idesc, k > 0 ? 1u : 0u);
#pragma unroll
                        for (int k = 0; k < ROT / 16; ++k) mma_f16(d, q1 + 2 * k, k1 + 2 * k, idesc, 1u);
                        mma_commit(bar(B_SFULL + 2 * t + (j & 1)));
                        if (t == 1 || nb[1] == 0) mma_commit(bar(B_KEMPTY + s));
                    }
                }
            }
        } else if (warp == 3) {
            const unsigned idesc = instr_desc(BQ, DV) | (1u << 16);                 // V as it lies, a row a key: MN-major
            bool ok = true;
            for (int j = 0; j < nb_max && ok; ++j) {
                const int s = j % KSTAGES;
                if (!(ok = mbar_wait_warp(bar(B_VFULL + s), (unsigned)(j / KSTAGES) & 1u, err, 56))) break;
                const unsigned long long v0d = smem_desc(v_s + s * V_BYTES);
#pragma unroll
                for (int t = 0; t < TILES; ++t) {
                    if (!ok || j >= nb[t]) continue;
                    if (!(ok = mbar_wait_warp(bar(B_PFULL + 2 * t + (j & 1)), (unsigned)(j >> 1) & 1u, err, 58))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const unsigned p = tmem_base + (unsigned)(2 * t + (j & 1)) * BKV, d = tmem_base + O_COL0 + (unsigned)t * DV;
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < BKV / 16; ++k)                  // 16 keys are 16 rows of 128 bytes
#pragma unroll
                            for (int part = 0; part < 2; ++part)
                                mma_f16_ts(d, p + part * (BKV / 2) + k * 8, v0d + k * 128, idesc, (j > 0 || part > 0 || k > 0) ? 1u : 0u);
                        mma_commit(bar(B_PVDONE + 2 * t + (j & 1)));
                        if (t == 1 || nb[1] == 0) mma_commit(bar(B_VEMPTY + s));
                    }
                }
            }
        } else if (warp == 2) {
            unsigned phases = 0;                                         // a bit a stage
            for (int j = 0; j < nb_max; ++j) {
                if (!partly_seen(j)) continue;
                const int s = j % KSTAGES;
                if (!mbar_wait_warp(bar(B_VFIX + s), (phases >> s) & 1u, err, 59)) break;
                phases ^= 1u << s;
                if (clean_values(smem + L::V_AT + s * V_BYTES, j == 0 ? rows_before : 0, j == nb_max - 1 ? last_rows : BKV, lane) && lane == 0) *found = 1;
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(B_VFULL + s));
            }
            if (lane == 0) mbar_arrive(bar(B_LOOKED));
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
        const int t = (warp - 4) >> 2, quarter = warp & 3;
        const int r = quarter * 32 + lane;                               // this thread's query row within the tile
        const int pos = pos0 + t * BQ + r, tile_first = pos0 + t * BQ, tile_last = tile_first + BQ - 1;
        const unsigned lane_addr = tmem_base + ((unsigned)(quarter * 32) << 16);
        const unsigned o_addr = lane_addr + O_COL0 + (unsigned)t * DV;
        const int my_nb = t ? nb[1] : nb[0];
        const float sink = sinks ? sinks[h] : -INFINITY;
        bool far = sink > -INFINITY;                                     // the sink is not in m and l
        float m = -INFINITY, l[4] = {0.f, 0.f, 0.f, 0.f};                // m: the reference of the row's exponentials
        bool ok = true;
        for (int j = 0; j < my_nb; ++j) {
            if (!(ok = mbar_wait_warp(bar(B_SFULL + 2 * t + (j & 1)), (unsigned)(j >> 1) & 1u, err, 60))) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned s_addr = lane_addr + (unsigned)(2 * t + (j & 1)) * BKV;
            unsigned s0[32], s1[32];
            tmem_ld32(s_addr, s0);
            tmem_ld32(s_addr + 32, s1);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            const int key0 = key_first + j * BKV;
            // the same for all rows of the tile: the block reaches past its first query, or before its last one's window
            if (key0 + BKV - 1 > tile_first || (window > 0 && key0 <= tile_last - window)) {
                const int upto = pos - key0 + 1, from = window > 0 ? upto - window : 0;
                mask_chunk(s0, 0, from, upto);
                mask_chunk(s1, 32, from, upto);
            }
            const float mx = __fmul_rn(fmaxf(chunk_max(s0), chunk_max(s1)), scale);      // (scale > 0)
            float corr = 1.0f;
            if (far && !(sink - fmaxf(m, mx) > FAR_BELOW)) {
                // the sink joins: what there is is brought to its scale
                far = false;
                corr = m == -INFINITY ? 0.f : ex2((m - sink) * LOG2E);
#pragma unroll
                for (int i = 0; i < 4; ++i) l[i] *= corr;
                l[0] += 1.f;
                m = sink;
            }
            const float mn = fmaxf(m, mx), ref = mn == -INFINITY ? 0.f : mn;
            const float c = m == -INFINITY ? 0.f : ex2(__fmul_rn(__fsub_rn(m, ref), LOG2E));
            m = mn;
            corr *= c;
            float sum[4] = {0.f, 0.f, 0.f, 0.f};
            chunk_weights(s0, scale, ref, s_addr, sum);
            chunk_weights(s1, scale, ref, s_addr + 16, sum);
#pragma unroll
            for (int i = 0; i < 4; ++i) l[i] = fmaf(l[i], c, sum[i]);
            if (j > 0 && __any_sync(0xffffffffu, corr != 1.0f)) {
                // O is the block before's until its product is done
                if (!(ok = mbar_wait_warp(bar(B_PVDONE + 2 * t + ((j - 1) & 1)), (unsigned)((j - 1) >> 1) & 1u, err, 61))) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int d = 0; d < DV; d += 32) {
                    unsigned v[32];
                    tmem_ld32(o_addr + (unsigned)d, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        const float2 x = mul2(make_float2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), make_float2(corr, corr));
                        v[i] = __float_as_uint(x.x);
                        v[i + 1] = __float_as_uint(x.y);
                    }
                    tmem_st32(o_addr + (unsigned)d, v);
                }
            }
            // P written (and O rescaled): tell the MMA warp
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(B_PFULL + 2 * t + (j & 1)));
        }
        if (ok && my_nb > 0) ok = mbar_wait_warp(bar(B_PVDONE + 2 * t + ((my_nb - 1) & 1)), (unsigned)((my_nb - 1) >> 1) & 1u, err, 62);
        if (ok && my_nb > 0) ok = mbar_wait_warp(bar(B_LOOKED), 0, err, 63);
        if (ok && my_nb > 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float den = __fadd_rn(__fadd_rn(l[0], l[1]), __fadd_rn(l[2], l[3])), by;     // the row is O by
            if (far) {
                const float f = exp2f((m - sink) * LOG2E);
                by = f / fmaf(den, f, 1.f);
            } else {
                by = den > 0.f ? 1.f / den : 0.f;
            }
            const bool live = t * BQ + r < nq;
            const size_t n = (size_t)(row0 + (live ? t * BQ + r : 0));
            if (gate && gate_heads) by *= 1.0f / (1.0f + expf(-gate[n * ld_gate + h]));
            const float* g = gate && !gate_heads ? gate + n * ld_gate + (size_t)h * DV : nullptr;
            const bool gate_vec = (((uintptr_t)gate | (uintptr_t)(ld_gate * 4)) & 15) == 0;      // (element by element a block's gates took longer than its softmax)
            __nv_bfloat16* dst = o + (n * nh + h) * DV;
#pragma unroll
            for (int c = 0; c < DV; c += 32) {
                NotFinite seen;
                if (*found && live)
                    for (int j = 0; j < my_nb; ++j) {
                        const int key0 = key_first + j * BKV;
                        if (partly_seen(j))
                            seen = look_up(seen, kx + (long long)(key_row + j * BKV) * ld_kx + v0 + h * DV + c, ld_kx,
                                           window > 0 ? max(0, pos - window + 1 - key0) : 0, min(BKV, pos + 1 - key0), 32);
                    }
                unsigned v[32];
                tmem_ld32(o_addr + (unsigned)c, v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (live) {
                    if (seen.any()) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) + seen.value(i));
                    }
#pragma unroll
                    for (int d = 0; d < 32; d += 8) {
                        float x[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e) x[e] = __uint_as_float(v[d + e]) * by;
                        if (g) {
                            float gl[8];
                            if (gate_vec) {
                                mv_load8(g + c + d, gl);
                            } else {
#pragma unroll
                                for (int e = 0; e < 8; ++e) gl[e] = g[c + d + e];
                            }
#pragma unroll
                            for (int e = 0; e < 8; ++e) x[e] *= 1.0f / (1.0f + expf(-gl[e]));
                        }
                        unsigned w4[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) w4[e] = bits(__floats2bfloat162_rn(x[2 * e], x[2 * e + 1]));
                        *reinterpret_cast<uint4*>(dst + c + d) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
                    }
                }
            }
        }
    }
    // Only now may the next kernel's blocks be given multiprocessors: signalled earlier, they would take the places of this
    // grid's own later blocks and sit there waiting.
    mv_pdl_launch_dependents();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

template <int ROT>
int launch(const void* q, const void* kx, int rows, int ld_kx, int v0, const void* rk, const int* cu, const int* starts,
           const float* sinks, const float* gate, int ld_gate, int gate_heads, void* o, int N, int B, int nh, float scale, int window,
           int* err, cudaStream_t stream) {
    CUtensorMap mq, mqr, mkx, mr;
    if (!tensor_map(q, N, nh * (DIM + ROT), BQ, &mq) || !tensor_map(q, N, nh * (DIM + ROT), BQ, &mqr, ROT) ||
        !tensor_map(kx, rows, ld_kx, BKV, &mkx) || !tensor_map(rk, rows, ROT, BKV, &mr, ROT))
        return (int)cudaErrorInvalidValue;
    const cudaError_t attr = mv_allow_smem<latent_attention_tc_kernel<ROT>>(LtLayout<ROT>::TOTAL);
    if (attr != cudaSuccess) return (int)attr;
    const dim3 grid(nh, (N + TILES * BQ - 1) / (TILES * BQ) + B);      // an upper bound of the pairs; spare blocks return at once
    if (grid.y > 65535u) return (int)cudaErrorInvalidValue;
    latent_attention_tc_kernel<ROT><<<grid, LT_THREADS, LtLayout<ROT>::TOTAL, stream>>>(
        mq, mqr, mkx, mr, (const __nv_bfloat16*)kx, ld_kx, v0, cu, starts, sinks, gate, ld_gate, gate_heads, (__nv_bfloat16*)o, B, nh, scale, window, err);
    return mv_launch_status();
}

}  // namespace

// bfloat16; heads of 64 + rot (32 or 64) channels, values of 64; scale > 0; q, kx and r on 16 bytes, kx's rows (ld_kx) and v0 in
// steps of 8.  `rows`: how many rows kx and r have.
MV_API int mv_latent_attention_tc(const void* q, const void* kx, int rows, int ld_kx, int v0, const void* r, const int* cu,
                                  const int* starts, const float* sinks, const float* gate, int ld_gate, int gate_heads,
                                  void* o, int N, int B, int nh, int rot, float scale, int window, int* err, cudaStream_t stream) {
    if (N <= 0) return 0;
    if ((rot != 32 && rot != 64) || !(scale > 0.f) || rows < 1 || ld_kx % 8 || v0 % 8 || v0 < nh * DIM || ld_kx < v0 + nh * DV || window < 0 ||
        (((uintptr_t)q | (uintptr_t)kx | (uintptr_t)r | (uintptr_t)o) & 15))
        return (int)cudaErrorInvalidValue;
    if (rot == 32) return launch<32>(q, kx, rows, ld_kx, v0, r, cu, starts, sinks, gate, ld_gate, gate_heads, o, N, B, nh, scale, window, err, stream);
    return launch<64>(q, kx, rows, ld_kx, v0, r, cu, starts, sinks, gate, ld_gate, gate_heads, o, N, B, nh, scale, window, err, stream);
}
