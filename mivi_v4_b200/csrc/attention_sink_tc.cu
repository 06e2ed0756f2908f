// attention_sink_prefill.cu's attention (a sink, capped scores, windows that keep the first tokens, chunks, biases by distance, gates) for steps that bring a
// sequence many tokens, on the fifth-generation tensor cores: key sizes up to 128 and value sizes up to 64 in steps of 16, pages of whole blocks of 64
// rows, an even number of heads to a kv head, bfloat16.  The plan is latent_attention_tc.cu's; what differs:
//
//   * the two tiles of a block are 128 query tokens of two heads of one kv head: they walk the same keys, so no tile walks blocks for the other's sake (two
//     tiles of one head's queries 128 apart would both walk a window's 128 more keys), and short sequences fill a block sooner;
//   * keys and values come by TMA straight out of the pages, a block of 64 rows a copy (64 channels a copy; channels beyond a row's end arrive as zeros);
//   * the key blocks are those of the kept first tokens, then those of the window.
//
//   warp 0      TMA: the Q tiles once, then keys and values into rings of four stages each;
//   warp 1      S = Q K^T (128 x 64 x dk);
//   warp 3      O += P V (128 x 64 x 64; with SPLIT twice, P being two bfloat16 numbers), P read from tensor memory;
//   warp 2      looks through the values of the blocks that some row of the tile does not see whole (attention_tc.cuh): rows after the last query become
//               zeros, and so do infinities and NaNs, which would pass through a weight of 0;
//   warps 4-11  softmax, four warps a tile, one query row a thread.
//
// Every sum is added and every score rounded as attention_sink_prefill.cu does it, so that a row's result does not hang on which of the two kernels its
// step took: both kinds of tensor-core instruction add alike; key blocks lie at multiples of 64, and a block that shows a row nothing changes nothing; a
// row's reference is its running maximum after every block; its denominator is four sums, of every eighth key and its neighbour; whether a block lies wholly
// beyond the distance table is decided for the same 16 queries.  (Of values that are not finite the other kernel lets a tile's 64 queries see all that one of them sees.)
//
// Bound by the exponential unit where scores are capped (three of its results a score; 61 % busy over one prompt of 2,048 tokens, two rounds of tiles of unequal length), else by the
// softmax's instructions (schedulers 30 to 35 % busy over the same).  This kernel /
// attention_sink_prefill.cu: one prompt of 2,048 tokens, 32 heads of 80 / 64 in groups of 4, capped, a window of 1,024 75 / 115 us; of 64 with chunks of
// 1,024 32 / 63; capped, a table of 241 distances, split weights 100 / 153.
#include "attention_tc.cuh"

namespace {

constexpr int ST_THREADS = 384;
constexpr int BQ = 128, TILES = 2, BKV = 64, DV = 64, KSTAGES = 4, SBUFS = 4;
constexpr int V_BYTES = BKV * DV * 2;
constexpr int DIST_SMEM = 2048;                    // numbers of a head's distance table that are kept in shared memory at most
constexpr unsigned O_COL0 = SBUFS * BKV;           // tile t: O at O_COL0 + 64 t
constexpr float LOG2E = 1.4426950408889634f;

// PARTS: parts of 64 channels that queries and keys lie in
template <int PARTS> struct StLayout {
    static constexpr int Q_PART = BQ * BK * 2, Q_BYTES = PARTS * Q_PART, K_PART = BKV * BK * 2, K_BYTES = PARTS * K_PART;
    static constexpr int K_AT = TILES * Q_BYTES, V_AT = K_AT + KSTAGES * K_BYTES, BAR_AT = V_AT + KSTAGES * V_BYTES, DIST_AT = BAR_AT + 512;
    static constexpr int TOTAL = DIST_AT + 1024;   // (with the alignment of the start; two heads' distance tables come on top)
};

// barriers, 8 bytes each.  Scores, weights and products have two a tile, by the key block's parity.
enum { B_Q = 0, B_KFULL = 1, B_KEMPTY = B_KFULL + KSTAGES, B_VFULL = B_KEMPTY + KSTAGES, B_VEMPTY = B_VFULL + KSTAGES,
       B_SFULL = B_VEMPTY + KSTAGES, B_PFULL = B_SFULL + 2 * TILES, B_PVDONE = B_PFULL + 2 * TILES, B_VFIX = B_PVDONE + 2 * TILES,
       B_LOOKED = B_VFIX + KSTAGES, B_COUNT };
static_assert(B_COUNT * 8 + 8 <= 512, "barrier area");

__device__ __forceinline__ float rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void tma_load_3d(unsigned dst, const CUtensorMap* map, int x, int y, int z, unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}

__device__ __forceinline__ float2 both(float x) { return make_float2(x, x); }

// 32 scores of a row: scaled and capped, in units of log 2
__device__ __forceinline__ void scale_chunk(unsigned (&s)[32], bool capped, float scale_l, float cap_l, float top) {
    if (capped) {
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
            const float2 y = mul2(make_float2(__uint_as_float(s[i]), __uint_as_float(s[i + 1])), both(scale_l));
            const float2 e = add2(both(1.0f), make_float2(ex2(y.x), ex2(y.y)));
            const float2 x = fma2(both(-2.0f * cap_l), make_float2(rcp(e.x), rcp(e.y)), both(top));
            s[i] = __float_as_uint(x.x);
            s[i + 1] = __float_as_uint(x.y);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
            const float2 x = fma2(make_float2(__uint_as_float(s[i]), __uint_as_float(s[i + 1])), both(scale_l), both(top));
            s[i] = __float_as_uint(x.x);
            s[i + 1] = __float_as_uint(x.y);
        }
    }
}
// n: the row's distance from the chunk's first key
__device__ __forceinline__ void table_chunk(unsigned (&s)[32], const float* by_dist, int last, float unit, int n) {
#pragma unroll
    for (int i = 0; i < 32; ++i)
        if (n - i >= 0) s[i] = __float_as_uint(fmaf(by_dist[min(n - i, last)], unit, __uint_as_float(s[i])));
}
__device__ __forceinline__ void log_chunk(unsigned (&s)[32], float db1, float db2, int n) {
#pragma unroll
    for (int i = 0; i < 32; ++i) s[i] = __float_as_uint(fmaf(-db1, __logf(fmaf(db2, (float)(n - i), 1.0f)), __uint_as_float(s[i])));
}
// scores of the keys from `upto` on, and of those before `from` but not before `keep`, become -inf; the chunk's first key is key c of the block
__device__ __forceinline__ void mask_chunk(unsigned (&s)[32], int c, int from, int keep, int upto) {
#pragma unroll
    for (int i = 0; i < 32; ++i)
        if (c + i >= upto || (c + i < from && c + i >= keep)) s[i] = 0xff800000u;
}
__device__ __forceinline__ float chunk_max(const unsigned (&s)[32]) {
    float a[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int i = 0; i < 32; i += 8)
#pragma unroll
        for (int e = 0; e < 4; ++e) a[e] = fmaxf(a[e], fmaxf(__uint_as_float(s[i + e]), __uint_as_float(s[i + 4 + e])));
    return fmaxf(fmaxf(a[0], a[1]), fmaxf(a[2], a[3]));
}
// the weights of 32 keys of a row into the row's columns p, with SPLIT what the rounding left of them into p + BKV / 2; keys 8 i + 2 t and 8 i + 2 t + 1 are
// added to sum t
template <bool SPLIT>
__device__ __forceinline__ void chunk_weights(const unsigned (&s)[32], float ref, unsigned p, float (&sum)[4]) {
    unsigned hi[16], lo[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float2 x = add2(make_float2(__uint_as_float(s[2 * i]), __uint_as_float(s[2 * i + 1])), both(-ref));
        const float2 w = make_float2(ex2(x.x), ex2(x.y));
        sum[i & 3] = __fadd_rn(sum[i & 3], __fadd_rn(w.x, w.y));
        hi[i] = bits(__floats2bfloat162_rn(w.x, w.y));
        if (SPLIT) {
            const float2 rest = add2(w, make_float2(-__uint_as_float(hi[i] << 16), -__uint_as_float(hi[i] & 0xffff0000u)));
            lo[i] = bits(__floats2bfloat162_rn(rest.x, rest.y));
        }
    }
    tmem_st16(p, hi);
    if (SPLIT) tmem_st16(p + BKV / 2, lo);
}

struct StArgs {
    const int *page_table, *cu, *starts;
    const float *sinks, *gate, *r1, *r2, *dist;
    const __nv_bfloat16* values;                       // the first page's; ld_v a row
    long long page_stride;
    __nv_bfloat16* o;
    float* o_all;
    int* err;
    int table_stride, page_shift, B, nh, nkv, dk, dv, ld_gate, window, keep_first, chunk, dist_len, gate_wide, ld_v;
    float scale, cap;
};

template <int PARTS, bool SPLIT>
__global__ void __launch_bounds__(ST_THREADS, 1)
attention_sink_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                         const __grid_constant__ CUtensorMap map_v, const __grid_constant__ StArgs a) {
    using L = StLayout<PARTS>;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const unsigned q_s = smem_u32(smem), k_s = q_s + L::K_AT, v_s = q_s + L::V_AT;
    unsigned long long* bars = (unsigned long long*)(smem + L::BAR_AT);
    unsigned* tmem_holder = (unsigned*)(bars + B_COUNT);
    volatile int* found = (volatile int*)(tmem_holder + 1);               // warp 2 has met a value that is not finite
    float* dist_s = (float*)(smem + L::DIST_AT);
    const unsigned bar0 = smem_u32(bars);
    auto bar = [&](int i) { return bar0 + 8u * (unsigned)i; };

    // pairs of heads first, then tiles of queries, the late (long) ones of a sequence first
    int b = 0, tile = (int)(gridDim.y - 1 - blockIdx.y);
    for (; b < a.B; ++b) {
        const int tiles = (a.cu[b + 1] - a.cu[b] + BQ - 1) / BQ;
        if (tile < tiles) break;
        tile -= tiles;
    }
    if (b >= a.B) return;
    // with o_all the grid's x counts (pair of heads, kv head whose values are read)
    const int h0 = TILES * (a.o_all ? (int)blockIdx.x / a.nkv : (int)blockIdx.x), g = h0 / (a.nh / a.nkv);
    const int vg = a.o_all ? (int)blockIdx.x % a.nkv : g;
    const int row0 = a.cu[b] + tile * BQ;
    const int nq = min(BQ, a.cu[b + 1] - row0);
    const int pos0 = a.starts[b] + tile * BQ, last_pos = pos0 + nq - 1;
    const int first_key = a.chunk > 0 ? pos0 - pos0 % a.chunk : (a.window > 0 ? max(0, pos0 - a.window + 1) : 0);
    const int kb_begin = first_key / BKV, kb_end = last_pos / BKV + 1;
    const int n_kept = (a.chunk == 0 && a.window > 0 && a.keep_first > 0) ? min((a.keep_first + BKV - 1) / BKV, kb_begin) : 0;
    const int n_iter = n_kept + kb_end - kb_begin;
    auto block_of = [&](int j) { return j < n_kept ? j : kb_begin + (j - n_kept); };
    const int last_rows = last_pos + 1 - (kb_end - 1) * BKV;             // rows of the last block up to the last query's
    const int keep = a.chunk == 0 && a.window > 0 ? a.keep_first : 0;
    // some row of the tile does not see all of block j: from the block on that reaches past the first query, from the last kept block on to where the last
    // query's window or chunk starts (a block with rows after the last query is one of these)
    const int last_from = a.chunk > 0 ? last_pos - last_pos % a.chunk : a.window > 0 ? max(0, last_pos - a.window + 1) : 0;
    const int seen_to = n_kept + (pos0 + 1) / BKV - kb_begin, kept_to = min(keep / BKV, n_kept);
    const int seen_from = n_kept + max(0, (last_from + BKV - 1) / BKV - kb_begin);
    auto partly_seen = [&](int j) { return j >= seen_to || (j >= kept_to && j < seen_from); };
    const int* table = a.page_table + (size_t)b * a.table_stride;
    const int page_size = 1 << a.page_shift;
    const int warp = warp_index(), lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int i = 0; i < B_COUNT; ++i) mbar_init(bar(i), i >= B_PFULL && i < B_PFULL + 2 * TILES ? 4 : 1);
        *found = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (a.dist && a.dist_len <= DIST_SMEM)
        for (int i = threadIdx.x; i < TILES * a.dist_len; i += ST_THREADS) dist_s[i] = a.dist[(size_t)h0 * a.dist_len + i] * LOG2E;
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
                for (int t = 0; t < TILES; ++t)
                    for (int p = 0; p < PARTS; ++p) tma_load_3d(q_s + t * L::Q_BYTES + p * L::Q_PART, &map_q, p * BK, h0 + t, row0, bar(B_Q));
            }
            for (int j = 0; j < n_iter; ++j) {
                const int s = j % KSTAGES, t0 = block_of(j) * BKV;
                const unsigned ph = (unsigned)(j / KSTAGES) & 1u;
                const int page = mv_read_page(table[t0 >> a.page_shift]), in_page = t0 & (page_size - 1);
                if (!mbar_wait_warp(bar(B_KEMPTY + s), ph ^ 1u, a.err, 81)) break;
                if (elect_one()) {
                    mbar_expect_tx(bar(B_KFULL + s), L::K_BYTES);
                    for (int p = 0; p < PARTS; ++p)
                        tma_load_3d(k_s + s * L::K_BYTES + p * L::K_PART, &map_k, p * BK, g * page_size + in_page, page, bar(B_KFULL + s));
                }
                if (!mbar_wait_warp(bar(B_VEMPTY + s), ph ^ 1u, a.err, 82)) break;
                // blocks that are partly seen go by way of warp 2, which then says that they are there
                const unsigned full = bar((partly_seen(j) ? B_VFIX : B_VFULL) + s);
                if (elect_one()) {
                    mbar_expect_tx(full, V_BYTES);
                    tma_load_3d(v_s + s * V_BYTES, &map_v, 0, vg * page_size + in_page, page, full);
                }
            }
        } else if (warp == 1) {
            // S(t, j) = Q_t K_j^T as soon as the keys are there and the buffer's weights, those of the tile's block before the last, are used
            const unsigned idesc = instr_desc(BQ, BKV);
            const int steps = a.dk / 16;
            bool ok = mbar_wait_warp(bar(B_Q), 0, a.err, 83);
            for (int j = 0; j < n_iter && ok; ++j) {
                const int s = j % KSTAGES;
                if (!(ok = mbar_wait_warp(bar(B_KFULL + s), (unsigned)(j / KSTAGES) & 1u, a.err, 84))) break;
#pragma unroll
                for (int t = 0; t < TILES; ++t) {
                    if (!ok) continue;
                    if (j > 1 && !(ok = mbar_wait_warp(bar(B_PVDONE + 2 * t + (j & 1)), (unsigned)((j - 2) >> 1) & 1u, a.err, 85))) continue;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const unsigned d = tmem_base + (unsigned)(2 * t + (j & 1)) * BKV;
                    const unsigned qa = q_s + t * L::Q_BYTES, ka = k_s + s * L::K_BYTES;
                    if (elect_one()) {
#pragma unroll
                        for (int p = 0; p < PARTS; ++p) {
                            const unsigned long long qd = smem_desc(qa + p * L::Q_PART), kd = smem_desc(ka + p * L::K_PART);
                            // 16 channels are 32 bytes, two units of a descriptor's address
#pragma unroll
                            for (int k = 0; k < BK / 16; ++k)
                                if (p * (BK / 16) + k < steps) mma_f16(d, qd + 2 * k, kd + 2 * k, idesc, p > 0 || k > 0 ? 1u : 0u);
                        }
                        mma_commit(bar(B_SFULL + 2 * t + (j & 1)));
                        if (t == 1) mma_commit(bar(B_KEMPTY + s));
                    }
                }
            }
        } else if (warp == 3) {
            const unsigned idesc = instr_desc(BQ, DV) | (1u << 16);                 // V as it lies, a row a key: MN-major
            bool ok = true;
            for (int j = 0; j < n_iter && ok; ++j) {
                const int s = j % KSTAGES;
                if (!(ok = mbar_wait_warp(bar(B_VFULL + s), (unsigned)(j / KSTAGES) & 1u, a.err, 86))) break;
                const unsigned long long v0d = smem_desc(v_s + s * V_BYTES);
#pragma unroll
                for (int t = 0; t < TILES; ++t) {
                    if (!ok) continue;
                    if (!(ok = mbar_wait_warp(bar(B_PFULL + 2 * t + (j & 1)), (unsigned)(j >> 1) & 1u, a.err, 88))) continue;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const unsigned p = tmem_base + (unsigned)(2 * t + (j & 1)) * BKV, d = tmem_base + O_COL0 + (unsigned)t * DV;
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < BKV / 16; ++k)                  // 16 keys are 16 rows of 128 bytes
#pragma unroll
                            for (int part = 0; part < (SPLIT ? 2 : 1); ++part)
                                mma_f16_ts(d, p + part * (BKV / 2) + k * 8, v0d + k * 128, idesc, (j > 0 || part > 0 || k > 0) ? 1u : 0u);
                        mma_commit(bar(B_PVDONE + 2 * t + (j & 1)));
                        if (t == 1) mma_commit(bar(B_VEMPTY + s));
                    }
                }
            }
        } else if (warp == 2) {
            unsigned phases = 0;                                         // a bit a stage
            for (int j = 0; j < n_iter; ++j) {
                if (!partly_seen(j)) continue;
                const int s = j % KSTAGES;
                if (!mbar_wait_warp(bar(B_VFIX + s), (phases >> s) & 1u, a.err, 89)) break;
                phases ^= 1u << s;
                if (clean_values(smem + L::V_AT + s * V_BYTES, 0, j == n_iter - 1 ? last_rows : BKV, lane) && lane == 0) *found = 1;
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(B_VFULL + s));
            }
            if (lane == 0) mbar_arrive(bar(B_LOOKED));
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
        const int t = (warp - 4) >> 2, quarter = warp & 3, h = h0 + t;
        const int r = quarter * 32 + lane;                               // this thread's query row within the tile
        const int pos = pos0 + r, tile_last = pos0 + BQ - 1;
        const unsigned lane_addr = tmem_base + ((unsigned)(quarter * 32) << 16);
        const unsigned o_addr = lane_addr + O_COL0 + (unsigned)t * DV;
        // scores, maxima and biases are held in units of log 2: the weights are powers of two then
        const bool capped = a.cap > 0.f;
        const float cap_l = a.cap * LOG2E, scale_l = capped ? 2.0f * LOG2E * a.scale / a.cap : a.scale * LOG2E;
        const float db1 = a.r1 ? a.r1[h] * LOG2E : 0.f, db2 = a.r1 ? a.r2[h] : 0.f;
        const float* by_dist = a.dist ? a.dist + (size_t)h * a.dist_len : nullptr;
        const float beyond = a.dist ? by_dist[a.dist_len - 1] * LOG2E : 0.f;
        const float dist_unit = a.dist_len <= DIST_SMEM ? 1.0f : LOG2E;
        const int pos16 = pos0 + (r & ~15);                              // the first of the 16 queries that share the choice of the far end
        const int from_pos = a.chunk > 0 ? pos - pos % a.chunk : (a.window > 0 ? pos - a.window + 1 : 0);
        const int masked_to = a.chunk > 0 ? tile_last - tile_last % a.chunk : (a.window > 0 ? tile_last - a.window + 1 : 0);
        float m = a.sinks ? a.sinks[h] * LOG2E : -INFINITY;              // the reference of the row's exponentials; a sink starts it
        float l[4] = {a.sinks ? 1.f : 0.f, 0.f, 0.f, 0.f};
        bool ok = true;
        for (int j = 0; j < n_iter; ++j) {
            if (!(ok = mbar_wait_warp(bar(B_SFULL + 2 * t + (j & 1)), (unsigned)(j >> 1) & 1u, a.err, 90))) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned s_addr = lane_addr + (unsigned)(2 * t + (j & 1)) * BKV;
            unsigned s0[32], s1[32];
            tmem_ld32(s_addr, s0);
            tmem_ld32(s_addr + 32, s1);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            const int key0 = block_of(j) * BKV, n = pos - key0;
            const bool near = a.dist != nullptr && pos16 - (key0 + BKV - 1) < a.dist_len - 1;
            const float add = a.dist != nullptr && !near ? beyond : 0.f;
            const float top = capped ? fmaf(a.cap, LOG2E, add) : add;
            scale_chunk(s0, capped, scale_l, cap_l, top);
            scale_chunk(s1, capped, scale_l, cap_l, top);
            if (near) {
                if (a.dist_len <= DIST_SMEM) {
                    const float* row = dist_s + t * a.dist_len;
                    table_chunk(s0, row, a.dist_len - 1, 1.0f, n);
                    table_chunk(s1, row, a.dist_len - 1, 1.0f, n - 32);
                } else {
                    table_chunk(s0, by_dist, a.dist_len - 1, dist_unit, n);
                    table_chunk(s1, by_dist, a.dist_len - 1, dist_unit, n - 32);
                }
            } else if (a.r1) {
                log_chunk(s0, db1, db2, n);
                log_chunk(s1, db1, db2, n - 32);
            }
            // the same for all rows of the tile: the block reaches past its first query, or before what its last one sees
            if (j < n_kept || key0 + BKV - 1 > pos0 || key0 < masked_to) {
                mask_chunk(s0, 0, from_pos - key0, keep - key0, n + 1);
                mask_chunk(s1, 32, from_pos - key0, keep - key0, n + 1);
            }
            const float mn = fmaxf(m, fmaxf(chunk_max(s0), chunk_max(s1))), ref = mn == -INFINITY ? 0.f : mn;
            const float c = m == -INFINITY ? 0.f : ex2(__fsub_rn(m, ref));
            m = mn;
            float sum[4] = {0.f, 0.f, 0.f, 0.f};
            chunk_weights<SPLIT>(s0, ref, s_addr, sum);
            chunk_weights<SPLIT>(s1, ref, s_addr + 16, sum);
#pragma unroll
            for (int i = 0; i < 4; ++i) l[i] = fmaf(l[i], c, sum[i]);
            if (j > 0 && __any_sync(0xffffffffu, c != 1.0f)) {
                // O is the block before's until its product is done
                if (!(ok = mbar_wait_warp(bar(B_PVDONE + 2 * t + ((j - 1) & 1)), (unsigned)((j - 1) >> 1) & 1u, a.err, 91))) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int d = 0; d < DV; d += 32) {
                    unsigned v[32];
                    tmem_ld32(o_addr + (unsigned)d, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        const float2 x = mul2(make_float2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])), both(c));
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
        if (ok) ok = mbar_wait_warp(bar(B_PVDONE + 2 * t + ((n_iter - 1) & 1)), (unsigned)((n_iter - 1) >> 1) & 1u, a.err, 92);
        if (ok) ok = mbar_wait_warp(bar(B_LOOKED), 0, a.err, 93);
        if (ok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const bool live = r < nq;
            const size_t row = (size_t)(row0 + (live ? r : 0));
            float by = 1.0f / __fadd_rn(__fadd_rn(l[0], l[1]), __fadd_rn(l[2], l[3]));
            if (a.gate && !a.gate_wide) by *= 1.0f / (1.0f + expf(-a.gate[row * a.ld_gate + h]));
            const float* gr = a.gate && a.gate_wide ? a.gate + row * a.ld_gate + (size_t)h * a.dv : nullptr;
            const bool gate_vec = (((uintptr_t)a.gate | (uintptr_t)(a.ld_gate * 4)) & 15) == 0;
            __nv_bfloat16* dst = a.o_all ? nullptr : a.o + (row * a.nh + h) * a.dv;
            float* dst_all = a.o_all ? a.o_all + ((row * a.nh + h) * a.nkv + vg) * a.dv : nullptr;
#pragma unroll
            for (int c = 0; c < DV; c += 32) {
                NotFinite seen;
                if (*found && live && c < a.dv)
                    for (int j = 0; j < n_iter; ++j) {
                        if (!partly_seen(j)) continue;
                        const int key0 = block_of(j) * BKV, upto = min(BKV, pos + 1 - key0), n = min(32, a.dv - c);
                        const __nv_bfloat16* rows = a.values + (size_t)mv_read_page(table[key0 >> a.page_shift]) * a.page_stride +
                                                    (size_t)(vg * page_size + (key0 & (page_size - 1))) * a.ld_v + c;
                        seen = look_up(seen, rows, a.ld_v, 0, min(keep - key0, upto), n);
                        seen = look_up(seen, rows, a.ld_v, max(0, from_pos - key0), upto, n);
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
                        if (c + d < a.dv) {
                            float x[8];
#pragma unroll
                            for (int e = 0; e < 8; ++e) x[e] = __uint_as_float(v[d + e]) * by;
                            if (gr) {
                                float gl[8];
                                if (gate_vec) {
                                    mv_load8(gr + c + d, gl);
                                } else {
#pragma unroll
                                    for (int e = 0; e < 8; ++e) gl[e] = gr[c + d + e];
                                }
#pragma unroll
                                for (int e = 0; e < 8; ++e) x[e] *= 1.0f / (1.0f + expf(-gl[e]));
                            }
                            if (a.o_all) {
                                *reinterpret_cast<float4*>(dst_all + c + d) = make_float4(x[0], x[1], x[2], x[3]);
                                *reinterpret_cast<float4*>(dst_all + c + d + 4) = make_float4(x[4], x[5], x[6], x[7]);
                            } else {
                                unsigned w4[4];
#pragma unroll
                                for (int e = 0; e < 4; ++e) w4[e] = bits(__floats2bfloat162_rn(x[2 * e], x[2 * e + 1]));
                                *reinterpret_cast<uint4*>(dst + c + d) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
                            }
                        }
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

// [planes][rows][cols] of bfloat16, rows cols apart and planes `plane` elements, read in boxes of 64 columns by box_rows rows by box_planes planes
bool tensor_map_3d(const void* ptr, int planes, int rows, int cols, long long plane, int box_rows, int box_planes, CUtensorMap* out) {
    EncodeTiled enc = encoder();
    if (!enc) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)planes};
    const cuuint64_t strides[2] = {(cuuint64_t)cols * 2, (cuuint64_t)plane * 2};
    const cuuint32_t box[3] = {(cuuint32_t)BK, (cuuint32_t)box_rows, (cuuint32_t)box_planes};
    const cuuint32_t elem[3] = {1, 1, 1};
    return enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int PARTS, bool SPLIT>
int launch(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const StArgs& a, dim3 grid, cudaStream_t stream) {
    const int tables = a.dist && a.dist_len <= DIST_SMEM ? TILES * a.dist_len * (int)sizeof(float) : 0;
    const cudaError_t attr = mv_allow_smem<attention_sink_tc_kernel<PARTS, SPLIT>>(StLayout<PARTS>::TOTAL + TILES * DIST_SMEM * (int)sizeof(float));
    if (attr != cudaSuccess) return (int)attr;
    attention_sink_tc_kernel<PARTS, SPLIT><<<grid, ST_THREADS, StLayout<PARTS>::TOTAL + tables, stream>>>(mq, mk, mv, a);
    return mv_launch_status();
}

}  // namespace

MV_GUARD_SETTER(attention_sink_tc)

// bfloat16; dk up to 128 and dv up to 64 in steps of 16, page_size a power of two of at least 64, nh / nkv even; q and the pool on 16 bytes, page_stride in
// steps of 8.
MV_API int mv_attention_sink_tc(const void* q, const void* pool, int n_pages, long long page_stride, const int* page_table,
                                int table_stride, int page_size, const int* cu, const int* starts,
                                const float* sinks, const float* gate, int ld_gate, void* o, int N, int B, int nh,
                                int nkv, int dk, int dv, float scale, float cap, int window, int keep_first,
                                int chunk, const float* r1, const float* r2, const float* dist, int dist_len, int v_in_k,
                                int gate_wide, float* o_all, int split, int* err, cudaStream_t stream) {
    if (N <= 0) return 0;
    if (nkv < 1 || nh % (TILES * nkv) || page_size < BKV || (page_size & (page_size - 1)) || dk % 16 || dv % 16 || dk < 16 || dv < 16 || dk > 2 * BK ||
        dv > DV || (v_in_k && dv > dk) || (r1 && !r2) || (dist && (dist_len < 1 || r1)) || n_pages < 1 || page_stride % 8 ||
        (((uintptr_t)q | (uintptr_t)pool | (uintptr_t)o | (uintptr_t)o_all) & 15))
        return (int)cudaErrorInvalidValue;
    const long long rows = (long long)nkv * page_size;
    CUtensorMap mq, mk, mv;
    const __nv_bfloat16* values = (const __nv_bfloat16*)pool + (v_in_k ? 0 : rows * dk);
    if (!tensor_map_3d(q, N, nh, dk, (long long)nh * dk, 1, BQ, &mq) || !tensor_map_3d(pool, n_pages, (int)rows, dk, page_stride, BKV, 1, &mk) ||
        !tensor_map_3d(values, n_pages, (int)rows, v_in_k ? dk : dv, page_stride, BKV, 1, &mv))
        return (int)cudaErrorInvalidValue;
    int page_shift = 0;
    while ((1 << page_shift) < page_size) ++page_shift;
    const dim3 grid(nh / TILES * (o_all ? nkv : 1), (N + BQ - 1) / BQ + B);      // an upper bound of the tiles; spare blocks return at once
    if (grid.y > 65535u) return (int)cudaErrorInvalidValue;
    const StArgs a = {page_table, cu, starts, sinks, gate, r1, r2, dist, values, page_stride, (__nv_bfloat16*)o, o_all, err, table_stride, page_shift,
                      B, nh, nkv, dk, dv, ld_gate, window, keep_first, chunk, dist_len, gate_wide, v_in_k ? dk : dv, scale, cap};
    if (dk <= BK) return split ? launch<1, true>(mq, mk, mv, a, grid, stream) : launch<1, false>(mq, mk, mv, a, grid, stream);
    return split ? launch<2, true>(mq, mk, mv, a, grid, stream) : launch<2, false>(mq, mk, mv, a, grid, stream);
}
