// Y[M, N] = X[M, K] . W[N, K]^T of float32 operands on the tensor cores, for products of many rows.
//
// Every operand, times 2^39, is split into three bfloat16 numbers, h + m + l (each what rounding left of the one before; together its 24 bits), and
// six of the nine products are added up: h h, then h m + m h, m m, h l + l h; what is left out is below 2^-25 of |x w|.  The tensor cores cut
// off what they add, to the last place of the largest number there is: a long chain of it loses places (K = 1,024 in one: 1e-6), and where all terms have one sign the loss adds up.  So h h
// is added over 64 of K in tensor memory and then in float32 registers; the five others, 2^-8 of it, have an accumulator of their own over all of K.
//
// Error against 64 bits in the 2-norm, 256 x 512, this kernel / float32 multiply-adds (gemm_simt.cu), 1e-7, at K = 1,024 | 2,048 | 4,608: terms of both signs 1.1 / 1.6 | 1.3 / 2.1 | 1.8 / 3.1;
// of one sign 1.1 / 0.6 | 1.2 / 0.7 | 1.5 / 0.8; X with magnitudes spread over e^9 (sigma of the logarithm 3) 1.5 / 1.3 | 1.2 / 1.4 | 2.2 / 3.1, and with W of one
// sign 3.5 / 1.1 | 4.0 / 2.5 | 3.6 / 3.2.  Model weights have both signs: there it is the more exact of the two, where all terms have one sign the less exact, by half of float32's
// last place.  (Runs of 128 of K: both signs 1.3 | 1.5 | 1.8, one sign 1.8 | 1.8 | 1.9, the last form 7.0 | 9.7 | 8.2, in the same time.  Runs that begin at minus half of what they will add, with what the
// sum's rounding left, 0.9 and 0.5 | 0.5 | 0.5: the products take 16 to 23 % longer.)
//
// Block = a tile of 128 rows of X by TN of W, 32 of K at a time:
//   warp 0       TMA: the float32 tiles of X and W into a ring of four stages;
//   warp 1       the products, twelve 128 x TN x 16 a stage;
//   warps 4-7    add the finished 64 of K of h h (two accumulators take turns) to their registers, TN columns of a row a thread;
//   warps 8-15   split X, a row a thread, out of a stage of the ring into tensor memory, from where the products read it;
//   warps 16-23  split W, a row a thread, into shared memory, in the layout that the products read.
// At the end the tile goes through shared memory, is multiplied by 2^-78, and all warps store it by rows.  The scale keeps all parts of all float32 numbers in bfloat16's range, down
// to the smallest subnormal one (without it what is left of a number below 2^-110 after its first eight bits falls out, which shows beside large numbers in the other operand).  Infinities,
// NaNs, operands from 2^88 on and sums from 2^50 on end as results that are not finite: these, and no others, are worked out again by float32
// multiply-adds, in a function of its own that leaves the others' way its registers.
//
// Bound by the splitting and its waits (720 instructions of every scheduler in a stage's 1,375 clocks for 128 x 128, 580 in 1,060 for 128 x 96; tensor cores busy 55 and 41 %), then by
// shared memory (a stage of 128 columns writes and reads 32 KB of float32 tiles, writes 24 KB and has the products read 48 KB of W's planes: 1,060 clocks at 128 bytes a clock).  1,165 rows against 9,216 x 1,024 516 -> 129 us (170 TFLOP/s), against 1,024 x 4,608 280 -> 86.  With X's planes in shared memory too, which the products then read at all
// its bandwidth, 174 us; with the two groups of splitting warps on the same stage 145.
#include "tc_common.cuh"

namespace {

constexpr int F3_THREADS = 768;
constexpr int TM = 128, KB = 32, RAW = 4, CHUNK = 2;     // CHUNK stages of KB: how long h h is added up in tensor memory
constexpr int X_BYTES = TM * KB * 4;
constexpr unsigned X_PLANE = KB / 2;                                 // columns of tensor memory

template <int TN> struct F3Layout {
    static constexpr int RAW_STAGE = X_BYTES + TN * KB * 4, PLANE = TN * KB * 2, PLANE_STAGE = 3 * PLANE;
    // tensor memory: two accumulators of h h, one of the others, and X's planes in two stages or four
    static constexpr unsigned LOW_COL = 2 * TN, X_COL = 3 * TN;
    static constexpr int PLANES = 512 - 3 * TN >= 4 * 3 * (int)X_PLANE ? 4 : 2;
    static constexpr int PLANES_AT = RAW * RAW_STAGE, BARS_AT = PLANES_AT + PLANES * PLANE_STAGE, TOTAL = BARS_AT + 256 + 1024;
    static constexpr int OUT_LD = TN + 4;                            // the tile at the end: 16-byte words of 8 rows in 8 bank groups
    static_assert(TN % 16 == 0 && TN <= 128 && TM * OUT_LD * 4 <= BARS_AT, "the tile fits the rings");
};
constexpr float SCALE = 549755813888.0f, UNSCALE = 3.3087224502121107e-24f;      // 2^39, 2^-78

constexpr int MAX_PLANES = 4;
enum { B_RAWFULL = 0, B_RAWEMPTY = B_RAWFULL + RAW, B_PLFULL = B_RAWEMPTY + RAW, B_PLEMPTY = B_PLFULL + MAX_PLANES, B_ACCFULL = B_PLEMPTY + MAX_PLANES,
       B_ACCEMPTY = B_ACCFULL + 2, B_COUNT = B_ACCEMPTY + 2 };
static_assert(B_COUNT * 8 + 8 <= 256, "barrier area");

// a packed pair's bfloat16 numbers as floats, and what they leave of (a, b)
__device__ __forceinline__ float2 rest(float2 x, unsigned h) {
    float2 y = make_float2(__uint_as_float(h << 16), __uint_as_float(h & 0xffff0000u)), minus = make_float2(-1.f, -1.f);
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(*reinterpret_cast<unsigned long long*>(&y)), "l"(*reinterpret_cast<unsigned long long*>(&minus)),
        "l"(*reinterpret_cast<unsigned long long*>(&x)));
    return *reinterpret_cast<float2*>(&r);
}
// two floats times SCALE -> their three bfloat16 numbers, packed by plane
__device__ __forceinline__ void split2(float2 a, unsigned& h, unsigned& m, unsigned& l) {
    const float2 x = mul2(a, make_float2(SCALE, SCALE));
    h = bits(__floats2bfloat162_rn(x.x, x.y));
    const float2 y = rest(x, h);
    m = bits(__floats2bfloat162_rn(y.x, y.y));
    const float2 z = rest(y, m);
    l = bits(__floats2bfloat162_rn(z.x, z.y));
}

struct F3Args {
    const float *X, *W, *bias;
    void* out;
    int mode, M, N, K, ldo;
    __device__ __forceinline__ void put(size_t o, int n, float v) const {
        if (bias) v += bias[n];
        if (mode == 1) ((__nv_bfloat16*)out)[o] = __float2bfloat16_rn(v);
        else ((float*)out)[o] = mode == 2 ? ((float*)out)[o] + v : v;
    }
};
__device__ __forceinline__ bool finite4(float4 v) { return fabsf(v.x) + fabsf(v.y) + fabsf(v.z) + fabsf(v.w) < INFINITY; }
// A thread's results that are not finite, by multiply-adds, K in its order.
template <int TN>
__device__ __noinline__ void multiply_again(const F3Args& g, const float* tile, int m0, int n0) {
    const int lane = threadIdx.x & 31, n = n0 + 4 * lane;
    for (int r = threadIdx.x >> 5; r < TM && m0 + r < g.M; r += F3_THREADS / 32) {
        const float* at = tile + r * F3Layout<TN>::OUT_LD + 4 * lane;
        if (finite4(*reinterpret_cast<const float4*>(at))) continue;
        for (int e = 0; e < 4 && n + e < g.N; ++e) {
            float v = at[e];
            if (!(fabsf(v) < INFINITY)) {
                const float *x = g.X + (size_t)(m0 + r) * g.K, *w = g.W + (size_t)(n + e) * g.K;
                v = 0.f;
                for (int k = 0; k < g.K; k += 4) {
                    const float4 a = *reinterpret_cast<const float4*>(x + k), b = *reinterpret_cast<const float4*>(w + k);
                    v = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, v))));
                }
            }
            g.put((size_t)(m0 + r) * g.ldo + n + e, n + e, v);
        }
    }
}

template <int TN>
__global__ void __launch_bounds__(F3_THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ F3Args g,
                   int* __restrict__ err) {
    using L = F3Layout<TN>;
    constexpr int PLANES = L::PLANES;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned long long* bars = (unsigned long long*)(smem + L::BARS_AT);
    unsigned* tmem_holder = (unsigned*)(bars + B_COUNT);
    const unsigned base = smem_u32(smem), bar0 = smem_u32(bars);
    auto bar = [&](int i) { return bar0 + 8u * (unsigned)i; };
    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
    const int nkb = (g.K + KB - 1) / KB, chunks = (nkb + CHUNK - 1) / CHUNK;

    if (threadIdx.x == 0) {
        for (int i = 0; i < B_COUNT; ++i) {
            const bool split = (i >= B_RAWEMPTY && i < B_RAWEMPTY + RAW) || (i >= B_PLFULL && i < B_PLFULL + MAX_PLANES);
            mbar_init(bar(i), split ? 8 : i >= B_ACCEMPTY ? 4 : 1);
        }
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
    float* tile = reinterpret_cast<float*>(smem);
    bool ok = true;

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
        if (warp == 0) {
            for (int kb = 0; kb < nkb; ++kb) {
                const int s = kb % RAW;
                if (!mbar_wait_warp(bar(B_RAWEMPTY + s), ((unsigned)(kb / RAW) & 1u) ^ 1u, err, 71)) break;
                const unsigned dst = base + s * L::RAW_STAGE;
                if (elect_one()) {
                    mbar_expect_tx(bar(B_RAWFULL + s), L::RAW_STAGE);
                    tma_load_2d(dst, &map_x, kb * KB, m0, bar(B_RAWFULL + s));
                    tma_load_2d(dst + X_BYTES, &map_w, kb * KB, n0, bar(B_RAWFULL + s));
                }
            }
        } else if (warp == 1) {
            const unsigned idesc = instr_desc(TM, TN);
            for (int kb = 0; kb < nkb; ++kb) {
                const int s = kb % PLANES, chunk = kb / CHUNK, acc = chunk & 1;
                const bool first = kb % CHUNK == 0;
                if (first && !mbar_wait_warp(bar(B_ACCEMPTY + acc), ((unsigned)(chunk >> 1) & 1u) ^ 1u, err, 72)) break;
                if (!mbar_wait_warp(bar(B_PLFULL + s), (unsigned)(kb / PLANES) & 1u, err, 73)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned p = base + L::PLANES_AT + s * L::PLANE_STAGE;
                const unsigned long long wh = smem_desc_64(p), wm = smem_desc_64(p + L::PLANE), wl = smem_desc_64(p + 2 * L::PLANE);
                const unsigned xh = tmem_base + L::X_COL + (unsigned)s * 3 * X_PLANE, xm = xh + X_PLANE, xl = xm + X_PLANE;
                const unsigned d = tmem_base + (unsigned)acc * TN, e = tmem_base + L::LOW_COL;
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < KB / 16; ++k) {       // 16 of K: 8 columns of tensor memory; 32 bytes, two units of a descriptor's address
                        mma_f16_ts(e, xh + 8 * k, wl + 2 * k, idesc, kb > 0 || k > 0 ? 1u : 0u);
                        mma_f16_ts(e, xl + 8 * k, wh + 2 * k, idesc, 1u);
                        mma_f16_ts(e, xm + 8 * k, wm + 2 * k, idesc, 1u);
                        mma_f16_ts(e, xh + 8 * k, wm + 2 * k, idesc, 1u);
                        mma_f16_ts(e, xm + 8 * k, wh + 2 * k, idesc, 1u);
                        mma_f16_ts(d, xh + 8 * k, wh + 2 * k, idesc, !first || k > 0 ? 1u : 0u);
                    }
                    mma_commit(bar(B_PLEMPTY + s));
                    if (kb % CHUNK == CHUNK - 1 || kb == nkb - 1) mma_commit(bar(B_ACCFULL + acc));
                }
            }
        }
    } else if (warp < 8) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
        const int quarter = warp & 3, r = quarter * 32 + lane;
        const unsigned lane_addr = tmem_base + ((unsigned)(quarter * 32) << 16);
        float2 sum[TN / 2];
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) sum[j] = make_float2(0.f, 0.f);
        auto add = [&](unsigned col) {
#pragma unroll
            for (int c = 0; c < TN; c += 16) {
                unsigned v[16];
                tmem_ld16(lane_addr + col + (unsigned)c, v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int j = 0; j < 8; ++j) sum[c / 2 + j] = add2(sum[c / 2 + j], make_float2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])));
            }
        };
        for (int chunk = 0; chunk < chunks; ++chunk) {
            const int acc = chunk & 1;
            if (!(ok = mbar_wait_warp(bar(B_ACCFULL + acc), (unsigned)(chunk >> 1) & 1u, err, 74))) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            add((unsigned)acc * TN);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(B_ACCEMPTY + acc));
        }
        if (ok) {
            // all products are done, and with them all reading of the rings
            add(L::LOW_COL);
#pragma unroll
            for (int j = 0; j < TN; j += 4)
                *reinterpret_cast<float4*>(tile + r * L::OUT_LD + j) =
                    make_float4(sum[j / 2].x * UNSCALE, sum[j / 2].y * UNSCALE, sum[j / 2 + 1].x * UNSCALE, sum[j / 2 + 1].y * UNSCALE);
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        // Two groups of four warps for X and two for W take turns stage by stage, so that one's waits run under the other's arithmetic (all of them on
        // half a row of the same stage: 1,200 clocks a stage whatever TN).  Both rings have an even number of stages: a group sees every phase of its barriers.
        const bool is_x = warp < 16;
        const int r = (warp & 3) * 32 + lane, group = (warp >> 2) & 1;     // this thread's row of the tile of X or W
        const bool live = is_x || r < TN;
        const unsigned at0 = tmem_base + ((unsigned)((warp & 3) * 32) << 16) + L::X_COL;
        for (int kb = group; kb < nkb; kb += 2) {
            const int s = kb % RAW, d = kb % PLANES;
            if (!mbar_wait_warp(bar(B_RAWFULL + s), (unsigned)(kb / RAW) & 1u, err, 75)) break;
            // 16-byte word w of 8 a row lies at w ^ (r % 8); in a plane word q of 4 at q ^ (r / 2 % 4)
            const unsigned char* src = smem + s * L::RAW_STAGE + (is_x ? 0 : X_BYTES) + r * 128;
            unsigned char* dst = smem + L::PLANES_AT + d * L::PLANE_STAGE + r * 64;
            const unsigned at = at0 + (unsigned)d * 3 * X_PLANE;
            bool free = true;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                unsigned h[8], m[8], l[8];
                if (live) {
#pragma unroll
                    for (int w = 0; w < 4; ++w) {
                        const float4 a = *reinterpret_cast<const float4*>(src + (((4 * half + w) ^ (r & 7)) << 4));
                        split2(make_float2(a.x, a.y), h[2 * w], m[2 * w], l[2 * w]);
                        split2(make_float2(a.z, a.w), h[2 * w + 1], m[2 * w + 1], l[2 * w + 1]);
                    }
                }
                if (half == 0) {
                    free = mbar_wait_warp(bar(B_PLEMPTY + d), ((unsigned)(kb / PLANES) & 1u) ^ 1u, err, 76);
                    if (!free) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                }
                if (is_x) {
                    tmem_st8(at + 8 * half, h);
                    tmem_st8(at + 8 * half + X_PLANE, m);
                    tmem_st8(at + 8 * half + 2 * X_PLANE, l);
                } else if (live) {
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        unsigned char* to = dst + (((2 * half + q) ^ ((r >> 1) & 3)) << 4);
                        *reinterpret_cast<uint4*>(to) = make_uint4(h[4 * q], h[4 * q + 1], h[4 * q + 2], h[4 * q + 3]);
                        *reinterpret_cast<uint4*>(to + L::PLANE) = make_uint4(m[4 * q], m[4 * q + 1], m[4 * q + 2], m[4 * q + 3]);
                        *reinterpret_cast<uint4*>(to + 2 * L::PLANE) = make_uint4(l[4 * q], l[4 * q + 1], l[4 * q + 2], l[4 * q + 3]);
                    }
                }
            }
            if (!free) break;
            if (is_x) {
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            } else {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(bar(B_PLFULL + d));
                mbar_arrive(bar(B_RAWEMPTY + s));
            }
        }
    }
    mv_pdl_launch_dependents();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    // a row's TN columns by a warp, four neighbours a lane
    const int n = 4 * lane < TN ? n0 + 4 * lane : g.N;
    const bool vec = n + 3 < g.N && (g.ldo & 3) == 0 && ((uintptr_t)g.out & 15) == 0 && g.mode != 1;
    bool left = false;
    for (int r = warp; r < TM && m0 + r < g.M; r += F3_THREADS / 32) {
        if (n >= g.N) continue;
        const float4 got = *reinterpret_cast<const float4*>(tile + r * L::OUT_LD + 4 * lane);
        if (!finite4(got)) {
            left = true;
            continue;
        }
        float v[4] = {got.x, got.y, got.z, got.w};
        const size_t o = (size_t)(m0 + r) * g.ldo + n;
        if (vec) {
            if (g.bias) {
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] += g.bias[n + e];
            }
            float4* p = reinterpret_cast<float4*>((float*)g.out + o);
            if (g.mode == 2) {
                const float4 old = *p;
                v[0] += old.x; v[1] += old.y; v[2] += old.z; v[3] += old.w;
            }
            *p = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (n + e < g.N) g.put(o + e, n + e, v[e]);
        }
    }
    if (left) multiply_again<TN>(g, tile, m0, n0);
    if (warp == 1) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

template <int TN>
int launch(const float* X, const float* W, const float* bias, void* out, int mode, int M, int N, int K, int ldo, int* err, cudaStream_t stream) {
    CUtensorMap mx, mw;
    if (!tensor_map(X, M, K, TM, &mx, KB, 4) || !tensor_map(W, N, K, TN, &mw, KB, 4)) return (int)cudaErrorInvalidValue;
    const cudaError_t attr = mv_allow_smem<gemm_f32_tc_kernel<TN>>(F3Layout<TN>::TOTAL);
    if (attr != cudaSuccess) return (int)attr;
    gemm_f32_tc_kernel<TN><<<dim3((N + TN - 1) / TN, (M + TM - 1) / TM), F3_THREADS, F3Layout<TN>::TOTAL, stream>>>(
        mx, mw, F3Args{X, W, bias, out, mode, M, N, K, ldo}, err);
    return mv_launch_status();
}

// The width of a tile, 128 or 96 columns: the one whose rounds over the device's multiprocessors take less, a round of 1,024 of K 26.4 or
// 21.9 us (1,165 rows: 9,216 columns in 133 / 154 us, 1,024 columns of 4,608 in 96 / 84, 2,048 in 51 / 50; tiles of 80 columns take as long as those of 96, of 64 95 %).
int tile_width(int M, int N, int sms) {
    auto cost = [&](int tn, int units) { return (((long long)((M + TM - 1) / TM) * ((N + tn - 1) / tn) + sms - 1) / sms) * units; };
    return cost(96, 83) < cost(128, 100) ? 96 : 128;
}

}  // namespace

// float32 X, W and sums; modes and bias as mv_gemm_simt's.  K a multiple of 4, X and W on 16 bytes, rows without gaps; `sms`: the device's multiprocessors.
MV_API int mv_gemm_f32_tc(const float* X, const float* W, const float* bias, void* out, int mode, int M, int N, int K, int ldo, int sms, int* err,
                          cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K < 4 || K % 4 || mode < 0 || mode > 2 || (((uintptr_t)X | (uintptr_t)W) & 15) || (M + TM - 1) / TM > 65535 || sms < 1) return (int)cudaErrorInvalidValue;
    return tile_width(M, N, sms) == 128 ? launch<128>(X, W, bias, out, mode, M, N, K, ldo, err, stream)
                                        : launch<96>(X, W, bias, out, mode, M, N, K, ldo, err, stream);
}
