// Y[M, N] = X[M, K] . W[N, K]^T on the CUDA cores, any sizes, operands in
// float32 or bfloat16, accumulation in float32 with fused multiply-add.
//
// This is the matrix product of the true 32-bit path (no tensor-core mode is
// involved, so no reduced-precision matrix mode can slip in; large ones go to gemm_f32_tc.cu, which is no less exact), and the product
// of last resort for shapes that the tensor-core kernels refuse.  It computes
// what the reference's matvec / matmul rows do
// (crates/mivi-quant/src/lib.rs:75-135, 143-245): out[b, n] = sum_d in[b, d] * W[n, d].
//
// Epilogues: 0 store float32, 1 store bfloat16, 2 add into a float32 matrix
// (the residual stream).  A bias [N] may be added in every mode.
//
// Float32 operands whose rows start on 16 bytes (K a multiple of 4) take one of two kernels: up to 8 rows of X
// gemm_f32_stream_kernel, which is bound by reading W once, above that gemm_f32_tile_kernel, which is bound by the
// fused multiply-adds (with 16 rows in the first a lane's words of X outweigh those of W: 36 us against 28 for
// 1,024 x 4,608).  Everything else takes gemm_simt_kernel.
#include "common.cuh"

#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace {

__device__ __forceinline__ void f32_store(void* out, int mode, size_t o, float v) {
    if (mode == 0) ((float*)out)[o] = v;
    else if (mode == 1) ((__nv_bfloat16*)out)[o] = __float2bfloat16_rn(v);
    else ((float*)out)[o] += v;
}

// two multiply-adds in one instruction: (d.x, d.y) = (a.x * b.x + d.x, a.y * b.y + d.y), each rounded once
__device__ __forceinline__ void f32_fma2(float2& d, const float2& a, const float2& b) {
    unsigned long long& dd = reinterpret_cast<unsigned long long&>(d);
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(dd) : "l"(reinterpret_cast<const unsigned long long&>(a)),
        "l"(reinterpret_cast<const unsigned long long&>(b)));
}

// ---- many rows -------------------------------------------------------------------------------------------
// A block of 128 threads computes a tile of BM x 128 (BM 64 or 32) over its share of K; the blocks of a cluster share K
// and add their tiles in rank order through distributed shared memory, so a product gives the same bits in every run.
// A thread has TM x 8 results, each as two sums (even and odd k) so that one packed instruction takes two steps of k and
// the 16-byte words that shared memory holds ([row][k], 36 floats a row: eight neighbouring rows fall into eight different
// bank groups) are its operands as they are.  Three stages of 32 k by cp.async, two blocks a multiprocessor.
// Bound by the multiply-adds and the loads from shared memory that feed them: 1,165 rows against 9,216 x 1,024 in 510 us, 43
// TFLOP/s, where gemm_simt_kernel took 1,770 (12.4).  Against 64 bits its error is 3e-7 to 6e-7, the one-sum-per-result
// kernel's about 1e-6: a result is added up in 2 (cut: up to 16) parts.
constexpr int FT_BN = 128, FT_BK = 32, FT_LD = FT_BK + 4, FT_STAGES = 3, FT_THREADS = 128;

template <int TM>
__global__ void __launch_bounds__(FT_THREADS, 2)
gemm_f32_tile_kernel(const float* __restrict__ X, const float* __restrict__ W, const float* __restrict__ bias,
                     void* __restrict__ out, int mode, int M, int N, int K, int ldo, int kb_per_rank) {
    constexpr int BM = TM * 8, ROWS = BM + FT_BN;
    extern __shared__ __align__(16) float smem[];                   // FT_STAGES x [ROWS][FT_LD], then the tile [BM][FT_BN]
    mv_pdl_begin();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tm = (warp & 1) * 4 + (lane >> 3), tn = (warp >> 1) * 8 + (lane & 7);     // 8 x 16 threads
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * FT_BN;
    const int kb_all = (K + FT_BK - 1) / FT_BK;
    const int kb0 = min(blockIdx.z * kb_per_rank, kb_all), kb1 = min(kb0 + kb_per_rank, kb_all);

    auto load = [&](int kb, int stage) {
        float* dst = smem + (size_t)stage * ROWS * FT_LD;
        const int k0 = kb * FT_BK;
#pragma unroll
        for (int e = 0; e < ROWS * (FT_BK / 4) / FT_THREADS; ++e) {
            const int idx = tid + e * FT_THREADS, r = idx >> 3, c = (idx & 7) * 4;
            const bool x_row = r < BM;
            const int row = x_row ? m0 + r : n0 + r - BM;
            const bool in = row < (x_row ? M : N) && k0 + c < K;
            const float* src = (x_row ? X : W) + (in ? (size_t)row * K + k0 + c : 0);
            const unsigned to = (unsigned)__cvta_generic_to_shared(dst + r * FT_LD + c);
            const int bytes = in ? 16 : 0;                          // the rest of the 16 is filled with zeros
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(src), "r"(bytes) : "memory");
        }
    };
    float2 acc[TM][8];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll
    for (int s = 0; s < FT_STAGES - 1; ++s) {
        if (kb0 + s < kb1) load(kb0 + s, s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    int stage = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
        asm volatile("cp.async.wait_group %0;" ::"n"(FT_STAGES - 2) : "memory");
        __syncthreads();                                            // this stage is there; the one before is done with
        {
            const int ahead = stage + FT_STAGES - 1 >= FT_STAGES ? stage - 1 : stage + FT_STAGES - 1;
            if (kb + FT_STAGES - 1 < kb1) load(kb + FT_STAGES - 1, ahead);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        const float* xs = smem + (size_t)stage * ROWS * FT_LD + tm * FT_LD;
        const float* ws = smem + (size_t)stage * ROWS * FT_LD + (BM + tn) * FT_LD;
#pragma unroll
        for (int kk = 0; kk < FT_BK; kk += 4) {
            float4 a[TM], b[8];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(xs + i * 8 * FT_LD + kk);
#pragma unroll
            for (int j = 0; j < 8; ++j) b[j] = *reinterpret_cast<const float4*>(ws + j * 16 * FT_LD + kk);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    f32_fma2(acc[i][j], make_float2(a[i].x, a[i].y), make_float2(b[j].x, b[j].y));
                    f32_fma2(acc[i][j], make_float2(a[i].z, a[i].w), make_float2(b[j].z, b[j].w));
                }
        }
        stage = stage + 1 == FT_STAGES ? 0 : stage + 1;
    }
    if (gridDim.z == 1) {
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int gm = m0 + tm + 8 * i;
            if (gm >= M) continue;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int gn = n0 + tn + 16 * j;
                if (gn >= N) continue;
                f32_store(out, mode, (size_t)gm * ldo + gn, acc[i][j].x + acc[i][j].y + (bias ? bias[gn] : 0.f));
            }
        }
        return;
    }
    // the cluster's shares of K: every block leaves its tile in its shared memory, then adds its rows of all of them
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) smem[(tm + 8 * i) * FT_BN + tn + 16 * j] = acc[i][j].x + acc[i][j].y;
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    const int ranks = (int)gridDim.z, rank = (int)blockIdx.z;
    for (int idx = tid; idx < BM / ranks * FT_BN; idx += FT_THREADS) {
        const int r = rank * (BM / ranks) + idx / FT_BN, c = idx & (FT_BN - 1);
        float v = 0.f;
        for (int q = 0; q < ranks; ++q) v += cluster.map_shared_rank(smem, q)[r * FT_BN + c];
        const int gm = m0 + r, gn = n0 + c;
        if (gm < M && gn < N) f32_store(out, mode, (size_t)gm * ldo + gn, v + (bias ? bias[gn] : 0.f));
    }
    cluster.sync();                                                 // nobody leaves while its tile is read
}

// Two blocks a multiprocessor run at once.  K is cut over 1, 2, 4 or 8 blocks so that the rounds of such blocks, each as long as a
// share of K and about four steps of filling and (cut) adding up, end soonest; a tile of 32 rows takes 0.63 of the time of one of
// 64 (half the products, fewer of them a read).  In 64ths of a step; `ranks` gets the cut.
inline long gemm_f32_tile_cost(int bm, int M, int N, int K, int* ranks) {
    const long tiles = (long)((N + FT_BN - 1) / FT_BN) * ((M + bm - 1) / bm);
    const int kb = (K + FT_BK - 1) / FT_BK;
    long best = 0;
    for (int r = 1; r <= 8; r *= 2) {
        const long cost = (tiles * r + 295) / 296 * ((kb + r - 1) / r + 4 + (r > 1 ? 2 : 0)) * (bm == 64 ? 64 : 40);
        if (r == 1 || cost < best) { best = cost; *ranks = r; }
    }
    return best;
}

template <int TM>
int gemm_f32_tile_launch(const float* X, const float* W, const float* bias, void* out, int mode, int M, int N, int K, int ldo,
                         cudaStream_t stream) {
    constexpr int BM = TM * 8;
    constexpr size_t smem = sizeof(float) * FT_STAGES * (BM + FT_BN) * FT_LD;
    static_assert(sizeof(float) * BM * FT_BN <= smem, "the tile takes the stages' place");
    const cudaError_t attr = mv_allow_smem<gemm_f32_tile_kernel<TM>>(smem);
    if (attr != cudaSuccess) return (int)attr;
    const int gx = (N + FT_BN - 1) / FT_BN, gy = (M + BM - 1) / BM, kb = (K + FT_BK - 1) / FT_BK;
    int ranks = 1;
    gemm_f32_tile_cost(BM, M, N, K, &ranks);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(gx, gy, ranks);
    cfg.blockDim = dim3(FT_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 1; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = (unsigned)ranks;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = mv_pdl_enabled() ? 2 : 1;
    cudaLaunchKernelEx(&cfg, gemm_f32_tile_kernel<TM>, X, W, bias, out, mode, M, N, K, ldo, (kb + ranks - 1) / ranks);
    return mv_launch_status();
}

// ---- few rows --------------------------------------------------------------------------------------------
// A block has 8 rows of W (4 for more than one row of X), its eight warps share K word by word (a warp reads 512 bytes of every row at a time), a lane keeps
// FS_ROWS x MP sums.  They are added over the lanes by halving (31 shuffles for 32 sums) and over the warps in order.  The first
// words of W are requested before the kernel before has ended: they do not depend on it.  Bound by reading W
// (16,384 x 2,048 against one row: 22 us, 6.1 TB/s; against 4 rows 34 us, where gemm_simt_kernel took 500).
constexpr int FS_WARPS = 8;

template <int MP, int FS_ROWS>
__global__ void __launch_bounds__(FS_WARPS * 32)
gemm_f32_stream_kernel(const float* __restrict__ X, const float* __restrict__ W, const float* __restrict__ bias,
                       void* __restrict__ out, int mode, int M, int N, int K, int ldo) {
    constexpr int SUMS = FS_ROWS * MP;
    __shared__ float part[FS_WARPS][SUMS];
    mv_pdl_launch_dependents();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n0 = blockIdx.x * FS_ROWS, K4 = K >> 2;
    const float4* W4 = reinterpret_cast<const float4*>(W);
    const float4* X4 = reinterpret_cast<const float4*>(X);
    float2 acc[FS_ROWS][MP];
#pragma unroll
    for (int r = 0; r < FS_ROWS; ++r)
#pragma unroll
        for (int m = 0; m < MP; ++m) acc[r][m] = make_float2(0.f, 0.f);
    float4 w[FS_ROWS];
    auto request = [&](int k4) {
#pragma unroll
        for (int r = 0; r < FS_ROWS; ++r)
            w[r] = (k4 < K4 && n0 + r < N) ? __ldcs(W4 + (size_t)(n0 + r) * K4 + k4) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    int k4 = warp * 32 + lane;
    request(k4);
    mv_pdl_wait();
    for (; k4 < K4; k4 += FS_WARPS * 32) {
        float4 now[FS_ROWS];
#pragma unroll
        for (int r = 0; r < FS_ROWS; ++r) now[r] = w[r];
        request(k4 + FS_WARPS * 32);
#pragma unroll
        for (int m = 0; m < MP; ++m) {
            const float4 x = m < M ? X4[(size_t)m * K4 + k4] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int r = 0; r < FS_ROWS; ++r) {
                f32_fma2(acc[r][m], make_float2(now[r].x, now[r].y), make_float2(x.x, x.y));
                f32_fma2(acc[r][m], make_float2(now[r].z, now[r].w), make_float2(x.z, x.w));
            }
        }
    }
    float v[SUMS];
#pragma unroll
    for (int r = 0; r < FS_ROWS; ++r)
#pragma unroll
        for (int m = 0; m < MP; ++m) v[r * MP + m] = acc[r][m].x + acc[r][m].y;
    // sums of a group of 32 (or of all, if fewer): each halving leaves a lane half of the sums over twice the lanes
    constexpr int GROUP = SUMS < 32 ? SUMS : 32;
#pragma unroll
    for (int g = 0; g < SUMS; g += GROUP) {
        int bit = 16;
#pragma unroll
        for (int n = GROUP / 2; n >= 1; n /= 2) {
            const bool high = lane & bit;
#pragma unroll
            for (int i = 0; i < n; ++i) {
                const float send = high ? v[g + i] : v[g + n + i], keep = high ? v[g + n + i] : v[g + i];
                v[g + i] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
            }
            bit >>= 1;
        }
        for (; bit >= 1; bit >>= 1) v[g] += __shfl_xor_sync(0xffffffffu, v[g], bit);
        // the lane's sum: its bits from the highest say which half was kept each time
        if (GROUP == 32) part[warp][g + lane] = v[g];
        else if ((lane & (32 / GROUP - 1)) == 0) part[warp][g + lane / (32 / GROUP)] = v[g];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < SUMS; i += FS_WARPS * 32) {
        const int r = i / MP, m = i - r * MP;
        float sum = 0.f;
#pragma unroll
        for (int q = 0; q < FS_WARPS; ++q) sum += part[q][i];
        if (m < M && n0 + r < N) f32_store(out, mode, (size_t)m * ldo + n0 + r, sum + (bias ? bias[n0 + r] : 0.f));
    }
}

template <int MP, int FS_ROWS>
int gemm_f32_stream_launch(const float* X, const float* W, const float* bias, void* out, int mode, int M, int N, int K, int ldo,
                           cudaStream_t stream) {
    mv_launch(gemm_f32_stream_kernel<MP, FS_ROWS>, (N + FS_ROWS - 1) / FS_ROWS, FS_WARPS * 32, 0, stream, X, W, bias, out, mode, M, N, K,
              ldo);
    return mv_launch_status();
}

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

template <typename T>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const T* __restrict__ X, const T* __restrict__ W, const float* __restrict__ bias,
                 void* __restrict__ out, int mode, int M, int N, int K, int ldo) {
    mv_pdl_begin();
    __shared__ float Xs[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;          // 16 x 16 threads
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += BK) {
        // 64 x 16 elements of each operand, 4 per thread
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int idx = tid + e * 256;
            const int r = idx >> 4, c = idx & 15;
            const int gm = m0 + r, gn = n0 + r, gk = k0 + c;
            Xs[c][r] = (gm < M && gk < K) ? mv_to_f32(X[(size_t)gm * K + gk]) : 0.f;
            Ws[c][r] = (gn < N && gk < K) ? mv_to_f32(W[(size_t)gn * K + gk]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = Xs[kk][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = Ws[kk][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + ty * TM + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gn = n0 + tx * TN + j;
            if (gn >= N) continue;
            float v = acc[i][j];
            if (bias) v += bias[gn];
            const size_t o = (size_t)gm * ldo + gn;
            if (mode == 0) ((float*)out)[o] = v;
            else if (mode == 1) ((__nv_bfloat16*)out)[o] = __float2bfloat16_rn(v);
            else ((float*)out)[o] += v;
        }
    }
}

}  // namespace

// The tile's rows (32 or 64) that a float32 product of more than 8 rows is cut into, plus the number of blocks that share K.
MV_API int mv_gemm_f32_plan(int M, int N, int K) {
    int r32 = 1, r64 = 1;
    const bool small = gemm_f32_tile_cost(32, M, N, K, &r32) < gemm_f32_tile_cost(64, M, N, K, &r64);
    return small ? 32 + r32 : 64 + r64;
}

MV_API int mv_gemm_simt(const void* X, const void* W, int in_dtype, const float* bias, void* out,
                        int mode, int M, int N, int K, int ldo, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (in_dtype == MV_DT_F32 && K >= 4 && K % 4 == 0 && ((uintptr_t)X | (uintptr_t)W) % 16 == 0 && (M + 31) / 32 <= 65535) {
        const float *x = (const float*)X, *w = (const float*)W;
        if (M == 1) return gemm_f32_stream_launch<1, 8>(x, w, bias, out, mode, M, N, K, ldo, stream);
        if (M == 2) return gemm_f32_stream_launch<2, 4>(x, w, bias, out, mode, M, N, K, ldo, stream);
        if (M <= 4) return gemm_f32_stream_launch<4, 4>(x, w, bias, out, mode, M, N, K, ldo, stream);
        if (M <= 8) return gemm_f32_stream_launch<8, 4>(x, w, bias, out, mode, M, N, K, ldo, stream);
        // 1,165 rows against 1,024 x 4,608: 152 tiles of 64 rows leave one block on a multiprocessor (305 us with K cut in four), 296
        // of 32 rows fill them (273; against 1,024 x 1,024: 109 and 63)
        if (mv_gemm_f32_plan(M, N, K) < 64)
            return gemm_f32_tile_launch<4>(x, w, bias, out, mode, M, N, K, ldo, stream);
        return gemm_f32_tile_launch<8>(x, w, bias, out, mode, M, N, K, ldo, stream);
    }
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (in_dtype == MV_DT_BF16)
        mv_launch(gemm_simt_kernel<__nv_bfloat16>, grid, 256, 0, stream, (const __nv_bfloat16*)X, (const __nv_bfloat16*)W,
                                                   bias, out, mode, M, N, K, ldo);
    else
        mv_launch(gemm_simt_kernel<float>, grid, 256, 0, stream, (const float*)X, (const float*)W, bias, out, mode,
                                                   M, N, K, ldo);
    return mv_launch_status();
}
