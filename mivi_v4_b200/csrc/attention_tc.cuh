// What the tcgen05 attentions share whose blocks of keys are masked for some of their rows (latent_attention_tc.cu, attention_sink_tc.cu).
//
// A product of weights and values takes all rows of a tile past every key, with a weight of 0 where a row does not see the key, and 0 times an
// infinity or a NaN is a NaN.  So the values of a block that some row does not see whole go by way of one warp, which puts zeros in the place of numbers that are not
// finite; if there were any, every row looks up in memory which of them it sees, and adds those to its sums at the end.  (A value that is not finite
// reaches the rows that see it and no others.  Looking through a block is some 120 instructions of that warp beside the softmax's 4,000.  Us without it and with it: latent attention, a
// prompt of 6,000 tokens 366 / 372, of 2,048 73 / 73, with a window of 512 64 / 64; with a sink, 2,048 tokens with chunks 40 / 40, 32 prompts of 128 52 / 54.)
#pragma once
#include "tc_common.cuh"

namespace {

// the halves of a pair of bfloat16 numbers that are not finite, as bits 15 and 31
__device__ __forceinline__ unsigned not_finite2(unsigned x) { return ((x & 0x7f807f80u) + 0x00800080u) & 0x80008000u; }

// By a whole warp: 64 rows of 64 values in shared memory, 128 bytes each.  Rows before `head` and from `tail` on become zeros, and so do numbers that are not
// finite in the others; whether there were any.  (The largest magnitude tells, a NaN kept: an instruction a pair of numbers.)
__device__ __forceinline__ bool clean_values(unsigned char* rows, int head, int tail, int lane) {
    uint4* p = reinterpret_cast<uint4*>(rows) + lane;
    if (head > 0 || tail < 64)
        for (int i = lane; i < 64 * 8; i += 32)
            if (i < head * 8 || i >= tail * 8) p[i - lane] = make_uint4(0u, 0u, 0u, 0u);
    __nv_bfloat162 top[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) top[e] = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 64 * 8; i += 32) {
        const uint4 x = p[i];
        top[0] = __hmax2_nan(top[0], __habs2(*reinterpret_cast<const __nv_bfloat162*>(&x.x)));
        top[1] = __hmax2_nan(top[1], __habs2(*reinterpret_cast<const __nv_bfloat162*>(&x.y)));
        top[2] = __hmax2_nan(top[2], __habs2(*reinterpret_cast<const __nv_bfloat162*>(&x.z)));
        top[3] = __hmax2_nan(top[3], __habs2(*reinterpret_cast<const __nv_bfloat162*>(&x.w)));
    }
    const __nv_bfloat162 most = __hmax2_nan(__hmax2_nan(top[0], top[1]), __hmax2_nan(top[2], top[3]));
    if (!__any_sync(0xffffffffu, not_finite2(*reinterpret_cast<const unsigned*>(&most)) != 0)) return false;
#pragma unroll 1
    for (int i = 0; i < 64 * 8; i += 32) {
        uint4 x = p[i];
        x.x &= ~((not_finite2(x.x) >> 15) * 0xffffu);
        x.y &= ~((not_finite2(x.y) >> 15) * 0xffffu);
        x.z &= ~((not_finite2(x.z) >> 15) * 0xffffu);
        x.w &= ~((not_finite2(x.w) >> 15) * 0xffffu);
        p[i] = x;
    }
    return true;
}

// Which of 32 channels have a NaN, an infinity, a negative infinity in the rows that a query sees.
struct NotFinite {
    unsigned nan = 0, pos = 0, neg = 0;
    __device__ __forceinline__ bool any() const { return (nan | pos | neg) != 0; }
    // what the rows add to the sum of channel i
    __device__ __forceinline__ float value(int i) const {
        const unsigned bit = 1u << i;
        return (nan & bit) || (pos & neg & bit) ? __int_as_float(0x7fffffff) : pos & bit ? INFINITY : neg & bit ? -INFINITY : 0.f;
    }
};
// rows [from, upto) of `ld` numbers each, channels [0, n) of them (n in steps of 8 up to 32, 16-byte aligned)
__device__ __noinline__ NotFinite look_up(NotFinite f, const __nv_bfloat16* rows, long long ld, int from, int upto, int n) {
    for (int r = from; r < upto; ++r) {
        const __nv_bfloat16* row = rows + (long long)r * ld;
        for (int w = 0; w < n / 8; ++w) {
            const uint4 x = *reinterpret_cast<const uint4*>(row + 8 * w);
            const unsigned v[4] = {x.x, x.y, x.z, x.w};
            if (!(not_finite2(x.x) | not_finite2(x.y) | not_finite2(x.z) | not_finite2(x.w))) continue;
            for (int e = 0; e < 8; ++e) {
                const unsigned b = (v[e >> 1] >> (16 * (e & 1))) & 0xffffu, bit = 1u << (8 * w + e);
                if ((b & 0x7f80u) != 0x7f80u) continue;
                if (b & 0x7fu) f.nan |= bit;
                else if (b & 0x8000u) f.neg |= bit;
                else f.pos |= bit;
            }
        }
    }
    return f;
}

}  // namespace
