// Operand rows of the tcgen05 grouped GEMM (grouped_tc.cu): an activation row as two rows of fp16, hi and lo parts of the row times
// a power of two that puts its largest element into [512, 1024), in the order in which the weights of the format are decoded;
// then the sums of its 32-element sub-blocks (Q4_K: for the mins) and, in the hi row, what undoes the scaling.  Written a
// 256-element block per warp at a time, by the RMSNorm kernel as it goes or from fp32 rows.
#pragma once
#include <cuda_fp16.h>

#include "dnb_common.cuh"

namespace dnb {
namespace tg {

__host__ __device__ __forceinline__ int x_cols(int n_in) { return (n_in / 32 + 63) / 64 * 64; }
__host__ __device__ __forceinline__ int row_pitch(int n_in) { return n_in + x_cols(n_in) + 8; }  // + the row's scale (a float) and padding

// The two groups of four elements that lane `lane` holds of the block at `b`: its 16-byte unit of the row.
template <int T>
__device__ __forceinline__ void operand_elems(int b, int lane, int& e0, int& e1) {
    e0 = T == T_Q4_K ? b + 64 * (lane >> 3) + 4 * (lane & 7) : b + 8 * lane;
    e1 = T == T_Q4_K ? e0 + 32 : e0 + 4;
}
__device__ __forceinline__ uint32_t operand_max(uint32_t mx, const float4& v) {  // bits of the largest |x|
    return max(mx, max(max(__float_as_uint(fabsf(v.x)), __float_as_uint(fabsf(v.y))), max(__float_as_uint(fabsf(v.z)), __float_as_uint(fabsf(v.w)))));
}
__device__ __forceinline__ float operand_scale(uint32_t amax_bits) {
    const int ex = (int)(amax_bits >> 23), s = ex == 0 ? 0 : max(-126, min(126, 9 - (ex - 127)));
    return __uint_as_float((uint32_t)(127 + s) << 23);
}
// Two numbers as hi and lo.  The tensor core adds with truncation, and as a block's sum of hi starts from that of lo, their addition is truncated,
// too (two accumulators, as there were before, are added in fp32): sums come out 3.4e-8 of themselves short, beside what the sums of hi lose
// either way.  So a lo part carries that much of its number, unless it is zero (then nothing is cut off).  Error against 64 bits, of what it was
// with two accumulators, without / with this: normal inputs 1.003 / 0.91, a mean of 3 (IQ3_XXS) 1.06 / 0.89, products of two normal numbers 0.997 /
// 0.91, one element in 16 1.16 / 0.93, one in 256 1.18 / 0.97; over 20 kinds of input, two formats, K of 512 and 2048 0.86 to 0.98, and 1.000 where
// lo is zero throughout.
constexpr float kShort = 0x1.2p-25f;
__device__ __forceinline__ void operand_split(float a, float b, uint32_t& h, uint32_t& l) {
    const __half2 hv = __floats2half2_rn(a, b);
    const float2 hf = __half22float2(hv);
    float la = a - hf.x, lb = b - hf.y;
    if (la != 0.f) la = fmaf(a, kShort, la);
    if (lb != 0.f) lb = fmaf(b, kShort, lb);
    const __half2 lv = __floats2half2_rn(la, lb);
    h = *reinterpret_cast<const uint32_t*>(&hv);
    l = *reinterpret_cast<const uint32_t*>(&lv);
}
// A warp: the block at b of the row whose hi part starts at `hi`.
template <int T>
__device__ __forceinline__ void operand_block(float4 v0, float4 v1, float up, int b, int K, int pitch, int lane, uint16_t* hi) {
    uint16_t* lo = hi + pitch;
    v0.x *= up; v0.y *= up; v0.z *= up; v0.w *= up;
    v1.x *= up; v1.y *= up; v1.z *= up; v1.w *= up;
    uint32_t h[4], l[4];
    if constexpr (T == T_Q4_K) {  // a word of nibbles yields its bytes 0, 2 and 1, 3
        operand_split(v0.x, v0.z, h[0], l[0]);
        operand_split(v0.y, v0.w, h[1], l[1]);
        operand_split(v1.x, v1.z, h[2], l[2]);
        operand_split(v1.y, v1.w, h[3], l[3]);
    } else {
        operand_split(v0.x, v0.y, h[0], l[0]);
        operand_split(v0.z, v0.w, h[1], l[1]);
        operand_split(v1.x, v1.y, h[2], l[2]);
        operand_split(v1.z, v1.w, h[3], l[3]);
    }
    *reinterpret_cast<uint4*>(hi + b + 8 * lane) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4*>(lo + b + 8 * lane) = make_uint4(l[0], l[1], l[2], l[3]);
    if constexpr (T == T_Q4_K) {
        float a = (v0.x + v0.y) + (v0.z + v0.w), c = (v1.x + v1.y) + (v1.z + v1.w);  // sub-blocks 2 g, 2 g + 1 of group g = lane / 8
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            c += __shfl_xor_sync(0xffffffffu, c, o);
        }
        if ((lane & 7) == 0) {
            uint32_t sh, sl;
            operand_split(a, c, sh, sl);
            const int at = K + b / 32 + 2 * (lane >> 3);
            *reinterpret_cast<uint32_t*>(hi + at) = sh;
            *reinterpret_cast<uint32_t*>(lo + at) = sl;
            if (K % 2048 && K % 2048 <= 1024 && b >= K / 2048 * 2048) {  // the stage with both halves of the mins reads the sums twice
                *reinterpret_cast<uint32_t*>(hi + at + 32) = sh;
                *reinterpret_cast<uint32_t*>(lo + at + 32) = sl;
            }
        }
    }
}
// A warp, once per row: columns without a sub-block are zero; the scale.
template <int T>
__device__ __forceinline__ void operand_tail(float up, int K, int pitch, int lane, uint16_t* hi) {
    const int xc = x_cols(K);
    if constexpr (T == T_Q4_K) {
        const int nsub = K / 32, g0 = nsub / 64 * 64, rest = nsub - g0;  // the last, partial group of 64
        for (int i = lane; i < xc - g0; i += 32)
            if (rest <= 32 ? (i & 31) >= rest : i >= rest) hi[K + g0 + i] = hi[pitch + K + g0 + i] = 0;
    }
    if (lane == 0) *reinterpret_cast<float*>(hi + K + xc) = __uint_as_float((254u << 23) - __float_as_uint(up));  // 1 / up
}

}  // namespace tg
}  // namespace dnb
