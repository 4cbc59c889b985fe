// Packed quants into exact fp16 pairs, for the tensor-core kernel whose scales follow the sum (grouped_tc.cu): Q4_K words as
// sc * q, IQ3_XXS codebook entries with their signs.  Each translation unit that includes this header owns a copy of the
// IQ3_XXS tables and uploads it once per device.
#pragma once
#include "dnb_common.cuh"
#include "formats.cuh"
#include "dnb_iq_tables.h"

namespace dnb {

// Q4_K: the scales of two sub-blocks in both halves, 2^10 sc of the even one (64,512 at most), 2^6 sc of the odd one.
struct KScales { uint32_t s0, s1; };
// A word of packed bytes as 2^-14 sc * q: low nibbles are the even sub-block, high nibbles the odd one.  A nibble where it lies is the fp16
// number 2^-24 q or 2^-20 q below the normal ones, which multiplies like any other, and the product is exact and normal: a mask and a
// multiplication a pair.  (As 1024 + q and 64 + q, with a multiply-add, the mask and the exponent took two logic instructions, for want of
// registers for the constants: 58.8 M warp instructions of a launch -> 53.2 M.)
__device__ __forceinline__ void k_word(uint32_t w, const KScales& s, uint32_t (&p)[4]) {
    const uint32_t w8 = w >> 8;
    p[0] = h2mul(w & 0x000f000fu, s.s0);
    p[1] = h2mul(w8 & 0x000f000fu, s.s0);
    p[2] = h2mul(w & 0x00f000f0u, s.s1);
    p[3] = h2mul(w8 & 0x00f000f0u, s.s1);
}

// IQ3_XXS tables in shared memory, kLutRep copies each (a lane reads copy lane % kLutRep: no bank conflicts).
//   grid: the codebook as fp16 pairs, 128 bytes from entry to entry
//   sgn : the eight signs of a 7-bit code (the eighth makes their number even), 32 copies (half as many and two lanes of most reads meet on
//         a bank: a chunk of 512 tokens 426 -> 421 us): pair q of the eight weights at bits 15 - q and
//         31 - q, so that a shift by q and a mask give the sign bits of a pair
// The tables sit on a 32 KB boundary of the shared-memory address space: an entry's address is a shift and one and-or.
struct MmCodebook { uint2 grid[256 * kLutRep]; uint32_t sgn[128 * 32]; };
constexpr uint32_t kMmBookAlign = 32768;
static __device__ __align__(16) MmCodebook g_mm_codebook;
static TablesOnce g_mm_tables;

static int upload_mm_tables(int device) {
    return tables_once(g_mm_tables, device, [] {
        static MmCodebook tb;
        for (int e = 0; e < 256; ++e) {
            uint32_t h[4];
            for (int j = 0; j < 4; ++j) h[j] = __half_as_ushort(__float2half((float)((dnb_iq3xxs_grid[e] >> (8 * j)) & 0xFFu)));
            for (int r = 0; r < kLutRep; ++r) tb.grid[e * kLutRep + r] = make_uint2(h[0] | (h[1] << 16), h[2] | (h[3] << 16));
        }
        for (uint32_t code = 0; code < 128; ++code) {
            const uint32_t sg = code | ((uint32_t)(__builtin_popcount(code) & 1) << 7);
            uint32_t u = 0;
            for (int q = 0; q < 4; ++q) u |= ((sg >> (2 * q)) & 1u) << (15 - q) | ((sg >> (2 * q + 1)) & 1u) << (31 - q);
            for (int r = 0; r < 32; ++r) tb.sgn[code * 32 + r] = u;
        }
        DNB_CUDA(cudaMemcpyToSymbol(g_mm_codebook, &tb, sizeof(tb)));
        return DNB_OK;
    });
}

// Eight weights of an IQ3_XXS sub-block as four signed fp16 pairs.  gl, sl: shared addresses of the lane's copies; idx: the two
// codebook indices; code: the sub-block word rotated so that the quarter's 7-bit sign code starts at bit 7.
__device__ __forceinline__ void iq3_pairs_h(uint32_t gl, uint32_t sl, uint32_t idx, uint32_t code, uint32_t (&p)[4]) {
    uint32_t u, g0, g1, g2, g3;
    asm("ld.shared.u32 %0, [%1];" : "=r"(u) : "r"((code & 0x3f80u) | sl));  // constant tables: plain asm, free to move
    asm("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(g0), "=r"(g1) : "r"(((idx << 7) & 0x7f80u) | gl));
    asm("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(g2), "=r"(g3) : "r"(((idx >> 1) & 0x7f80u) | gl));
    p[0] = g0 ^ (u & 0x80008000u);
    p[1] = g1 ^ ((u << 1) & 0x80008000u);
    p[2] = g2 ^ ((u << 2) & 0x80008000u);
    p[3] = g3 ^ ((u << 3) & 0x80008000u);
}

}  // namespace dnb
