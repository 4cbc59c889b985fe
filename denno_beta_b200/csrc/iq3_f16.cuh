// Packed quants into exact fp16 pairs, for the tensor-core kernels whose scales follow the sum (grouped_mma.cu on mma.sync,
// grouped_tc.cu on tcgen05): Q4_K / Q5_K words as sc * q, IQ3_XXS codebook entries with their signs.  Each translation unit
// that includes this header owns a copy of the IQ3_XXS tables and uploads it once per device.
#pragma once
#include "dnb_common.cuh"
#include "formats.cuh"
#include "dnb_iq_tables.h"

namespace dnb {

__device__ __forceinline__ uint32_t h2fma(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ uint32_t h2sub(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t h2mul(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
// Q4_K / Q5_K: a lane's scales of one row of a block.  s0 / s1: the scale of its even / odd sub-block in both halves,
// k0 / k1: -1024 * s0 and -64 * s1, mm: the pair of mins.
struct KScales { float d, dmin; uint32_t s0, s1, k0, k1, mm; };
__device__ __forceinline__ KScales k_scales(const uint8_t* row, int t) {
    const uint4 h = *reinterpret_cast<const uint4*>(row);
    const int sh = 16 * (t & 1);
    const uint32_t a = h.y >> sh, b = h.z >> sh, c = h.w >> sh;
    const bool low = t < 2;  // kquant.rs:878-887
    const uint32_t sc = low ? (a & 0x3f3fu) : ((c & 0x0f0fu) | ((a >> 2) & 0x3030u));
    const uint32_t mn = low ? (b & 0x3f3fu) : (((c >> 4) & 0x0f0fu) | ((b >> 2) & 0x3030u));
    KScales r;
    r.d = h2f((uint16_t)h.x);
    r.dmin = h2f((uint16_t)(h.x >> 16));
    r.s0 = h2sub(__byte_perm(sc, 0x64646464u, 0x4040u), 0x64006400u);
    r.s1 = h2sub(__byte_perm(sc, 0x64646464u, 0x4141u), 0x64006400u);
    r.k0 = h2mul(r.s0, 0xE400E400u);  // * -1024
    r.k1 = h2mul(r.s1, 0xD400D400u);  // * -64
    r.mm = h2sub(__byte_perm(mn, 0x64646464u, 0x4140u), 0x64006400u);
    return r;
}
// Word i of a lane's 32 bytes: low nibbles are the even sub-block, high nibbles the odd one.  hq (Q5_K): the word of fifth
// bits shifted so that bit 0 of a byte belongs to the low and bit 1 to the high nibble.
template <bool FIVE>
__device__ __forceinline__ void k_word(uint32_t w, uint32_t hq, const KScales& s, uint32_t (&p)[4]) {
    const uint32_t w8 = w >> 8;
    uint32_t a = (w & 0x000f000fu) | 0x64006400u, b = (w8 & 0x000f000fu) | 0x64006400u;    // 1024 + q
    uint32_t c = (w & 0x00f000f0u) | 0x54005400u, d = (w8 & 0x00f000f0u) | 0x54005400u;    // 64 + q
    if constexpr (FIVE) {
        const uint32_t h8 = hq >> 8;
        a |= (hq << 4) & 0x00100010u;
        b |= (h8 << 4) & 0x00100010u;
        c |= (hq << 7) & 0x01000100u;
        d |= (h8 << 7) & 0x01000100u;
    }
    p[0] = h2fma(a, s.s0, s.k0);
    p[1] = h2fma(b, s.s0, s.k0);
    p[2] = h2fma(c, s.s1, s.k1);
    p[3] = h2fma(d, s.s1, s.k1);
}

// IQ3_XXS tables in shared memory, kLutRep copies each (a lane reads copy lane % kLutRep: no bank conflicts).
//   grid: the codebook as fp16 pairs, 128 bytes from entry to entry
//   sgn : the eight signs of a 7-bit code (the eighth makes their number even): pair q of the eight weights at bits 15 - q and
//         31 - q, so that a shift by q and a mask give the sign bits of a pair
// The tables sit on a 32 KB boundary of the shared-memory address space: an entry's address is a shift and one and-or.
struct MmCodebook { uint2 grid[256 * kLutRep]; uint32_t sgn[128 * kLutRep]; };
constexpr uint32_t kMmBookAlign = 32768;
constexpr uint32_t kMmSmemBase = 1024;  // where dynamic shared memory starts (what the system keeps of an SM's shared memory per CTA)
static __device__ __align__(16) MmCodebook g_mm_codebook;
static bool g_mm_tables[64] = {false};

static int upload_mm_tables(int device) {
    if (device < 0 || device >= 64) return DNB_ERR_ARG;
    if (g_mm_tables[device]) return DNB_OK;
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
        for (int r = 0; r < kLutRep; ++r) tb.sgn[code * kLutRep + r] = u;
    }
    DNB_CUDA(cudaMemcpyToSymbol(g_mm_codebook, &tb, sizeof(tb)));
    g_mm_tables[device] = true;
    return DNB_OK;
}

// Eight weights of an IQ3_XXS sub-block as four signed fp16 pairs.  gl, sl: shared addresses of the lane's copies; idx: the two
// codebook indices; code: the sub-block word rotated so that the quarter's 7-bit sign code starts at bit 6.
__device__ __forceinline__ void iq3_pairs_h(uint32_t gl, uint32_t sl, uint32_t idx, uint32_t code, uint32_t (&p)[4]) {
    uint32_t u, g0, g1, g2, g3;
    asm("ld.shared.u32 %0, [%1];" : "=r"(u) : "r"((code & 0x1fc0u) | sl));  // constant tables: plain asm, free to move
    asm("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(g0), "=r"(g1) : "r"(((idx << 7) & 0x7f80u) | gl));
    asm("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(g2), "=r"(g3) : "r"(((idx >> 1) & 0x7f80u) | gl));
    p[0] = g0 ^ (u & 0x80008000u);
    p[1] = g1 ^ ((u << 1) & 0x80008000u);
    p[2] = g2 ^ ((u << 2) & 0x80008000u);
    p[3] = g3 ^ ((u << 3) & 0x80008000u);
}

}  // namespace dnb
