// IQ3_XXS decode into mma.sync fragments: what the one-token kernels of gemv_mma.cu and
// decode_fused.cu share.  Each translation unit that includes this header owns a copy of
// the bf16 codebook and uploads it once per device.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "dnb_common.cuh"
#include "formats.cuh"
#include "bulk.cuh"
#include "dnb_iq_tables.h"

namespace dnb {

constexpr int kGmRows = 8;     // rows of one matrix per group (x2 matrices = the 16 mma rows)
constexpr int kGmKs = 4;       // warps that split K within a group
constexpr int kGmGroups = 5;   // groups a CTA can hold
constexpr int kGmThreads = kGmGroups * kGmKs * 32;
constexpr int kGmSplit = 3;    // bf16 terms per activation value
constexpr int kIq3Unroll = 4;  // sub-blocks of the K loops unrolled together

// What a CTA copies into shared memory in one bulk copy, kLutRep copies of each entry (a lane reads copy lane % kLutRep):
//   grid: the IQ3_XXS codebook as bf16 pairs, .x = elements 0,1, .y = elements 2,3
//   sgn : the eight signs of a 7-bit code (the eighth makes their number even): pair q of the eight weights at bits 15 - q and
//         31 - q, so that a shift by q and a mask give the sign bits of a pair
struct Iq3Tables {
    uint2 grid[256 * kLutRep];
    uint32_t sgn[128 * kLutRep];
};
static __device__ __align__(16) Iq3Tables g_iq3_tables;
static TablesOnce g_tables_m;

static int upload_tables_m(int device) {
    return tables_once(g_tables_m, device, [] {
        static Iq3Tables tb;
        for (int e = 0; e < 256; ++e) {
            const uint32_t w = dnb_iq3xxs_grid[e];
            uint32_t h[4];
            for (int j = 0; j < 4; ++j) {
                const float f = (float)((w >> (8 * j)) & 0xFFu);  // <= 62: its fp32 pattern has nothing below bit 16
                uint32_t bits;
                memcpy(&bits, &f, 4);
                h[j] = bits >> 16;
            }
            for (int r = 0; r < kLutRep; ++r) tb.grid[e * kLutRep + r] = make_uint2(h[0] | (h[1] << 16), h[2] | (h[3] << 16));
        }
        for (uint32_t code = 0; code < 128; ++code) {
            const uint32_t sg = code | ((uint32_t)(__builtin_popcount(code) & 1) << 7);
            uint32_t u = 0;
            for (int q = 0; q < 4; ++q) u |= ((sg >> (2 * q)) & 1u) << (15 - q) | ((sg >> (2 * q + 1)) & 1u) << (31 - q);
            for (int r = 0; r < kLutRep; ++r) tb.sgn[code * kLutRep + r] = u;
        }
        DNB_CUDA(cudaMemcpyToSymbol(g_iq3_tables, &tb, sizeof(tb)));
        return DNB_OK;
    });
}
// A lane's view of the tables in shared memory: the addresses of its own copies
struct Iq3Lane {
    uint32_t grid, sgn;
    __device__ __forceinline__ Iq3Lane(const Iq3Tables* tb, int lane)
        : grid((uint32_t)__cvta_generic_to_shared(tb->grid + (lane & (kLutRep - 1)))), sgn((uint32_t)__cvta_generic_to_shared(tb->sgn + (lane & (kLutRep - 1)))) {}
};

__device__ __forceinline__ uint32_t bf16_bits(float v) { return __bfloat16_as_ushort(__float2bfloat16_rn(v)); }
__device__ __forceinline__ float silu_m(float v) { return v / (1.0f + expf(-v)); }
__device__ __forceinline__ float bf16_val(uint32_t h) { return __uint_as_float(h << 16); }

__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Eight weights of one IQ3_XXS sub-block as four signed bf16 pairs (without the scale): idx = the two codebook indices of this
// lane's quarter, code: the sub-block word rotated so that the quarter's 7-bit sign code starts at bit 6.
__device__ __forceinline__ void iq3_pairs(const Iq3Lane& L, uint32_t idx, uint32_t code, uint32_t (&p)[4]) {
    uint32_t u, g0, g1, g2, g3;
    asm("ld.shared.u32 %0, [%1];" : "=r"(u) : "r"((code & 0x1fc0u) + L.sgn));  // constant tables: plain asm, free to move
    asm("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(g0), "=r"(g1) : "r"((idx & 0xffu) * (kLutRep * 8u) + L.grid));
    asm("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(g2), "=r"(g3) : "r"((idx >> 8) * (kLutRep * 8u) + L.grid));
    p[0] = g0 ^ (u & 0x80008000u);
    p[1] = g1 ^ ((u << 1) & 0x80008000u);
    p[2] = g2 ^ ((u << 2) & 0x80008000u);
    p[3] = g3 ^ ((u << 3) & 0x80008000u);
}

// C = A * B with a zero accumulator
__device__ __forceinline__ void mma_bf16_z(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                          uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

// (d / 4) * (2 s + 1) of the sub-block word's top four bits (kquant.rs:667), exact: with v = 1 + s / 16 read off the word's bits it
// is 8 d v - 7.75 d, and d has 11 significant bits.  (A conversion from integer would be a quarter-rate instruction.)
struct Iq3Scale {
    float m, a;
    __device__ __forceinline__ explicit Iq3Scale(float d) : m(8.0f * d), a(-7.75f * d) {}
    __device__ __forceinline__ float of(uint32_t aux) const { return fmaf(__uint_as_float(((aux >> 9) & 0x00780000u) | 0x3f800000u), m, a); }
};

// One block (256 elements) of two IQ3_XXS rows against the B columns, sub-block by sub-block: the lane (g, t) decodes elements
// 8t .. 8t+7 of row `ba` (mma rows 0-7) and of row `bb` (mma rows 8-15); `y(ib)` gives the lane's B column for those eight elements.
// use(c, sa, sb): c[0], c[1] = row g of `ba`, columns 2t, 2t+1; c[2], c[3] = row g of `bb`; sa, sb the sub-block's scales.
// The eight sub-block words of a row come as aligned words shifted into place (a block starts on any even byte).
// What bounds it: the chain and the issue slots of the decode, 24 warps with a sub-block each in flight.  Signs from a table and
// scales without a conversion: gate and up of a one-token block (2048 x 512, 11 experts) 4.1 -> 3.6 us.
template <class Y, class Use>
__device__ __forceinline__ void iq3_block_mma(const uint8_t* ba, const uint8_t* bb, int t, const Iq3Lane& lutp, Y&& y_of, Use&& use) {
    const Iq3Scale da(h2f(ld16(ba))), db(h2f(ld16(bb)));
    const uint32_t ma = ((uint32_t)__cvta_generic_to_shared(ba) + 2u) & 2u, mb = ((uint32_t)__cvta_generic_to_shared(bb) + 2u) & 2u;
    const uint32_t* wa = reinterpret_cast<const uint32_t*>(ba + 66 - ma);
    const uint32_t* wb = reinterpret_cast<const uint32_t*>(bb + 66 - mb);
    const uint32_t sa = ma * 8u, sb = mb * 8u;
    const int st = (7 * t + 26) & 31;
    const uint8_t* ia = ba + 2 + 2 * t;
    const uint8_t* ib2 = bb + 2 + 2 * t;
    uint32_t la = wa[0], lb = wb[0];
#pragma unroll kIq3Unroll
    for (int ib = 0; ib < 8; ++ib) {
        // the ninth word belongs to the row only where the words are shifted
        const uint32_t na = wa[min(ib + 1, 7 + (int)(ma >> 1))], nb = wb[min(ib + 1, 7 + (int)(mb >> 1))];
        const uint32_t xa = __funnelshift_r(la, na, sa), xb = __funnelshift_r(lb, nb, sb);
        la = na;
        lb = nb;
        const uint4 y = y_of(ib);
        uint32_t p[4], q[4];
        float c[4];
        iq3_pairs(lutp, ld16(ia + 8 * ib), __funnelshift_r(xa, xa, st), p);
        iq3_pairs(lutp, ld16(ib2 + 8 * ib), __funnelshift_r(xb, xb, st), q);
        mma_bf16_z(c, p[0], q[0], p[1], q[1], y.x, y.y);
        mma_bf16(c, p[2], q[2], p[3], q[3], y.z, y.w);
        use(c, da.of(xa), db.of(xb));
    }
}

// Three-way bf16 split of an fp32 value: three 8-bit mantissas carry its 24 bits, and bf16 has fp32's
// exponent range, so v = h0 + h1 + h2 holds for every finite v (the subtractions are exact).
__device__ __forceinline__ void split3(float v, uint32_t (&h)[kGmSplit]) {
#pragma unroll
    for (int n = 0; n < kGmSplit; ++n) {
        h[n] = bf16_bits(v);
        v -= bf16_val(h[n]);
    }
}
// A gate/up group's share of one warp: blocks [b0, b1) of 8 gate rows (rowg: this lane's row g)
// and 8 up rows.  After the call lanes t = 0 and t = 1 of every row hold the row's two totals.
__device__ __forceinline__ void gate_up_warp(const uint8_t* rowg, const uint8_t* rowu, const Iq3Lane& lutp,
                                             const uint16_t* xb, bool has_col, int b0, int b1, int t, float& accg,
                                             float& accu) {
#pragma unroll 1
    for (int b = b0; b < b1; ++b)
        iq3_block_mma(
            rowg + b * 98, rowu + b * 98, t, lutp,
            [&](int ib) { return has_col ? *reinterpret_cast<const uint4*>(xb + (b * 8 + ib) * 32) : make_uint4(0u, 0u, 0u, 0u); },
            [&](const float (&c)[4], float sg, float su) {
                accg = fmaf(sg, c[0] + c[1], accg);
                accu = fmaf(su, c[2] + c[3], accu);
            });
    // lane t = 0 holds the hi and lo columns, t = 1 the lo2 column, t = 2, 3 nothing
    accg += __shfl_xor_sync(0xffffffffu, accg, 1);
    accu += __shfl_xor_sync(0xffffffffu, accu, 1);
}

// Barrier of the kGmKs warps of gate/up group q (named barriers 1 .. kGmGroups).  The ids are
// immediates so that the kernel reserves only the barriers it uses, not all sixteen.
__device__ __forceinline__ void group_barrier(int q) {
    switch (q) {
        case 0: asm volatile("bar.sync 1, %0;" ::"n"(kGmKs * 32) : "memory"); break;
        case 1: asm volatile("bar.sync 2, %0;" ::"n"(kGmKs * 32) : "memory"); break;
        case 2: asm volatile("bar.sync 3, %0;" ::"n"(kGmKs * 32) : "memory"); break;
        case 3: asm volatile("bar.sync 4, %0;" ::"n"(kGmKs * 32) : "memory"); break;
        default: asm volatile("bar.sync 5, %0;" ::"n"(kGmKs * 32) : "memory"); break;
    }
}

}  // namespace dnb
