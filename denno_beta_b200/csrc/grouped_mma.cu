// Grouped dequant matmul for few tokens per expert: decode batches, short prompts, caller-given selections, single
// matrices with a few vectors.  Q4_K, Q5_K, Q6_K, Q8_0 and IQ3_XXS on mma.sync with bytes (s8 or u8 x s8, integer sums).
//
// Reference kernels of this role: kernels_seg_k.cu:201-241, kernels_exp_iq_v2.cu:259-319 (one warp per row, fp32 FMA);
// block layouts kquant.rs:341-887.
//
// What bounds a call like this is instructions, not bytes: at HBM speed an SM has about four lane-instructions per weight
// of a 4-bit format, and an FMA kernel spends two (convert, multiply) per weight AND token.  Here a weight costs its
// decoding only, whatever the number of tokens, and it is decoded no further than to a byte:
//   * a lane turns packed bytes into the A fragment in registers (Q4_K: q, or 16 q where the nibble lies; Q5_K: q; Q6_K: 4 (q - 32);
//     Q8_0: q; IQ3_XXS: the codebook magnitude <= 62 with its sign), so no weight is rounded;
//   * the integer scales multiply the integer sums of a sub-block (Q4_K, Q5_K: sc, IQ3_XXS: 2 s + 1, 32 elements; Q6_K: 16 elements) and
//     add up over a 256-element block without rounding; d then multiplies in fp32.  (Q8_0 has a d per 32 elements.)  The mins of Q4_K
//     and Q5_K are one fp16 K step of m against the sub-block sums of the activations;
//   * an activation is an integer of 32 bits, of its 256-element block times a power of two, as four digits in base 256 in
//     four columns of B: rounded to 2^-31 of the block's largest.  Where that could be felt, in a block whose elements are of very
//     different size, what is left over is one more digit, of one more column tile.
// Why bytes: the logic and byte-permute instructions, fp16x2 and integer multiplies take two issue cycles of a scheduler here (FFMA and
// integer adds one), and an mma.sync of bytes (K = 32) eight, as one of fp16 (K = 16) does.  With fp16 weights a Q4_K weight pair was 2.3
// logic instructions and one fp16x2 multiply, now 0.6; 16 weights of an IQ3_XXS lane 34, now 25, and 12 instead of 18 shared-memory wavefronts.
//
// Work: an item is (segment, token tile, block of row groups); a row group is 16 A rows: 16 rows of one matrix, or 8 gate
// and 8 up rows of the same indices, whose results meet in one lane for silu(g) * u.  A persistent CTA of 16 warps stages
// an item's activations once; a warp then streams its row groups through a private ring of cp.async stages (one
// 256-element block of the 16 rows each) without any CTA-wide barrier.  Few row groups for the chip: KS warps share a row
// group, each takes a part of K, and their sums are added in a fixed order.  A row's result depends on the row and on KS, not on
// the tile, the column or the CTA; for decode batches KS is a constant of the shape, so that a token's bits do not depend on its batch.
//
// Measured, us of a launch, gate/up + down of 2048 x 512, top 10 of 512: fp16 operands in two or three parts -> bytes -> two blocks a stage and a
// loop for each number of column tiles -> 32 bits an activation and the remainders of wide blocks.  8 tokens: IQ3_XXS 49 + 31 -> 44 + 29 -> 41 + 27 -> 41 +
// 27, Q4_K 44 + 28 -> 33 + 23 -> 32 + 21 -> 32 + 23; 32 tokens: IQ3_XXS 115 + 68 -> 108 + 66 -> 101 + 62 -> 104 + 64, Q4_K 98 + 56 -> 75 + 45 -> 71 + 42 -> 71 + 49,
// Q8_0 151 + 92 -> 134 + 74 -> 111 + 64 -> 113 + 65; 200 tokens under a skewed router: Q4_K and Q6_K 302 + 175 -> 263 + 119 -> 154 + 120 -> 157 + 138, Q8_0 395 +
// 169 -> 249 + 135 -> 176 + 103 -> 189 + 105.  (One loop with unused column tiles switched off took the
// time of all of them, or not, as the compiler chose.)  Decoding alone is 30 (Q4_K) to 66 (IQ3_XXS) cycles of a scheduler for 16 rows x 32
// elements; bytes from HBM take 50 and 34.  Distance from the 64-bit result: see mm_stage_block.
#include <algorithm>
#include <type_traits>

#include "dnb_common.cuh"
#include "formats.cuh"
#include "tc_ptx.cuh"
#include "dnb_iq_tables.h"

namespace dnb {

constexpr int kMmWarps = 16;
constexpr int kMmThreads = kMmWarps * 32;
constexpr int kMmSegMax = 1088;  // segments of a launch at most
constexpr int kMmFixed = ((kMmSegMax + 4 + 16) * 4 + 127) / 128 * 128;  // segment table and the like in shared memory
// Where dynamic shared memory has to start for IQ3_XXS, whose tables' address is part of the instructions (as a register it costs 1.5 to 2 % of a
// batch).  The context knows where it starts (smem_base), and elsewhere mm_handles leaves the format to other kernels.
constexpr uint32_t kMmSmemBase = 1024;
constexpr int kMmTok = 2;        // tokens of a column tile: eight columns, four digits a token

// 256 elements of a row: bytes, and the pitch of a stage's rows with one and with two of them (a multiple of 16; a format whose blocks are
// not may start anywhere in its first 16 bytes).  The rows that are read together fall on different banks.
template <int T> struct Mq;
template <> struct Mq<T_Q4_K> { static constexpr int BB = 144, P1 = 160, P2 = 288; static constexpr bool ALIGNED = true; };
template <> struct Mq<T_Q5_K> { static constexpr int BB = 176, P1 = 176, P2 = 352; static constexpr bool ALIGNED = true; };
template <> struct Mq<T_Q6_K> { static constexpr int BB = 210, P1 = 240, P2 = 464; static constexpr bool ALIGNED = false; };
template <> struct Mq<T_IQ3_XXS> { static constexpr int BB = 98, P1 = 112, P2 = 240; static constexpr bool ALIGNED = false; };
template <> struct Mq<T_Q8_0> { static constexpr int BB = 272, P1 = 272, P2 = 544; static constexpr bool ALIGNED = true; };

template <int T> constexpr bool mq_mins = (T == T_Q4_K || T == T_Q5_K);

// ---- activations -----------------------------------------------------------------------------------------------------------
// A 256-element block of one token: [4 digits][256 bytes, unit u and lane t at 32 u + 8 t, kXDigit bytes apart: four digits of a
// lane's eight bytes fall on different banks; the 32 bytes between them: what is left over (mm_left_at)][3 parts][8] sub-block sums as fp16
// (formats with mins), then what undoes the scaling (two floats), and whether the block is wide.
constexpr int kXDigit = 288, kXSums = 4 * kXDigit, kXInv = kXSums + 48, kXWide = kXInv + 8, kXBlock = kXInv + 16;
__device__ __forceinline__ int mm_left_at(int u, int t) { return (u >> 1) * kXDigit + 256 + (u & 1) * 16 + 4 * t; }

// First element (of 256) of the two groups of four that unit u = 0..7 of lane t takes.
template <int T>
__device__ __forceinline__ void mm_unit_elems(int u, int t, int& e0, int& e1) {
    if constexpr (T == T_Q6_K) {
        e0 = (u >> 2) * 128 + (u & 1) * 32 + ((u >> 1) & 1) * 16 + 4 * t;
        e1 = e0 + 64;
    } else if constexpr (T == T_Q8_0) {
        e0 = 32 * u + 4 * t;
        e1 = e0 + 16;
    } else {
        e0 = 32 * u + 8 * t;
        e1 = e0 + 4;
    }
}
// The digits of four elements: d[j] = byte j of each.
__device__ __forceinline__ void mm_digits(const int (&v)[4], uint32_t (&d)[4]) {
    const uint32_t a = __byte_perm(v[0], v[1], 0x5140), b = __byte_perm(v[2], v[3], 0x5140);
    const uint32_t c = __byte_perm(v[0], v[1], 0x7362), e = __byte_perm(v[2], v[3], 0x7362);
    d[0] = __byte_perm(a, b, 0x5410);
    d[1] = __byte_perm(a, b, 0x7632);
    d[2] = __byte_perm(c, e, 0x5410);
    d[3] = __byte_perm(c, e, 0x7632);
}
// Two values as three fp16 pairs whose sums are the values: every bit of the elements above 1/1024 of the block's largest, and 2^-34 of the
// largest below, where the third part meets fp16's smallest number.
__device__ __forceinline__ void mm_split(float a, float b, uint32_t (&h)[3]) {
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        const __half2 v = __floats2half2_rn(a, b);
        h[p] = *reinterpret_cast<const uint32_t*>(&v);
        if (p < 2) {
            const float2 f = __half22float2(v);
            a -= f.x;
            b -= f.y;
        }
    }
}
__device__ __forceinline__ float mm_pow2(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }  // -126 <= e <= 127

// A lane's eight of the 256 elements at xr.
struct MmIn { float4 a, b; };
template <int T>
__device__ __forceinline__ MmIn mm_load_block(const float* xr, int lane) {
    int e0, e1;
    mm_unit_elems<T>(lane >> 2, lane & 3, e0, e1);
    return {*reinterpret_cast<const float4*>(xr + e0), *reinterpret_cast<const float4*>(xr + e1)};
}

// One warp: a token's 256 elements into their place in shared memory.  The block times 2^s, which puts its largest element into [2^30,
// 2^31), or into half of that where it would be above 0x7f7f7f7f, is rounded to integers; their four digits in base 256 are balanced (-128 ..
// 127), so that sum_j 256^j * d_j is the integer.
// That rounds elements below 2^24 (2^-7 to 2^-6 of the block's largest) to 2^-31 of the largest, which is less than what the sums are rounded
// by, unless hardly any weight hears the large elements.  So a block is called wide, and four more bits are kept of what the rounding left
// over, if fewer than 8 of its 32 lanes hold an element of 2^24 or more, or none of some unit's four (the 32 elements of a scale, which may be
// zero for the others), and other lanes are not zero.  Relative error against 64 bits with one element 2^j times the others in each block that
// no weight hears, Q8_0, K = 2048, in 1e-7, three fp16 parts of a row (as this kernel had before) / integers of 31 bits / these, j = 6: 0.91 /
// 0.88 / 0.83; 8: 0.91 / 1.6 / 0.82; 10: 0.97 / 5.6 / 0.84; 12: 1.7 / 22 / 1.05; 16: 22 / 354 / 12.  Over five formats, K of 512 to 4096, normal and
// heavy-tailed inputs, such outliers and small sub-blocks: at most 0.97 of the fp16 parts' error in any.
// Normal inputs have no wide blocks; of what the down projection meets, none or, behind a Q4_K or Q5_K layer whose mins drive most of a
// token's gates negative, a few in a hundred.  An item that has one costs a fifth more: a batch of 8 469 -> 472 us a pass, of 32 1,041 -> 1,050, a
// prompt of 77 357 -> 372 (before there were rests: 461, 1,023, 348).
// Returns whether the block is wide.
template <int T>
__device__ __forceinline__ bool mm_stage_block(const MmIn& in, uint8_t* dst, int lane) {
    const int u = lane >> 2, t = lane & 3;
    float x[8] = {in.a.x, in.a.y, in.a.z, in.a.w, in.b.x, in.b.y, in.b.z, in.b.w};
    uint32_t mine = 0u;
#pragma unroll
    for (int i = 0; i < 8; ++i) mine = max(mine, __float_as_uint(fabsf(x[i])));
    const uint32_t mx = __reduce_max_sync(0xffffffffu, mine);
    const int ex = (int)((mx + 0x10101u) >> 23);  // biased exponent of the largest |x|, one more where its mantissa is too large
    const int s = min(149, 157 - ex), s1 = min(s, 120);  // 149: every fp32 is an integer, subnormal ones too
    const float up = mm_pow2(s1);
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] *= up;
    if (s > s1) {  // a block below 2^-90 throughout: a second power of two
        const float up2 = mm_pow2(s - s1);
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] *= up2;
    }
    // lanes that have an element of 2^24 or more, lanes that have one at all; a unit is four lanes
    const uint32_t large = __ballot_sync(0xffffffffu, mine >= (uint32_t)(151 - s) << 23), some = __ballot_sync(0xffffffffu, mine != 0u);
    const uint32_t large4 = large | large >> 1 | large >> 2 | large >> 3, some4 = some | some >> 1 | some >> 2 | some >> 3;
    const bool wide = (some4 & ~large4 & 0x11111111u) != 0u || (__popc(large) < 8 && large != some);
    if constexpr (mq_mins<T>) {  // a sub-block is a unit: its sum over the four lanes, in units of 2^21
        float a = ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
        a += __shfl_xor_sync(0xffffffffu, a, 1);
        a += __shfl_xor_sync(0xffffffffu, a, 2);
        a *= 0x1p-21f;
        const float b = __shfl_xor_sync(0xffffffffu, a, 4);
        uint32_t h[3];
        mm_split(a, b, h);
        if ((lane & 7) == 0) {
#pragma unroll
            for (int p = 0; p < 3; ++p) *reinterpret_cast<uint32_t*>(dst + kXSums + p * 16 + (lane >> 3) * 4) = h[p];
        }
    }
    int v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = (int)(((uint32_t)__float2int_rn(x[i]) + 0x00808080u) ^ 0x00808080u);
    uint32_t d0[4], d1[4];
    mm_digits({v[0], v[1], v[2], v[3]}, d0);
    mm_digits({v[4], v[5], v[6], v[7]}, d1);
#pragma unroll
    for (int j = 0; j < 4; ++j) *reinterpret_cast<uint2*>(dst + j * kXDigit + lane * 8) = make_uint2(d0[j], d1[j]);
    // 2^-s for the low two digits, 2^(16 - s) for the high two; a block with an infinity or a NaN makes a NaN of every sum
    if (lane < 2) {
        const int e = 16 * lane - s;
        reinterpret_cast<float*>(dst + kXInv)[lane] = mx >= 0x7f800000u ? __uint_as_float(0x7fc00000u) : e >= -126 ? mm_pow2(e) : __uint_as_float(1u << (149 + e));
    }
    if (lane == 2) *reinterpret_cast<uint32_t*>(dst + kXWide) = wide ? 1u : 0u;
    if (__builtin_expect(wide, 0)) {
        // what is left over in fifteenths, -7 .. 7 (not to -8: with a bias, weights that are all positive would add it up); elements 4 .. 7 in the
        // lower nibbles of the bytes, 0 .. 3 in the upper
        uint32_t left = 0u;
#pragma unroll
        for (int i = 0; i < 8; ++i) left |= ((uint32_t)max(-7, min(7, __float2int_rn((x[i] - rintf(x[i])) * 15.f))) & 15u) << (8 * (i & 3) + (i < 4 ? 4 : 0));
        *reinterpret_cast<uint32_t*>(dst + mm_left_at(u, t)) = left;
    }
    return wide;
}

// ---- integer products --------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void mma_u8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint2 b) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b.x), "r"(b.y), "r"(0));
}
template <int C0>  // every element of C
__device__ __forceinline__ void mma_s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint2 b) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b.x), "r"(b.y), "r"(C0));
}
__device__ __forceinline__ void mma_s8_k16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b) {
    asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a0), "r"(a1), "r"(b), "r"(0));
}
__device__ __forceinline__ void mma_f16_z(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ uint32_t ld32u(const uint8_t* p) { return ld16(p) | (ld16(p + 2) << 16); }  // 2-byte aligned

// Q4_K / Q5_K header of a row: d, dmin, the eight scales (a byte each) and the pair of mins of sub-blocks 2 t, 2 t + 1 (kquant.rs:878-887).
struct MmK { float d, dmin; uint32_t sc[2], mm; };
__device__ __forceinline__ MmK mm_k_header(const uint8_t* row, int t) {
    const uint4 h = *reinterpret_cast<const uint4*>(row);
    MmK r;
    r.d = h2f((uint16_t)h.x);
    r.dmin = h2f((uint16_t)(h.x >> 16));
    r.sc[0] = h.y & 0x3f3f3f3fu;
    r.sc[1] = (h.w & 0x0f0f0f0fu) | ((h.y >> 2) & 0x30303030u);
    const int sh = 16 * (t & 1);
    const uint32_t mn = (t < 2 ? h.z & 0x3f3f3f3fu : ((h.w >> 4) & 0x0f0f0f0fu) | ((h.z >> 2) & 0x30303030u)) >> sh;
    r.mm = h2sub(__byte_perm(mn, 0x64646464u, 0x4140u), 0x64006400u);
    return r;
}

// IQ3_XXS tables in shared memory, 128 bytes from entry to entry, so that a lane's copies are on banks of its own:
//   grid: the four magnitudes of a codebook entry, a byte each (lane i reads copy i)
//   sgn : the signs of a 7-bit code (the eighth makes their number even) as 0 or 1 in a byte each: weights 0-3, 4-7 (copy i mod 16)
// They are the first thing in shared memory, an address that the instructions hold.
struct MmTables { uint32_t grid[256 * 32]; uint2 sgn[128 * 16]; };
static __device__ __align__(16) MmTables g_mm_s8;
static TablesOnce g_mm_s8_up;

static int upload_mm_s8(int device) {
    return tables_once(g_mm_s8_up, device, [] {
        static MmTables tb;
        for (int e = 0; e < 256; ++e)
            for (int r = 0; r < 32; ++r) tb.grid[e * 32 + r] = dnb_iq3xxs_grid[e];
        for (uint32_t code = 0; code < 128; ++code) {
            const uint32_t sg = code | ((uint32_t)(__builtin_popcount(code) & 1) << 7);
            uint2 u = make_uint2(0u, 0u);
            for (int i = 0; i < 4; ++i) {
                u.x |= ((sg >> i) & 1u) << (8 * i);
                u.y |= ((sg >> (4 + i)) & 1u) << (8 * i);
            }
            for (int r = 0; r < 16; ++r) tb.sgn[code * 16 + r] = u;
        }
        DNB_CUDA(cudaMemcpyToSymbol(g_mm_s8, &tb, sizeof(tb)));
        return DNB_OK;
    });
}

// Eight weights of an IQ3_XXS sub-block as signed bytes.  gl, sl: where the lane's copies are in an entry; idx: the two codebook indices; code:
// the sub-block word rotated so that the quarter's 7-bit sign code starts at bit 7.  A negative byte is ~v + 1 (v >= 4: nothing carries).
__device__ __forceinline__ void iq3_s8(uint32_t gl, uint32_t sl, uint32_t idx, uint32_t code, uint32_t& p0, uint32_t& p1) {
    uint32_t o0, o1, g0, g1;  // constant tables: plain asm, free to move
    asm("ld.shared.v2.u32 {%0, %1}, [%2 + %3];" : "=r"(o0), "=r"(o1) : "r"((code & 0x3f80u) | sl), "n"(kMmSmemBase + 256 * 32 * 4));
    asm("ld.shared.u32 %0, [%1 + %2];" : "=r"(g0) : "r"(((idx << 7) & 0x7f80u) | gl), "n"(kMmSmemBase));
    asm("ld.shared.u32 %0, [%1 + %2];" : "=r"(g1) : "r"(((idx >> 1) & 0x7f80u) | gl), "n"(kMmSmemBase));
    p0 = (g0 ^ (o0 * 255u)) + o0;
    p1 = (g1 ^ (o1 * 255u)) + o1;
}
// A CTA's copy of the tables; complete after the caller's barrier.
__device__ __forceinline__ void mm_tables_in(uint8_t* dst, int tid, int threads) {
    for (int i = tid; i < (int)(sizeof(MmTables) / 16); i += threads)
        tcp::cp_async16<false>(dst + 16 * i, reinterpret_cast<const uint8_t*>(&g_mm_s8) + 16 * i);
    tcp::cp_async_commit();
}

// ---- weights ---------------------------------------------------------------------------------------------------------------------
// A warp's ring of stages: one or two blocks of each of 16 rows, in 16-byte copies: a lane copies unit lane % 8 (+ 8, 16, ..) of rows
// lane / 8 + 0, 4, 8, 12.  Two blocks a stage halve what is spent on addresses and counters, and lift what copies alone reach from 4.6 to 5.7
// TB/s.  What a copy costs is its cache lines: four lanes to a row, with half the addresses, are 10 % slower, and so is one copy of all rows' last
// units where a block leaves one over (Q8_0 by 10 %).  (Bulk copies per row reach 5.6 TB/s, but each costs the warp a turn of a loop of a dozen
// instructions, a request of sixteen rows as many as decoding a block.)
struct MmRing { int nst, bps, pitch; };
template <int T>
struct MmStream {
    using Q = Mq<T>;
    uint8_t* mem;  // of this warp
    int nst, bps, pitch;
    uint32_t at;   // of this lane in a stage
    int lane, in = 0, out = 0;  // slots that are filled and read next
    const uint8_t *sa, *sb;       // rows lane / 8 and lane / 8 + 8
    uint32_t o1, o3;              // from there to rows lane / 8 + 4 and + 12
    __device__ __forceinline__ MmStream(uint8_t* m, const MmRing& r, int ln)
        : mem(m), nst(r.nst), bps(r.bps), pitch(r.pitch), at((ln >> 3) * r.pitch + (ln & 7) * 16), lane(ln), sa(nullptr), sb(nullptr), o1(0), o3(0) {}
    // the next requests are for rows r, r + 1, ... of w, or (pair) eight rows from r on of wa and of wb; no row beyond `last`
    template <bool PAIR>
    __device__ __forceinline__ void point(const uint8_t* wa, const uint8_t* wb, int r, int last, uint32_t rb) {
        const int q = lane >> 3;
        if constexpr (PAIR) {
            const size_t off = (size_t)(r + q) * rb;
            sa = wa + off;
            sb = wb + off;
            o1 = o3 = 4u * rb;
        } else {
            const int r0 = min(r + q, last), r2 = min(r + q + 8, last);
            sa = wa + (size_t)r0 * rb;
            sb = wa + (size_t)r2 * rb;
            o1 = (uint32_t)(min(r + q + 4, last) - r0) * rb;
            o3 = (uint32_t)(min(r + q + 12, last) - r2) * rb;
        }
    }
    __device__ __forceinline__ void request(int n) {  // n blocks of them; an empty request keeps the count of groups
        if (n > 0) {
            const int c16 = (lane & 7) * 16;
            uint8_t* dst = mem + in * 16 * pitch + at;
#pragma unroll
            for (int j = 0; j < 4; ++j, dst += 4 * pitch) {
                const uint8_t* src = (j < 2 ? sa : sb) + (j == 1 ? o1 : j == 3 ? o3 : 0u);
                int bytes = n * Q::BB;
                if constexpr (!Q::ALIGNED) {
                    bytes += (int)((uintptr_t)src & 15);
                    src = reinterpret_cast<const uint8_t*>((uintptr_t)src & ~(uintptr_t)15);
                }
#pragma unroll
                for (int cc = 0; cc < 2 * Q::BB + (Q::ALIGNED ? 0 : 14); cc += 128)
                    if (cc + 128 <= Q::BB || cc + c16 < bytes) tcp::cp_async16(dst + cc, src + c16 + cc);
            }
            sa += n * Q::BB;
            sb += n * Q::BB;
            if (++in == nst) in = 0;
        }
        tcp::cp_async_commit();
    }
    __device__ __forceinline__ void skip(int bytes) {  // between requests
        sa += bytes;
        sb += bytes;
    }
    __device__ __forceinline__ const uint8_t* wait() {  // rows 0-15 of the next stage; every lane has left the one before
        if (nst == 2) asm volatile("cp.async.wait_group 0;" ::: "memory");
        else if (nst == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 2;" ::: "memory");
        __syncwarp();
        return mem + out * 16 * pitch;
    }
    __device__ __forceinline__ void next() {
        if (++out == nst) out = 0;
    }
};

// One 256-element block of 16 rows (this lane: rows `ra` and `rb`) against NT column tiles; bq(i, u): unit u of the lane's B column of tile
// i at this block; inv, sumw: of the token whose columns the lane's accumulators hold, and of its B column.
// acc[i] += scales * sums: rows `ra` and `rb`, digits 0 and 1 of a token (t even) or 2 and 3 (t odd).
// REST: one more column tile, NT, whose columns are eight tokens; left: rows `ra` and `rb` of columns 2 t, 2 t + 1, without an `inv`.
template <int T, int NT, bool REST, class B>
__device__ __forceinline__ void mm_block(const uint8_t* ra, const uint8_t* rb, int t, uint32_t gl, uint32_t sl, const B& bq, const uint32_t (&sumw)[NT], const float (&inv)[NT], float (&acc)[NT][2], float (&left)[2][2]) {
    constexpr int N1 = NT + (REST ? 1 : 0);
    if constexpr (T == T_Q8_0) {
        float s[NT][2];
#pragma unroll
        for (int n = 0; n < NT; ++n) s[n][0] = s[n][1] = 0.f;
#pragma unroll
        for (int ib = 0; ib < 8; ++ib) {
            // the bytes start 2 or 4 bytes behind an aligned word; a lane takes words t and t + 4 of them
            uint32_t p[2], q[2];
            const uint8_t *a = ra + 34 * ib + 4 * t, *b = rb + 34 * ib + 4 * t;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (ib & 1) {
                    p[h] = *reinterpret_cast<const uint32_t*>(a + 2 + 16 * h);
                    q[h] = *reinterpret_cast<const uint32_t*>(b + 2 + 16 * h);
                } else {
                    p[h] = __byte_perm(*reinterpret_cast<const uint32_t*>(a + 16 * h), *reinterpret_cast<const uint32_t*>(a + 16 * h + 4), 0x5432);
                    q[h] = __byte_perm(*reinterpret_cast<const uint32_t*>(b + 16 * h), *reinterpret_cast<const uint32_t*>(b + 16 * h + 4), 0x5432);
                }
            }
            const float fa = h2f(ld16(ra + 34 * ib)), fb = h2f(ld16(rb + 34 * ib));
#pragma unroll
            for (int n = 0; n < N1; ++n) {
                // sums start at the bits of 1.5 * 2^23, so that they are floats as they stand (|sum| <= 2^19)
                int D[4];
                mma_s8<0x4B400000>(D, p[0], q[0], p[1], q[1], bq(n, ib));
                const float m = 12582912.f;
                if (REST && n == NT) {
                    left[0][0] = fmaf(fa, __int_as_float(D[0]) - m, left[0][0]);
                    left[0][1] = fmaf(fa, __int_as_float(D[1]) - m, left[0][1]);
                    left[1][0] = fmaf(fb, __int_as_float(D[2]) - m, left[1][0]);
                    left[1][1] = fmaf(fb, __int_as_float(D[3]) - m, left[1][1]);
                    continue;
                }
                s[n][0] = fmaf(fa, fmaf(256.f, __int_as_float(D[1]) - m, __int_as_float(D[0]) - m), s[n][0]);
                s[n][1] = fmaf(fb, fmaf(256.f, __int_as_float(D[3]) - m, __int_as_float(D[2]) - m), s[n][1]);
            }
        }
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            acc[n][0] = fmaf(s[n][0], inv[n], acc[n][0]);
            acc[n][1] = fmaf(s[n][1], inv[n], acc[n][1]);
        }
    } else {
        int c[N1][4];
#pragma unroll
        for (int n = 0; n < N1; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) c[n][i] = 0;
        // one sub-block: its sums times its scales
        auto add = [&](int n, const int (&D)[4], int fa, int fb) {
            c[n][0] += fa * D[0];
            c[n][1] += fa * D[1];
            c[n][2] += fb * D[2];
            c[n][3] += fb * D[3];
        };
        float da, db, dma = 0.f, dmb = 0.f;
        uint32_t mma = 0u, mmb = 0u;
        if constexpr (mq_mins<T>) {
            // bounds of a block's sums: Q4_K 8 * 16 * 63 * 32 * 15 * 128 < 2^29 (see below for the 16), Q5_K 8 * 63 * 32 * 31 * 128 < 2^26
            const MmK ka = mm_k_header(ra, t), kb = mm_k_header(rb, t);
            da = ka.d; db = kb.d; dma = ka.dmin; dmb = kb.dmin; mma = ka.mm; mmb = kb.mm;
            constexpr bool FIVE = T == T_Q5_K;
            uint2 ha = make_uint2(0u, 0u), hb = ha;
            if constexpr (FIVE) {
                ha = *reinterpret_cast<const uint2*>(ra + 16 + 8 * t);
                hb = *reinterpret_cast<const uint2*>(rb + 16 + 8 * t);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {  // sub-blocks 2 j (low nibbles) and 2 j + 1 (high)
                const uint2 qa = *reinterpret_cast<const uint2*>(ra + (FIVE ? 48 : 16) + 32 * j + 8 * t);
                const uint2 qb = *reinterpret_cast<const uint2*>(rb + (FIVE ? 48 : 16) + 32 * j + 8 * t);
                const uint32_t wa = ka.sc[j >> 1] >> (16 * (j & 1)), wb = kb.sc[j >> 1] >> (16 * (j & 1));
                int fa[2] = {(int)(wa & 0xffu), (int)((wa >> 8) & 0xffu)}, fb[2] = {(int)(wb & 0xffu), (int)((wb >> 8) & 0xffu)};
                uint32_t a[2][2], b[2][2];
                if constexpr (FIVE) {
                    auto fifth = [&](uint32_t h, int u) { return (u < 4 ? h << (4 - u) : h >> (u - 4)) & 0x10101010u; };
                    a[0][0] = (qa.x & 0x0f0f0f0fu) | fifth(ha.x, 2 * j);
                    a[0][1] = (qa.y & 0x0f0f0f0fu) | fifth(ha.y, 2 * j);
                    b[0][0] = (qb.x & 0x0f0f0f0fu) | fifth(hb.x, 2 * j);
                    b[0][1] = (qb.y & 0x0f0f0f0fu) | fifth(hb.y, 2 * j);
                    a[1][0] = ((qa.x >> 4) & 0x0f0f0f0fu) | fifth(ha.x, 2 * j + 1);
                    a[1][1] = ((qa.y >> 4) & 0x0f0f0f0fu) | fifth(ha.y, 2 * j + 1);
                    b[1][0] = ((qb.x >> 4) & 0x0f0f0f0fu) | fifth(hb.x, 2 * j + 1);
                    b[1][1] = ((qb.y >> 4) & 0x0f0f0f0fu) | fifth(hb.y, 2 * j + 1);
                } else {  // the high nibbles stay where they are, 16 times too large, and the even sub-blocks' scales take the 16, too
                    a[0][0] = qa.x & 0x0f0f0f0fu; a[0][1] = qa.y & 0x0f0f0f0fu;
                    b[0][0] = qb.x & 0x0f0f0f0fu; b[0][1] = qb.y & 0x0f0f0f0fu;
                    a[1][0] = qa.x & 0xf0f0f0f0u; a[1][1] = qa.y & 0xf0f0f0f0u;
                    b[1][0] = qb.x & 0xf0f0f0f0u; b[1][1] = qb.y & 0xf0f0f0f0u;
                    fa[0] *= 16;
                    fb[0] *= 16;
                }
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int n = 0; n < N1; ++n) {
                        int D[4];
                        mma_u8(D, a[h][0], b[h][0], a[h][1], b[h][1], bq(n, 2 * j + h));
                        add(n, D, fa[h], fb[h]);
                    }
            }
            if constexpr (!FIVE) {
                da *= 0.0625f;
                db *= 0.0625f;
            }
        } else if constexpr (T == T_IQ3_XXS) {  // (d / 4) * (2 s + 1) (kquant.rs:667); sums: 8 * 31 * 32 * 62 * 128 < 2^26
            da = 0.25f * h2f(ld16(ra));
            db = 0.25f * h2f(ld16(rb));
            // the eight sub-block words of a row as aligned words, shifted into place (a block starts on any even byte)
            const uint32_t ma = (tcp::s32(ra) + 2u) & 2u, mb = (tcp::s32(rb) + 2u) & 2u;
            const uint32_t* wa = reinterpret_cast<const uint32_t*>(ra + 66 - ma);
            const uint32_t* wb = reinterpret_cast<const uint32_t*>(rb + 66 - mb);
            const uint32_t sa = ma * 8u, sb = mb * 8u;
            const uint8_t* ia = ra + 2 + 2 * t;
            const uint8_t* ib2 = rb + 2 + 2 * t;
            const int st = (7 * t + 25) & 31;
            uint32_t la = wa[0], lb = wb[0];
#pragma unroll
            for (int ib = 0; ib < 8; ++ib) {
                // the ninth word belongs to the row only where the words are shifted
                const uint32_t naw = wa[ib < 7 ? ib + 1 : 7 + (ma >> 1)], nbw = wb[ib < 7 ? ib + 1 : 7 + (mb >> 1)];
                const uint32_t xa = __funnelshift_r(la, naw, sa), xb = __funnelshift_r(lb, nbw, sb);
                la = naw;
                lb = nbw;
                uint32_t p[2], q[2];
                iq3_s8(gl, sl, ld16(ia + 8 * ib), __funnelshift_r(xa, xa, st), p[0], p[1]);
                iq3_s8(gl, sl, ld16(ib2 + 8 * ib), __funnelshift_r(xb, xb, st), q[0], q[1]);
                const int fa = (int)(2u * (xa >> 28) + 1u), fb = (int)(2u * (xb >> 28) + 1u);
#pragma unroll
                for (int n = 0; n < N1; ++n) {
                    int D[4];
                    mma_s8<0>(D, p[0], q[0], p[1], q[1], bq(n, ib));
                    add(n, D, fa, fb);
                }
            }
        } else {  // Q6_K: a K step is one 16-element group of one scale; bytes are 4 * (q - 32), sums 16 * 128 * 16 * 128 * 128 < 2^30
            da = 0.25f * h2f(ld16(ra + 208));
            db = 0.25f * h2f(ld16(rb + 208));
#pragma unroll
            for (int g = 0; g < 4; ++g) {  // (half, is)
                const int half = g >> 1, is = g & 1;
                // the upper bit of each pair inverted: q - 32 in two's complement
                const uint32_t ha = ld32u(ra + 128 + 32 * half + 16 * is + 4 * t) ^ 0xaaaaaaaau, hb = ld32u(rb + 128 + 32 * half + 16 * is + 4 * t) ^ 0xaaaaaaaau;
#pragma unroll
                for (int w = 0; w < 2; ++w) {
                    const uint32_t qa = ld32u(ra + 64 * half + 32 * w + 16 * is + 4 * t), qb = ld32u(rb + 64 * half + 32 * w + 16 * is + 4 * t);
                    uint2 y[N1];
#pragma unroll
                    for (int n = 0; n < N1; ++n)
                        y[n] = bq(n, 2 * g + w);
#pragma unroll
                    for (int hi = 0; hi < 2; ++hi) {
                        const int sh = 6 - 2 * w - 4 * hi;  // the pair of bits to the top of its byte
                        const uint32_t va = ((hi ? qa >> 2 : qa << 2) & 0x3c3c3c3cu) | ((ha << sh) & 0xc0c0c0c0u);
                        const uint32_t vb = ((hi ? qb >> 2 : qb << 2) & 0x3c3c3c3cu) | ((hb << sh) & 0xc0c0c0c0u);
                        const int sc = 192 + 8 * half + is + 2 * w + 4 * hi;
                        const int fa = *reinterpret_cast<const int8_t*>(ra + sc), fb = *reinterpret_cast<const int8_t*>(rb + sc);
#pragma unroll
                        for (int n = 0; n < N1; ++n) {
                            int D[4];
                            mma_s8_k16(D, va, vb, hi ? y[n].y : y[n].x);
                            add(n, D, fa, fb);
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            float va = da * fmaf(256.f, (float)c[n][1], (float)c[n][0]), vb = db * fmaf(256.f, (float)c[n][3], (float)c[n][2]);
            if constexpr (mq_mins<T>) {
                float M[4];
                mma_f16_z(M, mma, mmb, 0u, 0u, sumw[n], 0u);
                const float k = (t & 1) ? 32.f : 0x1p21f;  // columns 0, 1 of a token stand beside its low digits, column 2 beside the high ones
                va = fmaf(-dma, (M[0] + M[1]) * k, va);
                vb = fmaf(-dmb, (M[2] + M[3]) * k, vb);
            }
            acc[n][0] = fmaf(va, inv[n], acc[n][0]);
            acc[n][1] = fmaf(vb, inv[n], acc[n][1]);
        }
        if constexpr (REST) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                left[0][i] = da * (float)c[NT][i];
                left[1][i] = db * (float)c[NT][2 + i];
            }
        }
    }
}

struct MmArgs {
    const SegDesc* seg;        // or null: `single`
    const int32_t* nseg_dev;   // or null: nseg_max segments
    SegDesc single;
    int nseg_max;
    int n_in, n_out, rb;       // rb: bytes of a row
    const float* x;            // fp32 rows
    int ldx;
    const int32_t* row_token;  // packed row -> x row, or null
    float* out;                // [packed row][n_out]
    int ks;                    // warps that split K
    MmRing ring;
    int skip;                  // row groups' time that a tile's activations take
    int* status;
};

__device__ __forceinline__ void mm_barrier(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// What a warp does of an item.
struct MmItem {
    const uint8_t *wa, *wb;    // the segment's matrices
    const uint8_t* acts;       // [m tokens][nb blocks][kXBlock]
    float* red;                // [2][16 warps][tiles * 2][32] when ks > 1
    float* out;                // the first token's results
    int m, nb, kb0, kbn;       // tokens; blocks of K, first and number of this warp's
    int rg, nrg, nslot;        // first row group and number of them, every nslot-th
    int n_out, rb, ks, slot, kpart;
};

// The warp's weight stream: the next blocks of the next row group.
template <int T, bool FUSED>
struct MmFeed {
    MmStream<T> w;
    int rg, b;
    __device__ __forceinline__ void prefetch(const MmItem& I) {
        int n = 0;
        if (rg < I.rg + I.nrg * I.nslot) {
            if (b == 0) {
                const uint32_t boff = (uint32_t)I.kb0 * Mq<T>::BB;
                w.template point<FUSED>(I.wa + boff, FUSED ? I.wb + boff : nullptr, rg * (FUSED ? 8 : 16), I.n_out - 1, (uint32_t)I.rb);
            }
            n = min(w.bps, I.kbn - b);
            b += n;
            if (b == I.kbn) {
                b = 0;
                rg += I.nslot;
            }
        }
        w.request(n);
    }
};

// One block of the 16 rows with what is left over of the wide ones among the tokens: one more column tile, token g's bytes are sixteen
// times the fifteenths.  token(k): token k's block.
template <int T, int N, class Token>
__device__ __forceinline__ void mm_block_wide(const uint8_t* ra, const uint8_t* rb, int lane, const Token& token, const uint8_t* const (&bp)[N],
                                              const uint32_t (&sumw)[N], const float (&inv)[N], float (&acc)[N][2]) {
    const int g = lane >> 2, t = lane & 3;
    auto is_wide = [&](int k) { return *reinterpret_cast<const uint32_t*>(token(k) + kXWide) != 0u; };
    const uint8_t* rest = token(g) + mm_left_at(0, t);
    const uint32_t mask = is_wide(g) ? 0xf0f0f0f0u : 0u;
    auto column = [&](int n, int u) {
        if (n < N) return *reinterpret_cast<const uint2*>(bp[n < N ? n : 0] + u * 32);
        const uint32_t v = *reinterpret_cast<const uint32_t*>(rest + mm_left_at(u, 0) - mm_left_at(0, 0));
        return make_uint2(v & mask, (v << 4) & mask);
    };
    float left[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
    mm_block<T, N, true>(ra, rb, t, 4 * lane, 8 * (lane & 15), column, sumw, inv, acc, left);
#pragma unroll
    for (int n = 0; n < N; ++n) {  // from lane t = n to the lanes that hold the low digits' sums of tokens 2 n, 2 n + 1
        const bool add = !(t & 1) && is_wide(n * kMmTok + (t >> 1));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float v0 = __shfl_sync(0xffffffffu, left[h][0], (g << 2) + n), v1 = __shfl_sync(0xffffffffu, left[h][1], (g << 2) + n);
            if (add) acc[n][h] = fmaf(t ? v1 : v0, (1.f / 240.f) * inv[n], acc[n][h]);
        }
    }
}

// The item's row groups with N column tiles (those behind the last token repeat it); REST: with what is left over of wide blocks, too.
template <int T, bool FUSED, int N, bool REST>
__device__ __forceinline__ void mm_row_groups(const MmItem& I, MmFeed<T, FUSED>& F) {
    using Q = Mq<T>;
    const int lane = F.w.lane, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const uint32_t gl = 4 * lane, sl = 8 * (lane & 15);
    auto token = [&](int k) { return I.acts + (size_t)min(k, I.m - 1) * I.nb * kXBlock; };
    const uint8_t *colb[N], *colv[N];  // the token of this lane's B column, and of its accumulators
#pragma unroll
    for (int n = 0; n < N; ++n) {
        colb[n] = token(n * kMmTok + (g >> 2));
        colv[n] = token(n * kMmTok + (t >> 1)) + kXInv + (t & 1) * 4;
    }
    float acc[N][2];
    for (int round = 0, rg = I.rg; round < I.nrg; ++round, rg += I.nslot) {
        // where a row's blocks start (only the position inside 16 bytes matters)
        uint32_t offa = 0, offb = 0;
        if constexpr (!Q::ALIGNED) {
            const uint32_t r0 = FUSED ? rg * 8 + g : min(rg * 16 + g, I.n_out - 1), r1 = FUSED ? r0 : (uint32_t)min(rg * 16 + 8 + g, I.n_out - 1);
            offa = r0 * (uint32_t)I.rb + (uint32_t)I.kb0 * Q::BB;
            offb = r1 * (uint32_t)I.rb + (uint32_t)I.kb0 * Q::BB;
        }
#pragma unroll
        for (int n = 0; n < N; ++n) acc[n][0] = acc[n][1] = 0.f;
#pragma unroll 1
        for (int b = 0; b < I.kbn;) {
            const uint8_t* st = F.w.wait();  // and every lane has left the slot that is filled next
            F.prefetch(I);
            const uint8_t *ra = st + g * F.w.pitch + (Q::ALIGNED ? 0u : offa & 15u), *rb = st + (g + 8) * F.w.pitch + (Q::ALIGNED ? 0u : offb & 15u);
            const int stop = min(b + F.w.bps, I.kbn);
            offa += (stop - b) * Q::BB;
            offb += (stop - b) * Q::BB;
#pragma unroll 1
            for (; b < stop; ++b, ra += Q::BB, rb += Q::BB) {
                const uint8_t* bp[N];
                uint32_t sumw[N];
                float inv[N];
                const int at_b = (I.kb0 + b) * kXBlock;
#pragma unroll
                for (int n = 0; n < N; ++n) {
                    bp[n] = colb[n] + at_b + (g & 3) * kXDigit + t * 8;
                    inv[n] = *reinterpret_cast<const float*>(colv[n] + at_b);
                    sumw[n] = 0u;  // the fourth column of a token takes no sums
                    if constexpr (mq_mins<T>) {
                        if ((g & 3) < 3) sumw[n] = *reinterpret_cast<const uint32_t*>(colb[n] + at_b + kXSums + (g & 3) * 16 + t * 4);
                    }
                }
                if constexpr (!REST) {
                    float none[2][2];
                    mm_block<T, N, false>(ra, rb, t, gl, sl, [&](int n, int u) { return *reinterpret_cast<const uint2*>(bp[n] + u * 32); }, sumw, inv, acc, none);
                } else {
                    mm_block_wide<T, N>(ra, rb, lane, [&](int k) { return token(k) + at_b; }, bp, sumw, inv, acc);
                }
            }
            F.w.next();
        }
        bool mine = true;
        if (I.ks > 1) {  // the warps of the row group meet; the first adds the others' sums in order
            float* rp = I.red + ((size_t)(round & 1) * kMmWarps + warp) * N * 2 * 32 + lane;
            mine = I.kpart == 0;
            if (!mine) {
#pragma unroll
                for (int n = 0; n < N; ++n)
#pragma unroll
                    for (int c = 0; c < 2; ++c) rp[(n * 2 + c) * 32] = acc[n][c];
            }
            mm_barrier(1 + I.slot, I.ks * 32);
            if (mine) {
                for (int k2 = 1; k2 < I.ks; ++k2) {
                    rp += N * 2 * 32;
#pragma unroll
                    for (int n = 0; n < N; ++n)
#pragma unroll
                        for (int c = 0; c < 2; ++c) acc[n][c] += rp[(n * 2 + c) * 32];
                }
            }
        }
        if (mine) {
#pragma unroll
            for (int n = 0; n < N; ++n) {
                // the low two digits' sums and the high two's meet: both lanes have both rows of the token
                float a = acc[n][0], b = acc[n][1];
                a += __shfl_xor_sync(0xffffffffu, a, 1);
                b += __shfl_xor_sync(0xffffffffu, b, 1);
                const int tok = n * kMmTok + (t >> 1);
                if (tok < I.m) {
                    float* o = I.out + (size_t)tok * I.n_out;
                    if constexpr (FUSED) {
                        if (!(t & 1)) o[rg * 8 + g] = a / (1.0f + expf(-a)) * b;
                    } else {
                        const int r = rg * 16 + g;
                        if (!(t & 1) && r < I.n_out) o[r] = a;
                        if ((t & 1) && r + 8 < I.n_out) o[r + 8] = b;
                    }
                }
            }
        }
    }
}
// Where things are in a CTA's shared memory, behind the IQ3_XXS tables.
struct MmShared {
    int* pre;        // [kMmSegMax + 1] first token tile of a segment
    int* wsum;       // [16]
    float* red;      // [2][16 warps][NT * 2][32] when ks > 1
    uint8_t* acts;   // [tokens of an item][blocks][kXBlock]
    uint8_t* ring;   // of the warp
};
template <int T, int NT>
__device__ __forceinline__ MmShared mm_shared(uint8_t* smem, const MmArgs& A) {
    MmShared S;
    uint8_t* p = smem + (T == T_IQ3_XXS ? sizeof(MmTables) : 0);
    S.pre = reinterpret_cast<int*>(p);
    S.wsum = S.pre + kMmSegMax + 4;
    p += kMmFixed;
    S.red = reinterpret_cast<float*>(p);
    if (A.ks > 1) p += 2 * kMmWarps * NT * 2 * 32 * sizeof(float);
    S.acts = p;
    S.ring = p + (size_t)NT * kMmTok * (A.n_in >> 8) * kXBlock + (size_t)(threadIdx.x >> 5) * A.ring.nst * 16 * A.ring.pitch;
    return S;
}

// The CTA's items.
template <int T, bool FUSED, int NT>
__device__ __forceinline__ void mm_items(const MmArgs& A, const MmShared& S, int nseg) {
    constexpr int TT = NT * kMmTok;  // tokens of an item
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nb = A.n_in >> 8;
    MmFeed<T, FUSED> F{MmStream<T>(S.ring, A.ring, lane), 0, 0};
    const int nslot = kMmWarps / A.ks, slot = warp / A.ks, kpart = warp - slot * A.ks;
    const int kb0 = nb * kpart / A.ks, kbn = nb * (kpart + 1) / A.ks - kb0;
    const int n_rg = FUSED ? A.n_out / 8 : (A.n_out + 15) / 16;
    // This CTA's share of all (tile, row group) pairs: a range of pairs in a row.  Another tile means another set of activations,
    // which takes as long as A.skip row groups: each tile is that much longer, and a CTA that has two gets so much less of them.
    const int span = n_rg + A.skip, total = S.pre[nseg] * span;
    const int share = total / (int)gridDim.x, extra = total - share * (int)gridDim.x;
    const int at1 = share * ((int)blockIdx.x + 1) + min((int)blockIdx.x + 1, extra);
    for (int at = share * (int)blockIdx.x + min((int)blockIdx.x, extra); at < at1;) {
        const int gtile = at / span, in = at - gtile * span;
        const int rg_begin = max(in - A.skip, 0), rg_end = min(in + (at1 - at), span) - A.skip;
        at += span - in;
        if (rg_end <= rg_begin) continue;
        int lo = 0, hi = nseg;  // the segment: pre[lo] <= gtile < pre[lo + 1]
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (S.pre[mid] <= gtile) lo = mid; else hi = mid;
        }
        const SegDesc sd = A.seg ? A.seg[lo] : A.single;
        const int tile = gtile - S.pre[lo];
        const int m = min(TT, (int)sd.m - tile * TT);
        const uint32_t row0 = sd.row0 + tile * TT;
        const int rg = rg_begin + slot;
        const MmItem I = {sd.wa, sd.wb, S.acts, S.red, A.out + (size_t)row0 * A.n_out, m, nb, kb0, kbn, rg, rg < rg_end ? (rg_end - rg + nslot - 1) / nslot : 0, nslot,
                          A.n_out, A.rb, A.ks, slot, kpart};
        F.rg = rg;
        F.b = 0;
        for (int i = 1; i < F.w.nst; ++i) F.prefetch(I);

        // ---- activations: a 256-element block of a token per warp ----
        bool wide = false;
        for (int gi = warp; gi < m * nb; gi += kMmWarps) {
            const int tok = gi / nb, b = gi - tok * nb;
            const uint32_t pr = row0 + tok;
            const float* xr = A.x + (size_t)(A.row_token ? A.row_token[pr] : (int32_t)pr) * A.ldx + b * 256;
            wide |= mm_stage_block<T>(mm_load_block<T>(xr, lane), S.acts + (size_t)gi * kXBlock, lane);
        }
        if (__builtin_expect(__syncthreads_or(wide), 0)) {
            mm_row_groups<T, FUSED, NT, true>(I, F);
        } else if (NT >= 4 && m > 2 * kMmTok) {
            mm_row_groups<T, FUSED, NT >= 4 ? 4 : 1, false>(I, F);
        } else if (NT >= 2 && m > kMmTok) {
            mm_row_groups<T, FUSED, NT >= 2 ? 2 : 1, false>(I, F);
        } else {
            mm_row_groups<T, FUSED, 1, false>(I, F);
        }
        __syncthreads();  // every warp has left the activations
    }
    tcp::cp_async_wait_all();
}
template <int T, bool FUSED, int NT>
__global__ void __launch_bounds__(kMmThreads, 1) mm_kernel(const MmArgs A) {
    constexpr int TT = NT * kMmTok;  // tokens of an item
    extern __shared__ __align__(128) uint8_t smem[];
    if (T == T_IQ3_XXS && tcp::s32(smem) != kMmSmemBase) {  // the tables' addresses would not be right: the context was told wrong
        if (threadIdx.x == 0) status_set(A.status, 26);
        return;
    }
    const MmShared S = mm_shared<T, NT>(smem, A);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if constexpr (T == T_IQ3_XXS) {
        mm_tables_in(smem, tid, kMmThreads);
        tcp::cp_async_wait_all();
    }
    pdl_wait();
    pdl_launch_dependents();

    // ---- first token tile of every segment ----
    const int nseg = A.nseg_dev ? min(*A.nseg_dev, A.nseg_max) : A.nseg_max;
    {
        const int per = (nseg + kMmThreads - 1) / kMmThreads;
        int sum = 0;
        for (int j = 0; j < per; ++j) {
            const int s = tid * per + j;
            if (s < nseg) sum += (int)(((A.seg ? A.seg[s].m : A.single.m) + TT - 1) / TT);
        }
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) S.wsum[warp] = incl;
        __syncthreads();
        int at = incl - sum;
        for (int w = 0; w < warp; ++w) at += S.wsum[w];
        for (int j = 0; j < per; ++j) {
            const int s = tid * per + j;
            if (s < nseg) {
                S.pre[s] = at;
                at += (int)(((A.seg ? A.seg[s].m : A.single.m) + TT - 1) / TT);
            }
        }
        if (tid == kMmThreads - 1) S.pre[nseg] = at;
        __syncthreads();
    }
    mm_items<T, FUSED, NT>(A, S, nseg);
}

template <int T, bool FUSED, int NT>
static int launch_mm_t(dnb_ctx* c, cudaStream_t st, MmArgs A, size_t smem, int grid, const char* name) {
    auto kern = mm_kernel<T, FUSED, NT>;
    static SmemGrant grant;
    DNB_CUDA(grant_smem(grant, c->device, kern, smem));
    ProfScope prof_(c, st, name);
    DNB_CUDA(launch_k(kern, dim3(grid), dim3(kMmThreads), smem, st, c->use_pdl, A));
    c->launches++;
    return DNB_OK;
}

bool mm_handles(const dnb_ctx* c, int type, int n_in) {
    return (type == T_Q4_K || type == T_Q5_K || type == T_Q6_K || type == T_Q8_0 || (type == T_IQ3_XXS && c->smem_base == (int)kMmSmemBase)) && n_in % 256 == 0 &&
           n_in > 0;
}

template <int T>
static int mm_launch_type(dnb_ctx* c, cudaStream_t st, bool fused, int nt, MmArgs& A, size_t smem, int grid, const char* name) {
#define DNB_MM(F, N) return launch_mm_t<T, F, N>(c, st, A, smem, grid, name)
    if (fused) { if (nt == 1) DNB_MM(true, 1); if (nt == 2) DNB_MM(true, 2); DNB_MM(true, 4); }
    if (nt == 1) DNB_MM(false, 1);
    if (nt == 2) DNB_MM(false, 2);
    DNB_MM(false, 4);
#undef DNB_MM
}

// The ring of each of `warps` warps that fits beside `base` bytes (`base_two`: with two blocks a stage): two blocks a stage where a warp has that many,
// three stages, then two; else one block, four stages to two.  Bytes of shared memory in all, or 0.
static size_t mm_ring(int type, int blocks, int warps, size_t base, size_t base_two, size_t cap, MmRing& r) {
    static const int form[5][2] = {{2, 3}, {2, 2}, {1, 4}, {1, 3}, {1, 2}};
    for (const auto& f : form) {
        if (f[0] > blocks) continue;
        r.bps = f[0];
        r.nst = f[1];
        switch (type) {
#define DNB_P(TT) case TT: r.pitch = f[0] == 2 ? Mq<TT>::P2 : Mq<TT>::P1; break;
            DNB_P(T_Q4_K) DNB_P(T_Q5_K) DNB_P(T_Q6_K) DNB_P(T_Q8_0) DNB_P(T_IQ3_XXS)
#undef DNB_P
            default: return 0;
        }
        const size_t smem = (f[0] == 2 ? base_two : base) + (size_t)warps * r.nst * 16 * r.pitch;
        if (smem <= cap) return smem;
    }
    return 0;
}

// batch: K is split as a constant of the shape.  rows: token rows of the launch in total; nseg_est: segments that will have rows (an estimate when the device counts them).
int launch_mm(dnb_ctx* c, cudaStream_t st, int type, bool fused, bool batch, const SegDesc* seg, const int32_t* nseg_dev, int nseg_max,
              int nseg_est, int rows, int n_in, int n_out, const float* x, int ldx, const int32_t* row_token, float* out,
              const SegDesc* single, const char* name) {
    if (!mm_handles(c, type, n_in) || n_out < 1 || (fused && n_out % 8) || nseg_max < 1 || nseg_max > kMmSegMax || rows < 1) return DNB_DECLINED;
    if (!seg && !single) return DNB_ERR_ARG;
    if ((((uintptr_t)x) & 15) || ldx % 4 || (single && ((((uintptr_t)single->wa) & 15) || (fused && (((uintptr_t)single->wb) & 15))))) return DNB_DECLINED;
    int rc = type == T_IQ3_XXS ? upload_mm_s8(c->device) : DNB_OK;
    if (rc) return rc;
    const int bb = type == T_Q4_K ? 144 : type == T_Q5_K ? 176 : type == T_Q6_K ? 210 : type == T_Q8_0 ? 272 : 98;
    MmArgs A = {};
    A.seg = seg; A.nseg_dev = nseg_dev; A.nseg_max = nseg_max;
    if (single) A.single = *single;
    A.n_in = n_in; A.n_out = n_out; A.rb = bb * (n_in / 256);
    A.x = x; A.ldx = ldx; A.row_token = row_token; A.out = out;
    // Column tiles: the fewest that hold an average segment (a wider instance costs registers and shared memory, a narrower
    // one decodes a segment's weights once more per tile).
    constexpr int tpt = kMmTok, max_nt = 4;
    const float avg = (float)rows / (float)std::max(1, nseg_est);
    int nt = 1;
    while (nt < max_nt && avg > 0.75f * nt * tpt) nt *= 2;
    const int n_rg = fused ? n_out / 8 : (n_out + 15) / 16, nb = n_in / 256;
    int split = batch && nb >= 4 ? 2 : 1;  // of a batch
    for (;; nt /= 2) {
        const long tiles = std::max(nseg_est, (rows + nt * tpt - 1) / (nt * tpt));
        // A CTA's row groups go round its slots of `ks` warps; the last round is partly empty, so K is split until there are
        // about six rounds (at most eight ways: each split costs an exchange of the sums).  A decode batch: two ways from four blocks on,
        // else not at all.  us a layer, gate/up of 2048 x 512, top 10 of 512, IQ3_XXS, 1 / 2 / 4 / 8 ways: 2 tokens 48.8 / 45.2 / 45.1 / 45.2,
        // 8 tokens 94.3 / 92.8 / 93.9 / 96.0, 32 tokens 206.8 / 204.1 / 213.1 / 222.7; down (two blocks) 1 / 2 ways: 8 tokens 93.1 / 93.8, 32 tokens
        // 206.6 / 209.8.  (Two sums in one warp, added like two warps' sums, would let K go unsplit with the same bits from 48 tokens on: 16 more
        // registers or as much shared memory, 10 to 20 % of a prompt's time.)
        const long per_cta = tiles * n_rg / c->sm_count;
        int ks = split;
        if (!batch)
            while (ks < 8 && ks * 2 <= nb && per_cta * ks < 6 * kMmWarps) ks *= 2;
        A.ks = ks;
        size_t base = kMmFixed + (ks > 1 ? (size_t)2 * kMmWarps * nt * 2 * 32 * 4 : 0) + (size_t)nt * tpt * nb * kXBlock;
        if (type == T_IQ3_XXS) base += sizeof(MmTables);
        const size_t smem = mm_ring(type, nb / ks, kMmWarps, base, base, 225 * 1024, A.ring);
        if (smem) {
            A.status = c->status;
            // Activations of a tile 2.5 - 3 us, a row group 1.1 us at K = 2048 and a quarter of that at K = 512 (IQ3_XXS).  us a layer of 2048 x 512, top
            // 10 of 512, with this many row groups / half / twice / four times as many: 8 tokens IQ3_XXS 80.1 / 82.0 / 79.7 / 83.0, Q4_K 67.9 / 69.5 / 68.0 /
            // 68.7, Q8_0 87.8 / 90.2 / 86.8 / 88.0; 32 tokens IQ3_XXS 182.5 / 183.0 / 182.7 / 185.9, Q4_K 135.8 / 136.5 / 136.6 / 136.3; Q4_K and Q6_K 77
            // tokens skewed 187.6 / 188.8 / 187.9 / 191.6, 200 even 482 / 485 / 484 / 486; 1024 x 768, 8 tokens Q4_K 58.0 / 59.1 / 57.7 / 58.5.
            A.skip = std::max(1, 5120 / n_in);
            if ((double)(nseg_max + (rows + nt * tpt - 1) / (nt * tpt)) * (n_rg + A.skip) > 2e9) return DNB_DECLINED;
            const int grid = nseg_dev ? c->sm_count : (int)std::min<long>(c->sm_count, std::max<long>(1, tiles * n_rg * ks / kMmWarps));
            switch (type) {
                case T_Q4_K: return mm_launch_type<T_Q4_K>(c, st, fused, nt, A, smem, grid, name);
                case T_Q5_K: return mm_launch_type<T_Q5_K>(c, st, fused, nt, A, smem, grid, name);
                case T_Q6_K: return mm_launch_type<T_Q6_K>(c, st, fused, nt, A, smem, grid, name);
                case T_Q8_0: return mm_launch_type<T_Q8_0>(c, st, fused, nt, A, smem, grid, name);
                default: return mm_launch_type<T_IQ3_XXS>(c, st, fused, nt, A, smem, grid, name);
            }
        }
        if (nt > 1) continue;
        if (split == 1) return DNB_DECLINED;
        split = 1;  // K so long that the exchange has no room beside it
        nt = 2;
    }
}

// ---- one matrix, a few vectors ---------------------------------------------------------------------------------------
// The same arithmetic for the GEMV of a single matrix (cuda.rs:21028 maybe_gpu_gguf_gemv_into).  What bounds it: a 4096 x 4096
// matrix is 64 KB per SM, so the time is how soon the bytes are asked for and how little follows once the vector is there; a large
// matrix is bytes or decoding.  Hence CTAs of eight warps, two per SM (the next GEMV's CTAs come in while this one's last are at
// work); a warp takes every ks-th block of K of 16 rows and asks for its first stages before it waits for the kernel in front of
// it, whose output the vector may be; it converts its own blocks of the vector, each with a power of two of its own, so that no
// CTA-wide step stands between vector and math; the warps' partial sums meet once per 16 rows, in a fixed order.
// Measured back to back, us, with fp16 operands -> with bytes: 4096 x 4096 Q4_K 5.6 -> 4.7; 65536 x 4096 Q8_0 71.8 -> 61 (4.7 TB/s), Q4_K 54 -> 37, IQ3_XXS
// 64 -> 55.  (The register-decode GEMV before took 8.4 for the small one, 103 for Q8_0.)
constexpr int kGvWarps = 8;

struct GvArgs {
    const uint8_t* w;
    const float* x;      // [tok][k]
    float* out;          // [tok][n]
    int k, n, rb, ks;
    MmRing ring;
    int nvec;            // a grid row takes TOK of them
    int* status;
};

template <int T, int TOK>
__global__ void __launch_bounds__(kGvWarps * 32, 2) gemv_mma_single_kernel(const GvArgs A) {
    using Q = Mq<T>;
    constexpr int XB = TOK * kXBlock;  // bytes of a converted block
    extern __shared__ __align__(128) uint8_t smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int nb = A.k >> 8, nslot = kGvWarps / A.ks, slot = warp / A.ks, kw = warp - slot * A.ks;
    // this warp's blocks: every ks-th stage of K, so that neighbours ask for neighbouring bytes at the same time
    const int bps = A.ring.bps, units = (nb + bps - 1) / bps, nst = (units - kw + A.ks - 1) / A.ks, kb_max = (units + A.ks - 1) / A.ks * bps;
    auto first = [&](int i) { return (kw + i * A.ks) * bps; };         // block of stage i
    auto count = [&](int i) { return min(bps, nb - first(i)); };
    uint8_t* p = smem + (T == T_IQ3_XXS ? sizeof(MmTables) : 0);
    float* red = reinterpret_cast<float*>(p);                                      // [2][8 warps][16 rows][TOK]
    p += 2 * kGvWarps * 16 * TOK * 4;
    uint8_t* xs = p + (size_t)warp * kb_max * XB;
    p += (size_t)kGvWarps * kb_max * XB;
    if (T == T_IQ3_XXS && tcp::s32(smem) != kMmSmemBase) {  // the tables' addresses would not be right: the context was told wrong
        if (tid == 0) status_set(A.status, 26);
        return;
    }
    MmStream<T> W(p + (size_t)warp * A.ring.nst * 16 * A.ring.pitch, A.ring, lane);
    const int n_rg = (A.n + 15) / 16, last = A.n - 1, rg_step = gridDim.x * nslot;
    const int rounds = (n_rg - (int)blockIdx.x * nslot + rg_step - 1) / rg_step;  // of the CTA; a slot's last one may be empty
    const int rg0 = blockIdx.x * nslot + slot;
    const int nrg = rg0 < n_rg ? (n_rg - rg0 + rg_step - 1) / rg_step : 0;

    // ---- weight stream (as in mm_kernel) ----
    int pf_rg = rg0, pf_i = 0;
    const int rg_stop = rg0 + nrg * rg_step;
    auto prefetch = [&]() {
        int n = 0;
        if (pf_rg < rg_stop) {
            if (pf_i == 0) W.template point<false>(A.w + (uint32_t)first(0) * Q::BB, nullptr, pf_rg * 16, last, (uint32_t)A.rb);
            n = count(pf_i);
        }
        W.request(n);
        if (n > 0) {
            W.skip((A.ks - 1) * bps * Q::BB);
            if (++pf_i == nst) {
                pf_i = 0;
                pf_rg += rg_step;
            }
        }
    };
    for (int i = 1; i < W.nst; ++i) prefetch();
    if constexpr (T == T_IQ3_XXS) mm_tables_in(smem, tid, kGvWarps * 32);
    pdl_wait();
    pdl_launch_dependents();

    // ---- this warp's blocks of the vectors ----
    const int v0 = blockIdx.y * TOK;
    bool wide = false;
    // A block's elements are asked for before the one in front of it is converted, those of two vectors together: what a conversion stores keeps
    // the compiler from doing so.  us, one after the other -> so: 2816 x 649, two vectors, Q4_K 4.9 -> 3.8, Q8_0 5.4 -> 4.2; 4096 x 4096 Q4_K 4.83 -> 4.78.
    // (In mm_kernel, where a warp rarely has two of them, it costs registers and 1 to 2 %.)
    {
        const int mine = (nst - 1) * bps + count(nst - 1);
        auto load = [&](int n, MmIn (&in)[TOK]) {
            const float* xr = A.x + (first(n >> (bps - 1)) + (n & (bps - 1))) * 256;
#pragma unroll
            for (int q = 0; q < TOK; ++q) in[q] = mm_load_block<T>(xr + (size_t)min(v0 + q, A.nvec - 1) * A.k, lane);
        };
        MmIn now[TOK], next[TOK];
        load(0, next);
#pragma unroll 1
        for (int n = 0; n < mine; ++n) {
#pragma unroll
            for (int q = 0; q < TOK; ++q) now[q] = next[q];
            if (n + 1 < mine) load(n + 1, next);
#pragma unroll
            for (int q = 0; q < TOK; ++q) wide |= mm_stage_block<T>(now[q], xs + n * XB + q * kXBlock, lane);
        }
    }
    if constexpr (T == T_IQ3_XXS) {  // the tables came in parts from all threads
        tcp::cp_async_wait_all();
        __syncthreads();
    }
    __syncwarp();

    // ---- the row groups ----
    const uint32_t gl = 4 * lane, sl = 8 * (lane & 15);
    const uint8_t *colb = xs + (TOK == 2 ? g >> 2 : 0) * kXBlock, *colv = xs + (TOK == 2 ? t >> 1 : 0) * kXBlock + kXInv + (t & 1) * 4;
    for (int rd = 0, rg = rg0; rd < rounds; ++rd, rg += rg_step) {
        float acc[1][2] = {{0.f, 0.f}};
        if (rd < nrg) {
            uint32_t offa = 0, offb = 0;
            if constexpr (!Q::ALIGNED) {
                offa = (uint32_t)(uintptr_t)A.w + (uint32_t)min(rg * 16 + g, last) * A.rb + (uint32_t)first(0) * Q::BB;
                offb = (uint32_t)(uintptr_t)A.w + (uint32_t)min(rg * 16 + 8 + g, last) * A.rb + (uint32_t)first(0) * Q::BB;
            }
            auto all_of_k = [&](auto rest) {
#pragma unroll 1
                for (int i = 0; i < nst; ++i) {
                    const uint8_t* st = W.wait();
                    prefetch();
                    const uint8_t *ra = st + g * W.pitch + (Q::ALIGNED ? 0u : offa & 15u), *rb = st + (g + 8) * W.pitch + (Q::ALIGNED ? 0u : offb & 15u);
                    offa += A.ks * bps * Q::BB;
                    offb += A.ks * bps * Q::BB;
                    const int n = count(i);
#pragma unroll 1
                    for (int j = 0; j < n; ++j, ra += Q::BB, rb += Q::BB) {
                        const int b = i * bps + j;
                        const uint8_t* bp = colb + b * XB + (g & 3) * kXDigit + t * 8;
                        const uint32_t sumw[1] = {mq_mins<T> && (g & 3) < 3 ? *reinterpret_cast<const uint32_t*>(colb + b * XB + kXSums + (g & 3) * 16 + t * 4) : 0u};
                        const float inv[1] = {*reinterpret_cast<const float*>(colv + b * XB)};
                        if constexpr (decltype(rest)::value) {
                            const uint8_t* const columns[1] = {bp};
                            mm_block_wide<T, 1>(ra, rb, lane, [&](int k) { return xs + b * XB + min(k, TOK - 1) * kXBlock; }, columns, sumw, inv, acc);
                        } else {
                            float none[2][2];
                            mm_block<T, 1, false>(ra, rb, t, gl, sl, [&](int, int u) { return *reinterpret_cast<const uint2*>(bp + u * 32); }, sumw, inv, acc, none);
                        }
                    }
                    W.next();
                }
            };
            if (__builtin_expect(wide, 0)) all_of_k(std::true_type());
            else all_of_k(std::false_type());
        }
        // lanes t = 0, 1 hold the first vector's low and high digits, t = 2, 3 the second's
        float a = acc[0][0], b = acc[0][1];
        a += __shfl_xor_sync(0xffffffffu, a, 1);
        b += __shfl_xor_sync(0xffffffffu, b, 1);
        float* rp = red + ((rd & 1) * kGvWarps + warp) * 16 * TOK;
        if ((t >> 1) < TOK) rp[(t >> 1) * 16 + ((t & 1) ? 8 + g : g)] = (t & 1) ? b : a;
        __syncthreads();  // (two buffers: a warp is at most one round ahead of the sums below)
        if (tid < nslot * 16 * TOK) {
            const int sl2 = tid / (16 * TOK), e = tid - sl2 * 16 * TOK, q = e >> 4;
            const int row = (blockIdx.x * nslot + rd * rg_step + sl2) * 16 + (e & 15);
            const float* r0 = red + ((rd & 1) * kGvWarps + sl2 * A.ks) * 16 * TOK + e;
            float v = r0[0];
            for (int w2 = 1; w2 < A.ks; ++w2) v += r0[w2 * 16 * TOK];
            if (row < A.n && v0 + q < A.nvec) A.out[(size_t)(v0 + q) * A.n + row] = v;
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

template <int T, int TOK>
static int launch_gv_t(dnb_ctx* c, cudaStream_t st, GvArgs A) {
    const int nb = A.k / 256;
    int ks = 1;
    while (ks < kGvWarps && ks * 2 <= nb) ks *= 2;
    // room for a warp's share of the vectors: whole stages of the form that is taken (2048 x 2048 IQ3_XXS with four vectors is two CTAs an SM, 4.4 us;
    // with room for two blocks where there is one it was one, and the call went to mm_kernel, 8.4 us)
    const size_t fixed = 2 * kGvWarps * 16 * TOK * 4 + (T == T_IQ3_XXS ? sizeof(MmTables) : 0), share = (size_t)kGvWarps * TOK * kXBlock;
    const size_t base = fixed + share * ((nb + ks - 1) / ks), base_two = fixed + share * ((nb + 2 * ks - 1) / (2 * ks) * 2);
    const size_t two = 113 * 1024;  // two CTAs per SM where they fit
    A.ks = ks;
    const int nslot = kGvWarps / ks, n_rg = (A.n + 15) / 16, ctas = (n_rg + nslot - 1) / nslot, rows = (A.nvec + TOK - 1) / TOK;
    // Two blocks a stage give the warps whole stages of K.  Where that makes the longest share longer (18 to 24 blocks: four instead of three)
    // and no SM has more than one CTA, whose longest share is then the time, it is one.  us, two / one: 1024 x 20 blocks Q4_K 5.5 / 4.5, 649 x 20, two
    // vectors, Q8_0 6.1 / 5.0, Q6_K 6.4 / 5.7, IQ3_XXS 6.8 / 6.1; with CTAs enough not always: 65536 x 20 blocks Q4_K 55 / 57, 24 blocks 59 / 66, 19 57 /
    // 55, other formats alike; and where the shares are as long: 1024 x 16 blocks 3.5 / 3.7, 65536 x 16 41 / 49.
    const int units = (nb + 1) / 2, longest_one = (nb + ks - 1) / ks, longest_two = (units + ks - 1) / ks * 2 - ((units - 1) % ks == 0 ? nb & 1 : 0);
    const int blocks = longest_two > longest_one && (long)ctas * rows <= c->sm_count ? 1 : nb / ks;
    size_t smem = mm_ring(T, blocks, kGvWarps, base, base_two, two, A.ring);
    if (!smem) smem = mm_ring(T, blocks, kGvWarps, base, base_two, 225 * 1024, A.ring);
    if (!smem) return DNB_DECLINED;
    A.status = c->status;
    auto kern = gemv_mma_single_kernel<T, TOK>;
    static SmemGrant grant;
    DNB_CUDA(grant_smem(grant, c->device, kern, smem));
    const int room = (smem <= two ? 2 : 1) * c->sm_count;
    // more vectors in grid rows of their own, each decoding the weights again: while they only fill SMs that would idle
    if (rows > 1 && (long)ctas * rows > room) return DNB_DECLINED;
    const int grid = std::min(ctas, room);
    ProfScope prof_(c, st, "gemv_mma");
    DNB_CUDA(launch_k(kern, dim3(grid, rows), dim3(kGvWarps * 32), smem, st, c->use_pdl, A));
    c->launches++;
    return DNB_OK;
}

int launch_gemv_mma(dnb_ctx* c, cudaStream_t st, int type, const uint8_t* w, int k, int n, const float* x, float* out, int nvec) {
    if (!mm_handles(c, type, k) || n < 1 || nvec < 1 || (((uintptr_t)w) & 15) || (((uintptr_t)x) & 15)) return DNB_DECLINED;
    const int rc = type == T_IQ3_XXS ? upload_mm_s8(c->device) : DNB_OK;
    if (rc) return rc;
    GvArgs A = {};
    A.w = w; A.x = x; A.out = out; A.k = k; A.n = n; A.nvec = nvec; A.rb = (int)row_bytes(type, k);
#define DNB_GV(TT) case TT: return nvec == 1 ? launch_gv_t<TT, 1>(c, st, A) : launch_gv_t<TT, 2>(c, st, A);
    switch (type) {
        DNB_GV(T_Q4_K)
        DNB_GV(T_Q5_K)
        DNB_GV(T_Q6_K)
        DNB_GV(T_Q8_0)
        default: return nvec == 1 ? launch_gv_t<T_IQ3_XXS, 1>(c, st, A) : launch_gv_t<T_IQ3_XXS, 2>(c, st, A);
    }
#undef DNB_GV
}

}  // namespace dnb
