// Grouped dequant matmul for few tokens per expert: decode batches, short prompts, caller-given selections, single
// matrices with a few vectors.  Q4_K, Q5_K, Q6_K, Q8_0 and IQ3_XXS on mma.sync.m16n8k16 (fp16, fp32 accumulators).
//
// Reference kernels of this role: kernels_seg_k.cu:201-241, kernels_exp_iq_v2.cu:259-319 (one warp per row, fp32 FMA);
// block layouts kquant.rs:341-887.
//
// What bounds a call like this is instructions, not bytes: at HBM speed an SM has about four lane-instructions per weight
// of a 4-bit format, and an FMA kernel spends two (convert, multiply) per weight AND token.  Here a weight costs its
// decoding only, whatever the number of tokens:
//   * a lane turns packed bytes into the fp16 A fragment in registers; the quantised value is an integer and exact
//     (Q4_K, Q5_K: sc * q <= 63 * 31 = 1953 < 2048, formed by one fp16 fma on the 1024 + q bit pattern; Q6_K: q - 32;
//     Q8_0: q; IQ3_XXS: the codebook magnitude <= 62 with its sign), so no weight is rounded;
//   * the scales multiply the fp32 sums of a 256-element block (Q4_K, Q5_K: d; their mins are one more K step of
//     m against the sub-block sums of the activations), of a 32-element block (Q8_0, IQ3_XXS) or of 16 elements (Q6_K);
//   * an activation is P fp16 numbers in P columns of B (P = 3 carries an fp32 to 2^-34 of the row's largest; P = 2 carries 22 bits and is
//     used where a call of this size had 16 before), of the row times a power of two that puts its largest element into
//     [512, 1024), so that nothing overflows and sub-block sums fit, too;
//   * K is walked in the order in which the packed bytes yield elements; the activations are staged in that order.
// A B column costs an mma per 16 weights of a lane's two rows and half a 16-byte shared-memory read.
//
// Work: an item is (segment, token tile, block of row groups); a row group is 16 A rows: 16 rows of one matrix, or 8 gate
// and 8 up rows of the same indices, whose results meet in one lane for silu(g) * u.  A persistent CTA of 16 warps stages
// an item's activations once; a warp then streams its row groups through a private ring of cp.async stages (one
// 256-element block of the 16 rows each) without any CTA-wide barrier.  Few row groups for the chip: KS warps share a row
// group, each takes a part of K, and their sums are added in a fixed order.  A row's result depends on the row, on P and on KS, not on
// the tile, the column or the CTA; for decode batches KS is a constant of the shape, so that a token's bits do not depend on its batch.
//
// Measured, us per layer of 2048 x 512, top 10 of 512, against one-row GEMVs (to 15 tokens) and tiled fp32 or bf16 tensor-core kernels:
// 8 tokens, IQ3_XXS 140 -> 95; 32 tokens 502 -> 204; 77 tokens under a skewed router, Q4_K with Q6_K down 895 -> 255.  Issue slots are
// 0.53 to 0.64 used, DRAM 0.12 to 0.20.
#include <algorithm>

#include "dnb_common.cuh"
#include "formats.cuh"
#include "tc_ptx.cuh"
#include "iq3_f16.cuh"

namespace dnb {

constexpr int kMmWarps = 16;
constexpr int kMmThreads = kMmWarps * 32;
constexpr int kMmSegMax = 1088;  // segments of a launch at most

// 256 elements of a row: bytes, 16-byte units of a stage row (blocks that are not 16-byte sized start anywhere in their first
// unit), and the unit stride of a stage row (chosen so that the eight rows a warp reads at once fall on different banks).
template <int T> struct Mq;
template <> struct Mq<T_Q4_K> { static constexpr int BB = 144, UNITS = 9, RS = 144; static constexpr bool ALIGNED = true; };
template <> struct Mq<T_Q5_K> { static constexpr int BB = 176, UNITS = 11, RS = 176; static constexpr bool ALIGNED = true; };
template <> struct Mq<T_Q6_K> { static constexpr int BB = 210, UNITS = 14, RS = 240; static constexpr bool ALIGNED = false; };
template <> struct Mq<T_IQ3_XXS> { static constexpr int BB = 98, UNITS = 7, RS = 112; static constexpr bool ALIGNED = false; };
template <> struct Mq<T_Q8_0> { static constexpr int BB = 272, UNITS = 17, RS = 272; static constexpr bool ALIGNED = true; };

template <int T> constexpr bool mq_mins = (T == T_Q4_K || T == T_Q5_K);

// First element (of 256) of the two groups of four that unit u = 0..7 of lane t takes; `swap`: a group's order is 0, 2, 1, 3.
template <int T>
__device__ __forceinline__ void mm_unit_elems(int u, int t, int& e0, int& e1) {
    if constexpr (mq_mins<T>) {
        e0 = 64 * t + 4 * u;
        e1 = e0 + 32;
    } else if constexpr (T == T_Q6_K) {
        e0 = (u >> 2) * 128 + (u & 1) * 32 + ((u >> 1) & 1) * 16 + 4 * t;
        e1 = e0 + 64;
    } else {
        e0 = 32 * u + 8 * t;
        e1 = e0 + 4;
    }
}

__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_f16_z(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ uint32_t ld32u(const uint8_t* p) { return ld16(p) | (ld16(p + 2) << 16); }  // 2-byte aligned

// One 256-element block of 16 rows (this lane: rows `ra` and `rb`) against NT column tiles; bp[i]: the lane's B column of tile
// i at this block; nt: tiles in use.  acc += scales * sums.
template <int T, int NT>
__device__ __forceinline__ void mm_block(const uint8_t* ra, const uint8_t* rb, int t, uint32_t gl, uint32_t sl, const uint8_t* const (&bp)[NT],
                                         const uint32_t (&sumw)[NT], int nt, float (&acc)[NT][4]) {
    if constexpr (mq_mins<T>) {
        const KScales sa = k_scales(ra, t), sb = k_scales(rb, t);
        constexpr bool FIVE = T == T_Q5_K;
        constexpr int QS = FIVE ? 48 : 16;
        float D[NT][4];
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) D[i][c] = 0.f;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const uint4 qa = *reinterpret_cast<const uint4*>(ra + QS + 32 * t + 16 * half);
            const uint4 qb = *reinterpret_cast<const uint4*>(rb + QS + 32 * t + 16 * half);
            uint4 ha = make_uint4(0, 0, 0, 0), hb = ha;
            if constexpr (FIVE) {
                ha = *reinterpret_cast<const uint4*>(ra + 16 + 16 * half);
                hb = *reinterpret_cast<const uint4*>(rb + 16 + 16 * half);
            }
            const uint32_t wa[4] = {qa.x, qa.y, qa.z, qa.w}, wb[4] = {qb.x, qb.y, qb.z, qb.w};
            const uint32_t fa[4] = {ha.x, ha.y, ha.z, ha.w}, fb[4] = {hb.x, hb.y, hb.z, hb.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint32_t p[4], q[4];
                k_word<FIVE>(wa[i], fa[i] >> (2 * t), sa, p);
                k_word<FIVE>(wb[i], fb[i] >> (2 * t), sb, q);
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    if (NT == 1 || n < nt) {
                        const uint4 y = *reinterpret_cast<const uint4*>(bp[n] + (half * 4 + i) * 64);
                        mma_f16(D[n], p[0], q[0], p[1], q[1], y.x, y.y);
                        mma_f16(D[n], p[2], q[2], p[3], q[3], y.z, y.w);
                    }
                }
            }
        }
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            if (NT == 1 || n < nt) {
                float M[4];
                mma_f16_z(M, sa.mm, sb.mm, 0u, 0u, sumw[n], 0u);
                acc[n][0] = fmaf(-sa.dmin, M[0], fmaf(sa.d, D[n][0], acc[n][0]));
                acc[n][1] = fmaf(-sa.dmin, M[1], fmaf(sa.d, D[n][1], acc[n][1]));
                acc[n][2] = fmaf(-sb.dmin, M[2], fmaf(sb.d, D[n][2], acc[n][2]));
                acc[n][3] = fmaf(-sb.dmin, M[3], fmaf(sb.d, D[n][3], acc[n][3]));
            }
        }
    } else if constexpr (T == T_IQ3_XXS) {
        // (d / 4) * (2 s + 1) (kquant.rs:667) = 8 d v - 7.75 d with v = 1 + s / 16 read off the bits: exact, d has 11 significant bits
        // (a conversion from integer would be a quarter-rate instruction)
        const float da = h2f(ld16(ra)), db = h2f(ld16(rb));
        const float ma8 = 8.f * da, na = -7.75f * da, mb8 = 8.f * db, nbs = -7.75f * db;
        // the eight sub-block words of a row as aligned words, shifted into place (a block starts on any even byte)
        const uint32_t ma = (tcp::s32(ra) + 2u) & 2u, mb = (tcp::s32(rb) + 2u) & 2u;
        const uint32_t* wa = reinterpret_cast<const uint32_t*>(ra + 66 - ma);
        const uint32_t* wb = reinterpret_cast<const uint32_t*>(rb + 66 - mb);
        const uint32_t sa = ma * 8u, sb = mb * 8u;
        const uint8_t* ia = ra + 2 + 2 * t;
        const uint8_t* ibp = rb + 2 + 2 * t;
        const int st = (7 * t + 26) & 31;
        uint32_t la = wa[0], lb = wb[0];
#pragma unroll
        for (int ib = 0; ib < 8; ++ib) {
            // the ninth word belongs to the row only where the words are shifted
            const uint32_t naw = wa[ib < 7 ? ib + 1 : 7 + (ma >> 1)], nbw = wb[ib < 7 ? ib + 1 : 7 + (mb >> 1)];
            const uint32_t xa = __funnelshift_r(la, naw, sa), xb = __funnelshift_r(lb, nbw, sb);
            la = naw;
            lb = nbw;
            uint32_t p[4], q[4];
            iq3_pairs_h(gl, sl, ld16(ia + 8 * ib), __funnelshift_r(xa, xa, st), p);
            iq3_pairs_h(gl, sl, ld16(ibp + 8 * ib), __funnelshift_r(xb, xb, st), q);
            const float fa = fmaf(__uint_as_float(((xa >> 9) & 0x00780000u) | 0x3f800000u), ma8, na);
            const float fb = fmaf(__uint_as_float(((xb >> 9) & 0x00780000u) | 0x3f800000u), mb8, nbs);
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                if (NT == 1 || n < nt) {
                    const uint4 y = *reinterpret_cast<const uint4*>(bp[n] + ib * 64);
                    float D[4];
                    mma_f16_z(D, p[0], q[0], p[1], q[1], y.x, y.y);
                    mma_f16(D, p[2], q[2], p[3], q[3], y.z, y.w);
                    acc[n][0] = fmaf(fa, D[0], acc[n][0]);
                    acc[n][1] = fmaf(fa, D[1], acc[n][1]);
                    acc[n][2] = fmaf(fb, D[2], acc[n][2]);
                    acc[n][3] = fmaf(fb, D[3], acc[n][3]);
                }
            }
        }
    } else if constexpr (T == T_Q8_0) {
        const uint32_t bias = 0x64806480u;  // 1024 + 128
#pragma unroll 4
        for (int ib = 0; ib < 8; ++ib) {
            const float fa = h2f(ld16(ra + 34 * ib)), fb = h2f(ld16(rb + 34 * ib));
            uint32_t p[4], q[4];
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                const uint32_t wa = ld32u(ra + 34 * ib + 2 + 8 * t + 4 * v) ^ 0x80808080u;
                const uint32_t wb = ld32u(rb + 34 * ib + 2 + 8 * t + 4 * v) ^ 0x80808080u;
                p[2 * v] = h2sub(__byte_perm(wa, 0x64646464u, 0x5140u), bias);
                p[2 * v + 1] = h2sub(__byte_perm(wa, 0x64646464u, 0x7362u), bias);
                q[2 * v] = h2sub(__byte_perm(wb, 0x64646464u, 0x5140u), bias);
                q[2 * v + 1] = h2sub(__byte_perm(wb, 0x64646464u, 0x7362u), bias);
            }
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                if (NT == 1 || n < nt) {
                    const uint4 y = *reinterpret_cast<const uint4*>(bp[n] + ib * 64);
                    float D[4];
                    mma_f16_z(D, p[0], q[0], p[1], q[1], y.x, y.y);
                    mma_f16(D, p[2], q[2], p[3], q[3], y.z, y.w);
                    acc[n][0] = fmaf(fa, D[0], acc[n][0]);
                    acc[n][1] = fmaf(fa, D[1], acc[n][1]);
                    acc[n][2] = fmaf(fb, D[2], acc[n][2]);
                    acc[n][3] = fmaf(fb, D[3], acc[n][3]);
                }
            }
        }
    } else {  // Q6_K: a K step is one 16-element group of one scale
        const float da = h2f(ld16(ra + 208)), db = h2f(ld16(rb + 208));
        const uint32_t bias = 0x64206420u;  // 1024 + 32
#pragma unroll 2
        for (int g = 0; g < 4; ++g) {  // (half, is)
            const int half = g >> 1, is = g & 1;
            const uint32_t ha = ld32u(ra + 128 + 32 * half + 16 * is + 4 * t), hb = ld32u(rb + 128 + 32 * half + 16 * is + 4 * t);
#pragma unroll
            for (int w = 0; w < 2; ++w) {
                const uint32_t qa = ld32u(ra + 64 * half + 32 * w + 16 * is + 4 * t), qb = ld32u(rb + 64 * half + 32 * w + 16 * is + 4 * t);
#pragma unroll
                for (int hi = 0; hi < 2; ++hi) {
                    const uint32_t va = ((qa >> (4 * hi)) & 0x0f0f0f0fu) | (((ha >> (2 * w + 4 * hi)) & 0x03030303u) << 4);
                    const uint32_t vb = ((qb >> (4 * hi)) & 0x0f0f0f0fu) | (((hb >> (2 * w + 4 * hi)) & 0x03030303u) << 4);
                    const uint32_t p0 = h2sub(__byte_perm(va, 0x64646464u, 0x5140u), bias), p1 = h2sub(__byte_perm(va, 0x64646464u, 0x7362u), bias);
                    const uint32_t q0 = h2sub(__byte_perm(vb, 0x64646464u, 0x5140u), bias), q1 = h2sub(__byte_perm(vb, 0x64646464u, 0x7362u), bias);
                    const int sc = 192 + 8 * half + is + 2 * w + 4 * hi;
                    const float fa = da * (float)(int)*reinterpret_cast<const int8_t*>(ra + sc), fb = db * (float)(int)*reinterpret_cast<const int8_t*>(rb + sc);
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        if (NT == 1 || n < nt) {
                            const uint2 y = *reinterpret_cast<const uint2*>(bp[n] + (2 * g + w) * 64 + 8 * hi);
                            float D[4];
                            mma_f16_z(D, p0, q0, p1, q1, y.x, y.y);
                            acc[n][0] = fmaf(fa, D[0], acc[n][0]);
                            acc[n][1] = fmaf(fa, D[1], acc[n][1]);
                            acc[n][2] = fmaf(fb, D[2], acc[n][2]);
                            acc[n][3] = fmaf(fb, D[3], acc[n][3]);
                        }
                    }
                }
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
    int ks, nst;               // warps that split K, stages of a warp's ring
    int col_stride;            // bytes between B columns
    int skip;                  // row groups' time that a tile's activations take
    uint32_t smem;             // bytes of dynamic shared memory
    int* status;
};

__device__ __forceinline__ void mm_barrier(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// Scale of a row: the power of two that puts its largest element into [512, 1024).
__device__ __forceinline__ float mm_row_scale(uint32_t amax_bits) {
    const int ex = (int)(amax_bits >> 23);  // biased exponent of the largest |x|
    const int s = ex == 0 ? 0 : max(-126, min(126, 9 - (ex - 127)));
    return __uint_as_float((uint32_t)(s + 127) << 23);
}
// Two values as P fp16 pairs whose sums are the values.  P = 2: 22 bits of the row's (one matrix: the block's) largest element; P = 3: every
// bit of the elements above 1/1024 of the largest, and 2^-34 of the largest below, where the third part meets fp16's smallest number.
template <int P>
__device__ __forceinline__ void mm_split(float a, float b, uint32_t (&h)[P]) {
#pragma unroll
    for (int p = 0; p < P; ++p) {
        const __half2 v = __floats2half2_rn(a, b);
        h[p] = *reinterpret_cast<const uint32_t*>(&v);
        if (p + 1 < P) {
            const float2 f = __half22float2(v);
            a -= f.x;
            b -= f.y;
        }
    }
}

template <int T, bool FUSED, int P, int NT>
__global__ void __launch_bounds__(kMmThreads, 1) mm_kernel(const MmArgs A) {
    using Q = Mq<T>;
    constexpr int TPT = P == 3 ? 2 : 4;  // tokens of a column tile (P = 3: columns 3 and 7 are copies nobody adds)
    constexpr int TT = NT * TPT;         // tokens of an item
    constexpr int STAGE = 16 * Q::RS;
    extern __shared__ __align__(128) uint8_t smem[];
    int* pre = reinterpret_cast<int*>(smem);                            // [kMmSegMax + 1] first token tile of a segment
    int* wsum = pre + kMmSegMax + 4;                                    // [16]
    uint32_t* amax = reinterpret_cast<uint32_t*>(wsum + 16);            // [2][16]
    uint8_t* p0 = smem + ((kMmSegMax + 4 + 16 + 32) * 4 + 127) / 128 * 128;
    float* red = reinterpret_cast<float*>(p0);                          // [2][16 warps][NT * 4][32] when ks > 1
    if (A.ks > 1) p0 += 2 * kMmWarps * NT * 4 * 32 * sizeof(float);
    uint8_t* acts = p0;
    p0 += (size_t)TT * P * A.col_stride;
    uint8_t* book = p0;
    if constexpr (T == T_IQ3_XXS) {
        book += (kMmBookAlign - (tcp::s32(p0) & (kMmBookAlign - 1))) & (kMmBookAlign - 1);
        p0 = book + sizeof(MmCodebook);
    }
    uint8_t* ring = p0;
    if (T == T_IQ3_XXS && (uint32_t)(ring - smem) + kMmWarps * A.nst * STAGE > A.smem) {  // only if shared memory started elsewhere
        if (threadIdx.x == 0) status_set(A.status, 26);
        return;
    }

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    ring += (size_t)warp * A.nst * STAGE;
    if constexpr (T == T_IQ3_XXS) {
        for (int i = tid; i < (int)(sizeof(MmCodebook) / 16); i += kMmThreads)
            tcp::cp_async16<false>(book + 16 * i, reinterpret_cast<const uint8_t*>(&g_mm_codebook) + 16 * i);
        tcp::cp_async_commit();
        tcp::cp_async_wait_all();
    }
    if (tid < 32) amax[tid] = 0u;
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
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        int at = incl - sum;
        for (int w = 0; w < warp; ++w) at += wsum[w];
        for (int j = 0; j < per; ++j) {
            const int s = tid * per + j;
            if (s < nseg) {
                pre[s] = at;
                at += (int)(((A.seg ? A.seg[s].m : A.single.m) + TT - 1) / TT);
            }
        }
        if (tid == kMmThreads - 1) pre[nseg] = at;
        __syncthreads();
    }
    const int nb = A.n_in >> 8;
    const int nslot = kMmWarps / A.ks, slot = warp / A.ks, kpart = warp - slot * A.ks;
    const int kb0 = nb * kpart / A.ks, kbn = nb * (kpart + 1) / A.ks - kb0;
    const int n_rg = FUSED ? A.n_out / 8 : (A.n_out + 15) / 16;
    const uint32_t gl = tcp::s32(book) + 8 * (lane & (kLutRep - 1)), sl = tcp::s32(book) + (uint32_t)sizeof(uint2) * 256 * kLutRep + 4 * (lane & (kLutRep - 1));
    int par = 0;
    // This CTA's share of all (tile, row group) pairs: a range of pairs in a row.  Another tile means another set of activations,
    // which takes as long as A.skip row groups: each tile is that much longer, and a CTA that has two gets so much less of them.
    const int span = n_rg + A.skip, total = pre[nseg] * span;
    const int share = total / (int)gridDim.x, extra = total - share * (int)gridDim.x;
    const int at1 = share * ((int)blockIdx.x + 1) + min((int)blockIdx.x + 1, extra);

    for (int at = share * (int)blockIdx.x + min((int)blockIdx.x, extra); at < at1; par ^= 1) {
        const int gtile = at / span, in = at - gtile * span;
        const int rg_begin = max(in - A.skip, 0), rg_end = min(in + (at1 - at), span) - A.skip;
        at += span - in;
        if (rg_end <= rg_begin) { par ^= 1; continue; }
        int lo = 0, hi = nseg;  // the segment: pre[lo] <= gtile < pre[lo + 1]
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (pre[mid] <= gtile) lo = mid; else hi = mid;
        }
        const SegDesc sd = A.seg ? A.seg[lo] : A.single;
        const int tile = gtile - pre[lo];
        const int m = min(TT, (int)sd.m - tile * TT);
        const uint32_t row0 = sd.row0 + tile * TT;
        int rg = rg_begin + slot;
        const int nrg = rg < rg_end ? (rg_end - rg + nslot - 1) / nslot : 0;
        const int nstage = nrg * kbn;

        // ---- the warp's weight stream: the next block of the next row group goes to ring slot pf_s ----
        // A lane copies unit `lane & 7` (+ 8, 16) of rows lane / 8 + 4 j; a format with one unit over has 16 lanes copy that one.
        int pf_rg = rg, pf_b = 0, pf_s = 0, pf_n = 0;
        const int r_in = lane >> 3, c16 = (lane & 7) * 16;
        constexpr bool TAIL = Q::ALIGNED && Q::UNITS % 8 == 1;
        const uint8_t *sa = nullptr, *sb = nullptr, *stl = nullptr;
        uint32_t o1 = 4u * A.rb, o2 = 0, o3 = 0;
        auto point = [&]() {  // row group pf_rg, first block
            const uint32_t boff = (uint32_t)kb0 * Q::BB;
            if constexpr (FUSED) {
                const size_t off = (size_t)(pf_rg * 8 + r_in) * A.rb + boff;
                sa = sd.wa + off;
                sb = sd.wb + off;
                if constexpr (TAIL) stl = (lane < 8 ? sd.wa : sd.wb) + (size_t)(pf_rg * 8 + (lane & 7)) * A.rb + boff + (Q::UNITS - 1) * 16;
            } else {
                const int row = pf_rg * 16 + r_in, last = A.n_out - 1;
                const int r0 = min(row, last);
                sa = sd.wa + (size_t)r0 * A.rb + boff;
                o1 = (uint32_t)(min(row + 4, last) - r0) * A.rb;
                o2 = (uint32_t)(min(row + 8, last) - r0) * A.rb;
                o3 = (uint32_t)(min(row + 12, last) - r0) * A.rb;
                if constexpr (TAIL) stl = sd.wa + (size_t)min(pf_rg * 16 + (lane & 15), last) * A.rb + boff + (Q::UNITS - 1) * 16;
            }
        };
        if (nstage > 0) point();
        auto prefetch = [&]() {
            if (pf_n < nstage) {
                uint8_t* dst = ring + pf_s * STAGE + r_in * Q::RS + c16;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint8_t* src = FUSED ? (j >= 2 ? sb : sa) + ((j & 1) ? o1 : 0u) : sa + (j == 0 ? 0u : j == 1 ? o1 : j == 2 ? o2 : o3);
                    if constexpr (!Q::ALIGNED) src = reinterpret_cast<const uint8_t*>((uintptr_t)src & ~(uintptr_t)15);
#pragma unroll
                    for (int cc = 0; cc < (TAIL ? Q::UNITS - 1 : Q::UNITS); cc += 8)
                        if (cc + 8 <= Q::UNITS || cc * 16 + c16 < Q::UNITS * 16) tcp::cp_async16(dst + j * 4 * Q::RS + cc * 16, src + cc * 16 + c16);
                }
                if constexpr (TAIL) {
                    if (lane < 16) tcp::cp_async16(ring + pf_s * STAGE + lane * Q::RS + (Q::UNITS - 1) * 16, stl);
                    stl += Q::BB;
                }
                ++pf_n;
                sa += Q::BB;
                if constexpr (FUSED) sb += Q::BB;
                if (++pf_b == kbn) {
                    pf_b = 0;
                    pf_rg += nslot;
                    if (pf_n < nstage) point();
                }
                if (++pf_s == A.nst) pf_s = 0;
            }
            tcp::cp_async_commit();
        };
        for (int i = 1; i < A.nst; ++i) prefetch();

        // ---- activations: largest element of each row, then the split into P columns ----
        for (int gi = warp; gi < m * nb; gi += kMmWarps) {  // one 256-element block of one token per warp
            const int tok = gi / nb, b = gi - tok * nb;
            const uint32_t pr = row0 + tok;
            const float* xr = A.x + (size_t)(A.row_token ? A.row_token[pr] : (int32_t)pr) * A.ldx + b * 256;
            const float4 v0 = *reinterpret_cast<const float4*>(xr + 4 * lane), v1 = *reinterpret_cast<const float4*>(xr + 128 + 4 * lane);
            uint32_t mx = max(max(__float_as_uint(fabsf(v0.x)), __float_as_uint(fabsf(v0.y))), max(__float_as_uint(fabsf(v0.z)), __float_as_uint(fabsf(v0.w))));
            mx = max(mx, max(max(__float_as_uint(fabsf(v1.x)), __float_as_uint(fabsf(v1.y))), max(__float_as_uint(fabsf(v1.z)), __float_as_uint(fabsf(v1.w)))));
            mx = __reduce_max_sync(0xffffffffu, mx);
            if (lane == 0) atomicMax(&amax[par * 16 + tok], mx);  // a maximum: any order gives the same
        }
        __syncthreads();
        for (int gi = warp; gi < m * nb; gi += kMmWarps) {
            const int tok = gi / nb, b = gi - tok * nb;
            const uint32_t pr = row0 + tok;
            const float* xr = A.x + (size_t)(A.row_token ? A.row_token[pr] : (int32_t)pr) * A.ldx + b * 256;
            const float s = mm_row_scale(amax[par * 16 + tok]);
            int e0, e1;
            mm_unit_elems<T>(g, t, e0, e1);  // lane = 4 * unit + quarter
            float4 v0 = *reinterpret_cast<const float4*>(xr + e0), v1 = *reinterpret_cast<const float4*>(xr + e1);
            v0.x *= s; v0.y *= s; v0.z *= s; v0.w *= s;
            v1.x *= s; v1.y *= s; v1.z *= s; v1.w *= s;
            uint32_t h[4][P];
            if constexpr (mq_mins<T>) {
                mm_split<P>(v0.x, v0.z, h[0]);
                mm_split<P>(v0.y, v0.w, h[1]);
                mm_split<P>(v1.x, v1.z, h[2]);
                mm_split<P>(v1.y, v1.w, h[3]);
            } else {
                mm_split<P>(v0.x, v0.y, h[0]);
                mm_split<P>(v0.z, v0.w, h[1]);
                mm_split<P>(v1.x, v1.y, h[2]);
                mm_split<P>(v1.z, v1.w, h[3]);
            }
            uint8_t* col = acts + (size_t)tok * P * A.col_stride;
#pragma unroll
            for (int p = 0; p < P; ++p)
                *reinterpret_cast<uint4*>(col + (size_t)p * A.col_stride + b * 512 + lane * 16) = make_uint4(h[0][p], h[1][p], h[2][p], h[3][p]);
            if constexpr (mq_mins<T>) {  // sums of the lane's two sub-blocks, over the eight units
                float a = (v0.x + v0.y) + (v0.z + v0.w), c = (v1.x + v1.y) + (v1.z + v1.w);
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) {
                    a += __shfl_xor_sync(0xffffffffu, a, o);
                    c += __shfl_xor_sync(0xffffffffu, c, o);
                }
                uint32_t sp[P];
                mm_split<P>(a, c, sp);
                if (g == 0) {
#pragma unroll
                    for (int p = 0; p < P; ++p) *reinterpret_cast<uint32_t*>(col + (size_t)p * A.col_stride + A.n_in * 2 + b * 16 + t * 4) = sp[p];
                }
            }
        }
        if (tid < 16) amax[(par ^ 1) * 16 + tid] = 0u;
        __syncthreads();

        // ---- the row groups ----
        const int nt = (m + TPT - 1) / TPT;
        const uint8_t* colb[NT];
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            const int tok = min(n * TPT + (P == 3 ? g >> 2 : g >> 1), m - 1), part = P == 3 ? min(g & 3, 2) : g & 1;
            colb[n] = acts + (size_t)(tok * P + part) * A.col_stride;
        }
        float acc[NT][4];
        int q_s = 0, q_b = 0, round = 0;
        uint32_t offa = 0, offb = 0;  // where a row's block starts (only the position inside 16 bytes matters)
        for (int q = 0; q < nstage; ++q) {
            if (A.nst == 2) asm volatile("cp.async.wait_group 0;" ::: "memory");
            else if (A.nst == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
            else asm volatile("cp.async.wait_group 2;" ::: "memory");
            __syncwarp();  // the stage is complete for every lane, and every lane has left the slot that is filled next
            prefetch();
            const uint8_t* st = ring + q_s * STAGE;
            const uint8_t* ra = st + g * Q::RS;
            const uint8_t* rb = st + (g + 8) * Q::RS;
            if constexpr (!Q::ALIGNED) {
                if (q_b == 0) {
                    const uint32_t r0 = FUSED ? rg * 8 + g : min(rg * 16 + g, A.n_out - 1), r1 = FUSED ? r0 : (uint32_t)min(rg * 16 + 8 + g, A.n_out - 1);
                    offa = r0 * (uint32_t)A.rb + (uint32_t)kb0 * Q::BB;
                    offb = r1 * (uint32_t)A.rb + (uint32_t)kb0 * Q::BB;
                }
                ra += offa & 15u;
                rb += offb & 15u;
                offa += Q::BB;
                offb += Q::BB;
            }
            if (q_b == 0) {
#pragma unroll
                for (int n = 0; n < NT; ++n)
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[n][c] = 0.f;
            }
            const uint8_t* bp[NT];
            uint32_t sumw[NT];
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                bp[n] = colb[n] + (kb0 + q_b) * 512 + t * 16;
                sumw[n] = 0u;
                if constexpr (mq_mins<T>) {
                    if (n < nt) sumw[n] = *reinterpret_cast<const uint32_t*>(colb[n] + A.n_in * 2 + (kb0 + q_b) * 16 + t * 4);
                }
            }
            mm_block<T, NT>(ra, rb, t, gl, sl, bp, sumw, nt, acc);
            if (++q_s == A.nst) q_s = 0;
            if (++q_b == kbn) {
                q_b = 0;
                bool mine = true;
                if (A.ks > 1) {  // the warps of the row group meet; the first adds the others' sums in order
                    float* rp = red + ((size_t)(round & 1) * kMmWarps + warp) * NT * 4 * 32 + lane;
                    mine = kpart == 0;
                    if (!mine) {
#pragma unroll
                        for (int n = 0; n < NT; ++n)
#pragma unroll
                            for (int c = 0; c < 4; ++c) rp[(n * 4 + c) * 32] = acc[n][c];
                    }
                    mm_barrier(1 + slot, A.ks * 32);
                    if (mine) {
                        for (int k2 = 1; k2 < A.ks; ++k2) {
                            rp += NT * 4 * 32;
#pragma unroll
                            for (int n = 0; n < NT; ++n)
#pragma unroll
                                for (int c = 0; c < 4; ++c) acc[n][c] += rp[(n * 4 + c) * 32];
                        }
                    }
                }
                if (mine) {
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
                        if (NT == 1 || n < nt) {
                            float a, b;  // this row of both halves of the tile, one token
                            int tok;
                            if constexpr (P == 3) {
                                a = (t & 1) ? acc[n][0] : acc[n][0] + acc[n][1];
                                b = (t & 1) ? acc[n][2] : acc[n][2] + acc[n][3];
                                a += __shfl_xor_sync(0xffffffffu, a, 1);
                                b += __shfl_xor_sync(0xffffffffu, b, 1);
                                tok = n * TPT + (t >> 1);
                            } else {
                                a = acc[n][0] + acc[n][1];
                                b = acc[n][2] + acc[n][3];
                                tok = n * TPT + t;
                            }
                            if (tok < m) {
                                const float s = mm_row_scale(amax[par * 16 + tok]);
                                const float inv = __uint_as_float((254u << 23) - __float_as_uint(s));  // 1 / 2^s: exponent 254 - e
                                a *= inv;
                                b *= inv;
                                float* o = A.out + (size_t)(row0 + tok) * A.n_out;
                                if constexpr (FUSED) {
                                    if (P == 2 || !(t & 1)) o[rg * 8 + g] = a / (1.0f + expf(-a)) * b;
                                } else {
                                    const int r = rg * 16 + g;
                                    if ((P == 2 || !(t & 1)) && r < A.n_out) o[r] = a;
                                    if ((P == 2 || (t & 1)) && r + 8 < A.n_out) o[r + 8] = b;
                                }
                            }
                        }
                    }
                }
                rg += nslot;
                ++round;
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // every warp has left the activations
    }
}

template <int T, bool FUSED, int P, int NT>
static int launch_mm_t(dnb_ctx* c, cudaStream_t st, MmArgs A, size_t smem, int grid, const char* name) {
    auto kern = mm_kernel<T, FUSED, P, NT>;
    static SmemGrant grant;
    DNB_CUDA(grant_smem(grant, c->device, kern, smem));
    ProfScope prof_(c, st, name);
    DNB_CUDA(launch_k(kern, dim3(grid), dim3(kMmThreads), smem, st, c->use_pdl, A));
    c->launches++;
    return DNB_OK;
}

bool mm_handles(int type, int n_in) {
    return (type == T_Q4_K || type == T_Q5_K || type == T_Q6_K || type == T_Q8_0 || type == T_IQ3_XXS) && n_in % 256 == 0 && n_in > 0;
}

template <int T>
static int mm_launch_type(dnb_ctx* c, cudaStream_t st, bool fused, int parts, int nt, MmArgs& A, size_t smem, int grid, const char* name) {
#define DNB_MM(F, P, N) return launch_mm_t<T, F, P, N>(c, st, A, smem, grid, name)
    if (parts == 2) {
        if constexpr (T == T_Q4_K || T == T_IQ3_XXS) {
            if (fused) { if (nt == 1) DNB_MM(true, 2, 1); DNB_MM(true, 2, 2); }
            if (nt == 1) DNB_MM(false, 2, 1);
            DNB_MM(false, 2, 2);
        }
        return DNB_DECLINED;
    }
    if (fused) { if (nt == 1) DNB_MM(true, 3, 1); if (nt == 2) DNB_MM(true, 3, 2); DNB_MM(true, 3, 4); }
    if (nt == 1) DNB_MM(false, 3, 1);
    if (nt == 2) DNB_MM(false, 3, 2);
    DNB_MM(false, 3, 4);
#undef DNB_MM
}

// batch: K is split as a constant of the shape.  rows: token rows of the launch in total; nseg_est: segments that will have rows (an estimate when the device counts them).
int launch_mm(dnb_ctx* c, cudaStream_t st, int type, bool fused, int parts, bool batch, const SegDesc* seg, const int32_t* nseg_dev, int nseg_max,
              int nseg_est, int rows, int n_in, int n_out, const float* x, int ldx, const int32_t* row_token, float* out,
              const SegDesc* single, const char* name) {
    if (!mm_handles(type, n_in) || n_out < 1 || (fused && n_out % 8) || nseg_max < 1 || nseg_max > kMmSegMax || rows < 1) return DNB_DECLINED;
    if (!seg && !single) return DNB_ERR_ARG;
    if ((((uintptr_t)x) & 15) || ldx % 4 || (single && ((((uintptr_t)single->wa) & 15) || (fused && (((uintptr_t)single->wb) & 15))))) return DNB_DECLINED;
    if (type != T_Q4_K && type != T_IQ3_XXS) parts = 3;
    int rc = type == T_IQ3_XXS ? upload_mm_tables(c->device) : DNB_OK;
    if (rc) return rc;
    const int bb = type == T_Q4_K ? 144 : type == T_Q5_K ? 176 : type == T_Q6_K ? 210 : type == T_Q8_0 ? 272 : 98;
    const int rs = type == T_Q4_K ? Mq<T_Q4_K>::RS : type == T_Q5_K ? Mq<T_Q5_K>::RS : type == T_Q6_K ? Mq<T_Q6_K>::RS
                 : type == T_Q8_0 ? Mq<T_Q8_0>::RS : Mq<T_IQ3_XXS>::RS;
    MmArgs A = {};
    A.seg = seg; A.nseg_dev = nseg_dev; A.nseg_max = nseg_max;
    if (single) A.single = *single;
    A.n_in = n_in; A.n_out = n_out; A.rb = bb * (n_in / 256);
    A.x = x; A.ldx = ldx; A.row_token = row_token; A.out = out;
    // columns 64 bytes apart modulo 128: the two columns a quarter-warp reads together fall on different banks
    A.col_stride = n_in * 2 + (n_in / 16 + 127) / 128 * 128 + 64;
    // Column tiles: the fewest that hold an average segment (a wider instance costs registers and shared memory, a narrower
    // one decodes a segment's weights once more per tile).
    const int tpt = parts == 3 ? 2 : 4, max_nt = parts == 3 ? 4 : 2;
    const float avg = (float)rows / (float)std::max(1, nseg_est);
    int nt = 1;
    while (nt < max_nt && avg > 0.75f * nt * tpt) nt *= 2;
    const int n_rg = fused ? n_out / 8 : (n_out + 15) / 16, nb = n_in / 256;
    const size_t fixed = ((kMmSegMax + 4 + 16 + 32) * 4 + 127) / 128 * 128;
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
        size_t base = fixed + (ks > 1 ? (size_t)2 * kMmWarps * nt * 4 * 32 * 4 : 0) + (size_t)nt * tpt * parts * A.col_stride;
        if (type == T_IQ3_XXS)  // the tables behind the activations, on their boundary (dynamic shared memory starts at kMmSmemBase)
            base = (base + kMmSmemBase + kMmBookAlign - 1) / kMmBookAlign * kMmBookAlign - kMmSmemBase + sizeof(MmCodebook);
        const size_t stage = (size_t)kMmWarps * 16 * rs, cap = 225 * 1024;
        for (A.nst = 4; A.nst >= 2 && base + A.nst * stage > cap; --A.nst) {}
        if (A.nst >= 2) {
            const size_t smem = base + A.nst * stage;
            A.smem = (uint32_t)smem;
            A.status = c->status;
            // activations of a tile 2.5 - 3 us, a row group 1.1 us at K = 2048 and a quarter of that at K = 512 (measured, IQ3_XXS)
            A.skip = std::max(1, 5120 / n_in);
            if ((double)(nseg_max + (rows + nt * tpt - 1) / (nt * tpt)) * (n_rg + A.skip) > 2e9) return DNB_DECLINED;
            const int grid = nseg_dev ? c->sm_count : (int)std::min<long>(c->sm_count, std::max<long>(1, tiles * n_rg * ks / kMmWarps));
            switch (type) {
                case T_Q4_K: return mm_launch_type<T_Q4_K>(c, st, fused, parts, nt, A, smem, grid, name);
                case T_Q5_K: return mm_launch_type<T_Q5_K>(c, st, fused, parts, nt, A, smem, grid, name);
                case T_Q6_K: return mm_launch_type<T_Q6_K>(c, st, fused, parts, nt, A, smem, grid, name);
                case T_Q8_0: return mm_launch_type<T_Q8_0>(c, st, fused, parts, nt, A, smem, grid, name);
                default: return mm_launch_type<T_IQ3_XXS>(c, st, fused, parts, nt, A, smem, grid, name);
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
// Measured back to back, us, register-decode GEMV before: 4096 x 4096 Q4_K 8.4 -> 5.7, IQ3_XXS 10.3 -> 6.4, Q8_0 8.9 -> 6.5; 65536 x
// 4096 Q8_0 103 -> 71 (4.0 TB/s), Q4_K 84 -> 47, IQ3_XXS 99 -> 56; two vectors of IQ3_XXS 62034 x 5632 466 -> 94.
constexpr int kGvWarps = 8;
constexpr int kGvPart = 576;  // bytes of a part of a block: 512, its sub-block sums (16), and padding that spreads neighbouring parts over the banks

struct GvArgs {
    const uint8_t* w;
    const float* x;      // [tok][k]
    float* out;          // [tok][n]
    int k, n, rb, ks, nst;
    int nvec;            // a grid row takes TOK of them
    uint32_t smem;
    int* status;
};

template <int T, int TOK>
__global__ void __launch_bounds__(kGvWarps * 32, 2) gemv_mma_single_kernel(const GvArgs A) {
    using Q = Mq<T>;
    constexpr int STAGE = 16 * Q::RS, XB = TOK * 3 * kGvPart;  // bytes of a converted block
    extern __shared__ __align__(128) uint8_t smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int nb = A.k >> 8, nslot = kGvWarps / A.ks, slot = warp / A.ks, kw = warp - slot * A.ks;
    const int kbn = (nb - kw + A.ks - 1) / A.ks, kb_max = (nb + A.ks - 1) / A.ks;  // this warp's blocks: kw, kw + ks, ...
    float* red = reinterpret_cast<float*>(smem);                                   // [2][8 warps][16 rows][TOK]
    float* inv = red + 2 * kGvWarps * 16 * TOK + warp * kb_max * TOK;              // [blocks][TOK] what undoes a block's scaling
    uint8_t* p = smem + ((2 * kGvWarps * 16 * TOK + kGvWarps * kb_max * TOK) * 4 + 127) / 128 * 128;
    uint8_t* xs = p + (size_t)warp * kb_max * XB;
    p += (size_t)kGvWarps * kb_max * XB;
    uint8_t* book = p;
    if constexpr (T == T_IQ3_XXS) {
        book += (kMmBookAlign - (tcp::s32(p) & (kMmBookAlign - 1))) & (kMmBookAlign - 1);
        p = book + sizeof(MmCodebook);
    }
    if (T == T_IQ3_XXS && (uint32_t)(p - smem) + kGvWarps * A.nst * STAGE > A.smem) {  // only if shared memory started elsewhere
        if (tid == 0) status_set(A.status, 26);
        return;
    }
    uint8_t* ring = p + (size_t)warp * A.nst * STAGE;
    const int n_rg = (A.n + 15) / 16, last = A.n - 1, rg_step = gridDim.x * nslot;
    const int rounds = (n_rg - (int)blockIdx.x * nslot + rg_step - 1) / rg_step;  // of the CTA; a slot's last one may be empty
    const int rg0 = blockIdx.x * nslot + slot;
    const int nrg = rg0 < n_rg ? (n_rg - rg0 + rg_step - 1) / rg_step : 0, nstage = nrg * kbn;

    // ---- weight stream (as in mm_kernel) ----
    int pf_rg = rg0, pf_b = 0, pf_s = 0, pf_n = 0;
    const int r_in = lane >> 3, c16 = (lane & 7) * 16;
    constexpr bool TAIL = Q::ALIGNED && Q::UNITS % 8 == 1;
    const uint8_t *sa = nullptr, *stl = nullptr;
    uint32_t o1 = 0, o2 = 0, o3 = 0;
    auto point = [&]() {
        const int row = pf_rg * 16 + r_in, r0 = min(row, last);
        sa = A.w + (size_t)r0 * A.rb + (uint32_t)kw * Q::BB;
        o1 = (uint32_t)(min(row + 4, last) - r0) * A.rb;
        o2 = (uint32_t)(min(row + 8, last) - r0) * A.rb;
        o3 = (uint32_t)(min(row + 12, last) - r0) * A.rb;
        if constexpr (TAIL) stl = A.w + (size_t)min(pf_rg * 16 + (lane & 15), last) * A.rb + (uint32_t)kw * Q::BB + (Q::UNITS - 1) * 16;
    };
    if (nstage > 0) point();
    auto prefetch = [&]() {
        if (pf_n < nstage) {
            uint8_t* dst = ring + pf_s * STAGE + r_in * Q::RS + c16;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint8_t* src = sa + (j == 0 ? 0u : j == 1 ? o1 : j == 2 ? o2 : o3);
                if constexpr (!Q::ALIGNED) src = reinterpret_cast<const uint8_t*>((uintptr_t)src & ~(uintptr_t)15);
#pragma unroll
                for (int cc = 0; cc < (TAIL ? Q::UNITS - 1 : Q::UNITS); cc += 8)
                    if (cc + 8 <= Q::UNITS || cc * 16 + c16 < Q::UNITS * 16) tcp::cp_async16(dst + j * 4 * Q::RS + cc * 16, src + cc * 16 + c16);
            }
            if constexpr (TAIL) {
                if (lane < 16) tcp::cp_async16(ring + pf_s * STAGE + lane * Q::RS + (Q::UNITS - 1) * 16, stl);
                stl += A.ks * Q::BB;
            }
            ++pf_n;
            sa += A.ks * Q::BB;
            if (++pf_b == kbn) {
                pf_b = 0;
                pf_rg += rg_step;
                if (pf_n < nstage) point();
            }
            if (++pf_s == A.nst) pf_s = 0;
        }
        tcp::cp_async_commit();
    };
    for (int i = 1; i < A.nst; ++i) prefetch();
    if constexpr (T == T_IQ3_XXS) {  // in the last of those groups' shadow: waited for with the first stage
        for (int i = tid; i < (int)(sizeof(MmCodebook) / 16); i += kGvWarps * 32)
            tcp::cp_async16<false>(book + 16 * i, reinterpret_cast<const uint8_t*>(&g_mm_codebook) + 16 * i);
        tcp::cp_async_commit();
    }
    pdl_wait();
    pdl_launch_dependents();

    // ---- this warp's blocks of the vectors ----
    const int v0 = blockIdx.y * TOK;
    for (int i = 0; i < kbn; ++i) {
#pragma unroll
        for (int q = 0; q < TOK; ++q) {
            const float* xr = A.x + (size_t)min(v0 + q, A.nvec - 1) * A.k + (kw + i * A.ks) * 256;
            int e0, e1;
            mm_unit_elems<T>(g, t, e0, e1);  // lane = 4 * unit + quarter
            float4 xa = *reinterpret_cast<const float4*>(xr + e0), xb = *reinterpret_cast<const float4*>(xr + e1);
            uint32_t mx = max(max(__float_as_uint(fabsf(xa.x)), __float_as_uint(fabsf(xa.y))), max(__float_as_uint(fabsf(xa.z)), __float_as_uint(fabsf(xa.w))));
            mx = max(mx, max(max(__float_as_uint(fabsf(xb.x)), __float_as_uint(fabsf(xb.y))), max(__float_as_uint(fabsf(xb.z)), __float_as_uint(fabsf(xb.w)))));
            const float s = mm_row_scale(__reduce_max_sync(0xffffffffu, mx));
            if (lane == 0) inv[i * TOK + q] = __uint_as_float((254u << 23) - __float_as_uint(s));
            xa.x *= s; xa.y *= s; xa.z *= s; xa.w *= s;
            xb.x *= s; xb.y *= s; xb.z *= s; xb.w *= s;
            uint32_t h[4][3];
            if constexpr (mq_mins<T>) {
                mm_split<3>(xa.x, xa.z, h[0]);
                mm_split<3>(xa.y, xa.w, h[1]);
                mm_split<3>(xb.x, xb.z, h[2]);
                mm_split<3>(xb.y, xb.w, h[3]);
            } else {
                mm_split<3>(xa.x, xa.y, h[0]);
                mm_split<3>(xa.z, xa.w, h[1]);
                mm_split<3>(xb.x, xb.y, h[2]);
                mm_split<3>(xb.z, xb.w, h[3]);
            }
            uint8_t* col = xs + i * XB + q * 3 * kGvPart;
#pragma unroll
            for (int c = 0; c < 3; ++c) *reinterpret_cast<uint4*>(col + c * kGvPart + lane * 16) = make_uint4(h[0][c], h[1][c], h[2][c], h[3][c]);
            if constexpr (mq_mins<T>) {
                float a = (xa.x + xa.y) + (xa.z + xa.w), b = (xb.x + xb.y) + (xb.z + xb.w);
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) {
                    a += __shfl_xor_sync(0xffffffffu, a, o);
                    b += __shfl_xor_sync(0xffffffffu, b, o);
                }
                uint32_t sp[3];
                mm_split<3>(a, b, sp);
                if (g == 0) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) *reinterpret_cast<uint32_t*>(col + c * kGvPart + 512 + t * 4) = sp[c];
                }
            }
        }
    }
    if constexpr (T == T_IQ3_XXS) {  // the tables came in parts from all threads
        tcp::cp_async_wait_all();
        __syncthreads();
    }
    __syncwarp();

    // ---- the row groups ----
    const uint32_t gl = tcp::s32(book) + 8 * (lane & (kLutRep - 1)), sl = tcp::s32(book) + (uint32_t)sizeof(uint2) * 256 * kLutRep + 4 * (lane & (kLutRep - 1));
    const uint8_t* colb = xs + ((TOK == 2 ? (g >> 2) : 0) * 3 + min(g & 3, 2)) * kGvPart;
    int q_s = 0, rg = rg0;
    for (int rd = 0; rd < rounds; ++rd, rg += rg_step) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        if (rd < nrg) {
            uint32_t offa = 0, offb = 0;
            if constexpr (!Q::ALIGNED) {
                offa = (uint32_t)(uintptr_t)A.w + (uint32_t)min(rg * 16 + g, last) * A.rb + (uint32_t)kw * Q::BB;
                offb = (uint32_t)(uintptr_t)A.w + (uint32_t)min(rg * 16 + 8 + g, last) * A.rb + (uint32_t)kw * Q::BB;
            }
            for (int i = 0; i < kbn; ++i) {
                if (A.nst == 2) asm volatile("cp.async.wait_group 0;" ::: "memory");
                else if (A.nst == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
                else asm volatile("cp.async.wait_group 2;" ::: "memory");
                __syncwarp();
                prefetch();
                const uint8_t* st = ring + q_s * STAGE;
                const uint8_t *ra = st + g * Q::RS, *rb = st + (g + 8) * Q::RS;
                if constexpr (!Q::ALIGNED) {
                    ra += offa & 15u;
                    rb += offb & 15u;
                    offa += A.ks * Q::BB;
                    offb += A.ks * Q::BB;
                }
                const uint8_t* const bp[1] = {colb + i * XB + t * 16};
                const uint32_t sumw[1] = {mq_mins<T> ? *reinterpret_cast<const uint32_t*>(colb + i * XB + 512 + t * 4) : 0u};
                float c[1][4] = {{0.f, 0.f, 0.f, 0.f}};
                mm_block<T, 1>(ra, rb, t, gl, sl, bp, sumw, 1, c);
                const float f = inv[i * TOK + (TOK == 2 ? t >> 1 : 0)];
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[j] = fmaf(f, c[0][j], acc[j]);
                if (++q_s == A.nst) q_s = 0;
            }
        }
        // columns 0-2 (lanes t = 0, 1) are the first vector's parts, 4-6 (t = 2, 3) the second's
        float a = (t & 1) ? acc[0] : acc[0] + acc[1], b = (t & 1) ? acc[2] : acc[2] + acc[3];
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
    const int nb = A.k / 256, rs = Mq<T>::RS;
    int ks = 1;
    while (ks < kGvWarps && ks * 2 <= nb) ks *= 2;
    const int kb_max = (nb + ks - 1) / ks;
    size_t base = ((2 * kGvWarps * 16 * TOK + kGvWarps * kb_max * TOK) * 4 + 127) / 128 * 128 + (size_t)kGvWarps * kb_max * TOK * 3 * kGvPart;
    if (T == T_IQ3_XXS) base = (base + kMmSmemBase + kMmBookAlign - 1) / kMmBookAlign * kMmBookAlign - kMmSmemBase + sizeof(MmCodebook);
    const size_t stage = (size_t)kGvWarps * 16 * rs, two = 113 * 1024, cap = 225 * 1024;  // two CTAs per SM where they fit
    A.ks = ks;
    for (A.nst = 4; A.nst > 2 && base + A.nst * stage > two; --A.nst) {}
    const size_t smem = base + A.nst * stage;
    if (smem > cap) return DNB_DECLINED;
    A.smem = (uint32_t)smem;
    A.status = c->status;
    auto kern = gemv_mma_single_kernel<T, TOK>;
    static SmemGrant grant;
    DNB_CUDA(grant_smem(grant, c->device, kern, smem));
    const int nslot = kGvWarps / ks, n_rg = (A.n + 15) / 16;
    const int room = (smem <= two ? 2 : 1) * c->sm_count, ctas = (n_rg + nslot - 1) / nslot, rows = (A.nvec + TOK - 1) / TOK;
    // more vectors in grid rows of their own, each decoding the weights again: while they only fill SMs that would idle
    if (rows > 1 && (long)ctas * rows > room) return DNB_DECLINED;
    const int grid = std::min(ctas, room);
    ProfScope prof_(c, st, "gemv_mma");
    DNB_CUDA(launch_k(kern, dim3(grid, rows), dim3(kGvWarps * 32), smem, st, c->use_pdl, A));
    c->launches++;
    return DNB_OK;
}

int launch_gemv_mma(dnb_ctx* c, cudaStream_t st, int type, const uint8_t* w, int k, int n, const float* x, float* out, int nvec) {
    if (!mm_handles(type, k) || n < 1 || nvec < 1 || (((uintptr_t)w) & 15) || (((uintptr_t)x) & 15)) return DNB_DECLINED;
    const int rc = type == T_IQ3_XXS ? upload_mm_tables(c->device) : DNB_OK;
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
