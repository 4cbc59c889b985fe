// Grouped per-expert GEMM of chunked prefill on tcgen05: Q4_K and IQ3_XXS experts as EXACT fp16 integers, block scales after
// the tensor-core sum.
//
// Reference kernels of this role: kernels_exp_k_pf.cu:188-258 (m-row fp32), kernels_gemm_grouped.cu:134-273 (fp32 FMA),
// kernels_exp_iq_tc.cu (bf16 wmma); block layouts kquant.rs:505-526, :659-680.
//
//     W . x  =  sum over 256-element blocks b of  s_b * [ sum_i w_i * x_i ]   ( - sum over sub-blocks of (dmin * m) * X )
//   Q4_K    : w = sc * q <= 945, s_b = d, and the mins: X = the sum of the sub-block's 32 activations
//   IQ3_XXS : w = codebook magnitude * sign * (2 s + 1) <= 1922, s_b = d / 4
// Every w is an integer below 2048 and exact in fp16, so a weight costs its decoding and nothing is rounded.  The mins are one
// more block of K = sub-blocks: A = -(dmin * m) * 2^10 as fp16 hi and lo, B = X.  An activation is fp16 hi + lo (22 bits) of the
// row times a power of two that puts its largest element into [512, 1024).
//
// What bounds it: per 64-element stage of two 128-row tiles the 16 producer warps issue about 900 instructions (Q4_K; 1.7 per
// weight) on four schedulers while the tensor core needs 8 MMAs of N = 2 x tokens; decoding and tensor work are of the same
// size at 32 tokens per tile, so both have to run all the time.  Hence:
//   * four producer groups of four warps, each on a stage of its own (a thread owns one row of both tiles: a 16-byte piece of
//     its 128-byte swizzled row goes to a different bank group in each of eight neighbouring lanes), a ring of four or five
//     stages: a group has the time of three other stages to wait for its bytes, decode and hand over.  (Two groups on a ring
//     of two or three stages of the same size left the MMA warp without work for half the time.)
//   * a thread's packed bytes for its next stage are requested before it waits for the ring;
//   * hi and lo rows of a token are neighbours in memory, in the B tile (N = 2 x tokens) and in TMEM: a weight tile is read
//     once per K step, and the epilogue adds the pair;
//   * gate/up reads its tokens through TMA row gathers from the token-major rows: no packed copy of the activations.
// Warps: 0-7 epilogue (thread = weight row, half of the token columns of both tiles; four TMEM buffers), 8-23 producers,
// 24 TMA, 25 MMA.  Persistent, one CTA per SM; items (segment, 32-token tile, 128 rows x 2) dealt round-robin.
#include <cuda.h>
#include <cuda_fp16.h>

#include "dnb_common.cuh"
#include "tc_ptx.cuh"
#include "iq3_f16.cuh"
#include "operand_rows.cuh"

namespace dnb {
namespace tg {
using namespace tcp;

constexpr int BK = 64;                  // K of a stage: one 128-byte swizzle row of fp16
constexpr int TILE_M = 128;
constexpr int NT = 32;                  // tokens of an item
constexpr int A_TILE = TILE_M * BK * 2; // 16 KB
constexpr int A_STAGE = 2 * A_TILE;
constexpr int B_STAGE = 2 * NT * BK * 2;// hi and lo rows: 8 KB
constexpr int NB = 4;                   // TMEM buffers
constexpr int BUF_COLS = 2 * 2 * NT;    // two tiles x (hi, lo) x tokens
constexpr int EWARPS = 8, GROUPS = 4, PWARPS = 4 * GROUPS;
constexpr int W_TMA = EWARPS + PWARPS, W_MMA = W_TMA + 1;
constexpr int NTHREADS = (W_MMA + 1) * 32;
constexpr int kMaxSeg = 1055;
constexpr int kLocalItems = 40;
constexpr float kMinScale = 1024.f;     // the mins' A values are scaled up so that the low halves stay normal fp16 numbers

template <int T> constexpr int kBB = T == T_Q4_K ? 144 : 98;

struct Maps { CUtensorMap box[3]; CUtensorMap row; };  // boxes of 16, 32, 64 operand rows; single rows for the gathers

struct Item {
    const uint8_t* pa;  // tile 0, first row
    const uint8_t* pb;  // tile 1
    int prow, m;        // first packed row, tokens (1..NT)
    int r0, pad;        // first output row
};

template <bool PAIR>
__device__ __forceinline__ Item decode_item(int item, int row_tiles, int rb, int nseg, const int* pre, const SegDesc* __restrict__ seg) {
    const int tile = item / row_tiles, rt = item - tile * row_tiles;
    int lo = 0, hi = nseg;  // pre[lo] <= tile < pre[lo + 1]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (pre[mid] <= tile) lo = mid; else hi = mid;
    }
    const SegDesc sd = seg[lo];
    const int t0 = (tile - pre[lo]) * NT;
    Item it;
    it.r0 = rt * (PAIR ? 2 * TILE_M : TILE_M);
    it.pa = sd.wa + (size_t)it.r0 * rb;
    it.pb = PAIR ? it.pa + (size_t)TILE_M * rb : sd.wb + (size_t)it.r0 * rb;
    it.prow = (int)sd.row0 + t0;
    it.m = min(NT, (int)sd.m - t0);
    it.pad = 0;
    return it;
}

// Tokens of the B tile: the smallest of 8, 16, 32 that holds the item.
__device__ __forceinline__ int tile_tokens(int m) { return m <= 8 ? 8 : m <= 16 ? 16 : 32; }

// Stages of an item: K / 64, then those of the mins (Q4_K): with up to 32 sub-blocks one stage holds the hi parts in its first
// 32 columns and the lo parts in the others (X is stored twice for it); with more, a stage of hi and one of lo per 64.
__host__ __device__ __forceinline__ int min_stages(int type, int n_in) {
    const int nsub = n_in / 32;
    return type != T_Q4_K ? 0 : nsub <= 32 ? 1 : 2 * ((nsub + 63) / 64);
}
struct Args {
    const SegDesc* seg;
    const int32_t* nseg_dev;
    int nseg_max, n_in, n_out, rb;
    const uint16_t* op;          // operand rows [2 * rows][pitch]
    const int32_t* row_token;    // packed row -> operand row, or null: itself
    float* out;
    float* const* row_dst;       // or null: out
    int* status;
    uint32_t smem;
};

__device__ __forceinline__ uint32_t chunk_off(int r, int c) {  // 16-byte column c of row r in a 128-byte-swizzled tile
    return (uint32_t)r * 128u + (uint32_t)((c ^ (r & 7)) << 4);
}

// ---- producers: one row of both tiles per thread -------------------------------------------------------------------------
template <int T> struct Raw;
template <> struct Raw<T_Q4_K> {
    uint4 h, a, b;
    __device__ __forceinline__ void load(const uint8_t* row, int c) {
        const uint8_t* p = row + (c >> 2) * 144;
        h = __ldg(reinterpret_cast<const uint4*>(p));
        a = __ldg(reinterpret_cast<const uint4*>(p + 16 + 32 * (c & 3)));
        b = __ldg(reinterpret_cast<const uint4*>(p + 32 + 32 * (c & 3)));
    }
};
template <> struct Raw<T_IQ3_XXS> {  // 16 index bytes and two sub-block words from the aligned words around them
    uint32_t i[5], x[3];
    __device__ __forceinline__ void load(const uint8_t* row, int c) {
        const uint8_t* p = row + (c >> 2) * 98 + 2 + 16 * (c & 3);
        const uint32_t* wi = reinterpret_cast<const uint32_t*>((uintptr_t)p & ~(uintptr_t)3);
        const uint32_t* wx = reinterpret_cast<const uint32_t*>((uintptr_t)(p + 64 - 8 * (c & 3)) & ~(uintptr_t)3);
#pragma unroll
        for (int k = 0; k < 5; ++k) i[k] = __ldg(wi + k);
#pragma unroll
        for (int k = 0; k < 3; ++k) x[k] = __ldg(wx + k);
    }
};

__device__ __forceinline__ void decode_stage(const Raw<T_Q4_K>& R, int c, uint8_t* tile, int r, uint32_t, uint32_t, const uint8_t*) {
    const int t = c & 3, sh = 16 * (t & 1);
    const uint32_t a = R.h.y >> sh, cc = R.h.w >> sh;
    const uint32_t sc = t < 2 ? (a & 0x3f3fu) : ((cc & 0x0f0fu) | ((a >> 2) & 0x3030u));  // kquant.rs:878-887
    KScales s;
    s.s0 = h2sub(__byte_perm(sc, 0x64646464u, 0x4040u), 0x64006400u);
    s.s1 = h2sub(__byte_perm(sc, 0x64646464u, 0x4141u), 0x64006400u);
    s.k0 = h2mul(s.s0, 0xE400E400u);
    s.k1 = h2mul(s.s1, 0xD400D400u);
    const uint32_t w[8] = {R.a.x, R.a.y, R.a.z, R.a.w, R.b.x, R.b.y, R.b.z, R.b.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        uint32_t p[4];
        k_word<false>(w[i], 0u, s, p);
        *reinterpret_cast<uint4*>(tile + chunk_off(r, i)) = make_uint4(p[0], p[1], p[2], p[3]);
    }
}
__device__ __forceinline__ void decode_stage(const Raw<T_IQ3_XXS>& R, int c, uint8_t* tile, int r, uint32_t gl, uint32_t sl, const uint8_t* row) {
    // index bytes and sub-block words of a block share their position within 4 bytes: 98 b + 2 + 16 c and 98 b + 66 + 8 c
    const uint32_t sh = (uint32_t)((uintptr_t)(row + (c >> 2) * 98 + 2) & 2u) * 8u;
#pragma unroll
    for (int hb = 0; hb < 2; ++hb) {
        const uint32_t aux = __funnelshift_r(R.x[hb], R.x[hb + 1], sh);
        const uint32_t s2 = h2sub((((aux >> 27) & 0x1Eu) | 0x6401u) * 0x10001u, 0x64006400u);  // 2 s + 1 in both halves
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t iw = __funnelshift_r(R.i[2 * hb + (q >> 1)], R.i[2 * hb + (q >> 1) + 1], sh) >> (16 * (q & 1));
            uint32_t p[4];
            iq3_pairs_h(gl, sl, iw, q == 0 ? aux << 6 : aux >> (7 * q - 6), p);
            *reinterpret_cast<uint4*>(tile + chunk_off(r, 4 * hb + q)) =
                make_uint4(h2mul(p[0], s2), h2mul(p[1], s2), h2mul(p[2], s2), h2mul(p[3], s2));
        }
    }
}
// Stage u of the mins of one Q4_K row.
__device__ __forceinline__ void mins_stage(const uint8_t* row, int nsub, int u, uint8_t* tile, int r) {
    const bool both = nsub <= 32;
    const int base = both ? 0 : 64 * (u >> 1);
#pragma unroll 1
    for (int c = 0; c < 8; ++c) {  // eight sub-blocks = one 256-element block per 16-byte column
        const int part = both ? c >> 2 : u & 1, blk = base / 8 + (both ? c & 3 : c);
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (blk * 8 < nsub) {
            const uint4 h = __ldg(reinterpret_cast<const uint4*>(row + blk * 144));
            const float dm = -kMinScale * h2f((uint16_t)(h.x >> 16));
            uint32_t o[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {  // sub-blocks 2 k, 2 k + 1
                const int sh = 16 * (k & 1);
                const uint32_t b = h.z >> sh, d = h.w >> sh;
                const uint32_t mn = k < 2 ? (b & 0x3f3fu) : (((d >> 4) & 0x0f0fu) | ((b >> 2) & 0x3030u));
                const float f0 = dm * (float)(mn & 0xffu), f1 = dm * (float)(mn >> 8);
                const __half2 hi = __floats2half2_rn(f0, f1);
                const float2 hf = __half22float2(hi);
                const __half2 lo = __floats2half2_rn(f0 - hf.x, f1 - hf.y);
                o[k] = part ? *reinterpret_cast<const uint32_t*>(&lo) : *reinterpret_cast<const uint32_t*>(&hi);
            }
            v = make_uint4(o[0], o[1], o[2], o[3]);
        }
        *reinterpret_cast<uint4*>(tile + chunk_off(r, c)) = v;
    }
}

__device__ __forceinline__ float swiglu_fast(float g, float u) { return __fdividef(g, 1.0f + __expf(-g)) * u; }

__device__ __forceinline__ void tma_gather4(void* dst, const CUtensorMap* map, int x, int y0, int y1, int y2, int y3, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(
            s32(dst)),
        "l"(map), "r"(x), "r"(y0), "r"(y1), "r"(y2), "r"(y3), "r"(s32(bar))
        : "memory");
}

// Shared memory: [barriers, segment table, items][B stages that fit below the tables][IQ3_XXS tables at a 32 KB boundary][A stages][other B stages]
template <int T> struct Layout {
    static constexpr int STAGES = T == T_Q4_K ? 5 : 4;
    static constexpr int LOW_B = T == T_Q4_K ? STAGES : 3;   // B stages in front
    static constexpr int HEAD = ((2 * STAGES + 2 * NB) * 8 + 16 + (kMaxSeg + 1) * 4 + kLocalItems * (int)sizeof(Item) + 1023) / 1024 * 1024;
};

template <int T, bool PAIR>  // PAIR: both tiles from seg.wa (256 rows, fp32 results); else gate and up rows, silu(g) * u
__global__ void __launch_bounds__(NTHREADS, 1) grouped_tc_kernel(const Args A, const __grid_constant__ Maps maps) {
    using L = Layout<T>;
    constexpr int STAGES = L::STAGES;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* base = smem_raw + ((1024u - (s32(smem_raw) & 1023u)) & 1023u);
    uint64_t* full = reinterpret_cast<uint64_t*>(base);
    uint64_t* empty = full + STAGES;
    uint64_t* tfull = empty + STAGES;
    uint64_t* tfree = tfull + NB;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfree + NB);
    int* pre = reinterpret_cast<int*>(tmem_slot + 4);  // [nseg + 1] first token tile of a segment
    Item* itab = reinterpret_cast<Item*>((reinterpret_cast<uintptr_t>(pre + kMaxSeg + 1) + 7) & ~(uintptr_t)7);
    uint8_t* b_low = base + L::HEAD;
    uint8_t* p = b_low + L::LOW_B * B_STAGE;
    uint8_t* book = p;
    if constexpr (T == T_IQ3_XXS) {
        book += (kMmBookAlign - (s32(p) & (kMmBookAlign - 1))) & (kMmBookAlign - 1);
        p = book + sizeof(MmCodebook);
    }
    uint8_t* a_base = p;
    uint8_t* b_high = a_base + STAGES * A_STAGE;
    if ((uint32_t)(b_high + (STAGES - L::LOW_B) * B_STAGE - smem_raw) > A.smem) {  // only if shared memory started elsewhere
        if (threadIdx.x == 0) status_set(A.status, 26);
        return;
    }
    auto b_tile = [&](int st) { return st < L::LOW_B ? b_low + st * B_STAGE : b_high + (st - L::LOW_B) * B_STAGE; };

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nchunks = A.n_in / BK, nmin = min_stages(T, A.n_in), nch = nchunks + nmin, nblk = A.n_in / 256, nsub = A.n_in / 32;
    const int row_tiles = A.n_out / (PAIR ? 2 * TILE_M : TILE_M);
    const int pitch = row_pitch(A.n_in), scale_col = A.n_in + x_cols(A.n_in);

    if (tid == 0) {
        for (int i = 0; i < STAGES; ++i) {
            mb_init(&full[i], 5);   // the four warps of a producer group + the TMA thread's expect_tx
            mb_init(&empty[i], 1);  // one tcgen05.commit
        }
        for (int i = 0; i < NB; ++i) {
            mb_init(&tfull[i], 1);
            mb_init(&tfree[i], EWARPS);
        }
        fence_mbarrier_init();
    }
    if constexpr (T == T_IQ3_XXS) {
        for (int i = tid; i < (int)(sizeof(MmCodebook) / 16); i += NTHREADS)
            cp_async16<false>(book + 16 * i, reinterpret_cast<const uint8_t*>(&g_mm_codebook) + 16 * i);
        cp_async_commit();
        cp_async_wait_all();
    }
    if (warp == W_MMA) tmem_alloc<NB * BUF_COLS>(tmem_slot);
    pdl_wait();
    pdl_launch_dependents();
    const int nseg = min(*A.nseg_dev, A.nseg_max);
    for (int i = tid; i < nseg; i += NTHREADS) pre[i + 1] = ((int)A.seg[i].m + NT - 1) / NT;
    __syncthreads();
    if (warp == 0) {
        int carry = 0;
        for (int b = 0; b < nseg; b += 32) {
            const int i = b + lane;
            int v = i < nseg ? pre[i + 1] : 0;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int o = __shfl_up_sync(0xffffffffu, v, d);
                if (lane >= d) v += o;
            }
            if (i < nseg) pre[i + 1] = carry + v;
            carry += __shfl_sync(0xffffffffu, v, 31);
        }
        if (lane == 0) pre[0] = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const int n_items = nseg > 0 ? pre[nseg] * row_tiles : 0;
    const int GR = gridDim.x;
    const int my_items = (int)blockIdx.x < n_items ? (n_items - (int)blockIdx.x + GR - 1) / GR : 0;
    if (tid < min(my_items, kLocalItems)) itab[tid] = decode_item<PAIR>((int)blockIdx.x + tid * GR, row_tiles, A.rb, nseg, pre, A.seg);
    __syncthreads();
    auto item = [&](int k) {
        return k < kLocalItems ? itab[k] : decode_item<PAIR>((int)blockIdx.x + k * GR, row_tiles, A.rb, nseg, pre, A.seg);
    };
    bool ok = true;

    if (warp < EWARPS) {
        // ---------------- epilogue: TMEM lane = weight row ----------------
        const int quad = warp & 3, hsel = warp >> 2;
        const int r = quad * 32 + lane;
        const uint32_t tlane = tmem_base + ((uint32_t)(quad * 32) << 16);
        int buf = 0;
        uint32_t pb = 0;
        uint16_t dn[2] = {0, 0};
        auto fetch_d = [&](const Item& it, int blk) {  // this row's block scale in both tiles
            dn[0] = __ldg(reinterpret_cast<const uint16_t*>(it.pa + (size_t)r * A.rb + blk * kBB<T>));
            dn[1] = __ldg(reinterpret_cast<const uint16_t*>(it.pb + (size_t)r * A.rb + blk * kBB<T>));
        };
        Item nx = my_items > 0 ? item(0) : Item{};
        if (my_items > 0) fetch_d(nx, 0);
        for (int k = 0; k < my_items && ok; ++k) {
            const Item it = nx;
            if (k + 1 < my_items) nx = item(k + 1);
            const int nte = tile_tokens(it.m), half = nte >> 1;
            float rs = 0.f;  // lane j: what undoes the scaling of token j of this warp's half
            if (lane < half) {
                const int pr = it.prow + min(hsel * half + lane, it.m - 1);
                const int orow = A.row_token ? A.row_token[pr] : pr;
                rs = *reinterpret_cast<const float*>(A.op + (size_t)(2 * orow) * pitch + scale_col);
            }
            float acc[2][16];
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[mt][j] = 0.f;
            for (int blk = 0; blk < nblk + (nmin ? 1 : 0); ++blk) {
                float s[2] = {1.f / kMinScale, 1.f / kMinScale};
                if (blk < nblk) {
                    constexpr float f = T == T_IQ3_XXS ? 0.25f : 1.f;
                    s[0] = f * h2f(dn[0]);
                    s[1] = f * h2f(dn[1]);
                    if (blk + 1 < nblk) fetch_d(it, blk + 1);
                    else if (k + 1 < my_items) fetch_d(nx, 0);
                }
                ok = warp_all(mb_wait(&tfull[buf], pb, A.status, 3));
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                    for (int h = 0; h < 2; ++h) {  // eight tokens each; 32-token tiles have two per warp
                        if (h == 0 || nte == 32) {
                            uint32_t v[16];
                            tmem_ld16(tlane + (uint32_t)(buf * BUF_COLS + mt * 2 * NT + hsel * nte + 16 * h), v);
                            tmem_ld_wait();
#pragma unroll
                            for (int j = 0; j < 8; ++j)
                                acc[mt][8 * h + j] = fmaf(s[mt], __uint_as_float(v[2 * j]) + __uint_as_float(v[2 * j + 1]), acc[mt][8 * h + j]);
                        }
                    }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mb_arrive(&tfree[buf]);
                if (++buf == NB) { buf = 0; pb ^= 1u; }
            }
            if (!ok) break;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const float f = __shfl_sync(0xffffffffu, rs, j);
                const int t = hsel * half + j;
                if (j < half && t < it.m) {
                    const float a0 = acc[0][j] * f, a1 = acc[1][j] * f;
                    if constexpr (!PAIR) {
                        A.out[(size_t)(it.prow + t) * A.n_out + it.r0 + r] = swiglu_fast(a0, a1);
                    } else {
                        // expert parallel: the owner's (token, slot) row
                        float* o = A.row_dst ? A.row_dst[it.prow + t] + it.r0 + r : A.out + (size_t)(it.prow + t) * A.n_out + it.r0 + r;
                        o[0] = a0;
                        o[TILE_M] = a1;
                    }
                }
            }
        }
    } else if (warp < W_TMA) {
        // ---------------- producers ----------------
        const int pw = warp - EWARPS, grp = pw >> 2, r = (pw & 3) * 32 + lane;
        const uint32_t gl = s32(book) + 8 * (lane & (kLutRep - 1)), sl = s32(book) + (uint32_t)sizeof(uint2) * 256 * kLutRep + 4 * (lane & (kLutRep - 1));
        int k = 0, c = grp, st = grp;  // stage number grp, grp + GROUPS, ... -> (item, stage of the item, ring slot)
        uint32_t ph = 1u;              // parity of the empty barrier to wait for; the first turn of the ring finds it free
        while (c >= nch && k < my_items) { c -= nch; ++k; }
        const uint8_t *pa = nullptr, *pb = nullptr;
        Raw<T> ra, rb;
        auto aim = [&]() {
            const Item it = item(k);
            pa = it.pa + (size_t)r * A.rb;
            pb = it.pb + (size_t)r * A.rb;
        };
        auto fetch = [&]() {
            if (k < my_items && c < nchunks) {
                ra.load(pa, c);
                rb.load(pb, c);
            }
        };
        if (k < my_items) aim();
        fetch();
        while (k < my_items) {
            ok = warp_all(mb_wait(&empty[st], ph, A.status, 2));
            if (!ok) break;
            uint8_t* tile = a_base + st * A_STAGE;
            if (c < nchunks) {
                decode_stage(ra, c, tile, r, gl, sl, pa);
                decode_stage(rb, c, tile + A_TILE, r, gl, sl, pb);
            } else {
                mins_stage(pa, nsub, c - nchunks, tile, r);
                mins_stage(pb, nsub, c - nchunks, tile + A_TILE, r);
            }
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mb_arrive(&full[st]);
            c += GROUPS;
            if (c >= nch) {
                do { c -= nch; ++k; } while (c >= nch && k < my_items);
                if (k < my_items) aim();
            }
            st += GROUPS;
            if (st >= STAGES) { st -= STAGES; ph ^= 1u; }
            fetch();
        }
    } else if (warp == W_TMA) {
        // ---------------- TMA: hi and lo rows of the tokens ----------------
        int st = 0;
        uint32_t ph = 1u;
        for (int k = 0; k < my_items && ok; ++k) {
            const Item it = item(k);
            const int nte = tile_tokens(it.m), sel = nte == 8 ? 0 : nte == 16 ? 1 : 2;
            int y0 = 0, y1 = 0;  // gathers: lane l brings tokens 2 l and 2 l + 1
            if (A.row_token && lane < nte / 2) {
                y0 = 2 * A.row_token[it.prow + min(2 * lane, it.m - 1)];
                y1 = 2 * A.row_token[it.prow + min(2 * lane + 1, it.m - 1)];
            }
            for (int c = 0; c < nch; ++c) {
                ok = warp_all(mb_wait(&empty[st], ph, A.status, 4));
                if (!ok) break;
                const int u = c - nchunks, col = c < nchunks ? c * BK : A.n_in + 64 * (u >> 1);
                if (lane == 0) mb_expect_tx(&full[st], (uint32_t)(2 * nte * BK * 2));
                __syncwarp();
                if (A.row_token) {
                    if (lane < nte / 2) tma_gather4(b_tile(st) + lane * 512, &maps.row, col, y0, y0 + 1, y1, y1 + 1, &full[st]);
                } else if (elect_one()) {
                    tma_load_2d(b_tile(st), &maps.box[sel], col, 2 * it.prow, &full[st]);
                }
                __syncwarp();
                if (++st == STAGES) { st = 0; ph ^= 1u; }
            }
        }
    } else {
        // ---------------- MMA issue ----------------
        int st = 0, buf = 0;
        uint32_t ph = 0u, pf = 1u;
        for (int k = 0; k < my_items && ok; ++k) {
            const Item it = item(k);
            const int nte = tile_tokens(it.m);
            const uint32_t idesc = (1u << 4) | ((uint32_t)((2 * nte) >> 3) << 17) | ((uint32_t)(TILE_M >> 4) << 24);  // fp16 x fp16 -> fp32
            for (int c = 0; c < nch; ++c) {
                ok = warp_all(mb_wait(&full[st], ph, A.status, 5));
                if (!ok) break;
                const bool first = c < nchunks ? (c & 3) == 0 : c == nchunks;
                const bool last = c < nchunks ? (c & 3) == 3 : c == nch - 1;
                if (first) ok = warp_all(mb_wait(&tfree[buf], pf, A.status, 6));
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t a_lo = desc_lo(s32(a_base + st * A_STAGE)), b_lo = desc_lo(s32(b_tile(st)));
                    const uint32_t d0 = tmem_base + (uint32_t)(buf * BUF_COLS);
                    // a stage of mins uses the K steps that hold sub-blocks (hi and lo halves side by side when both fit)
                    const int u = c - nchunks;
                    const int live = c < nchunks ? 4 : nsub <= 32 ? (nsub + 15) / 16 : min(4, (nsub - 64 * (u >> 1) + 15) / 16);
                    uint32_t acc = first ? 0u : 1u;
                    for (int ks = 0; ks < 4; ++ks) {
                        if (c >= nchunks && (nsub <= 32 ? (ks & 1) >= live : ks >= live)) continue;
                        mma_bf16(d0, desc_of(a_lo + 2u * ks), desc_of(b_lo + 2u * ks), idesc, acc);
                        mma_bf16(d0 + 2 * NT, desc_of(a_lo + (A_TILE >> 4) + 2u * ks), desc_of(b_lo + 2u * ks), idesc, acc);
                        acc = 1u;
                    }
                    mma_commit(&empty[st]);
                    if (last) mma_commit(&tfull[buf]);
                }
                __syncwarp();
                if (last && ++buf == NB) { buf = 0; pf ^= 1u; }
                if (++st == STAGES) { st = 0; ph ^= 1u; }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == W_MMA) {
        tc_fence_after();
        tmem_free<NB * BUF_COLS>(tmem_base);
    }
}

// ---- operand rows ----------------------------------------------------------------------------------------------------------
// Row p of x as fp16 hi and lo of the row times a power of two (largest element in [512, 1024)), in the order in which the
// weights of `type` are decoded, then the sums of its 32-element sub-blocks (Q4_K) and what undoes the scaling.  A warp per row.
template <int T>
__global__ void __launch_bounds__(256) operand_rows_kernel(const float* __restrict__ x, int ldx, int rows, const int32_t* rows_dev, int K, int pitch,
                                                               uint16_t* __restrict__ op) {
    pdl_wait();
    pdl_launch_dependents();
    const int p = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (p >= rows || (rows_dev && p >= *rows_dev)) return;
    const float* xr = x + (size_t)p * ldx;
    uint32_t mx = 0u;
    for (int i = 4 * lane; i < K; i += 128) {
        const float4 v = *reinterpret_cast<const float4*>(xr + i);
        mx = max(mx, max(max(__float_as_uint(fabsf(v.x)), __float_as_uint(fabsf(v.y))), max(__float_as_uint(fabsf(v.z)), __float_as_uint(fabsf(v.w)))));
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    const float up = operand_scale(mx);
    uint16_t* hi = op + (size_t)(2 * p) * pitch;
    for (int b = 0; b < K; b += 256) {
        int e0, e1;
        operand_elems<T>(b, lane, e0, e1);
        operand_block<T>(*reinterpret_cast<const float4*>(xr + e0), *reinterpret_cast<const float4*>(xr + e1), up, b, K, pitch, lane, hi);
    }
    operand_tail<T>(up, K, pitch, lane, hi);
}
}  // namespace tg

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

// [rows][cols] 16-bit row-major, box = 64 columns x box_rows rows, 128-byte swizzle.
int tc_make_map(void* m, void* base, uint64_t rows, uint64_t cols, uint32_t box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) {
        set_error("cuTensorMapEncodeTiled is not available from this driver");
        return DNB_ERR_CUDA;
    }
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {cols * 2};
    const cuuint32_t box[2] = {64, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(reinterpret_cast<CUtensorMap*>(m), CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed (%d) for %llu x %llu box %u", (int)r, (unsigned long long)rows,
                  (unsigned long long)cols, box_rows);
        return DNB_ERR_CUDA;
    }
    return DNB_OK;
}

size_t tc_row_pitch(int n_in) { return (size_t)tg::row_pitch(n_in); }

// Tensor maps over `rows` operand rows (2 * rows map rows of `pitch` fp16).
int tc_make_maps(void* op, uint64_t rows, int n_in, TcMaps* out) {
    static_assert(sizeof(TcMaps) == sizeof(tg::Maps), "TcMaps must mirror tg::Maps");
    tg::Maps* m = reinterpret_cast<tg::Maps*>(out);
    int rc;
    for (int i = 0; i < 3; ++i)
        if ((rc = tc_make_map(&m->box[i], op, 2 * rows, (uint64_t)tg::row_pitch(n_in), 16u << i))) return rc;
    return tc_make_map(&m->row, op, 2 * rows, (uint64_t)tg::row_pitch(n_in), 1);
}

int launch_operand_rows(dnb_ctx* c, cudaStream_t st, int type, const float* x, int ldx, int rows, int n_in, uint16_t* op, const char* name,
                        const int32_t* rows_dev) {
    if (n_in % 256 || ldx % 4) return DNB_DECLINED;
    ProfScope prof_(c, st, name);
    auto kern = type == T_Q4_K ? tg::operand_rows_kernel<T_Q4_K> : tg::operand_rows_kernel<T_IQ3_XXS>;
    DNB_CUDA(launch_k(kern, dim3((rows + 7) / 8), dim3(256), 0, st, c->use_pdl, x, ldx, rows, rows_dev, n_in, tg::row_pitch(n_in), op));
    c->launches++;
    return DNB_OK;
}

bool tc_handles(int type, int n_in, int n_out, bool fused) {
    return (type == T_Q4_K || type == T_IQ3_XXS) && n_in % 256 == 0 && n_out % (fused ? tg::TILE_M : 2 * tg::TILE_M) == 0;
}

template <int T, bool PAIR>
static int launch_tc_t(dnb_ctx* c, cudaStream_t st, tg::Args& A, const tg::Maps& M) {
    using L = tg::Layout<T>;
    size_t at = kMmSmemBase + L::HEAD + L::LOW_B * tg::B_STAGE;
    if (T == T_IQ3_XXS) at = (at + kMmBookAlign - 1) / kMmBookAlign * kMmBookAlign + sizeof(MmCodebook);
    const size_t smem = at + L::STAGES * tg::A_STAGE + (L::STAGES - L::LOW_B) * tg::B_STAGE - kMmSmemBase;
    A.smem = (uint32_t)smem;
    auto kern = tg::grouped_tc_kernel<T, PAIR>;
    static SmemGrant grant;
    DNB_CUDA(grant_smem(grant, c->device, kern, smem));
    ProfScope prof_(c, st, PAIR ? "tc_down" : "tc_gate_up");
    DNB_CUDA(launch_k(kern, dim3(c->sm_count), dim3(tg::NTHREADS), smem, st, c->use_pdl, A, M));
    c->launches++;
    return DNB_OK;
}

int launch_grouped_tc(dnb_ctx* c, cudaStream_t st, int type, bool fused, const SegDesc* seg, const int32_t* nseg_dev, int nseg_max, int n_in,
                      int n_out, const uint16_t* op, const TcMaps* maps, const int32_t* row_token, float* out, float* const* row_dst) {
    if (!tc_handles(type, n_in, n_out, fused) || nseg_max > tg::kMaxSeg) return DNB_DECLINED;
    int rc = type == T_IQ3_XXS ? upload_mm_tables(c->device) : DNB_OK;
    if (rc) return rc;
    tg::Args A = {};
    A.seg = seg; A.nseg_dev = nseg_dev; A.nseg_max = nseg_max; A.n_in = n_in; A.n_out = n_out; A.rb = (int)row_bytes(type, n_in);
    A.op = op; A.row_token = row_token; A.out = out; A.row_dst = row_dst; A.status = c->status;
    const tg::Maps& M = *reinterpret_cast<const tg::Maps*>(maps);
    if (type == T_Q4_K) return fused ? launch_tc_t<T_Q4_K, false>(c, st, A, M) : launch_tc_t<T_Q4_K, true>(c, st, A, M);
    return fused ? launch_tc_t<T_IQ3_XXS, false>(c, st, A, M) : launch_tc_t<T_IQ3_XXS, true>(c, st, A, M);
}

}  // namespace dnb
