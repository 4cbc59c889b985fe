// Grouped per-expert GEMM of chunked prefill on tcgen05: Q4_K and IQ3_XXS experts as EXACT fp16 integers, block scales after
// the tensor-core sum.
//
// Reference kernels of this role: kernels_exp_k_pf.cu:188-258 (m-row fp32), kernels_gemm_grouped.cu:134-273 (fp32 FMA),
// kernels_exp_iq_tc.cu (bf16 wmma); block layouts kquant.rs:505-526, :659-680.
//
//     W . x  =  sum over 256-element blocks b of  s_b * [ sum_i w_i * x_i ]   ( - sum over sub-blocks of (dmin * m) * X )
//   Q4_K    : w = sc * q <= 945 (times 2^-14, which s_b takes back), s_b = d, and the mins: X = the sum of the sub-block's 32 activations
//   IQ3_XXS : w = codebook magnitude * sign * (2 s + 1) <= 1922, s_b = d / 4
// Every w is an integer below 2048 and exact in fp16, so a weight costs its decoding and nothing is rounded.  The mins are one
// more block of K = sub-blocks: A = -(dmin * m) as fp16 hi and lo, times a power of two of the row's own that fits its largest
// dmin into fp16's range whatever its size, B = X.  An activation is fp16 hi + lo (22 bits) of the row times a power of two that
// puts its largest element into [512, 1024).
//
// What bounds it: instructions.  A 64-element stage of two 128-row tiles is 900 to 1,500 warp instructions of decoding on four schedulers, a
// copy, a wait or a hand-over of some warp as much again, and 16 MMAs of N = tokens (8 N cycles in all); 0.7 of the issue slots are taken.
// Shared memory is next: with A tiles in it (32 KB written and 32 KB read per stage, B read once per tile) a stage took 840 cycles, all of
// them shared-memory bandwidth.  So A goes from the producers' registers to tensor memory (tcgen05.st, thread = row = lane) and the MMA
// takes it from there.  One role per warp, each with a ring of its own in front:
//   * two warps copy packed rows (a 256-element block of all 256 rows, a tile a warp: 9 or 7 neighbouring lanes per row) into a raw ring.
//     (A thread that fetches its own row's bytes touches 32 cache lines per instruction; that alone took 0.5 us per stage.)
//   * four warps copy the tokens' lo (two) and hi rows into swizzled B tiles, two stages at a time, gathered from the token-major rows: no
//     packed copy of the activations.  (TMA row gathers took 80 cycles per four rows; a proxy fence in the copying warp waits for the copies
//     still on their way, so it is the MMA thread that executes it.  Two warps were behind the others in IQ3_XXS.)
//   * four groups of four producer warps, (even or odd stages) x (tile), a thread one row: decodes 64 weights into registers, THEN
//     waits for its slot (tensor memory holds only a block; with the decoding inside its turn-around a stage took 1,100
//     cycles) and stores them.  The block's scales go to a small ring, its mins to shared memory of the thread's own.
//   * two MMA threads, a tile each.  A block's weights stay in tensor memory while they are multiplied with the lo rows and then with the hi
//     rows, into the same columns: with 64 tokens there are two accumulator buffers (with sums of hi and lo apart there was room for
//     one, and the tensor core waited 350 cycles of a stage's 1,060 while it was read), and as lo comes first, the sums are rounded once more
//     than those of hi alone (what that costs is in operand_rows.cuh, and why the result is no less exact).  A wait, a fence and a commit are some 200
//     cycles of a thread's time, so two stages share them, and one thread for both tiles would be the bottleneck.
//   * eight epilogue warps, two accumulator buffers (thread = weight row, half of the token columns of both tiles).
// Persistent, one CTA per SM; items (segment, up to 64 tokens, 128 rows x 2) dealt round-robin.
// The code of all roles has to stay small: eight warps of a scheduler run five different loops.  Waiting loops that the compiler
// had unrolled made 150 KB of it, and no_instruction was a stall as frequent as the arithmetic pipes' (75 KB: Q4_K 434 -> 409 us a pass of the
// below); one copy of the decoding instead of two, and one of the MMA loop, 493 -> 434.
//
// Measured, 512 tokens of 2048 x 512, top 10 of 512 under a skewed router, two layers, us a pass: items of 32 (Q4_K) or 64 tokens with hi and lo
// sums apart -> these -> the shared expert's items first, nibbles as numbers below the normal ones, 32 copies of the signs: Q4_K 501 -> 409 -> 384,
// IQ3_XXS 473 -> 429 -> 421; a prompt of 14,018 tokens 6,865 -> 5,684 -> 5,285; the last round dealt backwards: 381, 416 and 5,216.
#include <cuda_fp16.h>

#include <type_traits>

#include "dnb_common.cuh"
#include "tc_ptx.cuh"
#include "iq3_f16.cuh"
#include "operand_rows.cuh"

namespace dnb {
namespace tg {
using namespace tcp;

constexpr int BK = 64;                  // K of a stage: one 128-byte swizzle row of fp16
constexpr int TILE_M = 128;
constexpr int A_COLS = BK / 2;          // tensor-memory columns of an A tile (two fp16 each)
constexpr int EWARPS = 8, PWARPS = 16, RWARPS = 2, BWARPS = 4;
constexpr int W_RAW = EWARPS + PWARPS, W_B = W_RAW + RWARPS, W_MMA = W_B + BWARPS;  // two warps, a tile each
constexpr int NTHREADS = 1024;
// Tokens of an item at most; N of its MMAs follows it in sixteens.  Against items of up to 32 (or, from some rows a segment on, 64), us a layer of
// 2048 x 512, evenly routed and skewed by -1.1 ln rank: Q4_K, 64 experts top 10, 512 tokens 212, 212 -> 186, 188; 128 top 8, 700 tokens 223, 239 ->
// 183, 207; 512 top 10, 512 tokens 434, 253 -> 439, 207; 64 tokens 306, 103 -> 307, 105.  IQ3_XXS 215, 214 -> 195, 195; 217, 240 -> 192, 218;
// 510, 242 -> 452, 217; 331, 106 -> 319, 108.
constexpr int NT = 64;
constexpr int NB = 2, BUF_COLS = 2 * NT;  // accumulator buffers: two tiles x tokens
constexpr int SLOTS = 4;                // of A (tensor memory) and of each half of B: stage c of a block has slot c
constexpr int PAIRS = SLOTS / 2;        // two stages have a barrier in common
constexpr int B_SLOT = NT * BK * 2, B_BYTES = 2 * SLOTS * B_SLOT;  // lo rows, then hi rows
// Registers per thread of the warpgroups once their roles are known; launched with 64, and no more than that in sum.
constexpr int REG_EPI = 112, REG_PROD = 56, REG_COPY = 32;
static_assert(2 * REG_EPI + 4 * REG_PROD + 2 * REG_COPY <= 8 * 64, "register split");
static_assert(EWARPS % 4 == 0 && W_RAW % 4 == 0 && (W_MMA + 2) * 32 == NTHREADS, "a register split falls between warpgroups");
static_assert(EWARPS == 8 && PWARPS == 16 && RWARPS == 2 && BWARPS == 4, "what the roles' index arithmetic and the register split are written for");
constexpr int kMaxSeg = 1055;
constexpr int kLocalItems = 40;
constexpr int A_COL0 = NB * BUF_COLS, TMEM_COLS = A_COL0 + SLOTS * 2 * A_COLS;
static_assert(TMEM_COLS == 512, "tensor memory");
constexpr int SCL = 8;                  // ring of block scales (the mins count as a block): producers are at most three blocks ahead of the epilogue

template <int T> constexpr int kBB = T == T_Q4_K ? 144 : 98;

struct Item {
    const uint8_t* pa;  // tile 0, first row
    const uint8_t* pb;  // tile 1
    int prow, m;        // first packed row, tokens
    int r0, pad;        // first output row
};

template <bool PAIR>
__device__ __forceinline__ Item decode_item(int item, int row_tiles, int rb, int nseg, int first, const int* pre, const SegDesc* __restrict__ seg) {
    int tile = item / row_tiles;
    const int rt = item - tile * row_tiles;
    tile += first;
    if (tile >= pre[nseg]) tile -= pre[nseg];
    int lo = 0, hi = nseg;  // pre[lo] <= tile < pre[lo + 1]
#pragma unroll 1
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

// Tokens of the B tile, N of its MMAs: the item's in sixteens.
__device__ __forceinline__ int tile_tokens(int m) { return (m + 15) & ~15; }

// An item's stages: for every eight blocks (or the rest) their 64-element stages, then those of the mins (Q4_K): with up to four
// blocks one stage holds the hi parts of the up to 32 mins in its first 32 columns and the lo parts in the others (the operand row
// has those sums twice), with more there is a stage of hi and one of lo.
template <int T> __host__ __device__ __forceinline__ int min_stages(int blocks) { return T != T_Q4_K ? 0 : blocks <= 4 ? 1 : 2; }

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

template <int N> __device__ __forceinline__ void reg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void reg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// ---- producers: one row of both tiles per thread -------------------------------------------------------------------------
template <int T> struct Raw;  // what stage `c` (0..3) of a block needs of a row's packed bytes
template <> struct Raw<T_Q4_K> {
    static constexpr int UNITS = 9, RS = 144;
    uint4 h, a, b;
    __device__ __forceinline__ void load(const uint8_t* p, int c) {
        h = *reinterpret_cast<const uint4*>(p);
        a = *reinterpret_cast<const uint4*>(p + 16 + 32 * c);
        b = *reinterpret_cast<const uint4*>(p + 32 + 32 * c);
    }
    __device__ __forceinline__ float scale() const { return 16384.0f * h2f((uint16_t)h.x); }  // the weights are 2^-14 of theirs
};
template <> struct Raw<T_IQ3_XXS> {  // 16 index bytes and two sub-block words from the aligned words around them
    static constexpr int UNITS = 7, RS = 112;
    uint32_t i[5], x[3];
    uint32_t d, sh;
    __device__ __forceinline__ void load(const uint8_t* p, int c) {  // p: the block, on an even address
        sh = ((s32(p) + 2u) & 2u) * 8u;
        d = ld16(p);
        const uint32_t* wi = reinterpret_cast<const uint32_t*>(p + 2 + 16 * c - (sh >> 3));
        const uint32_t* wx = reinterpret_cast<const uint32_t*>(p + 66 + 8 * c - (sh >> 3));
#pragma unroll
        for (int k = 0; k < 4; ++k) i[k] = wi[k];
        i[4] = wi[sh ? 4 : 3];  // the word after is the row's only where the words are shifted
        x[0] = wx[0];
        x[1] = wx[1];
        x[2] = wx[sh ? 2 : 1];
    }
    __device__ __forceinline__ float scale() const { return 0.25f * h2f((uint16_t)d); }
};

// 32 columns of this thread's tensor-memory lane.
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,"
        "%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
        "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
        "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
template <int N> using Int = std::integral_constant<int, N>;
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[16]) { tmem_ld16(taddr, r); }
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
// D (+)= A * B with A in tensor memory.
__device__ __forceinline__ void mma_f16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
}

__device__ __forceinline__ void decode_stage(const Raw<T_Q4_K>& R, int c, uint32_t (&o)[32], uint32_t, uint32_t) {
    const int sh = 16 * (c & 1);
    const uint32_t a = R.h.y >> sh, cc = R.h.w >> sh;
    const uint32_t sc = c < 2 ? (a & 0x3f3fu) : ((cc & 0x0f0fu) | ((a >> 2) & 0x3030u));  // kquant.rs:878-887
    KScales s;
    s.s0 = h2mul(h2sub(__byte_perm(sc, 0x64646464u, 0x4040u), 0x64006400u), 0x64006400u);
    s.s1 = h2mul(h2sub(__byte_perm(sc, 0x64646464u, 0x4141u), 0x64006400u), 0x54005400u);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint4 q = h ? R.b : R.a;
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint32_t p[4];
            k_word(w[i], s, p);
#pragma unroll
            for (int j = 0; j < 4; ++j) o[16 * h + 4 * i + j] = p[j];
        }
    }
}
__device__ __forceinline__ void decode_stage(const Raw<T_IQ3_XXS>& R, int, uint32_t (&o)[32], uint32_t gl, uint32_t sl) {
#pragma unroll
    for (int hb = 0; hb < 2; ++hb) {
        const uint32_t aux = __funnelshift_r(R.x[hb], R.x[hb + 1], R.sh);
        const uint32_t s2 = h2sub((((aux >> 27) & 0x1Eu) | 0x6401u) * 0x10001u, 0x64006400u);  // 2 s + 1 in both halves
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t iw = __funnelshift_r(R.i[2 * hb + (q >> 1)], R.i[2 * hb + (q >> 1) + 1], R.sh) >> (16 * (q & 1));
            uint32_t p[4];
            iq3_pairs_h(gl, sl, iw, q == 0 ? aux << 7 : aux >> (7 * q - 7), p);
#pragma unroll
            for (int j = 0; j < 4; ++j) o[16 * hb + 4 * q + j] = h2mul(p[j], s2);
        }
    }
}
// Stage u of the mins of one Q4_K row.  mm, dd: the last eight mins bytes of each block's header and its dmin, as the thread saved
// them (PWARPS * 32 entries from block to block); ex: exponent field of the scale, a power of two.
__device__ __forceinline__ void mins_stage(const uint2* mm, const uint16_t* dd, int blocks, int u, uint32_t ex, uint32_t (&o)[32]) {
    const bool both = blocks <= 4;
    const uint32_t neg = ((ex << 10) | 0x8000u) * 0x10001u;
#pragma unroll
    for (int c = 0; c < 8; ++c) {  // the eight sub-blocks of a block: four columns
        const bool low = both ? c >= 4 : u != 0;
        const int blk = both ? c & 3 : c;
        const bool live = blk < blocks;
        const uint2 h = mm[(live ? blk : 0) * PWARPS * 32];
        const uint32_t d = live ? dd[blk * PWARPS * 32] : 0u;
        const uint32_t dm = h2mul(d * 0x10001u, neg);  // -scale * dmin
        const uint32_t mn[2] = {h.x & 0x3f3f3f3fu, ((h.y >> 4) & 0x0f0f0f0fu) | ((h.x >> 2) & 0x30303030u)};  // kquant.rs:878-887
#pragma unroll
        for (int k = 0; k < 4; ++k) {  // sub-blocks 2 k, 2 k + 1: dmin * m rounded, or exactly what that left over
            const uint32_t m2 = h2sub(__byte_perm(mn[k >> 1], 0x64646464u, (k & 1) ? 0x4342u : 0x4140u), 0x64006400u);
            const uint32_t hi = h2mul(dm, m2);
            o[4 * c + k] = low ? h2fma(dm, m2, hi ^ 0x80008000u) : hi;
        }
    }
}

__device__ __forceinline__ float swiglu_fast(float g, float u) { return __fdividef(g, 1.0f + __expf(-g)) * u; }

__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {  // an arrival once this thread's copies so far are complete
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(s32(bar)) : "memory");
}
template <int N> __device__ __forceinline__ void cp_async_wait_group() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Shared memory: [barriers, segment table, items][block scales][B ring][IQ3_XXS tables at a 32 KB boundary][raw ring][Q4_K: mins]
template <int T> struct Layout {
    static constexpr int RSTAGES = 3;
    static constexpr int RAW_TILE = TILE_M * Raw<T>::RS, RAW_STAGE = 2 * RAW_TILE;
    static constexpr int BARS = 8 * PAIRS + 2 * (RSTAGES + NB);
    static constexpr int HEAD = (BARS * 8 + 16 + (kMaxSeg + 1) * 4 + 8 + kLocalItems * (int)sizeof(Item) + 127) / 128 * 128;
    static constexpr int LOW = (HEAD + SCL * 2 * TILE_M * 4 + 1023) / 1024 * 1024;  // where the B ring starts
    static constexpr int MINS = T == T_Q4_K ? PWARPS * 32 * 8 * 10 : 0;  // 8 + 2 bytes per block and producer thread
    static constexpr int TAIL = RSTAGES * RAW_STAGE + MINS;
};

template <int T, bool PAIR>  // PAIR: both tiles from seg.wa (256 rows, fp32 results); else gate and up rows, silu(g) * u
__global__ void __launch_bounds__(NTHREADS, 1) grouped_tc_kernel(const Args A) {
    using L = Layout<T>;
    using R = Raw<T>;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* base = smem_raw + ((1024u - (s32(smem_raw) & 1023u)) & 1023u);
    uint64_t* full = reinterpret_cast<uint64_t*>(base);  // [tile][PAIRS] A and the lo rows of B, [PAIRS] the hi rows
    uint64_t* empty = full + 4 * PAIRS;                  // [tile][PAIRS] the lo rows of B, [PAIRS] A and the hi rows
    uint64_t* rfull = empty + 4 * PAIRS;
    uint64_t* rempty = rfull + L::RSTAGES;
    uint64_t* tfull = rempty + L::RSTAGES;
    uint64_t* tfree = tfull + NB;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfree + NB);
    int* pre = reinterpret_cast<int*>(tmem_slot + 4);  // [nseg + 1] first token tile of a segment
    Item* itab = reinterpret_cast<Item*>((reinterpret_cast<uintptr_t>(pre + kMaxSeg + 1) + 7) & ~(uintptr_t)7);
    float* scl = reinterpret_cast<float*>(base + L::HEAD);  // [SCL][2][128]
    uint8_t* b_ring = base + L::LOW;
    uint8_t* p = b_ring + B_BYTES;
    uint8_t* book = p;
    if constexpr (T == T_IQ3_XXS) {
        book += (kMmBookAlign - (s32(p) & (kMmBookAlign - 1))) & (kMmBookAlign - 1);
        p = book + sizeof(MmCodebook);
    }
    uint8_t* raw_base = p;
    if ((uint32_t)(raw_base + L::TAIL - smem_raw) > A.smem) {  // only if shared memory starts elsewhere than the context was told
        if (threadIdx.x == 0) status_set(A.status, 26);
        return;
    }

    // The warp's number, told to be the same for its lanes: what depends on it leaves the 64 registers a thread.
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int nblk = A.n_in / 256;
    const int row_tiles = A.n_out / (PAIR ? 2 * TILE_M : TILE_M);
    const int pitch = row_pitch(A.n_in), scale_col = A.n_in + x_cols(A.n_in);

    if (tid == 0) {
        for (int i = 0; i < 4 * PAIRS; ++i) {
            mb_init(&full[i], (i & PAIRS ? 0 : PWARPS / 2) + BWARPS / 2 * 32);  // a tile's producers, and the lanes of two B warps
            mb_init(&empty[i], 1);                                              // a commit
        }
        for (int i = 0; i < L::RSTAGES; ++i) { mb_init(&rfull[i], RWARPS * 32); mb_init(&rempty[i], PWARPS); }
        for (int i = 0; i < NB; ++i) { mb_init(&tfull[i], 2); mb_init(&tfree[i], EWARPS); }
        fence_mbarrier_init();
    }
    if constexpr (T == T_IQ3_XXS) {
        for (int i = tid; i < (int)(sizeof(MmCodebook) / 16); i += NTHREADS)
            cp_async16<false>(book + 16 * i, reinterpret_cast<const uint8_t*>(&g_mm_codebook) + 16 * i);
        cp_async_commit();
        cp_async_wait_all();
    }
    if (warp == W_MMA) tmem_alloc<TMEM_COLS>(tmem_slot);
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
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    const int n_items = nseg > 0 ? pre[nseg] * row_tiles : 0;
    // The segments come by descending tokens, but for the shared expert's, which is the last: the largest has to be dealt first, not into the
    // last round of items.
    const int first = nseg > 1 && A.seg[nseg - 1].m > A.seg[0].m ? pre[nseg - 1] : 0;
    const int GR = gridDim.x;
    // Items are dealt round by round, the last round backwards, so that the CTAs that get one more are those that had the smaller ones: 1.4 % of
    // the passes below.  (Beyond the table, where a round is one of forty, straight on: what it took to know the last one there cost registers and
    // more than it gave, Q4_K 383 -> 412 us.)
    const int last = (n_items + GR - 1) / GR - 1, tail = last * GR + GR - 1 - (int)blockIdx.x;
    const bool back = last < kLocalItems;
    const int my_items = back ? last + (tail < n_items ? 1 : 0) : (n_items - (int)blockIdx.x + GR - 1) / GR;
    if (tid < min(my_items, kLocalItems)) itab[tid] = decode_item<PAIR>(back && tid == last ? tail : (int)blockIdx.x + tid * GR, row_tiles, A.rb, nseg, first, pre, A.seg);
    __syncthreads();
    auto item = [&](int k) {
        return k < kLocalItems ? itab[k] : decode_item<PAIR>((int)blockIdx.x + k * GR, row_tiles, A.rb, nseg, first, pre, A.seg);
    };
    bool ok = true;

    if (warp < EWARPS) {
        // ---------------- epilogue: TMEM lane = weight row ----------------
        reg_inc<REG_EPI>();
        const int quad = warp & 3, hsel = warp >> 2;
        const int r = quad * 32 + lane;
        const uint32_t tlane = tmem_base + ((uint32_t)(quad * 32) << 16);
        int buf = 0, sc = 0;
        uint32_t pb = 0;
        auto row_scale = [&](int k) {  // lane j: what undoes the scaling of token j of this warp's half (asked for an item ahead)
            const Item it = item(k);
            const int half = tile_tokens(it.m) >> 1, pr = it.prow + min(hsel * half + min(lane, half - 1), it.m - 1);
            const int orow = A.row_token ? A.row_token[pr] : pr;
            return *reinterpret_cast<const float*>(A.op + (size_t)(2 * orow) * pitch + scale_col);
        };
        float rs_next = my_items > 0 ? row_scale(0) : 0.f;
#pragma unroll 1
        for (int k = 0; k < my_items && ok; ++k) {
            const Item it = item(k);
            const int nte = tile_tokens(it.m), half = nte >> 1;
            const float rs = rs_next;
            rs_next = k + 1 < my_items ? row_scale(k + 1) : 0.f;
            float acc[2][NT / 2];  // the tile's first or second half of the tokens
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int j = 0; j < NT / 2; ++j) acc[mt][j] = 0.f;
#pragma unroll 1
            for (int b0 = 0; b0 < nblk && ok; b0 += 8) {
                const int bn = min(8, nblk - b0);
#pragma unroll 1
                for (int b = 0; b < bn + (T == T_Q4_K ? 1 : 0); ++b) {  // the last one: the mins
                    ok = warp_all(mb_wait(&tfull[buf], pb, A.status, 3));
                    if (!ok) break;
                    tc_fence_after();
                    const float s[2] = {scl[(sc * 2) * TILE_M + r], scl[(sc * 2 + 1) * TILE_M + r]};
                    sc = (sc + 1) & (SCL - 1);
                    const uint32_t col = tlane + (uint32_t)(buf * BUF_COLS + hsel * half);
                    auto sums = [&](auto at, auto width) {  // of `width` tokens; the last of them hand the buffer back before the arithmetic
                        constexpr int O = decltype(at)::value, W = decltype(width)::value;
                        uint32_t v[2][W];
                        tmem_ld(col + O, v[0]);
                        tmem_ld(col + NT + O, v[1]);
                        tmem_ld_wait();
                        if (O + W >= half) {
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mb_arrive(&tfree[buf]);
                        }
#pragma unroll
                        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                            for (int j = 0; j < W; ++j) acc[mt][O + j] = fmaf(s[mt], __uint_as_float(v[mt][j]), acc[mt][O + j]);
                    };
                    if (half == 8) sums(Int<0>(), Int<8>()); else sums(Int<0>(), Int<16>());
                    if (half == 24) sums(Int<16>(), Int<8>()); else if (half == 32) sums(Int<16>(), Int<16>());
                    if (++buf == NB) { buf = 0; pb ^= 1u; }
                }
            }
            if (!ok) break;
            const int t0 = hsel * half, cnt = min(half, it.m - t0);
            float* o = A.out + (size_t)(it.prow + t0) * A.n_out + it.r0 + r;
#pragma unroll
            for (int j0 = 0; j0 < NT / 2; j0 += 8) {
                if (j0 >= cnt) break;
#pragma unroll
                for (int j = j0; j < j0 + 8; ++j) {  // eight results first (independent chains), then the stores
                    const float f = __shfl_sync(0xffffffffu, rs, j);
                    acc[0][j] *= f;
                    acc[1][j] *= f;
                    if constexpr (!PAIR) acc[0][j] = swiglu_fast(acc[0][j], acc[1][j]);
                }
                if (PAIR && A.row_dst) {  // expert parallel: the owner's (token, slot) row
#pragma unroll
                    for (int j = j0; j < j0 + 8; ++j)
                        if (j < cnt) {
                            float* d = A.row_dst[it.prow + t0 + j] + it.r0 + r;
                            d[0] = acc[0][j];
                            d[TILE_M] = acc[1][j];
                        }
                } else {
#pragma unroll
                    for (int j = j0; j < j0 + 8; ++j, o += A.n_out)
                        if (j < cnt) {
                            o[0] = acc[0][j];
                            if constexpr (PAIR) o[TILE_M] = acc[1][j];
                        }
                }
            }
        }
    } else if (warp < W_RAW) {
        // ---------------- producers ----------------
        reg_dec<REG_PROD>();
        const int pw = warp - EWARPS, odd = pw >> 3, tile = (pw >> 2) & 1, r = (pw & 3) * 32 + lane;
        const uint32_t tlane = tmem_base + A_COL0 + (uint32_t)(tile * A_COLS) + ((uint32_t)((pw & 3) * 32) << 16);
        const uint32_t gl = s32(book) + 8 * (lane & (kLutRep - 1)), sl = s32(book) + (uint32_t)sizeof(uint2) * 256 * kLutRep + 4 * lane;
        uint2* mm = reinterpret_cast<uint2*>(raw_base + L::RSTAGES * L::RAW_STAGE) + pw * 32 + lane;
        uint16_t* dd = reinterpret_cast<uint16_t*>(raw_base + L::RSTAGES * L::RAW_STAGE + PWARPS * 32 * 8 * 8) + pw * 32 + lane;
        int rst = 0, sc = 0;
        uint32_t rph = 0u;
        uint32_t turn = ~0u;  // parities of the pairs
        auto claim = [&](int h) {  // slot odd + 2 h
            ok = warp_all(mb_wait(&empty[(2 * tile + 1) * PAIRS + h], (turn >> h) & 1u, A.status, 2));
            turn ^= 1u << h;
        };
        auto hand_over = [&](const uint32_t (&o)[32], int h) {
            claim(h);
            if (!ok) return;
            tc_fence_after();
            tmem_st32(tlane + (odd + 2 * h) * (2 * A_COLS), o);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mb_arrive(&full[2 * tile * PAIRS + h]);
        };
#pragma unroll 1
        for (int k = 0; k < my_items && ok; ++k) {
            const Item it = item(k);
            uint32_t off = 0;  // where the row's block starts within 16 bytes
            if constexpr (T == T_IQ3_XXS) off = (uint32_t)(uintptr_t)(tile ? it.pb : it.pa) + (uint32_t)r * A.rb;
#pragma unroll 1
            for (int b0 = 0; b0 < nblk && ok; b0 += 8) {
                const int bn = min(8, nblk - b0);
                uint32_t top = 0u;  // bits of the largest |dmin|, in the upper half
#pragma unroll 1
                for (int b = 0; b < bn; ++b) {
                    ok = warp_all(mb_wait(&rfull[rst], rph, A.status, 7));
                    if (!ok) break;
                    const uint8_t* raw = raw_base + rst * L::RAW_STAGE + tile * L::RAW_TILE + r * R::RS + (off & 15u);
                    if constexpr (T == T_IQ3_XXS) off += kBB<T>;
#pragma unroll 1
                    for (int h = 0; h < 2; ++h) {
                        R in;
                        in.load(raw, odd + 2 * h);
                        if (h == 0) {
                            if (!odd) {
                                scl[(sc * 2 + tile) * TILE_M + r] = in.scale();
                                sc = (sc + 1) & (SCL - 1);
                            }
                            if constexpr (T == T_Q4_K) {
                                top = max(top, in.h.x & 0x7fff0000u);
                                mm[b * PWARPS * 32] = make_uint2(in.h.z, in.h.w);
                                dd[b * PWARPS * 32] = (uint16_t)(in.h.x >> 16);
                            }
                        } else {
                            __syncwarp();
                            if (lane == 0) mb_arrive(&rempty[rst]);
                            if (++rst == L::RSTAGES) { rst = 0; rph ^= 1u; }
                        }
                        uint32_t o[32];
                        decode_stage(in, odd + 2 * h, o, gl, sl);
                        hand_over(o, h);
                        if (!ok) break;
                    }
                    if (!ok) break;
                }
                if (!ok) break;
                if constexpr (T == T_Q4_K) {
                    if (odd < min_stages<T>(bn)) {
                        // e = top >> 26, the exponent field of the largest |dmin| < 2^(e - 14): times 2^(24 - e) (2^15 at most) it is below
                        // 2^10, and dmin * m <= 63 * dmin below fp16's largest number
                        const uint32_t ex = min(30u, 39u - (top >> 26));
                        if (!odd) {
                            scl[(sc * 2 + tile) * TILE_M + r] = __uint_as_float((142u - ex) << 23);  // 2^-(ex - 15): undoes the scale
                            sc = (sc + 1) & (SCL - 1);
                        }
                        uint32_t o[32];
                        mins_stage(mm, dd, bn, odd, ex, o);
                        hand_over(o, 0);
                    } else {
                        claim(0);
                        if (ok && lane == 0) mb_arrive(&full[2 * tile * PAIRS]);
                    }
                }
            }
        }
    } else {
        reg_dec<REG_COPY>();  // one instruction for both warpgroups, above the roles: all warps of a warpgroup execute the same setmaxnreg
        if (warp < W_B) {
        // ---------------- raw rows, a tile per warp: lane = unit lane % 8 of row lane / 8 (+ 4 per step); Q4_K: the ninth units afterwards ----------------
        const int rw = warp - W_RAW, c16 = (lane & 7) * 16;
        int rst = 0;
        uint32_t rph = 1u;
#pragma unroll 1
        for (int k = 0; k < my_items && ok; ++k) {
            const Item it = item(k);
            const uint8_t* tile = rw ? it.pb : it.pa;
#pragma unroll 1
            for (int b0 = 0; b0 < nblk && ok; b0 += 8) {
                const int bn = min(8, nblk - b0);
#pragma unroll 1
                for (int b = 0; b < bn; ++b) {
                    ok = warp_all(mb_wait(&rempty[rst], rph, A.status, 8));
                    if (!ok) break;
                    uint8_t* dst = raw_base + rst * L::RAW_STAGE + (rw ? L::RAW_TILE : 0);
                    const uint32_t step = 4u * A.rb;
                    const uint8_t* src = tile + (size_t)(lane >> 3) * A.rb + (size_t)(b0 + b) * kBB<T>;
                    uint8_t* d = dst + (lane >> 3) * R::RS + c16;
#pragma unroll
                    for (int i = 0; i < TILE_M / 4; ++i, src += step) {
                        if constexpr (T == T_Q4_K) {
                            cp_async16(d + i * 4 * R::RS, src + c16);
                        } else {
                            const uint8_t* s16 = reinterpret_cast<const uint8_t*>((uintptr_t)src & ~(uintptr_t)15);
                            if (c16 < R::UNITS * 16) cp_async16(d + i * 4 * R::RS, s16 + c16);
                        }
                    }
                    if constexpr (T == T_Q4_K) {
                        const uint8_t* s9 = tile + (size_t)lane * A.rb + (size_t)(b0 + b) * kBB<T> + 128;
#pragma unroll
                        for (int i = 0; i < TILE_M / 32; ++i) cp_async16(dst + (lane + 32 * i) * R::RS + 128, s9 + (size_t)(32 * i) * A.rb);
                    }
                    cp_async_arrive(&rfull[rst]);
                    if (++rst == L::RSTAGES) { rst = 0; rph ^= 1u; }
                }
            }
        }
        cp_async_wait_all();
        } else if (warp < W_MMA) {
        // ---------------- B tiles: two warps the tokens' lo rows, two the hi rows; lane = unit lane % 8 of row lane / 8 (+ 8 per step, the
        // half's other warp takes the four between) ----------------
        const int hi = (warp - W_B) >> 1, brow = 4 * ((warp - W_B) & 1) + (lane >> 3);
        const uint32_t at = hi * SLOTS * B_SLOT + chunk_off(brow, lane & 7);  // rows r and r + 8 swizzle alike
        uint32_t turn = ~0u;  // parities of the pairs
#pragma unroll 1
        for (int k = 0; k < my_items && ok; ++k) {
            const Item it = item(k);
            const int steps = (it.m - 4 * ((warp - W_B) & 1) + 7) >> 3;  // columns of B behind the item's tokens may hold anything: nobody reads their sums
            uint32_t src[NT / 8];  // operand array rows of this lane's B rows, in 16-byte units
#pragma unroll
            for (int i = 0; i < NT / 8; ++i) {
                const int pr = it.prow + min(8 * i + brow, it.m - 1);
                const uint32_t orow = i < steps ? (uint32_t)(A.row_token ? A.row_token[pr] : pr) : 0u;
                src[i] = (2u * orow + 1u - hi) * (uint32_t)(pitch >> 3) + (lane & 7);
            }
            auto pair = [&](int off, int h, int stages, int next) {  // off: elements from the row's start; next: from one stage to the other
                const uint32_t t = (turn >> h) & 1u;
                ok = warp_all(mb_wait(&empty[hi * PAIRS + h], t, A.status, 4) && mb_wait(&empty[(2 + hi) * PAIRS + h], t, A.status, 4));
                if (!ok) return;
                turn ^= 1u << h;
                uint8_t* d = b_ring + 2 * h * B_SLOT + at;
                const uint16_t* from = A.op + off;
#pragma unroll
                for (int i = 0; i < NT / 8; ++i)
                    if (i < steps) {
                        const uint16_t* row = from + (size_t)src[i] * 8;
                        cp_async16(d + i * 1024, row);
                        if (stages > 1) cp_async16(d + B_SLOT + i * 1024, row + next);
                    }
                cp_async_arrive(&full[hi * PAIRS + h]);
                cp_async_arrive(&full[(2 + hi) * PAIRS + h]);
            };
#pragma unroll 1
            for (int b0 = 0; b0 < nblk && ok; b0 += 8) {
                const int bn = min(8, nblk - b0);
#pragma unroll 1
                for (int b = 0; b < bn && ok; ++b) {
#pragma unroll 1
                    for (int h = 0; h < PAIRS && ok; ++h) pair((b0 + b) * 256 + h * 2 * BK, h, 2, BK);
                }
                if (T == T_Q4_K && ok) pair(A.n_in + 8 * b0, 0, min_stages<T>(bn), 0);  // the mins read the sums behind the row
            }
        }
        cp_async_wait_all();
        } else if (elect_one()) {
            // ---------------- MMA issue: a thread per tile ----------------
            const int tile = warp - W_MMA;
            const uint32_t b_lo0 = desc_lo(s32(b_ring)), d0 = tmem_base + (uint32_t)(tile * NT), ta0 = tmem_base + A_COL0 + (uint32_t)(tile * A_COLS);
            uint32_t turn = 0u;  // parities
            uint64_t *fu = full + tile * 2 * PAIRS, *em = empty + tile * 2 * PAIRS;
            int buf = 0;
            uint32_t pf = 1u;
#pragma unroll 1
            for (int k = 0; k < my_items && ok; ++k) {
                const uint32_t idesc = (1u << 4) | ((uint32_t)(tile_tokens(item(k).m) >> 3) << 17) | ((uint32_t)(TILE_M >> 4) << 24);  // fp16 x fp16 -> fp32
                auto begin = [&]() { return mb_wait(&tfree[buf], pf, A.status, 6); };
                auto end = [&]() {
                    mma_commit(&tfull[buf]);
                    if (++buf == NB) { buf = 0; pf ^= 1u; }
                };
                // two stages against the lo (p < PAIRS) or hi rows; acc: of the first K step
                auto pair = [&](int p, uint32_t acc, auto mins, int steps, int hop) {
                    ok = mb_wait(&fu[p], (turn >> p) & 1u, A.status, 5);
                    if (!ok) return;
                    turn ^= 1u << p;
                    tc_fence_after();    // A: written to tensor memory by the producers
                    fence_async_smem();  // B: written to shared memory by the B warps' copies
                    const uint32_t d = d0 + (uint32_t)(buf * BUF_COLS);
                    const uint32_t ta = ta0 + (uint32_t)((p % PAIRS) * 4 * A_COLS), b_lo = b_lo0 + (uint32_t)(p * (2 * B_SLOT >> 4));
                    if constexpr (!decltype(mins)::value) {
#pragma unroll
                        for (int ks = 0; ks < 8; ++ks)
                            mma_f16_ta(d, ta + (uint32_t)(ks >> 2) * 2 * A_COLS + 8u * (ks & 3), desc_of(b_lo + (uint32_t)(ks >> 2) * (B_SLOT >> 4) + 2u * (ks & 3)), idesc,
                                       ks == 0 ? acc : 1u);
                    } else {  // `steps` K steps of hi mins, then of lo mins: `hop` further on
#pragma unroll 1
                        for (int i = 0; i < 2 * steps; ++i) {
                            const int ks = i < steps ? i : hop + i - steps;
                            mma_f16_ta(d, ta + (uint32_t)(ks >> 2) * 2 * A_COLS + 8u * (ks & 3), desc_of(b_lo + (uint32_t)(ks >> 2) * (B_SLOT >> 4) + 2u * (ks & 3)), idesc,
                                       i == 0 ? acc : 1u);
                        }
                    }
                    mma_commit(&em[p]);
                };
#pragma unroll 1
                for (int b0 = 0; b0 < nblk && ok; b0 += 8) {
                    const int bn = min(8, nblk - b0);
#pragma unroll 1
                    for (int b = 0; b < bn && ok; ++b) {
                        ok = begin();
                        if (!ok) break;
                        // everything against the lo rows, then against the hi rows: the hi sums are rounded as often as alone
#pragma unroll 1
                        for (int p = 0; p < 2 * PAIRS && ok; ++p)
                            pair(p, p ? 1u : 0u, Int<0>(), 0, 0);
                        if (ok) end();
                    }
                    if (T != T_Q4_K || !ok) continue;
                    // The mins: K steps without sub-blocks are left out (hi and lo side by side when both fit into one stage).
                    const int steps = (bn * 8 + 15) / 16, hop = min_stages<T>(bn) == 1 ? 2 : 4;
                    ok = begin();
                    if (ok) pair(0, 0u, Int<1>(), steps, hop);
                    if (ok) pair(PAIRS, 1u, Int<1>(), steps, hop);
                    if (ok) end();
                }
            }
        }
        __syncwarp();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == W_MMA) {
        tc_fence_after();
        tmem_free<TMEM_COLS>(tmem_base);
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

size_t tc_row_pitch(int n_in) { return (size_t)tg::row_pitch(n_in); }

int launch_operand_rows(dnb_ctx* c, cudaStream_t st, int type, const float* x, int ldx, int rows, int n_in, uint16_t* op, const char* name,
                        const int32_t* rows_dev) {
    if (n_in % 256 || ldx % 4) return DNB_DECLINED;
    ProfScope prof_(c, st, name);
    auto kern = type == T_Q4_K ? tg::operand_rows_kernel<T_Q4_K> : tg::operand_rows_kernel<T_IQ3_XXS>;
    DNB_CUDA(launch_k(kern, dim3((rows + 7) / 8), dim3(256), 0, st, c->use_pdl, x, ldx, rows, rows_dev, n_in, tg::row_pitch(n_in), op));
    c->launches++;
    return DNB_OK;
}

bool tc_handles(const dnb_ctx* c, int type, int n_in, int n_out, bool fused) {
    return c->smem_base > 0 && (type == T_Q4_K || type == T_IQ3_XXS) && n_in % 256 == 0 && n_out % (fused ? tg::TILE_M : 2 * tg::TILE_M) == 0;
}

template <int T, bool PAIR>
static int launch_tc_t(dnb_ctx* c, cudaStream_t st, tg::Args& A) {
    using L = tg::Layout<T>;
    const size_t base = c->smem_base;  // the parts are on 1 KB and 32 KB boundaries of the address space, wherever the CTA's part of it starts
    size_t at = (base + 1023) / 1024 * 1024 + L::LOW + tg::B_BYTES;
    if (T == T_IQ3_XXS) at = (at + kMmBookAlign - 1) / kMmBookAlign * kMmBookAlign + sizeof(MmCodebook);
    const size_t smem = at + L::TAIL - base;
    static_assert(L::BARS * 8 + 16 + (tg::kMaxSeg + 1) * 4 + 8 + tg::kLocalItems * sizeof(tg::Item) <= L::HEAD, "head too small");
    A.smem = (uint32_t)smem;
    auto kern = tg::grouped_tc_kernel<T, PAIR>;
    static SmemGrant grant;
    DNB_CUDA(grant_smem(grant, c->device, kern, smem));
    ProfScope prof_(c, st, PAIR ? "tc_down" : "tc_gate_up");
    DNB_CUDA(launch_k(kern, dim3(c->sm_count), dim3(tg::NTHREADS), smem, st, c->use_pdl, A));
    c->launches++;
    return DNB_OK;
}

int launch_grouped_tc(dnb_ctx* c, cudaStream_t st, int type, bool fused, const SegDesc* seg, const int32_t* nseg_dev, int nseg_max, int n_in,
                      int n_out, const uint16_t* op, const int32_t* row_token, float* out, float* const* row_dst) {
    if (!tc_handles(c, type, n_in, n_out, fused) || nseg_max > tg::kMaxSeg) return DNB_DECLINED;
    int rc = type == T_IQ3_XXS ? upload_mm_tables(c->device) : DNB_OK;
    if (rc) return rc;
    tg::Args A = {};
    A.seg = seg; A.nseg_dev = nseg_dev; A.nseg_max = nseg_max; A.n_in = n_in; A.n_out = n_out; A.rb = (int)row_bytes(type, n_in);
    A.op = op; A.row_token = row_token; A.out = out; A.row_dst = row_dst; A.status = c->status;
    if (type == T_Q4_K) return fused ? launch_tc_t<T_Q4_K, false>(c, st, A) : launch_tc_t<T_Q4_K, true>(c, st, A);
    return fused ? launch_tc_t<T_IQ3_XXS, false>(c, st, A) : launch_tc_t<T_IQ3_XXS, true>(c, st, A);
}

}  // namespace dnb
