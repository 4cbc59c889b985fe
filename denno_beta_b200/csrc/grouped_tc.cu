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
// more block of K = sub-blocks: A = -(dmin * m) as fp16 hi and lo, times a power of two of the row's own that fits its largest
// dmin into fp16's range whatever its size, B = X.  An activation is fp16 hi + lo (22 bits) of the row times a power of two that
// puts its largest element into [512, 1024).
//
// What bounds it: a 64-element stage of two 128-row tiles is about 900 warp instructions of decoding (Q4_K; 1.7 per weight) on
// four schedulers and 8 MMAs of N = 2 x tokens, the same order of time at 32 tokens; everything else has to stay out of the
// way of both.  Shared memory is the tightest: with A tiles in it (32 KB written and 32 KB read per stage, B read once per tile) a
// stage took 840 cycles, all of them shared-memory bandwidth.  So A goes from the producers' registers to tensor memory
// (tcgen05.st, thread = row = lane) and the MMA takes it from there.  One role per warp, each with a ring of its own in front:
//   * four warps copy packed rows (a 256-element block of all 256 rows: 9 or 7 neighbouring lanes per row) into a raw ring.  (A
//     thread that fetches its own row's bytes touches 32 cache lines per instruction; that alone took 0.5 us per stage.)
//   * two warps copy the tokens' hi and lo rows into swizzled B tiles, a stage each in turn, gathered from the token-major rows:
//     no packed copy of the activations.  (TMA row gathers took 80 cycles per four rows; a proxy fence in the copying warp
//     waits for the copies still on their way, so it is the MMA thread that executes it.)
//   * four groups of four producer warps, (even or odd stages) x (tile), a thread one row: decodes 64 weights into registers, THEN
//     waits for a ring slot (tensor memory holds only four stages; with the decoding inside its turn-around a stage took 1,100
//     cycles) and stores them.  The block's scales go to a small ring, its mins to shared memory of the thread's own.
//     A stage has one full barrier for both operands, on which producers and B copies arrive (a second wait a stage: 2 to 3 % more time).
//   * one MMA thread; hi and lo rows of a token are neighbours in the B tile (N = 2 x tokens) and in TMEM, so a weight tile is read
//     once per K step.
//   * eight epilogue warps, two accumulator buffers (thread = weight row, half of the token columns of both tiles).
// Persistent, one CTA per SM; items (segment, 32- or 64-token tile, 128 rows x 2) dealt round-robin.
//
// Measured, 512 tokens of 2048 x 512, top 10 of 512 under a skewed router, us gate/up + down as bracketed by events: Q4_K 175 + 84 (three
// bf16 products, a seventh of the accuracy) -> 122 + 83, IQ3_XXS 343 + 180 -> 122 + 73.  A stage takes about 950 cycles: the issuing thread's waits, fence, issue and
// commit; without the decoding a copy of the kernel was only 7 % faster.
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
constexpr int A_COLS = BK / 2;          // tensor-memory columns of an A tile (two fp16 each)
constexpr int EWARPS = 8, PWARPS = 16, RWARPS = 4, BWARPS = 2;
constexpr int W_RAW = EWARPS + PWARPS, W_B = W_RAW + RWARPS, W_MMA = W_B + BWARPS;
constexpr int NTHREADS = 1024;          // 32 warps, the last one idle
// What depends on the tokens of an item.  64 tokens a weight tile halve the decoding of an expert with many, but there is room for one
// accumulator buffer only (the tensor core waits while a block's sums are read) and for four B tiles instead of eight.
template <int NT> struct Tok {
    static constexpr int B_STAGE = 2 * NT * BK * 2;  // hi and lo rows: 8 or 16 KB
    static constexpr int NB = 64 / NT;               // accumulator buffers
    static constexpr int BUF_COLS = 2 * 2 * NT;      // two tiles x (hi, lo) x tokens
    static constexpr int BSLOTS = 256 / NT;          // ring of B in shared memory (its copies take over a microsecond)
    // Registers per thread of the warpgroups once their roles are known; launched with 64, and no more than that in sum.
    static constexpr int REG_EPI = NT == 64 ? 112 : 96, REG_PROD = NT == 64 ? 56 : 64, REG_RAW = 24, REG_MISC = 40;
    static_assert(2 * REG_EPI + 4 * REG_PROD + REG_RAW + REG_MISC <= 8 * 64, "register split");
};
constexpr int B_BYTES = 65536;          // of the B ring
static_assert(EWARPS == 8 && PWARPS == 16 && RWARPS == 4 && W_MMA == 30, "roles fill warpgroups");
constexpr int kMaxSeg = 1055;
constexpr int kLocalItems = 40;
constexpr int STAGES = 4, BSTAGES = 2 * STAGES;  // ring of A (tensor memory); barriers of a stage, which is known by its number mod BSTAGES
constexpr int A_COL0 = 256, TMEM_COLS = A_COL0 + STAGES * 2 * A_COLS;
static_assert(Tok<32>::NB * Tok<32>::BUF_COLS == A_COL0 && Tok<64>::NB * Tok<64>::BUF_COLS == A_COL0, "accumulators");
static_assert(Tok<32>::BSLOTS * Tok<32>::B_STAGE == B_BYTES && Tok<64>::BSLOTS * Tok<64>::B_STAGE == B_BYTES, "B ring");
static_assert(Tok<32>::BSLOTS == BSTAGES && Tok<64>::BSLOTS == STAGES, "a B slot is freed by the stage BSTAGES or STAGES earlier");
static_assert(TMEM_COLS == 512, "tensor memory");
constexpr int SCL = 8;                  // ring of block scales (the mins count as a block): producers are at most five blocks ahead of the epilogue

template <int T> constexpr int kBB = T == T_Q4_K ? 144 : 98;

struct Item {
    const uint8_t* pa;  // tile 0, first row
    const uint8_t* pb;  // tile 1
    int prow, m;        // first packed row, tokens
    int r0, pad;        // first output row
};

template <bool PAIR, int NT>
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

// Tokens of the B tile: the smallest of 8, 16, 32, 64 that holds the item.
__device__ __forceinline__ int tile_tokens(int m) { return m <= 8 ? 8 : m <= 16 ? 16 : m <= 32 ? 32 : 64; }

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
    __device__ __forceinline__ float scale() const { return h2f((uint16_t)h.x); }
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
    s.s0 = h2sub(__byte_perm(sc, 0x64646464u, 0x4040u), 0x64006400u);
    s.s1 = h2sub(__byte_perm(sc, 0x64646464u, 0x4141u), 0x64006400u);
    s.k0 = h2mul(s.s0, 0xE400E400u);
    s.k1 = h2mul(s.s1, 0xD400D400u);
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
            iq3_pairs_h(gl, sl, iw, q == 0 ? aux << 6 : aux >> (7 * q - 6), p);
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
    static constexpr int BARS = 2 * BSTAGES + 2 * (RSTAGES + 2);
    static constexpr int HEAD = (BARS * 8 + 16 + (kMaxSeg + 1) * 4 + 8 + kLocalItems * (int)sizeof(Item) + 127) / 128 * 128;
    static constexpr int LOW = (HEAD + SCL * 2 * TILE_M * 4 + 1023) / 1024 * 1024;  // where the B ring starts
    static constexpr int MINS = T == T_Q4_K ? PWARPS * 32 * 8 * 10 : 0;  // 8 + 2 bytes per block and producer thread
    static constexpr int TAIL = RSTAGES * RAW_STAGE + MINS;
};

// A stage number as its user sees it.  A group's stages are up to six apart and the groups may be a block apart from one another:
// with one `empty` barrier per slot a group could look at a slot whose last but one stage is still in use and take its parity for
// the last one's.  Stage n therefore commits to barrier n mod 2 * STAGES, and its slot's next user waits for exactly that commit.
struct StageCount {
    int q;          // stage number mod 2 * STAGES
    uint32_t turn;  // parity of its turn
    __device__ __forceinline__ explicit StageCount(int first) : q(first), turn(0u) {}
    __device__ __forceinline__ void advance(int n) {
        q += n;
        if (q >= 2 * STAGES) { q -= 2 * STAGES; turn ^= 1u; }
    }
    __device__ __forceinline__ int slot() const { return q & (STAGES - 1); }
    __device__ __forceinline__ bool wait(uint64_t* empty, int* status, int code) const {  // the stage STAGES earlier is done with its slot
        return q < STAGES ? mb_wait(&empty[q + STAGES], turn ^ 1u, status, code) : mb_wait(&empty[q - STAGES], turn, status, code);
    }
};

template <int T, bool PAIR, int NT>  // NT: tokens of an item; PAIR: both tiles from seg.wa (256 rows, fp32 results); else gate and up rows, silu(g) * u
__global__ void __launch_bounds__(NTHREADS, 1) grouped_tc_kernel(const Args A) {
    using L = Layout<T>;
    using R = Raw<T>;
    using K = Tok<NT>;
    constexpr int NB = K::NB, BUF_COLS = K::BUF_COLS, B_STAGE = K::B_STAGE;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* base = smem_raw + ((1024u - (s32(smem_raw) & 1023u)) & 1023u);
    uint64_t* full = reinterpret_cast<uint64_t*>(base);
    uint64_t* empty = full + BSTAGES;         // both: one per B slot, two per A slot
    uint64_t* rfull = empty + BSTAGES;
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
    if ((uint32_t)(raw_base + L::TAIL - smem_raw) > A.smem) {  // only if shared memory started elsewhere
        if (threadIdx.x == 0) status_set(A.status, 26);
        return;
    }

    // The warp's number, told to be the same for its lanes: what depends on it leaves the 64 registers a thread.  Spills in bytes, stores +
    // loads: Q4_K 48 + 88 -> 0 at 32 tokens, 112 + 148 -> 72 + 68 at 64; IQ3_XXS at 64 64 + 100 -> 36 + 28.  us gate/up + down, 64 experts top 10,
    // 1024 tokens evenly routed: Q4_K at 64 166 + 106 -> 145 + 103, IQ3_XXS 160 + 97 -> 150 + 97.  IQ3_XXS down at 32 never spilled and loses:
    // 128 -> 135.
    constexpr bool kUniform = !(T == T_IQ3_XXS && PAIR && NT == 32);
    const int tid = threadIdx.x, warp = kUniform ? __shfl_sync(0xffffffffu, tid >> 5, 0) : tid >> 5, lane = tid & 31;
    const int nblk = A.n_in / 256;
    const int row_tiles = A.n_out / (PAIR ? 2 * TILE_M : TILE_M);
    const int pitch = row_pitch(A.n_in), scale_col = A.n_in + x_cols(A.n_in);

    if (tid == 0) {
        for (int i = 0; i < BSTAGES; ++i) mb_init(&full[i], 8 + BWARPS * 32);  // two producer groups' warps, a tile each, and the B warps' lanes
        for (int i = 0; i < BSTAGES; ++i) mb_init(&empty[i], 1);               // a commit
        for (int i = 0; i < L::RSTAGES; ++i) { mb_init(&rfull[i], RWARPS * 32); mb_init(&rempty[i], PWARPS); }
        for (int i = 0; i < NB; ++i) { mb_init(&tfull[i], 1); mb_init(&tfree[i], EWARPS); }
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
    const uint32_t tmem_base = *tmem_slot;
    const int n_items = nseg > 0 ? pre[nseg] * row_tiles : 0;
    const int GR = gridDim.x;
    const int my_items = (int)blockIdx.x < n_items ? (n_items - (int)blockIdx.x + GR - 1) / GR : 0;
    if (tid < min(my_items, kLocalItems)) itab[tid] = decode_item<PAIR, NT>((int)blockIdx.x + tid * GR, row_tiles, A.rb, nseg, pre, A.seg);
    __syncthreads();
    auto item = [&](int k) {
        return k < kLocalItems ? itab[k] : decode_item<PAIR, NT>((int)blockIdx.x + k * GR, row_tiles, A.rb, nseg, pre, A.seg);
    };
    bool ok = true;

    if (warp < EWARPS) {
        // ---------------- epilogue: TMEM lane = weight row ----------------
        reg_inc<K::REG_EPI>();
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
        for (int k = 0; k < my_items && ok; ++k) {
            const Item it = item(k);
            const int nte = tile_tokens(it.m), half = nte >> 1;
            const float rs = rs_next;
            rs_next = k + 1 < my_items ? row_scale(k + 1) : 0.f;
            float acc[2][NT / 2];
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int j = 0; j < NT / 2; ++j) acc[mt][j] = 0.f;
            for (int b0 = 0; b0 < nblk && ok; b0 += 8) {
                const int bn = min(8, nblk - b0);
                for (int b = 0; b < bn + (T == T_Q4_K ? 1 : 0); ++b) {  // the last one: the mins
                    ok = warp_all(mb_wait(&tfull[buf], pb, A.status, 3));
                    if (!ok) break;
                    tc_fence_after();
                    const float s[2] = {scl[(sc * 2) * TILE_M + r], scl[(sc * 2 + 1) * TILE_M + r]};
                    sc = (sc + 1) & (SCL - 1);
                    const uint32_t col = tlane + (uint32_t)(buf * BUF_COLS + hsel * nte);
#pragma unroll
                    for (int h = 0; h < NT / 16; ++h) {  // eight tokens a load; a warp has half of the tile's
                        if (h == 0 || 16 * h < nte) {
                            uint32_t v[2][16];
                            tmem_ld16(col + 16 * h, v[0]);
                            tmem_ld16(col + 2 * NT + 16 * h, v[1]);
                            tmem_ld_wait();
                            if (16 * h + 16 >= nte) {  // read: hand the buffer back before the arithmetic
                                tc_fence_before();
                                __syncwarp();
                                if (lane == 0) mb_arrive(&tfree[buf]);
                            }
#pragma unroll
                            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                                for (int j = 0; j < 8; ++j)
                                    acc[mt][8 * h + j] =
                                        fmaf(s[mt], __uint_as_float(v[mt][2 * j]) + __uint_as_float(v[mt][2 * j + 1]), acc[mt][8 * h + j]);
                        }
                    }
                    if (++buf == NB) { buf = 0; pb ^= 1u; }
                }
            }
            if (!ok) break;
            const int t0 = hsel * half, cnt = min(half, it.m - t0);
            float* o = A.out + (size_t)(it.prow + t0) * A.n_out + it.r0 + r;
#pragma unroll
            for (int j = 0; j < NT / 2; ++j) {  // all results first (independent chains), then the stores
                const float f = __shfl_sync(0xffffffffu, rs, j);
                acc[0][j] *= f;
                acc[1][j] *= f;
                if constexpr (!PAIR) acc[0][j] = swiglu_fast(acc[0][j], acc[1][j]);
            }
            if (PAIR && A.row_dst) {  // expert parallel: the owner's (token, slot) row
#pragma unroll
                for (int j = 0; j < NT / 2; ++j)
                    if (j < cnt) {
                        float* d = A.row_dst[it.prow + t0 + j] + it.r0 + r;
                        d[0] = acc[0][j];
                        d[TILE_M] = acc[1][j];
                    }
            } else {
#pragma unroll
                for (int j = 0; j < NT / 2; ++j, o += A.n_out)
                    if (j < cnt) {
                        o[0] = acc[0][j];
                        if constexpr (PAIR) o[TILE_M] = acc[1][j];
                    }
            }
        }
    } else if (warp < W_RAW) {
        // ---------------- producers ----------------
        reg_dec<K::REG_PROD>();
        const int pw = warp - EWARPS, odd = pw >> 3, tile = (pw >> 2) & 1, r = (pw & 3) * 32 + lane;
        const uint32_t tlane = tmem_base + A_COL0 + (uint32_t)(tile * A_COLS) + ((uint32_t)((pw & 3) * 32) << 16);
        const uint32_t gl = s32(book) + 8 * (lane & (kLutRep - 1)), sl = s32(book) + (uint32_t)sizeof(uint2) * 256 * kLutRep + 4 * (lane & (kLutRep - 1));
        uint2* mm = reinterpret_cast<uint2*>(raw_base + L::RSTAGES * L::RAW_STAGE) + pw * 32 + lane;
        uint16_t* dd = reinterpret_cast<uint16_t*>(raw_base + L::RSTAGES * L::RAW_STAGE + PWARPS * 32 * 8 * 8) + pw * 32 + lane;
        int rst = 0, sc = 0;
        uint32_t rph = 0u;
        StageCount q(odd);
        auto hand_over = [&](const uint32_t (&o)[32]) {  // into the ring slot of stage q
            ok = warp_all(q.wait(empty, A.status, 2));
            if (!ok) return;
            tc_fence_after();
            tmem_st32(tlane + q.slot() * (2 * A_COLS), o);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mb_arrive(&full[q.q]);
        };
        for (int k = 0; k < my_items && ok; ++k) {
            const Item it = item(k);
            uint32_t off = 0;  // where the row's block starts within 16 bytes
            if constexpr (T == T_IQ3_XXS) off = (uint32_t)(uintptr_t)(tile ? it.pb : it.pa) + (uint32_t)r * A.rb;
            for (int b0 = 0; b0 < nblk && ok; b0 += 8) {
                const int bn = min(8, nblk - b0);
                uint32_t top = 0u;  // bits of the largest |dmin|, in the upper half
                for (int b = 0; b < bn; ++b) {
                    ok = warp_all(mb_wait(&rfull[rst], rph, A.status, 7));
                    if (!ok) break;
                    const uint8_t* raw = raw_base + rst * L::RAW_STAGE + tile * L::RAW_TILE + r * R::RS + (off & 15u);
                    if constexpr (T == T_IQ3_XXS) off += kBB<T>;
#pragma unroll
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
                        hand_over(o);
                        if (!ok) break;
                        q.advance(2);
                    }
                    if (!ok) break;
                }
                if (!ok) break;
                if constexpr (T == T_Q4_K) {
                    const int nm = min_stages<T>(bn);
                    if (odd < nm) {
                        // e = top >> 26, the exponent field of the largest |dmin| < 2^(e - 14): times 2^(24 - e) (2^15 at most) it is below
                        // 2^10, and dmin * m <= 63 * dmin below fp16's largest number
                        const uint32_t ex = min(30u, 39u - (top >> 26));
                        if (!odd) {
                            scl[(sc * 2 + tile) * TILE_M + r] = __uint_as_float((142u - ex) << 23);  // 2^-(ex - 15): undoes the scale
                            sc = (sc + 1) & (SCL - 1);
                        }
                        uint32_t o[32];
                        mins_stage(mm, dd, bn, odd, ex, o);
                        hand_over(o);
                    }
                    q.advance(nm);
                }
            }
        }
    } else if (warp < W_B) {
        reg_dec<K::REG_RAW>();
        // ---------------- raw rows: lane = unit lane % 8 of row lane / 8 (+ 4 per step); Q4_K: the ninth units afterwards ----------------
        const int rw = warp - W_RAW, c16 = (lane & 7) * 16, row0 = (rw & 1) * (TILE_M / 2);  // half a tile per warp
        int rst = 0;
        uint32_t rph = 1u;
        for (int k = 0; k < my_items && ok; ++k) {
            const Item it = item(k);
            const uint8_t* half = ((rw & 2) ? it.pb : it.pa) + (size_t)row0 * A.rb;
            for (int b0 = 0; b0 < nblk && ok; b0 += 8) {
                const int bn = min(8, nblk - b0);
                for (int b = 0; b < bn; ++b) {
                    ok = warp_all(mb_wait(&rempty[rst], rph, A.status, 8));
                    if (!ok) break;
                    uint8_t* dst = raw_base + rst * L::RAW_STAGE + ((rw & 2) ? L::RAW_TILE : 0) + row0 * R::RS;
                    const uint32_t step = 4u * A.rb;
                    const uint8_t* src = half + (size_t)(lane >> 3) * A.rb + (size_t)(b0 + b) * kBB<T>;
                    uint8_t* d = dst + (lane >> 3) * R::RS + c16;
#pragma unroll
                    for (int i = 0; i < TILE_M / 8; ++i, src += step) {
                        if constexpr (T == T_Q4_K) {
                            cp_async16(d + i * 4 * R::RS, src + c16);
                        } else {
                            const uint8_t* s16 = reinterpret_cast<const uint8_t*>((uintptr_t)src & ~(uintptr_t)15);
                            if (c16 < R::UNITS * 16) cp_async16(d + i * 4 * R::RS, s16 + c16);
                        }
                    }
                    if constexpr (T == T_Q4_K) {
                        const uint8_t* s9 = half + (size_t)lane * A.rb + (size_t)(b0 + b) * kBB<T> + 128;
#pragma unroll
                        for (int i = 0; i < TILE_M / 64; ++i) cp_async16(dst + (lane + 32 * i) * R::RS + 128, s9 + (size_t)(32 * i) * A.rb);
                    }
                    cp_async_arrive(&rfull[rst]);
                    if (++rst == L::RSTAGES) { rst = 0; rph ^= 1u; }
                }
            }
        }
        cp_async_wait_all();
    } else {
        reg_dec<K::REG_MISC>();
        if (warp < W_MMA) {
        // ---------------- B tiles: rows 2 t, 2 t + 1 = hi and lo of token t; lane = unit lane % 8 of row lane / 8 (+ 8 per step, the
        // other warp takes the four between) ----------------
        StageCount q(0);
        const int brow = 4 * (warp - W_B) + (lane >> 3);
        const uint32_t at = chunk_off(brow, lane & 7);  // rows r and r + 8 swizzle alike
        for (int k = 0; k < my_items && ok; ++k) {
            const Item it = item(k);
            const int steps = tile_tokens(it.m) / 4;  // 8 rows each
            uint32_t src[NT / 4];  // operand array rows of this lane's B rows, in 16-byte units
#pragma unroll
            for (int i = 0; i < NT / 4; ++i) {
                const int br = 8 * i + brow, pr = it.prow + min(br >> 1, it.m - 1);
                const uint32_t orow = i < steps ? (uint32_t)(A.row_token ? A.row_token[pr] : pr) : 0u;
                src[i] = (2u * orow + (br & 1)) * (uint32_t)(pitch >> 3) + (lane & 7);
            }
            auto stage = [&](int off) {  // off: elements from the row's start
                ok = warp_all(NT == 64 ? q.wait(empty, A.status, 4) : mb_wait(&empty[q.q], q.turn ^ 1u, A.status, 4));
                if (!ok) return;
                uint8_t* d = b_ring + (NT == 64 ? q.slot() : q.q) * B_STAGE + at;
                const uint16_t* from = A.op + off;
#pragma unroll
                for (int i = 0; i < NT / 4; ++i)
                    if (i < steps) cp_async16(d + i * 1024, from + (size_t)src[i] * 8);
                cp_async_arrive(&full[q.q]);
                q.advance(1);
            };
            for (int b0 = 0; b0 < nblk && ok; b0 += 8) {
                const int bn = min(8, nblk - b0);
                for (int b = 0; b < bn && ok; ++b) {
#pragma unroll 1
                    for (int c = 0; c < 4 && ok; ++c) stage((b0 + b) * 256 + c * BK);
                }
                const int sums = A.n_in + 8 * b0;  // the mins read the sums behind the row
                for (int u = 0; u < min_stages<T>(bn) && ok; ++u) stage(sums);
            }
        }
        cp_async_wait_all();
        } else if (warp == W_MMA && elect_one()) {
            // ---------------- MMA issue: one thread ----------------
            const uint32_t b_lo0 = desc_lo(s32(b_ring));
            StageCount q(0);
            int buf = 0;
            uint32_t pf = 1u;
            for (int k = 0; k < my_items && ok; ++k) {
                const int nte = tile_tokens(item(k).m);
                const uint32_t idesc = (1u << 4) | ((uint32_t)((2 * nte) >> 3) << 17) | ((uint32_t)(TILE_M >> 4) << 24);  // fp16 x fp16 -> fp32
                for (int b0 = 0; b0 < nblk && ok; b0 += 8) {
                    const int bn = min(8, nblk - b0);
                    for (int b = 0; b < bn + (T == T_Q4_K ? 1 : 0) && ok; ++b) {
                        // a block's four stages; or those of the mins, whose K steps without sub-blocks are left out (hi and lo side
                        // by side when both fit into one stage)
                        const bool mins = b == bn, pair = mins && bn <= 4;
                        const int stages = mins ? min_stages<T>(bn) : 4, live = mins ? (bn * 8 + 15) / 16 : 4;
                        ok = mb_wait(&tfree[buf], pf, A.status, 6);
                        const uint32_t d = tmem_base + (uint32_t)(buf * BUF_COLS);
                        for (int c = 0; c < stages && ok; ++c) {
                            ok = mb_wait(&full[q.q], q.turn, A.status, 5);
                            if (!ok) break;
                            tc_fence_after();    // A: written to tensor memory by the producers
                            fence_async_smem();  // B: written to shared memory by the B warps' copies
                            const uint32_t ta = tmem_base + A_COL0 + (uint32_t)(q.slot() * 2 * A_COLS), b_lo = b_lo0 + (uint32_t)((NT == 64 ? q.slot() : q.q) * (B_STAGE >> 4));
                            uint32_t acc = c == 0 ? 0u : 1u;
#pragma unroll
                            for (int ks = 0; ks < 4; ++ks) {
                                if ((pair ? ks & 1 : ks) >= live) continue;
                                mma_f16_ta(d, ta + 8u * ks, desc_of(b_lo + 2u * ks), idesc, acc);
                                mma_f16_ta(d + 2 * NT, ta + A_COLS + 8u * ks, desc_of(b_lo + 2u * ks), idesc, acc);
                                acc = 1u;
                            }
                            mma_commit(&empty[q.q]);
                            q.advance(1);
                        }
                        if (!ok) break;
                        mma_commit(&tfull[buf]);
                        if (++buf == NB) { buf = 0; pf ^= 1u; }
                    }
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

bool tc_handles(int type, int n_in, int n_out, bool fused) {
    return (type == T_Q4_K || type == T_IQ3_XXS) && n_in % 256 == 0 && n_out % (fused ? tg::TILE_M : 2 * tg::TILE_M) == 0;
}

template <int T, bool PAIR, int NT>
static int launch_tc_t(dnb_ctx* c, cudaStream_t st, tg::Args& A) {
    using L = tg::Layout<T>;
    size_t at = kMmSmemBase + L::LOW + tg::B_BYTES;
    if (T == T_IQ3_XXS) at = (at + kMmBookAlign - 1) / kMmBookAlign * kMmBookAlign + sizeof(MmCodebook);
    const size_t smem = at + L::TAIL - kMmSmemBase;
    static_assert(L::BARS * 8 + 16 + (tg::kMaxSeg + 1) * 4 + 8 + tg::kLocalItems * sizeof(tg::Item) <= L::HEAD, "head too small");
    A.smem = (uint32_t)smem;
    auto kern = tg::grouped_tc_kernel<T, PAIR, NT>;
    static SmemGrant grant;
    DNB_CUDA(grant_smem(grant, c->device, kern, smem));
    ProfScope prof_(c, st, PAIR ? "tc_down" : "tc_gate_up");
    DNB_CUDA(launch_k(kern, dim3(c->sm_count), dim3(tg::NTHREADS), smem, st, c->use_pdl, A));
    c->launches++;
    return DNB_OK;
}

int launch_grouped_tc(dnb_ctx* c, cudaStream_t st, int type, bool fused, const SegDesc* seg, const int32_t* nseg_dev, int nseg_max, int n_in,
                      int n_out, const uint16_t* op, const int32_t* row_token, float* out, float* const* row_dst, int tokens, int rows) {
    if (!tc_handles(type, n_in, n_out, fused) || nseg_max > tg::kMaxSeg) return DNB_DECLINED;
    int rc = type == T_IQ3_XXS ? upload_mm_tables(c->device) : DNB_OK;
    if (rc) return rc;
    tg::Args A = {};
    A.seg = seg; A.nseg_dev = nseg_dev; A.nseg_max = nseg_max; A.n_in = n_in; A.n_out = n_out; A.rb = (int)row_bytes(type, n_in);
    A.op = op; A.row_token = row_token; A.out = out; A.row_dst = row_dst; A.status = c->status;
    // Items of 64 tokens, or of 32.  Where no expert has more than 32 tokens, 64 save no decoding and cost a second accumulator and half of
    // the B ring: 11 to 14 % of a layer (Q4_K), 5 to 8 % (IQ3_XXS); where experts have more, they gain up to 30 %.  That depends on how the
    // tokens spread, which the host does not know.  With 40 rows a segment (IQ3_XXS: 24) 64 are the better choice either way; with fewer Q4_K
    // stays at 32, while IQ3_XXS, which loses little where 64 do not help, takes them from 256 tokens on.  us a layer, 32 / 64 tokens an
    // item, even routing, and skewed by -1.1 ln rank, 2048 x 512:
    //   Q4_K, 512 experts top 10: 512 tokens (11 rows a segment) 431 / 493, 248 / 238; 1024 tokens (22) 490 / 558, 416 / 364
    //         128 experts top 8: 384 tokens (27) 163 / 190, 181 / 179; 512 (36) 210 / 205, 211 / 197; 700 (49) 270 / 220, 256 / 238
    //         64 experts top 10: 200 tokens (34) 139 / 132, 144 / 156; 1024 (173) 381 / 315, 381 / 317
    //   IQ3_XXS, 512 experts top 10: 200 tokens 438 / 474, 166 / 151; 256 tokens 440 / 477, 176 / 160; 512 tokens 479 / 511, 275 / 238
    //         128 experts top 8: 200 tokens (14) 166 / 177, 139 / 144; 384 (27) 179 / 191, 199 / 179; 512 (36) 234 / 201, 233 / 199
    // Over six such shapes and 48 to 1024 tokens the rule is 0.1 % / 1.7 % (Q4_K, even / skewed) and 1.6 % / 1.0 % (IQ3_XXS) behind the better.
    // (Tried: the choice on the device, from the segments' token counts.  Both kernels launched, one without items: 1.5 us each.  One
    // kernel with both bodies, or with items of either size: 7 to 15 % slower, in registers and code.)
    const bool q4 = type == T_Q4_K, wide = rows >= (q4 ? 40 : 24) * nseg_max || (!q4 && tokens >= 256);
#define DNB_TC(TY, PAIR) return wide ? launch_tc_t<TY, PAIR, 64>(c, st, A) : launch_tc_t<TY, PAIR, 32>(c, st, A)
    if (type == T_Q4_K) { if (fused) DNB_TC(T_Q4_K, false); DNB_TC(T_Q4_K, true); }
    if (fused) DNB_TC(T_IQ3_XXS, false);
    DNB_TC(T_IQ3_XXS, true);
#undef DNB_TC
}

}  // namespace dnb
