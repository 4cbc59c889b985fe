// Softmax, top-k and renorm of one token by 128 threads: the routing of every path (tensor.rs:1171-1183; moe.rs:188-279;
// qwen4exp.rs:11802-11821; GPU form kernels_router225.cu:36-171 of the reference).
#pragma once
#include "dnb_common.cuh"

#ifndef DNB_STAMP
#define DNB_STAMP(i) do { } while (0)
#endif

namespace dnb {

constexpr int kFdCand = 64;  // entries the parallel ranking takes

// Shared memory of the routing of one token.
struct RouteSmem {
    float probs[1024];
    uint32_t tmax[128];
    int wcnt[4];
    uint32_t cand_k[kFdCand];
    int cand_x[kFdCand];
    float red[128];
    float cmax[4];
    float bcast;
    float inv;
    int nan_any;
    int total;
    int sel[32];
    float pv[32];
    int ssel[32];
    float spv[32];
};

__device__ __forceinline__ uint32_t order_key(float v) {  // larger float -> larger key; never 0 for a probability
    const uint32_t ub = __float_as_uint(v);
    return (ub & 0x80000000u) ? ~ub : (ub | 0x80000000u);
}

// Softmax, top-k and renorm of one token's logits (global memory) by 128 threads, tid = 0..127; route_sync is their barrier.
// Leaves the selection ascending in R.ssel and the routing weights in wts_s[0..k), which may be read after one more barrier; *rowsum
// takes the sum of the selected probabilities.  nsplit > 1: `logits` points at the first of nsplit partial sums of the row,
// split_stride floats apart (the tensor-core router's K splits), added in ascending order, then the bias: router_reduce_kernel's adds.
//
// Thread v holds entries v, v + 128, ...  Everything that depends on evaluation order is fixed, so a token gets the same bits on
// every path:
//   softmax denominator: per-thread partials in ascending index, then the tree ((s[l]+s[l+64]) + (s[l+32]+s[l+96])) and a
//     32-lane xor tree;
//   selection: the CPU scan's rule (moe.rs:256-279) -- a strictly larger value wins, ties go to the lower index, and a NaN is taken
//     only when it is the first unused entry;
//   renorm: the selected probabilities summed in ascending expert index, one add at a time, as on the CPU.
// Six 128-thread barriers: what could be one warp's work and a broadcast (the sum's tree, the threshold) every warp does for itself.
template <class Sync>
__device__ __forceinline__ void route_topk(RouteSmem& R, const float* __restrict__ logits, int ne, int k, int norm_topk,
                                           float* wts_s, int tid, Sync route_sync, float* rowsum = nullptr, int nsplit = 1,
                                           size_t split_stride = 0, const float* __restrict__ bias = nullptr) {
    const int lane = tid & 31, warp = tid >> 5;
    float p[8];
    float mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int idx = j * 128 + tid;
        p[j] = -INFINITY;
        if (idx < ne) {
            p[j] = __ldcg(logits + idx);  // L2: other CTAs of this launch may have written them
            if (nsplit > 1) {
                float part[kRouterSplitMax];  // all requested before the first is used
#pragma unroll
                for (int s = 1; s < kRouterSplitMax; ++s) part[s] = s < nsplit ? __ldcg(logits + (size_t)s * split_stride + idx) : 0.f;
#pragma unroll
                for (int s = 1; s < kRouterSplitMax; ++s)
                    if (s < nsplit) p[j] = __fadd_rn(p[j], part[s]);
                if (bias) p[j] = __fadd_rn(p[j], bias[idx]);
            }
        }
        mx = fmaxf(mx, p[j]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) R.cmax[warp] = mx;
    if (tid == 0) R.nan_any = 0;
    DNB_STAMP(16);
    route_sync();
    mx = fmaxf(fmaxf(R.cmax[0], R.cmax[1]), fmaxf(R.cmax[2], R.cmax[3]));
    {
        float part = 0.f;
        bool any_nan = false;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (j * 128 + tid < ne) {
                p[j] = expf(p[j] - mx);
                part += p[j];
                any_nan |= (p[j] != p[j]);
            }
        }
        R.red[tid] = part;
        if (any_nan) R.nan_any = 1;
    }
    DNB_STAMP(17);
    route_sync();
    // the tree of topk_block; the xor butterfly leaves the same bits in every lane of every warp
    float sum = (R.red[lane] + R.red[lane + 64]) + (R.red[lane + 32] + R.red[lane + 96]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const bool has_nan = R.nan_any != 0;
    uint32_t key[8];
    uint32_t km = 0u;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int idx = j * 128 + tid;
        key[j] = 0u;
        if (idx < ne) {
            p[j] = sum > 0.f ? p[j] / sum : p[j];
            R.probs[idx] = p[j];
            key[j] = order_key(p[j]);
            km = max(km, key[j]);
        }
    }
    R.tmax[tid] = km;
    DNB_STAMP(18);
    route_sync();
    // ---- selection ----
    // Fast form (no NaN): the entries fall into 32 classes by index mod 32 (= lane); t = the k-th largest
    // of the class maxima.  At least k entries reach t, so every one of the top k does; the entries that
    // reach it (a dozen or two) are ranked among themselves by (value descending, index ascending) -- the
    // CPU scan's rule.
    bool fast = !has_nan && k <= 32;
    int total = 0;
    if (fast) {
        const uint32_t v = max(max(R.tmax[lane], R.tmax[lane + 32]), max(R.tmax[lane + 64], R.tmax[lane + 96]));
        int above = 0;
#pragma unroll
        for (int j = 0; j < 32; ++j) above += (__shfl_sync(0xffffffffu, v, j) > v) ? 1 : 0;
        uint32_t t = __reduce_min_sync(0xffffffffu, (above < k && v != 0u) ? v : 0xffffffffu);
        const int have = __popc(__ballot_sync(0xffffffffu, v != 0u));
        if (have < k) t = 1u;  // fewer maxima than selections: every entry is a candidate
        uint32_t smask = 0u;
#pragma unroll
        for (int j = 0; j < 8; ++j) smask |= (key[j] != 0u && key[j] >= t) ? (1u << j) : 0u;
        const int cnt = __popc(smask);
        int incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        if (lane == 31) R.wcnt[warp] = incl;
        DNB_STAMP(19);
        route_sync();
        int before = incl - cnt;
        for (int w2 = 0; w2 < 4; ++w2) {
            const int c = R.wcnt[w2];
            if (w2 < warp) before += c;
            total += c;
        }
        fast = total >= k && total <= kFdCand;
        if (fast) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if ((smask >> j) & 1u) {
                    R.cand_k[before] = key[j];
                    R.cand_x[before] = j * 128 + tid;
                    ++before;
                }
        }
        DNB_STAMP(20);
        route_sync();
        if (fast && tid < total) {
            const uint32_t ck = R.cand_k[tid];
            const int cx = R.cand_x[tid];
            int rank = 0;
            for (int j = 0; j < total; ++j) {
                const uint32_t ok = R.cand_k[j];
                const int ox = R.cand_x[j];
                rank += (ok > ck || (ok == ck && ox < cx)) ? 1 : 0;
            }
            if (rank < k) {
                R.sel[rank] = cx;
                R.pv[rank] = R.probs[cx];
            }
        }
    }
    if (!fast) {
        // General form, warp 0: k rounds of the CPU scan (moe.rs:256-279) with the entries dealt to
        // the lanes.  A strictly larger value wins, ties go to the lower index, and a NaN is taken
        // only when it is the first unused entry.
        if (warp == 0) {
            uint32_t used = 0u;  // bit m: entry 32 m + lane
#pragma unroll 1
            for (int round = 0; round < k; ++round) {
                float best = -INFINITY;
                int best_i = 0x7fffffff, first = 0x7fffffff;
#pragma unroll 1
                for (int m = 0; 32 * m + lane < ne; ++m) {
                    if ((used >> m) & 1u) continue;
                    const int idx = 32 * m + lane;
                    first = min(first, idx);
                    const float v = R.probs[idx];
                    if (v == v && (best_i == 0x7fffffff || v > best)) {
                        best = v;
                        best_i = idx;
                    }
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
                    const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
                    first = min(first, __shfl_xor_sync(0xffffffffu, first, o));
                    if (oi != 0x7fffffff && (best_i == 0x7fffffff || ov > best || (ov == best && oi < best_i))) {
                        best = ov;
                        best_i = oi;
                    }
                }
                int win = best_i;
                if (has_nan || best_i == 0x7fffffff) {
                    const float fv = first != 0x7fffffff ? R.probs[first] : 0.f;
                    if (fv != fv || best_i == 0x7fffffff) win = first;
                }
                if ((win & 31) == lane) used |= 1u << (win >> 5);
                if (lane == 0) {
                    R.sel[round] = win;
                    R.pv[round] = R.probs[win];
                }
            }
        }
    }
    DNB_STAMP(21);
    route_sync();
    if (tid < k) {
        const int mine = R.sel[tid];
        int rank = 0;
        for (int j = 0; j < k; ++j) rank += (R.sel[j] < mine) ? 1 : 0;
        R.ssel[rank] = mine;
        R.spv[rank] = R.pv[tid];
    }
    route_sync();
    if (tid < k) {
        float s = 0.f;  // the selected probabilities in ascending expert index, one add at a time
        for (int j = 0; j < k; ++j) s = __fadd_rn(s, R.spv[j]);
        float w;
        if (!norm_topk) w = R.spv[tid];
        else if (isfinite(s) && s > 0.f) w = R.spv[tid] / s;
        else w = 1.0f / (float)k;
        wts_s[tid] = w;
        if (rowsum && tid == 0) *rowsum = s;
    }
    DNB_STAMP(22);
}

}  // namespace dnb
