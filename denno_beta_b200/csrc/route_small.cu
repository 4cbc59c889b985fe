// Routing of a decode batch (2-15 tokens) in two launches: RMSNorm + router logits, then softmax / top-k / renorm and the
// expert-major tables.  cuda.rs:48695 pf_router_dev_topk and moe_expert.rs:8309-8390 build_grouped_batch of the reference; values,
// selections and tables are those of the general kernels (moe_kernels.cu), operation for operation.
//
// What bounds it: latencies.  As four kernels (RMSNorm, logits by 16 CTAs, a CTA per token, a CTA per eight experts) the routing of
// eight tokens took 34 us of a 109 us layer, most of it launches, cold first loads and half-empty chips; the 4 MB of router rows are
// 0.7 us.  Here a warp holds its router row in registers before it waits for the kernel in front, and the tables are built where the
// selections are: a layer of eight tokens 109 -> 96 us.
#include <algorithm>

#include "dnb_common.cuh"
#include "route_topk.cuh"
#include "tc_ptx.cuh"

namespace dnb {

constexpr int kRsTok = 15;      // tokens at most (from 16 the tensor-core router takes over)
constexpr int kRsGroup = 4;     // tokens of a 128-thread group of the logits kernel at once
constexpr int kRsPass = 2 * kRsGroup;

// Barrier of 128-thread group g of a CTA (named barriers 1..8).
struct GroupSync {
    int id;
    __device__ __forceinline__ void operator()() const { asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory"); }
};

// CTA of 256 threads = four router rows; group g of 128 threads serves tokens g * kRsGroup .. of a pass of kRsPass, so that a thread
// computes the sums that prep_kernel's and router_logits_kernel's thread of the same number computes.  NV = n_embd / 128: float4 words
// of a row per lane, held in registers (the two groups' loads of a row meet in L1).
template <int NV>
__global__ void __launch_bounds__(256)
router_batch_kernel(const float* __restrict__ h, const float* __restrict__ norm_w, float eps, int nt, int e, const float* __restrict__ w_r,
                    const float* __restrict__ bias, int ne, float* __restrict__ xn, float* __restrict__ logits) {
    extern __shared__ __align__(16) float smem[];  // [kRsPass][e]
    __shared__ float red[kRsPass][4];
    const int tid = threadIdx.x & 127, grp = threadIdx.x >> 7, lane = tid & 31, warp = tid >> 5;
    const int row = blockIdx.x * 4 + warp;
    const GroupSync sync{1 + grp};
    float* xs = smem + (size_t)grp * kRsGroup * e;
    float4 wv[NV];
    const float4* wr = reinterpret_cast<const float4*>(w_r + (size_t)min(row, ne - 1) * e);
#pragma unroll
    for (int j = 0; j < NV; ++j) wv[j] = __ldg(wr + lane + 32 * j);
    pdl_wait();
    pdl_launch_dependents();
    for (int t0 = grp * kRsGroup; t0 < nt; t0 += kRsPass) {
        const int n = min(kRsGroup, nt - t0);
        sync();  // the pass before has been read
        for (int i = tid; i < n * (e >> 2); i += 128) tcp::cp_async16<false>(xs + 4 * i, h + (size_t)t0 * e + 4 * i);
        tcp::cp_async_commit();
        tcp::cp_async_wait_all();
        sync();
        if (norm_w) {
            // rms_inv_128's sum: thread v adds x[v]^2, x[v + 128]^2, ... by fma, a 32-lane xor tree, (w0 + w1) + (w2 + w3)
            float ss[kRsGroup];
#pragma unroll
            for (int q = 0; q < kRsGroup; ++q) ss[q] = 0.f;
#pragma unroll 4
            for (int i = tid; i < e; i += 128) {
#pragma unroll
                for (int q = 0; q < kRsGroup; ++q)
                    if (q < n) ss[q] = fmaf(xs[q * e + i], xs[q * e + i], ss[q]);
            }
#pragma unroll
            for (int q = 0; q < kRsGroup; ++q) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) ss[q] += __shfl_xor_sync(0xffffffffu, ss[q], o);
                if (lane == 0) red[grp * kRsGroup + q][warp] = ss[q];
            }
            sync();
#pragma unroll
            for (int q = 0; q < kRsGroup; ++q) {
                const float* r = red[grp * kRsGroup + q];
                ss[q] = 1.0f / sqrtf(((r[0] + r[1]) + (r[2] + r[3])) / (float)e + eps);
            }
#pragma unroll 4
            for (int i = tid; i < e; i += 128) {
                const float nw = __ldg(norm_w + i);
#pragma unroll
                for (int q = 0; q < kRsGroup; ++q) {
                    if (q < n) {
                        const float v = __fmul_rn(__fmul_rn(xs[q * e + i], ss[q]), nw);
                        xs[q * e + i] = v;
                        if ((int)blockIdx.x == t0 + q) xn[(size_t)(t0 + q) * e + i] = v;  // CTA t publishes token t
                    }
                }
            }
            sync();
        }
        float acc[kRsGroup];
#pragma unroll
        for (int q = 0; q < kRsGroup; ++q) acc[q] = 0.f;
#pragma unroll
        for (int j = 0; j < NV; ++j) {
#pragma unroll
            for (int q = 0; q < kRsGroup; ++q) {
                if (q < n) {
                    const float4 xv = reinterpret_cast<const float4*>(xs + (size_t)q * e)[lane + 32 * j];
                    acc[q] = fmaf(wv[j].x, xv.x, acc[q]);
                    acc[q] = fmaf(wv[j].y, xv.y, acc[q]);
                    acc[q] = fmaf(wv[j].z, xv.z, acc[q]);
                    acc[q] = fmaf(wv[j].w, xv.w, acc[q]);
                }
            }
        }
        const float b = bias && row < ne ? bias[row] : 0.f;
#pragma unroll
        for (int q = 0; q < kRsGroup; ++q) {
            if (q < n) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
                if (lane == 0 && row < ne) logits[(size_t)(t0 + q) * ne + row] = bias ? acc[q] + b : acc[q];
            }
        }
    }
}

struct TableArgs {
    const float* logits;      // null: the selections are given in sels
    int nt, k, ne, norm_topk;
    int32_t* sels;
    float* wts;
    const uint8_t *gate, *up, *down, *sg, *su, *sdn;
    size_t eb_g, eb_u, eb_d;
    SegDesc *seg_gu, *seg_dn;
    int32_t *row_token, *pos, *nseg;
};

// One CTA: a group of 128 threads per token (in turn from the ninth on), then the tables: segments by token count descending, ties
// by expert ascending, the rows of an expert in ascending token order; the shared expert last.
__global__ void __launch_bounds__(1024) topk_tables_kernel(const TableArgs A) {
    extern __shared__ __align__(16) uint8_t sm[];
    RouteSmem* R = reinterpret_cast<RouteSmem*>(sm);                       // [8] groups (only with logits)
    __shared__ int sel[kRsTok * 32];
    __shared__ float wt[8][32];
    __shared__ uint32_t tok[1024];                                         // tokens of an expert, a bit each
    __shared__ int active[kRsTok * 32], first[kRsTok * 32];                // the active experts in ascending order, their first rows
    __shared__ __align__(16) int key[kRsTok * 32 + 4];
    __shared__ int wsum[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, grp = tid >> 7;
    tok[tid] = 0u;
    pdl_wait();
    pdl_launch_dependents();
    const int pairs = A.nt * A.k;
    if (A.logits) {
        for (int t = grp; t < A.nt; t += 8) {
            const GroupSync sync{1 + grp};
            route_topk(R[grp], A.logits + (size_t)t * A.ne, A.ne, A.k, A.norm_topk, wt[grp], tid & 127, sync);
            sync();
            if ((tid & 127) < A.k) {
                const int i = t * A.k + (tid & 127);
                const int ex = R[grp].ssel[tid & 127];
                sel[i] = ex;
                A.sels[i] = ex;
                A.wts[i] = wt[grp][tid & 127];
            }
            sync();
        }
    } else if (tid < pairs) {
        sel[tid] = A.sels[tid];
    }
    __syncthreads();
    if (tid < pairs) {
        const int ex = sel[tid];
        if (ex >= 0 && ex < A.ne) atomicOr(&tok[ex], 1u << (tid / A.k));
    }
    __syncthreads();
    // active experts in ascending order
    const bool on = tid < A.ne && tok[tid] != 0u;
    const uint32_t bal = __ballot_sync(0xffffffffu, on);
    if (lane == 0) wsum[warp] = __popc(bal);
    __syncthreads();
    const int before = __reduce_add_sync(0xffffffffu, lane < warp ? wsum[lane] : 0), n_active = __reduce_add_sync(0xffffffffu, wsum[lane]);
    // An expert's key: larger = earlier among the segments (more tokens, then the lower index).
    if (on) {
        const int a = before + __popc(bal & ((1u << lane) - 1u));
        active[a] = tid;
        key[a] = __popc(tok[tid]) << 10 | (1023 - a);
    }
    if (tid < 4) key[n_active + tid] = 0;  // (read in fours)
    __syncthreads();
    if (tid < n_active) {
        const int ex = active[tid], mine = key[tid], c = mine >> 10;
        int rank = 0, row = 0;
        for (int o = 0; o < n_active; o += 4) {
            const int4 k4 = *reinterpret_cast<const int4*>(key + o);
            rank += (k4.x > mine) + (k4.y > mine) + (k4.z > mine) + (k4.w > mine);
            row += (k4.x > mine ? k4.x >> 10 : 0) + (k4.y > mine ? k4.y >> 10 : 0) + (k4.z > mine ? k4.z >> 10 : 0) + (k4.w > mine ? k4.w >> 10 : 0);
        }
        A.seg_gu[rank] = SegDesc{A.gate + (size_t)ex * A.eb_g, A.up + (size_t)ex * A.eb_u, (uint32_t)c, (uint32_t)row};
        A.seg_dn[rank] = SegDesc{A.down + (size_t)ex * A.eb_d, nullptr, (uint32_t)c, (uint32_t)row};
        first[tid] = row;
        uint32_t w = tok[ex];
        for (int at = row; w; ++at) {
            A.row_token[at] = __ffs((int)w) - 1;
            w &= w - 1u;
        }
    }
    __syncthreads();
    if (tid < pairs) {
        const int ex = sel[tid], t = tid / A.k;
        if (ex >= 0 && ex < A.ne) {
            int lo = 0, hi = n_active;  // active[lo] == ex
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (active[mid] <= ex) lo = mid; else hi = mid;
            }
            A.pos[tid] = first[lo] + __popc(tok[ex] & ((1u << t) - 1u));
        }
    }
    if (A.sg && tid < A.nt) A.row_token[pairs + tid] = tid;
    if (tid == 0) {
        if (A.sg) {
            A.seg_gu[n_active] = SegDesc{A.sg, A.su, (uint32_t)A.nt, (uint32_t)pairs};
            A.seg_dn[n_active] = SegDesc{A.sdn, nullptr, (uint32_t)A.nt, (uint32_t)pairs};
        }
        *A.nseg = n_active + (A.sg ? 1 : 0);
    }
}

bool route_small_handles(int nt, int e, int ne, int k) {
    return nt >= 1 && nt <= kRsTok && ne <= 1024 && k <= 32 && (e == 512 || e == 1024 || e == 2048 || e == 2560 || e == 4096);
}

template <int NV>
static int launch_router_batch_t(dnb_ctx* c, cudaStream_t st, const float* h, int nt, const Model& M, const Layer& L, Workspace& w) {
    const size_t smem = (size_t)std::min(nt, kRsPass) * M.e * sizeof(float);
    auto kern = router_batch_kernel<NV>;
    static SmemGrant grant;
    DNB_CUDA(grant_smem(grant, c->device, kern, smem));
    ProfScope prof_(c, st, "router_batch");
    DNB_CUDA(launch_k(kern, dim3((M.ne + 3) / 4), dim3(256), smem, st, c->use_pdl, h, (const float*)L.norm_w, M.eps, nt, M.e, (const float*)L.router_w,
                      (const float*)L.router_bias, M.ne, w.xn, w.logits));
    c->launches++;
    return DNB_OK;
}

// RMSNorm (w.xn, when the layer has a norm) and router logits (w.logits) of a decode batch.  DNB_DECLINED: shape not covered.
int launch_router_batch(dnb_ctx* c, cudaStream_t st, const float* h, int nt, const Model& M, const Layer& L, Workspace& w) {
    // CTA t publishes token t, so there have to be as many CTAs as tokens
    if (!route_small_handles(nt, M.e, M.ne, M.k) || (M.ne + 3) / 4 < nt || (((uintptr_t)h) & 15)) return DNB_DECLINED;
    switch (M.e / 128) {
        case 4: return launch_router_batch_t<4>(c, st, h, nt, M, L, w);
        case 8: return launch_router_batch_t<8>(c, st, h, nt, M, L, w);
        case 16: return launch_router_batch_t<16>(c, st, h, nt, M, L, w);
        case 20: return launch_router_batch_t<20>(c, st, h, nt, M, L, w);
        default: return launch_router_batch_t<32>(c, st, h, nt, M, L, w);
    }
}

// Top-k of w.logits (logits = false: the selections are in `sels` already) and the tables of the batch.
int launch_topk_tables(dnb_ctx* c, cudaStream_t st, bool logits, int nt, int k, int ne, int norm_topk, int32_t* sels, float* wts, const Layer& L,
                       Workspace& w, bool fold_shared) {
    if (nt < 1 || nt > kRsTok || ne > 1024 || k < 1 || k > 32) return DNB_DECLINED;
    TableArgs A = {};
    A.logits = logits ? w.logits : nullptr;
    A.nt = nt; A.k = k; A.ne = ne; A.norm_topk = norm_topk; A.sels = sels; A.wts = wts;
    A.gate = L.m[0].dev; A.up = L.m[1].dev; A.down = L.m[2].dev;
    A.eb_g = L.m[0].expert_bytes; A.eb_u = L.m[1].expert_bytes; A.eb_d = L.m[2].expert_bytes;
    A.sg = fold_shared ? L.m[3].dev : nullptr; A.su = fold_shared ? L.m[4].dev : nullptr; A.sdn = fold_shared ? L.m[5].dev : nullptr;
    A.seg_gu = w.seg_gu; A.seg_dn = w.seg_dn; A.row_token = w.row_token; A.pos = w.pos; A.nseg = w.nseg;
    const size_t smem = logits ? 8 * sizeof(RouteSmem) : 0;
    static SmemGrant grant;
    DNB_CUDA(grant_smem(grant, c->device, topk_tables_kernel, smem));
    ProfScope prof_(c, st, "topk_tables");
    DNB_CUDA(launch_k(topk_tables_kernel, dim3(1), dim3(1024), smem, st, c->use_pdl, A));
    c->launches++;
    return DNB_OK;
}

}  // namespace dnb
