// Hyper-connection mix and combine either side of the MoE block (model/hyper.rs of the reference;
// call sites model/qwen4exp.rs:3722-3765: hc_mix_quant -> moe_ffn_quant -> hc_combine_inplace; GPU forms
// kernels/kernels_mix_*.cu).  A layer carries hc parallel residual streams of n_embd values per token:
//
//   mix      xn[s]    = rmsnorm(res[s]) * w_norm[s]                       per stream (tensor.rs:1125-1135)
//            raw      = w_down_inject @ concat_s xn[s]                    [low_rank + hc] rows of hc*n_embd
//            lo[r]    = silu(raw[r] / hc),  r < low_rank                  silu(v) = v * (1 / (1 + exp(-v)))
//            inject[s] = raw[low_rank + s] / hc                           (no silu)
//            gate     = w_up @ lo                                         [hc*n_embd] rows of low_rank
//            mixed[d] = (1/hc) * sum_s xn[s][d] * sigmoid(gate[s][d])     ascending s, 1/hc after the sum
//   block    = MoE block (mixed)                                          no further norm
//   combine  out[s][d] = res[s][d] + block[d] * (2 * sigmoid(inject[s]))
//
// The order of operations inside an element (division by hc after the matmul, the form of silu, the
// ascending-s sum) follows hyper.rs:13-36, which states it as the numeric contract; the dot products are
// lane-split with a fixed xor tree (deterministic; the CPU's are sequential, so they differ by rounding).
// Weights are kept as fp32 (the checkpoints store them as BF16, whose expansion to fp32 is exact).
#include <algorithm>

#include "dnb_common.cuh"

namespace dnb {

struct HcLayer {
    int hc = 0, low_rank = 0;
    float* w_norm = nullptr;  // [hc][e]
    float* w_down = nullptr;  // [low_rank + hc][hc*e]
    float* w_up = nullptr;    // [hc*e][low_rank]
};
struct HcState {
    std::vector<HcLayer> layers;
    Scratch xn, raw, mixed, blk, res, out;  // device scratch, grow-only
    Scratch host_in, host_out;              // pinned staging of the host-buffer entry point
};

__device__ __forceinline__ float hc_sigmoid(float v) { return 1.0f / (1.0f + expf(-v)); }

// One token's mix is three dependent kernels over 21 MB of fp32 weights, and a call of one token is their latencies: each kernel
// therefore starts while its predecessor still runs (programmatic launch) and holds its first weights in registers before it waits.
// A call of one token (hc 4, n_embd 2048, rank 320, host buffers, the block included): 100 -> 57 us.

// one CTA of 128 threads per (token, stream): the summation tree of rms_inv_128 (moe_kernels.cu).  `res` may be pinned host memory;
// then res_dev (else null) receives a copy for the combine, and the row crosses the bus once.
__global__ void __launch_bounds__(128)
hc_norm_kernel(const float* res, float* res_dev, const float* __restrict__ w_norm, float eps, int hc, int e, float* __restrict__ xn) {
    __shared__ float red[4];
    const int s = blockIdx.x % hc;
    pdl_wait();
    pdl_launch_dependents();
    const float* xr = res + (size_t)blockIdx.x * e;
    if (res_dev) {
        float* rd = res_dev + (size_t)blockIdx.x * e;
        for (int i0 = threadIdx.x; i0 < e; i0 += 128 * 16) {  // sixteen words on their way per thread
            float v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = i0 + 128 * j < e ? __ldcv(xr + i0 + 128 * j) : 0.f;
#pragma unroll
            for (int j = 0; j < 16; ++j)
                if (i0 + 128 * j < e) rd[i0 + 128 * j] = v[j];
        }
        xr = rd;  // a thread reads back what it has written itself
    }
    float ss = 0.f;
    for (int i = threadIdx.x; i < e; i += 128) ss = fmaf(xr[i], xr[i], ss);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    const float inv = 1.0f / sqrtf(((red[0] + red[1]) + (red[2] + red[3])) / (float)e + eps);
    const float* g = w_norm + (size_t)s * e;
    float* o = xn + (size_t)blockIdx.x * e;
    for (int i = threadIdx.x; i < e; i += 128) o[i] = __fmul_rn(__fmul_rn(xr[i], inv), g[i]);
}

// raw[t][r] = w_down[r] . xn[t]; then lo / inject as above.  A CTA per row, its 256 threads split K (a warp per row left 324 warps
// on the chip, each with one load on its way: 27 us for 10.6 MB); up to eight tokens per CTA share the row's weights in registers.
constexpr int kHcDownTok = 8;
__global__ void __launch_bounds__(256)
hc_down_kernel(const float* __restrict__ w_down, const float* __restrict__ xn, int nt, int hc_dim, int low_rank, int hc,
               float* __restrict__ raw) {
    __shared__ float red[8][kHcDownTok];
    const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rows = low_rank + hc, n4 = hc_dim >> 2;
    const int t0 = blockIdx.y * kHcDownTok, ntok = min(kHcDownTok, nt - t0);
    const float4* wr = reinterpret_cast<const float4*>(w_down + (size_t)row * hc_dim);
    float acc[kHcDownTok];
#pragma unroll
    for (int q = 0; q < kHcDownTok; ++q) acc[q] = 0.f;
    for (int base = 0; base < n4; base += 2048) {
        float4 wv[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int i = base + tid + 256 * j;
            wv[j] = i < n4 ? __ldg(wr + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (base == 0) {  // the weights are constants of the layer, xn comes from the kernel before
            pdl_wait();
            pdl_launch_dependents();
        }
#pragma unroll
        for (int q = 0; q < kHcDownTok; ++q) {
            if (q < ntok) {
                const float4* x4 = reinterpret_cast<const float4*>(xn + (size_t)(t0 + q) * hc_dim);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int i = base + tid + 256 * j;
                    if (i < n4) {
                        const float4 xv = x4[i];
                        acc[q] = fmaf(wv[j].x, xv.x, acc[q]);
                        acc[q] = fmaf(wv[j].y, xv.y, acc[q]);
                        acc[q] = fmaf(wv[j].z, xv.z, acc[q]);
                        acc[q] = fmaf(wv[j].w, xv.w, acc[q]);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int q = 0; q < kHcDownTok; ++q) {
        if (q < ntok) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
            if (lane == 0) red[warp][q] = acc[q];
        }
    }
    __syncthreads();
    if (tid < ntok) {
        float a = red[0][tid];
#pragma unroll
        for (int w = 1; w < 8; ++w) a += red[w][tid];
        const float v = __fmul_rn(a, 1.0f / (float)hc);  // 1/hc after the matmul (hyper.rs:21-22)
        raw[(size_t)(t0 + tid) * rows + row] = row < low_rank ? __fmul_rn(v, hc_sigmoid(v)) : v;
    }
}

// gate[s][d] = w_up[s*e + d] . lo[t]; mixed[t][d] = (1/hc) * sum_s xn[t][s][d] * sigmoid(gate[s][d]).  One warp per d.
__global__ void __launch_bounds__(128)
hc_up_mixed_kernel(const float* __restrict__ w_up, const float* __restrict__ raw, const float* __restrict__ xn, int nt, int hc, int e,
                   int low_rank, float* __restrict__ mixed) {
    extern __shared__ float lo[];  // [low_rank] of the CTA's token
    const int t = blockIdx.y;
    const int rows = low_rank + hc;
    for (int i = threadIdx.x; i < low_rank; i += 128) lo[i] = raw[(size_t)t * rows + i];
    __syncthreads();
    const int d = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (d >= e) return;
    const float inv_hc = 1.0f / (float)hc;
    float m = 0.f;
    for (int s = 0; s < hc; ++s) {
        const float* wr = w_up + ((size_t)s * e + d) * low_rank;
        float acc = 0.f;
        for (int i = lane; i < low_rank; i += 32) acc = fmaf(__ldg(wr + i), lo[i], acc);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        const float term = __fmul_rn(xn[((size_t)t * hc + s) * e + d], hc_sigmoid(acc));
        m = s == 0 ? term : __fadd_rn(m, term);
    }
    if (lane == 0) mixed[(size_t)t * e + d] = __fmul_rn(m, inv_hc);
}

// The same for up to HC streams and a rank of at most 128 * N4 (a multiple of 4): a warp's rows of w_up sit in its registers before
// the wait and serve up to eight tokens.
constexpr int kHcUpTok = 8;
template <int HC, int N4>
__global__ void __launch_bounds__(128)
hc_up_mixed_reg_kernel(const float* __restrict__ w_up, const float* __restrict__ raw, const float* __restrict__ xn, int nt, int hc, int e,
                       int low_rank, float* __restrict__ mixed) {
    extern __shared__ __align__(16) float lo[];  // [tokens][low_rank]
    const int t0 = blockIdx.y * kHcUpTok, ntok = min(kHcUpTok, nt - t0), rows = low_rank + hc, r4 = low_rank >> 2;
    const int d = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    float4 wv[HC][N4];
#pragma unroll
    for (int s = 0; s < HC; ++s)
#pragma unroll
        for (int j = 0; j < N4; ++j)
            wv[s][j] = d < e && s < hc && lane + 32 * j < r4 ? __ldg(reinterpret_cast<const float4*>(w_up + ((size_t)s * e + d) * low_rank) + lane + 32 * j)
                                                             : make_float4(0.f, 0.f, 0.f, 0.f);
    pdl_wait();
    pdl_launch_dependents();
    for (int i = threadIdx.x; i < ntok * low_rank; i += 128) {
        const int q = i / low_rank;
        lo[i] = raw[(size_t)(t0 + q) * rows + (i - q * low_rank)];
    }
    __syncthreads();
    if (d >= e) return;
    const float inv_hc = 1.0f / (float)hc;
    for (int q = 0; q < ntok; ++q) {
        const float4* l4 = reinterpret_cast<const float4*>(lo + (size_t)q * low_rank);
        float acc[HC];
#pragma unroll
        for (int s = 0; s < HC; ++s) acc[s] = 0.f;
#pragma unroll
        for (int j = 0; j < N4; ++j) {
            if (lane + 32 * j < r4) {
                const float4 v = l4[lane + 32 * j];
#pragma unroll
                for (int s = 0; s < HC; ++s) {
                    acc[s] = fmaf(wv[s][j].x, v.x, acc[s]);
                    acc[s] = fmaf(wv[s][j].y, v.y, acc[s]);
                    acc[s] = fmaf(wv[s][j].z, v.z, acc[s]);
                    acc[s] = fmaf(wv[s][j].w, v.w, acc[s]);
                }
            }
        }
#pragma unroll
        for (int s = 0; s < HC; ++s)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc[s] += __shfl_xor_sync(0xffffffffu, acc[s], o);
        float m = 0.f;
#pragma unroll
        for (int s = 0; s < HC; ++s) {
            if (s < hc) {
                const float term = __fmul_rn(xn[((size_t)(t0 + q) * hc + s) * e + d], hc_sigmoid(acc[s]));
                m = s == 0 ? term : __fadd_rn(m, term);
            }
        }
        if (lane == 0) mixed[(size_t)(t0 + q) * e + d] = __fmul_rn(m, inv_hc);
    }
}

__global__ void hc_combine_kernel(const float* __restrict__ res, const float* __restrict__ blk, const float* __restrict__ raw, int hc, int e,
                                  int low_rank, float* __restrict__ out) {
    pdl_wait();
    pdl_launch_dependents();
    const int ts = blockIdx.x;  // token * hc + stream
    const int t = ts / hc, s = ts - t * hc;
    const float w = __fmul_rn(2.0f, hc_sigmoid(raw[(size_t)t * (low_rank + hc) + low_rank + s]));
    const float* r = res + (size_t)ts * e;
    const float* b = blk + (size_t)t * e;
    float* o = out + (size_t)ts * e;
    for (int d = threadIdx.x; d < e; d += blockDim.x) o[d] = __fadd_rn(r[d], __fmul_rn(b[d], w));
}

static int hc_grow(Scratch& s, size_t bytes, bool pinned = false) {
    if (bytes <= s.cap) return DNB_OK;
    if (s.p) { if (pinned) cudaFreeHost(s.p); else cudaFree(s.p); }
    s.p = nullptr;
    s.cap = 0;
    if (pinned) DNB_CUDA(cudaMallocHost(&s.p, bytes)); else DNB_CUDA(cudaMalloc(&s.p, bytes));
    s.cap = bytes;
    return DNB_OK;
}

void hc_release(dnb_ctx* c) {
    HcState* h = static_cast<HcState*>(c->hc);
    if (!h) return;
    for (auto& L : h->layers) {
        if (L.w_norm) cudaFree(L.w_norm);
        if (L.w_down) cudaFree(L.w_down);
        if (L.w_up) cudaFree(L.w_up);
    }
    for (Scratch* s : {&h->xn, &h->raw, &h->mixed, &h->blk, &h->res, &h->out})
        if (s->p) cudaFree(s->p);
    if (h->host_in.p) cudaFreeHost(h->host_in.p);
    if (h->host_out.p) cudaFreeHost(h->host_out.p);
    delete h;
    c->hc = nullptr;
}

// Enqueues the whole layer.  res_dev: where a `res` in pinned host memory is copied to on the device, or null.
static int hc_enqueue(dnb_ctx* c, HcState* H, int layer, const float* res, float* res_dev, int nt, float* out) {
    const Model& M = c->model;
    const HcLayer& L = H->layers[layer];
    const int hc = L.hc, lr = L.low_rank, e = M.e, hc_dim = hc * e;
    cudaStream_t st = c->stream;
    int rc;
    float* xn = (float*)H->xn.p;
    float* raw = (float*)H->raw.p;
    float* mixed = (float*)H->mixed.p;
    float* blk = (float*)H->blk.p;
    {
        ProfScope p_(c, st, "hc_norm");
        DNB_CUDA(launch_k(hc_norm_kernel, dim3(nt * hc), dim3(128), 0, st, c->use_pdl, res, res_dev, (const float*)L.w_norm, M.eps, hc, e, xn));
    }
    {
        ProfScope p_(c, st, "hc_down");
        DNB_CUDA(launch_k(hc_down_kernel, dim3(lr + hc, (nt + kHcDownTok - 1) / kHcDownTok), dim3(256), 0, st, c->use_pdl, (const float*)L.w_down,
                          (const float*)xn, nt, hc_dim, lr, hc, raw));
    }
    {
        ProfScope p_(c, st, "hc_up_mixed");
        if (hc <= 4 && lr % 4 == 0 && lr <= 384) {  // four rows of 384 are 48 registers: what a warp can hold beside its work
            const dim3 grid((e + 3) / 4, (nt + kHcUpTok - 1) / kHcUpTok);
            const size_t smem = (size_t)std::min(nt, kHcUpTok) * lr * 4;
            auto kern = lr <= 128 ? hc_up_mixed_reg_kernel<4, 1> : lr <= 256 ? hc_up_mixed_reg_kernel<4, 2> : hc_up_mixed_reg_kernel<4, 3>;
            DNB_CUDA(launch_k(kern, grid, dim3(128), smem, st, c->use_pdl, (const float*)L.w_up, (const float*)raw, (const float*)xn, nt, hc, e, lr, mixed));
        } else {
            hc_up_mixed_kernel<<<dim3((e + 3) / 4, nt), 128, (size_t)lr * 4, st>>>(L.w_up, raw, xn, nt, hc, e, lr, mixed);
        }
    }
    c->launches += 3;
    DNB_CUDA(cudaGetLastError());
    if ((rc = enqueue_block(c, layer, mixed, nt, blk))) return rc;
    {
        ProfScope p_(c, st, "hc_combine");
        DNB_CUDA(launch_k(hc_combine_kernel, dim3(nt * hc), dim3(256), 0, st, c->use_pdl, res_dev ? (const float*)res_dev : res, (const float*)blk,
                          (const float*)raw, hc, e, lr, out));
    }
    c->launches++;
    DNB_CUDA(cudaGetLastError());
    return DNB_OK;
}

static int hc_scratch(dnb_ctx* c, HcState* H, int layer, int nt) {
    const HcLayer& L = H->layers[layer];
    const int e = c->model.e, hc_dim = L.hc * e;
    int rc;
    if (!moe_layer_ready(c, layer)) {
        set_error("hc_moe_block: layer %d is not fully registered", layer);
        return DNB_DECLINED;
    }
    const void* before[4] = {H->xn.p, H->raw.p, H->mixed.p, H->blk.p};
    if ((rc = ensure_workspace(c, nt)) || (rc = hc_grow(H->xn, (size_t)nt * hc_dim * 4)) || (rc = hc_grow(H->raw, (size_t)nt * (L.low_rank + L.hc) * 4)) ||
        (rc = hc_grow(H->mixed, (size_t)nt * e * 4)) || (rc = hc_grow(H->blk, (size_t)nt * e * 4)))
        return rc;
    if (before[0] != H->xn.p || before[1] != H->raw.p || before[2] != H->mixed.p || before[3] != H->blk.p) forget_graphs(c);  // they hold the old addresses
    return DNB_OK;
}

}  // namespace dnb

using namespace dnb;

extern "C" int dnb_register_hc(dnb_ctx* c, int layer, int hc, int low_rank, const float* w_norm, const float* w_down_inject,
                               const float* w_up) {
    if (!c || !w_norm || !w_down_inject || !w_up) return DNB_ERR_ARG;
    const Model& M = c->model;
    if (layer < 0 || layer >= M.n_layer || hc < 1 || hc > 16 || low_rank < 1 || low_rank > 8192 || M.e % 4) {
        set_error("register_hc: layer %d / hc %d / low_rank %d outside the configured model or the kernels' range", layer, hc, low_rank);
        return DNB_ERR_ARG;
    }
    DNB_CUDA(cudaSetDevice(c->device));
    if (!c->hc) c->hc = new HcState();
    HcState* H = static_cast<HcState*>(c->hc);
    H->layers.resize(M.n_layer);
    HcLayer& L = H->layers[layer];
    DNB_CUDA(cudaDeviceSynchronize());
    forget_graphs(c);
    if (L.w_norm) cudaFree(L.w_norm);
    if (L.w_down) cudaFree(L.w_down);
    if (L.w_up) cudaFree(L.w_up);
    L = HcLayer();
    const size_t hc_dim = (size_t)hc * M.e;
    const size_t n_norm = hc_dim, n_down = (size_t)(low_rank + hc) * hc_dim, n_up = hc_dim * low_rank;
    DNB_CUDA(cudaMalloc((void**)&L.w_norm, n_norm * 4));
    DNB_CUDA(cudaMalloc((void**)&L.w_down, n_down * 4));
    DNB_CUDA(cudaMalloc((void**)&L.w_up, n_up * 4));
    DNB_CUDA(cudaMemcpy(L.w_norm, w_norm, n_norm * 4, cudaMemcpyHostToDevice));
    DNB_CUDA(cudaMemcpy(L.w_down, w_down_inject, n_down * 4, cudaMemcpyHostToDevice));
    DNB_CUDA(cudaMemcpy(L.w_up, w_up, n_up * 4, cudaMemcpyHostToDevice));
    L.hc = hc;
    L.low_rank = low_rank;
    return DNB_OK;
}

static HcState* hc_ready(dnb_ctx* c, int layer) {
    HcState* H = c ? static_cast<HcState*>(c->hc) : nullptr;
    if (!H || layer < 0 || layer >= (int)H->layers.size() || !H->layers[layer].w_norm) {
        set_error("hc_moe_block: layer %d has no hyper-connection weights registered", layer);
        return nullptr;
    }
    return H;
}

extern "C" int dnb_hc_moe_block_dev(dnb_ctx* c, int layer, const float* res_dev, int nt, float* out_dev) {
    if (!c || !res_dev || !out_dev || nt < 1) return DNB_ERR_ARG;
    HcState* H = hc_ready(c, layer);
    if (!H) return DNB_DECLINED;
    DNB_CUDA(cudaSetDevice(c->device));
    const int rc = hc_scratch(c, H, layer, nt);
    if (rc) return rc;
    return graphed(c, GraphKey{7, layer, nt, res_dev, out_dev}, [&]() { return hc_enqueue(c, H, layer, res_dev, nullptr, nt, out_dev); });
}

extern "C" int dnb_hc_moe_block(dnb_ctx* c, int layer, const float* res, int nt, float* out) {
    if (!c || !res || !out || nt < 1) return DNB_ERR_ARG;
    HcState* H = hc_ready(c, layer);
    if (!H) return DNB_DECLINED;
    DNB_CUDA(cudaSetDevice(c->device));
    const size_t bytes = (size_t)nt * H->layers[layer].hc * c->model.e * 4;
    int rc;
    const void* before[4] = {H->res.p, H->out.p, H->host_in.p, H->host_out.p};
    if ((rc = hc_grow(H->res, bytes)) || (rc = hc_grow(H->out, bytes)) || (rc = hc_grow(H->host_in, bytes, true)) ||
        (rc = hc_grow(H->host_out, bytes, true)))
        return rc;
    if (before[0] != H->res.p || before[1] != H->out.p || before[2] != H->host_in.p || before[3] != H->host_out.p) forget_graphs(c);
    if ((rc = hc_scratch(c, H, layer, nt))) return rc;
    memcpy(H->host_in.p, res, bytes);
    // A few tokens: the first kernel reads the pinned rows and the last one writes pinned rows (both are device-addressable);
    // copies of their own and the dependencies around them cost more than the 32 KB of a token.
    const bool direct = bytes <= 256 * 1024;
    rc = graphed(c, GraphKey{8, layer, nt, nullptr, nullptr}, [&]() -> int {
        if (direct) return hc_enqueue(c, H, layer, (const float*)H->host_in.p, (float*)H->res.p, nt, (float*)H->host_out.p);
        DNB_CUDA(cudaMemcpyAsync(H->res.p, H->host_in.p, bytes, cudaMemcpyHostToDevice, c->stream));
        const int r = hc_enqueue(c, H, layer, (const float*)H->res.p, nullptr, nt, (float*)H->out.p);
        if (r) return r;
        DNB_CUDA(cudaMemcpyAsync(H->host_out.p, H->out.p, bytes, cudaMemcpyDeviceToHost, c->stream));
        return DNB_OK;
    });
    if (rc) return rc;
    DNB_CUDA(wait_for_stream(c->stream));
    const int st = *reinterpret_cast<volatile int*>(c->status_host);
    if (st != 0) {  // a bounded device wait gave up: nothing is written (see dnb_device_status)
        *reinterpret_cast<volatile int*>(c->status_host) = 0;
        set_error("hc_moe_block: a bounded device wait gave up (status %d); the result was discarded", st);
        return DNB_DECLINED;
    }
    memcpy(out, H->host_out.p, bytes);
    return DNB_OK;
}
