// warmnet.cu -- the learned warm start: a small convolutional network that
// maps the costs of a pyramid level to the messages its nodes should start
// from (on the beliefs' scale), with
// hand-written tensor-core kernels -- the forward, data-gradient and
// weight-gradient convolutions on tcgen05 with tensor-memory accumulators
// (conv_tc.cu) -- the loss, ReLU, bias-gradient and Adam kernels, and a
// checkpoint format.
//
// Network (L labels, h hidden channels): conv3x3(L->h) ReLU, conv3x3(h->h)
// ReLU, conv3x3(h->h) ReLU, conv3x3(h->L); zero padding; activations NHWC.
// Input x = D_t / 4^t (the level's costs per fine node), output
// y = x + net(x), trained towards (D_t + m) / 4^t, m the message sums of a
// long hierarchical BP run (the finest level's, averaged per block, or the
// level's own).  Rounding points (mirrored by oracle/warmnet_ref.py):
// x, weights and hidden activations in BF16; sums in FP32; the output and
// every gradient in FP32, rounded to BF16 where they feed a tensor-core
// product.  The reference has no learned component: this whole file is new.
#include <cuda_bf16.h>

#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "ginf_gb300.h"
#include "ginf_internal.h"
#include "ptx.cuh"

namespace ginf_gpu {

cudaError_t conv_first_tc(int cin, const float *x, __nv_bfloat16 *x_bf16, const __nv_bfloat16 *w, const float *bias,
                          int nimg, int h, int wd, __nv_bfloat16 *out, int *status, cudaStream_t s);
cudaError_t conv_fwd_tc(int cin, int cout, bool relu, const __nv_bfloat16 *in, const __nv_bfloat16 *w,
                        const float *bias, int nimg, int h, int wd, void *out, const float *res, int *status,
                        cudaStream_t s);
cudaError_t conv_loss_tc(int cout, const __nv_bfloat16 *in, const __nv_bfloat16 *w, const float *bias, int nimg, int h,
                         int wd, const float *x, const float *target, bool wide_squares, float scale,
                         __nv_bfloat16 *grad, float *bias_part, double *loss_part, int *parts, int *status,
                         cudaStream_t s);
cudaError_t conv_dgrad_tc(int cin, const __nv_bfloat16 *in, const __nv_bfloat16 *w, int nimg, int h, int wd,
                          const __nv_bfloat16 *act, __nv_bfloat16 *grad, float *bias_part, int *parts, int *status,
                          cudaStream_t s);
cudaError_t conv_wgrad_tc(int cin, int cout, const __nv_bfloat16 *dout, const __nv_bfloat16 *in, int nimg, int h,
                          int wd, float *partials, int max_parts, int *parts, int *status, cudaStream_t s);

namespace {

constexpr int kThreads = 256;

inline unsigned nblocks(size_t n, int per = kThreads) { return (unsigned)((n + per - 1) / per); }

__device__ __forceinline__ uint32_t pack_bf16(__nv_bfloat16 lo, __nv_bfloat16 hi) {
    return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}


struct Geo {
    int n, h, w;  // images, rows, columns
};

// A layer's gradients from the per-CTA partial sums: out[i] = sum over k of
// w_part[k][i] for the nw weights, then the nb biases (which follow them in
// the parameter vector) from b_part.  Eight threads per output take every
// eighth partial, 32 neighbouring outputs reading one 128-byte line, and are
// added in a fixed order.  One thread per output, in order, was a chain of
// 304 (bias: 768) loads on a few blocks: 16 and 28 us a layer at 16x256x192x64,
// now about 7 us a layer.
//
// With loss_part, one more block (its warp 0) sums the loss: lane l takes
// loss_part[l], loss_part[l + 32], ..., then the lanes combine in a fixed
// order.
constexpr int kSlices = 8;
__global__ void __launch_bounds__(256) k_reduce_grads(const float *__restrict__ w_part, int w_parts, int nw,
                                                       const float *__restrict__ b_part, int b_parts, int nb,
                                                       float *__restrict__ out, const double *loss_part,
                                                       double denom, float *loss) {
    __shared__ float red[kSlices][32];
    const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
    grid_dependency_wait();
    launch_dependents();
    if (loss_part && blockIdx.x == gridDim.x - 1) {
        if (slice != 0) return;
        double s = 0.0;
        for (int i = lane; i < b_parts; i += 32) s += loss_part[i];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) *loss = (float)(s / denom);
        return;
    }
    const int i = blockIdx.x * 32 + lane;
    float s = 0.f;
    if (i < nw + nb) {
        const bool bias = i >= nw;
        const float *p = bias ? b_part + (i - nw) : w_part + i;
        const int n = bias ? nb : nw, parts = bias ? b_parts : w_parts;
        int k = slice;
        for (; k + 7 * kSlices < parts; k += 8 * kSlices) {
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = p[(size_t)(k + j * kSlices) * n];
#pragma unroll
            for (int j = 0; j < 8; ++j) s += v[j];
        }
        for (; k < parts; k += kSlices) s += p[(size_t)k * n];
    }
    red[slice][lane] = s;
    __syncthreads();
    if (slice == 0 && i < nw + nb) {
#pragma unroll
        for (int q = 1; q < kSlices; ++q) s += red[q][lane];
        out[i] = s;
    }
}

// Round to BF16, eight values per thread (two 16-byte loads, one 16-byte
// store) when both buffers are 16-byte aligned, grid-stride, scalar tail.
__global__ void k_f32_to_bf16(const float *__restrict__ a, __nv_bfloat16 *__restrict__ b, size_t n) {
    const size_t n8 = (((uintptr_t)a | (uintptr_t)b) & 15) == 0 ? n / 8 : 0;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (size_t i = t; i < n8; i += stride) {
        const float4 lo = reinterpret_cast<const float4 *>(a)[2 * i], hi = reinterpret_cast<const float4 *>(a)[2 * i + 1];
        reinterpret_cast<uint4 *>(b)[i] =
            make_uint4(pack_bf16(__float2bfloat16_rn(lo.x), __float2bfloat16_rn(lo.y)),
                       pack_bf16(__float2bfloat16_rn(lo.z), __float2bfloat16_rn(lo.w)),
                       pack_bf16(__float2bfloat16_rn(hi.x), __float2bfloat16_rn(hi.y)),
                       pack_bf16(__float2bfloat16_rn(hi.z), __float2bfloat16_rn(hi.w)));
    }
    for (size_t i = n8 * 8 + t; i < n; i += stride) b[i] = __float2bfloat16_rn(a[i]);
}

void f32_to_bf16(const float *a, __nv_bfloat16 *b, size_t n, cudaStream_t s) {
    const size_t blocks = (n / 8 + kThreads - 1) / kThreads;
    k_f32_to_bf16<<<(unsigned)(blocks < 1 ? 1 : (blocks > 4096 ? 4096 : blocks)), kThreads, 0, s>>>(a, b, n);
}

// Adam (bias-corrected) on FP32 master weights, refreshing the BF16 copy.
__global__ void k_adam(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m, float *__restrict__ v,
                       int n, float lr, float b1, float b2, float eps, float c1, float c2,
                       __nv_bfloat16 *__restrict__ pb) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float upd = lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    const float np = p[i] - upd;
    p[i] = np;
    if (pb) pb[i] = __float2bfloat16_rn(np);
}

uint64_t splitmix(uint64_t &s) {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

uint64_t fnv1a(const void *data, size_t n, uint64_t h = 1469598103934665603ull) {
    const unsigned char *p = static_cast<const unsigned char *>(data);
    for (size_t i = 0; i < n; ++i) {
        h ^= p[i];
        h *= 1099511628211ull;
    }
    return h;
}

}  // namespace

}  // namespace ginf_gpu

using namespace ginf_gpu;

// ---------------------------------------------------------------------------
// The network object.

struct ginf_warmnet {
    int device = -1;  // the device its parameters and buffers live on
    int L = 0, hidden = 0;
    int cin[4], cout[4];
    size_t woff[4], boff[4], nparams = 0;  // offsets into the flat FP32 parameter vector
    float *params = nullptr;               // FP32 master weights and biases (device)
    float *adam_m = nullptr, *adam_v = nullptr;
    float *grads = nullptr;
    __nv_bfloat16 *wbf = nullptr;  // BF16 copy of the weights (same offsets)
    int64_t step = 0;
    // activations / gradients, grown to the largest batch seen
    size_t cap_pix = 0;
    __nv_bfloat16 *a[4] = {};  // a[0] = x (L ch), a[1..3] hidden
    float *y = nullptr;        // output (L ch)
    __nv_bfloat16 *gb[2] = {};  // output gradients of one layer and the next (max channels)
    float *partials = nullptr;   // weight-gradient partial sums, one per CTA (two per SM)
    float *bias_part = nullptr;  // bias-gradient partial sums
    size_t cap_partials = 0;
    double *loss_part = nullptr;
    // The loss and the status word (DEV_ERR_* from the convolution kernels'
    // bounded waits) on the device, and where one copy leaves both on the host.
    struct Report {
        float loss;
        int status;
    };
    Report *report = nullptr, *report_host = nullptr;
    int *status = nullptr;  // &report->status
};

namespace {

ginf_status wfail(ginf_status s, const std::string &m) {
    ginf_gpu::set_last_error(m.c_str());
    return s;
}

#define GINF_WCK(call)                                                                       \
    do {                                                                                     \
        cudaError_t e_ = (call);                                                             \
        if (e_ != cudaSuccess) {                                                             \
            cudaGetLastError();                                                              \
            return wfail(GINF_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
        }                                                                                    \
    } while (0)

void layout(ginf_warmnet *n) {
    const int ch[5] = {n->L, n->hidden, n->hidden, n->hidden, n->L};
    size_t off = 0;
    for (int l = 0; l < 4; ++l) {
        n->cin[l] = ch[l];
        n->cout[l] = ch[l + 1];
        n->woff[l] = off;
        off += (size_t)n->cout[l] * 9 * n->cin[l];
        n->boff[l] = off;
        off += n->cout[l];
    }
    n->nparams = off;
}

ginf_status alloc_params(ginf_warmnet *n) {
    GINF_WCK(cudaMalloc(&n->params, n->nparams * sizeof(float)));
    GINF_WCK(cudaMalloc(&n->adam_m, n->nparams * sizeof(float)));
    GINF_WCK(cudaMalloc(&n->adam_v, n->nparams * sizeof(float)));
    GINF_WCK(cudaMalloc(&n->grads, n->nparams * sizeof(float)));
    GINF_WCK(cudaMalloc(&n->wbf, n->nparams * sizeof(__nv_bfloat16)));
    GINF_WCK(cudaMemset(n->adam_m, 0, n->nparams * sizeof(float)));
    GINF_WCK(cudaMemset(n->adam_v, 0, n->nparams * sizeof(float)));
    GINF_WCK(cudaMemset(n->grads, 0, n->nparams * sizeof(float)));
    GINF_WCK(cudaMalloc(&n->loss_part, 1024 * sizeof(double)));
    GINF_WCK(cudaMalloc(&n->report, sizeof(ginf_warmnet::Report)));
    GINF_WCK(cudaMemset(n->report, 0, sizeof(ginf_warmnet::Report)));
    GINF_WCK(cudaMallocHost(&n->report_host, sizeof(ginf_warmnet::Report)));
    n->status = &n->report->status;
    return GINF_OK;
}

// The end of a call: the loss (when asked for) and the status word in one
// copy ahead of the synchronisation, then a wait in a convolution kernel that
// ran out.
ginf_status finish(ginf_warmnet *n, float *loss, cudaStream_t s) {
    GINF_WCK(cudaMemcpyAsync(n->report_host, n->report, sizeof(ginf_warmnet::Report), cudaMemcpyDeviceToHost, s));
    GINF_WCK(cudaStreamSynchronize(s));
    if (loss) *loss = n->report_host->loss;
    const int st = n->report_host->status;
    if (st == 0) return GINF_OK;
    GINF_WCK(cudaMemset(n->status, 0, sizeof(int)));
    return wfail(GINF_ERR_TIMEOUT, "warm-start convolution: a device wait ran out (status " + std::to_string(st) + ")");
}

ginf_status refresh_bf16(ginf_warmnet *n, cudaStream_t s) {
    f32_to_bf16(n->params, n->wbf, n->nparams, s);
    GINF_WCK(cudaGetLastError());
    return GINF_OK;
}

ginf_status ensure_batch(ginf_warmnet *n, size_t pix) {
    if (pix <= n->cap_pix) return GINF_OK;
    for (int l = 0; l < 4; ++l) cudaFree(n->a[l]);
    cudaFree(n->y);
    cudaFree(n->gb[0]);
    cudaFree(n->gb[1]);
    const size_t cmax = (size_t)std::max(n->L, n->hidden);
    GINF_WCK(cudaMalloc(&n->a[0], pix * n->L * sizeof(__nv_bfloat16)));
    for (int l = 1; l < 4; ++l) GINF_WCK(cudaMalloc(&n->a[l], pix * n->hidden * sizeof(__nv_bfloat16)));
    GINF_WCK(cudaMalloc(&n->y, pix * n->L * sizeof(float)));
    for (int k = 0; k < 2; ++k) GINF_WCK(cudaMalloc(&n->gb[k], pix * cmax * sizeof(__nv_bfloat16)));
    n->cap_pix = pix;
    // Partial sums: one per CTA of a gradient kernel (up to two per SM).
    int sms = 0;
    GINF_WCK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, n->device));
    size_t need = 0;
    for (int l = 0; l < 4; ++l) need = std::max(need, (size_t)2 * sms * n->cout[l] * 9 * n->cin[l]);
    if (need > n->cap_partials) {
        cudaFree(n->partials);
        cudaFree(n->bias_part);
        GINF_WCK(cudaMalloc(&n->partials, need * sizeof(float)));
        GINF_WCK(cudaMalloc(&n->bias_part, (size_t)2 * sms * cmax * sizeof(float)));
        n->cap_partials = need;
    }
    return GINF_OK;
}

// The hidden layers, from x; its BF16 rounding into a[0] when `keep` asks for
// it (the first weight gradient reads it).
ginf_status forward_hidden(ginf_warmnet *n, const float *x, Geo g, bool keep, int *status, cudaStream_t s) {
    const size_t pix = (size_t)g.n * g.h * g.w;
    ginf_status st = ensure_batch(n, pix);
    if (st != GINF_OK) return st;
    GINF_WCK(conv_first_tc(n->L, x, keep ? n->a[0] : nullptr, n->wbf + n->woff[0], n->params + n->boff[0], g.n, g.h,
                           g.w, n->a[1], status, s));
    for (int l = 1; l < 3; ++l)
        GINF_WCK(conv_fwd_tc(n->cin[l], n->cout[l], true, n->a[l], n->wbf + n->woff[l], n->params + n->boff[l], g.n, g.h,
                             g.w, n->a[l + 1], nullptr, status, s));
    return GINF_OK;
}

// y = x + net(x) into y_out (the network's own buffer when null); the last
// layer reads x itself as its residual.
ginf_status forward(ginf_warmnet *n, const float *x, Geo g, int *status, cudaStream_t s, float *y_out = nullptr) {
    ginf_status st = forward_hidden(n, x, g, false, status, s);
    if (st != GINF_OK) return st;
    GINF_WCK(conv_fwd_tc(n->cin[3], n->cout[3], false, n->a[3], n->wbf + n->woff[3], n->params + n->boff[3], g.n, g.h,
                         g.w, y_out ? y_out : n->y, x, status, s));
    return GINF_OK;
}

// Loss and every parameter gradient (into n->grads) for one batch.  The last
// layer's output stays in its kernel: the loss, the BF16 output gradient and
// its bias sums leave from the epilogue, and each data gradient passes its
// ReLU and leaves bias sums the same way, so no FP32 gradient is written.
// 16x256x192x64: 519 us a call, 500 of them in its fifteen kernels (34 kernels
// with separate ones for loss, conversions, ReLU, flipped weights and bias sums
// took 1335).
ginf_status gradients(ginf_warmnet *n, const float *x, const float *target, Geo g, cudaStream_t s) {
    const size_t pix = (size_t)g.n * g.h * g.w, ny = pix * n->L;
    ginf_status st = ensure_batch(n, pix);
    if (st != GINF_OK) return st;
    // The kernel reads the target 16 bytes at a time.  The loss is an FP64 sum:
    // of FP32 squares, four at a time, for an aligned target, of single FP64
    // squares otherwise (16x256x192x64: 531 and 705 us a call; the FP64 unit's
    // rate shows in the second only).
    const bool aligned = ((uintptr_t)target & 15) == 0;
    if (!aligned) {
        GINF_WCK(cudaMemcpyAsync(n->y, target, ny * sizeof(float), cudaMemcpyDeviceToDevice, s));
        target = n->y;
    }
    if ((st = forward_hidden(n, x, g, true, n->status, s)) != GINF_OK) return st;
    int bias_parts = 0;
    GINF_WCK(conv_loss_tc(n->L, n->a[3], n->wbf + n->woff[3], n->params + n->boff[3], g.n, g.h, g.w, x, target,
                          !aligned, 2.f / (float)ny, n->gb[0], n->bias_part, n->loss_part, &bias_parts, n->status, s));
    int cur = 0;
    for (int l = 3; l >= 0; --l) {
        const int ci = n->cin[l], co = n->cout[l], nw = co * 9 * ci;
        int w_parts = 0;
        GINF_WCK(conv_wgrad_tc(ci, co, n->gb[cur], n->a[l], g.n, g.h, g.w, n->partials, (int)(n->cap_partials / nw),
                               &w_parts, n->status, s));
        const bool last = l == 3;  // with the loss
        GINF_WCK(launch_after(k_reduce_grads, (nw + co + 31) / 32 + last, 256, 0, s, n->partials, w_parts, nw,
                              n->bias_part, bias_parts, co, n->grads + n->woff[l], last ? n->loss_part : nullptr,
                              (double)ny, &n->report->loss));
        if (l == 0) break;
        // Data gradient, through the ReLU of layer l-1's output.
        GINF_WCK(conv_dgrad_tc(co, n->gb[cur], n->wbf + n->woff[l], g.n, g.h, g.w, n->a[l], n->gb[cur ^ 1], n->bias_part,
                               &bias_parts, n->status, s));
        cur ^= 1;
    }
    return GINF_OK;
}

ginf_status check_geo(const ginf_warmnet *n, int nimg, int h, int w) {
    if (!n) return wfail(GINF_ERR_INVALID_ARGUMENT, "warmnet is NULL");
    if (nimg < 1 || h < 1 || w < 1) return wfail(GINF_ERR_INVALID_ARGUMENT, "bad batch geometry");
    int dev = 0;
    GINF_WCK(cudaGetDevice(&dev));
    if (dev != n->device)
        return wfail(GINF_ERR_INVALID_ARGUMENT, "network was created on device " + std::to_string(n->device) +
                                                    ", the calling thread's current device is " + std::to_string(dev));
    return GINF_OK;
}

const char kMagic[8] = {'G', 'I', 'N', 'F', 'W', 'N', 'E', 'T'};
constexpr uint32_t kVersion = 1;

}  // namespace

namespace ginf_gpu {
// Used by the learned HBP solve in capi.cu: forward pass on level-t inputs.
// Device waits that run out are recorded in `status` (the network's own
// word when null).
ginf_status warmnet_forward(ginf_warmnet *n, const float *x, int nimg, int h, int w, float **y_out, int *status,
                            cudaStream_t s) {
    ginf_status st = check_geo(n, nimg, h, w);
    if (st != GINF_OK) return st;
    Geo g{nimg, h, w};
    st = forward(n, x, g, status ? status : n->status, s);
    if (st != GINF_OK) return st;
    *y_out = n->y;
    return GINF_OK;
}

// The C-ABI forward: the last layer writes the caller's buffer.
ginf_status warmnet_forward_into(ginf_warmnet *n, const float *x, int nimg, int h, int w, float *out, cudaStream_t s) {
    ginf_status st = check_geo(n, nimg, h, w);
    if (st != GINF_OK) return st;
    Geo g{nimg, h, w};
    return forward(n, x, g, n->status, s, out);
}
int warmnet_labels(const ginf_warmnet *n) { return n ? n->L : 0; }
}  // namespace ginf_gpu

extern "C" {

ginf_status ginf_warmnet_create(ginf_warmnet **out, int32_t num_labels, int32_t hidden, uint64_t seed) {
    ginf_gpu::set_last_error("");
    if (!out) return wfail(GINF_ERR_INVALID_ARGUMENT, "out is NULL");
    if ((num_labels != 16 && num_labels != 32 && num_labels != 64) || hidden != 32)
        return wfail(GINF_ERR_UNSUPPORTED, "the warm-start network is compiled for L in {16, 32, 64} and 32 hidden channels");
    ginf_warmnet *n = new ginf_warmnet();
    n->L = num_labels;
    n->hidden = hidden;
    layout(n);
    ginf_status st = cudaGetDevice(&n->device) == cudaSuccess ? alloc_params(n)
                                                               : wfail(GINF_ERR_NO_DEVICE, "no current CUDA device");
    if (st != GINF_OK) {
        ginf_warmnet_destroy(n);
        return st;
    }
    // He-uniform weights (last layer scaled by 0.1), zero biases.
    std::vector<float> p(n->nparams, 0.f);
    uint64_t s = seed * 0x9E3779B97F4A7C15ull + 12345;
    for (int l = 0; l < 4; ++l) {
        const float bound = std::sqrt(6.f / (9.f * n->cin[l])) * (l == 3 ? 0.1f : 1.f);
        for (size_t i = 0; i < (size_t)n->cout[l] * 9 * n->cin[l]; ++i) {
            const double u = (double)(splitmix(s) >> 11) * (1.0 / 9007199254740992.0);
            p[n->woff[l] + i] = (float)((2.0 * u - 1.0) * bound);
        }
    }
    if (cudaMemcpy(n->params, p.data(), p.size() * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess ||
        refresh_bf16(n, nullptr) != GINF_OK || cudaDeviceSynchronize() != cudaSuccess) {
        cudaGetLastError();
        ginf_warmnet_destroy(n);
        return wfail(GINF_ERR_CUDA, "warmnet initialisation failed");
    }
    *out = n;
    return GINF_OK;
}

ginf_status ginf_warmnet_destroy(ginf_warmnet *n) {
    if (!n) return GINF_OK;
    cudaFree(n->params);
    cudaFree(n->adam_m);
    cudaFree(n->adam_v);
    cudaFree(n->grads);
    cudaFree(n->wbf);
    for (int l = 0; l < 4; ++l) cudaFree(n->a[l]);
    cudaFree(n->y);
    cudaFree(n->gb[0]);
    cudaFree(n->gb[1]);
    cudaFree(n->partials);
    cudaFree(n->bias_part);
    cudaFree(n->loss_part);
    cudaFree(n->report);
    cudaFreeHost(n->report_host);
    delete n;
    return GINF_OK;
}

ginf_status ginf_warmnet_num_params(const ginf_warmnet *n, int64_t *count) {
    if (!n || !count) return wfail(GINF_ERR_INVALID_ARGUMENT, "NULL argument");
    *count = (int64_t)n->nparams;
    return GINF_OK;
}

ginf_status ginf_warmnet_get_params(const ginf_warmnet *n, float *host) {
    if (!n || !host) return wfail(GINF_ERR_INVALID_ARGUMENT, "NULL argument");
    GINF_WCK(cudaMemcpy(host, n->params, n->nparams * sizeof(float), cudaMemcpyDeviceToHost));
    return GINF_OK;
}

ginf_status ginf_warmnet_set_params(ginf_warmnet *n, const float *host) {
    if (!n || !host) return wfail(GINF_ERR_INVALID_ARGUMENT, "NULL argument");
    GINF_WCK(cudaMemcpy(n->params, host, n->nparams * sizeof(float), cudaMemcpyHostToDevice));
    ginf_status st = refresh_bf16(n, nullptr);
    if (st != GINF_OK) return st;
    GINF_WCK(cudaDeviceSynchronize());
    return GINF_OK;
}

ginf_status ginf_warmnet_forward(ginf_warmnet *n, const float *x, int32_t nimg, int32_t h, int32_t w, float *out,
                                 void *stream) {
    ginf_gpu::set_last_error("");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    ginf_status st = warmnet_forward_into(n, x, nimg, h, w, out, s);
    if (st != GINF_OK) return st;
    return finish(n, nullptr, s);
}

ginf_status ginf_warmnet_gradients(ginf_warmnet *n, const float *x, const float *target, int32_t nimg, int32_t h,
                                   int32_t w, float *loss, float *grads_host, void *stream) {
    ginf_gpu::set_last_error("");
    ginf_status st = check_geo(n, nimg, h, w);
    if (st != GINF_OK) return st;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    Geo g{nimg, h, w};
    if ((st = gradients(n, x, target, g, s)) != GINF_OK) return st;
    if (grads_host)
        GINF_WCK(cudaMemcpyAsync(grads_host, n->grads, n->nparams * sizeof(float), cudaMemcpyDeviceToHost, s));
    return finish(n, loss, s);
}

ginf_status ginf_warmnet_train_step(ginf_warmnet *n, const float *x, const float *target, int32_t nimg, int32_t h,
                                    int32_t w, float lr, float *loss, void *stream) {
    ginf_gpu::set_last_error("");
    ginf_status st = check_geo(n, nimg, h, w);
    if (st != GINF_OK) return st;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    Geo g{nimg, h, w};
    if ((st = gradients(n, x, target, g, s)) != GINF_OK) return st;
    n->step += 1;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - std::pow(b1, (float)n->step), c2 = 1.f - std::pow(b2, (float)n->step);
    k_adam<<<nblocks(n->nparams), kThreads, 0, s>>>(n->params, n->grads, n->adam_m, n->adam_v, (int)n->nparams, lr,
                                                    b1, b2, 1e-8f, c1, c2, n->wbf);
    GINF_WCK(cudaGetLastError());
    return finish(n, loss, s);
}

// Checkpoint: magic "GINFWNET", u32 version, u32 L, u32 hidden, i64 Adam step,
// u64 parameter count, then parameters, Adam m and Adam v as FP32, then the
// FNV-1a 64 checksum of everything before it.
ginf_status ginf_warmnet_save(const ginf_warmnet *n, const char *path) {
    if (!n || !path) return wfail(GINF_ERR_INVALID_ARGUMENT, "NULL argument");
    std::vector<unsigned char> buf;
    auto put = [&](const void *p, size_t k) {
        const unsigned char *c = static_cast<const unsigned char *>(p);
        buf.insert(buf.end(), c, c + k);
    };
    const uint32_t ver = kVersion, L = (uint32_t)n->L, hid = (uint32_t)n->hidden;
    const uint64_t np = n->nparams;
    put(kMagic, 8);
    put(&ver, 4);
    put(&L, 4);
    put(&hid, 4);
    put(&n->step, 8);
    put(&np, 8);
    std::vector<float> tmp(np);
    for (float *src : {n->params, n->adam_m, n->adam_v}) {
        GINF_WCK(cudaMemcpy(tmp.data(), src, np * sizeof(float), cudaMemcpyDeviceToHost));
        put(tmp.data(), np * sizeof(float));
    }
    const uint64_t sum = fnv1a(buf.data(), buf.size());
    put(&sum, 8);
    FILE *f = std::fopen(path, "wb");
    if (!f) return wfail(GINF_ERR_INVALID_ARGUMENT, std::string("cannot write ") + path);
    const bool ok = std::fwrite(buf.data(), 1, buf.size(), f) == buf.size();
    std::fclose(f);
    if (!ok) return wfail(GINF_ERR_INVALID_ARGUMENT, std::string("short write to ") + path);
    return GINF_OK;
}

ginf_status ginf_warmnet_load(ginf_warmnet **out, const char *path) {
    ginf_gpu::set_last_error("");
    if (!out || !path) return wfail(GINF_ERR_INVALID_ARGUMENT, "NULL argument");
    FILE *f = std::fopen(path, "rb");
    if (!f) return wfail(GINF_ERR_INVALID_ARGUMENT, std::string("cannot read ") + path);
    std::vector<unsigned char> buf;
    unsigned char tmp[65536];
    size_t k;
    while ((k = std::fread(tmp, 1, sizeof(tmp), f)) > 0) buf.insert(buf.end(), tmp, tmp + k);
    std::fclose(f);
    const size_t head = 8 + 4 + 4 + 4 + 8 + 8;
    if (buf.size() < head + 8 || std::memcmp(buf.data(), kMagic, 8) != 0)
        return wfail(GINF_ERR_INVALID_ARGUMENT, "not a warm-start network file");
    uint64_t sum;
    std::memcpy(&sum, buf.data() + buf.size() - 8, 8);
    if (sum != fnv1a(buf.data(), buf.size() - 8))
        return wfail(GINF_ERR_INVALID_ARGUMENT, "warm-start network file: checksum mismatch");
    uint32_t ver, L, hid;
    int64_t step;
    uint64_t np;
    std::memcpy(&ver, buf.data() + 8, 4);
    std::memcpy(&L, buf.data() + 12, 4);
    std::memcpy(&hid, buf.data() + 16, 4);
    std::memcpy(&step, buf.data() + 20, 8);
    std::memcpy(&np, buf.data() + 28, 8);
    if (ver != kVersion) return wfail(GINF_ERR_UNSUPPORTED, "warm-start network file: unknown version");
    ginf_warmnet *n = nullptr;
    ginf_status st = ginf_warmnet_create(&n, (int32_t)L, (int32_t)hid, 0);
    if (st != GINF_OK) return st;
    if (np != n->nparams || buf.size() != head + 3 * np * sizeof(float) + 8) {
        ginf_warmnet_destroy(n);
        return wfail(GINF_ERR_INVALID_ARGUMENT, "warm-start network file: size mismatch");
    }
    const unsigned char *p = buf.data() + head;
    float *dst[3] = {n->params, n->adam_m, n->adam_v};
    for (int i = 0; i < 3; ++i) {
        if (cudaMemcpy(dst[i], p + (size_t)i * np * sizeof(float), np * sizeof(float), cudaMemcpyHostToDevice) !=
            cudaSuccess) {
            cudaGetLastError();
            ginf_warmnet_destroy(n);
            return wfail(GINF_ERR_CUDA, "warm-start network upload failed");
        }
    }
    n->step = step;
    if ((st = refresh_bf16(n, nullptr)) != GINF_OK || cudaDeviceSynchronize() != cudaSuccess) {
        ginf_warmnet_destroy(n);
        return st != GINF_OK ? st : wfail(GINF_ERR_CUDA, "warm-start network upload failed");
    }
    *out = n;
    return GINF_OK;
}

}  // extern "C"
