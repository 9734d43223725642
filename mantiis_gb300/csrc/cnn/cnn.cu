// Kernels of the warm-start encoder-decoder network (include/mantiis_cnn.h):
// 3x3 convolutions (forward, data gradient, weight gradient) with BF16
// weights and FP32 accumulation, pooling / upsampling / ReLU adjoints, the
// masked loss and the Adam update.  sm_103a.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <type_traits>

#include "../../../include/mantiis_cnn.h"
#include "conv_fma.cuh"
#include "conv_tc.cuh"

namespace
{
__global__ void k_relu_bw(float *dy, const float *y, int64_t count)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count && !(y[i] > 0.f)) dy[i] = 0.f;
}

__global__ void k_add(float *y, const float *x, int64_t count)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) y[i] += x[i];
}

// Pooling, upsampling and their adjoints.  What bounds them is memory (L2 for
// most layers), as long as the index arithmetic is short: with 64-bit divisions
// and one float per thread, upsampling 64 planes of 256^2 to 512^2 took 62 us, now
// 13 (84 MB).  Each plane follows the last, so all are one image of coarse rows:
// thread i takes V neighbouring pixels of a coarse row and the 2 x 2 V pixels of
// the fine image that belong to them, as vectors (V = 2) where widths and
// addresses allow; indices are 32-bit as long as they reach the end.  The passes
// that followed one another over the same activations (the skip connection's sum,
// ReLU adjoints, copies of a gradient for its two uses) are fused with these or
// into the convolutions: of a training step on 8 x 128^2 they took 420 us, now 130.
template <typename I, int V> struct Pixels
{
    I coarse, fine; // of the first pixel; the second fine row is 2 w further on
    __device__ __forceinline__ Pixels(I i, int w)
    {
        const I per = (I)(w / V), r = i / per, c = (i - r * per) * V;
        coarse = r * (I)w + c;
        fine = r * 4 * (I)w + 2 * c;
    }
    static __device__ __forceinline__ void load(const float *p, float v[V])
    {
        if constexpr (V == 2)
        {
            const float2 q = *reinterpret_cast<const float2 *>(p);
            v[0] = q.x, v[1] = q.y;
        }
        else v[0] = p[0];
    }
    static __device__ __forceinline__ void store(float *p, const float v[V])
    {
        if constexpr (V == 2) *reinterpret_cast<float2 *>(p) = make_float2(v[0], v[1]);
        else p[0] = v[0];
    }
    static __device__ __forceinline__ void load_fine(const float *p, float v[2 * V])
    {
        if constexpr (V == 2)
        {
            const float4 q = *reinterpret_cast<const float4 *>(p);
            v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
        }
        else v[0] = p[0], v[1] = p[1];
    }
    static __device__ __forceinline__ void store_fine(float *p, const float v[2 * V])
    {
        if constexpr (V == 2) *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
        else p[0] = v[0], p[1] = v[1];
    }
};

// y (coarse) = mean of the 2x2 blocks of x
template <typename I, int V> __global__ void k_pool_fw(const float *x, float *y, I count, int w)
{
    typedef Pixels<I, V> P;
    const I i = (I)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const P p(i, w);
    float a[2 * V], b[2 * V], m[V];
    P::load_fine(x + p.fine, a);
    P::load_fine(x + p.fine + 2 * w, b);
#pragma unroll
    for (int k = 0; k < V; k++) m[k] = 0.25f * (a[2 * k] + a[2 * k + 1] + b[2 * k] + b[2 * k + 1]);
    P::store(y + p.coarse, m);
}

// its adjoint, dx (fine) = dy / 4
template <typename I, int V> __global__ void k_pool_bw(const float *dy, float *dx, I count, int w)
{
    typedef Pixels<I, V> P;
    const I i = (I)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const P p(i, w);
    float g[V], f[2 * V];
    P::load(dy + p.coarse, g);
#pragma unroll
    for (int k = 0; k < V; k++) f[2 * k] = f[2 * k + 1] = 0.25f * g[k];
    P::store_fine(dx + p.fine, f);
    P::store_fine(dx + p.fine + 2 * w, f);
}

// ... added to the gradient that the skip connection brought, and through the
// ReLU that gave the fine y: dx = dx + dy / 4 where y > 0, else 0
template <typename I, int V>
__global__ void k_pool_bw_add_relu(const float *dy, const float *y, float *dx, I count, int w)
{
    typedef Pixels<I, V> P;
    const I i = (I)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const P p(i, w);
    float g[V];
    P::load(dy + p.coarse, g);
#pragma unroll
    for (int r = 0; r < 2; r++)
    {
        float v[2 * V], m[2 * V];
        P::load_fine(y + p.fine + r * 2 * w, m);
        P::load_fine(dx + p.fine + r * 2 * w, v);
#pragma unroll
        for (int k = 0; k < 2 * V; k++) v[k] = m[k] > 0.f ? v[k] + __fmul_rn(0.25f, g[k / 2]) : 0.f;
        P::store_fine(dx + p.fine + r * 2 * w, v);
    }
}

// y (fine) = nearest upsampling of x
template <typename I, int V> __global__ void k_up_fw(const float *x, float *y, I count, int w)
{
    typedef Pixels<I, V> P;
    const I i = (I)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const P p(i, w);
    float v[V], f[2 * V];
    P::load(x + p.coarse, v);
#pragma unroll
    for (int k = 0; k < V; k++) f[2 * k] = f[2 * k + 1] = v[k];
    P::store_fine(y + p.fine, f);
    P::store_fine(y + p.fine + 2 * w, f);
}

// its adjoint, dx (coarse, may be null) = sum of the 2x2 blocks of dy; with y, also
// masked = dx through the ReLU that gave y
template <typename I, int V>
__global__ void k_up_bw(const float *dy, float *dx, const float *y, float *masked, I count, int w)
{
    typedef Pixels<I, V> P;
    const I i = (I)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const P p(i, w);
    float a[2 * V], b[2 * V], s[V];
    P::load_fine(dy + p.fine, a);
    P::load_fine(dy + p.fine + 2 * w, b);
#pragma unroll
    for (int k = 0; k < V; k++) s[k] = a[2 * k] + a[2 * k + 1] + b[2 * k] + b[2 * k + 1];
    if (dx) P::store(dx + p.coarse, s);
    if (!y) return;
    float m[V];
    P::load(y + p.coarse, m);
#pragma unroll
    for (int k = 0; k < V; k++) s[k] = m[k] > 0.f ? s[k] : 0.f;
    P::store(masked + p.coarse, s);
}

__global__ void __launch_bounds__(256) k_mse(const float *p, const float *t, const float *mask, float *dp, float *loss,
                                             int n, int c, int h, int wd, float norm)
{
    __shared__ float red[256];
    const int64_t plane = (int64_t)h * wd, count = (int64_t)n * c * plane;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    float l = 0.f;
    if (i < count)
    {
        const int64_t img = i / (c * plane), pix = i % plane;
        const float m = mask[img * plane + pix];
        const float d = m * (p[i] - t[i]);
        dp[i] = 2.f * d / norm;
        l = d * d / norm;
    }
    red[threadIdx.x] = l;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1)
    {
        if ((int)threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) atomicAdd(loss, red[0]);
}

struct AdamRates
{
    float lr, b1, b2, eps, c1, c2;
};
__device__ __forceinline__ void adam_one(float *w, const float *g, float *m, float *v, uint16_t *w16, int64_t i,
                                         const AdamRates &a)
{
    const float gi = g[i];
    const float mi = a.b1 * m[i] + (1.f - a.b1) * gi;
    const float vi = a.b2 * v[i] + (1.f - a.b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - a.lr * (mi / a.c1) / (sqrtf(vi / a.c2) + a.eps);
    w[i] = wi;
    if (w16) w16[i] = __bfloat16_as_ushort(__float2bfloat16_rn(wi));
}

// One launch for up to kListed tensors: block b belongs to the last tensor whose
// first block is not after b.  The network's 22 tensors took 22 launches of 3 to
// 6 us for the update and 22 of 2 us to clear the gradients; one of each: 19 and 10.
constexpr int kListed = 32;
struct TensorList
{
    cnn_tensor t[kListed];
    unsigned first[kListed]; // block
    int count;
};
__device__ __forceinline__ bool listed(const TensorList &list, int &k, int64_t &i)
{
    k = 0;
    while (k + 1 < list.count && blockIdx.x >= list.first[k + 1]) k++;
    i = (int64_t)(blockIdx.x - list.first[k]) * blockDim.x + threadIdx.x;
    return i < list.t[k].count;
}

__global__ void __launch_bounds__(256) k_adam(const __grid_constant__ TensorList list, AdamRates rates)
{
    int k;
    int64_t i;
    if (!listed(list, k, i)) return;
    const cnn_tensor &t = list.t[k];
    adam_one(t.w, t.g, t.m, t.v, t.w16, i, rates);
}

__global__ void __launch_bounds__(256) k_zero_grad(const __grid_constant__ TensorList list)
{
    int k;
    int64_t i;
    if (listed(list, k, i)) list.t[k].g[i] = 0.f;
}

__global__ void k_to_bf16(const float *x, uint16_t *y, int64_t count)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) y[i] = __bfloat16_as_ushort(__float2bfloat16_rn(x[i]));
}

int done()
{
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? 0 : -(int)e;
}

unsigned blocks(int64_t count) { return (unsigned)((count + 255) / 256); }

// f(index type, pixels per thread, threads): two coarse pixels a thread where the
// coarse width is even and all addresses (or'd together) are on 16 bytes
template <typename F> int each_coarse(int64_t rows, int w, uintptr_t addresses, F f)
{
    const int64_t count = rows * w;
    const bool narrow = 4 * count + 1024 < (int64_t)1 << 32;
    if (w % 2 == 0 && addresses % 16 == 0)
    {
        if (narrow) f(uint32_t(), std::integral_constant<int, 2>(), count / 2);
        else f(int64_t(), std::integral_constant<int, 2>(), count / 2);
    }
    else
    {
        if (narrow) f(uint32_t(), std::integral_constant<int, 1>(), count);
        else f(int64_t(), std::integral_constant<int, 1>(), count);
    }
    return done();
}
inline uintptr_t address(const void *p) { return (uintptr_t)p; }

// the list in launches of up to kListed tensors
template <typename F> int each_listed(const cnn_tensor *tensors, int count, F launch)
{
    TensorList list;
    int64_t total = 0;
    list.count = 0;
    for (int k = 0; k < count; k++)
    {
        const int64_t n = ((tensors[k].count > 0 ? tensors[k].count : 0) + 255) / 256;
        if (list.count == kListed || total + n > INT32_MAX)
        {
            if (total) launch(list, (unsigned)total);
            list.count = 0;
            total = 0;
        }
        if (n == 0) continue;
        list.t[list.count] = tensors[k];
        list.first[list.count++] = (unsigned)total;
        total += n;
    }
    if (total) launch(list, (unsigned)total);
    return done();
}

// the tensor-core convolutions take more than 48 KB of dynamic shared memory
int tc_attributes()
{
    static int rc = 1;
    if (rc == 1)
    {
        cudaError_t e = cudaFuncSetAttribute(cnn_tc::k_conv3x3_tc<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)cnn_tc::kSmemBytes);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(cnn_tc::k_conv3x3_tc<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)cnn_tc::kSmemBytes);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(cnn_tc::k_conv3x3_wgrad_tc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)cnn_tc::kWSmemBytes);
        rc = e == cudaSuccess ? 0 : -(int)e;
    }
    return rc;
}

// output channels per CTA of the tensor-core convolutions: all (up to 256) when
// the pixel tiles alone fill the GPU, else fewer (multiples of 16), so that the
// launch has about two CTAs per SM
int tc_ntile(int pixel_ctas, int cout)
{
    static int sms = 0;
    if (!sms)
    {
        int dev = 0;
        sms = 148;
        if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    }
    int nt = std::min(cout, cnn_tc::kNMax);
    nt = (nt + 15) & ~15;
    while (nt > 16 && (int64_t)pixel_ctas * ((cout + nt - 1) / nt) < 2 * sms) nt = ((nt / 2) + 15) & ~15;
    return nt;
}

// SMs of the current device, asked for once per device
int sm_count()
{
    static std::atomic<int> known[64];
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) != cudaSuccess) return sms;
    std::atomic<int> *slot = dev < 64 ? &known[dev] : nullptr;
    if (slot && slot->load(std::memory_order_relaxed)) return slot->load(std::memory_order_relaxed);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && slot)
        slot->store(sms, std::memory_order_relaxed);
    return sms;
}

// raises a kernel's dynamic shared memory limit, once per device
cudaError_t allow_smem(const void *kernel, size_t bytes, std::atomic<uint64_t> &done)
{
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = 1ull << (dev & 63);
    if (done.load(std::memory_order_relaxed) & bit) return cudaSuccess;
    const cudaError_t r = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (r == cudaSuccess) done.fetch_or(bit, std::memory_order_relaxed);
    return r;
}

template <typename T, bool TRANSPOSE>
int launch_conv(const float *x, const uint16_t *w, const float *b, float *y, const float *extra, float *y2, int n, int cin,
                int cout, int h, int wd, int relu, cudaStream_t st)
{
    static std::atomic<uint64_t> ready{0};
    const auto kernel = cnn_fma::k_conv3x3_fma<T, TRANSPOSE>;
    const cudaError_t e = allow_smem((const void *)kernel, T::kSmem, ready);
    if (e != cudaSuccess) return -(int)e;
    const dim3 grid((unsigned)(((wd + T::TW - 1) / T::TW) * ((h + T::TH - 1) / T::TH)),
                    (unsigned)((cout + T::CO - 1) / T::CO), (unsigned)n);
    kernel<<<grid, T::kThreads, T::kSmem, st>>>(x, w, b, y, extra, y2, cin, cout, h, wd, relu);
    return done();
}

// Register tiles of the FP32 convolutions, largest first: 512 pixels x 32
// channels (64 sums a thread), 256 x 32 (32), 128 x 32 (16), 64 x 16 (8), and
// 256 x 8 for layers of few output channels.
using ConvA = cnn_fma::ConvTile<32, 16, 2, 4, 8, 8>;
using ConvB = cnn_fma::ConvTile<32, 8, 1, 4, 8, 8>;
using ConvC = cnn_fma::ConvTile<16, 8, 1, 8, 4, 8>;
using ConvD = cnn_fma::ConvTile<8, 8, 1, 8, 2, 16>;
using ConvE = cnn_fma::ConvTile<32, 8, 1, 2, 4, 8>;

// Time of a tile on a layer in units of one FMA per sum: rounds of blocks over
// the SMs x sums per block x the tile's cost per FMA, which comes from sweeps of
// every tile over the network's layers (a full GPU of A runs at 45-51 TFLOP/s, B
// 43-50, C 29-34, D 20; layers that fill the GPU with A fall to 5-10 TFLOP/s at
// 16^2 and 8^2 pixels, where C and D reach 25 and 12.5)
template <typename T> double conv_cost(int n, int cout, int h, int wd, int sms, double per_fma)
{
    const int64_t blocks = (int64_t)((wd + T::TW - 1) / T::TW) * ((h + T::TH - 1) / T::TH) * ((cout + T::CO - 1) / T::CO) * n;
    return (double)((blocks + sms - 1) / sms) * T::ACC * T::kThreads * per_fma;
}

template <bool TRANSPOSE>
int conv(const float *x, const uint16_t *w, const float *b, float *y, const float *extra, float *y2, int n, int cin,
         int cout, int h, int wd, int relu, cudaStream_t st)
{
    const int sms = sm_count();
    const double cost[5] = {conv_cost<ConvA>(n, cout, h, wd, sms, 1.0), conv_cost<ConvB>(n, cout, h, wd, sms, 1.06),
                            conv_cost<ConvC>(n, cout, h, wd, sms, 1.5), conv_cost<ConvD>(n, cout, h, wd, sms, 2.3),
                            conv_cost<ConvE>(n, cout, h, wd, sms, 1.5)};
    switch ((int)(std::min_element(cost, cost + 5) - cost))
    {
    case 0: return launch_conv<ConvA, TRANSPOSE>(x, w, b, y, extra, y2, n, cin, cout, h, wd, relu, st);
    case 1: return launch_conv<ConvB, TRANSPOSE>(x, w, b, y, extra, y2, n, cin, cout, h, wd, relu, st);
    case 2: return launch_conv<ConvC, TRANSPOSE>(x, w, b, y, extra, y2, n, cin, cout, h, wd, relu, st);
    case 3: return launch_conv<ConvD, TRANSPOSE>(x, w, b, y, extra, y2, n, cin, cout, h, wd, relu, st);
    default: return launch_conv<ConvE, TRANSPOSE>(x, w, b, y, extra, y2, n, cin, cout, h, wd, relu, st);
    }
}

// two blocks per SM share a channel group's pixel tiles
int64_t wgrad_split(int64_t groups, int64_t tiles, int sms)
{
    return std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(tiles, 65535), 2 * sms / groups));
}

template <typename T>
int launch_wgrad(const float *x, const float *dy, float *dw, float *db, int n, int cin, int cout, int h, int wd,
                 cudaStream_t st)
{
    static std::atomic<uint64_t> ready{0};
    const auto kernel = cnn_fma::k_conv3x3_wgrad_fma<T>;
    const cudaError_t e = allow_smem((const void *)kernel, T::kSmem, ready);
    if (e != cudaSuccess) return -(int)e;
    const int64_t groups = (int64_t)((cout + T::CO - 1) / T::CO) * ((cin + T::LCI - 1) / T::LCI);
    const int64_t tiles = (int64_t)((wd + T::TW - 1) / T::TW) * ((h + T::TH - 1) / T::TH) * n;
    kernel<<<dim3((unsigned)groups, (unsigned)wgrad_split(groups, tiles, sm_count())), cnn_fma::kThreads, T::kSmem, st>>>(x, dy, dw, db, n, cin, cout, h, wd);
    return done();
}

// The weight gradient's tile for a layer by a model of its time, in packed FMAs of a
// thread: rounds of blocks over the SMs, each block's tiles one after the other (FMAs of
// its thread, 41 per copy of inputs and 31 of gradients that a thread stages; two blocks
// on an SM halve its rate; no tile below 182), and the sums at the end.  The numbers
// are fitted to every tile's times on 634 layers.
struct WgradChoice
{
    typedef int (*Launch)(const float *, const float *, float *, float *, int, int, int, int, int, cudaStream_t);
    int n, cin, cout, h, wd, sms;
    double cost = 0.0, limit = 0.0;
    Launch launch = nullptr;
    template <typename T> double time() const
    {
        const int64_t groups = (int64_t)((cout + T::CO - 1) / T::CO) * ((cin + T::LCI - 1) / T::LCI);
        const int64_t tiles = (int64_t)((wd + T::TW - 1) / T::TW) * ((h + T::TH - 1) / T::TH) * n;
        const int64_t split = wgrad_split(groups, tiles, sms), blocks = groups * split;
        const double share = blocks <= sms ? 1.0 : 2.0, rounds = (double)std::max<int64_t>(1, (blocks + 2 * sms - 1) / (2 * sms));
        const double fma = 18.0 * T::TW * T::TH / T::SPLIT;
        const double x = T::LCI * (T::TH + 2) * (wd % 4 == 0 ? T::TW / 4 + 2 : T::TW + 2) / (double)cnn_fma::kThreads;
        const double y = T::CO * T::TW * T::TH / (double)cnn_fma::kThreads;
        const double tile = std::max(182.0, share * (fma + 41.0 * x + 31.0 * y));
        return rounds * (double)((tiles + split - 1) / split) * tile + 35.0 + 3.1 * T::CO * T::RUN / cnn_fma::kThreads;
    }
    template <typename T> void start()
    {
        cost = time<T>();
        // (where every block has one tile and all run at once, the model is closer)
        const int64_t groups = (int64_t)((cout + T::CO - 1) / T::CO) * ((cin + T::LCI - 1) / T::LCI);
        const int64_t tiles = (int64_t)((wd + T::TW - 1) / T::TW) * ((h + T::TH - 1) / T::TH) * n;
        limit = (groups * tiles <= 2 * sms ? 0.8 : 0.575) * cost;
        launch = launch_wgrad<T>;
    }
    template <typename T> void other()
    {
        const double c = time<T>();
        if (c >= limit || c >= cost) return;
        cost = c;
        launch = launch_wgrad<T>;
    }
};
} // namespace

extern "C" {

int cnn_conv3x3_forward(const float *x, const uint16_t *w, const float *b, float *y, int n, int cin, int cout, int h,
                        int wd, int relu, void *stream)
{
    if (n <= 0 || cin <= 0 || cout <= 0 || h <= 0 || wd <= 0) return -1;
    return conv<false>(x, w, b, y, nullptr, nullptr, n, cin, cout, h, wd, relu, (cudaStream_t)stream);
}

int cnn_conv3x3_forward_add(const float *x, const uint16_t *w, const float *b, float *y, const float *skip, float *sum,
                            int n, int cin, int cout, int h, int wd, int relu, void *stream)
{
    if (n <= 0 || cin <= 0 || cout <= 0 || h <= 0 || wd <= 0 || !skip || !sum) return -1;
    return conv<false>(x, w, b, y, skip, sum, n, cin, cout, h, wd, relu, (cudaStream_t)stream);
}

int cnn_conv3x3_backward_data(const float *dy, const uint16_t *w, float *dx, int n, int cin, int cout, int h, int wd,
                              void *stream)
{
    if (n <= 0 || cin <= 0 || cout <= 0 || h <= 0 || wd <= 0) return -1;
    // a convolution from the cout gradient channels to the cin input channels
    return conv<true>(dy, w, nullptr, dx, nullptr, nullptr, n, cout, cin, h, wd, 0, (cudaStream_t)stream);
}

int cnn_conv3x3_backward_data_relu(const float *dy, const uint16_t *w, float *dx, const float *x, float *masked, int n,
                                   int cin, int cout, int h, int wd, void *stream)
{
    if (n <= 0 || cin <= 0 || cout <= 0 || h <= 0 || wd <= 0 || !x || !masked) return -1;
    return conv<true>(dy, w, nullptr, dx, x, masked, n, cout, cin, h, wd, 0, (cudaStream_t)stream);
}

int cnn_conv3x3_forward_tc(const float *x, const uint16_t *w, const float *b, float *y, int n, int cin, int cout,
                           int h, int wd, int relu, void *stream)
{
    if (n <= 0 || cin <= 0 || cout <= 0 || h <= 0 || wd <= 0) return -1;
    const int rc = tc_attributes();
    if (rc) return rc;
    const int tiles = (h * wd + cnn_tc::kM - 1) / cnn_tc::kM;
    const int nt = tc_ntile(tiles * n, cout);
    const dim3 grid((unsigned)tiles, (unsigned)((cout + nt - 1) / nt), (unsigned)n);
    cnn_tc::k_conv3x3_tc<false><<<grid, cnn_tc::kThreads, cnn_tc::kSmemBytes, (cudaStream_t)stream>>>(
        x, w, b, y, cin, cout, h, wd, relu, nt);
    return done();
}

int cnn_conv3x3_backward_data_tc(const float *dy, const uint16_t *w, float *dx, int n, int cin, int cout, int h, int wd,
                                 void *stream)
{
    if (n <= 0 || cin <= 0 || cout <= 0 || h <= 0 || wd <= 0) return -1;
    const int rc = tc_attributes();
    if (rc) return rc;
    const int tiles = (h * wd + cnn_tc::kM - 1) / cnn_tc::kM;
    const int nt = tc_ntile(tiles * n, cin);
    const dim3 grid((unsigned)tiles, (unsigned)((cin + nt - 1) / nt), (unsigned)n);
    // a convolution from the cout gradient channels to the cin input channels
    cnn_tc::k_conv3x3_tc<true><<<grid, cnn_tc::kThreads, cnn_tc::kSmemBytes, (cudaStream_t)stream>>>(
        dy, w, nullptr, dx, cout, cin, h, wd, 0, nt);
    return done();
}

int cnn_conv3x3_backward_weight_tc(const float *x, const float *dy, float *dw, float *db, int n, int cin, int cout,
                                   int h, int wd, void *stream)
{
    if (n <= 0 || cin <= 0 || cout <= 0 || h <= 0 || wd <= 0) return -1;
    const int rc = tc_attributes();
    if (rc) return rc;
    const int64_t total = (int64_t)n * h * wd;
    const int mt = (cout + cnn_tc::kM - 1) / cnn_tc::kM, nt = (cin + cnn_tc::kCC - 1) / cnn_tc::kCC;
    // split K: about four CTAs per SM over the whole launch, slices of at least
    // 1024 pixels (a multiple of the 64-pixel chunk)
    int sms = 148;
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int64_t slices = std::max<int64_t>(1, (int64_t)4 * sms / (mt * nt));
    int64_t slice = (total + slices - 1) / slices;
    slice = std::max<int64_t>(1024, (slice + cnn_tc::kWK - 1) / cnn_tc::kWK * cnn_tc::kWK);
    slices = (total + slice - 1) / slice;
    const dim3 grid((unsigned)mt, (unsigned)nt, (unsigned)slices);
    cnn_tc::k_conv3x3_wgrad_tc<<<grid, cnn_tc::kThreads, cnn_tc::kWSmemBytes, (cudaStream_t)stream>>>(
        x, dy, dw, n, cin, cout, h, wd, (int)slice);
    if (db) cnn_tc::k_bias_grad<<<cout, 256, 0, (cudaStream_t)stream>>>(dy, db, n, cout, h * wd);
    return done();
}

int cnn_tc_error(void)
{
    unsigned int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, cnn_tc::g_tc_error, sizeof(v)) != cudaSuccess) return -1;
    if (v && cudaMemcpyToSymbol(cnn_tc::g_tc_error, &zero, sizeof(zero)) != cudaSuccess) return -1;
    return (int)v;
}

int cnn_conv3x3_backward_weight(const float *x, const float *dy, float *dw, float *db, int n, int cin, int cout, int h,
                                int wd, void *stream)
{
    if (n <= 0 || cin <= 0 || cout <= 0 || h <= 0 || wd <= 0) return -1;
    const cudaStream_t st = (cudaStream_t)stream;
    using namespace cnn_fma;
    WgradChoice pick{n, cin, cout, h, wd, sm_count()};
    // 16 x 8 pixel tiles and 32 x 32 channels, 8 x 8 where the image is no wider; with few
    // output (input) channels the warps (lanes) share the pixels instead of channels
    if (cout <= 8)
    {
        if (wd > 8) pick.start<WgradTile<16, 8, 1, 32>>();
        else pick.start<WgradTile<8, 8, 1, 32>>();
    }
    else if (cin <= 4) pick.start<WgradTile<16, 8, 8, 4>>();
    else if (wd > 8) pick.start<WgradTile<16, 8, 8, 32>>();
    else pick.start<WgradTile<8, 8, 8, 32>>();
    // Smaller tiles where few blocks, or channels that are not there, leave those waiting: 4
    // or 8 output channels x 8 input channels, 16 x 16 on 16 x 8 or 8 x 8 pixels.  Only where
    // the model sees a good deal to gain: of 634 layers (1 to 8 images, 1 to 256 channels, 4 to
    // 140 pixels) none was more than 1.5 % slower for it, and the choice is 4 % from the best of 21
    // tiles on the average (30 % without).  us, with the tile above / now / with tiles of 16^2 pixels and
    // channels before these kernels: 11 -> 34 channels at 57^2 (5 images) 33 / 19 / 22, 34 -> 13 at 102 x 25
    // (6) 33 / 19 / 23, 2 -> 5 at 129^2 (8) 50 / 17 / 40, 251 -> 12 at 20^2 (6) 22 / 14.5 / 28.
    pick.other<WgradTile<16, 8, 1, 8>>();
    pick.other<WgradTile<16, 8, 2, 8>>();
    pick.other<WgradTile<16, 8, 4, 16>>();
    pick.other<WgradTile<8, 8, 4, 16>>();
    return pick.launch(x, dy, dw, db, n, cin, cout, h, wd, st);
}

int cnn_relu_backward(float *dy, const float *y, int64_t count, void *stream)
{
    if (count <= 0) return 0;
    k_relu_bw<<<blocks(count), 256, 0, (cudaStream_t)stream>>>(dy, y, count);
    return done();
}

int cnn_avgpool2_forward(const float *x, float *y, int nc, int h, int wd, void *stream)
{
    if (nc <= 0 || h <= 0 || wd <= 0 || h % 2 || wd % 2) return -1;
    return each_coarse((int64_t)nc * (h / 2), wd / 2, address(x) | address(y), [&](auto i, auto v, int64_t count) {
        typedef decltype(i) I;
        k_pool_fw<I, v><<<blocks(count), 256, 0, (cudaStream_t)stream>>>(x, y, (I)count, wd / 2);
    });
}

int cnn_avgpool2_backward(const float *dy, float *dx, int nc, int h, int wd, void *stream)
{
    if (nc <= 0 || h <= 0 || wd <= 0 || h % 2 || wd % 2) return -1;
    return each_coarse((int64_t)nc * (h / 2), wd / 2, address(dy) | address(dx), [&](auto i, auto v, int64_t count) {
        typedef decltype(i) I;
        k_pool_bw<I, v><<<blocks(count), 256, 0, (cudaStream_t)stream>>>(dy, dx, (I)count, wd / 2);
    });
}

int cnn_avgpool2_backward_add_relu(const float *dy, const float *y, float *dx, int nc, int h, int wd, void *stream)
{
    if (nc <= 0 || h <= 0 || wd <= 0 || h % 2 || wd % 2) return -1;
    return each_coarse((int64_t)nc * (h / 2), wd / 2, address(dy) | address(y) | address(dx),
                       [&](auto i, auto v, int64_t count) {
                           typedef decltype(i) I;
                           k_pool_bw_add_relu<I, v><<<blocks(count), 256, 0, (cudaStream_t)stream>>>(dy, y, dx, (I)count, wd / 2);
                       });
}

int cnn_upsample2_forward(const float *x, float *y, int nc, int h, int wd, void *stream)
{
    if (nc <= 0 || h <= 0 || wd <= 0) return -1;
    return each_coarse((int64_t)nc * h, wd, address(x) | address(y), [&](auto i, auto v, int64_t count) {
        typedef decltype(i) I;
        k_up_fw<I, v><<<blocks(count), 256, 0, (cudaStream_t)stream>>>(x, y, (I)count, wd);
    });
}

static int upsample2_backward(const float *dy, float *dx, const float *y, float *masked, int nc, int h, int wd, void *stream)
{
    if (nc <= 0 || h <= 0 || wd <= 0) return -1;
    return each_coarse((int64_t)nc * h, wd, address(dy) | address(dx) | address(y) | address(masked),
                       [&](auto i, auto v, int64_t count) {
                           typedef decltype(i) I;
                           k_up_bw<I, v><<<blocks(count), 256, 0, (cudaStream_t)stream>>>(dy, dx, y, masked, (I)count, wd);
                       });
}

int cnn_upsample2_backward(const float *dy, float *dx, int nc, int h, int wd, void *stream)
{
    return upsample2_backward(dy, dx, nullptr, nullptr, nc, h, wd, stream);
}

int cnn_upsample2_backward_relu(const float *dy, float *dx, const float *y, float *masked, int nc, int h, int wd, void *stream)
{
    if (!y || !masked) return -1;
    return upsample2_backward(dy, dx, y, masked, nc, h, wd, stream);
}

int cnn_add(float *y, const float *x, int64_t count, void *stream)
{
    if (count <= 0) return 0;
    k_add<<<blocks(count), 256, 0, (cudaStream_t)stream>>>(y, x, count);
    return done();
}

int cnn_mse(const float *p, const float *t, const float *mask, float *dp, float *loss, int n, int c, int h, int wd,
            float norm, void *stream)
{
    if (n <= 0 || c <= 0 || h <= 0 || wd <= 0 || !(norm > 0.f)) return -1;
    k_mse<<<blocks((int64_t)n * c * h * wd), 256, 0, (cudaStream_t)stream>>>(p, t, mask, dp, loss, n, c, h, wd, norm);
    return done();
}

int cnn_adam_many(const cnn_tensor *tensors, int count, float lr, float beta1, float beta2, float eps, int step, void *stream)
{
    if (step < 1) return -1;
    const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
    return each_listed(tensors, count, [&](const TensorList &list, unsigned blocks) {
        k_adam<<<blocks, 256, 0, (cudaStream_t)stream>>>(list, AdamRates{lr, beta1, beta2, eps, c1, c2});
    });
}

int cnn_adam(float *w, const float *g, float *m, float *v, uint16_t *w16, int64_t count, float lr, float beta1,
             float beta2, float eps, int step, void *stream)
{
    if (count <= 0) return 0;
    const cnn_tensor t{w, const_cast<float *>(g), m, v, w16, count};
    return cnn_adam_many(&t, 1, lr, beta1, beta2, eps, step, stream);
}

int cnn_zero_grad_many(const cnn_tensor *tensors, int count, void *stream)
{
    return each_listed(tensors, count, [&](const TensorList &list, unsigned blocks) {
        k_zero_grad<<<blocks, 256, 0, (cudaStream_t)stream>>>(list);
    });
}

int cnn_to_bf16(const float *x, uint16_t *y, int64_t count, void *stream)
{
    if (count <= 0) return 0;
    k_to_bf16<<<blocks(count), 256, 0, (cudaStream_t)stream>>>(x, y, count);
    return done();
}
} // extern "C"
