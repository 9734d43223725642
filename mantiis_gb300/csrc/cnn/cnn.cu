// Kernels of the warm-start encoder-decoder network (include/mantiis_cnn.h):
// 3x3 convolutions (forward, data gradient, weight gradient) with BF16
// weights and FP32 accumulation, pooling / upsampling / ReLU adjoints, the
// masked loss and the Adam update.  sm_103a.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>

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

// per (image * channel) plane: y (h/2, wd/2) = mean of the 2x2 blocks
__global__ void k_pool_fw(const float *x, float *y, int nc, int h, int wd)
{
    const int ho = h / 2, wo = wd / 2;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)nc * ho * wo) return;
    const int64_t c = i / ((int64_t)ho * wo);
    const int r = (int)(i % ((int64_t)ho * wo)), yy = r / wo, xx = r % wo;
    const float *p = x + c * h * wd + (int64_t)(2 * yy) * wd + 2 * xx;
    y[i] = 0.25f * (p[0] + p[1] + p[wd] + p[wd + 1]);
}

__global__ void k_pool_bw(const float *dy, float *dx, int nc, int h, int wd)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)nc * h * wd) return;
    const int64_t c = i / ((int64_t)h * wd);
    const int r = (int)(i % ((int64_t)h * wd)), yy = r / wd, xx = r % wd;
    dx[i] = 0.25f * dy[c * (h / 2) * (wd / 2) + (int64_t)(yy / 2) * (wd / 2) + xx / 2];
}

// nearest upsampling of an (h, wd) map to (2h, 2wd)
__global__ void k_up_fw(const float *x, float *y, int nc, int h, int wd)
{
    const int ho = 2 * h, wo = 2 * wd;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)nc * ho * wo) return;
    const int64_t c = i / ((int64_t)ho * wo);
    const int r = (int)(i % ((int64_t)ho * wo)), yy = r / wo, xx = r % wo;
    y[i] = x[c * h * wd + (int64_t)(yy / 2) * wd + xx / 2];
}

__global__ void k_up_bw(const float *dy, float *dx, int nc, int h, int wd)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)nc * h * wd) return;
    const int64_t c = i / ((int64_t)h * wd);
    const int r = (int)(i % ((int64_t)h * wd)), yy = r / wd, xx = r % wd;
    const int wo = 2 * wd;
    const float *p = dy + c * (4 * (int64_t)h * wd) + (int64_t)(2 * yy) * wo + 2 * xx;
    dx[i] = p[0] + p[1] + p[wo] + p[wo + 1];
}

__global__ void k_add(float *y, const float *x, int64_t count)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) y[i] += x[i];
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

__global__ void k_adam(float *w, const float *g, float *m, float *v, uint16_t *w16, int64_t count, float lr, float b1,
                       float b2, float eps, float c1, float c2)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    w[i] = wi;
    if (w16) w16[i] = __bfloat16_as_ushort(__float2bfloat16_rn(wi));
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

int sm_count()
{
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
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
int launch_conv(const float *x, const uint16_t *w, const float *b, float *y, int n, int cin, int cout, int h, int wd,
                int relu, cudaStream_t st)
{
    static std::atomic<uint64_t> ready{0};
    const auto kernel = cnn_fma::k_conv3x3_fma<T, TRANSPOSE>;
    const cudaError_t e = allow_smem((const void *)kernel, T::kSmem, ready);
    if (e != cudaSuccess) return -(int)e;
    const dim3 grid((unsigned)(((wd + T::TW - 1) / T::TW) * ((h + T::TH - 1) / T::TH)),
                    (unsigned)((cout + T::CO - 1) / T::CO), (unsigned)n);
    kernel<<<grid, T::kThreads, T::kSmem, st>>>(x, w, b, y, cin, cout, h, wd, relu);
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
int conv(const float *x, const uint16_t *w, const float *b, float *y, int n, int cin, int cout, int h, int wd, int relu,
         cudaStream_t st)
{
    const int sms = sm_count();
    const double cost[5] = {conv_cost<ConvA>(n, cout, h, wd, sms, 1.0), conv_cost<ConvB>(n, cout, h, wd, sms, 1.06),
                            conv_cost<ConvC>(n, cout, h, wd, sms, 1.5), conv_cost<ConvD>(n, cout, h, wd, sms, 2.3),
                            conv_cost<ConvE>(n, cout, h, wd, sms, 1.5)};
    switch ((int)(std::min_element(cost, cost + 5) - cost))
    {
    case 0: return launch_conv<ConvA, TRANSPOSE>(x, w, b, y, n, cin, cout, h, wd, relu, st);
    case 1: return launch_conv<ConvB, TRANSPOSE>(x, w, b, y, n, cin, cout, h, wd, relu, st);
    case 2: return launch_conv<ConvC, TRANSPOSE>(x, w, b, y, n, cin, cout, h, wd, relu, st);
    case 3: return launch_conv<ConvD, TRANSPOSE>(x, w, b, y, n, cin, cout, h, wd, relu, st);
    default: return launch_conv<ConvE, TRANSPOSE>(x, w, b, y, n, cin, cout, h, wd, relu, st);
    }
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
    // two blocks per SM share a channel group's pixel tiles
    const int64_t split = std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(tiles, 65535), 2 * sm_count() / groups));
    kernel<<<dim3((unsigned)groups, (unsigned)split), cnn_fma::kThreads, T::kSmem, st>>>(x, dy, dw, db, n, cin, cout, h, wd);
    return done();
}
} // namespace

extern "C" {

int cnn_conv3x3_forward(const float *x, const uint16_t *w, const float *b, float *y, int n, int cin, int cout, int h,
                        int wd, int relu, void *stream)
{
    if (n <= 0 || cin <= 0 || cout <= 0 || h <= 0 || wd <= 0) return -1;
    return conv<false>(x, w, b, y, n, cin, cout, h, wd, relu, (cudaStream_t)stream);
}

int cnn_conv3x3_backward_data(const float *dy, const uint16_t *w, float *dx, int n, int cin, int cout, int h, int wd,
                              void *stream)
{
    if (n <= 0 || cin <= 0 || cout <= 0 || h <= 0 || wd <= 0) return -1;
    // a convolution from the cout gradient channels to the cin input channels
    return conv<true>(dy, w, nullptr, dx, n, cout, cin, h, wd, 0, (cudaStream_t)stream);
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
    // 16 x 8 pixel tiles, 8 x 8 where the image is no wider; with few output
    // (input) channels the warps (lanes) share the pixels instead of channels
    using namespace cnn_fma;
    if (cout <= 8)
        return wd > 8 ? launch_wgrad<WgradTile<16, 8, 1, 32>>(x, dy, dw, db, n, cin, cout, h, wd, st)
                      : launch_wgrad<WgradTile<8, 8, 1, 32>>(x, dy, dw, db, n, cin, cout, h, wd, st);
    if (cin <= 4) return launch_wgrad<WgradTile<16, 8, 8, 4>>(x, dy, dw, db, n, cin, cout, h, wd, st);
    return wd > 8 ? launch_wgrad<WgradTile<16, 8, 8, 32>>(x, dy, dw, db, n, cin, cout, h, wd, st)
                  : launch_wgrad<WgradTile<8, 8, 8, 32>>(x, dy, dw, db, n, cin, cout, h, wd, st);
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
    k_pool_fw<<<blocks((int64_t)nc * h * wd / 4), 256, 0, (cudaStream_t)stream>>>(x, y, nc, h, wd);
    return done();
}

int cnn_avgpool2_backward(const float *dy, float *dx, int nc, int h, int wd, void *stream)
{
    if (nc <= 0 || h <= 0 || wd <= 0 || h % 2 || wd % 2) return -1;
    k_pool_bw<<<blocks((int64_t)nc * h * wd), 256, 0, (cudaStream_t)stream>>>(dy, dx, nc, h, wd);
    return done();
}

int cnn_upsample2_forward(const float *x, float *y, int nc, int h, int wd, void *stream)
{
    if (nc <= 0 || h <= 0 || wd <= 0) return -1;
    k_up_fw<<<blocks((int64_t)nc * h * wd * 4), 256, 0, (cudaStream_t)stream>>>(x, y, nc, h, wd);
    return done();
}

int cnn_upsample2_backward(const float *dy, float *dx, int nc, int h, int wd, void *stream)
{
    if (nc <= 0 || h <= 0 || wd <= 0) return -1;
    k_up_bw<<<blocks((int64_t)nc * h * wd), 256, 0, (cudaStream_t)stream>>>(dy, dx, nc, h, wd);
    return done();
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

int cnn_adam(float *w, const float *g, float *m, float *v, uint16_t *w16, int64_t count, float lr, float beta1,
             float beta2, float eps, int step, void *stream)
{
    if (count <= 0) return 0;
    if (step < 1) return -1;
    const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
    k_adam<<<blocks(count), 256, 0, (cudaStream_t)stream>>>(w, g, m, v, w16, count, lr, beta1, beta2, eps, c1, c2);
    return done();
}

int cnn_to_bf16(const float *x, uint16_t *y, int64_t count, void *stream)
{
    if (count <= 0) return 0;
    k_to_bf16<<<blocks(count), 256, 0, (cudaStream_t)stream>>>(x, y, count);
    return done();
}
} // extern "C"
