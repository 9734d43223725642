// 3x3 convolutions on the FP32 pipe, register tiled: forward and data gradient
// (k_conv3x3_fma) and weight gradient (k_conv3x3_wgrad_fma).  Activations FP32
// NCHW, weights BF16, FP32 accumulation.
//
// What bounds them is the FP32 pipe (128 FMA per clock and SM) as long as the
// operands come out of shared memory fast enough.  A thread therefore keeps a
// tile of outputs in registers: per input channel it reads (PY + 2) x 6 inputs
// once for its 4 x PY pixels and 9 x CT weights (the same for a whole warp, so
// broadcast), and makes PY x 4 x CT x 9 FMAs with them, two to an instruction
// (fma.rn.f32x2), which leaves issue slots for the loads.  Measured on a GB300
// (8 images, 32 -> 32 channels at 128^2 / 256 -> 128 at 32^2 / 256 -> 256 at
// 16^2 pixels): forward 55 / 123 / 94 us (44 / 39 / 26 TFLOP/s), weight gradient
// 60 / 119 / 68 us; with one pixel x 16 channels a thread, one shared-memory
// load per FMA, they took 171 / 461 / 226 and 125 / 420 / 218 us.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace cnn_fma
{
constexpr int kPX = 4; // output pixels per thread and row

__device__ __forceinline__ void copy4_async(float *dst, const float *src, bool valid)
{
    // 4-byte asynchronous copy; nothing is read and zero is written where !valid
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int n = valid ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void copy16_async(float *dst, const float *src, bool valid)
{
    // the same for 16 bytes, both addresses on 16 bytes
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int n = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ float bf_float(uint16_t v) { return __uint_as_float((uint32_t)v << 16); }

// two FP32 FMAs in one instruction, each rounded as fmaf
__device__ __forceinline__ void fma2(uint64_t &acc, uint64_t a, uint64_t b)
{
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ void add2(uint64_t &acc, uint64_t a)
{
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(acc) : "l"(a));
}
__device__ __forceinline__ uint64_t both(float v)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float half_of(uint64_t v, int hi)
{
    return __uint_as_float((uint32_t)(hi ? v >> 32 : v));
}

// Tile of one block: TW x TH pixels of one image and CG * CT output channels;
// thread = (pixel group of 4 x PY, channel group of CT).
template <int TW_, int TH_, int PY_, int CG_, int CT_, int CI_> struct ConvTile
{
    static constexpr int TW = TW_, TH = TH_, PY = PY_, CG = CG_, CT = CT_;
    static constexpr int CI = CI_;                       // input channels per chunk
    static constexpr int CO = CG * CT;                   // output channels per block
    static constexpr int NX = TW / kPX, NP = NX * (TH / PY);
    static constexpr int kThreads = NP * CG;
    // a staged row: columns tx0 - 4 .. tx0 + TW + 3, so that the tile's own
    // columns start on 16 bytes
    static constexpr int RS = TW + 8, ROWS = TH + 2;
    static constexpr int XF = CI * ROWS * RS;            // floats of a staged input chunk
    static constexpr int WF = CI * 9 * CO;               // floats of a staged weight chunk
    static constexpr int ACC = PY * kPX * CT;            // accumulators per thread
    static constexpr size_t kSmem = (size_t)2 * (XF + WF) * 4;
    static_assert(kThreads % 32 == 0 && CT % 2 == 0 && CO % 8 == 0 && CI % 8 == 0, "tile");
};

// y[co] = sum_ci sum_k w[co][ci][k] x[ci](p + offset(k)), offsets (kx - 1, ky - 1)
// with k = 3 ky + kx, zero outside the image; summed with ci ascending, then k
// ascending, whatever the tile.  TRANSPOSE: the data gradient of such a
// convolution, i.e. the same with w[ci][co][8 - k]; cin and cout are this
// convolution's own input / output channel counts.  With y2 (y may then be null)
// the pass over the result that follows in the network is done on the way out:
// y2 = y + extra (the decoder's skip connection) or, TRANSPOSE, y2 = y where
// extra > 0, else 0 (the adjoint of the ReLU that gave extra).
template <typename T, bool TRANSPOSE>
__global__ void __launch_bounds__(T::kThreads, 512 / T::kThreads)
    k_conv3x3_fma(const float *__restrict__ x, const uint16_t *__restrict__ w, const float *__restrict__ b,
                  float *__restrict__ y, const float *__restrict__ extra, float *__restrict__ y2, int cin, int cout,
                  int h, int wd, int relu)
{
    extern __shared__ __align__(16) float smem[];
    const int tid = (int)threadIdx.x;
    const int tiles_x = (wd + T::TW - 1) / T::TW;
    const int tx0 = ((int)blockIdx.x % tiles_x) * T::TW, ty0 = ((int)blockIdx.x / tiles_x) * T::TH;
    const int co0 = (int)blockIdx.y * T::CO;
    const int img = (int)blockIdx.z;
    const size_t plane = (size_t)h * wd;
    const float *xi = x + (size_t)img * cin * plane;
    const int pg = tid % T::NP, cg = tid / T::NP;
    const int px = (pg % T::NX) * kPX, py = (pg / T::NX) * T::PY;
    auto sx = [&](int st) { return smem + st * T::XF; };
    auto sw = [&](int st) { return smem + 2 * T::XF + st * T::WF; };

    // Inputs of a chunk: TW / 4 vectors and the two halo columns of each row
    // where rows start on 16 bytes, else single floats.
    const bool xvec = (wd & 3) == 0 && ((uintptr_t)x & 15u) == 0;
    auto stage_x = [&](int ci0, int st) {
        if (xvec)
        {
            constexpr int NV = T::TW / 4 + 2;
            for (int i = tid; i < T::CI * T::ROWS * NV; i += T::kThreads)
            {
                const int v = i % NV, r = i / NV, c = r / T::ROWS, yy = r % T::ROWS;
                const int gy = ty0 + yy - 1, gc = ci0 + c;
                const bool row = gc < cin && gy >= 0 && gy < h;
                const float *src = xi + (row ? (size_t)gc * plane + (size_t)gy * wd : 0);
                float *dst = sx(st) + r * T::RS;
                if (v < T::TW / 4)
                {
                    const bool ok = row && tx0 + 4 * v < wd; // rows are whole vectors
                    copy16_async(dst + 4 + 4 * v, ok ? src + tx0 + 4 * v : x, ok);
                }
                else
                {
                    const int gx = v == T::TW / 4 ? tx0 - 1 : tx0 + T::TW;
                    const bool ok = row && gx >= 0 && gx < wd;
                    copy4_async(dst + (gx - tx0 + 4), ok ? src + gx : x, ok);
                }
            }
        }
        else
            for (int i = tid; i < T::CI * T::ROWS * (T::TW + 2); i += T::kThreads)
            {
                const int v = i % (T::TW + 2), r = i / (T::TW + 2), c = r / T::ROWS, yy = r % T::ROWS;
                const int gy = ty0 + yy - 1, gx = tx0 + v - 1, gc = ci0 + c;
                const bool ok = gc < cin && gy >= 0 && gy < h && gx >= 0 && gx < wd;
                copy4_async(sx(st) + r * T::RS + 3 + v, ok ? xi + (size_t)gc * plane + (size_t)gy * wd + gx : x, ok);
            }
        copies_commit();
    };
    // Weights of a chunk pass through registers: converted, and transposed to
    // [channel][tap][output channel], so that a thread's CT lie together.  In
    // memory the chunk is CO runs of CI * 9 values (TRANSPOSE: CI runs of
    // CO * 9); with channel counts in whole eights these are 16-byte vectors of
    // 8 values (2-byte loads of the same weights took 15 % of the kernel).
    constexpr int RUN = TRANSPOSE ? T::CO * 9 : T::CI * 9, NRUN = TRANSPOSE ? T::CI : T::CO;
    constexpr int NWV = (RUN / 8 * NRUN + T::kThreads - 1) / T::kThreads;
    const bool wvec = (cin & 7) == 0 && (cout & 7) == 0 && ((uintptr_t)w & 15u) == 0;
    uint4 wreg[NWV];
    // vector j of this thread: run `run`, first value 8 * v of it.  TRANSPOSE
    // runs lie across the threads, the others' runs side by side (lane = output
    // channel: conflict-free stores)
    auto wplace = [&](int j, int &run, int &v) {
        const int i = tid + j * T::kThreads;
        run = TRANSPOSE ? i / (RUN / 8) : i % NRUN;
        v = TRANSPOSE ? i % (RUN / 8) : i / NRUN;
        return i < RUN / 8 * NRUN;
    };
    auto load_w = [&](int ci0) {
#pragma unroll
        for (int j = 0; j < NWV; j++)
        {
            int run, v;
            wreg[j] = make_uint4(0, 0, 0, 0);
            if (!wplace(j, run, v)) continue;
            // a run ends with the channels there are (whole eights)
            const int g0 = TRANSPOSE ? ci0 + run : co0 + run, left = TRANSPOSE ? cout - co0 : cin - ci0;
            if (g0 >= (TRANSPOSE ? cin : cout) || 8 * v >= left * 9) continue;
            const size_t at = TRANSPOSE ? ((size_t)g0 * cout + co0) * 9 : ((size_t)g0 * cin + ci0) * 9;
            wreg[j] = __ldg(reinterpret_cast<const uint4 *>(w + at) + v);
        }
    };
    auto store_w = [&](int st) {
#pragma unroll
        for (int j = 0; j < NWV; j++)
        {
            int run, v;
            if (!wplace(j, run, v)) continue;
            const uint32_t u[4] = {wreg[j].x, wreg[j].y, wreg[j].z, wreg[j].w};
#pragma unroll
            for (int e = 0; e < 8; e++)
            {
                const float f = __uint_as_float(e & 1 ? u[e / 2] & 0xffff0000u : u[e / 2] << 16);
                const int q = 8 * v + e;
                if (TRANSPOSE) sw(st)[(run * 9 + 8 - q % 9) * T::CO + q / 9] = f;
                else sw(st)[q * T::CO + run] = f;
            }
        }
    };
    // the same one value at a time, for any channel counts
    auto stage_w_scalar = [&](int ci0, int st) {
        for (int i = tid; i < T::WF; i += T::kThreads)
        {
            const int co = i % T::CO, r = i / T::CO, c = r / 9, k = r % 9;
            const int gco = co0 + co, gci = ci0 + c;
            uint16_t v = 0;
            if (gco < cout && gci < cin)
                v = TRANSPOSE ? __ldg(&w[((size_t)gci * cout + gco) * 9 + (8 - k)])
                              : __ldg(&w[((size_t)gco * cin + gci) * 9 + k]);
            sw(st)[i] = bf_float(v);
        }
    };

    uint64_t acc[T::PY][kPX][T::CT / 2]; // pairs of output channels
#pragma unroll
    for (int a = 0; a < T::PY; a++)
#pragma unroll
        for (int p = 0; p < kPX; p++)
#pragma unroll
            for (int c = 0; c < T::CT / 2; c++) acc[a][p][c] = 0;

    stage_x(0, 0);
    if (wvec)
    {
        load_w(0);
        store_w(0);
    }
    else stage_w_scalar(0, 0);
    copies_wait();
    __syncthreads();
    int st = 0;
    for (int ci0 = 0; ci0 < cin; ci0 += T::CI, st ^= 1)
    {
        const bool more = ci0 + T::CI < cin;
        if (more)
        {
            stage_x(ci0 + T::CI, st ^ 1);
            if (wvec) load_w(ci0 + T::CI);
            else stage_w_scalar(ci0 + T::CI, st ^ 1);
        }
        const int cmax = min(T::CI, cin - ci0);
#pragma unroll 1
        for (int c = 0; c < cmax; c++)
        {
            float xr[T::PY + 2][6];
            const float *px0 = sx(st) + (c * T::ROWS + py) * T::RS + px + 3;
#pragma unroll
            for (int r = 0; r < T::PY + 2; r++)
            {
                const float4 v = *reinterpret_cast<const float4 *>(px0 + r * T::RS + 1);
                xr[r][0] = px0[r * T::RS];
                xr[r][1] = v.x, xr[r][2] = v.y, xr[r][3] = v.z, xr[r][4] = v.w;
                xr[r][5] = px0[r * T::RS + 5];
            }
            const float *wp = sw(st) + c * 9 * T::CO + cg * T::CT;
#pragma unroll
            for (int k = 0; k < 9; k++)
            {
                uint64_t wv[T::CT / 2];
                if (T::CT >= 4)
                {
#pragma unroll
                    for (int o = 0; o < T::CT / 4; o++)
                    {
                        const ulonglong2 q = *reinterpret_cast<const ulonglong2 *>(wp + k * T::CO + 4 * o);
                        wv[2 * o] = q.x;
                        wv[2 * o + 1] = q.y;
                    }
                }
                else wv[0] = *reinterpret_cast<const unsigned long long *>(wp + k * T::CO);
#pragma unroll
                for (int a = 0; a < T::PY; a++)
#pragma unroll
                    for (int p = 0; p < kPX; p++)
                    {
                        const uint64_t xx = both(xr[a + k / 3][p + k % 3]);
#pragma unroll
                        for (int o = 0; o < T::CT / 2; o++) fma2(acc[a][p][o], wv[o], xx);
                    }
            }
        }
        if (more && wvec) store_w(st ^ 1);
        copies_wait();
        __syncthreads();
    }

    const int gx = tx0 + px;
    if (gx >= wd) return;
    // whole groups of 4 pixels are one store where rows start on 16 bytes
    const bool vec = (wd & 3) == 0 && (((uintptr_t)y | (uintptr_t)extra | (uintptr_t)y2) & 15u) == 0;
    auto put = [&](float *dst, const float v[kPX]) {
        if (vec) *reinterpret_cast<float4 *>(dst) = make_float4(v[0], v[1], v[2], v[3]);
        else
        {
#pragma unroll
            for (int p = 0; p < kPX; p++)
                if (gx + p < wd) dst[p] = v[p];
        }
    };
#pragma unroll
    for (int o = 0; o < T::CT; o++)
    {
        const int gco = co0 + cg * T::CT + o;
        if (gco >= cout) break;
        const float bias = b ? __ldg(&b[gco]) : 0.f;
#pragma unroll
        for (int a = 0; a < T::PY; a++)
        {
            const int gy = ty0 + py + a;
            if (gy >= h) break;
            float v[kPX];
#pragma unroll
            for (int p = 0; p < kPX; p++)
            {
                v[p] = half_of(acc[a][p][o / 2], o & 1) + bias;
                if (relu) v[p] = fmaxf(v[p], 0.f);
            }
            const size_t at = ((size_t)img * cout + gco) * plane + (size_t)gy * wd + gx;
            if (y) put(y + at, v);
            if (!y2) continue;
            float e[kPX];
            if (vec)
            {
                const float4 q = *reinterpret_cast<const float4 *>(extra + at);
                e[0] = q.x, e[1] = q.y, e[2] = q.z, e[3] = q.w;
            }
            else
            {
#pragma unroll
                for (int p = 0; p < kPX; p++) e[p] = gx + p < wd ? extra[at + p] : 0.f;
            }
#pragma unroll
            for (int p = 0; p < kPX; p++) v[p] = TRANSPOSE ? (e[p] > 0.f ? v[p] : 0.f) : v[p] + e[p];
            put(y2 + at, v);
        }
    }
}

constexpr int kThreads = 256; // of the weight gradient

// Weight gradient: dw[co][ci][k] += sum_pixels dy[co](p) x[ci](p + offset(k)),
// db[co] += sum dy[co].  A block takes LCI input channels (its lanes) x CGW * 4
// output channels (4 per warp) and walks TW x TH pixel tiles; a thread keeps the
// 4 x 9 sums of its channels in registers over all of them and, down a strip of
// 4 columns, the three input rows of the window, so that 144 FMAs take 6 new
// inputs and 4 x 4 gradients (the same for the warp: broadcast; staged with the
// output channel innermost, so that they come as pairs for the packed FMA).
// Where there are few channels the tile's strips are split instead: over the
// 8 / CGW warps of a channel group (few output channels), over the 32 / LCI
// lanes of an input channel (the network's two-channel input).
template <int TW_, int TH_, int CGW_, int LCI_> struct WgradTile
{
    static constexpr int TW = TW_, TH = TH_, CGW = CGW_, LCI = LCI_;
    static constexpr int CO = CGW * 4;
    static constexpr int PS = 8 / CGW, LS = 32 / LCI; // warps / lanes that share the pixels of a tile
    static constexpr int RS = TW + 8, ROWS = TH + 2;  // rows hold columns -4 .. TW + 3 of the tile
    // plane strides of 4 mod 32 words: 16-byte loads of lanes one channel apart
    // touch all banks
    static constexpr int XP = (ROWS * RS - 4 + 31) / 32 * 32 + 4;
    static constexpr int YS = CO + 4;                 // floats per pixel of the staged gradients
    static constexpr int XF = LCI * XP, YF = TW * TH * YS;
    static constexpr int NCOL = TW / kPX;             // strips of 4 columns
    static constexpr int SPLIT = PS * LS;
    static constexpr int BANDS = SPLIT > NCOL ? SPLIT / NCOL : 1, BH = TH / BANDS; // row bands of a strip
    static constexpr int RUN = LCI * 9;               // sums of one output channel in a block
    static constexpr size_t kStage = (size_t)2 * (XF + YF) * 4;
    static constexpr size_t kReduce = (size_t)8 * 4 * RUN * 4;
    static constexpr size_t kSmem = kStage > kReduce ? kStage : kReduce;
    static_assert(TH % BANDS == 0, "bands");
};

template <typename T>
__global__ void __launch_bounds__(kThreads, 2) k_conv3x3_wgrad_fma(const float *__restrict__ x,
                                                                   const float *__restrict__ dy, float *__restrict__ dw,
                                                                   float *__restrict__ db, int n, int cin, int cout,
                                                                   int h, int wd)
{
    extern __shared__ __align__(16) float smem[];
    const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nci = (cin + T::LCI - 1) / T::LCI;
    const int co0 = ((int)blockIdx.x / nci) * T::CO, ci0 = ((int)blockIdx.x % nci) * T::LCI;
    const int tiles_x = (wd + T::TW - 1) / T::TW, tiles_y = (h + T::TH - 1) / T::TH;
    const int tiles = tiles_x * tiles_y * n;
    const size_t plane = (size_t)h * wd;
    const int cw = warp % T::CGW, ps = warp / T::CGW, lci = lane % T::LCI, ls = lane / T::LCI;
    const bool xvec = (wd & 3) == 0 && ((uintptr_t)x & 15u) == 0;
    auto sx = [&](int st) { return smem + st * T::XF; };
    auto sy = [&](int st) { return smem + 2 * T::XF + st * T::YF; };
    auto stage = [&](int t, int st) {
        const int img = t / (tiles_x * tiles_y), r0 = t % (tiles_x * tiles_y);
        const int tx0 = (r0 % tiles_x) * T::TW, ty0 = (r0 / tiles_x) * T::TH;
        const float *xi = x + (size_t)img * cin * plane, *yi = dy + (size_t)img * cout * plane;
        if (xvec)
        {
            constexpr int NV = T::TW / 4 + 2;
            for (int i = tid; i < T::LCI * T::ROWS * NV; i += kThreads)
            {
                const int v = i % NV, r = i / NV, yy = r % T::ROWS, c = r / T::ROWS;
                const int gy = ty0 + yy - 1, gc = ci0 + c;
                const bool row = gc < cin && gy >= 0 && gy < h;
                const float *src = xi + (row ? (size_t)gc * plane + (size_t)gy * wd : 0);
                float *dst = sx(st) + c * T::XP + yy * T::RS;
                if (v < T::TW / 4)
                {
                    const bool ok = row && tx0 + 4 * v < wd;
                    copy16_async(dst + 4 + 4 * v, ok ? src + tx0 + 4 * v : x, ok);
                }
                else
                {
                    const int gx = v == T::TW / 4 ? tx0 - 1 : tx0 + T::TW;
                    const bool ok = row && gx >= 0 && gx < wd;
                    copy4_async(dst + (gx - tx0 + 4), ok ? src + gx : x, ok);
                }
            }
        }
        else
            for (int i = tid; i < T::LCI * T::ROWS * (T::TW + 2); i += kThreads)
            {
                const int v = i % (T::TW + 2), r = i / (T::TW + 2), yy = r % T::ROWS, c = r / T::ROWS;
                const int gx = tx0 + v - 1, gy = ty0 + yy - 1, gc = ci0 + c;
                const bool ok = gc < cin && gx >= 0 && gx < wd && gy >= 0 && gy < h;
                copy4_async(sx(st) + c * T::XP + yy * T::RS + 3 + v,
                            ok ? xi + (size_t)gc * plane + (size_t)gy * wd + gx : x, ok);
            }
        for (int i = tid; i < T::CO * T::TH * T::TW; i += kThreads)
        {
            const int xx = i % T::TW, r = i / T::TW, yy = r % T::TH, c = r / T::TH;
            const int gx = tx0 + xx, gy = ty0 + yy, gc = co0 + c;
            const bool ok = gc < cout && gx < wd && gy < h;
            copy4_async(sy(st) + (yy * T::TW + xx) * T::YS + c,
                        ok ? yi + (size_t)gc * plane + (size_t)gy * wd + gx : x, ok);
        }
        copies_commit();
    };

    uint64_t acc[2][9]; // pairs of output channels: sums since the last fold
    uint64_t sum[2][9]; // the folded sums
    // lane l: output channel l of the block, the warp's share of the pixels; a tile's
    // sum in FP32, the tiles' and the warps' in FP64, so that one rounded value per
    // block is added to db (one per warp, 2400 for 128^2 images, lost a third of a digit)
    double bsum = 0.0;
#pragma unroll
    for (int o = 0; o < 2; o++)
#pragma unroll
        for (int k = 0; k < 9; k++) acc[o][k] = sum[o][k] = 0;
    // sums of 64 pixels, added up: one chain of FP32 sums over all pixels of a block
    // was 1.4 times less exact on 8^2 to 32^2 pixels (error of dw against FP64) and
    // 2 to 4 % faster
    auto fold = [&]() {
#pragma unroll
        for (int o = 0; o < 2; o++)
#pragma unroll
            for (int k = 0; k < 9; k++)
            {
                add2(sum[o][k], acc[o][k]);
                acc[o][k] = 0;
            }
    };
    int t = (int)blockIdx.y, st = 0;
    if (t < tiles) stage(t, 0);
    copies_wait();
    __syncthreads();
    for (; t < tiles; t += (int)gridDim.y, st ^= 1)
    {
        if (t + (int)gridDim.y < tiles) stage(t + (int)gridDim.y, st ^ 1);
        const float *xp = sx(st) + lci * T::XP + 3;
        const float *yp = sy(st) + cw * 4;
        auto row = [&](const float *p, uint64_t v[6]) {
            const float4 a = *reinterpret_cast<const float4 *>(p + 1);
            v[0] = both(p[0]), v[1] = both(a.x), v[2] = both(a.y), v[3] = both(a.z), v[4] = both(a.w), v[5] = both(p[5]);
        };
        for (int s = ps * T::LS + ls; s < T::NCOL * T::BANDS; s += T::SPLIT)
        {
            const int x0 = (s % T::NCOL) * kPX, y0 = (s / T::NCOL) * T::BH;
            uint64_t xr[3][6]; // row y0 - 1 + j in xr[j % 3]
            row(xp + y0 * T::RS + x0, xr[0]);
            row(xp + (y0 + 1) * T::RS + x0, xr[1]);
#pragma unroll
            for (int j = 0; j < T::BH; j++)
            {
                row(xp + (y0 + j + 2) * T::RS + x0, xr[(j + 2) % 3]);
#pragma unroll
                for (int p = 0; p < kPX; p++)
                {
                    const ulonglong2 g = *reinterpret_cast<const ulonglong2 *>(yp + ((y0 + j) * T::TW + x0 + p) * T::YS);
#pragma unroll
                    for (int k = 0; k < 9; k++)
                    {
                        fma2(acc[0][k], g.x, xr[(j + k / 3) % 3][p + k % 3]);
                        fma2(acc[1][k], g.y, xr[(j + k / 3) % 3][p + k % 3]);
                    }
                }
            }
            if ((s / T::SPLIT) & 1) fold();
        }
        fold();
        if (db && ci0 == 0 && lane < T::CO)
        {
            float part = 0.f;
            for (int i = warp; i < T::TW * T::TH; i += 8) part += sy(st)[i * T::YS + lane];
            bsum += (double)part;
        }
        copies_wait();
        __syncthreads();
    }
    // sums of the lanes that share an input channel, then of the warps that
    // share output channels, in shared memory as [output channel][ci][k] (one
    // run of 9 LCI floats per output channel), added to dw in that order
    __shared__ double bred[8][T::CO];
    if (lane < T::CO) bred[warp][lane] = bsum;
    float *red = smem + warp * 4 * T::RUN;
#pragma unroll
    for (int o = 0; o < 4; o++)
#pragma unroll
        for (int k = 0; k < 9; k++)
        {
            float v = half_of(sum[o / 2][k], o & 1);
#pragma unroll
            for (int d = T::LCI; d < 32; d <<= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
            if (ls == 0) red[o * T::RUN + lci * 9 + k] = v;
        }
    __syncthreads();
    const int run = min(T::LCI, cin - ci0) * 9;
    for (int i = tid; i < T::CO * T::RUN; i += kThreads)
    {
        const int o = i / T::RUN, r = i % T::RUN, gco = co0 + o;
        if (gco >= cout || r >= run) continue;
        float v = 0.f;
#pragma unroll
        for (int s = 0; s < T::PS; s++) v += smem[((s * T::CGW + o / 4) * 4 + (o & 3)) * T::RUN + r];
        atomicAdd(&dw[((size_t)gco * cin + ci0) * 9 + r], v);
    }
    if (db && ci0 == 0 && tid < T::CO && co0 + tid < cout)
    {
        double v = 0.0;
#pragma unroll
        for (int k = 0; k < 8; k++) v += bred[k][tid];
        atomicAdd(&db[co0 + tid], (float)v);
    }
}
} // namespace cnn_fma
