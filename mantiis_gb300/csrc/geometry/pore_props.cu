// Local pore size and Knudsen number of a pore image on the GPU: the pipeline
// of Shape::calculateProperties (include/shape.hpp:127-251), kernel by kernel.
//
//   1. The image is padded by n columns on each side (void beside rows
//      1..n-2, include/shape.hpp:131-147) and thinned with the Zhang-Suen rule
//      of utils::thinning (include/utils.hpp:438-536).  Of the 3n x 3n padded
//      image only rows n-1..2n can ever be non-zero, so the kernels keep that
//      band of n+2 rows, bit-packed: bit k of word w of a row is column
//      32 w + k.  One thread evaluates the deletion rule for 32 pixels at
//      once with bitwise logic (the neighbour counts A and B come from a
//      bit-sliced adder over the eight neighbour masks).  Each sub-iteration
//      reads one buffer and writes the other, which is the reference's
//      "mark, then delete" order.  A launch runs 16 iterations (pairs of
//      sub-iterations) of each tile of the band in shared memory, the tile
//      with a halo of the 32 pixels that can reach it.  The loop stops after
//      the first iteration that deletes nothing, as the launches' change
//      flags tell; the extra iterations issued by then change nothing.
//   2. Exact Euclidean distance transforms (the float distance of the exact
//      integer squared distance) to the nearest solid pixel and to the
//      nearest skeleton pixel, in two separable passes: the vertical distance
//      to the nearest zero pixel of the column (from a bit mask of 32 rows per
//      word), then the row minimum of t^2 + g(j +- t)^2 scanned outwards from
//      the pixel until t^2 exceeds the best value found.
//   3. Per void pixel, the first skeleton pixel in raster order at the
//      skeleton distance (utils::distanceToNearestWallIndex,
//      include/utils.hpp:116-135, visited in O(D) by nearest_skeleton_at),
//      LocPore = 2 x its wall distance and Kn = mfp / LocPore / dx.
#include <cuda_runtime.h>
#include <sys/mman.h>
#include <unistd.h>

#include <cfloat>
#include <cstdint>
#include <stdexcept>
#include <string>

#include "../host/medial_search.hpp"
#include "pore_props.hpp"

namespace mantiis
{
namespace
{
struct GeomCudaError : std::runtime_error
{
    using std::runtime_error::runtime_error;
};

#define GK(call)                                                                                                       \
    do                                                                                                                 \
    {                                                                                                                  \
        cudaError_t e_ = (call);                                                                                       \
        if (e_ != cudaSuccess)                                                                                         \
            throw GeomCudaError(std::string(#call) + ": " + cudaGetErrorString(e_) + " (" + __FILE__ + ":" +         \
                                std::to_string(__LINE__) + ")");                                                       \
    } while (0)

template <typename T> struct GBuf
{
    T *p = nullptr;
    explicit GBuf(size_t n) { GK(cudaMalloc(&p, (n ? n : 1) * sizeof(T))); }
    ~GBuf() { cudaFree(p); }
    GBuf(const GBuf &) = delete;
    GBuf &operator=(const GBuf &) = delete;
};

constexpr int kThreads = 256;
// thinning iterations per launch, and launches issued between two reads of the
// change flags
constexpr int kChunk = 16, kLaunches = 8;

inline unsigned blocks_for(int64_t n) { return (unsigned)((n + kThreads - 1) / kThreads); }

// ---------------------------------------------------------------- thinning

// band row b (0..n+1) is padded row n-1+b, i.e. image row i = b-1; band
// column c (0..3n-1) is image column j = c-n.  Void image pixels, and the
// padding beside image rows 1..n-2, are 1.
__global__ void k_band_init(const int32_t *__restrict__ pore, uint32_t *__restrict__ band, int n, int wpr)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)(n + 2) * wpr) return;
    const int b = (int)(t / wpr), w = (int)(t % wpr);
    const int i = b - 1;
    uint32_t word = 0;
    if (i >= 0 && i < n)
    {
        const bool pad = i >= 1 && i <= n - 2;
        for (int k = 0; k < 32; k++)
        {
            const int c = 32 * w + k;
            if (c >= 3 * n) break;
            const int j = c - n;
            const bool v = (j >= 0 && j < n) ? pore[(int64_t)i * n + j] == 1 : pad;
            word |= (uint32_t)v << k;
        }
    }
    band[t] = word;
}

__device__ __forceinline__ uint32_t majority(uint32_t a, uint32_t b, uint32_t c) { return (a & b) | (c & (a ^ b)); }

// A row's words seen from its neighbours: c the word, e and w its pixels' right
// and left neighbours (bit k holds the neighbour of column 32 w + k).
struct RowWords
{
    uint32_t c, e, w;
    __device__ __forceinline__ void load(const uint32_t *at)
    {
        c = at[0];
        e = __funnelshift_r(c, at[1], 1);
        w = __funnelshift_l(at[-1], c, 1);
    }
};

// One Zhang-Suen sub-iteration (include/utils.hpp:438-514) of the 32 pixels P.c
// between the rows u and d: the deleted pixels.  A pixel is deleted when A == 1,
// 2 <= B <= 5 and both of the sub-iteration's triple products are zero.
// Every line is one or two three-input logic operations on 32 pixels.
__device__ __forceinline__ uint32_t thin_word(const RowWords &u, const RowWords &P, const RowWords &d, bool second)
{
    // A: 0 -> 1 transitions around the ring no, ne, ea, se, so, sw, we, nw.  Of two
    // adjacent steps a -> b -> c at most one is a transition, so four such pairs count them.
    const uint32_t x0 = (~u.c & u.e) | (~u.e & P.e), x1 = (~P.e & d.e) | (~d.e & d.c);
    const uint32_t x2 = (~d.c & d.w) | (~d.w & P.w), x3 = (~P.w & u.w) | (~u.w & u.c);
    const uint32_t none = ~(x0 | x1 | x2), one = (x0 ^ x1 ^ x2) & ~(x0 & x1 & x2);
    const uint32_t a_is_one = (x3 & none) | (~x3 & one);
    // B = b0 + 2 b1 + 4 b2 + 8 b3 of the eight neighbours, by full adders; b0 is not
    // needed, and 2 <= B <= 5 is ~b3 & (b1 ^ b2)
    const uint32_t s0 = u.c ^ u.e ^ P.e, c0 = majority(u.c, u.e, P.e);
    const uint32_t s1 = d.e ^ d.c ^ d.w, c1 = majority(d.e, d.c, d.w);
    const uint32_t s2 = P.w ^ u.w, c2 = P.w & u.w;
    const uint32_t c3 = majority(s0, s1, s2), t = c0 ^ c1 ^ c2, c4 = majority(c0, c1, c2);
    const uint32_t b1 = t ^ c3, b2 = c4 ^ (t & c3), b3 = c4 & t & c3;
    const uint32_t b_in_2_5 = ~b3 & (b1 ^ b2);
    const uint32_t m1 = second ? (u.c & P.e & P.w) : (u.c & P.e & d.c);
    const uint32_t m2 = second ? (u.c & d.c & P.w) : (P.e & d.c & P.w);
    return P.c & a_is_one & b_in_2_5 & ~(m1 | m2);
}

// kChunk iterations of one tile of kTileRows x kTileWords words, in shared memory
// with a halo of kHalo rows and one word (32 pixels): after s sub-iterations the
// outer s pixels of the halo are no longer the band's, the tile still is.  What
// is read beside the halo's words (the next row's end) is as wrong as that.
//
// A launch per sub-iteration took 3.6 us for a microsecond of work (1024 launches
// at n = 1024: 3.7 ms).  What bounds the tiles is their instructions, so a thread
// takes kStrip rows of a word column, each row loaded and shifted once, and the
// rule is 22 three-input operations (with 110 instructions a word and one word a
// thread: 50 us a launch at n = 1024, now 26; 32 launches, 0.83 ms).  44 rows are
// 144 tiles at n = 1024, one per SM; smaller tiles compute more halo, and shorter
// chunks pay their loads and launches more often.  Other n take the same tile (14 tiles at
// 300, 315 at 1500, 564 at 2048): the whole pipeline is 3.1, 4.3 and 4.2 times as fast
// there as with a launch per sub-iteration, 4.5 at 1024, 3.9 at 4096, 3.4 at 8192.  A tile is passed over where
// neither it nor its neighbours changed in the chunk before: it cannot change (a
// change elsewhere is at least a tile's height or width away, no less than the
// chunk's 32 sub-iterations), and dst holds its content already.
constexpr int kHalo = 2 * kChunk, kTileRows = 44, kTileWords = 16;
constexpr int kHaloRows = kTileRows + 2 * kHalo, kHaloWords = kTileWords + 2;
constexpr int kStrip = 2; // rows per thread
constexpr int kStrips = (kHaloRows - 2 + kStrip - 1) / kStrip;
constexpr int kTileThreads = (kStrips * kHaloWords + 31) / 32 * 32;
static_assert(kHalo <= 32 && kTileRows >= kHalo, "a change travels one pixel per sub-iteration");
static_assert(kTileThreads <= 1024, "one thread per strip");

__global__ void __launch_bounds__(kTileThreads) k_thin_tiles(const uint32_t *__restrict__ src, uint32_t *__restrict__ dst,
                                                             int n, int wpr, const uint8_t *__restrict__ was,
                                                             uint8_t *__restrict__ now, uint32_t *__restrict__ flags)
{
    constexpr int kWords = kHaloRows * kHaloWords;
    // a word before, and one and the last strip's missing rows after the tile
    __shared__ uint32_t buf[2][1 + kWords + (kStrip - 1) * kHaloWords + 1];
    __shared__ uint32_t s_changed;
    const int tx = (int)blockIdx.x, ty = (int)blockIdx.y, nx = (int)gridDim.x, ny = (int)gridDim.y;
    if (was)
    {
        bool any = false;
        for (int y = max(ty - 1, 0); y <= min(ty + 1, ny - 1); y++)
            for (int x = max(tx - 1, 0); x <= min(tx + 1, nx - 1); x++) any |= was[y * nx + x] != 0;
        if (!any)
        {
            if (threadIdx.x == 0) now[ty * nx + tx] = 0;
            return;
        }
    }
    // band rows 1..n are thinned; rows 0 and n + 1 and everything outside are zero
    const int row0 = 1 + ty * kTileRows - kHalo, word0 = tx * kTileWords - 1;
    for (int t = (int)threadIdx.x; t < (int)(sizeof(buf[0]) / sizeof(uint32_t)); t += kTileThreads)
    {
        const int k = t - 1, b = row0 + k / kHaloWords, w = word0 + k % kHaloWords;
        const bool in = k >= 0 && k < kWords && b >= 1 && b <= n && w >= 0 && w < wpr;
        buf[0][t] = in ? src[(int64_t)b * wpr + w] : 0u;
        buf[1][t] = buf[0][t]; // the first and last rows are not computed
    }
    if (threadIdx.x == 0) s_changed = 0u;
    const int x = (int)threadIdx.x % kHaloWords, y0 = 1 + (int)threadIdx.x / kHaloWords * kStrip;
    const int w = word0 + x, last = 3 * n - 1;
    // padded columns 0 and 3n-1 are never examined by the reference's raster loop
    uint32_t keep = 0u;
    if (w == 0) keep |= 1u;
    if (w == last / 32) keep |= 1u << (last % 32);
    const bool own_word = x >= 1 && x <= kTileWords;
    __syncthreads();
    uint32_t changed = 0; // bit k: this thread deleted a pixel of the tile in iteration k
    auto sub_iteration = [&](const uint32_t *in, uint32_t *out, bool second, int s) {
        // rows s + 1 .. kHaloRows - s - 2 have neighbours that are still the band's
        if (y0 + kStrip > s + 1 && y0 < kHaloRows - s - 1 && y0 < kHaloRows - 1)
        {
            const uint32_t *at = in + 1 + (y0 - 1) * kHaloWords + x;
            RowWords r[3];
            r[0].load(at);
            r[1].load(at + kHaloWords);
#pragma unroll
            for (int k = 0; k < kStrip; k++)
            {
                r[(k + 2) % 3].load(at + (k + 2) * kHaloWords);
                const RowWords &P = r[(k + 1) % 3];
                const uint32_t del = thin_word(r[k % 3], P, r[(k + 2) % 3], second) & ~keep;
                const int y = y0 + k;
                if (y < kHaloRows - 1) out[1 + y * kHaloWords + x] = P.c & ~del;
                if (del && own_word && y >= kHalo && y < kHalo + kTileRows) changed |= 1u << (s >> 1);
            }
        }
        __syncthreads();
    };
    for (int s = 0; s < 2 * kChunk; s += 2)
    {
        sub_iteration(buf[0], buf[1], false, s);
        sub_iteration(buf[1], buf[0], true, s + 1);
    }
    for (int t = (int)threadIdx.x; t < kTileRows * kTileWords; t += kTileThreads)
    {
        const int y = t / kTileWords, tw = t % kTileWords;
        const int b = row0 + kHalo + y, bw = word0 + 1 + tw;
        if (b <= n && bw < wpr) dst[(int64_t)b * wpr + bw] = buf[0][1 + (kHalo + y) * kHaloWords + 1 + tw];
    }
    changed = __reduce_or_sync(0xffffffffu, changed);
    if ((threadIdx.x & 31) == 0 && changed) atomicOr(&s_changed, changed);
    __syncthreads();
    if (threadIdx.x == 0)
    {
        now[ty * nx + tx] = s_changed != 0u;
        if (s_changed) atomicOr(flags, s_changed);
    }
}

// skeleton of the image: the band's image columns n..2n-1 of rows 1..n
struct BandSkeleton
{
    const uint32_t *band;
    int n, wpr;
    __device__ __forceinline__ bool at(int i, int j) const
    {
        const int c = j + n;
        return (band[(int64_t)(i + 1) * wpr + c / 32] >> (c % 32)) & 1u;
    }
    __device__ __forceinline__ bool operator[](int64_t k) const { return at((int)(k / n), (int)(k % n)); }
};

// ---------------------------------------------------------- distance transform

// Zero pixels of the two transforms, bit k of word (b, j) row 32 b + k of column
// j.  SKELETON false: zero image pixels (distance to the nearest solid pixel,
// include/shape.hpp:183-196); true: skeleton pixels (distance to the skeleton,
// :198-212).
template <bool SKELETON>
__global__ void k_zero_bits(const int32_t *__restrict__ pore, BandSkeleton skel, uint32_t *__restrict__ zero, int n)
{
    const int j = (int)(blockIdx.x * blockDim.x + threadIdx.x), b = (int)blockIdx.y;
    if (j >= n) return;
    uint32_t m = 0;
    for (int k = 0; k < 32 && 32 * b + k < n; k++)
    {
        const int i = 32 * b + k;
        m |= (uint32_t)(SKELETON ? skel.at(i, j) : pore[(int64_t)i * n + j] == 0) << k;
    }
    zero[(int64_t)b * n + j] = m;
}

// vertical distance to the nearest zero pixel of the column, -1 if none
__global__ void k_edt_columns(const uint32_t *__restrict__ zero, int32_t *__restrict__ g, int n)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)n * n) return;
    const int i = (int)(t / n), j = (int)(t % n), nb = (n + 31) / 32, k = i & 31;
    int best = INT32_MAX;
    uint32_t m = zero[(int64_t)(i >> 5) * n + j];
    uint32_t up = m & (0xFFFFFFFFu >> (31 - k)), down = m >> k; // rows up to i, rows from i on
    if (down) best = __ffs((int)down) - 1;
    if (up) best = min(best, k - (31 - __clz((int)up)));
    for (int b = (i >> 5) - 1; !up && b >= 0 && i - (32 * b + 31) < best; b--)
    {
        up = zero[(int64_t)b * n + j];
        if (up) best = min(best, i - (32 * b + 31 - __clz((int)up)));
    }
    for (int b = (i >> 5) + 1; !down && b < nb && 32 * b - i < best; b++)
    {
        down = zero[(int64_t)b * n + j];
        if (down) best = min(best, 32 * b + __ffs((int)down) - 1 - i);
    }
    g[t] = best == INT32_MAX ? -1 : best;
}

// exact squared distance = min over columns c of (j - c)^2 + g(c)^2, scanned
// outwards from j until (j - c)^2 reaches the best value; INT32_MAX where the
// image has no zero pixel (sides are at most 16384: sums stay below 2^30)
__global__ void k_edt_rows(const int32_t *__restrict__ g, int32_t *__restrict__ out, int n)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)n * n) return;
    const int i = (int)(t / n), j = (int)(t % n);
    const int32_t *row = g + (int64_t)i * n;
    const int32_t none = INT32_MAX;
    int32_t best = row[j] >= 0 ? row[j] * row[j] : none;
    for (int s = 1; s < n; s++)
    {
        const int32_t s2 = s * s;
        if (s2 >= best) break;
        const bool left = j - s >= 0, right = j + s < n;
        if (!left && !right) break;
        const int32_t a = left ? row[j - s] : -1, b = right ? row[j + s] : -1;
        if (a >= 0) best = min(best, s2 + a * a);
        if (b >= 0) best = min(best, s2 + b * b);
    }
    out[t] = best;
}

// ------------------------------------------------------------ local pore size

// float distance: sqrtf of the exact integer, the float maximum where there is none
__device__ __forceinline__ float edt_distance(int32_t s) { return s == INT32_MAX ? FLT_MAX : sqrtf((float)s); }

__global__ void k_local_pore(const int32_t *__restrict__ pore, BandSkeleton skel, const int32_t *__restrict__ wall,
                             const int32_t *__restrict__ medial, double *__restrict__ locpore, double *__restrict__ kn,
                             int n, double dx, double mfp)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)n * n) return;
    if (pore[t] != 1)
    {
        locpore[t] = 0.0;
        kn[t] = 0.0;
        return;
    }
    const int i = (int)(t / n), j = (int)(t % n);
    const int32_t s = medial[t];
    const int64_t hit = s <= kExactSquares ? nearest_skeleton_at_square(skel, n, i, j, s)
                                           : nearest_skeleton_at(skel, n, i, j, (double)edt_distance(s));
    const double mid = (double)edt_distance(wall[hit >= 0 ? hit : t]);
    const double lp = 2.0 * mid;
    locpore[t] = lp;
    kn[t] = mfp / lp / dx;
}
} // namespace

// The outputs are often fresh memory, whose pages the system gives out (and
// clears) at the first write: that is done while the kernels run, not by the copy
// that they end with.  The system is asked for the pages, nothing is written here:
// the outputs keep their content until the results arrive, and memory that it does
// not manage (outputs on the GPU, pinned ones) is left alone.
static void populate_pages(void *p, size_t bytes)
{
#ifdef MADV_POPULATE_WRITE
    const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE), first = ((uintptr_t)p + page - 1) / page * page,
                    end = ((uintptr_t)p + bytes) / page * page;
    if (first < end)
        (void)madvise(reinterpret_cast<void *>(first), end - first, MADV_POPULATE_WRITE); // refused: the copy does it
#else
    (void)p;
    (void)bytes;
#endif
}

void gpu_pore_properties(const int32_t *pore, int n, double dx, double mfp, double *locpore, double *kn,
                         int64_t *iterations, cudaStream_t stream)
{
    if (!pore || !locpore || !kn) throw std::invalid_argument("gpu_pore_properties: null argument");
    if (n <= 3 || n > kMaxPorePropsSide)
        throw std::invalid_argument("gpu_pore_properties: image side must be in 4.." +
                                    std::to_string(kMaxPorePropsSide));
    const int64_t nn = (int64_t)n * n;
    const int wpr = (3 * n + 31) / 32, nb = (n + 31) / 32;
    const int64_t band_words = (int64_t)(n + 2) * wpr;
    const dim3 tiles((unsigned)((wpr + kTileWords - 1) / kTileWords), (unsigned)((n + kTileRows - 1) / kTileRows));
    const int64_t ntiles = (int64_t)tiles.x * tiles.y;
    // one allocation for every buffer (each on 256 bytes)
    size_t total = 0;
    auto place = [&](size_t bytes) {
        const size_t at = total;
        total += (bytes + 255) / 256 * 256;
        return at;
    };
    const size_t o_lp = place(nn * sizeof(double)), o_kn = place(nn * sizeof(double)), o_pore = place(nn * 4),
                 o_g = place(nn * 4), o_wall = place(nn * 4), o_medial = place(nn * 4), o_a = place(band_words * 4),
                 o_b = place(band_words * 4), o_zero = place((size_t)nb * n * 4), o_flags = place(kLaunches * 4),
                 o_was = place(ntiles), o_now = place(ntiles);
    GBuf<unsigned char> mem(total);
    auto at = [&](size_t o) { return static_cast<void *>(mem.p + o); };
    double *d_lp = static_cast<double *>(at(o_lp)), *d_kn = static_cast<double *>(at(o_kn));
    int32_t *d_pore = static_cast<int32_t *>(at(o_pore)), *d_g = static_cast<int32_t *>(at(o_g)),
            *d_wall = static_cast<int32_t *>(at(o_wall)), *d_medial = static_cast<int32_t *>(at(o_medial));
    uint32_t *band[2] = {static_cast<uint32_t *>(at(o_a)), static_cast<uint32_t *>(at(o_b))};
    uint32_t *d_zero = static_cast<uint32_t *>(at(o_zero)), *flags = static_cast<uint32_t *>(at(o_flags));
    uint8_t *changed[2] = {static_cast<uint8_t *>(at(o_was)), static_cast<uint8_t *>(at(o_now))};
    GK(cudaMemcpyAsync(d_pore, pore, nn * sizeof(int32_t), cudaMemcpyHostToDevice, stream));

    k_band_init<<<blocks_for(band_words), kThreads, 0, stream>>>(d_pore, band[0], n, wpr);
    GK(cudaGetLastError());
    // each iteration deletes at least one pixel of the band or ends the loop
    const int64_t max_iterations = (int64_t)(n + 2) * 3 * n + kChunk * kLaunches;
    int64_t done = 0, converged_at = -1;
    int cur = 0; // the band's current buffer
    bool first = true;
    while (converged_at < 0)
    {
        if (done > max_iterations) throw std::runtime_error("gpu_pore_properties: thinning did not converge");
        GK(cudaMemsetAsync(flags, 0, kLaunches * sizeof(uint32_t), stream));
        for (int k = 0; k < kLaunches; k++, cur ^= 1, first = false)
            k_thin_tiles<<<tiles, kTileThreads, 0, stream>>>(band[cur], band[cur ^ 1], n, wpr,
                                                             first ? nullptr : changed[cur ^ 1], changed[cur], flags + k);
        GK(cudaGetLastError());
        if (done == 0)
        {
            populate_pages(locpore, nn * sizeof(double));
            populate_pages(kn, nn * sizeof(double));
        }
        uint32_t host_flags[kLaunches];
        GK(cudaMemcpyAsync(host_flags, flags, sizeof(host_flags), cudaMemcpyDeviceToHost, stream));
        GK(cudaStreamSynchronize(stream));
        for (int k = 0; k < kLaunches * kChunk && converged_at < 0; k++)
            if (!((host_flags[k / kChunk] >> (k % kChunk)) & 1u)) converged_at = done + k + 1;
        done += kLaunches * kChunk;
    }
    if (iterations) *iterations = converged_at;

    const unsigned gp = blocks_for(nn);
    const BandSkeleton skel{band[cur], n, wpr};
    const dim3 gz(blocks_for(n), (unsigned)nb);
    for (int mode = 0; mode < 2; mode++)
    {
        if (mode == 0) k_zero_bits<false><<<gz, kThreads, 0, stream>>>(d_pore, skel, d_zero, n);
        else k_zero_bits<true><<<gz, kThreads, 0, stream>>>(d_pore, skel, d_zero, n);
        k_edt_columns<<<gp, kThreads, 0, stream>>>(d_zero, d_g, n);
        k_edt_rows<<<gp, kThreads, 0, stream>>>(d_g, mode == 0 ? d_wall : d_medial, n);
    }
    k_local_pore<<<gp, kThreads, 0, stream>>>(d_pore, skel, d_wall, d_medial, d_lp, d_kn, n, dx, mfp);
    GK(cudaGetLastError());
    GK(cudaMemcpyAsync(locpore, d_lp, nn * sizeof(double), cudaMemcpyDeviceToHost, stream));
    GK(cudaMemcpyAsync(kn, d_kn, nn * sizeof(double), cudaMemcpyDeviceToHost, stream));
    GK(cudaStreamSynchronize(stream));
}

bool is_geometry_cuda_error(const std::exception &e) { return dynamic_cast<const GeomCudaError *>(&e) != nullptr; }
} // namespace mantiis
